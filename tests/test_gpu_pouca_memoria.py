"""A fused-engine handle where the device has room for the plain engine's arrays alone: it is made, and steps as the
plain engine does, bit for bit."""
import numpy as np
import pytest

from tanque import Cena, SimulacaoGPU, _abi
from tanque.cenarios import semear_retangulo_rapido

pytestmark = pytest.mark.gpu


def test_motor_simples_no_lugar_do_fundido(lib_gpu):
    import torch
    nx, ny, h = 3000, 2000, 0.01
    cena = Cena(nx, ny, h)
    agua = semear_retangulo_rapido(2 * h, 2 * h, 40 * h, 30 * h, h, s=5)

    def passo(sim):
        sim.adicionar(agua, False)
        sim.subpasso(1 / 480)
        return {c: sim.campo(c) for c in ("tipo", "q", "u", "v")}

    livre, uso = lambda: torch.cuda.mem_get_info()[0], {}
    for motor in (_abi.TQ_ENGINE_PLAIN, _abi.TQ_ENGINE_FUSED):
        antes = livre()
        sim = SimulacaoGPU(cena, {"engine": motor, "capacity": 65536})
        uso[motor] = antes - livre()
        if motor == _abi.TQ_ENGINE_PLAIN:
            certo = passo(sim)
        sim.fechar()
    simples, fundido = uso[_abi.TQ_ENGINE_PLAIN], uso[_abi.TQ_ENGINE_FUSED]
    assert fundido - simples > 64 << 20
    cheio = torch.empty(livre() - (simples + fundido) // 2, dtype=torch.uint8, device="cuda")
    try:
        sim = SimulacaoGPU(cena, {"engine": _abi.TQ_ENGINE_FUSED, "capacity": 65536})
        campos = passo(sim)
        sim.fechar()
    finally:
        del cheio
        torch.cuda.empty_cache()
    for c in certo:
        assert np.array_equal(campos[c], certo[c]), c
