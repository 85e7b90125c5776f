"""The right-hand side kernel where a thread takes several cells: one round of 888 blocks of 256 threads
exactly, one column more, and several rounds, with walls and trapped air, against the oracle: cell flags,
labels, bubble volumes bit-exact; div to 1e-5, qAr to 1e-4 (the bounds of the substep's parity tests), the
bubbles' right-hand sides to 1e-4 of the FP64 oracle's (its FP32 build rounds a large bubble's sum at each of
thousands of cells; the terms' velocities and volumes are exact, and qAr to 1e-4)."""
import numpy as np
import pytest

from estado import copiar_estado, erro_relativo
from oraculo import CenaOraculo, SimulacaoOraculo
from tanque import Cena, SimulacaoGPU, _abi
from tanque.cenarios import semear_retangulo_rapido
from tanque.constantes import CAMPOS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ar", [True, False], ids=["ar", "sem-ar"])
@pytest.mark.parametrize("nx,ny", [(592, 384), (593, 384), (1010, 470)], ids=str)
def test_lado_direito(lib_gpu, nx, ny, ar):
    h = 0.01
    cena_o, cena_g = CenaOraculo(nx, ny, h), Cena(nx, ny, h)
    for c in (cena_o, cena_g):
        c.tracar(0.3 * nx * h, 0.3 * ny * h, 0.3 * nx * h, 0.5 * ny * h, 0.6 * h)
        c.tracar(0.75 * nx * h, 0.1 * ny * h, 0.75 * nx * h, 0.3 * ny * h, 5 * h)
    cena_g.sdf[:] = cena_o.sdf
    opc = {"air": int(ar)}
    o, g = SimulacaoOraculo(cena_o, dict(opc, p2g_mode=_abi.TQ_P2G_FIXED)), SimulacaoGPU(cena_g, dict(opc))
    agua = semear_retangulo_rapido(2 * h, 2 * h, (nx - 2) * h, 0.6 * ny * h, h, s=5).reshape(-1, CAMPOS)
    x, y = agua[:, 0] / (nx * h), agua[:, 1] / (ny * h)
    agua[:, 2] = 0.3 * np.sin(9 * y)
    agua[:, 3] = 0.2 * np.cos(7 * x)
    agua = np.ascontiguousarray(agua[((x - 0.5) ** 2 + (y - 0.25) ** 2 > 0.01) & ((x - 0.15) ** 2 + (y - 0.4) ** 2 > 0.001)])
    for s in (o, g):
        s.adicionar(agua.ravel(), False)
    for s in (o, g):
        s.atualizarAr()
    copiar_estado(o, g)
    d = SimulacaoOraculo(cena_o, dict(opc, p2g_mode=_abi.TQ_P2G_FIXED), fp64=True)
    copiar_estado(o, d)
    for s in (o, g, d):
        s.avancar(1 / 240, 1)
    for campo in ["tipo", "rotulo", "volumeBolha"]:
        assert np.array_equal(g.campo(campo), o.campo(campo)), campo
    assert not ar or np.count_nonzero(o.campo("volumeBolha")) >= 2
    for campo, ref, tol in [("div", o, 1e-5), ("qAr", o, 1e-4), ("rhsBolha", d, 1e-4)]:
        e = erro_relativo(g.campo(campo), ref.campo(campo))
        assert e <= tol, f"{campo} relative error {e:.3g} > {tol}"
