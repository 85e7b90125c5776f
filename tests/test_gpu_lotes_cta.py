"""The fused solver's [DA] and [B] with few CTAs, each taking its cells in several batches (of 4 x 384 cells a
CTA): one cell less than whole batches, whole batches, one row more, and tens of them, with bubbles and
dry batches.  Three iterations of a substep against the oracle's: integers bit-exact, q, u and v to 1e-4,
bubble pressures to 1e-3 (the bounds of the fixed-count substeps)."""
import numpy as np
import pytest

from estado import INTEIROS, copiar_estado, erro_relativo
from oraculo import CenaOraculo, SimulacaoOraculo
from tanque import Cena, SimulacaoGPU, _abi
from tanque.cenarios import semear_retangulo_rapido
from tanque.constantes import CAMPOS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", [_abi.TQ_PRECOND_REFERENCE, _abi.TQ_PRECOND_BLOCK_1], ids=["ref", "bloco1"])
@pytest.mark.parametrize("nx,ny,ctas", [(96, 48, 1), (95, 97, 2), (96, 96, 2), (96, 97, 2), (307, 45, 3), (320, 241, 1),
                                        (322, 203, 7)], ids=str)
def test_lotes(lib_gpu, nx, ny, ctas, precond):
    h = 0.01
    opc = {"preconditioner": precond, "iterations": 3}
    cena_o, cena_g = CenaOraculo(nx, ny, h), Cena(nx, ny, h)
    for c in (cena_o, cena_g):
        c.tracar(0.3 * nx * h, 0.2 * ny * h, 0.3 * nx * h, 0.5 * ny * h, 0.6 * h)
    cena_g.sdf[:] = cena_o.sdf
    o = SimulacaoOraculo(cena_o, dict(opc, p2g_mode=_abi.TQ_P2G_FIXED))
    g = SimulacaoGPU(cena_g, dict(opc, engine=_abi.TQ_ENGINE_FUSED, fused_ctas=ctas))
    agua = semear_retangulo_rapido(2 * h, 2 * h, (nx - 2) * h, 0.6 * ny * h, h, s=5).reshape(-1, CAMPOS)
    x, y = agua[:, 0] / (nx * h), agua[:, 1] / (ny * h)
    agua[:, 2] = 0.3 * np.sin(9 * y)
    agua[:, 3] = 0.2 * np.cos(7 * x)
    fora = np.zeros(len(agua), bool)
    for cx, cy, r in [(0.15, 0.3, 0.08), (0.5, 0.25, 0.1), (0.8, 0.4, 0.05)]:  # trapped air
        fora |= (x - cx) ** 2 + (y - cy) ** 2 < r * r
    agua = np.ascontiguousarray(agua[~fora])
    for s in (o, g):
        s.adicionar(agua.ravel(), False)
    for quadro in range(2):
        copiar_estado(o, g)
        for s in (o, g):
            s.avancar(1 / 240, 1)
        for campo in INTEIROS:
            assert np.array_equal(g.campo(campo), o.campo(campo)), f"{quadro}: {campo}"
        assert np.any(o.campo("rotulo") >= 2)
        for campo, tol in {"q": 1e-4, "u": 1e-4, "v": 1e-4, "pressaoBolha": 1e-3}.items():
            e = erro_relativo(g.campo(campo), o.campo(campo))
            assert e <= tol, f"{quadro}: {campo} relative error {e:.3g} > {tol}"
