"""The labels' propagation with many cells pending: no label known, a few seeds, one cell in ten labelled, and
chains along walls, on lists below, at and above the block's 1,024 cells, against the oracle bit for bit."""
import numpy as np
import pytest

from oraculo import CenaOraculo, SimulacaoOraculo
from tanque import Cena, SimulacaoGPU, _abi
from tanque.cenarios import semear_retangulo_rapido

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sementes", [0.0, 0.001, 0.1])
@pytest.mark.parametrize("nx,ny", [(12, 9), (36, 36), (40, 37), (161, 77), (300, 200)], ids=str)
def test_propagacao(lib_gpu, nx, ny, sementes):
    h = 0.01
    cena_o, cena_g = CenaOraculo(nx, ny, h), Cena(nx, ny, h)
    for c in (cena_o, cena_g):
        c.tracar(0.4 * nx * h, 0.5 * ny * h, 0.4 * nx * h, 0.85 * ny * h, 0.8 * h)
        c.tracar(0.4 * nx * h, 0.85 * ny * h, 0.8 * nx * h, 0.85 * ny * h, 0.8 * h)
    cena_g.sdf[:] = cena_o.sdf
    o, g = SimulacaoOraculo(cena_o, {"p2g_mode": _abi.TQ_P2G_FIXED}), SimulacaoGPU(cena_g, {})
    agua = semear_retangulo_rapido(2 * h, 2 * h, 0.6 * nx * h, 0.4 * ny * h, h, s=5)
    rng = np.random.default_rng(nx)
    rot = np.where(rng.random(nx * ny) < sementes, rng.integers(1, 40, nx * ny), 0).astype(np.uint32)
    for s in (o, g):
        s.definirParticulas(agua)
        s.definirCampo("rotulo", rot)
    for passo in range(3):
        for s in (o, g):
            s.subpasso(1 / 480)
        for campo in ["tipo", "rotulo"]:
            assert np.array_equal(g.campo(campo), o.campo(campo)), f"{passo}: {campo}"
        o.definirParticulas(g.p)
