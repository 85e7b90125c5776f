"""The velocity extrapolation's two layers around scattered drops: faces one, two and more steps from water, at
the grid's edges and corners, on grids from 3x3 cells on, with the tank's frame and without any wall, against
the oracle: cell flags and the faces' valid flags bit-exact, u and v to 1e-4 (the substep's parity bound)."""
import numpy as np
import pytest

from estado import erro_relativo
from oraculo import SimulacaoOraculo
from tanque import Cena, SimulacaoGPU, _abi
from tanque.constantes import CAMPOS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("paredes", [True, False], ids=["moldura", "aberto"])
@pytest.mark.parametrize("nx,ny", [(3, 3), (4, 7), (9, 5), (16, 16), (33, 31), (130, 70), (257, 64)], ids=str)
def test_camadas(lib_gpu, nx, ny, paredes):
    h = 0.01
    cena = Cena(nx, ny, h)
    if not paredes:
        cena.sdf[:] = 3.0
    rng = np.random.default_rng(nx * ny)
    celulas = rng.random((ny, nx)) < 0.05
    if not paredes:  # the corners too
        celulas[0, 0] = celulas[-1, -1] = True
    j, i = np.nonzero(celulas)
    agua = np.zeros((4 * len(i), CAMPOS), np.float32)
    dx, dy = np.tile([0.25, 0.75, 0.25, 0.75], len(i)), np.tile([0.25, 0.25, 0.75, 0.75], len(i))
    agua[:, 0], agua[:, 1] = (np.repeat(i, 4) + dx) * h, (np.repeat(j, 4) + dy) * h
    agua[:, 2:4] = 0.2 * rng.standard_normal((len(agua), 2))
    opc = {"air": 0, "gravity": (0.0, 0.0)}
    o, g = SimulacaoOraculo(cena, dict(opc, p2g_mode=_abi.TQ_P2G_FIXED)), SimulacaoGPU(cena, dict(opc))
    for s in (o, g):
        s.definirParticulas(agua.ravel())
        s.subpasso(1 / 480)
    for campo in ["tipo", "uValida", "vValida"]:
        assert np.array_equal(g.campo(campo), o.campo(campo)), campo
    for campo in ["u", "v"]:
        e = erro_relativo(g.campo(campo), o.campo(campo))
        assert e <= 1e-4, f"{campo} relative error {e:.3g}"
