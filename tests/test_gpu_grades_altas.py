"""A grid of more than 65,535 rows of 32 cells, the surface's tiles (a launch's limit on its second dimension): a
substep's surface fields and right-hand side around some water at its bottom and at its top are those of a
short grid, bit for bit."""
import numpy as np
import pytest

from tanque import Cena, SimulacaoGPU
from tanque.constantes import CAMPOS

pytestmark = pytest.mark.gpu


def test_superficie(lib_gpu):
    nx, baixo, h = 4, 512, 2.0**-6  # (a power of two: positions two million rows up are exact)
    alto = baixo + 32 * 65_536
    campos = {}
    for ny in (baixo, alto):
        cena = Cena(nx, ny, h)
        cena.sdf[:] = 3.0  # no wall
        sim = SimulacaoGPU(cena, {"air": 0, "iterations": 1, "capacity": 4096, "gravity": (0.0, 0.0)})
        agua = np.zeros((4 * nx * 20, CAMPOS), np.float32)
        q = np.arange(4 * nx * 20)
        i, j, s = q // 4 % nx, q // (4 * nx), q % 4
        x, y = i + 0.25 + 0.5 * (s & 1), j + 0.25 + 0.5 * (s >> 1)
        agua[:, 0], agua[:, 1] = x * h, (y + 30) * h
        topo = agua.copy()
        topo[:, 1] = (y + ny - 60) * h
        sim.definirParticulas(np.concatenate([agua, topo]).ravel())
        sim.subpasso(1e-4)
        campos[ny] = {}
        for c in ["tipo", "fase", "normalY", "curvatura", "div"]:
            f = sim.campo(c).reshape(ny, nx)
            campos[ny][c] = np.stack([f[:200], f[-200:]])
        sim.fechar()
    for c in campos[baixo]:
        assert np.any(campos[baixo][c][0]) and np.any(campos[baixo][c][1]), c
        assert np.array_equal(campos[alto][c], campos[baixo][c]), c
