"""tq_clear_walls on grids whose mask has less than one point a thread of a launch's round of blocks, as many, one row more,
and several a thread: the mask of an empty tank and its wall cells, bit for bit as the package's Cena makes them."""
import numpy as np
import pytest

from tanque import Cena, SimulacaoGPU

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(3, 3), (31, 17), (296, 256), (297, 256), (1501, 600)], ids=str)
def test_limpar_paredes(lib_gpu, nx, ny):
    h = 0.01
    g = SimulacaoGPU(Cena(nx, ny, h), {"capacity": 64})
    g.tracarParede(0.1 * nx * h, 0.2 * ny * h, 0.9 * nx * h, 0.7 * ny * h, 2 * h)
    g.limparParedes()
    vazio = np.asarray(Cena(nx, ny, h).sdf, np.float32)
    assert np.array_equal(g.campo("sdf").view(np.uint32), vazio.view(np.uint32))
    m = vazio.astype(np.float64).reshape(ny, 2, nx, 2).sum(axis=(1, 3))
    assert np.array_equal(g.campo("solidoCelula"), (m < 0).astype(np.uint8).ravel())
    g.fechar()
