"""The plain solve's first kernel counts the bubbles' cells a warp at a time: bubbles that end inside a warp, several in
one warp beside water, and in the last, incomplete warp of the grid, with the V-cycle seeing them.  Three iterations
against the oracle: q to 1e-4, norms and bubble pressures to 1e-3 (the bounds of the fixed-count solves)."""
import numpy as np
import pytest

from estado import erro_relativo
from oraculo import carregar_oraculo
from tanque import resolver_pressao
from tanque.constantes import AGUA, AR, SOLIDO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(7, 5), (13, 9), (33, 31), (37, 23), (64, 40), (1001, 303)], ids=str)
def test_celulas_das_bolhas(lib_gpu, nx, ny):
    rng = np.random.default_rng(nx * ny)
    tipo = np.full((ny, nx), AGUA, np.uint8)
    tipo[0] = tipo[:, 0] = tipo[:, -1] = SOLIDO
    tipo[-1] = AR  # free surface
    rotulo = np.zeros((ny, nx), np.uint32)
    # bubbles of 1 x 1 to 3 x 2 cells all over the grid, and the last cells of the grid
    for b in range(2, 2 + max(3, nx * ny // 40)):
        i, j = int(rng.integers(1, nx - 1)), int(rng.integers(1, ny - 1))
        w, h = int(rng.integers(1, 4)), int(rng.integers(1, 3))
        livre = tipo[j:j + h, i:min(i + w, nx - 1)] == AGUA
        tipo[j:j + h, i:min(i + w, nx - 1)][livre] = AR
        rotulo[j:j + h, i:min(i + w, nx - 1)][livre] = min(b, 4095)
    rotulo[-1, -3:] = 2
    div = np.where(tipo == AGUA, 0.1 * rng.standard_normal((ny, nx)), 0).astype(np.float32)
    rhs = (0.05 * rng.standard_normal(4096)).astype(np.float32)
    saidas = []
    for lig in (None, carregar_oraculo()):
        q = np.zeros((ny, nx), np.float32)
        bolhas = {"rotulo": rotulo, "rhs": rhs, "y": np.zeros(4096, np.float32)}
        normas = resolver_pressao(tipo, div, q, 3, 0.0, bolhas, ligacao=lig)
        saidas.append((q, bolhas["y"], normas))
    (qg, yg, ng), (qo, yo, no) = saidas
    assert erro_relativo(qg, qo) < 1e-4
    assert erro_relativo(yg, yo) < 1e-3
    assert erro_relativo(ng, no) < 1e-3
