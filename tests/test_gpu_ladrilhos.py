"""The V-cycle's level legs on tiles (tq_vcycle) at the sizes where a tile, a block or the coarse section
ends, against the oracle's cicloV: FP32 to 2e-5 relative (the bound of the V-cycle's other tests).  The
right side is NaN off water: a caller's values there must not reach the result."""
import numpy as np
import pytest

from estado import erro_relativo
from oraculo import carregar_oraculo
from tanque import ciclo_v, resolver_pressao
from tanque.constantes import AGUA, AR, SOLIDO

pytestmark = pytest.mark.gpu

TAMANHOS = [(3, 3), (13, 13), (16, 16), (17, 31), (32, 32), (33, 33), (64, 64), (65, 129), (129, 48), (300, 14),
            (2100, 14), (500, 333), (1030, 770)]


@pytest.mark.parametrize("fundo", ["paredes-soltas", "agua-parada"])
@pytest.mark.parametrize("nx,ny", TAMANHOS, ids=str)
def test_legs(lib_gpu, nx, ny, fundo):
    rng = np.random.default_rng(nx * ny)
    tipo = np.full((ny, nx), AGUA, np.uint8)
    if fundo == "paredes-soltas":
        tipo[rng.random((ny, nx)) < 0.08] = SOLIDO
        tipo[: ny // 6] = AR
    else:  # a tank's frame, still water to 60 %, a wall in it
        tipo[int(ny * 0.6):] = AR
        tipo[ny // 4: ny // 4 + 3, nx // 5: nx // 2] = SOLIDO
        if min(nx, ny) > 4:
            tipo[:2] = tipo[-2:] = SOLIDO
            tipo[:, :2] = tipo[:, -2:] = SOLIDO
    b = rng.standard_normal((ny, nx)).astype(np.float32)
    ref = ciclo_v(tipo, np.where(tipo == AGUA, b, 0).astype(np.float32), ligacao=carregar_oraculo())
    b[tipo != AGUA] = np.nan
    x = ciclo_v(tipo, b)
    assert np.all(np.isfinite(x))
    assert erro_relativo(x, ref) < 2e-5


@pytest.mark.parametrize("nx,ny", [(40, 9), (13, 13), (33, 47), (257, 65), (700, 520)], ids=str)
def test_pcg_com_bolhas(lib_gpu, nx, ny):
    """The plain engine's three kernels an iteration on one level, at block edges and with several cells a
    thread, bubbles of one cell to many: q to 1e-4, norms and bubble pressures to 1e-3 of the oracle's
    (the bounds of the fixed-count solves)."""
    rng = np.random.default_rng(nx + ny)
    tipo = np.full((ny, nx), AGUA, np.uint8)
    tipo[int(ny * 0.75):] = AR
    tipo[0] = tipo[-1] = SOLIDO
    tipo[:, 0] = tipo[:, -1] = SOLIDO
    rotulo = np.where(tipo == AR, 1, 0).astype(np.uint32)
    for b, (i, j, w, h) in enumerate([(2, 2, 1, 1), (nx // 2, ny // 3, 4, 2), (nx // 3, 2, min(40, nx // 4), 2)]):
        tipo[j:j + h, i:i + w] = AR
        rotulo[j:j + h, i:i + w] = 2 + 5 * b
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
