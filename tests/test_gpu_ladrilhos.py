"""The V-cycle's level legs on tiles (tq_vcycle) at the sizes where a tile, a block or the coarse section
ends, against the oracle's cicloV: FP32 to 2e-5 relative (the bound of the V-cycle's other tests).  The
right side is NaN off water: a caller's values there must not reach the result."""
import numpy as np
import pytest

from estado import erro_relativo
from oraculo import carregar_oraculo
from tanque import ciclo_v
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
