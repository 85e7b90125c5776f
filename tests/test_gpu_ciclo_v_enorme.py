"""A V-cycle on a grid whose levels hold more than 2^31 cells together: around a few sources, its values are
those of a small grid with the same cells in the same places of every level's blocks, bit for bit."""
import numpy as np
import pytest

from tanque import ciclo_v
from tanque.constantes import AGUA

pytestmark = pytest.mark.gpu

# 832 columns halve to 7 whatever the rows, and both numbers of rows are multiples of 1,024: the same blocks
# around the first and the last rows on every level
NX, BAIXO, ALTO = 832, 4096, 1_945_600


def memoria_livre():
    for linha in open("/proc/meminfo"):
        if linha.startswith("MemAvailable"):
            return int(linha.split()[1]) * 1024
    return 0


def test_mais_de_2_31_celulas(lib_gpu):
    import torch
    if memoria_livre() < 48 << 30 or torch.cuda.mem_get_info()[0] < 90 << 30:
        pytest.skip("needs 48 GB of host memory and 90 GB on the device")
    fonte = np.random.default_rng(5).standard_normal((40, 40)).astype(np.float32)
    x = {}
    for ny in (BAIXO, ALTO):
        # water around the sources alone, so the coarse levels' values are the same
        tipo = np.zeros((ny, NX), np.uint8)
        b = np.zeros((ny, NX), np.float32)
        for j in (0, ny - 1024):
            tipo[j + 100:j + 900, 50:780] = AGUA
            b[j + 300:j + 340, 400:440] = fonte
        r = ciclo_v(tipo, b)
        x[ny] = r[:1024].copy(), r[-1024:].copy()
        del tipo, b, r
    for k in range(2):
        assert np.any(x[BAIXO][k])
        assert np.array_equal(x[ALTO][k], x[BAIXO][k])
