"""16-bit V-cycles whose coarsest level is itself stored in 16 bits (16,384 cells or more on at most 12 rows), in
shared memory and beyond it, against the oracle's cicloV.  The coarsest solve sweeps in FP32 and stores its
result once.  On a grid of that level alone, with a right side of one sign, that is two roundings to storage
(the right side's and the result's): twice the type's unit roundoff, and FP32's 2e-5; with levels above it the
16-bit bounds of the V-cycle's other tests."""
import numpy as np
import pytest

from estado import erro_relativo
from oraculo import carregar_oraculo
from tanque import _abi, ciclo_v
from tanque.constantes import AGUA, AR

pytestmark = pytest.mark.gpu

PRECS = [pytest.param(_abi.TQ_PREC_FP16, 2.0**-11, 2e-3, id="fp16"), pytest.param(_abi.TQ_PREC_BF16, 2.0**-8, 2e-2, id="bf16")]


@pytest.mark.parametrize("prec,u,tol", PRECS)
@pytest.mark.parametrize("nx,ny", [(1400, 12), (3000, 12), (12, 2000), (2800, 24), (6001, 23)], ids=str)
def test_nivel_mais_grosso(lib_gpu, nx, ny, prec, u, tol):
    tipo = np.full((ny, nx), AGUA, np.uint8)
    tipo[int(0.85 * ny):] = AR
    j, i = np.mgrid[0:ny, 0:nx]
    b = np.where(tipo == AGUA, 1 + 0.5 * np.sin(i / 40.0) * np.cos(j / 3.0), 0).astype(np.float32)
    ref = ciclo_v(tipo, b, ligacao=carregar_oraculo())
    x = ciclo_v(tipo, b, precisao=prec)
    assert erro_relativo(x, ref) < (2 * u + 2e-5 if min(nx, ny) <= 12 else tol)
