"""The V-cycle's level legs in the variants that only larger grids reach, against the oracle: 16-bit storage on level 1
and below, and the block preconditioners (closed faces between water cells on the coarse levels, one pass a leg)
on tiles of more than one block.  The 16-bit V-cycle's bounds are those of its other tests; three plain
iterations: q to 1e-4, norms to 1e-3 (the bounds of the fixed-count solves)."""
import numpy as np
import pytest

from estado import erro_relativo
from oraculo import carregar_oraculo
from tanque import _abi, ciclo_v, resolver_pressao
from tanque.constantes import AGUA, AR, SOLIDO

pytestmark = pytest.mark.gpu


def problema(nx, ny):
    """Water under air, loose wall cells, and walls one cell thick along and across the water."""
    rng = np.random.default_rng(nx + 7 * ny)
    tipo = np.full((ny, nx), AGUA, np.uint8)
    tipo[rng.random((ny, nx)) < 0.03] = SOLIDO
    for k in range(1, 6):
        tipo[k * ny // 8, nx // 10: 9 * nx // 10] = SOLIDO
        tipo[ny // 10: 7 * ny // 10, k * nx // 6] = SOLIDO
    tipo[int(0.8 * ny):] = AR
    return tipo, np.where(tipo == AGUA, rng.standard_normal((ny, nx)), 0).astype(np.float32)


@pytest.mark.parametrize("prec,tol", [(_abi.TQ_PREC_FP16, 2e-3), (_abi.TQ_PREC_BF16, 2e-2)], ids=["fp16", "bf16"])
@pytest.mark.parametrize("nx,ny", [(500, 333), (1030, 770)], ids=str)
def test_16_bits(lib_gpu, nx, ny, prec, tol):
    tipo, b = problema(nx, ny)
    assert erro_relativo(ciclo_v(tipo, b, precisao=prec), ciclo_v(tipo, b, ligacao=carregar_oraculo())) < tol


@pytest.mark.parametrize("precond", [_abi.TQ_PRECOND_BLOCK, _abi.TQ_PRECOND_BLOCK_1], ids=["bloco", "bloco-1"])
@pytest.mark.parametrize("nx,ny", [(1030, 770), (1499, 701)], ids=str)
def test_blocos(lib_gpu, nx, ny, precond):
    tipo, b = problema(nx, ny)
    saidas = []
    for lig in (None, carregar_oraculo()):
        q = np.zeros((ny, nx), np.float32)
        saidas.append((resolver_pressao(tipo, 0.1 * b, q, 3, 0.0, precond=precond, ligacao=lig), q))
    (ng, qg), (no, qo) = saidas
    assert erro_relativo(qg, qo) < 1e-4
    assert erro_relativo(ng, no) < 1e-3
