"""The fused solver's phases at the sizes where a thread's four cells, a warp's 30 coarse columns or a
run of cells ends, with and without bubbles (none, a few, more than one batch of a sum's terms), against
the oracle's solve: three iterations in FP32, q to 1e-4, norms and bubble pressures to 1e-3; to the
residual 1e-6 in every precision, q to 1e-3 (the bounds of the other fixed-count and tolerance tests)."""
import numpy as np
import pytest

from estado import erro_relativo
from oraculo import carregar_oraculo
from tanque import _abi, resolver_pressao
from tanque.constantes import AGUA, AR, SOLIDO

pytestmark = pytest.mark.gpu


def problema(nx, ny, bolhas):
    rng = np.random.default_rng(nx * 7 + ny)
    tipo = np.full((ny, nx), AGUA, np.uint8)
    tipo[int(ny * 0.75):] = AR
    tipo[0] = tipo[-1] = SOLIDO
    tipo[:, 0] = tipo[:, -1] = SOLIDO
    rotulo = np.where(tipo == AR, 1, 0).astype(np.uint32)
    lugares = [(i, j) for j in range(2, int(ny * 0.75) - 3, 4) for i in range(2, nx - 4, 4)][:bolhas]
    for b, (i, j) in enumerate(lugares):
        w = 1 + b % 2
        tipo[j:j + w, i:i + w] = AR
        rotulo[j:j + w, i:i + w] = 2 + b
    div = np.where(tipo == AGUA, 0.1 * rng.standard_normal((ny, nx)), 0).astype(np.float32)
    rhs = (0.05 * rng.standard_normal(4096)).astype(np.float32)
    return tipo, rotulo, div, rhs


def resolver(p, iters, tol, prec, lig):
    tipo, rotulo, div, rhs = p
    q = np.zeros(tipo.shape, np.float32)
    b = {"rotulo": rotulo, "rhs": rhs, "y": np.zeros(4096, np.float32)}
    normas = resolver_pressao(tipo, div, q, iters, tol, b, prec, _abi.TQ_ENGINE_FUSED, ligacao=lig)
    return q, b["y"], normas


@pytest.mark.parametrize("bolhas", [0, 3, 800])
@pytest.mark.parametrize("nx,ny", [(26, 26), (61, 45), (62, 33), (120, 90), (123, 241), (322, 203), (900, 700)], ids=str)
def test_fases(lib_gpu, nx, ny, bolhas):
    p = problema(nx, ny, bolhas)
    (qg, yg, ng), (qo, yo, no) = (resolver(p, 3, 0.0, _abi.TQ_PREC_FP32, lig) for lig in (None, carregar_oraculo()))
    assert erro_relativo(qg, qo) < 1e-4
    assert erro_relativo(ng, no) < 1e-3
    if bolhas:
        assert erro_relativo(yg, yo) < 1e-3
    if nx < 400:
        qo = resolver(p, 1000, 1e-6, _abi.TQ_PREC_FP32, carregar_oraculo())[0]
        for prec in (_abi.TQ_PREC_FP32, _abi.TQ_PREC_FP16, _abi.TQ_PREC_BF16):
            assert erro_relativo(resolver(p, 1000, 1e-6, prec, None)[0], qo) < 1e-3
