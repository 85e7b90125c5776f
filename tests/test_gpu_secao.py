"""The fused solver's coarse section where its variants meet: sections built as a matrix by one CTA,
few CTAs and the whole GPU, coarsest levels below and above the stored-matrix size, and coarsest
levels of one to many cells a thread.  A substep solved to the true residual 1e-6 against the
oracle's: integers bit-exact, q, u and v to 1e-3 relative (the bound of the 840x536 scene's test)."""
import numpy as np
import pytest

from estado import INTEIROS, erro_relativo
from oraculo import CenaOraculo, SimulacaoOraculo
from tanque import Cena, SimulacaoGPU, _abi
from tanque.cenarios import semear_retangulo_rapido

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [1, 4, 0])
@pytest.mark.parametrize("nx,ny,precond", [
    (30, 26, _abi.TQ_PRECOND_REFERENCE),    # one level above a 15x13 coarsest
    (256, 92, _abi.TQ_PRECOND_BLOCK),       # section 64x23 over 32x12, above the stored-matrix size
    (161, 77, _abi.TQ_PRECOND_BLOCK_1),     # one pass a leg in the section
    (700, 70, _abi.TQ_PRECOND_REFERENCE),   # coarsest 88x9
    (2900, 20, _abi.TQ_PRECOND_BLOCK),      # coarsest 1450x10: several cells a thread
], ids=str)
def test_secao_grossa(lib_gpu, ctas, nx, ny, precond):
    h = 0.004
    opc = {"tolerance": 1e-6, "iterations": 1000, "preconditioner": precond}
    cena_g, cena_o = Cena(nx, ny, h), CenaOraculo(nx, ny, h)
    for c in (cena_g, cena_o):
        c.tracar(0.5 * nx * h, 3 * h, 0.5 * nx * h, 0.6 * ny * h, 1.6 * h)
    g = SimulacaoGPU(cena_g, dict(opc, engine=_abi.TQ_ENGINE_FUSED, fused_ctas=ctas))
    o = SimulacaoOraculo(cena_o, dict(opc, p2g_mode=_abi.TQ_P2G_FIXED))
    agua = semear_retangulo_rapido(2 * h, 2 * h, 0.7 * nx * h, 0.7 * ny * h, h, s=5)
    for s in (g, o):
        s.adicionar(agua, False)
        s.avancar(1 / 480, 1)
    for campo in INTEIROS:
        assert np.array_equal(g.campo(campo), o.campo(campo)), campo
    for campo in ["q", "u", "v"]:
        e = erro_relativo(g.campo(campo), o.campo(campo))
        assert e <= 1e-3, f"{campo} relative error {e:.3g}"
    for s in (g, o):
        assert s.escalar(_abi.TQ_SCALAR_PCG_CONVERGED) == 1
