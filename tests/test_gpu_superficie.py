"""The grid stages of a substep (surface tile, right-hand side, gradient, extrapolation) at grid sizes around
their tiles' and blocks' edges, with thin and thick walls, trapped air and dye, against the oracle:
integers bit-exact, fields to the tolerances of the substep's parity test."""
import numpy as np
import pytest

from estado import INTEIROS, copiar_estado, erro_relativo
from oraculo import CenaOraculo, SimulacaoOraculo
from tanque import Cena, SimulacaoGPU, _abi
from tanque.cenarios import semear_retangulo
from tanque.constantes import CAMPOS

pytestmark = pytest.mark.gpu

FLUTUANTES = {"u": 1e-4, "v": 1e-4, "q": 1e-4, "div": 1e-5, "fase": 1e-6, "curvatura": 1e-4, "qAr": 1e-4,
              "normalX": 1e-4, "normalY": 1e-4, "pressaoBolha": 1e-3, "volumeAlvo": 0.0}


@pytest.mark.parametrize("ar", [True, False], ids=["ar", "sem-ar"])
@pytest.mark.parametrize("nx,ny", [(11, 9), (31, 33), (32, 32), (45, 64), (65, 31), (97, 66), (700, 240)], ids=str)
def test_etapas_da_grade(lib_gpu, nx, ny, ar):
    h = 0.01
    cena_o, cena_g = CenaOraculo(nx, ny, h), Cena(nx, ny, h)
    for c in (cena_o, cena_g):  # a wall of one cell, one of ten, and a cup over the water
        c.tracar(0.3 * nx * h, 0.3 * ny * h, 0.3 * nx * h, 0.5 * ny * h, 0.6 * h)
        c.tracar(0.75 * nx * h, 0.1 * ny * h, 0.75 * nx * h, 0.3 * ny * h, min(5, nx // 10) * h)
        c.tracar(0.45 * nx * h, 0.62 * ny * h, 0.6 * nx * h, 0.62 * ny * h, 0.8 * h)
    cena_g.sdf[:] = cena_o.sdf
    opc = {"air": int(ar)}
    o, g = SimulacaoOraculo(cena_o, dict(opc, p2g_mode=_abi.TQ_P2G_FIXED)), SimulacaoGPU(cena_g, dict(opc))
    agua = semear_retangulo(2 * h, 2 * h, (nx - 2) * h, 0.6 * ny * h, h, (0.3, 0.0, 0.1)).reshape(-1, CAMPOS)
    x, y = agua[:, 0] / (nx * h), agua[:, 1] / (ny * h)
    agua[:, 2] = 0.3 * np.sin(9 * y)
    agua[:, 3] = 0.2 * np.cos(7 * x)
    agua = agua[(x - 0.5) ** 2 + (y - 0.25) ** 2 > 0.01]  # trapped air
    for s in (o, g):
        s.adicionar(agua.ravel(), False)
    for quadro in range(3):
        copiar_estado(o, g)
        for s in (o, g):
            s.avancar(1 / 240, 1)
        for campo in INTEIROS:
            assert np.array_equal(g.campo(campo), o.campo(campo)), f"{quadro}: {campo}"
        for campo, tol in FLUTUANTES.items():
            e = erro_relativo(g.campo(campo), o.campo(campo))
            assert e <= tol, f"{quadro}: {campo} relative error {e:.3g} > {tol}"
