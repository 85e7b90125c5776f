"""tq_splat into a caller's buffer on and off a 16-byte boundary, at image sizes with every remainder of the
values a thread takes, against the oracle's splat: bit for bit, as the splat's other test."""
import numpy as np
import pytest

from estado import cena_bolha
from oraculo import mancha_oraculo
from tanque import Cena, SimulacaoGPU
from tanque.constantes import CAMPOS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("desvio", [0, 1])
@pytest.mark.parametrize("w,hp", [(1, 1), (2, 3), (33, 17), (64, 40), (211, 97)], ids=str)
def test_mancha_no_buffer_do_chamador(lib_gpu, w, hp, desvio):
    import torch
    cena, agua = cena_bolha(Cena)
    g = SimulacaoGPU(cena, {"iterations": 3})
    g.adicionar(agua, False)
    buf = torch.full((5 * w * hp + 2,), -7.0, dtype=torch.float32, device="cuda")
    g.mancha(w, hp, buf[desvio:desvio + 5 * w * hp])
    torch.cuda.synchronize()
    img = buf.cpu().numpy()
    ref = mancha_oraculo(g.p.reshape(-1, CAMPOS), cena.nx, cena.ny, cena.h, w, hp)
    assert np.array_equal(img[desvio:desvio + 5 * w * hp].view(np.uint32), ref.ravel().view(np.uint32))
    assert np.all(img[:desvio] == -7.0) and np.all(img[desvio + 5 * w * hp:] == -7.0)
    g.fechar()
