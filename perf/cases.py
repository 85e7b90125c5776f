"""The work that programs give this framework, as cases that can be timed: frames of a tank through
the simulation handle, a batch of tanks, and the entry points that stand alone (the pressure solve,
the V-cycle, the gradient, the splat).

A frame case is a rollout: the state goes in (particles, the pressure guess, the air labels reset), a
frame of some substeps runs, and every particle and the pressure come back to the host, as a program
does that tries several continuations of one state, restarts a scene, or drives the simulation from a
host that keeps the particles.  Every pass of it therefore does the same work.

Inputs come from the seed: particle velocities, affine terms and positions inside their cells,
right-hand sides, and the target and velocities of the gradient's scene.  The scenes (walls, fill) are
the case's own.
"""
from __future__ import annotations

import ctypes as C
import functools
import math
import os
import sys

import numpy as np
import torch

_PACOTE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tanque-de-agua_b200")
if _PACOTE not in sys.path:
    sys.path.insert(0, _PACOTE)

from tanque import Cena, SimulacaoGPU, _abi, resolver_pressao  # noqa: E402
from tanque.adjunto import AdjuntoGPU, Contexto, PassoDiferenciavel  # noqa: E402
from tanque.cenarios import (cena_adjunto, cena_ar_preso, cena_barragem_160, cena_ultra,  # noqa: E402
                             semear_retangulo_rapido, semente)
from tanque.constantes import CAMPOS, MAX_BOLHAS  # noqa: E402
from tanque.lote import Lote, gerar_tanques  # noqa: E402

PLAIN, FUSED = _abi.TQ_ENGINE_PLAIN, _abi.TQ_ENGINE_FUSED
REF, BLOCO, BLOCO_1 = _abi.TQ_PRECOND_REFERENCE, _abi.TQ_PRECOND_BLOCK, _abi.TQ_PRECOND_BLOCK_1
FP32, FP16, BF16 = _abi.TQ_PREC_FP32, _abi.TQ_PREC_FP16, _abi.TQ_PREC_BF16
SOLIDO, AGUA, AR = 0, 1, 2


def _quadro(name, cena, nx, ny, h, sub, motor=PLAIN, prec=FP32, precond=REF, tol=0.0, iters=3, quadros_s=60.0,
            grafo=False, corante=False, cena_s=1):
    """A rollout of one frame of 1 / quadros_s seconds in `sub` substeps."""
    d = dict(tipo="quadro", cena=cena, nx=nx, ny=ny, h=h, sub=sub, motor=motor, prec=prec, precond=precond, tol=tol,
             iters=iters, quadros_s=quadros_s, grafo=grafo, corante=corante, cena_s=cena_s)
    return dict(d, name=name) if name else d


def listed():
    return [
        # the reference's own engine settings (three PCG iterations, the default engine), from its
        # smallest quality to its largest: what a program gets that sets no option
        _quadro("frame_dam_160x100", "barragem", 160, 100, 0.00625, 4),
        _quadro("frame_tank_251x127_dye", "tanque", 251, 127, 0.004, 5, corante=True),
        _quadro("frame_air_480x270", "ar_preso", 480, 270, 0.0022, 9),
        _quadro("frame_ultra_840x536", "ultra", 840, 536, 0.0016, 14),
        # accurate pressure (true residual 1e-6), the settings of the test suite and the benchmark:
        # trapped air with the reference's preconditioner, and the 450k-cell scene as benchmarked
        _quadro("frame_air_480x270_tol", "ar_preso", 480, 270, 0.0022, 4, FUSED, FP32, REF, 1e-6, 1000, 135.0),
        _quadro("frame_ultra_tol_fp16", "ultra", 840, 536, 0.0016, 4, FUSED, FP16, BLOCO_1, 1e-6, 1000, 210.0, True),
        # a batch of uneven tanks side by side in atlases, each tank to its own tolerance
        dict(name="batch_32_tanks_tol", tipo="lote", n=32, cena_s=4, h=0.003, sub=4, quadros_s=240.0, prec=FP16,
             limite=1000),
        # resolverPCG as a function on host arrays: the drop-in for a host that keeps its own grid, with
        # enclosed air and the reference's three iterations; and an accurate solve at the largest size
        dict(name="solve_333x219_bubbles", tipo="solve", nx=333, ny=219, bolhas=True, motor=PLAIN, prec=FP32, tol=0.0,
             iters=3, cena_s=7),
        dict(name="solve_840x536_tol", tipo="solve", nx=840, ny=536, bolhas=True, motor=FUSED, prec=FP32, tol=1e-6,
             iters=1000, cena_s=8),
        # one V-cycle on device buffers, as a solver of the caller's own takes it as preconditioner
        dict(name="vcycle_641x359_fp16", tipo="vciclo", nx=641, ny=359, prec=FP16, cena_s=9),
        # the gradient of a control problem (forward and backward): the adjoint scene, a third of its steps
        dict(name="gradient_256x160", tipo="adjunto", nx=256, ny=160, passos=20, jato=6),
        # the splat of the particles into an image on the device, twice the grid's resolution
        dict(name="splat_960x540", tipo="mancha", cena="ar_preso", nx=480, ny=270, h=0.0022, w=960, alt=540,
             corante=True, cena_s=1),
    ]


def draw(rng):
    def lado(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    tipo = rng.choices(["quadro", "quadro_tol", "lote", "solve", "vciclo", "adjunto", "mancha"],
                       [6, 3, 1, 3, 2, 1, 2])[0]
    s = rng.randrange(1 << 20)
    if tipo == "quadro":
        nx, ny = lado(100, 800), lado(64, 500)
        h = rng.choice([0.0016, 0.0022, 0.003, 0.004, 0.006])
        return _quadro(None, "tanque", nx, ny, h, rng.randint(2, 10), rng.choice([PLAIN, PLAIN, FUSED]),
                       rng.choice([FP32, FP32, FP16, BF16]), grafo=rng.random() < 0.3, corante=rng.random() < 0.3,
                       cena_s=s)
    if tipo == "quadro_tol":
        nx, ny = lado(100, 600), lado(64, 400)
        h = rng.choice([0.0016, 0.0022, 0.003])
        return _quadro(None, "tanque", nx, ny, h, rng.randint(1, 3), FUSED, rng.choice([FP32, FP16]),
                       rng.choice([REF, BLOCO, BLOCO_1]), 1e-6, 1000, 200.0, rng.random() < 0.5, cena_s=s)
    if tipo == "lote":
        return dict(tipo="lote", n=rng.randint(6, 24), cena_s=s, h=0.003, sub=rng.randint(1, 3), quadros_s=300.0,
                    prec=rng.choice([FP32, FP16]), limite=rng.choice([500, 1000, 3000]))
    if tipo == "solve":
        acurado = rng.random() < 0.4
        return dict(tipo="solve", nx=lado(64, 800), ny=lado(64, 500), bolhas=rng.random() < 0.6,
                    motor=FUSED if acurado else rng.choice([PLAIN, PLAIN, FUSED]), prec=FP32,
                    tol=1e-6 if acurado else 0.0, iters=1000 if acurado else rng.randint(3, 12), cena_s=s)
    if tipo == "vciclo":
        return dict(tipo="vciclo", nx=lado(64, 1200), ny=lado(64, 640), prec=rng.choice([FP32, FP16, BF16]), cena_s=s)
    if tipo == "adjunto":
        return dict(tipo="adjunto", nx=lado(96, 256), ny=lado(64, 160), passos=rng.randint(4, 16),
                    jato=rng.randint(2, 8))
    nx, ny = lado(100, 480), lado(80, 270)
    k = rng.choice([1, 1.5, 2])
    return dict(tipo="mancha", cena="tanque", nx=nx, ny=ny, h=0.003, w=int(nx * k), alt=int(ny * k),
                corante=rng.random() < 0.5, cena_s=s)


# ------------------------------------------------------------------ scenes
@functools.lru_cache(maxsize=4)
def _cena(nome, nx, ny, h, s):
    """(walls, particles at rest) of a scene: the repository's own, or a tank with up to three wall
    segments and a water block over its floor, drawn as the batch draws its tanks."""
    if nome == "barragem":
        return cena_barragem_160(Cena)
    if nome == "ar_preso":
        return cena_ar_preso(Cena, nx, ny, h)
    if nome == "ultra":
        cena, _, agua, _ = cena_ultra(Cena, nx, ny, h)
        return cena, agua
    t = gerar_tanques(1, s, h, (nx, nx), (ny, ny))[0]
    cena = Cena(nx, ny, h)
    for k in t["tracos"]:
        cena.tracar(k["x0"], k["y0"], k["x1"], k["y1"], k["raio"])
    return cena, semear_retangulo_rapido(*t["agua"], h, s=t["semente"])


def _em_movimento(agua, h, seed, corante):
    """The particles of a scene in motion, in pinned memory: a smooth swirl of some tenths of a metre a
    second with its affine terms, small random velocities, jittered positions, and dye on one side."""
    r = np.random.default_rng(seed)
    buf = torch.empty(agua.size, dtype=torch.float32, pin_memory=True)
    p = buf.numpy().reshape(-1, CAMPOS)
    p[:] = agua.reshape(-1, CAMPOS)
    x, y = p[:, 0].copy(), p[:, 1].copy()
    L = np.float32(max(float(x.max(initial=h)), float(y.max(initial=h))))
    for _ in range(3):
        k = (r.uniform(2, 9, 2) / L).astype(np.float32)
        f = r.uniform(0, 2 * math.pi, 2).astype(np.float32)
        A = np.float32(r.uniform(0.05, 0.2))
        sx, cx, sy, cy = np.sin(k[0] * x + f[0]), np.cos(k[0] * x + f[0]), np.sin(k[1] * y + f[1]), np.cos(k[1] * y + f[1])
        p[:, 2] += A * sx * cy
        p[:, 3] -= A * (k[0] / k[1]) * cx * sy
        p[:, 4] += A * k[0] * cx * cy
        p[:, 5] -= A * k[1] * sx * sy
        p[:, 6] += A * k[0] * (k[0] / k[1]) * sx * sy
        p[:, 7] -= A * k[0] * cx * cy
    p[:, 2:4] += 0.02 * r.standard_normal((len(p), 2), dtype=np.float32)
    p[:, 0:2] += np.float32(0.05 * h) * (r.random((len(p), 2), dtype=np.float32) - np.float32(0.5))
    if corante:
        p[x < np.median(x), 9:12] = (0.9, 0.3, 0.1)
    return buf.numpy(), buf


def _grade(case):
    """Cell types and air labels of a pressure problem: the frame, wall segments in the water, a wavy
    surface, and round bubbles (labels from 2) below it."""
    nx, ny = case["nx"], case["ny"]
    al = semente(case["cena_s"])
    cena = Cena(nx, ny, 1.0)
    for _ in range(3):
        x0, y0 = (0.15 + 0.6 * al()) * nx, (0.15 + 0.35 * al()) * ny
        if al() < 0.5:
            cena.tracar(x0, y0, x0 + 0.12 * nx, y0, 2.0)
        else:
            cena.tracar(x0, y0, x0, y0 + 0.12 * ny, 2.0)
    m = cena.sdf.reshape(ny, 2, nx, 2).astype(np.float64)
    solido = m.sum(axis=(1, 3)) < 0
    j, i = np.mgrid[0:ny, 0:nx]
    nivel = (0.62 + 0.06 * np.sin((2 + 4 * al()) * math.pi * i / nx + 6 * al())) * ny
    tipo = np.where(j < nivel, AGUA, AR).astype(np.uint8)
    rotulo = np.where(tipo == AR, 1, 0).astype(np.uint32)
    if case.get("bolhas"):
        for b in range(max(2, min(12, nx * ny // 6000))):
            rr = 2.5 + 7 * al()
            cx, cy = rr + 3 + al() * (nx - 2 * rr - 6), rr + 3 + al() * max(0.45 * ny - 2 * rr - 6, 1)
            dentro = (i - cx) ** 2 + (j - cy) ** 2 < rr * rr
            tipo[dentro] = AR
            rotulo[dentro] = 2 + b
    tipo[solido] = SOLIDO
    rotulo[solido] = 0
    return tipo, rotulo


# ------------------------------------------------------------------ what a program has in hand
def _opcoes(case):
    return {"iteracoes": case.get("iters", 1000), "engine": case.get("motor", FUSED), "precision": case["prec"],
            "preconditioner": case.get("precond", BLOCO), "tolerance": case.get("tol", 1e-6)}


def _conduzir(sim, agua, h, seed, corante=False):
    """A handle with the scene's particles (those that the walls leave room for) in motion, and the host
    buffers they go in from and come back to."""
    if not sim.n:
        sim.adicionar(agua, False)
    p0, guarda = _em_movimento(sim.p, h, seed, corante)
    n = p0.size // CAMPOS
    saida = torch.empty(p0.size, dtype=torch.float32, pin_memory=True)
    q = torch.empty(sim.nx * sim.ny, dtype=torch.float32, pin_memory=True)
    return dict(sim=sim, p0=p0, n=n, saida=saida.numpy(), q=q.numpy(), q0=np.zeros(sim.nx * sim.ny, np.float32),
                guarda=(guarda, saida, q))


def prepare(case, seed):
    t = case["tipo"]
    if t == "quadro":
        cena, agua = _cena(case["cena"], case["nx"], case["ny"], case["h"], case["cena_s"])
        sim = SimulacaoGPU(cena, _opcoes(case))
        return dict(case=case, partes=[_conduzir(sim, agua, case["h"], seed, case["corante"])])
    if t == "lote":
        tanques = gerar_tanques(case["n"], case["cena_s"], case["h"])
        lote = Lote(lambda c, o: SimulacaoGPU(c, o), Cena, tanques, case["h"], _opcoes(case),
                    limite_grosso=case["limite"],
                    sms=torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count)
        partes = [_conduzir(sim, at["particulas"], case["h"], seed + 1000 * k)
                  for k, (sim, at) in enumerate(zip(lote.sims, lote.atlas))]
        return dict(case=case, lote=lote, partes=partes)
    if t == "mancha":
        cena, agua = _cena(case["cena"], case["nx"], case["ny"], case["h"], case["cena_s"])
        sim = SimulacaoGPU(cena)
        p, _ = _em_movimento(agua, case["h"], seed, case["corante"])
        p = p.reshape(-1, CAMPOS).copy()
        # foam where the water is fast, as a running simulation has it
        p[:, 8] = np.clip(np.hypot(p[:, 2], p[:, 3]) * 2 - 0.6, 0, 1)
        sim.definirParticulas(p)
        return dict(case=case, sim=sim, p=p,
                    imagem=torch.empty(5 * case["w"] * case["alt"], dtype=torch.float32, device="cuda"))
    if t == "adjunto":
        cena = cena_adjunto(case["nx"], case["ny"], 0.004, case["passos"], 1 / 240, case["jato"], seed)
        return dict(case=case, adj=AdjuntoGPU(cena), v0=cena["v0"], theta=cena["theta0"])
    tipo, rotulo = _grade(case)
    r = np.random.default_rng(seed)
    j, i = np.mgrid[0:case["ny"], 0:case["nx"]]
    # a divergence as a step leaves it: smooth where the flow is pushed, small and random elsewhere
    div = 0.02 * r.standard_normal((case["ny"], case["nx"]))
    for _ in range(4):
        a, b = r.uniform(1, 12, 2)
        div += 0.05 * np.sin(a * i / case["nx"] * 6 + r.uniform(0, 6)) * np.sin(b * j / case["ny"] * 6 + r.uniform(0, 6))
    div = np.where(tipo == AGUA, div, 0).astype(np.float32)
    if t == "vciclo":
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        b = dev(-div)
        return dict(case=case, tipo=dev(tipo), b=b, x=torch.empty_like(b), f=_vciclo())
    s = dict(case=case, tipo=tipo, div=div, q0=(0.1 * r.standard_normal(div.shape) * (tipo == AGUA)).astype(np.float32))
    s["q"] = s["q0"].copy()
    if case["bolhas"]:
        s["rotulo"] = rotulo
        s["rhs"] = np.zeros(MAX_BOLHAS, np.float32)
        s["rhs"][2:64] = 0.3 * r.standard_normal(62)
        s["y0"] = np.zeros(MAX_BOLHAS, np.float32)
        s["y0"][2:64] = 0.1 * r.standard_normal(62)
    return s


def _vciclo():
    f = _abi.carregar().lib.tq_vcycle_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_int32, C.c_int32, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int32, C.c_void_p]
    return f


# ------------------------------------------------------------------ one pass
def _entrar(h):
    h["sim"].definirParticulas(h["p0"])
    h["sim"].definirCampo("q", h["q0"])
    h["sim"].reiniciarAr()


def _sair(h):
    lig, n = _abi.carregar(), C.c_int32(0)
    lig("get_particles", h["sim"]._h, h["saida"].ctypes.data, h["n"], C.byref(n))
    lig("get_field", h["sim"]._h, _abi.CAMPOS_ENUM["q"], h["q"].ctypes.data, h["q"].nbytes)
    return {"p": h["saida"][: n.value * CAMPOS].reshape(-1, CAMPOS), "q": h["q"].reshape(h["sim"].ny, h["sim"].nx)}


def run(state):
    case = state["case"]
    t = case["tipo"]
    if t in ("quadro", "lote"):
        for h in state["partes"]:
            _entrar(h)
        dt = 1.0 / case["quadros_s"]
        if t == "lote":
            state["lote"].avancar(dt, case["sub"], grafo=True)
        elif case["grafo"]:
            state["partes"][0]["sim"].avancarGrafo(dt, case["sub"])
        else:
            state["partes"][0]["sim"].avancar(dt, case["sub"])
        return [_sair(h) for h in state["partes"]]
    if t == "mancha":
        return state["sim"].mancha(case["w"], case["alt"], state["imagem"])
    if t == "adjunto":
        ctx = Contexto()
        perda = PassoDiferenciavel.forward(ctx, state["adj"], state["v0"], state["theta"])
        _, dv0, dtheta = PassoDiferenciavel.backward(ctx, 1.0)
        return {"perda": perda, "dv0": dv0, "dtheta": dtheta}
    if t == "vciclo":
        st = state["f"](case["nx"], case["ny"], state["tipo"].data_ptr(), state["b"].data_ptr(), state["x"].data_ptr(),
                        case["prec"], torch.cuda.current_stream().cuda_stream)
        if st != _abi.TQ_OK:
            raise RuntimeError(f"tq_vcycle_noalloc: status {st}")
        return state["x"]
    q = state["q"]
    np.copyto(q, state["q0"])
    bolhas = None
    if case["bolhas"]:
        bolhas = {"rotulo": state["rotulo"], "rhs": state["rhs"], "y": state["y0"].copy()}
    resolver_pressao(state["tipo"], state["div"], q, case["iters"], case["tol"], bolhas, case["prec"], case["motor"])
    return {"q": q, "y": bolhas["y"] if bolhas else None}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    t = case["tipo"]
    if t == "quadro" or t == "lote":
        if t == "quadro":
            _, agua = _cena(case["cena"], case["nx"], case["ny"], case["h"], case["cena_s"])
            n, N = agua.size // CAMPOS, case["nx"] * case["ny"]
        else:
            tq = gerar_tanques(case["n"], case["cena_s"], case["h"])
            N = sum(k["nx"] * k["ny"] for k in tq)
            n = int(sum(4 * (k["agua"][2] - k["agua"][0]) * (k["agua"][3] - k["agua"][1]) / case["h"] ** 2 for k in tq))
        # in and out once; each substep reads and writes the particles, the wall SDF, the face
        # velocities and the pressure
        bytes_ = 96 * n + 8 * N + case["sub"] * (96 * n + (16 + 16 + 8 + 2) * N)
        # transfers and micro-steps per particle; surface, divergence and gradient per cell; a V-cycle
        # (4 passes of 4 sweeps a level) and a CG step per cell and iteration, where the count is fixed
        iters = case["iters"] if case.get("tol", 1e-6) == 0 else 30
        return {"bytes": bytes_, "flops": case["sub"] * (350 * n + (150 + 200 * iters) * N)}
    if t == "mancha":
        _, agua = _cena(case["cena"], case["nx"], case["ny"], case["h"], case["cena_s"])
        n = agua.size // CAMPOS
        px = math.pi * 2.1 ** 2 * (case["w"] / case["nx"]) * (case["alt"] / case["ny"])
        return {"bytes": 32 * n + 20 * case["w"] * case["alt"], "flops": n * px * (15 if case["corante"] else 10)}
    if t == "adjunto":
        N, n = case["nx"] * case["ny"], int(0.3 * 0.35 * 4 * case["nx"] * case["ny"])
        # forward, the recomputation and the reverse step each touch the state and the grid once and
        # (forward, recomputed, reversed) solve once, in doubles
        return {"bytes": case["passos"] * 3 * (128 * n + 60 * N), "flops": case["passos"] * 3 * (400 * n + 20 * 220 * N)}
    N = case["nx"] * case["ny"]
    if t == "vciclo":
        return {"bytes": 9 * N, "flops": 200 * N}
    iters = case["iters"] if case["tol"] == 0 else 30
    return {"bytes": (13 + (4 if case["bolhas"] else 0)) * N, "flops": 210 * iters * N}


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    """The splat, the V-cycle and the pressure solve in doubles with torch.  The frames have no such value
    (a frame of particles is chaotic in its last digits) and the gradient would be the whole step again."""
    if case["tipo"] == "mancha":
        return _mancha64(case, prepare(case, seed)["p"])
    if case["tipo"] == "vciclo":
        s = prepare(case, seed)
        return _Multigrade(s["tipo"].cpu().numpy()).ciclo(s["b"].double())
    if case["tipo"] == "solve":
        return _solve64(case, prepare(case, seed))
    return None


def _mancha64(case, p):
    w, alt, nx, ny, h = case["w"], case["alt"], case["nx"], case["ny"], case["h"]
    p = torch.from_numpy(p).cuda().double()
    raio, px, py, H = 2.1 * h, nx * h / w, ny * h / alt, ny * h
    i0, j0 = (p[:, 0] / px - 0.5).floor().long(), ((H - p[:, 1]) / py - 0.5).floor().long()
    ri, rj = int(raio / px) + 2, int(raio / py) + 2
    canais = torch.stack([torch.ones_like(p[:, 8]), p[:, 8], p[:, 9], p[:, 10], p[:, 11]])
    img = torch.zeros(5, alt * w, dtype=torch.float64, device="cuda")
    for dj in range(-rj, rj + 1):
        for di in range(-ri, ri + 1):
            i, j = i0 + di, j0 + dj
            u = ((i + 0.5) * px - p[:, 0]) / raio
            v = ((H - (j + 0.5) * py) - p[:, 1]) / raio
            r2 = u * u + v * v
            ok = (r2 < 1) & (i >= 0) & (j >= 0) & (i < w) & (j < alt)
            img.index_add_(1, (j * w + i)[ok], canais[:, ok] * (1 - r2[ok]) ** 2)
    return img.reshape(-1)


class _Multigrade:
    """cicloV (js/pressao-cpu.js:241-255) in doubles on the grid of cell types `tipo`."""

    def __init__(self, tipo):
        self.n = []
        while True:
            self.n.append(self._nivel(tipo))
            ny, nx = tipo.shape
            if min(nx, ny) <= 12:
                break
            f = np.full((2 * ((ny + 1) // 2), 2 * ((nx + 1) // 2)), SOLIDO, np.uint8)
            f[:ny, :nx] = tipo
            f = f.reshape(f.shape[0] // 2, 2, f.shape[1] // 2, 2)
            tipo = np.where((f == AR).any(axis=(1, 3)), AR, np.where((f == AGUA).any(axis=(1, 3)), AGUA, SOLIDO))
            tipo = tipo.astype(np.uint8)

    @staticmethod
    def _nivel(tipo):
        t = torch.from_numpy(np.ascontiguousarray(tipo)).cuda().long()
        ny, nx = t.shape
        livre = torch.nn.functional.pad((t != SOLIDO).double(), (1, 1, 1, 1))
        viz = [livre[1:-1, :-2], livre[1:-1, 2:], livre[:-2, 1:-1], livre[2:, 1:-1]]
        k = sum(viz)
        i, j = torch.arange(nx, device="cuda"), torch.arange(ny, device="cuda")
        return dict(agua=t == AGUA, viz=viz, k=k, muda=(t == AGUA) & (k > 0), inv=1 / k.clamp(min=1), i=i, j=j,
                    cor=(i[None, :] + j[:, None] + 1) & 1, nx=nx, ny=ny)

    @staticmethod
    def _viz(x):
        p = torch.nn.functional.pad(x, (1, 1, 1, 1))
        return p[1:-1, :-2], p[1:-1, 2:], p[:-2, 1:-1], p[2:, 1:-1]

    def _suavizar(self, n, x, b, desl, ordem):
        ci, cj = ((n["i"] + desl) % 16)[None, :], ((n["j"] + desl) % 16)[:, None]
        dentro = [ci != 0, ci != 15, cj != 0, cj != 15]
        fora = sum(v * torch.where(d, 0.0, s) for v, d, s in zip(n["viz"], dentro, self._viz(x)))
        q = x
        for h in range(8):
            cor = (h & 1) ^ ordem
            s = fora + sum(v * torch.where(d, c, 0.0) for v, d, c in zip(n["viz"], dentro, self._viz(q)))
            q = torch.where(n["muda"] & (n["cor"] == cor), (s + b) * n["inv"], q)
        return torch.where(n["agua"], q, 0.0)

    def ciclo(self, b, l=0):
        n = self.n[l]
        x = torch.zeros_like(b)
        if l == len(self.n) - 1:
            for k in range(64):
                for o in range(2):
                    cor = 1 - o if k & 1 else o
                    s = sum(v * c for v, c in zip(n["viz"], self._viz(x)))
                    x = torch.where(n["muda"] & (n["cor"] == cor), (s + b) * n["inv"], x)
            return x
        x = self._suavizar(n, x, b, 0, 0)
        x = self._suavizar(n, x, b, 8, 0)
        r = torch.where(n["agua"], b - (n["k"] * x - sum(v * c for v, c in zip(n["viz"], self._viz(x)))), 0.0)
        g = self.n[l + 1]
        r = torch.nn.functional.pad(r, (1, 2 * g["nx"] - n["nx"] + 1, 1, 2 * g["ny"] - n["ny"] + 1))
        w = torch.tensor([0.25, 0.75, 0.75, 0.25], dtype=torch.float64, device="cuda")
        bg = torch.nn.functional.conv2d(r[None, None], (w[:, None] * w[None, :])[None, None], stride=2)[0, 0]
        e = self.ciclo(torch.where(g["agua"], bg, 0.0), l + 1)
        e = torch.nn.functional.pad(torch.where(g["agua"], e, 0.0), (1, 1, 1, 1))

        def base(i):
            return torch.where(i & 1 == 0, (i >> 1) - 1, (i - 1) >> 1) + 1, torch.where(i & 1 == 0, 0.25, 0.75).double()
        (I, wi), (J, wj) = base(n["i"]), base(n["j"])
        wi, wj = wi[None, :], wj[:, None]
        up = (e[J][:, I] * wi * wj + e[J][:, I + 1] * (1 - wi) * wj + e[J + 1][:, I] * wi * (1 - wj)
              + e[J + 1][:, I + 1] * (1 - wi) * (1 - wj))
        x = torch.where(n["agua"], x + up, x)
        x = self._suavizar(n, x, b, 8, 1)
        return self._suavizar(n, x, b, 0, 1)


def _solve64(case, s):
    """resolverPCG (js/pressao-cpu.js:296-402) in doubles; with a tolerance, to a residual of 1e-13."""
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    tipo = dev(s["tipo"]).long()
    agua, ar = tipo == AGUA, tipo == AR
    com = case["bolhas"]
    rot = dev(s["rotulo"].astype(np.int64)) if com else torch.zeros_like(tipo)
    V = _Multigrade._viz
    livre = V((tipo != SOLIDO).double())
    # faces between a bubble's interior cells and water
    miolo = torch.zeros_like(agua)
    miolo[1:-1, 1:-1] = True
    b_int = ar & (rot >= 2) & miolo
    nag = V(agua.double())
    faces = torch.zeros(MAX_BOLHAS, dtype=torch.float64, device="cuda")
    faces.index_add_(0, rot[b_int], sum(nag)[b_int])
    ativa = faces > 0
    b_cel = ar & (rot >= 2) & ativa[rot]
    b_int &= b_cel
    cels = torch.zeros_like(faces).index_add_(0, rot[b_cel], torch.ones_like(rot[b_cel]).double())

    def A(q, y):
        g = torch.where(b_cel, y[rot], torch.where(agua, q, 0.0))
        aq = torch.where(agua, sum(livre) * q - sum(f * c for f, c in zip(livre, V(g))), 0.0)
        so = torch.zeros_like(y).index_add_(0, rot[b_int], sum(V(torch.where(agua, q, 0.0)))[b_int])
        return aq, torch.where(ativa, faces * y - so, 0.0)

    mg = _Multigrade(np.where(s["tipo"] == AR, np.where(rot.cpu().numpy() >= 2, AGUA, AR), s["tipo"]).astype(np.uint8))

    def M(r, rb):
        b = torch.where(b_cel, (rb / cels.clamp(min=1))[rot], r)
        x = mg.ciclo(b)
        zb = torch.zeros_like(rb).index_add_(0, rot[b_cel], (x / cels.clamp(min=1)[rot])[b_cel])
        return torch.where(agua, x, 0.0), zb

    q = torch.where(agua, dev(s["q0"]).double(), 0.0)
    y = torch.where(ativa, dev(s["y0"]).double(), 0.0) if com else torch.zeros_like(faces)
    rhs = dev(s["rhs"]).double() if com else torch.zeros_like(faces)
    aq, ay = A(q, y)
    r, rb = torch.where(agua, -dev(s["div"]).double() - aq, 0.0), torch.where(ativa, rhs - ay, 0.0)
    ponto = lambda a, ab, b, bb: float((a * b).sum() + (ab * bb).sum())  # noqa: E731
    n0 = math.sqrt(ponto(r, rb, r, rb))
    z, zb = M(r, rb)
    p, pb = z, zb
    rz = ponto(r, rb, z, zb)
    for it in range(case["iters"] if case["tol"] == 0 else 400):
        ap, apb = A(p, pb)
        pap = ponto(p, pb, ap, apb)
        al = rz / pap if abs(pap) > 1e-30 else 0.0
        q, y, r, rb = q + al * p, y + al * pb, r - al * ap, rb - al * apb
        if case["tol"] > 0 and math.sqrt(ponto(r, rb, r, rb)) <= 1e-13 * n0:
            break
        zo, zbo = z, zb
        z, zb = M(r, rb)
        novo = ponto(r, rb, z, zb)
        be = max(0.0, (novo - ponto(r, rb, zo, zbo)) / rz) if abs(rz) > 1e-30 else 0.0
        rz = novo
        p, pb = z + be * p, zb + be * pb
    if not com:
        return {"q": q, "y": None}
    return {"q": q, "y": torch.where(ativa, y, dev(s["y0"]).double())}
