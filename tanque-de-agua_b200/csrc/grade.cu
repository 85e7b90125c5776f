// grade.cu — per-cell and per-face kernels of the substep between the particle transfers and
// around the pressure solve: wall cells, cell flags, air-label propagation, surface fraction /
// normal / curvature, surface-tension air pressure, divergence with density correction,
// bubble right-hand sides, air pressure after the solve, pressure gradient and velocity
// extrapolation.
//
// Built with -fmad=false and written in double arithmetic with f32 stores, the way the
// reference's JavaScript computes (double locals, Float32Array stores): these stages then
// agree with the oracle bit for bit except where a transcendental (hypot) is involved.
#include "common.cuh"
#include "kernels.cuh"

namespace tq {

// Cena.celulaSolida (js/cena.js:119-127) for every cell: SimulacaoCPU.atualizarParedes.
__global__ void k_solidos(Dev d) {
  aposAnterior();
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.N) return;
  int i = c % d.nx, j = c / d.nx;
  int a = i * RES_MASCARA, b = j * RES_MASCARA;
  const float* s = d.sdf;
  double soma = (double)s[(size_t)b * d.mw + a] + (double)s[(size_t)b * d.mw + a + 1] +
                (double)s[(size_t)(b + 1) * d.mw + a] + (double)s[(size_t)(b + 1) * d.mw + a + 1];
  d.solido[c] = soma < 0 ? 1 : 0;
}

// Cena#moldura (js/cena.js:131-137): distance (cells) from mask point (x, y) to the frame's
// inner edge, positive inside the tank, clamped to +-SDF_MAX.
__device__ double molduraMascara(int x, int y, int mw, int mh) {
  const double m = MOLDURA * RES_MASCARA - 0.5;
  const double d = fmin(fmin(x - m, (double)(mw - 1) - m - x), fmin(y - m, (double)(mh - 1) - m - y)) / RES_MASCARA;
  return d > SDF_MAX ? SDF_MAX : d < -SDF_MAX ? -SDF_MAX : d;
}

// Cena.tracar (js/cena.js:43-72) on the device mask: one thread per mask point of the
// segment's box (x0, y0, nbx x nby), the capsule distance in double precision as the reference
// computes it, min into the mask (draw) or max of its negation capped by the frame (erase).
__global__ void k_tracar(float* sdf, int mw, int mh, int x0, int y0, int nbx, int nby, double ax, double ay, double dx,
                         double dy, double len2, double rp, int apagar) {
  aposAnterior();
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= nbx * nby) return;
  const int x = x0 + idx % nbx, y = y0 + idx / nbx;
  double t = len2 > 0 ? ((x - ax) * dx + (y - ay) * dy) / len2 : 0;
  t = t < 0 ? 0 : t > 1 ? 1 : t;
  const double px = ax + t * dx - x, py = ay + t * dy - y;
  double d = (sqrt(px * px + py * py) - rp) / RES_MASCARA;
  if (d > SDF_MAX) d = SDF_MAX;
  else if (d < -SDF_MAX) d = -SDF_MAX;
  const size_t k = (size_t)y * mw + x;
  double v = apagar ? fmax((double)sdf[k], -d) : fmin((double)sdf[k], d);
  if (apagar) v = fmin(v, molduraMascara(x, y, mw, mh));
  sdf[k] = (float)v;
}

// Cena#zerar (js/cena.js:139-144): the mask of an empty tank, the frame alone.  One round of blocks, several
// points a thread: a block's wait for the kernel before costs more than its points (a call on 7,221x316 cells took
// 63 us with a point a thread, 47 now).
constexpr int BLOCOS_ZERAR = 1184;  // 8 a SM
__global__ void __launch_bounds__(256) k_zerar_mascara(float* sdf, int mw, int mh) {
  aposAnterior();
  for (int idx = blockIdx.x * 256 + threadIdx.x; idx < mw * mh; idx += gridDim.x * 256)
    sdf[idx] = (float)molduraMascara(idx % mw, idx / mw, mw, mh);
}

// Adds 1 to *cont for every lane with `sim` and returns the lane's slot: one atomic a warp.
__device__ __forceinline__ int reservar(int* cont, bool sim) {
  const unsigned m = __ballot_sync(0xffffffffu, sim);
  if (!m) return 0;
  const int lane = threadIdx.x & 31, lider = __ffs(m) - 1;
  int base = 0;
  if (lane == lider) base = atomicAdd(cont, __popc(m));
  return __shfl_sync(0xffffffffu, base, lider) + __popc(m & ((1u << lane) - 1u));
}

// #tipos (js/fisica-cpu.js:293-299) and, with `faces`, the face velocities: the sums' quotient, gravity
// where a particle contributed, zero on wall faces (js/fisica-cpu.js:265-266 + :271-291 in the integer form of
// js/gpu/fisica.js:135-160).  With `ar`, the first step of #propagarRotulos (:412, non-air cells lose
// their label) and the list of the cells its first pass may label (see k_rotulos_resolver).
__global__ void __launch_bounds__(256) k_tipos(Dev d, int faces, float gdx, float gdy, int ar) {
  aposAnterior();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int nx = d.nx, ny = d.ny;
  if (faces) {
    if (k < d.nu) {
      const int i = k % (nx + 1), j = k / (nx + 1);
      const int2 a = d.accU[k];
      float val = 0.0f;
      if (a.y > 0) val = __fadd_rn(__fdiv_rn((float)a.x, (float)a.y), gdx);
      const bool s = i == 0 || i == nx || d.solido[i - 1 + j * nx] || d.solido[i + j * nx];
      d.u[k] = s ? 0.0f : val;
    }
    if (k < d.nv) {
      const int i = k % nx, j = k / nx;
      const int2 a = d.accV[k];
      float val = 0.0f;
      if (a.y > 0) val = __fadd_rn(__fdiv_rn((float)a.x, (float)a.y), gdy);
      const bool s = j == 0 || j == ny || d.solido[i + (j - 1) * nx] || d.solido[i + j * nx];
      d.v[k] = s ? 0.0f : val;
    }
  }
  bool p = false;
  if (k < d.N) {
    const uint8_t t = d.solido[k] ? SOLIDO : d.accCel[k].y > 0 ? AGUA : AR;
    d.tipo[k] = t;
    if (!faces) {  // the flags alone: the water fraction too (in a substep k_superficie makes it)
      const double dens = (float)d.accCel[k].x * (1.0f / 65536.0f);
      d.fase[k] = t == SOLIDO ? 0.0f : (float)fmin(1.0, dens / PARTICULAS_POR_CELULA);
    }
    if (ar) {
      if (t != AR) d.rotulo[k] = 0;
      const int i = k % nx, j = k / nx;
      p = i >= 1 && j >= 1 && i < nx - 1 && j < ny - 1 && t == AR && d.rotulo[k] == 0;
      d.pend[k] = p ? 1 : 0;
    }
  }
  if (ar) {
    const int slot = reservar(&d.esc->pendentes, p);
    if (p) d.lista[slot] = k;
  }
}

// ---------------------------------------------------------------- label propagation
// #propagarRotulos (js/fisica-cpu.js:409-422): two in-place raster passes over the interior;
// an unlabelled air cell takes the first non-zero of (left, right, down, up).  In raster order
// the left and lower neighbours already hold this pass's value while the right and upper ones
// hold the value from before the pass.  That makes each pass a system whose dependencies
// point only backwards in raster order, so it has exactly one solution, and repeating the
// update until nothing changes reaches it whatever order the cells are visited in.  Only the
// cells that were unlabelled air at the start of the pass ("pending") change; for a pending
// right/upper neighbour the before-the-pass value is 0.  One CTA does both passes: the second's
// pending cells are those of the first's list that are still unlabelled.  A step before any label is known
// has all air pending, a step of a running simulation a few cells.  All pending, no label / one cell in a
// thousand / in ten labelled, on 480x270 cells: 118 / 4890 / 802 us with the whole list walked in the second
// pass and each cell asked whether it is pending, 56 / 4100 / 624 now (107 / 3970 / 581 as four launches).
__global__ void __launch_bounds__(1024) k_rotulos_resolver(Dev d) {
  aposAnterior();
  __shared__ int mudou, ficam;
  int n = d.esc->pendentes;
  const int nx = d.nx;
  uint32_t* rot = d.rotulo;
  uint8_t* pend = d.pend;
  for (int passada = 0; passada < 2; passada++) {
    // Each sweep fixes at least one more cell of the longest dependency chain; n + 2 sweeps
    // always suffice.
    bool igual = true;
    for (int volta = 0; volta < n + 2; volta++) {
      if (threadIdx.x == 0) mudou = 0;
      __syncthreads();
      for (int t = threadIdx.x; t < n; t += blockDim.x) {
        const int c = d.lista[t];
        uint32_t r = rot[c - 1];
        if (!r) r = pend[c + 1] ? 0u : rot[c + 1];
        if (!r) r = rot[c - nx];
        if (!r) r = pend[c + nx] ? 0u : rot[c + nx];
        if (r != rot[c]) {
          rot[c] = r;
          mudou = 1;
        }
      }
      __syncthreads();
      if (!mudou) break;
      igual = false;
      __syncthreads();
    }
    if (passada == 1 || igual) break;  // (a pass that changed nothing would be repeated as it was)
    // the cells still unlabelled to the list's front, a block's worth at a time
    if (threadIdx.x == 0) ficam = 0;
    for (int t0 = 0; t0 < n; t0 += blockDim.x) {
      const int t = t0 + threadIdx.x, c = t < n ? d.lista[t] : 0;
      const bool fica = t < n && rot[c] == 0;
      if (t < n && !fica) pend[c] = 0;
      __syncthreads();
      const int slot = reservar(&ficam, fica);
      if (fica) d.lista[slot] = c;
      __syncthreads();
    }
    n = ficam;
    __syncthreads();
  }
  if (threadIdx.x == 0) d.esc->pendentes = 0;
}

// ---------------------------------------------------------------- surface
// #superficie (js/fisica-cpu.js:306-345) on one tile of 16x16 or 32x32 cells a CTA, in shared memory: the water fraction of
// every cell, three times carried into the walls (#estenderNaParede, :353-374: three layers, each a
// wall cell taking the mean of its neighbours that are no wall or were filled in an earlier layer) with
// two separable (1 2 1)/4 blurs in between (:314-328), the normals grad f / |grad f| and the
// curvature -div n / (2h) on the interior (:330-345; border cells are never written, they stay 0).  A
// tile also computes the 13 cells around it that its result depends on, each stage needing one or
// three fewer.  The 24 launches over the grid that this replaces took 105 us a substep on 160x100 cells,
// where each waited for the one before, and 128 us on 840x536.  What bounds it is the chain of its 20-odd
// stages, each a meeting of the CTA: the wall cells of the three layers are listed once, so an extension
// takes its own cells and not the whole region; the blurs walk a segment of a row or column a thread, so
// each value is converted to double once; and a grid whose 16x16 tiles fill the GPU at most once
// takes those (twice the cells around a tile, half the work of a CTA; with more tiles the larger
// ones' fewer cells win).  160x100 cells: 35 us with 32x32 tiles of 256 threads that scanned the region
// for each layer, 13 us now; 840x536: 48 -> 31 us.
constexpr int SUP_H = 13, SUP_THREADS = 512, SUP_LINHAS = 64, SUP_SEGS = SUP_THREADS / SUP_LINHAS;
constexpr int SUP_TILES = 592;  // 4 CTAs on each of 148 SMs
constexpr int SUP_LINHAS_MAX = 65535;  // rows of tiles in a launch's second dimension; more go to the third
constexpr uint8_t SUP_LIVRE = 0, SUP_FUNDO = 200, SUP_FORA = 255;  // marks: no wall; wall beyond layer 3; off the grid

template <int SUP_T>
__global__ void __launch_bounds__(SUP_THREADS) k_superficie(Dev d) {
  aposAnterior();
  constexpr int SUP_W = SUP_T + 2 * SUP_H, SUP_P = SUP_W + 1;  // odd pitch: no bank conflicts
  constexpr int SUP_SEG = (SUP_W + SUP_SEGS - 1) / SUP_SEGS;   // cells of a line a thread blurs
  static_assert(SUP_W <= SUP_LINHAS, "a thread a line");
  __shared__ float f[SUP_W * SUP_P], g[SUP_W * SUP_P];
  __shared__ uint8_t mk[SUP_W * SUP_P];  // SUP_LIVRE, the layer a wall cell is filled in (1-3), SUP_FUNDO, SUP_FORA
  __shared__ uint16_t lista[SUP_W * SUP_W];  // the wall cells of layers 1, 2 and 3
  __shared__ int nLista;
  const int nx = d.nx, ny = d.ny, x0 = blockIdx.x * SUP_T - SUP_H;
  const int y0 = (blockIdx.y + blockIdx.z * SUP_LINHAS_MAX) * SUP_T - SUP_H;
  if (y0 + SUP_H >= ny) return;  // (uniform over the CTA)
  if (threadIdx.x == 0) nLista = 0;
  bool parede = false;
  for (int t = threadIdx.x; t < SUP_W * SUP_W; t += SUP_THREADS) {
    const int i = t % SUP_W, j = t / SUP_W, gx = x0 + i, gy = y0 + j, o = j * SUP_P + i;
    float v = 0.0f;
    uint8_t m = SUP_FORA;
    if (gx >= 0 && gy >= 0 && gx < nx && gy < ny) {
      const int c = gx + gy * nx;
      m = d.tipo[c] == SOLIDO ? SUP_FUNDO : SUP_LIVRE;
      // the initial water fraction (:309)
      const double dens = (float)d.accCel[c].x * (1.0f / 65536.0f);
      if (m == SUP_LIVRE) v = (float)fmin(1.0, dens / PARTICULAS_POR_CELULA);
      else parede = true;
    }
    f[o] = v;
    g[o] = 0.0f;
    mk[o] = m;
  }
  // the layer each wall cell is filled in follows from the types alone: a wall cell beside a cell of
  // the layer before
  int fim[4] = {0, 0, 0, 0};
  if (__syncthreads_or(parede))
#pragma unroll
    for (int L = 1; L <= 3; L++) {
      const int w = SUP_W - 2 * L;
      for (int t = threadIdx.x; t < w * w; t += SUP_THREADS) {
        const int o = (L + t / w) * SUP_P + L + t % w;
        if (mk[o] == SUP_FUNDO && (mk[o - 1] == L - 1 || mk[o + 1] == L - 1 || mk[o - SUP_P] == L - 1 || mk[o + SUP_P] == L - 1)) {
          mk[o] = (uint8_t)L;
          lista[atomicAdd(&nLista, 1)] = (uint16_t)o;
        }
      }
      __syncthreads();
      fim[L] = nLista;
      __syncthreads();
    }
  // one extension: layer L reads the layers before it (cells nearer the region's edge than the stage
  // reaches get values that nothing reads)
  auto estender = [&] {
#pragma unroll
    for (int L = 1; L <= 3; L++) {
      if (fim[L] == fim[L - 1]) continue;
      for (int t = fim[L - 1] + threadIdx.x; t < fim[L]; t += SUP_THREADS) {
        const int o = lista[t];
        double s = 0;
        int k = 0;
        const int nb[4] = {o - 1, o + 1, o - SUP_P, o + SUP_P};
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (mk[nb[q]] < L) {
            s += (double)f[nb[q]];
            k++;
          }
        f[o] = (float)(s / k);
      }
      __syncthreads();
    }
  };
  const int seg = threadIdx.x / SUP_LINHAS, linha = threadIdx.x % SUP_LINHAS;
  // blur of the cells `b` inside: rows into g, then columns back into f (b + 1 inside)
  auto borrar = [&](int b) {
    if (linha >= b && linha < SUP_W - b) {
      const int i0 = max(seg * SUP_SEG, b + 1), i1 = min((seg + 1) * SUP_SEG, SUP_W - b - 1), r = linha * SUP_P;
      double a = i0 < i1 ? (double)f[r + i0 - 1] : 0.0, c = i0 < i1 ? (double)f[r + i0] : 0.0;
      for (int i = i0; i < i1; i++) {
        const double n = (double)f[r + i + 1];
        const int gx = x0 + i;
        g[r + i] = (float)(((gx > 0 ? a : c) + 2 * c + (gx < nx - 1 ? n : c)) * 0.25);
        a = c;
        c = n;
      }
    }
    __syncthreads();
    if (linha >= b + 1 && linha < SUP_W - b - 1) {
      const int j0 = max(seg * SUP_SEG, b + 1), j1 = min((seg + 1) * SUP_SEG, SUP_W - b - 1);
      double a = j0 < j1 ? (double)g[(j0 - 1) * SUP_P + linha] : 0.0, c = j0 < j1 ? (double)g[j0 * SUP_P + linha] : 0.0;
      for (int j = j0; j < j1; j++) {
        const double n = (double)g[(j + 1) * SUP_P + linha];
        const int gy = y0 + j;
        f[j * SUP_P + linha] = (float)(((gy > 0 ? a : c) + 2 * c + (gy < ny - 1 ? n : c)) * 0.25);
        a = c;
        c = n;
      }
    }
    __syncthreads();
  };
  estender();
  borrar(3);
  estender();
  borrar(7);
  estender();
  // f is done on the tile and 2 cells around it; the normals' components (g and h) on 1 cell around it
  __shared__ float h[(SUP_T + 2) * (SUP_T + 3)];
  constexpr int HP = SUP_T + 3;
  for (int t = threadIdx.x; t < (SUP_T + 2) * (SUP_T + 2); t += SUP_THREADS) {
    const int i = t % (SUP_T + 2), j = t / (SUP_T + 2), o = (j + 12) * SUP_P + i + 12, gx_ = x0 + i + 12, gy_ = y0 + j + 12;
    float a = 0.0f, b = 0.0f;
    if (gx_ >= 1 && gy_ >= 1 && gx_ < nx - 1 && gy_ < ny - 1) {
      const double gx = ((double)f[o + 1] - (double)f[o - 1]) * 0.5, gy = ((double)f[o + SUP_P] - (double)f[o - SUP_P]) * 0.5;
      const double n = hypot(gx, gy);
      a = n > 1e-3 ? (float)(gx / n) : 0.0f;
      b = n > 1e-3 ? (float)(gy / n) : 0.0f;
    }
    g[o] = a;
    h[j * HP + i] = b;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < SUP_T * SUP_T; t += SUP_THREADS) {
    const int i = t % SUP_T, j = t / SUP_T, gx = x0 + SUP_H + i, gy = y0 + SUP_H + j;
    if (gx >= nx || gy >= ny) continue;
    const int c = gx + gy * nx, o = (j + SUP_H) * SUP_P + i + SUP_H, oh = (j + 1) * HP + i + 1;
    d.fase[c] = f[o];
    if (gx < 1 || gy < 1 || gx >= nx - 1 || gy >= ny - 1) continue;
    const double a = ((double)g[o + 1] - (double)g[o - 1]) + ((double)h[oh + HP] - (double)h[oh - HP]);
    d.nX[c] = g[o];
    d.nY[c] = h[oh];
    d.kap[c] = (float)(-a / (2 * d.h));
  }
}

// #pressaoDoAr (js/fisica-cpu.js:381-403): the surface-tension jump of cell c, interior air (0 elsewhere),
// in units of q = p*dt/(rho*h).
__device__ inline float pressaoDoAr(const Dev& d, int c, int i, int j, double dt, double tensao) {
  const int nx = d.nx;
  if (!(i >= 1 && j >= 1 && i < nx - 1 && j < d.ny - 1) || d.tipo[c] != AR) return 0.0f;
  double pp = 0;
  if (tensao > 0) {
    const float* kap = d.kap;
    double s = kap[c];
    int k = 1;
    if (d.tipo[c - 1] == AGUA) { s += (double)kap[c - 1]; k++; }
    if (d.tipo[c + 1] == AGUA) { s += (double)kap[c + 1]; k++; }
    if (d.tipo[c - nx] == AGUA) { s += (double)kap[c - nx]; k++; }
    if (d.tipo[c + nx] == AGUA) { s += (double)kap[c + nx]; k++; }
    double kMax = 1 / d.h;
    if (k > 1) pp += tensao * fmax(-kMax, fmin(kMax, s / k));
  }
  return (float)(pp * (dt / (DENSIDADE_AGUA * d.h)));
}

// #pressaoDoAr, #classificar + #miolo (js/fisica-cpu.js:456-494) and the cells' part of
// #ladoDireitoDasBolhas (:429-454) in one pass over the grid: the air's pressure; the right-hand side of
// the projection, divergence minus the density correction minus the known air pressure of the
// neighbours (each neighbour's made again here, few cells have one); per bubble the water flowing
// into it now minus the surface-tension term of each water face, and its cells.  The per-bubble sums
// are 64-bit fixed point (2^-32) so their value does not depend on the order cells arrive in.  The last
// block closes the bubbles' right-hand sides: the volume recovery term and the initial pressure.
// One round of blocks, 6 an SM at 40 registers: with a block a 256 cells and 79 registers (3 an SM) each
// block's ticket waited for its writes, which took 15.4 us on 480x270 cells, 32 on 840x536, 150 on 9000x400
// and 447 on 38,370x316; 13.5, 22, 62 and 142 now (three kernels for the same work: 26, 40, 80 and 207).
constexpr int BLOCOS_LADO = 888;
__global__ void __launch_bounds__(256, 6) k_lado_direito(Dev d, double dt, double tensao, double tau, int bolhas) {
  aposAnterior();
  const int nx = d.nx, ny = d.ny;
  static_assert(MAX_BOLHAS % 256 == 0, "the last block's labels");
  for (int c0 = blockIdx.x * blockDim.x; c0 < d.N; c0 += gridDim.x * blockDim.x) {  // (uniform over the block)
    const int c = c0 + threadIdx.x;
    uint32_t b = 0;
    if (c < d.N) {
      const int i = c % nx, j = c / nx, t0 = d.tipo[c];
      const float qa = pressaoDoAr(d, c, i, j, dt, tensao);
      d.qAr[c] = qa;
      if (t0 != AGUA) {
        d.div[c] = 0.0f;
        d.q[c] = 0.0f;
      } else {
        double alvo = d.h / fmax(tau, dt);
        double dv = (double)d.u[i + 1 + j * (nx + 1)] - (double)d.u[i + j * (nx + 1)] +
                    (double)d.v[i + (j + 1) * nx] - (double)d.v[i + j * nx];
        double dens = (float)d.accCel[c].x * (1.0f / 65536.0f);
        double excesso = dens / PARTICULAS_POR_CELULA - 1;
        if (excesso < 0) {
          bool miolo = i >= 1 && j >= 1 && i < nx - 1 && j < ny - 1;
          for (int b2 = -1; b2 <= 1 && miolo; b2++)
            for (int a = -1; a <= 1; a++) {
              int n = i + a + (j + b2) * nx;
              if (d.solido[n] || d.accCel[n].y == 0) { miolo = false; break; }
            }
          if (!miolo) excesso = 0;
        }
        excesso = fmin(EXCESSO_MAX, fmax(EXCESSO_MIN, excesso));
        double ar = 0;
        long N = d.N;
        const int nb[4] = {c - 1, c + 1, c - nx, c + nx};  // flat neighbours, as the reference reads them
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (tipoEm(d.tipo, (long)nb[k], N, AR)) ar += (double)pressaoDoAr(d, nb[k], nb[k] % nx, nb[k] / nx, dt, tensao);
        d.div[c] = (float)(dv - alvo * excesso - ar);
      }
      if (bolhas && t0 == AR && i >= 1 && j >= 1 && i < nx - 1 && j < ny - 1) {
        const uint32_t r = d.rotulo[c];
        if (r >= 2 && r < (uint32_t)MAX_BOLHAS) {
          b = r;
          double t = qa;
          double s = 0;
          if (d.tipo[c - 1] == AGUA) s += (double)d.u[i + j * (nx + 1)] - t;
          if (d.tipo[c + 1] == AGUA) s += -(double)d.u[i + 1 + j * (nx + 1)] - t;
          if (d.tipo[c - nx] == AGUA) s += (double)d.v[i + j * nx] - t;
          if (d.tipo[c + nx] == AGUA) s += -(double)d.v[i + (j + 1) * nx] - t;
          somaFixa(&d.accB[r], s, ESCALA_BOLHA);
        }
      }
    }
    if (bolhas && __any_sync(0xffffffffu, b != 0)) {  // the cells of a bubble lie together: an atomic a warp and bubble
      const unsigned g = __match_any_sync(0xffffffffu, b);
      if (b && (int)(threadIdx.x & 31) == __ffs(g) - 1) atomicAdd(&d.volB[b], (unsigned)__popc(g));
    }
  }
  if (!bolhas) return;  // uniform over the grid
  __shared__ bool ultimo;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    ultimo = atomicAdd(&d.esc->tickets[1], 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!ultimo) return;
  __threadfence();
  if (threadIdx.x == 0) d.esc->tickets[1] = 0;
  // a thread's labels all at once: a label after the other waited for memory 16 times over (the kernel on
  // 160x100 cells: 15 -> 11 us).  What only bubbles with cells have is loaded for those alone: batches of it
  // for every label took the kernel's registers from 40 to 79, which left an SM 3 blocks.
  constexpr int K = MAX_BOLHAS / 256;
  uint32_t vol[K];
#pragma unroll
  for (int k = 0; k < K; k++) vol[k] = __ldcg(&d.volB[threadIdx.x + k * 256]);
#pragma unroll
  for (int k = 0; k < K; k++) {
    const int r = threadIdx.x + k * 256;
    float rhs = 0.0f;
    if (vol[k]) {  // (labels 0 and 1 are counted nowhere)
      rhs = (float)((double)__ldcg(&d.accB[r]) / ESCALA_BOLHA);
      rhs = (float)((double)rhs + VOLTA_VOLUME_BOLHA * ((double)d.volumeAlvo[r] - (double)vol[k]) * d.h / dt);
      d.yBolhaF[r] = (float)((double)d.pressaoBolha[r] * (dt / (DENSIDADE_AGUA * d.h)));
    }
    d.volumeBolhaF[r] = (float)vol[k];
    d.rhsBolhaF[r] = rhs;
  }
}

// #pressao after resolverPCG (js/fisica-cpu.js:503-514) and #gradiente (:519-545) in one pass: air cells get
// the surface-tension pressure plus their bubble's pressure; bubbles keep their pressure in Pa
// (clamped); the faces beside water take the gradient, into uTmp / vTmp.  A face reads an air cell's
// pressure from its parts, so no thread waits for the q another writes.
__global__ void __launch_bounds__(256) k_gradiente(Dev d, double dt, int ar) {
  aposAnterior();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int nx = d.nx, ny = d.ny;
  const uint8_t* tipo = d.tipo;
  auto qDoAr = [&](int c) {
    const uint32_t r = d.rotulo[c];
    const bool bolha = ar && r >= 2 && r < (uint32_t)MAX_BOLHAS && d.volumeBolhaF[r] != 0.0f;
    return (float)((double)d.qAr[c] + (bolha ? (double)d.yBolhaF[r] : 0.0));
  };
  auto qDe = [&](int c, uint8_t t) { return t == AR ? qDoAr(c) : d.q[c]; };
  if (k < d.N && tipo[k] == AR) d.q[k] = qDoAr(k);
  if (ar && k >= 2 && k < MAX_BOLHAS && d.volumeBolhaF[k] != 0.0f) {
    const double paraPa = (DENSIDADE_AGUA * d.h) / dt;
    d.pressaoBolha[k] = (float)fmax(-PRESSAO_BOLHA_MAX, fmin(PRESSAO_BOLHA_MAX, (double)d.yBolhaF[k] * paraPa));
  }
  if (k == 0) d.esc->vmaxBits = 0;  // k_g2p's largest speed starts from 0
  if (k < d.nu) {
    const int i = k % (nx + 1), j = k / (nx + 1);
    const uint8_t tl = i > 0 ? tipo[i - 1 + j * nx] : SOLIDO;
    const uint8_t tr = i < nx ? tipo[i + j * nx] : SOLIDO;
    float u = d.u[k];
    int val = 0;
    if (tl == SOLIDO || tr == SOLIDO) {
      u = 0.0f;
      val = 1;
    } else if (tl == AGUA || tr == AGUA) {
      u = (float)((double)u - ((double)qDe(i + j * nx, tr) - (double)qDe(i - 1 + j * nx, tl)));
      val = 1;
    }
    d.uTmp[k] = u;
    d.uValTmp[k] = (uint8_t)val;
  }
  if (k < d.nv) {
    const int i = k % nx, j = k / nx;
    const uint8_t tb = j > 0 ? tipo[i + (j - 1) * nx] : SOLIDO;
    const uint8_t tt = j < ny ? tipo[i + j * nx] : SOLIDO;
    float v = d.v[k];
    int val = 0;
    if (tb == SOLIDO || tt == SOLIDO) {
      v = 0.0f;
      val = 1;
    } else if (tb == AGUA || tt == AGUA) {
      v = (float)((double)v - ((double)qDe(i + j * nx, tt) - (double)qDe(i + (j - 1) * nx, tb)));
      val = 1;
    }
    d.vTmp[k] = v;
    d.vValTmp[k] = (uint8_t)val;
  }
}

// extrapolarComponente (js/fisica-cpu.js:673-690), both layers for u and v: an invalid face takes the mean
// of its valid 4-neighbours, or, with none, of the neighbours that the first layer made valid (each
// made again here: few faces need it).  Reads uTmp / vTmp, writes u / v.
__device__ inline bool camadaExtrapolada(const float* a, const uint8_t* val, int k, int w, int hh, float* out) {
  const int i = k % w, j = k / w;
  double soma = 0;
  int n = 0;
  if (i > 0 && val[k - 1]) { soma += (double)a[k - 1]; n++; }
  if (i < w - 1 && val[k + 1]) { soma += (double)a[k + 1]; n++; }
  if (j > 0 && val[k - w]) { soma += (double)a[k - w]; n++; }
  if (j < hh - 1 && val[k + w]) { soma += (double)a[k + w]; n++; }
  if (n > 0) *out = (float)(soma / n);
  return n > 0;
}
__device__ inline void extrapolar2(const float* a, const uint8_t* val, float* ao, uint8_t* vo, int k, int w, int hh) {
  float x = a[k];
  bool ok = val[k] != 0;
  if (!ok) {
    const int i = k % w, j = k / w;
    const bool e = i > 0, d = i < w - 1, b = j > 0, c = j < hh - 1;
    // the flags around the face go out together: first its neighbours', then those around them (one by one, each
    // behind the branch on the one before, an air face waited 20 times: gradient and extrapolation took 103 us on
    // 9000x400 cells and 91 on 7,221x316, 81 and 80 now; 840x536 stays at 24)
    const int perto = (e ? val[k - 1] : 0) | (d ? val[k + 1] : 0) | (b ? val[k - w] : 0) | (c ? val[k + w] : 0);
    if (perto) {
      ok = camadaExtrapolada(a, val, k, w, hh, &x);
    } else {
      const int longe = (i > 1 ? val[k - 2] : 0) | (i < w - 2 ? val[k + 2] : 0) | (j > 1 ? val[k - 2 * w] : 0) |
                        (j < hh - 2 ? val[k + 2 * w] : 0) | (e && b ? val[k - w - 1] : 0) | (d && b ? val[k - w + 1] : 0) |
                        (e && c ? val[k + w - 1] : 0) | (d && c ? val[k + w + 1] : 0);
      if (longe) {
        double soma = 0;
        int n = 0;
        float y = 0.0f;
        if (e && camadaExtrapolada(a, val, k - 1, w, hh, &y)) { soma += (double)y; n++; }
        if (d && camadaExtrapolada(a, val, k + 1, w, hh, &y)) { soma += (double)y; n++; }
        if (b && camadaExtrapolada(a, val, k - w, w, hh, &y)) { soma += (double)y; n++; }
        if (c && camadaExtrapolada(a, val, k + w, w, hh, &y)) { soma += (double)y; n++; }
        if (n > 0) {
          x = (float)(soma / n);
          ok = true;
        }
      }
    }
  }
  ao[k] = x;
  vo[k] = ok ? 1 : 0;
}
__global__ void __launch_bounds__(256) k_extrapolar(Dev d) {
  aposAnterior();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < d.nu) extrapolar2(d.uTmp, d.uValTmp, d.u, d.uVal, k, d.nx + 1, d.ny);
  if (k < d.nv) extrapolar2(d.vTmp, d.vValTmp, d.v, d.vVal, k, d.nx, d.ny + 1);
}

// ---------------------------------------------------------------- host launchers
void lancarSolidos(const Dev& d, cudaStream_t s) { lanca(k_solidos, blocos(d.N, 256), 256, 0, s, d); }
void lancarTracar(const Dev& d, double x0m, double y0m, double x1m, double y1m, double raio, bool apagar,
                  cudaStream_t s) {
  // the box and the segment in mask points, on the host in the same double arithmetic
  const double r = RES_MASCARA, esc = r / d.h;
  const double ax = x0m * esc - 0.5, ay = y0m * esc - 0.5, bx = x1m * esc - 0.5, by = y1m * esc - 0.5;
  const double rp = raio * esc;
  const double alc = rp + SDF_MAX * r + 1;
  const double xmin = fmax(0.0, floor(fmin(ax, bx) - alc)), xmax = fmin((double)(d.mw - 1), ceil(fmax(ax, bx) + alc));
  const double ymin = fmax(0.0, floor(fmin(ay, by) - alc)), ymax = fmin((double)(d.mh - 1), ceil(fmax(ay, by) + alc));
  if (!(xmin <= xmax) || !(ymin <= ymax)) return;
  const int nbx = (int)(xmax - xmin) + 1, nby = (int)(ymax - ymin) + 1;
  const double dx = bx - ax, dy = by - ay;
  lanca(k_tracar, blocos(nbx * nby, 256), 256, 0, s, (float*)d.sdf, d.mw, d.mh, (int)xmin, (int)ymin, nbx, nby, ax, ay, dx, dy,
        dx * dx + dy * dy, rp, apagar ? 1 : 0);
}
void lancarZerarMascara(const Dev& d, cudaStream_t s) {
  lanca(k_zerar_mascara, min(blocos(d.mw * d.mh, 256), BLOCOS_ZERAR), 256, 0, s, (float*)d.sdf, d.mw, d.mh);
}
void lancarTipos(const Dev& d, bool faces, float gdx, float gdy, bool ar, cudaStream_t s) {
  const int m = !faces ? d.N : d.nu > d.nv ? d.nu : d.nv;
  lanca(k_tipos, blocos(m, 256), 256, 0, s, d, faces ? 1 : 0, gdx, gdy, ar ? 1 : 0);
}
void lancarPropagarRotulos(const Dev& d, cudaStream_t s) { lanca(k_rotulos_resolver, 1, 1024, 0, s, d); }
void lancarSuperficie(const Dev& d, cudaStream_t s) {
  auto ladrilhos = [&](int t) {
    const int linhas = blocos(d.ny, t);
    return dim3(blocos(d.nx, t), min(linhas, SUP_LINHAS_MAX), blocos(linhas, SUP_LINHAS_MAX));
  };
  if (blocos(d.nx, 16) * blocos(d.ny, 16) <= SUP_TILES) lanca(k_superficie<16>, ladrilhos(16), SUP_THREADS, 0, s, d);
  else lanca(k_superficie<32>, ladrilhos(32), SUP_THREADS, 0, s, d);
}
void lancarLadoDireito(const Dev& d, double dt, double tensao, double tau, bool bolhas, cudaStream_t s) {
  // accB, facesB, celsB and volB are one block of memory
  if (bolhas) cudaMemsetAsync(d.accB, 0, MAX_BOLHAS * (sizeof(long long) + 3 * sizeof(uint32_t)), s);
  lanca(k_lado_direito, min(blocos(d.N, 256), BLOCOS_LADO), 256, 0, s, d, dt, tensao, tau, bolhas ? 1 : 0);
}
void lancarGradiente(const Dev& d, double dt, bool ar, cudaStream_t s) {
  int m = d.nu > d.nv ? d.nu : d.nv;
  m = m > MAX_BOLHAS ? m : MAX_BOLHAS;
  lanca(k_gradiente, blocos(m, 256), 256, 0, s, d, dt, ar ? 1 : 0);
}
void lancarExtrapolar(const Dev& d, cudaStream_t s) {
  int m = d.nu > d.nv ? d.nu : d.nv;
  lanca(k_extrapolar, blocos(m, 256), 256, 0, s, d);
}

}  // namespace tq
