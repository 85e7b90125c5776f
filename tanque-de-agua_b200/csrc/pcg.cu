// pcg.cu — MGPCG pressure projection: PCG with a multigrid V-cycle preconditioner, each
// enclosed air pocket one extra unknown ("supercell").  Restates js/pressao-cpu.js
// (resolverPCG :296-402, cicloV :241-255 and its parts) on the device.
//
// This file is the PLAIN engine: separate launches, the iteration loop on the host.  A V-cycle takes
// one launch a leg of each level (suavizador.cuh) and one for its coarse levels.  The V-cycle vectors (b, x, tmp of every level) are stored as T = float, __half or
// __nv_bfloat16 (levels below 16k cells stay float); arithmetic is FP32; dot products and
// norms are FP64 with a fixed reduction order (bitwise reproducible); per-bubble sums are
// 64-bit fixed point.
#include <mutex>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "pcg_interno.cuh"
#include "suavizador.cuh"
#include <type_traits>

namespace tq {

// Level 0's masks also carry, during a solve, whether the cell is air of an active bubble that the
// V-cycle sees as water (it takes its bubble's mean residual and gives its share of z back) and
// whether it is water to the operator.
constexpr int V0_BOLHA = 32, V0_AGUA = 64;

// ---------------------------------------------------------------- types and neighbours
// The preconditioner's level-0 types: bubble air counts as water (js/pressao-cpu.js:305-308); with
// TQ_PRECOND_BLOCK (bloco) it stays air.  And the operator's free neighbours (bits 0-3) of every
// cell, from the true types.
__global__ void k_mg_tipo0(const uint8_t* tipo, const uint32_t* rot, uint8_t* t0, uint8_t* vizOp, int nx, int ny,
                           int bolhas, int bloco) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nx * ny) return;
  const int i = c % nx, j = c / nx;
  uint8_t t = tipo[c];
  int m = 0;
  if (i > 0 && tipo[c - 1] != SOLIDO) m |= 1;
  if (i < nx - 1 && tipo[c + 1] != SOLIDO) m |= 2;
  if (j > 0 && tipo[c - nx] != SOLIDO) m |= 4;
  if (j < ny - 1 && tipo[c + nx] != SOLIDO) m |= 8;
  vizOp[c] = (uint8_t)m;
  if (bolhas && !bloco && t == AR && rot[c] >= 2) t = AGUA;
  t0[c] = t;
}

// The levels' sizes and arrays for the two kernels that prepare them.
struct Niveis {
  int L;
  int nx[MAX_NIVEIS], ny[MAX_NIVEIS];
  int ini[MAX_NIVEIS + 1];  // k_niveis_viz: first thread of each level
  uint8_t *tipo[MAX_NIVEIS], *viz[MAX_NIVEIS];
};

// tiposGrossos (js/pressao-cpu.js:63-81) of levels l0 + 1 .. l0 + 6: air if any child is air, else
// water if any is water.  A CTA takes 64x64 cells of level l0 and halves them in shared memory (a
// launch a level took 2.4-3.6 us each).
constexpr int NIVEIS_POR_VEZ = 6;
__global__ void __launch_bounds__(256) k_niveis_tipos(Niveis n, int l0) {
  __shared__ uint8_t t[2][32 * 32];
  auto mais = [](int a, int b) { return a == AR || b == AR ? (int)AR : a == AGUA || b == AGUA ? (int)AGUA : (int)SOLIDO; };
  const int L = min(n.L - 1, l0 + NIVEIS_POR_VEZ);
  for (int l = l0 + 1; l <= L; l++) {
    const int w = 64 >> (l - l0);  // the CTA's side on level l
    const uint8_t* f = t[(l - l0 - 1) & 1];
    for (int c = threadIdx.x; c < w * w; c += 256) {
      const int i = c % w, j = c / w, I = blockIdx.x * w + i, J = blockIdx.y * w + j;
      int r = SOLIDO;
      if (l == l0 + 1) {
        const int fx = n.nx[l0], fy = n.ny[l0];
        const uint8_t* src = n.tipo[l0];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int x = 2 * I + (q & 1), y = 2 * J + (q >> 1);
          if (x < fx && y < fy) r = mais(r, src[x + (size_t)y * fx]);
        }
      } else {
        const uint8_t* o = f + 2 * j * 2 * w + 2 * i;
        r = mais(mais(o[0], o[1]), mais(o[2 * w], o[2 * w + 1]));
      }
      t[(l - l0) & 1][c] = (uint8_t)r;
      if (I < n.nx[l] && J < n.ny[l]) n.tipo[l][I + (size_t)J * n.nx[l]] = (uint8_t)r;
    }
    __syncthreads();
  }
}

// Level 0's masks in a solve: k_niveis_viz's bits and V0_AGUA; V0_BOLHA where `bolhas` (celsB counted).
__global__ void k_viz0(Dev d, const uint8_t* tipo0, uint8_t* viz, int bolhas) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.N) return;
  int i = c % d.nx, j = c / d.nx;
  int m = 0;
  if (i > 0 && tipo0[c - 1] != SOLIDO) m |= 1;
  if (i < d.nx - 1 && tipo0[c + 1] != SOLIDO) m |= 2;
  if (j > 0 && tipo0[c - d.nx] != SOLIDO) m |= 4;
  if (j < d.ny - 1 && tipo0[c + d.nx] != SOLIDO) m |= 8;
  if (tipo0[c] == AGUA) m |= 16;
  const int t = d.tipo[c];
  if (t == AGUA) m |= V0_AGUA;
  else if (bolhas && t == AR) {
    const uint32_t b = d.rotulo[c];
    if (b >= 2 && b < (uint32_t)MAX_BOLHAS && d.celsB[b] > 0) m |= V0_BOLHA;
  }
  viz[c] = (uint8_t)m;
}

// prepararVizinhos (js/pressao-cpu.js:44-60) of every level from l0 on in one launch, packed in one byte:
// bits 0-3 = free (non-wall) left/right/down/up neighbours, bit 4 = the cell itself is water.  With
// `bloco` (TQ_PRECOND_BLOCK) the coarse levels' bits 0-3 are open where a fine face across the coarse
// face joins two non-wall fine cells (both coarse cells not wall).
__global__ void k_niveis_viz(Niveis n, int l0, int bloco) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  int l = l0;
  while (l < n.L && g >= n.ini[l + 1]) l++;
  if (l >= n.L) return;
  const int c = g - n.ini[l], nx = n.nx[l], ny = n.ny[l], i = c % nx, j = c / nx;
  const uint8_t* tipo = n.tipo[l];
  int m = 0;
  if (bloco && l >= 1) {
    if (tipo[c] != SOLIDO) {
      const uint8_t* tf = n.tipo[l - 1];
      const int fnx = n.nx[l - 1], fny = n.ny[l - 1];
      auto livre = [&](int x, int y) { return x >= 0 && y >= 0 && x < fnx && y < fny && tf[x + y * fnx] != SOLIDO; };
      auto horiz = [&](int i0, int i1) {
        return (livre(i0, 2 * j) && livre(i1, 2 * j)) || (livre(i0, 2 * j + 1) && livre(i1, 2 * j + 1));
      };
      auto vert = [&](int j0, int j1) {
        return (livre(2 * i, j0) && livre(2 * i, j1)) || (livre(2 * i + 1, j0) && livre(2 * i + 1, j1));
      };
      if (i > 0 && tipo[c - 1] != SOLIDO && horiz(2 * i - 1, 2 * i)) m |= 1;
      if (i < nx - 1 && tipo[c + 1] != SOLIDO && horiz(2 * i + 1, 2 * i + 2)) m |= 2;
      if (j > 0 && tipo[c - nx] != SOLIDO && vert(2 * j - 1, 2 * j)) m |= 4;
      if (j < ny - 1 && tipo[c + nx] != SOLIDO && vert(2 * j + 1, 2 * j + 2)) m |= 8;
    }
  } else {
    if (i > 0 && tipo[c - 1] != SOLIDO) m |= 1;
    if (i < nx - 1 && tipo[c + 1] != SOLIDO) m |= 2;
    if (j > 0 && tipo[c - nx] != SOLIDO) m |= 4;
    if (j < ny - 1 && tipo[c + nx] != SOLIDO) m |= 8;
  }
  if (tipo[c] == AGUA) m |= 16;
  n.viz[l][c] = (uint8_t)m;
}

// ---------------------------------------------------------------- V-cycle kernels
// What level 0's right side is made from: v, scaled by *escala (null: 1), cells of active bubbles
// their bubble's mean residual (precondicionar, js/pressao-cpu.js:353-355).
struct Fonte {
  const float* v;
  const double* escala = nullptr;
  const uint32_t* rotulo = nullptr;
  const double* rb = nullptr;
  const uint32_t* celsB = nullptr;
};

constexpr int T_LADRILHO = 512;

// The way down a level on one tile a CTA (descerLadrilho): both passes and the restriction.
template <class T, class TG, bool NIVEL0>
__global__ void __launch_bounds__(T_LADRILHO) k_descer(NivelDev<T> n, NivelDev<TG> g, int kx, int ky, int uma, int masc,
                                                       Fonte F) {
  extern __shared__ __align__(16) float mem[];
  if (n.parar && *n.parar) return;  // uniform over the CTA
  const Ladrilho L{(int)blockIdx.x * 16 * kx, (int)blockIdx.y * 16 * ky, kx, ky, n.nx, n.ny, n.viz};
  const float e = NIVEL0 && F.escala ? (float)*F.escala : 1.0f;
  descerLadrilho<T>(
      L, g.nx, g.ny, g.viz, uma != 0, masc != 0, VARREDURAS, mem,
      [&](int c) { return NIVEL0 ? __ldca(F.v + c) : carregar(n.b[c]); },
      [&](int c, int v, float bv, bool meu) {
        if (!NIVEL0) return bv;
        if (v & V0_BOLHA) {
          const uint32_t r = F.rotulo[c];
          bv = (float)(F.rb[r] / F.celsB[r]);
        }
        const T bt = guardar<T>(bv * e);
        if (meu) n.b[c] = bt;
        return carregar(bt);
      },
      [&](int c, float x) { n.x[c] = guardar<T>(x); }, [&](int C, float v) { g.b[C] = guardar<TG>(v); });
}

// The way up a level: x + the coarse correction and both passes, the level's result in n.tmp, or
// (saida not null) as floats in saida.
template <class T, class TG>
__global__ void __launch_bounds__(T_LADRILHO) k_subir(NivelDev<T> n, NivelDev<TG> g, const TG* xg, int kx, int ky,
                                                      int uma, int masc, float* saida) {
  extern __shared__ __align__(16) float mem[];
  if (n.parar && *n.parar) return;
  const Ladrilho L{(int)blockIdx.x * 16 * kx, (int)blockIdx.y * 16 * ky, kx, ky, n.nx, n.ny, n.viz};
  subirLadrilho<T>(
      L, g.nx, g.ny, uma != 0, masc != 0, VARREDURAS, mem, [&](int c) { return carregar(n.x[c]); },
      [&](int C) { return carregar(xg[C]); }, [&](int c) { return carregar(n.b[c]); },
      [&](const int (&cel)[2][4], const int (&v)[2][4], const float (&x)[2][4]) {
#pragma unroll
        for (int cr = 0; cr < 2; cr++)
#pragma unroll
          for (int m = 0; m < 4; m++)
            if (cel[cr][m] >= 0) {
              if (saida) saida[cel[cr][m]] = arredondar<T>(x[cr][m]);
              else n.tmp[cel[cr][m]] = guardar<T>(x[cr][m]);
            }
      });
}

// The coarse levels of at most SECAO_PLANA cells in one CTA, in shared memory: x as swept, its snapshot
// before the pass (what a block's outer neighbours hold), the right side.  A thread takes two cells
// side by side, one of each colour, so every thread works in every half-sweep and half the warps
// meet at its barrier: four shared loads, the sum, a store.  The coarsest level's half-sweeps that
// repeat the one before (the last colour of a sweep is the first of the next, and a colour reads
// only the other) are left out, 65 of 128.  8 us with a coarsest level of
// 49 cells alone, 17 us for three levels from 943 cells, where six launches a level and the 42-46 us of
// one CTA's 128 half-sweeps were.
constexpr int SECAO_PLANA = 1024, SECAO_PLANA_NIVEIS = 6, SECAO_PLANA_TOTAL = 1536, T_SECAO = 576;
struct SecaoPlana {
  int L, uma;
  int off[SECAO_PLANA_NIVEIS];
  NivelDev<float> n[SECAO_PLANA_NIVEIS];
  float* saida;
};
// t / k correctly rounded, as resolverGrosso's division, from i = 1/k rounded: t i is exact for 1, 2 and
// 4, and for 3 one correction by the residual t - 3 q rounds right (Markstein's theorem on the final
// step of a division; checked against t / 3.0f for all 2^23 significands).  An infinite quotient
// stays as it is.  No branch on k: one in the half-sweeps' loop took 137 of its 200 cycles.
__device__ __forceinline__ float dividirViz(float t, float k, float i) {
  const float q = t * i, r = fmaf(fmaf(-k, q, t), i, q);
  return fabsf(q) < INFINITY ? r : q;
}
__global__ void __launch_bounds__(T_SECAO) k_secao(SecaoPlana s) {
  // one array, addressed by offsets: x, the snapshots, the right sides, and a 0 for closed neighbours
  constexpr int S = SECAO_PLANA_TOTAL, B = 2 * SECAO_PLANA_TOTAL, ZERO = 3 * SECAO_PLANA_TOTAL;
  __shared__ float X[ZERO + 1];
  __shared__ uint8_t V[SECAO_PLANA_TOTAL];
  if (s.n[0].parar && *s.n[0].parar) return;
  const int t = threadIdx.x, nt = blockDim.x;
  for (int l = 0; l < s.L; l++) {
    const int N = s.n[l].nx * s.n[l].ny, o = s.off[l];
    for (int c = t; c < N; c += nt) {
      V[o + c] = s.n[l].viz[c];
      X[o + c] = X[S + o + c] = 0.0f;  // a pass takes the snapshots of the cells that change alone
      if (l == 0) X[B + o + c] = s.n[0].b[c];
    }
  }
  if (t == 0) X[ZERO] = 0.0f;
  __syncthreads();
  const float pes[4] = {0.25f, 0.75f, 0.75f, 0.25f};
  // The thread's two cells of a level (cells 2s and 2s + 1 of a row, colour e ^ ordem at [e]): index
  // (-1: none that changes), neighbours, free neighbours, right side.
  struct Par {
    int c[2], v[2][4], k[2];
    float b[2];
  };
  auto threads = [&](int l) { return (((s.n[l].nx + 1) >> 1) * s.n[l].ny + 31) & ~31; };
  auto par = [&](int l, int ordem, int desl, bool blocos) {  // desl: the blocks' shift; blocos: snapshots
    Par p;
    const int nx = s.n[l].nx, ny = s.n[l].ny, hw = (nx + 1) >> 1, o = s.off[l], j = t / hw;
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int i = 2 * (t % hw) + (((e ^ ordem) + 1 + j) & 1);
      const bool dentro = j < ny && i < nx;
      const int c = dentro ? o + i + j * nx : o, vz = dentro ? V[c] : 0, mk = vz & 15;
      const int bi = (i + desl) & 15, bj = (j + desl) & 15;
      // a neighbour of the cell's block is read as swept, one outside it from the snapshot
      p.c[e] = (vz & 16) && mk ? c : -1;
      p.v[e][0] = !(mk & 1) ? ZERO : (blocos && bi == 0 ? S : 0) + c - 1;
      p.v[e][1] = !(mk & 2) ? ZERO : (blocos && bi == 15 ? S : 0) + c + 1;
      p.v[e][2] = !(mk & 4) ? ZERO : (blocos && bj == 0 ? S : 0) + c - nx;
      p.v[e][3] = !(mk & 8) ? ZERO : (blocos && bj == 15 ? S : 0) + c + nx;
      p.k[e] = __popc(mk);
      p.b[e] = X[B + c];
    }
    return p;
  };
  auto sinc = [&](int n) {
    if (n == 32) __syncwarp();
    else asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory");
  };
  // one pass over level l by its first threads (whole warps over its cells)
  auto passo = [&](int l, int desl, int ordem) {
    const int n = threads(l);
    if (t >= n) return;
    const Par p = par(l, ordem, desl, true);
    float q[2], iq[2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
      q[e] = p.c[e] >= 0 ? X[p.c[e]] : 0.0f;
      iq[e] = inversoVizinhos(p.k[e]);
      if (p.c[e] >= 0) X[S + p.c[e]] = q[e];
    }
    sinc(n);
#pragma unroll 1
    for (int h = 0; h < VARREDURAS; h++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const float sm = ((X[p.v[e][0]] + X[p.v[e][1]]) + X[p.v[e][2]]) + X[p.v[e][3]];
        q[e] = q[e] + fmaf(sm + p.b[e], iq[e], -q[e]);
        if (p.c[e] >= 0) X[p.c[e]] = q[e];
        sinc(n);
      }
  };
  for (int l = 0; l < s.L - 1; l++) {
    if (!s.uma) {
      passo(l, 0, 0);
      __syncthreads();
    }
    passo(l, 8, 0);
    const int nx = s.n[l].nx, ny = s.n[l].ny, N = nx * ny, o = s.off[l];
    __syncthreads();
    for (int k = t; k < N; k += nt) {  // residuals into the snapshot array
      const int c = o + k, vz = V[c];
      float sm = 0.0f;
      sm += (vz & 1) ? X[c - 1] : 0.0f;
      sm += (vz & 2) ? X[c + 1] : 0.0f;
      sm += (vz & 4) ? X[c - nx] : 0.0f;
      sm += (vz & 8) ? X[c + nx] : 0.0f;
      X[S + c] = (vz & 16) ? X[B + c] - fmaf((float)__popc(vz & 15), X[c], -sm) : 0.0f;
    }
    __syncthreads();
    const int gx = s.n[l + 1].nx, G = gx * s.n[l + 1].ny, og = s.off[l + 1];
    for (int C = t; C < G; C += nt) {
      const int I = C % gx, J = C / gx;
      float sm = 0.0f;
      if (V[og + C] & 16)
#pragma unroll
        for (int bb = 0; bb < 4; bb++)
#pragma unroll
          for (int aa = 0; aa < 4; aa++) {
            const int i = 2 * I - 1 + aa, j = 2 * J - 1 + bb;
            if (i >= 0 && j >= 0 && i < nx && j < ny)
              sm = __fadd_rn(sm, __fmul_rn(X[S + o + i + j * nx], pes[aa] * pes[bb]));
          }
      X[B + og + C] = sm;
    }
    __syncthreads();
  }
  {  // resolverGrosso (js/pressao-cpu.js:217-238)
    const int n = threads(s.L - 1);
    if (t < n) {
      const Par p = par(s.L - 1, 0, 0, false);
      const float kf[2] = {(float)p.k[0], (float)p.k[1]};
      const float iq[2] = {inversoVizinhos(p.k[0]), inversoVizinhos(p.k[1])};
      auto meia = [&](auto E) {
        constexpr int e = decltype(E)::value;
        const float sm = ((X[p.v[e][0]] + X[p.v[e][1]]) + X[p.v[e][2]]) + X[p.v[e][3]];
        if (p.c[e] >= 0) X[p.c[e]] = dividirViz(sm + p.b[e], kf[e], iq[e]);
        sinc(n);
      };
#pragma unroll 1
      for (int h = 0; h < VARREDURAS_GROSSO / 2; h++) {
        meia(std::integral_constant<int, 0>{});
        meia(std::integral_constant<int, 1>{});
      }
      meia(std::integral_constant<int, 0>{});
    }
    __syncthreads();
  }
  for (int l = s.L - 2; l >= 0; l--) {
    const int nx = s.n[l].nx, N = nx * s.n[l].ny, o = s.off[l];
    const int gx = s.n[l + 1].nx, gy = s.n[l + 1].ny, og = s.off[l + 1];
    for (int k = t; k < N; k += nt) {
      if (!(V[o + k] & 16)) continue;
      const int i = k % nx, j = k / nx, I0 = grossoBaseF(i), J0 = grossoBaseF(j);
      const float wx0 = pesoBaseF(i), wy0 = pesoBaseF(j);
      float e = 0.0f;
#pragma unroll
      for (int b = 0; b < 2; b++)
#pragma unroll
        for (int a = 0; a < 2; a++) {
          const int I = I0 + a, J = J0 + b;
          if (I >= 0 && J >= 0 && I < gx && J < gy)
            e = fmaf(X[og + I + J * gx], (a ? 1.0f - wx0 : wx0) * (b ? 1.0f - wy0 : wy0), e);
        }
      X[o + k] = X[o + k] + e;
    }
    __syncthreads();
    passo(l, 8, 1);
    __syncthreads();
    if (!s.uma) {
      passo(l, 0, 1);
      __syncthreads();
    }
  }
  for (int c = t; c < s.n[0].nx * s.n[0].ny; c += nt) s.saida[c] = X[c];
}

// resolverGrosso (js/pressao-cpu.js:217-238): VARREDURAS_GROSSO alternating red-black sweeps
// in place on a coarsest level of more than SECAO_PLANA cells, from x = 0, one CTA; the level lives
// in shared memory when it fits.  65 half-sweeps as in k_secao.
template <class T>
__global__ void __launch_bounds__(1024) k_grosso(NivelDev<T> n, int emShared) {
  extern __shared__ unsigned char dyn[];
  if (n.parar && *n.parar) return;  // uniform over the CTA
  const int N = n.nx * n.ny, nx = n.nx;
  float* xs = (float*)dyn;
  float* bs = xs + N;
  uint8_t* vs = (uint8_t*)(bs + N);
  const uint8_t* viz = n.viz;
  if (emShared)
    for (int c = threadIdx.x; c < N; c += blockDim.x) {
      xs[c] = 0.0f;
      bs[c] = carregar(n.b[c]);
      vs[c] = viz[c];
    }
  else
    for (int c = threadIdx.x; c < N; c += blockDim.x) n.x[c] = guardar<T>(0.0f);
  __syncthreads();
  for (int h = 0; h <= VARREDURAS_GROSSO; h++) {
    const int cor = h & 1;
    for (int c = threadIdx.x; c < N; c += blockDim.x) {
      int i = c % nx, j = c / nx;
      int vz = emShared ? vs[c] : viz[c];
      if (!(vz & 16) || ((i + j + 1) & 1) != cor) continue;
      int q = __popc(vz & 15);
      if (!q) continue;
      auto x = [&](int k) { return emShared ? xs[k] : carregar(n.x[k]); };
      float s = 0.0f;
      if (vz & 1) s += x(c - 1);
      if (vz & 2) s += x(c + 1);
      if (vz & 4) s += x(c - nx);
      if (vz & 8) s += x(c + nx);
      const float r = dividirViz(s + (emShared ? bs[c] : carregar(n.b[c])), (float)q, inversoVizinhos(q));
      if (emShared) xs[c] = r;
      else n.x[c] = guardar<T>(r);
    }
    __syncthreads();
  }
  if (emShared)
    for (int c = threadIdx.x; c < N; c += blockDim.x) n.x[c] = guardar<T>(xs[c]);
}

// ---------------------------------------------------------------- PCG kernels
// Value a water cell's neighbour contributes to A*v (js/pressao-cpu.js:84-93 after difundir,
// :318-324): water -> v, air of an active bubble -> that bubble's value (as stored in the
// f32 grid), anything else -> 0.
__device__ inline float valorViz(const Dev& d, const float* v, const float* vbf, int n, bool bolhas) {
  uint8_t t = d.tipo[n];
  if (t == AGUA) return v[n];
  if (bolhas && t == AR) {
    uint32_t r = d.rotulo[n];
    if (r >= 2 && r < (uint32_t)MAX_BOLHAS && d.facesB[r] > 0) return vbf[r];
  }
  return 0.0f;
}
__device__ inline float aplicarA(const Dev& d, const uint8_t* vizOp, const float* v, const float* vbf, int c, bool bolhas) {
  int vz = vizOp[c];
  float s = 0.0f;
  if (vz & 1) s += valorViz(d, v, vbf, c - 1, bolhas);
  if (vz & 2) s += valorViz(d, v, vbf, c + 1, bolhas);
  if (vz & 4) s += valorViz(d, v, vbf, c - d.nx, bolhas);
  if (vz & 8) s += valorViz(d, v, vbf, c + d.nx, bolhas);
  return (float)__popc(vz & 15) * v[c] - s;
}

// r = -div - A q on water cells (js/pressao-cpu.js:331-338); q = 0 elsewhere.
__global__ void k_pcg_inicio(Dev d, const uint8_t* vizOp, int bolhas, double* q64) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.N) return;
  if (d.tipo[c] != AGUA) {
    d.q[c] = 0.0f;
    d.r[c] = 0.0f;
    return;
  }
  d.r[c] = -d.div[c] - aplicarA(d, vizOp, d.q, d.ybf, c, bolhas != 0);
  if (q64) q64[c] = (double)d.q[c];  // tolerance mode: the FP64 iterate
}

// Active bubbles (montarBolhas, js/pressao-cpu.js:271-288): faces = number of (interior bubble
// cell, water neighbour) pairs; cels = every air cell carrying an active label (:345-351).
__global__ void k_bolhas_faces(Dev d) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.N) return;
  const int nx = d.nx;
  int i = c % nx, j = c / nx;
  if (i < 1 || j < 1 || i >= nx - 1 || j >= d.ny - 1) return;
  uint32_t b = d.rotulo[c];
  if (b < 2 || b >= (uint32_t)MAX_BOLHAS || d.tipo[c] != AR) return;
  unsigned k = (d.tipo[c - 1] == AGUA) + (d.tipo[c + 1] == AGUA) + (d.tipo[c - nx] == AGUA) + (d.tipo[c + nx] == AGUA);
  if (k) atomicAdd(&d.facesB[b], k);
}
__global__ void k_bolhas_celulas(Dev d) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.N) return;
  uint32_t b = d.rotulo[c];
  if (b < 2 || b >= (uint32_t)MAX_BOLHAS || d.tipo[c] != AR || d.facesB[b] == 0) return;
  atomicAdd(&d.celsB[b], 1u);
}
// Initial bubble values: y from the caller (f32), zero for inactive labels.
__global__ void k_bolhas_inicio(Dev d) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= MAX_BOLHAS) return;
  bool at = b >= 2 && d.facesB[b] > 0;
  double y = at ? (double)d.yBolhaF[b] : 0.0;
  d.yB[b] = y;
  d.ybf[b] = (float)y;
  d.rb[b] = d.zb[b] = d.zvb[b] = d.pb[b] = d.apb[b] = 0.0;
  d.pbf[b] = 0.0f;
}

// Bubble rows of A*v (aplicarBolhas, js/pressao-cpu.js:325-328): out[b] = faces[b]*vb[b] -
// sum over the bubble's water faces of v[water cell].  The sum is 64-bit fixed point (2^-40).
constexpr double ESCALA_PCG = 1099511627776.0;  // 2^40
__global__ void k_bolhas_somar_v(Dev d, const float* v) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.N || d.esc->pronto) return;
  const int nx = d.nx;
  int i = c % nx, j = c / nx;
  if (i < 1 || j < 1 || i >= nx - 1 || j >= d.ny - 1) return;
  uint32_t b = d.rotulo[c];
  if (b < 2 || b >= (uint32_t)MAX_BOLHAS || d.tipo[c] != AR) return;
  double s = 0;
  if (d.tipo[c - 1] == AGUA) s += (double)v[c - 1];
  if (d.tipo[c + 1] == AGUA) s += (double)v[c + 1];
  if (d.tipo[c - nx] == AGUA) s += (double)v[c - nx];
  if (d.tipo[c + nx] == AGUA) s += (double)v[c + nx];
  if (s != 0) somaFixa(&d.accB[b], s, ESCALA_PCG);
}
// modo 0: rb = rhs - (faces*y - sum)  (initial bubble residual, :339-341)
// modo 1: apb = faces*pb - sum
__global__ void k_bolhas_linhas(Dev d, int modo) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= MAX_BOLHAS || d.esc->pronto) return;
  if (b < 2 || d.facesB[b] == 0) return;
  double soma = (double)d.accB[b] / ESCALA_PCG;
  if (modo == 0) d.rb[b] = (double)d.rhsBolhaF[b] - (d.facesB[b] * d.yB[b] - soma);
  else d.apb[b] = d.facesB[b] * d.pb[b] - soma;
}

// Level 0's right side made from F on a grid of one level (k_descer makes it elsewhere).
template <class T>
__global__ void k_fonte(NivelDev<T> n0, Fonte F) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n0.nx * n0.ny || (n0.parar && *n0.parar)) return;
  float v = F.v[c];
  if (n0.viz[c] & V0_BOLHA) v = (float)(F.rb[F.rotulo[c]] / F.celsB[F.rotulo[c]]);
  n0.b[c] = guardar<T>(v * (F.escala ? (float)*F.escala : 1.0f));
}
// After the V-cycle (precondicionar, js/pressao-cpu.js:357-361): z = x, except active bubble
// cells, whose mean correction becomes the bubble's z (the transpose of spreading) and whose grid
// value is zeroed.
template <class T>
__global__ void k_pre_juntar(Dev d, const uint8_t* viz0, const T* x0) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.N || d.esc->pronto) return;
  float inv = (float)(1.0 / d.esc->escalaMG);
  float x = carregar(x0[c]) * inv;
  if (viz0[c] & V0_BOLHA) {
    const uint32_t b = d.rotulo[c];
    somaFixa(&d.accB[b], (double)x / d.celsB[b], ESCALA_PCG);
    d.z[c] = 0.0f;
    return;
  }
  d.z[c] = x;
}
// The bubbles' z: the gathered mean correction, or with TQ_PRECOND_BLOCK (bloco) a Jacobi step on
// the bubble's row, r_b / faces_b.
__global__ void k_pre_bolhas(Dev d, int bloco) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= MAX_BOLHAS || d.esc->pronto) return;
  const bool at = b >= 2 && d.facesB[b] > 0;
  d.zb[b] = !at ? 0.0 : bloco ? d.rb[b] / (double)d.facesB[b] : (double)d.accB[b] / ESCALA_PCG;
}

// ap = A p on water cells (js/pressao-cpu.js:367-373).
__global__ void k_aplicar(Dev d, const uint8_t* vizOp, int bolhas) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.N || d.esc->pronto) return;
  d.ap[c] = d.tipo[c] == AGUA ? aplicarA(d, vizOp, d.p, d.pbf, c, bolhas != 0) : 0.0f;
}

// q += alpha p, r -= alpha Ap on water; bubbles likewise (js/pressao-cpu.js:377-385).
__global__ void k_atualizar(Dev d, double* q64) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (d.esc->pronto) return;
  double alfa = d.esc->alpha;
  if (c < MAX_BOLHAS && c >= 2 && d.facesB[c] > 0) {
    d.yB[c] += alfa * d.pb[c];
    d.rb[c] -= alfa * d.apb[c];
    d.ybf[c] = (float)d.yB[c];
  }
  if (c >= d.N || d.tipo[c] != AGUA) return;
  float a = (float)alfa;
  if (q64) q64[c] += alfa * (double)d.p[c];
  else d.q[c] = d.q[c] + a * d.p[c];
  d.r[c] = d.r[c] - a * d.ap[c];
}

__device__ inline double somaBloco(double v, double* sh);  // block sum (valid in thread 0), below

// Tolerance mode replaces the recursive FP32 residual by the true one each time the recursive one
// has fallen by this factor since the last replacement (as the fused engine and the oracle do).
constexpr double FATOR_TROCA = 1e-3;

// Tolerance mode, once the recursive residual met the tolerance (Escalares::verificar): the true
// residual in FP64 from the FP64 iterate and the bubble pressures.  Water cells: rt = -div - A q
// into d.ap (free until the next A p) and rt^2 into per-CTA partials; interior air of active
// bubbles: the sum of q over its water faces into the bubble's fixed-point sum (accB, zeroed
// before).  k_verdade_fim finishes the norm and decides.
__global__ void __launch_bounds__(256) k_verdade(Dev d, const uint8_t* vizOp, const double* q64, int bolhas) {
  __shared__ double sh[32];
  if (!d.esc->verificar || d.esc->pronto) return;  // uniform over the grid
  double s = 0;
  const int nx = d.nx;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < d.N; c += gridDim.x * blockDim.x) {
    const uint8_t t = d.tipo[c];
    if (t == AGUA) {
      const int vz = vizOp[c];
      double sv = 0;
      const int nb[4] = {c - 1, c + 1, c - nx, c + nx};
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (!(vz & (1 << q))) continue;
        const uint8_t tn = d.tipo[nb[q]];
        if (tn == AGUA) sv += q64[nb[q]];
        else if (bolhas && tn == AR) {
          const uint32_t r = d.rotulo[nb[q]];
          if (r >= 2 && r < (uint32_t)MAX_BOLHAS && d.facesB[r] > 0) sv += d.yB[r];
        }
      }
      const double rt = -(double)d.div[c] - ((double)__popc(vz & 15) * q64[c] - sv);
      d.ap[c] = (float)rt;
      s += rt * rt;
    } else if (bolhas && t == AR) {
      const int i = c % nx, j = c / nx;
      if (i < 1 || j < 1 || i >= nx - 1 || j >= d.ny - 1) continue;
      const uint32_t b = d.rotulo[c];
      if (b < 2 || b >= (uint32_t)MAX_BOLHAS || d.facesB[b] == 0) continue;
      double t2 = 0;
      if (d.tipo[c - 1] == AGUA) t2 += q64[c - 1];
      if (d.tipo[c + 1] == AGUA) t2 += q64[c + 1];
      if (d.tipo[c - nx] == AGUA) t2 += q64[c - nx];
      if (d.tipo[c + nx] == AGUA) t2 += q64[c + nx];
      if (t2 != 0) somaFixa(&d.accB[b], t2, ESCALA_PCG);
    }
  }
  const double tb = somaBloco(s, sh);
  if (threadIdx.x == 0) d.parciais[2 * blockIdx.x] = tb;
}
// One CTA: the true norm (partials in block order, then the bubble rows rhs - (faces y - sum)),
// and the decision: converged or at the cap -> pronto; else the bubble rows take their true
// residual, reiniciar is set (k_substituir copies the water part into r).
__global__ void __launch_bounds__(256) k_verdade_fim(Dev d, int blocosVerdade, int cap, double tol, int bolhas,
                                                    int meiaPrecisao) {
  __shared__ double sh[32];
  __shared__ int substituir;
  Escalares* e = d.esc;
  if (!e->verificar || e->pronto) return;
  double p1 = 0, q1 = 0;
  for (int k = threadIdx.x; k < blocosVerdade; k += blockDim.x) p1 += d.parciais[2 * k];
  auto rbv = [&](int b) { return (double)d.rhsBolhaF[b] - (d.facesB[b] * d.yB[b] - (double)d.accB[b] / ESCALA_PCG); };
  if (bolhas)
    for (int b = threadIdx.x; b < MAX_BOLHAS; b += blockDim.x)
      if (b >= 2 && d.facesB[b] > 0) {
        const double v = rbv(b);
        q1 += v * v;
      }
  const double T1 = somaBloco(p1, sh), B1 = somaBloco(q1, sh);
  if (threadIdx.x == 0) {
    const double nv = sqrt(T1 + B1);
    const bool ok = nv <= tol * e->norma0;
    e->normaVerd = nv;
    e->verificar = 0;
    substituir = 0;
    if (ok || e->iters >= cap) {
      e->pronto = 1;
      e->convergiu = ok ? 1 : 0;
    } else {
      e->reiniciar = 1;
      e->trocas++;
      e->proxTroca = nv * FATOR_TROCA;
      e->norma = nv;
      e->escalaMG = (meiaPrecisao && nv > 0) ? 1.0 / nv : 1.0;
      substituir = 1;
    }
  }
  __syncthreads();
  if (substituir && bolhas)
    for (int b = threadIdx.x; b < MAX_BOLHAS; b += blockDim.x)
      if (b >= 2 && d.facesB[b] > 0) d.rb[b] = rbv(b);
}
// After a replacement: r = the true residual on water cells.
__global__ void k_substituir(Dev d) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.N || !d.esc->reiniciar || d.esc->pronto) return;
  if (d.tipo[c] == AGUA) d.r[c] = d.ap[c];
}

// p = z + beta p on water (0 elsewhere); bubbles likewise (js/pressao-cpu.js:395-396).
__global__ void k_direcao(Dev d) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (d.esc->pronto) return;
  double beta = d.esc->beta;
  if (c < MAX_BOLHAS && c >= 2 && d.facesB[c] > 0) {
    d.pb[c] = d.zb[c] + beta * d.pb[c];
    d.pbf[c] = (float)d.pb[c];
  }
  if (c >= d.N) return;
  d.p[c] = d.tipo[c] == AGUA ? d.z[c] + (float)beta * d.p[c] : 0.0f;
}
// p = z, pb = zb (js/pressao-cpu.js:363-364)
__global__ void k_copiar_pz(Dev d) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < MAX_BOLHAS) {
    d.pb[c] = d.zb[c];
    d.pbf[c] = (float)d.zb[c];
    d.zvb[c] = 0.0;
  }
  if (c < d.N) d.p[c] = d.z[c];
}
// zOld = z, zvb = zb (js/pressao-cpu.js:388-389)
__global__ void k_guardar_z(Dev d) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (d.esc->pronto) return;
  if (c < MAX_BOLHAS) d.zvb[c] = d.zb[c];
  if (c < d.N) d.zOld[c] = d.z[c];
}
// End of the solve: non-water q = 0; bubbles hand back their pressure (js/pressao-cpu.js:399-400).
// Tolerance mode: q = the FP64 iterate rounded; the solve's convergence record (thread 0).
__global__ void k_pcg_fim(Dev d, int bolhas, const double* q64, double tol) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (bolhas && c >= 2 && c < MAX_BOLHAS && d.facesB[c] > 0) d.yBolhaF[c] = (float)d.yB[c];
  if (c < d.N) {
    if (d.tipo[c] != AGUA) d.q[c] = 0.0f;
    else if (q64) d.q[c] = (float)q64[c];
  }
  if (c == 0) {
    Escalares* e = d.esc;
    if (!q64) {
      e->normaVerd = -1.0;
      e->convergiu = 0;
    }
    e->solves++;
    if (q64 && !e->convergiu) e->capados++;
    e->itersAcum += e->iters;
    e->trocasAcum += e->trocas;
    if (q64 && e->norma0 > 0 && e->normaVerd / e->norma0 > e->maxRel) e->maxRel = e->normaVerd / e->norma0;
  }
}

// ---------------------------------------------------------------- dot products
// Two FP64 dot products over water cells (a*b1, a*b2) plus the bubble terms, in a fixed
// reduction order; the last block to finish does the scalar step of the running solve.
enum ModoProduto { NORMA0 = 0, RZ0 = 1, PAP = 2, NORMA = 3, BETA = 4 };

constexpr int DOT_BLOCOS = 296;
constexpr int DOT_T = 256;

__device__ inline double somaBloco(double v, double* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double t = 0;
  if (w == 0) {
    t = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  }
  __syncthreads();
  return t;  // valid in thread 0
}

__global__ void __launch_bounds__(DOT_T) k_produto(Dev d, int modo, const float* a, const float* b1, const float* b2,
                                                 int it, double tol, int bolhas, int meiaPrecisao, int cap) {
  __shared__ double sh[32];
  __shared__ bool ultimo;
  if (modo != NORMA0 && d.esc->pronto) return;  // uniform over the grid
  double s1 = 0, s2 = 0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < d.N; c += gridDim.x * blockDim.x) {
    if (d.tipo[c] != AGUA) continue;
    double av = a[c];
    s1 += av * (double)b1[c];
    if (b2) s2 += av * (double)b2[c];
  }
  double t1 = somaBloco(s1, sh);
  double t2 = b2 ? somaBloco(s2, sh) : 0.0;
  if (threadIdx.x == 0) {
    d.parciais[2 * blockIdx.x] = t1;
    d.parciais[2 * blockIdx.x + 1] = t2;
    __threadfence();
    unsigned v = atomicAdd(&d.esc->tickets[0], 1u);
    ultimo = v == gridDim.x - 1;
  }
  __syncthreads();
  if (!ultimo) return;
  __threadfence();
  // the last block: partials in block order, then the bubble terms in label order
  double p1 = 0, p2 = 0;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) {
    p1 += __ldcg(&d.parciais[2 * k]);
    p2 += __ldcg(&d.parciais[2 * k + 1]);
  }
  double q1 = 0, q2 = 0;
  if (bolhas) {
    for (int b = threadIdx.x; b < MAX_BOLHAS; b += blockDim.x) {
      if (b < 2 || d.facesB[b] == 0) continue;
      switch (modo) {
        case NORMA0:
        case NORMA: q1 += d.rb[b] * d.rb[b]; break;
        case RZ0: q1 += d.rb[b] * d.zb[b]; break;
        case PAP: q1 += d.pb[b] * d.apb[b]; break;
        case BETA: q1 += d.rb[b] * d.zb[b]; q2 += d.rb[b] * d.zvb[b]; break;
      }
    }
  }
  double T1 = somaBloco(p1, sh), T2 = somaBloco(p2, sh);
  double B1 = somaBloco(q1, sh), B2 = somaBloco(q2, sh);
  if (threadIdx.x == 0) {
    Escalares* e = d.esc;
    e->tickets[0] = 0;
    double x1 = T1 + B1, x2 = T2 + B2;
    switch (modo) {
      case NORMA0: {
        double nr = sqrt(x1);
        e->norma0 = e->norma = nr;
        e->normas[0] = nr;
        e->iters = 0;
        e->pronto = 0;
        e->verificar = 0;
        e->reiniciar = 0;
        e->trocas = 0;
        e->convergiu = 0;
        e->normaVerd = -1.0;
        e->proxTroca = nr * FATOR_TROCA;
        e->escalaMG = (meiaPrecisao && nr > 0) ? 1.0 / nr : 1.0;
        break;
      }
      case RZ0: e->rz = x1; break;
      case PAP: e->pap = x1; e->alpha = fabs(x1) < 1e-30 ? 0.0 : e->rz / x1; break;
      case NORMA: {
        double nr = sqrt(x1);
        e->norma = nr;
        if (it + 1 < 1024) e->normas[it + 1] = nr;
        e->iters = it + 1;
        // tolerance mode: the recursive residual met the tolerance, or fell by FATOR_TROCA since
        // the last replacement, or the cap came: the true residual decides (k_verdade,
        // k_verdade_fim)
        e->verificar = tol > 0 && (nr <= tol * e->norma0 || nr <= e->proxTroca || it + 1 >= cap);
        e->escalaMG = (meiaPrecisao && nr > 0) ? 1.0 / nr : 1.0;
        break;
      }
      case BETA: {
        double rzNovo = x1, cruzado = x2;
        // (after a residual replacement the direction carries on: no restart)
        e->beta = fabs(e->rz) < 1e-30 ? 0.0 : fmax(0.0, (rzNovo - cruzado) / e->rz);
        e->reiniciar = 0;
        e->rz = rzNovo;
        break;
      }
    }
  }
}

// ---------------------------------------------------------------- the solver object


Pcg* criarPcg(int nx, int ny, int precisao, int motor, int ctasFundido) {
  Pcg* p = new Pcg();
  p->ctasFundido = ctasFundido;
  p->nx = nx;
  p->ny = ny;
  p->N = nx * ny;
  p->precisao = precisao;
  p->motor = motor;
  // montarNiveis (js/pressao-cpu.js:24-41): halve (ceil) while min(nx, ny) > 12
  int L = 0;
  int a = nx, b = ny;
  p->nxL[0] = a;
  p->nyL[0] = b;
  L = 1;
  while ((a < b ? a : b) > 12 && L < MAX_NIVEIS) {
    a = (a + 1) / 2;
    b = (b + 1) / 2;
    p->nxL[L] = a;
    p->nyL[L] = b;
    L++;
  }
  p->L = L;
  bool ok = true;
  for (int l = 0; l < L; l++) {
    size_t n = (size_t)p->nxL[l] * p->nyL[l];
    p->meia[l] = precisao != TQ_PREC_FP32 && n >= (size_t)MEIA_MIN_CELULAS;
    const size_t e = 4;  // room for FP32 whatever the engine stores
    ok &= cudaMalloc(&p->tipoL[l], n) == cudaSuccess;
    ok &= cudaMalloc(&p->vizL[l], n) == cudaSuccess;
    ok &= cudaMalloc(&p->bL[l], n * e) == cudaSuccess;
    ok &= cudaMalloc(&p->xL[l], n * e) == cudaSuccess;
    ok &= cudaMalloc(&p->tmpL[l], n * e) == cudaSuccess;
  }
  ok &= cudaMalloc(&p->vizOp, p->N) == cudaSuccess;
  size_t nc = (size_t)p->nxL[L - 1] * p->nyL[L - 1];
  p->smemGrosso = nc * 9 <= 200 * 1024 ? nc * 9 : 0;
  if (p->smemGrosso) {
    // The attribute is per kernel, shared by every solver in the process: it is always raised
    // to the 200 KB cap, never set to this grid's size, which would fail the launches of a
    // solver on a grid with a larger coarsest level.
    auto subir = [](auto* k) {
      return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) == cudaSuccess;
    };
    if (!subir(k_grosso<float>) || !subir(k_grosso<__half>) || !subir(k_grosso<__nv_bfloat16>)) p->smemGrosso = 0;
  }
  if (ok && motor == TQ_ENGINE_FUSED) {
    // Grids with a single level (min(nx, ny) <= 12) have nothing to hand to the coarse
    // section: they run on the plain engine.
    p->fundido = criarFundido(p);
    if (!p->fundido) {
      cudaGetLastError();
      p->motor = TQ_ENGINE_PLAIN;
    }
  }
  if (!ok) {
    destruirPcg(p);
    return nullptr;
  }
  return p;
}

void destruirPcg(Pcg* p) {
  if (!p) return;
  destruirFundido(p->fundido);
  for (int l = 0; l < p->L; l++) {
    cudaFree(p->tipoL[l]);
    cudaFree(p->vizL[l]);
    cudaFree(p->bL[l]);
    cudaFree(p->xL[l]);
    cudaFree(p->tmpL[l]);
  }
  cudaFree(p->vizOp);
  if (p->q64) cudaFree(p->q64);
  destruirRegioes(p->regioes);
  delete p;
}

// Level descriptor with the storage type chosen at run time.
template <class T>
static NivelDev<T> nivel(Pcg* p, int l) {
  NivelDev<T> n;
  n.nx = p->nxL[l];
  n.ny = p->nyL[l];
  n.tipo = p->tipoL[l];
  n.viz = p->vizL[l];
  n.b = (T*)p->bL[l];
  n.x = (T*)p->xL[l];
  n.tmp = (T*)p->tmpL[l];
  n.parar = p->parar;
  return n;
}

// Dispatch on the storage type of level l.
template <class F>
static void comTipo(Pcg* p, int l, F f) {
  if (!p->meia[l]) f((float*)nullptr);
  else if (p->precisao == TQ_PREC_FP16) f((__half*)nullptr);
  else f((__nv_bfloat16*)nullptr);
}

// Dispatch on the storage types of levels l and l + 1 (16-bit down to some level, FP32 below it).
template <class F>
static void comTipos(Pcg* p, int l, F f) {
  comTipo(p, l, [&](auto* tf) {
    if (p->meia[l] && p->meia[l + 1]) f(tf, tf);
    else f(tf, (float*)nullptr);
  });
}

// The tile of a leg: by blocks a side, the launch's length in rounds of block sweeps, a CTA an SM
// (two of the smallest tile's) with 16 warps, is waves x rounds; the shortest wins, the smaller tile
// of equals (a smaller tile sweeps more blocks around it, a larger one leaves SMs without a tile).
static int escolherLadrilho(int nx, int ny, bool subir, bool uma) {
  constexpr int SMS = 148;
  int melhor = 1;
  long custo = -1;
  for (int k = 1; k <= 4; k++) {
    const long n = (long)blocos(nx, 16 * k) * blocos(ny, 16 * k);
    const long ondas = (n + SMS * (k == 1 ? 2 : 1) - 1) / (SMS * (k == 1 ? 2 : 1));
    auto voltas = [&](int b) { return (b * b + (k == 1 ? 8 : 15)) / (k == 1 ? 9 : 16); };
    const int r = uma ? voltas(subir ? k : k + 1) : subir ? voltas(k + 1) + voltas(k) : voltas(k + 2) + voltas(k + 1);
    const long c = ondas * (r + 2);
    if (custo < 0 || c < custo) {
      custo = c;
      melhor = k;
    }
  }
  return melhor;
}

template <class K>
static size_t prepararLadrilho(K kern, int k) {
  const size_t b = bytesLadrilho(k, k);
  if (b > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytesLadrilho(4, 4));
  return b;
}
static int threadsLadrilho(int k) { return k == 1 ? 288 : T_LADRILHO; }

// masc: the coarse levels of TQ_PRECOND_BLOCK, whose masks close faces between water cells
static void descerNivel(Pcg* p, int l, bool bloco, bool uma, const Fonte& F, cudaStream_t s) {
  uma = uma && l >= 1;
  const int k = escolherLadrilho(p->nxL[l], p->nyL[l], false, uma);
  const dim3 gr(blocos(p->nxL[l], 16 * k), blocos(p->nyL[l], 16 * k));
  comTipos(p, l, [&](auto* tf, auto* tg) {
    using TF = std::remove_pointer_t<decltype(tf)>;
    using TG = std::remove_pointer_t<decltype(tg)>;
    const NivelDev<TF> f = nivel<TF>(p, l);
    const NivelDev<TG> g = nivel<TG>(p, l + 1);
    auto kern = l == 0 ? k_descer<TF, TG, true> : k_descer<TF, TG, false>;
    const size_t b = prepararLadrilho(kern, k);
    lanca(kern, gr, threadsLadrilho(k), b, s, f, g, k, k, uma ? 1 : 0, bloco && l >= 1 ? 1 : 0, F);
  });
}
// xg: the coarse level's x (its result)
static void subirNivel(Pcg* p, int l, const void* xg, bool bloco, bool uma, float* saida, cudaStream_t s) {
  uma = uma && l >= 1;
  const int k = escolherLadrilho(p->nxL[l], p->nyL[l], true, uma), d = uma ? 8 : 0;
  const dim3 gr(blocos(p->nxL[l] + d, 16 * k), blocos(p->nyL[l] + d, 16 * k));
  comTipos(p, l, [&](auto* tf, auto* tg) {
    using TF = std::remove_pointer_t<decltype(tf)>;
    using TG = std::remove_pointer_t<decltype(tg)>;
    const size_t b = prepararLadrilho(k_subir<TF, TG>, k);
    lanca(k_subir<TF, TG>, gr, threadsLadrilho(k), b, s, nivel<TF>(p, l), nivel<TG>(p, l + 1), (const TG*)xg, k, k,
          uma ? 1 : 0, bloco && l >= 1 ? 1 : 0, saida);
  });
}

// cicloV (js/pressao-cpu.js:241-255) on a right side made from F (level 0's b is written); every
// level's result ends in its tmp, level 0's returned, or as floats in saida when there is one.
// umaPassada (TQ_PRECOND_BLOCK_1): the levels above 0 take one smoother pass a leg (shift 8).
static const void* cicloV(Pcg* p, const Fonte& F, cudaStream_t s, bool bloco, bool umaPassada, float* saida) {
  const int L = p->L;
  // the section: the coarse levels of at most SECAO_PLANA cells (not level 0)
  int Ls = L, total = 0;
  while (Ls > 1 && L - Ls < SECAO_PLANA_NIVEIS && p->nxL[Ls - 1] * p->nyL[Ls - 1] <= SECAO_PLANA &&
         ((p->nxL[Ls - 1] + 1) / 2) * p->nyL[Ls - 1] <= T_SECAO &&
         total + p->nxL[Ls - 1] * p->nyL[Ls - 1] <= SECAO_PLANA_TOTAL)
    Ls--, total += p->nxL[Ls] * p->nyL[Ls];
  const int Lf = Ls < L ? Ls : L - 1;  // the levels with tile legs: 0 .. Lf - 1
  for (int l = 0; l < Lf; l++) descerNivel(p, l, bloco, umaPassada, F, s);
  const void* x;
  if (Ls < L) {
    SecaoPlana sp{};
    sp.L = L - Ls;
    sp.uma = umaPassada ? 1 : 0;
    int off = 0;
    for (int l = Ls; l < L; l++) {
      sp.n[l - Ls] = nivel<float>(p, l);
      sp.off[l - Ls] = off;
      off += p->nxL[l] * p->nyL[l];
    }
    sp.saida = (float*)p->tmpL[Ls];
    x = sp.saida;
    lanca(k_secao, 1, (((p->nxL[Ls] + 1) / 2) * p->nyL[Ls] + 31) & ~31, 0, s, sp);
  } else {
    comTipo(p, L - 1, [&](auto* t) {
      using T = std::remove_pointer_t<decltype(t)>;
      lanca(k_grosso<T>, 1, 1024, p->smemGrosso, s, nivel<T>(p, L - 1), p->smemGrosso ? 1 : 0);
    });
    x = p->xL[L - 1];
  }
  for (int l = Lf - 1; l >= 0; l--) {
    subirNivel(p, l, x, bloco, umaPassada, l == 0 ? saida : nullptr, s);
    x = p->tmpL[l];
  }
  return x;
}

static void fonteNivelUnico(Pcg* p, const Fonte& F, cudaStream_t s) {
  if (p->L > 1) return;
  comTipo(p, 0, [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    lanca(k_fonte<T>, blocos(p->N, 256), 256, 0, s, nivel<T>(p, 0), F);
  });
}

// Types and neighbour masks of every level for this solve (bloco: TQ_PRECOND_BLOCK's coarse
// masks from the fine faces).
static void prepararNiveis(Pcg* p, const uint8_t* tipo0, bool bloco, cudaStream_t s, bool comNivel0 = true) {
  if (tipo0 != p->tipoL[0]) cudaMemcpyAsync(p->tipoL[0], tipo0, p->N, cudaMemcpyDeviceToDevice, s);
  Niveis n{};
  n.L = p->L;
  const int l0 = comNivel0 ? 0 : 1;
  for (int l = 0; l < p->L; l++) {
    n.nx[l] = p->nxL[l];
    n.ny[l] = p->nyL[l];
    n.tipo[l] = p->tipoL[l];
    n.viz[l] = p->vizL[l];
    n.ini[l + 1] = n.ini[l] + (l >= l0 ? n.nx[l] * n.ny[l] : 0);
  }
  for (int l = 0; l < p->L - 1; l += NIVEIS_POR_VEZ)
    lanca(k_niveis_tipos, dim3(blocos(n.nx[l], 64), blocos(n.ny[l], 64)), 256, 0, s, n, l);
  if (n.ini[p->L] > 0) lanca(k_niveis_viz, blocos(n.ini[p->L], 256), 256, 0, s, n, l0, bloco ? 1 : 0);
}

static void precondicionar(Pcg* p, const Dev& d, bool bolhas, bool bloco, bool umaPassada, cudaStream_t s) {
  int nb = blocos(d.N, 256);
  Fonte F{d.r, &d.esc->escalaMG, d.rotulo, d.rb, d.celsB};
  fonteNivelUnico(p, F, s);
  const void* x = cicloV(p, F, s, bloco, umaPassada, nullptr);
  const bool espalhar = bolhas && !bloco;  // with BLOCK the V-cycle does not see the bubbles
  if (espalhar) cudaMemsetAsync(d.accB, 0, MAX_BOLHAS * sizeof(long long), s);
  comTipo(p, 0, [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    lanca(k_pre_juntar<T>, nb, 256, 0, s, d, p->vizL[0], (const T*)x);
  });
  if (bolhas) lanca(k_pre_bolhas, blocos(MAX_BOLHAS, 256), 256, 0, s, d, bloco ? 1 : 0);
}

static void produto(Pcg* p, const Dev& d, int modo, const float* a, const float* b1, const float* b2, int it,
                    double tol, bool bolhas, int cap, cudaStream_t s) {
  lanca(k_produto, DOT_BLOCOS, DOT_T, 0, s, d, modo, a, b1, b2, it, tol, bolhas ? 1 : 0,
        p->precisao != TQ_PREC_FP32 ? 1 : 0, cap);
}

// Iterations the plain engine queues between two reads of the stop flag.  Every kernel of an
// iteration returns at once after the flag is set, so the result is the same as stopping at the
// exact iteration, with one host round trip per LOTE_VERIFICACAO iterations instead of one each.
constexpr int LOTE_VERIFICACAO = 8;

int reservarTolerancia(Pcg* p) {
  if (!p->regioes && !(p->regioes = criarRegioes(p->N))) return TQ_E_NOMEM;
  if (p->motor != TQ_ENGINE_FUSED && !p->q64 && cudaMalloc(&p->q64, (size_t)p->N * sizeof(double)) != cudaSuccess)
    return TQ_E_NOMEM;
  return TQ_OK;
}

int resolverPressao(Pcg* p, const Dev& d0, int iteracoes, double tol, bool bolhas, int precond, cudaStream_t s) {
  Dev d = d0;
  double* q64 = nullptr;
  if (tol > 0) {
    if (reservarTolerancia(p)) return TQ_E_NOMEM;
    projetarFechadas(p->regioes, d0, bolhas, s, &d);  // d reads the projected right-hand sides
    q64 = p->q64;
  }
  if (p->motor == TQ_ENGINE_FUSED) return resolverPressaoFundido(p, d, iteracoes, tol, bolhas, precond, s);
  const bool bloco = precond == TQ_PRECOND_BLOCK || precond == TQ_PRECOND_BLOCK_1;
  const bool umaPassada = precond == TQ_PRECOND_BLOCK_1;
  const int nb = blocos(d.N, 256);
  const int nbx = blocos(d.N > MAX_BOLHAS ? d.N : MAX_BOLHAS, 256);
  // operator (true types) and preconditioner types
  lanca(k_mg_tipo0, nb, 256, 0, s, d.tipo, d.rotulo, p->tipoL[0], p->vizOp, d.nx, d.ny, bolhas ? 1 : 0, bloco ? 1 : 0);
  prepararNiveis(p, p->tipoL[0], bloco, s, false);
  cudaMemsetAsync(d.facesB, 0, MAX_BOLHAS * sizeof(uint32_t), s);
  cudaMemsetAsync(d.celsB, 0, MAX_BOLHAS * sizeof(uint32_t), s);
  // the previous solve left its stop flag set: clear it before the first kernel that tests it
  // (the initial bubble sums and rows below; NORMA0 resets the rest of the record)
  cudaMemsetAsync(&d.esc->pronto, 0, sizeof(int), s);
  if (bolhas) {
    lanca(k_bolhas_faces, nb, 256, 0, s, d);
    lanca(k_bolhas_celulas, nb, 256, 0, s, d);
  }
  lanca(k_viz0, nb, 256, 0, s, d, p->tipoL[0], p->vizL[0], bolhas && !bloco ? 1 : 0);
  lanca(k_bolhas_inicio, blocos(MAX_BOLHAS, 256), 256, 0, s, d);
  lanca(k_pcg_inicio, nb, 256, 0, s, d, p->vizOp, bolhas ? 1 : 0, q64);
  if (bolhas) {
    cudaMemsetAsync(d.accB, 0, MAX_BOLHAS * sizeof(long long), s);
    lanca(k_bolhas_somar_v, nb, 256, 0, s, d, d.q);
    lanca(k_bolhas_linhas, blocos(MAX_BOLHAS, 256), 256, 0, s, d, 0);
  }
  produto(p, d, NORMA0, d.r, d.r, nullptr, 0, tol, bolhas, iteracoes, s);
  p->parar = &d.esc->pronto;  // the V-cycle kernels return once the solve has stopped
  precondicionar(p, d, bolhas, bloco, umaPassada, s);
  lanca(k_copiar_pz, nbx, 256, 0, s, d);
  produto(p, d, RZ0, d.r, d.z, nullptr, 0, tol, bolhas, iteracoes, s);
  int it = 0;
  for (; it < iteracoes; it++) {
    lanca(k_aplicar, nb, 256, 0, s, d, p->vizOp, bolhas ? 1 : 0);
    if (bolhas) {
      cudaMemsetAsync(d.accB, 0, MAX_BOLHAS * sizeof(long long), s);
      lanca(k_bolhas_somar_v, nb, 256, 0, s, d, d.p);
      lanca(k_bolhas_linhas, blocos(MAX_BOLHAS, 256), 256, 0, s, d, 1);
    }
    produto(p, d, PAP, d.p, d.ap, nullptr, it, tol, bolhas, iteracoes, s);
    lanca(k_atualizar, nbx, 256, 0, s, d, q64);
    produto(p, d, NORMA, d.r, d.r, nullptr, it, tol, bolhas, iteracoes, s);
    if (q64) {  // the true residual, when NORMA found the recursive one within the tolerance
      if (bolhas) cudaMemsetAsync(d.accB, 0, MAX_BOLHAS * sizeof(long long), s);
      lanca(k_verdade, DOT_BLOCOS, 256, 0, s, d, p->vizOp, q64, bolhas ? 1 : 0);
      lanca(k_verdade_fim, 1, 256, 0, s, d, DOT_BLOCOS, iteracoes, tol, bolhas ? 1 : 0,
            p->precisao != TQ_PREC_FP32 ? 1 : 0);
      lanca(k_substituir, nb, 256, 0, s, d);
    }
    if (it == iteracoes - 1) break;
    if (tol > 0 && it % LOTE_VERIFICACAO == LOTE_VERIFICACAO - 1) {
      int pronto = 0;
      if (cudaMemcpyAsync(&pronto, &d.esc->pronto, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
          cudaStreamSynchronize(s) != cudaSuccess) {
        p->parar = nullptr;
        return TQ_E_CUDA;
      }
      if (pronto) break;
    }
    lanca(k_guardar_z, nbx, 256, 0, s, d);
    precondicionar(p, d, bolhas, bloco, umaPassada, s);
    produto(p, d, BETA, d.r, d.z, d.zOld, it, tol, bolhas, iteracoes, s);
    lanca(k_direcao, nbx, 256, 0, s, d);
  }
  p->parar = nullptr;
  lanca(k_pcg_fim, nbx, 256, 0, s, d, bolhas ? 1 : 0, q64, tol);
  return cudaGetLastError() == cudaSuccess ? TQ_OK : TQ_E_CUDA;
}

// The residual history of the last solve (Escalares::normas), read from the device.
int normasPcg(Pcg* p, const Dev& d, double* out, int cap, cudaStream_t s) {
  (void)p;
  int iters = 0;
  if (cudaMemcpyAsync(&iters, &d.esc->iters, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return -1;
  int n = iters + 1 < 1024 ? iters + 1 : 1024;
  int k = n < cap ? n : cap;
  if (k > 0 && (cudaMemcpyAsync(out, d.esc->normas, sizeof(double) * k, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
                cudaStreamSynchronize(s) != cudaSuccess))
    return -1;
  return n;
}
int erroPcg(Pcg* p, cudaStream_t s) {
  const int e = erroFundido(p->fundido, s);
  return e ? e : erroRegioes(p->regioes, s);
}
int motorPcg(Pcg* p) { return p->motor; }
void perfilPcg(Pcg* p, bool ligar) { perfilFundido(p->fundido, ligar); }
int lerPerfilPcg(Pcg* p, unsigned long long* out, int cap) { return lerPerfilFundido(p->fundido, out, cap); }

// One V-cycle on caller-provided device buffers (tq_vcycle).
template <class T>
__global__ void k_descarregar_x(const T* x0, float* x, int N) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < N) x[c] = carregar(x0[c]);
}
int cicloVDispositivo(Pcg* p, const uint8_t* tipo, const float* b, float* x, cudaStream_t s, bool preparar,
                      const int* parar) {
  if (preparar) prepararNiveis(p, tipo, false, s);
  p->parar = parar;  // the cycle's kernels return at once while *parar != 0
  Fonte F{b};
  fonteNivelUnico(p, F, s);
  const void* r = cicloV(p, F, s, false, false, x);
  if (p->L == 1)
    comTipo(p, 0, [&](auto* tag) {
      using T = std::remove_pointer_t<decltype(tag)>;
      lanca(k_descarregar_x<T>, blocos(p->N, 256), 256, 0, s, (const T*)r, x, p->N);
    });
  p->parar = nullptr;
  return cudaGetLastError() == cudaSuccess ? TQ_OK : TQ_E_CUDA;
}

// ---------------------------------------------------------------- V-cycle without allocation
// The level hierarchy of tq_vcycle_noalloc lives in this file-scope device array instead of
// cudaMalloc'd buffers.  Level 0 reads the caller's types in place; every other array is
// carved from the scratch on 256-byte boundaries.  The call writes every scratch byte it
// reads before reading it (types and masks of every level, level-0 b and x = 0, the
// restriction's b and x = 0 on each coarse level), so nothing has to start at zero and
// nothing carries over from one call to the next.
static __device__ __align__(256) unsigned char g_scratchVCiclo[BYTES_SCRATCH_VCICLO];

namespace {
constexpr size_t ALINHA_SCRATCH = 256;
inline size_t alinhar(size_t n) { return (n + ALINHA_SCRATCH - 1) & ~(ALINHA_SCRATCH - 1); }

// The level sizes of montarNiveis (js/pressao-cpu.js:24-41), as criarPcg builds them.
int niveisDe(int nx, int ny, int* nxL, int* nyL) {
  int L = 1, a = nx, b = ny;
  nxL[0] = a;
  nyL[0] = b;
  while ((a < b ? a : b) > 12 && L < MAX_NIVEIS) {
    a = (a + 1) / 2;
    b = (b + 1) / 2;
    nxL[L] = a;
    nyL[L] = b;
    L++;
  }
  return L;
}
}  // namespace

size_t bytesScratchVCiclo(int nx, int ny) {
  int nxL[MAX_NIVEIS], nyL[MAX_NIVEIS];
  const int L = niveisDe(nx, ny, nxL, nyL);
  size_t total = 0;
  for (int l = 0; l < L; l++) {
    const size_t n = (size_t)nxL[l] * nyL[l];
    if (l > 0) total += alinhar(n);  // types (level 0 uses the caller's)
    total += alinhar(n) + 3 * alinhar(n * 4);  // masks, b, x, tmp
  }
  return total;
}

// Device address of the scratch on the current device.  The address is looked up with
// cudaGetSymbolAddress once per device and context: the cache holds, per device ordinal, the
// context the address belongs to, and a different current context (the device was reset, or the
// primary context was released and created again, which loads the module anew) looks it up
// again instead of handing out a stale address.  The current context comes from the driver's
// cuCtxGetCurrent, reached through cudaGetDriverEntryPoint (no link to libcuda).
namespace {
using CtxGetCurrent = int (*)(void**);
CtxGetCurrent ctxGetCurrent() {
  static CtxGetCurrent fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      f = nullptr;
    }
    return (CtxGetCurrent)f;
  }();
  return fn;
}
}  // namespace

int enderecoScratchVCiclo(void** out) {
  static std::mutex mtx;
  static void* base[64] = {};
  static void* ctxDe[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TQ_E_NODEV;
  std::lock_guard<std::mutex> g(mtx);
  void* ctx = nullptr;
  CtxGetCurrent f = ctxGetCurrent();
  if (!f) return TQ_E_CUDA;
  if (!base[dev] || f(&ctx) != 0 || !ctx || ctx != ctxDe[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_scratchVCiclo) != cudaSuccess || !p) {
      cudaGetLastError();
      base[dev] = nullptr;
      return TQ_E_CUDA;
    }
    // the lookup makes the runtime's primary context current if none was: read it after
    if (f(&ctx) != 0 || !ctx) return TQ_E_CUDA;
    base[dev] = p;
    ctxDe[dev] = ctx;
  }
  *out = base[dev];
  return TQ_OK;
}

int cicloVSemAlocar(void* scratch, int nx, int ny, const uint8_t* tipo, const float* b, float* x, int precisao,
                    cudaStream_t s) {
  Pcg p{};
  p.nx = nx;
  p.ny = ny;
  p.N = nx * ny;
  p.precisao = precisao;
  p.motor = TQ_ENGINE_PLAIN;
  p.L = niveisDe(nx, ny, p.nxL, p.nyL);
  unsigned char* cur = (unsigned char*)scratch;
  for (int l = 0; l < p.L; l++) {
    const size_t n = (size_t)p.nxL[l] * p.nyL[l];
    p.meia[l] = precisao != TQ_PREC_FP32 && n >= (size_t)MEIA_MIN_CELULAS;
    if (l == 0) {
      p.tipoL[0] = const_cast<uint8_t*>(tipo);  // only read (prepararNiveis copies nothing)
    } else {
      p.tipoL[l] = cur;
      cur += alinhar(n);
    }
    p.vizL[l] = cur;
    cur += alinhar(n);
    p.bL[l] = cur;
    cur += alinhar(n * 4);
    p.xL[l] = cur;
    cur += alinhar(n * 4);
    p.tmpL[l] = cur;
    cur += alinhar(n * 4);
  }
  // The coarsest solve stages its level in shared memory only within the default 48 KB, which
  // needs no function attribute.
  const size_t nc = (size_t)p.nxL[p.L - 1] * p.nyL[p.L - 1];
  p.smemGrosso = nc * 9 <= 48 * 1024 ? nc * 9 : 0;
  return cicloVDispositivo(&p, tipo, b, x, s);
}

}  // namespace tq
