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
// TQ_PRECOND_BLOCK (bloco) it stays air.  The operator's free neighbours (bits 0-3) of every cell,
// from the true types.  And the bubbles' faces (montarBolhas, js/pressao-cpu.js:271-288): the (interior
// bubble cell, water neighbour) pairs of each label; a label with any is an active bubble.
__global__ void k_plano_tipos(Dev d, uint8_t* t0, uint8_t* vizOp, int bolhas, int bloco) {
  aposAnterior();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.N) return;
  const int nx = d.nx, ny = d.ny, i = c % nx, j = c / nx;
  const int viz[4] = {i > 0 ? d.tipo[c - 1] : SOLIDO, i < nx - 1 ? d.tipo[c + 1] : SOLIDO,
                      j > 0 ? d.tipo[c - nx] : SOLIDO, j < ny - 1 ? d.tipo[c + nx] : SOLIDO};
  uint8_t t = d.tipo[c];
  int m = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) m |= (viz[q] != SOLIDO) << q;
  vizOp[c] = (uint8_t)m;
  if (bolhas && t == AR) {
    const uint32_t b = d.rotulo[c];
    if (b >= 2) {
      if (!bloco) t = AGUA;
      if (b < (uint32_t)MAX_BOLHAS && i >= 1 && j >= 1 && i < nx - 1 && j < ny - 1) {
        const unsigned k = (viz[0] == AGUA) + (viz[1] == AGUA) + (viz[2] == AGUA) + (viz[3] == AGUA);
        if (k) atomicAdd(&d.facesB[b], k);
      }
    }
  }
  t0[c] = t;
}

// The levels' sizes and arrays for the two kernels that prepare them.
struct Niveis {
  int L;
  int nx[MAX_NIVEIS], ny[MAX_NIVEIS];
  long long ini[MAX_NIVEIS + 1];  // k_niveis_viz: first thread of each level (all levels' cells may pass 2^31)
  uint8_t *tipo[MAX_NIVEIS], *viz[MAX_NIVEIS];
};

// tiposGrossos (js/pressao-cpu.js:63-81) of levels l0 + 1 .. l0 + 6: air if any child is air, else
// water if any is water.  A CTA takes 64x64 cells of level l0 and halves them in shared memory (a
// launch a level took 2.4-3.6 us each).
constexpr int NIVEIS_POR_VEZ = 6;
__global__ void __launch_bounds__(256) k_niveis_tipos(Niveis n, int l0) {
  aposAnterior();
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

// prepararVizinhos (js/pressao-cpu.js:44-60) of every level from l0 on in one launch, packed in one byte:
// bits 0-3 = free (non-wall) left/right/down/up neighbours, bit 4 = the cell itself is water.  With
// `bloco` (TQ_PRECOND_BLOCK) the coarse levels' bits 0-3 are open where a fine face across the coarse
// face joins two non-wall fine cells (both coarse cells not wall).
__global__ void k_niveis_viz(Niveis n, int l0, int bloco) {
  aposAnterior();
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int l = l0;
  while (l < n.L && g >= n.ini[l + 1]) l++;
  if (l >= n.L) return;
  const int c = (int)(g - n.ini[l]), nx = n.nx[l], ny = n.ny[l], i = c % nx, j = c / nx;
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
  aposAnterior();
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

// Level 0's right side made from F on a grid of one level (k_descer makes it elsewhere).
template <class T>
__global__ void k_fonte(NivelDev<T> n0, Fonte F) {
  aposAnterior();
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n0.nx * n0.ny || (n0.parar && *n0.parar)) return;
  float v = F.v[c];
  if (n0.viz[c] & V0_BOLHA) v = (float)(F.rb[F.rotulo[c]] / F.celsB[F.rotulo[c]]);
  n0.b[c] = guardar<T>(v * (F.escala ? (float)*F.escala : 1.0f));
}

// The coarse levels of at most SECAO_PLANA cells in one CTA, in shared memory: x as swept, its snapshot
// before the pass (what a block's outer neighbours hold), the right side.  A thread takes two cells
// side by side, one of each colour, so every thread works in every half-sweep and half the warps
// meet at its barrier: four shared loads, the sum, a store.  The coarsest level's half-sweeps that
// repeat the one before (the last colour of a sweep is the first of the next, and a colour reads
// only the other) are left out, 65 of 128.  8 us with a coarsest level of
// 49 cells alone, 17 us for three levels from 943 cells, where six launches a level and the 42-46 us of
// one CTA's 128 half-sweeps were.  What a pass needs to know of a cell (where it is, which neighbours are
// open, which lie in another block) is packed in a word once a launch for all levels together, and a
// cell that does not change stores to a place of its own kind (FORA) instead of branching: with the
// words made again in each pass (1,250 cycles of it, its half-sweeps 900 to 1,900) and the branches, three
// levels from 1,000 cells took 22 us, 20 us now.
constexpr int SECAO_PLANA = 1024, SECAO_PLANA_NIVEIS = 6, SECAO_PLANA_TOTAL = 1536, T_SECAO = 576;
constexpr int SECAO_PARES = 1024;  // pairs of cells of all levels, each level's from a multiple of 32 on
struct SecaoPlana {
  int L, uma;
  int off[SECAO_PLANA_NIVEIS + 1];  // a level's first cell; after the last level, their number
  int par[SECAO_PLANA_NIVEIS + 1];  // a level's first pair
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
  aposAnterior();
  // one array, addressed by offsets: x, the snapshots, the right sides, and a 0 for closed neighbours
  constexpr int S = SECAO_PLANA_TOTAL, B = 2 * SECAO_PLANA_TOTAL, ZERO = 3 * SECAO_PLANA_TOTAL, FORA = ZERO + 1;
  __shared__ float X[ZERO + 2];
  __shared__ uint8_t V[SECAO_PLANA_TOTAL];
  // a pair's cells (of colour 0, of colour 1): bits 0-10 the cell, 11-14 open neighbours, 15-18 and 19-22 those
  // in another block at shift 0 and 8, 23 it changes
  __shared__ uint2 D[SECAO_PARES];
  if (s.n[0].parar && *s.n[0].parar) return;
  // the levels' sizes, first cells and first pairs: a load from the arguments by a level's number takes several
  // times one from shared memory
  __shared__ int NX[SECAO_PLANA_NIVEIS], NY[SECAO_PLANA_NIVEIS], OFF[SECAO_PLANA_NIVEIS + 1], PAR[SECAO_PLANA_NIVEIS + 1];
  const int t = threadIdx.x, nt = blockDim.x, total = s.off[s.L];
  if (t <= s.L) {
    OFF[t] = s.off[t];
    PAR[t] = s.par[t];
    if (t < s.L) {
      NX[t] = s.n[t].nx;
      NY[t] = s.n[t].ny;
    }
  }
  auto nivelDe = [&](const int* inicio, int k) {
    int l = 0;
    while (l + 1 < s.L && k >= inicio[l + 1]) l++;
    return l;
  };
  for (int k0 = t; k0 < total; k0 += 3 * nt) {  // every load of the three out before its store
    uint8_t v[3];
    float b[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const int k = k0 + q * nt;
      v[q] = 0;
      b[q] = 0.0f;
      if (k < total) {
        const int l = nivelDe(s.off, k);
        v[q] = s.n[l].viz[k - s.off[l]];
        if (l == 0) b[q] = s.n[0].b[k];
      }
    }
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const int k = k0 + q * nt;
      if (k < total) {
        V[k] = v[q];
        X[k] = X[S + k] = 0.0f;  // a pass takes the snapshots of the cells that change alone
        X[B + k] = b[q];
      }
    }
  }
  if (t == 0) X[ZERO] = 0.0f;
  __syncthreads();
  for (int k = t; k < PAR[s.L]; k += nt) {
    const int l = nivelDe(PAR, k), nx = NX[l], ny = NY[l], hw = (nx + 1) >> 1, r = k - PAR[l], j = r / hw;
    unsigned w[2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int i = 2 * (r - j * hw) + ((e + 1 + j) & 1);
      w[e] = 0;
      if (j < ny && i < nx) {
        const int c = OFF[l] + i + j * nx, vz = V[c];
        const int i8 = (i + 8) & 15, j8 = (j + 8) & 15, i0 = i & 15, j0 = j & 15;
        w[e] = c | (vz & 15) << 11 | ((i0 == 0) | (i0 == 15) << 1 | (j0 == 0) << 2 | (j0 == 15) << 3) << 15 |
               ((i8 == 0) | (i8 == 15) << 1 | (j8 == 0) << 2 | (j8 == 15) << 3) << 19 |
               ((vz & 16) && (vz & 15) ? 1u << 23 : 0u);
      }
    }
    D[k] = make_uint2(w[0], w[1]);
  }
  __syncthreads();
  const float pes[4] = {0.25f, 0.75f, 0.75f, 0.25f};
  // The thread's two cells of a level, colour e ^ ordem at [e]: where it stores (FORA: it does not change),
  // neighbours, free neighbours, right side.
  struct Par {
    int c[2], v[2][4], k[2];
    float b[2];
  };
  auto threads = [&](int l) { return PAR[l + 1] - PAR[l]; };
  auto par = [&](int l, int ordem, int desl, bool blocos) {  // desl: the blocks' shift; blocos: snapshots
    Par p;
    const int nx = NX[l];
    const uint2 d = D[PAR[l] + t];
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const unsigned w = e ^ ordem ? d.y : d.x, fora = blocos ? w >> (desl ? 19 : 15) : 0u;
      const int c = w & 0x7ff;
      // a neighbour of the cell's block is read as swept, one outside it from the snapshot
      p.c[e] = w >> 23 & 1 ? c : FORA;
      p.v[e][0] = w >> 11 & 1 ? c - 1 + (fora & 1 ? S : 0) : ZERO;
      p.v[e][1] = w >> 12 & 1 ? c + 1 + (fora & 2 ? S : 0) : ZERO;
      p.v[e][2] = w >> 13 & 1 ? c - nx + (fora & 4 ? S : 0) : ZERO;
      p.v[e][3] = w >> 14 & 1 ? c + nx + (fora & 8 ? S : 0) : ZERO;
      p.k[e] = __popc(w >> 11 & 15);
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
      q[e] = p.c[e] != FORA ? X[p.c[e]] : 0.0f;
      iq[e] = inversoVizinhos(p.k[e]);
      if (p.c[e] != FORA) X[S + p.c[e]] = q[e];
    }
    sinc(n);
#pragma unroll 1
    for (int h = 0; h < VARREDURAS; h++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const float sm = ((X[p.v[e][0]] + X[p.v[e][1]]) + X[p.v[e][2]]) + X[p.v[e][3]];
        q[e] = q[e] + fmaf(sm + p.b[e], iq[e], -q[e]);
        X[p.c[e]] = q[e];
        sinc(n);
      }
  };
  for (int l = 0; l < s.L - 1; l++) {
    if (!s.uma) {
      passo(l, 0, 0);
      __syncthreads();
    }
    passo(l, 8, 0);
    const int nx = NX[l], ny = NY[l], N = nx * ny, o = OFF[l];
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
    const int gx = NX[l + 1], G = gx * NY[l + 1], og = OFF[l + 1];
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
        X[p.c[e]] = dividirViz(sm + p.b[e], kf[e], iq[e]);
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
    const int nx = NX[l], N = nx * NY[l], o = OFF[l];
    const int gx = NX[l + 1], gy = NY[l + 1], og = OFF[l + 1];
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
  for (int c = t; c < NX[0] * NY[0]; c += nt) s.saida[c] = X[c];
}

// resolverGrosso (js/pressao-cpu.js:217-238): VARREDURAS_GROSSO alternating red-black sweeps
// in place on a coarsest level of more than SECAO_PLANA cells, from x = 0, one CTA; the level lives
// in shared memory when it fits.  65 half-sweeps as in k_secao.
template <class T>
__global__ void __launch_bounds__(1024) k_grosso(NivelDev<T> n, int emShared) {
  aposAnterior();
  extern __shared__ unsigned char dyn[];
  if (n.parar && *n.parar) return;  // uniform over the CTA
  const int N = n.nx * n.ny, nx = n.nx;
  float* xs = (float*)dyn;
  float* bs = xs + N;
  uint8_t* vs = (uint8_t*)(bs + N);
  const uint8_t* viz = n.viz;
  // in global memory a 16-bit level sweeps in its free array, which has room for FP32
  float* xg = sizeof(T) == 4 ? (float*)n.x : (float*)n.tmp;
  if (emShared)
    for (int c = threadIdx.x; c < N; c += blockDim.x) {
      xs[c] = 0.0f;
      bs[c] = carregar(n.b[c]);
      vs[c] = viz[c];
    }
  else
    for (int c = threadIdx.x; c < N; c += blockDim.x) xg[c] = 0.0f;
  __syncthreads();
  for (int h = 0; h <= VARREDURAS_GROSSO; h++) {
    const int cor = h & 1;
    for (int c = threadIdx.x; c < N; c += blockDim.x) {
      int i = c % nx, j = c / nx;
      int vz = emShared ? vs[c] : viz[c];
      if (!(vz & 16) || ((i + j + 1) & 1) != cor) continue;
      int q = __popc(vz & 15);
      if (!q) continue;
      auto x = [&](int k) { return emShared ? xs[k] : xg[k]; };
      float s = 0.0f;
      if (vz & 1) s += x(c - 1);
      if (vz & 2) s += x(c + 1);
      if (vz & 4) s += x(c - nx);
      if (vz & 8) s += x(c + nx);
      const float r = dividirViz(s + (emShared ? bs[c] : carregar(n.b[c])), (float)q, inversoVizinhos(q));
      if (emShared) xs[c] = r;
      else xg[c] = r;
    }
    __syncthreads();
  }
  if (emShared || sizeof(T) == 2)
    for (int c = threadIdx.x; c < N; c += blockDim.x) n.x[c] = guardar<T>(emShared ? xs[c] : xg[c]);
}

// ---------------------------------------------------------------- PCG kernels
// One iteration is three kernels and a V-cycle: p = z + beta p with A p and p.Ap (k_plano_da), the
// q / r / bubble updates with r.r (k_plano_b), and the V-cycle, whose first kernel spreads r and whose
// last one gathers z with r.z and r.zOld.  Each sums its dot products in blocks, and its last block to
// finish adds the blocks' partials in block order and the active bubbles' terms in label order, makes
// the scalar and updates the bubbles: the next kernel finds alpha, the norm or beta ready.  (A launch
// for every step, with the dot products each a pass over the grid and a walk of the 4,096 labels,
// took 15 launches of 3-20 us beside the V-cycle.)
constexpr double ESCALA_PCG = 1099511627776.0;  // 2^40, the bubbles' fixed-point sums
// Tolerance mode replaces the recursive FP32 residual by the true one each time the recursive one
// has fallen by this factor since the last replacement (as the fused engine and the oracle do).
constexpr double FATOR_TROCA = 1e-3;
constexpr int T_PCG = 256;
constexpr int BLOCOS_PCG = 1184;  // 8 a SM; with more cells each thread takes several
static int blocosPcg(int N) { return blocos(N, T_PCG) < BLOCOS_PCG ? blocos(N, T_PCG) : BLOCOS_PCG; }

// What the solve's kernels share beside Dev: the operator's descriptor of every cell, the active
// bubbles (count first, then labels ascending) and the blocks' partial sums (two a block).
struct Plano {
  uint16_t* op;
  int* ativos;
  double* parc;
  int bolhas, bloco, meia;  // air labels in use, TQ_PRECOND_BLOCK, 16-bit V-cycle storage
};
// Bits 0-3 the neighbour is water, OP_AGUA water, OP_FACE interior air of an active bubble, OP_VIZ_BOLHA
// a neighbour is air of an active bubble; bits 8-10 the number of free neighbours.
constexpr int OP_AGUA = 16, OP_FACE = 32, OP_VIZ_BOLHA = 64;

__device__ inline bool bolhaAtiva(const Dev& d, uint32_t b) {
  return b >= 2 && b < (uint32_t)MAX_BOLHAS && d.facesB[b] > 0;
}

// Block sum of a double (valid in thread 0).
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
  return t;
}

// The block's partials of one or two sums; true in every thread of the block that finishes last,
// whose writes by the other blocks are then visible.
__device__ inline bool ultimoBloco(const Dev& d, const Plano& P, int bloco, int blocosTot, double s1, double s2,
                                   bool dois, double* sh) {
  __shared__ bool ultimo;
  const double t1 = somaBloco(s1, sh), t2 = dois ? somaBloco(s2, sh) : 0.0;
  if (threadIdx.x == 0) {
    P.parc[2 * bloco] = t1;
    if (dois) P.parc[2 * bloco + 1] = t2;
    __threadfence();
    ultimo = atomicAdd(&d.esc->tickets[0], 1u) == (unsigned)blocosTot - 1;
  }
  __syncthreads();
  if (!ultimo) return false;
  __threadfence();
  if (threadIdx.x == 0) d.esc->tickets[0] = 0;
  return true;
}
// Sums of the blocks' partials and of a term per active bubble (valid in thread 0): the last block.
template <class F>
__device__ inline void somasFinais(const Plano& P, int blocosTot, bool dois, double out[2], double* sh, F termo) {
  double p1 = 0, p2 = 0;
  for (int k = threadIdx.x; k < blocosTot; k += blockDim.x) {
    p1 += __ldcg(&P.parc[2 * k]);
    if (dois) p2 += __ldcg(&P.parc[2 * k + 1]);
  }
  double q1 = 0, q2 = 0;
  const int nAt = P.bolhas ? P.ativos[0] : 0;
  for (int k = threadIdx.x; k < nAt; k += blockDim.x) termo(P.ativos[1 + k], q1, q2);
  out[0] = somaBloco(p1, sh);
  out[0] += somaBloco(q1, sh);
  if (dois) {
    out[1] = somaBloco(p2, sh);
    out[1] += somaBloco(q2, sh);
  }
}

// Level 0's masks and descriptors, the bubbles' cells (every air cell of an active label,
// js/pressao-cpu.js:345-351), r = -div - A q on water with r.r (:331-338) and the bubbles' sums of q over
// their water faces.  The last block lists the active bubbles and closes their rows,
// rb = rhs - (faces y - sum) (:339-341), and the initial norm.
__global__ void __launch_bounds__(T_PCG) k_plano_inicio(Dev d, Plano P, const uint8_t* vizOp, const uint8_t* tipo0,
                                                        uint8_t* viz0, double* q64) {
  aposAnterior();
  __shared__ double sh[32];
  const int nx = d.nx, N = d.N;
  double s = 0;
  if (P.bolhas)  // (the last block writes the active labels' over these)
    for (int b = blockIdx.x * T_PCG + threadIdx.x; b < MAX_BOLHAS; b += gridDim.x * T_PCG)
      d.pb[b] = d.zb[b] = d.yB[b] = d.rb[b] = 0.0;
  auto celula = [&](int c) {  // the label of the active bubble that the cell is air of, or 0
    const int nb[4] = {c - 1, c + 1, c - nx, c + nx};
    const int t = d.tipo[c], livres = vizOp[c];
    int v0 = tipo0[c] == AGUA ? 16 : 0, op = __popc(livres) << 8;
    float sv = 0.0f;
    double face = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (!(livres & (1 << k))) continue;
      v0 |= 1 << k;  // (the preconditioner's types are wall where the true ones are)
      const int tn = d.tipo[nb[k]];
      if (tn == AGUA) {
        op |= 1 << k;
        const float qn = d.q[nb[k]];
        sv += qn;
        face += (double)qn;
      } else if (P.bolhas && tn == AR) {
        const uint32_t r = d.rotulo[nb[k]];
        if (bolhaAtiva(d, r)) {
          op |= OP_VIZ_BOLHA;
          sv += d.yBolhaF[r];
        }
      }
    }
    uint32_t b = 0;
    if (t == AGUA) {
      op |= OP_AGUA;
      v0 |= V0_AGUA;
      const float q = d.q[c], r = -d.div[c] - ((float)__popc(livres) * q - sv);
      d.r[c] = r;
      if (q64) q64[c] = (double)q;  // tolerance mode: the FP64 iterate
      s += (double)r * (double)r;
    } else {
      d.r[c] = 0.0f;
      if (P.bolhas && t == AR) {
        const uint32_t r = d.rotulo[c];
        if (bolhaAtiva(d, r)) {
          b = r;
          if (!P.bloco) v0 |= V0_BOLHA;
          const int i = c % nx, j = c / nx;
          if (i >= 1 && j >= 1 && i < nx - 1 && j < d.ny - 1) {
            op |= OP_FACE;
            if (face != 0) somaFixa(&d.accB[b], face, ESCALA_PCG);
          }
        }
      }
    }
    P.op[c] = (uint16_t)op;
    viz0[c] = (uint8_t)v0;
    return b;
  };
  const int lane = threadIdx.x & 31;
  for (int c0 = blockIdx.x * T_PCG + threadIdx.x - lane; c0 < N; c0 += gridDim.x * T_PCG) {  // a warp's trips are the same
    const uint32_t b = c0 + lane < N ? celula(c0 + lane) : 0u;
    if (__any_sync(0xffffffffu, b != 0)) {  // cells of one bubble lie together
      const unsigned g = __match_any_sync(0xffffffffu, b);
      if (b && lane == __ffs(g) - 1) atomicAdd(&d.celsB[b], (unsigned)__popc(g));
    }
  }
  if (!ultimoBloco(d, P, blockIdx.x, gridDim.x, s, 0, false, sh)) return;
  if (P.bolhas) {
    // the active labels in ascending order (K runs of T_PCG labels, a run's warps by ballot), their loads in
    // flight together; what only active labels have is touched for those alone (16 labels in a row a thread,
    // each waiting for the one before, took half of the kernel: 21 -> 8 us on 160x100 cells)
    constexpr int K = MAX_BOLHAS / T_PCG, W = T_PCG / 32;
    static_assert(K * W <= T_PCG, "a count a thread");
    __shared__ int pref[K * W + 1];
    const int w = threadIdx.x >> 5;
    unsigned at[K];
#pragma unroll
    for (int k = 0; k < K; k++) at[k] = __ldcg(&d.facesB[k * T_PCG + threadIdx.x]);
#pragma unroll
    for (int k = 0; k < K; k++) {
      at[k] = __ballot_sync(0xffffffffu, at[k] > 0 && k * T_PCG + threadIdx.x >= 2);
      if (lane == 0) pref[k * W + w] = __popc(at[k]);
    }
    __syncthreads();
    if (w == 0) {  // exclusive prefix of the K * W counts, K * W / 32 a lane
      constexpr int E = K * W / 32;
      int v[E], t = 0;
#pragma unroll
      for (int e = 0; e < E; e++) {
        v[e] = t;
        t += pref[lane * E + e];
      }
      int u = t;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, u, o);
        if (lane >= o) u += a;
      }
#pragma unroll
      for (int e = 0; e < E; e++) pref[lane * E + e] = v[e] + u - t;
      if (lane == 31) pref[K * W] = u;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; k++)
      if (at[k] >> lane & 1) P.ativos[1 + pref[k * W + w] + __popc(at[k] & ((1u << lane) - 1u))] = k * T_PCG + threadIdx.x;
    const int n = pref[K * W];
    if (threadIdx.x == 0) P.ativos[0] = n;
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += T_PCG) {
      const int b = P.ativos[1 + k];
      const double y = (double)d.yBolhaF[b];
      d.yB[b] = y;
      d.rb[b] = (double)d.rhsBolhaF[b] - (__ldcg(&d.facesB[b]) * y - (double)__ldcg(&d.accB[b]) / ESCALA_PCG);
      d.accB[b] = 0;
    }
    __syncthreads();
  }
  double x[2];
  somasFinais(P, gridDim.x, false, x, sh, [&](int b, double& q1, double&) { q1 += d.rb[b] * d.rb[b]; });
  if (threadIdx.x == 0) {
    Escalares* e = d.esc;
    const double nr = sqrt(x[0]);
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
    e->escalaMG = (P.meia && nr > 0) ? 1.0 / nr : 1.0;
  }
}

// p = z + beta p (z on the first iteration), A p and p.Ap (js/pressao-cpu.js:84-93, 363-373, 395-396); air of an
// active bubble gives a water cell its bubble's p, and takes the sum of p over its water faces.
// The last block: the bubbles' p and rows, p.Ap and alpha.
__global__ void __launch_bounds__(T_PCG) k_plano_da(Dev d, Plano P, const float* z, const float* pv, float* pn, int prim) {
  aposAnterior();
  __shared__ double sh[32];
  if (d.esc->pronto) return;  // uniform over the grid
  const int nx = d.nx, N = d.N;
  const double beta = prim ? 0.0 : d.esc->beta;
  const float bf = (float)beta;
  auto pbNovo = [&](int b) { return prim ? d.zb[b] : d.zb[b] + beta * d.pb[b]; };
  double s = 0;
  for (int c = blockIdx.x * T_PCG + threadIdx.x; c < N; c += gridDim.x * T_PCG) {
    const int m = P.op[c];
    // the five z and p go out with the descriptor (an index past the grid's end reads c itself; the
    // descriptor picks the neighbours that count)
    const int nb[5] = {c, c > 0 ? c - 1 : c, c < N - 1 ? c + 1 : c, c >= nx ? c - nx : c, c < N - nx ? c + nx : c};
    float pq[5];
#pragma unroll
    for (int k = 0; k < 5; k++) pq[k] = prim ? z[nb[k]] : z[nb[k]] + bf * pv[nb[k]];
    if (m & OP_AGUA) {
      float sv = 0.0f;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if (m & (1 << k)) sv += pq[k + 1];
        else if (m & OP_VIZ_BOLHA) {
          const int i = c % nx, j = c / nx;
          const bool existe = k == 0 ? i > 0 : k == 1 ? i < nx - 1 : k == 2 ? j > 0 : j < d.ny - 1;
          if (existe && d.tipo[nb[k + 1]] == AR) {
            const uint32_t r = d.rotulo[nb[k + 1]];
            if (bolhaAtiva(d, r)) sv += (float)pbNovo(r);
          }
        }
      }
      const float ap = (float)(m >> 8) * pq[0] - sv;
      pn[c] = pq[0];
      d.ap[c] = ap;
      s += (double)pq[0] * (double)ap;
    } else if (m & OP_FACE) {
      double t = 0;
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (m & (1 << k)) t += (double)pq[k + 1];
      if (t != 0) somaFixa(&d.accB[d.rotulo[c]], t, ESCALA_PCG);
    }
  }
  if (!ultimoBloco(d, P, blockIdx.x, gridDim.x, s, 0, false, sh)) return;
  double x[2];
  somasFinais(P, gridDim.x, false, x, sh, [&](int b, double& q1, double&) {
    const double pb = pbNovo(b), ap = d.facesB[b] * pb - (double)__ldcg(&d.accB[b]) / ESCALA_PCG;
    d.pb[b] = pb;
    d.apb[b] = ap;
    d.accB[b] = 0;
    q1 += pb * ap;
  });
  if (threadIdx.x == 0) {
    Escalares* e = d.esc;
    e->pap = x[0];
    e->alpha = fabs(x[0]) < 1e-30 ? 0.0 : e->rz / x[0];
  }
}

// q += alpha p, r -= alpha Ap on water with r.r; the last block the bubbles and the norm
// (js/pressao-cpu.js:377-386).
__global__ void __launch_bounds__(T_PCG) k_plano_b(Dev d, Plano P, const float* p, double* q64, int it, double tol, int cap) {
  aposAnterior();
  __shared__ double sh[32];
  if (d.esc->pronto) return;
  const double alfa = d.esc->alpha;
  const float a = (float)alfa;
  double s = 0;
  for (int c = blockIdx.x * T_PCG + threadIdx.x; c < d.N; c += gridDim.x * T_PCG) {
    const int m = P.op[c];
    const float pc = p[c], rc = d.r[c], apc = d.ap[c];
    const double qd = q64 ? q64[c] : 0.0;
    const float qf = q64 ? 0.0f : d.q[c];
    if (!(m & OP_AGUA)) continue;
    if (q64) q64[c] = qd + alfa * (double)pc;
    else d.q[c] = qf + a * pc;
    const float r = rc - a * apc;
    d.r[c] = r;
    s += (double)r * (double)r;
  }
  if (!ultimoBloco(d, P, blockIdx.x, gridDim.x, s, 0, false, sh)) return;
  double x[2];
  somasFinais(P, gridDim.x, false, x, sh, [&](int b, double& q1, double&) {
    d.yB[b] += alfa * d.pb[b];
    const double rb = d.rb[b] - alfa * d.apb[b];
    d.rb[b] = rb;
    q1 += rb * rb;
  });
  if (threadIdx.x == 0) {
    Escalares* e = d.esc;
    const double nr = sqrt(x[0]);
    e->norma = nr;
    if (it + 1 < 1024) e->normas[it + 1] = nr;
    e->iters = it + 1;
    // tolerance mode: the recursive residual met the tolerance, or fell by FATOR_TROCA since
    // the last replacement, or the cap came: the true residual decides (k_verdade, k_verdade_fim)
    e->verificar = tol > 0 && (nr <= tol * e->norma0 || nr <= e->proxTroca || it + 1 >= cap);
    e->escalaMG = (P.meia && nr > 0) ? 1.0 / nr : 1.0;
  }
}

// The gather of z after the V-cycle (precondicionar, js/pressao-cpu.js:357-361): z = x / escala; cells of an
// active bubble give their mean correction to the bubble's z (the transpose of spreading) and keep 0.
struct Juncao {
  Dev d;
  Plano P;
  const float* zVelho;  // null on the first iteration
  float* zNovo;
};
template <class T>
__device__ __forceinline__ void juntarCelula(const Juncao& J, int c, int v, float x, float inv, float r, float zv,
                                             double& s1, double& s2) {
  const float z = arredondar<T>(x) * inv;
  if (v & V0_BOLHA) {
    const uint32_t b = J.d.rotulo[c];
    somaFixa(&J.d.accB[b], (double)z / J.d.celsB[b], ESCALA_PCG);
    J.zNovo[c] = 0.0f;
    return;
  }
  J.zNovo[c] = z;
  if (v & V0_AGUA) {
    s1 += (double)r * (double)z;
    s2 += (double)r * (double)zv;
  }
}
// After the gather: r.z and r.zOld, and by the last block the bubbles' z (with TQ_PRECOND_BLOCK a Jacobi
// step on the bubble's row) and beta (js/pressao-cpu.js:388-394).
__device__ inline void fimJuncao(const Juncao& J, int bloco, int blocosTot, double s1, double s2) {
  __shared__ double sh[32];
  const Dev& d = J.d;
  if (!ultimoBloco(d, J.P, bloco, blocosTot, s1, s2, true, sh)) return;
  double x[2];
  somasFinais(J.P, blocosTot, true, x, sh, [&](int b, double& q1, double& q2) {
    const double zv = d.zb[b];
    const double zb = J.P.bloco ? d.rb[b] / (double)d.facesB[b] : (double)__ldcg(&d.accB[b]) / ESCALA_PCG;
    d.zb[b] = zb;
    d.accB[b] = 0;
    q1 += d.rb[b] * zb;
    q2 += d.rb[b] * zv;
  });
  if (threadIdx.x == 0) {
    Escalares* e = d.esc;
    // (after a residual replacement the direction carries on: no restart)
    e->beta = !J.zVelho || fabs(e->rz) < 1e-30 ? 0.0 : fmax(0.0, (x[0] - x[1]) / e->rz);
    e->reiniciar = 0;
    e->rz = x[0];
  }
}
// The gather on a grid of one level (k_subir's last launch does it elsewhere).
template <class T>
__global__ void __launch_bounds__(T_PCG) k_juntar(Juncao J, const uint8_t* viz0, const T* x0) {
  aposAnterior();
  const Dev& d = J.d;
  if (d.esc->pronto) return;
  const float inv = (float)(1.0 / d.esc->escalaMG);
  double s1 = 0, s2 = 0;
  for (int c = blockIdx.x * T_PCG + threadIdx.x; c < d.N; c += gridDim.x * T_PCG)
    juntarCelula<T>(J, c, viz0[c], carregar(x0[c]), inv, d.r[c], J.zVelho ? J.zVelho[c] : 0.0f, s1, s2);
  fimJuncao(J, blockIdx.x, gridDim.x, s1, s2);
}

// The way up a level: x + the coarse correction and both passes, the level's result in n.tmp, or
// (saida not null) as floats in saida, or (JUNTA, level 0 of a solve) gathered into z.
template <class T, class TG, bool JUNTA>
__global__ void __launch_bounds__(T_LADRILHO) k_subir(NivelDev<T> n, NivelDev<TG> g, const TG* xg, int kx, int ky,
                                                      int uma, int masc, float* saida,
                                                      const __grid_constant__ Juncao J) {
  aposAnterior();
  extern __shared__ __align__(16) float mem[];
  if (n.parar && *n.parar) return;
  const Ladrilho L{(int)blockIdx.x * 16 * kx, (int)blockIdx.y * 16 * ky, kx, ky, n.nx, n.ny, n.viz};
  double s1 = 0, s2 = 0;
  const float inv = JUNTA ? (float)(1.0 / J.d.esc->escalaMG) : 1.0f;
  subirLadrilho<T>(
      L, g.nx, g.ny, uma != 0, masc != 0, VARREDURAS, mem, [&](int c) { return carregar(n.x[c]); },
      [&](int C) { return carregar(xg[C]); }, [&](int c) { return carregar(n.b[c]); },
      [&](const int (&cel)[2][4], const int (&v)[2][4], const float (&x)[2][4]) {
        if constexpr (JUNTA) {
          float r[2][4], zv[2][4];
#pragma unroll
          for (int cr = 0; cr < 2; cr++)
#pragma unroll
            for (int m = 0; m < 4; m++) {
              const int c = cel[cr][m] < 0 ? 0 : cel[cr][m];
              r[cr][m] = J.d.r[c];
              zv[cr][m] = J.zVelho ? J.zVelho[c] : 0.0f;
            }
#pragma unroll
          for (int cr = 0; cr < 2; cr++)
#pragma unroll
            for (int m = 0; m < 4; m++)
              if (cel[cr][m] >= 0)
                juntarCelula<T>(J, cel[cr][m], v[cr][m], x[cr][m], inv, r[cr][m], zv[cr][m], s1, s2);
        } else {
#pragma unroll
          for (int cr = 0; cr < 2; cr++)
#pragma unroll
            for (int m = 0; m < 4; m++)
              if (cel[cr][m] >= 0) {
                if (saida) saida[cel[cr][m]] = arredondar<T>(x[cr][m]);
                else n.tmp[cel[cr][m]] = guardar<T>(x[cr][m]);
              }
        }
      });
  if (JUNTA) fimJuncao(J, blockIdx.x + blockIdx.y * gridDim.x, gridDim.x * gridDim.y, s1, s2);
}

// Tolerance mode, once the recursive residual met the tolerance (Escalares::verificar): the true
// residual in FP64 from the FP64 iterate and the bubble pressures.  Water cells: rt = -div - A q
// into d.ap (free until the next A p) and rt^2 into per-CTA partials; interior air of active
// bubbles: the sum of q over its water faces into the bubble's fixed-point sum (accB, zeroed
// before).  k_verdade_fim finishes the norm and decides.
constexpr int BLOCOS_VERDADE = 296;  // 2 a SM
__global__ void __launch_bounds__(256) k_verdade(Dev d, const uint8_t* vizOp, const double* q64, int bolhas) {
  aposAnterior();
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
  aposAnterior();
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
  if (bolhas)
    for (int b = threadIdx.x; b < MAX_BOLHAS; b += blockDim.x) {
      if (substituir && b >= 2 && d.facesB[b] > 0) d.rb[b] = rbv(b);
      d.accB[b] = 0;  // the next iteration's sums start from 0
    }
}
// After a replacement: r = the true residual on water cells.
__global__ void k_substituir(Dev d) {
  aposAnterior();
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.N || !d.esc->reiniciar || d.esc->pronto) return;
  if (d.tipo[c] == AGUA) d.r[c] = d.ap[c];
}

// End of the solve: non-water q = 0; bubbles hand back their pressure (js/pressao-cpu.js:399-400).
// Tolerance mode: q = the FP64 iterate rounded; the solve's convergence record (thread 0).
__global__ void k_pcg_fim(Dev d, int bolhas, const double* q64, double tol) {
  aposAnterior();
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

// ---------------------------------------------------------------- the solver object
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



Pcg* criarPcg(int nx, int ny, int precisao, int motor, Arena& A, int ctasFundido) {
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
  for (int l = 0; l < L; l++) {
    size_t n = (size_t)p->nxL[l] * p->nyL[l];
    p->meia[l] = precisao != TQ_PREC_FP32 && n >= (size_t)MEIA_MIN_CELULAS;
    A.pedir(&p->tipoL[l], n);
    A.pedir(&p->vizL[l], n);
    // room for FP32 whatever the engine stores
    A.pedir((float**)&p->bL[l], n);
    A.pedir((float**)&p->xL[l], n);
    A.pedir((float**)&p->tmpL[l], n);
  }
  A.pedir(&p->vizOp, p->N);
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
  if (motor == TQ_ENGINE_FUSED) {
    // Grids with a single level (min(nx, ny) <= 12) have nothing to hand to the coarse
    // section: they run on the plain engine.
    p->fundido = criarFundido(p, A);
    if (!p->fundido) {
      cudaGetLastError();
      p->motor = TQ_ENGINE_PLAIN;
    }
  }
  if (p->motor == TQ_ENGINE_PLAIN) {
    // the partial sums of k_plano_da / k_plano_b's blocks, or of the gather's tiles if more
    const int k = escolherLadrilho(nx, ny, true, false);
    const size_t lad = (size_t)blocos(nx, 16 * k) * blocos(ny, 16 * k);
    A.pedir(&p->op, p->N);
    A.pedir(&p->p2, p->N);
    A.pedir(&p->parc, 2 * (lad > (size_t)BLOCOS_PCG ? lad : (size_t)BLOCOS_PCG));
    A.pedir(&p->ativos, MAX_BOLHAS + 1);
  }
  return p;
}

bool iniciarPcg(Pcg* p, cudaStream_t s) { return !p->fundido || iniciarFundido(p->fundido, p, s); }

void destruirPcg(Pcg* p) {
  if (!p) return;
  destruirFundido(p->fundido);
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
// (saida, J: level 0's alone)
static void subirNivel(Pcg* p, int l, const void* xg, bool bloco, bool uma, float* saida, const Juncao* J,
                       cudaStream_t s) {
  uma = uma && l >= 1;
  const int k = escolherLadrilho(p->nxL[l], p->nyL[l], true, uma), d = uma ? 8 : 0;
  const dim3 gr(blocos(p->nxL[l] + d, 16 * k), blocos(p->nyL[l] + d, 16 * k));
  comTipos(p, l, [&](auto* tf, auto* tg) {
    using TF = std::remove_pointer_t<decltype(tf)>;
    using TG = std::remove_pointer_t<decltype(tg)>;
    auto kern = J ? k_subir<TF, TG, true> : k_subir<TF, TG, false>;
    const size_t b = prepararLadrilho(kern, k);
    lanca(kern, gr, threadsLadrilho(k), b, s, nivel<TF>(p, l), nivel<TG>(p, l + 1), (const TG*)xg, k, k, uma ? 1 : 0,
          bloco && l >= 1 ? 1 : 0, saida, J ? *J : Juncao{});
  });
}

// cicloV (js/pressao-cpu.js:241-255) on a right side made from F (level 0's b is written); every
// level's result ends in its tmp, level 0's returned, or as floats in saida, or gathered by J, when
// there is one (on more than one level).
// umaPassada (TQ_PRECOND_BLOCK_1): the levels above 0 take one smoother pass a leg (shift 8).
static const void* cicloV(Pcg* p, const Fonte& F, cudaStream_t s, bool bloco, bool umaPassada, float* saida,
                          const Juncao* J) {
  const int L = p->L;
  // the section: the coarse levels of at most SECAO_PLANA cells (not level 0)
  int Ls = L, total = 0, pares = 0;
  auto paresDe = [&](int l) { return (((p->nxL[l] + 1) / 2) * p->nyL[l] + 31) & ~31; };
  while (Ls > 1 && L - Ls < SECAO_PLANA_NIVEIS && p->nxL[Ls - 1] * p->nyL[Ls - 1] <= SECAO_PLANA &&
         ((p->nxL[Ls - 1] + 1) / 2) * p->nyL[Ls - 1] <= T_SECAO &&
         total + p->nxL[Ls - 1] * p->nyL[Ls - 1] <= SECAO_PLANA_TOTAL && pares + paresDe(Ls - 1) <= SECAO_PARES)
    Ls--, total += p->nxL[Ls] * p->nyL[Ls], pares += paresDe(Ls);
  const int Lf = Ls < L ? Ls : L - 1;  // the levels with tile legs: 0 .. Lf - 1
  for (int l = 0; l < Lf; l++) descerNivel(p, l, bloco, umaPassada, F, s);
  const void* x;
  if (Ls < L) {
    SecaoPlana sp{};
    sp.L = L - Ls;
    sp.uma = umaPassada ? 1 : 0;
    for (int l = Ls; l < L; l++) {
      sp.n[l - Ls] = nivel<float>(p, l);
      sp.off[l - Ls + 1] = sp.off[l - Ls] + p->nxL[l] * p->nyL[l];
      sp.par[l - Ls + 1] = sp.par[l - Ls] + paresDe(l);
    }
    sp.saida = (float*)p->tmpL[Ls];
    x = sp.saida;
    lanca(k_secao, 1, paresDe(Ls), 0, s, sp);
  } else {
    comTipo(p, L - 1, [&](auto* t) {
      using T = std::remove_pointer_t<decltype(t)>;
      lanca(k_grosso<T>, 1, 1024, p->smemGrosso, s, nivel<T>(p, L - 1), p->smemGrosso ? 1 : 0);
    });
    x = p->xL[L - 1];
  }
  for (int l = Lf - 1; l >= 0; l--) {
    subirNivel(p, l, x, bloco, umaPassada, l == 0 ? saida : nullptr, l == 0 ? J : nullptr, s);
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

// z = the preconditioned residual (J.zNovo), the bubbles' z, r.z and beta.
static void precondicionar(Pcg* p, const Juncao& J, bool bloco, bool umaPassada, cudaStream_t s) {
  const Dev& d = J.d;
  Fonte F{d.r, &d.esc->escalaMG, d.rotulo, d.rb, d.celsB};
  fonteNivelUnico(p, F, s);
  const void* x = cicloV(p, F, s, bloco, umaPassada, nullptr, &J);
  if (p->L == 1)
    comTipo(p, 0, [&](auto* tag) {
      using T = std::remove_pointer_t<decltype(tag)>;
      lanca(k_juntar<T>, blocosPcg(d.N), T_PCG, 0, s, J, p->vizL[0], (const T*)x);
    });
}

// Iterations the plain engine queues between two reads of the stop flag.  Every kernel of an
// iteration returns at once after the flag is set, so the result is the same as stopping at the
// exact iteration, with one host round trip per LOTE_VERIFICACAO iterations instead of one each.
constexpr int LOTE_VERIFICACAO = 8;

int reservarTolerancia(Pcg* p, cudaStream_t s) {
  if (!p->regioes && !(p->regioes = criarRegioes(p->N, s))) return TQ_E_NOMEM;
  if (p->motor != TQ_ENGINE_FUSED && !p->q64 && cudaMalloc(&p->q64, (size_t)p->N * sizeof(double)) != cudaSuccess)
    return TQ_E_NOMEM;
  return TQ_OK;
}

int resolverPressao(Pcg* p, const Dev& d0, int iteracoes, double tol, bool bolhas, int precond, cudaStream_t s) {
  Dev d = d0;
  double* q64 = nullptr;
  if (tol > 0) {
    if (reservarTolerancia(p, s)) return TQ_E_NOMEM;
    projetarFechadas(p->regioes, d0, bolhas, s, &d);  // d reads the projected right-hand sides
    q64 = p->q64;
  }
  if (p->motor == TQ_ENGINE_FUSED) return resolverPressaoFundido(p, d, iteracoes, tol, bolhas, precond, s);
  const bool bloco = precond == TQ_PRECOND_BLOCK || precond == TQ_PRECOND_BLOCK_1;
  const bool umaPassada = precond == TQ_PRECOND_BLOCK_1;
  const int nb = blocos(d.N, 256), nbp = blocosPcg(d.N);
  const int nbx = blocos(d.N > MAX_BOLHAS ? d.N : MAX_BOLHAS, 256);
  const Plano P{p->op, p->ativos, p->parc, bolhas ? 1 : 0, bloco ? 1 : 0, p->precisao != TQ_PREC_FP32 ? 1 : 0};
  zerarBolhas(d, s);
  // operator (true types) and preconditioner types, the levels', level 0's masks with r and its norm
  lanca(k_plano_tipos, nb, 256, 0, s, d, p->tipoL[0], p->vizOp, bolhas ? 1 : 0, bloco ? 1 : 0);
  prepararNiveis(p, p->tipoL[0], bloco, s, false);
  lanca(k_plano_inicio, nbp, T_PCG, 0, s, d, P, p->vizOp, p->tipoL[0], p->vizL[0], q64);
  p->parar = &d.esc->pronto;  // the V-cycle kernels return once the solve has stopped
  float *zc = d.z, *zo = d.zOld, *pv = d.p, *pn = p->p2;  // z, p and the previous ones swap buffers
  precondicionar(p, Juncao{d, P, nullptr, zc}, bloco, umaPassada, s);
  int it = 0;
  for (; it < iteracoes; it++) {
    lanca(k_plano_da, nbp, T_PCG, 0, s, d, P, zc, pv, pn, it == 0 ? 1 : 0);
    std::swap(pv, pn);
    lanca(k_plano_b, nbp, T_PCG, 0, s, d, P, pv, q64, it, tol, iteracoes);
    if (q64) {  // the true residual, when the recursive one is within the tolerance
      lanca(k_verdade, BLOCOS_VERDADE, 256, 0, s, d, p->vizOp, q64, bolhas ? 1 : 0);
      lanca(k_verdade_fim, 1, 256, 0, s, d, BLOCOS_VERDADE, iteracoes, tol, bolhas ? 1 : 0,
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
    precondicionar(p, Juncao{d, P, zc, zo}, bloco, umaPassada, s);
    std::swap(zc, zo);
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
  aposAnterior();
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < N) x[c] = carregar(x0[c]);
}
int cicloVDispositivo(Pcg* p, const uint8_t* tipo, const float* b, float* x, cudaStream_t s, bool preparar,
                      const int* parar) {
  if (preparar) prepararNiveis(p, tipo, false, s);
  p->parar = parar;  // the cycle's kernels return at once while *parar != 0
  Fonte F{b};
  fonteNivelUnico(p, F, s);
  const void* r = cicloV(p, F, s, false, false, x, nullptr);
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
