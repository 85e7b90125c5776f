// pcg_fundido.cu — FUSED engine of the MGPCG pressure projection: the whole solve of
// resolverPCG (js/pressao-cpu.js:296-402) in ONE persistent cooperative launch.
//
// One CTA of 384 threads per SM (12 warps: room for ~170 registers a thread); phases are separated by a grid barrier (monotonic arrival
// counter, release-add / acquire-poll) whose waits are bounded: a wait that exceeds ~1 s sets
// an error flag, every CTA returns, and the host reports TQ_E_TIMEOUT.
// Per PCG iteration: [DA] beta and p = z + beta p fused with A p and p.Ap, [B] alpha and the q/r/bubble
// updates with r.r, [C] the convergence test fused with spreading the residual into the V-cycle's
// right-hand side, the V-cycle, and the gather of z with r.z and r.zOld.
// The V-cycle is the reference's preconditioner (cicloV, js/pressao-cpu.js:241-255):
//   - grid levels: the snapshot block smoother with one WARP per 16x16 block (8 cells per
//     lane, warp-synchronous red-black sweeps in registers); the prolongation of the coarse
//     correction is folded into the loads of the first smoother pass on the way up; the
//     restriction marches up the fine rows in registers;
//   - the coarse levels (the largest suffix of levels fitting in ~200 KB) run inside CTA 0's
//     shared memory, warps mapped to rows, while the other CTAs wait at the barrier.
// Scalars (alpha, beta, norms) are FP64 sums of per-CTA partials in a fixed order, computed
// redundantly by every CTA after the barrier, so all CTAs hold the same bits without another
// barrier; per-bubble sums are 64-bit fixed point as in the plain engine.
#include <cstdio>
#include <cstdlib>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "pcg_interno.cuh"
#include "suavizador.cuh"

namespace tq {

constexpr int TF = 384;
constexpr int WARPS = TF / 32;
constexpr long long LIMITE_CICLOS = 2000000000LL;  // ~1 s at 1.9 GHz
constexpr double ESC = 1099511627776.0;            // 2^40, per-bubble fixed point
constexpr size_t SMEM_GROSSO_MAX = 200 * 1024;
// Levels up to this many cells run in CTA 0's coarse section; larger ones as grid phases,
// where their 16x16 blocks spread over the SMs instead of queueing on one SM's warps.
constexpr size_t SECAO_MAX_CELULAS = 2048;
// The coarsest solve as a stored matrix: up to DENSO_MAX changing cells (water with a free
// neighbour) on a coarsest level of at most DENSO_MAPA_MAX cells.  Layout at offDenso: the
// matrix (DENSO_MAX^2 floats), the cells (int), their neighbours' list indices (4 int each),
// 1/k (float), and a header (count, count of colour 0).
constexpr int DENSO_MAX = 128;
constexpr int DENSO_MAPA_MAX = DENSO_MAX * DENSO_MAX;
constexpr size_t DENSO_BYTES = (size_t)DENSO_MAX * DENSO_MAX * 4 + (size_t)DENSO_MAX * 4 * 6 + 16;
constexpr size_t SMEM_CTA_MAX = 227 * 1024 - 2048;  // dynamic shared memory cap (static share aside)
// The whole coarse section (levels Lc..L-1 of the V-cycle, from x = 0) is a linear map of level
// Lc's right side, fixed during a solve.  For a top section level of at most SECAO_DENSA_MAX
// cells, a solve that may run at least SECAO_DENSA_MIN_ITERS iterations builds that map once (a
// column per water cell, every CTA running the section on unit vectors) and applies it as one
// grid-wide matrix-vector product per V-cycle, instead of CTA 0 running the section alone.
constexpr int SECAO_DENSA_MAX = 2048;
constexpr int SECAO_DENSA_MIN_ITERS = 30;
// The build runs up to SECAO_EQUIPES teams of warps a CTA, a column each, and takes from a column's top
// level only the blocks its unit vector reaches (secaoGrossa): 370 -> 215 us a solve on the 480x270
// scene, 205 -> 145 us on the 840x536 scene, 15.8 -> 2.7 ms on a 256x92 tank atlas with 4 CTAs.
constexpr int SECAO_EQUIPES = 3;
// A section has at most 5 levels: they halve while both sides exceed 12, from SECAO_MAX_CELULAS cells.
constexpr int SECAO_NIVEIS = 6;
// The coarsest level's sweeps hold their cells in registers, up to GROSSO_REG a colour and thread.
constexpr int GROSSO_REG = 4;
// Partial sums a CTA leaves for the next phase: channels 0 and 1 of the gather, the true residual and the
// start, 2 of [DA], 3 of [B].  A phase that reads a channel writes another: a fast CTA may end it before a
// slow one has read.
constexpr int NPARC = 4;
// Tolerance mode replaces the recursive FP32 residual by the true one (FP64) each time the
// recursive one has fallen by this factor since the last replacement: the rounding it gathers,
// about 1e-7 of the residual it started from per iteration, then stays far below the tolerance.
constexpr double FATOR_TROCA = 1e-3;
// With tanks (tq_set_tanks) the whole grid's recursive residual below the tolerance only starts
// the per-tank checks of the true residual: one every VERIF_TANQUES iterations.  Measured on the
// 256-tank batch: 4,069 tank-substeps/s every 2 iterations, 3,993 every one (more checks), 3,955
// every 4 (more iterations past the stop).
constexpr int VERIF_TANQUES = 2;
constexpr int PERFIL_MAX = 1 << 16;                // phase-trace capacity
constexpr int PERFIL_SECAO = 1 << 14;              // coarse-section stamps (after the phase trace)
// per-warp shared-memory areas (floats)
constexpr int CT = 121;                            // 11x11 coarse tile for the folded prolongation
constexpr int SUAV_W = CT + 7;                     // the coarse tile of a PROL pass
// per-bubble tables a CTA keeps in its areas between two grid barriers ([DA]: two doubles a label)
constexpr size_t AREA_BOLHAS = (size_t)MAX_BOLHAS * 16;
constexpr size_t AREA_TERMOS = (size_t)(TF - 32) * 16;  // after them, terms of a sum over the bubbles

struct NivelF {
  int nx, ny, meia, pad;
  uint8_t* viz;
  uint8_t* tipo;
  void *b, *x, *tmp;
};

// Blocks of a level for a smoother pass with shift `desl`.
__host__ __device__ __forceinline__ int blocosNivel(int nx, int ny, int desl) {
  return ((nx + desl + 15) >> 4) * ((ny + desl + 15) >> 4);
}

struct Fundido {
  int G = 0, Lc = 0;
  uint8_t* solidos = nullptr;  // wall-block flags (Args::sol) of the levels that use them
  bool comParedes[MAX_NIVEIS] = {};  // level l skips wall blocks (its flags exist)
  uint8_t* sol[MAX_NIVEIS] = {};      // level l's flags in `solidos` (Args::sol)
  size_t smem = 0;
  NivelF* niveis = nullptr;  // level table (device)
  double* parc = nullptr;
  unsigned* bar = nullptr;
  int* erro = nullptr;
  long long* accZ = nullptr;
  double *zb2 = nullptr, *pb2 = nullptr;
  int* ativos = nullptr;
  int* nAtivos = nullptr;
  float *p2 = nullptr, *z2 = nullptr;
  float *xc = nullptr, *bc = nullptr;
  int offDenso = -1;  // byte offset of the coarsest level's matrix in CTA 0's shared memory
  bool secaoDensa = false;  // the section's matrix can be built (buffers below allocated)
  int equipes = 1, bytesSecao = 0;  // Args::equipes, Args::bytesSecao
  float* mSecao = nullptr;   // nW x nW, row i = water cell i of level Lc
  int *wSecao = nullptr, *wInv = nullptr, *nW = nullptr;  // water cells of level Lc, cell -> row, count
  unsigned* densoG = nullptr;  // the coarsest level's matrix, list and header, copied to the CTAs that use it
  uint16_t *op = nullptr, *rotP = nullptr;
  unsigned long long* rotB = nullptr;
  void* kern = nullptr;
  unsigned long long* perfil = nullptr;
  bool perfilar = false;
  double* q64 = nullptr;     // the FP64 iterate of a tolerance-mode solve
  long long* accV = nullptr; // per-bubble fixed-point sums of the true residual
  // Bounded-wait test hooks, read from the environment when the solver is created:
  // TQ_BARRIER_WAIT_CYCLES sets the grid barrier's limit (SM clock cycles); TQ_BARRIER_HOLD_CTA
  // and TQ_BARRIER_HOLD_CYCLES make that CTA wait that many cycles before it arrives at the
  // first barrier of the NEXT solve only (one-shot), so the other CTAs' waits run out.
  long long limite = LIMITE_CICLOS;
  int segurarCta = -1;
  long long segurarCiclos = 0;
  // red-black sweeps per smoother pass with the block preconditioner: measured on the 840x536
  // scene, 2 to 8 sweeps change the solve's time by under 5 % (fewer iterations, costlier
  // passes), so the reference's count stays
  int varredurasBloco = VARREDURAS;
};

struct Args {
  Dev d;
  int L, Lc;
  const NivelF* niv;
  uint8_t* vizOp;
  int iteracoes;
  double tol;
  int bolhas, escalar;
  double* parc;
  unsigned* bar;
  int* erro;
  long long* accZ;
  double *zb2, *pb2;
  int* ativos;
  int* nAtivos;
  float *p2, *z2;
  float *xc, *bc;
  int offDenso;  // coarsest-level matrix in CTA 0's dynamic shared memory (-1: sweeps)
  int secaoDensa;  // 1: the section may be replaced by its matrix
  int equipes, bytesSecao;  // teams of a CTA that build its columns, and the shared bytes of each
  float* mSecao;
  int *wSecao, *wInv, *nWp;
  unsigned* densoG;
  uint16_t* op;  // per-cell operator descriptor of level 0 (OP_*)
  // per-cell bubble labels of level 0, 12 bits each: bits 0-11 the cell's own (air of an active
  // bubble), 12-23 / 24-35 / 36-47 / 48-59 its left / right / down / up neighbour's (0: none)
  unsigned long long* rotB;
  uint16_t* rotP;  // the cell's own label where the V-cycle spreads to and gathers from it, else 0
  unsigned long long* perfil;  // [0] count, [1..] %globaltimer at each barrier (null: off)
  // per level: 1 per 16x16 block whose cells are all wall (out-of-grid cells count as wall), the
  // blocks of shift 0 then those of shift 8; null where the level does not skip wall blocks
  uint8_t* sol[MAX_NIVEIS];
  long long limite;          // grid barrier wait limit (cycles)
  int segurarCta;            // test hook: this CTA arrives late at the first barrier (-1: none)
  long long segurarCiclos;   // ... after waiting this many cycles (bounded)
  int bloco;  // TQ_PRECOND_BLOCK: bubble rows Jacobi, V-cycle on water, coarse masks from faces
  int varreduras;  // red-black sweeps per smoother pass (VARREDURAS, the reference's, unless BLOCK)
  int umaPassada;  // BLOCK_1: one smoother pass a leg on the grid levels above 0 (see cicloV)
  // tolerance mode: q accumulates in FP64 (q64) and the solve stops on the true residual
  // ||b - A q64|| (FP64), with residual replacement; null in fixed-count mode
  double* q64;
  long long* accV;
};

// The level table, copied into shared memory at kernel start: every phase reads its level's
// sizes and pointers without an L2 round trip in front of its first data load.
__shared__ NivelF s_niv[MAX_NIVEIS];

// Phase trace of the fused solve (the %globaltimer at every grid barrier of the last solve).
void perfilFundido(Fundido* f, bool ligar) {
  if (!f) return;
  f->perfilar = ligar;
  if (ligar && !f->perfil) {
    if (cudaMalloc(&f->perfil, (PERFIL_MAX + 2 + PERFIL_SECAO) * sizeof(unsigned long long)) != cudaSuccess) {
      f->perfil = nullptr;
      f->perfilar = false;
    }
  }
}
int lerPerfilFundido(Fundido* f, unsigned long long* out, int cap) {
  if (!f || !f->perfil) return 0;
  if (cap < 0) {  // the coarse-section stamps instead of the phase trace
    unsigned long long n = 0;
    if (cudaMemcpy(&n, f->perfil + PERFIL_MAX + 1, sizeof n, cudaMemcpyDeviceToHost) != cudaSuccess) return 0;
    if (n > PERFIL_SECAO) n = PERFIL_SECAO;
    int k = (int)(n < (unsigned long long)(-cap) ? n : (unsigned long long)(-cap));
    if (k > 0 && cudaMemcpy(out, f->perfil + PERFIL_MAX + 2, k * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 0;
    return k;
  }
  unsigned long long n = 0;
  if (cudaMemcpy(&n, f->perfil, sizeof n, cudaMemcpyDeviceToHost) != cudaSuccess) return 0;
  if (n > PERFIL_MAX) n = PERFIL_MAX;
  int k = (int)(n < (unsigned long long)cap ? n : (unsigned long long)cap);
  if (k > 0 && cudaMemcpy(out, f->perfil + 1, k * sizeof(unsigned long long), cudaMemcpyDeviceToHost) != cudaSuccess)
    return 0;
  return k;
}

// ---------------------------------------------------------------- small helpers
template <class T>
__device__ __forceinline__ T ldcg(const T* p) { return __ldcg(p); }
template <>
__device__ __forceinline__ __half ldcg<__half>(const __half* p) {
  return __ushort_as_half(__ldcg((const unsigned short*)p));
}
template <>
__device__ __forceinline__ __nv_bfloat16 ldcg<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __ushort_as_bfloat16(__ldcg((const unsigned short*)p));
}
__device__ __forceinline__ int ldcg8(const uint8_t* p) { return (int)__ldcg((const unsigned char*)p); }
// Loads of a smoother pass's snapshot, right-hand side and masks: through L1 (ld.ca), where
// the lines a warp shares with the blocks beside it may already be.  These arrays were last
// written before the grid barrier that opens the pass, whose acquire orders the loads after
// those writes (PTX memory model; the cache operator is a hint), and the pass writes other
// arrays.  Measured: 1,085 against 1,099 us per iteration on the 38,370x316 atlas, no change
// on the 840x536 scene.
template <class T>
__device__ __forceinline__ T ldsv(const T* p) { return __ldca(p); }
template <>
__device__ __forceinline__ __half ldsv<__half>(const __half* p) {
  return __ushort_as_half(__ldca((const unsigned short*)p));
}
template <>
__device__ __forceinline__ __nv_bfloat16 ldsv<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __ushort_as_bfloat16(__ldca((const unsigned short*)p));
}
__device__ __forceinline__ int ldsv8(const uint8_t* p) { return (int)__ldca((const unsigned char*)p); }

__device__ __forceinline__ void gravarN(int meia, void* v, int c, float x) {
  if (meia == 0) ((float*)v)[c] = x;
  else if (meia == 1) ((__half*)v)[c] = __float2half_rn(x);
  else ((__nv_bfloat16*)v)[c] = __float2bfloat16_rn(x);
}

__device__ __forceinline__ unsigned lerAdquirir(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void somarLiberar(unsigned* p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Grid barrier: every CTA adds 1 (release) to a counter that only grows during the solve and
// waits (acquire) until it reaches epoch * gridDim.  The wait is bounded.  Returns false when
// this CTA gave up (its wait ran out, or it saw another CTA's error flag while waiting); a CTA
// that gave up returns, so the others give up at their next barrier.
__device__ bool barreira(const Args& a, unsigned& epoca) {
  __shared__ int falhou;
  __syncthreads();
  if (threadIdx.x == 0) {
    if (epoca == 0 && (int)blockIdx.x == a.segurarCta) {  // test hook: a late arrival, bounded
      const long long t = clock64();
      while (clock64() - t < a.segurarCiclos) __nanosleep(1000);
    }
    epoca++;
    const unsigned alvo = epoca * gridDim.x;
    somarLiberar(a.bar, 1u);
    long long t0 = clock64();
    int f = 0;
    for (unsigned voltas = 0;; voltas++) {
      if (lerAdquirir(a.bar) >= alvo) break;
      if ((voltas & 255u) == 255u) {
        if (*(volatile int*)a.erro) {
          f = 1;
          break;
        }
        if (clock64() - t0 > a.limite) {
          atomicExch(a.erro, 1);
          f = 1;
          break;
        }
      }
    }
    falhou = f;
    if (a.perfil && blockIdx.x == 0) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      unsigned long long k = a.perfil[0]++;
      if (k < PERFIL_MAX) a.perfil[1 + k] = t;
    }
  }
  __syncthreads();
  return falhou == 0;
}

// What bounds the short phases is latency and code: an iteration runs through more of it than the SM's
// instruction cache holds (about 128 KB; code outside it is fetched at 6 to 15 cycles an instruction, 2
// inside).  So chains of dependent steps stay rolled loops, and rare work takes little code.

// Block sums of two doubles (valid in thread 0).
__device__ __forceinline__ double2 somaBloco2(double u, double v, double* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll 1
  for (int o = 16; o > 0; o >>= 1) {
    u += __shfl_down_sync(0xffffffffu, u, o);
    v += __shfl_down_sync(0xffffffffu, v, o);
  }
  __syncthreads();
  if (lane == 0) {
    sh[w] = u;
    sh[16 + w] = v;
  }
  __syncthreads();
  if (w == 0) {
    u = lane < WARPS ? sh[lane] : 0.0;
    v = lane < WARPS ? sh[16 + lane] : 0.0;
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) {
      u += __shfl_down_sync(0xffffffffu, u, o);
      v += __shfl_down_sync(0xffffffffu, v, o);
    }
  }
  return make_double2(u, v);
}
__device__ __forceinline__ double somaBloco(double v, double* sh) { return somaBloco2(v, 0.0, sh).x; }

// Warp 0's sums of the per-CTA partials of two channels, in CTA order (valid in lane 0).  Loads go out
// in batches before the sums (a rolled load-add loop waits one L2 round trip per step); each lane
// still adds its terms in ascending order.
__device__ __forceinline__ double2 somaParciais(const double* parc) {
  const int t = threadIdx.x, G = gridDim.x;
  double v0 = 0, v1 = 0;
  constexpr int UC = 5;  // 5 x 32 slots cover one CTA per SM
#pragma unroll 1
  for (int k0 = t; k0 < G; k0 += 32 * UC) {
    double2 p[UC];
#pragma unroll
    for (int u = 0; u < UC; u++)
      p[u] = k0 + 32 * u < G ? __ldcg((const double2*)(parc + (k0 + 32 * u) * NPARC)) : make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < UC; u++) {
      v0 += p[u].x;
      v1 += p[u].y;
    }
  }
  __syncwarp();
#pragma unroll 1
  for (int o = 16; o > 0; o >>= 1) {
    v0 += __shfl_down_sync(0xffffffffu, v0, o);
    v1 += __shfl_down_sync(0xffffffffu, v1, o);
  }
  return make_double2(v0, v1);
}

// Sums, in CTA order, of the per-CTA partials of channel CANAL (DOIS: and the next), plus up to two sums over
// the active bubbles (ascending labels): termos(b, t0, t1) makes bubble b's terms.  Warp 0 of every CTA
// sums the same data in the same order, so every CTA obtains the same bits; the other warps make the
// terms meanwhile (and what else termos stores in shared memory, visible after the call), a bubble a
// thread: code for one bubble, not for a batch of them.  Called only after a grid barrier, whose last step
// is a __syncthreads(): sh is free, and the next writer of sh (a block sum) synchronises first.
constexpr int LOTE_TERMOS = TF - 32;  // a multiple of 32: lane l of warp 0 adds terms l, l + 32, ...
template <bool DOIS, int CANAL, class F>
__device__ __forceinline__ void somasGlobais(const Args& a, int nAt, F termos, double* sh, double out[4], float* areas) {
  double* T = (double*)(areas + AREA_BOLHAS / 4);
  const int t = threadIdx.x;
  double2 v = make_double2(0.0, 0.0);
  double b0 = 0, b1 = 0;
  if (t < 32) v = somaParciais(a.parc + (CANAL & 2));
  if (CANAL & 1) v.x = v.y;
#pragma unroll 1
  for (int k0 = 0; k0 < nAt; k0 += LOTE_TERMOS) {
    const int n = min(LOTE_TERMOS, nAt - k0);
    if (t >= 32 && t - 32 < n) {
      double t0 = 0, t1 = 0;
      termos(__ldcg(&a.ativos[k0 + t - 32]), t0, t1);
      T[t - 32] = t0;
      if (DOIS) T[LOTE_TERMOS + t - 32] = t1;
    }
    __syncthreads();
    if (t < 32)
#pragma unroll 1
      for (int u = t; u < n; u += 32) {
        b0 += T[u];
        if (DOIS) b1 += T[LOTE_TERMOS + u];
      }
    if (k0 + LOTE_TERMOS < nAt) __syncthreads();
  }
  if (t < 32) {
    if (nAt > 0)
#pragma unroll 1
      for (int o = 16; o > 0; o >>= 1) {
        b0 += __shfl_down_sync(0xffffffffu, b0, o);
        if (DOIS) b1 += __shfl_down_sync(0xffffffffu, b1, o);
      }
    if (t == 0) {
      sh[0] = v.x;
      sh[1] = v.y;
      sh[2] = b0;
      sh[3] = b1;
    }
  }
  __syncthreads();
  out[0] = sh[0];
  out[1] = sh[1];
  out[2] = sh[2];
  out[3] = sh[3];
}

__device__ __forceinline__ bool bolhaAtiva(const Args& a, uint32_t r) {
  return r >= 2 && r < (uint32_t)MAX_BOLHAS && __ldcg(&a.d.facesB[r]) > 0;
}

// The preconditioned residual z_b of active bubble b: REFERENCE, the mean V-cycle correction
// over its cells (the gather's fixed-point sum, precondicionar js/pressao-cpu.js:357-361);
// BLOCK, a Jacobi step on its row, r_b / faces_b (its diagonal).
__device__ __forceinline__ double zbDe(const Args& a, int b) {
  return a.bloco ? __ldcg(&a.d.rb[b]) / (double)__ldcg(&a.d.facesB[b]) : (double)__ldcg(&a.accZ[b]) / ESC;
}

// Free-neighbour bits (0-3: left, right, down, up) of coarse cell (I, J) of level g from the
// faces of its finer level f (TQ_PRECOND_BLOCK): a coarse face is open when both coarse cells
// are not wall and a fine face across it (between fine columns 2I+1 and 2I+2 in rows 2J, 2J+1,
// or the vertical counterpart) joins two non-wall fine cells.  Walls thinner than a coarse cell
// then still separate the water on either side.
__device__ __noinline__ int vizinhosPorFaces(const NivelF& f, const NivelF& g, int I, int J) {
  const int C = I + J * g.nx;
  if (ldcg8(g.tipo + C) == SOLIDO) return 0;
  auto livre = [&](int i, int j) {
    return i >= 0 && j >= 0 && i < f.nx && j < f.ny && ldcg8(f.tipo + i + j * f.nx) != SOLIDO;
  };
  auto horiz = [&](int i0, int i1) {
    return (livre(i0, 2 * J) && livre(i1, 2 * J)) || (livre(i0, 2 * J + 1) && livre(i1, 2 * J + 1));
  };
  auto vert = [&](int j0, int j1) {
    return (livre(2 * I, j0) && livre(2 * I, j1)) || (livre(2 * I + 1, j0) && livre(2 * I + 1, j1));
  };
  int m = 0;
  if (I > 0 && ldcg8(g.tipo + C - 1) != SOLIDO && horiz(2 * I - 1, 2 * I)) m |= 1;
  if (I < g.nx - 1 && ldcg8(g.tipo + C + 1) != SOLIDO && horiz(2 * I + 1, 2 * I + 2)) m |= 2;
  if (J > 0 && ldcg8(g.tipo + C - g.nx) != SOLIDO && vert(2 * J - 1, 2 * J)) m |= 4;
  if (J < g.ny - 1 && ldcg8(g.tipo + C + g.nx) != SOLIDO && vert(2 * J + 1, 2 * J + 2)) m |= 8;
  return m;
}

// Per-cell operator descriptor of level 0 (built once per solve): bits 0-3 the left, right,
// down and up neighbours are water; OP_AGUA the cell is water; OP_FACE interior air of an
// active bubble (its water faces enter the bubble's row); OP_VIZ_BOLHA a free neighbour is
// air of an active bubble; OP_BOLHA air of an active bubble; bits 8-10 the number of free
// (non-wall) neighbours.
constexpr int OP_AGUA = 16, OP_FACE = 32, OP_VIZ_BOLHA = 64, OP_BOLHA = 128;
// Level 0's neighbour masks also carry, above bits 0-4, the cell's OP_BOLHA and OP_AGUA.
constexpr int V0_BOLHA = 32, V0_AGUA = 64;

// Adds v to bubble lab's fixed-point sum (lab 0: nothing), by the whole warp: one atomic a label and warp.
// A large bubble's cells would otherwise queue thousands of atomics on one address, which bounded the
// phases that make these sums.  Integer sums: any grouping gives the same result.
__device__ __forceinline__ void somarBolhaWarp(long long* acc, int lab, long long v) {
  unsigned resto = __ballot_sync(0xffffffffu, lab && v);
#pragma unroll 1
  while (resto) {
    const int l0 = __shfl_sync(0xffffffffu, lab, __ffs(resto) - 1);
    const bool meu = lab == l0;
    long long t = meu ? v : 0;
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0 && t) atomicAdd((unsigned long long*)&acc[l0], (unsigned long long)t);
    resto &= ~__ballot_sync(0xffffffffu, meu);
  }
}

// ---------------------------------------------------------------- grid-level smoother
// Modes of a smoother pass over a grid level:
//   M_NORMAL   snapshot = src, right side = b; with `zero`, snapshot = 0: the first pass on the way
//              down, whose x the restriction leaves at 0 (js/pressao-cpu.js:186);
//   M_PROL     snapshot = x + P(x_coarse) (prolongar, js/pressao-cpu.js:191-214), built while
//              loading: the first pass on the way up;
//   M_ESPALHAR level 0, first pass: snapshot 0 (:354); also spreads the residual into b
//              (precondicionar, js/pressao-cpu.js:353-355), b = escala * r, bubble cells their bubble's mean;
//   M_JUNTAR   level 0, last pass: instead of storing x, gathers z = x / escala (:357-361),
//              bubble cells' share into the bubble's fixed-point sum, and the partials of r.z
//              and r.zOld.
enum { M_NORMAL = 0, M_PROL = 1, M_ESPALHAR = 2, M_JUNTAR = 3 };

// What the spread and the gather need (level 0).
struct Reuniao {
  float escala;          // b = escala * residual; z = x / escala
  float* zNovo;
  const float* zVelho;   // previous z (r.zOld), or null
};

// Bilinear coarse correction at fine cell (sx, sy) from the 11x11 coarse tile ct whose origin is
// (cx0, cy0) (prolongar, js/pressao-cpu.js:191-214).
__device__ __forceinline__ float correcaoGrossa(const float* ct, int cx0, int cy0, int sx, int sy) {
  const int I0 = grossoBaseF(sx) - cx0, J0 = grossoBaseF(sy) - cy0;
  const float wx0 = pesoBaseF(sx), wy0 = pesoBaseF(sy);
  float e = 0.0f;
#pragma unroll
  for (int b = 0; b < 2; b++) {
    const float wy = b ? 1.0f - wy0 : wy0;
#pragma unroll
    for (int aa = 0; aa < 2; aa++) e += ct[(J0 + b) * 11 + I0 + aa] * ((aa ? 1.0f - wx0 : wx0) * wy);
  }
  return e;
}

// suavizar (js/pressao-cpu.js:99-150) for one 16x16 block, by one warp, in registers (see
// meiaReg).  Every global load of the block (cells, frame, flags, right side; with PROL the
// coarse tile) goes out in one batch.
template <class T, int MODO>
__device__ __forceinline__ void suavizarBloco(const Args& a, const NivelF& n, int blk, int nbx, int desl, bool masc, bool zero, int ordem,
                                              const T* src, T* dst, float* area, const NivelF& g,
                                              const float* xcSecao, const Reuniao& ru, double& s0, double& s1) {
  constexpr bool PROL = MODO == M_PROL;
  const bool ZERO = MODO == M_ESPALHAR || (MODO == M_NORMAL && zero);
  const int lane = threadIdx.x & 31, gl = lane >> 3, k = lane & 7;
  const int bx = blk % nbx, by = blk / nbx;
  const int ox = bx * 16 - desl, oy = by * 16 - desl;
  const int nx = n.nx, ny = n.ny;
  const T* b = (const T*)n.b;
  // PROL: the coarse tile (columns from (ox-2)>>1, rows from (oy-2)>>1, 11x11) is loaded first,
  // so that every load of the block is in flight before any result is used.  Coarse x is 0 off
  // water (a grid level's snapshot, or the section's output, zeroed before the solve off water),
  // so the tile needs no water flags.
  const int cx0 = (ox - 2) >> 1, cy0 = (oy - 2) >> 1;
  float cv[4];
  if (PROL) {
    int C[4];
    bool ok[4];
#pragma unroll
    for (int kk = 0; kk < 4; kk++) {
      const int s = lane + 32 * kk;
      const int I = cx0 + s % 11, J = cy0 + s / 11;
      ok[kk] = s < CT && I >= 0 && J >= 0 && I < g.nx && J < g.ny;
      C[kk] = ok[kk] ? I + J * g.nx : 0;
    }
    // the coarse values' storage type is chosen once (warp-uniform), so the four loads are
    // straight-line code in flight together
    // (a level below the section is stored as T, see criarFundido)
    if (xcSecao) {
#pragma unroll
      for (int kk = 0; kk < 4; kk++) cv[kk] = ok[kk] ? __ldcg(xcSecao + C[kk]) : 0.0f;
    } else {
      T cR[4];
#pragma unroll
      for (int kk = 0; kk < 4; kk++) {
        cR[kk] = guardar<T>(0.0f);
        if (ok[kk]) cR[kk] = ldcg((const T*)g.x + C[kk]);
      }
#pragma unroll
      for (int kk = 0; kk < 4; kk++) cv[kk] = carregar(cR[kk]);
    }
  }
  float x[2][4], bq[2][4];  // [colour][m], see meiaReg
  T bR[2][4], xR[2][4];     // as stored
  int v[2][4], cel[2][4];
  int om[2][4];  // M_ESPALHAR, M_JUNTAR: the cells' own bubble labels (0: not bubble air)
  float rv[2][4], zv[2][4];  // M_JUNTAR: the residual and the previous z
  unsigned cels[2][4];       // M_JUNTAR: the cells of the cell's bubble
  Moldura f;
  unsigned aguaF = 0;  // PROL: water flags of the frame cells (bits 0-3 left, 4-7 right, 8-9 below, 10-11 above)
#pragma unroll
  for (int cr = 0; cr < 2; cr++)
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int gx = ox + 2 * k + ((cr + 1 + m) & 1), gy = oy + 4 * gl + m;
      const bool dentro = gx >= 0 && gy >= 0 && gx < nx && gy < ny;
      const int c = gx + gy * nx;
      cel[cr][m] = dentro ? c : -1;
      v[cr][m] = 0;
      bq[cr][m] = 0.0f;
      bR[cr][m] = xR[cr][m] = guardar<T>(0.0f);
      // as stored: a load under a branch that also converts waits inside the branch, which cost the
      // 16-bit kernels 2 to 3 us a phase
      if (dentro) {
        v[cr][m] = ldsv8(n.viz + c);
        if (MODO == M_ESPALHAR) bq[cr][m] = __ldcg(a.d.r + c);
        else bR[cr][m] = ldsv(b + c);
      }
    }
  if (!ZERO)
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++)
        if (cel[cr][m] >= 0) xR[cr][m] = ldsv(src + cel[cr][m]);
  // the warp-uniform tests (bubbles the V-cycle sees, a previous z) stay outside the loads, so each
  // group of loads is straight-line code in flight with the block's
  if (MODO == M_ESPALHAR || MODO == M_JUNTAR) {
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++) om[cr][m] = 0;
    if (a.bolhas && !a.bloco)
#pragma unroll
      for (int cr = 0; cr < 2; cr++)
#pragma unroll
        for (int m = 0; m < 4; m++) om[cr][m] = cel[cr][m] >= 0 ? (int)__ldcg(a.rotP + cel[cr][m]) : 0;
  }
  if (MODO == M_JUNTAR) {
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++) {
        rv[cr][m] = cel[cr][m] >= 0 ? __ldcg(a.d.r + cel[cr][m]) : 0.0f;
        zv[cr][m] = 0.0f;
      }
    if (ru.zVelho)
#pragma unroll
      for (int cr = 0; cr < 2; cr++)
#pragma unroll
        for (int m = 0; m < 4; m++) zv[cr][m] = cel[cr][m] >= 0 ? __ldcg(ru.zVelho + cel[cr][m]) : 0.0f;
  }
  // The block's frame: lane i loads the left (i < 16) or right column's row i & 15 and the
  // bottom (i < 16) or top row's column i & 15; the lanes next to the frame (k = 0 / 7 for the
  // columns, g = 0 / 3 for the rows) take their values by shuffle.  With PROL the same two cells'
  // water flags come along (gathered by ballot below).
  int vzLR = 0, vzBT = 0;
  {
    const int fr = lane & 15;
    const int gxA = lane < 16 ? ox - 1 : ox + 16, gyA = oy + fr;
    const int gxB = ox + fr, gyB = lane < 16 ? oy - 1 : oy + 16;
    const bool okA = gxA >= 0 && gxA < nx && gyA >= 0 && gyA < ny;
    const bool okB = gxB >= 0 && gxB < nx && gyB >= 0 && gyB < ny;
    if (PROL) {
      vzLR = okA ? ldsv8(n.viz + gxA + gyA * nx) : 0;
      vzBT = okB ? ldsv8(n.viz + gxB + gyB * nx) : 0;
    }
    T fA = guardar<T>(0.0f), fB = guardar<T>(0.0f);
    if (!ZERO) {
      if (okA) fA = ldsv(src + gxA + gyA * nx);
      if (okB) fB = ldsv(src + gxB + gyB * nx);
    }
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++) {
        if (MODO != M_ESPALHAR) bq[cr][m] = carregar(bR[cr][m]);
        x[cr][m] = ZERO ? 0.0f : carregar(xR[cr][m]);
      }
    if (ZERO) {
#pragma unroll
      for (int m = 0; m < 4; m++) f.esq[m] = f.dir[m] = 0.0f;
#pragma unroll
      for (int j = 0; j < 2; j++) f.bai[j] = f.cim[j] = 0.0f;
    } else {
      const float xA = carregar(fA), xB = carregar(fB);
#pragma unroll
      for (int m = 0; m < 4; m++) f.esq[m] = f.dir[m] = __shfl_sync(0xffffffffu, xA, (k == 7 ? 16 : 0) + 4 * gl + m);
#pragma unroll
      for (int j = 0; j < 2; j++) f.bai[j] = f.cim[j] = __shfl_sync(0xffffffffu, xB, (gl == 3 ? 16 : 0) + 2 * k + j);
    }
  }
  if (MODO == M_ESPALHAR) {
    // cells of active bubbles take their bubble's mean residual; b is stored in the storage
    // type and the sweep uses the stored value
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++) {
        if (cel[cr][m] < 0) continue;
        float val = bq[cr][m];
        if (om[cr][m]) val = area[om[cr][m]];
        const T bt = guardar<T>(val * ru.escala);
        ((T*)n.b)[cel[cr][m]] = bt;
        bq[cr][m] = carregar(bt);
      }
  }
  if (PROL) {
    // the frame's water flags of this lane's frame cells: bits 0-3 left rows 4g..4g+3 (k = 0),
    // 4-7 right (k = 7), 8-9 below columns 2k, 2k+1 (g = 0), 10-11 above (g = 3)
    const unsigned mLR = __ballot_sync(0xffffffffu, (vzLR & 16) != 0);
    const unsigned mBT = __ballot_sync(0xffffffffu, (vzBT & 16) != 0);
    if (k == 0) aguaF |= (mLR >> (4 * gl)) & 0xFu;
    if (k == 7) aguaF |= ((mLR >> (16 + 4 * gl)) & 0xFu) << 4;
    if (gl == 0) aguaF |= ((mBT >> (2 * k)) & 3u) << 8;
    if (gl == 3) aguaF |= ((mBT >> (16 + 2 * k)) & 3u) << 10;
    // coarse tile: columns from (ox-2)>>1, rows from (oy-2)>>1, 11x11 (x, 0 off water and off
    // the grid); the snapshot of every fine water cell, frame included, is x + P(x_coarse)
    float* ct = area;
#pragma unroll
    for (int kk = 0; kk < 4; kk++) {
      const int s = lane + 32 * kk;
      if (s < CT) ct[s] = cv[kk];
    }
    __syncwarp();
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++)
        if (v[cr][m] & 16) x[cr][m] += correcaoGrossa(ct, cx0, cy0, ox + 2 * k + ((cr + 1 + m) & 1), oy + 4 * gl + m);
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int gy = oy + 4 * gl + m;
      if (aguaF >> m & 1) f.esq[m] += correcaoGrossa(ct, cx0, cy0, ox - 1, gy);
      if (aguaF >> (4 + m) & 1) f.dir[m] += correcaoGrossa(ct, cx0, cy0, ox + 16, gy);
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int gx = ox + 2 * k + j;
      if (aguaF >> (8 + j) & 1) f.bai[j] += correcaoGrossa(ct, cx0, cy0, gx, oy - 1);
      if (aguaF >> (10 + j) & 1) f.cim[j] += correcaoGrossa(ct, cx0, cy0, gx, oy + 16);
    }
    __syncwarp();
  }
  if (MODO == M_JUNTAR)
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++) cels[cr][m] = om[cr][m] ? __ldcg(a.d.celsB + om[cr][m]) : 1u;
  // a block with no cell to update (air, solid, walled-in water) keeps its values: the warp skips
  // the sweeps (fmaf(0, d, q) = q for every cell of the block)
  bool mexe = false;
#pragma unroll
  for (int cr = 0; cr < 2; cr++)
#pragma unroll
    for (int m = 0; m < 4; m++) mexe |= (v[cr][m] & 16) && (v[cr][m] & 15);
  // (level 0's masks close no face between water cells: x = 0 off water, so it needs no masking)
  if (__any_sync(0xffffffffu, mexe))
    varrerReg(x, v, bq, f, ordem, MODO != M_ESPALHAR && MODO != M_JUNTAR && masc, a.varreduras);
  if (MODO == M_JUNTAR) {
    const float inv = 1.0f / ru.escala;
    bool bolha = false;
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++) {
        const int c = cel[cr][m];
        bolha |= om[cr][m] != 0;
        const float xz = carregar(guardar<T>((v[cr][m] & 16) ? x[cr][m] : 0.0f)) * inv;
        x[cr][m] = xz;
        if (c < 0) continue;
        ru.zNovo[c] = om[cr][m] ? 0.0f : xz;
        if ((v[cr][m] & V0_AGUA) && !om[cr][m]) {
          s0 += (double)rv[cr][m] * (double)xz;
          if (ru.zVelho) s1 += (double)rv[cr][m] * (double)zv[cr][m];
        }
      }
    if (__any_sync(0xffffffffu, bolha)) {
      // a bubble cell's share of z goes to its bubble's fixed-point sum; the lane adds its
      // consecutive cells of one bubble before the atomic (integer sums: same result).  A rolled loop
      // over the cells, through shared memory: the FP64 division's code once.
#pragma unroll
      for (int cr = 0; cr < 2; cr++)
#pragma unroll
        for (int m = 0; m < 4; m++) {
          float* o = area + (4 * cr + m) * 32 + lane;
          o[0] = x[cr][m];
          ((int*)o)[256] = om[cr][m];
          ((unsigned*)o)[512] = cels[cr][m];
        }
      int labA = 0;
      long long acc = 0;
#pragma unroll 1
      for (int q = 0; q < 8; q++) {
        const float* o = area + q * 32 + lane;
        const int lab = ((const int*)o)[256];
        if (!lab) continue;
        if (lab != labA) {
          if (labA && acc) atomicAdd((unsigned long long*)&a.accZ[labA], (unsigned long long)acc);
          labA = lab;
          acc = 0;
        }
        acc += __double2ll_rn((double)o[0] / ((const unsigned*)o)[512] * ESC);
      }
      somarBolhaWarp(a.accZ, labA, acc);
    }
  } else {
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++)
        if (cel[cr][m] >= 0) dst[cel[cr][m]] = guardar<T>((v[cr][m] & 16) ? x[cr][m] : 0.0f);
  }
}

template <class T, int MODO>
__device__ __forceinline__ void faseSuavizarT(const Args& a, int l, int desl, bool paraTmp, bool zero, int ordem,
                                           float* areas, const Reuniao& ru, double* sh) {
  const NivelF n = s_niv[l];
  const int nbx = (n.nx + desl + 15) >> 4, nby = (n.ny + desl + 15) >> 4;
  const int nb = nbx * nby;
  const int w = threadIdx.x >> 5;
  // the spread reads the CTA's bubble means, the gather takes 3 words a cell of its block
  float* area = MODO == M_ESPALHAR ? areas : areas + w * (MODO == M_JUNTAR ? 768 : SUAV_W);
  const T* src = (const T*)(paraTmp ? n.x : n.tmp);
  T* dst = (T*)(paraTmp ? n.tmp : n.x);
  NivelF g{};
  if (MODO == M_PROL) g = s_niv[l + 1];
  const float* xcSecao = (MODO == M_PROL && l + 1 == a.Lc) ? a.xc : nullptr;
  double s0 = 0.0, s1 = 0.0;
  // with more blocks than warps (exc > 0), the warps that take two blocks take the last 2 exc
  // blocks of the row-major order, the top rows: air above the water in a tank, whose blocks
  // skip their sweeps, so the pass lasts about one water block
  const int tot = WARPS * gridDim.x, exc = nb - tot;
  const int tw = w * gridDim.x + blockIdx.x;  // the warp's first block index
  auto blocoDe = [&](int t) { return exc > 0 ? nb - 1 - (t + exc) % nb : t; };
  // Blocks of wall alone are skipped on the levels that flag them: their cells hold x = 0 in both
  // snapshots (zeroed before the solve, and a pass writes 0 off water) and b = 0, so a pass would
  // rewrite the same zeros.  The flags of the warp's first 32 blocks come in one load, lane k's for
  // its k-th.
  const uint8_t* fl = a.sol[l] ? a.sol[l] + (desl ? blocosNivel(n.nx, n.ny, 0) : 0) : nullptr;
  unsigned paredes = 0;
  if (fl) {
    const int tk = tw + (threadIdx.x & 31) * tot;
    paredes = __ballot_sync(0xffffffffu, tk < nb && ldcg8(fl + blocoDe(tk)) != 0);
  }
  const bool masc = a.bloco && l >= 1;
  int k = 0, zr = zero;
#pragma unroll 1
  for (int t = tw; t < nb; t += tot, k++) {
    const int blk = blocoDe(t);
    if (fl && (k < 32 ? (paredes >> k) & 1u : ldcg8(fl + blk) != 0)) continue;
    if (MODO == M_NORMAL) asm volatile("" : "+r"(zr));  // or the compiler makes a copy of the loop for each leg
    suavizarBloco<T, MODO>(a, n, blk, nbx, desl, masc, zr != 0, ordem, src, dst, area, g, xcSecao, ru, s0, s1);
  }
  if (MODO == M_JUNTAR) {
    const double2 t = somaBloco2(s0, s1, sh);
    if (threadIdx.x == 0) {
      a.parc[blockIdx.x * NPARC + 0] = t.x;
      a.parc[blockIdx.x * NPARC + 1] = t.y;
    }
  }
}

// ---------------------------------------------------------------- restriction
// Two neighbouring cells of a row from an even column on, as stored (nothing is converted before every
// load is out): one load where the level's rows start on even cells (par); zeros outside the level (d: the
// first cell is inside, d1: the second).
template <class T>
struct Par {
  unsigned w;
  T a, b;
};
template <>
struct Par<float> {
  float2 w;
  float a, b;
};
template <class T>
__device__ __forceinline__ void lerPar(Par<T>& r, const T* p, int c, bool d, bool d1, bool par) {
  r.w = {};
  r.a = r.b = guardar<T>(0.0f);
  if (par) {
    if (d) r.w = __ldcg((const decltype(r.w)*)(p + c));
  } else {
    if (d) r.a = ldcg(p + c);
    if (d1) r.b = ldcg(p + c + 1);
  }
}
template <class T>
__device__ __forceinline__ float2 valores(const Par<T>& r, bool par) {
  if constexpr (sizeof(T) == 4) {
    return par ? r.w : make_float2(r.a, r.b);
  } else {
    T a, b;
    if constexpr (std::is_same<T, __half>::value) {
      a = __ushort_as_half((unsigned short)r.w);
      b = __ushort_as_half((unsigned short)(r.w >> 16));
    } else {
      a = __ushort_as_bfloat16((unsigned short)r.w);
      b = __ushort_as_bfloat16((unsigned short)(r.w >> 16));
    }
    return make_float2(carregar(par ? a : r.a), carregar(par ? b : r.b));
  }
}

// restringir (js/pressao-cpu.js:159-188) as a gather in registers: a warp takes 30 coarse columns (a lane
// each, lanes 0 and 31 the fine columns beside them) and marches up R coarse rows.  A lane holds its two
// fine columns of the rows in use; the neighbours' come by shuffle, and every value is loaded once a
// warp, the next row's before this row's sums.  R: one round of the grid's warps, up to 4 rows (a
// larger grid takes more rounds).  Measured on level 0 of 840x536 cells: 9.0 -> 5.2 us in FP32, 10.9 -> 5.7
// in FP16, against a footprint staged in shared memory a value a load.
template <class T>
__device__ __forceinline__ void faseRestringir(const Args& a, int l) {
  const NivelF f = s_niv[l];
  const NivelF g = s_niv[l + 1];
  const bool secao = l + 1 == a.Lc, par = !(f.nx & 1);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nseg = (g.nx + 29) / 30, tot = WARPS * gridDim.x;
  const int R = min(4, (nseg * g.ny + tot - 1) / tot), total = nseg * ((g.ny + R - 1) / R);
  const T *fx = (const T*)f.x, *fb = (const T*)f.b;
  // A region whose coarse cells lie in wall blocks of the coarse level (its shift-0 flags) is skipped:
  // those cells keep b = 0.  The flags of the warp's first 32 regions come in one go, lane k's for its
  // k-th.
  const uint8_t* flg = a.sol[l + 1];
  const int gbx = (g.nx + 15) >> 4;
  auto paredeReg = [&](int reg) {
    const int J = reg / nseg * R, I = reg % nseg * 30, bx1 = min(I + 29, g.nx - 1) >> 4, by1 = min(J + R - 1, g.ny - 1) >> 4;
    int p = 1;
#pragma unroll 1
    for (int by = J >> 4; by <= by1; by++)
#pragma unroll 1
      for (int bx = I >> 4; bx <= bx1; bx++) p &= ldcg8(flg + by * gbx + bx);
    return p != 0;
  };
  const int t0 = w * gridDim.x + blockIdx.x;
  unsigned paredes = 0;
  if (flg) {
    const int tk = t0 + lane * tot;
    paredes = __ballot_sync(0xffffffffu, tk < total && paredeReg(tk));
  }
  int kr = 0;
#pragma unroll 1
  for (int reg = t0; reg < total; reg += tot, kr++) {
    if (flg && (kr < 32 ? (paredes >> kr) & 1u : paredeReg(reg))) continue;
    const int J0 = reg / nseg * R, I = reg % nseg * 30 + lane - 1, i = 2 * I, J1 = min(J0 + R, g.ny);
    // xr: x of rows 2J .. 2J + 3; bn, vn: right side and masks of rows 2J + 1 and 2J + 2
    const bool dI = i >= 0 && i < f.nx, dI1 = dI && i + 1 < f.nx;
    float2 xr[4];
    Par<T> xn[2], bn[2];
    int vn[2], vm[2], gv = 0;
    auto lerX = [&](Par<T>& r, int j) {
      const bool d = j >= 0 && j < f.ny;
      lerPar<T>(r, fx, i + j * f.nx, d && dI, d && dI1, par);
    };
    auto ler = [&](int J) {
      gv = I >= 0 && I < g.nx && J >= J0 ? ldcg8(g.viz + I + J * g.nx) : 0;
#pragma unroll
      for (int q = 0; q < 2; q++) {
        lerX(xn[q], 2 * J + 2 + q);
        const int j = 2 * J + 1 + q, c = i + j * f.nx;
        const bool d = j >= 0 && j < f.ny && dI, d1 = d && dI1;
        lerPar<T>(bn[q], fb, c, d, d1, par);
        vn[q] = vm[q] = 0;
        if (par) {
          if (d) vn[q] = (int)__ldcg((const unsigned short*)(f.viz + c));
        } else {
          if (d) vn[q] = ldcg8(f.viz + c);
          if (d1) vm[q] = ldcg8(f.viz + c + 1);
        }
      }
    };
    {
      Par<T> u[2];
      lerX(u[0], 2 * J0 - 2);
      lerX(u[1], 2 * J0 - 1);
      ler(J0 - 1);
      xr[2] = valores<T>(u[0], par);
      xr[3] = valores<T>(u[1], par);
    }
    float rs[4][4];  // residuals of rows 2J - 1 .. 2J + 2 in columns 2I - 1 .. 2I + 2
#pragma unroll
    for (int q = 0; q < 4; q++) rs[2][q] = rs[3][q] = 0.0f;
#pragma unroll 1
    for (int J = J0 - 1; J < J1; J++) {
      xr[0] = xr[2];
      xr[1] = xr[3];
      float2 b[2];
      int v[2];
#pragma unroll
      for (int q = 0; q < 2; q++) {
        xr[2 + q] = valores<T>(xn[q], par);
        b[q] = valores<T>(bn[q], par);
        v[q] = vn[q] | vm[q] << 8;
      }
      const int gvz = gv;
      if (J + 1 < J1) ler(J + 1);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        rs[0][q] = rs[2][q];
        rs[1][q] = rs[3][q];
      }
      // b - A x on water cells, 0 elsewhere (TQ_PRECOND_BLOCK's coarse masks can close a face between
      // two water cells; elsewhere x is 0 past a closed face)
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const float2 x = xr[1 + q];
        const float xe = __shfl_up_sync(0xffffffffu, x.y, 1), xd = __shfl_down_sync(0xffffffffu, x.x, 1);
        auto residuo = [&](int m, float bb, float c, float e, float d, float bai, float cim) {
          const float t = ((((m & 1) ? e : 0.0f) + ((m & 2) ? d : 0.0f)) + ((m & 4) ? bai : 0.0f)) + ((m & 8) ? cim : 0.0f);
          return (m & 16) ? bb - fmaf((float)__popc(m & 15), c, -t) : 0.0f;
        };
        const float r0 = residuo(v[q] & 255, b[q].x, x.x, xe, x.y, xr[q].x, xr[2 + q].x);
        const float r1 = residuo(v[q] >> 8, b[q].y, x.y, x.x, xd, xr[q].y, xr[2 + q].y);
        rs[2 + q][0] = __shfl_up_sync(0xffffffffu, r1, 1);
        rs[2 + q][1] = r0;
        rs[2 + q][2] = r1;
        rs[2 + q][3] = __shfl_down_sync(0xffffffffu, r0, 1);
      }
      if (J < J0 || lane < 1 || lane > 30 || I >= g.nx) continue;
      const float pes[4] = {0.25f, 0.75f, 0.75f, 0.25f};
      float soma = 0.0f;
#pragma unroll
      for (int bb = 0; bb < 4; bb++)
#pragma unroll
        for (int aa = 0; aa < 4; aa++) soma = fmaf(rs[bb][aa], pes[aa] * pes[bb], soma);
      if (!(gvz & 16)) soma = 0.0f;
      const int C = I + J * g.nx;
      if (secao) a.bc[C] = soma;
      else gravarN(g.meia, g.b, C, soma);
    }
  }
}

// ---------------------------------------------------------------- coarse section (CTA 0)
// Level arrays live in CTA 0's dynamic shared memory and are addressed by offsets from the
// `extern __shared__` array, so every access compiles to a shared-memory access.
struct NivelS {
  int nx, ny;
  int xa, xb, b;  // float offsets
  int v;          // byte offset
};

// The threads that run a coarse section together: the CTA, or one of a.equipes teams of whole
// warps (named barrier 1 + id), thread ti of nt.
struct Equipe {
  int ti, nt, id;
};
__device__ __forceinline__ void sincEquipe(const Equipe& q) {
  if (q.nt == TF) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(q.id + 1), "r"(q.nt) : "memory");
}

// One smoother pass over a level held in shared memory: the level's 16x16 blocks (those of the
// rectangle r of block coordinates) are taken in turn by the team's warps, each sweeping its
// block in registers (varrerReg) from the snapshot `src` and writing `dst`.
struct Ret {
  int x0, y0, x1, y1;  // inclusive
};
__device__ __noinline__ void passoS(float* F, const uint8_t* U, const NivelS n, int desl, int ordem, int src, int dst, bool masc,
                       int nVarr, const Equipe& eq, const Ret& r) {
  const int lane = threadIdx.x & 31, w = eq.ti >> 5, gl = lane >> 3, k = lane & 7;
  const int nx = n.nx, ny = n.ny;
  const int nbr = r.x1 - r.x0 + 1;
  for (int b = w; b < nbr * (r.y1 - r.y0 + 1); b += eq.nt >> 5) {
    const int ox = (r.x0 + b % nbr) * 16 - desl, oy = (r.y0 + b / nbr) * 16 - desl;
    float x[2][4], bq[2][4];  // [colour][m], see meiaReg
    int v[2][4], cel[2][4];
    Moldura f;
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++) {
        const int gx = ox + 2 * k + ((cr + 1 + m) & 1), gy = oy + 4 * gl + m;
        const bool dentro = gx >= 0 && gy >= 0 && gx < nx && gy < ny;
        const int c = gx + gy * nx;
        cel[cr][m] = dentro ? c : -1;
        v[cr][m] = dentro ? (U[n.v + c] | 128) : 0;
        x[cr][m] = dentro ? F[src + c] : 0.0f;
        bq[cr][m] = dentro ? F[n.b + c] : 0.0f;
      }
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int gy = oy + 4 * gl + m;
      const bool okL = k == 0 && ox - 1 >= 0 && gy >= 0 && gy < ny;
      const bool okR = k == 7 && ox + 16 < nx && gy >= 0 && gy < ny;
      f.esq[m] = okL ? F[src + ox - 1 + gy * nx] : 0.0f;
      f.dir[m] = okR ? F[src + ox + 16 + gy * nx] : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int gx = ox + 2 * k + j;
      const bool okB = gl == 0 && gx >= 0 && gx < nx && oy - 1 >= 0;
      const bool okT = gl == 3 && gx >= 0 && gx < nx && oy + 16 < ny;
      f.bai[j] = okB ? F[src + gx + (oy - 1) * nx] : 0.0f;
      f.cim[j] = okT ? F[src + gx + (oy + 16) * nx] : 0.0f;
    }
    varrerReg(x, v, bq, f, ordem, masc, nVarr);
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++)
        if (cel[cr][m] >= 0) F[dst + cel[cr][m]] = (v[cr][m] & 16) ? x[cr][m] : 0.0f;
  }
  sincEquipe(eq);
}

// The coarsest solve (resolverGrosso, js/pressao-cpu.js:217-238) is VARREDURAS_GROSSO
// red-black sweeps from x = 0: a linear map of the right side, fixed for the whole PCG solve
// because the cell types are.  The grid builds that map once per solve: column j is the sweeps
// applied to b = e_j (stored at M[i * nL + j], so a warp applying a row touches consecutive
// words).  Each V-cycle then applies it as a matrix-vector product.  Leaves the header count > DENSO_MAX when the level has more changing
// cells, and the section keeps the sweeps.
struct Denso {
  float* M;
  int* celula;  // cell | free-neighbour mask << 24, colour 0 first
  int* viz4;    // list index of each free neighbour (left, right, down, up) or -1
  float* inv;   // 1/k
  int* cab;     // [0] count, [1] count of colour 0
};
__device__ __forceinline__ Denso denso(unsigned char* dyn, int off) {
  Denso z;
  z.M = (float*)(dyn + off);
  z.celula = (int*)(z.M + DENSO_MAX * DENSO_MAX);
  z.viz4 = z.celula + DENSO_MAX;
  z.inv = (float*)(z.viz4 + 4 * DENSO_MAX);
  z.cab = (int*)(z.inv + DENSO_MAX);
  return z;
}

// The half-sweeps of resolverGrosso as (colour) steps: sweep k takes colour 0 then 1 when k is even
// and 1 then 0 when k is odd, and a half-sweep of one colour reads the other colour alone, so the
// first half of each sweep after the first repeats the half-sweep before it and changes nothing.
// Left out are only those repeats: 65 alternating half-sweeps give the bits of all 128.
constexpr int MEIAS_GROSSO = VARREDURAS_GROSSO + 1;

// Every CTA lists the cells and neighbours; column j is swept by one warp of the grid (CTA
// j % gridDim.x), lanes over the rows, in its own shared column, and goes to the global copy
// a.densoG, which the CTAs that apply the matrix load after the next grid barrier.  One thread a
// column on CTA 0 alone took 231-299 us of every solve while the other CTAs waited.
__device__ __noinline__ void montarDenso(const Args& a, unsigned char* dyn) {
  const Denso z = denso(dyn, a.offDenso);
  const NivelF n = s_niv[a.L - 1];
  const int nx = n.nx, N = n.nx * n.ny;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int* mapa = (int*)z.M;  // cell -> list index, while the matrix is not written yet
  if (w == 0) {
    int base = 0, n0 = 0;
    for (int cor = 0; cor < 2; cor++) {
      for (int c0 = 0; c0 < N; c0 += 32) {
        const int c = c0 + lane;
        const bool minha = c < N && ((((c % nx) + (c / nx) + 1) & 1) == cor);
        const int vz = minha ? ldcg8(n.viz + c) : 0;
        const bool ok = minha && (vz & 16) && (vz & 15);
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        const int pos = base + __popc(m & ((1u << lane) - 1u));
        if (minha) mapa[c] = ok ? pos : -1;
        if (ok && pos < DENSO_MAX) z.celula[pos] = c | ((vz & 15) << 24);
        base += __popc(m);
      }
      if (cor == 0) n0 = base;
    }
    if (lane == 0) {
      z.cab[0] = base;
      z.cab[1] = n0;
    }
  }
  __syncthreads();
  const int nL = z.cab[0];
  if (nL <= DENSO_MAX) {
    for (int i = threadIdx.x; i < nL; i += TF) {
      const int e = z.celula[i], c = e & 0xffffff, mk = e >> 24;
      z.viz4[4 * i + 0] = (mk & 1) ? mapa[c - 1] : -1;
      z.viz4[4 * i + 1] = (mk & 2) ? mapa[c + 1] : -1;
      z.viz4[4 * i + 2] = (mk & 4) ? mapa[c - nx] : -1;
      z.viz4[4 * i + 3] = (mk & 8) ? mapa[c + nx] : -1;
      z.inv[i] = inversoVizinhos(__popc(mk));
    }
    __syncthreads();
    const int n0 = z.cab[1];
    float* col = z.M + w * (DENSO_MAX + 32);  // the warp's column; entry nL stays 0 (a closed neighbour)
    for (int j = w * gridDim.x + blockIdx.x; j < nL; j += WARPS * gridDim.x) {
      for (int i = lane; i <= nL; i += 32) col[i] = 0.0f;
      __syncwarp();
      for (int h = 0; h < MEIAS_GROSSO; h++) {
        const int i0 = (h & 1) ? n0 : 0, i1 = (h & 1) ? nL : n0;
        for (int i = i0 + lane; i < i1; i += 32) {
          float t = 0.0f;
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const int v = z.viz4[4 * i + q];
            t += col[v >= 0 ? v : nL];
          }
          col[i] = (t + (i == j ? 1.0f : 0.0f)) * z.inv[i];
        }
        __syncwarp();
      }
      for (int i = lane; i < nL; i += 32) a.densoG[i * nL + j] = __float_as_uint(col[i]);
      __syncwarp();
    }
  }
  if (blockIdx.x == 0) {  // the list and the header after the matrix
    __syncthreads();
    const unsigned* src = (const unsigned*)z.celula;
    constexpr int M = DENSO_MAX * DENSO_MAX;
    for (int k = threadIdx.x; k < (int)(DENSO_BYTES / 4) - M; k += TF) a.densoG[M + k] = src[k];
  }
  __syncthreads();
}

// The matrix (its used part), list and header from the global copy into this CTA's shared memory.
__device__ void carregarDenso(const Args& a, unsigned char* dyn) {
  unsigned* dst = (unsigned*)(dyn + a.offDenso);
  constexpr int M = DENSO_MAX * DENSO_MAX, R = (int)(DENSO_BYTES / 4) - M;
  const int nL = (int)__ldcg(a.densoG + M + R - 4);
  const int usado = nL <= DENSO_MAX ? nL * nL : 0;
  for (int k = threadIdx.x; k < usado; k += TF) dst[k] = __ldcg(a.densoG + k);
  for (int k = threadIdx.x; k < R; k += TF) dst[M + k] = __ldcg(a.densoG + M + k);
  __syncthreads();
}

// x = M b on the coarsest level (one warp per row, lanes over the row, fixed-order warp sum).
__device__ void aplicarDenso(const Denso& z, float* F, int xa, int b, const Equipe& eq) {
  const int lane = threadIdx.x & 31, w = eq.ti >> 5;
  const int nL = z.cab[0];
  for (int i = w; i < nL; i += eq.nt >> 5) {
    float s = 0.0f;
    for (int j = lane; j < nL; j += 32) s += z.M[i * nL + j] * F[b + (z.celula[j] & 0xffffff)];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) F[xa + (z.celula[i] & 0xffffff)] = s;
  }
}

// Stamp of the coarse-section trace (CTA 0, thread 0, when tracing).
__device__ __forceinline__ void marcaSecao(const Args& a, bool marcar = true) {
  if (marcar && a.perfil && threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    unsigned long long* base = a.perfil + PERFIL_MAX + 1;
    unsigned long long k = base[0]++;
    if (k < PERFIL_SECAO) base[1 + k] = t;
  }
}

// Levels Lc..L-1 of the V-cycle inside a CTA: loads b of level Lc (a.bc), runs the down
// passes and restrictions, the coarsest red-black solve, the prolongations and up passes, and
// stores x of level Lc (a.xc).  With coluna >= 0, the same for b = the unit vector of the section's
// water cell `coluna`, by one team, into that column of the section's matrix.  From a unit vector
// the top level's down passes and restriction change the blocks around the cell alone (every
// other block sweeps zeros into zeros), so a column takes only those; its later levels are whole.
// smem holds the team's level arrays, dyn the CTA's (the coarsest level's matrix at a.offDenso).
__device__ __noinline__ void secaoGrossa(const Args& a, unsigned char* smem, unsigned char* dyn, NivelS* tab, int coluna,
                                         const Equipe eq, bool primeira) {
  const bool marcar = coluna < 0 && blockIdx.x == 0;
  NivelS* s = tab - a.Lc;  // level l at s[l]
  float* F = (float*)smem;
  uint8_t* U = smem;
  const int lane = threadIdx.x & 31, w = eq.ti >> 5, nw = eq.nt >> 5;
  marcaSecao(a, marcar);
  if (eq.ti == 0) {
    int off = 0;  // bytes
    for (int l = a.Lc; l < a.L; l++) {
      const NivelF n = s_niv[l];
      const int N = n.nx * n.ny;
      NivelS& t = s[l];
      t.nx = n.nx;
      t.ny = n.ny;
      t.xa = off / 4;
      off += (N * 4 + 15) & ~15;
      t.xb = off / 4;
      off += (N * 4 + 15) & ~15;
      t.b = off / 4;
      off += (N * 4 + 15) & ~15;
      t.v = off;
      off += (N + 15) & ~15;
    }
  }
  sincEquipe(eq);
  const int celJ = coluna >= 0 ? __ldcg(a.wSecao + coluna) : -1;  // column build: b = unit vector
  for (int l = a.Lc; l < a.L; l++) {
    const NivelS t = s[l];
    const uint8_t* viz = s_niv[l].viz;
    const int N = t.nx * t.ny;
    if (coluna >= 0)
      for (int c = eq.ti; c < N; c += eq.nt) {
        F[t.xa + c] = F[t.xb + c] = 0.0f;
        F[t.b + c] = l == a.Lc && c == celJ ? 1.0f : 0.0f;
      }
    if (!primeira) continue;
    for (int c0 = 0; c0 < N; c0 += 4 * eq.nt) {  // loads in batches of 4 per thread
      int vv[4];
      float bb[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int c = c0 + eq.ti + k * eq.nt;
        vv[k] = c < N ? ldcg8(viz + c) : 0;
        bb[k] = (c < N && l == a.Lc && coluna < 0) ? __ldcg(a.bc + c) : 0.0f;
      }
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int c = c0 + eq.ti + k * eq.nt;
        if (c < N) {
          U[t.v + c] = (uint8_t)vv[k];
          if (coluna >= 0) continue;
          F[t.xa + c] = 0.0f;
          if (l == a.Lc) F[t.b + c] = bb[k];
        }
      }
    }
  }
  sincEquipe(eq);
  marcaSecao(a, marcar);
  const float pes[4] = {0.25f, 0.75f, 0.75f, 0.25f};
  // the block preconditioner's single pass (see cicloV) ends in xb: the level's two buffers swap
  // roles in this CTA's table (rebuilt at each call)
  auto todos = [](const NivelS& n, int desl) {
    return Ret{0, 0, ((n.nx + desl + 15) >> 4) - 1, ((n.ny + desl + 15) >> 4) - 1};
  };
  auto trocarS = [&](int l) {
    if (eq.ti == 0) {
      const int t = s[l].xa;
      s[l].xa = s[l].xb;
      s[l].xb = t;
    }
    sincEquipe(eq);
  };
  for (int l = a.Lc; l < a.L - 1; l++) {
    NivelS f = s[l];
    const NivelS g = s[l + 1];
    // the blocks and (for the restriction) cells that can hold anything but 0: all, or around celJ
    Ret r0 = todos(f, 0), r8 = todos(f, 8), rc{0, 0, f.nx - 1, f.ny - 1}, rg{0, 0, g.nx - 1, g.ny - 1};
    if (coluna >= 0 && l == a.Lc) {
      const int i = celJ % f.nx, j = celJ / f.nx;
      r0 = {i >> 4, j >> 4, i >> 4, j >> 4};
      // shift 8: the cell's block, or (after the pass of shift 0) the four over its shift-0 block
      if (a.umaPassada) r8 = {(i + 8) >> 4, (j + 8) >> 4, (i + 8) >> 4, (j + 8) >> 4};
      else r8 = {r0.x0, r0.y0, min(r0.x0 + 1, r8.x1), min(r0.y0 + 1, r8.y1)};
      // the cells of those blocks and their neighbours, and the coarse cells whose windows meet them
      rc = {max(16 * r8.x0 - 9, 0), max(16 * r8.y0 - 9, 0), min(16 * r8.x1 + 8, f.nx - 1), min(16 * r8.y1 + 8, f.ny - 1)};
      rg = {max((rc.x0 - 2) >> 1, 0), max((rc.y0 - 2) >> 1, 0), min((rc.x1 + 2) >> 1, g.nx - 1),
            min((rc.y1 + 2) >> 1, g.ny - 1)};
    }
    if (a.umaPassada) {
      passoS(F, U, f, 8, 0, f.xa, f.xb, a.bloco != 0, a.varreduras, eq, r8);
      trocarS(l);
      f = s[l];
    } else {
      passoS(F, U, f, 0, 0, f.xa, f.xb, a.bloco != 0, a.varreduras, eq, r0);
      marcaSecao(a, marcar);
      passoS(F, U, f, 8, 0, f.xb, f.xa, a.bloco != 0, a.varreduras, eq, r8);
    }
    marcaSecao(a, marcar);
    // restringir: residuals of the fine level into its free x buffer, then the 4x4 gathers.
    // Out-of-range and dry neighbours enter with weight or value 0, which adds +0 to a sum.
    {
      const int wf = rc.x1 - rc.x0 + 1, Nf = wf * (rc.y1 - rc.y0 + 1);
      const float* x = F + f.xa;
      for (int k = eq.ti; k < Nf; k += eq.nt) {
        const int c = rc.x0 + k % wf + (rc.y0 + k / wf) * f.nx;
        const int vz = U[f.v + c];
        const float a0 = x[(vz & 1) ? c - 1 : c], a1 = x[(vz & 2) ? c + 1 : c];
        const float a2 = x[(vz & 4) ? c - f.nx : c], a3 = x[(vz & 8) ? c + f.nx : c];
        const float xc = x[c], bc = F[f.b + c];
        float t = 0.0f;
        t += (vz & 1) ? a0 : 0.0f;
        t += (vz & 2) ? a1 : 0.0f;
        t += (vz & 4) ? a2 : 0.0f;
        t += (vz & 8) ? a3 : 0.0f;
        F[f.xb + c] = (vz & 16) ? bc - ((float)__popc(vz & 15) * xc - t) : 0.0f;
      }
      sincEquipe(eq);
      const float* r = F + f.xb;
      const int wg = rg.x1 - rg.x0 + 1, Ng = wg * (rg.y1 - rg.y0 + 1);
      for (int k = eq.ti; k < Ng; k += eq.nt) {
        const int I = rg.x0 + k % wg, J = rg.y0 + k / wg, C = I + J * g.nx;
        float rv[16];
#pragma unroll
        for (int bb = 0; bb < 4; bb++) {
          const int j = min(max(2 * J - 1 + bb, 0), f.ny - 1);
#pragma unroll
          for (int aa = 0; aa < 4; aa++) rv[bb * 4 + aa] = r[min(max(2 * I - 1 + aa, 0), f.nx - 1) + j * f.nx];
        }
        float sum = 0.0f;
#pragma unroll
        for (int bb = 0; bb < 4; bb++) {
          const int j = 2 * J - 1 + bb;
#pragma unroll
          for (int aa = 0; aa < 4; aa++) {
            const int i = 2 * I - 1 + aa;
            const bool dentro = i >= 0 && j >= 0 && i < f.nx && j < f.ny;
            sum += dentro ? rv[bb * 4 + aa] * (pes[aa] * pes[bb]) : 0.0f;
          }
        }
        F[g.b + C] = (U[g.v + C] & 16) ? sum : 0.0f;
        F[g.xa + C] = 0.0f;
      }
    }
    sincEquipe(eq);
    marcaSecao(a, marcar);
  }
  const bool comDenso = a.offDenso >= 0 && denso(dyn, a.offDenso).cab[0] <= DENSO_MAX;
  if (comDenso) {
    const NivelS n = s[a.L - 1];
    aplicarDenso(denso(dyn, a.offDenso), F, n.xa, n.b, eq);
  } else {
    // resolverGrosso (js/pressao-cpu.js:217-238) on every warp of the team
    const NivelS n = s[a.L - 1];
    const int nx = n.nx, N = n.nx * n.ny;
    float* x = F + n.xa;
    // The cells that change (water with a free neighbour), listed per colour in the free x
    // buffer as cell | mask << 24, colour 0 first, in cell order: each warp lists a slice of
    // the cells (a multiple of 32) at the offset of the slices before it.
    int* lista = (int*)(F + n.xb);
    __shared__ unsigned short contWs[SECAO_EQUIPES][2][WARPS];
    auto& contW = contWs[eq.id];
    const int fatia = ((N + eq.nt - 1) / eq.nt) * 32;
    const int lo = min(w * fatia, N), hi = min(lo + fatia, N);
    auto muda = [&](int c, int cor) {
      const int vz = c < hi ? U[n.v + c] : 0;
      const bool ok = c < hi && (vz & 16) && (vz & 15) && ((((c % nx) + (c / nx) + 1) & 1) == cor);
      return ok ? (c | ((vz & 15) << 24)) : -1;
    };
#pragma unroll
    for (int cor = 0; cor < 2; cor++) {
      int k = 0;
      for (int c0 = lo; c0 < hi; c0 += 32) k += __popc(__ballot_sync(0xffffffffu, muda(c0 + lane, cor) >= 0));
      if (lane == 0) contW[cor][w] = (unsigned short)k;
    }
    sincEquipe(eq);
    int cont[2] = {0, 0}, base[2] = {0, 0};
    for (int q = 0; q < nw; q++)
#pragma unroll
      for (int cor = 0; cor < 2; cor++) {
        if (q == w) base[cor] = cont[cor];
        cont[cor] += contW[cor][q];
      }
    base[1] += cont[0];
#pragma unroll
    for (int cor = 0; cor < 2; cor++) {
      int b = base[cor];
      for (int c0 = lo; c0 < hi; c0 += 32) {
        const int e = muda(c0 + lane, cor);
        const unsigned m = __ballot_sync(0xffffffffu, e >= 0);
        if (e >= 0) lista[b + __popc(m & ((1u << lane) - 1u))] = e;
        b += __popc(m);
      }
    }
    sincEquipe(eq);
    if (cont[0] <= GROSSO_REG * eq.nt && cont[1] <= GROSSO_REG * eq.nt) {
      const int ne = ((cont[0] > cont[1] ? cont[0] : cont[1]) + eq.nt - 1) / eq.nt;  // uniform
      // Up to GROSSO_REG cells a colour and thread: index, neighbours, right side and 1/k stay in
      // registers, so a half-sweep is four shared loads, the sum and a store.  (One warp walking
      // the list took 98-150 us a V-cycle on 930 to 1,000-cell levels.)  A closed neighbour
      // reads the list's first word, 0 once every thread has its cells.
      int cel[2][GROSSO_REG], vz[2][GROSSO_REG][4];
      float bq[2][GROSSO_REG], iq[2][GROSSO_REG];
      const int zero = n.xb - n.xa;
#pragma unroll
      for (int cor = 0; cor < 2; cor++)
#pragma unroll
        for (int e = 0; e < GROSSO_REG; e++) {
          const int k = eq.ti + e * eq.nt;
          const int E = k < cont[cor] ? lista[(cor ? cont[0] : 0) + k] : -1;
          const int c = E < 0 ? 0 : E & 0xffffff, mk = E < 0 ? 0 : E >> 24;
          cel[cor][e] = E < 0 ? -1 : c;
          vz[cor][e][0] = (mk & 1) ? c - 1 : zero;
          vz[cor][e][1] = (mk & 2) ? c + 1 : zero;
          vz[cor][e][2] = (mk & 4) ? c - nx : zero;
          vz[cor][e][3] = (mk & 8) ? c + nx : zero;
          bq[cor][e] = E < 0 ? 0.0f : F[n.b + c];
          iq[cor][e] = inversoVizinhos(__popc(mk));
        }
      sincEquipe(eq);
      if (eq.ti == 0) F[n.xb] = 0.0f;
      sincEquipe(eq);
      auto meia = [&](auto COR) {
        constexpr int cor = decltype(COR)::value;
#pragma unroll
        for (int e = 0; e < GROSSO_REG; e++)
          if (e < ne && cel[cor][e] >= 0) {
            float t = 0.0f;
#pragma unroll
            for (int q = 0; q < 4; q++) t += x[vz[cor][e][q]];
            x[cel[cor][e]] = (t + bq[cor][e]) * iq[cor][e];
          }
        sincEquipe(eq);
      };
#pragma unroll 1
      for (int h = 0; h < MEIAS_GROSSO; h++) {
        if (h & 1) meia(std::integral_constant<int, 1>{});
        else meia(std::integral_constant<int, 0>{});
      }
    } else {
#pragma unroll 1
      for (int h = 0; h < MEIAS_GROSSO; h++) {
        const int cor = h & 1;
        const int ini = cor ? cont[0] : 0, n_ = cont[cor];
        for (int e0 = eq.ti; e0 < n_; e0 += 2 * eq.nt) {
          const int eA = e0, eB = e0 + eq.nt;
          const int EA = lista[ini + eA], EB = eB < n_ ? lista[ini + eB] : -1;
          float va[5], vb[5];
          {
            const int c = EA & 0xffffff, mk = EA >> 24;
            va[0] = x[(mk & 1) ? c - 1 : c];
            va[1] = x[(mk & 2) ? c + 1 : c];
            va[2] = x[(mk & 4) ? c - nx : c];
            va[3] = x[(mk & 8) ? c + nx : c];
            va[4] = F[n.b + c];
          }
          {  // an idle entry (-1) reads cell 0
            const int c = EB < 0 ? 0 : EB & 0xffffff, mk = EB < 0 ? 0 : EB >> 24;
            vb[0] = x[(mk & 1) ? c - 1 : c];
            vb[1] = x[(mk & 2) ? c + 1 : c];
            vb[2] = x[(mk & 4) ? c - nx : c];
            vb[3] = x[(mk & 8) ? c + nx : c];
            vb[4] = F[n.b + c];
          }
          {
            const int mk = EA >> 24;
            float t = 0.0f;
            t += (mk & 1) ? va[0] : 0.0f;
            t += (mk & 2) ? va[1] : 0.0f;
            t += (mk & 4) ? va[2] : 0.0f;
            t += (mk & 8) ? va[3] : 0.0f;
            x[EA & 0xffffff] = (t + va[4]) * inversoVizinhos(__popc(mk));
          }
          if (EB >= 0) {
            const int mk = EB >> 24;
            float t = 0.0f;
            t += (mk & 1) ? vb[0] : 0.0f;
            t += (mk & 2) ? vb[1] : 0.0f;
            t += (mk & 4) ? vb[2] : 0.0f;
            t += (mk & 8) ? vb[3] : 0.0f;
            x[EB & 0xffffff] = (t + vb[4]) * inversoVizinhos(__popc(mk));
          }
        }
        sincEquipe(eq);
      }
    }
  }
  sincEquipe(eq);
  marcaSecao(a, marcar);
  for (int l = a.L - 2; l >= a.Lc; l--) {
    const NivelS g = s[l + 1];
    const NivelS f = s[l];
    // prolongar: coarse x is 0 on every dry coarse cell, out-of-range corners get weight 0
    for (int c = eq.ti; c < f.nx * f.ny; c += eq.nt) {
      const int i = c % f.nx, j = c / f.nx;
      const int I0 = grossoBaseF(i), J0 = grossoBaseF(j);
      const float wx0 = pesoBaseF(i), wy0 = pesoBaseF(j);
      float gv[4];
#pragma unroll
      for (int b = 0; b < 2; b++) {
        const int J = min(max(J0 + b, 0), g.ny - 1);
#pragma unroll
        for (int aa = 0; aa < 2; aa++) gv[b * 2 + aa] = F[g.xa + min(max(I0 + aa, 0), g.nx - 1) + J * g.nx];
      }
      const float xf = F[f.xa + c];
      float e = 0.0f;
#pragma unroll
      for (int b = 0; b < 2; b++) {
        const int J = J0 + b;
        const float wy = b ? 1.0f - wy0 : wy0;
#pragma unroll
        for (int aa = 0; aa < 2; aa++) {
          const int I = I0 + aa;
          const bool dentro = I >= 0 && J >= 0 && I < g.nx && J < g.ny;
          e += dentro ? gv[b * 2 + aa] * ((aa ? 1.0f - wx0 : wx0) * wy) : 0.0f;
        }
      }
      if (U[f.v + c] & 16) F[f.xa + c] = xf + e;
    }
    sincEquipe(eq);
    marcaSecao(a, marcar);
    passoS(F, U, f, 8, 1, f.xa, f.xb, a.bloco != 0, a.varreduras, eq, todos(f, 8));
    if (a.umaPassada) {
      trocarS(l);
    } else {
      marcaSecao(a, marcar);
      passoS(F, U, f, 0, 1, f.xb, f.xa, a.bloco != 0, a.varreduras, eq, todos(f, 0));
    }
    marcaSecao(a, marcar);
  }
  const NivelS t = s[a.Lc];
  const int Nc = t.nx * t.ny;
  if (coluna < 0) {
    for (int c = eq.ti; c < Nc; c += eq.nt) a.xc[c] = F[t.xa + c];
  } else {  // column `coluna` of the section's matrix, rows = water cells of level Lc
    const int nW = __ldcg(a.nWp);
    for (int c = eq.ti; c < Nc; c += eq.nt) {
      const int r = __ldcg(a.wInv + c);
      if (r >= 0) a.mSecao[(size_t)r * nW + coluna] = F[t.xa + c];
    }
  }
  sincEquipe(eq);  // the next column rewrites the table and the arrays
}

// x of level Lc = M b over its water cells, every CTA staging b in shared memory and each warp
// producing rows (lanes over the row, fixed-order warp sum).  Entries off water stay 0.
__device__ void aplicarSecaoDensa(const Args& a, unsigned char* dyn) {
  const int nW = __ldcg(a.nWp);
  float* bs = (float*)dyn;
  for (int j = threadIdx.x; j < nW; j += TF) bs[j] = __ldcg(a.bc + __ldcg(a.wSecao + j));
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int i = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; i < nW; i += WARPS * gridDim.x) {
    const float* Mi = a.mSecao + (size_t)i * nW;
    float sm = 0.0f;
#pragma unroll 8
    for (int j = lane; j < nW; j += 32) sm += __ldcg(Mi + j) * bs[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sm += __shfl_xor_sync(0xffffffffu, sm, o);
    if (lane == 0) a.xc[__ldcg(a.wSecao + i)] = sm;
  }
}

// ---------------------------------------------------------------- the V-cycle
// After a single smoother pass (x -> tmp) the pass's output becomes the level's x: every CTA
// swaps the two snapshots in its own copy of the level table, at the same point of the solve.
// The barrier that follows (it opens with __syncthreads) publishes the swap to the CTA.
__device__ __forceinline__ void trocarXTmp(int l) {
  __syncthreads();
  if (threadIdx.x == 0) {
    void* t = s_niv[l].x;
    s_niv[l].x = s_niv[l].tmp;
    s_niv[l].tmp = t;
  }
}

// cicloV (js/pressao-cpu.js:241-255) between the spread of the residual (first pass) and the
// gather of z (last pass): 5 Lc + 1 phases, each ending at a grid barrier.  With
// TQ_PRECOND_BLOCK_1 the grid levels above 0 take one smoother pass a leg (shift 8, red-black
// down and black-red up, so the cycle stays symmetric): 3 Lc + 3 phases.
// A loop over the phases with one place for each kind of phase and one barrier, everything inlined:
// across a call, the caller's values go through local memory, which each barrier's acquire drops from
// L1, and a function reads the kernel's arguments through memory too.  With the loads taken as stored
// (suavizarBloco, faseRestringir): 112 -> 95 us an iteration on 840x536 cells (BLOCK_1, FP16), 130 -> 115
// (REFERENCE, FP32), 93 -> 83 on 480x270.
template <class T>
__device__ __forceinline__ bool cicloV(const Args& a, unsigned& ep, float* areas, unsigned char* smem, NivelS* tabS,
                                       const Reuniao& ru, double* sh, bool secaoDensa) {
  // a level's phases: 0 and 1 its passes on the way down, 2 its restriction, 4 and 5 its passes on the way
  // up; 3 the section
  int l = 0, f = 0;
#pragma unroll 1
  for (;;) {
    const bool uma = a.umaPassada && l >= 1;
    if (f == 2) {
      faseRestringir<T>(a, l);
    } else if (f == 3) {
      if (secaoDensa) aplicarSecaoDensa(a, smem);
      else if (blockIdx.x == 0) secaoGrossa(a, smem, smem, tabS, -1, Equipe{(int)threadIdx.x, TF, 0}, true);
    } else if (f == 4) {
      faseSuavizarT<T, M_PROL>(a, l, 8, true, false, 1, areas, ru, sh);
    } else if (f == 0 && l == 0) {
      faseSuavizarT<T, M_ESPALHAR>(a, 0, 0, true, false, 0, areas, ru, sh);
    } else if (f == 5 && l == 0) {
      faseSuavizarT<T, M_JUNTAR>(a, 0, 0, false, false, 1, areas, ru, sh);
    } else {
      faseSuavizarT<T, M_NORMAL>(a, l, f == 1 || uma ? 8 : 0, f == 0, f == 0, f == 5, areas, ru, sh);
    }
    if (uma && (f == 0 || f == 4)) trocarXTmp(l);
    if (!barreira(a, ep)) return false;
    if (f == 5 && l == 0) return true;
    if (f == 2) {
      l++;
      f = l < a.Lc ? 0 : 3;
    } else if (f == 3 || f == 5 || (f == 4 && uma)) {
      l--;
      f = 4;
    } else {
      f = f == 0 && uma ? 2 : f + 1;
    }
  }
}

// ---------------------------------------------------------------- PCG pieces
// A*v at water cell c (js/pressao-cpu.js:84-93 after difundir): neighbours that are water give
// val(n), active-bubble air gives valB(label), anything else 0.
template <class FV, class FB>
__device__ __forceinline__ float aplicarF(const Args& a, int c, FV val, FB valB) {
  const Dev& d = a.d;
  const int vz = ldcg8(a.vizOp + c);
  float s = 0.0f;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (!(vz & (1 << k))) continue;
    const int n = k == 0 ? c - 1 : k == 1 ? c + 1 : k == 2 ? c - d.nx : c + d.nx;
    const int t = ldcg8(d.tipo + n);
    if (t == AGUA) s += val(n);
    else if (a.bolhas && t == AR) {
      uint32_t r = __ldcg(d.rotulo + n);
      if (bolhaAtiva(a, r)) s += valB(r);
    }
  }
  return (float)__popc(vz & 15) * val(c) - s;
}

// A hint to bring the line into L1.
__device__ __forceinline__ void paraL1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

constexpr int KDA = 4;  // cells a thread and batch of [DA], [B] and the true residual

// [DA] of a PCG iteration over this CTA's cells: beta, p = z + beta p (z alone on the first
// iteration), A p (js/pressao-cpu.js:84-93, bubble neighbours through their p), the partial of
// p.Ap (channel 2) and, for air of active bubbles, the sums over their water faces.  Bound by the
// latency of its loads: cells go in batches of KDA a thread, a stride of the grid apart, with every load
// ahead; the left and right neighbours come by shuffle (a warp's cells are consecutive).  The first
// batch's lines are on their way to L1 while the global sums behind beta are made (a hint, as values
// held in registers across the sums cost spills); the bubbles' z and previous p wait in shared memory
// (areas), put there by the warps that do not sum.
// z and p come through L1: they were last written before the grid barrier that opens this phase,
// whose acquire orders these loads after those writes.
// Measured, [DA] / [B] a phase with its barrier (FP16), against four consecutive cells a thread whose products the CTA
// passed on through shared memory: 840x536 cells 10.8 / 8.0 -> 8.4 / 6.0 us, 38,370x316 222 / 169 -> 100 / 84 (an
// iteration 1,005 -> 784).  Direct loads of the left and right neighbours took 7 us more on the last and 0.3 on
// 840x536; the lines of the next batch ahead as well 3 and 0.5.
__device__ __forceinline__ void faseDA(const Args& a, const float* zc, const float* pv, float* pn, bool prim, int nAt,
                                       const double* pbVelho, double* pbNovo, const double* zbOld, double* zbCur,
                                       double& rz, double* sh, float* areas) {
  const Dev& d = a.d;
  const int N = d.N, nx = d.nx, lane = threadIdx.x & 31, GT = gridDim.x * TF;
  double* zbS = (double*)areas;
  double* pbS = zbS + MAX_BOLHAS;
  auto bolha = [&](int b) {
    zbS[b] = zbDe(a, b);
    if (!prim) pbS[b] = __ldcg(&pbVelho[b]);
  };
  double beta = 0.0, s = 0.0;
  auto pbNovoV = [&](int b) { return prim ? zbS[b] : zbS[b] + beta * pbS[b]; };
  auto somar = [&] {
    if (prim) {
      if (nAt > 0) {
#pragma unroll 1
        for (int k = threadIdx.x; k < nAt; k += TF) bolha(__ldcg(&a.ativos[k]));
        __syncthreads();
      }
      return;
    }
    double somas[4];
    somasGlobais<true, 0>(a, nAt, [&](int b, double& t0, double& t1) {
      bolha(b);
      const double r = __ldcg(&d.rb[b]);
      t0 = r * zbS[b];
      t1 = r * __ldcg(&zbOld[b]);
    }, sh, somas, areas);
    const double rzNovo = somas[0] + somas[2], cruz = somas[1] + somas[3];
    beta = fabs(rz) < 1e-30 ? 0.0 : fmax(0.0, (rzNovo - cruz) / rz);
    rz = rzNovo;
  };
  int m[KDA];
  float z[KDA][3], w[KDA][3], zl[KDA], wl[KDA];
  // a batch's cells, those below and above (an index across a row's end reads a value that no flag selects),
  // and one beside the cell: lane 31's to the right, the others' to the left (of which lane 0's counts; a
  // branch would wait for its load).  The first iteration loads the previous p as well and leaves it out: behind
  // a branch those loads waited for the ones before it (120 against 100 us on 38,370x316 cells)
  auto ler = [&](int c0) {
#pragma unroll
    for (int k = 0; k < KDA; k++) m[k] = c0 + k * GT < N ? __ldca(a.op + c0 + k * GT) : 0;
#pragma unroll
    for (int k = 0; k < KDA; k++) {
      const int c = c0 + k * GT < N ? c0 + k * GT : 0;
      z[k][0] = __ldca(zc + c);
      z[k][1] = __ldca(zc + (c >= nx ? c - nx : c));
      z[k][2] = __ldca(zc + (c < N - nx ? c + nx : c));
      zl[k] = __ldca(zc + (lane == 31 ? min(c + 1, N - 1) : max(c - 1, 0)));
    }
#pragma unroll
    for (int k = 0; k < KDA; k++) {
      const int c = c0 + k * GT < N ? c0 + k * GT : 0;
      w[k][0] = __ldca(pv + c);
      w[k][1] = __ldca(pv + (c >= nx ? c - nx : c));
      w[k][2] = __ldca(pv + (c < N - nx ? c + nx : c));
      wl[k] = __ldca(pv + (lane == 31 ? min(c + 1, N - 1) : max(c - 1, 0)));
    }
  };
  float betaf = 0.0f;
  auto fazer = [&](int c0) {
    unsigned long long rl[KDA];
#pragma unroll
    for (int k = 0; k < KDA; k++)
      rl[k] = (m[k] & OP_VIZ_BOLHA) || ((m[k] & OP_FACE) && (m[k] & 15)) ? __ldcg(a.rotB + c0 + k * GT) : 0ull;
    int labA = 0;
    long long acc = 0;
#pragma unroll
    for (int k = 0; k < KDA; k++) {
      const int mk = m[k], c = c0 + k * GT;
      const float p = prim ? z[k][0] : z[k][0] + betaf * w[k][0];
      const float pl = prim ? zl[k] : zl[k] + betaf * wl[k];
      const float pe = __shfl_up_sync(0xffffffffu, p, 1), pd = __shfl_down_sync(0xffffffffu, p, 1);
      float pq[4] = {lane == 0 ? pl : pe, lane == 31 ? pl : pd, prim ? z[k][1] : z[k][1] + betaf * w[k][1],
                     prim ? z[k][2] : z[k][2] + betaf * w[k][2]};
#pragma unroll
      for (int q = 0; q < 4; q++) pq[q] = (mk >> q) & 1 ? pq[q] : 0.0f;
      if (mk & OP_AGUA) {
        if (mk & OP_VIZ_BOLHA)  // a neighbour that is air of an active bubble contributes that bubble's p
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const int b = (int)(rl[k] >> (12 + 12 * q)) & 0xfff;
            if (b && !((mk >> q) & 1)) pq[q] = (float)pbNovoV(b);
          }
        const float ap = (float)(mk >> 8) * p - (((pq[0] + pq[1]) + pq[2]) + pq[3]);
        pn[c] = p;
        d.ap[c] = ap;
        s += (double)p * ap;
      } else if ((mk & OP_FACE) && (mk & 15)) {
        // (p and Ap off water are never read) the bubble's row: the sum of p over its water faces
        const double f = (((double)pq[0] + (double)pq[1]) + (double)pq[2]) + (double)pq[3];
        const int lab = (int)(rl[k] & 0xfff);
        if (lab != labA) {
          if (acc) atomicAdd((unsigned long long*)&d.accB[labA], (unsigned long long)acc);
          labA = lab;
          acc = 0;
        }
        acc += __double2ll_rn(f * ESC);
      }
    }
    if (__any_sync(0xffffffffu, labA)) somarBolhaWarp((long long*)d.accB, labA, acc);
  };
#pragma unroll
  for (int k = 0; k < KDA; k++) {
    const int c = blockIdx.x * TF + threadIdx.x + k * GT;
    if (c < N) {
      paraL1(a.op + c);
      paraL1(zc + c), paraL1(zc + max(c - nx, 0)), paraL1(zc + min(c + nx, N - 1));
      if (!prim) paraL1(pv + c), paraL1(pv + max(c - nx, 0)), paraL1(pv + min(c + nx, N - 1));
    }
  }
  somar();
  betaf = (float)beta;
  if (blockIdx.x == 0)
#pragma unroll 1
    for (int k = threadIdx.x; k < nAt; k += TF) {
      const int b = __ldcg(&a.ativos[k]);
      zbCur[b] = zbS[b];
      pbNovo[b] = pbNovoV(b);
    }
#pragma unroll 1
  for (int base = blockIdx.x * TF; base < N; base += KDA * GT) {
    const int c0 = base + threadIdx.x;
    ler(c0);
    fazer(c0);
  }
  const double tb = somaBloco(s, sh);
  if (threadIdx.x == 0) a.parc[blockIdx.x * NPARC + 2] = tb;
}

// Per-tank sums of v^2 over the water cells of each tank of an atlas (tq_set_tanks) into destino:
// a warp-uniform loop over 32-cell segments; a segment inside one tank is reduced by shuffles and
// added with one FP64 atomic, a segment across tanks adds lane by lane.  Summation order varies
// with the schedule (FP64 rounding, far below the tolerance); every CTA later reads the same sums.
__device__ __noinline__ void somarPorTanque(const Args& a, const float* v, double* destino) {
  const Dev& d = a.d;
  const int N = d.N, GT = gridDim.x * TF, lane = threadIdx.x & 31;
  for (int c0 = blockIdx.x * TF + (threadIdx.x & ~31); c0 < N; c0 += GT) {
    const int c = c0 + lane;
    int t = -1;
    double x = 0.0;
    if (c < N && d.tipo[c] == AGUA) {
      t = tanqueDe(d, c);
      if (t >= 0) {
        x = (double)__ldcg(v + c);
        x *= x;
      }
    }
    const int t0 = __shfl_sync(0xffffffffu, t, 0);
    if (__all_sync(0xffffffffu, t == t0)) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0 && t0 >= 0 && x != 0.0) atomicAdd(destino + t0, x);
    } else if (t >= 0 && x != 0.0) {
      atomicAdd(destino + t, x);
    }
  }
}

// Every tank's true residual within the tolerance of its own initial one: ||r_t||^2 = the water
// sums (d.rvT) plus the squared true rows of the tank's bubbles, against tol^2 ||r0_t||^2.  Thread
// t takes tanks t, t + TF, ..., adding its bubbles in the active list's order, so every CTA
// reaches the same answer from the same global values (the barrier before made them visible).
// Nothing is written here: every CTA reads d.rvT in this phase.  With `gravar` (CTA 0 alone,
// after the solve's last barrier) the totals go to d.rvT for tq_get_tank_residuals.
template <class FB>
__device__ bool tanquesConvergiram(const Args& a, int nAt, FB rbVerd, bool gravar = false) {
  const Dev& d = a.d;
  bool ok = true;
  for (int t = threadIdx.x; t < d.nTanques; t += TF) {
    double s = __ldcg(d.rvT + t);
    for (int k = 0; k < nAt; k++) {
      const int b = __ldcg(&a.ativos[k]);
      if (__ldcg(d.tanqueBolha + b) != t) continue;
      const double v = rbVerd(b);
      s += v * v;
    }
    const double r0 = __ldcg(d.r0T + t);
    ok = ok && s <= a.tol * a.tol * r0;
    if (gravar) d.rvT[t] = s;
  }
  return __syncthreads_and(ok) != 0;
}

// The true residual of a tolerance-mode solve, in FP64 from the FP64 iterate q64 and the bubble
// pressures yB: on water cells r = -div - A q (js/pressao-cpu.js:331-338, bubble neighbours
// through their y), written to d.r in FP32 (the replacement, when it comes to that) and summed
// squared into channel 0; on the interior air of active bubbles, the sum of q over the bubble's
// water faces into its fixed-point sum accV (the bubble row, :339-341, is finished after the
// next barrier).
__device__ __noinline__ void faseVerdade(const Args& a, double* sh) {
  const Dev& d = a.d;
  const int N = d.N, nx = d.nx;
  const int gt0 = blockIdx.x * TF + threadIdx.x, GT = gridDim.x * TF;
  double s = 0;
  // batches of KDA cells a thread, as in [DA]: descriptors, then the five q of each cell (through
  // L1, written before this phase's barrier) and its divergence, then the bubble labels where
  // the descriptor needs them
  for (int c0 = gt0; c0 < N; c0 += KDA * GT) {
    int m[KDA];
#pragma unroll
    for (int k = 0; k < KDA; k++) m[k] = c0 + k * GT < N ? __ldcg(a.op + c0 + k * GT) : 0;
    double qv[KDA][5];
    float dv[KDA];
#pragma unroll
    for (int k = 0; k < KDA; k++) {
      const int c = c0 + k * GT < N ? c0 + k * GT : 0;
      const int nb[5] = {c, c > 0 ? c - 1 : c, c < N - 1 ? c + 1 : c, c >= nx ? c - nx : c, c < N - nx ? c + nx : c};
#pragma unroll
      for (int q = 0; q < 5; q++) qv[k][q] = __ldca(a.q64 + nb[q]);
      dv[k] = __ldcg(d.div + c);
    }
    unsigned long long rl[KDA];
#pragma unroll
    for (int k = 0; k < KDA; k++)
      rl[k] = (a.bolhas && (m[k] & (OP_VIZ_BOLHA | OP_FACE))) ? __ldcg(a.rotB + c0 + k * GT) : 0ull;
#pragma unroll
    for (int k = 0; k < KDA; k++) {
      const int mk = m[k], c = c0 + k * GT;
      if (!(mk & (OP_AGUA | OP_FACE))) continue;
      if (mk & OP_AGUA) {
        double sv = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          if (mk & (1 << q)) sv += qv[k][q + 1];
          else if (mk & OP_VIZ_BOLHA) {
            const int r = (int)(rl[k] >> (12 + 12 * q)) & 0xfff;
            if (r) sv += __ldcg(d.yB + r);
          }
        }
        const double rt = -(double)dv[k] - ((double)(mk >> 8) * qv[k][0] - sv);
        d.r[c] = (float)rt;
        s += rt * rt;
      } else {
        double t = 0;
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (mk & (1 << q)) t += qv[k][q + 1];
        if (t != 0) somaFixa(&a.accV[(int)(rl[k] & 0xfff)], t, ESC);
      }
    }
  }
  const double tb = somaBloco(s, sh);
  if (threadIdx.x == 0) {
    a.parc[blockIdx.x * NPARC + 0] = tb;
    a.parc[blockIdx.x * NPARC + 1] = 0.0;
  }
  if (d.nTanques) somarPorTanque(a, d.r, d.rvT);  // d.r holds the true residual now (FP32)
}

// The wall-block flags of the levels that have them (Args::sol), both shifts: one warp per
// block, 8 cells a lane; a block is wall when every cell of it in the grid is.
__device__ __noinline__ void marcarParedes(const Args& a) {
  const int lane = threadIdx.x & 31, wg = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, nw = WARPS * gridDim.x;
  for (int l = 0; l < a.Lc; l++) {
    const NivelF n = s_niv[l];
    if (!a.sol[l]) continue;
    for (int desl = 0; desl <= 8; desl += 8) {
      const int nbx = (n.nx + desl + 15) >> 4, nb = blocosNivel(n.nx, n.ny, desl);
      uint8_t* fl = a.sol[l] + (desl ? blocosNivel(n.nx, n.ny, 0) : 0);
      for (int blk = wg; blk < nb; blk += nw) {
        const int ox = (blk % nbx) * 16 - desl, oy = (blk / nbx) * 16 - desl;
        const int gy = oy + (lane >> 1), gx0 = ox + (lane & 1) * 8;
        bool parede = true;
        for (int k = 0; k < 8; k++) {
          const int gx = gx0 + k;
          if (gx >= 0 && gy >= 0 && gx < n.nx && gy < n.ny) parede &= ldcg8(n.tipo + gx + gy * n.nx) == SOLIDO;
        }
        const bool todos = __all_sync(0xffffffffu, parede);
        if (lane == 0) fl[blk] = todos ? 1 : 0;
      }
    }
  }
}

// ---------------------------------------------------------------- the kernel
template <class T>
__global__ void __launch_bounds__(TF, 1) k_mgpcg(const __grid_constant__ Args a) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ double sh[32];
  __shared__ NivelS tabS[SECAO_EQUIPES][SECAO_NIVEIS];
  float* areas = (float*)dyn;
  const Dev& d = a.d;
  const int N = d.N, nx = d.nx, ny = d.ny;
  const int gt0 = blockIdx.x * TF + threadIdx.x;
  const int GT = gridDim.x * TF;
  unsigned ep = 0;
  double somas[4];
  if (threadIdx.x < a.L) s_niv[threadIdx.x] = a.niv[threadIdx.x];
  __syncthreads();

  // ---- setup: level-0 preconditioner types, operator masks, bubble faces
  {
    uint8_t* t0 = s_niv[0].tipo;
    for (int c = gt0; c < N; c += GT) {
      const int t = d.tipo[c];
      const uint32_t rot = d.rotulo[c];
      // REFERENCE: enclosed air of a bubble is water to the V-cycle (js/pressao-cpu.js:305-308);
      // BLOCK: it stays air (free surface), the bubble rows take a Jacobi step instead
      t0[c] = (a.bolhas && !a.bloco && t == AR && rot >= 2) ? AGUA : (uint8_t)t;
      const int i = c % nx, j = c / nx;
      int m = 0;
      if (i > 0 && d.tipo[c - 1] != SOLIDO) m |= 1;
      if (i < nx - 1 && d.tipo[c + 1] != SOLIDO) m |= 2;
      if (j > 0 && d.tipo[c - nx] != SOLIDO) m |= 4;
      if (j < ny - 1 && d.tipo[c + nx] != SOLIDO) m |= 8;
      if (t == AGUA) m |= 16;
      a.vizOp[c] = (uint8_t)m;
      if (a.bolhas && t == AR && rot >= 2 && rot < (uint32_t)MAX_BOLHAS && i >= 1 && j >= 1 && i < nx - 1 &&
          j < ny - 1) {
        unsigned k = (d.tipo[c - 1] == AGUA) + (d.tipo[c + 1] == AGUA) + (d.tipo[c - nx] == AGUA) +
                     (d.tipo[c + nx] == AGUA);
        if (k) atomicAdd(&d.facesB[rot], k);
      }
    }
  }
  if (!barreira(a, ep)) return;
  // ---- coarse types (tiposGrossos, js/pressao-cpu.js:63-81), one level per phase
  for (int l = 1; l < a.L; l++) {
    const NivelF f = s_niv[l - 1];
    const NivelF g = s_niv[l];
    for (int C = gt0; C < g.nx * g.ny; C += GT) {
      const int I = C % g.nx, J = C / g.nx;
      bool ar = false, agua = false;
      for (int b = 0; b < 2; b++)
        for (int aa = 0; aa < 2; aa++) {
          int i = 2 * I + aa, j = 2 * J + b;
          if (i >= f.nx || j >= f.ny) continue;
          int t = ldcg8(f.tipo + i + j * f.nx);
          if (t == AR) ar = true;
          else if (t == AGUA) agua = true;
        }
      g.tipo[C] = ar ? AR : agua ? AGUA : SOLIDO;
    }
    if (!barreira(a, ep)) return;
  }
  // ---- neighbour masks of every level, bubble cell counts, active list, initial y
  for (int l = 0; l < a.L; l++) {
    const NivelF n = s_niv[l];
    for (int c = gt0; c < n.nx * n.ny; c += GT) {
      const int i = c % n.nx, j = c / n.nx;
      const uint8_t* tp = n.tipo;
      int m = 0;
      if (l >= 1 && a.bloco) {
        m = vizinhosPorFaces(s_niv[l - 1], n, i, j);
      } else {
        if (i > 0 && ldcg8(tp + c - 1) != SOLIDO) m |= 1;
        if (i < n.nx - 1 && ldcg8(tp + c + 1) != SOLIDO) m |= 2;
        if (j > 0 && ldcg8(tp + c - n.nx) != SOLIDO) m |= 4;
        if (j < n.ny - 1 && ldcg8(tp + c + n.nx) != SOLIDO) m |= 8;
      }
      if (ldcg8(tp + c) == AGUA) m |= 16;
      if (l == 0) {  // the descriptor's water and bubble-air bits (OP_AGUA, OP_BOLHA) for the
                     // spread and the gather; every other reader masks bits 0-4.  With BLOCK
                     // the V-cycle does not see bubbles: no cell spreads or gathers for one.
        const int t = d.tipo[c];
        if (t == AGUA) m |= V0_AGUA;
        else if (a.bolhas && !a.bloco && t == AR && bolhaAtiva(a, d.rotulo[c])) m |= V0_BOLHA;
      }
      n.viz[c] = (uint8_t)m;
    }
  }
  marcarParedes(a);
  for (int c = gt0; c < N; c += GT) {  // the operator descriptor (bubble faces are complete)
    const int i = c % nx, j = c / nx;
    const int t = d.tipo[c];
    int m = 0, livres = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const bool existe = k == 0 ? i > 0 : k == 1 ? i < nx - 1 : k == 2 ? j > 0 : j < ny - 1;
      if (!existe) continue;
      const int nb = k == 0 ? c - 1 : k == 1 ? c + 1 : k == 2 ? c - nx : c + nx;
      const int tn = d.tipo[nb];
      if (tn != SOLIDO) livres++;
      if (tn == AGUA) m |= 1 << k;
      else if (a.bolhas && tn == AR && bolhaAtiva(a, d.rotulo[nb])) m |= OP_VIZ_BOLHA;
    }
    if (t == AGUA) m |= OP_AGUA;
    if (a.bolhas && t == AR && bolhaAtiva(a, d.rotulo[c])) {
      m |= OP_BOLHA;
      if (i >= 1 && j >= 1 && i < nx - 1 && j < ny - 1) m |= OP_FACE;
    }
    a.op[c] = (uint16_t)(m | (livres << 8));
    if (d.nTanques && (m & OP_FACE)) d.tanqueBolha[d.rotulo[c] & 0xfffu] = tanqueDe(d, c);  // same for all its cells
    unsigned long long rl = 0;
    if (a.bolhas && (m & (OP_BOLHA | OP_VIZ_BOLHA))) {
      if (m & OP_BOLHA) rl = d.rotulo[c] & 0xfffu;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const bool existe = k == 0 ? i > 0 : k == 1 ? i < nx - 1 : k == 2 ? j > 0 : j < ny - 1;
        if (!existe) continue;
        const int nb = k == 0 ? c - 1 : k == 1 ? c + 1 : k == 2 ? c - nx : c + nx;
        if (d.tipo[nb] == AR && bolhaAtiva(a, d.rotulo[nb]))
          rl |= (unsigned long long)(d.rotulo[nb] & 0xfffu) << (12 + 12 * k);
      }
    }
    a.rotB[c] = rl;
    a.rotP[c] = a.bloco ? 0 : (uint16_t)(rl & 0xfffu);
  }
  if (a.bolhas) {
    for (int c = gt0; c < N; c += GT) {
      uint32_t b = d.rotulo[c];
      if (b >= 2 && b < (uint32_t)MAX_BOLHAS && d.tipo[c] == AR && __ldcg(&d.facesB[b]) > 0)
        atomicAdd(&d.celsB[b], 1u);
    }
    if (blockIdx.x == 0) {
      if (threadIdx.x < 32) {  // active labels in ascending order (one warp, ballot-compacted)
        int base = 0;
        for (int b0 = 0; b0 < MAX_BOLHAS; b0 += 32) {
          int b = b0 + threadIdx.x;
          bool at = b >= 2 && __ldcg(&d.facesB[b]) > 0;
          unsigned m = __ballot_sync(0xffffffffu, at);
          if (at) a.ativos[base + __popc(m & ((1u << threadIdx.x) - 1u))] = b;
          base += __popc(m);
        }
        if (threadIdx.x == 0) *a.nAtivos = base;
      }
      for (int b = threadIdx.x; b < MAX_BOLHAS; b += TF) {
        bool at = b >= 2 && __ldcg(&d.facesB[b]) > 0;
        d.yB[b] = at ? (double)d.yBolhaF[b] : 0.0;
        d.rb[b] = 0.0;
        d.zb[b] = a.zb2[b] = 0.0;
        d.pb[b] = a.pb2[b] = 0.0;
      }
    }
  } else if (blockIdx.x == 0 && threadIdx.x == 0) {
    *a.nAtivos = 0;
  }
  if (!barreira(a, ep)) return;
  const int nAt = a.bolhas ? __ldcg(a.nAtivos) : 0;

  // ---- r = -div - A q (js/pressao-cpu.js:331-338), bubble aq sums
  {
    double s = 0;
    for (int c = gt0; c < N; c += GT) {
      if (d.tipo[c] != AGUA) {
        d.q[c] = 0.0f;
        d.r[c] = 0.0f;
        continue;
      }
      float ar = aplicarF(a, c, [&](int n) { return __ldcg(d.q + n); },
                          [&](uint32_t r) { return (float)__ldcg(d.yB + r); });
      float rv = -d.div[c] - ar;
      d.r[c] = rv;
      if (a.q64) a.q64[c] = (double)d.q[c];
      s += (double)rv * rv;
    }
    if (a.bolhas)
      for (int c = gt0; c < N; c += GT) {
        const int i = c % nx, j = c / nx;
        if (i < 1 || j < 1 || i >= nx - 1 || j >= ny - 1) continue;
        uint32_t b = d.rotulo[c];
        if (d.tipo[c] != AR || !bolhaAtiva(a, b)) continue;
        double t = 0;
        if (d.tipo[c - 1] == AGUA) t += (double)__ldcg(d.q + c - 1);
        if (d.tipo[c + 1] == AGUA) t += (double)__ldcg(d.q + c + 1);
        if (d.tipo[c - nx] == AGUA) t += (double)__ldcg(d.q + c - nx);
        if (d.tipo[c + nx] == AGUA) t += (double)__ldcg(d.q + c + nx);
        if (t != 0) somaFixa(&d.accB[b], t, ESC);
      }
    double tb = somaBloco(s, sh);
    if (threadIdx.x == 0) {
      a.parc[blockIdx.x * NPARC + 0] = tb;
      a.parc[blockIdx.x * NPARC + 1] = 0.0;
    }
  }
  // the coarsest level's matrix (its neighbour masks are complete since the last barrier)
  if (a.offDenso >= 0) montarDenso(a, dyn);
  if (a.secaoDensa && blockIdx.x == (gridDim.x > 1 ? 1 : 0) && threadIdx.x < 32) {
    // the water cells of level Lc, in cell order (one warp, ballot-compacted)
    const NivelF n = s_niv[a.Lc];
    const int Nc = n.nx * n.ny;
    int base = 0;
    for (int c0 = 0; c0 < Nc; c0 += 32) {
      const int c = c0 + threadIdx.x;
      const bool agua = c < Nc && (ldcg8(n.viz + c) & 16);
      const unsigned m = __ballot_sync(0xffffffffu, agua);
      const int pos = base + __popc(m & ((1u << threadIdx.x) - 1u));
      if (c < Nc) a.wInv[c] = agua ? pos : -1;
      if (agua) a.wSecao[pos] = c;
      base += __popc(m);
    }
    if (threadIdx.x == 0) *a.nWp = base;
  }
  if (!barreira(a, ep)) return;
  // each tank's ||r0||^2, water rows (r is complete since the barrier; read at the checks, many
  // barriers later)
  if (d.nTanques && a.q64) somarPorTanque(a, d.r, d.r0T);
  // rb = rhs - (faces*y - sum) (js/pressao-cpu.js:339-341); norm0
  auto rbInicial = [&](int b) {
    return (double)d.rhsBolhaF[b] - (__ldcg(&d.facesB[b]) * __ldcg(&d.yB[b]) - (double)__ldcg(&d.accB[b]) / ESC);
  };
  somasGlobais<false, 0>(a, nAt, [&](int b, double& t, double&) { const double v = rbInicial(b); t = v * v; }, sh, somas,
                      areas);
  const double norma0 = sqrt(somas[0] + somas[2]);
  if (blockIdx.x == 0) {
    for (int k = threadIdx.x; k < nAt; k += TF) {
      int b = __ldcg(&a.ativos[k]);
      d.rb[b] = rbInicial(b);
      if (d.nTanques && a.q64) {  // the bubble rows of each tank's ||r0||^2
        const int t = __ldcg(d.tanqueBolha + b);
        if (t >= 0) atomicAdd(d.r0T + t, d.rb[b] * d.rb[b]);
      }
    }
    if (threadIdx.x == 0) {
      d.esc->norma0 = d.esc->norma = norma0;
      d.esc->normas[0] = norma0;
      d.esc->iters = 0;
      d.esc->pronto = 0;
    }
  }
  if (!barreira(a, ep)) return;  // rb visible before spreading
  // ---- the section's matrix: every CTA builds its share of the columns with its own copy of
  // the coarsest level's matrix
  const int nW = a.secaoDensa ? __ldcg(a.nWp) : 0;
  const bool secaoDensa = a.secaoDensa && a.iteracoes >= SECAO_DENSA_MIN_ITERS;
  if (a.offDenso >= 0 && (secaoDensa || blockIdx.x == 0)) carregarDenso(a, dyn);
  if (secaoDensa) {
    const int nt = TF / a.equipes, g = threadIdx.x / nt;
    const Equipe eq{(int)threadIdx.x - g * nt, nt, g};
    bool primeira = true;  // a team's masks stay in its area from its first column on
    for (int col = g * gridDim.x + blockIdx.x; col < nW; col += a.equipes * gridDim.x, primeira = false)
      secaoGrossa(a, dyn + (size_t)g * a.bytesSecao, dyn, tabS[g], col, eq, primeira);
    __syncthreads();
    const NivelF nc = s_niv[a.Lc];
    for (int c = gt0; c < nc.nx * nc.ny; c += GT) a.xc[c] = 0.0f;  // off water, x of level Lc stays 0
    if (!barreira(a, ep)) return;
  }
  float escala = (a.escalar && norma0 > 0) ? (float)(1.0 / norma0) : 1.0f;
  if (blockIdx.x == 0)
    for (int b = threadIdx.x; b < MAX_BOLHAS; b += TF) {
      a.accZ[b] = 0;
      d.accB[b] = 0;
    }
  // the spread reads each active bubble's mean residual from the CTA's areas (the V-cycle sees no
  // bubbles with BLOCK)
  auto mediaBolha = [&](int b) { areas[b] = (float)(__ldcg(&d.rb[b]) / __ldcg(&d.celsB[b])); };
  auto mediasBolhas = [&] {
    if (a.bloco) return;
#pragma unroll 1
    for (int k = threadIdx.x; k < nAt; k += TF) mediaBolha(__ldcg(&a.ativos[k]));
  };
  mediasBolhas();
  __syncthreads();
  Reuniao ru{escala, d.z, nullptr};
  int cz = 0, cp = 0;  // which of the two z / p buffers holds the latest values
  auto zbAtual = [&](int b) { return zbDe(a, b); };
  double rz = 0.0;
  bool primeira = true;
  int itersFeitas = 0, trocas = 0;
  bool convergiu = false;
  double normaVerd = -1.0;
  double proxTroca = norma0 * FATOR_TROCA;  // the next residual replacement's threshold
  int proxVerif = 0;                          // with tanks: the next iteration that may check
  auto rbVerd = [&](int b) {  // a bubble's true row, from faseVerdade's sums
    return (double)d.rhsBolhaF[b] - (__ldcg(&d.facesB[b]) * __ldcg(&d.yB[b]) - (double)__ldcg(&a.accV[b]) / ESC);
  };

  for (int it = -1;;) {
    if (!cicloV<T>(a, ep, areas, dyn, tabS[0], ru, sh, secaoDensa)) return;
    if (it < 0) {
      somasGlobais<false, 0>(a, nAt, [&](int b, double& t, double&) { t = __ldcg(&d.rb[b]) * zbAtual(b); }, sh, somas, areas);
      rz = somas[0] + somas[2];
      __syncthreads();
    } else {
      cz ^= 1;
      cp ^= 1;
      primeira = false;
    }
    if (++it >= a.iteracoes) break;
    float* zc = cz ? a.z2 : d.z;
    float* zo = cz ? d.z : a.z2;
    const float* pv = cp ? a.p2 : d.p;
    float* pn = cp ? d.p : a.p2;
    const double* zbOld = cz ? d.zb : a.zb2;
    double* zbCur = cz ? a.zb2 : d.zb;
    const double* pbVelho = cp ? a.pb2 : d.pb;
    double* pbNovo = cp ? d.pb : a.pb2;
    // ---- [DA] beta, p = z + beta p, A p, p.Ap, bubble rows
    faseDA(a, zc, pv, pn, primeira, nAt, pbVelho, pbNovo, zbOld, zbCur, rz, sh, areas);
    if (!barreira(a, ep)) return;
    // ---- [B] alpha; q += alpha p, r -= alpha Ap; bubbles; r.r
    auto apbV = [&](int b) {
      return __ldcg(&d.facesB[b]) * __ldcg(&pbNovo[b]) - (double)__ldcg(&d.accB[b]) / ESC;
    };
    double alfa;
    {
      somasGlobais<false, 2>(a, nAt, [&](int b, double& t, double&) { t = __ldcg(&pbNovo[b]) * apbV(b); }, sh, somas, areas);
      const double pap = somas[0] + somas[2];
      alfa = fabs(pap) < 1e-30 ? 0.0 : rz / pap;
      const float af = (float)alfa;
      double s = 0;
#pragma unroll 1
      for (int c0 = gt0; c0 < N; c0 += KDA * GT) {  // all loads of a batch first
        int m[KDA];
        float qv[KDA], pnv[KDA], rv[KDA], apv[KDA];
        double qd[KDA];
#pragma unroll
        for (int k = 0; k < KDA; k++) {
          const int c = c0 + k * GT < N ? c0 + k * GT : 0;
          m[k] = c0 + k * GT < N ? __ldcg(a.op + c) : 0;
          if (a.q64) qd[k] = __ldcg(a.q64 + c);
          else qv[k] = __ldcg(d.q + c);
          pnv[k] = __ldcg(pn + c);
          rv[k] = __ldcg(d.r + c);
          apv[k] = __ldcg(d.ap + c);
        }
#pragma unroll
        for (int k = 0; k < KDA; k++) {
          if (!(m[k] & OP_AGUA)) continue;
          const int c = c0 + k * GT;
          if (a.q64) a.q64[c] = qd[k] + alfa * (double)pnv[k];
          else d.q[c] = qv[k] + af * pnv[k];
          const float r = rv[k] - af * apv[k];
          d.r[c] = r;
          s += (double)r * r;
        }
      }
      if (blockIdx.x == 0) {
        double sb = 0;
        for (int k = threadIdx.x; k < nAt; k += TF) {
          int b = __ldcg(&a.ativos[k]);
          d.yB[b] += alfa * __ldcg(&pbNovo[b]);
          double rbn = __ldcg(&d.rb[b]) - alfa * apbV(b);
          d.rb[b] = rbn;
          sb += rbn * rbn;
        }
        s += sb;
        for (int b = threadIdx.x; b < MAX_BOLHAS; b += TF) {
          a.accZ[b] = 0;
          if (a.q64) a.accV[b] = 0;
        }
        if (a.q64)
          for (int t = threadIdx.x; t < d.nTanques; t += TF) d.rvT[t] = 0.0;
      }
      double tb = somaBloco(s, sh);
      if (threadIdx.x == 0) a.parc[blockIdx.x * NPARC + 3] = tb;
    }
    if (!barreira(a, ep)) return;
    // ---- [C] norm, convergence, spread the residual
    somasGlobais<false, 3>(a, a.bloco ? 0 : nAt, [&](int b, double&, double&) { mediaBolha(b); }, sh, somas, areas);
    double norma = sqrt(somas[0]);
    itersFeitas = it + 1;
    const bool ultima = it == a.iteracoes - 1;
    bool fim = ultima || (a.tol > 0 && norma <= a.tol * norma0);
    if (fim && !ultima && d.nTanques && it < proxVerif && norma > proxTroca) fim = false;
    if (a.q64 && (fim || norma <= proxTroca)) {
      // tolerance mode: the true residual of the FP64 iterate decides, and replaces the
      // recursive one unless the solve ends here
      proxVerif = it + VERIF_TANQUES;
      faseVerdade(a, sh);
      if (!barreira(a, ep)) return;
      somasGlobais<false, 0>(a, nAt, [&](int b, double& t, double&) { const double v = rbVerd(b); t = v * v; }, sh, somas,
                          areas);
      normaVerd = sqrt(somas[0] + somas[2]);
      // with tanks, each tank's own residual decides; without, the whole grid's
      convergiu = d.nTanques ? tanquesConvergiram(a, nAt, rbVerd) : normaVerd <= a.tol * norma0;
      fim = convergiu || ultima;
      if (!fim) {
        // replacement: r (water) was rewritten by faseVerdade, the bubble rows follow; the
        // iteration goes on with the same search direction
        trocas++;
        proxTroca = normaVerd * FATOR_TROCA;
        norma = normaVerd;
        if (blockIdx.x == 0)
          for (int k = threadIdx.x; k < nAt; k += TF) {
            const int b = __ldcg(&a.ativos[k]);
            d.rb[b] = rbVerd(b);
          }
        if (!barreira(a, ep)) return;  // rb visible before the spread
        mediasBolhas();
        __syncthreads();
      }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      if (it + 1 < 1024) d.esc->normas[it + 1] = norma;
      d.esc->iters = it + 1;
      d.esc->norma = norma;
      d.esc->pronto = fim ? 1 : 0;
    }
    if (fim) break;
    escala = (a.escalar && norma > 0) ? (float)(1.0 / norma) : 1.0f;
    if (blockIdx.x == 0)
      for (int b = threadIdx.x; b < MAX_BOLHAS; b += TF) d.accB[b] = 0;
    ru = Reuniao{escala, zo, zc};
  }
  // ---- end: q = 0 off water (the FP64 iterate rounded on water); bubbles hand back their
  // pressure; the solve's convergence record
  if (!barreira(a, ep)) return;
  for (int c = gt0; c < N; c += GT) {
    if (d.tipo[c] != AGUA) d.q[c] = 0.0f;
    else if (a.q64) d.q[c] = (float)__ldcg(a.q64 + c);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    Escalares* e = d.esc;
    const bool ok = a.q64 && convergiu;
    e->normaVerd = a.q64 ? normaVerd : -1.0;
    e->convergiu = ok ? 1 : 0;
    e->trocas = trocas;
    e->solves++;
    if (a.q64 && !ok) e->capados++;
    e->itersAcum += itersFeitas;
    e->trocasAcum += trocas;
    if (a.q64 && norma0 > 0 && normaVerd / norma0 > e->maxRel) e->maxRel = normaVerd / norma0;
  }
  if (blockIdx.x == 0 && d.nTanques && a.q64) tanquesConvergiram(a, nAt, rbVerd, true);  // each tank's total
  if (blockIdx.x == 0)
    for (int k = threadIdx.x; k < nAt; k += TF) {
      int b = __ldcg(&a.ativos[k]);
      d.yBolhaF[b] = (float)__ldcg(&d.yB[b]);
    }
}

// ---------------------------------------------------------------- host side
template <class T>
static void* kernelDe() { return (void*)k_mgpcg<T>; }

Fundido* criarFundido(Pcg* p, Arena& A) {
  if (p->L < 2) return nullptr;  // no coarse level to hand to the coarse section
  Fundido* f = new Fundido();
  // coarse section: the longest suffix of levels (not level 0) fitting the shared budget
  int Lc = p->L;
  size_t bytes = 0;
  for (int l = p->L - 1; l >= 1; l--) {
    size_t n = (size_t)p->nxL[l] * p->nyL[l];
    size_t b = 3 * ((n * 4 + 15) & ~(size_t)15) + ((n + 15) & ~(size_t)15);
    if (bytes + b > SMEM_GROSSO_MAX || (n > SECAO_MAX_CELULAS && l < p->L - 1)) break;
    bytes += b;
    Lc = l;
  }
  if (Lc >= p->L || p->L - Lc > SECAO_NIVEIS) {  // even the coarsest level does not fit
    delete f;
    return nullptr;
  }
  f->Lc = Lc;
  // 16-bit storage on every grid level below the coarse section (the smallest included), so the
  // kernel's passes exist in one storage type only (faseSuavizarT); the level buffers hold 4 bytes
  // an element whatever they store
  if (p->precisao != TQ_PREC_FP32)
    for (int l = 0; l < Lc; l++) p->meia[l] = true;
  const size_t areas = AREA_BOLHAS + AREA_TERMOS;
  static_assert(areas >= WARPS * 768 * 4 && areas >= WARPS * SUAV_W * 4, "the warps' areas");
  f->smem = bytes > areas ? bytes : areas;
  f->bytesSecao = (int)bytes;
  // teams that build the section's matrix side by side, where their areas and the coarsest
  // level's matrix fit in a CTA's shared memory
  for (int q = SECAO_EQUIPES; q > 1; q--)
    if (TF % (32 * q) == 0 && q * bytes + DENSO_BYTES + 16 <= SMEM_CTA_MAX) {
      f->equipes = q;
      if (q * bytes > f->smem) f->smem = q * bytes;
      break;
    }
  {  // the coarsest level's matrix after everything else, when the level is small enough
    const size_t nGrosso = (size_t)p->nxL[p->L - 1] * p->nyL[p->L - 1];
    const size_t off = (f->smem + 15) & ~(size_t)15;
    if (nGrosso <= (size_t)DENSO_MAPA_MAX && off + DENSO_BYTES <= SMEM_CTA_MAX) {
      f->offDenso = (int)off;
      f->smem = off + DENSO_BYTES;
    }
  }
  const size_t nSecao = (size_t)p->nxL[Lc] * p->nyL[Lc];
  f->secaoDensa = f->offDenso >= 0 && nSecao <= (size_t)SECAO_DENSA_MAX && Lc < p->L - 1;
  f->kern = p->precisao == TQ_PREC_FP16   ? kernelDe<__half>()
            : p->precisao == TQ_PREC_BF16 ? kernelDe<__nv_bfloat16>()
                                          : kernelDe<float>();
  int dev = 0, sms = 0, porSM = 0;
  // The attribute is per kernel and shared by every solver in the process: raise it to the
  // largest size any grid uses (f->smem <= SMEM_CTA_MAX), never lower it to this grid's.
  const size_t smemMax = SMEM_CTA_MAX;
  bool ok = cudaGetDevice(&dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
            cudaFuncSetAttribute(f->kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemMax) == cudaSuccess &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&porSM, f->kern, TF, f->smem) == cudaSuccess && porSM >= 1;
  if (!ok) {
    cudaGetLastError();
    delete f;
    return nullptr;
  }
  // one CTA per SM (co-resident, as the grid barrier needs), or the requested fewer
  f->G = p->ctasFundido > 0 && p->ctasFundido < sms ? p->ctasFundido : sms;
  // Wall blocks are skipped on levels of at least two full rounds of the grid's warps (a
  // tank atlas's finest levels): there the flags' one extra load per warp and pass is paid
  // back; a level of one round (the 450k-cell scene's) keeps no flags.
  // TQ_WALL_SKIP_MIN_BLOCKS in the environment (read when the handle is created) sets the
  // threshold in blocks; the tests use 1 to skip on every grid level and 0x7fffffff for none.
  long long limiar = 2LL * WARPS * f->G;
  if (const char* e = getenv("TQ_WALL_SKIP_MIN_BLOCKS")) limiar = atoll(e);
  if (const char* e = getenv("TQ_BARRIER_WAIT_CYCLES")) {
    const long long v = atoll(e);
    if (v > 0 && v <= LIMITE_CICLOS) f->limite = v;
  }
  if (const char* e = getenv("TQ_BARRIER_HOLD_CTA")) f->segurarCta = atoi(e);
  if (const char* e = getenv("TQ_BARRIER_HOLD_CYCLES")) {
    const long long v = atoll(e);
    f->segurarCiclos = v > 0 && v <= 4 * LIMITE_CICLOS ? v : 0;
  }
  size_t nFlags = 0;
  for (int l = 0; l < Lc; l++) {
    f->comParedes[l] = blocosNivel(p->nxL[l], p->nyL[l], 0) >= limiar;
    if (f->comParedes[l]) nFlags += blocosNivel(p->nxL[l], p->nyL[l], 0) + blocosNivel(p->nxL[l], p->nyL[l], 8);
  }
  const size_t N = p->N, nLc = (size_t)p->nxL[Lc] * p->nyL[Lc];
  A.pedir(&f->niveis, MAX_NIVEIS);
  A.pedir(&f->parc, (size_t)f->G * NPARC);
  A.pedir(&f->bar, 2);
  A.pedir(&f->erro, 1);
  A.pedir(&f->accZ, MAX_BOLHAS);
  A.pedir(&f->zb2, MAX_BOLHAS);
  A.pedir(&f->pb2, MAX_BOLHAS);
  A.pedir(&f->ativos, MAX_BOLHAS);
  A.pedir(&f->nAtivos, 1);
  A.pedir(&f->p2, N);
  A.pedir(&f->z2, N);
  A.pedir(&f->xc, nLc);
  A.pedir(&f->bc, nLc);
  A.pedir(&f->op, N);
  A.pedir(&f->rotP, N);
  A.pedir(&f->rotB, N);
  A.pedir(&f->q64, N);
  A.pedir(&f->accV, MAX_BOLHAS);
  if (nFlags) A.pedir(&f->solidos, nFlags);
  if (f->secaoDensa) {
    A.pedir(&f->mSecao, nLc * nLc);
    A.pedir(&f->wSecao, nLc);
    A.pedir(&f->wInv, nLc);
    A.pedir(&f->nW, 1);
  }
  if (f->offDenso >= 0) A.pedir(&f->densoG, DENSO_BYTES / 4);
  return f;
}

// The level table on the device and the wall flags' places, once the arena is reserved.
bool iniciarFundido(Fundido* f, const Pcg* p, cudaStream_t s) {
  NivelF tab[MAX_NIVEIS] = {};
  for (int l = 0; l < p->L; l++) {
    NivelF& n = tab[l];
    n.nx = p->nxL[l];
    n.ny = p->nyL[l];
    n.meia = (l < f->Lc && p->meia[l]) ? (p->precisao == TQ_PREC_FP16 ? 1 : 2) : 0;
    n.viz = p->vizL[l];
    n.tipo = p->tipoL[l];
    n.b = p->bL[l];
    n.x = p->xL[l];
    n.tmp = p->tmpL[l];
  }
  size_t off = 0;
  for (int l = 0; l < f->Lc; l++) {
    if (!f->comParedes[l]) continue;
    f->sol[l] = f->solidos + off;
    off += blocosNivel(p->nxL[l], p->nyL[l], 0) + blocosNivel(p->nxL[l], p->nyL[l], 8);
  }
  return cudaMemcpyAsync(f->niveis, tab, sizeof tab, cudaMemcpyHostToDevice, s) == cudaSuccess;
}

void destruirFundido(Fundido* f) {
  if (!f) return;
  if (f->perfil) cudaFree(f->perfil);
  delete f;
}

// Queues the solve on `s` and returns without waiting: the iteration count, the residual history
// and the convergence record stay on the device (Escalares), and a bounded wait that gave up
// leaves f->erro set for erroFundido to report.  Nothing here waits for the device, so a frame
// of substeps can be captured in a CUDA graph.
int resolverPressaoFundido(Pcg* p, const Dev& d, int iteracoes, double tol, bool bolhas, int precond,
                           cudaStream_t s) {
  Fundido* f = p->fundido;
  Args a{};
  a.bloco = precond == TQ_PRECOND_BLOCK || precond == TQ_PRECOND_BLOCK_1 ? 1 : 0;
  a.varreduras = a.bloco ? f->varredurasBloco : VARREDURAS;
  a.umaPassada = precond == TQ_PRECOND_BLOCK_1 ? 1 : 0;
  a.limite = f->limite;
  a.segurarCta = f->segurarCta;
  a.segurarCiclos = f->segurarCiclos;
  f->segurarCta = -1;  // the hold is one-shot
  a.q64 = tol > 0 ? f->q64 : nullptr;
  a.accV = f->accV;
  a.d = d;
  a.L = p->L;
  a.Lc = f->Lc;
  a.niv = f->niveis;
  a.vizOp = p->vizOp;
  a.iteracoes = iteracoes;
  a.tol = tol;
  a.bolhas = bolhas ? 1 : 0;
  a.escalar = p->precisao != TQ_PREC_FP32 ? 1 : 0;
  a.parc = f->parc;
  a.bar = f->bar;
  a.erro = f->erro;
  a.accZ = f->accZ;
  a.zb2 = f->zb2;
  a.pb2 = f->pb2;
  a.ativos = f->ativos;
  a.nAtivos = f->nAtivos;
  a.p2 = f->p2;
  a.z2 = f->z2;
  for (int l = 0; l < MAX_NIVEIS; l++) a.sol[l] = f->sol[l];
  a.xc = f->xc;
  a.bc = f->bc;
  a.offDenso = f->offDenso;
  a.secaoDensa = f->secaoDensa ? 1 : 0;
  a.equipes = f->equipes;
  a.bytesSecao = f->bytesSecao;
  a.mSecao = f->mSecao;
  a.wSecao = f->wSecao;
  a.wInv = f->wInv;
  a.nWp = f->nW;
  a.densoG = f->densoG;
  a.op = f->op;
  a.rotB = f->rotB;
  a.rotP = f->rotP;
  a.perfil = f->perfilar ? f->perfil : nullptr;
  if (a.perfil) {
    cudaMemsetAsync(f->perfil, 0, sizeof(unsigned long long), s);
    cudaMemsetAsync(f->perfil + PERFIL_MAX + 1, 0, sizeof(unsigned long long), s);
  }
  zerarBolhas(d, s);
  if (d.nTanques && tol > 0) cudaMemsetAsync(d.r0T, 0, (size_t)d.nTanques * sizeof(double), s);
  cudaMemsetAsync(f->bar, 0, 2 * sizeof(unsigned), s);
  // f->erro is not cleared here: a solve that gave up keeps it set until erroFundido reads it,
  // and every later solve of the frame then stops at its first barrier instead of waiting.
  // The levels that skip wall blocks start the solve with their snapshots and right side at 0,
  // and with level 0 so do both z vectors (a pass never writes anything else off water).
  for (int l = 0; l < f->Lc; l++) {
    if (!f->comParedes[l]) continue;
    const size_t bytes = (size_t)p->nxL[l] * p->nyL[l] * (p->meia[l] ? 2 : 4);
    cudaMemsetAsync(p->xL[l], 0, bytes, s);
    cudaMemsetAsync(p->tmpL[l], 0, bytes, s);
    cudaMemsetAsync(p->bL[l], 0, bytes, s);
  }
  if (f->comParedes[0]) {
    cudaMemsetAsync(d.z, 0, (size_t)d.N * 4, s);
    cudaMemsetAsync(f->z2, 0, (size_t)d.N * 4, s);
  }
  void* args[] = {&a};
  contarLancamento();
  cudaError_t e = cudaLaunchCooperativeKernel(f->kern, dim3(f->G), dim3(TF), args, f->smem, s);
  if (e != cudaSuccess) return TQ_E_CUDA;
  return TQ_OK;
}

// TQ_E_TIMEOUT when a solve since the last call gave up on a bounded wait (the flag is cleared),
// else TQ_OK.  Waits for the stream.
int erroFundido(Fundido* f, cudaStream_t s) {
  if (!f) return TQ_OK;
  int h = 0;
  if (cudaMemcpyAsync(&h, f->erro, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return TQ_E_CUDA;
  if (!h) return TQ_OK;
  if (cudaMemsetAsync(f->erro, 0, sizeof(int), s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess)
    return TQ_E_CUDA;
  return TQ_E_TIMEOUT;
}

}  // namespace tq
