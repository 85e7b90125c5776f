// suavizador.cuh — the multigrid smoother's block sweep in registers, and a whole leg of a V-cycle's
// level on a tile in shared memory, shared by the plain engine (pcg.cu) and the fused engine
// (pcg_fundido.cu).
#pragma once
#include "common.cuh"

namespace tq {

__device__ __forceinline__ int grossoBaseF(int i) { return (i & 1) == 0 ? (i >> 1) - 1 : (i - 1) >> 1; }
__device__ __forceinline__ float pesoBaseF(int i) { return (i & 1) == 0 ? 0.25f : 0.75f; }

// ---------------------------------------------------------------- block sweeps
// 1/k for k free neighbours (k = 1..4), the correctly rounded float constants.
__device__ __forceinline__ float inversoVizinhos(int k) {
  return k == 1 ? 1.0f : k == 2 ? 0.5f : k == 3 ? (1.0f / 3.0f) : 0.25f;
}

// ---------------------------------------------------------------- register-resident block sweep
// Lane l of the warp that owns a 16x16 block holds, for each colour c and m = 0..3, the cell of
// colour c in row 4g + m (g = l >> 3) among the columns 2k, 2k + 1 (k = l & 7): its column is
// (c + 1 + m) & 1, since a cell's colour is (row + column + 1) & 1 (js/pressao-cpu.js:120).  It
// also holds the block's frame next to its cells: left and right of its rows (k = 0, k = 7),
// below and above its columns (g = 0, g = 3).  In a half-sweep of colour COR every neighbour of
// an updated cell has the other colour: the lane's own other cell in the row, the rows m -/+ 1
// of the lane (same column), the row in lane l -/+ 1, the row below row 0 in lane l - 8 (its
// m = 3), the row above row 3 in lane l + 8 (its m = 0), or the frame: 6 shuffles a half-sweep,
// which keeps the shuffle pipe, shared by the SM's warps, half as busy as rows g + 4m would.
// A half-sweep reads no value that it writes.
// Every snapshot holds x = 0 on cells that are not water (the passes store 0 there, the frame
// outside the grid is 0), so a wall neighbour adds +0 and the sum needs no mask; only 1/k and
// whether the cell changes come from the mask.  The exception is TQ_PRECOND_BLOCK's coarse
// levels, whose masks close faces between two water cells across a thin wall: with `masc` the
// neighbours the mask leaves out enter the sum with weight 0 (masc is uniform over the grid; bits
// tested in each half-sweep instead cost 100 cycles of it).
struct Moldura {
  float esq[4], dir[4];  // frame left / right of the lane's rows (k = 0 / k = 7)
  float bai[2], cim[2];  // frame below / above the lane's columns (g = 0 / g = 3), by column
};

template <int COR, bool MASC>
__device__ __forceinline__ void meiaReg(float (&x)[2][4], const float (&bq)[2][4], const float (&iq)[2][4],
                                        const bool (&muda)[2][4], const Moldura& f, const float (&p)[2][4][4]) {
  const int lane = threadIdx.x & 31, g = lane >> 3, k = lane & 7;
  float H[4];
#pragma unroll
  for (int m = 0; m < 4; m++)  // row m's neighbour in lane l + 1 (colour COR in the odd column) or l - 1
    H[m] = __shfl_sync(0xffffffffu, x[1 - COR][m], (((COR + 1 + m) & 1) ? lane + 1 : lane - 1) & 31);
  const float D = __shfl_sync(0xffffffffu, x[1 - COR][3], (lane - 8) & 31);
  const float U = __shfl_sync(0xffffffffu, x[1 - COR][0], (lane + 8) & 31);
#pragma unroll
  for (int m = 0; m < 4; m++) {
    const int jc = (COR + 1 + m) & 1;  // the column of colour COR in row m
    const float y = x[1 - COR][m];
    float esq = jc ? y : (k == 0 ? f.esq[m] : H[m]);
    float dir = jc ? (k == 7 ? f.dir[m] : H[m]) : y;
    float baixo = m >= 1 ? x[1 - COR][m >= 1 ? m - 1 : 0] : (g >= 1 ? D : f.bai[jc]);
    float cima = m <= 2 ? x[1 - COR][m <= 2 ? m + 1 : 3] : (g <= 2 ? U : f.cim[jc]);
    // weights 1 and 0 in fused multiply-adds: the bits of the masked sum
    const float* w = p[COR][m];
    const float sm = MASC ? fmaf(w[3], cima, fmaf(w[2], baixo, fmaf(w[1], dir, w[0] * esq)))
                          : ((esq + dir) + baixo) + cima;
    const float q = x[COR][m];
    const float n = q + fmaf(sm + bq[COR][m], iq[COR][m], -q);
    x[COR][m] = muda[COR][m] ? n : q;
  }
}

// A sweep is the two half-sweeps one after the other in straight line: picking the colour by the
// loop's parity instead cost twice the time (262 against 98 cycles a half-sweep with one warp on
// an SM, 294 against 173 with 12).  The loop over the sweeps stays rolled: the code stays small in
// the instruction cache, which each phase enters cold.
template <bool MASC>
__device__ __forceinline__ void varrerOrdem(float (&x)[2][4], const int (&v)[2][4], const float (&bq)[2][4],
                                            const float (&iq)[2][4], const bool (&muda)[2][4], const Moldura& f,
                                            int ordem, int nVarr) {
  float p[2][4][4];  // MASC: 1 for an open face
  if (MASC)
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
      for (int m = 0; m < 4; m++)
#pragma unroll
        for (int q = 0; q < 4; q++) p[c][m][q] = (v[c][m] >> q) & 1 ? 1.0f : 0.0f;
  if (ordem == 0) {
#pragma unroll 1
    for (int h = 0; h < nVarr; h++) {
      meiaReg<0, MASC>(x, bq, iq, muda, f, p);
      meiaReg<1, MASC>(x, bq, iq, muda, f, p);
    }
  } else {
#pragma unroll 1
    for (int h = 0; h < nVarr; h++) {
      meiaReg<1, MASC>(x, bq, iq, muda, f, p);
      meiaReg<0, MASC>(x, bq, iq, muda, f, p);
    }
  }
}

// The VARREDURAS red-black sweeps (js/pressao-cpu.js:114-137) of the warp's block in registers;
// v = neighbour mask | 16 water | 128 in grid, bq = right side; ordem 0 sweeps colour 0 first.
__device__ __forceinline__ void varrerReg(float (&x)[2][4], const int (&v)[2][4], const float (&bq)[2][4],
                                         const Moldura& f, int ordem, bool masc, int nVarr) {
  float iq[2][4];
  bool muda[2][4];
#pragma unroll
  for (int c = 0; c < 2; c++)
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int mk = v[c][m] & 15;
      iq[c][m] = inversoVizinhos(__popc(mk));
      muda[c][m] = (v[c][m] & 16) && mk;
    }
  if (masc) varrerOrdem<true>(x, v, bq, iq, muda, f, ordem, nVarr);
  else varrerOrdem<false>(x, v, bq, iq, muda, f, ordem, nVarr);
}

// ---------------------------------------------------------------- a leg of a level on a tile
// Down a level, the V-cycle runs two smoother passes from x = 0 (blocks at shift 0, then shift 8)
// and restricts the residual; up, it adds the coarse correction and runs the two passes in
// reverse.  A CTA does a whole leg for a tile of kx x ky blocks: it also sweeps the blocks around
// its tile that the last pass and the restriction read, so the passes need no exchange with other
// CTAs.  That trades sweeps (on the way down (k+2)^2 + (k+1)^2 blocks instead of 2 k^2, up
// (k+1)^2 + k^2) for launches: one a leg instead of three, which bound these levels: the plain
// engine's V-cycle (tq_vcycle_noalloc, FP32) went from 182 to 65 us on 160x100 cells, 282 to
// 130 us on 840x536 (111 since the launches overlap), bits unchanged.
//
// Shared arrays hold the cells from (fx0 - 10, fy0 - 10) on, H rows of pitch P = 16 kx + 20 (4 mod
// 8: a warp's 64-bit accesses of four rows of a block then meet no bank twice).
struct Ladrilho {
  int fx0, fy0, kx, ky;  // first cell and size in blocks
  int nx, ny;            // the level
  const uint8_t* viz;
};
__host__ __device__ constexpr int passoLadrilho(int k) { return 16 * k + 20; }
// Floats of the arrays of one leg: x before and after a pass, the right side, the masks (bytes), and
// going up the coarse tile.
__host__ __device__ constexpr int areaLadrilho(int kx, int ky) { return passoLadrilho(kx) * passoLadrilho(ky); }
__host__ __device__ constexpr size_t bytesLadrilho(int kx, int ky) {
  return (size_t)areaLadrilho(kx, ky) * 13 + (size_t)(8 * kx + 10) * (8 * ky + 10) * 4;
}

// The value a level's storage type keeps of v.
template <class T>
__device__ __forceinline__ float arredondar(float v) { return carregar(guardar<T>(v)); }

// The column (0 or 1) of a lane's pair that colour cr has in row m (see meiaReg).
#define TQ_COL(cr, m) (((cr) + 1 + (m)) & 1)

// A lane's cells of the block at (ox, oy) and the block's frame from a shared array of tile L.
__device__ __forceinline__ void lerBlocoS(const Ladrilho& L, int ox, int oy, const float* xs, float (&x)[2][4],
                                          Moldura& f) {
  const int lane = threadIdx.x & 31, gl = lane >> 3, k = lane & 7, P = passoLadrilho(L.kx);
  const float* o = xs + (oy - L.fy0 + 10 + 4 * gl) * P + ox - L.fx0 + 10 + 2 * k;
#pragma unroll
  for (int m = 0; m < 4; m++) {
    const float2 v = *reinterpret_cast<const float2*>(o + m * P);
    x[(1 + m) & 1][m] = v.x;
    x[m & 1][m] = v.y;
    f.esq[m] = k == 0 ? o[m * P - 1] : 0.0f;
    f.dir[m] = k == 7 ? o[m * P + 2] : 0.0f;
  }
#pragma unroll
  for (int j = 0; j < 2; j++) {
    f.bai[j] = gl == 0 ? o[j - P] : 0.0f;
    f.cim[j] = gl == 3 ? o[j + 4 * P] : 0.0f;
  }
}
// A lane's cells into a shared array (the part of the block inside the array).
__device__ __forceinline__ void gravarBlocoS(const Ladrilho& L, int ox, int oy, float* xs, const float (&x)[2][4]) {
  const int lane = threadIdx.x & 31, gl = lane >> 3, k = lane & 7, P = passoLadrilho(L.kx), H = passoLadrilho(L.ky);
  const int cx = ox - L.fx0 + 10 + 2 * k, cy = oy - L.fy0 + 10 + 4 * gl;
  if (cx < 0 || cx >= P) return;
#pragma unroll
  for (int m = 0; m < 4; m++)
    if (cy + m >= 0 && cy + m < H)
      *reinterpret_cast<float2*>(xs + (cy + m) * P + cx) = make_float2(x[(1 + m) & 1][m], x[m & 1][m]);
}
__device__ __forceinline__ void gravarBlocoS(const Ladrilho& L, int ox, int oy, uint8_t* vs, const int (&v)[2][4]) {
  const int lane = threadIdx.x & 31, gl = lane >> 3, k = lane & 7, P = passoLadrilho(L.kx), H = passoLadrilho(L.ky);
  const int cx = ox - L.fx0 + 10 + 2 * k, cy = oy - L.fy0 + 10 + 4 * gl;
  if (cx < 0 || cx >= P) return;
#pragma unroll
  for (int m = 0; m < 4; m++)
    if (cy + m >= 0 && cy + m < H)
      *reinterpret_cast<uchar2*>(vs + (cy + m) * P + cx) =
          make_uchar2((unsigned char)v[(1 + m) & 1][m], (unsigned char)v[m & 1][m]);
}
__device__ __forceinline__ void lerMascarasS(const Ladrilho& L, int ox, int oy, const uint8_t* vs, int (&v)[2][4]) {
  const int lane = threadIdx.x & 31, gl = lane >> 3, k = lane & 7, P = passoLadrilho(L.kx);
  const uint8_t* o = vs + (oy - L.fy0 + 10 + 4 * gl) * P + ox - L.fx0 + 10 + 2 * k;
#pragma unroll
  for (int m = 0; m < 4; m++) {
    const uchar2 q = *reinterpret_cast<const uchar2*>(o + m * P);
    v[(1 + m) & 1][m] = q.x;
    v[m & 1][m] = q.y;
  }
}
// Whether a lane's cell of the block is the tile's own (each cell of the level belongs to one tile).
__device__ __forceinline__ bool proprio(const Ladrilho& L, int gx, int gy) {
  return gx >= L.fx0 && gy >= L.fy0 && gx < L.fx0 + 16 * L.kx && gy < L.fy0 + 16 * L.ky;
}
__device__ __forceinline__ bool mexe(const int (&v)[2][4]) {
  bool a = false;
#pragma unroll
  for (int cr = 0; cr < 2; cr++)
#pragma unroll
    for (int m = 0; m < 4; m++) a |= (v[cr][m] & 16) && (v[cr][m] & 15);
  return __any_sync(0xffffffffu, a);
}

// The way down on tile L by the whole CTA: lerB(c) loads what the right side of cell c is made from and
// fazerB(c, mask, value, own) makes the stored right side of it (own: the tile's own cell),
// gravarX(c, x) takes the tile's own cells' x, gravarG(C, s) the coarse cells' restricted residual
// (0 on dry ones).  uma: TQ_PRECOND_BLOCK_1's single pass, blocks at shift 8.
template <class T, class LB, class FB, class GX, class GG>
__device__ __forceinline__ void descerLadrilho(const Ladrilho& L, int gnx, int gny, const uint8_t* gviz, bool uma,
                                               bool masc, int nVarr, float* mem, LB lerB, FB fazerB, GX gravarX,
                                               GG gravarG) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5, gl = lane >> 3, k = lane & 7;
  const int nx = L.nx, ny = L.ny, P = passoLadrilho(L.kx), A = areaLadrilho(L.kx, L.ky);
  float *x1 = mem, *x2 = mem + A, *bs = mem + 2 * A;
  uint8_t* vs = (uint8_t*)(mem + 3 * A);
  {
    const int desl = uma ? 8 : 16, bx = L.kx + (uma ? 1 : 2), nb = bx * (L.ky + (uma ? 1 : 2));
    for (int b = w; b < nb; b += nw) {
      const int ox = L.fx0 - desl + 16 * (b % bx), oy = L.fy0 - desl + 16 * (b / bx);
      float x[2][4], bq[2][4];
      int v[2][4];
#pragma unroll
      for (int cr = 0; cr < 2; cr++)
#pragma unroll
        for (int m = 0; m < 4; m++) {
          const int gx = ox + 2 * k + TQ_COL(cr, m), gy = oy + 4 * gl + m;
          const bool dentro = gx >= 0 && gy >= 0 && gx < nx && gy < ny;
          v[cr][m] = dentro ? (int)__ldca(L.viz + gx + gy * nx) : 0;
          bq[cr][m] = dentro ? lerB(gx + gy * nx) : 0.0f;
          x[cr][m] = 0.0f;
        }
#pragma unroll
      for (int cr = 0; cr < 2; cr++)
#pragma unroll
        for (int m = 0; m < 4; m++) {
          const int gx = ox + 2 * k + TQ_COL(cr, m), gy = oy + 4 * gl + m;
          const bool dentro = gx >= 0 && gy >= 0 && gx < nx && gy < ny;
          if (dentro) bq[cr][m] = fazerB(gx + gy * nx, v[cr][m], bq[cr][m], proprio(L, gx, gy));
        }
      Moldura f{};
      if (mexe(v)) varrerReg(x, v, bq, f, 0, masc, nVarr);
#pragma unroll
      for (int cr = 0; cr < 2; cr++)
#pragma unroll
        for (int m = 0; m < 4; m++) {
          x[cr][m] = (v[cr][m] & 16) ? arredondar<T>(x[cr][m]) : 0.0f;
          const int gx = ox + 2 * k + TQ_COL(cr, m), gy = oy + 4 * gl + m;
          if (uma && proprio(L, gx, gy) && gx < nx && gy < ny) gravarX(gx + gy * nx, x[cr][m]);
        }
      gravarBlocoS(L, ox, oy, uma ? x2 : x1, x);
      gravarBlocoS(L, ox, oy, bs, bq);
      gravarBlocoS(L, ox, oy, vs, v);
    }
  }
  __syncthreads();
  if (!uma) {
    const int bx = L.kx + 1, nb = bx * (L.ky + 1);
    for (int b = w; b < nb; b += nw) {
      const int ox = L.fx0 - 8 + 16 * (b % bx), oy = L.fy0 - 8 + 16 * (b / bx);
      float x[2][4], bq[2][4];
      int v[2][4];
      Moldura f, nada;
      lerBlocoS(L, ox, oy, x1, x, f);
      lerBlocoS(L, ox, oy, bs, bq, nada);
      lerMascarasS(L, ox, oy, vs, v);
      if (mexe(v)) varrerReg(x, v, bq, f, 0, masc, nVarr);
#pragma unroll
      for (int cr = 0; cr < 2; cr++)
#pragma unroll
        for (int m = 0; m < 4; m++) {
          x[cr][m] = (v[cr][m] & 16) ? arredondar<T>(x[cr][m]) : 0.0f;
          const int gx = ox + 2 * k + TQ_COL(cr, m), gy = oy + 4 * gl + m;
          if (proprio(L, gx, gy) && gx < nx && gy < ny) gravarX(gx + gy * nx, x[cr][m]);
        }
      gravarBlocoS(L, ox, oy, x2, x);
    }
    __syncthreads();
  }
  // residuals of the tile's cells and the ring around them (a row a warp), into x1
  for (int j = w; j < 16 * L.ky + 2; j += nw)
    for (int i = lane; i < 16 * L.kx + 2; i += 32) {
      const int o = (j + 9) * P + i + 9, vz = vs[o];
      float s = 0.0f;
      s += (vz & 1) ? x2[o - 1] : 0.0f;
      s += (vz & 2) ? x2[o + 1] : 0.0f;
      s += (vz & 4) ? x2[o - P] : 0.0f;
      s += (vz & 8) ? x2[o + P] : 0.0f;
      x1[o] = (vz & 16) ? bs[o] - fmaf((float)__popc(vz & 15), x2[o], -s) : 0.0f;
    }
  __syncthreads();
  // restringir (js/pressao-cpu.js:159-188) as a gather over 4x4 windows
  const float pes[4] = {0.25f, 0.75f, 0.75f, 0.25f};
  const int cw = 8 * L.kx;
  for (int t = threadIdx.x; t < cw * 8 * L.ky; t += blockDim.x) {
    const int i = t % cw, j = t / cw, I = (L.fx0 >> 1) + i, J = (L.fy0 >> 1) + j;
    if (I >= gnx || J >= gny) continue;
    const float* r = x1 + (2 * j + 9) * P + 2 * i + 9;
    float s = 0.0f;
    if (__ldca(gviz + I + J * gnx) & 16) {
#pragma unroll
      for (int bb = 0; bb < 4; bb++)
#pragma unroll
        for (int aa = 0; aa < 4; aa++) s = __fadd_rn(s, __fmul_rn(r[bb * P + aa], pes[aa] * pes[bb]));
    }
    gravarG(I + J * gnx, s);
  }
}

// The way up on tile L by the whole CTA: lerX(c) the cell's x, lerC(C) the coarse level's x (0 on dry
// cells), lerB(c) its right side; gravar(cel, v, x) takes each lane's cells of a swept block (cel -1
// outside the grid), the level's result.  uma: a single pass, and the tile's blocks are those of shift 8.
template <class T, class LX, class LC, class LB, class GV>
__device__ __forceinline__ void subirLadrilho(const Ladrilho& L, int gnx, int gny, bool uma, bool masc, int nVarr,
                                              float* mem, LX lerX, LC lerC, LB lerB, GV gravar) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5, gl = lane >> 3, k = lane & 7;
  const int nx = L.nx, ny = L.ny, P = passoLadrilho(L.kx), A = areaLadrilho(L.kx, L.ky);
  float *x1 = mem, *x2 = mem + A, *cs = mem + 2 * A;
  const int cw = 8 * L.kx + 10, chh = 8 * L.ky + 10;
  uint8_t* vs = (uint8_t*)(cs + cw * chh);
  const int cx0 = (L.fx0 >> 1) - 5, cy0 = (L.fy0 >> 1) - 5;
  // every load of a batch goes out before its first store
  const int xw = 16 * L.kx + 18, nX = xw * (16 * L.ky + 18), nC = cw * chh;
  constexpr int KC = 2, KX = 5;
  for (int c0 = threadIdx.x, t0 = threadIdx.x; c0 < nC || t0 < nX; c0 += KC * blockDim.x, t0 += KX * blockDim.x) {
    float cv[KC], xv[KX];
    int vz[KX], o[KX];
#pragma unroll
    for (int q = 0; q < KC; q++) {
      const int t = c0 + q * blockDim.x, I = cx0 + t % cw, J = cy0 + t / cw;
      cv[q] = t < nC && I >= 0 && J >= 0 && I < gnx && J < gny ? lerC(I + J * gnx) : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < KX; q++) {
      const int t = t0 + q * blockDim.x, i = t % xw, j = t / xw, gx = L.fx0 - 9 + i, gy = L.fy0 - 9 + j;
      const bool dentro = t < nX && gx >= 0 && gy >= 0 && gx < nx && gy < ny;
      o[q] = t < nX ? (j + 1) * P + i + 1 : -1;
      vz[q] = dentro ? (int)__ldca(L.viz + gx + gy * nx) : 0;
      xv[q] = dentro ? lerX(gx + gy * nx) : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < KC; q++)
      if (c0 + q * (int)blockDim.x < nC) cs[c0 + q * blockDim.x] = cv[q];
#pragma unroll
    for (int q = 0; q < KX; q++)
      if (o[q] >= 0) {
        vs[o[q]] = (uint8_t)vz[q];
        x1[o[q]] = xv[q];
      }
  }
  __syncthreads();
  // prolongar (js/pressao-cpu.js:191-214): water cells take the bilinear coarse correction
  for (int j = w; j < 16 * L.ky + 18; j += nw)
    for (int i = lane; i < 16 * L.kx + 18; i += 32) {
      const int o = (j + 1) * P + i + 1;
      if (!(vs[o] & 16)) continue;
      const int gx = L.fx0 - 9 + i, gy = L.fy0 - 9 + j;
      const float* c = cs + (grossoBaseF(gy) - cy0) * cw + grossoBaseF(gx) - cx0;
      const float wx0 = pesoBaseF(gx), wy0 = pesoBaseF(gy);
      float e = 0.0f;
      e = fmaf(c[0], wx0 * wy0, e);
      e = fmaf(c[1], (1.0f - wx0) * wy0, e);
      e = fmaf(c[cw], wx0 * (1.0f - wy0), e);
      e = fmaf(c[cw + 1], (1.0f - wx0) * (1.0f - wy0), e);
      x1[o] = arredondar<T>(x1[o] + e);
    }
  __syncthreads();
  auto passo = [&](int ox, int oy, const float* xs, float (&x)[2][4], int (&v)[2][4], int (&cel)[2][4]) {
    float bq[2][4];
    Moldura f;
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++) {
        const int gx = ox + 2 * k + TQ_COL(cr, m), gy = oy + 4 * gl + m;
        const bool dentro = gx >= 0 && gy >= 0 && gx < nx && gy < ny;
        cel[cr][m] = dentro ? gx + gy * nx : -1;
        bq[cr][m] = dentro ? lerB(cel[cr][m]) : 0.0f;
      }
    lerBlocoS(L, ox, oy, xs, x, f);
    lerMascarasS(L, ox, oy, vs, v);
    if (mexe(v)) varrerReg(x, v, bq, f, 1, masc, nVarr);
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++) x[cr][m] = (v[cr][m] & 16) ? x[cr][m] : 0.0f;
  };
  const int bx = L.kx + (uma ? 0 : 1), nb = bx * (L.ky + (uma ? 0 : 1));
  for (int b = w; b < nb; b += nw) {
    const int ox = L.fx0 - 8 + 16 * (b % bx), oy = L.fy0 - 8 + 16 * (b / bx);
    float x[2][4];
    int v[2][4], cel[2][4];
    passo(ox, oy, x1, x, v, cel);
    if (uma) {
      gravar(cel, v, x);
      continue;
    }
#pragma unroll
    for (int cr = 0; cr < 2; cr++)
#pragma unroll
      for (int m = 0; m < 4; m++) x[cr][m] = arredondar<T>(x[cr][m]);
    gravarBlocoS(L, ox, oy, x2, x);
  }
  if (uma) return;
  __syncthreads();
  for (int b = w; b < L.kx * L.ky; b += nw) {
    const int ox = L.fx0 + 16 * (b % L.kx), oy = L.fy0 + 16 * (b / L.kx);
    float x[2][4];
    int v[2][4], cel[2][4];
    passo(ox, oy, x2, x, v, cel);
    gravar(cel, v, x);
  }
}

}  // namespace tq
