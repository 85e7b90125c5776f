// pcg_interno.cuh — the pressure-solver object shared by the plain engine (pcg.cu) and the
// fused engine (pcg_fundido.cu).
#pragma once
#include <vector>

#include "arena.cuh"
#include "common.cuh"

namespace tq {

// Levels with at least this many cells store the V-cycle vectors in 16-bit when a
// half-precision mode is selected (the small coarse levels stay FP32).
constexpr int MEIA_MIN_CELULAS = 16384;

struct Fundido;

struct Pcg {
  int nx, ny, N, precisao, motor;
  int ctasFundido = 0;  // the fused engine's CTA count (0: one per SM)
  int L;
  int nxL[MAX_NIVEIS], nyL[MAX_NIVEIS];
  bool meia[MAX_NIVEIS];  // level stored in half precision
  uint8_t* tipoL[MAX_NIVEIS];
  uint8_t* vizL[MAX_NIVEIS];
  void *bL[MAX_NIVEIS], *xL[MAX_NIVEIS], *tmpL[MAX_NIVEIS];  // 4 bytes per element allocated
  uint8_t* vizOp;
  double* q64 = nullptr;  // the plain engine's FP64 iterate (tolerance mode), allocated on first use
  // the plain engine's operator descriptors, second p, partial sums and active bubbles (pcg.cu, Plano)
  uint16_t* op = nullptr;
  float* p2 = nullptr;
  double* parc = nullptr;
  int* ativos = nullptr;
  const int* parar = nullptr;  // the running plain solve's stop flag (NivelDev::parar)
  size_t smemGrosso = 0;
  Fundido* fundido = nullptr;
  Regioes* regioes = nullptr;  // tolerance mode's closed-region projection, allocated on first use
};

// The bubbles' face and cell counts and fixed-point sums to 0: one block of memory (Dev::accB, facesB, celsB).
inline void zerarBolhas(const Dev& d, cudaStream_t s) {
  cudaMemsetAsync(d.accB, 0, MAX_BOLHAS * (sizeof(long long) + 2 * sizeof(uint32_t)), s);
}

// pcg_fundido.cu
Fundido* criarFundido(Pcg* p, Arena& A);
bool iniciarFundido(Fundido* f, const Pcg* p, cudaStream_t s);
void destruirFundido(Fundido* f);
int resolverPressaoFundido(Pcg* p, const Dev& d, int iteracoes, double tol, bool bolhas, int precond,
                           cudaStream_t s);
int erroFundido(Fundido* f, cudaStream_t s);
void perfilFundido(Fundido* f, bool ligar);
int lerPerfilFundido(Fundido* f, unsigned long long* out, int cap);

}  // namespace tq
