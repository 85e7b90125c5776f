// arena.cuh — the device memory of one object as one allocation: its arrays are asked for first, then
// reserved together and zeroed on the object's stream.  A handle's 110 arrays allocated and freed one by
// one took 40 ms on 840x536 cells, four fifths of a tq_solve_pressure call.
#pragma once
#include <cuda_runtime.h>

#include <vector>

namespace tq {

class Arena {
 public:
  Arena() = default;
  Arena(const Arena&) = delete;
  Arena& operator=(const Arena&) = delete;
  ~Arena() {
    if (base) cudaFree(base);
  }
  // *p gets n elements (on a 256-byte boundary, with 16 bytes to spare) when the arena is reserved; p
  // itself must stay where it is until then.
  template <class T>
  void pedir(T** p, size_t n) {
    pedidos.push_back({reinterpret_cast<void**>(p), total});
    total += (n * sizeof(T) + 16 + 255) & ~(size_t)255;
  }
  // One allocation for everything asked for, zeroed on s; false when there is no room.
  bool reservar(cudaStream_t s) {
    if (cudaMalloc(&base, total) != cudaSuccess) {
      cudaGetLastError();
      base = nullptr;
      return false;
    }
    for (auto& q : pedidos) *q.p = static_cast<char*>(base) + q.off;
    pedidos.clear();
    return cudaMemsetAsync(base, 0, total, s) == cudaSuccess;
  }

 private:
  struct Pedido {
    void** p;
    size_t off;
  };
  std::vector<Pedido> pedidos;
  size_t total = 0;
  void* base = nullptr;
};

}  // namespace tq
