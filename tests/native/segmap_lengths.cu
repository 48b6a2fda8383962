// Test kernels for the segmented map (built to lib/libsgs_segmap_test.so): a
// frontier of given lengths, zero-length entries among them, mapped with an op
// that notes who visits each slot.
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "sgs_segmap.cuh"

namespace {

using namespace sgs;

__global__ void k_append(const uint32_t *len, uint32_t n, FrontierView f) {
  for (uint32_t b = 0; b < n; b += 32) {  // one warp: entry i is vertex i
    const uint32_t i = b + threadIdx.x;
    frontier_append(f, i < n, i, i < n ? len[i] : 0u);
  }
}

// Adds one to seen[first[v] + j] for every visited slot j of v, as `width` wide
// an op as the engine's: one slot or four at a time.
template <bool Quad>
struct NoteOp {
  static constexpr bool kAppends = false;
  static constexpr bool kQuad = Quad;
  struct Payload {
    uint64_t first;
  };
  const uint64_t *first;
  uint32_t *seen;
  uint64_t total;
  __device__ __forceinline__ Payload load(uint32_t, uint32_t v) const { return Payload{first[v]}; }
  __device__ __forceinline__ uint32_t visit(uint32_t, const Payload &p, uint32_t j, bool &, uint32_t &,
                                            uint32_t &) const {
    if (p.first + j < total) atomicAdd(&seen[p.first + j], 1u);
    return 1;
  }
  __device__ __forceinline__ uint32_t visit4(uint32_t v, const Payload &p, uint32_t j0, uint32_t len, bool (&a)[4],
                                             uint32_t (&b)[4], uint32_t (&c)[4]) const {
    uint32_t n = 0;
    for (int k = 0; k < 4; ++k)
      if (j0 + k < len) n += visit(v, p, j0 + k, a[k], b[k], c[k]);
    return n;
  }
};

template <class T>
struct Dev {
  T *p = nullptr;
  explicit Dev(size_t n) {
    if (cudaMalloc((void **)&p, (n ? n : 1) * sizeof(T)) != cudaSuccess) p = nullptr;
    if (p) cudaMemset(p, 0, (n ? n : 1) * sizeof(T));
  }
  ~Dev() { cudaFree(p); }
};

}  // namespace

// Visits per slot (entry after entry) of a map over `n` entries of `len` slots;
// *counted = the map's own count.  Returns a cudaError_t.
extern "C" __attribute__((visibility("default"))) int sgs_test_segmap(uint32_t n, const uint32_t *len, int quad,
                                                                      uint32_t ctas, uint32_t *seen,
                                                                      uint64_t *counted) {
  std::vector<uint64_t> first(n + 1, 0);
  uint64_t padded = 0;
  for (uint32_t i = 0; i < n; ++i) {
    first[i + 1] = first[i] + len[i];
    padded += (len[i] + 3u) & ~3u;
  }
  const uint64_t total = first[n];
  const uint32_t units = (uint32_t)(padded / UNIT + 2);
  Dev<uint32_t> d_len(n), vtx(n + 1), flen(n + 1), ustart(units), d_seen(total);
  Dev<uint64_t> ebase(n + 1), d_first(n + 1);
  Dev<unsigned long long> counters(3);
  for (const void *p : {(const void *)d_len.p, (const void *)vtx.p, (const void *)flen.p, (const void *)ustart.p,
                        (const void *)d_seen.p, (const void *)ebase.p, (const void *)d_first.p,
                        (const void *)counters.p})
    if (!p) return (int)cudaErrorMemoryAllocation;
  cudaMemcpy(d_len.p, len, n * sizeof(uint32_t), cudaMemcpyHostToDevice);
  cudaMemcpy(d_first.p, first.data(), (n + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice);
  FrontierView f{vtx.p, flen.p, ebase.p, ustart.p, (uint64_t *)counters.p, units};
  FrontierView out{vtx.p, flen.p, ebase.p, ustart.p, (uint64_t *)(counters.p + 1), units};  // never appended to
  k_append<<<1, 32>>>(d_len.p, n, f);
  if (quad) seg_map<<<ctas, RELAX_THREADS>>>(f, out, NoteOp<true>{d_first.p, d_seen.p, total}, counters.p + 2);
  else seg_map<<<ctas, RELAX_THREADS>>>(f, out, NoteOp<false>{d_first.p, d_seen.p, total}, counters.p + 2);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(seen, d_seen.p, total * sizeof(uint32_t), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(counted, counters.p + 2, sizeof(uint64_t), cudaMemcpyDeviceToHost);
  return (int)e;
}
