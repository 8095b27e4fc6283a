// ntt_tc.cu -- the tensor-core pass kernels (ntt_tc.cuh): matrices, instances, and when they run.
#include <cuda_runtime.h>

#include <cstdint>

#include "ntt_host.cuh"
#include "ntt_tc.cuh"

namespace bc {

namespace tc {
// One block per matrix, one thread per entry.
__global__ void __launch_bounds__(256) fill_images_kernel(uint8_t *img) {
  const uint32_t b = blockIdx.x, V = b % 4 + 1, o = threadIdx.x >> 4, i = threadIdx.x & 15;
  const bool dif = (b / 8) != 0, inv = (b / 4) % 2 != 0;
  const uint64_t m = (o >> V) == (i >> V) ? pow2_mod((uint32_t)entry_exp(dif, inv, (int)V, o, i)) : 0;
  put_entry(img + b * IMG_BYTES, o, i, m);
}
} // namespace tc

cudaError_t tc_fill_images(uint8_t *img) {
  tc::fill_images_kernel<<<tc::IMAGES, 256>>>(img);
  return cudaGetLastError();
}

// A natural -> bit-reversed inverse scales by bit-reversed indexes in its pass at
// bit 0, which is not this kernel's, and does not gain from it with 9 bits above
// (launch_ntt): no instances.
template <int K, bool LOW> static PassKernel tk(bool b2n, bool inverse) {
  if (b2n) return inverse ? tc::pass_kernel_tc<K, LOW, true, true> : tc::pass_kernel_tc<K, LOW, true, false>;
  if (!inverse) return tc::pass_kernel_tc<K, LOW, false, false>;
  if constexpr (!LOW && K != 9)
    return tc::pass_kernel_tc<K, LOW, false, true>;
  else
    return nullptr;
}

PassKernel pick_pass_kernel_tc(int K, bool low, bool b2n, bool inverse) {
  if (low) {
    switch (K) {
    case 8: return tk<8, true>(b2n, inverse);
    case 9: return tk<9, true>(b2n, inverse);
    case 10: return tk<10, true>(b2n, inverse);
    case 11: return tk<11, true>(b2n, inverse);
    case 12: return tk<12, true>(b2n, inverse);
    }
  } else {
    switch (K) {
    case 4: return tk<4, false>(b2n, inverse);
    case 5: return tk<5, false>(b2n, inverse);
    case 8: return tk<8, false>(b2n, inverse);
    case 9: return tk<9, false>(b2n, inverse);
    case 10: return tk<10, false>(b2n, inverse);
    }
  }
  return nullptr;
}

size_t tc_pass_smem(int K) {
  switch (K) {
  case 4: return tc::pass_smem_bytes<4>();
  case 5: return tc::pass_smem_bytes<5>();
  case 8: return tc::pass_smem_bytes<8>();
  case 9: return tc::pass_smem_bytes<9>();
  case 10: return tc::pass_smem_bytes<10>();
  case 11: return tc::pass_smem_bytes<11>();
  case 12: return tc::pass_smem_bytes<12>();
  }
  return 0;
}

// Columns of a tile (log2) of a window of K bits.
uint32_t tc_log_g(int K, bool low) { return low ? tc::TILE_BITS - K : 0; }

// Whether the tensor-core kernel has the window [lb, lb + K) and fills its tiles
// with the columns there are.
bool tc_window_ok(int K, uint32_t lb, uint32_t cols, bool b2n, bool inverse) {
  const bool low = lb == 0;
  if (!low && lb < (uint32_t)(tc::TILE_BITS - K)) return false;
  const uint64_t g = 1ull << tc_log_g(K, low), tiles = (cols + g - 1) / g;
  if (4ull * cols < 3 * tiles * g) return false;
  if (cols > 65535) return false; // grid.y: one column a CTA at least (the other kernels tile columns)
  return pick_pass_kernel_tc(K, low, b2n, inverse) != nullptr;
}

bool tc_pass_ok(const PassLaunch &q) {
  // whole scalings by base^i belong to the other kernels; n^-1 alone on a
  // bit-reversed -> natural pass's outputs is this one's
  if (q.load_scale) return false;
  if (q.store_scale && (!q.b2n || (q.has_coset && q.share == SHARE_NONE))) return false;
  if (((uint64_t)q.cols << q.log_groups) > 65535) return false;
  return tc_window_ok(q.K, q.lb, q.cols, q.b2n, q.inverse);
}

} // namespace bc
