// lde_tc.cu -- the tensor-core top-window kernels (lde_tc.cuh): their tables, instances, and when they run.
#include <cuda_runtime.h>

#include <cstdint>

#include "lde_tc.cuh"

namespace bc {

namespace tc {
// Coset matrices: block H, one thread per entry.
__global__ void __launch_bounds__(256) fill_coset_images_kernel(uint8_t *img, const DevTables tabs) {
  const uint32_t H = blockIdx.x, o = threadIdx.x >> 4, i = threadIdx.x & 15;
  const uint64_t m = pow2_mod((uint32_t)entry_exp(false, false, 4, o, i));
  put_entry(img + H * IMG_BYTES, o, i, gl::mul_canon(m, gl::pow(twiddle(tabs, 0, H << 3), i)));
}

// The 32-point matrix: w_32^(i brev5(o)), w_32 = 2^78.
__global__ void __launch_bounds__(256) fill_wide_image_kernel(uint8_t *img) {
  const uint32_t t = blockIdx.x * 256 + threadIdx.x, o = t >> 5, i = t & 31;
  const uint64_t m = pow2_mod((78u * ((i * (__brev(o) >> 27)) & 31)) % 192);
  put_entry(img + (i >> 4) * (WIDE_IMG_BYTES / 2), o, i & 15, m);
}

// Power tables of prefix H: those of a 10-bit window of two 5-bit rounds, and PowerTable<8>.
__global__ void __launch_bounds__(256) fill_top_powers_kernel(uint64_t *wide, uint64_t *pw8, const DevTables tabs) {
  const uint32_t H = blockIdx.x;
  for (uint32_t t = threadIdx.x; t < 1024; t += 256)
    wide[H * 1024 + t] = gl::canon(gl::pow(twiddle(tabs, 0, (H << 9) + (t >> 5 << 4)), t & 31));
  fill_power_table<8>(pw8 + H * PowerTable<8>::words, tabs, 0, H, Scale{false, 0, 0}, 0);
}
} // namespace tc

size_t tc_table_bytes() { return tc::TOP_TABLE_END; }

cudaError_t tc_fill_tables(uint8_t *img, const DevTables &tabs) {
  using namespace tc;
  cudaError_t e = tc_fill_images(img);
  if (e != cudaSuccess) return e;
  fill_coset_images_kernel<<<TOP_PREFIXES, 256>>>(img + COSET_IMG_OFF, tabs);
  fill_wide_image_kernel<<<4, 256>>>(img + WIDE_IMG_OFF);
  fill_top_powers_kernel<<<TOP_PREFIXES, 256>>>(reinterpret_cast<uint64_t *>(img + WIDE_PW_OFF),
                                                reinterpret_cast<uint64_t *>(img + PW8_OFF), tabs);
  return cudaGetLastError();
}

TopKernel pick_top_tc(int K) {
  switch (K) {
  case 4: return tc::top_kernel_tc<4, false>;
  case 5: return tc::top_kernel_tc<5, true>;
  case 8: return tc::top_kernel_tc<8, false>;
  case 10: return tc::top_kernel_tc<10, true>;
  }
  return nullptr;
}

size_t tc_top_smem(int K) {
  switch (K) {
  case 4: return tc::top_tc_smem_bytes<4, false>();
  case 5: return tc::top_tc_smem_bytes<5, true>();
  case 8: return tc::top_tc_smem_bytes<8, false>();
  case 10: return tc::top_tc_smem_bytes<10, true>();
  }
  return 0;
}

bool tc_top_ok(int K, uint32_t lb, uint32_t log_blowup) {
  return log_blowup < 32 && (1u << log_blowup) <= tc::TOP_PREFIXES && lb >= (uint32_t)(tc::TILE_BITS - K) && pick_top_tc(K);
}

} // namespace bc
