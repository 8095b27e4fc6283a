// ntt_tc.cuh -- a pass of ntt_pass.cuh with its rounds on the tensor cores (tc.cuh).
//
// Same windows, twiddles, tile positions and results as pass_body; a tile is
// always 4096 elements (256 threads).  Rounds take 4 window bits from the top;
// with K mod 4 bits left, a short round at the bottom (its matrix block
// diagonal).  Per round: one MMA pair over the tile, then every thread folds
// its row's 16 outputs, multiplies them by powers where the next (DIT) or
// this (DIF) round has them, and stores each where the next round's operand
// wants it.  The window's top round has one s for the whole tile: s^j, the
// coset step and n^-1 are multiplied into its matrix instead, once per CTA.
//
// Split.  128 registers, 2 CTAs an SM (their accumulators are all of tensor
// memory): while one CTA waits for its MMAs the other folds.  The matrix of
// the top round is built per CTA (about 130 instructions a thread) because it
// saves 15 of 16 multiplications per element of a round in every column.
#pragma once
#include "ntt_host.cuh"
#include "ntt_pass.cuh"
#include "tc.cuh"

namespace bc {
namespace tc {

// Shared memory of a pass: tile, matrices (top round, full round, short round),
// power table, barrier and tensor-memory address; 1 KB to align the tile.
template <int K> __host__ __device__ constexpr uint32_t pass_images() { return K % 4 ? 3 : 2; }
template <int K> __host__ __device__ constexpr uint32_t pass_smem_bytes() {
  return 1024 + TILE_BYTES + pass_images<K>() * IMG_BYTES + PowerTable<K>::words * 8 + 32;
}

// A thread whose wait ran out waits for nothing more and goes on to the end:
// what it then reads and overwrites early is its own CTA's tile and
// accumulators, so the launch's results are invalid (and reported) but nothing
// else is touched.  The issuing thread also issues nothing more.  Telling the
// whole CTA at its next barrier instead cost 1 to 5 % of every kernel.
struct Ctx {
  uint32_t bar, tmem, phase;
  uint32_t tries; // bound of a wait
  uint32_t bad;   // 0, or 1 + the barrier's phase whose wait ran out
};

// Barrier and tensor memory of a CTA; ends with a barrier.  slot: 16 bytes of shared memory.
__device__ __forceinline__ Ctx begin(uint64_t *slot, uint32_t tries) {
  Ctx c;
  c.bar = smem_u32(slot);
  c.phase = 0;
  c.tries = tries;
  c.bad = 0;
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot + 1)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(c.bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  c.tmem = *reinterpret_cast<volatile uint32_t *>(slot + 1);
  return c;
}

// Frees the tensor memory.  Products that the issuing thread gave up on may
// still be running: it waits for them once more first, so that they do not end
// in the memory of whoever is given it next.
__device__ __forceinline__ void end(const Ctx &c, uint32_t *error) {
  if (c.bad) {
    if (threadIdx.x == 0) mbar_wait(c.bar, c.bad - 1, WAIT_TRIES);
    if (error) *(volatile uint32_t *)error = 1u;
  }
  fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem), "r"(TMEM_COLS));
}

// Whether this CTA is of the first `wave` of its launch (0: launched without
// overlap): only those can start before the predecessor has ended.
__device__ __forceinline__ bool in_first_wave(uint32_t wave) { return blockIdx.y * gridDim.x + blockIdx.x < wave; }

// One round's products, issued by one thread: orders this CTA's shared-memory
// stores before, and returns when every operand has been read and all sums are
// in tensor memory (or, c.bad, without).
template <class F> __device__ __forceinline__ void products(Ctx &c, F &&issue) {
  fence_smem_to_mma();
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  if (threadIdx.x == 0 && !c.bad) {
    issue();
    mma_commit(c.bar);
  }
  __syncwarp();
  if (!c.bad && !mbar_wait(c.bar, c.phase, c.tries)) c.bad = 1 + c.phase;
  c.phase ^= 1;
  __syncwarp();
  fence_after_sync();
}

// The tile times the matrix at img.
__device__ __forceinline__ void multiply(Ctx &c, uint32_t tile, uint32_t img) {
  products(c, [&] {
    const uint64_t b = operand_desc(img);
    mma_128x128(c.tmem, operand_desc(tile), b);
    mma_128x128(c.tmem + 128, operand_desc(tile + TILE_BYTES / 2), b);
  });
}

// use(o, y) for the 16 outputs of the thread's row, the reads of four outputs
// in flight while the previous four are folded.
template <class F> __device__ __forceinline__ void outputs(const Ctx &c, F &&use) {
  const uint32_t warp = threadIdx.x >> 5;
  const uint32_t a = c.tmem + ((warp & 3) << 21) + (warp >> 2) * 128;
  uint32_t d0[32], d1[32];
  ld_digits32(d0, a);
  wait_ld(d0);
  ld_digits32(d1, a + 32);
#pragma unroll
  for (int o = 0; o < 4; o++) use(o, fold_digits(d0 + 8 * o));
  wait_ld(d1);
  ld_digits32(d0, a + 64);
#pragma unroll
  for (int o = 0; o < 4; o++) use(4 + o, fold_digits(d1 + 8 * o));
  wait_ld(d0);
  ld_digits32(d1, a + 96);
#pragma unroll
  for (int o = 0; o < 4; o++) use(8 + o, fold_digits(d0 + 8 * o));
  wait_ld(d1);
#pragma unroll
  for (int o = 0; o < 4; o++) use(12 + o, fold_digits(d1 + 8 * o));
}

// Scaling by base^i, i the natural index in the column: DIT rounds multiply
// their input j and DIF rounds their output j by s_R^j, and j is a field of
// the natural index at bit lb + B, so (s_R base^(2^(lb + B)))^j scales by that
// field's share: no multiplication of its own.
struct Scale {
  bool on;
  uint32_t inv, kshift; // coset_power's arguments: base = c or c^-1
  __device__ __forceinline__ uint64_t power(const DevTables &t, uint32_t bit) const {
    return coset_power(t, inv, 1u << bit, kshift);
  }
};

// Power table of tile prefix H: every round below the top one.
template <int K, int B = PowerTable<K>::next(K - 4)>
__device__ __forceinline__ void fill_power_table(uint64_t *pw, const DevTables &tabs, uint32_t inv, uint32_t H,
                                                 const Scale &sc, uint32_t lb, uint32_t first = 0) {
  if constexpr (B >= 0) {
    using T = PowerTable<K>;
    constexpr int V = T::V(B), NP = 1 << V;
    for (uint32_t r = (threadIdx.x + THREADS - first) % THREADS; r < T::rows(B); r += THREADS) {
      uint64_t p[NP];
      p[0] = 1;
      p[1] = twiddle(tabs, inv, (H << (K - B - 1)) + (r << (V - 1)));
      if (sc.on) p[1] = mul(p[1], sc.power(tabs, lb + B));
#pragma unroll
      for (int j = 2; j < NP; j++) p[j] = (j & 1) ? mul(p[j - 1], p[1]) : mul(p[j / 2], p[j / 2]);
      uint64_t *row = pw + T::base(B) + r * (NP + 1);
#pragma unroll
      for (int j = 0; j < NP; j++) row[j] = p[j];
    }
    fill_power_table<K, T::next(B)>(pw, tabs, inv, H, sc, lb, (first + T::rows(B)) % THREADS);
  }
}

// The full round's matrix with input i (DIT) or output o (DIF) scaled by
// kappa sigma^i: 256 entries, one a thread.
template <bool DIF, bool INV>
__device__ __forceinline__ void build_matrix(uint8_t *img, uint64_t sigma, uint64_t kappa) {
  const uint32_t o = threadIdx.x >> 4, i = threadIdx.x & 15;
  const uint64_t m = pow2_mod((uint32_t)entry_exp(DIF, INV, 4, o, i));
  put_entry(img, o, i, gl::mul_canon(m, gl::mul(kappa, gl::pow(sigma, DIF ? o : i))));
}

__device__ __forceinline__ void copy_image(uint8_t *dst, const uint8_t *src) {
#pragma unroll
  for (uint32_t i = 0; i < IMG_BYTES / 16 / THREADS; i++)
    reinterpret_cast<uint4 *>(dst)[threadIdx.x + THREADS * i] = __ldg(reinterpret_cast<const uint4 *>(src) + threadIdx.x + THREADS * i);
}

// log2 of the run of low positions a tile spans: windows above bit 0 take as
// long a run as fills the tile with one column (256 bytes and more of every
// row for K <= 8, and no waste for odd column counts).
__host__ __device__ constexpr int run_log(int K, bool low) { return low ? 0 : TILE_BITS - K; }

// Address of the element at tile index e from that of the tile's element 0.
// For a constant e: an immediate offset when the window starts at bit 0
// (C = 1), else one multiply-add by the window step.
template <int K, int LC, class T>
__device__ __forceinline__ T *elem_at(T *base, uint32_t e, uint64_t stride, uint32_t step_bytes) {
  const uint32_t w = (e >> LC) & ((1u << K) - 1), lc = e & ((1u << LC) - 1);
  if constexpr (K + LC < TILE_BITS) {
    const uint32_t g = e >> (K + LC);
    if (g) base += (uint64_t)g * stride;
  }
  if constexpr (LC == 0) return base + w;
  return reinterpret_cast<T *>(mad_wide(w, step_bytes, reinterpret_cast<uint64_t>(base + lc)));
}

// Store address of a constant part c of a linear tile address with thread part
// a: only the chunk bits can be set in both.
__device__ __forceinline__ uint32_t xor_part(uint32_t a, uint32_t c) { return (a ^ (c & 0x70u)) + (c & ~0x70u); }

// Round I of the execution order to its end: outputs multiplied by powers and
// stored for round I + 1.
template <int K, int LC, bool DIF, int I>
__device__ __forceinline__ void middle_round(Ctx &c, uint8_t *tile, const uint64_t *pw, uint32_t img) {
  multiply(c, smem_u32(tile), img);
  // DIT rounds take powers on their inputs: those of the next round; DIF
  // rounds on their outputs: their own
  using RS = Rounds<K, LC>;
  constexpr int B = RS::make(DIF, DIF ? I : I + 1).B;
  constexpr uint32_t WM = (1u << K) - 1;
  const uint32_t e0 = elem_of_row<K, LC, DIF, I>(threadIdx.x);
  const uint32_t a0 = addr_of<K, LC, DIF, I + 1>(e0);
  const uint64_t *pp = pw + PowerTable<K>::index(B, (e0 >> LC) & WM);
  outputs(c, [&](int o, uint64_t y) {
    const uint32_t eo = elem_of_slot<K, LC, DIF, I>((uint32_t)o);
    const uint32_t po = PowerTable<K>::index(B, (eo >> LC) & WM) - PowerTable<K>::base(B);
    if (!DIF || (o & ((1 << RS::make(DIF, I).V) - 1)) != 0) y = mul(y, pp[po]); // DIF: not the s^0
    *reinterpret_cast<uint64_t *>(tile + xor_part(a0, addr_of<K, LC, DIF, I + 1>(eo))) = y;
  });
}

template <int K, int LC, bool DIF, int I>
__device__ __forceinline__ void middle_rounds(Ctx &c, uint8_t *tile, const uint64_t *pw, uint32_t img_top,
                                              uint32_t img_full, uint32_t img_short) {
  using RS = Rounds<K, LC>;
  if constexpr (I + 1 < RS::N) {
    constexpr Layout q = RS::make(DIF, I);
    middle_round<K, LC, DIF, I>(c, tile, pw, q.V < 4 ? img_short : q.B == K - 4 ? img_top : img_full);
    middle_rounds<K, LC, DIF, I + 1>(c, tile, pw, img_top, img_full, img_short);
  }
}

// One CTA's work: tile position bx, column chunk by (as pass_body, tiles of
// 4096 elements).  store_scale (DIF): n^-1; base^i by p.share.
template <int K, bool LOW, bool B2N, bool INV>
__device__ __forceinline__ void pass_body_tc(const PassParams &p, uint32_t bx, uint32_t by, uint8_t *smem, Ctx &ctx,
                                             bool tables_first) {
  constexpr int LC = run_log(K, LOW), LG = TILE_BITS - K - LC;
  using RS = Rounds<K, LC>;
  constexpr int LAST = RS::N - 1;
  constexpr uint32_t G = 1u << LG;
  uint8_t *tile = smem, *img0 = smem + TILE_BYTES;
  uint64_t *pw = reinterpret_cast<uint64_t *>(img0 + pass_images<K>() * IMG_BYTES);
  const uint32_t img_top = smem_u32(img0), img_full = img_top + IMG_BYTES, img_short = img_full + IMG_BYTES;
  const uint32_t tid = threadIdx.x;
  TileGeom tg;
  tg.H = bx >> (p.lb - LC);
  tg.base_off = ((uint64_t)tg.H << (p.lb + K)) + ((uint64_t)(bx & ((1u << (p.lb - LC)) - 1)) << LC);
  tg.group = by / p.chunks_per_group;
  tg.col_begin = (by - tg.group * p.chunks_per_group) * p.cols_per_cta;
  tg.col_end = min(p.group_cols, tg.col_begin + p.cols_per_cta);
  const uint32_t Hbig = tg.H + (brev_bits(tg.group, p.log_groups) << (p.log_n - p.lb - K));
  const uint64_t *in = p.in + tg.group * p.group_stride_in + tg.base_off;
  uint64_t *out = p.out + tg.group * p.group_stride_out + tg.base_off;

  const uint32_t step_bytes = 8u << p.lb; // one window position
  // the thread's row in the first and the last round
  const uint32_t e_in = elem_of_row<K, LC, B2N, 0>(tid), e_out = elem_of_row<K, LC, B2N, LAST>(tid);
  const uint32_t a_in = addr_of<K, LC, B2N, 0>(e_in);

  // The tile of column group c0, asynchronously (cp.async): a window at bit 0 of
  // a DIF pass as it lies, 16 bytes at a time; else each thread its row's 16
  // words (neighbouring threads take neighbouring addresses).  Issued as soon as
  // the last round's products are done, so it overlaps that round's folding and
  // stores.  Slots of columns past the chunk keep what they hold: rows and
  // diagonal blocks do not mix columns.
  constexpr bool AS_IT_LIES = B2N && LOW;
  // DIT passes at bit 0 without a short round end with a row's 16 consecutive
  // words in each thread.  Stored straight from there, a warp's 16-byte stores
  // would each touch 32 lines (12-bit passes 11 % slower), so these go through
  // the tile, whose next words meanwhile wait in registers.
  constexpr bool STAGED = !B2N && LOW && K % 4 == 0;
  uint64_t x[STAGED ? 16 : 1];
  auto first = [&](uint32_t c0) {
    if constexpr (STAGED) {
      const uint64_t *src = elem_at<K, LC>(in + (uint64_t)c0 * p.stride_in, e_in, p.stride_in, step_bytes);
#pragma unroll
      for (uint32_t s = 0; s < 16; s++) {
        const uint32_t es = elem_of_slot<K, LC, B2N, 0>(s);
        x[s] = c0 + ((e_in | es) >> (K + LC)) < tg.col_end ? __ldcg(elem_at<K, LC>(src, es, p.stride_in, step_bytes)) : 0;
      }
    } else if constexpr (AS_IT_LIES) {
#pragma unroll
      for (uint32_t i = 0; i < 8; i++) {
        const uint32_t e = 2 * (tid + THREADS * i);
        const uint32_t col = c0 + (e >> (K + LC));
        if (col < tg.col_end) {
          const uint64_t *src = elem_at<K, LC>(in + (uint64_t)c0 * p.stride_in, e, p.stride_in, step_bytes);
          uint8_t *dst = tile + addr_of<K, LC, B2N, 0>(e);
          if (p.vec_in) {
            cp_async16(dst, src);
          } else {
            cp_async8(dst, src);
            cp_async8(dst + 8, src + 1);
          }
        }
      }
    } else {
      const uint64_t *src = elem_at<K, LC>(in + (uint64_t)c0 * p.stride_in, e_in, p.stride_in, step_bytes);
#pragma unroll
      for (uint32_t s = 0; s < 16; s++) {
        const uint32_t es = elem_of_slot<K, LC, B2N, 0>(s);
        if (c0 + ((e_in | es) >> (K + LC)) < tg.col_end)
          cp_async8(tile + xor_part(a_in, addr_of<K, LC, B2N, 0>(es)), elem_at<K, LC>(src, es, p.stride_in, step_bytes));
      }
    }
    cp_async_commit();
  };
  // the first column's words: before the tables, whose set-up then hides their
  // latency, or after them when the predecessor may still be running
  if (!tables_first) {
    if (p.overlap) wait_previous();
    first(tg.col_begin);
  }

  {
    uint64_t sigma = Hbig ? twiddle(p.tabs, INV, Hbig << 3) : 1, kappa = 1;
    const Scale sc{p.share != SHARE_NONE, p.share == SHARE_COSET_INV, p.share == SHARE_G ? 0 : p.coset_kshift};
    if (B2N && p.store_scale) kappa = p.tabs.inv_pow2[p.log_n];
    if (sc.on) sigma = mul(sigma, sc.power(p.tabs, K - 4 + p.lb));
    build_matrix<B2N, INV>(img0, sigma, kappa);
    copy_image(img0 + IMG_BYTES, p.tabs.tc_img + img_index(B2N, INV, 4) * IMG_BYTES);
    if constexpr (K % 4 != 0) copy_image(img0 + 2 * IMG_BYTES, p.tabs.tc_img + img_index(B2N, INV, K % 4) * IMG_BYTES);
    fill_power_table<K>(pw, p.tabs, INV, Hbig, sc, p.lb);
  }
  if (tables_first) {
    wait_previous();
    first(tg.col_begin);
  }

#pragma unroll 1
  for (uint32_t c0 = tg.col_begin; c0 < tg.col_end; c0 += G) {
    if constexpr (STAGED) {
#pragma unroll
      for (uint32_t s = 0; s < 16; s += 2)
        *reinterpret_cast<ulonglong2 *>(tile + xor_part(a_in, addr_of<K, LC, B2N, 0>(elem_of_slot<K, LC, B2N, 0>(s)))) =
            make_ulonglong2(x[s], x[s + 1]);
    } else {
      cp_async_wait<0>();
    }
    middle_rounds<K, LC, B2N, 0>(ctx, tile, pw, img_top, img_full, img_short);
    constexpr Layout ql = RS::make(B2N, LAST);
    multiply(ctx, smem_u32(tile), ql.V < 4 ? img_short : ql.B == K - 4 ? img_top : img_full);
    const bool more = c0 + G < tg.col_end;
    if constexpr (STAGED) {
      const uint32_t a_out = addr_of<K, LC, B2N, LAST>(e_out);
      uint64_t even = 0;
      outputs(ctx, [&](int o, uint64_t y) {
        if (p.canon_out) y = gl::canon(y);
        const uint32_t ee = elem_of_slot<K, LC, B2N, LAST>((uint32_t)o & ~1u);
        if (o & 1)
          *reinterpret_cast<ulonglong2 *>(tile + xor_part(a_out, addr_of<K, LC, B2N, LAST>(ee))) = make_ulonglong2(even, y);
        else
          even = y;
      });
      if (more) first(c0 + G);
      __syncthreads();
#pragma unroll
      for (uint32_t i = 0; i < 8; i++) {
        const uint32_t e = 2 * (tid + THREADS * i);
        if (c0 + (e >> (K + LC)) >= tg.col_end) continue;
        const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(tile + addr_of<K, LC, B2N, LAST>(e));
        uint64_t *d = elem_at<K, LC>(out + (uint64_t)c0 * p.stride_out, e, p.stride_out, step_bytes);
        if (p.vec_out) {
          *reinterpret_cast<ulonglong2 *>(d) = v;
        } else {
          d[0] = v.x;
          d[1] = v.y;
        }
      }
      __syncthreads(); // the tile is free
      continue;
    }
    if (more) first(c0 + G); // the operands have been read: the tile is free
    // straight from registers: neighbouring threads write neighbouring addresses,
    // or (DIT, bit 0, short last round) a thread its row's runs of 2^V words, 16
    // bytes at a time (10-bit passes: 10 % faster than through the tile), the
    // threads' runs one after the other
    static_assert(rows_ascend(RS::make(B2N, LAST)), "neighbouring threads store to neighbouring addresses");
    uint64_t *dst = elem_at<K, LC>(out + (uint64_t)c0 * p.stride_out, e_out, p.stride_out, step_bytes);
    uint64_t even = 0;
    outputs(ctx, [&](int o, uint64_t y) {
      if (p.canon_out) y = gl::canon(y);
      const uint32_t eo = elem_of_slot<K, LC, B2N, LAST>((uint32_t)o);
      if constexpr (!B2N && LOW) {
        if (!(o & 1)) {
          even = y;
          return;
        }
        const uint32_t ee = elem_of_slot<K, LC, B2N, LAST>((uint32_t)o - 1);
        if (c0 + ((e_out | ee) >> (K + LC)) >= tg.col_end) return;
        uint64_t *d = elem_at<K, LC>(dst, ee, p.stride_out, step_bytes);
        if (p.vec_out) {
          __stcg(reinterpret_cast<ulonglong2 *>(d), make_ulonglong2(even, y));
        } else {
          __stcg(d, even);
          __stcg(d + 1, y);
        }
      } else {
        if (c0 + ((e_out | eo) >> (K + LC)) < tg.col_end) __stcg(elem_at<K, LC>(dst, eo, p.stride_out, step_bytes), y);
      }
    });
  }
  cp_async_wait<0>();
}

// LOW: the window starts at bit 0.
template <int K, bool LOW, bool B2N, bool INV> __global__ void __launch_bounds__(THREADS, 2) pass_kernel_tc(const PassParams p) {
  extern __shared__ __align__(1024) uint8_t tc_smem[];
  uint8_t *smem = tc_smem + ((1024 - (smem_u32(tc_smem) & 1023)) & 1023);
  uint64_t *slot = reinterpret_cast<uint64_t *>(smem + TILE_BYTES + pass_images<K>() * IMG_BYTES) + ((PowerTable<K>::words + 1) & ~1u);
  Ctx ctx = begin(slot, p.tabs.wait_tries);
  allow_next(); // with its tensor memory in hand: no CTA of this launch can wait for one of the next
  pass_body_tc<K, LOW, B2N, INV>(p, blockIdx.x, blockIdx.y, smem, ctx, in_first_wave(p.overlap));
  end(ctx, p.tabs.wait_error);
}

} // namespace tc
} // namespace bc
