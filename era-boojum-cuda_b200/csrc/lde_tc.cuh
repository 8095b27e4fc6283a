// lde_tc.cuh -- the fused LDE's top-window kernel on the tensor cores.
//
// Same step as lde_top_kernel (lde.cuh): the inverse transform's rounds on the
// top window, then for every coset the forward ones, each coset stored once.
// The window is cut into equal rounds, of 4 bits (matrices of tc.cuh) or, WIDE,
// of 5: then one M = 128, N = K = 256 product per tile with a 64 KB matrix, and
// two threads share a row (outputs 0..15 and 16..31, by thread bit 7; the
// accumulator columns a thread reads are the same as for 4-bit rounds).  A
// 10-bit window takes two wide rounds instead of three, i.e. two digit folds
// and one multiplication by powers per element and direction.
//
// One matrix for both directions.  The inverse round is y_t = sum_u x_u
// w^(-t brev(u)); with the forward matrix w^(i brev(o)) that is word i =
// brev(u) and output o with brev(o) = -t: the inverse layouts number their
// words by reversed bits, and outputs are relabelled at compile time.
//
// Scaling n^-1 g^i costs nothing here: the passes below have multiplied by n^-1
// and the share of the low bits (SHARE_G), the inverse rounds'
// powers carry the share of their output fields (tc::Scale), and the top
// field's share goes with the coset factors.  Coset k's forward rounds have
// the twiddle prefix H = brev(k): the top round's sigma_H^j is multiplied into
// its matrix (4-bit rounds: precomputed per H) or into the coefficients (WIDE:
// a 64 KB matrix per coset does not fit), the other round has a power table per H.
#pragma once
#include "lde.cuh"
#include "ntt_tc.cuh"

namespace bc {
namespace tc {

// Device tables of this kernel, behind the images (DevTables::tc_img).
constexpr uint32_t TOP_PREFIXES = 16; // H < 16: blowups up to 16
constexpr uint32_t WIDE_IMG_BYTES = 65536;
constexpr uint32_t COSET_IMG_OFF = IMAGES * IMG_BYTES;                    // [H]: full round, input i times T[8 H]^i
constexpr uint32_t WIDE_IMG_OFF = COSET_IMG_OFF + TOP_PREFIXES * IMG_BYTES;
constexpr uint32_t WIDE_PW_OFF = WIDE_IMG_OFF + WIDE_IMG_BYTES;           // [H][R][j]: T[(H << 9) + (R << 4)]^j
constexpr uint32_t PW8_OFF = WIDE_PW_OFF + TOP_PREFIXES * 1024 * 8;       // [H]: PowerTable<8>
constexpr uint32_t TOP_TABLE_END = PW8_OFF + TOP_PREFIXES * PowerTable<8>::words * 8;

struct TopLayout {
  int B;      // lowest window bit of the round
  int reg[4]; // tile index bits of a thread's 16 words
  int row[8]; // tile index bits of the thread bits (WIDE: row[7] is the fifth word bit)
  int out7;   // tile index bit that thread bit 7 is in the outputs
};

constexpr __host__ __device__ uint32_t brev4(uint32_t v) {
  return (v & 1) << 3 | (v & 2) << 1 | (v & 4) >> 1 | (v & 8) >> 3;
}

// Rounds 0 .. N - 1 are the inverse's (bottom-up), N .. 2 N - 1 a coset's (top-down).
template <int K, int LC, bool WIDE> struct TopRounds {
  static constexpr int LR = WIDE ? 5 : 4, N = K / LR;
  static_assert(N * LR == K, "the window is cut into equal rounds");
  static constexpr __host__ __device__ int bank(const TopLayout &q, int b) {
    int m = 0;
    for (int t = 0; t < 4; t++)
      if (q.reg[t] == b) m ^= 1 << t;
    for (int t = 0; t < 3; t++)
      if (q.row[t] == b) m ^= 2 << t;
    return m;
  }
  static constexpr __host__ __device__ TopLayout make(int i) {
    TopLayout q{};
    const bool inv = i < N;
    q.B = inv ? i * LR : K - LR * (i - N + 1);
    const int lo = LC + q.B;
    for (int t = 0; t < 4; t++) q.reg[t] = inv ? lo + LR - 1 - t : lo + t;
    int rest[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    int n = 0;
    for (int b = 0; b < TILE_BITS; b++)
      if (b < lo || b >= lo + LR) rest[n++] = b;
    for (int t = 0; t < n; t++) q.row[t] = rest[t];
    if (i + 1 < 2 * N) {
      const TopLayout nx = make(i + 1);
      if (i == N - 1) { // same field, same rows: a thread stores its own row
        for (int t = 0; t < n; t++) q.row[t] = nx.row[t];
      } else {
        bool found = false;
        for (int m = 0; m < (1 << n) && !found; m++) {
          int pick[4] = {0, 0, 0, 0}, cnt = 0;
          for (int t = 0; t < n; t++)
            if (m >> t & 1) {
              if (cnt < 4) pick[cnt] = rest[t];
              cnt++;
            }
          if (cnt != 4 || !spans16(bank(nx, pick[0]), bank(nx, pick[1]), bank(nx, pick[2]), bank(nx, pick[3]))) continue;
          found = true;
          int o = 4;
          for (int t = 0; t < 4; t++) q.row[t] = pick[t];
          for (int t = 0; t < n; t++)
            if (rest[t] != pick[0] && rest[t] != pick[1] && rest[t] != pick[2] && rest[t] != pick[3])
              q.row[o++] = rest[t];
        }
      }
    }
    if (WIDE) q.row[7] = inv ? lo : lo + 4;
    q.out7 = WIDE ? lo + 4 : q.row[7];
    return q;
  }
};

// Tile index of thread t's word 0 (as operand rows / as outputs), of word s,
// and tile address (linear over XOR, as addr_of).
template <int K, int LC, bool WIDE, int I> __host__ __device__ constexpr uint32_t top_in_elem(uint32_t t) {
  constexpr TopLayout q = TopRounds<K, LC, WIDE>::make(I);
  uint32_t e = 0;
#pragma unroll
  for (int b = 0; b < 8; b++) e |= (t >> b & 1u) << q.row[b];
  return e;
}
template <int K, int LC, bool WIDE, int I> __host__ __device__ constexpr uint32_t top_out_elem(uint32_t t) {
  constexpr TopLayout q = TopRounds<K, LC, WIDE>::make(I);
  uint32_t e = 0;
#pragma unroll
  for (int b = 0; b < 7; b++) e |= (t >> b & 1u) << q.row[b];
  return e | (t >> 7 & 1u) << q.out7;
}
template <int K, int LC, bool WIDE, int I> __host__ __device__ constexpr uint32_t top_word_elem(uint32_t s) {
  constexpr TopLayout q = TopRounds<K, LC, WIDE>::make(I);
  uint32_t e = 0;
#pragma unroll
  for (int b = 0; b < 4; b++) e |= (s >> b & 1u) << q.reg[b];
  return e;
}
template <int K, int LC, bool WIDE, int I> __host__ __device__ constexpr uint32_t top_addr(uint32_t e) {
  constexpr TopLayout q = TopRounds<K, LC, WIDE>::make(I);
  uint32_t r = 0, s = 0;
#pragma unroll
  for (int b = 0; b < 8; b++) r |= (e >> q.row[b] & 1u) << b;
#pragma unroll
  for (int b = 0; b < 4; b++) s |= (e >> q.reg[b] & 1u) << b;
  return r << 7 | ((s >> 1) ^ (r & 7u)) << 4 | (s & 1u) << 3;
}

// Field value of a thread's v-th output.  Forward: v.  Inverse, 4 bits:
// accumulator v is t = -brev4(v).  Inverse, WIDE: the thread of half h takes
// accumulators h + 2 v, whose brev5 is 16 h + brev4(v): t = -(16 h + brev4(v))
// mod 32, i.e. low bits -brev4(v), and bit 4 = h for v = 0, 1 - h otherwise;
// the bit is left to the caller (flips).
__host__ __device__ constexpr uint32_t inv_field(uint32_t v) { return (16u - brev4(v)) & 15u; }
__host__ __device__ constexpr bool flips(uint32_t v) { return v != 0; }

// The wide product: K = 256 bytes in two panels of 128, N = 256.
constexpr uint32_t MMA_DESC_WIDE = (2u << 4) | ((256u >> 3) << 17) | ((128u >> 4) << 24);
template <bool WIDE> __device__ __forceinline__ void top_multiply(Ctx &c, uint32_t tile, uint32_t img) {
  if constexpr (!WIDE) {
    multiply(c, tile, img);
  } else {
    products(c, [&] {
#pragma unroll
      for (uint32_t k = 0; k < 8; k++) {
        const uint64_t a = operand_desc(tile + (k >> 2) * (TILE_BYTES / 2)) + 2 * (k & 3);
        const uint64_t b = operand_desc(img + (k >> 2) * (WIDE_IMG_BYTES / 2)) + 2 * (k & 3);
        asm volatile("{\n\t"
                     ".reg .pred acc;\n\t"
                     "setp.ne.u32 acc, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, acc;\n\t"
                     "}" ::"r"(c.tmem),
                     "l"(a), "l"(b), "r"(MMA_DESC_WIDE), "r"(k)
                     : "memory");
      }
    });
  }
}

// use(v, y) for the thread's outputs of an inverse round.
template <bool WIDE, class F> __device__ __forceinline__ void inverse_outputs(const Ctx &c, F &&use) {
  if constexpr (!WIDE) {
    outputs(c, use);
  } else {
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t a = c.tmem + ((warp & 3) << 21) + (warp >> 2) * 8;
#pragma unroll
    for (uint32_t g = 0; g < 4; g++) {
      uint32_t d[32];
      ld_digits8x4(d, a + 64 * g); // accumulators 8 g + h + {0, 2, 4, 6}
      wait_ld(d);
#pragma unroll
      for (int o = 0; o < 4; o++) use((int)(4 * g) + o, fold_digits(d + 8 * o));
    }
  }
}

// Shared memory: tile, matrices (4 bits: full round, inverse top round, two
// coset slots; WIDE: the one), power tables, barrier.
template <int K, bool WIDE> __host__ __device__ constexpr uint32_t top_tc_images() {
  return WIDE ? WIDE_IMG_BYTES : 4 * IMG_BYTES;
}
template <int K, bool WIDE> __host__ __device__ constexpr uint32_t top_tc_pw_words() {
  // WIDE: inverse table (rows of 33), coset powers (16 x 32); 4 bits: inverse, two coset slots
  return WIDE ? (K > 5 ? 32 * 33 : 0) + TOP_PREFIXES * 32 : 3 * PowerTable<K>::words;
}
template <int K, bool WIDE> __host__ __device__ constexpr uint32_t top_tc_smem_bytes() {
  return 1024 + TILE_BYTES + top_tc_images<K, WIDE>() + top_tc_pw_words<K, WIDE>() * 8 + 32;
}

template <int K, bool WIDE>
__device__ __forceinline__ void top_body_tc(const LdeTopParams &p, uint32_t bx, uint32_t by, uint8_t *smem, Ctx &ctx,
                                            bool tables_first) {
  constexpr int LC = run_log(K, false);
  using TR = TopRounds<K, LC, WIDE>;
  constexpr int N = TR::N, LR = TR::LR;
  static_assert(N <= 2, "one or two rounds");
  uint8_t *tile = smem, *img0 = smem + TILE_BYTES;
  uint64_t *pw = reinterpret_cast<uint64_t *>(img0 + top_tc_images<K, WIDE>());
  const uint32_t t_tile = smem_u32(tile), t_full = smem_u32(img0);
  const uint32_t tid = threadIdx.x, half = tid >> 7;
  const uint64_t base_off = (uint64_t)bx << LC;
  const uint32_t col_begin = by * p.cols_per_cta, col_end = min(p.num_cols, col_begin + p.cols_per_cta);
  const uint32_t nb = 1u << p.log_blowup, step_bytes = 8u << p.lb;
  const uint8_t *gt = p.tabs.tc_img;

  // operand words of the first round: each thread its row's 16, asynchronously
  const uint32_t e_in = top_in_elem<K, LC, WIDE, 0>(tid), a_in = top_addr<K, LC, WIDE, 0>(e_in);
  auto load = [&](uint32_t c0) {
    const uint64_t *src = elem_at<K, LC>(p.in + (uint64_t)c0 * p.stride_in + base_off, e_in, p.stride_in, step_bytes);
#pragma unroll
    for (uint32_t s = 0; s < 16; s++) {
      const uint32_t es = top_word_elem<K, LC, WIDE, 0>(s);
      cp_async8(tile + xor_part(a_in, top_addr<K, LC, WIDE, 0>(es)), elem_at<K, LC>(src, es, p.stride_in, step_bytes));
    }
    cp_async_commit();
  };

  if (!tables_first) {
    if (p.overlap) wait_previous();
    load(col_begin);
  }

  // the coset's matrix and power table, one coset ahead (4-bit rounds)
  auto fetch_coset = [&](uint32_t k, uint32_t slot) {
    const uint32_t H = brev_bits(k, p.log_blowup);
    uint8_t *dst = img0 + (2 + slot) * IMG_BYTES;
    const uint8_t *src = gt + COSET_IMG_OFF + H * IMG_BYTES;
#pragma unroll
    for (uint32_t i = 0; i < IMG_BYTES / 16 / THREADS; i++) cp_async16(dst + 16 * (tid + THREADS * i), src + 16 * (tid + THREADS * i));
    if constexpr (N == 2) {
      const uint8_t *ps = gt + PW8_OFF + H * PowerTable<K>::words * 8;
      uint8_t *pd = reinterpret_cast<uint8_t *>(pw + (1 + slot) * PowerTable<K>::words);
      if (tid < PowerTable<K>::words / 2) cp_async16(pd + 16 * tid, ps + 16 * tid);
    }
    cp_async_commit();
  };
  uint64_t *const coset_pw = pw + (N == 2 ? 32 * 33 : 0); // WIDE: [k][j]: (sigma_H G)^j
  if constexpr (WIDE) {
    for (uint32_t i = tid; i < WIDE_IMG_BYTES / 16; i += THREADS) cp_async16(img0 + 16 * i, gt + WIDE_IMG_OFF + 16 * i);
    cp_async_commit();
    // inverse table: R (32) x j (32), T_inv[R << 4]^j times the field's share of g^i
    if constexpr (N == 2) {
      const uint64_t share = g_power(p.tabs, 0, 1u << p.lb);
      const uint32_t R = tid >> 3, j0 = (tid & 7) * 4;
      const uint64_t s = mul(twiddle(p.tabs, 1, R << 4), share);
      uint64_t q = gl::pow(s, j0);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        pw[R * 33 + j0 + j] = q;
        q = mul(q, s);
      }
    }
    const uint64_t G5 = g_power(p.tabs, 0, 1u << (p.lb + K - 5));
    for (uint32_t i = tid; i < nb * 32; i += THREADS) {
      const uint32_t H = brev_bits(i >> 5, p.log_blowup);
      const uint64_t s = H ? mul(twiddle(p.tabs, 0, H << 4), G5) : G5;
      coset_pw[i] = gl::pow(s, i & 31);
    }
  } else {
    fetch_coset(0, 0);
    copy_image(img0, gt + img_index(false, false, 4) * IMG_BYTES);
    { // inverse top round: output t times the field's share of g^i
      const uint32_t o = tid >> 4, i = tid & 15;
      const uint64_t share = g_power(p.tabs, 0, 1u << (p.lb + K - 4));
      const uint64_t m = pow2_mod((uint32_t)entry_exp(false, false, 4, o, i));
      put_entry(img0 + IMG_BYTES, o, i, gl::mul_canon(m, gl::pow(share, inv_field(o))));
    }
    if constexpr (N == 2) fill_power_table<K>(pw, p.tabs, 1, 0, Scale{true, 0, 0}, p.lb);
  }
  if (tables_first) {
    wait_previous();
    load(col_begin);
  }
  uint32_t step = 0; // coset slots used so far

#pragma unroll 1
  for (uint32_t c0 = col_begin; c0 < col_end; c0++) {
    const bool more = c0 + 1 < col_end;
    cp_async_wait<0>();
    if constexpr (N == 2) { // inverse, bottom round
      top_multiply<WIDE>(ctx, t_tile, t_full);
      constexpr int FB = LC; // tile index bit of the field
      const uint32_t e0 = top_out_elem<K, LC, WIDE, 0>(tid);
      const uint32_t R = (e0 >> (LC + LR)) & ((1u << LR) - 1);
      const uint32_t ef = WIDE ? e0 ^ (16u << FB) : e0; // the flipped half
      const uint32_t a0 = top_addr<K, LC, WIDE, 1>(e0), af = top_addr<K, LC, WIDE, 1>(ef);
      const uint64_t *p0 = pw + (WIDE ? R * 33 + 16 * half : R * 17), *pf = WIDE ? pw + R * 33 + 16 * (half ^ 1) : p0;
      inverse_outputs<WIDE>(ctx, [&](int v, uint64_t y) {
        const uint32_t f = inv_field((uint32_t)v);
        if (WIDE || f != 0) y = mul(y, (flips((uint32_t)v) ? pf : p0)[f]);
        *reinterpret_cast<uint64_t *>(tile + xor_part(flips((uint32_t)v) ? af : a0, top_addr<K, LC, WIDE, 1>(f << FB))) = y;
      });
    }
    // inverse, top round: the coefficients (4 bits: scaled by the matrix; WIDE: with the coset factors)
    uint64_t coef[16]; // by field value (WIDE: its low 4 bits)
    top_multiply<WIDE>(ctx, t_tile, WIDE ? t_full : t_full + IMG_BYTES);
    inverse_outputs<WIDE>(ctx, [&](int v, uint64_t y) { coef[inv_field((uint32_t)v)] = y; });
    // forward: the thread's own row; coefficient 0 in its half, the others in the other one (WIDE)
    const uint32_t e1 = top_out_elem<K, LC, WIDE, N - 1>(tid);
    const uint32_t h0 = top_addr<K, LC, WIDE, N>(e1);
    const uint32_t hf = WIDE ? top_addr<K, LC, WIDE, N>(e1 ^ (16u << (LC + K - LR))) : h0;

#pragma unroll 1
    for (uint32_t k = 0; k < nb; k++) {
      const uint32_t slot = step & 1;
      if constexpr (WIDE) {
        const uint64_t *c0p = coset_pw + k * 32 + 16 * half, *cfp = coset_pw + k * 32 + 16 * (half ^ 1);
        *reinterpret_cast<uint64_t *>(tile + h0) = mul(coef[0], c0p[0]);
        *reinterpret_cast<uint64_t *>(tile + xor_part(hf, top_addr<K, LC, WIDE, N>(top_word_elem<K, LC, WIDE, N>(1)))) =
            mul(coef[1], cfp[1]);
#pragma unroll
        for (int s = 2; s < 16; s += 2)
          *reinterpret_cast<ulonglong2 *>(tile + xor_part(hf, top_addr<K, LC, WIDE, N>(top_word_elem<K, LC, WIDE, N>(s)))) =
              make_ulonglong2(mul(coef[s], cfp[s]), mul(coef[s + 1], cfp[s + 1]));
      } else {
#pragma unroll
        for (int s = 0; s < 16; s += 2)
          *reinterpret_cast<ulonglong2 *>(tile + xor_part(h0, top_addr<K, LC, WIDE, N>(top_word_elem<K, LC, WIDE, N>(s)))) =
              make_ulonglong2(coef[s], coef[s + 1]);
        cp_async_wait<0>(); // this coset's matrix and powers
        const uint32_t kn = k + 1 == nb ? 0 : k + 1;
        if (kn || more) fetch_coset(kn, slot ^ 1);
      }
      step++;
      top_multiply<WIDE>(ctx, t_tile, WIDE ? t_full : t_full + (2 + slot) * IMG_BYTES);
      if constexpr (N == 2) { // top round to bottom round
        constexpr int FB = LC + K - LR;
        const uint32_t e0 = top_out_elem<K, LC, WIDE, N>(tid);
        const uint32_t a0 = top_addr<K, LC, WIDE, N + 1>(e0);
        const uint32_t j = (e0 >> LC) & ((1u << LR) - 1);
        const uint64_t *pp = WIDE ? reinterpret_cast<const uint64_t *>(gt + WIDE_PW_OFF) +
                                        brev_bits(k, p.log_blowup) * 1024 + half * 512 + j
                                  : pw + (1 + slot) * PowerTable<K>::words +
                                        PowerTable<K>::index(0, (e0 >> LC) & ((1u << K) - 1));
        outputs(ctx, [&](int v, uint64_t y) {
          y = mul(y, WIDE ? __ldg(pp + 32 * v) : pp[17 * v]);
          *reinterpret_cast<uint64_t *>(tile + xor_part(a0, top_addr<K, LC, WIDE, N + 1>((uint32_t)v << FB))) = y;
        });
        top_multiply<WIDE>(ctx, t_tile, t_full);
      }
      if (more && k + 1 == nb) load(c0 + 1); // the tile is free
      const uint32_t eo = top_out_elem<K, LC, WIDE, 2 * N - 1>(tid);
      uint64_t *dst = elem_at<K, LC>(p.out + (uint64_t)k * p.coset_stride + (uint64_t)c0 * p.stride_out + base_off, eo,
                                     p.stride_out, step_bytes);
      outputs(ctx, [&](int v, uint64_t y) {
        __stcg(elem_at<K, LC>(dst, (uint32_t)v << LC, p.stride_out, step_bytes), y);
      });
    }
  }
  cp_async_wait<0>();
}

template <int K, bool WIDE> __global__ void __launch_bounds__(THREADS, 2) top_kernel_tc(const LdeTopParams p) {
  extern __shared__ __align__(1024) uint8_t tc_smem[];
  uint8_t *smem = tc_smem + ((1024 - (smem_u32(tc_smem) & 1023)) & 1023);
  uint64_t *slot = reinterpret_cast<uint64_t *>(smem + TILE_BYTES + top_tc_images<K, WIDE>()) +
                   ((top_tc_pw_words<K, WIDE>() + 1) & ~1u);
  Ctx ctx = begin(slot, p.tabs.wait_tries);
  allow_next(); // with its tensor memory in hand: no CTA of this launch can wait for one of the next
  top_body_tc<K, WIDE>(p, blockIdx.x, blockIdx.y, smem, ctx, in_first_wave(p.overlap));
  end(ctx, p.tabs.wait_error);
}

} // namespace tc
} // namespace bc
