// tc.cuh -- radix-16 rounds on the tensor cores (tcgen05, 8-bit integers).
//
// A round multiplies groups of 16 field elements by one constant 16 x 16
// matrix M.  Over the bytes of the operands that is an integer contraction:
// with x_i = sum_b x_{i,b} 2^(8b) (any u64 word, its bytes as they lie in
// memory) and M[o][i] 2^(8b) mod p = sum_j m_{o,j,i,b} 2^(8j),
//     y_o = sum_j 2^(8j) D_{o,j},   D_{o,j} = sum_{i,b} m_{o,j,i,b} x_{i,b},
// i.e. D = A B^T with A one 128-byte row per group (16 words), B the 128 x 128
// byte matrix m, and 32-bit sums D < 128 * 255^2 < 2^23: exact.  tcgen05.mma
// kind::i8 computes 128 groups x 128 digits at once (M = N = K = 128) from
// shared memory into tensor memory; a thread then reads the 8 digits of each
// of its group's 16 outputs back (tcgen05.ld, lane = group) and folds them
// into a u64 (fold_digits).
//
// Why: the pass kernels are bound by 32-bit integer issue.  A radix-16 network
// of shift butterflies is 42 instructions per element; folding eight digits is
// 15, and the tensor pipe, idle otherwise, does the sums (8180 multiply-adds
// per clock and SM measured for M = 128, N = 128, K = 32 instructions, 64
// cycles each).  Measured on B200, register-resident rounds: 850 G butterflies/s
// with the multiplications by powers (the butterfly network: 820) and 1560
// where a round needs none, which is why the kernels put as many powers as they
// can into the matrices.
//
// Layout of a tile (4096 elements, 12 index bits): 256 rows of 16 words in the
// K-major 128-byte-swizzle layout that the MMA's shared-memory descriptors
// name: word s of row r at byte 128 r + 16 ((s >> 1) ^ (r & 7)) + 8 (s & 1).
// Row and word number are bit fields of the element's tile index, chosen per
// round (Layout), so a round's outputs are stored straight where the next
// round's A operand needs them: one 8-byte store per element and round, no
// loads.
#pragma once
#include <cstdint>

#include "gl.cuh"
#include "tables.cuh"

namespace bc {
namespace tc {

constexpr int TILE_BITS = 12;
constexpr uint32_t TILE = 1u << TILE_BITS;      // elements
constexpr uint32_t TILE_BYTES = TILE * 8;       // two M = 128 operands
constexpr uint32_t THREADS = TILE / 16;         // one row a thread
constexpr uint32_t IMG_BYTES = 16384;           // one B matrix, 128 x 128 bytes
constexpr uint32_t TMEM_COLS = 256;             // accumulators: 2 x (128 lanes x 128 columns)
// Bound of a completion wait, in tries: one suspends the thread for about 4 us
// when nothing arrives (measured on B200, with or without a time hint), so 4 s.
constexpr uint32_t WAIT_TRIES = 1u << 20;

// ---------------------------------------------------------------- instructions
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Programmatic dependent launch: the kernels of one call overlap each other's
// prologue (tables, matrices).  allow_next once the CTA has its tensor memory
// (the next kernel's CTAs hold theirs while they wait); a kernel touches what its
// predecessor wrote (or reads) only after wait_previous, which returns when the
// predecessor has completed and its stores are visible.
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Shared-memory operand descriptor: K-major, 128-byte swizzle, groups of 8
// rows 1024 bytes apart.  K advances by 32 bytes = 2 units of the address field.
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3ffffu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)2 << 61;
}

// Instruction descriptor: u8 x u8 -> s32, M = 128, N = 128, both K-major.
constexpr uint32_t MMA_DESC = (2u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

// D[tmem] = A B^T over K = 128 bytes: four K = 32 instructions.  One thread.
__device__ __forceinline__ void mma_128x128(uint32_t d, uint64_t a, uint64_t b) {
#pragma unroll
  for (uint32_t k = 0; k < 4; k++)
    asm volatile("{\n\t"
                 ".reg .pred acc;\n\t"
                 "setp.ne.u32 acc, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, acc;\n\t"
                 "}" ::"r"(d),
                 "l"(a + 2 * k), "l"(b + 2 * k), "r"(MMA_DESC), "r"(k)
                 : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_smem_to_mma() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 32 accumulator columns of the warp's 32 lanes (completed by wait_ld).
__device__ __forceinline__ void ld_digits32(uint32_t (&r)[32], uint32_t addr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
               "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,"
               "%27,%28,%29,%30,%31}, [%32];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                 "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
                 "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
                 "=r"(r[30]), "=r"(r[31])
               : "r"(addr));
}

// Four runs of 8 accumulator columns, 16 apart.
__device__ __forceinline__ void ld_digits8x4(uint32_t (&r)[32], uint32_t addr) {
#pragma unroll
  for (int i = 0; i < 4; i++)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[8 * i]), "=r"(r[8 * i + 1]), "=r"(r[8 * i + 2]), "=r"(r[8 * i + 3]), "=r"(r[8 * i + 4]),
                   "=r"(r[8 * i + 5]), "=r"(r[8 * i + 6]), "=r"(r[8 * i + 7])
                 : "r"(addr + 16 * i));
}

// Completes the reads of r (and any before); r as operands so that no use of
// them moves above it.
__device__ __forceinline__ void wait_ld(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]),
                 "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]),
                 "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]),
                 "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]),
                 "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               ::"memory");
}

// Waits for the completion of phase `parity`; false when the tries ran out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t tries) {
  for (uint32_t i = 0; i < tries; i++) {
    uint32_t ok;
    asm volatile("{\n\t"
                 ".reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t"
                 "}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    if (ok) return true;
  }
  return false;
}

// ---------------------------------------------------------------- field pieces
__device__ __forceinline__ uint64_t mad_wide(uint32_t a, uint32_t b, uint64_t c) {
  uint64_t r;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}

// sum_j d[j] 2^(8j) (mod p) as a u64, for d[j] <= 256 * 255^2 < 2^24 (32 words
// a row; 16 give half of that).  Pairs first: p = d + 2^8 d' < 2^32; L = p0 +
// 2^16 p1 and H = p2 + 2^16 p3 < 2^49.  With
// H = h0 + h1 2^32: L + h0 2^32 + h1 2^64 = (L + h1 EPS) + h0 2^32, where
// L + h1 EPS < 2^50, so one carry can leave the top word and the fold of its
// EPS cannot carry again (the top word wrapped to less than 2^18).
__device__ __forceinline__ uint64_t fold_digits(const uint32_t *d) {
  const uint32_t p0 = d[0] + (d[1] << 8), p1 = d[2] + (d[3] << 8), p2 = d[4] + (d[5] << 8), p3 = d[6] + (d[7] << 8);
  const uint64_t l = mad_wide(p1, 65536u, p0), h = mad_wide(p3, 65536u, p2);
  const uint64_t t = mad_wide(gl::hi32(h), 0xffffffffu, l);
  uint64_t r;
  asm("{\n\t"
      ".reg .u32 t0, t1, c;\n\t"
      ".reg .u64 t;\n\t"
      "mov.b64 {t0, t1}, %1;\n\t"
      "add.cc.u32 t1, t1, %2;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "mov.b64 t, {t0, t1};\n\t"
      "mad.wide.u32 %0, c, 0xffffffff, t;\n\t"
      "}"
      : "=l"(r)
      : "l"(t), "r"(gl::lo32(h)));
  return r;
}

// a * b (mod p) as a u64: the 128-bit product r0..r3, then
// r0 + r1 2^32 + r2 EPS - r3.  z = r0 + r2 EPS < 2^64; adding r1 to its top
// word and subtracting r3 leave k in {-1, 0, 1} times 2^64 = EPS (k = 1: the
// rest is at most 2^64 - 2^33 + 1; k = -1: it is at least 2^64 - 2^32), so
// k (2^32 - 1) goes in without a further carry.  36.4 cycles a warp and
// sub-partition in a register loop, gl::mul_chain 40.0, gl::mul 44.5 (B200).
__device__ __forceinline__ uint64_t mul(uint64_t a, uint64_t b) {
  const unsigned __int128 q = (unsigned __int128)a * b;
  const uint64_t lo = (uint64_t)q, hi = (uint64_t)(q >> 64);
  const uint64_t z = mad_wide(gl::lo32(hi), 0xffffffffu, (uint64_t)gl::lo32(lo));
  uint64_t r;
  asm("{\n\t"
      ".reg .u32 z0, z1, c, k;\n\t"
      ".reg .u64 t;\n\t"
      "mov.b64 {z0, z1}, %1;\n\t"
      "add.cc.u32 z1, z1, %2;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "sub.cc.u32 z0, z0, %3;\n\t"
      "subc.cc.u32 z1, z1, 0;\n\t"
      "subc.u32 k, c, 0;\n\t"
      "add.u32 z1, z1, k;\n\t"
      "mov.b64 t, {z0, z1};\n\t"
      "mad.wide.s32 %0, k, -1, t;\n\t"
      "}"
      : "=l"(r)
      : "l"(z), "r"(gl::hi32(lo)), "r"(gl::hi32(hi)));
  return r;
}

// ---------------------------------------------------------------- layouts
// The rounds of a window of K bits over runs of 2^LC low positions, in
// execution order (DIT: from the top, the short round of K mod 4 bits last;
// DIF: the reverse).  The tile index is [columns | window | low positions].
// A round's 16 words are four bits of it: slot[0..V) its own bits, the others
// (short rounds) passed through; row[] holds the remaining eight, a row number's
// bit i being tile index bit row[i]; thread t works on row t.
struct Layout {
  int V;       // stages of the round
  int B;       // window bit it starts at
  int slot[4]; // tile index bits of the word number
  int row[8];  // tile index bits of the row number
};

__host__ __device__ constexpr bool in4(const int *s, int b) { return s[0] == b || s[1] == b || s[2] == b || s[3] == b; }

// Bank group (4 bits: half of a 16-byte chunk, and which chunk) that tile
// index bit b moves in layout q: word bit 0 is the half, word bits 1..3 and row
// bits 0..2 both select the chunk.
__host__ __device__ constexpr int bank_of(const Layout &q, int b) {
  int m = 0;
  for (int t = 0; t < 4; t++)
    if (q.slot[t] == b) m ^= 1 << t;
  for (int t = 0; t < 3; t++)
    if (q.row[t] == b) m ^= 2 << t;
  return m;
}

__host__ __device__ constexpr bool spans16(int a, int b, int c, int d) {
  int seen = 0;
  for (int i = 0; i < 16; i++) {
    const int v = (i & 1 ? a : 0) ^ (i & 2 ? b : 0) ^ (i & 4 ? c : 0) ^ (i & 8 ? d : 0);
    seen |= 1 << v;
  }
  return seen == 0xffff;
}

// Whether the rows of a layout count its other tile index bits upwards, so that
// neighbouring threads hold neighbouring elements.
__host__ __device__ constexpr bool rows_ascend(const Layout &q) {
  for (int i = 0; i < 7; i++)
    if (q.row[i] >= q.row[i + 1]) return false;
  return true;
}

template <int K, int LC> struct Rounds {
  static constexpr int R = K % 4, NF = K / 4, N = NF + (R ? 1 : 0);
  // layout of round i of the execution order, row order as the bank rule of the
  // round after it needs it: the 16 threads of a half-warp store to 16
  // different 8-byte bank groups of the next layout (lowest bits that do,
  // which also keeps a warp's global accesses on neighbouring addresses)
  static __host__ __device__ constexpr Layout make(bool dif, int i) {
    Layout q{};
    const int top_down = dif ? N - 1 - i : i; // position from the window's top
    const bool is_short = R && top_down == N - 1;
    q.V = is_short ? R : 4;
    q.B = is_short ? 0 : K - 4 * (top_down + 1);
    for (int t = 0; t < 4; t++) q.slot[t] = t < q.V ? LC + q.B + t : TILE_BITS - 4 + t; // short: the tile's top bits
    int nrow = 0;
    int rest[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int b = 0; b < TILE_BITS; b++)
      if (!in4(q.slot, b)) rest[nrow++] = b;
    for (int t = 0; t < 8; t++) q.row[t] = rest[t];
    if (i + 1 < N) {
      const Layout n = make(dif, i + 1);
      bool found = false;
      for (int m = 0; m < 256 && !found; m++) {
        int pick[4] = {0, 0, 0, 0}, cnt = 0;
        for (int t = 0; t < 8; t++)
          if (m >> t & 1) {
            if (cnt < 4) pick[cnt] = rest[t];
            cnt++;
          }
        if (cnt != 4) continue;
        if (!spans16(bank_of(n, pick[0]), bank_of(n, pick[1]), bank_of(n, pick[2]), bank_of(n, pick[3]))) continue;
        found = true;
        int o = 4;
        for (int t = 0; t < 4; t++) q.row[t] = pick[t];
        for (int t = 0; t < 8; t++)
          if (rest[t] != pick[0] && rest[t] != pick[1] && rest[t] != pick[2] && rest[t] != pick[3]) q.row[o++] = rest[t];
      }
    }
    return q;
  }
};

// Byte offset in the tile of the element with tile index e: linear over XOR,
// so e may be split into a thread's part and a constant part.
template <int K, int LC, bool DIF, int I> __host__ __device__ constexpr uint32_t addr_of(uint32_t e) {
  constexpr Layout q = Rounds<K, LC>::make(DIF, I);
  uint32_t r = 0, s = 0;
#pragma unroll
  for (int t = 0; t < 8; t++) r |= (e >> q.row[t] & 1u) << t;
#pragma unroll
  for (int t = 0; t < 4; t++) s |= (e >> q.slot[t] & 1u) << t;
  return r << 7 | ((s >> 1) ^ (r & 7u)) << 4 | (s & 1u) << 3;
}

// Tile index of row r's word 0, and of word s alone.
template <int K, int LC, bool DIF, int I> __host__ __device__ constexpr uint32_t elem_of_row(uint32_t r) {
  constexpr Layout q = Rounds<K, LC>::make(DIF, I);
  uint32_t e = 0;
#pragma unroll
  for (int t = 0; t < 8; t++) e |= (r >> t & 1u) << q.row[t];
  return e;
}
template <int K, int LC, bool DIF, int I> __host__ __device__ constexpr uint32_t elem_of_slot(uint32_t s) {
  constexpr Layout q = Rounds<K, LC>::make(DIF, I);
  uint32_t e = 0;
#pragma unroll
  for (int t = 0; t < 4; t++) e |= (s >> t & 1u) << q.slot[t];
  return e;
}

// Power table of a tile position: s_R^j of every round but the window's top one
// (its single R is the tile's prefix, whose powers go into its matrix).  The
// round on window bits [B, B + V) keeps s_R^j (j = 0 .. 2^V - 1; s_R =
// T[R << (V - 1)], R the prefix and the window bits above) at
// pw_base(B) + R_local (2^V + 1) + j, rounds nearer the top first: the odd
// stride puts one j of 16 consecutive R on 16 different banks.
template <int K> struct PowerTable {
  static __host__ __device__ constexpr int V(int B) { return B == 0 && K % 4 ? K % 4 : 4; }
  static __host__ __device__ constexpr uint32_t rows(int B) { return 1u << (K - B - V(B)); } // R_local values
  static __host__ __device__ constexpr int next(int B) { return B >= 4 ? B - 4 : (B > 0 ? 0 : -1); }
  static __host__ __device__ constexpr uint32_t base(int B) {
    uint32_t o = 0;
    for (int b = next(K - 4); b > B; b = next(b)) o += rows(b) * ((1u << V(b)) + 1);
    return o;
  }
  static constexpr uint32_t words = base(-1);
  // entry of window value w in the round on [B, B + V)
  static __host__ __device__ constexpr uint32_t index(int B, uint32_t w) {
    return base(B) + (w >> (B + V(B))) * ((1u << V(B)) + 1) + ((w >> B) & ((1u << V(B)) - 1));
  }
};

// Order of the matrices in DevTables::tc_img: per direction and twiddle table
// (variant = 2 B2N + INV), those of V = 1..4 stages (16 / 2^V blocks on the diagonal).
__host__ __device__ constexpr uint32_t img_index(bool b2n, bool inv, int V) { return (2 * b2n + inv) * 4 + V - 1; }
constexpr uint32_t IMAGES = 16;

// Writes the 8 x 8 digit block of matrix entry (o, i) = c (canonical): row
// 8 o + j, column 8 i + b holds digit j of c 2^(8b) mod p.
__device__ __forceinline__ void put_entry(uint8_t *img, uint32_t o, uint32_t i, uint64_t c) {
  uint32_t v[16]; // v[2 b], v[2 b + 1]: words of c 2^(8b)
#pragma unroll
  for (int b = 0; b < 8; b++) {
    v[2 * b] = gl::lo32(c);
    v[2 * b + 1] = gl::hi32(c);
    c = gl::mul_pow2<8, true>(c);
  }
#pragma unroll
  for (int half = 0; half < 2; half++) { // digits 0..3 from the low words, 4..7 from the high ones
    uint32_t q[2][4];                    // q[b / 4][j]: digit j of four consecutive b
#pragma unroll
    for (int g = 0; g < 2; g++) {
      const uint32_t w0 = v[8 * g + half], w1 = v[8 * g + 2 + half], w2 = v[8 * g + 4 + half], w3 = v[8 * g + 6 + half];
      const uint32_t a0 = __byte_perm(w0, w1, 0x5140), a1 = __byte_perm(w2, w3, 0x5140);
      const uint32_t b0 = __byte_perm(w0, w1, 0x7362), b1 = __byte_perm(w2, w3, 0x7362);
      q[g][0] = __byte_perm(a0, a1, 0x5410);
      q[g][1] = __byte_perm(a0, a1, 0x7632);
      q[g][2] = __byte_perm(b0, b1, 0x5410);
      q[g][3] = __byte_perm(b0, b1, 0x7632);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t row = 8 * o + 4 * half + j;
      *reinterpret_cast<uint2 *>(img + row * 128 + (((i >> 1) ^ (row & 7)) << 4) + (i & 1) * 8) =
          make_uint2(q[0][j], q[1][j]);
    }
  }
}

// Entry (o, i) of a round's matrix.  DIT (natural -> bit-reversed): output o,
// input i: w^(i brev(o)); DIF: w^(o brev(i)); w = w_{2^V} (inverse twiddles:
// its inverse), all of them powers of two: w_16 = 2^156.  The bits above V pick
// the block on the diagonal.
__host__ __device__ constexpr int entry_exp(bool dif, bool inv, int V, uint32_t o, uint32_t i) {
  const uint32_t m = (1u << V) - 1;
  const uint32_t a = dif ? o & m : i & m, r = dif ? i & m : o & m;
  uint32_t b = 0;
  for (int t = 0; t < V; t++) b |= (r >> t & 1u) << (V - 1 - t);
  const int e = (int)((156u * ((a * b) << (4 - V))) % 192u);
  return inv ? (192 - e) % 192 : e;
}

// 2^e mod p, e < 192.
__device__ __forceinline__ uint64_t pow2_mod(uint32_t e) {
  const bool neg = e >= 96;
  if (neg) e -= 96;
  uint64_t r;
  if (e < 64) {
    r = 1ull << e;
    if (r >= gl::P) r -= gl::P;
  } else {
    r = (gl::EPS << (e - 64)); // 2^64 = EPS; EPS 2^(e - 64) < 2^64 for e < 96
    r = gl::canon(r);
  }
  return neg ? (r ? gl::P - r : 0) : r;
}

} // namespace tc
} // namespace bc
