// ntt.cu -- per-device tables, pass plans, and the plain batched-NTT C ABI.
//
// C-ABI entry points mirror the reference's Rust surface in src/ntt.rs and
// src/context.rs (declared in include/bc_ntt.h with the line each replaces).
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <mutex>
#include <vector>

#include "../../include/bc_ntt.h"
#include "ntt_host.cuh"
#include "ntt_pass.cuh"
#include "tc.cuh"

namespace bc {

// ---------------------------------------------------------------- host field
namespace hostf {
constexpr uint64_t P = 0xffffffff00000001ull;
typedef unsigned __int128 u128;
inline uint64_t mul(uint64_t a, uint64_t b) { return (uint64_t)(((u128)a * b) % P); }
inline uint64_t pow(uint64_t b, uint64_t e) {
  uint64_t r = 1;
  b %= P;
  while (e) {
    if (e & 1) r = mul(r, b);
    b = mul(b, b);
    e >>= 1;
  }
  return r;
}
inline uint64_t inv(uint64_t a) { return pow(a, P - 2); }
inline uint64_t root(unsigned log_size) { return pow(pow(7, (P - 1) >> 32), 1ull << (32 - log_size)); }
inline uint32_t brev(uint32_t x, unsigned bits) {
  uint32_t r = 0;
  for (unsigned i = 0; i < bits; i++) r |= ((x >> i) & 1u) << (bits - 1 - i);
  return r;
}
} // namespace hostf

// ---------------------------------------------------------------- context
namespace {
constexpr int MAX_DEVICES = 64;
constexpr size_t TC_TAIL_TABS = 16; // offset of the copy of the tables behind the matrices; the error word before it

struct DeviceCtx {
  bool live = false;
  uint64_t *block = nullptr;
  uint64_t *top_pw = nullptr; // precomputed top-window power tables
  uint64_t *top_pw_st = nullptr; // the same for the short-round-on-top partition
  uint8_t *tc = nullptr; // tensor-core matrices, then the wait-error word and a copy of tabs
  DevTables tabs{};
  int sms = 0;
};
DeviceCtx g_ctx[MAX_DEVICES];
std::mutex g_ctx_mutex;

constexpr size_t N_TW_LO = 1u << TW_FINE, N_TW_HI = 1u << (TW_LOG - 1 - TW_FINE);
constexpr size_t N_G_LO = 1u << G_FINE, N_G_HI = 1u << (TW_LOG - G_FINE);
constexpr size_t N_W_LO = 1u << PW_FINE, N_W_HI = 1u << (PW_LOG - PW_FINE);
constexpr size_t TABLE_WORDS = 2 * (N_TW_LO + N_TW_HI + N_G_LO + N_G_HI + N_W_LO + N_W_HI);
constexpr int MAX_TOP_K = 12; // largest window of a pass

void build_host_tables(std::vector<uint64_t> &h, size_t off[12]) {
  using namespace hostf;
  h.assign(TABLE_WORDS, 0);
  size_t o = 0;
  auto seg = [&](int idx, size_t len) {
    off[idx] = o;
    o += len;
  };
  for (int inv_ = 0; inv_ < 2; inv_++) {
    seg(0 + inv_, N_TW_LO);
    seg(2 + inv_, N_TW_HI);
    seg(4 + inv_, N_G_LO);
    seg(6 + inv_, N_G_HI);
    seg(8 + inv_, N_W_LO);
    seg(10 + inv_, N_W_HI);
  }
  for (int inv_ = 0; inv_ < 2; inv_++) {
    const uint64_t w_lo_root = inv_ ? inv(root(TW_FINE + 1)) : root(TW_FINE + 1);
    const uint64_t w_hi_root = inv_ ? inv(root(TW_LOG)) : root(TW_LOG);
    for (uint32_t r = 0; r < N_TW_LO; r++) h[off[0 + inv_] + r] = pow(w_lo_root, brev(r, TW_FINE));
    for (uint32_t r = 0; r < N_TW_HI; r++) h[off[2 + inv_] + r] = pow(w_hi_root, brev(r, TW_LOG - 1 - TW_FINE));
    const uint64_t g = inv_ ? inv(7) : 7;
    uint64_t acc = 1;
    for (size_t i = 0; i < N_G_LO; i++, acc = mul(acc, g)) h[off[4 + inv_] + i] = acc;
    const uint64_t g_step = pow(g, N_G_LO);
    acc = 1;
    for (size_t i = 0; i < N_G_HI; i++, acc = mul(acc, g_step)) h[off[6 + inv_] + i] = acc;
    const uint64_t w = inv_ ? inv(root(PW_LOG)) : root(PW_LOG);
    acc = 1;
    for (size_t i = 0; i < N_W_LO; i++, acc = mul(acc, w)) h[off[8 + inv_] + i] = acc;
    const uint64_t w_step = pow(w, N_W_LO);
    acc = 1;
    for (size_t i = 0; i < N_W_HI; i++, acc = mul(acc, w_step)) h[off[10 + inv_] + i] = acc;
  }
}
} // namespace

int current_device() {
  int d = -1;
  if (cudaGetDevice(&d) != cudaSuccess) return -1;
  return d;
}

const DevTables *device_tables() {
  const int d = current_device();
  if (d < 0 || d >= MAX_DEVICES || !g_ctx[d].live) return nullptr;
  return &g_ctx[d].tabs;
}

const DevTables *device_tables_on_gpu() {
  const DevTables *t = device_tables();
  return t ? reinterpret_cast<const DevTables *>(t->tc_img + tc_table_bytes() + TC_TAIL_TABS) : nullptr;
}

int sm_count() {
  const int d = current_device();
  if (d >= 0 && d < MAX_DEVICES && g_ctx[d].sms) return g_ctx[d].sms;
  int n = 148;
  if (d >= 0) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, d);
  return n;
}

// Layout of the top-window power tables: per K (1..12) the inverse table, then
// for b = 1 .. TOP_PW_LOG - K the 2^b forward tables, 2^K words each, i.e.
// 2^K (2^(TOP_PW_LOG + 1 - K) - 1) = 2^16 - 2^K words per K.  Table t of a K
// (t = 0 the inverse one, t = 2^b - 1 + k the forward one of coset k of b).
size_t top_pw_base(int K) { return (size_t)(K - 1) * (1u << (TOP_PW_LOG + 1)) - ((1u << K) - 2); }
size_t top_pw_words() { return top_pw_base(MAX_TOP_K + 1); }

// One block per table t of window size K, rounds of partition PART.
template <int K, int PART> __global__ void top_pw_fill_kernel(const DevTables tabs, uint64_t *base) {
  const uint32_t t = blockIdx.x;
  uint32_t inv = 1, H = 0;
  if (t > 0) {
    const uint32_t b = 31 - __clz(t + 1), k = t + 1 - (1u << b);
    inv = 0;
    H = brev_bits(k, b);
  }
  fill_powers<K, 0, PART>(base + (size_t)t * (1u << K), tabs, inv, H, threadIdx.x, blockDim.x);
}

template <int K, int PART> cudaError_t top_pw_fill(const DevTables &tabs, uint64_t *all) {
  const uint32_t tables = (1u << (TOP_PW_LOG + 1 - K)) - 1;
  top_pw_fill_kernel<K, PART><<<tables, 256>>>(tabs, all + top_pw_base(K));
  if constexpr (K < MAX_TOP_K) return top_pw_fill<K + 1, PART>(tabs, all);
  return cudaGetLastError();
}

cudaError_t context_create_current() {
  std::lock_guard<std::mutex> lock(g_ctx_mutex);
  const int d = current_device();
  if (d < 0 || d >= MAX_DEVICES) return cudaErrorInvalidDevice;
  DeviceCtx &c = g_ctx[d];
  if (c.live) return cudaSuccess;
  std::vector<uint64_t> h;
  size_t off[12];
  build_host_tables(h, off);
  // the pass kernels apply T[u], u < 8, as shifts by small_tw_exp
  for (int inv_ = 0; inv_ < 2; inv_++)
    for (int u = 0; u < 8; u++)
      if (h[off[0 + inv_] + u] != hostf::pow(2, (uint64_t)small_tw_exp(inv_ != 0, u))) return cudaErrorInvalidValue;
  cudaError_t e = cudaMalloc(&c.block, TABLE_WORDS * sizeof(uint64_t));
  if (e != cudaSuccess) return e;
  e = cudaMemcpy(c.block, h.data(), TABLE_WORDS * sizeof(uint64_t), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(c.block);
    c.block = nullptr;
    return e;
  }
  for (int inv_ = 0; inv_ < 2; inv_++) {
    c.tabs.tw_lo[inv_] = c.block + off[0 + inv_];
    c.tabs.tw_hi[inv_] = c.block + off[2 + inv_];
    c.tabs.g_lo[inv_] = c.block + off[4 + inv_];
    c.tabs.g_hi[inv_] = c.block + off[6 + inv_];
    c.tabs.w_lo[inv_] = c.block + off[8 + inv_];
    c.tabs.w_hi[inv_] = c.block + off[10 + inv_];
  }
  const uint64_t two_inv = hostf::inv(2);
  uint64_t acc = 1;
  for (int k = 0; k <= TW_LOG; k++, acc = hostf::mul(acc, two_inv)) c.tabs.inv_pow2[k] = acc;
  e = cudaMalloc(&c.top_pw, top_pw_words() * sizeof(uint64_t));
  if (e == cudaSuccess) e = cudaMalloc(&c.top_pw_st, top_pw_words() * sizeof(uint64_t));
  if (e == cudaSuccess) e = top_pw_fill<1, 0>(c.tabs, c.top_pw);
  if (e == cudaSuccess) e = top_pw_fill<1, 1>(c.tabs, c.top_pw_st);
  if (e == cudaSuccess) e = cudaMalloc(&c.tc, tc_table_bytes() + TC_TAIL_TABS + sizeof(DevTables));
  if (e == cudaSuccess) e = cudaMemset(c.tc + tc_table_bytes(), 0, TC_TAIL_TABS);
  if (e == cudaSuccess) e = tc_fill_tables(c.tc, c.tabs);
  c.tabs.tc_img = c.tc;
  c.tabs.wait_error = reinterpret_cast<uint32_t *>(c.tc + tc_table_bytes());
  c.tabs.wait_tries = tc::WAIT_TRIES;
  if (e == cudaSuccess)
    e = cudaMemcpy(c.tc + tc_table_bytes() + TC_TAIL_TABS, &c.tabs, sizeof(DevTables), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    cudaFree(c.block);
    cudaFree(c.top_pw);
    cudaFree(c.top_pw_st);
    cudaFree(c.tc);
    c.block = c.top_pw = c.top_pw_st = nullptr;
    c.tc = nullptr;
    return e;
  }
  cudaDeviceGetAttribute(&c.sms, cudaDevAttrMultiProcessorCount, d);
  c.live = true;
  return cudaSuccess;
}

const uint64_t *top_power_tables(uint32_t K, uint32_t log_blowup, bool inverse, bool short_top) {
  const int d = current_device();
  if (d < 0 || d >= MAX_DEVICES || !g_ctx[d].live || K < 1 || K > (uint32_t)MAX_TOP_K) return nullptr;
  const uint64_t *base = (short_top ? g_ctx[d].top_pw_st : g_ctx[d].top_pw) + top_pw_base((int)K);
  if (inverse) return base;
  if (log_blowup < 1 || K + log_blowup > (uint32_t)TOP_PW_LOG) return nullptr;
  return base + ((size_t)(1u << log_blowup) - 1) * (1u << K);
}

cudaError_t context_destroy_current() {
  std::lock_guard<std::mutex> lock(g_ctx_mutex);
  const int d = current_device();
  if (d < 0 || d >= MAX_DEVICES) return cudaErrorInvalidDevice;
  DeviceCtx &c = g_ctx[d];
  if (!c.live) return cudaSuccess;
  c.live = false;
  cudaError_t e = cudaFree(c.block);
  const cudaError_t e2 = cudaFree(c.top_pw);
  const cudaError_t e3 = cudaFree(c.top_pw_st);
  const cudaError_t e4 = cudaFree(c.tc);
  if (e == cudaSuccess) e = e2;
  if (e == cudaSuccess) e = e3;
  if (e == cudaSuccess) e = e4;
  c.block = c.top_pw = c.top_pw_st = nullptr;
  c.tc = nullptr;
  return e;
}

// ---------------------------------------------------------------- plans
Plan two_pass(int top, int low) {
  Plan pl{};
  pl.npasses = 2;
  pl.pass[0] = {(uint8_t)top, (uint8_t)(top <= 9 ? 8 : top == 10 ? 4 : 2)};
  pl.pass[1] = {(uint8_t)low, 1};
  return pl;
}

// Default pass plans.  The pass that owns bit 0 takes up to 12 bits (contiguous
// 32 KB tiles); the others use windows whose shared-memory rounds are free of
// bank conflicts: 4, 5, 8 or 9 bits with runs of 8 (64-byte rows), 10 bits with
// runs of 4, 11 bits with runs of 2.  On the tensor cores a window of 4 j + 1
// bits spends a round on its last bit: upper windows of 5 and 9 bits lost to 4
// and 8 (B200, plain forward: 64 x 2^14 21.0 us as 5 + 9, 19.0 as 4 + 10; 16 x
// 2^18 86 as 9 + 9, 76 as 8 + 10), and on the other kernels these splits are no
// slower at 18..20 bits.
Plan default_plan(uint32_t log_n) {
  Plan pl{};
  // top window bits for 13..23 (index log_n - 13)
  static const uint8_t top2[11] = {5, 4, 4, 8, 8, 8, 8, 8, 9, 10, 11};
  if (log_n <= 12) {
    pl.npasses = 1;
    pl.pass[0] = {(uint8_t)log_n, 1};
  } else if (log_n <= 23) {
    pl = two_pass(top2[log_n - 13], (int)log_n - top2[log_n - 13]);
  } else {
    // 24..27: two upper windows from {4, 5, 8, 9, 10} over the bits above 12
    static const uint8_t a3[4] = {4, 5, 5, 5}, b3[4] = {8, 8, 9, 10};
    pl.npasses = 3;
    pl.pass[0] = {a3[log_n - 24], 8};
    pl.pass[1] = {b3[log_n - 24], (uint8_t)(b3[log_n - 24] == 10 ? 4 : 8)};
    pl.pass[2] = {12, 1};
  }
  return pl;
}

// A plan whose lowest window is below 12 bits tiles columns together on the
// tensor cores (2^(12 - K) of them).  With fewer columns than fill such a tile
// (tc_window_ok) that pass, and with it the fused top window, would run on the
// other kernels: a two-pass split with a larger low window that is filled is
// taken instead, 12 bits at most, else one bit more in the low window (2^13: 4
// + 9 bits instead of 5 + 8, 6 % faster on the other kernels).  Upper windows
// of 4, 8 or 10 bits before 5 or 9 when whole_rounds (plain transforms, 16 bits
// as 4 + 12 against 5 + 11, 2..100 columns: 10 to 15 % faster).
static bool fit_split(int low, uint32_t log_n, uint32_t cols, bool whole_rounds, Plan &pl) {
  for (int any = whole_rounds ? 0 : 1; any < 2; any++)
    for (int k = low + 1; k <= 12; k++) {
      const int top = (int)log_n - k;
      const bool has = top == 4 || top == 8 || top == 10 || (any && (top == 5 || top == 9));
      if (has && tc_window_ok(k, 0, cols, true, true)) {
        const Knobs knobs = pl.knobs;
        pl = two_pass(top, k);
        pl.knobs = knobs;
        return true;
      }
    }
  return false;
}
static bool fit_one_more(Plan &pl) {
  const int top = pl.pass[0].K, low = pl.pass[1].K;
  if (pl.npasses != 2 || (top != 5 && top != 9) || low >= 12) return false;
  const Knobs knobs = pl.knobs;
  pl = two_pass(top - 1, low + 1);
  pl.knobs = knobs;
  return true;
}

Plan fit_plan(Plan pl, uint32_t log_n, uint32_t cols) {
  const int low = pl.pass[pl.npasses - 1].K;
  if (cols > 65535) return pl; // the tensor-core kernels' limit, not few
  if (pl.npasses < 2 || pl.pass[pl.npasses - 1].C != 1 || low < 8 || tc_window_ok(low, 0, cols, true, true)) return pl;
  if (!fit_split(low, log_n, cols, false, pl)) fit_one_more(pl);
  return pl;
}

// The same for a plain transform, where the kinds of call differ in what they
// can run on the tensor cores.  Times on B200, of calls captured into a graph,
// 1..100 columns of 2^13..2^21 in every mode.
Plan fit_ntt_plan(Plan pl, uint32_t log_n, uint32_t cols, bool b2n, bool inverse, bool coset) {
  if (log_n <= 12 || cols > 65535) return pl;
  const int low = pl.pass[pl.npasses - 1].K;
  if (low < 8 || low > 12) return pl;
  const uint32_t g = 1u << tc_log_g(low, true), slots = (cols + g - 1) / g * g, tiles = cols << (log_n - 12);
  // Three passes gain from a short low window only when its tiles are full: two
  // otherwise (12 x 2^21: 428 us as 9 + 12, 476 as 4 + 8 + 9).
  const bool two = pl.npasses < 3 || (log_n <= 22 && 8 * cols < 7 * slots);
  // One pass of these keeps the integer kernel (tc_pass_ok): the last of a
  // natural -> bit-reversed inverse, the first of a bit-reversed -> natural
  // forward transform of a coset.  Columns that do not fill a tile are nothing
  // to it, and the splits are those that suit it best (3 x 2^16 inverse: 16 us
  // as 8 + 8, 20 as 5 + 11; of a coset, 12 x 2^13: 20 as 5 + 8, 25 as 4 + 9; 3 x
  // 2^21: 159 as 9 + 12, 170 as 4 + 8 + 9), with three CTAs an SM in low windows
  // of 9..11 bits (33 x 2^17: 120 against 131).
  if (b2n != inverse && (inverse || coset)) {
    if (!two || log_n > 22) return pl;
    int top = (int)(log_n < 21 ? 8 : log_n - 12);
    if (log_n < 16) top = b2n ? (log_n == 13 ? 5 : 4) : coset ? 5 : 4;
    Plan q = two_pass(top, (int)log_n - top);
    if (inverse && q.pass[1].K >= 9 && q.pass[1].K <= 11) q.knobs.occ = BC_PASS_MIN_BLOCKS_B2N;
    return q;
  }
  if (two && pl.npasses == 3) return default_plan(log_n);
  if (tc_window_ok(low, 0, cols, b2n, inverse)) return pl;
  Plan q = pl;
  if (fit_split(low, log_n, cols, true, q)) {
    // half a wave of 12-bit tiles (5 x 2^16 forward: 15.3 us as 8 + 8, 16.5 as 4 + 12; 3 x 2^16: 15.0 and 12.2)
    const bool half_wave = q.pass[1].K == 12 && tiles > 64 && tiles <= 128;
    return half_wave && !b2n && !coset ? pl : q;
  }
  // All on the integer kernels if the coset's powers cannot be spread over the
  // passes; their split also when the columns are more than half of the tiles
  // under a 4-bit window (forward, 5 x 2^13: 11.8 us as 5 + 8, 12.8 as 4 + 9; of
  // a coset 13 and 15).
  if (!b2n && log_n <= 15) {
    const uint32_t g4 = 1u << tc_log_g((int)log_n - 4, true), slots4 = (cols + g4 - 1) / g4 * g4;
    if (coset || 2 * cols > slots4) return two_pass(5, (int)log_n - 5);
  }
  fit_one_more(pl);
  return pl;
}

static bool shape_supported(int K, int C) {
  if (C == 1) return K >= 1 && K <= 12;
  if (C == 8) return K >= 1 && K <= 9;
  if (C == 4) return K == 10;
  if (C == 2) return K == 11;
  return false;
}

bool plan_valid(const Plan &pl, uint32_t log_n) {
  if (pl.npasses < 1 || pl.npasses > 4) return false;
  uint32_t sum = 0;
  for (int i = 0; i < pl.npasses; i++) {
    const int K = pl.pass[i].K, C = pl.pass[i].C;
    if (!shape_supported(K, C)) return false;
    sum += K;
  }
  if (sum != log_n) return false;
  // window of pass i starts at lb = log_n - (K_0 + ... + K_i); C must fit below it
  uint32_t top = log_n;
  for (int i = 0; i < pl.npasses; i++) {
    const uint32_t lb = top - pl.pass[i].K;
    const int C = pl.pass[i].C;
    if (C == 1 && lb != 0) return false;
    if (C > 1 && (1u << lb) < (uint32_t)C) return false;
    top = lb;
  }
  return true;
}

// ---------------------------------------------------------------- kernels

template <int K, int C, bool B2N, bool INV> static PassKernel kptr() { return ntt_pass_kernel<K, C, B2N, INV>; }

template <bool B2N, bool INV> static PassKernel pick_c1(int K) {
  switch (K) {
  case 1: return kptr<1, 1, B2N, INV>();
  case 2: return kptr<2, 1, B2N, INV>();
  case 3: return kptr<3, 1, B2N, INV>();
  case 4: return kptr<4, 1, B2N, INV>();
  case 5: return kptr<5, 1, B2N, INV>();
  case 6: return kptr<6, 1, B2N, INV>();
  case 7: return kptr<7, 1, B2N, INV>();
  case 8: return kptr<8, 1, B2N, INV>();
  case 9: return kptr<9, 1, B2N, INV>();
  case 10: return kptr<10, 1, B2N, INV>();
  case 11: return kptr<11, 1, B2N, INV>();
  case 12: return kptr<12, 1, B2N, INV>();
  default: return nullptr;
  }
}

template <bool B2N, bool INV> static PassKernel pick_c8(int K) {
  switch (K) {
  case 1: return kptr<1, 8, B2N, INV>();
  case 2: return kptr<2, 8, B2N, INV>();
  case 3: return kptr<3, 8, B2N, INV>();
  case 4: return kptr<4, 8, B2N, INV>();
  case 5: return kptr<5, 8, B2N, INV>();
  case 6: return kptr<6, 8, B2N, INV>();
  case 7: return kptr<7, 8, B2N, INV>();
  case 8: return kptr<8, 8, B2N, INV>();
  case 9: return kptr<9, 8, B2N, INV>();
  default: return nullptr;
  }
}

template <bool B2N, bool INV> static PassKernel pick(int K, int C) {
  if (C == 1) return pick_c1<B2N, INV>(K);
  if (C == 8) return pick_c8<B2N, INV>(K);
  if (C == 4 && K == 10) return kptr<10, 4, B2N, INV>();
  if (C == 2 && K == 11) return kptr<11, 2, B2N, INV>();
  return nullptr;
}

// The other occupancy variant of the C = 1 passes of 9..12 bits: 3 CTAs per SM
// for natural->bit-reversed (default 2), 2 for bit-reversed->natural (default 3).
template <bool B2N, bool INV> static PassKernel pick_occ(int K) {
  constexpr int M = B2N ? BC_PASS_MIN_BLOCKS : BC_PASS_MIN_BLOCKS_B2N;
  switch (K) {
  case 9: return ntt_pass_kernel<9, 1, B2N, INV, M>;
  case 10: return ntt_pass_kernel<10, 1, B2N, INV, M>;
  case 11: return ntt_pass_kernel<11, 1, B2N, INV, M>;
  case 12: return ntt_pass_kernel<12, 1, B2N, INV, M>;
  default: return nullptr;
  }
}

PassKernel pick_pass_kernel(int K, int C, bool b2n, bool inverse, int occ) {
  const int dflt = (b2n && K >= 9) ? BC_PASS_MIN_BLOCKS_B2N : BC_PASS_MIN_BLOCKS;
  if (occ && occ != dflt && C == 1 && K >= 9 && K <= 12) {
    const int other = b2n ? BC_PASS_MIN_BLOCKS : BC_PASS_MIN_BLOCKS_B2N;
    if (occ != other) return nullptr;
    if (b2n) return inverse ? pick_occ<true, true>(K) : pick_occ<true, false>(K);
    return inverse ? pick_occ<false, true>(K) : pick_occ<false, false>(K);
  }
  if (b2n) return inverse ? pick<true, true>(K, C) : pick<true, false>(K, C);
  return inverse ? pick<false, true>(K, C) : pick<false, false>(K, C);
}

static uint32_t log2_ceil(uint64_t x) {
  uint32_t l = 0;
  while ((1ull << l) < x) l++;
  return l;
}

bool ntt_args_ok(uint32_t log_n, uint64_t stride_in, uint64_t stride_out, uint32_t log_ext, uint32_t coset_idx) {
  if (log_n < 1 || log_n > (uint32_t)MAX_LOG_N || log_n + log_ext > (uint32_t)PW_LOG) return false;
  const uint64_t n = 1ull << log_n;
  if (n > stride_in || n > stride_out) return false;
  if (coset_idx > 0 && (log_ext == 0 || coset_idx >= (1u << log_ext))) return false;
  return true;
}

uint32_t plan_lb(const Plan &pl, uint32_t log_n, int i) {
  uint32_t top = log_n;
  for (int j = 0; j <= i; j++) top -= pl.pass[j].K;
  return top;
}

uint32_t choose_log_g(uint32_t wc_log, uint32_t cols) {
  // tile of ~4096 elements, at least 512 (one warp of 16 values each), never
  // more columns per iteration than the batch holds
  uint32_t log_g = wc_log < 12 ? 12 - wc_log : 0;
  const uint32_t lg_cols = log2_ceil(cols);
  if (log_g > lg_cols) log_g = lg_cols;
  if (wc_log + log_g < 9) log_g = 9 - wc_log;
  return log_g;
}

bool build_pass(const PassLaunch &pl, int cols_factor_max, PassParams &p, dim3 &grid, uint32_t &threads,
                size_t &smem_bytes) {
  const DevTables *tabs = device_tables();
  if (!tabs) return false;
  const int K = pl.K, C = pl.C;
  p = PassParams{};
  p.in = pl.in;
  p.out = pl.out;
  p.stride_in = pl.stride_in;
  p.stride_out = pl.stride_out;
  p.group_stride_in = pl.group_stride_in;
  p.group_stride_out = pl.group_stride_out;
  p.group_cols = pl.cols;
  p.log_groups = pl.log_groups;
  p.log_n = pl.log_n;
  p.lb = pl.lb;
  // window and run of a tile, log2; tensor-core tiles fill up with low positions, then columns
  const uint32_t wc_log = pl.tc ? 12 - tc_log_g(K, pl.lb == 0) : (uint32_t)K + log2_ceil((uint32_t)C);
  p.log_g = pl.full_tile || pl.tc ? (wc_log < 12 ? 12 - wc_log : 0) : choose_log_g(wc_log, pl.cols);
  const uint32_t G = 1u << p.log_g;
  const uint64_t tiles_per_col = (1ull << pl.log_n) >> wc_log;
  const uint64_t groups = 1ull << pl.log_groups;
  const uint64_t chunks = (pl.cols + G - 1) / G;
  uint64_t factor = (tiles_per_col * chunks * groups) / ((uint64_t)sm_count() * 8);
  if (factor < 1) factor = 1;
  if (factor > (uint64_t)cols_factor_max) factor = cols_factor_max;
  p.cols_per_cta = G * (uint32_t)factor;
  p.chunks_per_group = (pl.cols + p.cols_per_cta - 1) / p.cols_per_cta;
  p.inverse = pl.inverse;
  p.load_scale = pl.load_scale;
  p.store_scale = pl.store_scale;
  p.canon_out = pl.canon_out;
  p.share = pl.share;
  p.overlap = pl.overlap ? 2 * (uint32_t)sm_count() : 0;
  p.has_coset = pl.has_coset;
  p.coset_kshift = pl.coset_kshift;
  p.vec_in = ((uintptr_t)p.in % 16 == 0 && p.stride_in % 2 == 0 && p.group_stride_in % 2 == 0) ? 1 : 0;
  p.vec_out = ((uintptr_t)p.out % 16 == 0 && p.stride_out % 2 == 0 && p.group_stride_out % 2 == 0) ? 1 : 0;
  p.tabs = *tabs;
  const uint32_t tile = G << wc_log;
  threads = tile / 16;
  smem_bytes = pl.tc ? tc_pass_smem(K) : (size_t)pass_smem_words(tile, K) * sizeof(uint64_t);
  const uint64_t gy = groups * p.chunks_per_group;
  if (tiles_per_col > 0x7fffffffull || gy > 65535) return false;
  grid = dim3((uint32_t)tiles_per_col, (uint32_t)gy);
  return true;
}

cudaError_t launch_pass(const PassLaunch &pl, cudaStream_t stream) {
  if (!device_tables()) return cudaErrorInitializationError;
  if (pl.cols == 0) return cudaSuccess;
  PassParams p;
  dim3 grid;
  uint32_t threads;
  size_t smem;
  if (!build_pass(pl, pl.walk, p, grid, threads, smem)) return cudaErrorInvalidConfiguration;
  PassKernel kern = pl.tc ? pick_pass_kernel_tc(pl.K, pl.lb == 0, pl.b2n, pl.inverse)
                          : pick_pass_kernel(pl.K, pl.C, pl.b2n, pl.inverse, pl.occ);
  if (!kern) return cudaErrorInvalidValue;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  if (pl.tc) return launch_tc(kern, grid, smem, p, pl.overlap, stream);
  kern<<<grid, threads, smem, stream>>>(p);
  return cudaGetLastError();
}

// Whether pass i of a plain transform gains from the tensor-core kernel.
static bool tc_faster(const Plan &pl, int i, uint32_t cols, bool b2n, bool inverse, bool scaled) {
  const int K = pl.pass[i].K;
  if (pl.npasses == 1) {
    // A single pass has index prefix 0: the integer kernels skip the top
    // round's powers, and nothing hides this kernel's tables.  Measured at 1 to
    // 30000 columns of 2^8..2^12 (ratio of times, tensor cores / integer):
    // inverse 0.63-1.0; forward with a coset 1.0-1.15 up to a CTA an SM, then
    // 0.77-1.0; plain forward, natural -> bit-reversed, 1.0-1.36 (12 bits: 0.96
    // from some 4000 columns on), bit-reversed -> natural 1.0-1.2 with 9 bits,
    // 0.76-0.96 with 12, else 1.0-1.12 up to about 1000 tiles, then 0.87-1.0.
    const uint32_t g = 1u << tc_log_g(K, true), tiles = (cols + g - 1) / g;
    if (inverse) return true;
    if (scaled) return tiles > (uint32_t)sm_count();
    if (!b2n) return K == 12 && tiles > 2048;
    return K == 12 || (K != 9 && tiles > 1024);
  }
  // Upper windows of a plain natural -> bit-reversed transform that end in a
  // round of one bit: with 9 bits the integer kernel is up to 10 % faster (8 x
  // 2^18, 3 x 2^21), with 5 bits up to 16 % (64 x 2^15) unless the next pass is a
  // tensor-core one, whose tables are then built meanwhile (33 x 2^14: 12 % for
  // the tensor cores).  Scaled by a coset's powers they gain, as windows that
  // are whole rounds do.
  if (!b2n && !scaled && i + 1 < pl.npasses) {
    if (K == 9) return false;
    if (K == 5 && i + 2 == pl.npasses) return tc_window_ok(pl.pass[i + 1].K, 0, cols, b2n, inverse);
  }
  return true;
}

cudaError_t launch_ntt(const Plan &pl, const uint64_t *in, uint64_t *out, uint32_t log_n, uint32_t num_ntts,
                       uint64_t stride_in, uint64_t stride_out, bool bitrev_inputs, bool inverse, uint32_t log_ext,
                       uint32_t coset_idx, cudaStream_t stream) {
  if (!device_tables()) return cudaErrorInitializationError;
  if (num_ntts == 0) return cudaSuccess;
  // a coset transform's scaling is shared by its passes when all of them run on
  // the tensor cores, and otherwise applied whole by its first (forward) or
  // last (inverse) pass
  const bool scaled = log_ext > 0 && bitrev_inputs == inverse;
  bool on_tc[4], share = scaled;
  for (int i = 0; i < pl.npasses; i++) {
    on_tc[i] = tc_window_ok(pl.pass[i].K, plan_lb(pl, log_n, i), num_ntts, bitrev_inputs, inverse) &&
               tc_faster(pl, i, num_ntts, bitrev_inputs, inverse, scaled);
    share = share && on_tc[i];
  }
  bool prev_tc = false;
  for (int s = 0; s < pl.npasses; s++) {
    const int i = bitrev_inputs ? pl.npasses - 1 - s : s; // b2n runs the passes bottom-up
    const bool first = s == 0, last = s == pl.npasses - 1;
    PassLaunch q;
    q.K = pl.pass[i].K;
    q.C = pl.pass[i].C;
    q.b2n = bitrev_inputs;
    q.in = first ? in : out;
    q.out = out;
    q.stride_in = first ? stride_in : stride_out;
    q.stride_out = stride_out;
    q.cols = num_ntts;
    q.log_n = log_n;
    q.lb = plan_lb(pl, log_n, i);
    q.inverse = inverse;
    q.load_scale = first && !inverse && log_ext > 0 && !share;
    q.share = share ? (inverse ? SHARE_COSET_INV : SHARE_COSET) : SHARE_NONE;
    q.store_scale = last && inverse;
    q.canon_out = last;
    q.has_coset = log_ext > 0 ? 1 : 0;
    q.coset_kshift = coset_idx ? coset_idx << (PW_LOG - log_n - log_ext) : 0;
    q.walk = plan_walk(pl);
    q.occ = pl.knobs.occ;
    q.overlap = prev_tc;
    prev_tc = q.tc = on_tc[i] && tc_pass_ok(q);
    cudaError_t e = launch_pass(q, stream);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

} // namespace bc

using namespace bc;

// ---------------------------------------------------------------- C ABI
extern "C" cudaError_t bc_ntt_context_create(uint32_t powers_of_w_coarse_log_count,
                                             uint32_t powers_of_g_coarse_log_count) {
  // The reference splits its tables by these counts (src/context.rs:171-176);
  // the split here is fixed, the arguments keep the reference's bounds check.
  if (powers_of_w_coarse_log_count > 24 || powers_of_g_coarse_log_count > 24) return cudaErrorInvalidValue;
  return context_create_current();
}

extern "C" cudaError_t bc_ntt_context_destroy(void) { return context_destroy_current(); }

extern "C" cudaError_t bc_ntt_wait_status(uint32_t *status) {
  const DevTables *t = device_tables();
  if (!status) return cudaErrorInvalidValue;
  if (!t) return cudaErrorInitializationError;
  cudaError_t e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(status, t->wait_error, sizeof(uint32_t), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && *status) e = cudaMemset(t->wait_error, 0, sizeof(uint32_t));
  return e;
}

extern "C" cudaError_t bc_ntt_set_wait_limit(uint32_t tries) {
  DevTables *t = const_cast<DevTables *>(device_tables());
  if (!t) return cudaErrorInitializationError;
  cudaError_t e = cudaDeviceSynchronize(); // runs already enqueued finish with the old limit
  if (e != cudaSuccess) return e;
  t->wait_tries = tries > tc::WAIT_TRIES ? tc::WAIT_TRIES : tries;
  return cudaMemcpy(const_cast<DevTables *>(device_tables_on_gpu()), t, sizeof(DevTables), cudaMemcpyHostToDevice);
}

extern "C" cudaError_t bc_batch_ntt_internal(const uint64_t *inputs, uint64_t *outputs, uint32_t log_n,
                                             uint32_t num_ntts, uint64_t stride_in, uint64_t stride_out,
                                             bool bitrev_inputs, bool inverse, uint32_t log_extension_degree,
                                             uint32_t coset_index, cudaStream_t stream) {
  if (!ntt_args_ok(log_n, stride_in, stride_out, log_extension_degree, coset_index)) return cudaErrorInvalidValue;
  if (num_ntts && (!inputs || !outputs)) return cudaErrorInvalidValue;
  const Plan pl = call_ntt_plan(log_n, num_ntts, bitrev_inputs, inverse, log_extension_degree > 0);
  return launch_ntt(pl, inputs, outputs, log_n, num_ntts, stride_in, stride_out, bitrev_inputs, inverse,
                    log_extension_degree, coset_index, stream);
}

extern "C" cudaError_t bc_batch_ntt_out_of_place(const uint64_t *inputs_matrix, size_t inputs_len,
                                                 uint64_t *outputs_matrix, size_t outputs_len, uint32_t log_n,
                                                 uint32_t num_ntts, uint64_t inputs_offset, uint64_t outputs_offset,
                                                 uint64_t stride_in, uint64_t stride_out, bool bitrev_inputs,
                                                 bool inverse, uint32_t log_extension_degree, uint32_t coset_index,
                                                 cudaStream_t stream) {
  if (log_n < 1 || log_n > (uint32_t)MAX_LOG_N) return cudaErrorInvalidValue;
  const uint64_t n = 1ull << log_n;
  if (inputs_offset + n > stride_in || outputs_offset + n > stride_out) return cudaErrorInvalidValue;
  if (inputs_len < (uint64_t)num_ntts * stride_in || outputs_len < (uint64_t)num_ntts * stride_out)
    return cudaErrorInvalidValue;
  if (inputs_matrix == outputs_matrix) return cudaErrorInvalidValue;
  const uint64_t *in = inputs_matrix + inputs_offset;
  uint64_t *out = outputs_matrix + outputs_offset;
  if (in == out) return cudaErrorInvalidValue;
  return bc_batch_ntt_internal(in, out, log_n, num_ntts, stride_in, stride_out, bitrev_inputs, inverse,
                               log_extension_degree, coset_index, stream);
}

extern "C" cudaError_t bc_batch_ntt_in_place(uint64_t *inputs_matrix, size_t len, uint32_t log_n, uint32_t num_ntts,
                                             uint64_t inputs_offset, uint64_t stride, bool bitrev_inputs,
                                             bool inverse, uint32_t log_extension_degree, uint32_t coset_index,
                                             cudaStream_t stream) {
  if (log_n < 1 || log_n > (uint32_t)MAX_LOG_N) return cudaErrorInvalidValue;
  const uint64_t n = 1ull << log_n;
  if (inputs_offset + n > stride) return cudaErrorInvalidValue;
  if (len < (uint64_t)num_ntts * stride) return cudaErrorInvalidValue;
  uint64_t *p = inputs_matrix + inputs_offset;
  return bc_batch_ntt_internal(p, p, log_n, num_ntts, stride, stride, bitrev_inputs, inverse, log_extension_degree,
                               coset_index, stream);
}

extern "C" cudaError_t bc_batch_ntt_with_plan(const uint64_t *inputs, uint64_t *outputs, uint32_t log_n,
                                              uint32_t num_ntts, uint64_t stride_in, uint64_t stride_out,
                                              bool bitrev_inputs, bool inverse, uint32_t log_extension_degree,
                                              uint32_t coset_index, const uint8_t *pass_bits,
                                              const uint8_t *pass_runs, uint32_t npasses, cudaStream_t stream) {
  if (!ntt_args_ok(log_n, stride_in, stride_out, log_extension_degree, coset_index)) return cudaErrorInvalidValue;
  if (npasses < 1 || npasses > 4 || !pass_bits || !pass_runs) return cudaErrorInvalidValue;
  Plan pl{};
  pl.npasses = (int)npasses;
  for (uint32_t i = 0; i < npasses; i++) pl.pass[i] = {pass_bits[i], pass_runs[i]};
  if (!plan_valid(pl, log_n)) return cudaErrorInvalidValue;
  return launch_ntt(pl, inputs, outputs, log_n, num_ntts, stride_in, stride_out, bitrev_inputs, inverse,
                    log_extension_degree, coset_index, stream);
}
