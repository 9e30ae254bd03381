// Routed experts of several tokens over the 2-bit affine bank on the f16 tensor cores (tcgen05.mma kind::f16, weights
// as the TMEM operand).
//
// A weight is s*q + b with one fp16 pair (s, b) per group of 128 codes q in 0..3.  Written as
// s*(q-1) + (b+s), the first term is one of {-s, 0, s, 2s}: exact in fp16 (up to |s| = 32752), so the MMA multiplies
// the true weight and no scale has to be applied to partial sums.  The second term only needs the sums of the
// activations over the groups; they enter the same accumulator as further K columns: [b | s] against the group sums
// split into two fp16 halves (22 bits).  Activations are bf16, so after scaling a row by a power of two (its largest
// value into [2^7, 2^8)) they are exact in fp16 down to 2^-25 of the row's largest value.  Against float64 with the same
// bf16 roundings a call is off by 1e-4 to 1.8e-4 of its norm (values that rounded the other way), the one-token kernel,
// whose place it takes and which holds activations in fixed point, by 2.1e-4 to 2.7e-4.  The one-warp kernels, at 1.3e-5
// with groups of 64, keep the banks that the one-token kernel does not take.
//
// Rows are grouped by expert.  Two grouped GEMMs run per call, weights on the M side:
//   gate/up : [128 weight rows, <=64 routed rows] twice, K = hidden; g, u rounded to bf16, SwiGLU, router weight,
//             h rounded to bf16 (the reference's rounding points, model/expert_affine.py:65-81)
//   down    : K = inter, y rounded to bf16; a last kernel adds a token's k rows in route order.
// Before each, prep_rows_kernel writes the scaled fp16 rows with their group sums behind them, in the K order the
// unpacking produces (codes j and j+8 of a 16-code word side by side).
//
// What bounds it: an expert's 2-bit rows at 6.5 TB/s leave an SM 89 cycles per 128 x 64 codes, and unpacking them
// takes 100 instructions in each of the four warps that hold the tile's rows (one and + or, one FMA, one multiply per two
// codes); the MMAs of a unit of 64 rows take 128.  So the unpacked operand goes registers -> TMEM (tcgen05.st, 32 cycles a
// tile), not through shared memory, where writing and reading it again would take 256 cycles.  Sixteen warps unpack, four
// per scheduler: a tile's step takes 455 to 476 cycles in a loop of eight warps by themselves, and sixteen instead of
// eight took 2048 tokens from 4.85 to 4.28 ms.  In the kernel (64 experts, 3072 rows, gate/up) the schedulers issue in 65 %
// of the cycles, 1080 instructions per tile with scales, waits and addresses: issue slots bound it, not DRAM (18 %).
//
// Warp roles (768 threads): warp 0 TMA (weight tiles through a 3-D map {K/4 bytes, rows, slot}, activation rows
// sixteen at a time), warp 1 owns TMEM and issues the MMAs, warps 4-19 unpack (four per TMEM lane quarter),
// warps 20-23 drain.  Every wait is bounded (CACHALOT_STATUS_WAIT_EXPIRED).
#include "tensor_core.cuh"

namespace cachalot {
namespace {

constexpr int BM = 128;           // weight rows per tile (MMA M)
constexpr int NT = 64;            // routed rows per unit (MMA N): two accumulator buffers and four operand slots fill TMEM
constexpr int KST = 256;          // codes of K per shared-memory stage
constexpr int W_TILE = BM * KST / 4;
constexpr int X_PIECE = NT * 128;  // 64 fp16 of every row
constexpr int X_BOX = 16 * 128;    // one TMA box: 16 rows
constexpr int NTHREADS = 768;
constexpr int UNPACK0 = 4, DRAIN0 = 20;  // first unpacking and draining warp
constexpr int TMEM_COLS = 512;
constexpr int A_COL = 256;        // operand slots start behind the accumulators
constexpr int MAX_STAGES = 5, BAR_BYTES = 512;
constexpr int A_SLOTS = 4;        // of 64 columns: gate and up of one 64-code step, or two steps of down

__device__ __forceinline__ void tc_mma_f16_ts(uint32_t tacc, uint32_t ta, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(tacc),
      "r"(ta), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,"
      "%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
      "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// instruction descriptor of kind::f16: f16 x f16 -> f32, both K-major, M = 128, N = n
__device__ __forceinline__ uint32_t idesc_f16(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24); }

// K as the kernels see it: k codes, then the group sums' columns (high halves, low halves), `ext` each
struct KShape {
  int k, block, n_block, ext, pitch;
};
__host__ __device__ inline KShape k_shape(int k) {
  KShape s;
  s.k = k;
  s.block = k % 128 == 0 ? 128 : 64;  // rows that start in mid-group: half groups
  s.n_block = k / s.block;
  s.ext = (2 * s.n_block + 63) / 64 * 64;
  s.pitch = k + 2 * s.ext;
  return s;
}

struct F16Args {
  const uint8_t* bank;
  long long record_bytes;
  long long off_s[2], off_b[2];  // scale and bias arrays of the matrices inside a record
  const Unit* units;
  const int32_t* n_units;
  int n_rows, k;
  const float* row_scale;  // f32 [R]: what a row's accumulators are multiplied by
  const float* row_w;      // gate/up: router weight of every grouped row
  float limit;
  int n_stage;             // shared-memory stages
  int n_win;               // 16-byte windows that hold a row's scales (or biases) at any alignment
  __nv_bfloat16* out;      // bf16 [R, n_rows]: h or y
  int* status;
};

// 64 codes of one row (16 bytes) -> 32 registers of s*(q-1): register 8i+j holds codes j and j+8 of word i.  Written in
// PTX: through the half2 intrinsics the same arithmetic took 250 instructions instead of 100.
__device__ __forceinline__ void unpack64(const uint4 wv, uint32_t s2, uint32_t (&r)[32]) {
  const uint32_t w[4] = {wv.x, wv.y, wv.z, wv.w};
  // 4^-c and -(1024 * 4^-c + 1) as pairs of halves
  constexpr uint32_t mul[5] = {0x3C003C00u, 0x34003400u, 0x2C002C00u, 0x24002400u, 0x1C001C00u};
  constexpr uint32_t add[5] = {0xE401E401u, 0xDC04DC04u, 0xD410D410u, 0xCC40CC40u, 0xC500C500u};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t hi = w[i] >> 10;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int c = j < 5 ? j : j - 5;  // the two bits sit at 2c of a ten-bit mantissa: 1024 + 4^c q
      uint32_t t;
      asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(t) : "r"(j < 5 ? w[i] : hi), "r"(0x00030003u << (2 * c)), "r"(0x64006400u));
      asm("fma.rn.f16x2 %0, %0, %1, %2;" : "+r"(t) : "r"(mul[c]), "r"(add[c]));
      asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r[8 * i + j]) : "r"(t), "r"(s2));
    }
  }
}

template <int NA>
__global__ void __launch_bounds__(NTHREADS, 1)
grouped_f16_kernel(const __grid_constant__ CUtensorMap map_a0, const __grid_constant__ CUtensorMap map_a1,
                   const __grid_constant__ CUtensorMap map_b, F16Args A) {
  constexpr int STAGE_BYTES = NA * W_TILE + (KST / 64) * X_PIECE;
  constexpr int OFF_X = NA * W_TILE;
  constexpr int ACC_COLS = NA * NT;
  static_assert(2 * ACC_COLS <= A_COL && A_COL + A_SLOTS * 64 <= TMEM_COLS, "TMEM columns");
  const int n_stage = A.n_stage;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)n_stage * STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* a_full = empty + MAX_STAGES;
  uint64_t* a_empty = a_full + A_SLOTS;
  uint64_t* acc_full = a_empty + A_SLOTS;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* sc_full = acc_empty + 2;  // one per pair of unpacking warps
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(sc_full + 8);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_holder + 1);
  uint8_t* sc_base = smem + (size_t)n_stage * STAGE_BYTES + BAR_BYTES;  // scales and biases of this and the next item

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    // a stage is free when its last MMA is done: the unpacking warps that wait for the stage have read it before that
    for (int s = 0; s < n_stage; ++s) mbar_init(&full[s], 1), mbar_init(&empty[s], 1);
    for (int s = 0; s < A_SLOTS; ++s) mbar_init(&a_full[s], 8), mbar_init(&a_empty[s], 1);
    for (int b = 0; b < 2; ++b) mbar_init(&acc_full[b], 1), mbar_init(&acc_empty[b], 4);
    for (int b = 0; b < 8; ++b) mbar_init(&sc_full[b], 2);
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)), "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_holder;

  const int n_mt = (A.n_rows + BM - 1) / BM;
  const long long total = (long long)*A.n_units * n_mt;
  const KShape K = k_shape(A.k);
  const int n64 = A.k / 64, n_main = (n64 + 3) / 4;         // 64-code steps; stages of four
  const int e64 = K.ext / 64, n_ext = (e64 + 1) / 2;        // group-sum steps; stages of two (each: high and low half)
  const int n_st = n_main + n_ext;
  // 64-wide steps of stage ks
  auto steps_of = [&](int ks) { return ks < n_main ? min(4, n64 - ks * 4) : min(2, e64 - (ks - n_main) * 2); };

  if (warp == 0) {
    // ---- loads --------------------------------------------------------------------------------
    if (elect_one()) {
      uint64_t pol_w, pol_x;
      asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol_w));
      asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol_x));
      int s = 0;
      uint32_t ph = 0;
      bool wrapped = false, ok = true;
      for (long long w = blockIdx.x; w < total && ok; w += gridDim.x) {
        const Unit u = A.units[w / n_mt];
        const int row = (int)(w % n_mt) * BM;
        const int n16 = (u.ntok + 15) >> 4;
        for (int ks = 0; ks < n_st; ++ks) {
          if (wrapped && !mbar_wait(&empty[s], ph ^ 1u, abort)) { ok = false; break; }
          uint8_t* st = smem + (size_t)s * STAGE_BYTES;
          const int steps = steps_of(ks);
          const bool main = ks < n_main;
          const int pieces = main ? steps : 2 * steps;
          mbar_expect_tx(&full[s], (main ? NA * W_TILE : 0) + pieces * n16 * X_BOX);
          if (main) {
            tma_load_3d(st, &map_a0, ks * (KST / 4), row, u.slot, &full[s], pol_w);
            if (NA == 2) tma_load_3d(st + W_TILE, &map_a1, ks * (KST / 4), row, u.slot, &full[s], pol_w);
          }
          for (int j = 0; j < pieces; ++j) {
            // main: 64 codes each; group sums: high and low half of step 0, then of step 1
            const int kx = main ? (ks * 4 + j) * 64 : A.k + (j & 1) * K.ext + ((ks - n_main) * 2 + (j >> 1)) * 64;
            for (int i = 0; i < n16; ++i)
              tma_load_2d(st + OFF_X + j * X_PIECE + i * X_BOX, &map_b, kx * 2, u.row_start + 16 * i, &full[s], pol_x);
          }
          if (++s == n_stage) s = 0, ph ^= 1u, wrapped = true;
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMAs ---------------------------------------------------------------------------------
    if (elect_one()) {
      int s = 0, a = 0;
      uint32_t ph = 0, aph = 0;
      long long item = 0;
      bool ok = true;
      const uint64_t d_x0 = desc_sw128(smem_u32(smem) + OFF_X);
      for (long long w = blockIdx.x; w < total && ok; w += gridDim.x, ++item) {
        const Unit u = A.units[w / n_mt];
        const int buf = (int)(item & 1);
        const uint32_t id = idesc_f16((u.ntok + 15) & ~15);
        const uint32_t t_acc = tmem + buf * ACC_COLS;
        uint32_t accumulate = 0;
        if (item >= 2 && !mbar_wait(&acc_empty[buf], (uint32_t)((item >> 1) - 1) & 1u, abort)) { ok = false; break; }
        tc_fence_after();
        for (int ks = 0; ks < n_st && ok; ++ks) {
          if (!mbar_wait(&full[s], ph, abort)) { ok = false; break; }
          const uint64_t dx = d_x0 + (uint64_t)((uint32_t)(s * STAGE_BYTES) >> 4);
          const int steps = steps_of(ks);
          const bool main = ks < n_main;
          for (int st = 0; st < steps; st += (NA == 2 ? 1 : 2)) {
            if (!mbar_wait(&a_full[a], aph, abort)) { ok = false; break; }
            tc_fence_after();
            const uint32_t ta = tmem + A_COL + a * 64;
#pragma unroll
            for (int h = 0; h < 2; ++h) {  // half of the slot: matrix h, or step st + h
              if (NA == 1 && st + h >= steps) break;
              const int piece = (main ? 1 : 2) * (NA == 2 ? st : st + h);
              const uint32_t td = t_acc + (NA == 2 ? h * NT : 0);
              const uint64_t db = dx + (uint64_t)((uint32_t)(piece * X_PIECE) >> 4);
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                tc_mma_f16_ts(td, ta + h * 32 + kk * 8, db + kk * 2, id, (NA == 2 || h == 0) && kk == 0 ? accumulate : 1u);
              if (!main) {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) tc_mma_f16_ts(td, ta + h * 32 + kk * 8, db + (X_PIECE >> 4) + kk * 2, id, 1u);
              }
            }
            accumulate = 1;
            tc_commit(&a_empty[a]);
            if (++a == A_SLOTS) a = 0, aph ^= 1u;
          }
          tc_commit(&empty[s]);
          if (++s == n_stage) s = 0, ph ^= 1u;
        }
        if (ok) tc_commit(&acc_full[buf]);
      }
    }
  } else if (warp >= UNPACK0 && warp < DRAIN0) {
    // ---- codes -> fp16 operand in TMEM -----------------------------------------------------------
    // TMEM lane quarter; matrix (gate/up) or step of a slot (down); which of every two operand slots
    const int q = warp & 3, p = ((warp - UNPACK0) >> 2) & 1, hh = (warp - UNPACK0) >> 3;
    const int m = q * 32 + lane;                  // row of the tile
    const uint32_t t_dst = tmem + A_COL + ((uint32_t)(q * 32) << 16) + p * 32;
    // The scales and biases of the next item come by 16-byte asynchronous copies (a row of them starts at any even
    // address) into windows [buffer][set][array][window][row].  The two warps that unpack the same rows (hh) share them:
    // one brings the scales, the other the biases.
    const long long off_s = NA == 2 && p ? A.off_s[1] : A.off_s[0], off_b = NA == 2 && p ? A.off_b[1] : A.off_b[0];
    struct RowRef {
      uint32_t buf;        // shared-memory address
      int lead_s, lead_b;  // halfs in front of the row's first group
      int i0;              // the row's first 64-code step, counted over the matrix
      bool ok;             // the row exists
    };
    auto fetch = [&](long long w, int par) {
      RowRef r;
      const Unit u = A.units[w / n_mt];
      const uint8_t* rec = A.bank + (size_t)u.slot * A.record_bytes;
      const int n = (int)(w % n_mt) * BM + m;
      r.ok = n < A.n_rows;
      r.i0 = n * n64;
      const uint32_t dst = smem_u32(sc_base) + (uint32_t)((par * 2 + p) * 2 * A.n_win * BM + m) * 16;
      r.buf = dst;
      const long long g0 = r.i0 >> 1, g1 = (r.i0 + n64 - 1) >> 1;  // two steps of 64 codes to a group
#pragma unroll
      for (int arr = 0; arr < 2; ++arr) {
        const uintptr_t at = reinterpret_cast<uintptr_t>(rec + (arr ? off_b : off_s) + 2 * g0);
        const uintptr_t end = at + 2 * (g1 - g0 + 1);
        (arr ? r.lead_b : r.lead_s) = (int)(at & 15) >> 1;
        if (r.ok && arr == hh)
          for (int i = 0; i < A.n_win; ++i) {
            const uintptr_t from = (at & ~(uintptr_t)15) + 16 * i;
            if (from < end)
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (uint32_t)((arr * A.n_win + i) * BM * 16)), "l"(from) : "memory");
          }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      return r;
    };
    // half number i of the row's scales (arr 0) or biases (1)
    auto value = [&](const RowRef& r, int arr, int i) -> uint32_t {
      const int h = (arr ? r.lead_b : r.lead_s) + i;
      uint16_t v;
      asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(r.buf + (uint32_t)((arr * A.n_win + (h >> 3)) * BM * 16 + (h & 7) * 2)));
      return v;
    };
    auto ext_val = [&](const RowRef& r, int e) -> uint32_t {
      if (!r.ok || e >= 2 * K.n_block) return 0u;
      const bool is_s = e >= K.n_block;
      const int j = is_s ? e - K.n_block : e;
      return value(r, is_s ? 0 : 1, K.block == 128 ? j : ((r.i0 + j) >> 1) - (r.i0 >> 1));
    };
    int s = 0, a = 0;
    uint32_t ph = 0, aph = 1;  // the first pass over the slots finds them free
    bool ok = true;
    // one operand slot: free -> unpacked -> published
    auto begin = [&]() -> bool {
      if (!__all_sync(0xffffffffu, mbar_wait(&a_empty[a], aph, abort))) return false;
      tc_fence_after();
      return true;
    };
    auto publish = [&]() {
      tc_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_full[a]);
    };
    auto next_slot = [&]() {
      if (++a == A_SLOTS) a = 0, aph ^= 1u;
    };
    RowRef cur = {}, nxt = {};
    int par = 0;
    if (blockIdx.x < total) nxt = fetch(blockIdx.x, 0);
    for (long long w = blockIdx.x; w < total && ok; w += gridDim.x) {
      cur = nxt;
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&sc_full[p * 4 + q]);
      if (!__all_sync(0xffffffffu, mbar_wait(&sc_full[p * 4 + q], par, abort))) break;  // both warps: arrived, and done with the other buffer
      par ^= 1;
      if (w + gridDim.x < total) nxt = fetch(w + gridDim.x, par);
      auto stage = [&](int ks, int steps, bool codes) -> bool {
        if (!__all_sync(0xffffffffu, mbar_wait(&full[s], ph, abort))) return false;
        const uint32_t row = smem_u32(smem) + s * STAGE_BYTES + (NA == 2 ? p * W_TILE : 0) + m * (KST / 4);
        for (int i = 0; i < steps; i += (NA == 2 ? 1 : 2), next_slot()) {
          if ((a & 1) != hh) continue;
          const int step = NA == 2 ? i : i + p;
          if (!begin()) return false;
          if (step < steps) {
            uint32_t r[32];
            if (codes) {
              uint4 wv;
              asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                           : "=r"(wv.x), "=r"(wv.y), "=r"(wv.z), "=r"(wv.w)
                           : "r"(row + ((step ^ ((m >> 1) & 3)) << 4)));
              const uint32_t sv = cur.ok ? value(cur, 0, ((cur.i0 + ks * 4 + step) >> 1) - (cur.i0 >> 1)) : 0u;
              unpack64(wv, sv * 0x10001u, r);
            } else {
              const int e0 = ((ks - n_main) * 2 + step) * 64;
#pragma unroll
              for (int j = 0; j < 32; ++j) r[j] = ext_val(cur, e0 + 2 * j) | (ext_val(cur, e0 + 2 * j + 1) << 16);
            }
            tc_st32(t_dst + a * 64, r);
          }
          publish();
        }
        return true;
      };
      // Full stages of codes in a loop of their own (2048 tokens 4.28 -> 4.07 ms: four steps known to the compiler).
      int ks = 0;
      for (; ks < n64 / 4 && ok; ++ks) {
        ok = stage(ks, 4, true);
        if (++s == n_stage) s = 0, ph ^= 1u;
      }
      // A set of warps waits for the stages that it unpacks a slot of, and for no other: the MMAs that free a stage do not
      // wait for it there, so it could come after the stage's next fill, take that phase for the one before its own and
      // wait for good.  A phase that it did not wait for is over when it comes to that stage again: stages with one slot
      // are among the last n_ext + 1 of an item, at most n_stage (enough_stages), and between two items it meets
      // (sc_full) the warp of the other set that did wait.
      for (; ks < n_st && ok; ++ks) {
        const int steps = steps_of(ks);
        if (steps > (NA == 2 ? 1 : 2) || (a & 1) == hh) ok = stage(ks, steps, ks < n_main);
        else next_slot();
        if (++s == n_stage) s = 0, ph ^= 1u;
      }
    }
  } else if (warp >= DRAIN0) {
    // ---- accumulators -> h or y -------------------------------------------------------------------
    const int q = warp & 3;
    const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
    long long item = 0;
    for (long long w = blockIdx.x; w < total; w += gridDim.x, ++item) {
      const Unit u = A.units[w / n_mt];
      const int n0 = (int)(w % n_mt) * BM + q * 32;
      const int buf = (int)(item & 1);
      const bool rows_ok = n0 < A.n_rows;  // whole warps: n_rows is a multiple of 64
      if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[buf], (uint32_t)(item >> 1) & 1u, abort))) break;
      tc_fence_after();
      for (int j0 = 0; j0 < u.ntok; j0 += 16) {
        uint32_t g[16], up[16];
        tc_ld16(lane_base + buf * ACC_COLS + j0, g);
        if (NA == 2) tc_ld16(lane_base + buf * ACC_COLS + NT + j0, up);
        float rs = 0.f, wv = 0.f;
        if (lane < 16 && j0 + lane < u.ntok) {
          rs = A.row_scale[u.row_start + j0 + lane];
          if (NA == 2) wv = A.row_w[u.row_start + j0 + lane];
        }
        tc_ld_wait();
        if (!rows_ok) continue;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (j0 + j >= u.ntok) break;
          const float sc = __shfl_sync(0xffffffffu, rs, j);
          float v = bf16_round(__uint_as_float(g[j]) * sc);
          if (NA == 2) v = swiglu(v, bf16_round(__uint_as_float(up[j]) * sc), A.limit) * __shfl_sync(0xffffffffu, wv, j);
          A.out[(size_t)(u.row_start + j0 + j) * A.n_rows + n0 + lane] = __float2bfloat16_rn(v);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort) {
    if (threadIdx.x == 0 && A.status) atomicOr(A.status, CACHALOT_STATUS_WAIT_EXPIRED);
    // give loads and MMAs still in flight time to land before the shared memory goes away
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

__device__ __forceinline__ float finite_or_0(float v) { return fabsf(v) <= 3.4e38f ? v : 0.f; }

// One CTA per grouped row: bf16 row src[p] (or p) of [., k] -> fp16 row p times a power of two, codes j and j+8 of every
// sixteen side by side, behind it the sums of its blocks (twice: against the biases and the scales) as high and low
// halves.  out fp16 [rows, pitch], row_scale f32 [rows] = the inverse of the power of two.  An infinite or NaN value shows in
// its block's sum alone, against the bias alone, so that the product is bias * sum as in the one-token kernel: as an
// operand of its own it would meet zeros and both signs of s*(q-1).
__global__ void prep_rows_kernel(const __nv_bfloat16* __restrict__ x, const int32_t* __restrict__ src, KShape K, __half* __restrict__ out,
                                 float* __restrict__ row_scale) {
  __shared__ float part[32];
  const int p = blockIdx.x;
  const __nv_bfloat16* row = x + (size_t)(src ? src[p] : p) * K.k;
  __half* o = out + (size_t)p * K.pitch;
  const int n16 = K.k / 16;
  float amax = 0.f;
  for (int g = threadIdx.x; g < 2 * n16; g += blockDim.x) {
    const uint4 v = *reinterpret_cast<const uint4*>(row + g * 8);
    const uint32_t wds[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      amax = fmaxf(amax, fmaxf(fabsf(finite_or_0(__uint_as_float(wds[j] << 16))), fabsf(finite_or_0(__uint_as_float(wds[j] & 0xffff0000u)))));
  }
  amax = warp_max(amax);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = warp_max((threadIdx.x & 31) < (blockDim.x >> 5) ? part[threadIdx.x & 31] : 0.f);
  const int eb = (int)(__float_as_uint(amax) >> 23);
  const int e = eb == 0 ? 0 : min(134 - eb, 126);  // largest finite value into [2^7, 2^8); a row of zeros as it is
  const float sc = pow2f(e);
  if (threadIdx.x == 0) row_scale[p] = pow2f(-e);
  const int per = K.block / 16;  // sixteens per block: 4 or 8 neighbouring threads
  for (int g0 = 0; g0 < n16; g0 += blockDim.x) {
    const int g = g0 + threadIdx.x;
    float sum = 0.f;
    if (g < n16) {
      uint32_t wds[8];
      *reinterpret_cast<uint4*>(wds) = *reinterpret_cast<const uint4*>(row + g * 16);
      *reinterpret_cast<uint4*>(wds + 4) = *reinterpret_cast<const uint4*>(row + g * 16 + 8);
      __half h[16];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float a = __uint_as_float(wds[j] << 16), b = __uint_as_float(wds[j] & 0xffff0000u);
        h[2 * j] = __float2half_rn(finite_or_0(a) * sc);
        h[2 * j + 1] = __float2half_rn(finite_or_0(b) * sc);
        sum += (a - finite_or_0(a)) + (b - finite_or_0(b));  // 0 where both are finite
      }
      __half2 r[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        r[j] = __halves2half2(h[j], h[j + 8]);
        sum += __half2float(h[2 * j]) + __half2float(h[2 * j + 1]);
      }
      *reinterpret_cast<uint4*>(o + g * 16) = *reinterpret_cast<const uint4*>(r);
      *reinterpret_cast<uint4*>(o + g * 16 + 8) = *reinterpret_cast<const uint4*>(r + 4);
    }
    for (int d = 1; d < per; d <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if (g < n16 && g % per == 0) {
      const int j = g / per;
      const bool fin = fabsf(sum) <= 65504.f;
      const __half hi = __float2half_rn(sum), lo = __float2half_rn(fin ? sum - __half2float(hi) : 0.f);
      __half* e0 = o + K.k + j;
      e0[0] = hi, e0[K.n_block] = fin ? hi : __float2half_rn(0.f);
      e0[K.ext] = e0[K.ext + K.n_block] = lo;
    }
  }
  for (int j = 2 * K.n_block + threadIdx.x; j < K.ext; j += blockDim.x) o[K.k + j] = o[K.k + K.ext + j] = __float2half_rn(0.f);
}

constexpr size_t SMEM_LIMIT = 227 * 1024;
// windows of a row of scales: its halfs behind up to 14 bytes of lead-in, none where every row starts on 16 bytes
int windows(int k) {
  const int g = (k + 127) / 128 + (k % 128 ? 1 : 0);
  const bool aligned = k % 1024 == 0;
  return (2 * g + (aligned ? 0 : 14) + 15) / 16;
}
size_t scale_bytes(int n_win) { return (size_t)8 * n_win * BM * 16; }  // [buffer][set][scale, bias][window][row]
// as many stages as fit beside the scales
int stages(int na, int n_win) {
  const size_t fixed = scale_bytes(n_win) + BAR_BYTES + 1024;
  if (fixed >= SMEM_LIMIT) return 0;
  return (int)min((SMEM_LIMIT - fixed) / (size_t)(na * W_TILE + (KST / 64) * X_PIECE), (size_t)MAX_STAGES);
}
// enough stages: two for a pipeline, and those at the end of an item that may have one operand slot only, the group sums'
// and the last one of the codes, in different ones
bool enough_stages(int na, int k) { return stages(na, windows(k)) >= 1 + (k_shape(k).ext / 64 + 1) / 2; }
size_t smem_bytes(int na, int nstage, int n_win) {
  return (size_t)nstage * (na * W_TILE + (KST / 64) * X_PIECE) + scale_bytes(n_win) + BAR_BYTES + 1024;
}

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct F16Scratch {
  PlanArrays plan;
  float *x_scale, *h_scale;
  __half *xp, *hp;
  __nv_bfloat16 *h, *y;
  size_t total;
};
F16Scratch carve_f16(uint8_t* base, const BankView& v, size_t R, size_t n_seg) {
  F16Scratch s;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    uint8_t* p = base ? base + at : nullptr;
    at += align_up(bytes, 256);
    return p;
  };
  const size_t S = n_seg > R ? n_seg : R;
  s.plan.seg_off = reinterpret_cast<int32_t*>(take((S + 1) * 4));
  s.plan.seg_slot = reinterpret_cast<int32_t*>(take(S * 4));
  s.plan.inv = reinterpret_cast<int32_t*>(take(R * 4));
  s.plan.src_token = reinterpret_cast<int32_t*>(take(R * 4));
  s.plan.row_w = reinterpret_cast<float*>(take(R * 4));
  s.plan.n_units = reinterpret_cast<int32_t*>(take(256));
  s.plan.units = reinterpret_cast<Unit*>(take((R / NT + R + 1) * sizeof(Unit)));  // a segment with rows: ceil(rows / NT)
  s.x_scale = reinterpret_cast<float*>(take(R * 4));
  s.h_scale = reinterpret_cast<float*>(take(R * 4));
  // x is through when h is prepared, and h when y is written: two buffers serve the four
  s.xp = s.hp = reinterpret_cast<__half*>(take(R * max(k_shape(v.hidden).pitch, k_shape(v.inter).pitch) * 2));
  s.h = s.y = reinterpret_cast<__nv_bfloat16*>(take(R * max(v.hidden, v.inter) * 2));
  s.total = at;
  return s;
}

// planned rows -> s.y
int run_f16(const BankView& v, const F16Scratch& s, const void* x_bf16, long long R, float limit, int* status, cudaStream_t stream) {
  const int H = v.hidden, I = v.inter;
  const KShape kx = k_shape(H), kh = k_shape(I);
  CUtensorMap m_w1, m_w3, m_w2, m_x, m_h;
  int rc;
  if ((rc = make_map(&m_w1, v.base + v.off[0], H / 4, H / 4, I, v.record_bytes, v.n_slots, BM, KST / 4))) return rc;
  if ((rc = make_map(&m_w3, v.base + v.off[6], H / 4, H / 4, I, v.record_bytes, v.n_slots, BM, KST / 4))) return rc;
  if ((rc = make_map(&m_w2, v.base + v.off[3], I / 4, I / 4, H, v.record_bytes, v.n_slots, BM, KST / 4))) return rc;
  if ((rc = make_map(&m_x, s.xp, kx.pitch * 2, kx.pitch * 2, (int)R, 0, 0, 16, 128))) return rc;
  if ((rc = make_map(&m_h, s.hp, kh.pitch * 2, kh.pitch * 2, (int)R, 0, 0, 16, 128))) return rc;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  F16Args a = {};
  a.bank = v.base;
  a.record_bytes = v.record_bytes;
  a.units = s.plan.units;
  a.n_units = s.plan.n_units;
  a.row_w = s.plan.row_w;
  a.limit = limit;
  a.status = status;

  prep_rows_kernel<<<(unsigned)R, 256, 0, stream>>>((const __nv_bfloat16*)x_bf16, s.plan.src_token, kx, s.xp, s.x_scale);
  a.off_s[0] = v.off[1], a.off_b[0] = v.off[2];
  a.off_s[1] = v.off[7], a.off_b[1] = v.off[8];
  a.n_rows = I, a.k = H;
  a.row_scale = s.x_scale;
  a.out = s.h;
  auto launch = [&](auto kern, int na, const CUtensorMap& ma0, const CUtensorMap& ma1, const CUtensorMap& mb) {
    a.n_win = windows(a.k);
    a.n_stage = stages(na, a.n_win);
    smem_optin_once(kern, (int)SMEM_LIMIT);
    kern<<<sms, NTHREADS, smem_bytes(na, a.n_stage, a.n_win), stream>>>(ma0, ma1, mb, a);
  };
  launch(grouped_f16_kernel<2>, 2, m_w1, m_w3, m_x);
  if ((rc = check_launch("moe (2-bit, grouped) gate/up"))) return rc;

  prep_rows_kernel<<<(unsigned)R, 256, 0, stream>>>(s.h, nullptr, kh, s.hp, s.h_scale);
  a.off_s[0] = a.off_s[1] = v.off[4], a.off_b[0] = a.off_b[1] = v.off[5];
  a.n_rows = H, a.k = I;
  a.row_scale = s.h_scale;
  a.out = s.y;
  launch(grouped_f16_kernel<1>, 1, m_w2, m_w2, m_h);
  return check_launch("moe (2-bit, grouped) down");
}

}  // namespace

bool f16_supported(const BankView& v) {
  return v.format == CACHALOT_BANK_AFFINE && v.bits == 2 && v.group == 128 && v.scale_dtype == CACHALOT_F16 && enough_stages(2, v.hidden) &&
         enough_stages(1, v.inter);
}

// as few runs of whole tokens as the planning kernel's limit allows, as equal as they can be
int decode_f16_run(int rows, int k) {
  const int most = max(PLAN_ROWS_MAX / k, 1), runs = (rows + most - 1) / most;
  return (rows + runs - 1) / runs;
}

size_t decode_f16_workspace_bytes(const BankView& v, int rows, int k) {
  return carve_f16(nullptr, v, (size_t)decode_f16_run(rows, k) * k, 0).total;
}

// Routed experts of a decode batch, reference rounding points, run by run.
int launch_decode_f16(const BankView& v, const void* x_bf16, const int32_t* slots, const float* gate_w, int rows, int k, float limit,
                      void* workspace, void* out, int out_dtype, int* status, cudaStream_t stream) {
  const int chunk = decode_f16_run(rows, k);
  const F16Scratch s = carve_f16(static_cast<uint8_t*>(workspace), v, (size_t)chunk * k, 0);
  for (int r0 = 0; r0 < rows; r0 += chunk) {
    const int n = min(chunk, rows - r0), R = n * k;
    int rc;
    if ((rc = launch_decode_plan(s.plan, slots + (size_t)r0 * k, gate_w + (size_t)r0 * k, R, k, v.n_slots, 1, NT, status, stream))) return rc;
    if ((rc = run_f16(v, s, static_cast<const __nv_bfloat16*>(x_bf16) + (size_t)r0 * v.hidden, R, limit, status, stream))) return rc;
    uint8_t* o = static_cast<uint8_t*>(out) + (size_t)r0 * v.hidden * (out_dtype == CACHALOT_BF16 ? 2 : 4);
    if ((rc = launch_combine_rows(s.y, s.plan.inv, n, k, v.hidden, o, out_dtype, stream))) return rc;
  }
  return CACHALOT_OK;
}

size_t prefill_f16_workspace_bytes(const BankView& v, int tokens, int k, int n_experts) {
  return carve_f16(nullptr, v, (size_t)tokens * k, (size_t)n_experts).total;
}

int launch_prefill_f16(const BankView& v, const void* x_bf16, const int32_t* perm, const int32_t* offsets, const int32_t* slot_of_expert,
                       const float* gate_w, int tokens, int k, int n_experts, float limit, void* workspace, float* out, int* status,
                       cudaStream_t stream) {
  const long long R = (long long)tokens * k;
  const F16Scratch s = carve_f16(static_cast<uint8_t*>(workspace), v, (size_t)R, (size_t)n_experts);
  int rc;
  if ((rc = launch_prefill_plan(s.plan, perm, offsets, slot_of_expert, gate_w, R, k, n_experts, v.n_slots, NT, true, status, stream))) return rc;
  if ((rc = run_f16(v, s, x_bf16, R, limit, status, stream))) return rc;
  return launch_combine_rows(s.y, s.plan.inv, tokens, k, v.hidden, out, CACHALOT_F32, stream);
}

}  // namespace cachalot
