// FP64 contractions on the integer tensor pipe (tcgen05.mma kind::i8).
//
// Each row of an FP64 operand is held as a fixed-point number of 56 bits
// relative to a power of two above the row's largest entry, in seven balanced
// base-256 digits (signed bytes):
//   a_k = 2^(e - 55) sum_i d_i 256^(6 - i),   d_i in [-128, 127].
// A product of two rows is then
//   sum_k a_k b_k = 2^(ea + eb - 14) sum_t 256^-t D_t,
//   D_t = sum_k sum_(i + j = t) d_i[k] d'_j[k],
// where every D_t is an integer sum that the tensor core accumulates exactly
// in 32 bits (at most 7 products of magnitude 2^14 per k: exact up to KMAX
// values of k).  The D_t of t <= 6 are formed (Ozaki's error-free splitting;
// K. Ozaki et al., Numer. Algorithms 59 (2012) 95) and added up in 64-bit
// integers, then in FP64.  What is lost is the rounding of each entry to 2^-56
// of its row's bound and the digit products of t >= 7; no FP64 rounding
// occurs inside the sum over k, whereas the DMMA kernels err like one rounding per
// k.  Rows that this does not suit are noticed, and their products formed by the
// DMMA kernels (RoughRows, k_digit_rowdot_sum).
//
// Why: a DGEMM on the FP64 tensor pipe peaks at 35 TFLOP/s here; the integer
// pipe does the 28 products of digits at up to 4.5 POP/s.  At nmo 300 / naux 1000
// / 32 frequencies the contraction of all 45 150 pairs takes 15.0 ms (DMMA: 52.8
// ms) and P0 3.9 ms (13.0 ms) plus 0.9 ms for its digits; the tensor pipe is busy for
// 93 % of an SM's active cycles in P0 and 83 % in the contraction (a small case of each),
// at the 1.65 GHz that the power limit leaves.  P0's error is 4.6 to 7.1 x 2^-53 of
// the root-sum-square of the terms of an element from K = 1024 to 10 400, the DMMA
// kernel's 8.5 to 28.
//
// The kernel runs on CTA pairs (cta_group::2, M = 256, N = 128).  Why this
// tile: the seven accumulators of a tile are formed in two passes over K, D_4
// to D_6 and then D_3 to D_0 (4 x 128 columns fill TMEM), so that a digit
// slice loaded once per K block feeds up to seven products: 35 to 37 bytes per SM
// and cycle from L2, where one product per load would need 96.  Slices
// travel through a ring of nine 24 KB slots (this CTA's 128 rows of A and half
// of the B tile, 128 bytes of K each), in an order that lets early slices leave
// while late ones arrive (64-byte slices leave room for two whole blocks, but
// measured slower).  The
// accumulators end their sums one after the other, and each is handed to the
// epilogue at once, so that the four buffers go round without the MMAs
// waiting for a drain.  The epilogue keeps the 64-bit sums of its 128 x 128 tile
// in registers (64 per thread), as integers: FP64 instructions hardly get
// issued while the MMAs run at full rate.
#include <algorithm>
#include <cmath>

#include "digit_rowdot.cuh"
#include "qx_blas.cuh"
#include "qx_internal.cuh"
#include "tc_ptx.cuh"

namespace qx {

namespace dgt {
constexpr int NS = 7;                          // digits (slices) per operand
constexpr int BK = 128;                        // bytes of K per block
constexpr int TM = 128;                        // rows of A per CTA
constexpr int TN = 128;                        // N of the pair's tile
constexpr int A_BYTES = TM * BK;               // 16 KB
constexpr int B_BYTES = (TN / 2) * BK;         // 8 KB
constexpr int SLOT_BYTES = A_BYTES + B_BYTES;  // 24 KB
constexpr int SLOTS = 9;
constexpr int NBUF = 4;                        // TMEM accumulators of TN columns
constexpr int BAR_OFF = SLOTS * SLOT_BYTES;
constexpr int NEPI = 8;
constexpr int WARP0 = 4;                       // first epilogue warp (a warpgroup boundary)
constexpr int THREADS = 32 * (WARP0 + NEPI);
// Registers per thread after the split of the launch's 384 x 168: the first
// warpgroup (loads, MMA issue) gives to the two of the epilogue (64 FP64 sums
// each).  128 x 72 + 256 x 216 = 384 x 168.
constexpr int REGS_LAUNCH = 168, REGS_FRONT = 72, REGS_EPI = 216;
static_assert(128 * REGS_FRONT + 32 * NEPI * REGS_EPI <= THREADS * REGS_LAUNCH, "register split");
constexpr int CPW = TN / 2;                    // columns per epilogue warp
constexpr int TOTAL = BAR_OFF + 256 + 1024;    // + slack for the 1024-byte alignment
static_assert(TOTAL <= 232448, "shared memory of one CTA");
// Longest K of a launch: 7 * 2^14 * KMAX < 2^31.
constexpr int KMAX = 16384;
// Order in which a K block's slices are loaded, low pass (seven slices) and
// high pass (four).
__device__ __constant__ const int LOAD_LO[7] = {2, 3, 1, 4, 5, 0, 6};
__device__ __constant__ const int LOAD_HI[4] = {3, 0, 1, 2};
}  // namespace dgt

// One launch: C[w][m][n] = sum_k A[m][k] B[w][n][k] over digit operands.
struct DigitArgs {
  int M, N, K, nbatch;
  int rowdot;            // 1: part[2 nt + half][w][m] = sum_n b C; 0: store
  const double* scaleA;  // [M] 2^(e - 7)
  const double* scaleB;  // [nbatch][ldsb] 2^(e - 7), zeros from N on
  int ldsb;              // N rounded up to TN
  int sh;                // the epilogue's last shift: max(0, ceil(log2 K) - 8)
  // rowdot: the rows of A (b) as integers xt[m / 32][n][m % 32] (k_digit_xt),
  // B lower triangular (K <= n).
  const int2* xt;
  int wgroup;           // frequencies per group of the item order
  double* part;         // [2 n_tiles][nbatch][M]
  // store: lower tiles and their mirror (lower = 1, with delta_mn added; add:
  // onto what out holds, for a further range of K, no delta), or all tiles (wide:
  // out and ldo allow 32-byte stores).
  int lower, add, wide;
  // lower: A is the batched operand too (scaleA = scaleB).
  // Nothing to do when the lowest rho (as RoughRows has it) of A times that of B is
  // above the limit.
  const unsigned* lowA;
  const unsigned* lowB;
  float rough_limit;
  double* out;
  int ldo;
  size_t out_stride;
  int* err;
};

// Column tiles of a lower-triangular store in pairs of 128-row blocks: column
// nt holds T - nt blocks.
__host__ __device__ inline int digit_lower_pairs(int T) {
  int s = 0;
  for (int nt = 0; nt < T; ++nt) s += (T - nt + 1) / 2;
  return s;
}

struct DigitTile {
  int w, nt, mb, kbe;  // frequency, column tile, this CTA's row block, K blocks
};

__device__ __forceinline__ int digit_items(const DigitArgs& a) {
  const int T = (a.M + dgt::TM - 1) / dgt::TM, NT = (a.N + dgt::TN - 1) / dgt::TN;
  if (a.rowdot) return (a.nbatch + a.wgroup - 1) / a.wgroup * ((T + 1) / 2) * a.wgroup * NT;
  return (a.lower ? digit_lower_pairs(T) : (T + 1) / 2 * NT) * a.nbatch;
}

// Item -> tile; false for the padding items of the last frequency group.
__device__ __forceinline__ bool digit_tile(const DigitArgs& a, int it, int rank, DigitTile& t) {
  const int T = (a.M + dgt::TM - 1) / dgt::TM, NT = (a.N + dgt::TN - 1) / dgt::TN;
  const int kb = (a.K + dgt::BK - 1) / dgt::BK;
  if (a.rowdot) {
    // The frequencies of a group share each pair block while it is in L2;
    // the column tiles (of 1, 2, ... K blocks) are rotated from item to item
    // so that the clusters' strides see all of them.
    const int mp_n = (T + 1) / 2, per = mp_n * a.wgroup * NT;
    const int g = it / per, r = it - g * per;
    const int q = r / NT;
    t.nt = (r - q * NT + q) % NT;
    const int mp = q / a.wgroup;
    t.w = g * a.wgroup + (q - mp * a.wgroup);
    t.mb = 2 * mp + rank;
    t.kbe = min(kb, (t.nt + 1) * (dgt::TN / dgt::BK));
    return t.w < a.nbatch;
  }
  const int per = a.lower ? digit_lower_pairs(T) : (T + 1) / 2 * NT;
  t.w = it / per;
  int r = it - t.w * per;
  if (a.lower) {
    for (t.nt = 0; t.nt < T - 1; ++t.nt) {
      const int c = (T - t.nt + 1) / 2;
      if (r < c) break;
      r -= c;
    }
    t.mb = t.nt + 2 * r + rank;
  } else {
    // The smaller operand stays in L2, the larger passes once.
    const int mp = (T + 1) / 2;
    if (a.N <= a.M) {
      t.nt = r % NT;
      t.mb = r / NT * 2 + rank;
    } else {
      t.nt = r / mp;
      t.mb = (r - t.nt * mp) * 2 + rank;
    }
  }
  t.kbe = kb;
  return true;
}

__device__ __forceinline__ void umma_i8_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
// kind::i8: signed 8-bit A and B (format 1), 32-bit integer accumulator
// (format 2), both K-major, no saturation.
constexpr uint32_t kDigitIdesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(dgt::TN >> 3) << 17) |
                                 ((uint32_t)((2 * dgt::TM) >> 4) << 24);

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
      "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

__device__ __forceinline__ double pow2i(int k) { return __hiloint2double((1023 + k) << 20, 0); }  // |k| < 1023

// A 64-bit integer as FP64, rounded once: 2^84 + 2^32 (hi + 2^31) and 2^52 +
// lo as bit patterns (the conversion instruction is far slower).
__device__ __forceinline__ double i64_to_f64(long long s) {
  const double hi = __hiloint2double(0x45300000, (int)(s >> 32) ^ 0x80000000);
  const double lo = __hiloint2double(0x43300000, (int)(uint32_t)s);
  return (hi - (0x1p84 + 0x1p63 + 0x1p52)) + lo;
}

// s 2^q, -1020 <= q <= 900, rounded to nearest even, without FP64 instructions
// (the epilogue's get next to no issue slots while the MMAs run).
__device__ __forceinline__ double i64_scale(long long s, int q) {
  const unsigned long long sign = (unsigned long long)s & 0x8000000000000000ull;
  const unsigned long long m = s < 0 ? 0ull - (unsigned long long)s : (unsigned long long)s;
  if (m == 0) return 0.0;
  const int lz = __clzll((long long)m);
  const unsigned long long t = m << lz;
  const uint32_t lo = (uint32_t)t;
  const uint32_t up = (lo >> 10) & (uint32_t)(((lo & 0x3ff) != 0) | ((lo >> 11) & 1)) & 1;
  const int e = 1022 + 63 - lz + q;  // the leading bit of t >> 11 adds one
  return __longlong_as_double((long long)((((unsigned long long)(uint32_t)e << 52) + (t >> 11) + up) | sign));
}

__device__ __forceinline__ void st_v4(double* p, double a, double b, double c, double d) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};\n" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// A load that does not stay in L1.
__device__ __forceinline__ int2 ld_stream(const int2* p) {
  int2 v;
  asm volatile("ld.global.L1::no_allocate.v2.s32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

// The MMA issuer's view of the slot ring and the accumulators of one pass.
// All 32 lanes of the warp run it with the same values, and one elected lane
// issues: the descriptors then stay in uniform registers.  (With the whole loop
// inside one lane's branch every MMA waited for its descriptors to be moved
// there, ~105 cycles per MMA against the 64 it occupies the tensor core.)
struct DigitIssue {
  uint32_t a0;         // low descriptor word of slot 0's A tile
  uint64_t* full;
  uint64_t* empty;
  uint64_t* acc_full;
  uint64_t* acc_empty;
  volatile int* abort_flag;
  int* err;
  uint32_t tmem;
  uint32_t elected;    // this lane issues
  int slot0, phase0;   // slot and phase of the block's first slice
  int u0;              // sequence number of the pass's first accumulator
  bool ok;

  __device__ __forceinline__ int slot(int pos) const {
    const int s = slot0 + pos;
    return s >= dgt::SLOTS ? s - dgt::SLOTS : s;
  }
  // Wait for the slice at load position pos of this block.
  __device__ __forceinline__ void wait(int pos) {
    const int s = slot0 + pos;
    const int ph = s >= dgt::SLOTS ? phase0 ^ 1 : phase0;
    ok = __all_sync(0xffffffffu, ok && mbar_wait(&full[slot(pos)], ph, abort_flag, err, 44));
    tc_fence_after();
  }
  __device__ __forceinline__ void release(int pos) {
    if (ok && elected) umma_commit_pair_both(&empty[slot(pos)]);
  }
  // Hand accumulator c to the epilogue (after its last product of the pass).
  __device__ __forceinline__ void publish(int c, bool last) {
    if (last && ok && elected) umma_commit_pair_both(&acc_full[(u0 + c) & (dgt::NBUF - 1)]);
  }
  // Product of the slices at positions pa (of A) and pb (of B) into the
  // pass's accumulator c (0..3, in the order of first use); start: the first
  // product of the pass into it.
  __device__ __forceinline__ void mul(int pa, int pb, int c, bool start = false) {
    const int u = u0 + c, buf = u & (dgt::NBUF - 1);
    if (start && u >= dgt::NBUF) {
      ok = __all_sync(0xffffffffu,
                      ok && mbar_wait(&acc_empty[buf], ((u / dgt::NBUF) - 1) & 1, abort_flag, err, 43));
      tc_fence_after();
    }
    const uint32_t a = a0 + slot(pa) * (dgt::SLOT_BYTES >> 4);
    const uint32_t b = a0 + slot(pb) * (dgt::SLOT_BYTES >> 4) + (dgt::A_BYTES >> 4);
    const uint32_t d = tmem + buf * dgt::TN;
    if (ok && elected) {
#pragma unroll
      for (int kk = 0; kk < dgt::BK / 32; ++kk)
        umma_i8_pair(d, umma_desc_of(a + 2 * kk), umma_desc_of(b + 2 * kk), kDigitIdesc, start && kk == 0 ? 0u : 1u);
    }
    __syncwarp();
  }
};

// Low pass, one K block.  Positions of the slices in LOAD_LO: 2 -> 0, 3 -> 1,
// 1 -> 2, 4 -> 3, 5 -> 4, 0 -> 5, 6 -> 6.  Accumulators: D_4 -> 0, D_5 -> 1,
// D_6 -> 2, begun and ended in this order.  start, last: the first and the
// last K block of the pass.
__device__ __forceinline__ void digit_block_lo(DigitIssue& q, bool start, bool last) {
  q.wait(0);
  q.mul(0, 0, 0, start);  // 2 2
  q.wait(1);
  q.wait(2);
  q.mul(2, 1, 0);         // 1 3
  q.mul(1, 2, 0);         // 3 1
  q.mul(0, 1, 1, start);  // 2 3
  q.mul(1, 0, 1);         // 3 2
  q.mul(1, 1, 2, start);  // 3 3
  q.release(1);
  q.wait(3);
  q.mul(0, 3, 2);  // 2 4
  q.mul(3, 0, 2);  // 4 2
  q.release(0);
  q.mul(2, 3, 1);  // 1 4
  q.mul(3, 2, 1);  // 4 1
  q.wait(4);
  q.mul(2, 4, 2);  // 1 5
  q.mul(4, 2, 2);  // 5 1
  q.release(2);
  q.wait(5);
  q.mul(5, 3, 0);  // 0 4
  q.mul(3, 5, 0);  // 4 0
  q.release(3);
  q.publish(0, last);
  q.mul(5, 4, 1);  // 0 5
  q.mul(4, 5, 1);  // 5 0
  q.release(4);
  q.publish(1, last);
  q.wait(6);
  q.mul(5, 6, 2);  // 0 6
  q.mul(6, 5, 2);  // 6 0
  q.release(5);
  q.release(6);
  q.publish(2, last);
}

// High pass.  Positions in LOAD_HI: 3 -> 0, 0 -> 1, 1 -> 2, 2 -> 3.
// Accumulators: D_3 -> 0, D_2 -> 1, D_1 -> 2, D_0 -> 3.
__device__ __forceinline__ void digit_block_hi(DigitIssue& q, bool start, bool last) {
  q.wait(0);
  q.wait(1);
  q.mul(1, 0, 0, start);  // 0 3
  q.mul(0, 1, 0);         // 3 0
  q.release(0);
  q.wait(2);
  q.wait(3);
  q.mul(2, 3, 0);  // 1 2
  q.mul(3, 2, 0);  // 2 1
  q.publish(0, last);
  q.mul(1, 3, 1, start);  // 0 2
  q.mul(3, 1, 1);         // 2 0
  q.release(3);
  q.mul(2, 2, 1);  // 1 1
  q.publish(1, last);
  q.mul(1, 2, 2, start);  // 0 1
  q.mul(2, 1, 2);         // 1 0
  q.release(2);
  q.publish(2, last);
  q.mul(1, 1, 3, start);  // 0 0
  q.release(1);
  q.publish(3, last);
}

// MODE: the epilogue (and args.rowdot, args.lower accordingly).
enum { DIGIT_ROWDOT, DIGIT_LOWER, DIGIT_PLAIN };
template <int MODE>
__global__ void __launch_bounds__(dgt::THREADS, 1)
    k_digit_gemm(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, DigitArgs args) {
  namespace P = dgt;
  if (cluster_nctarank() != 2) {
    if (threadIdx.x == 0) atomicCAS(args.err, 0, 40);
    return;
  }
  if (MODE != DIGIT_ROWDOT && __uint_as_float(~*args.lowA) * __uint_as_float(~*args.lowB) > args.rough_limit) return;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + P::BAR_OFF);
  uint64_t* empty = full + P::SLOTS;
  uint64_t* acc_full = empty + P::SLOTS;    // [NBUF]
  uint64_t* acc_empty = acc_full + P::NBUF;  // [NBUF]
  uint64_t* drain_bar = acc_empty + P::NBUF;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const bool leader = rank == 0;
  const int n_items = digit_items(args);
  const int item0 = (int)cluster_id_x(), item_step = (int)cluster_count_x();

  if (threadIdx.x == 0) {
    for (int s = 0; s < P::SLOTS; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < P::NBUF; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 2 * P::NEPI);  // every epilogue warp of both CTAs
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)),
                 "r"(P::NBUF * P::TN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < P::WARP0) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(P::REGS_FRONT));
  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    if (lane == 0) {
      const uint32_t full_leader = mapa_rank(smem_u32(full), 0);
      int s = 0, ph = 0, used = 0;  // next slot, its phase, slots handed out (up to SLOTS)
      bool ok = true;
      auto load = [&](const DigitTile& t, int kb, int slice) {
        if (!ok) return;
        if (used >= P::SLOTS) {
          if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, args.err, 41)) {
            ok = false;
            return;
          }
        } else {
          ++used;
        }
        if (leader) mbar_expect_tx(&full[s], 2 * P::SLOT_BYTES);
        const uint32_t dst = smem_u32(smem + s * P::SLOT_BYTES);
        const uint32_t fb = full_leader + s * 8;
        tma_load_3d_pair(dst, &mapA, fb, kb * P::BK, t.mb * P::TM, (MODE == DIGIT_LOWER ? t.w * P::NS : 0) + slice);
        tma_load_3d_pair(dst + P::A_BYTES, &mapB, fb, kb * P::BK, t.nt * P::TN + (P::TN / 2) * rank,
                         t.w * P::NS + slice);
        if (++s == P::SLOTS) {
          s = 0;
          ph ^= 1;
        }
      };
      for (int it = item0; it < n_items && ok; it += item_step) {
        DigitTile t;
        if (!digit_tile(args, it, rank, t)) continue;
        for (int kb = 0; kb < t.kbe && ok; ++kb)
          for (int i = 0; i < 7; ++i) load(t, kb, P::LOAD_LO[i]);
        for (int kb = 0; kb < t.kbe && ok; ++kb)
          for (int i = 0; i < 4; ++i) load(t, kb, P::LOAD_HI[i]);
      }
      // The MMA commits of the last slots arrive on this CTA's empty[] too:
      // they have landed before the CTA leaves.
      for (int q = 0; q < used; ++q) {
        const int b = s - used + q;  // the last `used` slots, oldest first
        const int sl = b < 0 ? b + P::SLOTS : b;
        volatile int no_abort = 0;
        mbar_wait(&empty[sl], b < 0 ? ph ^ 1 : ph, &no_abort, args.err, 42);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (even CTA) ----------------
    if (leader) {
      DigitIssue q;
      q.a0 = umma_desc_lo(smem_u32(smem));
      q.full = full;
      q.empty = empty;
      q.acc_full = acc_full;
      q.acc_empty = acc_empty;
      q.abort_flag = abort_flag;
      q.err = args.err;
      q.tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
      q.elected = elect_one();
      q.slot0 = 0;
      q.phase0 = 0;
      q.u0 = 0;
      q.ok = true;
      auto advance = [&](int n) {
        q.slot0 += n;
        if (q.slot0 >= P::SLOTS) {
          q.slot0 -= P::SLOTS;
          q.phase0 ^= 1;
        }
      };
      for (int it = item0; it < n_items && q.ok; it += item_step) {
        DigitTile t;
        if (!digit_tile(args, it, rank, t)) continue;
        for (int kb = 0; kb < t.kbe && q.ok; ++kb) {
          digit_block_lo(q, kb == 0, kb == t.kbe - 1);
          advance(7);
        }
        q.u0 += 3;
        for (int kb = 0; kb < t.kbe && q.ok; ++kb) {
          digit_block_hi(q, kb == 0, kb == t.kbe - 1);
          advance(4);
        }
        q.u0 += 4;
      }
      if (q.elected) {
        umma_commit_pair_own(drain_bar);
        volatile int no_abort = 0;
        mbar_wait(drain_bar, 0, &no_abort, args.err, 45);
      }
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(P::REGS_EPI));
    // ---------------- epilogue (warps 4..11, both CTAs) ----------------
    const int quarter = warp & 3;
    const int half = (warp - P::WARP0) >> 2;
    int u = 0;
    bool ok = true;
    for (int it = item0; it < n_items && ok; it += item_step) {
      DigitTile t;
      if (!digit_tile(args, it, rank, t)) continue;
      const int m = t.mb * P::TM + quarter * 32 + lane;
      const int n0 = t.nt * P::TN + half * P::CPW;
      // The scales of this warp's columns: the first touch brings them to L1.
      const double* sb = args.scaleB + (size_t)t.w * args.ldsb + n0;
      asm volatile("prefetch.global.L1 [%0];\n" ::"l"(sb + 2 * lane));
      // Accumulator in -> the 64 columns of this thread's row.
      auto drain = [&](auto&& f) {
        if (!ok) return;
        const int buf = u & (P::NBUF - 1);
        // The lanes leave together: what follows is collective.
        ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[buf], (u / P::NBUF) & 1, abort_flag, args.err, 46));
        if (!ok) return;
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * P::TN + half * P::CPW;
#pragma unroll
        for (int j = 0; j < P::CPW / 32; ++j) {
          uint32_t r[32];
          tmem_ld32(taddr + 32 * j, r);
#pragma unroll
          for (int q = 0; q < 32; ++q) f(32 * j + q, (int)r[q]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (leader)
            mbar_arrive(&acc_empty[buf]);
          else
            mbar_arrive_rank(&acc_empty[buf], 0);
        }
        ++u;
      };
      // s = sum_t 256^(6 - t) D_t for t = 2..6, in the order of the
      // accumulators: |D_t| < (t + 1) 2^28, so |s| < 2^62.
      long long s[P::CPW];
      drain([&](int c, int d) { s[c] = (long long)d << 16; });
      drain([&](int c, int d) { s[c] += (long long)d << 8; });
      drain([&](int c, int d) { s[c] += d; });
      drain([&](int c, int d) { s[c] += (long long)d << 24; });
      // From here in units of 256 (rounded: less than what the dropped D_7
      // amounts to), with D_1: |s| < 2^54 + 2^61.
      drain([&](int c, int d) { s[c] = (s[c] + ((long long)d << 32) + 128) >> 8; });
      drain([&](int c, int d) { s[c] += (long long)d << 32; });
      // With D_0, in units of 2^(sh + 8) so that the sum stays below 2^63.
      const long long half_unit = args.sh ? 1ll << (args.sh - 1) : 0;
      constexpr int XB = rowdot::TERMS;
      const int2* x = nullptr;
      int2 b[2][XB];
      if (MODE == DIGIT_ROWDOT) {
        x = args.xt + ((size_t)(t.mb * (P::TM / 32) + quarter) * args.ldsb + n0) * 32 + lane;
#pragma unroll
        for (int q = 0; q < XB; ++q) b[0][q] = ld_stream(x + q * 32);
      }
      drain([&](int c, int d) { s[c] = ((s[c] + half_unit) >> args.sh) + ((long long)d << (40 - args.sh)); });
      if (!ok) break;
      const double sa = m < args.M ? args.scaleA[MODE == DIGIT_LOWER ? (size_t)t.w * args.ldsb + m : m] : 0.0;
      if (MODE == DIGIT_ROWDOT) {
        // Each thread contracts its row of C with its row of X, in integers:
        // FP64 instructions get next to no issue slots while the MMAs run at
        // full rate (with them this part of a tile took 16 000 to 36 000 cycles
        // and ended only when the next tile's low pass had, its high pass
        // waiting).  The row of s is shifted up until its largest entry takes 62
        // bits in units of the largest of the columns' scales; of each product X s
        // the part above 2^60 is kept.  X is laid out so that a load is 256
        // contiguous bytes per warp.
        // Exponent fields of the columns' scales (2047: a row that is not finite; 0:
        // a zero row or none), and how far each lies below the largest: column
        // 32 j + l in lane l.
        int dn[P::CPW / 32], emax = 0, spread = 0;
#pragma unroll
        for (int j = 0; j < P::CPW / 32; ++j) emax = max(emax, dn[j] = __double2hiint(__ldg(sb + 32 * j + lane)) >> 20);
        emax = __reduce_max_sync(0xffffffffu, emax);
#pragma unroll
        for (int j = 0; j < P::CPW / 32; ++j) {
          if (dn[j]) spread = max(spread, emax - dn[j]);
          dn[j] = min(emax - dn[j], 63);
        }
        spread = __reduce_max_sync(0xffffffffu, spread);
        int z;
        double v = 0.0;
        auto contract = [&](auto&& y) {
#pragma unroll
          for (int c0 = 0; c0 < P::CPW; c0 += XB) {
            const int h = (c0 / XB) & 1;
            if (c0 + XB < P::CPW) {
#pragma unroll
              for (int q = 0; q < XB; ++q) b[h ^ 1][q] = ld_stream(x + (c0 + XB + q) * 32);
            }
            rowdot::Sum acc;
#pragma unroll
            for (int q = 0; q < XB; ++q) acc.add(b[h][q].x, b[h][q].y, y(c0 + q));
            v += i64_to_f64(acc.result());
          }
        };
        // Scales within 2^3 of each other, as those of a dielectric matrix's rows:
        // the shift is taken from the sums as they are, which costs three bits at
        // most, and from their high words.  (The other form for all tiles took 1 to
        // 3 % longer for the whole call, nmo 121 to 300.)
        uint32_t high = 0;
#pragma unroll
        for (int c = 0; c < P::CPW; ++c) high |= (uint32_t)(rowdot::top_bits(s[c], 0) >> 32);
        z = rowdot::norm_shift((uint64_t)high << 32);
        if (__all_sync(0xffffffffu, spread <= rowdot::NEAR && z >= rowdot::NEAR && (high != 0 || m >= args.M || emax == 0))) {
          contract([&](int c) {  // (a zero column's shift does not matter)
            return (long long)((unsigned long long)s[c] << ((z - emax + (__double2hiint(__ldg(sb + c)) >> 20)) & 63));
          });
        } else {
          auto down = [&](int c) { return __shfl_sync(0xffffffffu, dn[c / 32], c % 32); };
          uint64_t top = 0;
#pragma unroll
          for (int c = 0; c < P::CPW; ++c) top |= rowdot::top_bits(s[c], down(c));
          z = rowdot::norm_shift(top);
          contract([&](int c) { return rowdot::aligned(s[c], z, down(c)); });
        }
        if (m < args.M) {
          // b = 2^(ea - 55) X, C = 2^(ea - 7) 2^(en - 7) 2^(sh - 40) s.
          v = emax == 2047 ? __longlong_as_double(0x7FF8000000000000ll)
                           : ldexp(v * sa, emax - 1023 + args.sh - (88 - rowdot::UNIT) - z) * sa;
          args.part[((size_t)(2 * t.nt + half) * args.nbatch + t.w) * args.M + m] = v;
        }
      } else if (MODE == DIGIT_LOWER) {
        if (m < args.M) {
          const double unit = sa * pow2i(args.sh - 40);  // C = s 2^(sh - 40), scaled
          double* out = args.out + (size_t)t.w * args.out_stride;
          double* orow = out + (size_t)m * args.ldo + n0;
#pragma unroll
          for (int c = 0; c < P::CPW; ++c) {
            const int n = n0 + c;
            if (n >= args.N || n > m) continue;
            double y = i64_to_f64(s[c]) * unit * __ldg(sb + c);
            if (args.add)
              y += orow[c];
            else if (n == m)
              y += 1.0;
            orow[c] = y;
            // The lower triangle and its mirror: the stored matrix is exactly symmetric.
            if (n != m) out[(size_t)n * args.ldo + m] = y;
          }
        }
      } else if (m < args.M) {
        // C = 2^(ea - 7) 2^(en - 7) 2^(sh - 40) s.  A tile of few K blocks is
        // bound by this part: integer arithmetic and stores of whole 32-byte
        // sectors where out allows them (16 800 x 5100 x 700: 2.0 ms with FP64
        // instructions and 8-byte stores, now 1.26).  The scales are
        // powers of two; one that is not a normal number (rows near the ends of
        // the range, or not finite) takes the multiplication.
        const int xs = (__double2hiint(sa) >> 20) & 2047;
        const int xa = (xs == 0 || xs == 2047 ? 1 << 20 : xs) - 2046 + args.sh - 40;
        const double unit = sa * pow2i(args.sh - 40);
        double* orow = args.out + (size_t)t.w * args.out_stride + (size_t)m * args.ldo + n0;
        auto value = [&](int c) {
          const double sc = __ldg(sb + c);
          const int xb = (__double2hiint(sc) >> 20) & 2047, q = xa + xb;
          if (xb == 0 || xb == 2047 || q < -1020 || q > 900) return i64_to_f64(s[c]) * unit * sc;
          return i64_scale(s[c], q);
        };
        if (args.wide && n0 + P::CPW <= args.N) {
#pragma unroll
          for (int c = 0; c < P::CPW; c += 4) st_v4(orow + c, value(c), value(c + 1), value(c + 2), value(c + 3));
        } else {
#pragma unroll
          for (int c = 0; c < P::CPW; ++c)
            if (n0 + c < args.N) orow[c] = value(c);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(P::NBUF * P::TN));
  }
}

// v[w][p] = 2 sum_q part[q][w][p]  (fixed order), and the items (w, block of
// REDO_ROWS pairs) that k_pair_contract_redo has to look at: list[0 .. *count), in any
// order.
//
// Fixed point loses what an entry lacks of its row's bound, so the error of v is
// not bounded by v's own terms when large entries of b meet small ones of W'.
// With 2^e and N the bound and the norm of row b, w_n and r_n those of the rows of W',
// K columns, the root-mean-square error of v is about
//   2 2^-56 (0.58 2^e |b r| + 1.16 2^e N rms(r) + (0.58 N + 0.82 sqrt(K) 2^e) |b w|),
// |b r|^2 = sum_n b_n^2 r_n^2: the entries' rounding (2^-55 / sqrt(12) of their bound)
// in b (in C, in the sum over n, and the epilogue's below it) and in W', and the six
// digit products of t = 7 (each sqrt(1 / 12) 2^8 twice).  Here N times the largest w
// and r stand for the sums (most), and up to 2 x 2^-53 of the sum of the magnitudes of
// v's half-tile sums a pair's digits stand: 1 for a dielectric matrix and normal b of
// any K, 2 where an entry of b is above four deviations.
constexpr int REDO_ROWS = kPairRedoRows;
struct DigitCheck {
  const double* scale;             // [npair] 2^(e - 7)
  const double* norm;              // [npair] r
  const unsigned long long* most;  // [nw] {W, R}
  double k082;                     // 0.82 sqrt(K)
  int* count;
  int* list;                       // w nblk + block
};
__global__ void __launch_bounds__(256) k_digit_rowdot_sum(const double* __restrict__ part, int np, int npair, int nw,
                                                          double* __restrict__ v, int ldv, DigitCheck ck) {
  __shared__ int bad[8];
  const int w = blockIdx.y, nblk = (npair + REDO_ROWS - 1) / REDO_ROWS;
  const double W = __longlong_as_double((long long)ck.most[2 * w]), R = __longlong_as_double((long long)ck.most[2 * w + 1]);
  for (int p0 = blockIdx.x * blockDim.x; p0 < npair; p0 += gridDim.x * blockDim.x) {
    const int p = p0 + threadIdx.x;
    bool fail = false;
    if (p < npair) {
      double s = 0.0, mag = 0.0;
      for (int q = 0; q < np; ++q) {
        const double h = part[((size_t)q * nw + w) * npair + p];
        s += h;
        mag += fabs(h);
      }
      v[(size_t)w * ldv + p] = 2.0 * s;
      const double bound = ck.scale[p] * 128.0, n2 = ck.norm[p] * bound;
      fail = !(n2 * (0.58 * (3.0 * bound * R + n2 * W) + ck.k082 * bound * W) <= 16.0 * mag);
    }
    const int any = __any_sync(0xffffffffu, fail);
    if ((threadIdx.x & 31) == 0) bad[threadIdx.x >> 5] = any;
    __syncthreads();
    if (threadIdx.x < 256 / REDO_ROWS && (bad[2 * threadIdx.x] | bad[2 * threadIdx.x + 1]))
      ck.list[atomicAdd(ck.count, 1)] = w * nblk + p0 / REDO_ROWS + threadIdx.x;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Splitting rows into digits.
// ---------------------------------------------------------------------------
// The row's scale from the bits of its largest magnitude: entries times
// f1 * f2 = 2^(55 - e) lie within the digits' range (the margin for the
// balanced top digit: below 0x7F7F7F7F7F7F80 = 0.996 * 2^55), sc = 2^(e - 7).
// A row with an infinity or a NaN gets zero digits and a NaN scale: what it
// enters becomes NaN.  A zero row gets the scale zero, so that it does not stand
// for the largest scale among rows of small entries.
struct RowScale {
  double f1, f2, sc;
};
constexpr int kNotFinite = 1 << 30;
// f1 and f2 from k = 55 - e (kNotFinite: zeros).
__device__ __forceinline__ RowScale scale_factors(int k) {
  RowScale r;
  const int k1 = k >> 1;
  r.f1 = k == kNotFinite ? 0.0 : pow2i(k1);
  r.f2 = k == kNotFinite ? 0.0 : pow2i(k - k1);
  r.sc = 0.0;
  return r;
}
__device__ __forceinline__ int digit_scale(unsigned long long amax, double& sc) {
  if (amax >= 0x7FF0000000000000ull) {
    sc = __longlong_as_double(0x7FF8000000000000ll);
    return kNotFinite;
  }
  if (amax == 0) {
    sc = 0.0;
    return 55;
  }
  int e = max(1, (int)(amax >> 52)) - 1022;
  if ((amax & 0xFFFFFFFFFFFFFull) >= 0xFC00000000000ull) ++e;
  sc = ldexp(1.0, e - 7);
  return 55 - e;
}
__device__ __forceinline__ RowScale digit_scale(unsigned long long amax) {
  double sc;
  RowScale r = scale_factors(digit_scale(amax, sc));
  r.sc = sc;
  return r;
}

// Eight entries (as their 56-bit integers) -> eight bytes of each digit slice.
// What is seen of a row while it is split: the sum of squares of its top digits
// (x ~ d_0 2^(e - 7)), and the entries without one (below 2^(e - 8)).
struct TopDigits {
  int squares = 0, zeros = 0;
  __device__ __forceinline__ void add(uint32_t four) {
    squares = __dp4a((int)four, (int)four, squares);
    zeros += __popc(~(((four & 0x7f7f7f7fu) + 0x7f7f7f7fu) | four) & 0x80808080u);
  }
};

__device__ __forceinline__ void digit_store8(const double (&x)[8], const RowScale& r, int8_t* dst, size_t slab,
                                             TopDigits& top) {
  constexpr unsigned long long BIAS = 0x80808080808080ull;
  uint32_t lo[8], hi[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    // A row with a non-finite entry stores zeros (its scale is NaN).
    const double y = r.f1 == 0.0 ? 0.0 : x[i] * r.f1 * r.f2;
    const unsigned long long z = ((unsigned long long)__double2ll_rn(y) + BIAS) ^ BIAS;
    lo[i] = (uint32_t)z;
    hi[i] = (uint32_t)(z >> 32);
  }
  uint32_t w[8][2];  // byte position (0 least significant) x four entries
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t *l = lo + 4 * h, *g = hi + 4 * h;
    uint32_t t0 = __byte_perm(l[0], l[1], 0x5140), t1 = __byte_perm(l[2], l[3], 0x5140);
    w[0][h] = __byte_perm(t0, t1, 0x5410);
    w[1][h] = __byte_perm(t0, t1, 0x7632);
    t0 = __byte_perm(l[0], l[1], 0x7362), t1 = __byte_perm(l[2], l[3], 0x7362);
    w[2][h] = __byte_perm(t0, t1, 0x5410);
    w[3][h] = __byte_perm(t0, t1, 0x7632);
    t0 = __byte_perm(g[0], g[1], 0x5140), t1 = __byte_perm(g[2], g[3], 0x5140);
    w[4][h] = __byte_perm(t0, t1, 0x5410);
    w[5][h] = __byte_perm(t0, t1, 0x7632);
    t0 = __byte_perm(g[0], g[1], 0x7362), t1 = __byte_perm(g[2], g[3], 0x7362);
    w[6][h] = __byte_perm(t0, t1, 0x5410);
    top.add(w[6][h]);
  }
#pragma unroll
  for (int i = 0; i < 7; ++i)
    *reinterpret_cast<uint2*>(dst + (size_t)i * slab) = make_uint2(w[6 - i][0], w[6 - i][1]);
}

__device__ __forceinline__ void load8(const double* p, int k, int lim, double (&x)[8]) {
  if (k + 8 <= lim) {
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const double2 v = *reinterpret_cast<const double2*>(p + k + i);
      x[i] = v.x;
      x[i + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = k + i < lim ? p[k + i] : 0.0;
  }
}
__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
}
__device__ __forceinline__ unsigned long long max_bits8(const double (&x)[8], unsigned long long m) {
#pragma unroll
  for (int i = 0; i < 8; ++i) m = max(m, abs_bits(x[i]));
  return m;
}
__device__ __forceinline__ unsigned long long warp_max(unsigned long long m) {
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}

// How far fixed point suits the rows, by blocks of 64: block[w nblk + r / 64] the
// largest rho of its rows, lowest the complement of the smallest of all (as bit
// patterns of floats, zero on entry).
//
// The rounding of an entry (2^-55 of the bound 2^e) and the dropped digit products
// make an error of a product of two rows, in 2^-53 of the root-sum-square of its
// terms, of about rho rho' / 10, rho = 2^e / rms.  The DMMA kernel's sums of K
// random terms make 0.28 sqrt(K).  Tiles stand for their digits up to rho rho' =
// 6.25 sqrt(K) in P0 and 10 sqrt(K) in gemm_nt_digits (rough_limit, of the blocks'
// largest rho: all but a few of a tile's elements lie well below), of rows that
// share most of their large entries: a row
// more than twice as many of whose entries have a zero top digit, |x| < 2^(e - 8),
// as of a normal row (0.8 rho / 256 of them; weighted ones 1.3, and the margin of a
// small K) has an infinite rho here, as one that is not finite.
// Measured for normal B and the weights of zero frequency, digits / DMMA, rms over the
// elements: K = 1024 4.6 / 8.5, 2020 5.5 / 12, 5270 5.9 / 19, 10 400 7.1 / 28.  In an
// exact model, K = 10 400: an entry of 30 rms in each row 42; rows of log-uniform
// entries over one decade, up where the other's are down, 24, over one and a half
// (infinite, as all that follow) 73, over four 2 10^4.
constexpr int ROUGH_ROWS = kRoughRows;
struct RoughRows {
  unsigned* block;
  unsigned* lowest;
  int nblk;
};
// A row's scale 2^(e - 7), sum of squares and number of zeros of its K top digits.
__device__ __forceinline__ void mark_rough(const RoughRows& g, int w, int r, double scale, long long squares, int zeros,
                                           int K) {
  if (scale == 0.0) return;  // a zero row
  const float k2 = sqrtf((float)K), rho = 128.0f * k2 / sqrtf((float)squares);
  const bool suits = isfinite(scale) && zeros <= 0x1p-8f * 1.6f * rho * K + 0.5f * k2;
  const unsigned bits = __float_as_uint(suits ? rho : INFINITY);
  atomicMax(g.block + (size_t)w * g.nblk + r / ROUGH_ROWS, bits);
  atomicMax(g.lowest, ~bits);
}

// What the split finds out about the rows besides their scales (each may be
// null): norm[w lds + r], |row r| relative to 2^e, from above (the top digits' and their
// rounding's); per batch the largest 2^e and the largest |row| (as bit patterns,
// zero on entry; a NaN is larger than all); the marked blocks of rows.
struct SplitStats {
  double* norm;
  unsigned long long* most;  // [batch][2]
  RoughRows rough;
};

// Sum over the TPR threads of a row (every thread of the block calls it).
template <int TPR>
__device__ __forceinline__ long long row_sum(int v, int* red) {
  v = __reduce_add_sync(0xffffffffu, v);
  if (TPR == 32) return v;
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  long long s = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) s += red[i];
  return s;
}

// Rows of src [batch][rows][ld] (K valid columns) -> digits
// [batch][7][rows][ldk].  TPR threads per row, blocks of 256.  lower: only the
// columns c <= r of row r are taken.
template <int TPR>
__global__ void __launch_bounds__(256) k_digit_split(const double* __restrict__ src, int rows, int K, int ld,
                                                     size_t src_stride, int lower, int8_t* __restrict__ dig, int ldk,
                                                     double* __restrict__ scale, int lds, SplitStats st) {
  static_assert(TPR == 32 || TPR == 256, "a warp or a block per row");
  constexpr int RPB = 256 / TPR;
  __shared__ unsigned long long red[8];
  __shared__ int redi[8];
  const int r = blockIdx.x * RPB + threadIdx.x / TPR, t = threadIdx.x % TPR, w = blockIdx.y;
  const bool live = r < rows;
  const double* p = src + (size_t)w * src_stride + (size_t)(live ? r : 0) * ld;
  const int lim = live ? (lower ? min(r + 1, K) : K) : 0;
  unsigned long long m = 0;
  double x[8];
  for (int k = 8 * t; k < lim; k += 8 * TPR) {
    load8(p, k, lim, x);
    m = max_bits8(x, m);
  }
  m = warp_max(m);
  if (TPR == 256) {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) m = max(m, red[i]);
  }
  const RowScale sc = digit_scale(m);
  const size_t slab = (size_t)rows * ldk;
  int8_t* d = dig + (size_t)w * 7 * slab + (size_t)r * ldk;
  // lower: the K blocks that the row's column tile reads.
  const int end = !live ? 0 : lower ? min(ldk, (r / dgt::TN + 1) * dgt::TN) : ldk;
  TopDigits top;
  for (int k = 8 * t; k < end; k += 8 * TPR) {
    load8(p, k, lim, x);
    digit_store8(x, sc, d + k, slab, top);
  }
  const long long squares = row_sum<TPR>(top.squares, redi);
  const long long zeros = TPR == 256 ? (__syncthreads(), row_sum<TPR>(top.zeros, redi)) : row_sum<TPR>(top.zeros, redi);
  if (live && t == 0) {
    scale[(size_t)w * lds + r] = sc.sc;
    const double norm = (sqrt((double)squares) + 0.5 * sqrt((double)lim)) * 0x1p-7, bound = sc.sc * 128.0;
    if (st.norm) st.norm[(size_t)w * lds + r] = norm;
    if (st.most) {
      atomicMax(st.most + 2 * w, (unsigned long long)__double_as_longlong(bound));
      atomicMax(st.most + 2 * w + 1, (unsigned long long)__double_as_longlong(bound * norm));
    }
    // (less the zeros from K to ldk)
    if (st.rough.block) mark_rough(st.rough, w, r, sc.sc, squares, (int)zeros - (end - lim), lim);
  }
}

// Rows of b [rows][ld] (K valid columns, scales sa as left by k_digit_split)
// as the integers that their digits stand for: xt[r / 32][k][r % 32] = {low word,
// high word} (rowdot::x_words), k < ldt, zero outside.  Blocks of 32 rows x 32
// columns through shared memory.
__global__ void __launch_bounds__(256) k_digit_xt(const double* __restrict__ b, int rows, int K, int ld,
                                                  const double* __restrict__ sa, int ldt, int2* __restrict__ xt) {
  __shared__ double tile[32][33];
  const int k0 = blockIdx.x * 32, r0 = blockIdx.y * 32, tx = threadIdx.x & 31;
  for (int y = threadIdx.x >> 5; y < 32; y += 8)
    tile[y][tx] = (r0 + y < rows && k0 + tx < K) ? b[(size_t)(r0 + y) * ld + k0 + tx] : 0.0;
  __syncthreads();
  // 2^(55 - e) in two factors, from the scale 2^(e - 7); zero for a row that is
  // not finite or zero.
  const double sc = r0 + tx < rows ? sa[r0 + tx] : 0.0;
  const bool fin = sc > 0.0 && isfinite(sc);
  const int k = 48 - (fin ? ilogb(sc) : 0), k1 = k >> 1;
  const double f1 = fin ? pow2i(k1) : 0.0, f2 = pow2i(k - k1);
  int2* dst = xt + ((size_t)blockIdx.y * ldt + k0) * 32;
  for (int y = threadIdx.x >> 5; y < 32; y += 8) {
    const double v = tile[tx][y];
    const rowdot::Words w = rowdot::x_words(fin ? __double2ll_rn(v * f1 * f2) : 0);
    dst[y * 32 + tx] = make_int2(w.lo, w.hi);
  }
}

// Digits of b[P][k] sqrt(chi[w][k]) for DG_R rows and DG_F frequencies per block:
// the row is read from L2 once for the frequencies, root = sqrt(chi) once for the
// rows.  The weights go to both operands of P0 by halves, which are then one: all on
// one side its rows have larger bounds (normal rows, zero frequency, K = 5270:
// 8.6 x 2^-53 instead of 6.3, for the DMMA's 9.9), and B_ov is split as well.
constexpr int DG_R = 2, DG_F = 4;
__global__ void __launch_bounds__(256, 2) k_digit_split_chi(const double* __restrict__ b, int rows, int K, int ld,
                                                         const double* __restrict__ root, int ldr, int nw,
                                                         int8_t* __restrict__ dig, int ldk,
                                                         double* __restrict__ scale, int lds, RoughRows rough) {
  constexpr int NC = DG_R * DG_F;
  __shared__ unsigned long long red[8][NC], squares[NC];
  __shared__ int zeros[NC];
  const int r0 = blockIdx.x * DG_R, w0 = blockIdx.y * DG_F;
  const int nr = min(DG_R, rows - r0), nf = min(DG_F, nw - w0);
  unsigned long long m[NC];
#pragma unroll
  for (int i = 0; i < NC; ++i) m[i] = 0;
  for (int k = 8 * threadIdx.x; k < K; k += 8 * 256) {
    double x[DG_R][8], c[8];
#pragma unroll
    for (int r = 0; r < DG_R; ++r) load8(b + (size_t)(r0 + min(r, nr - 1)) * ld, k, K, x[r]);
#pragma unroll
    for (int f = 0; f < DG_F; ++f) {
      load8(root + (size_t)(w0 + min(f, nf - 1)) * ldr, k, K, c);
#pragma unroll
      for (int r = 0; r < DG_R; ++r)
#pragma unroll
        for (int i = 0; i < 8; ++i) m[r * DG_F + f] = max(m[r * DG_F + f], abs_bits(x[r][i] * c[i]));
    }
  }
  if (threadIdx.x < NC) squares[threadIdx.x] = zeros[threadIdx.x] = 0;
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    const unsigned long long v = warp_max(m[i]);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][i] = v;
  }
  __syncthreads();
  int kexp[NC];
  TopDigits top[NC];
  double my_scale = 0.0;  // of combination threadIdx.x
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    unsigned long long v = 0;
    double scale_i;
#pragma unroll
    for (int j = 0; j < 8; ++j) v = max(v, red[j][i]);
    kexp[i] = digit_scale(v, scale_i);
    if (threadIdx.x == i) my_scale = scale_i;
  }
  const size_t slab = (size_t)rows * ldk;
  for (int k = 8 * threadIdx.x; k < ldk; k += 8 * 256) {
    double x[DG_R][8], c[8], y[8];
#pragma unroll
    for (int r = 0; r < DG_R; ++r) load8(b + (size_t)(r0 + min(r, nr - 1)) * ld, k, K, x[r]);
#pragma unroll
    for (int f = 0; f < DG_F; ++f) {
      if (f >= nf) break;
      load8(root + (size_t)(w0 + f) * ldr, k, K, c);
#pragma unroll
      for (int r = 0; r < DG_R; ++r) {
        if (r >= nr) break;
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] = x[r][i] * c[i];
        digit_store8(y, scale_factors(kexp[r * DG_F + f]), dig + (size_t)(w0 + f) * 7 * slab + (size_t)(r0 + r) * ldk + k,
                     slab, top[r * DG_F + f]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    const int q = __reduce_add_sync(0xffffffffu, top[i].squares), n = __reduce_add_sync(0xffffffffu, top[i].zeros);
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&squares[i], (unsigned long long)q);
      atomicAdd(&zeros[i], n);
    }
  }
  __syncthreads();
  if (threadIdx.x < NC) {
    const int r = threadIdx.x / DG_F, f = threadIdx.x % DG_F;
    if (r < nr && f < nf) {
      scale[(size_t)(w0 + f) * lds + r0 + r] = my_scale;
      // (less the zeros from K to ldk)
      mark_rough(rough, w0 + f, r0 + r, my_scale, (long long)squares[threadIdx.x], zeros[threadIdx.x] - (ldk - K), K);
    }
  }
}

// root[w][k] = sqrt(chi[w][k])
__global__ void k_digit_root(const double* __restrict__ chi, size_t n, double* __restrict__ root) {
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
    root[k] = sqrt(chi[k]);
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
// Digits [slabs][rows][ldk], box 128 bytes x box_rows with the 128-byte swizzle.
static CUtensorMap digit_map(const int8_t* base, int K, int rows, int ldk, int slabs, int box_rows) {
  QX_REQUIRE((reinterpret_cast<uintptr_t>(base) & 15) == 0 && ldk % 16 == 0, QX_ERR_INVALID_INPUT,
             "digit map base/stride not 16-byte aligned");
  CUtensorMap m;
  cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)slabs};
  cuuint64_t strides[2] = {(cuuint64_t)ldk, (cuuint64_t)ldk * rows};
  cuuint32_t box[3] = {(cuuint32_t)dgt::BK, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<int8_t*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  QX_REQUIRE(r == CUDA_SUCCESS, QX_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return m;
}

template <int MODE>
static void launch_digit_gemm(qx_ctx* ctx, const int8_t* a, int lda, const int8_t* b, int ldb, DigitArgs args) {
  args.rowdot = MODE == DIGIT_ROWDOT;
  args.lower = MODE == DIGIT_LOWER;
  const CUtensorMap ma = digit_map(a, args.K, args.M, lda, MODE == DIGIT_LOWER ? dgt::NS * args.nbatch : dgt::NS, dgt::TM);
  const CUtensorMap mb = digit_map(b, args.K, args.N, ldb, dgt::NS * args.nbatch, dgt::TN / 2);
  QX_REQUIRE(args.K > 0 && args.K <= dgt::KMAX, QX_ERR_INVALID_INPUT, "digit GEMM: K = %d", args.K);
  args.sh = 0;
  while ((256 << args.sh) < args.K) ++args.sh;
  args.err = status_words(ctx, 1);
  QX_CUDA(cudaMemsetAsync(args.err, 0, sizeof(int), ctx->stream));
  static PerDeviceOnce attr_once;
  static int max_clusters[PerDeviceOnce::kMaxDevices] = {};
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(dgt::THREADS);
  cfg.dynamicSmemBytes = dgt::TOTAL;
  cfg.stream = ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  attr_once(ctx->device, [&] {
    QX_CUDA(cudaFuncSetAttribute(k_digit_gemm<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, dgt::TOTAL));
    cfg.gridDim = dim3(2 * ctx->sm_count);
    int n = 0;
    QX_CUDA(cudaOccupancyMaxActiveClusters(&n, k_digit_gemm<MODE>, &cfg));
    max_clusters[ctx->device] = std::max(n, 1);
  });
  const int T = ceil_div(args.M, dgt::TM), NT = ceil_div(args.N, dgt::TN);
  const long long items =
      args.rowdot ? (long long)ceil_div(args.nbatch, args.wgroup) * ceil_div(T, 2) * args.wgroup * NT
                  : (long long)(args.lower ? digit_lower_pairs(T) : ceil_div(T, 2) * NT) * args.nbatch;
  QX_REQUIRE(items > 0 && items < (1ll << 30), QX_ERR_INVALID_INPUT, "digit GEMM: %lld tiles", items);
  cfg.gridDim = dim3(2 * (unsigned)std::min<long long>(items, max_clusters[ctx->device]));
  QX_CUDA(cudaLaunchKernelEx(&cfg, k_digit_gemm<MODE>, ma, mb, args));
  check_launch(ctx);
  ctx->pending.push_back({args.err, 1, 0});
}

// Reserve without throwing: false when the device has no room (the caller
// then takes the DMMA kernels, which need no operand copies).
static bool try_reserve(DevBuf& b, size_t bytes) {
  try {
    b.reserve(bytes);
    return true;
  } catch (const Error&) {
    cudaGetLastError();
    return false;
  }
}

static void split_rows(qx_ctx* ctx, const double* src, int rows, int K, int ld, size_t stride, int batch, int lower,
                       int8_t* dig, int ldk, double* scale, int lds, SplitStats st = {}) {
  if (K <= 2048)
    k_digit_split<32><<<dim3(ceil_div(rows, 8), batch), 256, 0, ctx->stream>>>(src, rows, K, ld, stride, lower, dig,
                                                                             ldk, scale, lds, st);
  else
    k_digit_split<256><<<dim3(rows, batch), 256, 0, ctx->stream>>>(src, rows, K, ld, stride, lower, dig, ldk, scale,
                                                                   lds, st);
  check_launch(ctx);
}

// ---------------------------------------------------------------------------
// Workspace.  A context holds at most its limit over the four slots: 3/8 for the
// batched operand's digits (WS_DIG_B), 1/4 for the other's (WS_DIG_A), 3/8 for the
// rest (scales, the pairs' integers and partial sums).  Larger problems run in
// chunks.  By default one frequency and 256 rows are always taken; within a limit
// that the caller has set, a product whose smallest chunk does not fit takes the
// DMMA kernels.  Chunks do not change a result: frequencies and rows are
// independent.
// ---------------------------------------------------------------------------
// 4 GB: P0 at nmo 300 / naux 1000 / 32 frequencies takes two chunks, its contraction of
// all pairs one.  Batch workers share the device: 1.25 GB.
size_t digit_limit(const qx_ctx* ctx) {
  return ctx->digit_limit ? ctx->digit_limit : ctx->worker ? (size_t)1280 << 20 : (size_t)4096 << 20;
}
struct DigitPlan {
  int fc = 0, rows = 0;       // frequencies and rows (pairs, or of A) per chunk; none: 0
  size_t a = 0, b = 0, s = 0, p = 0;  // bytes of the slots
};

static DigitPlan plan_p0(int naux, int nov, int ldov, int nw, size_t limit, bool strict) {
  DigitPlan d;
  const int ldk = round_up(nov, 16), lds = round_up(naux, dgt::TN), nblk = ceil_div(naux, ROUGH_ROWS);
  const size_t per = (size_t)7 * naux * ldk, per_s = ((size_t)lds + ldov + nblk) * sizeof(double);
  size_t f = std::min(limit / 8 * 3 / per, limit / 8 * 3 / per_s);
  if (f == 0 && strict) return d;
  f = std::max<size_t>(1, std::min<size_t>(f, nw));
  d.fc = ceil_div(nw, ceil_div(nw, (int)f));
  d.b = per * d.fc;
  d.s = per_s * d.fc + 64;
  return d;
}

static DigitPlan plan_contract(int npair, int naux, int nw, size_t limit, bool strict) {
  DigitPlan d;
  const int lds = round_up(naux, dgt::TN), NT = lds / dgt::TN;
  const size_t row = (size_t)7 * round_up(naux, 16), third = limit / 8 * 3;
  size_t f = third / (row * naux);
  if (f == 0 && strict) return d;
  d.fc = (int)std::max<size_t>(1, std::min<size_t>(f, nw));
  // Per pair: digits; partial sums, integers, scale, norm and list entries.
  const size_t per_p = ((size_t)2 * NT * d.fc + lds) * sizeof(double);
  const size_t fixed_s = ((size_t)(2 * lds + 2) * d.fc + 2) * sizeof(double);
  const size_t per_s = 2 * sizeof(double) + (size_t)ceil_div(d.fc, REDO_ROWS / (int)sizeof(int));
  size_t r = fixed_s < third ? std::min(limit / 4 / row, (third - fixed_s) / (per_p + per_s)) / 256 * 256 : 0;
  if (r == 0 && strict && npair > 0) {
    d.fc = 0;
    return d;
  }
  r = std::max<size_t>(256, r);
  d.rows = (int)std::min<size_t>(r, npair);
  const size_t padded = round_up(d.rows, 256);
  d.a = row * d.rows;
  d.b = row * naux * d.fc;
  d.p = ((size_t)2 * NT * d.fc * d.rows + padded * lds) * sizeof(double);
  d.s = fixed_s + (size_t)2 * d.rows * sizeof(double) + (size_t)ceil_div(d.rows, REDO_ROWS) * d.fc * sizeof(int);
  return d;
}

size_t digit_workspace_bytes(int naux, int nov, int npair, int nw, size_t limit) {
  const int ldov = round_up(nov, 8);
  const DigitPlan p0 = digits_for_p0(naux, nov) ? plan_p0(naux, nov, ldov, nw, limit, false) : DigitPlan{};
  const DigitPlan pc = digits_for_contraction(naux) ? plan_contract(npair, naux, nw, limit, false) : DigitPlan{};
  return std::max(p0.b, pc.b) + std::max(p0.s, pc.s) + pc.a + pc.p;
}

// From where the integer tensor pipe is the faster one: with 24 frequencies P0 took
// 137 (DMMA) and 152 us (digits) at naux 300 / nov 949, 295 and 209 us at 350 / 1411, 474
// and 264 us at 423 / 2020.  From K = 1024 on its error is half the DMMA's or less.
bool digits_for_p0(int naux, int nov) { return naux >= 256 && nov >= 1024; }

// eps[w] = I + B_ov diag(chi'[w]) B_ov^T, chi' >= 0.
bool launch_eps_digits(qx_ctx* ctx, const double* bov, int ldov, int naux, int nov, const double* chi, int nw,
                       double* eps, int ldn, size_t eps_stride) {
  const DigitPlan plan = plan_p0(naux, nov, ldov, nw, digit_limit(ctx), ctx->digit_limit != 0);
  if (!plan.fc) return false;
  const int ldk = round_up(nov, 16), fc = plan.fc;
  DevBuf &db = ctx->ws[WS_DIG_B], &ds = ctx->ws[WS_DIG_S];
  const int lds = round_up(naux, dgt::TN), nblk = ceil_div(naux, ROUGH_ROWS);
  const size_t n_scale = (size_t)lds * fc, n_flag = (size_t)nblk * fc + 1, n_root = (size_t)ldov * fc;
  if (!try_reserve(db, plan.b) || !try_reserve(ds, plan.s)) return false;
  // Roots of the weights; scales and the rows' rho (zeroed together).
  double* root = ds.as<double>();
  double* sb = root + n_root;
  unsigned* marks = reinterpret_cast<unsigned*>(sb + n_scale);
  const RoughRows rough{marks + 1, marks, nblk};
  const float limit = 6.25f * std::sqrt((float)nov);
  for (int w0 = 0; w0 < nw; w0 += fc) {
    const int n = std::min(fc, nw - w0);
    QX_CUDA(cudaMemsetAsync(sb, 0, n_scale * sizeof(double) + n_flag * sizeof(int), ctx->stream));
    const size_t nr = (size_t)n * ldov;
    k_digit_root<<<(unsigned)std::min<size_t>((nr + 255) / 256, 2048), 256, 0, ctx->stream>>>(
        chi + (size_t)w0 * ldov, nr, root);
    check_launch(ctx);
    k_digit_split_chi<<<dim3(ceil_div(naux, DG_R), ceil_div(n, DG_F)), 256, 0, ctx->stream>>>(
        bov, naux, nov, ldov, root, ldov, n, db.as<int8_t>(), ldk, sb, lds, rough);
    check_launch(ctx);
    DigitArgs a{};
    a.M = a.N = naux;
    a.nbatch = n;
    a.scaleA = a.scaleB = sb;
    a.ldsb = lds;
    a.out = eps + (size_t)w0 * eps_stride;
    a.ldo = ldn;
    a.out_stride = eps_stride;
    a.lowA = a.lowB = rough.lowest;
    a.rough_limit = limit;
    for (int k0 = 0; k0 < nov; k0 += dgt::KMAX) {
      a.K = std::min(dgt::KMAX, nov - k0);
      a.add = k0 > 0;
      launch_digit_gemm<DIGIT_LOWER>(ctx, db.as<int8_t>() + k0, ldk, db.as<int8_t>() + k0, ldk, a);
    }
    // The tiles above the limit by the DMMA kernel.
    launch_eps_dmma(ctx, bov, ldov, naux, nov, chi + (size_t)w0 * ldov, n, eps + (size_t)w0 * eps_stride, ldn,
                    eps_stride, rough.block, limit);
  }
  return true;
}

// C[m][n] = sum_k A[m][k] B[n][k].  The rows are read two entries at a time:
// operands that are not 16-byte aligned with even leading dimensions are left to
// the caller's other path, which refuses them.
bool gemm_nt_digits(qx_ctx* ctx, const double* A, int M, int lda, const double* B, int N, int ldb, int K, double* C,
                    int ldc) {
  // From K = 161 on (two K blocks) and a few tiles each way: below, the
  // padding and the digits cost what the faster products give.
  if (K <= 160 || K > dgt::KMAX || M < 2 * dgt::TM || N < 2 * dgt::TN) return false;
  if (lda % 2 || ldb % 2 || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return false;
  const int ldd = round_up(K, 16);
  const size_t row = (size_t)7 * ldd, limit = digit_limit(ctx);
  const int rows_a = (int)std::min<size_t>(limit / 4 / row, 1u << 30) / 256 * 256;
  const int rows_b = (int)std::min<size_t>(limit / 8 * 3 / row, 1u << 30) / 256 * 256;
  if (ctx->digit_limit && (rows_a == 0 || rows_b == 0)) return false;
  const int mc = std::min(M, std::max(256, rows_a)), nc = std::min(N, std::max(256, rows_b));
  const int lds = round_up(nc, dgt::TN), blkA = ceil_div(mc, ROUGH_ROWS), blkB = ceil_div(nc, ROUGH_ROWS);
  DevBuf &da = ctx->ws[WS_DIG_A], &db = ctx->ws[WS_DIG_B], &ds = ctx->ws[WS_DIG_S];
  const size_t b_bytes = lds * sizeof(double) + (size_t)round_up(blkB + 1, 2) * sizeof(int);
  const size_t a_bytes = mc * sizeof(double) + (size_t)(blkA + 1) * sizeof(int);
  if (!try_reserve(da, row * mc) || !try_reserve(db, row * nc) || !try_reserve(ds, b_bytes + a_bytes)) return false;
  // Scales of B and its rows' rho; the same of A.
  double* sb = ds.as<double>();
  unsigned* mb = reinterpret_cast<unsigned*>(sb + lds);
  double* sa = reinterpret_cast<double*>(ds.as<char>() + b_bytes);
  unsigned* ma = reinterpret_cast<unsigned*>(sa + mc);
  const RoughRows ra{ma + 1, ma, blkA}, rb{mb + 1, mb, blkB};
  for (int n0 = 0; n0 < N; n0 += nc) {
    const int n = std::min(nc, N - n0);
    QX_CUDA(cudaMemsetAsync(sb, 0, b_bytes, ctx->stream));
    split_rows(ctx, B + (size_t)n0 * ldb, n, K, ldb, 0, 1, 0, db.as<int8_t>(), ldd, sb, lds, {nullptr, nullptr, rb});
    for (int m0 = 0; m0 < M; m0 += mc) {
      const int m = std::min(mc, M - m0);
      if (n0 == 0 || mc < M) {
        QX_CUDA(cudaMemsetAsync(ma, 0, (size_t)(blkA + 1) * sizeof(int), ctx->stream));
        split_rows(ctx, A + (size_t)m0 * lda, m, K, lda, 0, 1, 0, da.as<int8_t>(), ldd, sa, 0, {nullptr, nullptr, ra});
      }
      DigitArgs a{};
      a.M = m;
      a.N = n;
      a.K = K;
      a.nbatch = 1;
      a.scaleA = sa;
      a.scaleB = sb;
      a.ldsb = lds;
      a.out = C + (size_t)m0 * ldc + n0;
      a.ldo = ldc;
      a.wide = ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 31) == 0;
      a.lowA = ma;
      a.lowB = mb;
      // The adjoint's rows of G have a large diagonal (rho 5 to 20): a matrix X X^T of
      // 400 columns times normal rows, K = 700, err by 10 (the DMMA's sums by 8.6, in
      // 2^-53 of the root-sum-square), its elements of rho rho' = 6 to 10 sqrt(K), 4 %
      // of them, by 19.  The gradient's error is the same either way (1.2 to 1.6 e-15).
      a.rough_limit = 10.0f * std::sqrt((float)K);
      launch_digit_gemm<DIGIT_PLAIN>(ctx, da.as<int8_t>(), ldd, db.as<int8_t>(), ldd, a);
      // The tiles above the limit by the DMMA kernel.
      GemmNT g{};
      g.M = m;
      g.N = n;
      g.K = K;
      g.A = A + (size_t)m0 * lda;
      g.lda = lda;
      g.B = B + (size_t)n0 * ldb;
      g.ldb = ldb;
      g.C = a.out;
      g.ldc = ldc;
      g.batch = 1;
      g.alpha = 1.0;
      g.splitk = 1;
      g.roughA = ra.block;
      g.roughB = rb.block;
      g.rough_limit = a.rough_limit;
      gemm_nt_f64(ctx, g);
    }
  }
  return true;
}

// The integer tensor pipe above one column tile: with 24 frequencies the
// contraction took 44 (DMMA) and 32 us (digits) at naux 139 with 160 pairs, 72 and 35
// us at naux 196 with 224, 178 and 84 us with 3136; at naux 86 the DMMA kernel was the
// faster one (24 against 27 us).  Its five launches more cost ~15 us on the host, so
// the line is drawn at 160.
bool digits_for_contraction(int naux) { return naux > 160 && naux <= dgt::KMAX; }

// v[w][p] = Bpt[p]^T Wc[w] Bpt[p] from W' (half-lower Wc).
bool launch_pair_contract_digits(qx_ctx* ctx, const double* bpt, int ldk, int npair, int naux, const double* wc,
                                 int ldn, size_t wc_stride, int nw, double* v, int ldv) {
  const DigitPlan plan = plan_contract(npair, naux, nw, digit_limit(ctx), ctx->digit_limit != 0);
  if (!plan.fc) return false;
  const int ldd = round_up(naux, 16), NT = ceil_div(naux, dgt::TN), fc = plan.fc, pc = plan.rows;
  const size_t row = (size_t)7 * ldd;
  const int lds = NT * dgt::TN;
  DevBuf &da = ctx->ws[WS_DIG_A], &db = ctx->ws[WS_DIG_B], &ds = ctx->ws[WS_DIG_S], &dp = ctx->ws[WS_DIG_P];
  if (!try_reserve(da, plan.a) || !try_reserve(db, plan.b) || !try_reserve(ds, plan.s) || !try_reserve(dp, plan.p))
    return false;
  int2* xt = reinterpret_cast<int2*>(dp.as<double>() + (size_t)2 * NT * fc * pc);
  // Scales of W', its largest bounds and norms, the count of the listed blocks (zeroed
  // together), its norms; scales and norms of the pairs, the list of blocks.
  double* sb = ds.as<double>();
  unsigned long long* most = reinterpret_cast<unsigned long long*>(sb + (size_t)lds * fc);
  int* redo_count = reinterpret_cast<int*>(most + 2 * fc);
  double* norm_w = reinterpret_cast<double*>(redo_count + 2);
  double* sa = norm_w + (size_t)lds * fc;
  double* norm = sa + pc;
  int* redo = reinterpret_cast<int*>(norm + pc);
  for (int p0 = 0; p0 < npair; p0 += pc) {
    const int np = std::min(pc, npair - p0);
    split_rows(ctx, bpt + (size_t)p0 * ldk, np, naux, ldk, 0, 1, 0, da.as<int8_t>(), ldd, sa, 0, {norm, nullptr, {}});
    k_digit_xt<<<dim3(lds / 32, ceil_div(np, 32)), 256, 0, ctx->stream>>>(bpt + (size_t)p0 * ldk, np, naux, ldk, sa, lds,
                                                                           xt);
    check_launch(ctx);
    for (int w0 = 0; w0 < nw; w0 += fc) {
      const int n = std::min(fc, nw - w0);
      if (p0 == 0 || fc < nw) {
        QX_CUDA(cudaMemsetAsync(sb, 0, ((size_t)(lds + 2) * fc + 1) * sizeof(double), ctx->stream));
        split_rows(ctx, wc + (size_t)w0 * wc_stride, naux, naux, ldn, wc_stride, n, 1, db.as<int8_t>(), ldd, sb, lds,
                   {norm_w, most, {}});
      } else {
        QX_CUDA(cudaMemsetAsync(redo_count, 0, sizeof(int), ctx->stream));
      }
      DigitArgs a{};
      a.M = np;
      a.N = naux;
      a.K = naux;
      a.nbatch = n;
      a.scaleA = sa;
      a.scaleB = sb;
      a.ldsb = lds;
      a.xt = xt;
      // Digits of W' of a frequency group within half of L2.
      a.wgroup = (int)std::max<size_t>(1, std::min<size_t>(n, ((size_t)60 << 20) / (row * naux)));
      a.part = dp.as<double>();
      launch_digit_gemm<DIGIT_ROWDOT>(ctx, da.as<int8_t>(), ldd, db.as<int8_t>(), ldd, a);
      const DigitCheck ck{sa, norm, most, 0.82 * std::sqrt((double)naux), redo_count, redo};
      k_digit_rowdot_sum<<<dim3(std::min(ceil_div(np, 256), 512), n), 256, 0, ctx->stream>>>(
          dp.as<double>(), 2 * NT, np, n, v + (size_t)w0 * ldv + p0, ldv, ck);
      check_launch(ctx);
      launch_pair_contract_redo(ctx, bpt + (size_t)p0 * ldk, ldk, np, naux, wc + (size_t)w0 * wc_stride, ldn, wc_stride,
                                n, v + (size_t)w0 * ldv + p0, ldv,
                                {redo_count, redo, sa, norm, sb, norm_w, lds, dp.as<double>(), 2 * NT});
    }
  }
  return true;
}

}  // namespace qx
