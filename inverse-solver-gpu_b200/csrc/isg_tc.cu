// Tensor-core engine for the dense leaf stages of the MLFMA matvec on sm_100a.
//
// Near field + L2P (kernels.cu:32-81, 292-319; solve.cpp:170-216) and P2M
// (kernels.cu:6-30; solve.cpp:80-92) are complex GEMMs with a shared,
// translation-invariant operand.  Each runs as a real GEMM through the
// embedding [re, im] x [[re, -im], [im, re]] on tcgen05 (kind::f16, FP32
// accumulation in TMEM).  FP32 accuracy comes from splitting both operands
// into FP16 pairs, v = hi + lo, after a power-of-two scaling of each tile into
// the FP16 range, and summing hi*hi + hi*lo + lo*hi (the lo*lo term is below
// FP32 rounding).
//
// Near-field CTA: 8, 16 or 32 x 8 leaves of one RHS.  Its halo of leaves is stored
// in shared memory in the K-major core-matrix layout [halo row][16-byte K chunk]
// [halo column], so the operand of each of the nine neighbour slots is the same
// halo seen through a descriptor shifted by one halo row / column.  The weights (9
// slots x 128 x 128 reals, then the L2P basis) stream through a ring of 16 KB stages
// filled by bulk async copies.
#include <cmath>
#include <cstring>
#include <vector>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "isg_context.hpp"
#include "isg_tc.cuh"

namespace isg {

namespace {

using namespace tc;

constexpr int kTX = 8, kTRMax = 32;              // leaf columns and most leaf rows of a near-field item
constexpr int kHR = kTRMax + 2, kHC = kTX + 2;   // its 34 x 10 halo
constexpr int kStageBytes = 16384;               // hi [128 x 32] + lo [128 x 32]
constexpr int kStageHalf = 8192;
constexpr int kNearStages = 36;                  // 9 slots x 4 K-chunks of 32 reals
constexpr int kLeafSampMax = 80;                 // samples of a leaf ring
constexpr int kErrNear = 101, kErrP2m = 111;

__device__ __forceinline__ float cabs1(float2 v) { return fmaxf(fabsf(v.x), fabsf(v.y)); }

// ---- near field + L2P, persistent and pipelined ----
// Items are TR x 8 leaves of one RHS (TR = 32, or 16 or 8 where 32 would leave
// SMs without an item, np_rows); a persistent CTA walks them in steps of
// gridDim.x.  An item's K dimension (9 neighbour slots x 128 source reals of
// the halo, then 2 ns reals of the leaf locals for L2P) is staged in shared
// memory one A-stage at a time: a halo K-group (32 source reals of every leaf
// of the item's (TR + 2) x 10-leaf halo) feeds the nine weight stages of its K
// range; an L2P stage (32 reals of the locals of the item's 8 TR leaves) feeds
// one.  Stage order: H0 H1 H2 H3 L0 ..
// L4; the weights are packed in the same order.  An A-stage arrives as FP32 by
// one tensor load whose rows are a leaf's 32 reals (128 contiguous bytes) into
// a staging buffer, and the converters write it as FP16 hi/lo in the MMA's
// core-matrix layout into an operand buffer.  The whole halo is never
// resident, so two staging buffers, two operand buffers and a three-deep
// weight ring fit in shared memory and the roles overlap:
//   warp 0      tensor loads of the A-stages (4-D maps, no multicast)
//   warp 1      bulk copies of the weight stages
//   warp 2      MMA issue (one elected lane)
//   warps 3..6  A-stage conversion to FP16 hi/lo
//   warps 7..14 epilogue, two per TMEM lane quarter (an item's upper and lower leaf rows)
// Near field and L2P accumulate into one TMEM accumulator per item: the input
// is scaled by the power of two that P2M's per-RHS maximum gives and the
// locals by M2L's, each lowered until both products carry the same power of
// two.  Two accumulator sets (256 columns each) alternate between
// items, so an item's epilogue runs under the next item's MMAs.
// Shared memory bounds the large items: the MMAs read 12 KB for their 128 cycles, and
// tensor loads, weight stages and converters come on top.  Both operand kinds are
// written at the halo's pitch of 10 leaves and read in an order that keeps a phase's
// lanes on different banks: 1024 x 1024 x 64 1185 -> 1086 us, 256 x 256 x 64 105.5 -> 101.5
// (L2P stages at a pitch of 8 leaves were 4-way conflicts).
constexpr int kNpKC = 4;                                       // 8-real K-chunks per A-stage
constexpr int kNpHaloSplit = kHR * kNpKC * kHC * 16;           // 21760: one FP16 split of a halo K-group
constexpr int kNpBuf = 2 * kNpHaloSplit;                       // 43520: an operand (hi, lo) or a staged A-stage
constexpr int kNpHaloBytes = kHR * kHC * 32 * 4;               // 43520: a halo K-group as FP32
constexpr int kNpL2pBytes = kTRMax * kTX * 32 * 4;             // 32768: an L2P stage as FP32
constexpr int kNpNS = 2, kNpNO = 2, kNpNB = 3;                 // staging, operand buffers, weight ring depth
constexpr int kNpConvWarp0 = 3, kNpConvWarps = 4, kNpEpiWarp0 = 7, kNpEpiWarps = 8;
constexpr int kNpThreads = 32 * (kNpEpiWarp0 + kNpEpiWarps);  // 480
constexpr int kNpConv = 32 * kNpConvWarps, kNpEpi = 32 * kNpEpiWarps;
struct NpSmem {
  static constexpr int s = 0;                                  // kNpNS FP32 staging buffers
  static constexpr int o = kNpNS * kNpBuf;                     // kNpNO FP16 hi/lo operand buffers
  static constexpr int b = o + kNpNO * kNpBuf;                 // kNpNB weight stages
  static constexpr int bars = b + kNpNB * kStageBytes;         // 19 mbarriers
  static constexpr int misc = bars + 24 * 8;                   // TMEM base, abort flag
  static constexpr int dscr = misc + 16;                       // [2][kNpEpiWarps][3] double
  static constexpr int total = dscr + 2 * kNpEpiWarps * 3 * 8;
};
static_assert(kNpBuf % 128 == 0 && NpSmem::o % 128 == 0, "tensor-load destinations are 128-byte aligned");
static_assert(kNpHaloBytes <= kNpBuf && kNpL2pBytes <= kNpBuf, "buffer sizes");
static_assert(NpSmem::total <= 227 * 1024, "shared memory of one CTA");

// A-stage a of an item: returns 0 (halo K-group a, a < 4) or 1 (L2P stage
// a - 4) and its index.  The L2P stages come last: tensor-core accumulation
// rounds each step against the running sum, and interleaving the L2P terms
// into the near-field sum measured 2x the operator error (5.5e-6 against
// 2.5e-6 relative to FP64 on random inputs).
__host__ __device__ inline int np_stage(int a, int &idx) {
  idx = a < 4 ? a : a - 4;
  return a < 4 ? 0 : 1;
}

// A dot product's terms over one epilogue chunk at FP32 instruction cost:
// each product a b is split exactly into its rounded value p and its rounding
// error fma(a, b, -p) (Dekker's TwoProduct); the p go round-robin into four
// independent FP32 partial sums (short dependency chains), the errors into a
// fifth, and the five are added into the FP64 sum once per chunk.  Each
// partial sum rounds three times over a 16-term chunk, below the rounding of
// the complex64 vectors themselves; the _rn intrinsics keep the compiler from
// contracting the exact split.  (Converting every product to FP64 cost 1.75
// ms of a 4.4 ms 256-RHS launch; Kahan compensation, a four-add dependency
// chain per term, cost more than that.)
struct Acc32 {
  float p[4] = {0.f, 0.f, 0.f, 0.f}, e = 0.f;
  __device__ __forceinline__ void add_prod(int j, float a, float b) {
    const float q = __fmul_rn(a, b);
    e = __fadd_rn(e, fmaf(a, b, -q));
    p[j & 3] = __fadd_rn(p[j & 3], q);
  }
  __device__ __forceinline__ double take() {
    const double v = (((double)p[0] + (double)p[1]) + ((double)p[2] + (double)p[3])) + (double)e;
    p[0] = p[1] = p[2] = p[3] = e = 0.f;
    return v;
  }
};

struct TcNearArgs {
  const float2 *x, *g;  // operator input (transformed by mode)
  const float2 *xe;     // x of the `x - ...` epilogue
  int64_t gstride;
  int mode;
  const int *active;
  const uint8_t *B;  // weight stages in A-stage order
  int nl2p;
  float sw, sb;      // power-of-two scales of the near-field weights and the L2P basis
  const unsigned *levmax, *locmax;  // [R][kLevStride]: P2M's input maximum (slot kInMaxSlot), M2L's locals
  int lvl_leaf;
  float2 *y;
  int epi, red;
  const float2 *dot_a;
  double *part;
  int nleaf, U, tiles_x, ppr, nitems;  // items of TR x kTX leaves: columns, per RHS, in all
  int *err;
};

// The item's operand scales: input s1 and locals s2 lowered to a common product scale p = s1 sw = s2 sb.
// A zero maximum (an all-zero input or locals) leaves the other operand's scale alone.
__device__ __forceinline__ void np_scales(const TcNearArgs &A, int rhs, float &s1, float &s2, float &p) {
  const float mx = __uint_as_float(A.levmax[rhs * kLevStride + kInMaxSlot]);
  const float ml = __uint_as_float(A.locmax[rhs * kLevStride + A.lvl_leaf]);
  const float a = mx > 0.f ? pow2_scale(mx) * A.sw : INFINITY;
  const float b = ml > 0.f ? pow2_scale(ml) * A.sb : INFINITY;
  p = fminf(a, b);
  if (!(p < INFINITY)) p = A.sw;
  s1 = p / A.sw;
  s2 = p / A.sb;
}

template <int TR>
__global__ void __launch_bounds__(kNpThreads, 1) k_tc_near_pipe(TcNearArgs A, const __grid_constant__ CUtensorMap tmh,
                                                                const __grid_constant__ CUtensorMap tml) {
  extern __shared__ __align__(1024) char sm[];
  uint64_t *sfull = (uint64_t *)(sm + NpSmem::bars);  // staging landed / read out
  uint64_t *sfree = sfull + kNpNS;
  uint64_t *ofull = sfree + kNpNS, *ofree = ofull + kNpNO;  // operand converted / consumed by the MMAs
  uint64_t *bfull = ofree + kNpNO, *bempty = bfull + kNpNB;
  uint64_t *tfull = bempty + kNpNB, *tfree = tfull + 2, *mdone = tfree + 2;
  uint32_t *tslot = (uint32_t *)(sm + NpSmem::misc);
  volatile int *abort = (volatile int *)(sm + NpSmem::misc + 4);
  double *dscr = (double *)(sm + NpSmem::dscr);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * kNpNS + 2 * kNpNO + 2 * kNpNB + 5; i++) mbar_init(sfull + i, 1);
    *abort = 0;
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(tslot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;  // set s: columns [256 s, +8 TR)
  const int na = 4 + A.nl2p;     // A-stages per item
  const int nb = 36 + A.nl2p;    // weight stages per item
  auto next_item = [&](int w) {
    do w += gridDim.x;
    while (w < A.nitems && A.active && !A.active[w / A.ppr]);
    return w;
  };
  const int blk = blockIdx.x + grid_wait();
  const int first = (A.active && blk < A.nitems && !A.active[blk / A.ppr]) ? next_item(blk) : blk;
  auto geom = [&](int w, int &rhs, int &ty0, int &tx0) {
    rhs = w / A.ppr;
    const int pr = w % A.ppr, pty = pr / A.tiles_x, ptx = pr % A.tiles_x;
    ty0 = pty * TR;
    tx0 = ptx * kTX;
  };
  const uint32_t halo_bytes = (uint32_t)(TR + 2) * kHC * 32 * 4, l2p_bytes = (uint32_t)TR * kTX * 32 * 4;

  if (warp == 0) {
    // ---- A-stage tensor loads into the staging buffers: rows of 32 reals ----
    if (lane == 0) {
      int ka = 0;
      const bool pre_x = A.epi == EPI_FWD || A.epi == EPI_ADJ || A.red == RED_TS;
      for (int w = first; w < A.nitems && !*abort; w = next_item(w)) {
        int rhs, ty0, tx0;
        geom(w, rhs, ty0, tx0);
        // the rows the epilogue will read for this item (x, the dot vector, g), into L2
        // about one item ahead of it: its loads then wait on L2, not on HBM
        {
          const uint32_t run = (uint32_t)min(kTX, A.nleaf - tx0) * kBB * 8;
          const size_t rb = (size_t)rhs * A.U;
          for (int r = 0; r < TR && ty0 + r < A.nleaf; r++) {
            const size_t at = (size_t)((ty0 + r) * A.nleaf + tx0) * kBB;
            if (pre_x) bulk_prefetch_l2(A.xe + rb + at, run);
            if (A.red == RED_DOT) bulk_prefetch_l2(A.dot_a + rb + at, run);
            if (A.epi == EPI_ADJ) bulk_prefetch_l2(A.g + rhs * A.gstride + at, run);
          }
        }
        for (int a = 0; a < na; a++, ka++) {
          const int i = ka % kNpNS;
          if (!mbar_wait_or(sfree + i, ((ka / kNpNS) & 1) ^ 1, abort, A.err, kErrNear)) break;
          char *dst = sm + NpSmem::s + i * kNpBuf;
          int idx;
          if (np_stage(a, idx) == 0) {
            mbar_expect_tx(sfull + i, halo_bytes);
            tma_load_4d(dst, &tmh, 32 * idx, tx0 - 1, ty0 - 1, rhs, sfull + i);
          } else {
            mbar_expect_tx(sfull + i, l2p_bytes);
            tma_load_4d(dst, &tml, 32 * idx, tx0, ty0, rhs, sfull + i);
          }
        }
      }
      // every load issued has landed before the CTA exits (bounded waits)
      for (int j = 1; j <= kNpNS && j <= ka; j++) {
        const int kk = ka - j;
        mbar_wait(sfull + kk % kNpNS, (kk / kNpNS) & 1, A.err, kErrNear);
      }
    }
  } else if (warp == 1) {
    // ---- weight stages through the ring, in A-stage order ----
    if (lane == 0) {
      int kb = 0;
      for (int w = first; w < A.nitems && !*abort; w = next_item(w)) {
        for (int t = 0; t < nb; t++, kb++) {
          const int b = kb % kNpNB;
          if (!mbar_wait_or(bempty + b, ((kb / kNpNB) & 1) ^ 1, abort, A.err, kErrNear)) break;
          mbar_expect_tx(bfull + b, kStageBytes);
          bulk_g2s(sm + NpSmem::b + b * kStageBytes, A.B + (size_t)t * kStageBytes, kStageBytes, bfull + b);
        }
      }
      for (int j = 1; j <= kNpNB && j <= kb; j++) {
        const int kk = kb - j;
        mbar_wait(bfull + kk % kNpNB, (kk / kNpNB) & 1, A.err, kErrNear);
      }
    }
  } else if (warp == 2) {
    // ---- MMA issue (the warp waits, one elected lane issues): D[128 target
    // reals][8 TR leaves of the item] += weights (A, M = 128) x data (B, N = 8 TR):
    // each weight stage is 2 K-steps x 3 split products.  A wait that expires may do so in
    // some lanes only, so the warp votes once per weight stage and branches on the vote ----
    const uint32_t idesc = idesc_f16_f32(128, kTX * TR), sbase = smem_u32(sm);
    int ka = 0, kb = 0, it = 0;
    bool ok = true;
    for (int w = first; w < A.nitems && ok; w = next_item(w), it++) {
      const int set = it & 1;
      const uint32_t d = tmem + (uint32_t)(set * 256);
      bool ready = mbar_wait_or(tfree + set, ((it >> 1) & 1) ^ 1, abort, A.err, kErrNear);
      for (int a = 0; a < na && ok; a++, ka++) {
        const int i = ka % kNpNO;
        ready = mbar_wait_or(ofull + i, (ka / kNpNO) & 1, abort, A.err, kErrNear) && ready;
        int idx;
        const int kind = np_stage(a, idx);
        const uint32_t obase = sbase + NpSmem::o + i * kNpBuf;
        constexpr uint32_t lbo = kHC * 16;  // K-adjacent core matrices
        const uint64_t dh0 = smem_desc(obase, lbo, kNpKC * lbo);
        const uint64_t dl0 = smem_desc(obase + kNpHaloSplit, lbo, kNpKC * lbo);
        const int nq = kind == 0 ? 9 : 1;
        for (int q = 0; q < nq; q++, kb++) {
          const int b = kb % kNpNB;
          ok = __all_sync(0xffffffffu, mbar_wait_or(bfull + b, (kb / kNpNB) & 1, abort, A.err, kErrNear) && ready);
          if (!ok) break;
          tc_fence_after();
          const uint32_t bb = sbase + NpSmem::b + b * kStageBytes;
          const uint64_t wh0 = smem_desc(bb, 128, 512), wl0 = smem_desc(bb + kStageHalf, 128, 512);
          // neighbour slot q: the item's leaf rows start at halo row 1 + dr, column 1 + dc
          const uint32_t doff0 = kind == 0 ? (uint32_t)((q / 3) * (kNpKC * kHC * 16) + (q % 3) * 16) : 0u;
          const uint64_t dh = desc_add(dh0, doff0), dl = desc_add(dl0, doff0);
          const int acc = (a | q) ? 1 : 0;
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 2; ks++) {
              const uint32_t doff = (uint32_t)ks * 2 * lbo;
              mma_f16(d, desc_add(wh0, ks * 256), desc_add(dh, doff), idesc, ks ? 1 : acc);
              mma_f16(d, desc_add(wh0, ks * 256), desc_add(dl, doff), idesc, 1);
              mma_f16(d, desc_add(wl0, ks * 256), desc_add(dh, doff), idesc, 1);
            }
            mma_commit(bempty + b);
            if (q == nq - 1) mma_commit(ofree + i);
            if (q == nq - 1 && a == na - 1) mma_commit(tfull + set);
          }
          __syncwarp();
        }
      }
    }
    // every MMA issued is complete before the CTA frees TMEM (bounded wait)
    if (elect_one()) mma_commit(mdone);
    __syncwarp();
    mbar_wait(mdone, 0, A.err, kErrNear);
  } else if (warp < kNpEpiWarp0) {
    // ---- converters: a staged FP32 A-stage becomes the FP16 hi/lo operand.  One
    // unit is a 4-complex chunk (32 bytes) of one leaf: staging [row][col][32 reals]
    // to operand [row][chunk][col][16 bytes], hi then lo ----
    const int ct = threadIdx.x - 32 * kNpConvWarp0;
    int ka = 0;
    for (int w = first; w < A.nitems; w = next_item(w)) {
      float s1, s2, p;
      np_scales(A, w / A.ppr, s1, s2, p);
      for (int a = 0; a < na; a++, ka++) {
        const int i = ka % kNpNS, o = ka % kNpNO;
        const bool ok = mbar_wait_or(sfull + i, (ka / kNpNS) & 1, abort, A.err, kErrNear) &&
                        mbar_wait_or(ofree + o, ((ka / kNpNO) & 1) ^ 1, abort, A.err, kErrNear);
        const float4 *st = (const float4 *)(sm + NpSmem::s + i * kNpBuf);
        char *hi = sm + NpSmem::o + o * kNpBuf, *lo = hi + kNpHaloSplit;
        int idx;
        const bool halo = np_stage(a, idx) == 0;
        const int cols = halo ? kHC : kTX, units = (halo ? TR + 2 : TR) * cols * kNpKC;
        const float sr = halo ? s1 : s2, si = halo && A.mode == IN_CONJ ? -s1 : sr;  // the imaginary parts' sign
        for (int e = ct; e < units && ok; e += kNpConv) {
          const int c = e & 3, row = halo ? (e >> 2) / kHC : (e >> 2) / kTX, col = (e >> 2) - row * cols;
          // staging offset ((row * cols + col) * 32 + 8 c) reals; every other leaf reads its
          // second half first, so that the 8 lanes of a load phase cover all banks
          const int f = (e >> 2) & 1;
          const float4 x0 = st[2 * e + f], x1 = st[2 * e + 1 - f];
          const float4 a0 = f ? x1 : x0, a1 = f ? x0 : x1;
          uint32_t h[4], l[4];
          split2u(a0.x * sr, a0.y * si, h[0], l[0]);
          split2u(a0.z * sr, a0.w * si, h[1], l[1]);
          split2u(a1.x * sr, a1.y * si, h[2], l[2]);
          split2u(a1.z * sr, a1.w * si, h[3], l[3]);
          const int off = ((row * kNpKC + c) * kHC + col) * 16;  // the pitch of 10 leaves keeps the banks apart
          st_shared_v4(hi + off, h);
          st_shared_v4(lo + off, l);
        }
        fence_proxy_async();
        named_sync(1, kNpConv);
        if (ct == 0) {
          mbar_arrive(sfree + i);
          mbar_arrive(ofull + o);
        }
      }
    }
  } else {
    // ---- epilogue: TMEM lane = target real (pixel 16 qd + lane / 2, real part on
    // even lanes), column = leaf of the item; the warp's 32 lanes are 128 contiguous
    // bytes of one leaf's output, so every load and store is one coalesced row.
    // Warps 7..10 take the item's first TR / 2 leaf rows (columns 0 .. 4 TR - 1), 11..14 the rest ----
    const int ew = warp - kNpEpiWarp0, qd = warp & 3, hh = ew >> 2;
    const bool odd = lane & 1;
    const bool need_x = A.epi == EPI_FWD || A.epi == EPI_ADJ || A.red == RED_TS;
    const float *xf = (const float *)A.xe, *af = (const float *)A.dot_a;
    float *yf = (float *)A.y;
    int it = 0;
    for (int w = first; w < A.nitems; w = next_item(w), it++) {
      int rhs, ty0, tx0;
      geom(w, rhs, ty0, tx0);
      const int set = it & 1;
      float s1, s2, p;
      np_scales(A, rhs, s1, s2, p);
      const float inv = 1.f / p;
      // a lane whose wait expired writes nothing, but takes part in the shuffles below
      const bool ok = mbar_wait_or(tfull + set, (it >> 1) & 1, abort, A.err, kErrNear);
      tc_fence_after();
      const size_t rbase = (size_t)rhs * A.U;
      const float *gf = A.g ? (const float *)(A.g + rhs * A.gstride) : nullptr;
      const float *xr = xf + 2 * rbase, *ar = af + 2 * rbase;
      float *yr = yf + 2 * rbase;
      double r0 = 0, r1 = 0, r2 = 0;
      Acc32 q0, q1, q2;
      const int nch = TR / 2, lyb = ty0 + hh * nch;  // the warp's leaf rows (an even number)
      if (lyb < A.nleaf) {  // warp-uniform
        // chunks of 8 leaves (one leaf row); the loads of chunk ch + 1 are in flight while
        // chunk ch is computed and stored
        auto fidx = [&](int ch, int j) { return 2 * ((lyb + ch) * A.nleaf + tx0 + j) * kBB + 32 * qd + lane; };
        auto load = [&](int ch, float (&xv)[8], float (&av)[8], float (&gv)[8], unsigned &live) {
          live = 0;
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const bool lv = lyb + ch < A.nleaf && tx0 + j < A.nleaf;
            live |= lv ? 1u << j : 0u;
            const int fi = fidx(ch, j);
            xv[j] = (need_x && lv) ? xr[fi] : 0.f;
            av[j] = (A.red == RED_DOT && lv) ? ar[fi] : 0.f;
            gv[j] = (A.epi == EPI_ADJ && lv) ? gf[fi] : 0.f;
          }
        };
        auto process = [&](int ch, const float (&xv)[8], const float (&av)[8], const float (&gv)[8], unsigned live) {
          float d[8];
          tmem_ld8(tmem + ((uint32_t)(32 * qd) << 16) + (uint32_t)(set * 256 + kTX * (hh * nch + ch)), d);
#pragma unroll
          for (int j = 0; j < 8; j++) {
            if (!((live >> j) & 1)) continue;  // warp-uniform
            const float o = d[j] * inv;
            float v = o;
            if (A.epi == EPI_FWD) {
              v = xv[j] - o;
            } else if (A.epi == EPI_ADJ) {  // x - conj(g o)
              const float op = __shfl_xor_sync(0xffffffffu, o, 1), gp = __shfl_xor_sync(0xffffffffu, gv[j], 1);
              v = odd ? xv[j] + (gp * o + gv[j] * op) : xv[j] - (gv[j] * o - gp * op);
            } else if (A.epi == EPI_CONJ) {
              v = odd ? -o : o;
            }
            if (ok) yr[fidx(ch, j)] = v;
            if (A.red == RED_DOT) {  // conj(a) y
              const float vp = __shfl_xor_sync(0xffffffffu, v, 1);
              q0.add_prod(j, av[j], v);
              q1.add_prod(j, odd ? -av[j] : av[j], vp);
            } else if (A.red == RED_TS) {  // conj(y) x and |y|^2
              const float xp = __shfl_xor_sync(0xffffffffu, xv[j], 1);
              q0.add_prod(j, v, xv[j]);
              q1.add_prod(j, odd ? -v : v, xp);
              q2.add_prod(j, v, v);
            }
          }
          if (A.red != RED_NONE && (ch & 1)) {  // two chunks' FP32 partial sums into the FP64 ones
            r0 += q0.take();
            r1 += q1.take();
            r2 += q2.take();
          }
        };
        float xa[8], aa[8], ga[8], xb[8], ab[8], gb[8];
        unsigned la, lb;
        load(0, xa, aa, ga, la);
#pragma unroll 1
        for (int ch = 0; ch < nch; ch += 2) {
          load(ch + 1, xb, ab, gb, lb);
          process(ch, xa, aa, ga, la);
          if (ch + 2 < nch) load(ch + 2, xa, aa, ga, la);
          process(ch + 1, xb, ab, gb, lb);
        }
      }
      if (A.red != RED_NONE) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          r0 += __shfl_xor_sync(0xffffffffu, r0, o);
          r1 += __shfl_xor_sync(0xffffffffu, r1, o);
          r2 += __shfl_xor_sync(0xffffffffu, r2, o);
        }
        if (lane == 0) {
          double *ds = dscr + (set * kNpEpiWarps + ew) * 3;
          ds[0] = r0;
          ds[1] = r1;
          ds[2] = r2;
        }
      }
      tc_fence_before();
      named_sync(2, kNpEpi);  // the accumulator set is read out, the warps' sums are in dscr
      if (ew == 0 && lane == 0) {
        mbar_arrive(tfree + set);
        if (A.red != RED_NONE && ok) {
          double s0 = 0, s1v = 0, s2v = 0;
          for (int k = 0; k < kNpEpiWarps; k++) {
            const double *ds = dscr + (set * kNpEpiWarps + k) * 3;
            s0 += ds[0];
            s1v += ds[1];
            s2v += ds[2];
          }
          // the item's sum goes to the record of its first 8 x 8 leaves, zero to the others'
          const int rows8 = (A.nleaf + 7) / 8;
          for (int r = ty0 / 8; r < min(rows8, (ty0 + TR) / 8); r++) {
            const bool first8 = r == ty0 / 8;
            double *pp = A.part + (((size_t)rhs * rows8 + r) * A.tiles_x + tx0 / kTX) * 4;
            pp[0] = first8 ? s0 : 0.0;
            pp[1] = first8 ? s1v : 0.0;
            pp[2] = first8 ? s2v : 0.0;
            pp[3] = 0.0;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// ---- P2M: persistent CTAs over (RHS, 128-leaf tile) items, N = 2 ns padded to 16 ----
constexpr int kP2mA = 16 * 2048;  // one FP16 split of the [128 x 128] operand

struct TcP2mArgs {
  const float2 *x;
  int conj;  // the input is conjugated
  const int *active;
  const uint8_t *B;  // 4 stages of [npad x 32] hi then lo
  int npad, stage_bytes;
  float inv_c;
  float2 *mul_leaf;
  size_t mp;
  int ns, nleaves, U, tiles, nitems;
  int *err;
  unsigned *levmax;  // [R][kLevStride]: this level's max |re|, |im| per RHS (FP32 bits)
  int lvl;
};

// Converter, MMA and epilogue roles over double-buffered A operands (128 leaves
// x 64 pixels x re, im, FP16 hi/lo) and TMEM accumulators; the coefficients (B,
// 4 stages) stay resident.  An item's pixels (one contiguous run) are bulk-copied
// as FP32 into the operand buffer they will fill; the converters take them into
// registers, take the item's maximum among themselves, and split them in place.  The epilogue reads each leaf's ring from its TMEM
// lane and turns lanes into contiguous runs through a small per-warp tile;
// it keeps the level maximum for the M2M above. ----
struct P2mPipeSmem {
  __host__ __device__ static size_t a(int b) { return (size_t)b * 2 * kP2mA; }  // hi, then lo kP2mA on
  __host__ __device__ static size_t bst() { return 4 * (size_t)kP2mA; }
  // per epilogue warp: 32 leaves x 8 complex (+1 pad)
  __host__ __device__ static size_t epi(int stage_bytes) { return bst() + 4 * (size_t)stage_bytes; }
  __host__ __device__ static size_t bar(int stage_bytes) { return epi(stage_bytes) + 8 * 32 * 9 * 8; }
  __host__ __device__ static size_t total(int stage_bytes) { return bar(stage_bytes) + 256; }
};
// Roles: converters warps 0..7, MMA warp 8, epilogue warps 9..16 (two per
// TMEM lane quarter warp % 4, each taking every other 16-column chunk).
constexpr int kP2mConvWarps = 8, kP2mMmaWarp = 8, kP2mEpiWarp0 = 9, kP2mThreads = 17 * 32;
constexpr int kP2mConv = 32 * kP2mConvWarps, kP2mEpi = kP2mThreads - 32 * kP2mEpiWarp0;
constexpr int kP2mUnits = 128 * 16;                             // (leaf, 4-pixel chunk) per item
constexpr int kP2mPer = (kP2mUnits + kP2mConv - 1) / kP2mConv;  // units per converter thread

__global__ void __launch_bounds__(kP2mThreads, 1) k_tc_p2m_pipe(TcP2mArgs A) {
  extern __shared__ __align__(1024) char sm[];
  const PipeBars Bq(sm + P2mPipeSmem::bar(A.stage_bytes));
  float *fscr = (float *)(Bq.abar + 16);  // [kP2mConvWarps] converter maxima
  float *sval = fscr + 16;                // [2] the scale of the item in buffer b
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 11; i++) mbar_init(Bq.abar + i, 1);
    *Bq.abort = 0;
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(Bq.tslot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *Bq.tslot;
  auto next_item = [&](int w) {
    do w += gridDim.x;
    while (w < A.nitems && A.active && !A.active[w / A.tiles]);
    return w;
  };
  if (threadIdx.x == 0) {  // the coefficients, which no earlier kernel writes
    mbar_expect_tx(Bq.abar, 4 * A.stage_bytes);
    for (int c = 0; c < 4; c++)
      bulk_g2s(sm + P2mPipeSmem::bst() + c * A.stage_bytes, A.B + (size_t)c * A.stage_bytes, A.stage_bytes, Bq.abar);
  }
  const int blk = blockIdx.x + grid_wait();
  const int first = (A.active && !A.active[blk / A.tiles]) ? next_item(blk) : blk;
  // an item's pixels (its leaves are one contiguous run) into operand buffer b, as FP32
  auto stage = [&](int w, int b) {
    const int rhs = w / A.tiles, leaf0 = (w % A.tiles) * 128;
    const uint32_t bytes = (uint32_t)min(128, A.nleaves - leaf0) * kBB * 8;
    mbar_expect_tx(Bq.zfull + b, bytes);
    bulk_g2s(sm + P2mPipeSmem::a(b), A.x + (size_t)rhs * A.U + (size_t)leaf0 * kBB, bytes, Bq.zfull + b);
  };

  if (warp < kP2mConvWarps) {
    // ---- converters ----
    if (threadIdx.x == 0) {
      if (first < A.nitems) {
        stage(first, 0);
        const int second = next_item(first);
        if (second < A.nitems) stage(second, 1);
      }
    }
    int w = first;
    for (int it = 0; w < A.nitems; it++) {
      const int b = it & 1, ph = (it >> 1) & 1;
      // the staged pixels, and the scale slot (free once the epilogue of item it - 2 is done)
      const bool fok = mbar_wait_or(Bq.zfull + b, ph, Bq.abort, A.err, kErrP2m) &&
                       mbar_wait_or(Bq.tfree + b, ph ^ 1, Bq.abort, A.err, kErrP2m);
      const int leaf0 = (w % A.tiles) * 128;
      const float4 *zst = (const float4 *)(sm + P2mPipeSmem::a(b));  // [leaf][32 float4]
      float2 v[kP2mPer][4];
      float mx = 0.f;
#pragma unroll
      for (int r = 0; r < kP2mPer; r++) {
        const int u = threadIdx.x + r * kP2mConv;
        const int m = ((u >> 7) << 3) | (u & 7), c = ((u >> 3) & 15) ^ (u & 7);
#pragma unroll
        for (int p = 0; p < 4; p++) v[r][p] = make_float2(0.f, 0.f);
        if (u < kP2mUnits && leaf0 + m < A.nleaves) {
          // the 8 leaves of a load phase, 512 bytes apart, take 8 different chunks, the
          // upper four of them their second half first: all banks, no conflict (with one
          // chunk for all, 4-way: P2M of 1024 x 1024 x 64 256 us, this 249)
          const int odd = (c >> 2) & 1;
          const float4 x0 = zst[m * 32 + 2 * c + odd], x1 = zst[m * 32 + 2 * c + 1 - odd];
          const float4 a0 = odd ? x1 : x0, a1 = odd ? x0 : x1;
          v[r][0] = make_float2(a0.x, a0.y);
          v[r][1] = make_float2(a0.z, a0.w);
          v[r][2] = make_float2(a1.x, a1.y);
          v[r][3] = make_float2(a1.z, a1.w);
#pragma unroll
          for (int p = 0; p < 4; p++) mx = fmaxf(mx, cabs1(v[r][p]));
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if (lane == 0) fscr[warp] = mx;
      named_sync(1, kP2mConv);  // every staged value is in registers: the buffer is rewritten in place
      float m2 = 0.f;
      for (int k = 0; k < kP2mConvWarps; k++) m2 = fmaxf(m2, fscr[k]);
      const float s = pow2_scale(m2), si = A.conj ? -s : s;
      // the input's maximum per RHS: the near-field kernel's scale for the same input
      if (threadIdx.x == 0 && fok && m2 > 0.f)
        atomicMax(&A.levmax[(w / A.tiles) * kLevStride + kInMaxSlot], __float_as_uint(m2));
      char *ahi = sm + P2mPipeSmem::a(b), *alo = ahi + kP2mA;
      if (fok) {
#pragma unroll
        for (int r = 0; r < kP2mPer; r++) {
          const int u = threadIdx.x + r * kP2mConv;
          if (u >= kP2mUnits) continue;
          const int off = (u >> 7) * 2048 + (((u >> 3) & 15) ^ (u & 7)) * 128 + (u & 7) * 16;
          uint32_t h[4], l[4];
#pragma unroll
          for (int p = 0; p < 4; p++) split2u(v[r][p].x * s, v[r][p].y * si, h[p], l[p]);
          st_shared_v4(ahi + off, h);
          st_shared_v4(alo + off, l);
        }
      }
      if (threadIdx.x == 0) sval[b] = s;
      fence_proxy_async();
      named_sync(1, kP2mConv);  // the operand is written; fscr may be reused
      if (threadIdx.x == 0) mbar_arrive(Bq.bfull + b);
      w = next_item(w);
    }
  } else if (warp == kP2mMmaWarp) {
    // ---- MMA issue: D[128 leaves][npad] = A[b] (hi/lo) x coefficients (hi/lo) ----
    const uint32_t idesc = idesc_f16_f32(128, A.npad), sbase = smem_u32(sm);
    const uint64_t bh0 = smem_desc(sbase + (uint32_t)P2mPipeSmem::bst(), 128, 512);
    const uint64_t bl0 = smem_desc(sbase + (uint32_t)P2mPipeSmem::bst() + A.stage_bytes / 2, 128, 512);
    const bool aok = mbar_wait_or(Bq.abar, 0, Bq.abort, A.err, kErrP2m);
    int w = first;
    for (int it = 0; w < A.nitems; it++) {
      const int b = it & 1, ph = (it >> 1) & 1;
      const bool ok = mbar_wait_or(Bq.bfull + b, ph, Bq.abort, A.err, kErrP2m) && aok;
      tc_fence_after();
      if (__all_sync(0xffffffffu, ok)) {
        const uint64_t ah0 = smem_desc(sbase + (uint32_t)P2mPipeSmem::a(b), 128, 2048);
        const uint64_t al0 = smem_desc(sbase + (uint32_t)P2mPipeSmem::a(b) + kP2mA, 128, 2048);
        const uint32_t d = tmem + (uint32_t)(b * 256);
        for (int pass = 0; pass < 2; pass++)  // the small products first, as in k_tc_l2l
          for (int c = 0; c < 4; c++) {
            const uint32_t aoff0 = (uint32_t)c * 512, boff0 = c * A.stage_bytes;
            if (elect_one()) {
#pragma unroll
              for (int ks = 0; ks < 2; ks++) {
                const uint32_t aoff = aoff0 + ks * 256, boff = boff0 + ks * 256;
                if (pass == 0) {
                  mma_f16(d, desc_add(ah0, aoff), desc_add(bl0, boff), idesc, (c | ks) ? 1 : 0);
                  mma_f16(d, desc_add(al0, aoff), desc_add(bh0, boff), idesc, 1);
                } else {
                  mma_f16(d, desc_add(ah0, aoff), desc_add(bh0, boff), idesc, 1);
                }
              }
            }
            __syncwarp();
          }
      }
      if (elect_one()) mma_commit(Bq.tfull + b);
      __syncwarp();
      w = next_item(w);
    }
  } else {
    // ---- epilogue: lane = leaf, columns 2k (re), 2k + 1 (im).  Each 16-column chunk
    // (8 samples of the warp's 32 consecutive leaves) goes through a padded
    // shared tile so that 8 lanes write one leaf's 64 contiguous bytes ----
    const int ew = warp - kP2mEpiWarp0, qd = warp & 3, eg = ew >> 2;  // lane quarter, chunk parity
    float2 *tile = (float2 *)(sm + P2mPipeSmem::epi(A.stage_bytes)) + ew * 32 * 9;
    int w = first, w2 = first < A.nitems ? next_item(next_item(first)) : A.nitems;
    for (int it = 0; w < A.nitems; it++) {
      const int b = it & 1, ph = (it >> 1) & 1;
      // tfull: the accumulator; bfull (already complete): the item's scale is visible
      const bool ok = mbar_wait_or(Bq.tfull + b, ph, Bq.abort, A.err, kErrP2m) &&
                      mbar_wait_or(Bq.bfull + b, ph, Bq.abort, A.err, kErrP2m);
      tc_fence_after();
      // the MMAs are done with operand buffer b: item it + 2's pixels go there now
      if (ew == 0 && lane == 0 && w2 < A.nitems) stage(w2, b);
      w2 = w2 < A.nitems ? next_item(w2) : A.nitems;
      const int rhs = w / A.tiles, leafw = (w % A.tiles) * 128 + 32 * qd;  // the warp's first leaf
      const float inv = A.inv_c / sval[b];
      float2 *outw = A.mul_leaf + (size_t)rhs * A.mp + (size_t)leafw * A.ns;
      float omx = 0.f;
      const uint32_t taddr = tmem + ((uint32_t)(32 * qd) << 16) + (uint32_t)(b * 256);
      for (int c0 = 16 * eg; c0 < A.npad; c0 += 32) {
        float d[16];
        tmem_ld16(taddr + c0, d);
        const int k0 = c0 / 2, nk = min(8, A.ns - k0);
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (j < nk) tile[lane * 9 + j] = make_float2(d[2 * j] * inv, d[2 * j + 1] * inv);
        __syncwarp();
        if (ok) {
#pragma unroll
          for (int r = 0; r < 8; r++) {  // element r * 32 + lane: leaf e / 8, sample e % 8
            const int e = r * 32 + lane, lf = e >> 3, j = e & 7;
            if (j < nk && leafw + lf < A.nleaves) {
              const float2 o = tile[lf * 9 + j];
              outw[(size_t)lf * A.ns + k0 + j] = o;
              omx = fmaxf(omx, fmaxf(fabsf(o.x), fabsf(o.y)));
            }
          }
        }
        __syncwarp();
      }
      tc_fence_before();
      named_sync(2, kP2mEpi);  // the accumulator is read out
      if (ew == 0 && lane == 0) mbar_arrive(Bq.tfree + b);
      const unsigned mbits = __reduce_max_sync(0xffffffffu, __float_as_uint(omx));  // omx >= 0
      if (lane == 0 && ok && mbits) atomicMax(&A.levmax[rhs * kLevStride + A.lvl], mbits);
      w = next_item(w);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// ---- host: operand construction ----

inline double pow2_scale_host(double maxabs) {
  if (!(maxabs > 0)) return 1.0;
  int e;
  std::frexp(maxabs, &e);
  return std::ldexp(1.0, 14 - e);
}

// Writes the [nrows x 32] K-major FP16 core-matrix block of reals(row, k0..k0+31)
// as hi then lo (each nrows/8 groups x 4 chunks x 8 rows x 8 halves).
template <class F>
void pack_stage(std::vector<uint8_t> &buf, size_t at, int nrows, int k0, double scale, F real_at) {
  const size_t half = (size_t)nrows * 32 * 2;
  __half *hi = (__half *)(buf.data() + at), *lo = (__half *)(buf.data() + at + half);
  for (int n = 0; n < nrows; n++)
    for (int k = 0; k < 32; k++) {
      const double v = real_at(n, k0 + k) * scale;
      const __half h = __double2half(v);
      const __half l = __double2half(v - (double)__half2float(h));
      const size_t idx = ((size_t)(n / 8) * 4 + k / 8) * 64 + (n % 8) * 8 + (k % 8);
      hi[idx] = h;
      lo[idx] = l;
    }
}

}  // namespace

struct TcPlan {
  uint8_t *nearB = nullptr;  // weight stages in the near field's A-stage order
  int nl2p = 0;
  float sw = 1, sb = 1;
  uint8_t *p2mB = nullptr;
  int npad = 0, p2m_stage = 0;
  float inv_c = 1;
  int *err = nullptr;
  bool ok = false;
  int near_pair = 0;  // near-field items picked by isg_autotune: of 16 leaf rows times this at most (0: 32)
};

bool tc_available(const isg_ctx *c) { return c->tc && c->tc->ok; }
void tc_set_near_pair(isg_ctx *c, int pair) {
  if (tc_available(c)) c->tc->near_pair = pair;
}
int tc_near_pair(const isg_ctx *c) { return tc_available(c) ? c->tc->near_pair : 0; }

}  // namespace isg

int *isg_ctx::tc_err_flag() const { return tc ? tc->err : nullptr; }

namespace isg {

// cuTensorMapEncodeTiled through the runtime's driver entry-point query, so
// that the library does not link the driver library (it still loads where
// there is no driver, for the checks that need none); null when unavailable.
// The lookup runs once per process; C++11 makes the static's initialisation
// thread-safe, so contexts on several host threads may race to it.
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return (PFN_cuTensorMapEncodeTiled_v12000)p;
    return nullptr;
  }();
  return fn;
}

isg_status tc_setup(isg_ctx *c) {
  int dev = 0, major = 0, minor = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
  cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev);
  const HostTables &T = c->T;
  const int ns = T.nsamp[T.L - 1];
  c->tc = new TcPlan();
  TcPlan &P = *c->tc;
  if (major != 10 || ns > kLeafSampMax || !tensor_map_encoder()) return ISG_OK;  // engine unavailable, SIMT remains
  // near field: real embedding of near[slot][t][b]; row n = 2t + d, K = 2b + e
  auto wreal = [&](int s, int n, int k) {
    const cd w = T.near[((size_t)s * kBB + n / 2) * kBB + k / 2];
    const int d = n & 1, e = k & 1;
    return d == 0 ? (e == 0 ? w.real() : -w.imag()) : (e == 0 ? w.imag() : w.real());
  };
  auto breal = [&](int n, int k) {
    if (k / 2 >= ns) return 0.0;
    const cd w = T.basis[(size_t)(n / 2) * ns + k / 2];
    const int d = n & 1, e = k & 1;
    return d == 0 ? (e == 0 ? w.real() : -w.imag()) : (e == 0 ? w.imag() : w.real());
  };
  double mw = 0, mb = 0, mc = 0;
  for (const cd &v : T.near) mw = std::max(mw, std::max(std::abs(v.real()), std::abs(v.imag())));
  for (const cd &v : T.basis) mb = std::max(mb, std::max(std::abs(v.real()), std::abs(v.imag())));
  for (const cd &v : T.coeff) mc = std::max(mc, std::max(std::abs(v.real()), std::abs(v.imag())));
  const double sw = pow2_scale_host(mw), sb = pow2_scale_host(mb), sc = pow2_scale_host(mc);
  const int kl = ((2 * ns + 31) / 32) * 32;  // L2P K padded to whole stages
  P.nl2p = kl / 32;
  P.sw = (float)sw;
  P.sb = (float)sb;
  // near field: per A-stage, a halo K-group's nine slots or one L2P stage
  std::vector<uint8_t> nb((size_t)(kNearStages + P.nl2p) * kStageBytes, 0);
  {
    size_t t = 0;
    for (int a = 0; a < 4 + P.nl2p; a++) {
      int idx;
      if (np_stage(a, idx) == 0) {
        for (int q = 0; q < 9; q++, t++)
          pack_stage(nb, t * kStageBytes, 128, idx * 32, sw, [&](int n, int k) { return wreal(q, n, k); });
      } else {
        pack_stage(nb, (t++) * kStageBytes, 128, idx * 32, sb, breal);
      }
    }
  }
  // P2M: row n = 2k + d over samples (padded to a multiple of 16), K = 2 pixel + e
  P.npad = ((2 * ns + 15) / 16) * 16;
  P.p2m_stage = P.npad * 32 * 2 * 2;
  auto creal = [&](int n, int k) {
    if (n / 2 >= ns) return 0.0;
    const cd w = T.coeff[(size_t)(n / 2) * kBB + k / 2];
    const int d = n & 1, e = k & 1;
    return d == 0 ? (e == 0 ? w.real() : -w.imag()) : (e == 0 ? w.imag() : w.real());
  };
  std::vector<uint8_t> pb((size_t)4 * P.p2m_stage, 0);
  for (int c2 = 0; c2 < 4; c2++) pack_stage(pb, (size_t)c2 * P.p2m_stage, P.npad, c2 * 32, sc, creal);
  P.inv_c = (float)(1.0 / sc);
  isg_status e;
  if ((e = cuda_check(c, cudaMalloc(&P.nearB, nb.size()), "tc alloc")) != ISG_OK) return e;
  if ((e = cuda_check(c, cudaMalloc(&P.p2mB, pb.size()), "tc alloc")) != ISG_OK) return e;
  if ((e = cuda_check(c, cudaMalloc(&P.err, sizeof(int)), "tc alloc")) != ISG_OK) return e;
  cudaMemcpy(P.nearB, nb.data(), nb.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(P.p2mB, pb.data(), pb.size(), cudaMemcpyHostToDevice);
  cudaMemset(P.err, 0, sizeof(int));
  for (auto k : {k_tc_near_pipe<8>, k_tc_near_pipe<16>, k_tc_near_pipe<32>})
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, NpSmem::total);
  cudaFuncSetAttribute(k_tc_p2m_pipe, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)P2mPipeSmem::total(P.p2m_stage));
  if ((e = cuda_check(c, cudaGetLastError(), "tc setup")) != ISG_OK) return e;
  P.ok = true;
  return ISG_OK;
}

void tc_destroy(isg_ctx *c) {
  if (!c->tc) return;
  cudaFree(c->tc->nearB);
  cudaFree(c->tc->p2mB);
  cudaFree(c->tc->err);
  delete c->tc;
  c->tc = nullptr;
}

int tc_near_blocks(const isg_ctx *c) {
  const int n8 = (c->P.nleaf + 7) / 8;
  return n8 * n8;
}

// Leaf rows per item of the pipelined near field: 32 (the most MMA columns, so
// each weight stage serves 256 leaves), unless 16 or 8 rows still give every
// item an SM of its own or the grid is no higher than that: the launch is then
// as long as one item, whose time falls with its rows.
static int np_rows(const DevPlan &P, int nrhs, int sms, int cap) {
  const int cols = (P.nleaf + kTX - 1) / kTX;
  for (int tr : {8, 16})
    if (tr >= cap || tr >= P.nleaf || (int64_t)cols * ((P.nleaf + tr - 1) / tr) * nrhs <= sms) return tr;
  return kTRMax;
}

int tc_error(isg_ctx *c) {
  if (!tc_available(c)) return 0;
  int h = 0;
  cudaMemcpy(&h, c->tc->err, sizeof(int), cudaMemcpyDeviceToHost);
  return h;
}

static bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }

static int device_sms(const isg_ctx *c) {
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->opts.device);
  return sms;
}

bool tc_near_tall(const isg_ctx *c, int nrhs) { return np_rows(c->P, nrhs, device_sms(c), kTRMax) == kTRMax; }

// The input is plain or conjugated (callers form g x first, run_matvec); its
// maximum and the locals' are known (P2M and M2L of the same matvec).  Leaf rings are
// multiples of 4 samples, so every row that the tensor maps address is 16-byte aligned.
isg_status tc_near(isg_ctx *c, const NearArgs &N, cudaStream_t st) {
  const DevPlan &P = c->P;
  const TcPlan &T = *c->tc;
  const float2 *loc_leaf = N.loc + P.lv[P.L - 1].off;
  if (!aligned16(N.in.x) || (N.x_epi && !aligned16(N.x_epi)) || (N.in.g && !aligned16(N.in.g)) || !aligned16(N.y) ||
      (N.dot_a && !aligned16(N.dot_a)) || (N.in.gstride % 2) || N.epi == EPI_L2P_ONLY || N.in.mode == IN_G ||
      !N.inmax || !N.locmax)
    return ISG_UNSUPPORTED;
  TcNearArgs A;
  A.x = N.in.x;
  A.xe = N.x_epi ? N.x_epi : N.in.x;
  A.g = N.in.g;
  A.gstride = N.in.gstride;
  A.mode = N.in.mode;
  A.active = N.in.active;
  A.B = T.nearB;
  A.nl2p = T.nl2p;
  A.sw = T.sw;
  A.sb = T.sb;
  A.levmax = N.inmax;
  A.locmax = N.locmax;
  A.lvl_leaf = P.L - 1;
  A.y = N.y;
  A.epi = N.epi;
  A.red = N.red;
  A.dot_a = N.dot_a;
  A.part = N.part;
  A.nleaf = P.nleaf;
  A.U = P.U;
  const int sms = device_sms(c);
  const bool tuned = T.near_pair > 0 && 4 * N.in.nrhs >= P.tuned_nrhs;
  const int tr = np_rows(P, N.in.nrhs, sms, tuned ? 16 * T.near_pair : kTRMax);
  A.tiles_x = (P.nleaf + kTX - 1) / kTX;
  A.ppr = A.tiles_x * ((P.nleaf + tr - 1) / tr);
  A.nitems = A.ppr * N.in.nrhs;
  A.err = T.err;
  // tmh: the input as [RHS][leaf row][leaf column][128 reals], a box is one halo
  // K-group (32 reals) of the item's (tr + 2) x 10 halo; tml: the leaf locals as
  // [RHS][leaf row][leaf column][2 ns reals], a box is one L2P stage of the item
  CUtensorMap tmh, tml;
  memset(&tmh, 0, sizeof(tmh));
  memset(&tml, 0, sizeof(tml));
  const cuuint32_t one[4] = {1, 1, 1, 1};
  const cuuint64_t hd[4] = {2 * kBB, (cuuint64_t)P.nleaf, (cuuint64_t)P.nleaf, (cuuint64_t)N.in.nrhs};
  const cuuint64_t hs[3] = {(cuuint64_t)kBB * 8, (cuuint64_t)P.nleaf * kBB * 8, (cuuint64_t)P.U * 8};
  const cuuint32_t hb[4] = {32, (cuuint32_t)kHC, (cuuint32_t)(tr + 2), 1};
  const cuuint64_t ld[4] = {(cuuint64_t)(2 * P.ns_leaf), (cuuint64_t)P.nleaf, (cuuint64_t)P.nleaf,
                            (cuuint64_t)N.in.nrhs};
  const cuuint64_t ls[3] = {(cuuint64_t)P.ns_leaf * 8, (cuuint64_t)P.nleaf * P.ns_leaf * 8, (cuuint64_t)P.mp * 8};
  const cuuint32_t lb[4] = {32, (cuuint32_t)kTX, (cuuint32_t)tr, 1};
  const PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
  if (encode(&tmh, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (void *)A.x, hd, hs, hb, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS ||
      encode(&tml, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (void *)loc_leaf, ld, ls, lb, one,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
    c->err = "near field: a tensor map was refused";
    return ISG_CUDA_ERROR;
  }
  count_launch();
  launch(tr == 32 ? k_tc_near_pipe<32> : tr == 16 ? k_tc_near_pipe<16> : k_tc_near_pipe<8>, std::min(A.nitems, sms),
         kNpThreads, NpSmem::total, st, A, tmh, tml);
  return cuda_check(c, cudaGetLastError(), "tc near launch");
}

isg_status tc_p2m(isg_ctx *c, const BatchArgs &B, float2 *mul, cudaStream_t st) {
  const DevPlan &P = c->P;
  const TcPlan &T = *c->tc;
  if (!aligned16(B.x) || B.mode == IN_G) return ISG_UNSUPPORTED;  // callers form g x first (run_matvec)
  TcP2mArgs A;
  A.x = B.x;
  A.conj = B.mode == IN_CONJ;
  A.active = B.active;
  A.B = T.p2mB;
  A.npad = T.npad;
  A.stage_bytes = T.p2m_stage;
  A.inv_c = T.inv_c;
  A.mul_leaf = mul + P.lv[P.L - 1].off;
  A.mp = P.mp;
  A.ns = P.ns_leaf;
  A.nleaves = P.nleaf * P.nleaf;
  A.U = P.U;
  A.tiles = (A.nleaves + 127) / 128;
  A.nitems = A.tiles * B.nrhs;
  A.err = T.err;
  A.levmax = c->levmax;
  A.lvl = P.L - 1;
  count_launch();
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->opts.device);
  launch(k_tc_p2m_pipe, std::min(A.nitems, sms), kP2mThreads, P2mPipeSmem::total(T.p2m_stage), st, A);
  return cuda_check(c, cudaGetLastError(), "tc p2m launch");
}

}  // namespace isg
