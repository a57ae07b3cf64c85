// Tensor-core chunk forward (64-token chunks, compact-WY form), two kernels or one that does the work of both:
//
//   chunk_prep_kernel   persistent, two CTAs per SM walking over the (sequence, chunk, head) units, all
//                       chunks independent.  The raw inputs of the next unit arrive by tiled TMA
//                       loads as their places become free, g under the inverse of the current one,
//                       k and q after its last product, beta behind its last store (a CTA that
//                       starts a unit with per-thread loads spends a quarter of its time issuing
//                       them: the load/store unit's queue, not HBM, is the limit).  Builds the WY
//                       factors of the chunk and writes them as row-major tiles:
//                       cumulative log-decay, block-anchored Gram products on tf32 tcgen05 MMAs,
//                       the inverse T of the unit lower-triangular system on CUDA cores (fp32; two
//                       32 x 32 blocks by substitution, the third by products), Y = T E on tf32
//                       tcgen05 MMAs.
//   chunk_scan_kernel   one CTA per (sequence, head) or half of its value rows, chunks in order.  The state
//                       lives transposed (S^T: value rows x key columns) in TMEM as the fp32 accumulator
//                       and is fed back as the tf32 A operand of the next MMAs without leaving TMEM:
//                           R^T  = Z^T T^T - S^T Y^T           (Z = w v)
//                           O^T  = S^T Qg^T + R^T Aqk^T
//                           S^T <- S^T diag(d) + R^T Kt
//                       The B operands are the prep kernel's row-major tiles, brought in by tiled
//                       TMA loads in the swizzled layout of their role (chunk_common.cuh).
//   chunk_joint_kernel  where few sequences and heads leave most SMs without a scan: some CTAs scan
//                       (after helping to prepare) while the others prepare, chunk by chunk.
//
// Math per chunk (reference: src/gdn2_sm120/reference.py:149-172, chunk.py:188-331, with the
// chunk length re-chosen as 64 and the decay normalisation anchored per 16-token block so that
// every exponent stays inside the contract "16-token prefix sums of g > -87"):
//   G_i = sum_{t<=i} g_t,  a_I = G at the start of block I = i / 16
//   L[i][j]   = sum_k beta k_i exp(G_i - a_I) * k_j exp(a_I - G_j)      (j < i)
//   Aqk[i][j] = sum_k scale q_i exp(G_i - a_I) * k_j exp(a_I - G_j)     (j <= i)
//   T = (I + L)^-1,  Y = T (beta k exp(G)),  R = T (w v) - Y S
//   Qg = scale q exp(G),  Kt = k exp(G_end - G),  d = exp(G_end)

#include <algorithm>
#include <type_traits>

#include "chunk_common.cuh"

namespace gdn2 {

using namespace tc;

namespace {

// ---------------------------------------------------------------------------------------------
// prep kernel
// ---------------------------------------------------------------------------------------------
// Persistent, two CTAs of 256 threads per SM.  A unit is a chain of a dozen phases of about a microsecond,
// each waiting for the one before (loads, exponentials, tensor cores, the inverse, stores): with one
// CTA per SM the issue slots were 35 % busy and a unit took 10.5 us.  Two CTAs fill each other's waits; for
// that a CTA has to live in 113 KB and 128 registers per thread, so the Gram operands are built and multiplied
// 32 channels at a time, and everything else shares their place.  (In two rounds of 64 channels the inputs
// waiting for the second spilled: 115 KB a unit through L2, as much as the tiles themselves.)
//
// What a unit takes is what passes through the load/store unit of shared memory (10 thousand wavefronts of 128 bytes a
// unit in an earlier form, where a unit took 14 thousand clocks of an SM), so the layouts below are chosen for few of
// them.  A thread owns 4 consecutive tokens x 2 channels of each round: tokens 8 warp + 4 (lane / 16), channels
// 2 (lane % 16).  Sums along the tokens need no shuffles, a 16-lane row of a store phase fills a 128-byte line, and what
// depends on a channel alone is read once for four tokens.
constexpr int kPrepThreads = 256;
constexpr int kJointParts = 2;
constexpr int kRound = 32, kRounds = kDim / kRound;  // channels per round
constexpr int kLdQ = 36;          // leading dimension of a transposed 32 x 32 block (16-byte rows, banks shift by 4)

// One region, by phase (bytes):
//   inputs       g at 0 (16 or 32 KiB), dense rows; k, q, beta (16 KiB each), 2 slabs of 64 lines of 64 channels,
//                16-byte pieces permuted by the line: the rows of both halves of a warp are then in other banks
//                (lines of 32 channels would be too, but the copy engine is paid by the line)
//   rounds       A operand [E_anchored ; Q_anchored], 128 lines of 32 channels, B operands K^I, 16 (I + 1) lines
//                each (K-major, 128-byte swizzle); E[j][k], tf32, MN-major operand, 4 swizzled slabs of 32
//                channels x 64 lines (tc05.cuh) over k and q: slab r is written once rounds r and r + 1 have
//                been read, hence the order 0, 2, 1, 3
//   inverse      -L^T over beta, T's diagonal blocks behind the next unit's g, T^T as a tf32 tile
//   last product Y^T on its way out, over -L^T and T^T
// The next unit's g arrives over the Gram operands under the inverse, its k and q after the last product, its beta
// once Y^T has left.
constexpr int kOffGramA = 0, kOffGramB = 16384;                         // + 20480
constexpr int kOffTable = 36864;                                        // decay table, 13 rows of 128
constexpr int kOffInG = 0, kOffInK = 44032, kOffInQ = kOffInK + 16384, kOffInBeta = kOffInQ + 16384;
constexpr int kOffE = kOffInK;
constexpr int kOffLt = kOffInBeta;                                      // -L^T, [64][64]
constexpr int kOffW = kOffLt + 32 * 64 * 4;                             // over its lines 32.., columns ..32: the block product
constexpr int kOffP = 32768, kOffQt = kOffP + 4096;                     // T[..32][..32], T[32..][32..] transposed
constexpr int kOffTt = kOffLt + 16384;                                  // T^T[j][i], MN-major operand, 2 swizzled slabs of 64 lines
constexpr int kOffY = kOffLt;                                           // Y^T[k][i], 2 swizzled slabs of 128 lines
constexpr int kPrepRegion = kOffTt + 16384;                             // 109568
static_assert(kOffTable + 13 * 512 <= kOffE && kOffQt + 32 * kLdQ * 4 <= kOffE && kOffY + 32768 <= kPrepRegion, "prep region");
static_assert(kOffE % 1024 == 0 && kOffGramB % 1024 == 0 && kOffTt % 1024 == 0 && kOffY % 1024 == 0,
              "swizzled tiles are 1024-byte aligned");

struct PrepSmem {
  alignas(1024) uint8_t region[kPrepRegion];
  float part[8][kDim];                 // sums of g over groups of 8 tokens, then what precedes them in their block
  float gend[kDim];
  alignas(8) uint64_t bar[2];          // MMA commits (the second one: and T^T has left)
  alignas(8) uint64_t bar_ld[2];       // raw inputs: {g} and {k, q, beta}
  int next[2];                         // joint launch: the unit after this one (two slots: one may still be read)
  uint32_t tmem_base;
};
static_assert(sizeof(PrepSmem) <= 115712, "two prep CTAs must fit an SM");
constexpr uint32_t kStageTile16 = kChunk * kDim * 2;                // a 16-bit input tile

struct PrepParams {
  uint8_t* ws;   // workspace (D, status)
  ForwardTiles tiles;  // the tile arrays (in the workspace for a training call, else in the scratch)
  int64_t n_ch;
  int H;
  float scale;
  int training;  // layout of the workspace
  int prologue;  // kPrologueNorm | kPrologueGate: the inputs are raw projections / gate pre-activations
};

__device__ __forceinline__ int gram_col(int I) { return (I == 0) ? 0 : (I == 1) ? 16 : (I == 2) ? 48 : 96; }

struct PrepMaps {
  CUtensorMap g, k, q, beta;
  CUtensorMap out_tt, out_yt;  // tiles that leave by tiled stores
};

// The units of one group of 256 threads (`tid` within it): first, first + stride, ..., or in a joint launch
// `first` and then whatever the queue gives; tensor memory columns tb .. tb + 255.  kPro: the instantiation
// that can apply the layer prologue to raw inputs (p.prologue says which parts); the plain instantiation
// carries none of that code.  kJoint: `quota` (0: all there are) units are taken in the order in which the scans
// running beside need them (chunk by chunk through all sequences), and a finished one is marked in its D array: at
// once with kSoon, else when the next unit's inputs are in registers.
template <typename T, typename G, typename Seqs, bool kPro, bool kJoint, bool kSoon>
__device__ __forceinline__ void prep_units(const PrepParams& p, const Seqs& seqs, const PrepMaps& tm, PrepSmem& sm,
                                           const int tid, const uint32_t tb, const int first, const int stride,
                                           const int barrier, int* queue, int quota) {
  uint8_t* const R = sm.region;
  const WsLayout ws{p.n_ch, p.training != 0};
  int* status = reinterpret_cast<int*>(p.ws + ws.off_status());
  BoundedWaiter waiter(status);
  const int warp = tid >> 5, lane = tid & 31;
  auto sync = [&] {
    if constexpr (kJoint) asm volatile("bar.sync %0, 256;" ::"r"(barrier) : "memory");
    else __syncthreads();
  };
  if (tid == 0) {
    mbar_init(&sm.bar[0], 1);
    mbar_init(&sm.bar[1], 2);
    mbar_init(&sm.bar_ld[0], 1);
    mbar_init(&sm.bar_ld[1], 1);
    fence_mbar_init();
  }
  constexpr int kMmaWarp = 6, kCopyWarp = 7;  // (the first warps have more to write)
  const int i0 = 8 * warp + 4 * (lane >> 4), cl = lane & 15;  // tokens i0 .. i0 + 3
  const int mb = warp >> 1;                   // 16-token block of this warp's tokens
  const int q4 = warp & 3, part = warp >> 2;  // TMEM lane quadrant of this warp, and its half of the columns

  // unit -> number of its tiles, head, first token row of the chunk, tokens that exist
  const int heads = p.H, n_ch = int(p.n_ch);
  struct Place { int ch, h, row, valid; };
  auto locate = [&](int unit) {
    if constexpr (kJoint) {
      const int per_chunk = seqs.count() * heads, c = int(uint32_t(unit) / uint32_t(per_chunk));
      const int r = unit - c * per_chunk, s_ = int(uint32_t(r) / uint32_t(heads));
      const SeqInfo sq = seqs.at(s_);
      unit = (sq.chunk0 + c) * heads + (r - s_ * heads);
      return Place{unit, r - s_ * heads, int(sq.row0) + c * kChunk, min(kChunk, sq.len - c * kChunk)};
    } else {
      const int chunk = int(uint32_t(unit) / uint32_t(heads));
      const SeqInfo sq = seqs.at(seqs.find(chunk));
      const int t_ = (chunk - sq.chunk0) * kChunk;
      return Place{unit, unit - chunk * heads, int(sq.row0) + t_, min(kChunk, sq.len - t_)};
    }
  };
  const uint32_t leader = elect_leader();
  auto issue_g = [&](const Place& at) {
    mbar_arrive_expect_tx(&sm.bar_ld[0], uint32_t(kChunk * kDim * sizeof(G)), leader);
    tma_load_3d(R + kOffInG, &tm.g, 0, at.h, at.row, &sm.bar_ld[0], leader);
  };
  auto issue_kq = [&](const Place& at) {
    mbar_arrive_expect_tx(&sm.bar_ld[1], 3 * kStageTile16, leader);  // (beta among them)
    tma_load_4d(R + kOffInK, &tm.k, 0, at.row, 0, at.h, &sm.bar_ld[1], leader);
    tma_load_4d(R + kOffInQ, &tm.q, 0, at.row, 0, at.h, &sm.bar_ld[1], leader);
  };
  auto issue_b = [&](const Place& at) { tma_load_4d(R + kOffInBeta, &tm.beta, 0, at.row, 0, at.h, &sm.bar_ld[1], leader); };
  sync();
  if (warp == kCopyWarp && first < n_ch) {
    const Place at = locate(first);
    issue_g(at);
    issue_kq(at);
    issue_b(at);
  }
  const bool pro_norm = kPro && (p.prologue & kPrologueNorm) != 0;
  const bool pro_gate = kPro && (p.prologue & kPrologueGate) != 0;
  using RawG = typename Raw2<G>::type;
  using RawT = typename Raw2<T>::type;
  uint32_t par = 0;
  // joint launch, the copying warp: the unit after this one, and one whose tiles are on their way out, with its mark
  [[maybe_unused]] int popped = 0, leaving = -1;
  [[maybe_unused]] float mark = 0.f;
  auto set_mark = [&] {
    if constexpr (kJoint) {
      bulk_wait_all();
      fence_async_all();
      // (the lane that committed the copies of T^T: a wait for copies is one for the thread's own, and which lane is
      // elected is not promised)
      if (leader && leaving >= 0) {
        store_release(reinterpret_cast<float*>(p.ws + ws.off_d() + int64_t(leaving) * kBlobD), mark);
      }
    }
  };
  for (int unit = first, unit_next; unit < n_ch; unit = unit_next, par ^= 1u) {
  // a queue and not a stride: an SM that shares its way to L2 with a scan prepares at little more than half
  // the pace of the others, and the scans wait for the slowest
  unit_next = unit + stride;
  if constexpr (kJoint) {
    if (warp == kCopyWarp && lane == 0) popped = --quota != 0 ? stride + atomicAdd(queue, 1) : n_ch;
  }
  // tokens of this chunk that exist: 64, fewer in the last chunk of a sequence.  The rest of the tile
  // belongs to somebody else and is replaced by the identity step (no decay, no key, no query).
  const Place here = locate(unit);
  const int ch = here.ch, n_valid = here.valid;
  const bool partial = n_valid < kChunk;
  // ---- log-decays, in units of ln 2 (a decay is one ex2): sums from the start of the 16-token block ----------
  float2 Gc[kRounds][4];
  waiter.wait(&sm.bar_ld[0], par);
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    RawG raw[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      raw[t] = *reinterpret_cast<const RawG*>(R + kOffInG + ((i0 + t) * kDim + kRound * r + 2 * cl) * sizeof(G));
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      float2 x = unpack2<G>(raw[t]);
      if (pro_gate) x = make_float2(prologue_log_decay(x.x), prologue_log_decay(x.y));
      x = (partial && i0 + t >= n_valid) ? twice(0.f) : mul2(x, twice(kLog2e));
      Gc[r][t] = t > 0 ? add2(Gc[r][t - 1], x) : x;
    }
    // the upper half of the warp goes on from the lower one
    const float2 x = make_float2(__shfl_up_sync(0xffffffffu, Gc[r][3].x, 16), __shfl_up_sync(0xffffffffu, Gc[r][3].y, 16));
    if (lane >= 16) {
#pragma unroll
      for (int t = 0; t < 4; ++t) Gc[r][t] = add2(Gc[r][t], x);
      *reinterpret_cast<float2*>(&sm.part[warp][kRound * r + 2 * cl]) = Gc[r][3];
    }
  }
  if (warp == kCopyWarp) {
    bulk_wait_read_all();  // the last unit's Y^T has left
    if (unit != first) issue_b(here);
  }
  sync();
  // A thread per channel: what precedes each group in its block, and the decay table, row by row:
  //   0..3 exp(a_I), a_I = sum up to block I   4..7 exp(a_{I+1} - a_I)   8..11 exp(a_end - a_{I+1})   12 exp(a_3 - a_1)
  float* const table = reinterpret_cast<float*>(R + kOffTable);
  if (tid < kDim) {
    float x[8], block[4];
#pragma unroll
    for (int t = 0; t < 8; ++t) x[t] = sm.part[t][tid];
#pragma unroll
    for (int I = 0; I < 4; ++I) {
      sm.part[2 * I][tid] = 0.f;
      sm.part[2 * I + 1][tid] = x[2 * I];
      block[I] = x[2 * I] + x[2 * I + 1];
    }
    const float a1 = block[0], a2 = a1 + block[1], a3 = a2 + block[2], end = a3 + block[3];
    sm.gend[tid] = end;
    // (element 0 of D doubles as the mark of a finished unit: see the end of the loop)
    if (!kJoint || tid > 0) reinterpret_cast<float*>(p.ws + ws.off_d() + int64_t(ch) * kBlobD)[tid] = exp2_approx(end);
    table[tid] = 1.f;
    table[kDim + tid] = exp2_approx(a1);
    table[2 * kDim + tid] = exp2_approx(a2);
    table[3 * kDim + tid] = exp2_approx(a3);
#pragma unroll
    for (int I = 0; I < 4; ++I) table[(4 + I) * kDim + tid] = exp2_approx(block[I]);
    table[8 * kDim + tid] = exp2_approx(block[1] + block[2] + block[3]);
    table[9 * kDim + tid] = exp2_approx(block[2] + block[3]);
    table[10 * kDim + tid] = exp2_approx(block[3]);
    table[11 * kDim + tid] = 1.f;
    table[12 * kDim + tid] = exp2_approx(block[1] + block[2]);
  }
  waiter.wait(&sm.bar_ld[1], par);
  RawT rk[4], rq[4], rb[4];
  auto read_raw = [&](int r) {
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int i = i0 + t, at = (r >> 1) * 8192 + i * 128 + ((((r & 1) * 4 + (cl >> 2)) ^ (i & 7)) << 4) + (cl & 3) * 4;
      rk[t] = *reinterpret_cast<const RawT*>(R + kOffInK + at);
      rq[t] = *reinterpret_cast<const RawT*>(R + kOffInQ + at);
      rb[t] = *reinterpret_cast<const RawT*>(R + kOffInBeta + at);
      if (partial && i0 + t >= n_valid) rk[t] = rq[t] = rb[t] = RawT{};
    }
  };
  float inv_q[4], inv_k[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) inv_q[t] = inv_k[t] = 1.f;
  if (pro_norm) {
    // sums of q^2 and k^2 over the channels: this thread's, then the sixteen lanes of a token
    float sq[4] = {}, sk[4] = {};
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      read_raw(r);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 x = unpack2<T>(rq[t]), y = unpack2<T>(rk[t]);
        sq[t] += x.x * x.x + x.y * x.y;
        sk[t] += y.x * y.x + y.y * y.y;
      }
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
#pragma unroll
      for (int off = 1; off < 16; off <<= 1) {
        sq[t] += __shfl_xor_sync(0xffffffffu, sq[t], off);
        sk[t] += __shfl_xor_sync(0xffffffffu, sk[t], off);
      }
      inv_q[t] = rsqrtf(sq[t] + kPrologueEps);
      inv_k[t] = rsqrtf(sk[t] + kPrologueEps);
    }
  }
  read_raw(0);
  sync();
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const float2 base = *reinterpret_cast<const float2*>(&sm.part[warp][kRound * r + 2 * cl]);
#pragma unroll
    for (int t = 0; t < 4; ++t) Gc[r][t] = add2(Gc[r][t], base);
  }

  if (!kSoon && warp == kCopyWarp) set_mark();

  // ---- Gram products P_I = [E_a ; Q_a] (K^I)^T on the tensor cores, 32 channels at a time ------------------
  float* const tile_q = reinterpret_cast<float*>(p.tiles.q + int64_t(ch) * kTileQ);
  float* const tile_kn = reinterpret_cast<float*>(p.tiles.kn + int64_t(ch) * kTileKn);
  // (a loop, with the round's sums shifted into place at its end: unrolled it would be 4 x the code, and the
  // compiler's moves across the rounds cost more registers than there are)
#pragma unroll 1
  for (int r = 0; r < kRounds; ++r) {
    const int kc0 = kRound * r + 2 * cl;
    auto row = [&](int t) { return *reinterpret_cast<const float2*>(table + t * kDim + kc0); };
    const float2 e_amb = row(mb);
    // before their rounding: beta k and scale q decayed from the block's anchor, k decayed to it and to the next one
    float2 ba[4], qa[4], ko[4], nb[4];
    {
      const float2 c_nx = row(4 + mb);  // decay over the whole 16-token block (<= 1)
      const float2 t_end = row(8 + mb);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 G2 = Gc[0][t];
        const float2 anchored = exp2_2(G2);                    // <= 1
        const float2 own = exp2_2(make_float2(-G2.x, -G2.y));  // >= 1, bounded by the 16-token contract
        float2 k = unpack2<T>(rk[t]), b = unpack2<T>(rb[t]), q = mul2(unpack2<T>(rq[t]), twice(p.scale));
        if (pro_gate) b = make_float2(prologue_sigmoid(b.x), prologue_sigmoid(b.y));
        if (pro_norm) {
          k = mul2(k, twice(inv_k[t]));
          q = mul2(q, twice(inv_q[t]));
        }
        ba[t] = mul2(mul2(b, k), anchored);
        qa[t] = mul2(q, anchored);
        ko[t] = mul2(k, own);
        nb[t] = mul2(k, mul2(own, c_nx));
        // token-major tiles Q[i][k] and Kn[i][k]: 16 lanes write 128 consecutive bytes
        *reinterpret_cast<float2*>(tile_q + (i0 + t) * kDim + kc0) = tf32_operand_2(mul2(qa[t], e_amb));
        *reinterpret_cast<float2*>(tile_kn + (i0 + t) * kDim + kc0) = tf32_operand_2(mul2(nb[t], t_end));
      }
    }
    if (r + 1 < kRounds) read_raw(r + 1);
    if (r > 0) waiter.wait(&sm.bar[0], (r - 1) & 1);  // the last round's operands have been multiplied
    {
      // 8 bytes of a 128-byte line, whose 16-byte pieces are permuted by the line (the row numbers of K^I start at
      // multiples of 16: one permutation for all)
      auto put = [&](int line0, const float2 (&x)[4]) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int i = i0 + t;
          *reinterpret_cast<float2*>(R + line0 * 128 + i * 128 + (((cl >> 1) ^ (i & 7)) << 4) + (cl & 1) * 8) =
              tf32_operand_2(x[t]);
        }
      };
      put(kOffGramA / 128, ba);
      put(kOffGramA / 128 + 64, qa);
      // token i is a row of every K^I, I >= its own block
      put(kOffGramB / 128 + gram_col(mb), ko);
      if (mb < 3) put(kOffGramB / 128 + gram_col(mb + 1), nb);
      if (mb < 2) {
        const float2 far = row(5 + mb);  // on over the next block
        float2 y[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) y[t] = mul2(nb[t], far);
        put(kOffGramB / 128 + gram_col(mb + 2), y);
      }
      if (mb < 1) {
        const float2 far = row(12);      // ... and the one after that
        float2 y[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) y[t] = mul2(nb[t], far);
        put(kOffGramB / 128 + gram_col(3), y);
      }
    }
    fence_async_smem();
    tc_fence_before();
    sync();
    if (warp == kMmaWarp) {
      tc_fence_after();
      // the four anchored copies K^0 .. K^3 are stacked (16 + 32 + 48 + 64 = 160 rows) and their products
      // sit side by side in TMEM, so one N = 160 instruction per k-step reads the A tile once for all four
      const uint32_t id = idesc(128, 160, kFmtTF32, kMajorK, kMajorK);
      const uint32_t a0 = smem_u32(R + kOffGramA), b0 = smem_u32(R + kOffGramB);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        mma_tf32_ss(tb, smem_desc_sw128_k(a0, 0, ks), smem_desc_sw128_k(b0, 0, ks), id, (r | ks) > 0 ? 1u : 0u, leader);
      }
      mma_commit(&sm.bar[0], leader);
    }
    // E[i][channels of this thread]: 8 bytes of line i of a slab, 32-byte pieces permuted by the line
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int i = i0 + t, slab = (r >> 1) | ((r & 1) << 1);
      *reinterpret_cast<float2*>(R + kOffE + slab * 8192 + i * 128 + (((cl >> 2) ^ (i & 3)) << 5) + (cl & 3) * 8) =
          tf32_operand_2(mul2(ba[t], e_amb));
    }
#pragma unroll
    for (int n = 0; n + 1 < kRounds; ++n) {
#pragma unroll
      for (int t = 0; t < 4; ++t) Gc[n][t] = Gc[n + 1][t];
    }
  }
  waiter.wait(&sm.bar[0], 1);
  tc_fence_after();
  float* const Lt = reinterpret_cast<float*>(R + kOffLt);     // [64][64]    -L transposed: Lt[m][r] = -L[r][m]
  float* const P = reinterpret_cast<float*>(R + kOffP);       // [32][32]    T[..32][..32]
  float* const Qt = reinterpret_cast<float*>(R + kOffQt);     // [32][kLdQ]  Qt[m][r] = T[32 + r][32 + m]
  float* const W = reinterpret_cast<float*>(R + kOffW);       // [32][64]    -L[32.., ..32) T[..32][..32]
  // -L (rows 0..63) goes into fp32 scratch, A_qk (rows 64..127) into the workspace; the two warps of a quadrant take 32
  // columns each.  A_qk is stored behind the barrier, beside the first step of the inverse, which its warps have no
  // part in: the stores queue behind those of the rounds, and the inverse would wait for them.
  const int gram_row = 32 * q4 + lane;  // TMEM lane = row of [E_a ; Q_a]
  float a_qk[2][16];
  {
    const int r = gram_row;
    const int i = r & 63;
    const int I_lo = (q4 & 1) * 2;
    const int my_I = I_lo + (lane >> 4);
#pragma unroll
    for (int sub = 0; sub < 2; ++sub) {
      const int c0 = 32 * part + 16 * sub;
      uint32_t lo[16], hi[16];
      const bool need_lo = c0 < 16 * (I_lo + 1), need_hi = c0 < 16 * (I_lo + 2);
      if (need_lo) tmem_ld16(tmem_addr(tb, 32 * q4, gram_col(I_lo) + c0), lo);
      if (need_hi) tmem_ld16(tmem_addr(tb, 32 * q4, gram_col(I_lo + 1) + c0), hi);
      tmem_wait_ld();
      float (&vals)[16] = a_qk[sub];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const bool mine_lo = (my_I == I_lo);
        const float x = mine_lo ? (need_lo ? __uint_as_float(lo[j]) : 0.f) : (need_hi ? __uint_as_float(hi[j]) : 0.f);
        const int col = c0 + j;
        vals[j] = (r < 64) ? ((col < i) ? -x : 0.f) : ((col <= i) ? to_tf32_operand(x) : 0.f);
      }
      if (r < 64 && need_hi) {  // (nobody reads the block of zeros)
#pragma unroll
        for (int j = 0; j < 16; ++j) Lt[(c0 + j) * kChunk + i] = vals[j];
      }
    }
  }
  tc_fence_before();
  sync();
  // the Gram operands are dead: the next unit's g may have their place
  if (warp == kCopyWarp) {
    if constexpr (kJoint) {
      unit_next = __shfl_sync(0xffffffffu, popped, 0);
      if (lane == 0) sm.next[par] = unit_next;
    }
    if (unit_next < n_ch) {
      const Place at = locate(unit_next);
      issue_g(at);
      // beta has to wait for Y^T to leave and is needed soon after: 393 -> 373 us (B8 T4096 H16).  In a joint launch, whose
      // Y^T leaves by itself, it is only in the way (B1 T8192 H16 225 -> 229 us).
      if (!kJoint) tma_prefetch_l2_4d(&tm.beta, 0, at.row, 0, at.h, leader);
    }
  }
  if (gram_row >= 64) {
    // A_qk leaves transposed, At[j][i]: the 32 lanes of a warp (rows i) fill one 128-byte line per column j;
    // the quadrant j >= 32, i < 32 is zero and stays unwritten (nobody reads it)
    float* tile_at = reinterpret_cast<float*>(p.tiles.at + int64_t(ch) * kTileAt) + gram_row - 64;
    if (part == 0 || gram_row >= 96) {
#pragma unroll
      for (int j = 0; j < 32; ++j) tile_at[(32 * part + j) * kChunk] = a_qk[j >> 4][j & 15];
    }
  }

  // ---- T = (I + L)^-1 ----------------------------------------------------------------------------------------
  // The two 32 x 32 diagonal blocks by substitution, a warp each and a lane per column: what a finished entry adds to
  // all later ones is independent, and the factor L is the same for all lanes, four rows of it a broadcast.  Then
  // T[32.., ..32) = -T[32.., 32..) (L[32.., ..32) T[..32, ..32)) in two products of four warps, a lane 4 rows x 2
  // columns.  (16 x 16 blocks, whose products read both factors lane by lane, were a third of all wavefronts, 6 barriers
  // and 6.4 thousand clocks a unit.)
  auto ld4 = [](const float* ptr) { return *reinterpret_cast<const float4*>(ptr); };
  // T^T[j][i .. i + 3]: lines of 32 tokens i, two slabs, 32-byte pieces permuted by the line
  auto put_t = [&](int j, int i, float2 lo, float2 hi) {
    lo = tf32_operand_2(lo);
    hi = tf32_operand_2(hi);
    *reinterpret_cast<float4*>(R + kOffTt + (i >> 5) * 8192 + j * 128 + ((((i & 31) >> 3) ^ (j & 3)) << 5) + (i & 4) * 4) =
        make_float4(lo.x, lo.y, hi.x, hi.y);
  };
  if (warp < 2) {
    const float* l0 = Lt + 32 * warp * (kChunk + 1);
    float2 x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) x[r] = make_float2(lane == 2 * r ? 1.f : 0.f, lane == 2 * r + 1 ? 1.f : 0.f);
#pragma unroll
    for (int m = 0; m < 31; ++m) {
      const float2 xm = twice((m & 1) ? x[m >> 1].y : x[m >> 1].x);
#pragma unroll
      for (int r4 = (m + 1) / 4; r4 < 8; ++r4) {  // (entries up to m meet zeros)
        const float4 l = ld4(l0 + m * kChunk + 4 * r4);
        x[2 * r4] = fma2(make_float2(l.x, l.y), xm, x[2 * r4]);
        x[2 * r4 + 1] = fma2(make_float2(l.z, l.w), xm, x[2 * r4 + 1]);
      }
    }
    if (warp == 0) {
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        P[2 * r * 32 + lane] = x[r].x;
        P[(2 * r + 1) * 32 + lane] = x[r].y;
      }
    } else {
#pragma unroll
      for (int r = 0; r < 16; r += 2) {
        *reinterpret_cast<float4*>(Qt + lane * kLdQ + 2 * r) = make_float4(x[r].x, x[r].y, x[r + 1].x, x[r + 1].y);
      }
    }
#pragma unroll
    for (int r = 0; r < 16; r += 2) put_t(32 * warp + lane, 32 * warp + 2 * r, x[r], x[r + 1]);
  } else if (warp < 6) {
    // the block of zeros, j >= 32, i < 32 (it does not leave)
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      *reinterpret_cast<float4*>(R + kOffTt + 4096 + (tid - 64 + 128 * x) * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  sync();
  // rows r0 .. r0 + 3, columns c0, c0 + 1 of a product: the sum over m of rows[m][r0 ..] cols[m][c0 ..], in two chains
  const int r0 = 8 * (warp - 2) + 4 * (lane >> 4), c0 = 2 * (lane & 15);
  auto product = [&](const float* rows, int ld_rows, const float* cols, int ld_cols, float2 (&out)[2][2]) {
    float2 acc[2][2][2] = {};
#pragma unroll
    for (int m = 0; m < 32; ++m) {
      const float4 a = ld4(rows + m * ld_rows + r0);
      const float2 b = *reinterpret_cast<const float2*>(cols + m * ld_cols + c0);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float2 bc = twice(c ? b.y : b.x);
        acc[m & 1][c][0] = fma2(make_float2(a.x, a.y), bc, acc[m & 1][c][0]);
        acc[m & 1][c][1] = fma2(make_float2(a.z, a.w), bc, acc[m & 1][c][1]);
      }
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
#pragma unroll
      for (int x = 0; x < 2; ++x) out[c][x] = add2(acc[0][c][x], acc[1][c][x]);
    }
  };
  const bool multiplies = warp >= 2 && warp < 6;
  if (multiplies) {
    float2 w[2][2];
    product(Lt + 32, kChunk, P, 32, w);
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      *reinterpret_cast<float2*>(W + (r0 + 2 * x) * kChunk + c0) = make_float2(w[0][x].x, w[1][x].x);
      *reinterpret_cast<float2*>(W + (r0 + 2 * x + 1) * kChunk + c0) = make_float2(w[0][x].y, w[1][x].y);
    }
  }
  sync();
  if (multiplies) {
    float2 t[2][2];
    product(Qt, kLdQ, W, kChunk, t);
    put_t(c0, 32 + r0, t[0][0], t[0][1]);
    put_t(c0 + 1, 32 + r0, t[1][0], t[1][1]);
  }
  fence_async_smem();
  tc_fence_before();
  sync();

  // ---- Y^T = E^T T^T (both read MN-major), while T^T leaves -----------------------------------------------------
  if (warp == kMmaWarp) {
    tc_fence_after();
    const uint32_t t0a = smem_u32(R + kOffTt), e0 = smem_u32(R + kOffE);
    const uint32_t id_y = idesc(128, 64, kFmtTF32, kMajorMN, kMajorMN);
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      mma_tf32_ss(tb, smem_desc_sw128_mn(e0, 8192, ks), smem_desc_sw128_mn(t0a, 8192, ks), id_y, ks > 0 ? 1u : 0u, leader);
    }
    mma_commit(&sm.bar[1], leader);
  }
  if (warp == kCopyWarp) {
    tma_store_4d(&tm.out_tt, 0, 0, 0, ch, R + kOffTt, leader);
    tma_store_4d(&tm.out_tt, 0, 0, 1, ch, R + kOffTt + 8192, leader);
    tma_store_4d(&tm.out_tt, 0, 32, 1, ch, R + kOffTt + 8192 + 4096, leader);
    bulk_commit();
    bulk_wait_read_all();
    mbar_arrive(&sm.bar[1], leader);
  }
  waiter.wait(&sm.bar[1], par);
  tc_fence_after();
  if (warp == kCopyWarp && unit_next < n_ch) issue_kq(locate(unit_next));
  {
    // lanes = key channels k, columns = tokens i: each warp takes 32 tokens of its quadrant, a lane 128 bytes of a row of
    // Yt[k][i].  They leave through shared memory, lines whose 16-byte pieces are permuted by their number: rows of their
    // own stored by the lanes take five times the wavefronts.  Not so in a joint launch, where the scans beside are held
    // up more than that is worth (B1 T32768 H16 805 us by the lanes, 861 through shared memory; T16384 416 and 440).
    const int kr = 32 * ((q4 >> 1) | ((q4 & 1) << 1)) + lane;  // (slabs in the order 0, 2, 1, 3)
    uint32_t r[32];
    tmem_ld32(tmem_addr(tb, 32 * q4, 32 * part), r);
    tmem_wait_ld();
    float y[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) y[j] = to_tf32_operand(__uint_as_float(r[j]));
    if constexpr (kJoint) {
      float* row = reinterpret_cast<float*>(p.tiles.yt + int64_t(ch) * kTileYt) + kr * kChunk + 32 * part;
      const bool wide_tiles = (reinterpret_cast<uintptr_t>(p.tiles.yt) & 31) == 0;  // (a tile is 32 KiB)
#pragma unroll
      for (int j = 0; j < 32; j += 8) {
        const float4 lo = make_float4(y[j], y[j + 1], y[j + 2], y[j + 3]);
        const float4 hi = make_float4(y[j + 4], y[j + 5], y[j + 6], y[j + 7]);
        // (buffers are 16-byte aligned by contract; from an allocator they are 32-byte aligned as well)
        if (wide_tiles) {
          store_global_32b(row + j, lo, hi);
        } else {
          *reinterpret_cast<float4*>(row + j) = lo;
          *reinterpret_cast<float4*>(row + j + 4) = hi;
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        *reinterpret_cast<float4*>(R + kOffY + part * 16384 + kr * 128 + (((j >> 2) ^ (kr & 7)) << 4)) =
            make_float4(y[j], y[j + 1], y[j + 2], y[j + 3]);
      }
    }
  }
  // (what the scan of a joint launch reads through the copy engine, another proxy than these stores)
  if constexpr (kJoint) fence_async_all();
  else fence_async_smem();
  tc_fence_before();  // the next unit's products replace these accumulators
  sync();
  if (!kJoint && warp == kCopyWarp) {
    tma_store_4d(&tm.out_yt, 0, 0, 0, ch, R + kOffY, leader);
    bulk_commit();
  }
  if constexpr (kJoint) {
    // A finished unit is marked by the sign of D[0] (a decay is never negative) once its tiles are in memory: the
    // copying warp looks to that here or when it has the next unit's sums.
    unit_next = sm.next[par];
    leaving = ch;
    mark = __uint_as_float(__float_as_uint(exp2_approx(sm.gend[0])) | 0x80000000u);
    if (kSoon && warp == kCopyWarp) set_mark();
  }
  }  // units of this group
  if (warp == kCopyWarp) {
    bulk_wait_all();  // the last tiles are in memory before the CTA goes on
    set_mark();       // (with kSoon once more the same)
  }
}

template <typename T, typename G, typename Seqs, bool kPro = false>
__global__ void __launch_bounds__(kPrepThreads, 2)
chunk_prep_kernel(const PrepParams p, const __grid_constant__ Seqs seqs, const __grid_constant__ PrepMaps tm) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  PrepSmem& sm = *reinterpret_cast<PrepSmem*>(smem_raw);
  if (threadIdx.x < 32) {
    tmem_alloc(&sm.tmem_base, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tb = sm.tmem_base;
  prep_units<T, G, Seqs, kPro, false, false>(p, seqs, tm, sm, threadIdx.x, tb, int(blockIdx.x), int(gridDim.x), 0, nullptr, 0);
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) tmem_dealloc(tb, 256);
}

// ---------------------------------------------------------------------------------------------
// scan kernel
// ---------------------------------------------------------------------------------------------
// Warp-specialised.  What bounds a scan of few heads is the latency of one chunk, which walks the chain
// S -> R -> S; in phases that all warps go through together a chunk took 3.8-5 us (every phase waited for
// the tensor cores and the tensor cores for every phase).  Here the MMAs of a chunk are issued back to
// back by one warp and everything else runs beside them:
//   warp 0       tiled TMA loads, each buffer refilled as soon as its MMA has read it (one lane)
//   warp 3       MMAs, per chunk:  R^T -= S^T Y^T | O^T = S^T Qg^T | S'^T += R^T Kt | O^T += R^T Aqk^T |
//                R'^T = Z'^T T^T of the next chunk.  MMAs of one shape on one accumulator run in order; every
//                other dependence (R -> S', S' -> R') is waited for, with independent MMAs in the queue meanwhile
//   warp 2       loads of v and w, whose buffer frees at another time than the others
//   warps 4..11  decay: S' <- S diag(d) into the other of two state buffers while R is formed (the output
//                still reads S); training: the chunk-start state, staged and sent by bulk stores
//   warps 12..19 Z = w v of the next chunk into tensor memory; training: R out
//   warps 20..23 O out (staged, one TMA store); in a joint launch, whose preparing CTAs need the registers, the Z
//                warps do it (where loads are late, Z waits for them and O behind it: 691 -> 743 us at
//                B4 T8192 H32 training, so not in a launch of its own)
// A passed mbarrier wait costs ~150 clocks, so what an MMA group needs arrives on one barrier: the bytes of
// its tiles, the threads that wrote its other operand and those that freed its accumulator.
// Tensor memory (columns): S 2 x 128, R 2 x 64, O 64, Z 64 = all 512.
// Where a CTA has only the first 64 value rows, a group has work for the two warps of four that reach them, and the
// single warps take the places of others: the MMA warp is then alone on its scheduler (3300 -> 2940 clocks a chunk;
// with working warps beside it an MMA is issued in 50 clocks instead of 25).  In a joint launch, which has this form
// only, one more warp watches the marks of prepared chunks (a look at one takes most of a microsecond); it is on the
// MMA warp's scheduler too, and asleep for 200 ns between looks.
template <int kParts>
struct ScanWarps {  // (first) warps of the groups
  static constexpr int kLoads = 0, kVw = 2, kMma = 3, kDecay0 = 4, kZ0 = 12, kOut0 = 20, kThreads = 768;
  static __device__ __forceinline__ bool works(int warp) { return warp >= kDecay0; }
};
template <>
struct ScanWarps<2> {
  static constexpr int kLoads = 2, kWatch = 7, kVw = 6, kMma = 3, kDecay0 = 0, kZ0 = 8, kOut0 = 16, kThreads = 576;
  static __device__ __forceinline__ bool works(int warp) { return (warp & 3) < 2; }
};

struct ScanSmem {
  // swizzled operand tiles, slabs of 32 columns (tc05.cuh): Q is read K-major, the others MN-major
  alignas(1024) uint8_t yt[32768];   // Yt[k][i]: 2 slabs of 128 lines
  alignas(1024) uint8_t q[32768];    // Q[i][k]:  4 slabs of 64 lines
  alignas(1024) uint8_t kn[32768];   // Kn[j][k]: 4 slabs of 64 lines
  alignas(1024) uint8_t at[16384];   // At[j][i]: 2 slabs of 64 lines
  alignas(1024) uint8_t tt[16384];   // Tt[j][i]: 2 slabs of 64 lines
  alignas(128) uint8_t v[16384];     // raw v, w of the chunk, [64][128] 16-bit rows (halves of two chunks)
  alignas(128) uint8_t w[16384];
  alignas(128) uint8_t o[16384];     // output rows [64][128] on their way out (one TMA store: 64-byte pieces
                                     // stored by threads at the stride of a token row drain at 2 bytes per clock)
  alignas(128) float ck[2][32 * kDim];  // training: 32 rows of the chunk-start state per half of the decay group
  alignas(16) float d[2][kDim];
  alignas(8) uint64_t full_vw[2], full_d[2];
  uint64_t go_u;      // Tt, Z written (and the R before the last read):          1 load + 8 warps
  uint64_t go_r;      // Yt, the state of the last chunk:                         1 load + 1 commit
  uint64_t go_o;      // Q, the O of the last chunk read:                         1 load + the warps of O
  uint64_t go_s;      // Kn, At, decayed state, R:                                2 loads + 8 warps + 1 commit
  uint64_t vw_read[2];  // v, w are in registers:                                   8 warps
  uint64_t u_done, r_done, q_done, s_done, o_done, all_done;  // MMA commits
  volatile int failed;
  volatile int prepared;  // chunks whose tiles may be loaded
  uint32_t tmem_base;
};
static_assert(sizeof(ScanSmem) <= 232448, "forward scan exceeds the 227 KiB shared-memory limit");

struct ScanParams {
  const uint8_t* d;    // chunk-end decays, 512 bytes per unit
  const float* s_in;   // [sequences,H,128,128] or null
  void* out;           // [rows,H,128]
  float* s_out;        // [sequences,H,128,128] or null
  float* bnd;          // chunk-start states, one slot more than chunks per sequence, or null
  float* rn;           // residual tiles (training) or null
  int* status;
  int H;
  int activate_w;      // w holds pre-activations
};
struct ScanMaps {
  CUtensorMap yt, q, kn, at, tt, v, w, out;
};

// One sequence and head, or a half of its value rows (kParts = 2: value_parts), by a whole CTA.  kJoint: the prep
// groups run beside in the same launch, and a chunk's tiles are loaded once its mark is there.
template <typename T, typename Seqs, bool kJoint, int kParts>
__device__ __forceinline__ void scan_sequence(const ScanParams& p, const Seqs& seqs, const ScanMaps& tm, ScanSmem& sm,
                                              const int item) {
  constexpr int kRows = kDim / kParts;  // value rows of this CTA: lanes 0 .. kRows - 1 of tensor memory
  constexpr int kVwSlots = kParts;      // halves of v and w leave room for those of the next chunk
  using W = ScanWarps<kParts>;
  constexpr int kThreads = kJoint ? 32 * W::kOut0 : W::kThreads;
  BoundedWaiter waiter(p.status, 1u << 20, &sm.failed);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int unit = item / kParts, v0 = (item - unit * kParts) * kRows;
  const int s = unit / p.H, h = unit - s * p.H;
  const SeqInfo sq = seqs.at(s);
  const int n_chunks = sq.n_chunks;
  constexpr uint32_t kColS = 0, kColR = 256, kColO = 384, kColZ = 448;
  auto ch_of = [&](int c) { return int64_t(sq.chunk0 + c) * p.H + h; };

  if (warp == W::kMma) {
    tmem_alloc(&sm.tmem_base, 512);
    tmem_relinquish();
  }
  if (tid == 0) {
    for (int i = 0; i < kVwSlots; ++i) {
      mbar_init(&sm.full_vw[i], 1);
      mbar_init(&sm.vw_read[i], 8 / kParts);
    }
    mbar_init(&sm.full_d[0], 1);
    mbar_init(&sm.full_d[1], 1);
    mbar_init(&sm.go_u, 1 + 8 / kParts);
    mbar_init(&sm.go_r, 1 + 1);
    mbar_init(&sm.go_o, 1 + (kJoint ? 8 : 4) / kParts);
    mbar_init(&sm.go_s, 2 + 8 / kParts + 1);
    mbar_init(&sm.u_done, 1); mbar_init(&sm.r_done, 1); mbar_init(&sm.q_done, 1);
    mbar_init(&sm.s_done, 1); mbar_init(&sm.o_done, 1); mbar_init(&sm.all_done, 1);
    mbar_arrive(&sm.go_r);  // no earlier chunk holds up the first one
    // a wait that ran out in the prep kernel left garbage tiles: results become NaN from the start
    sm.failed = *static_cast<volatile const int*>(p.status) != kStatusOk;
    sm.prepared = 0;
    fence_mbar_init();
  }
  // lines 32..63 of the first slab of At and Tt (j >= 32, i < 32) are never loaded: zero, once
  for (int e = tid; e < 4096 / 16; e += kThreads) {
    reinterpret_cast<float4*>(sm.at + 4096)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    reinterpret_cast<float4*>(sm.tt + 4096)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tb = sm.tmem_base;
  auto arrive = [&](uint64_t* bar) {  // one arrival per warp, after its tensor-memory accesses
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  };
  auto watches = [&] {
    if constexpr (kJoint) return warp == W::kWatch;
    return false;
  };

  // O of a chunk out, by whole sets of four warps (one per lane quadrant of tensor memory), each `kTokens` of
  // the 64 tokens from i0 on
  auto emit_o = [&](auto tokens, int c, int i0, int group0) {
    constexpr int kTokens = decltype(tokens)::value, kGroup = kRows * (kChunk / kTokens);
    const int vrow = 32 * (warp & 3) + lane;
    const bool sender = tid == group0 * 32;
    waiter.wait(&sm.o_done, uint32_t(c) & 1u);
    tc_fence_after();
    uint32_t x[kTokens];
#pragma unroll
    for (int j = 0; j < kTokens; j += 32) {
      tmem_ld32(tmem_addr(tb, 32u * (warp & 3), kColO + i0 + j), *reinterpret_cast<uint32_t(*)[32]>(&x[j]));
    }
    tmem_wait_ld();
    if (c + 1 < n_chunks) arrive(&sm.go_o);
    const bool failed = sm.failed != 0;
    if (sender) bulk_wait_read_all();  // the previous chunk's rows have left the buffer
    asm volatile("bar.sync 4, %0;" ::"n"(kGroup) : "memory");
    T* tile = reinterpret_cast<T*>(sm.o) + i0 * kRows + vrow;
#pragma unroll
    for (int j = 0; j < kTokens; j += 2) {
      typename Pair<T>::type y = Pair<T>::make(__uint_as_float(x[j]), __uint_as_float(x[j + 1]));
      if (failed) y = Pair<T>::make(poison_nan(), poison_nan());
      tile[j * kRows] = y.x;
      tile[(j + 1) * kRows] = y.y;
    }
    fence_async_smem();
    asm volatile("bar.sync 4, %0;" ::"n"(kGroup) : "memory");
    const int row = int(sq.row0) + c * kChunk, n_valid = min(kChunk, sq.len - c * kChunk);
    if (n_valid == kChunk) {
      if (sender) {
        tma_store_3d(&tm.out, v0, h, row, sm.o);
        bulk_commit();
      }
    } else {  // the rows behind a partial chunk (the last one) belong to somebody else
      constexpr int kPieces = kRows / 8;  // 16-byte pieces of a row
      const int first = (kTokens == kChunk ? 0 : (i0 / kTokens) * kRows) + vrow;
      for (int e = first; e < n_valid * kPieces; e += kGroup) {
        *reinterpret_cast<uint4*>(static_cast<T*>(p.out) + (int64_t(row + e / kPieces) * p.H + h) * kDim + v0 +
                                  8 * (e % kPieces)) = *reinterpret_cast<const uint4*>(sm.o + e * 16);
      }
    }
    if (sender && c + 1 == n_chunks) bulk_wait_all();  // the last rows are in global memory before the CTA retires
  };

  if (warp == W::kLoads) {
    // ---------------------------------------------------------------- loads
    const uint32_t leader = elect_leader();
    // Tt and At are zero for j >= 32, i < 32: three 32-row boxes, the fourth quadrant of the tile stays zero
    auto load_tri = [&](uint8_t* dst, const CUtensorMap* map, int ch, uint64_t* bar) {
      tma_load_4d(dst, map, 0, 0, 0, ch, bar, leader);
      tma_load_4d(dst + 8192, map, 0, 0, 1, ch, bar, leader);
      tma_load_4d(dst + 8192 + 4096, map, 0, 32, 1, ch, bar, leader);
    };
    auto load_t = [&](int c) {
      mbar_arrive_expect_tx(&sm.go_u, uint32_t(kTileTt - 4096), leader);
      load_tri(sm.tt, &tm.tt, int(ch_of(c)), &sm.go_u);
    };
    auto load_y = [&](int c) {
      mbar_arrive_expect_tx(&sm.go_r, uint32_t(kTileYt), leader);
      tma_load_4d(sm.yt, &tm.yt, 0, 0, 0, int(ch_of(c)), &sm.go_r, leader);
    };
    auto load_d = [&](int c) {
      mbar_arrive_expect_tx(&sm.full_d[c & 1], uint32_t(kBlobD), leader);
      bulk_g2s(sm.d[c & 1], p.d + ch_of(c) * kBlobD, uint32_t(kBlobD), &sm.full_d[c & 1], leader);
    };
    auto load_k = [&](int c) {
      mbar_arrive_expect_tx(&sm.go_s, uint32_t(kTileKn), leader);
      tma_load_4d(sm.kn, &tm.kn, 0, 0, 0, int(ch_of(c)), &sm.go_s, leader);
    };
    auto load_q = [&](int c) {
      mbar_arrive_expect_tx(&sm.go_o, uint32_t(kTileQ), leader);
      tma_load_4d(sm.q, &tm.q, 0, 0, 0, int(ch_of(c)), &sm.go_o, leader);
    };
    auto load_a = [&](int c) {
      mbar_arrive_expect_tx(&sm.go_s, uint32_t(kTileAt - 4096), leader);
      load_tri(sm.at, &tm.at, int(ch_of(c)), &sm.go_s);
    };
    int prepared = 0;  // chunks known to be prepared: a fence for each of them held up its first load by 1000 clocks
    auto ready = [&](int c) {
      if (!kJoint || c < prepared) return;
      // (the watching warp gives up by itself and then lets everything pass)
      for (uint32_t looks = 0; (prepared = sm.prepared) <= c && looks < (1u << 27); ++looks) __nanosleep(20);
      __threadfence_block();
      fence_async_all();
    };
    ready(0);
    load_t(0);
    load_y(0);
    load_d(0);
    load_q(0);
    load_k(0);
    load_a(0);
    for (int c = 1; c < n_chunks; ++c) {
      const uint32_t par = uint32_t(c - 1) & 1u;
      waiter.wait(&sm.u_done, par);
      ready(c);
      load_t(c);
      load_d(c);  // (the decay of chunk c - 2, which had the slot, has run)
      waiter.wait(&sm.r_done, par);
      load_y(c);
      waiter.wait(&sm.q_done, par);
      load_q(c);
      waiter.wait(&sm.s_done, par);
      load_k(c);
      waiter.wait(&sm.o_done, par);
      load_a(c);
    }
  } else if (warp == W::kMma) {
    // ---------------------------------------------------------------- MMAs
    // (the initial state must be in tensor memory: barrier 1, decay group and this warp)
    asm volatile("bar.sync 1, %0;" ::"n"(2 * kRows + 32) : "memory");
    tc_fence_after();
    const uint32_t leader = elect_leader();
    const uint32_t y0 = smem_u32(sm.yt), q0 = smem_u32(sm.q), a0 = smem_u32(sm.at);
    const uint32_t kn0 = smem_u32(sm.kn), t0 = smem_u32(sm.tt);
    const uint32_t id_neg_mn = idesc(128, 64, kFmtTF32, kMajorK, kMajorMN, 1, 0);
    const uint32_t id_pos_mn = idesc(128, 64, kFmtTF32, kMajorK, kMajorMN);
    const uint32_t id_pos_k = idesc(128, 64, kFmtTF32, kMajorK, kMajorK);
    const uint32_t id_s = idesc(128, 128, kFmtTF32, kMajorK, kMajorMN);
    // R^T = Z^T T^T    (A = Z columns, K = 64 tokens; B = Tt[j][i] read MN-major)
    auto issue_u = [&](int c) {
      const uint32_t r = tb + kColR + 64u * (uint32_t(c) & 1u);
      waiter.wait(&sm.go_u, uint32_t(c) & 1u);
      tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        mma_tf32_ts(r, tb + kColZ + ks * 8, smem_desc_sw128_mn(t0, 8192, ks), id_pos_mn, ks > 0 ? 1u : 0u, leader);
      }
      mma_commit(&sm.u_done, leader);
    };
    issue_u(0);
    for (int c = 0; c < n_chunks; ++c) {
      const uint32_t par = uint32_t(c) & 1u;
      const uint32_t s_old = tb + kColS + 128u * par, s_new = tb + kColS + 128u * (par ^ 1u);
      const uint32_t r = tb + kColR + 64u * par;
      waiter.wait(&sm.go_r, par);
      tc_fence_after();
      // R^T -= S^T Y^T   (A = state columns, K = 128 keys; B = Yt[k][i] read MN-major)
#pragma unroll
      for (int ks = 0; ks < 16; ++ks) {
        mma_tf32_ts(r, s_old + ks * 8, smem_desc_sw128_mn(y0, 16384, ks), id_neg_mn, 1u, leader);
      }
      mma_commit(&sm.r_done, leader);
      mma_commit(&sm.go_s, leader);
      waiter.wait(&sm.go_o, par);
      tc_fence_after();
      // O^T = S^T Qg^T   (B = Q[i][k] read K-major)
#pragma unroll
      for (int ks = 0; ks < 16; ++ks) {
        mma_tf32_ts(tb + kColO, s_old + ks * 8, smem_desc_sw128_k(q0, 8192, ks), id_pos_k, ks > 0 ? 1u : 0u, leader);
      }
      mma_commit(&sm.q_done, leader);
      waiter.wait(&sm.go_s, par);
      tc_fence_after();
      // S'^T += R^T Kt   (K = 64 tokens; B = Kn[j][k] read MN-major)
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        mma_tf32_ts(s_new, r + ks * 8, smem_desc_sw128_mn(kn0, 8192, ks), id_s, 1u, leader);
      }
      mma_commit(&sm.s_done, leader);
      if (c + 1 < n_chunks) mma_commit(&sm.go_r, leader);
      // O^T += R^T Aqk^T (B = At[j][i] read MN-major)
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        mma_tf32_ts(tb + kColO, r + ks * 8, smem_desc_sw128_mn(a0, 8192, ks), id_pos_mn, 1u, leader);
      }
      mma_commit(&sm.o_done, leader);
      if (c + 1 < n_chunks) issue_u(c + 1);
    }
    mma_commit(&sm.all_done, leader);
  } else if (warp == W::kVw) {
    // ---------------------------------------------------------------- v and w
    const uint32_t leader = elect_leader();
    auto load_vw = [&](int c) {
      const int row = int(sq.row0) + c * kChunk, slot = c % kVwSlots, at = slot * (16384 / kVwSlots);
      mbar_arrive_expect_tx(&sm.full_vw[slot], 2u * 16384u / kParts, leader);
      tma_load_3d(sm.v + at, &tm.v, v0, h, row, &sm.full_vw[slot], leader);
      tma_load_3d(sm.w + at, &tm.w, v0, h, row, &sm.full_vw[slot], leader);
    };
    for (int c = 0; c < n_chunks; ++c) {
      if (c >= kVwSlots) waiter.wait(&sm.vw_read[c % kVwSlots], uint32_t(c / kVwSlots - 1) & 1u);
      load_vw(c);
    }
  } else if (watches()) {
    // ---------------------------------------------------------------- marks of prepared chunks
    for (int c = 0; c < n_chunks;) {
      const int mine = min(c + lane, n_chunks - 1);
      const uint32_t missing = ~__ballot_sync(0xffffffffu, marked(reinterpret_cast<const float*>(p.d + ch_of(mine) * kBlobD)));
      const int there = missing == 0 ? 32 : __ffs(int(missing)) - 1;
      if (there == 0) {
        if (!waiter.look_again()) c = n_chunks;
        __nanosleep(200);
      } else {
        c = min(c + there, n_chunks);
        waiter.look_anew();
      }
      // (a wait of a preparer that ran out, or this one's own: results become NaN)
      if (*static_cast<volatile const int*>(p.status) != kStatusOk) sm.failed = 1;
      __syncwarp();
      if (lane == 0 && c > 0) {
        __threadfence_block();
        sm.prepared = c;
      }
    }
  } else if (!W::works(warp)) {
    // (nothing to do in this form)
  } else if (warp < W::kZ0) {
    // ---------------------------------------------------------------- decay of the state
    // thread = value row of the transposed state (TMEM lane) x one half of the 128 key columns
    const int q4 = warp & 3, half = (warp - W::kDecay0) >> 2;
    const int vrow = 32 * q4 + lane, k0 = 64 * half;
    const uint32_t lane_base = 32u * q4;
    const int64_t state = (int64_t(sq.sid) * p.H + h) * int64_t(kDim * kDim);
    const bool sender = lane == 0 && q4 == 0;  // sends this half's staged rows
    uint32_t lo[32], hi[32];
    const int64_t my_row = v0 + vrow;
    auto half_barrier = [&] { asm volatile("bar.sync %0, 128;" ::"r"(2 + half) : "memory"); };
    auto load_state = [&](uint32_t col) {
      tmem_ld32(tmem_addr(tb, lane_base, col + k0), lo);
      tmem_ld32(tmem_addr(tb, lane_base, col + k0 + 32), hi);
      tmem_wait_ld();
    };
    auto store_state = [&](uint32_t col) {
      tmem_st32(tmem_addr(tb, lane_base, col + k0), lo);
      tmem_st32(tmem_addr(tb, lane_base, col + k0 + 32), hi);
      tmem_wait_st();
    };
    // 32 key rows of the chunk-start state, 16 KiB, through the staging buffer of this half
    auto send_rows = [&](const uint32_t (&x)[32], int c, int kr) {
      if (sender) bulk_wait_read_all();  // the previous rows have left the buffer
      half_barrier();
      float* dst = sm.ck[half] + vrow;
#pragma unroll
      for (int j = 0; j < 32; ++j) dst[j * kDim] = __uint_as_float(x[j]);
      fence_async_smem();
      half_barrier();
      if (sender) {
        bulk_s2g(p.bnd + ((int64_t(sq.slot0 + c) * p.H + h) * kDim + kr) * kDim, sm.ck[half], 32u * kDim * 4u);
        bulk_commit();
      }
    };
    {
      const float* src = (p.s_in != nullptr) ? p.s_in + state + my_row : nullptr;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        lo[j] = (src != nullptr) ? __float_as_uint(src[(k0 + j) * kDim]) : 0u;
        hi[j] = (src != nullptr) ? __float_as_uint(src[(k0 + 32 + j) * kDim]) : 0u;
      }
      store_state(kColS);
      tc_fence_before();
      asm volatile("bar.sync 1, %0;" ::"n"(2 * kRows + 32) : "memory");
    }
    for (int c = 0; c < n_chunks; ++c) {
      const uint32_t par = uint32_t(c) & 1u;
      if (c > 0) {
        waiter.wait(&sm.s_done, par ^ 1u);
        tc_fence_after();
        load_state(kColS + 128u * par);
      }
      if (kParts == 1 && p.bnd != nullptr) send_rows(lo, c, k0);
      waiter.wait(&sm.full_d[par], uint32_t(c >> 1) & 1u);
#pragma unroll
      for (int j4 = 0; j4 < 8; ++j4) {
        const float4 da = *reinterpret_cast<const float4*>(&sm.d[par][k0 + 4 * j4]);
        const float4 db = *reinterpret_cast<const float4*>(&sm.d[par][k0 + 32 + 4 * j4]);
        lo[4 * j4 + 0] = __float_as_uint(__uint_as_float(lo[4 * j4 + 0]) * fabsf(da.x));
        lo[4 * j4 + 1] = __float_as_uint(__uint_as_float(lo[4 * j4 + 1]) * fabsf(da.y));
        lo[4 * j4 + 2] = __float_as_uint(__uint_as_float(lo[4 * j4 + 2]) * fabsf(da.z));
        lo[4 * j4 + 3] = __float_as_uint(__uint_as_float(lo[4 * j4 + 3]) * fabsf(da.w));
        hi[4 * j4 + 0] = __float_as_uint(__uint_as_float(hi[4 * j4 + 0]) * fabsf(db.x));
        hi[4 * j4 + 1] = __float_as_uint(__uint_as_float(hi[4 * j4 + 1]) * fabsf(db.y));
        hi[4 * j4 + 2] = __float_as_uint(__uint_as_float(hi[4 * j4 + 2]) * fabsf(db.z));
        hi[4 * j4 + 3] = __float_as_uint(__uint_as_float(hi[4 * j4 + 3]) * fabsf(db.w));
      }
      // (the other buffer: its readers, R and O of chunk c - 1, ran before the update that s_done stands for)
      store_state(kColS + 128u * (par ^ 1u));
      arrive(&sm.go_s);
      if (p.bnd != nullptr) {
        // the other rows, off the chain: the chunk-start state is still in its buffer, which this group alone
        // overwrites, one chunk later.  They leave by plain stores: the copy engine has 200 KB of a chunk to
        // move as it is (with these rows staged too, a chunk waited 2000 clocks for its buffer)
        float* ck = p.bnd + ((int64_t(sq.slot0 + c) * p.H + h) * kDim + k0) * kDim + my_row;
        if (kParts > 1) {  // (a part of a row is not contiguous: all of it in this way)
          tmem_ld32(tmem_addr(tb, lane_base, kColS + 128u * par + k0), lo);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) ck[j * kDim] = __uint_as_float(lo[j]);
        }
        tmem_ld32(tmem_addr(tb, lane_base, kColS + 128u * par + k0 + 32), hi);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j) ck[(32 + j) * kDim] = __uint_as_float(hi[j]);
      }
    }
    // ---- final state ---------------------------------------------------------------------------------
    waiter.wait(&sm.s_done, uint32_t(n_chunks - 1) & 1u);
    tc_fence_after();
    load_state(kColS + 128u * (uint32_t(n_chunks) & 1u));
    float* fin = (p.s_out != nullptr) ? p.s_out + state + my_row : nullptr;
    float* ck = (p.bnd != nullptr) ? p.bnd + (int64_t(sq.slot0 + n_chunks) * p.H + h) * int64_t(kDim * kDim) + my_row
                                   : nullptr;
    const bool failed = sm.failed != 0;
#pragma unroll
    for (int j = 0; j < 64; ++j) {
      const float x = failed ? poison_nan() : __uint_as_float(j < 32 ? lo[j & 31] : hi[j & 31]);
      if (fin != nullptr) fin[(k0 + j) * kDim] = x;
      if (ck != nullptr) ck[(k0 + j) * kDim] = x;
    }
    if (sender) bulk_wait_all();  // the last staged rows are in global memory before the CTA retires
  } else if (kJoint || warp < W::kOut0) {
    // ---------------------------------------------------------------- Z = w v (and in a joint launch O out)
    // thread = value row (TMEM lane) x one half of the 64 tokens
    const int q4 = warp & 3, half = (warp - W::kZ0) >> 2;
    const int vrow = 32 * q4 + lane, i0 = 32 * half;
    const uint32_t lane_base = 32u * q4;
    const T* vs = reinterpret_cast<const T*>(sm.v) + i0 * kRows + vrow;
    const T* wsrc = reinterpret_cast<const T*>(sm.w) + i0 * kRows + vrow;
    uint32_t a[32];
    // R of chunk c for backward, row-major R[j][v]: the 32 lanes of a warp fill one 128-byte line per token
    auto load_residual = [&](int c) {
      tmem_ld32(tmem_addr(tb, lane_base, kColR + 64u * (uint32_t(c) & 1u) + i0), a);
      tmem_wait_ld();
    };
    auto store_residual = [&](int c) {
      float* rn = p.rn + ch_of(c) * (kBlobRn / 4) + i0 * kDim + v0 + vrow;
#pragma unroll
      for (int j = 0; j < 32; ++j) rn[j * kDim] = to_tf32(__uint_as_float(a[j]));
    };
    auto build_z = [&](int c) {
      const int slot = c % kVwSlots, at = slot * (kChunk * kDim / kVwSlots);
      waiter.wait(&sm.full_vw[slot], uint32_t(c / kVwSlots) & 1u);
      const int n_valid = sq.len - c * kChunk;
      // 16 tokens at a time: more with their activations in flight would not fit the registers
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        T vr[16];
        float z[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          z[j] = to_float(wsrc[at + (16 * part + j) * kRows]);
          vr[j] = vs[at + (16 * part + j) * kRows];
        }
        if (part == 1) {
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.vw_read[slot]);
        }
        if (p.activate_w) {
#pragma unroll
          for (int j = 0; j < 16; ++j) z[j] = prologue_sigmoid(z[j]);
        }
        uint32_t zr[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) zr[j] = __float_as_uint(to_tf32_operand(to_float(vr[j]) * z[j]));
        if (n_valid < kChunk) {  // rows past the end of the sequence are somebody else's
#pragma unroll
          for (int j = 0; j < 16; ++j) zr[j] = (i0 + 16 * part + j < n_valid) ? zr[j] : 0u;
        }
        if (part == 0 && c > 0) {
          waiter.wait(&sm.u_done, uint32_t(c - 1) & 1u);  // and with it everything of chunk c - 2
          tc_fence_after();
        }
        tmem_st16(tmem_addr(tb, lane_base, kColZ + i0 + 16 * part), zr);
      }
      tmem_wait_st();
      if (p.rn != nullptr && c > 1) load_residual(c - 2);  // before its columns take the R of this chunk
      arrive(&sm.go_u);
      if (p.rn != nullptr && c > 1) store_residual(c - 2);
    };
    if constexpr (kJoint) arrive(&sm.go_o);  // no earlier chunk holds up the first output
    build_z(0);
    for (int c = 0; c < n_chunks; ++c) {
      if (c + 1 < n_chunks) build_z(c + 1);
      if constexpr (kJoint) emit_o(std::integral_constant<int, 32>{}, c, i0, W::kZ0);
    }
    if (p.rn != nullptr) {
      waiter.wait(&sm.all_done, 0);
      tc_fence_after();
      for (int c = max(0, n_chunks - 2); c < n_chunks; ++c) {
        load_residual(c);
        store_residual(c);
      }
    }
  } else {
    // ---------------------------------------------------------------- O out
    arrive(&sm.go_o);  // no earlier chunk holds up the first output
    for (int c = 0; c < n_chunks; ++c) emit_o(std::integral_constant<int, 64>{}, c, 0, W::kOut0);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == W::kMma) {
    tc_fence_after();
    tmem_dealloc(tb, 512);
  }
}

template <typename T, typename Seqs, int kParts>
__global__ void __launch_bounds__(ScanWarps<kParts>::kThreads, 1)
chunk_scan_kernel(const ScanParams p, const __grid_constant__ Seqs seqs, const __grid_constant__ ScanMaps tm) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if constexpr (std::is_same<Seqs, PackedSeqs>::value) let_others_begin();  // the token kernels of the short sequences
  scan_sequence<T, Seqs, false, kParts>(p, seqs, tm, *reinterpret_cast<ScanSmem*>(smem_raw), int(blockIdx.x));
}

// ---------------------------------------------------------------------------------------------
// prep and scan in one launch
// ---------------------------------------------------------------------------------------------
// With few sequences and heads the scan is a serial chain on a few SMs (1.6-2 us per chunk) while the others
// idle, and it starts when the last prep unit is done.  Here some CTAs scan and the others prepare, chunk by
// chunk; the tiles are still in L2 when the scan reads them.  The scans wait for the preparers, which wait
// for nobody; the launch is cooperative, so that all CTAs are resident together.
// The two SMs of a pair share their way to L2 (with a preparer beside it a scan took 3.3 us per chunk): the CTAs
// come in clusters of two, and those of a scanning pair take half of the value rows each.  512 threads leave a
// preparing group the 128 registers a thread that it has in a launch of its own.  us, against one scanning CTA a
// pair and 96 registers, when this form was made: B1 T8192 H16 364 -> 233, B1 T32768 H16 1521 -> 820 (raw 1112 -> 960).
// With a faster preparation and other numbers of CTAs it takes 224 and 802 (raw 921).
constexpr int kJointThreads = 512;
struct JointSmem {
  PrepSmem prep[2];
};
template <typename T, typename G, typename Seqs, bool kPro, bool kSoon>
__global__ void __launch_bounds__(kJointThreads, 1) __cluster_dims__(2, 1, 1)
chunk_joint_kernel(const PrepParams pp, const ScanParams sp, const __grid_constant__ Seqs seqs,
                   const __grid_constant__ PrepMaps tm_prep, const __grid_constant__ ScanMaps tm_scan,
                   const int quota) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int tid = threadIdx.x, n_scan = kJointParts * seqs.count() * sp.H;
  const bool scans = int(blockIdx.x) < n_scan;
  if (!scans || quota > 0) {
    // number of this CTA among those that prepare from the start
    const int nr = quota > 0 ? int(blockIdx.x) : int(blockIdx.x) - n_scan;
    const int n_groups = 2 * (quota > 0 ? int(gridDim.x) : int(gridDim.x) - n_scan);
    JointSmem& sm = *reinterpret_cast<JointSmem*>(smem_raw);
    if (tid < 32) {
      tmem_alloc(&sm.prep[0].tmem_base, 512);
      if (!scans) tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tb = sm.prep[0].tmem_base;
    const int group = tid >> 8;
    prep_units<T, G, Seqs, kPro, true, kSoon>(pp, seqs, tm_prep, sm.prep[group], tid & 255, tb + 256u * group,
                                       group * (n_groups / 2) + nr, n_groups, 1 + group, sp.status + kQueueWord,
                                       scans ? quota : 0);
    tc_fence_before();
    __syncthreads();
    if (tid < 32) {
      tc_fence_after();
      tmem_dealloc(tb, 512);
    }
    if (!scans) return;
    if ((tid & 255) == 0) {  // the scan's shared memory lies over these
      for (uint64_t* bar : {&sm.prep[group].bar[0], &sm.prep[group].bar[1], &sm.prep[group].bar_ld[0], &sm.prep[group].bar_ld[1]}) {
        mbar_inval(bar);
      }
    }
    __syncthreads();
  }
  scan_sequence<T, Seqs, true, kJointParts>(sp, seqs, tm_scan, *reinterpret_cast<ScanSmem*>(smem_raw), int(blockIdx.x));
}

// ---------------------------------------------------------------------------------------------
// test aid: a bounded wait that runs out
// ---------------------------------------------------------------------------------------------
// One CTA allocates tensor memory like the real kernels, waits with their BoundedWaiter on an
// mbarrier that nothing arms, and must come back by itself: status word set, tensor memory freed.
__global__ void __launch_bounds__(128, 1) debug_wait_expires_kernel(int* status, uint32_t max_polls) {
  __shared__ alignas(8) uint64_t bar;
  __shared__ uint32_t tmem_base;
  const int warp = threadIdx.x >> 5;
  if (warp == 0) {
    tmem_alloc(&tmem_base, 32);
    tmem_relinquish();
  }
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  BoundedWaiter waiter(status, max_polls);
  waiter.wait(&bar, 0);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, 32);
}

// One thread looks `looks` times in vain for each of `waits` things and then waits on an mbarrier that is complete: the
// status word tells whether any of it ran out.
__global__ void __launch_bounds__(32, 1) debug_looks_kernel(int* status, uint32_t limit, uint32_t looks, uint32_t waits) {
  __shared__ alignas(8) uint64_t bar;
  if (threadIdx.x != 0) return;
  mbar_init(&bar, 1);
  fence_mbar_init();
  mbar_arrive(&bar);
  BoundedWaiter waiter(status, limit);
  for (uint32_t i = 0; i < waits; ++i) {
    waiter.look_anew();
    for (uint32_t j = 0; j < looks && waiter.look_again(); ++j) {}
  }
  waiter.wait(&bar, 0);
}

}  // namespace

int launch_debug_looks(int* status, uint32_t limit, uint32_t looks, uint32_t waits, cudaStream_t stream) {
  debug_looks_kernel<<<1, 32, 0, stream>>>(status, limit, looks, waits);
  return check_launch();
}

int launch_debug_wait_expires(int* status, uint32_t max_polls, cudaStream_t stream) {
  debug_wait_expires_kernel<<<1, 128, 0, stream>>>(status, max_polls);
  return check_launch();
}

// ---- launcher ---------------------------------------------------------------------------------
int64_t chunk_workspace_bytes(int64_t batch, int64_t full_tokens, int64_t heads, int training) {
  const WsLayout ws{batch * (full_tokens / kChunk) * heads, training != 0};
  return ws.total();
}

// kind: 0 = forward of an inference call, 1 = backward, 2 = forward of a training call
int64_t chunk_scratch_bytes(int64_t batch, int64_t full_tokens, int64_t heads, int kind) {
  const ScratchLayout sc{batch * (full_tokens / kChunk) * heads};
  return kind == 1 ? sc.total_backward() : sc.total_forward(kind == 2);
}

int64_t chunk_status_offset(int64_t batch, int64_t full_tokens, int64_t heads) {
  const WsLayout ws{batch * (full_tokens / kChunk) * heads};
  return ws.off_status();
}

namespace {

struct ForwardCall {
  const void *q, *k, *v, *g, *beta, *w;
  const float* s_in;
  void* out;
  float *s_out, *bnd;
  uint8_t *workspace, *scratch;
  int64_t rows, H;  // token rows of the sequence tensors, heads
  int training, dtype, g_dtype;
  float scale;
  int prologue;
};

thread_local int t_forward_kernels = 0;  // of this thread's latest chunk forward

// One launch for both where it gains.  Apart they take n_ch * 6.7 us / SMs (the preparation), 1.6-2 us per chunk (the
// scans) and what two launches cost; together the scans' time and some 20 us, where the SMs that do not scan, or all in
// turn (quota), have the units ready in time.
// At most a sixth of the SMs scanning, two launches / one, us, inference, raw, forward of a training step:
//   400 units on    H16 T1792 84/73 94/87 98/91   H16 T2048 90/79 100/95 105/97   H16 T8192 295/226 324/261 338/296
//                   H8 T3200 109/101 117/120 131/132   H8 T4096 131/120 141/144 162/161   H8 T8192 248/210 262/249 301/290
//                   H12 T3200 123/103 133/124 145/134   H24 T1280 76/69 86/79 84/77   H24 T2048 111/91 123/110 121/105
//   below           H16 T1024 55/54 61/65 61/65   H16 T1280 70/60 76/73 78/73   H8 T2048 76/75 82/91 90/95   H8 T2560
//                   94/87 102/103 113/112   H24 T832 61/54 68/65 66/60
//   fewer scans     H1 T12288 279/292 287/349 354/413   H3 T12288 295/292 307/351 393/413   H4 T8192 211/206 225/247 272/286
//                   H6 T8192 231/208 246/249 293/288
//   the units are ready in time either way and a pair of CTAs scans no faster than it does alone, so 4 scans at least,
//   and 8 with a prologue or states to write
// With up to a quarter scanning (above that the preparation falls behind):
//   above the line  H25 T2560 133/108 145/134 146/122   H28 T2048 121/103 133/128 131/108   H32 T1792 115/105 127/118
//                   125/108   H32 T8192 397/368 455/431 447/425   H37 T2048 130/126 145/151 143/132   H37 T8192 430/423
//                   496/497 485/486
//   below           H25 T1536 90/83 100/91 102/87   H28 T1024 70/62 78/73 78/69   H28 T1792 106/91 119/112 115/97
//                   H32 T1280 88/85 98/103 96/87   H37 T1024 74/73 84/89 82/77   H37 T1280 94/87 102/103 102/95
// The lines were drawn for a form of the launch that cost more.  Above them it is the better one or within 3 %, but for raw
// calls of 35 to 37 scans and some 1100 units (145/151, 143/153).  Below them it would gain in most calls of more units
// than the preparing kernel takes at once, two an SM: they stand on the safe side.
bool prefer_joint(int64_t n_scan, int64_t n_ch, int64_t n_chunks, bool training, bool prologue, int sm_count) {
  if (4 * n_scan > sm_count || profiling()) return false;
  if (6 * n_scan <= sm_count) return n_ch >= 400 && n_scan >= (training || prologue ? 8 : 4);
  return 83 * n_ch > (350 + 4 * n_chunks) * sm_count;
}

template <typename T, typename G, typename Seqs, bool kPro>
int launch_joint(const PrepParams& pp, const ScanParams& sp, const Seqs& seqs, const PrepMaps& tm_prep,
                 const ScanMaps& tm_scan, int sm_count, cudaStream_t stream) {
  constexpr int smem = int(sizeof(JointSmem) > sizeof(ScanSmem) ? sizeof(JointSmem) : sizeof(ScanSmem));
  static_assert(smem <= 232448, "joint kernel exceeds the 227 KiB shared-memory limit");
  // the marks of finished units are in D, right before the status block: one fill clears both
  const WsLayout ws{pp.n_ch, pp.training != 0};
  cudaError_t err = cudaMemsetAsync(pp.ws + ws.off_d(), 0, size_t(pp.n_ch) * kBlobD + kStatusBytes, stream);
  if (err != cudaSuccess) { record_cuda_error(err); return GDN2_ERR_LAUNCH; }
  const int pairs = seqs.count() * sp.H;
  // Clusters of two CTAs.  No more preparers than pairs of units, nor than keep ahead of the scans: a unit takes an
  // SM 8.7 us (raw 11) and a chunk of a scan 1.6 us (1.8), and more of them get in the scans' way: three clusters a pair
  // up to eight pairs, then less, as the scans slow down themselves; raw, two more than three a pair.  us at T32768, with
  // one cluster less than the rule gives / the rule / one more, and from H16 on the same on a second and a third GPU, on
  // which the step up lies elsewhere by a cluster:
  //   H4 761/734/736   H6 744/738/745   H8 740/742/761   H10 759/745/763   H11 757/746/777   H12 773/755/785
  //   H14 785/769/814  H15 802/785/814  H16 816/800/816, 818/802/787, 818/849/861  H17 828/812/843, 833/814/837, 830/843/871
  //   H18 841/824/865, 845/827/861, 843/855/886   H19 853/837/869, 855/839/873, 855/886/902   H20 861/869/910, 865/849/894
  //   raw  H8 900/886/886   H10 904/890/892   H12 914/898/900   H14 912/904/900   H16 919/918/908   H18 941/935/933
  // (T8192 lies flatter and at the same places: H8 206/206/206, H12 214/212/212, H16 226/224/226, raw H16 259/257/257;
  // training within 1 %.)
  const int64_t paced = pp.prologue != 0 ? 3 * pairs + 2 : std::min({3 * pairs, (49 * pairs + 102) / 20, 2 * pairs + 11});
  const int64_t want = pairs + std::min((pp.n_ch + 3) / 4, paced);
  const int clusters = int(std::min(want, int64_t(sm_count / 2)));
  // Where the preparers alone would not keep up, the scanning CTAs first prepare `quota` units for each group of
  // theirs, so that everybody is done at the same time.  While a scan advances by a chunk a preparing SM makes
  // `pace` / 100 units: 1.7 us to 8.5, 1.9 to 12 with the prologue, 1.8 to 9 where the states are written out.  us, with
  // 18 / 20 / 21: T32768 H20 942/925/927, H24 1157/1142/1138, H32 1530/1535/1536, T8192 H32 391/386/400, H37
  // 445/448/462, training T4096 H32 (18 / 20 / 22) 233/220/221; raw, with 15 / 16 / 18: T8192 H32 441/447/467, H37
  // 510/515/533, T32768 H24 1341/1316/1320, B2 T4133 H16 238/236/238.
  const int64_t pace = pp.prologue != 0 && pp.training == 0 ? 16 : 20;
  const int64_t in_time = int64_t(2 * (clusters - pairs)) * seqs.n_chunks * pace / 100;
  const int quota = pp.n_ch > in_time ? int((pp.n_ch - in_time + 2 * clusters) / (4 * clusters)) : 0;
  // Where the preparers keep ahead by themselves, or nearly so, a unit is marked at once; elsewhere the microsecond that a
  // release waits for the unit's stores is taken from the next unit, and the mark waits until that one has its inputs.
  // us, at once / later: raw H8 T3200 115/119, T5000 163/167, H16 T2048 90/94, plain H16 T2048 75/78, H15 T32768 783/806.  By
  // the units that are in time: all but 1 % raw H18 T1472 74.3/77.7; 94 % plain H22 T1344 64.7/65.9; 93 % raw H19 T1600
  // 79.6/82.3; 86 % raw H20 T1600 82.9/83.2; 83 % plain H24 T1088 61.5/60.3; 81 % raw H21 T1600 85.1/84.4; 71 % raw H23
  // T1344 82.8/80.2; with a quota raw H24 T8192 332/327, H32 T4096 235/232, plain H24 T8192 278/271.  (Two kernels: with
  // both forms in one the raw calls that have a quota take 331 and 235.)
  const bool soon = quota == 0 && 100 * in_time >= 85 * pp.n_ch;
  auto kernel = soon ? chunk_joint_kernel<T, G, Seqs, kPro, true> : chunk_joint_kernel<T, G, Seqs, kPro, false>;
  err = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
  if (err != cudaSuccess) { record_cuda_error(err); return GDN2_ERR_LAUNCH; }
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(unsigned(2 * clusters));
  config.blockDim = dim3(kJointThreads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute together;
  together.id = cudaLaunchAttributeCooperative;
  together.val.cooperative = 1;
  config.attrs = &together;
  config.numAttrs = 1;
  err = cudaLaunchKernelEx(&config, kernel, pp, sp, seqs, tm_prep, tm_scan, quota);
  if (err == cudaErrorCooperativeLaunchTooLarge) {  // a context with fewer SMs than the device
    (void)cudaGetLastError();
    return GDN2_ERR_UNSUPPORTED;
  }
  if (err != cudaSuccess) { (void)cudaGetLastError(); record_cuda_error(err); return GDN2_ERR_LAUNCH; }
  return GDN2_OK;
}

template <typename T, typename Seqs>
int launch_scan(const ScanParams& p, const Seqs& seqs, const ScanMaps& tm, int64_t n_scan, int parts,
                cudaStream_t stream) {
  auto kernel = parts == 2 ? chunk_scan_kernel<T, Seqs, 2> : chunk_scan_kernel<T, Seqs, 1>;
  const int smem = int(sizeof(ScanSmem));
  const cudaError_t err = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
  if (err != cudaSuccess) { record_cuda_error(err); return GDN2_ERR_LAUNCH; }
  const int threads = parts == 2 ? ScanWarps<2>::kThreads : ScanWarps<1>::kThreads;
  kernel<<<unsigned(n_scan * parts), threads, smem, stream>>>(p, seqs, tm);
  return check_launch();
}

template <typename Seqs>
int launch_forward(const Seqs& seqs, const ForwardCall& a, cudaStream_t stream) {
  const int64_t n_ch = int64_t(seqs.total_chunks()) * a.H;
  // units, token rows and the grids of the scans are 31-bit numbers
  if (n_ch <= 0 || n_ch > int64_t(0x7fffffff) || a.rows > int64_t(0x7fffffff)) return GDN2_ERR_TOO_LARGE;
  int sm_count = 0;
  if (int st = multiprocessors(&sm_count); st != GDN2_OK) return st;
  const int64_t n_scan = int64_t(seqs.count()) * a.H;
  bool joint = false;
  if constexpr (std::is_same<Seqs, UniformSeqs>::value) {
    joint = prefer_joint(n_scan, n_ch, seqs.n_chunks, a.training != 0, a.prologue != 0, sm_count);
  }
  const int parts = joint ? kJointParts : value_parts(n_ch, n_scan, seqs.at(0).n_chunks, sm_count, 2);
  const WsLayout ws{n_ch, a.training != 0};
  int* status = reinterpret_cast<int*>(a.workspace + ws.off_status());
  const ForwardTiles tiles = forward_tiles(a.workspace, a.scratch, n_ch, a.training != 0);
  PrepMaps tm_prep;
  ScanMaps tm;
  // the sequence tensors, and the scan's operands: the prep kernel's tiles in the swizzle of their role
  if (!encode_sequence_map(&tm_prep.g, a.g, a.rows, a.H, a.g_dtype) ||
      !encode_half_map(&tm_prep.k, a.k, a.rows, a.H, a.dtype) ||
      !encode_half_map(&tm_prep.q, a.q, a.rows, a.H, a.dtype) ||
      !encode_half_map(&tm_prep.beta, a.beta, a.rows, a.H, a.dtype) ||
      !encode_tile_map(&tm_prep.out_tt, tiles.tt, n_ch, kChunk, kChunk, true, 32, 1) ||
      !encode_tile_map(&tm_prep.out_yt, tiles.yt, n_ch, kDim, kChunk, false) ||
      !encode_sequence_map(&tm.v, a.v, a.rows, a.H, a.dtype, kChunk, kDim / parts) ||
      !encode_sequence_map(&tm.w, a.w, a.rows, a.H, a.dtype, kChunk, kDim / parts) ||
      !encode_sequence_map(&tm.out, a.out, a.rows, a.H, a.dtype, kChunk, kDim / parts) ||
      !encode_tile_map(&tm.yt, tiles.yt, n_ch, kDim, kChunk, true) ||
      !encode_tile_map(&tm.q, tiles.q, n_ch, kChunk, kDim, false) ||
      !encode_tile_map(&tm.kn, tiles.kn, n_ch, kChunk, kDim, true) ||
      !encode_tile_map(&tm.at, tiles.at, n_ch, kChunk, kChunk, true, 32, 1) ||
      !encode_tile_map(&tm.tt, tiles.tt, n_ch, kChunk, kChunk, true, 32, 1)) {
    return GDN2_ERR_LAUNCH;
  }
  const PrepParams pp{a.workspace, tiles, n_ch, int(a.H), a.scale, a.training, a.prologue};
  const ScanParams sp{a.workspace + ws.off_d(), a.s_in, a.out, a.s_out, a.bnd,
                      a.training ? reinterpret_cast<float*>(a.workspace + ws.off_rn()) : nullptr,
                      status, int(a.H), (a.prologue & kPrologueGate) != 0};
  cudaError_t err;
  if constexpr (std::is_same<Seqs, UniformSeqs>::value) {
    if (joint) {
      int st = GDN2_OK;
      GDN2_DISPATCH_TYPES(a.dtype, a.g_dtype, {
        st = a.prologue != 0 ? launch_joint<T, G, Seqs, true>(pp, sp, seqs, tm_prep, tm, sm_count, stream)
                             : launch_joint<T, G, Seqs, false>(pp, sp, seqs, tm_prep, tm, sm_count, stream);
      });
      if (st != GDN2_ERR_UNSUPPORTED) {
        t_forward_kernels = 1;
        return st;
      }
    }
  }
  err = cudaMemsetAsync(status, 0, kStatusBytes, stream);
  if (err != cudaSuccess) { record_cuda_error(err); return GDN2_ERR_LAUNCH; }

  profile_mark(0, stream);
  const unsigned prep_grid = unsigned(n_ch < 2 * int64_t(sm_count) ? n_ch : 2 * int64_t(sm_count));
  GDN2_DISPATCH_TYPES(a.dtype, a.g_dtype, {
    auto kernel = a.prologue != 0 ? chunk_prep_kernel<T, G, Seqs, true> : chunk_prep_kernel<T, G, Seqs, false>;
    const int smem = int(sizeof(PrepSmem));
    err = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    if (err != cudaSuccess) { record_cuda_error(err); return GDN2_ERR_LAUNCH; }
    kernel<<<prep_grid, kPrepThreads, smem, stream>>>(pp, seqs, tm_prep);
  });
  int st = check_launch();
  if (st != GDN2_OK) return st;
  profile_mark(1, stream);

  st = a.dtype == GDN2_BF16 ? launch_scan<__nv_bfloat16>(sp, seqs, tm, n_scan, parts, stream)
                            : launch_scan<__half>(sp, seqs, tm, n_scan, parts, stream);
  profile_mark(2, stream);
  t_forward_kernels = 2;
  return st;
}

}  // namespace

int chunk_forward_kernels() { return t_forward_kernels; }
int chunk_value_parts(int64_t units, int64_t scans, int64_t longest, int sm_count, int most) {
  return value_parts(units, scans, longest, sm_count, most);
}
int64_t tensor_maps_encoded() { return g_tensor_maps_encoded.load(std::memory_order_relaxed); }

int launch_chunk_forward(const void* q, const void* k, const void* v, const void* g, const void* beta,
                         const void* w, const float* s_in, void* out, float* s_out, float* bnd,
                         uint8_t* workspace, uint8_t* scratch, int64_t B, int64_t T, int64_t H,
                         int64_t full_tokens, int training, int dtype, int g_dtype, float scale,
                         int prologue, cudaStream_t stream) {
  const int64_t n_chunks = full_tokens / kChunk;
  if (B * T > int64_t(0x7fffffff) || B * n_chunks * H > int64_t(0x7fffffff)) return GDN2_ERR_TOO_LARGE;
  const UniformSeqs seqs{0, T, int(full_tokens < T ? full_tokens : T), int(n_chunks), int(B)};
  const ForwardCall a{q, k, v, g, beta, w, s_in, out, s_out, bnd, workspace, scratch, B * T, H,
                      training, dtype, g_dtype, scale, prologue};
  return launch_forward(seqs, a, stream);
}

// `table` lists the sequences of at least one chunk, longest first; `rows` is the packed length.
int launch_packed_chunk_forward(const PackedSeqs& table, const void* q, const void* k, const void* v, const void* g,
                                const void* beta, const void* w, const float* s_in, void* out, float* s_out,
                                float* bnd, uint8_t* workspace, uint8_t* scratch, int64_t rows, int64_t H,
                                int training, int dtype, int g_dtype, float scale, int prologue,
                                cudaStream_t stream) {
  const ForwardCall a{q, k, v, g, beta, w, s_in, out, s_out, bnd, workspace, scratch, rows, H,
                      training, dtype, g_dtype, scale, prologue};
  return launch_forward(table, a, stream);
}

}  // namespace gdn2
