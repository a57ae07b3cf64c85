// Token-path kernels for one token or a few: exact fp32 recurrence.
//
//   token_step_kernel         one decode step of few heads (or of states that are not 16-byte aligned), and
//                             sequences of up to 9 tokens
//   token_decode_ring_kernel  one decode step of many heads, persistent
//   token_t1_zero_kernel      T == 1, zero initial state closed form (write-only state)
//
// Longer sequences run in spans of 16 tokens (token_span.cu).  These follow the recurrence of
// src/gdn2_sm120/reference.py:80-93 of the reference literally; the thread mapping is this library's own
// (the reference's token kernel is src/gdn2_sm120/recurrent.py:108-243).
//
// State tile ownership in the step kernel: one CTA = (batch, head, 32 value columns), 128 threads.
// Thread `tid` owns the float4 column group cg = tid & 7 of the key rows rg + 16*i, rg = tid >> 3,
// i = 0..7, so one warp touches four 128-byte row segments per i: fully coalesced 128-bit state I/O, 32
// fp32 state registers per thread, and every state element is read and written by exactly one thread
// (which is why an exact in-place state update is race-free).

#include <type_traits>

#include "common.cuh"
#include "seqs.cuh"
#include "tc05.cuh"

namespace gdn2 {

int launch_span_forward(const void*, const void*, const void*, const void*, const void*, const void*, const float*,
                        void*, float*, float*, int64_t, int64_t, int64_t, int64_t, int64_t, int, int, float, int,
                        cudaStream_t);

namespace {

// Fewest (batch, head) pairs for which a decode step runs on the persistent ring kernel (below it
// the ring has too few heads per SM to overlap anything; measured equal to the plain kernel at 160-192)
#ifndef GDN2_DECODE_RING_MIN_HEADS
#define GDN2_DECODE_RING_MIN_HEADS 256
#endif

constexpr int kTokThreads = 128;
constexpr int kTokVT = 32;                     // value columns per CTA
constexpr int kTokTiles = kDim / kTokVT;       // 4 CTAs per (batch, head)
constexpr int kRowsPerThread = 8;              // 128 rows / 16 row groups
constexpr int64_t kStateElems = int64_t(kDim) * kDim;

struct TokenStepParams {
  const void *q, *k, *v, *g, *beta, *w;
  const float* s_in;
  void* out;
  float* s_out;
  float* bnd;    // states before and after the tokens, or null
  int H;
  int first;     // sequences of the list before this one are not this launch's
  float scale;
  int prologue;  // kPrologueNorm | kPrologueGate: raw projections / gate pre-activations are activated here
};

__device__ __forceinline__ float4 ld_red4(const float (*red)[kTokVT], int col) {
  // sum of the four per-warp partial rows
  float4 s = *reinterpret_cast<const float4*>(&red[0][col]);
#pragma unroll
  for (int wv = 1; wv < 4; ++wv) {
    const float4 t = *reinterpret_cast<const float4*>(&red[wv][col]);
    s.x += t.x; s.y += t.y; s.z += t.z; s.w += t.w;
  }
  return s;
}

// kPro (here and in the two decode kernels below): the instantiation that can apply the layer prologue
// to raw inputs; the plain instantiation carries none of that code.
//
// Up to kTok tokens one after the other, their inputs read at the start; a token costs two barriers and two
// reductions over the CTA.  kTok = 1 is a decode step (T == 1).
template <typename T, typename G, typename Seqs, bool kPro, int kTok>
__global__ void __launch_bounds__(kTokThreads)
token_step_kernel(const TokenStepParams p, const __grid_constant__ Seqs seqs) {
  __shared__ float s_a[kTok][kDim], s_e[kTok][kDim], s_k[kTok][kDim], s_q[kTok][kDim];
  __shared__ float s_z[kTok][kTokVT];
  __shared__ __align__(16) float s_red[2][4][kTokVT];  // [erase|output][warp][column]
  __shared__ float s_nrm[kTok][4][2];                  // fused prologue: per warp sums of q^2, k^2

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cg = tid & 7, rg = tid >> 3;
  const int vt = int(blockIdx.x % kTokTiles);
  const int sh = int(blockIdx.x) / kTokTiles;
  const int s_ = kTok == 1 ? 0 : sh / p.H, h = sh - s_ * p.H;
  const SeqInfo sq = seqs.at(kTok == 1 ? 0 : p.first + s_);
  const int n = kTok == 1 ? 1 : sq.len;  // (0: an empty sequence of a packed batch, its state passes through)
  const int64_t bh = kTok == 1 ? sh : int64_t(sq.sid) * p.H + h;
  // (T == 1: the sequence row is the head's number)
  auto row_of = [&](int t) { return kTok == 1 ? bh * kDim : ((sq.row0 + t) * p.H + h) * kDim; };
  const int col0 = vt * kTokVT + cg * 4;
  const bool pro_norm = kPro && (p.prologue & kPrologueNorm) != 0;
  const bool pro_gate = kPro && (p.prologue & kPrologueGate) != 0;

  float S[kRowsPerThread][4];
  if (p.s_in != nullptr) {
    const float* src = p.s_in + bh * kStateElems;
    const bool vec = (reinterpret_cast<uintptr_t>(p.s_in) & 15) == 0;
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) load4(src + (rg + 16 * i) * kDim + col0, vec, S[i]);
  } else {
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) S[i][0] = S[i][1] = S[i][2] = S[i][3] = 0.f;
  }
  auto store_state = [&](float* dst) {
    const bool vec = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) store4(dst + (rg + 16 * i) * kDim + col0, vec, S[i]);
  };
  constexpr int kBatch = kTok < 4 ? kTok : 4;  // tokens read together (eight take the registers of other CTAs)
  auto stage = [&](int t0) {
    T rk[kBatch], rq[kBatch], rb[kBatch], rw[kBatch], rv[kBatch];
    G rg_[kBatch];
#pragma unroll
    for (int t = 0; t < kBatch; ++t) {  // (a token that does not exist: the last one is read in its place)
      const int64_t idx = row_of(min(t0 + t, n - 1));
      rk[t] = static_cast<const T*>(p.k)[idx + tid];
      rq[t] = static_cast<const T*>(p.q)[idx + tid];
      rg_[t] = static_cast<const G*>(p.g)[idx + tid];
      rb[t] = static_cast<const T*>(p.beta)[idx + tid];
      if (tid < kTokVT) {
        rw[t] = static_cast<const T*>(p.w)[idx + vt * kTokVT + tid];
        rv[t] = static_cast<const T*>(p.v)[idx + vt * kTokVT + tid];
      }
    }
#pragma unroll
    for (int x = 0; x < kBatch; ++x) {
      const int t = t0 + x;
      if (t >= n) break;
      const float kv = to_float(rk[x]), qv = to_float(rq[x]);
      float gv = to_float(rg_[x]), bv = to_float(rb[x]);
      if (pro_gate) { gv = prologue_log_decay(gv); bv = prologue_sigmoid(bv); }
      s_a[t][tid] = expf(gv);
      s_e[t][tid] = bv * kv;
      s_k[t][tid] = kv;
      s_q[t][tid] = p.scale * qv;
      if (tid < kTokVT) {
        float wv = to_float(rw[x]);
        if (pro_gate) wv = prologue_sigmoid(wv);
        s_z[t][tid] = wv * to_float(rv[x]);
      }
      if (pro_norm) {
        float sq_ = qv * qv, sk = kv * kv;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          sq_ += __shfl_xor_sync(0xffffffffu, sq_, off);
          sk += __shfl_xor_sync(0xffffffffu, sk, off);
        }
        if (lane == 0) { s_nrm[t][warp][0] = sq_; s_nrm[t][warp][1] = sk; }
      }
    }
  };
  if constexpr (kTok == kBatch) {
    if (n > 0) stage(0);
  } else {
#pragma unroll 1
    for (int t0 = 0; t0 < n; t0 += kBatch) stage(t0);
  }
  if (p.bnd != nullptr) store_state(p.bnd + (int64_t(sq.slot0) * p.H + h) * kStateElems);
  if (n == 0 && p.s_out != nullptr) store_state(p.s_out + bh * kStateElems);
  __syncthreads();

#pragma unroll 1
  for (int t = 0; t < n; ++t) {
    // reciprocal norms of the raw q and k (1 when the inputs are already normalised)
    float iq = 1.f, ik = 1.f;
    if (pro_norm) {
      iq = rsqrtf(s_nrm[t][0][0] + s_nrm[t][1][0] + s_nrm[t][2][0] + s_nrm[t][3][0] + kPrologueEps);
      ik = rsqrtf(s_nrm[t][0][1] + s_nrm[t][1][1] + s_nrm[t][2][1] + s_nrm[t][3][1] + kPrologueEps);
    }
    // X = a * S ; partial r = X^T e over this thread's rows
    float r[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) {
      const float a = s_a[t][rg + 16 * i], e = kPro ? s_e[t][rg + 16 * i] * ik : s_e[t][rg + 16 * i];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        S[i][c] *= a;
        r[c] = fmaf(S[i][c], e, r[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      r[c] += __shfl_xor_sync(0xffffffffu, r[c], 8);
      r[c] += __shfl_xor_sync(0xffffffffu, r[c], 16);
    }
    if (lane < 8) *reinterpret_cast<float4*>(&s_red[0][warp][cg * 4]) = make_float4(r[0], r[1], r[2], r[3]);
    __syncthreads();

    const float4 rs = ld_red4(s_red[0], cg * 4);
    const float u[4] = {s_z[t][cg * 4 + 0] - rs.x, s_z[t][cg * 4 + 1] - rs.y,
                        s_z[t][cg * 4 + 2] - rs.z, s_z[t][cg * 4 + 3] - rs.w};
    // S = X + k u^T ; partial o = S^T (scale q)
    float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) {
      const float kv = kPro ? s_k[t][rg + 16 * i] * ik : s_k[t][rg + 16 * i];
      const float qv = kPro ? s_q[t][rg + 16 * i] * iq : s_q[t][rg + 16 * i];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        S[i][c] = fmaf(kv, u[c], S[i][c]);
        o[c] = fmaf(S[i][c], qv, o[c]);
      }
    }
    if (t + 1 == n) {
      if (p.s_out != nullptr) store_state(p.s_out + bh * kStateElems);
      if (p.bnd != nullptr) store_state(p.bnd + (int64_t(sq.slot0 + 1) * p.H + h) * kStateElems);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      o[c] += __shfl_xor_sync(0xffffffffu, o[c], 8);
      o[c] += __shfl_xor_sync(0xffffffffu, o[c], 16);
    }
    if (lane < 8) *reinterpret_cast<float4*>(&s_red[1][warp][cg * 4]) = make_float4(o[0], o[1], o[2], o[3]);
    __syncthreads();
    if (tid < kTokVT) {
      const float ov = s_red[1][0][tid] + s_red[1][1][tid] + s_red[1][2][tid] + s_red[1][3][tid];
      stf<T>(p.out, row_of(t) + vt * kTokVT + tid, ov);
    }
  }
  if constexpr (std::is_same<Seqs, PackedSpans>::value) outlast_others();
}

// ---------------------------------------------------------------------------------
// Decode step (T == 1, 16-byte aligned states, many heads): persistent CTAs, one per SM, each
// walking over (batch, head) pairs.  A head's whole 64 KiB state travels global -> shared ->
// global as 1-D bulk asynchronous copies through a three-slot ring, so two loads and one store
// are in flight per SM while the current head is updated in place in shared memory.
// Thread = (value column v, key half): the sums over keys stay inside a thread except for one
// two-way combine, and shared-memory accesses to the state are conflict-free.
constexpr int kDecThreads = 256;
constexpr int kDecStages = 3;

struct DecodeSmem {
  alignas(128) float state[kDecStages][kDim * kDim];
  alignas(16) float ae[2][kDim], a[2][kDim], kk[2][kDim], qs[2][kDim], z[2][kDim];
  float red[2][2][kDim];   // [parity][key half][column]  erase partial sums
  float redo[2][2][kDim];  //                             output partial sums
  float nrm[2][4][2];      // fused prologue: [parity][warp of the key half][q | k] sums of squares
  alignas(8) uint64_t full[kDecStages];
};

struct DecodeParams {
  const void *q, *k, *v, *g, *beta, *w;
  const float* s_in;
  void* out;
  float* s_out;
  int64_t n_heads;  // batch * heads; T == 1 so sequence row index == head index
  float scale;
  int prologue;     // kPrologueNorm | kPrologueGate
};

template <typename T, typename G, bool kPro = false>
__global__ void __launch_bounds__(kDecThreads, 1) token_decode_ring_kernel(const DecodeParams p) {
  extern __shared__ __align__(128) unsigned char dec_smem_raw[];
  DecodeSmem& sm = *reinterpret_cast<DecodeSmem*>(dec_smem_raw);
  const int tid = threadIdx.x;
  const int col = tid & (kDim - 1), kh = tid >> 7;
  const int64_t first = blockIdx.x, stride = gridDim.x;
  const int64_t n_mine = (p.n_heads > first) ? (p.n_heads - first + stride - 1) / stride : 0;
  constexpr uint32_t kStateBytes = kDim * kDim * sizeof(float);

  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < kDecStages; ++s) tc::mbar_init(&sm.full[s], 1);
    tc::fence_mbar_init();
  }
  __syncthreads();

  auto issue_load = [&](int64_t n) {  // thread 0 only
    const int s = int(n % kDecStages);
    tc::mbar_arrive_expect_tx(&sm.full[s], kStateBytes);
    tc::bulk_g2s(sm.state[s], p.s_in + (first + n * stride) * int64_t(kDim) * kDim, kStateBytes, &sm.full[s]);
  };
  // per-head vectors: threads 0..127 own a key channel, threads 128..255 a value channel
  float va = 0.f, vb = 0.f, vc = 0.f, vd = 0.f;
  auto fetch_vectors = [&](int64_t n) {
    const int64_t idx = (first + n * stride) * kDim + col;
    if (kh == 0) {
      va = ldf<G>(p.g, idx); vb = ldf<T>(p.beta, idx); vc = ldf<T>(p.k, idx); vd = ldf<T>(p.q, idx);
    } else {
      va = ldf<T>(p.w, idx); vb = ldf<T>(p.v, idx);
    }
  };
  const bool pro_norm = kPro && (p.prologue & kPrologueNorm) != 0;
  const bool pro_gate = kPro && (p.prologue & kPrologueGate) != 0;
  auto stage_vectors = [&](int buf) {
    if (kh == 0) {
      if (pro_gate) { va = prologue_log_decay(va); vb = prologue_sigmoid(vb); }
      const float av = expf(va);
      sm.a[buf][col] = av;
      sm.ae[buf][col] = av * (vb * vc);
      sm.kk[buf][col] = vc;
      sm.qs[buf][col] = p.scale * vd;
      if (pro_norm) {  // warps 0..3 hold the 128 key channels
        float sq = vd * vd, sk = vc * vc;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          sq += __shfl_xor_sync(0xffffffffu, sq, off);
          sk += __shfl_xor_sync(0xffffffffu, sk, off);
        }
        if ((tid & 31) == 0) { sm.nrm[buf][tid >> 5][0] = sq; sm.nrm[buf][tid >> 5][1] = sk; }
      }
    } else {
      if (pro_gate) va = prologue_sigmoid(va);
      sm.z[buf][col] = va * vb;
    }
  };

  if (n_mine > 0) {
    if (tid == 0) {
      issue_load(0);
      if (n_mine > 1) issue_load(1);
    }
    fetch_vectors(0);
    stage_vectors(0);
  }
  __syncthreads();

  bool dead = false;
  for (int64_t n = 0; n < n_mine; ++n) {
    const int s = int(n % kDecStages), buf = int(n & 1);
    const int64_t bh = first + n * stride;
    if (n + 1 < n_mine) fetch_vectors(n + 1);
    if (!dead && !tc::mbar_wait(&sm.full[s], uint32_t((n / kDecStages) & 1), 1u << 20)) dead = true;

    float* S = sm.state[s] + col;
    const int k0 = 64 * kh;
    // pass 1: r[v] = sum_k S[k][v] * (a[k] e[k])
    float r0 = 0.f, r1 = 0.f, r2 = 0.f, r3 = 0.f;  // four chains: the sum is latency-bound otherwise
#pragma unroll 4
    for (int kq = 0; kq < 64; kq += 4) {
      const float4 f = *reinterpret_cast<const float4*>(&sm.ae[buf][k0 + kq]);
      r0 = fmaf(S[(k0 + kq) * kDim], f.x, r0);
      r1 = fmaf(S[(k0 + kq + 1) * kDim], f.y, r1);
      r2 = fmaf(S[(k0 + kq + 2) * kDim], f.z, r2);
      r3 = fmaf(S[(k0 + kq + 3) * kDim], f.w, r3);
    }
    sm.red[buf][kh][col] = (r0 + r1) + (r2 + r3);
    if (tid == 0 && n + 2 < n_mine) {
      // The slot of head n + 2 was last used by head n - 1, whose store was issued at the end of the
      // previous iteration: by now it has normally finished reading the slot, so this wait does not
      // hold up the warp (at the top of the iteration it stalled every head by the store's read time).
      tc::bulk_wait_read_all();
      issue_load(n + 2);
    }
    // a copy that never arrived, for any thread: the head's results are marked invalid for all
    dead = __syncthreads_or(dead ? 1 : 0) != 0;
    // raw q / k: the erase sum is linear in k, the output in q, so the reciprocal norms scale the sums
    float iq = 1.f, ik = 1.f;
    if (pro_norm) {
      iq = rsqrtf(sm.nrm[buf][0][0] + sm.nrm[buf][1][0] + sm.nrm[buf][2][0] + sm.nrm[buf][3][0] + kPrologueEps);
      ik = rsqrtf(sm.nrm[buf][0][1] + sm.nrm[buf][1][1] + sm.nrm[buf][2][1] + sm.nrm[buf][3][1] + kPrologueEps);
    }
    const float r_sum = sm.red[buf][0][col] + sm.red[buf][1][col];
    const float u = kPro ? (sm.z[buf][col] - ik * r_sum) * ik  // u * ik: S += (k ik) u
                         : sm.z[buf][col] - r_sum;
    // pass 2: S <- a S + k u^T ; o[v] = sum_k S[k][v] (scale q[k])
    float o = 0.f;
#pragma unroll 4
    for (int kq = 0; kq < 64; kq += 4) {
      const float4 fa = *reinterpret_cast<const float4*>(&sm.a[buf][k0 + kq]);
      const float4 fk = *reinterpret_cast<const float4*>(&sm.kk[buf][k0 + kq]);
      const float4 fq = *reinterpret_cast<const float4*>(&sm.qs[buf][k0 + kq]);
      float x0 = fmaf(fk.x, u, fa.x * S[(k0 + kq) * kDim]);
      float x1 = fmaf(fk.y, u, fa.y * S[(k0 + kq + 1) * kDim]);
      float x2 = fmaf(fk.z, u, fa.z * S[(k0 + kq + 2) * kDim]);
      float x3 = fmaf(fk.w, u, fa.w * S[(k0 + kq + 3) * kDim]);
      S[(k0 + kq) * kDim] = x0; S[(k0 + kq + 1) * kDim] = x1;
      S[(k0 + kq + 2) * kDim] = x2; S[(k0 + kq + 3) * kDim] = x3;
      o = fmaf(x0, fq.x, o); o = fmaf(x1, fq.y, o); o = fmaf(x2, fq.z, o); o = fmaf(x3, fq.w, o);
    }
    sm.redo[buf][kh][col] = o;
    if (n + 1 < n_mine) stage_vectors(buf ^ 1);
    tc::fence_async_smem();
    __syncthreads();
    // A head whose state never arrived is not written back: the caller's state (which an in-place
    // update would otherwise overwrite with garbage) survives and the NaN output says so.
    if (tid == 0 && !dead) {
      tc::bulk_s2g(p.s_out + bh * int64_t(kDim) * kDim, sm.state[s], kStateBytes);
      tc::bulk_commit();
    }
    if (kh == 0) {
      float ov = sm.redo[buf][0][col] + sm.redo[buf][1][col];
      if (kPro) ov *= iq;
      if (dead) ov = __int_as_float(0x7fc00000);  // a bulk copy never arrived: make the failure visible
      stf<T>(p.out, bh * kDim + col, ov);
    }
  }
  if (tid == 0) tc::bulk_wait_all();
}

// ---------------------------------------------------------------------------------
struct T1ZeroParams {
  const void *q, *k, *v, *w;
  void* out;
  float* s_out;
  int64_t H;
  float scale;
  int prologue;
};

template <typename T, bool kPro = false>
__global__ void __launch_bounds__(kTokThreads) token_t1_zero_kernel(const T1ZeroParams p) {
  __shared__ float s_k[kDim];
  __shared__ float s_z[kTokVT];
  __shared__ float s_part[4];
  __shared__ float s_nrm[4][2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cg = tid & 7, rg = tid >> 3;
  const int vt = int(blockIdx.x % kTokTiles);
  const int64_t bh = blockIdx.x / kTokTiles;
  const int64_t idx = bh * kDim;  // T == 1: [B, 1, H, 128]

  const bool pro_norm = kPro && (p.prologue & kPrologueNorm) != 0;
  const bool pro_gate = kPro && (p.prologue & kPrologueGate) != 0;
  const float kv = ldf<T>(p.k, idx + tid);
  const float qv = ldf<T>(p.q, idx + tid);
  float qk = p.scale * qv * kv;
  if (tid < kTokVT) {
    float wv = ldf<T>(p.w, idx + vt * kTokVT + tid);
    if (pro_gate) wv = prologue_sigmoid(wv);
    s_z[tid] = wv * ldf<T>(p.v, idx + vt * kTokVT + tid);
  }
  float sq = qv * qv, sk = kv * kv;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    qk += __shfl_xor_sync(0xffffffffu, qk, off);
    if (pro_norm) {
      sq += __shfl_xor_sync(0xffffffffu, sq, off);
      sk += __shfl_xor_sync(0xffffffffu, sk, off);
    }
  }
  if (lane == 0) {
    s_part[warp] = qk;
    s_nrm[warp][0] = sq;
    s_nrm[warp][1] = sk;
  }
  if (!pro_norm) s_k[tid] = kv;
  __syncthreads();
  qk = s_part[0] + s_part[1] + s_part[2] + s_part[3];
  if (pro_norm) {  // raw q, k: scale by the reciprocal norms
    const float ik = rsqrtf(s_nrm[0][1] + s_nrm[1][1] + s_nrm[2][1] + s_nrm[3][1] + kPrologueEps);
    qk *= ik * rsqrtf(s_nrm[0][0] + s_nrm[1][0] + s_nrm[2][0] + s_nrm[3][0] + kPrologueEps);
    s_k[tid] = kv * ik;
    __syncthreads();
  }

  float z[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) z[c] = s_z[cg * 4 + c];
  float* dst = p.s_out + bh * kStateElems + vt * kTokVT + cg * 4;
  const bool vec = (reinterpret_cast<uintptr_t>(p.s_out) & 15) == 0;
#pragma unroll
  for (int i = 0; i < kRowsPerThread; ++i) {
    const float kr = s_k[rg + 16 * i];
    const float row[4] = {kr * z[0], kr * z[1], kr * z[2], kr * z[3]};
    store4(dst + (rg + 16 * i) * kDim, vec, row);
  }
  if (tid < kTokVT) stf<T>(p.out, idx + vt * kTokVT + tid, qk * s_z[tid]);
}

inline bool grid_fits(int64_t blocks) { return blocks > 0 && blocks <= int64_t(0x7fffffff); }

// `most`: 1 (T == 1 without checkpoints), 4 or kStepTokens, the most tokens a sequence has
template <typename Seqs>
int launch_steps(const TokenStepParams& p, const Seqs& seqs, int64_t blocks, int most, int dtype, int g_dtype,
                 cudaStream_t stream, bool beside = false) {
  if (!grid_fits(blocks)) return GDN2_ERR_TOO_LARGE;
  auto run = [&](auto tok) {
    constexpr int kTok = decltype(tok)::value;
    int st = GDN2_OK;
    if (beside) {
      GDN2_DISPATCH_TYPES(dtype, g_dtype, {
        st = launch_beside(p.prologue != 0 ? token_step_kernel<T, G, Seqs, true, kTok>
                                           : token_step_kernel<T, G, Seqs, false, kTok>,
                           unsigned(blocks), kTokThreads, 0, stream, p, seqs);
      });
      return st;
    }
    GDN2_DISPATCH_TYPES(dtype, g_dtype, {
      if (p.prologue != 0) token_step_kernel<T, G, Seqs, true, kTok><<<unsigned(blocks), kTokThreads, 0, stream>>>(p, seqs);
      else token_step_kernel<T, G, Seqs, false, kTok><<<unsigned(blocks), kTokThreads, 0, stream>>>(p, seqs);
    });
    return check_launch();
  };
  if constexpr (std::is_same<Seqs, UniformSeqs>::value) {
    if (most == 1) return run(std::integral_constant<int, 1>{});
  }
  return most == 4 ? run(std::integral_constant<int, 4>{}) : run(std::integral_constant<int, kStepTokens>{});
}

}  // namespace

// ---- launchers (called from api.cu) --------------------------------------------------
int launch_token_forward(const void* q, const void* k, const void* v, const void* g,
                         const void* beta, const void* w, const float* s_in, void* out,
                         float* s_out, float* bnd, int64_t B, int64_t T, int64_t H,
                         int64_t t_begin, int64_t t_end, int dtype, int g_dtype, float scale,
                         int prologue, cudaStream_t stream) {
  const int64_t blocks = B * H * kTokTiles;
  if (!grid_fits(blocks)) return GDN2_ERR_TOO_LARGE;
  // decode fast path: one token, state in and out, 16-byte aligned, enough heads to fill the GPU
  if (T == 1 && t_begin == 0 && t_end == 1 && s_in != nullptr && s_out != nullptr && bnd == nullptr &&
      B * H >= GDN2_DECODE_RING_MIN_HEADS &&
      ((reinterpret_cast<uintptr_t>(s_in) | reinterpret_cast<uintptr_t>(s_out)) & 15) == 0) {
    int dev = 0, sms = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (err != cudaSuccess) { record_cuda_error(err); return GDN2_ERR_LAUNCH; }
    DecodeParams dp{q, k, v, g, beta, w, s_in, out, s_out, B * H, scale, prologue};
    const int smem = int(sizeof(DecodeSmem));
    const unsigned grid = unsigned(B * H < sms ? B * H : sms);
    GDN2_DISPATCH_TYPES(dtype, g_dtype, {
      auto kernel = prologue != 0 ? token_decode_ring_kernel<T, G, true> : token_decode_ring_kernel<T, G, false>;
      err = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
      if (err != cudaSuccess) { record_cuda_error(err); return GDN2_ERR_LAUNCH; }
      kernel<<<grid, kDecThreads, smem, stream>>>(dp);
    });
    return check_launch();
  }
  // A few tokens one by one (step_tokens says how many): the spans of token_span.cu cost nearly as much for one
  // token as for 16 (B32 H32, 2 tokens: 73 us there, 32 here).
  const int64_t tokens = t_end - t_begin;
  if (tokens >= 1 && tokens <= step_tokens(prologue)) {
    const TokenStepParams p{q, k, v, g, beta, w, s_in, out, s_out, bnd, int(H), 0, scale, prologue};
    const int most = T == 1 && bnd == nullptr ? 1 : tokens <= 4 ? 4 : kStepTokens;
    return launch_steps(p, UniformSeqs{t_begin, T, int(tokens), 1, int(B)}, blocks, most, dtype, g_dtype, stream);
  }
  return launch_span_forward(q, k, v, g, beta, w, s_in, out, s_out, bnd, B, T, H, t_begin, t_end, dtype, g_dtype,
                             scale, prologue, stream);
}

// the sequences from `first` on, none of more than step_tokens(prologue) tokens
int launch_packed_steps(const PackedSpans& table, int first, const void* q, const void* k, const void* v, const void* g,
                        const void* beta, const void* w, const float* s_in, void* out, float* s_out, float* bnd,
                        int64_t H, int dtype, int g_dtype, float scale, int prologue, bool beside,
                        cudaStream_t stream) {
  const TokenStepParams p{q, k, v, g, beta, w, s_in, out, s_out, bnd, int(H), first, scale, prologue};
  return launch_steps(p, table, (table.n - first) * H * kTokTiles, table.e[first].len <= 4 ? 4 : kStepTokens, dtype,
                      g_dtype, stream, beside);
}

int launch_token_t1_zero(const void* q, const void* k, const void* v, const void* w, void* out,
                         float* s_out, int64_t B, int64_t H, int dtype, float scale, int prologue,
                         cudaStream_t stream) {
  const int64_t blocks = B * H * kTokTiles;
  if (!grid_fits(blocks)) return GDN2_ERR_TOO_LARGE;
  T1ZeroParams p{q, k, v, w, out, s_out, H, scale, prologue};
  if (dtype == GDN2_BF16) {
    if (prologue != 0) token_t1_zero_kernel<__nv_bfloat16, true><<<unsigned(blocks), kTokThreads, 0, stream>>>(p);
    else token_t1_zero_kernel<__nv_bfloat16, false><<<unsigned(blocks), kTokThreads, 0, stream>>>(p);
  } else {
    if (prologue != 0) token_t1_zero_kernel<__half, true><<<unsigned(blocks), kTokThreads, 0, stream>>>(p);
    else token_t1_zero_kernel<__half, false><<<unsigned(blocks), kTokThreads, 0, stream>>>(p);
  }
  return check_launch();
}

}  // namespace gdn2
