// Token path, 16 tokens at a time: forward, reverse state scan and VJP in fp32 on the CUDA cores.
//
// These serve the sequences (and ragged tails) shorter than one tensor-core chunk.  Walking the recurrence
// token by token costs two block-wide reductions and two barriers per token whatever the arithmetic (1.4 us
// forward, 13 us backward).  A span of up to 16 tokens is the same linear map written once (the compact-WY
// form of src/gdn2_sm120/reference.py:149-172 at chunk length 16): everything that reads the state is one
// contraction over it for all tokens of the span, the serial part shrinks to a 16 x 16 triangular solve per
// value column.  Per span, with a = exp(g), P_ij = a_{j+1} .. a_i (products of numbers <= 1: no anchor and
// no bound on g is needed, unlike the tensor-core chunks), e = beta k, s = scale q:
//     L_ij = sum_k e_i P_ij k_j (j < i)    A_ij = sum_k s_i P_ij k_j (j <= i)
//     E_i = e_i P_i0 a_0    Q_i = s_i P_i0 a_0    K_j = k_j P_{n-1,j}    D = a_0 .. a_{n-1}
//   forward   r = E S    u_i = w_i v_i - r_i - sum_{j<i} L_ij u_j    o = Q S + A u    S' = D S + K^T u
//   reverse   y_j = K_j dS' + sum_{i>=j} A_ij do_i    x_j = y_j - sum_{i>j} L_ij x_i  (= d(w v))
//             dS = D dS' + Q^T do - E^T x
//   VJP       dv = x w, dw = x v, dE = -x S^T, dQ = do S^T, dK = u dS'^T, dL = -x u^T, dA = do u^T,
//             and back through the definitions of L, A, E, Q, K, D to q, k, beta and g.
// Reference counterparts: recurrent.py:108-303, backward_parallel.py:625-718, 1052-1421, backward.py:378-797.

#include <type_traits>

#include "common.cuh"
#include "seqs.cuh"

namespace gdn2 {

int launch_packed_steps(const PackedSpans&, int, const void*, const void*, const void*, const void*, const void*,
                        const void*, const float*, void*, float*, float*, int64_t, int, int, float, int, bool,
                        cudaStream_t);

namespace {

constexpr int kSpan = kTokenInterval;          // 16
constexpr int64_t kStateElems = int64_t(kDim) * kDim;

// what a span's tokens look like in shared memory (fp32)
struct SpanRows {
  float a[kSpan][kDim];    // exp(g)
  float e[kSpan][kDim];    // beta k      -> E after finish_gram
  float k[kSpan][kDim];    // k           -> K
  float s[kSpan][kDim];    // scale q     -> Q
  float d[kDim];           // D
  float l[kSpan][kSpan];   // L[i][j], zero for j >= i
  float m[kSpan][kSpan];   // A[i][j], zero for j > i
  float lt[kSpan][kSpan];  // L[j][i]
  float mt[kSpan][kSpan];  // A[j][i]
};

// The token path takes tensors of any element alignment.  Whether four elements can be read at once is asked
// once for all tensors and not per load: a branch at each load keeps the next one from being issued behind it
// (8.3k of the 27k clocks of a span).
template <typename T, bool kVec>
__device__ __forceinline__ typename Raw4<T>::type load_quad(const void* base, int64_t idx) {
  if (kVec) return load4_raw<T>(base, idx);
  typename Raw4<T>::type raw;
  T* h = reinterpret_cast<T*>(&raw);
#pragma unroll
  for (int c = 0; c < 4; ++c) h[c] = static_cast<const T*>(base)[idx + c];
  return raw;
}
template <typename T>
__device__ __forceinline__ bool quads_aligned(const void* base) {
  return (reinterpret_cast<uintptr_t>(base) & (4 * sizeof(T) - 1)) == 0;
}
__device__ __forceinline__ void put4(float* p, const float (&x)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
}
__device__ __forceinline__ float4 get4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// Rows of the tokens `row0 .. row0 + n - 1` of head h: a warp per token, a lane per 4 channels, the loads of
// all the warp's tokens in flight together.  Rows n..15 become identity steps.  kPro: raw inputs are
// activated / normalised (prologue flags) on the way.
template <typename T, typename G, bool kPro, int kWarps>
__device__ __forceinline__ void load_rows(SpanRows& sm, const void* q, const void* k, const void* g, const void* beta,
                                          int64_t row0, int H, int h, int n, float scale, int prologue, int warp,
                                          int lane) {
  constexpr int kEach = kSpan / kWarps;
  typename Raw4<G>::type raw_g[kEach];
  typename Raw4<T>::type raw_b[kEach], raw_k[kEach], raw_q[kEach];
  auto fetch = [&](auto vec) {
    constexpr bool kVec = decltype(vec)::value;
#pragma unroll
    for (int x = 0; x < kEach; ++x) {
      // (a token that does not exist: the last one is read in its place, so that no branch separates the loads)
      const int64_t idx = ((row0 + min(warp + x * kWarps, n - 1)) * H + h) * kDim + 4 * lane;
      raw_g[x] = load_quad<G, kVec>(g, idx);
      raw_b[x] = load_quad<T, kVec>(beta, idx);
      raw_k[x] = load_quad<T, kVec>(k, idx);
      raw_q[x] = load_quad<T, kVec>(q, idx);
    }
  };
  if (quads_aligned<G>(g) && quads_aligned<T>(beta) && quads_aligned<T>(k) && quads_aligned<T>(q)) fetch(std::true_type{});
  else fetch(std::false_type{});
  float gv[kEach][4], bv[kEach][4], kk[kEach][4], s[kEach][4];
#pragma unroll
  for (int x = 0; x < kEach; ++x) {
    const int t = warp + x * kWarps;
    unpack4<G>(raw_g[x], gv[x]);
    unpack4<T>(raw_b[x], bv[x]);
    unpack4<T>(raw_k[x], kk[x]);
    unpack4<T>(raw_q[x], s[x]);
    if (kPro && (prologue & kPrologueNorm) != 0) {
      float sk = kk[x][0] * kk[x][0] + kk[x][1] * kk[x][1] + kk[x][2] * kk[x][2] + kk[x][3] * kk[x][3];
      float sq = s[x][0] * s[x][0] + s[x][1] * s[x][1] + s[x][2] * s[x][2] + s[x][3] * s[x][3];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        sk += __shfl_xor_sync(0xffffffffu, sk, off);
        sq += __shfl_xor_sync(0xffffffffu, sq, off);
      }
      const float ik = rsqrtf(sk + kPrologueEps), iq = rsqrtf(sq + kPrologueEps);
#pragma unroll
      for (int c = 0; c < 4; ++c) { kk[x][c] *= ik; s[x][c] *= iq; }
    }
    if (kPro && (prologue & kPrologueGate) != 0) {
#pragma unroll
      for (int c = 0; c < 4; ++c) { gv[x][c] = prologue_log_decay(gv[x][c]); bv[x][c] = prologue_sigmoid(bv[x][c]); }
    }
    const bool there = t < n;
    float a[4], e[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      kk[x][c] = there ? kk[x][c] : 0.f;
      a[c] = there ? expf(gv[x][c]) : 1.f;
      e[c] = there ? bv[x][c] * kk[x][c] : 0.f;
      s[x][c] = there ? s[x][c] * scale : 0.f;
    }
    put4(&sm.a[t][4 * lane], a);
    put4(&sm.e[t][4 * lane], e);
    put4(&sm.k[t][4 * lane], kk[x]);
    put4(&sm.s[t][4 * lane], s[x]);
  }
}

// L and A.  A warp takes the columns j = warp + kWarps c together, so that a row of a, e, s is read once for
// all of them; a lane has 4 channels.  For each row i the partial sums of all columns go through one
// transposing reduction over the warp.
template <int kWarps>
__device__ __forceinline__ void gram(SpanRows& sm, int warp, int lane) {
  constexpr int kC = kSpan / kWarps;  // columns of this warp: 4 or 2
  float4 p[kC];
#pragma unroll
  for (int c = 0; c < kC; ++c) p[c] = make_float4(0.f, 0.f, 0.f, 0.f);
  // (results stay in registers to the end: the compiler would not move a row's loads above the store of the
  // row before, which waits for a chain of shuffles)
  float total[kSpan];
#pragma unroll
  for (int i = 0; i < kSpan; ++i) {
    const float4 a = get4(&sm.a[i][4 * lane]), e = get4(&sm.e[i][4 * lane]), s = get4(&sm.s[i][4 * lane]);
    const float4 k = get4(&sm.k[i][4 * lane]);
    float x[2 * kC];
#pragma unroll
    for (int c = 0; c < kC; ++c) {  // P_ij k_j is zero up to i = j, which starts it
      if (c <= i / kWarps) {
        p[c].x *= a.x; p[c].y *= a.y; p[c].z *= a.z; p[c].w *= a.w;
      }
      x[c] = c <= i / kWarps ? fmaf(e.x, p[c].x, e.y * p[c].y) + fmaf(e.z, p[c].z, e.w * p[c].w) : 0.f;
      if (c == i / kWarps && warp == i % kWarps) p[c] = k;
      x[kC + c] = c <= i / kWarps ? fmaf(s.x, p[c].x, s.y * p[c].y) + fmaf(s.z, p[c].z, s.w * p[c].w) : 0.f;
    }
    // 2 kC values over 32 lanes: halve the values while there are several, then fold the lanes that share one
    int m = 16;
#pragma unroll
    for (int w = kC; w > 0; w >>= 1, m >>= 1) {
      const bool up = (lane & m) != 0;
#pragma unroll
      for (int j = 0; j < w; ++j) {
        const float send = up ? x[j] : x[j + w];
        x[j] = (up ? x[j + w] : x[j]) + __shfl_xor_sync(0xffffffffu, send, m);
      }
    }
#pragma unroll
    for (int f = 32 / (4 * kC); f > 0; f >>= 1) x[0] += __shfl_xor_sync(0xffffffffu, x[0], f);
    total[i] = x[0];
  }
  constexpr int kShare = 32 / (2 * kC);  // lanes with the same total
  if ((lane & (kShare - 1)) == 0) {
    const int value = lane / kShare, j = warp + kWarps * (value & (kC - 1));  // value: L of kC columns, then A
    float* dst = (value < kC ? &sm.l[0][0] : &sm.m[0][0]) + j;
    float* dst_t = (value < kC ? &sm.lt[0][0] : &sm.mt[0][0]) + j * kSpan;
#pragma unroll
    for (int i = 0; i < kSpan; ++i) dst[i * kSpan] = total[i];
#pragma unroll
    for (int i = 0; i < kSpan; i += 4) {
      *reinterpret_cast<float4*>(dst_t + i) = make_float4(total[i], total[i + 1], total[i + 2], total[i + 3]);
    }
  }
}
// After a barrier: e, s, k become E, Q, K and D is formed; threads 0..127, a channel each.
__device__ __forceinline__ void finish_gram(SpanRows& sm, int c) {
  float a[kSpan], e[kSpan], s[kSpan], k[kSpan];
#pragma unroll
  for (int i = 0; i < kSpan; ++i) { a[i] = sm.a[i][c]; e[i] = sm.e[i][c]; s[i] = sm.s[i][c]; k[i] = sm.k[i][c]; }
  float p = 1.f;
#pragma unroll
  for (int i = 0; i < kSpan; ++i) {
    p *= a[i];
    sm.e[i][c] = e[i] * p;
    sm.s[i][c] = s[i] * p;
  }
  sm.d[c] = p;
  p = 1.f;
#pragma unroll
  for (int i = kSpan - 1; i >= 0; --i) {
    sm.k[i][c] = k[i] * p;
    p *= a[i];
  }
}
// row i of a 16 x 16 matrix, the same for every lane
__device__ __forceinline__ void matrix_row(const float (*m)[kSpan], int i, float (&x)[kSpan]) {
#pragma unroll
  for (int j = 0; j < kSpan; j += 4) {
    const float4 q = get4(&m[i][j]);
    x[j] = q.x; x[j + 1] = q.y; x[j + 2] = q.z; x[j + 3] = q.w;
  }
}

// ---- forward and reverse state scan: one CTA = (sequence, head, 64 value columns) ---------------------
// 256 threads hold the state: thread = 8 key rows x 4 value columns, in registers from start to end (8 warps and
// not 4 on 32 columns, which also halves the Gram products per column).  Half of a span's work, its rows and
// Gram products, does not touch the state: with kSplit a second group of 256 threads prepares the next span
// meanwhile, in the other of two buffers (B4 T48 H16 training: forward 30 -> 24 us, reverse 29 -> 22; B4 T32
// raw 20 -> 17).  That is the form for grids that leave a CTA its SM alone; larger ones run two CTAs of 256
// threads per SM, which fill each other's waits as well and need no registers for two groups (B32 T32 H16 raw
// 105 us, split 121; B16 T48 the same either way).
constexpr int kThreads = 256, kWarps = kThreads / 32;
// named barriers: 1, 2 within a group; ready / free of buffer b between the groups
constexpr int kBarReady = 3, kBarFree = 5;
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// Runs prepare(span, buffer) and advance(span, buffer) for the spans 0 .. n - 1 in order.
template <bool kSplit, typename Prepare, typename Advance>
__device__ __forceinline__ void walk_spans(int n, bool preparer, Prepare prepare, Advance advance) {
  if constexpr (!kSplit) {
    for (int i = 0; i < n; ++i) {
      prepare(i, 0);
      __syncthreads();
      advance(i, 0);
      __syncthreads();
    }
  } else if (preparer) {
    for (int i = 0; i < n; ++i) {
      if (i >= 2) bar_sync(kBarFree + (i & 1), 2 * kThreads);
      prepare(i, i & 1);
      bar_arrive(kBarReady + (i & 1), 2 * kThreads);
    }
  } else {
    for (int i = 0; i < n; ++i) {
      bar_sync(kBarReady + (i & 1), 2 * kThreads);
      advance(i, i & 1);
      if (i + 2 < n) bar_arrive(kBarFree + (i & 1), 2 * kThreads);
    }
  }
}
constexpr int kCols = 64, kTiles = kDim / kCols;

// Warps 0..3 hold columns 0..31 of the tile, warps 4..7 columns 32..63.
struct TileThread {
  int lane, warp, rg, cc, rw, col0;  // rows 8 rg .. 8 rg + 7, columns col0 .. col0 + 3 (cc within the tile)
  __device__ TileThread(int tid, int tile)
      : lane(tid & 31), warp(tid >> 5), rg((tid >> 3) & 15), cc(32 * (tid >> 7) + 4 * (tid & 7)), rw((tid >> 5) & 3),
        col0(tile * kCols + cc) {}
};
__device__ __forceinline__ void load_tile(const float* state, const TileThread& t, float (&S)[8][4]) {
  const bool vec = (reinterpret_cast<uintptr_t>(state) & 15) == 0;
#pragma unroll
  for (int r = 0; r < 8; ++r) load4(state + (8 * t.rg + r) * kDim + t.col0, vec, S[r]);
}
__device__ __forceinline__ void store_tile(float* state, const TileThread& t, const float (&S)[8][4]) {
  const bool vec = (reinterpret_cast<uintptr_t>(state) & 15) == 0;
#pragma unroll
  for (int r = 0; r < 8; ++r) store4(state + (8 * t.rg + r) * kDim + t.col0, vec, S[r]);
}
__device__ __forceinline__ void load8(const float* p, float (&x)[8]) {
  const float4 lo = get4(p), hi = get4(p + 4);
  x[0] = lo.x; x[1] = lo.y; x[2] = lo.z; x[3] = lo.w;
  x[4] = hi.x; x[5] = hi.y; x[6] = hi.z; x[7] = hi.w;
}
// acc[c] = sum over this thread's rows of x[row] S[row][c]
__device__ __forceinline__ void rows_times_tile(const float* x, const TileThread& t, const float (&S)[8][4],
                                                float (&acc)[4]) {
  float v[8];
  load8(x + 8 * t.rg, v);
#pragma unroll
  for (int c = 0; c < 4; ++c) acc[c] = v[0] * S[0][c];
#pragma unroll
  for (int r = 1; r < 8; ++r) {
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[c] = fmaf(v[r], S[r][c], acc[c]);
  }
}
// S[row][c] += x[row] y[c]
__device__ __forceinline__ void rank_one(const float* x, const float* y, const TileThread& t, float sign,
                                         float (&S)[8][4]) {
  float v[8];
  load8(x + 8 * t.rg, v);
  float4 w = get4(y + t.cc);
  w.x *= sign; w.y *= sign; w.z *= sign; w.w *= sign;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    S[r][0] = fmaf(v[r], w.x, S[r][0]);
    S[r][1] = fmaf(v[r], w.y, S[r][1]);
    S[r][2] = fmaf(v[r], w.z, S[r][2]);
    S[r][3] = fmaf(v[r], w.w, S[r][3]);
  }
}
__device__ __forceinline__ void decay_rows(const float* d, const TileThread& t, float (&S)[8][4]) {
  float v[8];
  load8(d + 8 * t.rg, v);
#pragma unroll
  for (int r = 0; r < 8; ++r) {
#pragma unroll
    for (int c = 0; c < 4; ++c) S[r][c] *= v[r];
  }
}

template <bool kSplit>
struct FwdSmem {
  SpanRows rows[kSplit ? 2 : 1];
  float z[kSplit ? 2 : 1][kSpan][kCols];  // w v
  float u[kSpan][kCols];
  float part[4][kSpan][2][kCols];        // per warp of a column half: E S and Q S
};
struct SpanFwdParams {
  const void *q, *k, *v, *g, *beta, *w;
  const float* s_in;
  void* out;
  float *s_out, *bnd;
  int H;
  float scale;
  int prologue;
};

template <typename T, typename G, typename Seqs, bool kPro, bool kSplit>
__global__ void __launch_bounds__(kSplit ? 2 * kThreads : kThreads)
token_span_forward_kernel(const SpanFwdParams p, const __grid_constant__ Seqs seqs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FwdSmem<kSplit>& sm = *reinterpret_cast<FwdSmem<kSplit>*>(smem_raw);
  if constexpr (std::is_same<Seqs, PackedSpans>::value) let_others_begin();
  const int tid = threadIdx.x % kThreads, tile = int(blockIdx.x) % kTiles;
  const bool preparer = kSplit && threadIdx.x >= kThreads;
  const TileThread t(tid, tile);
  const int sh = int(blockIdx.x) / kTiles, s_ = sh / p.H, h = sh - s_ * p.H;
  const SeqInfo sq = seqs.at(s_);
  const int64_t state = (int64_t(sq.sid) * p.H + h) * kStateElems;
  auto sync = [&] { bar_sync(preparer ? 2 : 1, kThreads); };

  float S[8][4];
  if (p.s_in != nullptr && !preparer) {
    load_tile(p.s_in + state, t, S);
  } else {
#pragma unroll
    for (int r = 0; r < 8; ++r) S[r][0] = S[r][1] = S[r][2] = S[r][3] = 0.f;
  }
  auto prepare = [&](int span, int buf) {
    const int j0 = span * kSpan, n = min(kSpan, sq.len - j0);
    const int64_t row0 = sq.row0 + j0;
    SpanRows& rows = sm.rows[buf];
    constexpr int kZ = kSpan * kCols / kThreads;
    float wv[kZ], vv[kZ];  // (issued before anything waits)
#pragma unroll
    for (int x = 0; x < kZ; ++x) {
      const int i = (tid + x * kThreads) / kCols, c = tid % kCols;
      const int64_t idx = ((row0 + min(i, n - 1)) * p.H + h) * kDim + tile * kCols + c;
      wv[x] = ldf<T>(p.w, idx);
      vv[x] = ldf<T>(p.v, idx);
    }
    load_rows<T, G, kPro, kWarps>(rows, p.q, p.k, p.g, p.beta, row0, p.H, h, n, p.scale, p.prologue, t.warp, t.lane);
#pragma unroll
    for (int x = 0; x < kZ; ++x) {
      const int i = (tid + x * kThreads) / kCols, c = tid % kCols;
      if (kPro && (p.prologue & kPrologueGate) != 0) wv[x] = prologue_sigmoid(wv[x]);
      sm.z[buf][i][c] = i < n ? wv[x] * vv[x] : 0.f;
    }
    sync();
    gram<kWarps>(rows, t.warp, t.lane);
    sync();
    if (tid < kDim) finish_gram(rows, tid);
  };
  auto advance = [&](int span, int buf) {
    const int j0 = span * kSpan, n = min(kSpan, sq.len - j0);
    const int64_t row0 = sq.row0 + j0;
    const SpanRows& rows = sm.rows[buf];
    if (p.bnd != nullptr) store_tile(p.bnd + (int64_t(sq.slot0 + span) * p.H + h) * kStateElems, t, S);
    // E S and Q S: over this thread's rows, then over the four row groups of the warp; four tokens at a time
    // (rows of tokens that do not exist are zero)
#pragma unroll 1
    for (int i0 = 0; i0 < n; i0 += 4) {
      const bool b16 = (t.lane & 16) != 0, b8 = (t.lane & 8) != 0;
      float x[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float r[4], o[4], y[4];
        rows_times_tile(rows.e[i0 + i], t, S, r);
        rows_times_tile(rows.s[i0 + i], t, S, o);
#pragma unroll
        for (int c = 0; c < 4; ++c) y[c] = (b16 ? o[c] : r[c]) + __shfl_xor_sync(0xffffffffu, b16 ? r[c] : o[c], 16);
#pragma unroll
        for (int c = 0; c < 2; ++c) x[i][c] = (b8 ? y[c + 2] : y[c]) + __shfl_xor_sync(0xffffffffu, b8 ? y[c] : y[c + 2], 8);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        *reinterpret_cast<float2*>(&sm.part[t.rw][i0 + i][b16 ? 1 : 0][t.cc + (b8 ? 2 : 0)]) = make_float2(x[i][0], x[i][1]);
      }
    }
    sync();
    if (tid < kCols) {  // a thread per column: (I + L) u = z - E S
      const int col = tid;
      float u[kSpan];
#pragma unroll
      for (int i = 0; i < kSpan; ++i) {
        u[i] = i < n ? sm.z[buf][i][col] - ((sm.part[0][i][0][col] + sm.part[1][i][0][col]) +
                                          (sm.part[2][i][0][col] + sm.part[3][i][0][col]))
                     : 0.f;
      }
#pragma unroll
      for (int i = 0; i < kSpan; ++i) {
        float l[kSpan];
        matrix_row(rows.l, i, l);
#pragma unroll
        for (int j = 0; j < i; ++j) u[i] = fmaf(-l[j], u[j], u[i]);
      }
#pragma unroll
      for (int i = 0; i < kSpan; ++i) sm.u[i][col] = u[i];
    }
    sync();
    {
      const int col = tid % kCols;
      float u[kSpan];
#pragma unroll
      for (int j = 0; j < kSpan; ++j) u[j] = sm.u[j][col];
#pragma unroll
      for (int x = 0; x < kSpan * kCols / kThreads; ++x) {
        const int i = (tid + x * kThreads) / kCols;
        if (i < n) {
          float m[kSpan];
          matrix_row(rows.m, i, m);
          float o = (sm.part[0][i][1][col] + sm.part[1][i][1][col]) +
                    (sm.part[2][i][1][col] + sm.part[3][i][1][col]);
          // tokens up to i alone: what follows must not reach this output, not even as 0 times an infinity
          static_assert(kThreads / kCols == 4, "rows i of this thread: 4 x + 0..3");
#pragma unroll
          for (int j = 0; j < 4 * x + 4; ++j) o = j <= i ? fmaf(m[j], u[j], o) : o;
          stf<T>(p.out, ((row0 + i) * p.H + h) * kDim + tile * kCols + col, o);
        }
      }
    }
    decay_rows(rows.d, t, S);
#pragma unroll 1
    for (int i0 = 0; i0 < n; i0 += 4) {
#pragma unroll
      for (int j = i0; j < i0 + 4; ++j) rank_one(rows.k[j], sm.u[j], t, 1.f, S);
    }
    if (kSplit) sync();  // (u and part are written again)
  };
  walk_spans<kSplit>(sq.n_chunks, preparer, prepare, advance);
  if (preparer) return;
  if (p.bnd != nullptr) store_tile(p.bnd + (int64_t(sq.slot0 + sq.n_chunks) * p.H + h) * kStateElems, t, S);
  if (p.s_out != nullptr) store_tile(p.s_out + state, t, S);
  if constexpr (std::is_same<Seqs, PackedSpans>::value) outlast_others();
}

// ---- reverse scan of the state cotangent -------------------------------------------------------------
template <bool kSplit>
struct RevSmem {
  SpanRows rows[kSplit ? 2 : 1];
  float d_out[kSplit ? 2 : 1][kSpan][kCols];
  float x[kSpan][kCols];                // d(w v)
  float part[4][kSpan][kCols];          // per warp of a column half: K dS'
};
struct SpanRevParams {
  const void *q, *k, *g, *beta, *d_out;
  const float* ds_final;
  float *d_bnd, *ds_init;
  int H;
  float scale;
};

template <typename T, typename G, typename Seqs, bool kSplit>
__global__ void __launch_bounds__(kSplit ? 2 * kThreads : kThreads)
token_span_reverse_kernel(const SpanRevParams p, const __grid_constant__ Seqs seqs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RevSmem<kSplit>& sm = *reinterpret_cast<RevSmem<kSplit>*>(smem_raw);
  if constexpr (std::is_same<Seqs, PackedSpans>::value) let_others_begin();  // the reverse scans of the longer sequences
  const int tid = threadIdx.x % kThreads, tile = int(blockIdx.x) % kTiles;
  const bool preparer = kSplit && threadIdx.x >= kThreads;
  const TileThread t(tid, tile);
  const int sh = int(blockIdx.x) / kTiles, s_ = sh / p.H, h = sh - s_ * p.H;
  const SeqInfo sq = seqs.at(s_);
  const int64_t state = (int64_t(sq.sid) * p.H + h) * kStateElems;
  auto sync = [&] { bar_sync(preparer ? 2 : 1, kThreads); };

  float dS[8][4];
  if (p.ds_final != nullptr && !preparer) {
    load_tile(p.ds_final + state, t, dS);
  } else {
#pragma unroll
    for (int r = 0; r < 8; ++r) dS[r][0] = dS[r][1] = dS[r][2] = dS[r][3] = 0.f;
  }
  // step `it` works on span n_chunks - 1 - it
  auto prepare = [&](int it, int buf) {
    const int j0 = (sq.n_chunks - 1 - it) * kSpan, n = min(kSpan, sq.len - j0);
    const int64_t row0 = sq.row0 + j0;
    SpanRows& rows = sm.rows[buf];
    constexpr int kZ = kSpan * kCols / kThreads;
    float o[kZ];  // (issued before anything waits)
#pragma unroll
    for (int x = 0; x < kZ; ++x) {
      const int i = (tid + x * kThreads) / kCols, c = tid % kCols;
      o[x] = ldf<T>(p.d_out, ((row0 + min(i, n - 1)) * p.H + h) * kDim + tile * kCols + c);
    }
    load_rows<T, G, false, kWarps>(rows, p.q, p.k, p.g, p.beta, row0, p.H, h, n, p.scale, 0, t.warp, t.lane);
#pragma unroll
    for (int x = 0; x < kZ; ++x) {
      const int i = (tid + x * kThreads) / kCols, c = tid % kCols;
      sm.d_out[buf][i][c] = i < n ? o[x] : 0.f;
    }
    sync();
    gram<kWarps>(rows, t.warp, t.lane);
    sync();
    if (tid < kDim) finish_gram(rows, tid);
  };
  auto advance = [&](int it, int buf) {
    const int span = sq.n_chunks - 1 - it, n = min(kSpan, sq.len - span * kSpan);
    const SpanRows& rows = sm.rows[buf];
    store_tile(p.d_bnd + (int64_t(sq.slot0 + span + 1) * p.H + h) * kStateElems, t, dS);
#pragma unroll 1
    for (int i0 = 0; i0 < n; i0 += 4) {
      const bool b16 = (t.lane & 16) != 0, b8 = (t.lane & 8) != 0;
      float x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float r[4], y[2];
        rows_times_tile(rows.k[i0 + i], t, dS, r);
#pragma unroll
        for (int c = 0; c < 2; ++c) y[c] = (b16 ? r[c + 2] : r[c]) + __shfl_xor_sync(0xffffffffu, b16 ? r[c] : r[c + 2], 16);
        x[i] = (b8 ? y[1] : y[0]) + __shfl_xor_sync(0xffffffffu, b8 ? y[0] : y[1], 8);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) sm.part[t.rw][i0 + i][t.cc + (b16 ? 2 : 0) + (b8 ? 1 : 0)] = x[i];
    }
    sync();
    if (tid < kCols) {  // a thread per column: (I + L)^T x = K dS' + A^T do
      const int col = tid;
      float x[kSpan], o[kSpan];
#pragma unroll
      for (int i = 0; i < kSpan; ++i) {
        o[i] = sm.d_out[buf][i][col];
        x[i] = i < n ? (sm.part[0][i][col] + sm.part[1][i][col]) + (sm.part[2][i][col] + sm.part[3][i][col])
                     : 0.f;
      }
#pragma unroll
      for (int i = kSpan - 1; i >= 0; --i) {
        float l[kSpan], m[kSpan];
        matrix_row(rows.mt, i, m);
        matrix_row(rows.lt, i, l);
#pragma unroll
        for (int j = i; j < kSpan; ++j) x[i] = fmaf(m[j], o[j], x[i]);
#pragma unroll
        for (int j = kSpan - 1; j > i; --j) x[i] = fmaf(-l[j], x[j], x[i]);
      }
#pragma unroll
      for (int i = 0; i < kSpan; ++i) sm.x[i][col] = x[i];
    }
    sync();
    decay_rows(rows.d, t, dS);
#pragma unroll 1
    for (int i0 = 0; i0 < n; i0 += 2) {
#pragma unroll
      for (int i = i0; i < i0 + 2; ++i) {
        rank_one(rows.s[i], sm.d_out[buf][i], t, 1.f, dS);
        rank_one(rows.e[i], sm.x[i], t, -1.f, dS);
      }
    }
    if (kSplit) sync();  // (x and part are written again)
  };
  walk_spans<kSplit>(sq.n_chunks, preparer, prepare, advance);
  if (preparer) return;
  store_tile(p.d_bnd + int64_t(sq.slot0 * int64_t(p.H) + h) * kStateElems, t, dS);
  if (p.ds_init != nullptr) store_tile(p.ds_init + state, t, dS);
}

// ---- VJP of one span ------------------------------------------------------------------------------------
// One CTA = (span, head), 256 threads.  A thread keeps an 8 x 8 block of S (span start) and of dS' (span end)
// in registers for both kinds of contraction: over keys (E S, K dS', partial sums of its rows) and over
// values (x S^T, do S^T, u dS'^T, partial sums of its columns); the sums over the other threads go through
// transposing shuffles and one array in shared memory.  Then a thread per key channel and token parity walks
// back through the definitions of L, A, E, Q, K.  320 multiply-adds per token and thread, issue bound.
constexpr int kVjpThreads = 256;
constexpr int kLdV = kDim + 4;  // rows of 128 values, shifted by 4 banks each

struct VjpSmem {
  SpanRows rows;
  float x[kSpan][kLdV], u[kSpan][kLdV], d_out[kSpan][kLdV];
  float2 dla[kSpan][kSpan];             // (dL, dA)[i][j]
  union {
    float keys[4][kSpan][2][kDim];      // per row group of four: E S, K dS'
    struct {
      float vals[2][kSpan][3][kDim];    // per column half: dE (negated), dQ, dK
      float dd[2][kDim];                // ... and sum_v S dS'
      float de[kSpan][kDim], ds[kSpan][kDim], dk[kSpan][kDim], dg[kSpan][kDim];  // the other parity's share
    };
  };
  float ends[2][kDim];                  // dG: key terms of tokens 0..7, query and erase terms of tokens 8..15
};
struct SpanVjpParams {
  const void *q, *k, *v, *g, *beta, *w, *d_out;
  const float *bnd, *d_bnd;
  void *dq, *dk, *dv, *dg, *dbeta, *dw;
  int H;
  float scale;
};

template <typename T, typename G, typename Seqs>
__global__ void __launch_bounds__(kVjpThreads, 1)
token_span_vjp_kernel(const SpanVjpParams p, const __grid_constant__ Seqs seqs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  VjpSmem& sm = *reinterpret_cast<VjpSmem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rgl = lane >> 3, cgl = lane & 7, rgh = warp >> 1, cgh = warp & 1;
  const int r0 = 8 * (4 * rgh + rgl), c0 = 8 * (8 * cgh + cgl);  // this thread's rows and columns
  const int span = int(blockIdx.x) / p.H, h = int(blockIdx.x) - span * p.H;
  const SeqInfo sq = seqs.at(seqs.find(span));
  const int j_ = span - sq.chunk0, n = min(kSpan, sq.len - j_ * kSpan);
  const int64_t row0 = sq.row0 + j_ * kSpan;

  float S[8][8], dS[8][8];
  {
    const float* s_src = p.bnd + (int64_t(sq.slot0 + j_) * p.H + h) * kStateElems + r0 * kDim + c0;
    const float* d_src = p.d_bnd + (int64_t(sq.slot0 + j_ + 1) * p.H + h) * kStateElems + r0 * kDim + c0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      load8(s_src + r * kDim, S[r]);
      load8(d_src + r * kDim, dS[r]);
    }
  }
  constexpr int kEach = kSpan / (kVjpThreads / 32);
  typename Raw4<T>::type raw_o[kEach];
  auto fetch_o = [&](auto vec) {
#pragma unroll
    for (int x = 0; x < kEach; ++x) {
      const int i = min(warp + x * (kVjpThreads / 32), n - 1);
      raw_o[x] = load_quad<T, decltype(vec)::value>(p.d_out, ((row0 + i) * p.H + h) * kDim + 4 * lane);
    }
  };
  if (quads_aligned<T>(p.d_out)) fetch_o(std::true_type{});
  else fetch_o(std::false_type{});
  load_rows<T, G, false, kVjpThreads / 32>(sm.rows, p.q, p.k, p.g, p.beta, row0, p.H, h, n, p.scale, 0, warp, lane);
#pragma unroll
  for (int x = 0; x < kEach; ++x) {
    const int i = warp + x * (kVjpThreads / 32);
    float o[4];
    unpack4<T>(raw_o[x], o);
    if (i >= n) o[0] = o[1] = o[2] = o[3] = 0.f;
    put4(&sm.d_out[i][4 * lane], o);
  }
  __syncthreads();
  gram<kVjpThreads / 32>(sm.rows, warp, lane);
  __syncthreads();
  if (tid < kDim) finish_gram(sm.rows, tid);
  __syncthreads();

  // ---- over keys: E S and K dS', two tokens at a time (rows of tokens that do not exist are zero) ---------
#pragma unroll 1
  for (int i0 = 0; i0 < n; i0 += 2) {
    const bool b16 = (lane & 16) != 0, b8 = (lane & 8) != 0;
    float y[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float e[8], k[8], x[16];
      load8(&sm.rows.e[i0 + i][r0], e);
      load8(&sm.rows.k[i0 + i][r0], k);
#pragma unroll
      for (int c = 0; c < 8; ++c) { x[c] = e[0] * S[0][c]; x[8 + c] = k[0] * dS[0][c]; }
#pragma unroll
      for (int r = 1; r < 8; ++r) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          x[c] = fmaf(e[r], S[r][c], x[c]);
          x[8 + c] = fmaf(k[r], dS[r][c], x[8 + c]);
        }
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) x[c] = (b16 ? x[8 + c] : x[c]) + __shfl_xor_sync(0xffffffffu, b16 ? x[c] : x[8 + c], 16);
#pragma unroll
      for (int c = 0; c < 4; ++c) y[i][c] = (b8 ? x[4 + c] : x[c]) + __shfl_xor_sync(0xffffffffu, b8 ? x[c] : x[4 + c], 8);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      *reinterpret_cast<float4*>(&sm.keys[rgh][i0 + i][b16 ? 1 : 0][c0 + (b8 ? 4 : 0)]) =
          make_float4(y[i][0], y[i][1], y[i][2], y[i][3]);
    }
  }
  __syncthreads();
  // ---- a thread per value column: u by the first 128 threads, x (with dv and dw) by the others ------------
  {
    const int col = tid & (kDim - 1);
    float wv[kSpan], vv[kSpan], y[kSpan];
#pragma unroll
    for (int i = 0; i < kSpan; ++i) {
      const int64_t idx = ((row0 + min(i, n - 1)) * p.H + h) * kDim + col;
      wv[i] = ldf<T>(p.w, idx);
      vv[i] = ldf<T>(p.v, idx);
    }
    const int kind = tid >> 7;
#pragma unroll
    for (int i = 0; i < kSpan; ++i) {
      y[i] = i < n ? (sm.keys[0][i][kind][col] + sm.keys[1][i][kind][col]) +
                         (sm.keys[2][i][kind][col] + sm.keys[3][i][kind][col])
                   : 0.f;
    }
    if (kind == 0) {
#pragma unroll
      for (int i = 0; i < kSpan; ++i) {
        y[i] = i < n ? fmaf(wv[i], vv[i], -y[i]) : 0.f;
        float l[kSpan];
        matrix_row(sm.rows.l, i, l);
#pragma unroll
        for (int j = 0; j < i; ++j) y[i] = fmaf(-l[j], y[j], y[i]);
      }
#pragma unroll
      for (int i = 0; i < kSpan; ++i) sm.u[i][col] = y[i];
    } else {
      float o[kSpan];
#pragma unroll
      for (int i = 0; i < kSpan; ++i) o[i] = sm.d_out[i][col];
#pragma unroll
      for (int i = kSpan - 1; i >= 0; --i) {
        float l[kSpan], m[kSpan];
        matrix_row(sm.rows.mt, i, m);
        matrix_row(sm.rows.lt, i, l);
#pragma unroll
        for (int j = i; j < kSpan; ++j) y[i] = fmaf(m[j], o[j], y[i]);
#pragma unroll
        for (int j = kSpan - 1; j > i; --j) y[i] = fmaf(-l[j], y[j], y[i]);
      }
#pragma unroll
      for (int i = 0; i < kSpan; ++i) {
        sm.x[i][col] = y[i];
        if (i < n) {
          const int64_t idx = ((row0 + i) * p.H + h) * kDim + col;
          stf<T>(p.dv, idx, y[i] * wv[i]);
          stf<T>(p.dw, idx, y[i] * vv[i]);
        }
      }
    }
  }
  __syncthreads();
  // ---- dL and dA: a thread per (i, j) --------------------------------------------------------------------
  {
    const int i = tid >> 4, j = tid & 15;
    float dl = 0.f, da = 0.f;
    if (j <= i) {
#pragma unroll 4
      for (int c = 0; c < kDim; c += 4) {
        const float4 x = get4(&sm.x[i][c]), o = get4(&sm.d_out[i][c]), u = get4(&sm.u[j][c]);
        dl = fmaf(x.x, u.x, fmaf(x.y, u.y, fmaf(x.z, u.z, fmaf(x.w, u.w, dl))));
        da = fmaf(o.x, u.x, fmaf(o.y, u.y, fmaf(o.z, u.z, fmaf(o.w, u.w, da))));
      }
    }
    sm.dla[i][j] = make_float2(j < i ? -dl : 0.f, da);
  }
  // ---- over values: x S^T (= -dE), do S^T, u dS'^T, and S . dS' ---------------------------------------------
  auto across_columns = [&](float (&y)[24], float (&sum)[3], int kinds) {
    // 24 sums (kind, row) over the eight lanes that share this thread's rows: lane cgl keeps row cgl of each
    const bool b4 = (lane & 4) != 0, b2 = (lane & 2) != 0, b1 = (lane & 1) != 0;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      if (q < kinds) {
        float z[8];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          z[r] = (b4 ? y[8 * q + 4 + r] : y[8 * q + r]) +
                 __shfl_xor_sync(0xffffffffu, b4 ? y[8 * q + r] : y[8 * q + 4 + r], 4);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) z[r] = (b2 ? z[2 + r] : z[r]) + __shfl_xor_sync(0xffffffffu, b2 ? z[r] : z[2 + r], 2);
        sum[q] = (b1 ? z[1] : z[0]) + __shfl_xor_sync(0xffffffffu, b1 ? z[0] : z[1], 1);
      }
    }
  };
#pragma unroll 1
  for (int i0 = 0; i0 < n; i0 += 2) {
    float sum[2][3];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float x[8], o[8], u[8], y[24];
      load8(&sm.x[i0 + i][c0], x);
      load8(&sm.d_out[i0 + i][c0], o);
      load8(&sm.u[i0 + i][c0], u);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        y[r] = x[0] * S[r][0];
        y[8 + r] = o[0] * S[r][0];
        y[16 + r] = u[0] * dS[r][0];
#pragma unroll
        for (int c = 1; c < 8; ++c) {
          y[r] = fmaf(x[c], S[r][c], y[r]);
          y[8 + r] = fmaf(o[c], S[r][c], y[8 + r]);
          y[16 + r] = fmaf(u[c], dS[r][c], y[16 + r]);
        }
      }
      across_columns(y, sum[i], 3);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
      for (int q = 0; q < 3; ++q) sm.vals[cgh][i0 + i][q][r0 + cgl] = sum[i][q];
    }
  }
  {
    float y[24], sum[3];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      y[r] = S[r][0] * dS[r][0];
#pragma unroll
      for (int c = 1; c < 8; ++c) y[r] = fmaf(S[r][c], dS[r][c], y[r]);
    }
    across_columns(y, sum, 1);
    sm.dd[cgh][r0 + cgl] = sum[0];
  }
  __syncthreads();

  // ---- a thread per key channel and column parity: through L and A -----------------------------------------
  const int c = tid & (kDim - 1), par = tid >> 7;
  float kk[kSpan], bb[kSpan], ss[kSpan], aa[kSpan];
#pragma unroll
  for (int i = 0; i < kSpan; ++i) {
    const int64_t idx = ((row0 + min(i, n - 1)) * p.H + h) * kDim + c;
    kk[i] = ldf<T>(p.k, idx);
    bb[i] = ldf<T>(p.beta, idx);
    ss[i] = p.scale * ldf<T>(p.q, idx);
    aa[i] = sm.rows.a[i][c];
  }
  // dG_t, t = 0..15, is a sum of terms that each hold a_t (through P), so that it is right to fp32 precision at
  // any decay: D S . dS', the query and erase terms of tokens i >= t with S, the key terms of tokens j < t with
  // dS', and of the pairs (i, j) those with j < t <= i.  (Row sums minus column sums of all pairs from t on are
  // the same number, but terms of order one cancel in it: relative error of dg 2e-4 at g = -10 a token and
  // 0.4 at -25, against 1.0e-7 and 0.7e-7 in this form, which costs 5 of 311 us at B16 T48 H16.)
  float de[kSpan], ds[kSpan], dk[kSpan / 2];
  float pair[kSpan], dg[kSpan];  // pair terms of row i with this thread's columns so far; their sums over i >= t
#pragma unroll
  for (int i = 0; i < kSpan; ++i) de[i] = ds[i] = pair[i] = dg[i] = 0.f;
  float behind = 0.f;            // sum of pair[i] over i > 2 jj
#pragma unroll
  for (int jj = 0; jj < kSpan / 2; ++jj) {
    // columns j = 2 jj + par; written for both parities so that every index is a constant (tokens that do not
    // exist have zero rows and columns in dL and dA)
    float kj = par ? kk[2 * jj + 1] : kk[2 * jj], p_ij = 1.f, col = 0.f;
#pragma unroll
    for (int i = 2 * jj; i < kSpan; ++i) {
      const bool mine = i > 2 * jj || par == 0;  // i >= j
      if (i > 2 * jj + 1 || (i == 2 * jj + 1 && par == 0)) p_ij *= aa[i];
      const float2 d = sm.dla[i][2 * jj + par];
      const float t = mine ? p_ij : 0.f, tk = t * kj;
      de[i] = fmaf(d.x, tk, de[i]);
      ds[i] = fmaf(d.y, tk, ds[i]);
      const float row = fmaf(d.x, bb[i] * kk[i], d.y * ss[i]);
      col = fmaf(row, t, col);
      if (i > 2 * jj) pair[i] = fmaf(row, i > 2 * jj + 1 || par == 0 ? tk : 0.f, pair[i]);  // (i > j)
    }
    dk[jj] = col;
    float rest = 0.f;
#pragma unroll
    for (int i = kSpan - 1; i > 2 * jj + 2; --i) rest += pair[i];
    const float from = jj + 1 < kSpan / 2 ? rest + pair[2 * jj + 2] : 0.f;
    if (jj + 1 < kSpan / 2) dg[2 * jj + 2] = from;
    dg[2 * jj + 1] = par ? behind : pair[2 * jj + 1] + from;  // (column 2 jj + 1 is not one of its columns)
    behind = rest;
  }
  // hand the other parity's thread what it finishes: tokens 0..7 are finished by parity 0, 8..15 by parity 1
#pragma unroll
  for (int i = 0; i < kSpan; ++i) {
    if ((i >= kSpan / 2) != (par == 1)) {
      sm.de[i][c] = de[i];
      sm.ds[i][c] = ds[i];
      sm.dg[i][c] = dg[i];
    }
    if ((i & 1) == par) sm.dk[i][c] = dk[i >> 1];
  }
  __syncthreads();
  float before = 1.f, after = 1.f;  // decays of the other half's tokens
#pragma unroll
  for (int i = 0; i < kSpan / 2; ++i) { before *= aa[i]; after *= aa[kSpan / 2 + i]; }
  const int half = par * (kSpan / 2);
  float run_c = par ? before : 1.f, total = 0.f, reads[kSpan / 2], keys[kSpan / 2], decay[kSpan / 2];
#pragma unroll
  for (int x = 0; x < kSpan / 2; ++x) decay[x] = par ? aa[kSpan / 2 + x] : aa[x];
  float tails[kSpan / 2];
  {
    float run = par ? 1.f : after;
#pragma unroll
    for (int x = kSpan / 2 - 1; x >= 0; --x) { tails[x] = run; run *= decay[x]; }
  }
#pragma unroll
  for (int x = 0; x < kSpan / 2; ++x) {
    const int i = half + x;
    run_c *= decay[x];
    const float k = par ? kk[kSpan / 2 + x] : kk[x], b = par ? bb[kSpan / 2 + x] : bb[x];
    const float s = par ? ss[kSpan / 2 + x] : ss[x], e = b * k;
    const float gde = (par ? de[kSpan / 2 + x] : de[x]) + sm.de[i][c];
    const float gds = (par ? ds[kSpan / 2 + x] : ds[x]) + sm.ds[i][c];
    const float gdk = sm.dk[i][c];
    float d_e = 0.f, d_q = 0.f, d_k = 0.f;
    if (i < n) {
      d_e = -(sm.vals[0][i][0][c] + sm.vals[1][i][0][c]);
      d_q = sm.vals[0][i][1][c] + sm.vals[1][i][1][c];
      d_k = sm.vals[0][i][2][c] + sm.vals[1][i][2][c];
    }
    const float ce = fmaf(d_e, run_c, gde), cs = fmaf(d_q, run_c, gds), ck = fmaf(d_k, tails[x], gdk);
    if (i < n) {
      const int64_t idx = ((row0 + i) * p.H + h) * kDim + c;
      stf<T>(p.dq, idx, p.scale * cs);
      stf<T>(p.dk, idx, fmaf(b, ce, ck));
      stf<T>(p.dbeta, idx, k * ce);
    }
    reads[x] = fmaf(e, d_e, s * d_q) * run_c;
    keys[x] = k * (d_k * tails[x]);
    total += par ? reads[x] : keys[x];
  }
  sm.ends[par][c] = total;
  __syncthreads();
  float state = before * after * (sm.dd[0][c] + sm.dd[1][c]);
  if (par) state += sm.ends[0][c];
  float sum[kSpan / 2];
#pragma unroll
  for (int x = 0; x < kSpan / 2; ++x) {
    sum[x] = state + ((par ? dg[kSpan / 2 + x] : dg[x]) + sm.dg[half + x][c]);
    state += keys[x];
  }
  float run = par ? 0.f : sm.ends[1][c];
#pragma unroll
  for (int x = kSpan / 2 - 1; x >= 0; --x) {
    run += reads[x];
    const int i = half + x;
    if (i < n) stf<G>(p.dg, ((row0 + i) * p.H + h) * kDim + c, sum[x] + run);
  }
  if constexpr (std::is_same<Seqs, PackedSpans>::value) outlast_others();
}

inline int64_t spans_for(int64_t tokens) { return (tokens + kSpan - 1) / kSpan; }
inline bool grid_fits(int64_t blocks) { return blocks > 0 && blocks <= int64_t(0x7fffffff); }

// batch rows' token ranges [t_begin, t_end); false when a grid or a slot number would not fit 31 bits
bool uniform_spans(int64_t B, int64_t T, int64_t H, int64_t t_begin, int64_t t_end, UniformSeqs* seqs) {
  const int64_t spans = spans_for(t_end - t_begin);
  if (t_end - t_begin > int64_t(0x7fffffff) || !grid_fits(B * H * kTiles) ||
      B * (spans + 1) * H > int64_t(0x7fffffff)) {
    return false;
  }
  *seqs = UniformSeqs{t_begin, T, int(t_end - t_begin), int(spans), int(B)};
  return true;
}

template <typename Kernel, typename Params, typename Seqs>
int launch(Kernel kernel, int64_t blocks, int threads, int smem, const Params& p, const Seqs& seqs,
           cudaStream_t stream, bool beside = false) {
  if (!grid_fits(blocks)) return GDN2_ERR_TOO_LARGE;
  const cudaError_t err = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
  if (err != cudaSuccess) { record_cuda_error(err); return GDN2_ERR_LAUNCH; }
  if (beside) return launch_beside(kernel, unsigned(blocks), threads, smem, stream, p, seqs);
  kernel<<<unsigned(blocks), threads, smem, stream>>>(p, seqs);
  return check_launch();
}

// kSplit needs a second span to prepare (a packed batch lists its longest sequence first) and an SM per CTA.
template <typename Seqs>
int prefer_split(const Seqs& seqs, int64_t H, bool* split) {
  int sm_count = 0;
  if (int st = multiprocessors(&sm_count); st != GDN2_OK) return st;
  *split = seqs.count() > 0 && seqs.at(0).len > kSpan && int64_t(seqs.count()) * H * kTiles <= sm_count;
  return GDN2_OK;
}
template <bool kPro, bool kSplit, typename Seqs>
int run_forward(const Seqs& seqs, const SpanFwdParams& p, int dtype, int g_dtype, cudaStream_t stream, bool beside) {
  const int64_t blocks = int64_t(seqs.count()) * p.H * kTiles;
  int st = GDN2_OK;
  GDN2_DISPATCH_TYPES(dtype, g_dtype, {
    st = launch(token_span_forward_kernel<T, G, Seqs, kPro, kSplit>, blocks, kSplit ? 2 * kThreads : kThreads,
                int(sizeof(FwdSmem<kSplit>)), p, seqs, stream, beside);
  });
  return st;
}
template <typename Seqs>
int run_forward(const Seqs& seqs, const SpanFwdParams& p, int dtype, int g_dtype, cudaStream_t stream,
                bool beside = false) {
  bool split = false;
  if (int st = prefer_split(seqs, p.H, &split); st != GDN2_OK) return st;
  auto run = p.prologue != 0 ? (split ? run_forward<true, true, Seqs> : run_forward<true, false, Seqs>)
                             : (split ? run_forward<false, true, Seqs> : run_forward<false, false, Seqs>);
  return run(seqs, p, dtype, g_dtype, stream, beside);
}
template <bool kSplit, typename Seqs>
int run_reverse(const Seqs& seqs, const SpanRevParams& p, int dtype, int g_dtype, cudaStream_t stream) {
  const int64_t blocks = int64_t(seqs.count()) * p.H * kTiles;
  int st = GDN2_OK;
  GDN2_DISPATCH_TYPES(dtype, g_dtype, {
    st = launch(token_span_reverse_kernel<T, G, Seqs, kSplit>, blocks, kSplit ? 2 * kThreads : kThreads,
                int(sizeof(RevSmem<kSplit>)), p, seqs, stream);
  });
  return st;
}
template <typename Seqs>
int run_reverse(const Seqs& seqs, const SpanRevParams& p, int dtype, int g_dtype, cudaStream_t stream) {
  bool split = false;
  if (int st = prefer_split(seqs, p.H, &split); st != GDN2_OK) return st;
  return (split ? run_reverse<true, Seqs> : run_reverse<false, Seqs>)(seqs, p, dtype, g_dtype, stream);
}
template <typename Seqs>
int run_vjp(const Seqs& seqs, const SpanVjpParams& p, int dtype, int g_dtype, cudaStream_t stream,
            bool beside = false) {
  const int64_t blocks = int64_t(seqs.total_chunks()) * p.H;
  int st = GDN2_OK;
  GDN2_DISPATCH_TYPES(dtype, g_dtype, {
    st = launch(token_span_vjp_kernel<T, G, Seqs>, blocks, kVjpThreads, int(sizeof(VjpSmem)), p, seqs, stream, beside);
  });
  return st;
}

}  // namespace

// ---- launchers (called from api.cu, packed.cu and token_kernels.cu) ---------------------------------------
int launch_span_forward(const void* q, const void* k, const void* v, const void* g, const void* beta, const void* w,
                        const float* s_in, void* out, float* s_out, float* bnd, int64_t B, int64_t T, int64_t H,
                        int64_t t_begin, int64_t t_end, int dtype, int g_dtype, float scale, int prologue,
                        cudaStream_t stream) {
  UniformSeqs seqs;
  if (!uniform_spans(B, T, H, t_begin, t_end, &seqs)) return GDN2_ERR_TOO_LARGE;
  return run_forward(seqs, SpanFwdParams{q, k, v, g, beta, w, s_in, out, s_out, bnd, int(H), scale, prologue}, dtype,
                     g_dtype, stream);
}

int launch_token_dstate_scan(const void* q, const void* k, const void* g, const void* beta,
                             const void* d_out, const float* ds_final, float* d_bnd,
                             float* ds_init, int64_t B, int64_t T, int64_t H, int64_t t_begin,
                             int64_t t_end, int dtype, int g_dtype, float scale,
                             cudaStream_t stream) {
  UniformSeqs seqs;
  if (!uniform_spans(B, T, H, t_begin, t_end, &seqs)) return GDN2_ERR_TOO_LARGE;
  return run_reverse(seqs, SpanRevParams{q, k, g, beta, d_out, ds_final, d_bnd, ds_init, int(H), scale}, dtype,
                     g_dtype, stream);
}

int launch_token_chunk_vjp(const void* q, const void* k, const void* v, const void* g,
                           const void* beta, const void* w, const void* d_out, const float* bnd,
                           const float* d_bnd, void* dq, void* dk, void* dv, void* dg,
                           void* dbeta, void* dw, int64_t B, int64_t T, int64_t H,
                           int64_t t_begin, int64_t t_end, int dtype, int g_dtype, float scale,
                           cudaStream_t stream) {
  UniformSeqs seqs;
  if (!uniform_spans(B, T, H, t_begin, t_end, &seqs)) return GDN2_ERR_TOO_LARGE;
  return run_vjp(seqs, SpanVjpParams{q, k, v, g, beta, w, d_out, bnd, d_bnd, dq, dk, dv, dg, dbeta, dw, int(H), scale},
                 dtype, g_dtype, stream);
}

int launch_packed_token_forward(const PackedSpans& table, const void* q, const void* k, const void* v, const void* g,
                                const void* beta, const void* w, const float* s_in, void* out, float* s_out,
                                float* bnd, int64_t H, int dtype, int g_dtype, float scale, int prologue, bool beside,
                                cudaStream_t stream) {
  // longest first: the sequences of a few tokens are the end of the list
  int spans = 0;
  while (spans < table.n && table.e[spans].len > step_tokens(prologue)) ++spans;
  if (spans > 0) {
    PackedSpans longer = table;
    longer.n = spans;
    const int st = run_forward(longer, SpanFwdParams{q, k, v, g, beta, w, s_in, out, s_out, bnd, int(H), scale, prologue},
                               dtype, g_dtype, stream, beside);
    if (st != GDN2_OK || spans == table.n) return st;
    beside = !profiling();
  }
  return launch_packed_steps(table, spans, q, k, v, g, beta, w, s_in, out, s_out, bnd, H, dtype, g_dtype, scale,
                             prologue, beside, stream);
}

int launch_packed_token_reverse(const PackedSpans& table, const void* q, const void* k, const void* g, const void* beta,
                                const void* d_out, const float* ds_final, float* d_bnd, float* ds_init, int64_t H,
                                int dtype, int g_dtype, float scale, cudaStream_t stream) {
  return run_reverse(table, SpanRevParams{q, k, g, beta, d_out, ds_final, d_bnd, ds_init, int(H), scale}, dtype, g_dtype,
                     stream);
}

int launch_packed_token_vjp(const PackedSpans& table, const void* q, const void* k, const void* v, const void* g,
                            const void* beta, const void* w, const void* d_out, const float* bnd, const float* d_bnd,
                            void* dq, void* dk, void* dv, void* dg, void* dbeta, void* dw, int64_t H, int dtype,
                            int g_dtype, float scale, bool beside, cudaStream_t stream) {
  if (table.chunks == 0) return GDN2_OK;
  return run_vjp(table, SpanVjpParams{q, k, v, g, beta, w, d_out, bnd, d_bnd, dq, dk, dv, dg, dbeta, dw, int(H), scale},
                 dtype, g_dtype, stream, beside);
}

}  // namespace gdn2
