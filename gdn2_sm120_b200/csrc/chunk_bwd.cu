// Tensor-core chunk backward (64-token chunks), two kernels that consume the WY tiles and
// residuals saved by the forward and the fp32 chunk-start states.  The reverse scan reads the very
// tiles the forward scan read, through tiled TMA loads in the other swizzle: what the forward
// contracted over columns it contracts over rows (K-major <-> MN-major operands, tc05.cuh).
//
//   chunk_bwd_scan_kernel  one CTA per (batch, head) or part of its value rows, chunks in reverse order.  The
//                          state cotangent lives transposed (dS^T: value rows x key columns) in TMEM:
//                              dR^T  = dO^T Aqk + dS^T Kt^T        dZ^T = dR^T T
//                              dS^T <- dS^T diag(d) + dO^T Qg - dR^T Y
//                          It writes dZ = T^T dR per chunk and the cotangent at every chunk start.
//   chunk_bwd_vjp_kernel   persistent, one CTA per SM walking over the (batch, chunk, head) units,
//                          all chunks independent.  With R = T (Z - E S_0) as the parametrisation
//                          (no Y / U needed):
//                              dv = dZ w, dw = dZ v             (dZ = T^T dR comes from the scan)
//                              [-dE ; dQg] = [dZ ; dO] S_0^T    dKt = R dS_1^T
//                              [-dL ; dA]  = [dZ ; dO] R^T      (strictly lower / lower part)
//                          then the Gram products' VJP with the same 16-token block anchors as the
//                          forward, and a per-channel chain (one thread = one key channel) that
//                          forms dq, dk, dbeta and the reverse cumulative sum for dg.
//                          Its joint form does the work of both, where few sequences and heads scan.
// A ragged length ends in a partial chunk: tokens past T - 1 carry no cotangent and get no gradient.
//
// Reference counterparts: boundary scan  src/gdn2_sm120/backward_parallel.py:721-1049,
// compact-WY VJP  src/gdn2_sm120/backward_wy.py:226-1168 (a 10-12 launch graph there).

#include <cuda.h>

#include <type_traits>

#include "chunk_common.cuh"

namespace gdn2 {

using namespace tc;

namespace {

constexpr int64_t kStateElems = int64_t(kDim) * kDim;

// =============================================================================================
// reverse scan
// =============================================================================================
// Warp-specialised like the forward scan (chunk_fwd.cu), for the same reason: the MMAs of a chunk are issued
// back to back by one warp, the rest runs beside them.
//   warp 16      tiled TMA loads, each buffer refilled as soon as its MMA has read it
//   warp 18      MMAs, per chunk:  dR^T += dS^T Kt^T | dS'^T += dO^T Qg | dS'^T -= dR^T Y | dZ^T = dR^T T |
//                dR'^T = dO'^T Aqk of the next chunk, the dependences between accumulators waited for
//   warps 0..7   decay: dS' <- dS diag(d) into the other of two buffers; the cotangent checkpoints, staged
//   warps 8..15  dO of the next chunk (the one before it in time) into tensor memory, dZ out (staged)
// Tensor memory (columns): dS 2 x 128, dR 2 x 64, dZ 64, dO 64 = all 512.
// (With a half or a quarter of the value rows two or one warp of four has work; the loads and the MMAs then take the
// places of others, see ScanWarps in chunk_fwd.cu.)
template <int kParts>
struct BScanWarps {
  static constexpr int kDo0 = 8, kLoads = kParts > 1 ? 2 : 16, kMma = kParts > 1 ? 3 : 18, kMark = 6;
  static constexpr int kThreads = kParts > 1 ? 512 : 608;
  static __device__ __forceinline__ bool works(int warp) { return warp < 16 && (warp & 3) < 4 / kParts; }
};
constexpr int kCsZ = 144, kRsZ = 32 * kCsZ;  // dZ tile: the padded strides of the VJP kernel's [dZ ; dO] stack

struct BScanSmem {
  // swizzled operand tiles, slabs of 32 columns (tc05.cuh): Q is read MN-major, the others K-major
  alignas(1024) uint8_t kn[32768];   // Kn[j][k]: 4 slabs of 64 lines
  alignas(1024) uint8_t q[32768];    // Q[i][k]:  4 slabs of 64 lines
  alignas(1024) uint8_t yt[32768];   // Yt[k][j]: 2 slabs of 128 lines
  alignas(1024) uint8_t at[16384];   // At[j][i]: 2 slabs of 64 lines
  alignas(1024) uint8_t tt[16384];   // Tt[j][i]: 2 slabs of 64 lines
  alignas(128) uint8_t d_out[16384]; // raw dO of the chunk, [64][128] 16-bit rows
  alignas(128) uint8_t dz[kBlobDZ];  // dZ staging, natural tile X[r = j][c = v] with the padded strides
  alignas(128) float ck[2][32 * kDim];  // 32 rows of the cotangent per half of the decay group
  alignas(16) float d[2][kDim];
  alignas(8) uint64_t full_o, full_d[2];
  uint64_t go_a;      // At, dO written:               1 load + 8 warps
  uint64_t full_k, full_y;
  uint64_t go_q;      // Q, decayed cotangent:         1 load + 8 warps
  uint64_t go_z;      // Tt, dZ of the last step read: 1 load + 8 warps
  uint64_t do_read;   // dO is in registers:                                 8 warps
  uint64_t a_done, k_done, z_done, do_done, s_done;  // MMA commits
  volatile int failed;
  volatile int stored[4], sent;  // joint launch: steps whose cotangents (by warp) and dZ are in memory
  uint32_t tmem_base;
};
static_assert(sizeof(BScanSmem) <= 232448, "reverse scan exceeds the 227 KiB shared-memory limit");

// Joint launch: the last 16 bytes of a dZ tile, behind its last row, belong to nobody.  Word 0 counts the CTAs
// of the scan that have left in memory what the VJP reads of the unit; the first unit's word 1 is the queue of units.
constexpr int64_t kMarkOffset = kBlobDZ - 16;
struct Marks {
  uint8_t* dz;
  __device__ __forceinline__ unsigned* of(int64_t ch) const {
    return reinterpret_cast<unsigned*>(dz + ch * kBlobDZ + kMarkOffset);
  }
  __device__ __forceinline__ void arrive(int64_t ch) const {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(of(ch)) : "memory");
  }
};

struct BScanParams {
  const uint8_t* d;         // chunk-end decays, 512 bytes per unit
  uint8_t* dz;              // dZ tiles
  const float* ds_final;    // [sequences,H,128,128] or null
  float* d_bnd;             // cotangents at the chunk starts, one slot more than chunks per sequence
  float* ds_init;           // [sequences,H,128,128] or null
  int* status;
  int H;
  Marks marks;              // joint launch
};
struct BScanMaps {
  CUtensorMap at, tt, kn, q, yt, d_out;
};

// One sequence and head, or a part of its value rows (value_parts), by a whole CTA.  kJoint: the VJP of finished
// chunks runs beside in the same launch, and this CTA joins it afterwards.
template <typename T, typename Seqs, bool kJoint, int kParts>
__device__ __forceinline__ void reverse_sequence(const BScanParams& p, const Seqs& seqs, const BScanMaps& tm,
                                                 BScanSmem& sm, const int item) {
  BoundedWaiter waiter(p.status, 1u << 20, &sm.failed);

  using W = BScanWarps<kParts>;
  constexpr int kRows = kDim / kParts;  // value rows of this CTA: lanes 0 .. kRows - 1 of tensor memory
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int unit = item / kParts, v0 = (item - unit * kParts) * kRows;
  const int s = unit / p.H, h = unit - s * p.H;
  const SeqInfo sq = seqs.at(s);
  const int n_chunks = sq.n_chunks;
  constexpr uint32_t kColS = 0, kColR = 256, kColZ = 384, kColDo = 448;
  // step `it` of the reverse scan works on chunk n_chunks - 1 - it
  auto chunk_of = [&](int it) { return n_chunks - 1 - it; };
  auto ch_of = [&](int it) { return int64_t(sq.chunk0 + chunk_of(it)) * p.H + h; };

  if (warp == W::kMma) {
    tmem_alloc(&sm.tmem_base, 512);
    if (!kJoint) tmem_relinquish();
  }
  if (tid == 0) {
    uint64_t* one[] = {&sm.full_o, &sm.full_d[0], &sm.full_d[1], &sm.full_k, &sm.full_y, &sm.a_done, &sm.k_done,
                       &sm.z_done, &sm.do_done, &sm.s_done};
#pragma unroll
    for (int i = 0; i < 10; ++i) mbar_init(one[i], 1);
    mbar_init(&sm.go_a, 1 + 8 / kParts);
    mbar_init(&sm.go_q, 1 + 8 / kParts);
    mbar_init(&sm.go_z, 1 + 8 / kParts);
    mbar_init(&sm.do_read, 8 / kParts);
    for (int i = 0; i < 4; ++i) sm.stored[i] = 0;
    sm.sent = 0;
    // a wait that ran out earlier (forward or backward) left garbage behind: results become NaN
    sm.failed = *static_cast<volatile const int*>(p.status) != kStatusOk;
    fence_mbar_init();
  }
  // lines 32..63 of the first slab of At and Tt (j >= 32, i < 32) are never loaded: zero, once
  for (int e = tid; e < 4096 / 16; e += W::kThreads) {
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

  if (warp == W::kLoads) {
    // ---------------------------------------------------------------- loads
    const uint32_t leader = elect_leader();
    auto load_o = [&](int it) {
      mbar_arrive_expect_tx(&sm.full_o, 16384u / kParts, leader);
      tma_load_3d(sm.d_out, &tm.d_out, v0, h, int(sq.row0) + chunk_of(it) * kChunk, &sm.full_o, leader);
    };
    // At and Tt are zero for j >= 32, i < 32: three 32-row boxes each, the fourth quadrant stays zero
    auto load_tri = [&](uint8_t* dst, const CUtensorMap* map, int it, uint64_t* bar) {
      const int ch = int(ch_of(it));
      mbar_arrive_expect_tx(bar, uint32_t(kTileAt - 4096), leader);
      tma_load_4d(dst, map, 0, 0, 0, ch, bar, leader);
      tma_load_4d(dst + 8192, map, 0, 0, 1, ch, bar, leader);
      tma_load_4d(dst + 8192 + 4096, map, 0, 32, 1, ch, bar, leader);
    };
    auto load_tile = [&](uint8_t* dst, const CUtensorMap* map, int it, uint64_t* bar) {
      mbar_arrive_expect_tx(bar, 32768u, leader);
      tma_load_4d(dst, map, 0, 0, 0, int(ch_of(it)), bar, leader);
    };
    auto load_d = [&](int it) {
      mbar_arrive_expect_tx(&sm.full_d[it & 1], uint32_t(kBlobD), leader);
      bulk_g2s(sm.d[it & 1], p.d + ch_of(it) * kBlobD, uint32_t(kBlobD), &sm.full_d[it & 1], leader);
    };
    load_o(0);
    load_tri(sm.at, &tm.at, 0, &sm.go_a);
    load_tile(sm.kn, &tm.kn, 0, &sm.full_k);
    load_d(0);
    load_tile(sm.q, &tm.q, 0, &sm.go_q);
    load_tile(sm.yt, &tm.yt, 0, &sm.full_y);
    load_tri(sm.tt, &tm.tt, 0, &sm.go_z);
    if (n_chunks > 1) load_d(1);
    for (int it = 1; it < n_chunks; ++it) {
      const uint32_t par = uint32_t(it - 1) & 1u;
      waiter.wait(&sm.do_read, par);
      load_o(it);
      waiter.wait(&sm.a_done, par);
      load_tri(sm.at, &tm.at, it, &sm.go_a);
      waiter.wait(&sm.k_done, par);
      load_tile(sm.kn, &tm.kn, it, &sm.full_k);
      waiter.wait(&sm.do_done, par);
      load_tile(sm.q, &tm.q, it, &sm.go_q);
      waiter.wait(&sm.s_done, par);
      load_tile(sm.yt, &tm.yt, it, &sm.full_y);
      if (it + 1 < n_chunks) load_d(it + 1);  // the decay of step it - 1 has run: its slot is free
      waiter.wait(&sm.z_done, par);
      load_tri(sm.tt, &tm.tt, it, &sm.go_z);
    }
  } else if (warp == W::kMma) {
    // ---------------------------------------------------------------- MMAs
    // (the terminal cotangent must be in tensor memory: barrier 1, decay group and this warp)
    asm volatile("bar.sync 1, %0;" ::"n"(2 * kRows + 32) : "memory");
    tc_fence_after();
    const uint32_t leader = elect_leader();
    const uint32_t a0 = smem_u32(sm.at), kn0 = smem_u32(sm.kn), tt0 = smem_u32(sm.tt);
    const uint32_t q0 = smem_u32(sm.q), y0 = smem_u32(sm.yt);
    const uint32_t id64 = idesc(128, 64, kFmtTF32, kMajorK, kMajorK);
    const uint32_t id_pos = idesc(128, 128, kFmtTF32, kMajorK, kMajorMN);
    const uint32_t id_neg = idesc(128, 128, kFmtTF32, kMajorK, kMajorK, 1, 0);
    const uint32_t d_o = tb + kColDo, z = tb + kColZ;
    // dR^T = dO^T Aqk   (A: dO columns, K = 64 tokens; B: At[j][i] read K-major)
    auto issue_a = [&](int it) {
      const uint32_t r = tb + kColR + 64u * (uint32_t(it) & 1u);
      waiter.wait(&sm.go_a, uint32_t(it) & 1u);
      tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        mma_tf32_ts(r, d_o + ks * 8, smem_desc_sw128_k(a0, 8192, ks), id64, ks > 0 ? 1u : 0u, leader);
      }
      mma_commit(&sm.a_done, leader);
    };
    issue_a(0);
    for (int it = 0; it < n_chunks; ++it) {
      const uint32_t par = uint32_t(it) & 1u;
      const uint32_t s_old = tb + kColS + 128u * par, s_new = tb + kColS + 128u * (par ^ 1u);
      const uint32_t r = tb + kColR + 64u * par;
      // dR^T += dS^T Kt^T (A: cotangent columns, K = 128 keys; B: Kn[j][k] read K-major)
      waiter.wait(&sm.full_k, par);
      if (it > 0) waiter.wait(&sm.s_done, par ^ 1u);
      tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < 16; ++ks) {
        mma_tf32_ts(r, s_old + ks * 8, smem_desc_sw128_k(kn0, 8192, ks), id64, 1u, leader);
      }
      mma_commit(&sm.k_done, leader);
      // dS'^T += dO^T Qg  (K = 64 tokens; B: Q[i][k] read MN-major)
      waiter.wait(&sm.go_q, par);
      tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        mma_tf32_ts(s_new, d_o + ks * 8, smem_desc_sw128_mn(q0, 8192, ks), id_pos, 1u, leader);
      }
      mma_commit(&sm.do_done, leader);
      // dS'^T -= dR^T Y   (A: dR^T columns, K = 64 tokens; B: Yt[k][j] read K-major)
      waiter.wait(&sm.full_y, par);
      waiter.wait(&sm.k_done, par);
      tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        mma_tf32_ts(s_new, r + ks * 8, smem_desc_sw128_k(y0, 16384, ks), id_neg, 1u, leader);
      }
      mma_commit(&sm.s_done, leader);
      // dZ^T = dR^T T     (A: dR^T columns, K = 64 tokens; B: Tt[j][i] read K-major)
      waiter.wait(&sm.go_z, par);
      tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        mma_tf32_ts(z, r + ks * 8, smem_desc_sw128_k(tt0, 8192, ks), id64, ks > 0 ? 1u : 0u, leader);
      }
      mma_commit(&sm.z_done, leader);
      if (it + 1 < n_chunks) issue_a(it + 1);
    }
  } else if (kJoint && warp == W::kMark) {
    // ---------------------------------------------------------------- marks of finished units
    // a warp of its own: what a mark has to wait for would hold up the others for half of a chunk's time
    for (int it = 0; it < n_chunks; ++it) {
      const volatile int* mine = lane < 4 ? &sm.stored[lane] : &sm.sent;
      // (the other warps of the scan give up by themselves)
      for (uint32_t looks = 0; !__all_sync(0xffffffffu, *mine > it) && looks < (1u << 27); ++looks) __nanosleep(40);
      __threadfence_block();
      // (the VJP reads through the copy engine, another proxy than the stores)
      fence_async_all();
      __syncwarp();  // what each lane saw is ordered before lane 0's release (a vote orders no memory)
      if (lane == 0) p.marks.arrive(ch_of(it));
    }
  } else if (!W::works(warp)) {
    // (nothing to do in this form)
  } else if (warp < W::kDo0) {
    // ---------------------------------------------------------------- decay of the cotangent
    // thread = value row of the transposed cotangent (TMEM lane) x one half of the 128 key columns
    const int q4 = warp & 3, half = warp >> 2;
    const int vrow = 32 * q4 + lane, k0 = 64 * half;
    const int64_t my_row = v0 + vrow;
    const uint32_t lane_base = 32u * q4;
    const int64_t state = (int64_t(sq.sid) * p.H + h) * kStateElems;
    const bool sender = lane == 0 && q4 == 0;  // sends this half's staged rows
    uint32_t lo[32], hi[32];
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
    // 32 key rows of the cotangent at the end of chunk c, 16 KiB, through the staging buffer of this half
    auto send_rows = [&](const uint32_t (&x)[32], int c, int kr) {
      if (sender) bulk_wait_read_all();  // the previous rows have left the buffer
      half_barrier();
      float* dst = sm.ck[half] + vrow;
#pragma unroll
      for (int j = 0; j < 32; ++j) dst[j * kDim] = __uint_as_float(x[j]);
      fence_async_smem();
      half_barrier();
      if (sender) {
        bulk_s2g(p.d_bnd + ((int64_t(sq.slot0 + c + 1) * p.H + h) * kDim + kr) * kDim, sm.ck[half], 32u * kDim * 4u);
        bulk_commit();
      }
    };
    {
      const float* src = (p.ds_final != nullptr) ? p.ds_final + state + my_row : nullptr;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        lo[j] = (src != nullptr) ? __float_as_uint(src[(k0 + j) * kDim]) : 0u;
        hi[j] = (src != nullptr) ? __float_as_uint(src[(k0 + 32 + j) * kDim]) : 0u;
      }
      store_state(kColS);
      tc_fence_before();
      asm volatile("bar.sync 1, %0;" ::"n"(2 * kRows + 32) : "memory");
    }
    for (int it = 0; it < n_chunks; ++it) {
      const uint32_t par = uint32_t(it) & 1u;
      if (it > 0) {
        waiter.wait(&sm.s_done, par ^ 1u);
        tc_fence_after();
        load_state(kColS + 128u * par);
      }
      waiter.wait(&sm.full_d[par], uint32_t(it >> 1) & 1u);
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
      store_state(kColS + 128u * (par ^ 1u));
      arrive(&sm.go_q);
      // the cotangent at the end of this chunk, off the chain: it is still in its buffer, which this group
      // alone overwrites, one step later
      load_state(kColS + 128u * par);
      if (kParts == 1) {
        send_rows(lo, chunk_of(it), k0);
        send_rows(hi, chunk_of(it), k0 + 32);
      } else {  // (a part of a row is not contiguous: plain stores)
        float* ck = p.d_bnd + ((int64_t(sq.slot0 + chunk_of(it) + 1) * p.H + h) * kDim + k0) * kDim + my_row;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          ck[j * kDim] = __uint_as_float(lo[j]);
          ck[(32 + j) * kDim] = __uint_as_float(hi[j]);
        }
        if constexpr (kJoint) {
          __threadfence_block();
          __syncwarp();
          if (lane == 0) sm.stored[2 * half + q4] = it + 1;
        }
      }
    }
    // ---- cotangent of the initial state: slot 0 and d_initial_state ----------------------------------
    waiter.wait(&sm.s_done, uint32_t(n_chunks - 1) & 1u);
    tc_fence_after();
    load_state(kColS + 128u * (uint32_t(n_chunks) & 1u));
    float* slot = p.d_bnd + (int64_t(sq.slot0) * p.H + h) * kStateElems + my_row;
    float* init = (p.ds_init != nullptr) ? p.ds_init + state + my_row : nullptr;
    const bool failed = sm.failed != 0;
#pragma unroll
    for (int j = 0; j < 64; ++j) {
      const float x = failed ? poison_nan() : __uint_as_float(j < 32 ? lo[j & 31] : hi[j & 31]);
      slot[(k0 + j) * kDim] = x;
      if (init != nullptr) init[(k0 + j) * kDim] = x;
    }
    if (sender) bulk_wait_all();  // the last staged rows are in global memory before the CTA retires
  } else {
    // ---------------------------------------------------------------- dO in, dZ out
    // thread = value row (TMEM lane) x one half of the 64 tokens
    const int q4 = warp & 3, half = (warp - W::kDo0) >> 2;
    const int vrow = 32 * q4 + lane, i0 = 32 * half;
    const uint32_t lane_base = 32u * q4;
    const bool sender = lane == 0 && q4 == 0 && half == 0;
    auto group_barrier = [&] { asm volatile("bar.sync 4, %0;" ::"n"(2 * kRows) : "memory"); };
    const T* src = reinterpret_cast<const T*>(sm.d_out) + i0 * kRows + vrow;
    auto build_do = [&](int it) {
      waiter.wait(&sm.full_o, uint32_t(it) & 1u);
      uint32_t x[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) x[j] = __float_as_uint(to_float(src[j * kRows]));
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.do_read);
      const int n_valid = sq.len - chunk_of(it) * kChunk;
      if (n_valid < kChunk) {  // past the end of the sequence there is no cotangent
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = (i0 + j < n_valid) ? x[j] : 0u;
      }
      if (it > 0) {
        waiter.wait(&sm.do_done, uint32_t(it - 1) & 1u);
        tc_fence_after();
      }
      tmem_st32(tmem_addr(tb, lane_base, kColDo + i0), x);
      tmem_wait_st();
      arrive(&sm.go_a);
    };
    arrive(&sm.go_z);  // no earlier step holds up the first dZ
    build_do(0);
    uint8_t* col = sm.dz + ((v0 + vrow) >> 2) * kCsZ + (vrow & 3) * 4;
    for (int it = 0; it < n_chunks; ++it) {
      if (it + 1 < n_chunks) build_do(it + 1);
      waiter.wait(&sm.z_done, uint32_t(it) & 1u);
      tc_fence_after();
      uint32_t r[32];
      tmem_ld32(tmem_addr(tb, lane_base, kColZ + i0), r);
      tmem_wait_ld();
      if (it + 1 < n_chunks) arrive(&sm.go_z);
      // dZ out: 32 token columns of value row v into the staging tile X[r = j][c = v], one bulk store
      const bool failed = sm.failed != 0;
      if (sender) {
        if constexpr (kJoint) {
          bulk_wait_all();  // the previous tile is in memory, long since
          __threadfence_block();
          sm.sent = it;
        } else {
          bulk_wait_read_all();  // the previous tile has left the staging buffer
        }
      }
      group_barrier();
#pragma unroll
      for (int jj = 0; jj < 32; ++jj) {
        const int j = i0 + jj;
        *reinterpret_cast<float*>(col + (j >> 3) * kRsZ + (j & 7) * 16) =
            failed ? poison_nan() : to_tf32(__uint_as_float(r[jj]));
      }
      fence_async_smem();
      group_barrier();
      if (sender) {
        uint8_t* dst = p.dz + ch_of(it) * kBlobDZ;
        if (kParts == 1) {
          bulk_s2g(dst, sm.dz, uint32_t(kBlobDZ));
        } else {  // this CTA's columns of each group of eight rows
#pragma unroll
          for (int jg = 0; jg < 8; ++jg) {
            const int at = jg * kRsZ + (v0 >> 2) * kCsZ;
            bulk_s2g(dst + at, sm.dz + at, uint32_t(kRows / 4 * kCsZ - 16));
          }
        }
        bulk_commit();
      }
    }
    if (sender) {
      bulk_wait_all();  // the last dZ tile is in global memory before the CTA retires
      if constexpr (kJoint) {
        __threadfence_block();
        sm.sent = n_chunks;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == W::kMma) {
    tc_fence_after();
    tmem_dealloc(tb, 512);
  }
  if (kJoint && tid == 0) {  // other shared memory lies over these from here on
    for (uint64_t* bar = &sm.full_o; bar <= &sm.s_done; ++bar) mbar_inval(bar);
  }
}

template <typename T, typename Seqs, int kParts>
__global__ void __launch_bounds__(BScanWarps<kParts>::kThreads, 1)
chunk_bwd_scan_kernel(const BScanParams p, const __grid_constant__ Seqs seqs, const __grid_constant__ BScanMaps tm) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  reverse_sequence<T, Seqs, false, kParts>(p, seqs, tm, *reinterpret_cast<BScanSmem*>(smem_raw), int(blockIdx.x));
  if constexpr (std::is_same<Seqs, PackedSeqs>::value) outlast_others();  // the short sequences' reverse kernel
}


// =============================================================================================
// chunk VJP
// =============================================================================================
// 512 threads.  Elementwise phases: warp = 4-token group tg, lane = 4-channel group c4.  TMEM phases:
// warp & 3 = lane quadrant, warp >> 2 = share of the columns.
// Final chain: thread = (key channel, 16-token block).
constexpr int kVjpThreads = 512;
constexpr int kCsN = 144;              // natural 128-column tiles: padded chunk stride
constexpr int kRsN = 32 * kCsN;        // 4608
constexpr int kRsT = 2064;             // transposed 64-column tiles: padded row-group stride
constexpr int kCsS = 144;              // 64-column tiles written by scattered 4-byte stores
constexpr int kRsS = 16 * kCsS;        // 2304

// dynamic shared memory map (bytes).  Phase B = products with the states, phase C = Gram VJP.
constexpr int kOffStack = 0;                      // B: [dZ ; dO] X[r = 128][c = v], RS kRsN     73728 (dZ rows: bulk copy)
constexpr int kOffRn = kOffStack + 16 * kRsN;     // B: R[j][v], 4 swizzled slabs of 64 lines    32768
constexpr int kOffS0 = kOffRn + 32768;            // B: S_0[k][v], 4 swizzled slabs of 128 lines  65536
constexpr int kOffDs1 = kOffS0 + 65536;           // B: dS_1[k][64 v] half, 2 swizzled slabs      32768
static_assert(kOffS0 % 1024 == 0 && kOffDs1 % 1024 == 0, "swizzled tiles are 1024-byte aligned");
constexpr int kEndB = kOffDs1 + 32768;            // 204800
constexpr int kOffStack2 = 0;                     // C: [dL_I ; dA_I] for I = 0..3, X[r = 128][c = j], RS 2048   32768
constexpr int kOffDLt = 32768;                    // C: dL^T X[r = j][c = i], RS kRsS            18432
constexpr int kOffDAt = kOffDLt + 8 * kRsS;       // C: dA^T                                     18432
constexpr int kOffKIt = kOffDAt + 8 * kRsS;       // C: (K^I)^T X[r = k][c = j < 16 (I+1)], RS 512 (I+1) + 16
constexpr int kKItBytes = 16 * (528 + 1040 + 1552 + 2064);  // 82944
constexpr int kOffEat = kOffKIt + kKItBytes;      // C: E_a^T X[r = k][c = i], RS kRsT           33024
constexpr int kOffQat = kOffEat + 16 * kRsT;      // C: Q_a^T                                    33024
constexpr int kEndC = kOffQat + 16 * kRsT;        // 218624
// final chain: k and q of the unit as 16-bit [64][128] tiles over the dO rows of the stack (dk and dq
// replace them in place and leave by tiled TMA stores), the log-decay prefix G as an fp32 tile over
// the dS_1 buffer.  The next unit's prefetch keeps clear of both until the chain is over.
constexpr int kOffTileK = kOffStack + 8 * kRsN;   // 36864
constexpr int kOffTileQ = kOffTileK + 16384;
constexpr int kOffTileG = kOffDs1;
// beta (dbeta in place) has no 16 KiB hole left: its 16-token blocks 0..2 sit behind the dS_1 buffer,
// block 3 in the last 4 KiB of the dO rows; a chain thread works on one block, so it sees one base
constexpr int kOffTileB012 = kEndB;               // 204800, 12 KiB
constexpr int kOffTileB3 = kOffTileQ + 16384;     // 69632, 4 KiB
static_assert(kOffTileB3 + 4096 <= kOffRn, "chain tiles exceed the dO rows of the stack");
static_assert(kOffTileB012 + 12288 <= kEndC, "beta tile exceeds the free space behind the dS_1 buffer");
__device__ __forceinline__ int beta_tile_offset(int blk) { return blk < 3 ? kOffTileB012 + blk * 4096 : kOffTileB3; }
constexpr int kOffMisc = (kEndB > kEndC ? kEndB : kEndC);
struct VjpMisc {
  float part[16][kDim];   // exclusive prefixes of the log-decay per 4-token group
  float gend[kDim];
  float xe[4][kDim];      // per-block sum_j Kt_j dKt_j
  float xt[4][kDim];      // partial sums of dd = sum_v dS_1 * S_0, then the per-block sums of dG
  alignas(8) uint64_t bar_a, bar_s, bar_r, bar_m, bar_d;
  uint32_t tmem_base;
  int next[2], ready[2];  // joint launch: the unit after this one, and whether the scan is done with it (two slots:
                          // one may still be read)
  int failed;             // joint launch: a wait of the scan ran out, or the wait for it
};
constexpr int kVjpSmemBytes = kOffMisc + int(sizeof(VjpMisc));
static_assert(kVjpSmemBytes <= 232448, "VJP kernel exceeds the 227 KiB shared-memory limit");

__device__ __forceinline__ int kit_rs(int I) { return 512 * (I + 1) + 16; }
__device__ __forceinline__ int kit_offset(int I) {
  return kOffKIt + 16 * ((I == 0) ? 0 : (I == 1) ? 528 : (I == 2) ? (528 + 1040) : (528 + 1040 + 1552));
}
__device__ __forceinline__ uint32_t d6_col(int I) { return (I == 3) ? 0u : (I == 2) ? 64u : (I == 1) ? 448u : 480u; }

struct VjpParams {
  const void *q, *k, *v, *g, *beta, *w, *d_out;
  const uint8_t* sc;    // scratch: dZ written by the reverse scan
  void *dq, *dk, *dv, *dg, *dbeta, *dw;
  int* status;
  int64_t n_ch;
  int H;
  float scale;
};
// tensor maps of the seven sequence tensors the VJP kernel reads (for L2 prefetches only)
struct VjpInputMaps {
  CUtensorMap q, k, v, g, beta, w, d_out;
};

template <typename T>
__device__ __forceinline__ void load4v(const void* base, int64_t idx, float (&out)[4]) {
  unpack4<T>(load4_raw<T>(base, idx), out);
}

template <typename T>
__device__ __forceinline__ void store4v(void* base, int64_t idx, float a, float b, float c, float d);
template <>
__device__ __forceinline__ void store4v<__nv_bfloat16>(void* base, int64_t idx, float a, float b, float c, float d) {
  *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(base) + idx) = make_uint2(pack_bf16(a, b), pack_bf16(c, d));
}
template <>
__device__ __forceinline__ void store4v<float>(void* base, int64_t idx, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(static_cast<float*>(base) + idx) = make_float4(a, b, c, d);
}
template <>
__device__ __forceinline__ void store4v<__half>(void* base, int64_t idx, float a, float b, float c, float d) {
  const __half2 lo = __floats2half2_rn(a, b), hi = __floats2half2_rn(c, d);
  *reinterpret_cast<uint2*>(static_cast<__half*>(base) + idx) =
      make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

__device__ __forceinline__ float2 tf32_2(float2 x) { return make_float2(to_tf32(x.x), to_tf32(x.y)); }

// The value of k times its anchored decay, `decay` alone or `decay * far` for row blocks beyond the next one:
// the chain calls this with the factors of the tile build, so that it multiplies the Gram cotangents by
// exactly the operand values the tensor cores saw.
__device__ __forceinline__ float2 anchored_k(float2 k, float2 decay, float2 far, bool use_far) {
  return mul2(k, use_far ? mul2(decay, far) : decay);
}

__device__ __forceinline__ void tmem_ld4x2(uint32_t taddr, float2 (&x)[4]) {
  uint32_t r[8];
  tmem_ld8(taddr, r);
  tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}

// kF32Grads: dq, dk, dv, dbeta, dw leave as fp32 instead of the sequence dtype (the values before
// their final rounding; used by tests to judge the arithmetic apart from the 16-bit cast).
// kRagged: some sequence length is not a multiple of 64, its last chunk is partial; only this
// instantiation carries the guards (they cost the others 6 %; a packed step of H16, 8192 tokens 1 %).
// kJoint: the reverse scans run in the same launch (below).  Units come from a queue in the order in which the scans
// finish them, and what the scans write of a unit is loaded once their marks are there.  The plain form carries none
// of that, and the body is the kernel's own: bound by instruction issue and short of registers, the plain kernel
// depends on how the compiler places what is nobody's business here.  As a function that both kernels called, with
// the next unit kept in a register and the flag of a failed scan in the plain form's condition as a constant, B4 T8192
// H32 took 1615 us; without these three 1585.
struct VjpMaps {
  CUtensorMap s0, ds, rn, dq, dk, dbeta;
  VjpInputMaps in;
};

// Reverse scan and VJP in one launch.  With few sequences and heads the reverse scan keeps a few SMs busy, 1.9-2.2 us
// per chunk, and the VJP of a chunk needs nothing but that chunk's share of it.  Here the scans run on pairs of CTAs (a
// half of the value rows each) and all other CTAs, and at last these too, take the units from a queue, last chunks
// first, waiting for the scans' marks.  The scans wait for nobody; the launch is cooperative, so that all CTAs are
// resident together: it begins when every SM is free.  (Pairs that draw scans from a queue, and need no others beside
// them, can begin on the SMs that are free; every step took 10-12 us more, B1 T2048 H16 207 -> 218, H32 T8192 1046 ->
// 1059.)  A unit's scratch tiles and cotangents are still in L2 when the VJP reads them.  Whatever waits for memory on
// behalf of a mark is kept off the scan's chain and the VJP's: by the scanning warps themselves it cost a chunk 1.2 us,
// by the thread that issues the VJP's copies a unit 1500 clocks.
constexpr int kJointParts = 2;
template <bool kJoint>
struct JointScan {
  BScanParams p;
  BScanMaps tm;
};
template <>
struct JointScan<false> {};

// The queue of units of a joint launch, and the marks of those that the scans have finished.
template <typename Seqs>
struct JointUnits {
  const VjpParams& p;
  const Seqs& seqs;
  const Marks marks;
  VjpMisc& ms;
  // the next unit of the queue, last chunks first
  __device__ __forceinline__ int pop() const {
    const unsigned u = atomicAdd(marks.of(0) + 1, 1u);
    if (u >= unsigned(p.n_ch)) return int(p.n_ch);
    const unsigned per_chunk = unsigned(seqs.count()) * unsigned(p.H), step = u / per_chunk, r = u - step * per_chunk;
    const SeqInfo sq = seqs.at(int(r / unsigned(p.H)));
    return (sq.chunk0 + sq.n_chunks - 1 - int(step)) * p.H + int(r % unsigned(p.H));
  }
  // have the scans finished a unit: a look, or a wait
  __device__ __forceinline__ bool finished(int64_t ch) const {
    unsigned x;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(marks.of(ch)) : "memory");
    if (x != unsigned(kJointParts)) return false;
    fence_async_all();
    // (a wait of the scan that ran out: gradients become NaN)
    if (*static_cast<volatile const int*>(p.status) != kStatusOk) ms.failed = 1;
    return true;
  }
  __device__ __forceinline__ void await(int64_t ch, BoundedWaiter& waiter) const {
    waiter.look_anew();
    while (!finished(ch)) {
      if (!waiter.look_again()) {
        ms.failed = 1;
        break;
      }
      __nanosleep(100);
    }
  }
};

template <typename T, typename G, typename Seqs, bool kF32Grads, bool kRagged, bool kJoint>
__global__ void __launch_bounds__(kVjpThreads, 1)
chunk_bwd_vjp_kernel(const VjpParams p, const __grid_constant__ Seqs seqs, const __grid_constant__ VjpMaps tm,
                     const __grid_constant__ JointScan<kJoint> scan) {
  using O = typename std::conditional<kF32Grads, float, T>::type;  // element type of dq, dk, dv, dbeta, dw
  extern __shared__ __align__(1024) uint8_t smem[];
  if constexpr (std::is_same<Seqs, PackedSeqs>::value) let_others_begin();  // the short sequences' VJP
  if constexpr (kJoint) {
    static_assert(BScanWarps<kJointParts>::kThreads == kVjpThreads, "a scanning CTA goes on with the VJP");
    if (int(blockIdx.x) < kJointParts * seqs.count() * p.H) {
      reverse_sequence<T, Seqs, true, kJointParts>(scan.p, seqs, scan.tm, *reinterpret_cast<BScanSmem*>(smem),
                                                   int(blockIdx.x));
      fence_async_smem();
      __syncthreads();
    }
  }
  const CUtensorMap &tm_s0 = tm.s0, &tm_ds = tm.ds, &tm_rn = tm.rn, &tm_dq = tm.dq, &tm_dk = tm.dk, &tm_dbeta = tm.dbeta;
  const VjpInputMaps& tm_in = tm.in;
  VjpMisc& ms = *reinterpret_cast<VjpMisc*>(smem + kOffMisc);
  const ScratchLayout sc{p.n_ch};
  BoundedWaiter waiter(p.status);
  // a wait that ran out earlier (forward or reverse scan) left garbage behind: gradients become NaN
  const bool upstream_failed = *static_cast<volatile const int*>(p.status) != kStatusOk;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q4 = warp & 3, part = warp >> 2;
  const int tg = warp, c4 = lane, kc0 = 4 * lane;

  if (warp == 0) {
    tmem_alloc(&ms.tmem_base, 512);
    tmem_relinquish();
  }
  if (tid == 0) {
    mbar_init(&ms.bar_a, 1);
    mbar_init(&ms.bar_r, 1);
    mbar_init(&ms.bar_m, 1);
    mbar_init(&ms.bar_d, 1);
    mbar_init(&ms.bar_s, 1);
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tb = ms.tmem_base;
  const uint32_t leader = elect_leader();
  uint32_t mma_phase = 0;
  constexpr uint32_t kColD2 = 64, kColD3 = 128, kColD4 = 256, kColD5 = 320;

  // Everything the first MMA batch of a chunk-head reads arrives asynchronously: the dZ rows of the
  // stack and the residual R as 1-D bulk copies, S_0 and the first 64 value columns of dS_1 as tiled TMA
  // loads (128-byte swizzle) that put the row-major fp32 checkpoints into shared memory as K-major
  // operands, 32 value columns per slab (the tensor cores read the fp32 containers as tf32).  No
  // register staging.  The kernel is persistent: one SM takes in bytes at a limited rate, so the copies
  // for the CTA's next chunk-head are issued as soon as the last MMA of the current one has read shared
  // memory, and land during its final chain.
  // The chain keeps the dO rows of the stack and the dS_1 buffer for its own tiles, so the copies come in
  // two parts: S_0, R and dZ before the chain, the dS_1 half after it (bar_s expects both from the start).
  // unit -> head, first token row, tokens that exist, checkpoint slot of the chunk start
  // (all 31-bit numbers, the launcher checks: 32-bit divisions, a fraction of the 64-bit routine)
  struct Place { int h, row, valid, slot; };
  auto locate = [&](int64_t ch_) {
    const int chunk = int(uint32_t(ch_) / uint32_t(p.H));
    const SeqInfo sq = seqs.at(seqs.find(chunk));
    const int c_ = chunk - sq.chunk0, h_ = int(ch_) - chunk * p.H;
    return Place{h_, int(sq.row0) + c_ * kChunk, min(kChunk, sq.len - c_ * kChunk), (sq.slot0 + c_) * p.H + h_};
  };
  auto issue_loads = [&](int64_t ch_, int slot_) {
    mbar_arrive_expect_tx(&ms.bar_s, uint32_t(65536 + 32768));
    tma_load_4d(smem + kOffS0, &tm_s0, 0, 0, 0, slot_, &ms.bar_s);
    mbar_arrive_expect_tx(&ms.bar_a, uint32_t(kBlobDZ + kBlobRn));
    tma_load_4d(smem + kOffRn, &tm_rn, 0, 0, 0, int(ch_), &ms.bar_a);
    if constexpr (!kJoint) bulk_g2s(smem + kOffStack, p.sc + sc.off_dz() + ch_ * kBlobDZ, uint32_t(kBlobDZ), &ms.bar_a);
  };
  auto issue_ds1 = [&](int slot_) {
    tma_load_4d(smem + kOffDs1, &tm_ds, 0, 0, 0, slot_ + p.H, &ms.bar_s);
  };
  int64_t first = blockIdx.x, joint_next = 0;
  if constexpr (kJoint) {
    if (tid == 0) {
      ms.failed = 0;
      ms.next[0] = JointUnits<Seqs>{p, seqs, scan.p.marks, ms}.pop();
    }
    __syncthreads();
    first = ms.next[0];
    __syncthreads();
  }
  if (tid == 0 && first < p.n_ch) {
    const int slot_ = locate(first).slot;
    issue_loads(first, slot_);
    if constexpr (kJoint) {
      JointUnits<Seqs>{p, seqs, scan.p.marks, ms}.await(first, waiter);
      bulk_g2s(smem + kOffStack, p.sc + sc.off_dz() + first * kBlobDZ, uint32_t(kBlobDZ), &ms.bar_a);
    }
    issue_ds1(slot_);
  }

  uint32_t iter = 0;
  for (int64_t ch = first; ch < p.n_ch; ch = kJoint ? joint_next : ch + gridDim.x, ++iter) {
  const uint32_t par = iter & 1u;
  [[maybe_unused]] int popped = 0;
  if constexpr (kJoint) {
    if (tid == 96) popped = JointUnits<Seqs>{p, seqs, scan.p.marks, ms}.pop();
  }
  const Place at = locate(ch);
  const int h = at.h;
  auto seq_idx = [&](int tok) { return (int64_t(at.row + tok) * p.H + h) * int64_t(kDim); };
  // tokens of this chunk that exist: 64 except in the last chunk of a sequence, whose missing tokens read
  // as zeros (the identity step) and whose gradients are not stored
  const int n_valid = kRagged ? at.valid : kChunk;
  auto there = [&](int tok) { return !kRagged || tok < n_valid; };            // does token `tok` of the chunk exist
  auto clamped = [&](int tok) { return kRagged ? min(tok, n_valid - 1) : tok; };  // a token that does
  const int ds1_slot = at.slot + p.H;
  // dd[k] += sum over the 64 value columns of half `hf` of dS_1[k][v] S_0[k][v], both read from their
  // shared-memory tiles.  The two tiles are swizzled alike (a line = 32 values of one key row, its
  // 16-byte pieces permuted by the row), so equal positions hold equal (k, v) and the order inside a
  // line does not matter for the sum.  Piece qd = tid + 512 x: line (qd >> 3) = slab * 128 + k, piece qd & 7.
  auto dd_half = [&](int hf) {
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int qd = tid + 512 * x;
      const int line = qd >> 3, slab = line >> 7, kr = line & 127;
      const float4 ds = *reinterpret_cast<const float4*>(smem + kOffDs1 + slab * 16384 + kr * 128 + (qd & 7) * 16);
      const float4 s0 = *reinterpret_cast<const float4*>(smem + kOffS0 + (2 * hf + slab) * 16384 + kr * 128 + (qd & 7) * 16);
      float acc = ds.x * s0.x + ds.y * s0.y + ds.z * s0.z + ds.w * s0.w;
      // the 8 lanes of a line
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      acc += __shfl_xor_sync(0xffffffffu, acc, 4);
      // one owner per (half, slab, key row): partial sums in fixed slots, no atomics, so that the result
      // does not depend on the timing of the warps (xt is free until the end of the chain)
      if ((lane & 7) == 0) ms.xt[2 * hf + slab][kr] = acc;
    }
  };

  // ---- phase A: dO rows of the stack (rows 64 + i), natural tile with padded chunk stride, and the
  // log-decay sums of this thread's tokens
  float Gc[4][4];
  {
    float dv4[4][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      // a token past the end of a ragged sequence: the last real token is read instead (no branch around
      // the loads, they are all issued back to back) and its value dropped below
      const int64_t idx = seq_idx(clamped(4 * tg + e)) + kc0;
      load4v<T>(p.d_out, idx, dv4[e]);
      load4v<G>(p.g, idx, Gc[e]);
    }
    if (kRagged && n_valid < kChunk) {  // CTA-uniform; false for every chunk but the last one of a sequence
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (!there(4 * tg + e)) {
#pragma unroll
          for (int f = 0; f < 4; ++f) dv4[e][f] = Gc[e][f] = 0.f;
        }
      }
    }
    if (!kF32Grads) {
      // the dk / dq tiles of the previous unit lie where the dO rows go: their stores must have read them
      if (tid == 0) bulk_wait_read_all();
      __syncthreads();
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = 4 * tg + e;
      *reinterpret_cast<float4*>(smem + kOffStack + ((64 + i) >> 3) * kRsN + c4 * kCsN + (i & 7) * 16) =
          make_float4(dv4[e][0], dv4[e][1], dv4[e][2], dv4[e][3]);
      // (log-decays in units of ln 2: a decay is one ex2)
#pragma unroll
      for (int f = 0; f < 4; ++f) Gc[e][f] = e > 0 ? fmaf(Gc[e][f], kLog2e, Gc[e - 1][f]) : Gc[e][f] * kLog2e;
    }
  }
  *reinterpret_cast<float4*>(&ms.part[tg][kc0]) = make_float4(Gc[3][0], Gc[3][1], Gc[3][2], Gc[3][3]);
  if constexpr (kJoint) {
    if (tid == 96) ms.next[par] = popped;
  }
  waiter.wait(&ms.bar_a, par);
  waiter.wait(&ms.bar_s, par);
  dd_half(0);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  if constexpr (kJoint) joint_next = ms.next[par];
  // ---- first MMA batch: M4 (first half) dKt^T = dS_1[:, v < 64] R[:, v < 64]^T ;
  //      M2 [-dL ; dA] = [dZ ; dO] R^T ;  M3 [-dE ; dQg]^T = S_0 [dZ ; dO]^T ------------------------------
  if (warp == 0) {
    tc_fence_after();
    const uint32_t st = smem_u32(smem + kOffStack), rn = smem_u32(smem + kOffRn);
    const uint32_t s0 = smem_u32(smem + kOffS0), d1 = smem_u32(smem + kOffDs1);
    const uint32_t id64 = idesc(128, 64, kFmtTF32, kMajorK, kMajorK);
    const uint32_t id128 = idesc(128, 128, kFmtTF32, kMajorK, kMajorK);
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      mma_tf32_ss(tb + kColD4, smem_desc_sw128_k(d1, 16384, ks), smem_desc_sw128_k(rn, 8192, ks), id64,
                  ks > 0 ? 1u : 0u, leader);
    }
    mma_commit(&ms.bar_r, leader);  // the dS_1 buffer may be refilled once these have run
#pragma unroll
    for (int ks = 0; ks < 16; ++ks) {
      mma_tf32_ss(tb + kColD2, smem_desc(st, kCsN, kRsN, ks * 2 * kCsN), smem_desc_sw128_k(rn, 8192, ks), id64,
                  ks > 0 ? 1u : 0u, leader);
    }
#pragma unroll
    for (int ks = 0; ks < 16; ++ks) {
      mma_tf32_ss(tb + kColD3, smem_desc_sw128_k(s0, 16384, ks), smem_desc(st, kCsN, kRsN, ks * 2 * kCsN), id128,
                  ks > 0 ? 1u : 0u, leader);
    }
    mma_commit(&ms.bar_m, leader);
    // the second 64 value columns of dS_1 replace the first as soon as their product has run
    waiter.wait(&ms.bar_r, 0);
    mbar_arrive_expect_tx(&ms.bar_d, 32768u, leader);
    tma_load_4d(smem + kOffDs1, &tm_ds, 0, 0, 2, ds1_slot, &ms.bar_d, leader);
  }
  // ---- under the tensor cores: log-decay prefixes, dv = dZ w, dw = dZ v, and the raw inputs of the
  // Gram operands.  Every load is issued before the first store: the outputs may alias the inputs as
  // far as the compiler knows, so a load placed after a store would wait for its round trip.
  if (tid < kDim) {
    float x[16], run = 0.f;  // (all read before the first is written: the reads wait together)
#pragma unroll
    for (int t = 0; t < 16; ++t) x[t] = ms.part[t][tid];
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      ms.part[t][tid] = run;
      run += x[t];
    }
    ms.gend[tid] = run;
  }
  const int mb = tg >> 2;
  float kk[4][4], qq[4][4], bb[4][4];
  {
    typename Raw4<T>::type wr[4], vr[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int64_t idx = seq_idx(clamped(4 * tg + e)) + kc0;  // see phase A
      wr[e] = load4_raw<T>(p.w, idx);
      vr[e] = load4_raw<T>(p.v, idx);
      load4v<T>(p.k, idx, kk[e]);
      load4v<T>(p.q, idx, qq[e]);
      load4v<T>(p.beta, idx, bb[e]);
    }
    if (kRagged && n_valid < kChunk) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (!there(4 * tg + e)) {
#pragma unroll
          for (int f = 0; f < 4; ++f) kk[e][f] = qq[e][f] = bb[e][f] = 0.f;
        }
      }
    }
    // (the ragged instantiation has the one, predicated copy of these stores: a second, unpredicated copy
    // for the warps whose tokens all exist made it slower, that kernel is close to the size of the
    // instruction cache)
    auto store_dv_dw = [&](auto guarded) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = 4 * tg + e;
        float4 dz = *reinterpret_cast<const float4*>(smem + kOffStack + (j >> 3) * kRsN + c4 * kCsN + (j & 7) * 16);
        if (upstream_failed || waiter.dead) dz = make_float4(poison_nan(), poison_nan(), poison_nan(), poison_nan());
        if constexpr (kJoint) {
          if (ms.failed != 0) dz = make_float4(poison_nan(), poison_nan(), poison_nan(), poison_nan());
        }
        const int64_t idx = seq_idx(j) + kc0;
        float wv[4], vv[4];
        unpack4<T>(wr[e], wv);
        unpack4<T>(vr[e], vv);
        if (!decltype(guarded)::value || j < n_valid) {
          store4v<O>(p.dv, idx, dz.x * wv[0], dz.y * wv[1], dz.z * wv[2], dz.w * wv[3]);
          store4v<O>(p.dw, idx, dz.x * vv[0], dz.y * vv[1], dz.z * vv[2], dz.w * vv[3]);
        }
      }
    };
    if (!kRagged) store_dv_dw(std::false_type{});
    else store_dv_dw(std::true_type{});
  }
  // The sequence tensors of the next chunk-head are read with per-thread loads, whose rate is set by the
  // bytes in flight over the latency: have its seven [64][128] tiles brought into L2, the four that are read
  // first from here on and the others with the tile copies.  (All behind the tile copies they wait for those
  // in the copy engine: B4 T8192 H32 1.72 ms against 1.63; all from here, ragged lengths lose 2 %.)
  if (tid == 64 && (kJoint ? joint_next : ch + gridDim.x) < p.n_ch) {
    const Place nx = locate(kJoint ? joint_next : ch + gridDim.x);
    tma_prefetch_l2_3d(&tm_in.d_out, 0, nx.h, nx.row);
    tma_prefetch_l2_3d(&tm_in.g, 0, nx.h, nx.row);
    tma_prefetch_l2_3d(&tm_in.w, 0, nx.h, nx.row);
    tma_prefetch_l2_3d(&tm_in.v, 0, nx.h, nx.row);
  }
  // (where all wait for the tensor cores anyway: a look takes 1500 clocks)
  if constexpr (kJoint) {
    if (tid == 96) {
      ms.ready[par] = joint_next < p.n_ch && JointUnits<Seqs>{p, seqs, scan.p.marks, ms}.finished(joint_next);
    }
  }
  // ---- M4 (second half) once the second half of dS_1 has landed -----------------------------------------
  waiter.wait(&ms.bar_d, par);
  dd_half(1);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    const uint32_t rn = smem_u32(smem + kOffRn), d1 = smem_u32(smem + kOffDs1);
    const uint32_t id64 = idesc(128, 64, kFmtTF32, kMajorK, kMajorK);
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      mma_tf32_ss(tb + kColD4, smem_desc_sw128_k(d1, 16384, ks), smem_desc_sw128_k(rn, 8192, 8 + ks), id64, 1u, leader);
    }
    mma_commit(&ms.bar_r, leader);
  }
  waiter.wait(&ms.bar_m, mma_phase & 1u);
  ++mma_phase;
  tc_fence_after();

  // ================================ phase C: Gram VJP =============================================
  // [-dL_raw ; dA_raw] out of TMEM: masked tiles [dL ; dA] (rows) and their transposes; the four
  // warps of a quadrant take 16 columns each.  These tiles lie over the [dZ ; dO] stack, whose last
  // readers (the first MMA batch and the dv / dw pass) are done; R and the dS_1 buffer may still be
  // read by the second half of M4 and are not touched before the wait further down.
  {
    const int r = 32 * q4 + lane, i = r & 63;
    // row of the stacked tile: the dL and dA rows of a 16-token block sit next to each other, so that
    // one N = 32 instruction multiplies both by (K^I)^T
    const int row2 = 32 * (i >> 4) + ((r < 64) ? 0 : 16) + (i & 15);
    uint8_t* tr_base = smem + ((r < 64) ? kOffDLt : kOffDAt);
    const int c0 = 16 * part;
    uint32_t raw[16];
    tmem_ld16(tmem_addr(tb, 32 * q4, kColD2 + c0), raw);
    tmem_wait_ld();
    float vals[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int col = c0 + j;
      const float x = __uint_as_float(raw[j]);
      vals[j] = to_tf32_operand((r < 64) ? ((col < i) ? -x : 0.f) : ((col <= i) ? x : 0.f));
      *reinterpret_cast<float*>(tr_base + (col >> 3) * kRsS + (i >> 2) * kCsS + (col & 7) * 16 + (i & 3) * 4) = vals[j];
    }
#pragma unroll
    for (int j4 = 0; j4 < 4; ++j4) {
      *reinterpret_cast<float4*>(smem + kOffStack2 + blk_off<4>(row2, c0 + 4 * j4, 2048, 128)) =
          make_float4(vals[4 * j4], vals[4 * j4 + 1], vals[4 * j4 + 2], vals[4 * j4 + 3]);
    }
  }
  // anchored Gram operands, transposed tiles X[r = channel][c = token] with padded row-group stride.
  // They overwrite R and the dS_1 buffer: the second half of M4 must have run.
  waiter.wait(&ms.bar_r, 1);
  tc_fence_after();
  {
    auto row4 = [&](const float* row, float (&x)[4]) {
      const float4 y = *reinterpret_cast<const float4*>(row + kc0);
      x[0] = y.x; x[1] = y.y; x[2] = y.z; x[3] = y.w;
    };
    float base[4], a_blk[4][4], end[4];
    row4(ms.part[tg], base);
#pragma unroll
    for (int I = 0; I < 4; ++I) row4(ms.part[4 * I], a_blk[I]);
    row4(ms.gend, end);
    // Ea, Qa: anchored at the start of the token's own block.  (K^I)^T for every row block I >= the own block
    // mb, two exponentials per element in all:
    //   I = mb      k exp(a_mb - G)                      (own block: >= 1, bounded by the 16-token contract)
    //   I = mb + 1  k exp(a_next - G)                    (a_next = start of the next block)
    //   I > mb + 1  k (exp(a_next - G) exp(a_I - a_next))
    // The final chain forms the same products with the same expressions (anchored_k above).
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const int kc = kc0 + f;
      const float a_mb = mb == 0 ? a_blk[0][f] : mb == 1 ? a_blk[1][f] : mb == 2 ? a_blk[2][f] : a_blk[3][f];
      const float a_nx = mb == 0 ? a_blk[1][f] : mb == 1 ? a_blk[2][f] : mb == 2 ? a_blk[3][f] : end[f];
      const float c_nx = exp2_approx(a_nx - a_mb);  // decay over the whole 16-token block
      float2 k2[2], own[2], nb[2], ea[2], qa[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const float2 G = add2(make_float2(Gc[2 * x][f], Gc[2 * x + 1][f]), twice(base[f]));
        Gc[2 * x][f] = G.x;
        Gc[2 * x + 1][f] = G.y;
        const float2 to_anchor = minus2(twice(a_mb), G);
        const float2 anchored = exp2_2(make_float2(-to_anchor.x, -to_anchor.y));
        k2[x] = make_float2(kk[2 * x][f], kk[2 * x + 1][f]);
        ea[x] = tf32_operand_2(mul2(mul2(make_float2(bb[2 * x][f], bb[2 * x + 1][f]), k2[x]), anchored));
        qa[x] = tf32_operand_2(mul2(mul2(twice(p.scale), make_float2(qq[2 * x][f], qq[2 * x + 1][f])), anchored));
        own[x] = exp2_2(to_anchor);
        nb[x] = mul2(own[x], twice(c_nx));           // exp(a_nx - G): the chain forms it the same way
      }
      const uint32_t off = blk_off<4>(kc, 4 * tg, kRsT, 128);
      *reinterpret_cast<float4*>(smem + kOffEat + off) = make_float4(ea[0].x, ea[0].y, ea[1].x, ea[1].y);
      *reinterpret_cast<float4*>(smem + kOffQat + off) = make_float4(qa[0].x, qa[0].y, qa[1].x, qa[1].y);
#pragma unroll
      for (int I = 0; I < 4; ++I) {
        if (I >= mb) {
          const float far = (I > mb + 1) ? exp2_approx(a_blk[I][f] - a_nx) : 1.f;
          float2 val[2];
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            val[x] = tf32_operand_2(anchored_k(k2[x], (I == mb) ? own[x] : nb[x], twice(far), I > mb + 1));
          }
          *reinterpret_cast<float4*>(smem + kit_offset(I) + blk_off<4>(kc, 4 * tg, kit_rs(I), 128)) =
              make_float4(val[0].x, val[0].y, val[1].x, val[1].y);
        }
      }
    }
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    const uint32_t s2 = smem_u32(smem + kOffStack2);
    const uint32_t dlt = smem_u32(smem + kOffDLt), dat = smem_u32(smem + kOffDAt);
    const uint32_t eat0 = smem_u32(smem + kOffEat), qat0 = smem_u32(smem + kOffQat);
    const uint32_t id32 = idesc(128, 32, kFmtTF32, kMajorK, kMajorK);
    // [dEa_I^T | dQa_I^T] (columns 32 I .. 32 I + 31) = (K^I)^T x the 32 stacked rows [dL_I ; dA_I]
#pragma unroll
    for (int I = 0; I < 4; ++I) {
#pragma unroll
      for (int ks = 0; ks < 2 * (I + 1); ++ks) {
        mma_tf32_ss(tb + kColD5 + 32 * I, smem_desc(smem_u32(smem), 128, kit_rs(I), kit_offset(I) + ks * 256),
                    smem_desc(s2, 128, 2048, 4 * I * 2048 + ks * 256), id32, ks > 0 ? 1u : 0u, leader);
      }
    }
    // (dK^I)^T = Ea^T[:, block I] dL[block I, :] + Qa^T[:, block I] dA[block I, :]
#pragma unroll
    for (int I = 0; I < 4; ++I) {
      const uint32_t idn = idesc(128, 16 * (I + 1), kFmtTF32, kMajorK, kMajorK);
#pragma unroll
      for (int pt = 0; pt < 2; ++pt) {
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
          mma_tf32_ss(tb + d6_col(I), smem_desc(pt ? qat0 : eat0, 128, kRsT, 4 * I * 128 + ks * 256),
                      smem_desc(pt ? dat : dlt, kCsS, kRsS, 4 * I * kCsS + ks * 2 * kCsS), idn, (pt | ks) ? 1u : 0u, leader);
        }
      }
    }
    mma_commit(&ms.bar_m, leader);
  }
  waiter.wait(&ms.bar_m, mma_phase & 1u);
  ++mma_phase;
  tc_fence_after();
  // shared memory (all but the small arrays of VjpMisc) is dead from here on: fetch the next chunk-head
  [[maybe_unused]] bool pending = false;  // (what the scan writes of the next unit is not there yet)
  if (tid == 0 && (kJoint ? joint_next : ch + gridDim.x) < p.n_ch) issue_loads((kJoint ? joint_next : ch + gridDim.x), locate(kJoint ? joint_next : ch + gridDim.x).slot);
  if constexpr (kJoint) {
    if (tid == 0 && joint_next < p.n_ch) {
      pending = ms.ready[par] == 0;
      if (!pending) bulk_g2s(smem + kOffStack, p.sc + sc.off_dz() + joint_next * kBlobDZ, uint32_t(kBlobDZ), &ms.bar_a);
    }
  }
  if (tid == 64 && (kJoint ? joint_next : ch + gridDim.x) < p.n_ch) {  // (see the other prefetches above)
    const Place nx = locate(kJoint ? joint_next : ch + gridDim.x);
    tma_prefetch_l2_3d(&tm_in.k, 0, nx.h, nx.row);
    tma_prefetch_l2_3d(&tm_in.q, 0, nx.h, nx.row);
    tma_prefetch_l2_3d(&tm_in.beta, 0, nx.h, nx.row);
  }
  // hand k, q and the log-decay prefix to the chain, which walks the tokens of one channel: these threads
  // hold them as 4 x 4 patches (the same values, and for G the same summation order, as the tiles above)
  {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int off = (4 * tg + e) * kDim + kc0;
      store4v<T>(smem + kOffTileK, off, kk[e][0], kk[e][1], kk[e][2], kk[e][3]);
      store4v<T>(smem + kOffTileQ, off, qq[e][0], qq[e][1], qq[e][2], qq[e][3]);
      store4v<T>(smem + beta_tile_offset(mb), (4 * (tg & 3) + e) * kDim + kc0, bb[e][0], bb[e][1], bb[e][2], bb[e][3]);
      store4v<float>(smem + kOffTileG, off, Gc[e][0], Gc[e][1], Gc[e][2], Gc[e][3]);
    }
    __syncthreads();
  }

  // ================================ per-channel chain ==============================================
  // One thread = one key channel over one 16-token block.  The log-decay G and the anchored operands
  // are re-evaluated with exactly the expressions (and summation order) used when the MMA tiles were
  // built, so that dG multiplies each Gram cotangent by the very tf32 value the tensor cores saw:
  // the row and column contributions of the Gram products to dG then cancel as they do exactly.
  {
    const int kc = tid & 127, blk = part;
    bool failed = upstream_failed || waiter.dead;
    if constexpr (kJoint) failed = failed || ms.failed != 0;
    const float gend = ms.gend[kc];
    // dd[k] = sum_v dS_1[k][v] S_0[k][v]: read here, before xt is reused for the block sums of dG
    const float dd_k = (ms.xt[0][kc] + ms.xt[1][kc]) + (ms.xt[2][kc] + ms.xt[3][kc]);
    const float a_me = ms.part[4 * blk][kc];
    const float a_nx = (blk < 3) ? ms.part[4 * (blk + 1)][kc] : gend;
    // per-thread constants: everything but three exponentials per token comes from these
    const float e_ame = exp2_approx(a_me);            // exp(G) = exp(G - a_me) e_ame
    const float c_nx = exp2_approx(a_nx - a_me);      // exp(a_next - G) = exp(a_me - G) c_nx, as in the tile build
    const float t_end = exp2_approx(gend - a_nx);     // exp(G_end - G) = exp(a_next - G) t_end
    const float far2 = (blk + 2 < 4) ? exp2_approx(ms.part[4 * (blk + 2)][kc] - a_nx) : 1.f;  // row block blk + 2
    const float far3 = (blk + 3 < 4) ? exp2_approx(ms.part[4 * (blk + 3)][kc] - a_nx) : 1.f;  // row block blk + 3
    // dG of a token goes back into the slot of the G tile this thread read its log-decay from (nobody else
    // touches it), and the two halves of the block run as a loop: the kernel is a long stretch of
    // straight-line code that every warp walks once per unit, and what it does not need to hold twice
    // saves instruction fetches
    // Two tokens per instruction throughout; -k in place of k where the contribution to dG is negative.
    float2 e_part = twice(0.f), tot = twice(0.f);  // (e_part: negated)
#pragma unroll 1
    for (int sb = 0; sb < 2; ++sb) {
      const int i0 = 16 * blk + 8 * sb;
      float2 ea[4], nk[4], kv[4], bv[4], sq[4], nb[4], P3[4], P2[4], dG[4], x[4], y[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int off = (i0 + 2 * t) * kDim + kc, off_b = (8 * sb + 2 * t) * kDim + kc;
        ea[t] = make_float2(ldf<float>(smem + kOffTileG, off), ldf<float>(smem + kOffTileG, off + kDim));
        kv[t] = make_float2(ldf<T>(smem + kOffTileK, off), ldf<T>(smem + kOffTileK, off + kDim));
        sq[t] = mul2(twice(p.scale), make_float2(ldf<T>(smem + kOffTileQ, off), ldf<T>(smem + kOffTileQ, off + kDim)));
        bv[t] = make_float2(ldf<T>(smem + beta_tile_offset(blk), off_b), ldf<T>(smem + beta_tile_offset(blk), off_b + kDim));
      }
      // row blocks I = blk + d that contain these tokens as columns, nearest first: the own block uses
      // exp(a_me - G), the others exp(a_next - G) (times the block-to-block factor from d = 2 on)
      tmem_ld4x2(tmem_addr(tb, 32 * q4, d6_col(blk) + i0), x);  // dK^blk
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 to_anchor = minus2(twice(a_me), ea[t]);
        const float2 own = exp2_2(to_anchor);
        nk[t] = make_float2(-kv[t].x, -kv[t].y);
        nb[t] = mul2(own, twice(c_nx));
        ea[t] = exp2_2(make_float2(-to_anchor.x, -to_anchor.y));  // the anchored decay exp(G - a_me)
        P3[t] = mul2(x[t], own);
        dG[t] = mul2(tf32_2(anchored_k(nk[t], own, twice(1.f), false)), x[t]);
      }
      tmem_ld4x2(tmem_addr(tb, 32 * q4, kColD4 + i0), x);  // dKt
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 et = mul2(nb[t], twice(t_end));
        const float2 nkt = mul2(nk[t], et);
        P3[t] = fma2(x[t], et, P3[t]);
        e_part = fma2(nkt, x[t], e_part);
        dG[t] = fma2(nkt, x[t], dG[t]);
      }
#pragma unroll
      for (int d = 1; d < 4; ++d) {
        if (blk + d < 4) {
          const float2 far = twice((d == 2) ? far2 : far3);
          tmem_ld4x2(tmem_addr(tb, 32 * q4, d6_col(blk + d) + i0), x);  // dK^(blk + d)
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            P3[t] = fma2(x[t], (d > 1) ? mul2(nb[t], far) : nb[t], P3[t]);
            dG[t] = fma2(tf32_2(anchored_k(nk[t], nb[t], far, d > 1)), x[t], dG[t]);
          }
        }
      }
      tmem_ld4x2(tmem_addr(tb, 32 * q4, kColD3 + i0), x);  // -dE (state part)
      tmem_ld4x2(tmem_addr(tb, 32 * q4, kColD5 + 32 * blk + 8 * sb), y);  // dEa
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 neg_eg = mul2(ea[t], twice(-e_ame));
        P2[t] = fma2(x[t], neg_eg, mul2(y[t], ea[t]));
        const float2 bk = mul2(bv[t], kv[t]);
        dG[t] = fma2(mul2(bk, neg_eg), x[t], dG[t]);
        dG[t] = fma2(tf32_2(mul2(bk, ea[t])), y[t], dG[t]);
      }
      tmem_ld4x2(tmem_addr(tb, 32 * q4, kColD3 + 64 + i0), x);  // dQg (state part)
      tmem_ld4x2(tmem_addr(tb, 32 * q4, kColD5 + 32 * blk + 16 + 8 * sb), y);  // dQa
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 eg = mul2(ea[t], twice(e_ame));
        float2 dq = mul2(twice(p.scale), fma2(x[t], eg, mul2(y[t], ea[t])));
        dG[t] = fma2(tf32_2(mul2(sq[t], ea[t])), y[t], fma2(mul2(sq[t], eg), x[t], dG[t]));
        float2 dk = fma2(bv[t], P2[t], P3[t]), db = mul2(kv[t], P2[t]);
        if (failed) dq = dk = db = twice(poison_nan());
        const int tok = i0 + 2 * t, off = tok * kDim + kc;
        if (kF32Grads) {
          const int64_t idx = seq_idx(tok) + kc, idx1 = seq_idx(tok + 1) + kc;
          if (there(tok)) { stf<O>(p.dq, idx, dq.x); stf<O>(p.dk, idx, dk.x); stf<O>(p.dbeta, idx, db.x); }
          if (there(tok + 1)) { stf<O>(p.dq, idx1, dq.y); stf<O>(p.dk, idx1, dk.y); stf<O>(p.dbeta, idx1, db.y); }
        } else {
          // in place over q and k (this thread's own slots, already read): the tiles leave by TMA stores
          const int off_b = (8 * sb + 2 * t) * kDim + kc;
          stf<T>(smem + kOffTileQ, off, dq.x);
          stf<T>(smem + kOffTileQ, off + kDim, dq.y);
          stf<T>(smem + kOffTileK, off, dk.x);
          stf<T>(smem + kOffTileK, off + kDim, dk.y);
          stf<T>(smem + beta_tile_offset(blk), off_b, db.x);
          stf<T>(smem + beta_tile_offset(blk), off_b + kDim, db.y);
        }
        stf<float>(smem + kOffTileG, off, dG[t].x);
        stf<float>(smem + kOffTileG, off + kDim, dG[t].y);
        tot = add2(tot, dG[t]);
      }
    }
    ms.xe[blk][kc] = -(e_part.x + e_part.y);
    float total = tot.x + tot.y;
    __syncthreads();
    if (blk == 3) {
      const float end_term = ms.xe[0][kc] + ms.xe[1][kc] + ms.xe[2][kc] + ms.xe[3][kc] + exp2_approx(gend) * dd_k;
      *reinterpret_cast<float*>(smem + kOffTileG + (63 * kDim + kc) * 4) += end_term;
      total += end_term;
    }
    ms.xt[blk][kc] = total;
    __syncthreads();
    float run = 0.f;
#pragma unroll
    for (int bq = 3; bq > 0; --bq) {
      if (bq > blk) run += ms.xt[bq][kc];
    }
    if (!kRagged) {
#pragma unroll
      for (int t = 15; t >= 0; --t) {
        run += ldf<float>(smem + kOffTileG, (16 * blk + t) * kDim + kc);
        stf<G>(p.dg, seq_idx(16 * blk + t) + kc, failed ? poison_nan() : run);
      }
    } else {
#pragma unroll
      for (int t = 15; t >= 0; --t) {
        run += ldf<float>(smem + kOffTileG, (16 * blk + t) * kDim + kc);
        if (16 * blk + t < n_valid) stf<G>(p.dg, seq_idx(16 * blk + t) + kc, failed ? poison_nan() : run);
      }
    }
  }
  // the next chunk-head reuses the arrays of VjpMisc and the TMEM columns
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // The rows behind a partial chunk belong to somebody else: its gradients leave row by row, those of a
  // whole chunk by TMA.  (bulk_wait_read_all above and the barriers of phase A guard the tiles' reuse.)
  if (!kF32Grads && kRagged && n_valid < kChunk) {
    for (int e = tid; e < n_valid * 16; e += kVjpThreads) {
      const int tok = e >> 4, piece = e & 15;
      const int64_t idx = seq_idx(tok) + 8 * piece;
      const int off = tok * 256 + piece * 16;
      *reinterpret_cast<uint4*>(static_cast<T*>(p.dq) + idx) = *reinterpret_cast<const uint4*>(smem + kOffTileQ + off);
      *reinterpret_cast<uint4*>(static_cast<T*>(p.dk) + idx) = *reinterpret_cast<const uint4*>(smem + kOffTileK + off);
      *reinterpret_cast<uint4*>(static_cast<T*>(p.dbeta) + idx) =
          *reinterpret_cast<const uint4*>(smem + beta_tile_offset(tok >> 4) + (tok & 15) * 256 + piece * 16);
    }
  }
  if (tid == 0) {
    if (!kF32Grads && !(kRagged && n_valid < kChunk)) {
      tma_store_3d(&tm_dq, 0, h, at.row, smem + kOffTileQ);
      tma_store_3d(&tm_dk, 0, h, at.row, smem + kOffTileK);
#pragma unroll
      for (int bq = 0; bq < 4; ++bq) {
        tma_store_3d(&tm_dbeta, 0, h, at.row + 16 * bq, smem + beta_tile_offset(bq));
      }
      bulk_commit();
    }
    // the G tile is dead: the dS_1 half of the next chunk-head may land on it
    if constexpr (kJoint) {
      if (pending) {
        JointUnits<Seqs>{p, seqs, scan.p.marks, ms}.await(joint_next, waiter);
        bulk_g2s(smem + kOffStack, p.sc + sc.off_dz() + joint_next * kBlobDZ, uint32_t(kBlobDZ), &ms.bar_a);
      }
    }
    if ((kJoint ? joint_next : ch + gridDim.x) < p.n_ch) issue_ds1(locate(kJoint ? joint_next : ch + gridDim.x).slot);
  }
  }  // chunk-head loop
  if (tid == 0) bulk_wait_all();  // the last dq / dk tiles are in global memory before the CTA retires
  if (warp == 0) tmem_dealloc(tb, 512);
}

}  // namespace

// ---- launcher ---------------------------------------------------------------------------------------
namespace {

struct BackwardCall {
  const void *q, *k, *v, *g, *beta, *w, *d_out;
  const float *ds_final, *bnd;
  float* d_bnd;
  const uint8_t* workspace;
  uint8_t* scratch;
  void *dq, *dk, *dv, *dg, *dbeta, *dw;
  float* ds_init;
  int64_t rows, H;  // token rows of the sequence tensors, heads
  int dtype, g_dtype;
  float scale;
  int grads_f32;
  bool ragged;      // some last chunk is partial
  bool beside;      // the launch before this call's is of the same backward and independent of it
};

template <typename T, typename G, typename Seqs, bool kF32Grads, bool kRagged>
int launch_vjp(const VjpParams& p, const Seqs& seqs, const VjpMaps& m, cudaStream_t stream) {
  auto kernel = chunk_bwd_vjp_kernel<T, G, Seqs, kF32Grads, kRagged, false>;
  cudaError_t err = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), kVjpSmemBytes);
  if (err != cudaSuccess) { record_cuda_error(err); return GDN2_ERR_LAUNCH; }
  int sm_count = 0;
  if (int st = multiprocessors(&sm_count); st != GDN2_OK) return st;
  const unsigned grid = unsigned(p.n_ch < int64_t(sm_count) ? p.n_ch : int64_t(sm_count));
  kernel<<<grid, kVjpThreads, kVjpSmemBytes, stream>>>(p, seqs, m, JointScan<false>{});
  return check_launch();
}

template <typename T, typename Seqs>
int launch_bscan(const BScanParams& p, const Seqs& seqs, const BScanMaps& tm, int64_t n_scan, int parts, bool beside,
                 cudaStream_t stream) {
  auto kernel = parts == 4 ? chunk_bwd_scan_kernel<T, Seqs, 4>
              : parts == 2 ? chunk_bwd_scan_kernel<T, Seqs, 2> : chunk_bwd_scan_kernel<T, Seqs, 1>;
  const int smem = int(sizeof(BScanSmem));
  const cudaError_t err = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
  if (err != cudaSuccess) { record_cuda_error(err); return GDN2_ERR_LAUNCH; }
  const int threads = parts > 1 ? BScanWarps<2>::kThreads : BScanWarps<1>::kThreads;
  if (beside) return launch_beside(kernel, unsigned(n_scan * parts), threads, smem, stream, p, seqs, tm);
  kernel<<<unsigned(n_scan * parts), threads, smem, stream>>>(p, seqs, tm);
  return check_launch();
}

thread_local int t_backward_kernels = 0;  // of this thread's latest chunk backward

// One launch for both where it gains: at most a quarter of the SMs with a scan, as in the forward, enough scans, and
// sequences long enough for the VJP to run behind them.  Training steps with two launches / one, us:
//   32 chunks on    H4 T2048 151/159   H4 T2560 198/192   H8 T2048 180/170   H12 T2560 246/224   H16 T2048 225/207
//                   H16 T2560 269/243   H24 T2048 262/249   H28 T2048 294/280   H32 T2048 312/309   H37 T2048 340/350
//                   H37 T2560 420/424   B2 T4133 H16 fp16 619/581
//   below           H4 T1024 98/100   H8 T1024 102/105   H8 T1280 137/130   H8 T1792 165/156   H16 T1024 131/133
//                   H16 T1280 169/161   H16 T1792 208/195   H24 T1280 184/180   H24 T1536 202/207   H32 T1024 187/185
//                   H32 T1792 287/278   H37 T1280 233/240   H37 T1792 300/306
//   fewer scans     H2 T2560 169/175   H3 T2560 174/181: all that the launch could hide is a few units, and quarters of
//                   the value rows, which only the scan kernel has, are worth more
// (Between 18 and 31 chunks 6 to 32 scans would gain 2-6 % where the units are more than one per SM; the line stands
// above that, where all but the two ends of the range gain.)
bool prefer_joint_backward(int64_t n_scan, int64_t n_chunks, int sm_count) {
  return 4 * n_scan <= sm_count && n_scan >= 4 && n_chunks >= 32 && !profiling();
}

template <typename T, typename G, bool kRagged>
int launch_joint(const BScanParams& sp, const VjpParams& vp, const UniformSeqs& seqs, const BScanMaps& tm_scan,
                 const VjpMaps& tm_vjp, int sm_count, cudaStream_t stream) {
  constexpr int smem = int(sizeof(BScanSmem)) > kVjpSmemBytes ? int(sizeof(BScanSmem)) : kVjpSmemBytes;
  auto kernel = chunk_bwd_vjp_kernel<T, G, UniformSeqs, false, kRagged, true>;
  cudaError_t err = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
  if (err != cudaSuccess) { record_cuda_error(err); return GDN2_ERR_LAUNCH; }
  err = cudaMemset2DAsync(sp.marks.dz + kMarkOffset, kBlobDZ, 0, 16, size_t(vp.n_ch), stream);
  if (err != cudaSuccess) { record_cuda_error(err); return GDN2_ERR_LAUNCH; }
  const int64_t want = int64_t(seqs.count()) * sp.H + (vp.n_ch + 1) / 2;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(2 * unsigned(want < sm_count / 2 ? want : sm_count / 2));
  config.blockDim = dim3(kVjpThreads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeCooperative;
  attributes[0].val.cooperative = 1;
  attributes[1].id = cudaLaunchAttributeClusterDimension;
  attributes[1].val.clusterDim.x = 2;
  attributes[1].val.clusterDim.y = attributes[1].val.clusterDim.z = 1;
  config.attrs = attributes;
  config.numAttrs = 2;
  err = cudaLaunchKernelEx(&config, kernel, vp, seqs, tm_vjp, JointScan<true>{sp, tm_scan});
  if (err == cudaErrorCooperativeLaunchTooLarge) {  // a context with fewer SMs than the device
    (void)cudaGetLastError();
    return GDN2_ERR_UNSUPPORTED;
  }
  if (err != cudaSuccess) { (void)cudaGetLastError(); record_cuda_error(err); return GDN2_ERR_LAUNCH; }
  return GDN2_OK;
}

template <typename Seqs>
int launch_backward(const Seqs& seqs, const BackwardCall& a, cudaStream_t stream) {
  if (a.grads_f32 && !(a.dtype == GDN2_BF16 && a.g_dtype == GDN2_FP32)) return GDN2_ERR_UNSUPPORTED;
  const int64_t n_ch = int64_t(seqs.total_chunks()) * a.H;
  const int64_t n_slots = (int64_t(seqs.total_chunks()) + seqs.count()) * a.H;
  if (n_ch <= 0 || n_slots > int64_t(0x7fffffff) || a.rows > int64_t(0x7fffffff)) return GDN2_ERR_TOO_LARGE;
  const WsLayout ws{n_ch, true};
  const ScratchLayout sc{n_ch};
  // the status word is the one the forward cleared: a forward failure stays visible to backward
  int* status = reinterpret_cast<int*>(const_cast<uint8_t*>(a.workspace) + ws.off_status());

  profile_mark(3, stream);
  int sm_count = 0;
  if (int err = multiprocessors(&sm_count); err != GDN2_OK) return err;
  const int64_t n_scan = int64_t(seqs.count()) * a.H;
  bool joint = false;
  if constexpr (std::is_same<Seqs, UniformSeqs>::value) {
    joint = !a.grads_f32 && prefer_joint_backward(n_scan, seqs.n_chunks, sm_count);
  }
  const int parts = joint ? kJointParts : value_parts(n_ch, n_scan, seqs.at(0).n_chunks, sm_count, 4);
  // the reverse scan's operands: the forward's tiles, each in the swizzle of the role backward reads it in
  BScanMaps tm;
  if (!encode_tile_map(&tm.at, a.workspace + ws.off_at(), n_ch, kChunk, kChunk, false, 32, 1) ||
      !encode_tile_map(&tm.tt, a.workspace + ws.off_tt(), n_ch, kChunk, kChunk, false, 32, 1) ||
      !encode_tile_map(&tm.kn, a.workspace + ws.off_kn(), n_ch, kChunk, kDim, false) ||
      !encode_tile_map(&tm.q, a.workspace + ws.off_q(), n_ch, kChunk, kDim, true) ||
      !encode_tile_map(&tm.yt, a.workspace + ws.off_yt(), n_ch, kDim, kChunk, false) ||
      !encode_sequence_map(&tm.d_out, a.d_out, a.rows, a.H, a.dtype, kChunk, kDim / parts)) {
    return GDN2_ERR_LAUNCH;
  }
  const Marks marks{a.scratch + sc.off_dz()};
  const BScanParams sp{a.workspace + ws.off_d(), a.scratch + sc.off_dz(), a.ds_final, a.d_bnd, a.ds_init, status,
                       int(a.H), marks};
  // dq, dk and dbeta leave the VJP kernel through tiled TMA stores; the maps of the inputs serve prefetches
  VjpMaps m;
  const int grad_dtype = a.grads_f32 ? GDN2_FP32 : a.dtype;
  if (!encode_tile_map(&m.s0, reinterpret_cast<const uint8_t*>(a.bnd), n_slots, kDim, kDim, false) ||
      !encode_tile_map(&m.ds, reinterpret_cast<const uint8_t*>(a.d_bnd), n_slots, kDim, kDim, false, 0, 2) ||
      !encode_tile_map(&m.rn, a.workspace + ws.off_rn(), n_ch, kChunk, kDim, false) ||
      !encode_sequence_map(&m.dq, a.dq, a.rows, a.H, grad_dtype) ||
      !encode_sequence_map(&m.dk, a.dk, a.rows, a.H, grad_dtype) ||
      !encode_sequence_map(&m.dbeta, a.dbeta, a.rows, a.H, grad_dtype, 16) ||
      !encode_sequence_map(&m.in.q, a.q, a.rows, a.H, a.dtype) ||
      !encode_sequence_map(&m.in.k, a.k, a.rows, a.H, a.dtype) ||
      !encode_sequence_map(&m.in.v, a.v, a.rows, a.H, a.dtype) ||
      !encode_sequence_map(&m.in.g, a.g, a.rows, a.H, a.g_dtype) ||
      !encode_sequence_map(&m.in.beta, a.beta, a.rows, a.H, a.dtype) ||
      !encode_sequence_map(&m.in.w, a.w, a.rows, a.H, a.dtype) ||
      !encode_sequence_map(&m.in.d_out, a.d_out, a.rows, a.H, a.dtype)) {
    return GDN2_ERR_LAUNCH;
  }
  const VjpParams vp{a.q, a.k, a.v, a.g, a.beta, a.w, a.d_out, a.scratch, a.dq, a.dk, a.dv, a.dg,
                     a.dbeta, a.dw, status, n_ch, int(a.H), a.scale};
  int st = GDN2_ERR_UNSUPPORTED;
  if constexpr (std::is_same<Seqs, UniformSeqs>::value) {
    if (joint) {
      GDN2_DISPATCH_TYPES(a.dtype, a.g_dtype, {
        st = a.ragged ? launch_joint<T, G, true>(sp, vp, seqs, tm, m, sm_count, stream)
                      : launch_joint<T, G, false>(sp, vp, seqs, tm, m, sm_count, stream);
      });
      if (st != GDN2_ERR_UNSUPPORTED) {
        t_backward_kernels = 1;
        return st;
      }
    }
  }
  st = a.dtype == GDN2_BF16 ? launch_bscan<__nv_bfloat16>(sp, seqs, tm, n_scan, parts, a.beside, stream)
                            : launch_bscan<__half>(sp, seqs, tm, n_scan, parts, a.beside, stream);
  if (st != GDN2_OK) return st;
  profile_mark(4, stream);
  if constexpr (std::is_same<Seqs, UniformSeqs>::value) {
    if (a.grads_f32) {
      st = a.ragged ? launch_vjp<__nv_bfloat16, float, Seqs, true, true>(vp, seqs, m, stream)
                    : launch_vjp<__nv_bfloat16, float, Seqs, true, false>(vp, seqs, m, stream);
    }
  }
  if (!a.grads_f32) {
    GDN2_DISPATCH_TYPES(a.dtype, a.g_dtype, {
      st = a.ragged ? launch_vjp<T, G, Seqs, false, true>(vp, seqs, m, stream)
                    : launch_vjp<T, G, Seqs, false, false>(vp, seqs, m, stream);
    });
  }
  profile_mark(5, stream);
  t_backward_kernels = 2;
  return st;
}

}  // namespace

int chunk_backward_kernels() { return t_backward_kernels; }

int launch_chunk_backward(const void* q, const void* k, const void* v, const void* g, const void* beta,
                          const void* w, const void* d_out, const float* ds_final, const float* bnd,
                          float* d_bnd, const uint8_t* workspace, uint8_t* scratch, void* dq, void* dk, void* dv, void* dg,
                          void* dbeta, void* dw, float* ds_init, int64_t B, int64_t T, int64_t H,
                          int64_t full_tokens, int dtype, int g_dtype, float scale, int grads_f32,
                          cudaStream_t stream) {
  const int64_t n_chunks = full_tokens / kChunk;
  if (B * T > int64_t(0x7fffffff) || B * n_chunks * H > int64_t(0x7fffffff)) return GDN2_ERR_TOO_LARGE;
  const UniformSeqs seqs{0, T, int(full_tokens < T ? full_tokens : T), int(n_chunks), int(B)};
  const BackwardCall a{q, k, v, g, beta, w, d_out, ds_final, bnd, d_bnd, workspace, scratch, dq, dk, dv, dg, dbeta,
                       dw, ds_init, B * T, H, dtype, g_dtype, scale, grads_f32, full_tokens > T, false};
  return launch_backward(seqs, a, stream);
}

// `table` as for launch_packed_chunk_forward.
int launch_packed_chunk_backward(const PackedSeqs& table, const void* q, const void* k, const void* v, const void* g,
                                 const void* beta, const void* w, const void* d_out, const float* ds_final,
                                 const float* bnd, float* d_bnd, const uint8_t* workspace, uint8_t* scratch, void* dq,
                                 void* dk, void* dv, void* dg, void* dbeta, void* dw, float* ds_init, int64_t rows,
                                 int64_t H, int dtype, int g_dtype, float scale, bool beside, cudaStream_t stream) {
  bool ragged = false;
  for (int i = 0; i < table.n; ++i) ragged = ragged || table.e[i].len % kChunk != 0;
  const BackwardCall a{q, k, v, g, beta, w, d_out, ds_final, bnd, d_bnd, workspace, scratch, dq, dk, dv, dg, dbeta,
                       dw, ds_init, rows, H, dtype, g_dtype, scale, 0, ragged, beside};
  return launch_backward(table, a, stream);
}

}  // namespace gdn2
