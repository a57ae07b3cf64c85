// Shared definitions of the 64-token tensor-core chunk path.
//
// For every unit ch = (b * n_chunks + c) * H + h (one 64-token chunk of one head) the prep kernel
// writes the WY factors as plain row-major fp32 matrices holding tf32 values ("tiles"), ONE copy of
// each.  The forward scan and the reverse scan both consume them: the forward contracts over one index
// of a tile and the backward over the other, so one kernel reads a tile as a K-major operand and the
// other as an MN-major operand.  Tiled TMA loads put the same global bytes into shared memory in the
// layout each role needs (K-major: 128-byte swizzle; MN-major tf32: 128-byte swizzle with 32-byte
// atoms, the only MN-major form the tensor cores accept for 32-bit operands).  The orientation of a
// tile in global memory is the one its producer can store with full 128-byte lines: token-major for
// tiles made from registers, transposed for tiles read out of tensor memory (lane = row).
//
//   Q    [token i (64)][key k (128)]     32 KiB   scale * gamma * q            fwd K-major,  bwd MN-major
//   Kn   [token j (64)][key k (128)]     32 KiB   k * gamma_end / gamma        fwd MN-major, bwd K-major
//   Yt   [key k (128)][token i (64)]     32 KiB   Y^T, Y = (I+L)^-1 E          fwd MN-major, bwd K-major
//   At   [token j (64)][token i (64)]    16 KiB   tril(Q_gamma Kbar^T)^T       fwd MN-major, bwd K-major
//   Tt   [token j (64)][token i (64)]    16 KiB   ((I+L)^-1)^T                 fwd MN-major, bwd K-major
//        (both are zero where j > i: the quadrant j >= 32, i < 32 is neither written nor read, the
//        consumers keep those lines of their shared-memory tile at zero; 12 KiB move)
//   D    float[128]                      512 B    gamma_end
//        (element 0 is negative when its unit was prepared beside a running scan: read magnitudes)
//
//   Rn   [token j (64)][value v (128)]   32 KiB   R = U - Y S_0   forward scan -> VJP kernel (K-major)
//
// One more per-unit array is a "blocked" tile (see tc05.cuh) that a bulk copy moves as it is:
//   dZ   X[r = token j (64)][c = value v (128)] RS = 4608, CS = 144   36 KiB   dZ = T^T dR
//        (reverse scan -> VJP kernel; the padded strides are those of the tile it is copied into.  The 16 bytes
//        behind the last row are padding too: where the two share a launch they hold the unit's mark and, in the
//        first tile, the queue of units)
//
// Buffers (caller-provided, struct of arrays, each array n_ch entries long):
//   workspace  D, a 256-byte status block, and for a training call what backward consumes:
//              Rn, Q, Kn, Yt, At, Tt
//   scratch    dead when the call returns: the forward tiles of an inference call (Q, Kn, Yt, At, Tt in
//              144 KiB per unit; a training call has them in its workspace and no forward scratch);
//              backward dZ
#pragma once

#include <cuda.h>

#include <atomic>
#include <mutex>

#include "common.cuh"
#include "seqs.cuh"
#include "tc05.cuh"

namespace gdn2 {

constexpr int64_t kTileQ = 32768, kTileKn = 32768, kTileYt = 32768;
constexpr int64_t kTileAt = 16384, kTileTt = 16384, kBlobD = 512;
constexpr int64_t kBlobRn = 32768, kBlobDZ = 8 * 4608;
constexpr int64_t kStatusBytes = 256;  // word 0: status
constexpr int kQueueWord = 16;         // joint launch: next unit to prepare
constexpr float kLog2e = 1.4426950408889634f;  // log-decays are summed in units of ln 2
// forward scratch per unit, sizes callers know: 144 KiB for an inference call (its tiles take 128 of
// them), 32 KiB reserved for a training call (NULL will do)
constexpr int64_t kFwdScratchInference = 147456, kFwdScratchTraining = 32768;

// workspace: what a training forward leaves for backward (inference: D and the status block only)
struct WsLayout {
  int64_t n_ch;
  bool training = false;
  __host__ __device__ int64_t off_d() const { return 0; }
  __host__ __device__ int64_t off_status() const { return n_ch * kBlobD; }
  // training-only arrays follow the status block
  __host__ __device__ int64_t off_rn() const { return off_status() + kStatusBytes; }
  __host__ __device__ int64_t off_q() const { return off_rn() + n_ch * kBlobRn; }
  __host__ __device__ int64_t off_kn() const { return off_q() + n_ch * kTileQ; }
  __host__ __device__ int64_t off_yt() const { return off_kn() + n_ch * kTileKn; }
  __host__ __device__ int64_t off_at() const { return off_yt() + n_ch * kTileYt; }
  __host__ __device__ int64_t off_tt() const { return off_at() + n_ch * kTileAt; }
  __host__ __device__ int64_t total() const { return training ? off_tt() + n_ch * kTileTt : off_rn(); }
};

// scratch of one call
struct ScratchLayout {
  int64_t n_ch;
  // inference calls only (a training call keeps these in its workspace)
  __host__ __device__ int64_t off_q() const { return 0; }
  __host__ __device__ int64_t off_kn() const { return off_q() + n_ch * kTileQ; }
  __host__ __device__ int64_t off_yt() const { return off_kn() + n_ch * kTileKn; }
  __host__ __device__ int64_t off_at() const { return off_yt() + n_ch * kTileYt; }
  __host__ __device__ int64_t off_tt() const { return off_at() + n_ch * kTileAt; }
  __host__ __device__ int64_t total_forward(bool training) const {
    return n_ch * (training ? kFwdScratchTraining : kFwdScratchInference);
  }
  __host__ __device__ int64_t off_dz() const { return 0; }
  __host__ __device__ int64_t total_backward() const { return n_ch * kBlobDZ; }
};
static_assert(kTileQ + kTileKn + kTileYt + kTileAt + kTileTt <= kFwdScratchInference, "tiles exceed the scratch");

// where the forward tile arrays of a call live
struct ForwardTiles {
  uint8_t *q, *kn, *yt, *at, *tt;
};
inline ForwardTiles forward_tiles(uint8_t* workspace, uint8_t* scratch, int64_t n_ch, bool training) {
  const WsLayout ws{n_ch, training};
  const ScratchLayout sc{n_ch};
  ForwardTiles t;
  if (training) {
    t.q = workspace + ws.off_q(); t.kn = workspace + ws.off_kn(); t.yt = workspace + ws.off_yt();
    t.at = workspace + ws.off_at(); t.tt = workspace + ws.off_tt();
  } else {
    t.q = scratch + sc.off_q(); t.kn = scratch + sc.off_kn(); t.yt = scratch + sc.off_yt();
    t.at = scratch + sc.off_at(); t.tt = scratch + sc.off_tt();
  }
  return t;
}

// device status codes written to the workspace status word (0 = ok)
enum : int { kStatusOk = 0, kStatusBarrierTimeout = 1 };

__device__ __forceinline__ float poison_nan() { return __int_as_float(0x7fc00000); }

// A wait that gives up: after `limit` failed polls the thread records kStatusBarrierTimeout in the
// status word (and in the CTA's flag when it has one, for the roles of a warp-specialised kernel) and
// every later wait of the thread returns immediately.  The kernel then runs to its end (shared
// resources such as TMEM are always released) and writes NaN instead of results, so the failure shows
// in the outputs themselves and not only in the status word.
struct BoundedWaiter {
  bool dead = false;
  int* status;
  uint32_t limit;
  volatile int* cta_flag;
  __device__ explicit BoundedWaiter(int* s, uint32_t max_polls = (1u << 20), volatile int* flag = nullptr)
      : status(s), limit(max_polls), cta_flag(flag) {}
  __device__ __forceinline__ void wait(uint64_t* bar, uint32_t parity) {
    if (dead) return;
    if (!tc::mbar_wait(bar, parity, limit)) expire();
  }
  // for loops that look at something other than an mbarrier: false once `limit` looks in a row were in vain.  What was
  // looked for has a count of its own, from look_anew on: a launch may look any number of times, and mbarrier waits
  // keep their limit.
  uint32_t looks = 0;
  __device__ __forceinline__ void look_anew() { looks = 0; }
  __device__ __forceinline__ bool look_again() {
    if (!dead && ++looks >= limit) expire();
    return !dead;
  }
  __device__ __forceinline__ void expire() {
    dead = true;
    if (cta_flag != nullptr) *cta_flag = 1;
    if (status != nullptr) atomicExch(status, kStatusBarrierTimeout);
  }
};

// ---- marks between CTAs of one launch: a float whose sign says that a unit is finished ------------
__device__ __forceinline__ void store_release(float* p, float x) {
  asm volatile("st.release.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(x) : "memory");
}
__device__ __forceinline__ bool marked(const float* p) {
  uint32_t x;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(p) : "memory");
  return (x >> 31) != 0;
}

// ---- tensor maps (host) -------------------------------------------------------------------------
// cuTensorMapEncodeTiled through the runtime's driver entry point query: the library does not link
// against the driver API for this one call.
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult query;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &query) != cudaSuccess ||
        query != cudaDriverEntryPointSuccess) {
      return EncodeTiledFn(nullptr);
    }
    return reinterpret_cast<EncodeTiledFn>(ptr);
  }();
  return fn;
}

// Encoding a tensor map costs the host some 20 microseconds and a call needs a dozen of them; the
// maps depend only on addresses and shapes, which repeat from call to call (allocators hand the same
// blocks out again), so the last few hundred are kept.  Four ways a set, the oldest of a set leaves; one mutex.
// (One map a set is not enough: a training step has some thirty, of which one pair in two steps met in 512 places.)
struct TensorMapKey {
  uintptr_t base;
  cuuint64_t dims[4], strides[3];
  cuuint32_t box[4];
  int rank, type, swizzle;
  bool operator==(const TensorMapKey& o) const {
    bool same = base == o.base && rank == o.rank && type == o.type && swizzle == o.swizzle;
    for (int i = 0; i < 4; ++i) same = same && dims[i] == o.dims[i] && box[i] == o.box[i];
    for (int i = 0; i < 3; ++i) same = same && strides[i] == o.strides[i];
    return same;
  }
  // every field counts: scans of split value rows and the VJP have maps of one tensor that differ in box[0] alone
  uint64_t hash() const {
    uint64_t h = base;
    auto mix = [&h](uint64_t x) { h = (h ^ x) * 0x9E3779B97F4A7C15ull; h ^= h >> 32; };
    for (int i = 0; i < 4; ++i) { mix(dims[i]); mix(box[i]); }
    for (int i = 0; i < 3; ++i) mix(strides[i]);
    mix(uint64_t(rank) << 32 | uint64_t(type) << 16 | uint64_t(swizzle));
    return h;
  }
};

inline std::atomic<int64_t> g_tensor_maps_encoded{0};  // by this process: those that were not kept

// rank 3 or 4; unused trailing entries of dims / strides / box are 1 / 0 / 1
inline bool encode_cached(CUtensorMap* tm, int rank, CUtensorMapDataType type, const void* base,
                          const cuuint64_t (&dims)[4], const cuuint64_t (&strides)[3], const cuuint32_t (&box)[4],
                          CUtensorMapSwizzle swizzle) {
  constexpr int kSets = 128, kWays = 4;
  struct Set {
    struct { bool used = false; TensorMapKey key; CUtensorMap map; } way[kWays];
    int oldest = 0;
  };
  static Set sets[kSets];
  static std::mutex mutex;
  const TensorMapKey key{reinterpret_cast<uintptr_t>(base), {dims[0], dims[1], dims[2], dims[3]},
                         {strides[0], strides[1], strides[2]}, {box[0], box[1], box[2], box[3]}, rank, int(type),
                         int(swizzle)};
  Set& set = sets[key.hash() % kSets];
  {
    std::lock_guard<std::mutex> lock(mutex);
    for (const auto& way : set.way) {
      if (way.used && way.key == key) { *tm = way.map; return true; }
    }
  }
  EncodeTiledFn encode = encode_tiled_fn();
  if (encode == nullptr) return false;
  const cuuint32_t elem_strides[4] = {1, 1, 1, 1};
  // OOB_FILL_NONE: the part of a load box outside the tensor reads as zero
  auto attempt = [&] {
    return encode(tm, type, cuuint32_t(rank), const_cast<void*>(base), dims, strides, box, elem_strides,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  if (!attempt()) {
    // a driver call needs the device's context in this thread, and a thread whose first CUDA call this is (an
    // autograd thread served from an allocator's cache) has none yet
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaSetDevice(device) != cudaSuccess || !attempt()) return false;
  }
  g_tensor_maps_encoded.fetch_add(1, std::memory_order_relaxed);
  std::lock_guard<std::mutex> lock(mutex);
  for (const auto& way : set.way) {
    if (way.used && way.key == key) return true;  // (another thread was first)
  }
  auto& way = set.way[set.oldest];
  set.oldest = (set.oldest + 1) % kWays;
  way.used = true; way.key = key; way.map = *tm;
  return true;
}

// A contiguous [rows, H, 128] sequence tensor (rows = batch * time, or the packed length) seen as
// (channel, head, row): a box (128, 1, 64) is one head's 64-token chunk, landing in shared memory as dense
// [64][128] rows (`box_rows` tokens and `box_cols` channels when given).  A partial chunk reads on into the rows of
// the next sequence (zeros past the end of the tensor): the kernels mask what is not theirs.
inline bool encode_sequence_map(CUtensorMap* tm, const void* base, int64_t rows, int64_t heads, int dtype,
                                int box_rows = kChunk, int box_cols = kDim) {
  const cuuint64_t es = (dtype == GDN2_FP32) ? 4 : 2;
  const CUtensorMapDataType type = (dtype == GDN2_FP32)   ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                   : (dtype == GDN2_BF16) ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                          : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const cuuint64_t dims[4] = {cuuint64_t(kDim), cuuint64_t(heads), cuuint64_t(rows), 1};
  const cuuint64_t strides[3] = {cuuint64_t(kDim) * es, cuuint64_t(heads) * kDim * es, 0};  // bytes, dimensions 1..2
  const cuuint32_t box[4] = {cuuint32_t(box_cols), 1, cuuint32_t(box_rows), 1};
  return encode_cached(tm, 3, type, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
}

// The same tensor (16-bit) seen as (channel within 64, row, half of the channels, head): a box (64, 64, 2, 1) is one
// head's chunk, landing as [half][64] lines of 128 bytes whose 16-byte pieces are permuted by the line.
inline bool encode_half_map(CUtensorMap* tm, const void* base, int64_t rows, int64_t heads, int dtype) {
  const cuuint64_t dims[4] = {64, cuuint64_t(rows), kDim / 64, cuuint64_t(heads)};
  const cuuint64_t strides[3] = {cuuint64_t(heads) * kDim * 2, 128, kDim * 2};
  const cuuint32_t box[4] = {64, kChunk, kDim / 64, 1};
  return encode_cached(tm, 4, dtype == GDN2_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                       base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

// An array of n_ch row-major fp32 tiles [rows][cols] seen as (column within a slab, row, slab of 32
// columns, unit).  A slab lands in shared memory as `rows` lines of 128 bytes; mn_major chooses the
// swizzle: 128-byte with 32-byte atoms (the tile is read as an MN-major operand, contraction over its
// rows) or plain 128-byte (K-major operand, contraction over its columns).  A box takes `box_slabs` slabs
// of `box_rows` rows (0: all of them): one copy instruction brings a whole tile.  Tiles whose zero
// quadrant is never moved go in boxes of one slab and half the rows.
inline bool encode_tile_map(CUtensorMap* tm, const uint8_t* base, int64_t n_ch, int rows, int cols, bool mn_major,
                            int box_rows = 0, int box_slabs = 0) {
  const cuuint64_t dims[4] = {32, cuuint64_t(rows), cuuint64_t(cols / 32), cuuint64_t(n_ch)};
  const cuuint64_t strides[3] = {cuuint64_t(cols) * 4, 128, cuuint64_t(rows) * cols * 4};
  const cuuint32_t box[4] = {32, cuuint32_t(box_rows > 0 ? box_rows : rows),
                             cuuint32_t(box_slabs > 0 ? box_slabs : cols / 32), 1};
  return encode_cached(tm, 4, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, base, dims, strides, box,
                       mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B);
}

// CTAs that share the value rows of one (sequence, head) in a scan.  A value row of the state never meets another
// one, so a scan may have 64 or 32 of the 128 rows (its MMAs still have 128; the lanes behind are idle) and gives
// the same bits.  What an SM takes in and puts out goes through a port of 48-50 bytes a clock (a probe that only
// copies: 48.2 in, 50 both ways), and a chunk of a training scan is 284 KB forward and 236 KB back, 2.9 and 2.5 us
// of its 3.0 and 2.6: halves of the rows move 212 and 178 KB each, quarters 176 and 149.  Scan times, us, with 1 / 2 /
// 4 parts: training B1 T2048 H16 100 / 70 / 73 forward, 86 / 64 / 60 back; B2 T4096 H16 193 / 143 / 152 and
// 162 / 128 / 123; inference B1 T2048 H32 70 / 68 / 73, B1 T32768 H16 971 / 866 / 920 (hence 2 at most forward).
// As many as leave the longest sequence the longest part of the call: with 128 sequences x heads of one length,
// where every SM has a scan as it is, halves take 749 -> 758 us (training B4 T8192 H32) and 221 -> 293 (inference
// B8 T4096); packed training of 911, 2300, 150, 1640, 77, 1202, 514, 1398 tokens, H16, 133 -> 114 and 109 -> 97.
// A CTA counts for five chunks more than it scans: it takes that long to start, to read its state and to end (a scan of
// one to four chunks takes 15-17 us).  Without them packed inference of 100, 200, 300 tokens, H32, was split into 192
// CTAs for 148 SMs: 51.8 -> 56.0 us, and 300, 300, 600 80.7 -> 84.1; 64, 128, 192, 256 at H24 39.0 -> 41.1.
constexpr int kScanOverhead = 5;
inline int value_parts(int64_t units, int64_t scans, int64_t longest, int sm_count, int most) {
  int parts = 1;
  while (parts < most && 2 * parts * (units + kScanOverhead * scans) <= (longest + kScanOverhead) * sm_count) parts *= 2;
  return parts;
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

}  // namespace gdn2
