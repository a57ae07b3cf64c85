// Packed variable-length sequences: one call for all of them.
//
// The sequences of a [1, total, H, 128] batch go to the same kernels as equally long ones, with a table
// of (first row, length, first piece, state row) in the kernels' parameters instead of a division:
// from 64 tokens on to the chunk kernels, below to the token kernels, as separate calls would.  A launch
// per kernel for the whole batch instead of one per sequence: a batch of 16 prompts spent most of its time
// on 90 launches whose grids filled a tenth of the GPU.

#include <algorithm>
#include <initializer_list>

#include "chunk_common.cuh"

namespace gdn2 {

int launch_packed_chunk_forward(const PackedSeqs&, const void*, const void*, const void*, const void*, const void*,
                                const void*, const float*, void*, float*, float*, uint8_t*, uint8_t*, int64_t, int64_t,
                                int, int, int, float, int, cudaStream_t);
int launch_packed_chunk_backward(const PackedSeqs&, const void*, const void*, const void*, const void*, const void*,
                                 const void*, const void*, const float*, const float*, float*, const uint8_t*,
                                 uint8_t*, void*, void*, void*, void*, void*, void*, float*, int64_t, int64_t, int,
                                 int, float, bool, cudaStream_t);
int launch_packed_token_forward(const PackedSpans&, const void*, const void*, const void*, const void*, const void*,
                                const void*, const float*, void*, float*, float*, int64_t, int, int, float, int, bool,
                                cudaStream_t);
int launch_packed_token_reverse(const PackedSpans&, const void*, const void*, const void*, const void*, const void*,
                                const float*, float*, float*, int64_t, int, int, float, cudaStream_t);
int launch_packed_token_vjp(const PackedSpans&, const void*, const void*, const void*, const void*, const void*,
                            const void*, const void*, const float*, const float*, void*, void*, void*, void*, void*,
                            void*, int64_t, int, int, float, bool, cudaStream_t);

namespace {

struct Tables {
  PackedSeqs chunks;   // sequences of 64 tokens and more, longest first
  PackedSpans spans;   // shorter ones, empty ones included (their state passes through)
};

// The tables follow from the bounds alone: forward and backward of a batch agree on every unit and slot.
int build_tables(const int64_t* bounds, int64_t n_seq, int64_t total, int64_t heads, Tables* t) {
  if (bounds == nullptr) return GDN2_ERR_NULL_POINTER;
  if (n_seq <= 0 || heads <= 0 || total < 0) return GDN2_ERR_BAD_SHAPE;
  if (n_seq > kMaxPacked || total > int64_t(0x7fffffff)) return GDN2_ERR_TOO_LARGE;
  int order[kMaxPacked];
  for (int i = 0; i < int(n_seq); ++i) {
    if (bounds[i] < 0 || bounds[i + 1] < bounds[i] || bounds[i + 1] > total) return GDN2_ERR_BAD_RANGE;
    order[i] = i;
  }
  std::stable_sort(order, order + n_seq, [&](int a, int b) {
    return bounds[a + 1] - bounds[a] > bounds[b + 1] - bounds[b];
  });
  t->chunks.n = t->chunks.chunks = t->spans.n = t->spans.chunks = 0;
  for (int i = 0; i < int(n_seq); ++i) {
    const int s = order[i], row0 = int(bounds[s]), len = int(bounds[s + 1] - bounds[s]);
    if (len >= kChunk) t->chunks.add(row0, len, s);
    else t->spans.add(row0, len, s);
  }
  // units and checkpoint slots are 31-bit numbers
  const int64_t most = int64_t(std::max(t->chunks.chunks, t->spans.chunks)) + n_seq;
  if (most * heads > int64_t(0x7fffffff) / 4) return GDN2_ERR_TOO_LARGE;
  return GDN2_OK;
}

int check_call(int dtype, int g_dtype, std::initializer_list<const void*> required,
               std::initializer_list<const void*> optional) {
  if (!valid_seq_dtype(dtype) || !valid_gate_dtype(g_dtype, dtype)) return GDN2_ERR_BAD_DTYPE;
  for (const void* ptr : required) {
    if (ptr == nullptr) return GDN2_ERR_NULL_POINTER;
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0) return GDN2_ERR_ALIGNMENT;
  }
  for (const void* ptr : optional) {
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0) return GDN2_ERR_ALIGNMENT;
  }
  return GDN2_OK;
}

}  // namespace
}  // namespace gdn2

using namespace gdn2;

extern "C" int gdn2_packed_sizes(const int64_t* bounds, int64_t n_seq, int64_t total, int64_t heads, int64_t* chunks,
                                 int64_t* chunk_slots, int64_t* span_slots) {
  if (chunks == nullptr || chunk_slots == nullptr || span_slots == nullptr) return GDN2_ERR_NULL_POINTER;
  Tables t;
  const int st = build_tables(bounds, n_seq, total, heads, &t);
  if (st != GDN2_OK) return st;
  *chunks = t.chunks.chunks;
  *chunk_slots = int64_t(t.chunks.chunks) + t.chunks.n;
  *span_slots = int64_t(t.spans.chunks) + t.spans.n;
  return GDN2_OK;
}

extern "C" int gdn2_packed_forward(const void* q, const void* k, const void* v, const void* g, const void* beta,
                                   const void* w, const float* initial_state, void* out, float* final_state,
                                   float* chunk_boundaries, float* span_boundaries, void* workspace, void* scratch,
                                   const int64_t* bounds, int64_t n_seq, int64_t total, int64_t heads, int training,
                                   int dtype, int g_dtype, float scale, int prologue, void* stream) {
  Tables t;
  int st = build_tables(bounds, n_seq, total, heads, &t);
  if (st != GDN2_OK) return st;
  if ((st = check_call(dtype, g_dtype, {q, k, v, g, beta, w, out},
                       {initial_state, final_state, chunk_boundaries, span_boundaries, workspace, scratch})) != GDN2_OK) {
    return st;
  }
  if ((prologue & ~(GDN2_PROLOGUE_NORMALIZE_QK | GDN2_PROLOGUE_ACTIVATE_GATES)) != 0 || (prologue != 0 && training)) {
    return GDN2_ERR_UNSUPPORTED;
  }
  const cudaStream_t cs = static_cast<cudaStream_t>(stream);
  if (t.chunks.n > 0) {
    if (workspace == nullptr || (training ? chunk_boundaries == nullptr : scratch == nullptr)) {
      return GDN2_ERR_NULL_POINTER;
    }
    st = launch_packed_chunk_forward(t.chunks, q, k, v, g, beta, w, initial_state, out, final_state,
                                     training ? chunk_boundaries : nullptr, static_cast<uint8_t*>(workspace),
                                     static_cast<uint8_t*>(scratch), total, heads, training, dtype, g_dtype, scale,
                                     prologue, cs);
    if (st != GDN2_OK) return st;
  }
  if (t.spans.n > 0) {
    if (training && span_boundaries == nullptr) return GDN2_ERR_NULL_POINTER;
    // Beside the scans, which leave the SMs to one another as they end, and some idle from the start.  (Packed inference
    // of 16 sequences, H16, 33 and 7 tokens among them: 268 -> 242 us.)
    st = launch_packed_token_forward(t.spans, q, k, v, g, beta, w, initial_state, out, final_state,
                                     training ? span_boundaries : nullptr, heads, dtype, g_dtype, scale, prologue,
                                     t.chunks.n > 0 && !profiling(), cs);
  }
  return st;
}

extern "C" int gdn2_packed_backward(const void* q, const void* k, const void* v, const void* g, const void* beta,
                                    const void* w, const void* d_out, const float* d_final_state,
                                    const float* chunk_boundaries, float* d_chunk_boundaries,
                                    const float* span_boundaries, float* d_span_boundaries, const void* workspace,
                                    void* scratch, void* dq, void* dk, void* dv, void* dg, void* dbeta, void* dw,
                                    float* d_initial_state, const int64_t* bounds, int64_t n_seq, int64_t total,
                                    int64_t heads, int dtype, int g_dtype, float scale, void* stream) {
  Tables t;
  int st = build_tables(bounds, n_seq, total, heads, &t);
  if (st != GDN2_OK) return st;
  if ((st = check_call(dtype, g_dtype, {q, k, v, g, beta, w, d_out, dq, dk, dv, dg, dbeta, dw},
                       {d_final_state, d_initial_state, chunk_boundaries, d_chunk_boundaries, span_boundaries,
                        d_span_boundaries, workspace, scratch})) != GDN2_OK) {
    return st;
  }
  const cudaStream_t cs = static_cast<cudaStream_t>(stream);
  if (t.chunks.n > 0 &&
      (workspace == nullptr || scratch == nullptr || chunk_boundaries == nullptr || d_chunk_boundaries == nullptr)) {
    return GDN2_ERR_NULL_POINTER;
  }
  // The reverse scans run beside the short sequences' reverse kernel, and the short sequences' VJP beside the other one.
  const bool beside = t.chunks.n > 0 && t.spans.n > 0 && !profiling();
  if (t.spans.n > 0) {
    if (span_boundaries == nullptr || d_span_boundaries == nullptr) return GDN2_ERR_NULL_POINTER;
    st = launch_packed_token_reverse(t.spans, q, k, g, beta, d_out, d_final_state, d_span_boundaries, d_initial_state,
                                     heads, dtype, g_dtype, scale, cs);
    if (st != GDN2_OK) return st;
  }
  if (t.chunks.n > 0) {
    st = launch_packed_chunk_backward(t.chunks, q, k, v, g, beta, w, d_out, d_final_state, chunk_boundaries,
                                      d_chunk_boundaries, static_cast<const uint8_t*>(workspace),
                                      static_cast<uint8_t*>(scratch), dq, dk, dv, dg, dbeta, dw, d_initial_state,
                                      total, heads, dtype, g_dtype, scale, beside, cs);
    if (st != GDN2_OK) return st;
  }
  if (t.spans.n > 0) {
    st = launch_packed_token_vjp(t.spans, q, k, v, g, beta, w, d_out, span_boundaries, d_span_boundaries, dq, dk, dv, dg,
                                 dbeta, dw, heads, dtype, g_dtype, scale, beside, cs);
  }
  return st;
}
