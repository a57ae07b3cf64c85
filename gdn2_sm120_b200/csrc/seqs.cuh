// Which token rows a chunk (64 tokens, chunk kernels) or a span (16 tokens, token kernels) consists of.
//
// A sequence is a run of token rows of the [rows][H][128] tensors (rows = batch * time, or the packed
// length) cut into pieces of kSpan tokens; the last one may be partial.  Pieces are numbered through all
// sequences, `chunk0` is a sequence's first one; unit = piece * H + h.  The state checkpoints have one
// slot more than pieces per sequence: slot of piece c = (chunk0 + order + c) * H + h.
#pragma once

#include "common.cuh"

namespace gdn2 {

constexpr int kChunk = GDN2_CHUNK;  // 64
constexpr int kStepTokens = 8;      // forward calls of sequences up to this long go token by token

struct SeqInfo {
  int64_t row0;   // first token row
  int len;        // tokens
  int chunk0;     // number of its first piece
  int n_chunks;
  int slot0;      // chunk0 + position of the sequence in the list
  int sid;        // row of its state in the [sequences][H][128][128] state tensors
};

// A batch of equally long sequences: everything follows from the sizes.
struct UniformSeqs {
  int64_t first, stride;  // row of the first token, token rows from one sequence to the next
  int len, n_chunks, n;
  __host__ __device__ int count() const { return n; }
  __host__ __device__ int total_chunks() const { return n * n_chunks; }
  __host__ __device__ __forceinline__ SeqInfo at(int s) const {
    return SeqInfo{first + s * stride, len, s * n_chunks, n_chunks, s * (n_chunks + 1), s};
  }
  __device__ __forceinline__ int find(int chunk) const { return int(uint32_t(chunk) / uint32_t(n_chunks)); }
};

// Sequences of several lengths, a table in kernel-parameter space (no copy to the device).  The host lists
// the longest first: the scans walk a sequence serially and the long ones must not start last.
constexpr int kMaxPacked = GDN2_PACKED_MAX_SEQUENCES;  // per launch: 4 KiB of parameters; longer lists take several
template <int kSpan>
struct PackedSeqsOf {
  struct Entry { int row0, len, chunk0, sid; };
  int n, chunks;
  Entry e[kMaxPacked];
  __host__ __device__ int count() const { return n; }
  __host__ __device__ int total_chunks() const { return chunks; }
  __host__ __device__ __forceinline__ SeqInfo at(int s) const {
    const Entry x = e[s];
    return SeqInfo{x.row0, x.len, x.chunk0, (x.len + kSpan - 1) / kSpan, x.chunk0 + s, x.sid};
  }
  __device__ __forceinline__ int find(int chunk) const {  // last entry with chunk0 <= chunk
    int lo = 0, hi = n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (e[mid].chunk0 <= chunk) lo = mid; else hi = mid - 1;
    }
    return lo;
  }
  void add(int row0, int len, int sid) {  // host; empty sequences own no piece
    e[n++] = Entry{row0, len, chunks, sid};
    chunks += (len + kSpan - 1) / kSpan;
  }
};
using PackedSeqs = PackedSeqsOf<kChunk>;
using PackedSpans = PackedSeqsOf<kTokenInterval>;

}  // namespace gdn2
