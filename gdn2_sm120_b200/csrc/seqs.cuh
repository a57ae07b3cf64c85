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
// Forward calls of sequences up to this long go token by token, longer ones in spans of 16 tokens.  The line is one
// for all grids, so that a sequence gives the same bits alone and in a batch.  us, steps / spans, for sequences x
// heads of 16, 64, 96, 128, 512, 1024 (at 64 and 128 the spans fill the SMs once and twice):
//   8 tokens            6.5/7.5   8.4/7.8  10.0/11.3  11.9/11.3  33.8/37.9  75.1/83.6
//   9 tokens            7.1/8.4   9.1/8.6  11.1/12.7  13.2/12.7  38.2/42.6  82.4/91.8
//   10 tokens           7.6/8.4   9.9/8.6  11.9/12.7  14.2/12.8  41.1/42.8  88.9/91.8
//   raw inputs, 7       7.3/8.2   9.3/8.4  11.1/12.0  13.2/12.1  39.5/39.8  80.7/83.4
//   raw inputs, 8       7.9/8.3  10.1/8.5  12.1/12.1  14.4/12.2  43.5/40.1  88.3/83.9
//   raw inputs, 9       8.9/9.1  11.2/9.3  13.6/13.5  16.0/13.5  48.9/45.1  99.5/92.8
constexpr int kStepTokens = 9, kStepTokensRaw = 8;
inline int step_tokens(int prologue) { return prologue != 0 ? kStepTokensRaw : kStepTokens; }

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
