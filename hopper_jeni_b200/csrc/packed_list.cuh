// The work list of a packed variable-length batch, laid out by every thread block for itself in shared memory: the sequences
// by length, longest first, and where the items of each begin in the list.
//
// Without it the list covers max_seqlen for every sequence in the order of the batch: most of it is empty when the lengths
// differ (every empty item costs a claim), and a long sequence late in the batch leaves most SMs idle at the end.  B200, us,
// causal: backward of 36 sequences of 128 to 8192 tokens, Hq12 Hkv4 D64 1 592 -> 1 532, of 128 of 16 to 2048, Hq4 Hkv1 D64
// 195 -> 138; forward of 32 of 16 to 2048, Hq4 Hkv1 D64 37.8 -> 28.2, of 28 of 128 to 8192, Hq32 Hkv8 D128 1 785 -> 1 746.
#pragma once

#include <stdint.h>

namespace gqa {

constexpr int kMaxListedSeqs = 512;       // larger batches keep the order of the batch
constexpr int kMaxListedUnits = 1 << 21;  // (twice that many * kMaxListedSeqs is a sort key of 31 bits)

// Whether a launch of one item per `rows` rows of a sequence for each of `heads` heads is listed.  Building the list delays the
// first item by a microsecond (28 sequences) to six (512).  Where every item finds an SM at once, or no sequence has more
// than one, there is nothing to order; and many short sequences take too little for it: 512 of which all but one have 1 to 64
// tokens, Hq4 D64 causal, are 41.7 us unlisted and 47.3 listed (backward 56.9 / 60.9), 512 of 16 to 2048 tokens 283 / 278
// (730 / 679).
inline bool list_pays(int n_seqs, int max_len, int tokens, int rows, int heads, int sms) {
    const long long max_units = ((long long)max_len + rows - 1) / rows;
    return n_seqs <= kMaxListedSeqs && max_units > 1 && max_units < kMaxListedUnits && n_seqs * max_units * heads > sms &&
           (long long)tokens / rows * heads * 64 >= (long long)n_seqs * sms;
}
// Sequences of (nearly) one length are in order as they are.
inline bool lengths_differ(int n_seqs, int max_len, int tokens) { return (long long)tokens * 8 < (long long)n_seqs * max_len * 7; }

struct alignas(16) PackedList {
    int first[kMaxListedSeqs + 1];         // first item of every run of `run` sequences; then the number of items
    unsigned short seq[kMaxListedSeqs];    // the sequences, longest first (equal lengths in the order of the batch)

    // To be called by every thread of the block.  A sequence has one unit per `unit_rows` rows, `max_units` at most, a run as
    // many per sequence as its longest one, and every unit `heads` items.
    // Places by comparison with every other sequence, four per load: 1 750 to 2 700 cycles at 28 sequences, 2 300 to 3 500 at 128,
    // 4 800 at 256 and 12 000 to 15 000 at 512 (26 000 with one per load).  A sort in registers and a binary search in the sorted
    // parts is shorter, but the backward kernel with it is 4 % slower at D = 64 (registers): 36 sequences of 128 to 8192 tokens
    // 1 532 -> 1 588 us.
    __device__ void build(const int* cu, int n_seqs, int unit_rows, int max_units, int heads, int run) {
        constexpr int kPer = 2;  // sequences per thread: two are enough from 256 threads on
        int key[kPer], rank[kPer];  // keys: longer first, then the order of the batch; 0 beyond the sequences
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int i = threadIdx.x + k * blockDim.x;
            key[k] = 0;
            if (i < n_seqs)
                key[k] = min(max(cu[i + 1] - cu[i] + unit_rows - 1, 0) / unit_rows, max_units) * kMaxListedSeqs + (kMaxListedSeqs - 1 - i);
            if (i < kMaxListedSeqs) first[i] = key[k];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int i = threadIdx.x + k * blockDim.x;
            rank[k] = 0;
            if (i < n_seqs)
                for (int o = 0; o < n_seqs; o += 4) {
                    const int4 v = *reinterpret_cast<const int4*>(first + o);
                    rank[k] += (v.x > key[k]) + (v.y > key[k]) + (v.z > key[k]) + (v.w > key[k]);
                }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int i = threadIdx.x + k * blockDim.x;
            if (i < n_seqs) {
                seq[rank[k]] = (unsigned short)i;
                if (rank[k] % run == 0) first[rank[k] / run + 1] = key[k] / kMaxListedSeqs * heads * min(run, n_seqs - rank[k]);
            }
        }
        if (threadIdx.x == 0) first[0] = 0;
        __syncthreads();
        if (threadIdx.x < 32) {  // running sums
            const int n_runs = (n_seqs + run - 1) / run;
            int carry = 0;
            for (int base = 1; base <= n_runs; base += 32) {
                const int i = base + (int)threadIdx.x;
                int v = i <= n_runs ? first[i] : 0;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const int o = __shfl_up_sync(0xffffffffu, v, off);
                    if ((int)threadIdx.x >= off) v += o;
                }
                v += carry;
                if (i <= n_runs) first[i] = v;
                carry = __shfl_sync(0xffffffffu, v, 31);
            }
        }
        __syncthreads();
    }
    // The run that item `idx` (below the number of items) belongs to.
    __device__ int run_of(int idx, int n_runs) const {
        int lo = 0, hi = n_runs;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (first[mid] <= idx) lo = mid;
            else hi = mid;
        }
        return lo;
    }
};

}  // namespace gqa
