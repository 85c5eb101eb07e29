// gmi_fx_kernels.hpp -- host interface of the fixed-point pair sums.
#pragma once

#include "gmi_context.hpp"

namespace gmi {

// One FP64-grade pair sum on caller-provided buffers: out (=|+=)
// sum_j M(i, j) F_j for targets [tgt_start, tgt_start + n_tgt).
struct FxPairSum {
    cudaStream_t stream;
    int sm_count;
    int kind;                      // kSS, kBB, kSB or kBS
    const double *xt;              // positions of the target set (AoS)
    int tgt_start, n_tgt;
    const double *xs, *fs;         // sources: positions, loads (6 values for kSS and kBS, else 3)
    int n_src;
    double as, ab, mu;             // segment and blob radius (equal kinds: the one radius twice)
    double *out;
    int accumulate;
    void *rec;                     // n_src records of fx_record_bytes(kind)
    double *partial;               // split partial sums
    size_t partial_bytes;          // bounds the number of splits
    unsigned *err;
    const int *skip;               // optional device flag: non-zero makes both kernels no-ops
    int *splits_out;               // optional: the caller adds the split partials (partial[p * 3 n_tgt + e],
                                   // p < *splits_out) itself; 1: the kernel wrote `out`
    int pdl;                       // the first kernel too may start while the previous one on the stream ends
    unsigned long long wait_ns;
    int max_splits;                // 0: no cap beyond the automatic choice
    bool staged;                   // out overlaps an input: it is written by a last kernel, from `partial` (one
                                   // split's place at least)
};

// Whether the formats hold this kind's radii (gmi_pairs_fx.cuh).
bool fx_supported(int kind, double as, double ab, double mu);
size_t fx_record_bytes(int kind);
// The source splits of the automatic choice (it sizes `partial`).
int fx_splits(int n_tgt, int n_src, int sm_count);
// Packs the sources and sums, in one to three launches (*launched counts them).
gmi_status launch_pair_fx(const FxPairSum &s, int *launched);

}  // namespace gmi
