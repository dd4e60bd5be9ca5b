// The complex64 BLOCK8 parity launch (h3d_b8slab.cu), called by the batched sweep.
#pragma once

#include "h3d_b8.cuh"

namespace h3d {

// Block records of an operator (per 12^3 block: 1/||a||^2 and the wavenumber box): size and set-up.
// wnc: the records of a batch with any complex wavenumber hold complex boxes.
size_t slab_record_bytes(int NI, int NJ, int NK, bool wnc);
int launch_slab_pack(const Op<float> &op, bool adj, int NI, int NJ, int NK, bool wnc, float *rec, cudaStream_t st);

// One block parity of a table of problems: r right-hand sides per CTA (1 or 2), wnc when any
// problem has a complex wavenumber, dir 0 forward, 1 backward, 2 both passes.  one: host copy
// of the descriptor of a single problem (nprob = 1), passed as a kernel parameter.  chained: the launch before on the
// stream is another parity of the same sweep, whose tail this launch may overlap with the part of its
// prologue that reads set-up data only (the block records must be complete before that launch).
int launch_slab(int r, bool wnc, const B8Prob<float> &one, const B8Prob<float> *probs, const int *starts, int nprob, long long nctas,
                cplx<float> *x, const cplx<float> *b, float w, const int *active, int par, int dir,
                bool chained, cudaStream_t st);

}  // namespace h3d
