// Host interface of the FP32 matching screened on the tensor cores
// (match_fp32_tc.cu).
#pragma once

#include <cuda_runtime.h>

namespace snapmrf {

struct ScreenRequest {
    float *maps;             // out [nvox][5]
    long long *index_out;    // optional out [nvox]
    const float2 *img;       // device [nvox][img_stride]
    long long img_stride;
    const float2 *atoms;     // device [NATOMS][atom_stride]
    long long atom_stride;
    const float *params;     // device [NATOMS][nparams]
    int nparams;
    long long nreps, NATOMS, natoms, nvox;
    int nblocks;
    const float *b1map;      // device [nvox] or null (one B1 value per block with it)
    bool imag;               // atoms purely imaginary
};

// Enqueues the call's matching on st and sets *done, or leaves *done false
// when the screen does not apply (no room for its operands, sizes past its
// index types): the caller then runs the FP32 kernel.
int match_fp32_screened(const ScreenRequest &q, cudaStream_t st, bool *done);

}  // namespace snapmrf
