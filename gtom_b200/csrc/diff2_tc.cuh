// The two forms of the dense squared differences.
#pragma once

#include "common.cuh"

namespace gtomrln {

constexpr int kDiffTile = 64;  // references and shifts per tile of the direct kernel

// Direct kernel (estep.cu).  flags (device, one int per [particle][reference
// tile][shift tile], may be NULL): only the tiles whose flag is set.
int diff2_direct(const float2* particle, const float* minvsigma2, const float* ctf, int64_t elements,
                 const float2* shifts, const float2* refs, float* diff2, unsigned nparticles, unsigned nrefs,
                 unsigned nshifts, bool cc, const int* flags, cudaStream_t stream);

// On the tensor cores (diff2_tc.cu), the direct kernel for tiles with close
// matches.
int diff2_tensor(const float2* particle, const float* minvsigma2, const float* ctf, int64_t elements,
                 const float2* shifts, const float2* refs, float* diff2, unsigned nparticles, unsigned nrefs,
                 unsigned nshifts, bool cc, cudaStream_t stream);

}  // namespace gtomrln
