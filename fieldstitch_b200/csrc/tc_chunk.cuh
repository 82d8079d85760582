// Candidate chunks of the tensor-core matcher: runs of TC_CHUNK targets.
#pragma once

#ifndef FSB_HD
#ifdef __CUDACC__
#define FSB_HD __host__ __device__ __forceinline__
#else
#define FSB_HD inline
#endif
#endif

namespace fsb {

constexpr int TC_CHUNK = 16;   // columns per candidate chunk

// How many of chunk ch's columns exist among nb >= 1 targets: none for an empty record (negative) or for any
// other value that is no chunk of theirs. Records that a dense kernel which gave up on a wait left
// unwritten hold whatever was in that memory, so the product with TC_CHUNK is formed only once it fits.
FSB_HD int chunk_columns(int ch, int nb) {
    if (ch < 0 || ch > (nb - 1) / TC_CHUNK) return 0;
    const int left = nb - ch * TC_CHUNK;
    return left < TC_CHUNK ? left : TC_CHUNK;
}

}  // namespace fsb
