// Host interface of the mixed-precision (tcgen05, int8-sliced) outgoing
// plane-wave pass, mixed.cu.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "plan.hpp"

namespace pdmk {

// particles per pipeline chunk of the mixed pass for n modes per axis half
int mixed_chunk(int nk);
// bytes of one chunk's table block (a multiple of 16)
int mixed_table_bytes(int nk);
// 2-D tensor map over the particle rows x, y, z, q (back to back, of an even
// stride), in boxes of kcp + 2 particles
void make_coord_map(CUtensorMap* map, const double* rows, int stride, int kcp);
// max |q| over n charges into *out (one block)
void launch_absmax(const double* sq, int n, double* out, cudaStream_t st);
// the mixed pass over device-resident lists: the table pass over nchunks
// (item, chunk) pairs into the items' chunk table blocks, then the
// contraction: the 128-row M tiles of each item, which share the
// item's blocks (ceil((s_end - s_begin) / chunk) of them); d_next: the counter
// the tiles are taken from, at zero
void dispatch_mixed(int nk, const CUtensorMap& tmap, const PwItem* d_items, int nitems, const int2* d_chunks,
                    int nchunks, int* d_next, const double* d_qmax, int* d_err, cudaStream_t st);

}  // namespace pdmk
