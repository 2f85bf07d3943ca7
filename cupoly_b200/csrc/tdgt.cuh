// Host interface of the tensor-core DGT (tdgt.cu).
#pragma once
#include "engine.cuh"

namespace cpoly {

constexpr int kTdgtListMax = 4096;  // rows of a work list per launch (their order lives in shared memory)

// One transform of npolys x nres residues (see run_transform in dgt.cu), the element blocks of
// 2^tlayout.logNc elements on the tensor cores.  With tlayout.S > 0 the blocks are the 2^S
// parts that the split stage leaves, without a twist.
int launch_tdgt(const Engine& e, ulonglong2* data, const ulonglong2* fsrc, const InvSrc& isrc, int nres, int rid_off,
                int npolys, long long poly_stride, bool inverse, cudaStream_t st, const int* rid_list);

}  // namespace cpoly
