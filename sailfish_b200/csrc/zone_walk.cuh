// Row and column of the zones z0, z0 + step, z0 + 2 step, ... of a grid of nj
// columns, without a division per zone: a 64-bit one takes about a hundred
// instructions, more than the work of most zone-wise kernels. It pays with the
// zones a thread takes: reductions over 1153 x 1153 zones (nine a thread) 48 ->
// 39 us, passes of one or two zones a thread unchanged.
#pragma once

#include <cuda_runtime.h>

namespace cbd {

struct ZoneWalk {
    int i, j;

    __device__ __forceinline__ ZoneWalk(long z0, long step, int nj) : nj_(nj)
    {
        if ((unsigned long)(z0 | step) >> 32) {
            i = (int)(z0 / nj);
            di_ = (int)(step / nj);
        } else {
            i = (int)((unsigned)z0 / (unsigned)nj);
            di_ = (int)((unsigned)step / (unsigned)nj);
        }
        j = (int)(z0 - (long)i * nj);
        dj_ = (int)(step - (long)di_ * nj);
    }
    __device__ __forceinline__ void next()
    {
        i += di_;
        if (j >= nj_ - dj_) {
            j -= nj_ - dj_;
            ++i;
        } else {
            j += dj_;
        }
    }

private:
    int nj_, di_, dj_;
};

}  // namespace cbd
