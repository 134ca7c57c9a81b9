// gx_history.cuh -- per-epoch sums of the askAdam loss history.
//
// A kernel that keeps its voxels in registers over many epochs has, every
// epoch, NQ values a thread to add up over a volume.  A butterfly per epoch
// costs 5 shuffles and, with several warps, a block barrier; here a warp
// transposes instead: two epochs' values are merged by one exchange (half of
// the lanes keep the sum of the first, half of the second), two such pairs by
// the next, and after 32 epochs each lane holds one epoch's whole sum, so an
// epoch costs about one exchange, and every 32 epochs there is one barrier and
// one row of FP64 additions.  A lane adds the same pairs in the same tree as the
// butterfly (distances 16, 8, 4, 2, 1), so the warp sums are the same bit for bit.
#pragma once

#include "gx_internal.h"

namespace gx {

template <int NQ>
struct HistorySums {
    float pend[5][NQ];
    int n = 0;        // epochs taken
    int e0;           // first epoch of the launch
    double* buf;      // shared: [2][warps][32][NQ]
    double* hist;     // row of epoch 0 of the volume
    double scale0;    // of the first quantity

    // shared memory, in doubles, of `warps` warps: two halves, alternating by flush
    __host__ __device__ static constexpr int buf_doubles(int warps) { return 2 * warps * 32 * NQ; }

    __device__ __forceinline__ HistorySums(double* shared, double* hist_row0, double s0, int first_epoch)
        : e0(first_epoch), buf(shared), hist(hist_row0), scale0(s0) {
#pragma unroll
        for (int l = 0; l < 5; ++l)
#pragma unroll
            for (int q = 0; q < NQ; ++q) pend[l][q] = 0.0f;
    }

    // The values of the next epoch.  Called by whole blocks (a barrier every 32 epochs).
    __device__ __forceinline__ void add(const float (&v)[NQ], int last_epoch) {
        const int lane = threadIdx.x & 31;
        float r[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) r[q] = v[q];
        bool whole = true;
#pragma unroll
        for (int l = 0; l < 5; ++l) {
            if (whole) {
                if ((n >> l) & 1) {
                    const int d = 16 >> l;
                    const bool second = (lane & d) != 0;
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        const float keep = second ? r[q] : pend[l][q], send = second ? pend[l][q] : r[q];
                        r[q] = keep + __shfl_xor_sync(0xffffffffu, send, d);
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < NQ; ++q) pend[l][q] = r[q];
                    whole = false;
                }
            }
        }
        ++n;
        if (whole) flush(r, last_epoch);
    }

    // After the last epoch: the sums of an unfinished group.
    __device__ __forceinline__ void finish(int last_epoch) {
        const float zero[NQ] = {};
#pragma unroll 1
        while (n & 31) add(zero, last_epoch);
    }

private:
    __device__ __forceinline__ void flush(const float (&r)[NQ], int last_epoch) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
        // lane l holds the epoch whose index in the group is l with its 5 bits reversed
        const int e = e0 + n - 32 + (int)(__brev((unsigned int)lane) >> 27);
        double* b = buf + ((n >> 5) & 1) * nw * 32 * NQ;
        if (nw > 1) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) b[(warp * 32 + lane) * NQ + q] = (double)r[q];
            __syncthreads();
            // warps take the quantities in turn
            for (int q = warp; q < NQ; q += nw) {
                double t = 0.0;
                for (int w = 0; w < nw; ++w) t += b[(w * 32 + lane) * NQ + q];
                if (q == 0) t *= scale0;
                if (e <= last_epoch && t != 0.0) atomicAdd(hist + (size_t)e * kHistW + q, t);
            }
        } else {
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                double t = (double)r[q];
                if (q == 0) t *= scale0;
                if (e <= last_epoch && t != 0.0) atomicAdd(hist + (size_t)e * kHistW + q, t);
            }
        }
    }
};

}  // namespace gx
