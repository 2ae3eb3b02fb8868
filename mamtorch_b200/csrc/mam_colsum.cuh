// Column sums of an fp32 matrix [M, N] (the bias gradient): out[n] = sum_m in[m][n].
//
// Bound by one read of the matrix.  torch's reduction over the outer dimension keeps too few loads in flight when N
// is small and M large: [401408, 128] takes it 211 us, 1.0 TB/s (this: 38 us, 5.5 TB/s).  Here 32 columns x 8 row lanes
// of a CTA read a slab of rows, each thread four rows apart in four accumulators, and a second launch adds the slabs'
// partial sums in the same manner: a fixed order, so two runs agree bit for bit.  An accumulator takes COLSUM_RUN
// additions in sequence before it is added to the thread's sum, which keeps long slabs exact ([401408, 1000], 21696 rows
// a slab: error 1.9e-7 against float64, torch 2.6e-7; without the runs, in slabs half as long, 3.3e-7).
// Four CTAs per SM with sixteen loads in flight a thread, all resident at once: 250 us there and 63 at [154303, 622];
// eight CTAs with eight loads 254 and 70, and where 1200 of them left sixteen for a second round 108.
#pragma once
#include <cuda_runtime.h>

namespace mamb200 {

constexpr int COLSUM_COLS = 32, COLSUM_LANES = 8, COLSUM_RUN = 16, COLSUM_CTAS = 4;

// grid (column groups, slabs): rows [slab*rows_per, +rows_per) into out[slab][n]
__global__ void __launch_bounds__(COLSUM_COLS * COLSUM_LANES, COLSUM_CTAS)
mam_colsum_kernel(const float* __restrict__ in, float* __restrict__ out, long long M, long long N,
                  long long rows_per) {
    __shared__ float part[COLSUM_LANES][COLSUM_COLS];
    const int c = threadIdx.x % COLSUM_COLS, l = threadIdx.x / COLSUM_COLS;
    const long long n = (long long)blockIdx.x * COLSUM_COLS + c;
    const long long m0 = (long long)blockIdx.y * rows_per, m1 = min(m0 + rows_per, M);
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    if (n < N) {
        long long m = m0 + l;
        for (; m + (4 * COLSUM_RUN - 1) * COLSUM_LANES < m1;) {
            float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
            for (int j = 0; j < COLSUM_RUN; ++j, m += 4 * COLSUM_LANES) {
#pragma unroll
                for (int i = 0; i < 4; ++i) t[i] += in[(m + i * COLSUM_LANES) * N + n];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) s[i] += t[i];
        }
#pragma unroll 2
        for (; m + 3 * COLSUM_LANES < m1; m += 4 * COLSUM_LANES) {
#pragma unroll
            for (int i = 0; i < 4; ++i) s[i] += in[(m + i * COLSUM_LANES) * N + n];
        }
        for (; m < m1; m += COLSUM_LANES) s[0] += in[m * N + n];
    }
    part[l][c] = (s[0] + s[1]) + (s[2] + s[3]);
    __syncthreads();
    if (l == 0 && n < N) {
        float t[COLSUM_LANES];
#pragma unroll
        for (int i = 0; i < COLSUM_LANES; ++i) t[i] = part[i][c];
        out[(long long)blockIdx.y * N + n] = ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
    }
}

}  // namespace mamb200
