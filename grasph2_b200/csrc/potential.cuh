// potential.cuh -- the FP64 pair potential sum_{i<j} m_i m_j / sqrt(r_ij^2 + eps^2) of the diagnostics.
//
// Row blocks of 128 I particles (I per thread, in registers) meet column blocks through shared memory. Row block a takes
// the column blocks a, a + 1, ... a + nb / 2 (mod nb), so every unordered pair of blocks is met once and every row
// block has the same work (a sweep over j > i gives the first block all of it and the last block none: 15 of 18 ms
// at N = 65,536 were spent waiting for the first blocks). Tasks of `chunk` consecutive offsets go round robin to a
// resident grid; a CTA keeps its sum in registers and leaves one partial, so the order of every sum is fixed.
//
// Bound: the FP64 pipe, 13 instructions per unordered pair (3 separation, 3 r^2 + eps^2, 5 x^(-1/2), mass, sum).
#pragma once

#include <algorithm>

#include "common.cuh"
#include "rsqrt64.cuh"

namespace gsph {

constexpr int kPotThreads = 128;
constexpr int kPotPerSM = 4;

// positions and masses of the two precisions
struct PotSource32 {
    const double* pos;  // [3][n_pad]
    const float4* posm;
    int64_t n_pad;
    __device__ __forceinline__ double4 at(int64_t i) const {
        return make_double4(pos[i], pos[n_pad + i], pos[2 * n_pad + i], static_cast<double>(posm[i].w));
    }
};
struct PotSource64 {
    const double4* posm;
    __device__ __forceinline__ double4 at(int64_t i) const { return posm[i]; }
};

template <typename Source, int I>
__global__ void __launch_bounds__(kPotThreads, kPotPerSM) k_pair_potential(Source src, int64_t n, int nb, int chunk, int ntasks,
                                                                double eps2, double* __restrict__ out) {
    constexpr int B = kPotThreads * I;
    __shared__ double2 Jxy[kPotThreads], Jzm[kPotThreads];
    __shared__ double red[kPotThreads / 32];
    const int tid = threadIdx.x;
    const int noff = nb / 2 + 1;  // offsets of a row block; for even nb the last one is met from the lower half only
    double total = 0.0;
    for (int t = blockIdx.x; t < ntasks; t += gridDim.x) {
        const int a = t % nb, d0 = t / nb * chunk, d1 = min(noff, d0 + chunk);
        double X[I], Y[I], Z[I], M[I], phi[I];
#pragma unroll
        for (int k = 0; k < I; ++k) {  // rows past the end: no mass, far away on the other side than the columns
            const int64_t i = static_cast<int64_t>(a) * B + k * kPotThreads + tid;
            const double4 q = i < n ? src.at(i) : make_double4(-1e18, -1e18, -1e18, 0.0);
            X[k] = q.x; Y[k] = q.y; Z[k] = q.z; M[k] = q.w;
            phi[k] = 0.0;
        }
        for (int d = d0; d < d1; ++d) {
            if (nb % 2 == 0 && d == nb / 2 && a >= nb / 2) continue;
            const int b = a + d < nb ? a + d : a + d - nb;
            for (int c = 0; c < I; ++c) {
                const int64_t j0 = static_cast<int64_t>(b) * B + c * kPotThreads;
                if (j0 >= n) break;
                const double4 q = j0 + tid < n ? src.at(j0 + tid) : make_double4(1e18, 1e18, 1e18, 0.0);
                __syncthreads();  // the previous tile's reads are done
                Jxy[tid] = make_double2(q.x, q.y);
                Jzm[tid] = make_double2(q.z, q.w);
                __syncthreads();
#pragma unroll 2
                for (int j = 0; j < kPotThreads; ++j) {
                    const double2 A = Jxy[j], Z2 = Jzm[j];
                    double x[I];
                    bool ok = true;
#pragma unroll
                    for (int k = 0; k < I; ++k) {
                        const double dx = A.x - X[k], dy = A.y - Y[k], dz = Z2.x - Z[k];
                        x[k] = fma(dz, dz, fma(dy, dy, fma(dx, dx, eps2)));
                        ok = ok && series_range64(x[k]);
                    }
                    if (ok) {
#pragma unroll
                        for (int k = 0; k < I; ++k) x[k] = Z2.y * inv_sqrt64(x[k]);
                    } else {
#pragma unroll
                        for (int k = 0; k < I; ++k) x[k] = Z2.y / sqrt(x[k]);
                    }
#pragma unroll
                    for (int k = 0; k < I; ++k)  // the block against itself: j > i
                        phi[k] += d > 0 || c * kPotThreads + j > k * kPotThreads + tid ? x[k] : 0.0;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < I; ++k) total = fma(M[k], phi[k], total);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    if ((tid & 31) == 0) red[tid >> 5] = total;
    __syncthreads();
    if (tid == 0) out[blockIdx.x] = (red[0] + red[1]) + (red[2] + red[3]);
}

// Fields 0 .. K-1 of `rows` rows of K block partials, one warp per field, and field 1 += scale * the sum of `npot`
// partials of the potential; out[k], in a fixed order.
template <int K>
__global__ void __launch_bounds__(32 * K) k_sum_partials(const double* __restrict__ part, int rows,
                                                         const double* __restrict__ pot, int npot, double scale,
                                                         double* __restrict__ out) {
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double s = 0.0;
#pragma unroll 4
    for (int r = lane; r < rows; r += 32) s += part[static_cast<int64_t>(r) * K + k];
    if (k == 1)
        for (int r = lane; r < npot; r += 32) s = fma(scale, pot[r], s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[k] = s;
}

inline int potential_sms() {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}
// partials of the potential (CTAs of its grid): at most this many for any n
inline int potential_partials() { return potential_sms() * kPotPerSM; }

// potential partials of n particles into out[0 .. grid); grid receives their number
template <typename Source>
cudaError_t launch_pair_potential(const Source& src, int64_t n, double eps2, double* out, int& grid, cudaStream_t s) {
    // I = 4 spends a quarter of the shared-memory reads of I = 1 per pair; smaller blocks where the pairs of 48
    // blocks would not fill the grid twice
    const int I = n >= kPotThreads * 4 * 48 ? 4 : (n >= kPotThreads * 2 * 48 ? 2 : 1);
    const int64_t B = static_cast<int64_t>(kPotThreads) * I;
    const int nb = static_cast<int>((n + B - 1) / B), noff = nb / 2 + 1;
    const int cap = potential_partials();
    const int chunk = static_cast<int>(std::max<int64_t>(1, static_cast<int64_t>(nb) * noff / (static_cast<int64_t>(cap) * 16)));
    const int64_t tasks = static_cast<int64_t>(nb) * ((noff + chunk - 1) / chunk);
    grid = static_cast<int>(std::min<int64_t>(tasks, cap));
    const int nt = static_cast<int>(tasks);
    switch (I) {
        case 1: k_pair_potential<Source, 1><<<grid, kPotThreads, 0, s>>>(src, n, nb, chunk, nt, eps2, out); break;
        case 2: k_pair_potential<Source, 2><<<grid, kPotThreads, 0, s>>>(src, n, nb, chunk, nt, eps2, out); break;
        default: k_pair_potential<Source, 4><<<grid, kPotThreads, 0, s>>>(src, n, nb, chunk, nt, eps2, out);
    }
    return cudaGetLastError();
}

}  // namespace gsph
