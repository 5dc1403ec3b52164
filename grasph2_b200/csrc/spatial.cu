// spatial.cu -- chunk bounding boxes, per-group near-chunk lists, and the Hilbert-curve reorder.
#include <algorithm>

#include <cub/device/device_radix_sort.cuh>

#include "spatial.cuh"

namespace gsph {

namespace {

inline unsigned blocks_for(int64_t n, int t) { return static_cast<unsigned>((n + t - 1) / t); }

// one warp per half chunk, two halves per chunk: min/max over the real particles (none: lo = +inf, hi = -inf)
static_assert(kChunk == 64, "two halves per chunk");
__global__ void __launch_bounds__(256) k_chunk_bounds(DevArrays a, SpatialArrays s, int64_t nsub) {
    __shared__ float4 box[8][2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t w = static_cast<int64_t>(blockIdx.x) * 8 + warp, i = w * 32 + lane;
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    wait_predecessor();
    if (i < a.n) {
        const float4 p = a.posm[i];
        mn[0] = mx[0] = p.x; mn[1] = mx[1] = p.y; mn[2] = mx[2] = p.z;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            mn[c] = fminf(mn[c], __shfl_xor_sync(0xffffffffu, mn[c], o));
            mx[c] = fmaxf(mx[c], __shfl_xor_sync(0xffffffffu, mx[c], o));
        }
    if (lane == 0) {
        box[warp][0] = make_float4(mn[0], mn[1], mn[2], 0.0f);
        box[warp][1] = make_float4(mx[0], mx[1], mx[2], 0.0f);
    }
    __syncthreads();
    if (lane != 0 || w >= nsub) return;
    const float4 l = box[warp][0], u = box[warp][1];
    s.sub_lo[w] = l;
    s.sub_hi[w] = u;
    if (warp & 1) return;
    const float4 m = box[warp + 1][0], v = box[warp + 1][1];
    s.box_lo[w / 2] = make_float4(fminf(l.x, m.x), fminf(l.y, m.y), fminf(l.z, m.z), 0.0f);
    s.box_hi[w / 2] = make_float4(fmaxf(u.x, v.x), fmaxf(u.y, v.y), fmaxf(u.z, v.z), 0.0f);
}

__device__ __forceinline__ float gap(float lo_a, float hi_a, float lo_b, float hi_b) {
    return fmaxf(0.0f, fmaxf(lo_b - hi_a, lo_a - hi_b));
}

// one warp per i-group: the ordered list of chunks within h of the group's box, 128 chunks per round
__global__ void __launch_bounds__(128) k_chunk_lists(const float4* lo, const float4* hi, int* list, int* count, int64_t ngroups,
                                                     int64_t nchunks, float h2m) {
    constexpr int per_group = kGroup / kChunk;
    wait_predecessor();
    const int lane = threadIdx.x & 31;
    const int64_t g = static_cast<int64_t>(blockIdx.x) * 4 + (threadIdx.x >> 5);
    if (g >= ngroups) return;
    float4 glo = lo[g * per_group], ghi = hi[g * per_group];
#pragma unroll
    for (int k = 1; k < per_group; ++k) {
        const float4 l = lo[g * per_group + k], u = hi[g * per_group + k];
        glo.x = fminf(glo.x, l.x); glo.y = fminf(glo.y, l.y); glo.z = fminf(glo.z, l.z);
        ghi.x = fmaxf(ghi.x, u.x); ghi.y = fmaxf(ghi.y, u.y); ghi.z = fmaxf(ghi.z, u.z);
    }
    int* out = list + g * nchunks;
    int n = 0;
    for (int64_t r = 0; r < nchunks; r += 128) {
        bool near[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int64_t c = r + 32 * k + lane;
            near[k] = false;
            if (c < nchunks) {
                const float4 l = lo[c], u = hi[c];
                const float dx = gap(glo.x, ghi.x, l.x, u.x), dy = gap(glo.y, ghi.y, l.y, u.y),
                            dz = gap(glo.z, ghi.z, l.z, u.z);
                near[k] = dx * dx + dy * dy + dz * dz <= h2m;
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned b = __ballot_sync(0xffffffffu, near[k]);
            if (near[k]) out[n + __popc(b & ((1u << lane) - 1u))] = static_cast<int>(r + 32 * k + lane);
            n += __popc(b);
        }
    }
    if (lane == 0) count[g] = n;
}

// The groups by falling near-chunk count (to a 256th of the largest), so that the warps of long lists start first and
// the short ones fill the last wave, and the chunks per item ceil(total near chunks / items), which sets the order of
// the SPH sums (pairs.cuh) and nothing else. One block: counting sort. The order within a bucket is not fixed, and need not be: every group's results are its own.
constexpr int kOrderThreads = 1024, kBuckets = 256;
__global__ void __launch_bounds__(kOrderThreads) k_group_order(const int* count, int* order,
                                                               int ngroups, int items) {
    __shared__ int most, bins[kBuckets], warp_sum[kBuckets / 32];
    __shared__ unsigned long long total;
    wait_predecessor();
    if (threadIdx.x == 0) {
        most = 1;
        total = 0;
    }
    if (threadIdx.x < kBuckets) bins[threadIdx.x] = 0;
    __syncthreads();
    int m = 0;
    unsigned long long sum = 0;
    for (int g = threadIdx.x; g < ngroups; g += kOrderThreads) {
        m = max(m, count[g]);
        sum += count[g];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&most, m);
        atomicAdd(&total, sum);
    }
    __syncthreads();
    if (threadIdx.x == 0) order[ngroups] = static_cast<int>(max(1ull, (total + items - 1) / items));
    const int top = most;
    auto bucket = [&](int g) {
        return kBuckets - 1 - static_cast<int>(static_cast<long long>(count[g]) * (kBuckets - 1) / top);
    };
    for (int g = threadIdx.x; g < ngroups; g += kOrderThreads) atomicAdd(&bins[bucket(g)], 1);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int v = 0, x = 0;
    if (threadIdx.x < kBuckets) {
        v = x = bins[threadIdx.x];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sum[warp] = x;
    }
    __syncthreads();
    if (threadIdx.x < kBuckets) {
        int before = x - v;
        for (int w = 0; w < warp; ++w) before += warp_sum[w];
        bins[threadIdx.x] = before;
    }
    __syncthreads();
    for (int g = threadIdx.x; g < ngroups; g += kOrderThreads) order[atomicAdd(&bins[bucket(g)], 1)] = g;
}

// ---- space-filling-curve reorder ----------------------------------------------------------------
__device__ __forceinline__ int f2o(float f) {  // float -> int with the same order
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float o2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

__global__ void k_bbox_init(int* bb) {
    if (threadIdx.x < 3) bb[threadIdx.x] = 0x7fffffff;
    else if (threadIdx.x < 6) bb[threadIdx.x] = static_cast<int>(0x80000000u);
}

__global__ void k_bbox(DevArrays a, int* bb) {
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < a.n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const float4 p = a.posm[i];
        const float v[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (isfinite(v[d])) {
                mn[d] = fminf(mn[d], v[d]);
                mx[d] = fmaxf(mx[d], v[d]);
            }
        }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mn[d] = fminf(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
            mx[d] = fmaxf(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(bb + d, f2o(mn[d]));
            atomicMax(bb + 3 + d, f2o(mx[d]));
        }
    }
}

__global__ void k_curve_keys(DevArrays a, const int* bb, unsigned* keys, int* vals) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n_pad) return;
    vals[i] = static_cast<int>(i);
    if (i >= a.n) {
        keys[i] = 0xffffffffu;  // padding stays behind every real particle
        return;
    }
    const float4 p = a.posm[i];
    const float v[3] = {p.x, p.y, p.z};
    unsigned q[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float lo = o2f(bb[d]), hi = o2f(bb[3 + d]);
        const float span = hi - lo;
        float t = (span > 0.0f && isfinite(v[d])) ? (v[d] - lo) / span : 0.0f;
        t = fminf(fmaxf(t, 0.0f), 1.0f);
        q[d] = static_cast<unsigned>(t * 1023.0f);
    }
    keys[i] = hilbert3(q[0], q[1], q[2]);
}

template <typename T>
__global__ void k_gather(const T* __restrict__ src, T* __restrict__ dst, const int* __restrict__ order, int64_t n) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[order[i]];
}

__global__ void k_iota(int* v, int64_t n) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) v[i] = static_cast<int>(i);
}

// All the arrays of a small context at once: gathered into scratch rows (BACK: copied from there), one array or group of
// arrays per blockIdx.y. With a gather and a copy per array, sixteen arrays of 4,096 particles took about 80 us of
// launches; from 65,536 particles on the copies themselves count and the rows would take 200 bytes per particle.
struct PermuteSet {
    float4* v4[10];
    double* v8;
    float *f0, *f1;
    int* ext;
};
template <bool BACK>
__global__ void __launch_bounds__(256) k_permute_all(PermuteSet s, float4* __restrict__ tmp, const int* __restrict__ order,
                                                     int64_t n) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int y = blockIdx.y;
    const int64_t o = BACK ? i : order[i];
    auto move = [&](auto* arr, auto* row) {
        if (BACK) arr[i] = row[i];
        else row[i] = arr[o];
    };
    if (y < 10) {
        float4* arr = s.v4[0];
#pragma unroll
        for (int k = 1; k < 10; ++k)
            if (y == k) arr = s.v4[k];
        move(arr, tmp + y * n);
    } else if (y == 10) {
        double* row = reinterpret_cast<double*>(tmp + 10 * n);
        for (int d = 0; d < 3; ++d) move(s.v8 + d * n, row + d * n);
    } else {
        float* row = reinterpret_cast<float*>(tmp + 12 * n);
        move(s.f0, row);
        move(s.f1, row + n);
        move(s.ext, reinterpret_cast<int*>(row + 2 * n));
    }
}

template <typename T>
cudaError_t permute(T* arr, T* tmp, const int* order, int64_t n, cudaStream_t st, int& launches) {
    k_gather<T><<<blocks_for(n, 256), 256, 0, st>>>(arr, tmp, order, n);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    ++launches;
    return cudaMemcpyAsync(arr, tmp, n * sizeof(T), cudaMemcpyDeviceToDevice, st);
}

}  // namespace

size_t spatial_sort_tmp_bytes(int64_t n_pad) {
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, bytes, static_cast<const unsigned*>(nullptr), static_cast<unsigned*>(nullptr),
                                    static_cast<const int*>(nullptr), static_cast<int*>(nullptr),
                                    static_cast<int>(n_pad));
    return bytes;
}

cudaError_t launch_chunk_bounds(const DevArrays& a, const SpatialArrays& s, cudaStream_t st) {
    const int64_t nsub = a.n_pad / 32;
    k_chunk_bounds<<<blocks_for(nsub, 8), 256, 0, st>>>(a, s, nsub);
    return cudaGetLastError();
}

cudaError_t launch_chunk_lists(const DevArrays& a, const SpatialArrays& s, float h, cudaStream_t st) {
    const int64_t nchunks = a.n_pad / kChunk, ngroups = a.n_pad / kGroup;
    const float hm = h * (1.0f + kMargin);
    return launch_kernel(true, k_chunk_lists, blocks_for(ngroups, 4), 128, st, s.box_lo, s.box_hi, s.list, s.count, ngroups,
                         nchunks, hm * hm);
}

cudaError_t launch_group_order(const DevArrays& a, const SpatialArrays& s, int items, cudaStream_t st) {
    return launch_kernel(true, k_group_order, 1, kOrderThreads, st, s.count, s.group_order,
                         static_cast<int>(a.n_pad / kGroup), items);
}

cudaError_t launch_identity_order(const SpatialArrays& s, int64_t n_pad, cudaStream_t st) {
    k_iota<<<blocks_for(n_pad, 256), 256, 0, st>>>(s.ext_of_int, n_pad);
    return cudaGetLastError();
}

cudaError_t curve_order(const DevArrays& a, const SpatialArrays& s, cudaStream_t st, int& launches) {
    const int64_t np = a.n_pad;
    k_bbox_init<<<1, 32, 0, st>>>(s.bbox);
    // four particles per thread, so that the warps' atomics stay few (256 CTAs on 4,096 particles took 10.4 us)
    k_bbox<<<std::min(256u, blocks_for(a.n, 1024)), 256, 0, st>>>(a, s.bbox);
    k_curve_keys<<<blocks_for(np, 256), 256, 0, st>>>(a, s.bbox, s.keys, s.order);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    launches += 3;
    size_t tb = s.sort_tmp_bytes;
    e = cub::DeviceRadixSort::SortPairs(s.sort_tmp, tb, s.keys, s.keys + np, s.order, s.order_out,
                                        static_cast<int>(np), 0, 32, st);
    if (e != cudaSuccess) return e;
    launches += 4;  // onesweep radix sort passes (approximate count for the launch counter)
    return e;
}

cudaError_t reorder_particles(const DevArrays& a, const SpatialArrays& s, cudaStream_t st, int& launches) {
    const cudaError_t e = curve_order(a, s, st, launches);
    if (e != cudaSuccess) return e;
    return permute_particles(a, s.order_out, s.tmp4, s.tmp8, s.ext_of_int, st, launches);
}

cudaError_t permute_particles(const DevArrays& a, const int* ord, float4* t4, double* t8, int* ext_of_int,
                              cudaStream_t st, int& launches) {
    const int64_t np = a.n_pad;
    cudaError_t e = cudaSuccess;
    if (permute_rows(np) > 1) {
        const PermuteSet set{{a.posm, a.velrho, a.acc, a.xvel, a.sA, a.sB, a.dA, a.dB, a.jA, a.jB},
                             a.pos64, a.rhodot, a.balsara, ext_of_int};
        const dim3 grid(blocks_for(np, 256), 12);
        k_permute_all<false><<<grid, 256, 0, st>>>(set, t4, ord, np);
        k_permute_all<true><<<grid, 256, 0, st>>>(set, t4, ord, np);
        launches += 2;
        return cudaGetLastError();
    }
    float4* f4s[] = {a.posm, a.velrho, a.acc, a.xvel, a.sA, a.sB, a.dA, a.dB, a.jA, a.jB};
    for (float4* arr : f4s) {
        e = permute(arr, t4, ord, np, st, launches);
        if (e != cudaSuccess) return e;
    }
    for (int d = 0; d < 3; ++d) {
        e = permute(a.pos64 + d * np, t8, ord, np, st, launches);
        if (e != cudaSuccess) return e;
    }
    float* tf = reinterpret_cast<float*>(t4);
    e = permute(a.rhodot, tf, ord, np, st, launches);
    if (e == cudaSuccess) e = permute(a.balsara, tf, ord, np, st, launches);
    if (e == cudaSuccess) e = permute(ext_of_int, reinterpret_cast<int*>(t4), ord, np, st, launches);
    return e;
}

}  // namespace gsph
