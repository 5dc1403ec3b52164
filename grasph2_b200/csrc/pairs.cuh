// pairs.cuh -- the all-pairs j-tile engine shared by the density, velocity-gradient, acceleration
// and gravity kernels.
//
// Replaces the reference's tile loop detail::do_for_each_pair_fast_impl
// (src/particles/algorithms.h:270-309) with:
//   * a 2-D grid: blockIdx.x = block of i-particles, blockIdx.y = segment of j-tiles (j-split),
//     so small N still fills 148 SMs and large N has no tail wave; each (i-block, segment)
//     writes its partial sums, which a finish kernel adds up in a fixed order (deterministic);
//   * j-tiles of `jt` particles staged in shared memory by 1-D bulk copies (cp.async.bulk, no
//     multicast), double-buffered against the i-loop and completed on mbarriers;
//   * arrays padded to a multiple of kPad with inert particles (zero mass, far away), so every tile
//     is full and the reference's remainder-tile bug (algorithms.h:285-301) cannot arise.
#pragma once

#include "common.cuh"
#include "spatial.cuh"

namespace gsph {

// Two-stage pipeline over the j-tiles [t_begin, t_end) of up to 4 float4 streams.
template <int NS>
struct JTilePipe {
    float4* buf;          // shared: [2][NS][jt]
    uint64_t* bar;        // shared: [2]
    const float4* src[NS];
    int jt;
    int64_t t_begin, t_end;  // tiles t_begin .. t_end-1
    int* status;

    __device__ __forceinline__ void issue(int b, int64_t t) {
        mbar_expect_tx(&bar[b], static_cast<uint32_t>(NS * jt * sizeof(float4)));
#pragma unroll
        for (int s = 0; s < NS; ++s)
            bulk_g2s(buf + (static_cast<int64_t>(b) * NS + s) * jt, src[s] + t * jt,
                     static_cast<uint32_t>(jt * sizeof(float4)), &bar[b]);
    }

    // init barriers and start the first two tiles; all threads must call it
    __device__ __forceinline__ void start() {
        if (threadIdx.x == 0) {
            mbar_init(&bar[0], 1);
            mbar_init(&bar[1], 1);
            fence_barrier_init();
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            if (t_begin < t_end) issue(0, t_begin);
            if (t_begin + 1 < t_end) issue(1, t_begin + 1);
        }
    }

    // for each tile: wait for it, run body(stage pointers), release the buffer and refill it
    template <typename Body>
    __device__ __forceinline__ void run(Body&& body) {
        int k = 0;
        for (int64_t t = t_begin; t < t_end; ++t, ++k) {
            const int b = k & 1;
            const bool ok = mbar_wait_bounded(&bar[b], static_cast<uint32_t>((k >> 1) & 1), status);
            if (__syncthreads_or(!ok)) {
                drain(k);
                return;
            }
            const float4* stage = buf + static_cast<int64_t>(b) * NS * jt;
            body(stage);
            __syncthreads();
            if (threadIdx.x == 0 && t + 2 < t_end) issue(b, t + 2);
        }
    }

    // after a timed-out wait: give copies still in flight a bounded time to land before exit
    __device__ __forceinline__ void drain(int k) {
        if (threadIdx.x == 0) {
            for (int extra = 0; extra < 2; ++extra) {
                const int kk = k + extra;
                const int64_t t = t_begin + kk;
                if (t >= t_end) break;
                mbar_wait_bounded(&bar[kk & 1], static_cast<uint32_t>((kk >> 1) & 1), status);
            }
        }
        __syncthreads();
    }
};

// ---- culled passes -------------------------------------------------------------------------------
// 32 consecutive particles at a time, lane l holds particle l. One pass finds the neighbours (four warps share its
// i-group's near chunks, half a chunk with a box of its own at a time) and stores their lists; the SPH passes walk
// them, one warp per 32 particles. No partial sums.
//
// Order of summation: the near chunks of a group form items of `per_item` chunks, an item's chunks form stages of
// kStageChunks. A particle's density is the sum over items of the sum over stages of the sum over neighbours (compensated:
// stages by two-sum, items in FP64); its SPH sums are the sum over items of the sum over neighbours (compensated: items in
// FP64, an item's neighbours in FP32 as in the plain form; in large contexts, from about 570,000 particles, an item can hold
// all of a group's near chunks, and the two forms are then one). It follows from the near chunks alone, not from the launch.
constexpr int kStageChunks = 4;
constexpr int kSub = 32;                 // particles per warp and per box
constexpr int kSubs = kGroup / kSub;
constexpr int kHalves = kChunk / kSub;   // boxes per chunk
constexpr int kItemsPerSM = 30;          // items aimed at in all (only the order of the SPH sums)

struct NearView {
    const int* list;     // near chunks of each i-group, row stride nchunks
    const int* count;
    const int* order;    // i-groups, the longest lists first; [ngroups]: chunks per item
    const float4 *lo, *hi;  // bounds of every 32 particles
    int ngroups;
    int64_t nchunks, n, n_pad;
    float hm2;           // (h (1 + kMargin))^2
    int* nb;             // neighbour lists [cap][n_pad]; the sign bit marks the first neighbour of an item ...
    int* nbcnt;          // ... and their lengths [n_pad]; more than cap: the list is incomplete
    int cap;
    __device__ __forceinline__ int group() const { return order[blockIdx.x / kSubs]; }
    __device__ __forceinline__ int64_t first(int g) const {
        return static_cast<int64_t>(g) * kGroup + (blockIdx.x % kSubs) * kSub;
    }
    __device__ __forceinline__ int per_item() const { return order[ngroups]; }
};
constexpr int kItemMark = static_cast<int>(0x80000000u);

// The near chunks of the 32 particles from s0 (group g): boxes farther than h (1 + kMargin) from the 32 particles' own
// box are skipped (32 of them per vote), the positions of the others go through the shared buffer `sh`, the next
// box's load in flight while one is tested, and body(mask, jb, c) gets each lane's mask of the neighbours (0 < r^2 <= H^2,
// bit k: particle jb + k, its record in sh[k]) and the chunk's place in the list.
template <typename Body>
__device__ __forceinline__ void near_scan(const NearView& v, const float4* posm, int g, int64_t s0,
                                          uint32_t span, float4 pi, float4* sh, Body&& body) {
    const int lane = threadIdx.x & 31;
    const float4 l = v.lo[s0 / kSub], u = v.hi[s0 / kSub];
    const int nh = v.count[g] * kHalves;
    const int* chunks = v.list + static_cast<int64_t>(g) * v.nchunks;
    for (int h0 = 0; h0 < nh; h0 += 32) {
        const int h = h0 + lane;
        int bx = 0;
        bool near = false;
        if (h < nh) {
            bx = chunks[h / kHalves] * kHalves + h % kHalves;
            const float4 bl = v.lo[bx], bu = v.hi[bx];
            const float gx = fmaxf(0.0f, fmaxf(bl.x - u.x, l.x - bu.x)), gy = fmaxf(0.0f, fmaxf(bl.y - u.y, l.y - bu.y)),
                        gz = fmaxf(0.0f, fmaxf(bl.z - u.z, l.z - bu.z));
            near = !(gx * gx + gy * gy + gz * gz > v.hm2);
        }
        unsigned todo = __ballot_sync(0xffffffffu, near);
        int jn = 0;
        float4 qn = make_float4(0, 0, 0, 0);
        if (todo) {
            jn = kSub * __shfl_sync(0xffffffffu, bx, __ffs(todo) - 1);
            qn = posm[jn + lane];
        }
        while (todo) {
            const int c = (h0 + __ffs(todo) - 1) / kHalves;
            todo &= todo - 1;
            const int jb = jn;
            const float4 q0 = qn;
            if (todo) {
                jn = kSub * __shfl_sync(0xffffffffu, bx, __ffs(todo) - 1);
                qn = posm[jn + lane];
            }
            __syncwarp();  // the previous box's reads are done
            sh[lane] = q0;
            __syncwarp();
            unsigned m4[4];  // four independent masks: no serial chain over the 32 tests
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                unsigned m = 0;
#pragma unroll
                for (int t = 0; t < 8; ++t) {
                    const float4 q = sh[8 * b + t];
                    const float dx = q.x - pi.x, dy = q.y - pi.y, dz = q.z - pi.z;
                    const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                    m |= static_cast<unsigned>((__float_as_uint(r2) - 1u) < span) << t;  // 0 < r2 <= H2
                }
                m4[b] = m;
            }
            body(m4[0] | (m4[1] << 8) | (m4[2] << 16) | (m4[3] << 24), jb, c);
        }
    }
}

// shared-memory bytes of a pipeline: 2 stages of NS streams plus the two barriers
__host__ __device__ inline size_t pipe_smem_bytes(int ns, int jt) {
    return static_cast<size_t>(2) * ns * jt * sizeof(float4) + 2 * sizeof(uint64_t);
}

// tile range of segment `seg` out of `nseg` over `ntiles` tiles (balanced to within one tile)
__device__ __forceinline__ void segment_tiles(int64_t ntiles, int seg, int nseg, int64_t& t0, int64_t& t1) {
    t0 = ntiles * seg / nseg;
    t1 = ntiles * (seg + 1) / nseg;
}

// ---- partial-sum fields of the SPH pair passes -----------------------------------------------
enum Field : int {
    F_GX = 0, F_GY, F_GZ,                    // gravity (G applied in the finish kernel)
    F_AX, F_AY, F_AZ,                        // stress + AV acceleration
    F_XV0, F_XV1, F_XV2,                     // XSPH
    F_E00, F_E11, F_E22, F_E01, F_E02, F_E12,  // strain rate (symmetric)
    F_W01, F_W02, F_W12,                     // rotation rate (antisymmetric)
    F_DIVV,                                  // velocity divergence
    F_C0, F_C1, F_C2,                        // velocity curl (fluid + Balsara)
    F_MAXV,                                  // max signal velocity (a max, not a sum)
    F_COUNT
};

enum Pass : int { PASS_VGRAD = 0, PASS_ACC = 1, PASS_FUSED = 2 };

template <int PASS, bool GRAV, bool SOLIDS>
__host__ __device__ constexpr uint32_t field_mask() {
    uint32_t m = 0;
    if (PASS != PASS_VGRAD) {
        m |= (1u << F_AX) | (1u << F_AY) | (1u << F_AZ) | (1u << F_XV0) | (1u << F_XV1) | (1u << F_XV2) |
             (1u << F_MAXV);
        if (GRAV) m |= (1u << F_GX) | (1u << F_GY) | (1u << F_GZ);
    }
    if (PASS != PASS_ACC) {
        m |= (1u << F_DIVV);
        if (SOLIDS)
            m |= (1u << F_E00) | (1u << F_E11) | (1u << F_E22) | (1u << F_E01) | (1u << F_E02) | (1u << F_E12) |
                 (1u << F_W01) | (1u << F_W02) | (1u << F_W12);
        else
            m |= (1u << F_C0) | (1u << F_C1) | (1u << F_C2);
    }
    return m;
}

__host__ __device__ constexpr int popc_c(uint32_t x) {  // no recursion: folds where the field is only known after unrolling
    x -= (x >> 1) & 0x55555555u;
    x = (x & 0x33333333u) + ((x >> 2) & 0x33333333u);
    return static_cast<int>((((x + (x >> 4)) & 0x0f0f0f0fu) * 0x01010101u) >> 24);
}

template <uint32_t MASK>
__host__ __device__ constexpr int field_offset(int f) {
    return popc_c(MASK & ((1u << f) - 1u));
}

// Optional event pair bracketing one pair-kernel launch (per-kernel timing, graph-capturable).
struct KTimer {
    cudaEvent_t start = nullptr, stop = nullptr;
};
cudaError_t timer_record(cudaEvent_t ev, cudaStream_t s);

// host launchers (pairs.cu)
// How the finish kernels read a particle's gravity partials: segments 0 .. nseg-1 of the one-sided
// kernel, or (sym_G > 0) the symmetric kernel's G + 1 slots, both [slot][component][particle].
struct GravSum {
    int nseg = 0;
    int sym_G = 0;
};

struct Launch {
    bool cull;       // SPH passes over near-chunk lists (spatial.cuh) + separate all-pairs gravity
    int threads;     // threads per CTA of the SPH pair kernels
    int jt;          // j-tile
    int nseg;        // j-split of the SPH pair kernels
    int grav_threads;
    int grav_ipt;    // i per thread of the gravity kernel
    int grav_jt;     // j-tile of the gravity kernel
    bool grav_x2;    // paired FP32 (f32x2) form of the gravity kernel
    int grav_nseg;
    int grav_sym_G = 0;   // > 0: symmetric gravity kernel over G groups of grav_sym_gs blocks
    int grav_sym_gs = 0;
    int grav_sym_shape = 0;  // block shape of the symmetric kernel (pairs.cu)
    int accum;       // GSPH_ACCUM_*
};

// the finish kernels' view of the gravity partials of launch shape L; nseg == 0: no gravity partials
inline GravSum grav_sum(const Launch& L, int nseg) {
    GravSum g;
    if (nseg <= 0) return g;
    if (L.grav_sym_G > 0) {
        g.sym_G = L.grav_sym_G;
    } else {
        g.nseg = nseg;
    }
    return g;
}
// groups of ceil(nblocks / target) blocks
inline void sym_groups(int64_t nblocks, int target, int& G, int& gs) {
    gs = static_cast<int>((nblocks + target - 1) / target);
    if (gs < 1) gs = 1;
    G = static_cast<int>((nblocks + gs - 1) / gs);
}
constexpr int kSymShapes = 4;
// the symmetric kernel's block shape and groups for n_pad particles (at most `groups`; 0: its own choice); with
// shape >= 0 that block shape
void sym_shape(int64_t n_pad, int sms, int groups, int shape, Launch& L);

// The density pass and the j-records of the new density. With `sp`: the neighbour search over the near chunks (with
// INTEGRATE_DENSITY the search alone), which stores the lists that the SPH passes of the step read.
cudaError_t launch_density(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s,
                           const KTimer* t = nullptr, const SpatialArrays* sp = nullptr);
// `early`: launched early (common.cuh) behind a kernel of the same step
cudaError_t launch_prepare(const DevArrays& a, const DevParams& p, cudaStream_t s, bool early = false);
// With `sp`, the SPH terms run over the neighbour lists of launch_density; the finish kernel then adds the gravity sums (a.gfold, from launch_gravity_partials), after waiting for
// `join` when it is given (the gravity kernel may run on another stream).
cudaError_t launch_pairs(int pass, const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s,
                         const KTimer* t = nullptr, const SpatialArrays* sp = nullptr, int gnseg = 0,
                         cudaEvent_t join = nullptr);
cudaError_t launch_gravity_partials(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s,
                                    const KTimer* t = nullptr);
cudaError_t launch_gravity(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s,
                           const KTimer* t = nullptr);
cudaError_t launch_fp32_peak(int sm_count, int iters, float* sink, cudaStream_t s);
cudaError_t launch_gravity_raw(const float4* posm_padded, float* part, int64_t n_pad, int ipt, int jt, int nseg,
                               float eps2, int* status, cudaStream_t s);
// the FP64 fold of `S` slots of a.gpart into a.gfold; far_G: groups of k_gravity_sym whose flags it asks (0: none)
cudaError_t launch_gravity_fold(const DevArrays& a, const Launch& L, int S, cudaStream_t s, bool early, int far_G = 0,
                                float eps2 = 0.0f);
int64_t fp32_peak_flops(int sm_count, int iters);

// the gravity partials and their fold with the kernels of the fixed order (gravity_fixed.cu)
cudaError_t launch_fixed_gravity(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s,
                                 const KTimer* t = nullptr);

size_t partial_floats(const DevParams& p, const Launch& L, int64_t n_pad);
size_t gravity_partial_floats(const Launch& L, int64_t n_pad);
int gravity_blocks_per_sm(int ipt, int threads, int jt, bool comp);

}  // namespace gsph
