// pairs.cu -- the all-pairs kernels of computeDerivatives (src/computeDerivatives.h:52-328).
//
//   k_density        calcDensity            (:52-91)    rho_i = sum_{0<r<=H} m_j W(r_ij)
//   k_pairs<VGRAD>   calcBalsaraDensityDTDStressDT (:96-162) strain/rotation rate, div v, curl
//   k_pairs<ACC>     calcAcceleration       (:167-313)  gravity + stress + AV (+XSPH, art. stress)
//   k_pairs<FUSED>   both in one pass, used whenever the acceleration does not need the Balsara
//                    values of the same step (the switch off): one N^2 sweep instead of two
//   k_gravity<I>     calcAcceleration with ENABLE_SPH off: register-blocked pure gravity
//   *_finish         sum the j-segment partials in a fixed order, then the per-particle epilogue
//                    (do_after of each job): density floor, Jaumann stress rate, drho/dt,
//                    Balsara switch, environment acceleration
//
// Arithmetic is FP32. GSPH_ACCUM_COMPENSATED accumulates each j-tile in FP32, folds the tile
// partial into a (sum, error) pair with a two-sum, and combines the j-segments in FP64.
#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "f32x2.cuh"
#include "gravity_sym.cuh"
#include "pairs.cuh"
#include "sph.cuh"

namespace gsph {

namespace {

// ================================================================================================
// density
// ================================================================================================
// The partial sums of particle i: j-segments [seg][field][n_pad] (the culled pass: one); KK = fields per slot (2K
// with compensation terms).
struct PartView {
    const float* part;
    int64_t n_pad;
    int nseg;
    int KK;
    bool err;  // compensation terms stored after the K sums (all-pairs segments, compensated)
    __device__ __forceinline__ float at(int slot, int o, int64_t i) const {
        return part[(static_cast<int64_t>(slot) * KK + o) * n_pad + i];
    }
};

// one tile of the density sum: rho += m_j W~(q) over 0 < r^2 <= H^2 (self term excluded), the
// spline prefactor applied by the finish kernel
__device__ __forceinline__ float density_tile(const float4* __restrict__ J, int nj, float4 pi, uint32_t span,
                                              float inv_h) {
    float rho = 0.0f;
#pragma unroll 8
    for (int j = 0; j < nj; ++j) {
        const float4 q = J[j];
        const float dx = q.x - pi.x, dy = q.y - pi.y, dz = q.z - pi.z;
        const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        if (in_open_closed(r2, 0u, span)) {  // calcDensity: r2 <= H2 && r2 > 0 (computeDerivatives.h:72)
            const float r = r2 * rsqrtf(r2);
            rho = fmaf(q.w, w_poly(r * inv_h), rho);
        }
    }
    return rho;
}

// all-pairs density sum: blockIdx.x = i-block, blockIdx.y = j-segment
template <bool COMP>
__global__ void __launch_bounds__(256) k_density(const float4* __restrict__ posm, float* __restrict__ part,
                                                  int64_t n_pad, int jt, int nseg, DevParams p, int* status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    JTilePipe<1> pipe;
    pipe.buf = reinterpret_cast<float4*>(smem_raw);
    pipe.bar = reinterpret_cast<uint64_t*>(smem_raw + 2 * jt * sizeof(float4));
    pipe.src[0] = posm;
    pipe.jt = jt;
    pipe.status = status;
    segment_tiles(n_pad / jt, blockIdx.y, nseg, pipe.t_begin, pipe.t_end);
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const float4 pi = posm[i];
    const uint32_t span = __float_as_uint(p.H2);
    float rho_s = 0.0f, rho_c = 0.0f;
    pipe.start();
    pipe.run([&](const float4* J) {
        const float t = density_tile(J, jt, pi, span, p.inv_h);
        if (COMP) fold(rho_s, rho_c, t);
        else rho_s += t;
    });
    const int64_t seg = blockIdx.y;
    part[(seg * (COMP ? 2 : 1)) * n_pad + i] = rho_s;
    if (COMP) part[(seg * 2 + 1) * n_pad + i] = rho_c;
}

// The neighbour search of 32 particles by W warps, with the density sum and its epilogue (DENS) or without (the
// density is integrated). The group's near chunks come in batches of up to 64, cut at a stage. A: the batch's boxes are
// tested against the 32 particles' own, 32 per warp. B: warp w takes the stages w, w + W, ...; the positions of a near
// box go through the warp's shared buffer, every lane gets the mask of its neighbours (0 < r^2 <= H^2) and adds
// their terms to the stage's sum. C: with the counts of all stages known, each warp writes its stages' neighbours to
// their places in the particle's list, and warp 0 adds the stage sums in their order.
//
// Bound: instruction issue (8 per test, about 2 % of the tests are neighbours). One warp alone took 154 us for 65,536
// particles of the impact and 29 us for the 4,096 of the fluid, whose 128 warps leave the chip idle. Eight warps help
// the search alone in few groups (a rubble step with 16,384 particles 178.7 -> 174.7 us, with 4,000 73.3 -> 66.7), not the
// search with the density sum (71.6 us for 68.5 in the fluid's step: the walk over the stages is each warp's own).
constexpr int kBatch = 64;
template <int W, bool DENS, bool COMP>
__global__ void __launch_bounds__(kSub * W) k_near(const float4* posm, float4* velrho,
                                                            DevParams p, NearView v) {
    __shared__ float4 sh[W][kSub];
    __shared__ unsigned mk[kBatch * kHalves][kSub];   // neighbour masks of the batch's boxes
    __shared__ float ts[DENS ? kBatch : 1][kSub];     // stage sums
    __shared__ unsigned short cs[kBatch][kSub];       // neighbours per stage
    __shared__ int bxs[kBatch * kHalves];
    __shared__ unsigned nm[kBatch * kHalves / 32];    // which boxes are near
    constexpr int kVotes = kBatch * kHalves / 32;  // one vote per batch in each of the first warps
    static_assert(kVotes <= W, "one vote per warp and batch");
    wait_predecessor();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = v.group(), ic = v.per_item(), nc = v.count[g];
    const int64_t s0 = v.first(g), i = s0 + lane;
    if (s0 >= v.n) return;
    const float4 pi = posm[i];
    const float4 l = v.lo[s0 / kSub], u = v.hi[s0 / kSub];
    const int* chunks = v.list + static_cast<int64_t>(g) * v.nchunks;
    const uint32_t span = __float_as_uint(p.H2);
    // stages of [c0, c1), item ends at `ie`: f(q, first chunk, end chunk, item ends with it)
    auto stages = [&](int c0, int c1, int ie, auto&& f) {
        for (int q = 0, b = c0; b < c1; ++q) {
            const int e = min(b + kStageChunks, min(ie, c1));
            f(q, b - c0, e - c0, e == ie);
            if (e == ie) ie += ic;
            b = e;
        }
        return ie;
    };
    int cnt = 0;                                 // neighbours so far
    bool seen = false;                           // ... any of them of the current item
    float rs = 0.0f, rc = 0.0f, tot = 0.0f;      // sums of the item (and its error term) and of the items before it
    double tot2 = 0.0;
    auto end_item = [&]() {
        if (COMP) tot2 += static_cast<double>(rs) + static_cast<double>(rc);
        else tot += rs;
        rs = rc = 0.0f;
    };
    int ie = ic;  // end of the item that holds c0
    for (int c0 = 0; c0 < nc;) {
        int c1 = min(nc, c0 + kBatch);
        if (c1 < nc) c1 -= c1 % ic % kStageChunks;  // whole stages
        if (warp < kVotes) {  // A
            const int h = threadIdx.x;
            int bx = 0;
            bool near = false;
            if (h < (c1 - c0) * kHalves) {
                bx = chunks[c0 + h / kHalves] * kHalves + h % kHalves;
                const float4 bl = v.lo[bx], bu = v.hi[bx];
                const float gx = fmaxf(0.0f, fmaxf(bl.x - u.x, l.x - bu.x)), gy = fmaxf(0.0f, fmaxf(bl.y - u.y, l.y - bu.y)),
                            gz = fmaxf(0.0f, fmaxf(bl.z - u.z, l.z - bu.z));
                near = !(gx * gx + gy * gy + gz * gz > v.hm2);
            }
            bxs[h] = bx;
            const unsigned b = __ballot_sync(0xffffffffu, near);
            if (lane == 0) nm[warp] = b;
        }
        __syncthreads();
        // B
        stages(c0, c1, ie, [&](int q, int b, int e, bool) {
            if (q % W != warp) return;
            float t = 0.0f;
            int n = 0;
            for (int h = b * kHalves; h < e * kHalves; ++h) {
                if (!(nm[h >> 5] >> (h & 31) & 1u)) continue;
                const float4 q0 = posm[bxs[h] * kSub + lane];
                __syncwarp();  // the previous box's reads are done
                sh[warp][lane] = q0;
                __syncwarp();
                unsigned m4[4];  // four independent masks: no serial chain over the 32 tests
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    unsigned m = 0;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const float4 r = sh[warp][8 * w + k];
                        const float dx = r.x - pi.x, dy = r.y - pi.y, dz = r.z - pi.z;
                        const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                        m |= static_cast<unsigned>((__float_as_uint(r2) - 1u) < span) << k;  // 0 < r2 <= H2
                    }
                    m4[w] = m;
                }
                unsigned m = m4[0] | (m4[1] << 8) | (m4[2] << 16) | (m4[3] << 24);
                mk[h][lane] = m;
                n += __popc(m);
                if (DENS) {
                    while (m) {
                        const float4 r = sh[warp][__ffs(m) - 1];
                        m &= m - 1;
                        const float dx = r.x - pi.x, dy = r.y - pi.y, dz = r.z - pi.z;
                        const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                        const float d = r2 * rsqrtf(r2);
                        t = fmaf(r.w, w_poly(d * p.inv_h), t);
                    }
                }
            }
            cs[q][lane] = static_cast<unsigned short>(n);
            if (DENS) ts[DENS ? q : 0][lane] = t;
        });
        __syncthreads();
        // C
        ie = stages(c0, c1, ie, [&](int q, int b, int e, bool item_ends) {
            const int n = cs[q][lane];
            if (q % W == warp && __any_sync(0xffffffffu, n > 0)) {
                int at = cnt;
                bool first = !seen;
                for (int h = b * kHalves; h < e * kHalves; ++h) {
                    if (!(nm[h >> 5] >> (h & 31) & 1u)) continue;
                    unsigned m = mk[h][lane];
                    const int jb = bxs[h] * kSub;
                    while (m) {
                        const int j = jb + __ffs(m) - 1;
                        m &= m - 1;
                        if (at < v.cap) v.nb[static_cast<int64_t>(at) * v.n_pad + i] = j | (first ? kItemMark : 0);
                        first = false;
                        ++at;
                    }
                }
            }
            cnt += n;
            seen = !item_ends && (seen || n > 0);
            if (DENS && warp == 0) {
                if (COMP) fold(rs, rc, ts[DENS ? q : 0][lane]);
                else rs += ts[DENS ? q : 0][lane];
                if (item_ends) end_item();
            }
        });
        __syncthreads();  // before the next batch
        c0 = c1;
    }
    if (warp != 0) return;
    v.nbcnt[i] = cnt;
    if (!DENS || i >= v.n) return;
    end_item();
    float rho = COMP ? static_cast<float>(tot2 * static_cast<double>(p.w_pref)) : tot * p.w_pref;
    if (has(p, GSPH_DEAL_WITH_NO_PARTNERS) && rho < 0.001f) rho = p.rho0 * 0.01f;  // computeDerivatives.h:85-88
    reinterpret_cast<float*>(velrho + i)[3] = rho;
}

// sum the slots, apply the prefactor and the optional floor (computeDerivatives.h:85-88), then
// build the j-record sigma/rho^2 of the new density
template <bool COMP>
__global__ void k_density_finish(DevArrays a, DevParams p, PartView pv) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    float rho;
    if (COMP) {
        double s = 0.0;
        for (int k = 0; k < pv.nseg; ++k) s += static_cast<double>(pv.at(k, 0, i)) + static_cast<double>(pv.at(k, 1, i));
        rho = static_cast<float>(s * static_cast<double>(p.w_pref));
    } else {
        float s = 0.0f;
        for (int k = 0; k < pv.nseg; ++k) s += pv.at(k, 0, i);
        rho = s * p.w_pref;
    }
    if (has(p, GSPH_DEAL_WITH_NO_PARTNERS) && rho < 0.001f) rho = p.rho0 * 0.01f;
    float4 vr = a.velrho[i];
    vr.w = rho;
    a.velrho[i] = vr;
    float4 jA, jB;
    make_jrecord(p, rho, a.sA[i], a.sB[i], a.balsara[i], jA, jB);
    a.jA[i] = jA;
    a.jB[i] = jB;
    if (a.jrec) {
        float4* r = a.jrec + 4 * i;
        r[0] = a.posm[i]; r[1] = vr; r[2] = jA; r[3] = jB;
    }
}

// j-records from the current density
__global__ void k_prepare(DevArrays a, DevParams p) {
    wait_predecessor();
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const float4 vr = a.velrho[i];
    float4 jA, jB;
    make_jrecord(p, vr.w, a.sA[i], a.sB[i], a.balsara[i], jA, jB);
    a.jA[i] = jA;
    a.jB[i] = jB;
    if (a.jrec) {
        float4* r = a.jrec + 4 * i;
        r[0] = a.posm[i]; r[1] = vr; r[2] = jA; r[3] = jB;
    }
}

// ================================================================================================
// SPH pair passes
// ================================================================================================
// The all-pairs body over nj staged j-records (P: posm, V: velrho, JA/JB: sigma/rho^2): gravity when
// GRAV != 0 (computeDerivatives.h:229-235, G applied by the finish kernel), then the SPH terms of
// every neighbour. GRAV: 0 off, 1 softened (eps > 0), 2 unsoftened (eps == 0: self pair gives 0).
template <int PASS, int GRAV, bool SOLIDS>
__device__ __forceinline__ void pair_tile(PairAcc& T, float& maxv, const ISph& I, const float4* __restrict__ P,
                                          const float4* __restrict__ V, const float4* __restrict__ JA,
                                          const float4* __restrict__ JB, int nj, const DevParams& p) {
    constexpr bool DO_A = PASS != PASS_VGRAD;
    const float eps2 = I.eps2;
#pragma unroll 4
    for (int j = 0; j < nj; ++j) {
        const float4 q = P[j];
        const float dx = q.x - I.pi.x, dy = q.y - I.pi.y, dz = q.z - I.pi.z;  // d = x_j - x_i = -r_ij
        const float r2e = fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, eps2)));
        if (GRAV != 0) {
            float inv = rsqrtf(r2e);
            if (GRAV == 2) inv = fminf(inv, 1e12f);
            const float s = q.w * inv * (inv * inv);
            T.f[F_GX] = fmaf(dx, s, T.f[F_GX]);
            T.f[F_GY] = fmaf(dy, s, T.f[F_GY]);
            T.f[F_GZ] = fmaf(dz, s, T.f[F_GZ]);
        }
        if (in_open_closed(r2e, I.lo, I.span))  // 0 < r2 <= H2
            sph_neighbour<PASS, SOLIDS>(T, maxv, I, q.w, dx, dy, dz, r2e - eps2, V[j],
                                        DO_A ? JA[j] : make_float4(0, 0, 0, 0), DO_A ? JB[j] : make_float4(0, 0, 0, 0),
                                        p);
    }
}

template <uint32_t MASK, bool COMP>
__device__ __forceinline__ void fold_tile(PairAcc& S, PairAcc& C, const PairAcc& T) {
#pragma unroll
    for (int f = 0; f < F_COUNT; ++f) {
        if (!((MASK >> f) & 1u) || f == F_MAXV) continue;
        if (COMP) fold(S.f[f], C.f[f], T.f[f]);
        else S.f[f] += T.f[f];
    }
}

// store one thread's partial sums: field o at out[o * stride] (sums) and out[(K + o) * stride]
// (compensation terms)
template <uint32_t MASK, bool COMP>
__device__ __forceinline__ void store_partials(float* out, int64_t stride, const PairAcc& S, const PairAcc& C,
                                               float maxv) {
    constexpr int K = popc_c(MASK);
#pragma unroll
    for (int f = 0; f < F_COUNT; ++f) {
        if (!((MASK >> f) & 1u)) continue;
        const int o = field_offset<MASK>(f);
        out[o * stride] = (f == F_MAXV) ? maxv : S.f[f];
        if (COMP) out[(K + o) * stride] = (f == F_MAXV) ? 0.0f : C.f[f];
    }
}

// All-pairs SPH pass: blockIdx.x = i-block, blockIdx.y = j-segment (partials [seg][field][n_pad]).
template <int PASS, int GRAV, bool SOLIDS, bool COMP>
__global__ void __launch_bounds__(256) k_pairs(DevArrays a, DevParams p, int jt, int nseg) {
    constexpr uint32_t MASK = field_mask<PASS, (GRAV != 0), SOLIDS>();
    constexpr int K = popc_c(MASK);
    constexpr int NS = (PASS == PASS_VGRAD) ? 2 : 4;

    extern __shared__ __align__(16) unsigned char smem_raw[];
    JTilePipe<NS> pipe;
    pipe.buf = reinterpret_cast<float4*>(smem_raw);
    pipe.bar = reinterpret_cast<uint64_t*>(smem_raw + 2 * NS * jt * sizeof(float4));
    pipe.src[0] = a.posm;
    pipe.src[1] = a.velrho;
    if constexpr (NS == 4) {
        pipe.src[2] = a.jA;
        pipe.src[3] = a.jB;
    }
    pipe.jt = jt;
    pipe.status = a.status;
    segment_tiles(a.n_pad / jt, blockIdx.y, nseg, pipe.t_begin, pipe.t_end);

    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const ISph I = load_isph<PASS, SOLIDS>(a, p, i, (GRAV == 1) ? p.eps2 : 0.0f);
    PairAcc S, C;
#pragma unroll
    for (int f = 0; f < F_COUNT; ++f) S.f[f] = C.f[f] = 0.0f;
    float maxv = 0.0f;

    pipe.start();
    pipe.run([&](const float4* stage) {
        PairAcc T;
#pragma unroll
        for (int f = 0; f < F_COUNT; ++f) T.f[f] = 0.0f;
        pair_tile<PASS, GRAV, SOLIDS>(T, maxv, I, stage, stage + jt, stage + 2 * jt, stage + 3 * jt, jt, p);
        fold_tile<MASK, COMP>(S, C, T);
    });
    store_partials<MASK, COMP>(a.part + static_cast<int64_t>(blockIdx.y) * (COMP ? 2 * K : K) * a.n_pad + i, a.n_pad,
                               S, C, maxv);
}

// Culled SPH pass (no gravity) over the neighbour lists, one warp per 32 particles: one packed 64-byte record per
// neighbour, the next record and the index after it in flight. A warp with an incomplete list goes back to the boxes.
//
// Bound: instruction issue and the L2 latency of the gathers. A lane goes through all its neighbours and adds an item's
// sums when its next neighbour belongs to another one, so a warp runs as long as its longest list (a warp per
// item of a few chunks kept 18.8 of 32 lanes active and left the items' partial sums to the finish kernel).
// In few groups there is one warp to a scheduler at most, and the chain of one neighbour's arithmetic behind another's is
// what it waits for. There the records of D = 4 neighbours are in flight (a rubble step with 16,384 particles 199 -> 194
// us), and the fused pass goes to two warps, one for the velocity gradient (PART 1) and one for the acceleration (PART 2):
// 208 -> 190 us for a step of the impact with 16,384 particles, 115 -> 98 with 4,000.
// a record of the kernel before (common.cuh), loaded where it is written: left to the compiler, plain loads of the next
// neighbours move down to their use (a rubble step with 5,000 particles 75.7 -> 81.3 us)
__device__ __forceinline__ float4 load_here(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
template <int PASS, bool SOLIDS, bool COMP, int D, int PART>
__device__ __forceinline__ void pairs_near(const DevArrays& a, const DevParams& p, const NearView& v) {
    constexpr uint32_t ALL = field_mask<PASS, false, SOLIDS>(), FIRST = field_mask<PASS_VGRAD, false, SOLIDS>();
    constexpr uint32_t MASK = PART == 0 ? ALL : (PART == 1 ? ALL & FIRST : ALL & ~FIRST);
    constexpr bool DO_A = PASS != PASS_VGRAD && PART != 1;
    using Sum = typename std::conditional<COMP, double, float>::type;
    __shared__ float4 sh[kSub];
    const int g = v.group(), ic = v.per_item();
    const int64_t s0 = v.first(g), i = s0 + threadIdx.x;
    if (s0 >= v.n) return;
    const ISph I = load_isph<PASS, SOLIDS>(a, p, i, 0.0f);
    const int* lst = v.nb + i;
    const int cnt = v.nbcnt[i];
    PairAcc T;                // the sums of the item
    Sum S[F_COUNT];           // ... and of the items before it
#pragma unroll
    for (int f = 0; f < F_COUNT; ++f) {
        T.f[f] = 0.0f;
        S[f] = 0;
    }
    float maxv = 0.0f;
    const float4 zero = make_float4(0, 0, 0, 0);
    auto end_item = [&]() {
#pragma unroll
        for (int f = 0; f < F_COUNT; ++f)
            if (((MASK >> f) & 1u) && f != F_MAXV) {
                S[f] += static_cast<Sum>(T.f[f]);
                T.f[f] = 0.0f;
            }
    };
    auto term = [&](float4 q, float4 vj, float4 ja, float4 jb) {
        const float dx = q.x - I.pi.x, dy = q.y - I.pi.y, dz = q.z - I.pi.z;
        const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        sph_neighbour<PASS, SOLIDS, PART>(T, maxv, I, q.w, dx, dy, dz, r2, vj, ja, jb, p);
    };
    if (!__any_sync(0xffffffffu, cnt > v.cap)) {
        int e[D] = {}, en[D] = {};  // the entries of the next D neighbours, and of the D after them
        float4 rec[D][4];
        auto load = [&](int d) {
            const float4* r = a.jrec + 4 * static_cast<int64_t>(e[d] & ~kItemMark);
            rec[d][0] = load_here(r);
            rec[d][1] = load_here(r + 1);
            rec[d][2] = DO_A ? load_here(r + 2) : zero;
            rec[d][3] = DO_A ? load_here(r + 3) : zero;
        };
#pragma unroll
        for (int d = 0; d < D; ++d) {
            e[d] = d < cnt ? lst[static_cast<int64_t>(d) * v.n_pad] : 0;
            en[d] = D + d < cnt ? lst[static_cast<int64_t>(D + d) * v.n_pad] : 0;
        }
#pragma unroll
        for (int d = 0; d < D; ++d) load(d);
        for (int k0 = 0; k0 < cnt; k0 += D) {
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const int k = k0 + d;
                if (k >= cnt) break;
                const float4 q = rec[d][0], vj = rec[d][1], ja = rec[d][2], jb = rec[d][3];
                const bool first = e[d] < 0;
                e[d] = en[d];
                if (k + D < cnt) load(d);
                if (k + 2 * D < cnt) en[d] = lst[static_cast<int64_t>(k + 2 * D) * v.n_pad];
                if (first) end_item();
                term(q, vj, ja, jb);
            }
        }
    } else {
        int item = 0, next = ic, last = -1;
        near_scan(v, a.posm, g, s0, I.span, I.pi, sh, [&](unsigned m, int jb, int c) {
            while (c >= next) {
                ++item;
                next += ic;
            }
            while (m) {
                const float4* r = a.jrec + 4 * static_cast<int64_t>(jb + __ffs(m) - 1);
                m &= m - 1;
                if (item != last) end_item();
                last = item;
                term(r[0], r[1], DO_A ? r[2] : zero, DO_A ? r[3] : zero);
            }
        });
    }
    end_item();
#pragma unroll
    for (int f = 0; f < F_COUNT; ++f)
        if ((MASK >> f) & 1u)
            a.part[static_cast<int64_t>(field_offset<ALL>(f)) * a.n_pad + i] = f == F_MAXV ? maxv : static_cast<float>(S[f]);
}

template <int PASS, bool SOLIDS, bool COMP, int D>
__global__ void __launch_bounds__(kSub) k_pairs_near(DevArrays a, DevParams p, NearView v) {
    wait_predecessor();
    pairs_near<PASS, SOLIDS, COMP, D, 0>(a, p, v);
}
template <bool SOLIDS, bool COMP>
__global__ void __launch_bounds__(kSub) k_pairs_near_split(DevArrays a, DevParams p, NearView v) {
    wait_predecessor();
    if (blockIdx.y == 0) pairs_near<PASS_FUSED, SOLIDS, COMP, 1, 2>(a, p, v);
    else pairs_near<PASS_FUSED, SOLIDS, COMP, 1, 1>(a, p, v);
}

// Sum the slots of one field in a fixed order: FP32 in plain mode, FP64 of (sum + error) in
// compensated mode. The max signal velocity is a max over slots.
template <uint32_t MASK, bool COMP>
__device__ __forceinline__ float seg_sum(const PartView& v, int64_t i, int f) {
    constexpr int K = popc_c(MASK);
    const int o = field_offset<MASK>(f);
    if (f == F_MAXV) {
        float m = 0.0f;
        for (int k = 0; k < v.nseg; ++k) m = fmaxf(m, v.at(k, o, i));
        return m;
    }
    if (COMP) {
        double s = 0.0;
        for (int k = 0; k < v.nseg; ++k) {
            s += static_cast<double>(v.at(k, o, i));
            if (v.err) s += static_cast<double>(v.at(k, K + o, i));
        }
        return static_cast<float>(s);
    }
    float s = 0.0f;
    for (int k = 0; k < v.nseg; ++k) s += v.at(k, o, i);
    return s;
}

// ---- the FP64 fold of the gravity partials ---------------------------------------------------------
// Both all-pairs gravity kernels leave per-particle partial sums [slot][component][n_pad]: the one-sided
// kernel's j-segments, or the symmetric kernel's G + 1 slots (its row and column sums, each written by
// one task). 32 particles per CTA: warp q sums the slots [q R, (q + 1) R) in FP64 (with the error terms of
// the compensated form), then the runs are added in the order q = 0, 1, 2, 3 -- a fixed order, so results
// are deterministic.
//
// Bound: the latency of the loads in small contexts, so all 17 slots of a run of 65 are in flight at once; DRAM in large ones, where a
// thread takes V = 4 particles in 16-byte loads. Measured (cold caches; before, with eight particles per warp and 32
// contiguous bytes): 4,096 particles 5.8 us (11.8), 65,536 16.7 (21.2), 262,144 80 (140), 100,003 compensated 46 (61).
constexpr int kFoldT = 4, kFoldThreads = 32 * kFoldT;
template <int V> struct FoldVec { using type = float; };
template <> struct FoldVec<4> { using type = float4; };
template <int V>
__device__ __forceinline__ float fold_get(const typename FoldVec<V>::type& x, int e) {
    if constexpr (V == 4) return e == 0 ? x.x : (e == 1 ? x.y : (e == 2 ? x.z : x.w));
    else return x;
}
// Where 1/r^3 does not suit the separations (gravity_sym.cuh), the slots of k_gravity_sym are of no use: a group of its
// particles reaches far, or the softening is out of range. The fold then sums over all particles itself, (m / r) (1 / r^2) as
// the one-sided kernels do, 256 at a time in FP32. Asking costs next to nothing (the groups' flags come with the slots, the
// vote is in its barrier), and the sweep keeps its registers: with the far sums in the sweep's kernel, looked up per tile or
// per task, its compensated form lost 1.5 to 3.5 us at 3,000 to 12,000 particles (9,000: 38.3 -> 40.1 us; now 38.3), unequal
// masses 2 % (45,000: 626 -> 638 us; now 625).
struct FarView {
    const int* groups = nullptr;  // flags of the G groups of the sweep (G = 0: slots that hold any separation)
    int G = 0;
    const float4* posm = nullptr;
    float eps2 = 0.0f;
};
template <int V>
__device__ __forceinline__ void far_sums(const FarView& v, int64_t n, int64_t i, int q, double (&s)[V][3]) {
    float x[V], y[V], z[V];
#pragma unroll
    for (int e = 0; e < V; ++e) {
        const float4 p = v.posm[i + e < n ? i + e : n - 1];
        x[e] = p.x; y[e] = p.y; z[e] = p.z;
        s[e][0] = s[e][1] = s[e][2] = 0.0;
    }
    const float most = v.eps2 > 0.0f ? INFINITY : 1e12f;  // eps == 0: the self pair gives 0
    const int64_t j1 = n * (q + 1) / kFoldT;
    for (int64_t j0 = n * q / kFoldT; j0 < j1; j0 += 256) {
        float t[V][3];
#pragma unroll
        for (int e = 0; e < V; ++e) t[e][0] = t[e][1] = t[e][2] = 0.0f;
#pragma unroll 4
        for (int64_t j = j0; j < min(j1, j0 + 256); ++j) {
            const float4 p = v.posm[j];
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const float dx = p.x - x[e], dy = p.y - y[e], dz = p.z - z[e];
                const float inv = fminf(rsqrtf(fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, v.eps2)))), most);
                const float w = p.w * inv * (inv * inv);
                t[e][0] = fmaf(dx, w, t[e][0]);
                t[e][1] = fmaf(dy, w, t[e][1]);
                t[e][2] = fmaf(dz, w, t[e][2]);
            }
        }
#pragma unroll
        for (int e = 0; e < V; ++e)
            for (int c = 0; c < 3; ++c) s[e][c] += static_cast<double>(t[e][c]);
    }
}
// f(i, sum) for the particles of this CTA, on the threads of warp 0
template <bool COMP, int V, typename F>
__device__ __forceinline__ void fold_slots(const float* part, int64_t n, int64_t n_pad, int S, const FarView& v, F&& f) {
    using Vec = typename FoldVec<V>::type;
    constexpr int K = COMP ? 6 : 3, U = (V == 4 ? 12 : 54) / K;
    __shared__ double run[kFoldT - 1][V][3][32];
    const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
    const int64_t i = (static_cast<int64_t>(blockIdx.x) * 32 + lane) * V;
    const int R = (S + kFoldT - 1) / kFoldT;
    const int k0 = min(S, q * R), k1 = min(S, k0 + R);
    const int flag = static_cast<int>(threadIdx.x) < v.G ? v.groups[threadIdx.x] : 0;  // looked at behind the slots' loads
    double s[V][3];
#pragma unroll
    for (int e = 0; e < V; ++e) s[e][0] = s[e][1] = s[e][2] = 0.0;
    if (i < n) {  // n_pad is a multiple of 1024: a vector of the last particles stays in its row
        for (int k = k0; k < k1; k += U) {
            Vec w[U][K];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float* p = part + static_cast<int64_t>(V == 1 ? k + u : min(k + u, k1 - 1)) * K * n_pad + i;
#pragma unroll
                for (int c = 0; c < K; ++c)
                    w[u][c] = V > 1 || k + u < k1 ? *reinterpret_cast<const Vec*>(p + c * n_pad) : Vec{};
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (V > 1 && k + u >= k1) break;
#pragma unroll
                for (int e = 0; e < V; ++e)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        s[e][c] += static_cast<double>(fold_get<V>(w[u][c], e));
                        if (COMP) s[e][c] += static_cast<double>(fold_get<V>(w[u][K - 3 + c], e));
                    }
            }
        }
    }
    auto hand_over = [&]() {
        if (q > 0)
#pragma unroll
            for (int e = 0; e < V; ++e)
#pragma unroll
                for (int c = 0; c < 3; ++c) run[q - 1][e][c][lane] = s[e][c];
    };
    hand_over();
    int far = flag;
    for (int k = threadIdx.x + kFoldThreads; k < v.G; k += kFoldThreads) far |= v.groups[k];
    if (__syncthreads_or(far || (v.G > 0 && v.eps2 > 0.0f && sym_far_eps<1>(v.eps2)))) {
        far_sums<V>(v, n, i, q, s);
        hand_over();
        __syncthreads();
    }
    if (q > 0) return;
#pragma unroll
    for (int e = 0; e < V; ++e) {
        if (i + e >= n) break;
        double t[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {  // runs 0 + 1 + 2 + 3, in this order
            t[c] = s[e][c];
#pragma unroll
            for (int r = 0; r < kFoldT - 1; ++r) t[c] += run[r][e][c][lane];
        }
        f(i + e, t);
    }
}
inline int fold_vec(int64_t n) { return n >= 32768 ? 4 : 1; }
inline unsigned fold_blocks(int64_t n) { return static_cast<unsigned>((n + 32 * fold_vec(n) - 1) / (32 * fold_vec(n))); }

// the culled path: the fold of the gravity partials into gfold[3][n_pad], on the gravity kernel's stream
template <bool COMP, int V>
__global__ void __launch_bounds__(kFoldThreads) k_gravity_fold(const float* part, int64_t n, int64_t n_pad, int S,
                                                               double* gfold, FarView v) {
    wait_predecessor();
    fold_slots<COMP, V>(part, n, n_pad, S, v, [&](int64_t i, const double (&t)[3]) {
        for (int c = 0; c < 3; ++c) gfold[c * n_pad + i] = t[c];
    });
}

template <int PASS, bool GRAV, bool SOLIDS, bool COMP>
__global__ void k_pairs_finish(DevArrays a, DevParams p, PartView pv, GravSum gsum) {
    constexpr uint32_t MASK = field_mask<PASS, GRAV, SOLIDS>();
    wait_predecessor();
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (PASS != PASS_VGRAD && has(p, GSPH_VARIABLE_TIMESTEP) && i == 0)
        a.dt_state[1] = p.max_dt;  // nextTS reset of calcAcceleration::do_after (:306-309)
    if (i >= a.n) return;
    float g[3] = {0.0f, 0.0f, 0.0f};
    bool grav = false;
    if (PASS != PASS_VGRAD) {
        if (GRAV) {
            g[0] = seg_sum<MASK, COMP>(pv, i, F_GX);
            g[1] = seg_sum<MASK, COMP>(pv, i, F_GY);
            g[2] = seg_sum<MASK, COMP>(pv, i, F_GZ);
            grav = true;
        } else if (gsum.nseg > 0 || gsum.sym_G > 0) {  // folded on the gravity stream (k_gravity_fold)
            for (int c = 0; c < 3; ++c) g[c] = static_cast<float>(a.gfold[c * a.n_pad + i]);
            grav = true;
        }
    }
    // the culled passes: one slot per field, all of them in flight at once (one after another, 4,000 particles took 18.4 us)
    if (pv.nseg == 1 && !pv.err) {
        float v[popc_c(MASK)];
#pragma unroll
        for (int o = 0; o < popc_c(MASK); ++o) v[o] = pv.at(0, o, i);
        sph_finish<PASS, SOLIDS>(a, p, i, [&](int f) { return 0.0f + v[field_offset<MASK>(f)]; }, grav, g);
        return;
    }
    sph_finish<PASS, SOLIDS>(a, p, i, [&](int f) { return seg_sum<MASK, COMP>(pv, i, f); }, grav, g);
}

// ================================================================================================
// pure gravity (ENABLE_SPH off): I i-particles per thread share every j read from shared memory
// ================================================================================================
// I (even) i-particles per thread in I/2 register pairs; same arithmetic order as k_gravity
template <int I, int GRAV, bool COMP>
__global__ void __launch_bounds__(128) k_gravity_x2(const float4* __restrict__ posm, float* __restrict__ part,
                                                     int64_t n_pad, int jt, int nseg, float eps2, int* status) {
    constexpr int P = I / 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    JTilePipe<1> pipe;
    pipe.buf = reinterpret_cast<float4*>(smem_raw);
    pipe.bar = reinterpret_cast<uint64_t*>(smem_raw + 2 * jt * sizeof(float4));
    pipe.src[0] = posm;
    pipe.jt = jt;
    pipe.status = status;
    segment_tiles(n_pad / jt, blockIdx.y, nseg, pipe.t_begin, pipe.t_end);

    const int64_t base = static_cast<int64_t>(blockIdx.x) * blockDim.x * I + threadIdx.x;
    float2 X[P], Y[P], Z[P], AX[P], AY[P], AZ[P], CX[P], CY[P], CZ[P];
#pragma unroll
    for (int k = 0; k < P; ++k) {
        const float4 a = posm[base + static_cast<int64_t>(2 * k) * blockDim.x];
        const float4 b = posm[base + static_cast<int64_t>(2 * k + 1) * blockDim.x];
        X[k] = make_float2(a.x, b.x); Y[k] = make_float2(a.y, b.y); Z[k] = make_float2(a.z, b.z);
        AX[k] = AY[k] = AZ[k] = make_float2(0.0f, 0.0f);
        CX[k] = CY[k] = CZ[k] = make_float2(0.0f, 0.0f);
    }
    const float2 E2 = make_float2(eps2, eps2);

    pipe.start();
    pipe.run([&](const float4* J) {
        float2 TX[P], TY[P], TZ[P];
#pragma unroll
        for (int k = 0; k < P; ++k) TX[k] = TY[k] = TZ[k] = make_float2(0.0f, 0.0f);
#pragma unroll 4
        for (int j = 0; j < jt; ++j) {
            const float4 q = J[j];
            const float2 qx = make_float2(q.x, q.x), qy = make_float2(q.y, q.y), qz = make_float2(q.z, q.z),
                         qm = make_float2(q.w, q.w);
#pragma unroll
            for (int k = 0; k < P; ++k) {
                const float2 dx = sub2(qx, X[k]), dy = sub2(qy, Y[k]), dz = sub2(qz, Z[k]);
                const float2 r2 = fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, E2)));
                float2 inv = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
                if (GRAV == 2) inv = make_float2(fminf(inv.x, 1e12f), fminf(inv.y, 1e12f));
                const float2 s = mul2(mul2(qm, inv), mul2(inv, inv));
                if (COMP) {
                    TX[k] = fma2(dx, s, TX[k]); TY[k] = fma2(dy, s, TY[k]); TZ[k] = fma2(dz, s, TZ[k]);
                } else {
                    AX[k] = fma2(dx, s, AX[k]); AY[k] = fma2(dy, s, AY[k]); AZ[k] = fma2(dz, s, AZ[k]);
                }
            }
        }
        if (COMP) {
#pragma unroll
            for (int k = 0; k < P; ++k) {
                fold(AX[k].x, CX[k].x, TX[k].x); fold(AX[k].y, CX[k].y, TX[k].y);
                fold(AY[k].x, CY[k].x, TY[k].x); fold(AY[k].y, CY[k].y, TY[k].y);
                fold(AZ[k].x, CZ[k].x, TZ[k].x); fold(AZ[k].y, CZ[k].y, TZ[k].y);
            }
        }
    });

    const int64_t seg = blockIdx.y;
    const int K = COMP ? 6 : 3;
#pragma unroll
    for (int k = 0; k < P; ++k) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float* out = part + seg * K * n_pad + base + static_cast<int64_t>(2 * k + h) * blockDim.x;
            out[0] = h ? AX[k].y : AX[k].x;
            out[n_pad] = h ? AY[k].y : AY[k].x;
            out[2 * n_pad] = h ? AZ[k].y : AZ[k].x;
            if (COMP) {
                out[3 * n_pad] = h ? CX[k].y : CX[k].x;
                out[4 * n_pad] = h ? CY[k].y : CY[k].x;
                out[5 * n_pad] = h ? CZ[k].y : CZ[k].x;
            }
        }
    }
}
// ================================================================================================
// symmetric all-pairs gravity (Newton's third law): every unordered pair evaluated once
// ================================================================================================
// Particles form blocks of B = R T (R rows per thread, T threads); blocks form G groups of `gs` consecutive blocks.
// CTA t is the task (ga, gb), ga <= gb (the G(G-1)/2 pairs of distinct groups first, then the G diagonal ones): for
// every row block a of group ga it sweeps the column blocks of group gb (those after a when ga == gb) in j-tiles
// through shared memory. One 1/r^3 serves both particles of a pair. The pairs inside a block run one-sided. Each
// particle has G + 1 slots, each written by one task (its row sums from tasks (g, gb), its column sums from tasks
// (ga, g), g its group); the fold adds a particle's slots in FP64 in a fixed order, so results do not depend on
// scheduling.
//
// An f32x2 instruction takes one row against two columns, 32 apart: rows are duplicated once per block, columns are
// staged as (x x' y y') (z z' m m') so that a 16-byte load brings two register pairs, and a column sum is an f32x2
// accumulator of its own. In round r of a block of 64 columns lane l takes the columns (l + r) % 32 and (l + r) % 32 + 32,
// adds its rows' shares and hands the sums to lane l - 1; after 32 rounds lane l holds the warp's sums of columns l and
// l + 32. (Two rows per instruction, as gravity_fixed.cu, costs a register move per operand for the duplicated column,
// zeroed accumulators and a horizontal add per column: 113 instructions per 512 interactions instead of 84.)
// Row sums are accumulated per j-tile and then added to running sums in shared memory (plain: one add; compensated: a
// two-sum fold whose error terms are there too).
//
// Where every row of the block has one mass and every column of the tile has one (the particle sources give equal
// masses; it is looked up in each tile, in the barrier that publishes it), the masses leave the pair loop: 14 FP32
// operations per unordered pair instead of 16.
//
// Bound: the register file. An f32x2 multiply-add of three different register pairs reads six registers and runs at
// 0.60 of the FMA rate, multiplies and adds (four) at 0.96; six of a pair's operations are such multiply-adds, which
// predicts 0.77 of the FMA rate; the pipe is 75 % busy with equal masses, 78 % with others.
// Measured (N = 262,144, 128 groups, one B200): row-packed 22.3 ms, column-packed 19.2 ms, equal masses 17.5 ms.
template <typename S, int GRAV, bool COMP>
__global__ void __launch_bounds__(S::T, S::CTAS) k_gravity_sym(const float4* __restrict__ posm, float* __restrict__ part,
                                                               int64_t n, int64_t n_pad, int G, int gs, float eps2, int* far_groups) {
    constexpr int R = S::R, T = S::T, B = S::B, JT = S::JT, PF = S::PF, W = S::W;
    constexpr int K = COMP ? 6 : 3;
    __shared__ float4 XY[JT / 2], ZM[JT / 2];
    __shared__ float js[W][3][JT];
    __shared__ float rsh[3 * R][T];             // the row particles' running sums ...
    __shared__ float csh[COMP ? 3 * R : 1][T];  // ... and, compensated, their rounding errors
    const int tid = threadIdx.x, warp = tid >> 5;
    int ga, gb;
    sym_task(static_cast<int>(blockIdx.x), G, ga, gb);
    const int nb = static_cast<int>(n_pad / B);
    const int ra0 = ga * gs, ra1 = min(nb, ra0 + gs);
    const int cg0 = gb * gs, cg1 = min(nb, cg0 + gs);
    const bool diag = ga == gb;
    // slots [slot][component][n_pad]: a particle of group g holds its row sums from tasks (g, gb), gb = g .. G-1, in
    // slots 0 .. G-1-g and its column sums from tasks (ga, g), ga = 0 .. g, in slots G-g .. G
    const int s_row = gb - ga, s_col = G - gb + ga;
    auto slot = [&](int64_t particle, int sl, int c) { return part + (static_cast<int64_t>(sl) * K + c) * n_pad + particle; };
    if (diag) {  // the group's first block is never a column here: its column slot is zero
        for (int e = tid; e < B; e += T)
            for (int c = 0; c < K; ++c) *slot(static_cast<int64_t>(ra0) * B + e, s_col, c) = 0.0f;
        bool far = false;  // for the fold; the padding lies far out too, but has no mass
        for (int64_t i = static_cast<int64_t>(ra0) * B + tid; i < min(n, static_cast<int64_t>(ra1) * B); i += T)
            far = sym_far(posm[i]) || far;
        const int any = __syncthreads_or(far);
        if (tid == 0) far_groups[ga] = any;
    }
    const float2 E2 = make_float2(eps2, eps2);

    for (int a = ra0; a < ra1; ++a) {
        const int64_t base = static_cast<int64_t>(a) * B + tid;
        SymRows<S> rows;
        const float mr = posm[static_cast<int64_t>(a) * B].w;
        bool same = true;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const float4 u = posm[base + static_cast<int64_t>(k) * T];
            rows.set(k, u);
            same = same && u.w == mr;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                rsh[c * R + k][tid] = 0.0f;
                if (COMP) csh[COMP ? c * R + k : 0][tid] = 0.0f;
            }
        }
        const bool rows_equal = __syncthreads_and(same);
        // tiles: the block's own (one-sided) when diagonal, then the columns
        const int64_t d0 = static_cast<int64_t>(a) * B;
        const int nd = diag ? B / JT : 0;
        const int64_t c0 = static_cast<int64_t>(diag ? a + 1 : cg0) * B, c1 = static_cast<int64_t>(cg1) * B;
        const int total = nd + (c1 > c0 ? static_cast<int>((c1 - c0) / JT) : 0);
        auto src = [&](int k) { return k < nd ? d0 + static_cast<int64_t>(k) * JT : c0 + static_cast<int64_t>(k - nd) * JT; };
        float4 pf[PF];
        float mn = 0.0f;  // the mass of the next tile's first column
#pragma unroll
        for (int h = 0; h < PF; ++h) pf[h] = make_float4(0, 0, 0, 0);
        if (total > 0) {
            mn = posm[src(0)].w;
#pragma unroll
            for (int h = 0; h < PF; ++h) pf[h] = posm[src(0) + h * T + tid];
        }
        for (int k = 0; k < total; ++k) {
            __syncthreads();  // the previous tile's reads of XY, ZM and js are done
            const float mc = mn;
            bool same_c = true;
#pragma unroll
            for (int h = 0; h < PF; ++h) {
                sym_stage(XY, ZM, tid + h * T, pf[h]);
                same_c = same_c && pf[h].w == mc;
            }
            const bool equal = __syncthreads_and(same_c) && rows_equal;
            if (k + 1 < total) {
                mn = posm[src(k + 1)].w;
#pragma unroll
                for (int h = 0; h < PF; ++h) pf[h] = posm[src(k + 1) + h * T + tid];
            }
            rows.clear();
            if (k < nd) sym_own<S, GRAV, false>(rows, XY, ZM, E2);
            else if (equal) sym_columns<S, GRAV, true>(rows, XY, ZM, E2, js[warp]);
            else sym_columns<S, GRAV, false>(rows, XY, ZM, E2, js[warp]);
            // the tile's row partials into the running sums: a two-sum fold (compensated), or one add (plain: a sum
            // of tile sums, not one running sum over the whole column group)
            const float wr = k >= nd && equal ? mc : 1.0f;
            auto row_add = [&](int o, float2 t) {
                float x = rsh[o][tid];
                if (COMP) {
                    float e = csh[COMP ? o : 0][tid];
                    fold(x, e, wr * (t.x + t.y));
                    csh[COMP ? o : 0][tid] = e;
                } else {
                    x = fmaf(wr, t.x + t.y, x);
                }
                rsh[o][tid] = x;
            };
#pragma unroll
            for (int m = 0; m < R; ++m) {
                row_add(m, rows.TX[m]);
                row_add(R + m, rows.TY[m]);
                row_add(2 * R + m, rows.TZ[m]);
            }
            if (k >= nd) {  // this tile's column sums over the CTA's row block, into the column slot
                __syncthreads();
                const float wc = equal ? -mr : 1.0f;
                const int64_t jb = c0 + static_cast<int64_t>(k - nd) * JT;
#pragma unroll
                for (int h = 0; h < PF; ++h) {
                    const int j = tid + h * T;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        float v = js[0][c][j] + js[1][c][j];
                        if constexpr (W == 4) v += js[2][c][j] + js[3][c][j];
                        v *= wc;
                        float* dst = slot(jb + j, s_col, c);
                        if (COMP) {
                            float* cdst = slot(jb + j, s_col, 3 + c);
                            if (a == ra0) {
                                *dst = v;
                                *cdst = 0.0f;
                            } else {
                                float sv = *dst, cv = *cdst;
                                fold(sv, cv, v);
                                *dst = sv;
                                *cdst = cv;
                            }
                        } else {
                            *dst = a == ra0 ? v : *dst + v;
                        }
                    }
                }
            }
        }
        // the row sums of block a into its row slot (a thread's own shared-memory values)
#pragma unroll
        for (int m = 0; m < R; ++m) {
            const int64_t pr = base + static_cast<int64_t>(m) * T;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                *slot(pr, s_row, c) = rsh[c * R + m][tid];
                if (COMP) *slot(pr, s_row, 3 + c) = csh[COMP ? c * R + m : 0][tid];
            }
        }
    }
}

// The shapes, by rows per thread, threads and CTAs per SM: larger blocks do less per column sum, smaller ones give more
// tasks (sym_shape).
using Sym8 = SymShape<8, 128, 3>;
using Sym4 = SymShape<4, 128, 4>;
using Sym2 = SymShape<2, 128, 6>;
using Sym1 = SymShape<2, 64, 12>;

template <int I, int GRAV, bool COMP>
__global__ void __launch_bounds__(128) k_gravity(const float4* __restrict__ posm, float* __restrict__ part,
                                                  int64_t n_pad, int jt, int nseg, float eps2, int* status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    JTilePipe<1> pipe;
    pipe.buf = reinterpret_cast<float4*>(smem_raw);
    pipe.bar = reinterpret_cast<uint64_t*>(smem_raw + 2 * jt * sizeof(float4));
    pipe.src[0] = posm;
    pipe.jt = jt;
    pipe.status = status;
    segment_tiles(n_pad / jt, blockIdx.y, nseg, pipe.t_begin, pipe.t_end);

    const int64_t base = static_cast<int64_t>(blockIdx.x) * blockDim.x * I + threadIdx.x;
    float xi[I], yi[I], zi[I], ax[I], ay[I], az[I], cx[I], cy[I], cz[I];
#pragma unroll
    for (int k = 0; k < I; ++k) {
        const float4 q = posm[base + static_cast<int64_t>(k) * blockDim.x];
        xi[k] = q.x; yi[k] = q.y; zi[k] = q.z;
        ax[k] = ay[k] = az[k] = 0.0f;
        cx[k] = cy[k] = cz[k] = 0.0f;
    }

    pipe.start();
    pipe.run([&](const float4* J) {
        float tx[I], ty[I], tz[I];
#pragma unroll
        for (int k = 0; k < I; ++k) tx[k] = ty[k] = tz[k] = 0.0f;
#pragma unroll 4
        for (int j = 0; j < jt; ++j) {
            const float4 q = J[j];
#pragma unroll
            for (int k = 0; k < I; ++k) {
                const float dx = q.x - xi[k], dy = q.y - yi[k], dz = q.z - zi[k];
                const float r2 = fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, eps2)));
                float inv = rsqrtf(r2);
                if (GRAV == 2) inv = fminf(inv, 1e12f);
                const float s = q.w * inv * (inv * inv);
                if (COMP) {
                    tx[k] = fmaf(dx, s, tx[k]);
                    ty[k] = fmaf(dy, s, ty[k]);
                    tz[k] = fmaf(dz, s, tz[k]);
                } else {
                    ax[k] = fmaf(dx, s, ax[k]);
                    ay[k] = fmaf(dy, s, ay[k]);
                    az[k] = fmaf(dz, s, az[k]);
                }
            }
        }
        if (COMP) {
#pragma unroll
            for (int k = 0; k < I; ++k) {
                fold(ax[k], cx[k], tx[k]);
                fold(ay[k], cy[k], ty[k]);
                fold(az[k], cz[k], tz[k]);
            }
        }
    });

    const int64_t seg = blockIdx.y;
    const int K = COMP ? 6 : 3;
#pragma unroll
    for (int k = 0; k < I; ++k) {
        float* out = part + seg * K * n_pad + base + static_cast<int64_t>(k) * blockDim.x;
        out[0] = ax[k];
        out[n_pad] = ay[k];
        out[2 * n_pad] = az[k];
        if (COMP) {
            out[3 * n_pad] = cx[k];
            out[4 * n_pad] = cy[k];
            out[5 * n_pad] = cz[k];
        }
    }
}

template <bool COMP, int V>
__global__ void __launch_bounds__(kFoldThreads) k_gravity_finish(DevArrays a, DevParams p, GravSum gsum) {
    wait_predecessor();
    if (has(p, GSPH_VARIABLE_TIMESTEP) && blockIdx.x == 0 && threadIdx.x == 0) a.dt_state[1] = p.max_dt;
    fold_slots<COMP, V>(a.part, a.n, a.n_pad, gsum.sym_G > 0 ? gsum.sym_G + 1 : gsum.nseg, FarView{a.gfar, gsum.sym_G, a.posm, p.eps2}, [&](int64_t i, const double (&t)[3]) {
        float acc[3];
#pragma unroll
        for (int c = 0; c < 3; ++c)
            acc[c] = COMP ? static_cast<float>(t[c] * static_cast<double>(p.G)) : p.G * static_cast<float>(t[c]);
        if (a.grav) a.grav[i] = make_float4(acc[0], acc[1], acc[2], 0.0f);
        environment(p, a.posm[i], a.velrho[i], acc[0], acc[1], acc[2]);
        a.acc[i] = make_float4(acc[0], acc[1], acc[2], 0.0f);
        a.xvel[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    });
}

inline unsigned blocks_for(int64_t n, int t) { return static_cast<unsigned>((n + t - 1) / t); }
constexpr int kEach = 128;  // threads per CTA of the per-particle kernels: 4,096 particles on 32 SMs

}  // namespace

// ---- host launchers ----------------------------------------------------------------------------
// Event record that also works while `s` is being captured into a graph (as an event-record node).
cudaError_t timer_record(cudaEvent_t ev, cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(s, &st);
    if (e != cudaSuccess) return e;
    if (st == cudaStreamCaptureStatusActive) return cudaEventRecordWithFlags(ev, s, cudaEventRecordExternal);
    return cudaEventRecord(ev, s);
}

#define GSPH_TIMER_MARK(t, which)                          \
    do {                                                   \
        if (t) {                                           \
            cudaError_t te_ = timer_record((t)->which, s); \
            if (te_ != cudaSuccess) return te_;            \
        }                                                  \
    } while (0)

namespace {
NearView near_view(const DevArrays& a, const DevParams& p, const SpatialArrays& sp) {
    NearView v;
    v.list = sp.list;
    v.count = sp.count;
    v.order = sp.group_order;
    v.lo = sp.sub_lo;
    v.hi = sp.sub_hi;
    v.ngroups = static_cast<int>(a.n_pad / kGroup);
    v.nchunks = a.n_pad / kChunk;
    v.n = a.n;
    v.n_pad = a.n_pad;
    const float hm = p.H * (1.0f + kMargin);
    v.hm2 = hm * hm;
    v.nb = sp.nb;
    v.nbcnt = sp.nbcnt;
    v.cap = sp.nb_cap;
    return v;
}
unsigned near_blocks(const DevArrays& a) { return static_cast<unsigned>(a.n_pad / kSub); }
template <int W>
cudaError_t near_launch(const DevArrays& a, const DevParams& p, const NearView& v, bool dens, bool comp, bool early,
                        cudaStream_t s) {
    auto kern = !dens ? k_near<W, false, false> : (comp ? k_near<W, true, true> : k_near<W, true, false>);
    return launch_kernel(early, kern, near_blocks(a), kSub * W, s, a.posm, a.velrho, p, v);
}
// at most one warp and a half per scheduler of the 148 SMs when a warp takes 32 particles
constexpr int kAhead = 4;  // records in flight then
bool few_groups(const DevArrays& a) { return a.n_pad / kSub <= 900; }
PartView seg_view(const DevArrays& a, int nseg, int KK, bool err) {
    return PartView{a.part, a.n_pad, nseg, KK, err};
}
}  // namespace

cudaError_t launch_density(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s, const KTimer* t,
                           const SpatialArrays* sp) {
    const bool comp = L.accum == GSPH_ACCUM_COMPENSATED;
    GSPH_TIMER_MARK(t, start);
    if (sp) {
        const NearView v = near_view(a, p, *sp);
        const bool dens = !has(p, GSPH_INTEGRATE_DENSITY);
        const cudaError_t le = !dens && few_groups(a) ? near_launch<8>(a, p, v, dens, comp, !t, s)
                                                                  : near_launch<4>(a, p, v, dens, comp, !t, s);
        if (le != cudaSuccess) return le;
    } else {
        const int T = 256;
        const dim3 grid(static_cast<unsigned>(a.n_pad / T), static_cast<unsigned>(L.nseg));
        const size_t smem = pipe_smem_bytes(1, L.jt);
        if (comp) k_density<true><<<grid, T, smem, s>>>(a.posm, a.part, a.n_pad, L.jt, L.nseg, p, a.status);
        else k_density<false><<<grid, T, smem, s>>>(a.posm, a.part, a.n_pad, L.jt, L.nseg, p, a.status);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    GSPH_TIMER_MARK(t, stop);
    if (sp) return launch_prepare(a, p, s, !t);  // the density is final: the j-records
    const PartView pv = seg_view(a, L.nseg, comp ? 2 : 1, comp);
    if (comp) k_density_finish<true><<<blocks_for(a.n, 256), 256, 0, s>>>(a, p, pv);
    else k_density_finish<false><<<blocks_for(a.n, 256), 256, 0, s>>>(a, p, pv);
    return cudaGetLastError();
}

cudaError_t launch_prepare(const DevArrays& a, const DevParams& p, cudaStream_t s, bool early) {
    return launch_kernel(early, k_prepare, blocks_for(a.n, kEach), kEach, s, a, p);
}

namespace {
template <int PASS, int GRAV, bool SOLIDS, bool COMP>
cudaError_t pairs_t(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s, const KTimer* t,
                    const SpatialArrays* sp, int gnseg, cudaEvent_t join) {
    constexpr int NS = (PASS == PASS_VGRAD) ? 2 : 4;
    if (sp) {  // SPH terms over the near chunks; gravity partials come from elsewhere
        constexpr uint32_t MASK = field_mask<PASS, false, SOLIDS>();
        constexpr int K = popc_c(MASK);
        GSPH_TIMER_MARK(t, start);
        const NearView v = near_view(a, p, *sp);
        void (*kern)(DevArrays, DevParams, NearView) = k_pairs_near<PASS, SOLIDS, COMP, 1>;
        dim3 grid(near_blocks(a));
        if (few_groups(a)) {
            if constexpr (PASS == PASS_FUSED) {
                kern = k_pairs_near_split<SOLIDS, COMP>;
                grid.y = 2;
            } else {
                kern = k_pairs_near<PASS, SOLIDS, COMP, kAhead>;
            }
        }
        cudaError_t e = launch_kernel(!t, kern, grid, kSub, s, a, p, v);
        if (e != cudaSuccess) return e;
        GSPH_TIMER_MARK(t, stop);
        if (join) {
            e = cudaStreamWaitEvent(s, join, 0);
            if (e != cudaSuccess) return e;
        }
        return launch_kernel(!t && !join, k_pairs_finish<PASS, false, SOLIDS, COMP>, blocks_for(a.n, kEach), kEach, s, a, p,
                             seg_view(a, 1, K, false), grav_sum(L, PASS == PASS_VGRAD ? 0 : gnseg));
    }
    constexpr uint32_t MASK = field_mask<PASS, (GRAV != 0), SOLIDS>();
    constexpr int K = popc_c(MASK);
    const size_t smem = pipe_smem_bytes(NS, L.jt);
    auto kern = k_pairs<PASS, GRAV, SOLIDS, COMP>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return e;
    }
    const dim3 grid(static_cast<unsigned>(a.n_pad / L.threads), static_cast<unsigned>(L.nseg));
    GSPH_TIMER_MARK(t, start);
    kern<<<grid, L.threads, smem, s>>>(a, p, L.jt, L.nseg);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    GSPH_TIMER_MARK(t, stop);
    k_pairs_finish<PASS, (GRAV != 0), SOLIDS, COMP><<<blocks_for(a.n, 256), 256, 0, s>>>(
        a, p, seg_view(a, L.nseg, COMP ? 2 * K : K, COMP), GravSum{});
    return cudaGetLastError();
}

template <int PASS, int GRAV>
cudaError_t pairs_g(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s, const KTimer* t,
                    const SpatialArrays* sp, int gnseg, cudaEvent_t join) {
    const bool solids = has(p, GSPH_SOLIDS);
    const bool comp = L.accum == GSPH_ACCUM_COMPENSATED;
    if (solids)
        return comp ? pairs_t<PASS, GRAV, true, true>(a, p, L, s, t, sp, gnseg, join)
                    : pairs_t<PASS, GRAV, true, false>(a, p, L, s, t, sp, gnseg, join);
    return comp ? pairs_t<PASS, GRAV, false, true>(a, p, L, s, t, sp, gnseg, join)
                : pairs_t<PASS, GRAV, false, false>(a, p, L, s, t, sp, gnseg, join);
}
}  // namespace

cudaError_t launch_pairs(int pass, const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s,
                         const KTimer* t, const SpatialArrays* sp, int gnseg, cudaEvent_t join) {
    if (sp) {  // the culled kernels carry no gravity
        switch (pass) {
            case PASS_VGRAD: return pairs_g<PASS_VGRAD, 0>(a, p, L, s, t, sp, 0, join);
            case PASS_ACC: return pairs_g<PASS_ACC, 0>(a, p, L, s, t, sp, gnseg, join);
            default: return pairs_g<PASS_FUSED, 0>(a, p, L, s, t, sp, gnseg, join);
        }
    }
    const int grav = !has(p, GSPH_SELF_GRAVITY) ? 0 : (p.eps2 > 0.0f ? 1 : 2);
    switch (pass) {
        case PASS_VGRAD: return pairs_g<PASS_VGRAD, 0>(a, p, L, s, t, nullptr, 0, nullptr);
        case PASS_ACC:
            return grav == 0 ? pairs_g<PASS_ACC, 0>(a, p, L, s, t, nullptr, 0, nullptr)
                             : (grav == 1 ? pairs_g<PASS_ACC, 1>(a, p, L, s, t, nullptr, 0, nullptr)
                                          : pairs_g<PASS_ACC, 2>(a, p, L, s, t, nullptr, 0, nullptr));
        default:
            return grav == 0 ? pairs_g<PASS_FUSED, 0>(a, p, L, s, t, nullptr, 0, nullptr)
                             : (grav == 1 ? pairs_g<PASS_FUSED, 1>(a, p, L, s, t, nullptr, 0, nullptr)
                                          : pairs_g<PASS_FUSED, 2>(a, p, L, s, t, nullptr, 0, nullptr));
    }
}

namespace {
template <typename S, int GRAV, bool COMP>
void sym_launch(const DevArrays& a, const DevParams& p, const Launch& L, float* out, cudaStream_t s) {
    const int G = L.grav_sym_G;
    k_gravity_sym<S, GRAV, COMP><<<static_cast<unsigned>(G * (G + 1) / 2), S::T, 0, s>>>(a.posm, out, a.n, a.n_pad, G,
                                                                                        L.grav_sym_gs, p.eps2, a.gfar);
}
template <int I, int GRAV, bool COMP>
cudaError_t gravity_t(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s, const KTimer* t,
                      bool finish) {
    const int T = L.grav_threads;
    const dim3 grid(static_cast<unsigned>(a.n_pad / (static_cast<int64_t>(T) * I)), static_cast<unsigned>(L.grav_nseg));
    const size_t smem = pipe_smem_bytes(1, L.grav_jt);
    GSPH_TIMER_MARK(t, start);
    if (L.grav_sym_G > 0) {
        float* out = finish ? a.part : a.gpart;
        switch (L.grav_sym_shape) {
            case 0: sym_launch<Sym8, GRAV, COMP>(a, p, L, out, s); break;
            case 1: sym_launch<Sym4, GRAV, COMP>(a, p, L, out, s); break;
            case 2: sym_launch<Sym2, GRAV, COMP>(a, p, L, out, s); break;
            default: sym_launch<Sym1, GRAV, COMP>(a, p, L, out, s);
        }
    } else if constexpr (I >= 2) {
        if (L.grav_x2)
            k_gravity_x2<I, GRAV, COMP><<<grid, T, smem, s>>>(a.posm, finish ? a.part : a.gpart, a.n_pad, L.grav_jt,
                                                               L.grav_nseg, p.eps2, a.status);
        else
            k_gravity<I, GRAV, COMP><<<grid, T, smem, s>>>(a.posm, finish ? a.part : a.gpart, a.n_pad, L.grav_jt,
                                                            L.grav_nseg, p.eps2, a.status);
    } else {
        k_gravity<I, GRAV, COMP><<<grid, T, smem, s>>>(a.posm, finish ? a.part : a.gpart, a.n_pad, L.grav_jt,
                                                        L.grav_nseg, p.eps2, a.status);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    GSPH_TIMER_MARK(t, stop);
    const int S = L.grav_sym_G > 0 ? L.grav_sym_G + 1 : L.grav_nseg;
    if (!finish) return launch_gravity_fold(a, L, S, s, !t, L.grav_sym_G, p.eps2);  // the culled path: the SPH finish reads a.gfold
    auto kern = fold_vec(a.n) == 4 ? k_gravity_finish<COMP, 4> : k_gravity_finish<COMP, 1>;
    return launch_kernel(!t, kern, fold_blocks(a.n), kFoldThreads, s, a, p, grav_sum(L, L.grav_nseg));
}
template <int GRAV, bool COMP>
cudaError_t gravity_i(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s, const KTimer* t,
                      bool finish) {
    switch (L.grav_ipt) {
        case 1: return gravity_t<1, GRAV, COMP>(a, p, L, s, t, finish);
        case 2: return gravity_t<2, GRAV, COMP>(a, p, L, s, t, finish);
        case 8: return gravity_t<8, GRAV, COMP>(a, p, L, s, t, finish);
        default: return gravity_t<4, GRAV, COMP>(a, p, L, s, t, finish);
    }
}
cudaError_t gravity_any(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s, const KTimer* t,
                        bool finish) {
    const bool comp = L.accum == GSPH_ACCUM_COMPENSATED;
    if (p.eps2 > 0.0f) return comp ? gravity_i<1, true>(a, p, L, s, t, finish) : gravity_i<1, false>(a, p, L, s, t, finish);
    return comp ? gravity_i<2, true>(a, p, L, s, t, finish) : gravity_i<2, false>(a, p, L, s, t, finish);
}
}  // namespace

cudaError_t launch_gravity(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s, const KTimer* t) {
    const bool comp = L.accum == GSPH_ACCUM_COMPENSATED;
    if (!has(p, GSPH_SELF_GRAVITY)) {  // neither gravity nor SPH: environment terms only
        auto kern = fold_vec(a.n) == 4 ? (comp ? k_gravity_finish<true, 4> : k_gravity_finish<false, 4>)
                                       : (comp ? k_gravity_finish<true, 1> : k_gravity_finish<false, 1>);
        return launch_kernel(false, kern, fold_blocks(a.n), kFoldThreads, s, a, p, GravSum{});
    }
    return gravity_any(a, p, L, s, t, true);
}

cudaError_t launch_gravity_partials(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s,
                                    const KTimer* t) {
    return gravity_any(a, p, L, s, t, false);
}

cudaError_t launch_gravity_fold(const DevArrays& a, const Launch& L, int S, cudaStream_t s, bool early, int far_G, float eps2) {
    const bool comp = L.accum == GSPH_ACCUM_COMPENSATED;
    auto kern = fold_vec(a.n) == 4 ? (comp ? k_gravity_fold<true, 4> : k_gravity_fold<false, 4>)
                                   : (comp ? k_gravity_fold<true, 1> : k_gravity_fold<false, 1>);
    return launch_kernel(early, kern, fold_blocks(a.n), kFoldThreads, s, a.gpart, a.n, a.n_pad, S, a.gfold,
                         FarView{a.gfar, far_G, a.posm, eps2});
}

// Gravity partials of caller-provided, already padded j-records into caller-provided partials
// (the allocation-free entry point, noalloc.cu): the plain-FP32 paired kernel.
cudaError_t launch_gravity_raw(const float4* posm_padded, float* part, int64_t n_pad, int ipt, int jt, int nseg,
                               float eps2, int* status, cudaStream_t s) {
    const int T = 128;
    const dim3 grid(static_cast<unsigned>(n_pad / (static_cast<int64_t>(T) * ipt)), static_cast<unsigned>(nseg));
    const size_t smem = pipe_smem_bytes(1, jt);
    const bool soft = eps2 > 0.0f;
    if (ipt == 4) {
        if (soft) k_gravity_x2<4, 1, false><<<grid, T, smem, s>>>(posm_padded, part, n_pad, jt, nseg, eps2, status);
        else k_gravity_x2<4, 2, false><<<grid, T, smem, s>>>(posm_padded, part, n_pad, jt, nseg, eps2, status);
    } else {
        if (soft) k_gravity_x2<2, 1, false><<<grid, T, smem, s>>>(posm_padded, part, n_pad, jt, nseg, eps2, status);
        else k_gravity_x2<2, 2, false><<<grid, T, smem, s>>>(posm_padded, part, n_pad, jt, nseg, eps2, status);
    }
    return cudaGetLastError();
}

// ---- FP32 FFMA throughput probe (roofline denominator) -------------------------------------------
namespace {
constexpr int kPeakThreads = 256;
constexpr int kPeakBlocksPerSM = 4;
constexpr int kPeakChains = 16;
constexpr int kPeakUnroll = 16;
__global__ void __launch_bounds__(kPeakThreads) k_fp32_peak(float* sink, int iters) {
    float x[kPeakChains];
#pragma unroll
    for (int c = 0; c < kPeakChains; ++c) x[c] = static_cast<float>(threadIdx.x + c) * 1e-3f;
    const float a = 0.999999f, b = 1e-7f;
    for (int k = 0; k < iters; ++k) {
#pragma unroll
        for (int u = 0; u < kPeakUnroll; ++u)
#pragma unroll
            for (int c = 0; c < kPeakChains; ++c) x[c] = fmaf(x[c], a, b);
    }
    float s = 0.0f;
#pragma unroll
    for (int c = 0; c < kPeakChains; ++c) s += x[c];
    if (s == -1.0f) sink[blockIdx.x] = s;  // never true; keeps the chains live
}
}  // namespace

cudaError_t launch_fp32_peak(int sm_count, int iters, float* sink, cudaStream_t s) {
    k_fp32_peak<<<sm_count * kPeakBlocksPerSM, kPeakThreads, 0, s>>>(sink, iters);
    return cudaGetLastError();
}

int64_t fp32_peak_flops(int sm_count, int iters) {
    return static_cast<int64_t>(sm_count) * kPeakBlocksPerSM * kPeakThreads * static_cast<int64_t>(iters) *
           kPeakUnroll * kPeakChains * 2;
}

size_t partial_floats(const DevParams& p, const Launch& L, int64_t n_pad) {
    const int mult = (L.accum == GSPH_ACCUM_COMPENSATED) ? 2 : 1;
    size_t k = 0;
    if (has(p, GSPH_SPH)) {
        const size_t kd = 1;
        const size_t kp = static_cast<size_t>(popc_c(field_mask<PASS_FUSED, true, true>()));
        k = std::max(kd, kp);
        k = std::max<size_t>(k, static_cast<size_t>(popc_c(field_mask<PASS_FUSED, true, false>())));
        k *= static_cast<size_t>(std::max(L.nseg, 1));
    } else {
        k = 3 * static_cast<size_t>(L.grav_sym_G > 0 ? L.grav_sym_G + 1 : std::max(L.grav_nseg, 1));
    }
    return k * mult * static_cast<size_t>(n_pad);
}

int gravity_blocks_per_sm(int ipt, int threads, int jt, bool comp) {
    const size_t smem = pipe_smem_bytes(1, jt);
    int nb = 0;
    cudaError_t e = cudaSuccess;
#define GSPH_OCC(I)                                                                                      \
    e = comp ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_gravity<I, 1, true>, threads, smem)  \
             : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_gravity<I, 1, false>, threads, smem)
    switch (ipt) {
        case 1: GSPH_OCC(1); break;
        case 2: GSPH_OCC(2); break;
        case 8: GSPH_OCC(8); break;
        default: GSPH_OCC(4); break;
    }
#undef GSPH_OCC
    return (e == cudaSuccess && nb > 0) ? nb : 4;
}

// Model of the shapes' times: an SM takes ceil(tasks / SMs) tasks, `ctas` at a time at `rate` interactions per clock (only
// their ratios count; the largest shape now does 13.5); a last round of fewer takes as long as 0.6 of a full one at least
// (a lone CTA does not fill the FMA pipe). Up to 128 groups: N = 262,144 in 17.5 ms against 18.4 ms with 64 (tasks four
// times as large, the last wave 68 % full); 64 above 4 M particles, where a particle's slots would take 1.5 KB.
void sym_shape(int64_t n_pad, int sms, int groups, int shape, Launch& L) {
    const int B[kSymShapes] = {Sym8::B, Sym4::B, Sym2::B, Sym1::B};
    const int ctas[kSymShapes] = {Sym8::CTAS, Sym4::CTAS, Sym2::CTAS, Sym1::CTAS};
    const double rate[kSymShapes] = {14.9, 13.4, 11.0, 10.0};
    const int target = groups ? groups : (n_pad <= (int64_t(1) << 22) ? 128 : 64);
    double best = 1e300;
    for (int k = 0; k < kSymShapes; ++k) {
        if (shape >= 0 && k != shape) continue;
        int G, gs;
        sym_groups(n_pad / B[k], target, G, gs);
        const int64_t per_sm = (static_cast<int64_t>(G) * (G + 1) / 2 + sms - 1) / sms;
        const int64_t full = per_sm / ctas[k], rest = per_sm % ctas[k];
        const double load = static_cast<double>(full * ctas[k]) + (rest ? std::max<double>(rest, 0.6 * ctas[k]) : 0.0);
        const double pairs = static_cast<double>(gs) * B[k] * gs * B[k];
        if (load * pairs / rate[k] < best) {
            best = load * pairs / rate[k];
            L.grav_sym_shape = k;
            L.grav_sym_G = G;
            L.grav_sym_gs = gs;
        }
    }
}

size_t gravity_partial_floats(const Launch& L, int64_t n_pad) {
    const int mult = (L.accum == GSPH_ACCUM_COMPENSATED) ? 2 : 1;
    const int slots = L.grav_sym_G > 0 ? L.grav_sym_G + 1 : std::max(L.grav_nseg, 1);
    return static_cast<size_t>(3) * mult * static_cast<size_t>(slots) * static_cast<size_t>(n_pad);
}

}  // namespace gsph
