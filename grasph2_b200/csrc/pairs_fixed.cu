// pairs_fixed.cu -- the derivatives of a network proposal, in a fixed order of summation.
//
// The surrogate's network (mlp.cu) takes its inputs and keeps its activations in BF16. A last-place change of the
// summed density or acceleration moves an input across a rounding boundary of BF16 every few thousand particles,
// and one such flip moves a particle's proposed stress by up to 5 % of its rms: the network's own rounding noise, but
// another proposal. A trained model is judged and shipped with the proposals it made, so network proposals keep the
// order of summation (and the launch shapes that set it) they have always had, whatever the plain steps do: work items
// of near chunks for the density and SPH sums, the row-packed symmetric gravity kernel. The plain passes (pairs.cu)
// are 1.2 (gravity) to 3 (SPH) times as fast; their results differ in the last places only.
#include <algorithm>

#include "f32x2.cuh"
#include "pairs.cuh"
#include "sph.cuh"

namespace gsph {

namespace {

constexpr int kStageChunks = 4;  // chunks staged per pipeline stage (256 j-particles)
constexpr int kItemNb = 96;      // neighbour-list slots per lane and work item (density pass -> SPH passes)

// Work item w of the culled passes: i-group g, positions [c0, c1) of g's near-chunk list. Items are
// numbered group by group (item_start[g] .. item_start[g+1]-1), at most item_chunks chunks each.
struct CullView {
    const int* list;
    const int* count;
    const int* item_start;  // [ngroups + 2]: first item of each group, the number of items, the
                            // chunks per item (chosen on the device from the total near-chunk count)
    int ngroups;
    int64_t nchunks;        // row stride of `list`
    float* part;            // [item][field][kGroup]
    int* nb;                // nullable: per item, each lane's neighbour indices [item][kItemNb][kGroup] ...
    int* nbcnt;             // ... and their count [item][kGroup] (kItemNb + 1: the list overflowed) ...
    int* nbover;            // ... and per item whether any lane's list overflowed
    const float4* box_lo;   // per-chunk bounding boxes (the culled density pass skips, warp by warp, the
    const float4* box_hi;   // chunks of an item that are farther than h (1 + kMargin) from the warp's box)
    __device__ __forceinline__ int items() const { return item_start[ngroups]; }
    __device__ __forceinline__ void item(int w, int& g, int& c0, int& c1) const {
        int lo = 0, hi = ngroups;  // item_start[lo] <= w < item_start[hi]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (item_start[mid] <= w) lo = mid;
            else hi = mid;
        }
        g = lo;
        const int ic = item_start[ngroups + 1];
        c0 = (w - item_start[g]) * ic;
        c1 = min(c0 + ic, count[g]);
    }
};

// Two-stage pipeline over a list of chunks, kStageChunks chunks per stage; the stage counter runs on
// across items so the mbarrier phases stay in step.
template <int NS>
struct ItemPipe {
    static constexpr int SJ = kStageChunks * kChunk;
    float4* buf;     // shared: [2][NS][SJ]
    uint64_t* bar;   // shared: [2]
    const float4* src[NS];
    int* status;
    uint32_t kst = 0;

    __device__ __forceinline__ void init() {
        if (threadIdx.x == 0) {
            mbar_init(&bar[0], 1);
            mbar_init(&bar[1], 1);
            fence_barrier_init();
        }
        __syncthreads();
    }
    __device__ __forceinline__ void issue(int b, const int* chunks, int first, int nc) {
        mbar_expect_tx(&bar[b], static_cast<uint32_t>(NS * nc * kChunk * sizeof(float4)));
        for (int c = 0; c < nc; ++c) {
            const int64_t ch = chunks[first + c];
#pragma unroll
            for (int s = 0; s < NS; ++s)
                bulk_g2s(buf + (static_cast<int64_t>(b) * NS + s) * SJ + c * kChunk, src[s] + ch * kChunk,
                         static_cast<uint32_t>(kChunk * sizeof(float4)), &bar[b]);
        }
    }
    // body(stage, nj) for every stage of the n chunks chunks[0..n); false if a wait gave up
    template <typename Body>
    __device__ __forceinline__ bool run(const int* chunks, int n, Body&& body) {
        const int nst = (n + kStageChunks - 1) / kStageChunks;
        if (threadIdx.x == 0)
            for (int st = 0; st < 2 && st < nst; ++st)
                issue((kst + st) & 1, chunks, st * kStageChunks, min(kStageChunks, n - st * kStageChunks));
        for (int st = 0; st < nst; ++st) {
            const int b = kst & 1;
            const bool ok = mbar_wait_bounded(&bar[b], (kst >> 1) & 1, status);
            if (__syncthreads_or(!ok)) {
                if (threadIdx.x == 0 && st + 1 < nst)
                    mbar_wait_bounded(&bar[(kst + 1) & 1], ((kst + 1) >> 1) & 1, status);
                __syncthreads();
                return false;
            }
            const int nc = min(kStageChunks, n - st * kStageChunks);
            body(buf + static_cast<int64_t>(b) * NS * SJ, nc * kChunk);
            __syncthreads();
            if (threadIdx.x == 0 && st + 2 < nst)
                issue(b, chunks, (st + 2) * kStageChunks, min(kStageChunks, n - (st + 2) * kStageChunks));
            ++kst;
        }
        return true;
    }
};


// culled density sum over the near-chunk work items (persistent grid); every lane also
// records the indices of its neighbours in this item (for the SPH passes of the same step)
template <bool COMP>
__global__ void __launch_bounds__(kGroup, 12) k_fixed_density(const float4* __restrict__ posm, DevParams p, CullView cv,
                                                          int* status) {
    constexpr int SJ = kStageChunks * kChunk;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ItemPipe<1> pipe;
    pipe.buf = reinterpret_cast<float4*>(smem_raw);
    pipe.bar = reinterpret_cast<uint64_t*>(smem_raw + 2 * SJ * sizeof(float4));
    pipe.src[0] = posm;
    pipe.status = status;
    pipe.init();
    const uint32_t span = __float_as_uint(p.H2);
    const int total = cv.items();
    __shared__ float4 wbox[kGroup / 32][2];  // each warp's bounding box for the current item
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        int g, c0, c1;
        cv.item(w, g, c0, c1);
        const float4 pi = posm[static_cast<int64_t>(g) * kGroup + threadIdx.x];
        float rho_s = 0.0f, rho_c = 0.0f;
        int cnt = 0;
        // the warp's bounding box: a chunk of the group's list that lies farther than h (1 + kMargin)
        // from it (the list's own conservative bound) holds no neighbour of the warp's 32 particles, and
        // the warp skips its tests (same sums, same lists; padding lanes only widen the box)
        {
            float wlo[3] = {pi.x, pi.y, pi.z}, whi[3] = {pi.x, pi.y, pi.z};
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    wlo[c] = fminf(wlo[c], __shfl_xor_sync(0xffffffffu, wlo[c], o));
                    whi[c] = fmaxf(whi[c], __shfl_xor_sync(0xffffffffu, whi[c], o));
                }
            __syncwarp();  // the previous item's reads of this warp's box are done
            if ((threadIdx.x & 31) == 0) {
                wbox[threadIdx.x >> 5][0] = make_float4(wlo[0], wlo[1], wlo[2], 0.0f);
                wbox[threadIdx.x >> 5][1] = make_float4(whi[0], whi[1], whi[2], 0.0f);
            }
            __syncwarp();
        }
        int* lst = cv.nb + static_cast<int64_t>(w) * kItemNb * kGroup + threadIdx.x;
        const int* chunks = cv.list + static_cast<int64_t>(g) * cv.nchunks + c0;
        int chunk_base = 0;
        if (!pipe.run(chunks, c1 - c0, [&](const float4* J, int nj) {
                float t = 0.0f;
                {
                    for (int s0 = 0; s0 < nj; s0 += kChunk) {
                        const int jc = chunks[chunk_base + s0 / kChunk], jb = jc * kChunk;
                        {
                            const float4 l = cv.box_lo[jc], u = cv.box_hi[jc];
                            const float4 wl = wbox[threadIdx.x >> 5][0], wh = wbox[threadIdx.x >> 5][1];
                            const float gx = fmaxf(0.0f, fmaxf(l.x - wh.x, wl.x - u.x)),
                                        gy = fmaxf(0.0f, fmaxf(l.y - wh.y, wl.y - u.y)),
                                        gz = fmaxf(0.0f, fmaxf(l.z - wh.z, wl.z - u.z));
                            const float hm = p.H * (1.0f + kMargin);
                            if (gx * gx + gy * gy + gz * gz > hm * hm) continue;  // warp-uniform
                        }
                        // the chunk's 64 tests into a bit mask without branches, then its set bits in
                        // ascending order (the neighbours, about 2 % of the tests)
                        unsigned m8[8];
#pragma unroll
                        for (int b = 0; b < 8; ++b) {
                            unsigned m = 0;
#pragma unroll
                            for (int u = 0; u < 8; ++u) {
                                const float4 q = J[s0 + b * 8 + u];
                                const float dx = q.x - pi.x, dy = q.y - pi.y, dz = q.z - pi.z;
                                const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                                m |= static_cast<unsigned>(in_open_closed(r2, 0u, span)) << u;
                            }
                            m8[b] = m;
                        }
                        uint64_t bits = static_cast<uint64_t>(m8[0] | (m8[1] << 8) | (m8[2] << 16) | (m8[3] << 24)) |
                                        (static_cast<uint64_t>(m8[4] | (m8[5] << 8) | (m8[6] << 16) | (m8[7] << 24)) << 32);
                        while (bits) {
                            const int j = __ffsll(static_cast<long long>(bits)) - 1;
                            bits &= bits - 1;
                            const float4 q = J[s0 + j];
                            const float dx = q.x - pi.x, dy = q.y - pi.y, dz = q.z - pi.z;
                            const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                            const float r = r2 * rsqrtf(r2);
                            t = fmaf(q.w, w_poly(r * p.inv_h), t);
                            if (cnt < kItemNb) lst[cnt * kGroup] = jb + j;
                            ++cnt;
                        }
                    }
                    chunk_base += nj / kChunk;
                }
                if (COMP) fold(rho_s, rho_c, t);
                else rho_s += t;
            }))
            return;
        float* out = cv.part + static_cast<int64_t>(w) * (COMP ? 2 : 1) * kGroup + threadIdx.x;
        out[0] = rho_s;
        if (COMP) out[kGroup] = rho_c;
        {
            cv.nbcnt[static_cast<int64_t>(w) * kGroup + threadIdx.x] = min(cnt, kItemNb + 1);
            const int over = __syncthreads_or(cnt > kItemNb);  // the SPH passes read one flag per item
            if (threadIdx.x == 0) cv.nbover[w] = over;
        }
    }
}


// the partial sums of an item: field o at out[o * kGroup]
template <uint32_t MASK>
__device__ __forceinline__ void store_item(float* out, const PairAcc& T, float maxv) {
#pragma unroll
    for (int f = 0; f < F_COUNT; ++f)
        if ((MASK >> f) & 1u) out[field_offset<MASK>(f) * kGroup] = (f == F_MAXV) ? maxv : T.f[f];
}

// Culled SPH pass (no gravity): a persistent grid walks the work items; item w covers some near
// chunks of one i-group and writes its partials to part[w][field][kGroup]. Phase 1 streams only the
// positions of those chunks through shared memory and lets every lane record the indices of its own
// neighbours (kNbCap per lane, flushed early when a lane's list is nearly full); phase 2 walks the
// per-lane lists and gathers each neighbour's records from L2, so the SPH terms run lane-dense.
constexpr int kNbCap = 64;
template <int PASS, bool SOLIDS>
__global__ void __launch_bounds__(kGroup, 5) k_fixed_pairs(DevArrays a, DevParams p, CullView cv) {
    constexpr uint32_t MASK = field_mask<PASS, false, SOLIDS>();
    constexpr int K = popc_c(MASK);
    constexpr bool DO_A = PASS != PASS_VGRAD;
    constexpr int SJ = kStageChunks * kChunk;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ItemPipe<1> pipe;
    pipe.buf = reinterpret_cast<float4*>(smem_raw);
    pipe.bar = reinterpret_cast<uint64_t*>(smem_raw + 2 * SJ * sizeof(float4));
    pipe.src[0] = a.posm;
    pipe.status = a.status;
    const int lane = threadIdx.x & 31;
    int* nb = reinterpret_cast<int*>(smem_raw + pipe_smem_bytes(1, SJ)) + (threadIdx.x >> 5) * (kNbCap * 32);
    pipe.init();
    const int total = cv.items();
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        int g, c0, c1;
        cv.item(w, g, c0, c1);
        const int64_t i = static_cast<int64_t>(g) * kGroup + threadIdx.x;
        const ISph I = load_isph<PASS, SOLIDS>(a, p, i, 0.0f);
        PairAcc T;
#pragma unroll
        for (int f = 0; f < F_COUNT; ++f) T.f[f] = 0.0f;
        float maxv = 0.0f;
        // the density pass's neighbour lists of this item, when every lane's list is complete (one flag
        // per item, so no block-wide vote: the warps of a block run through list items independently)
        if (cv.nb && cv.nbover[w] == 0) {
            const int lcnt = cv.nbcnt[static_cast<int64_t>(w) * kGroup + threadIdx.x];
            const int* lst = cv.nb + static_cast<int64_t>(w) * kItemNb * kGroup + threadIdx.x;
            const float4 zero = make_float4(0, 0, 0, 0);
            const int j0 = lcnt > 0 ? lst[0] : 0;
            int jn = lcnt > 1 ? lst[kGroup] : 0;  // the index of neighbour k+1
            const float4* r0 = a.jrec + 4 * static_cast<int64_t>(j0);  // one 64-byte record per neighbour
            float4 qn = __ldg(r0), vn = __ldg(r0 + 1);
            float4 an = DO_A ? __ldg(r0 + 2) : zero, bn = DO_A ? __ldg(r0 + 3) : zero;
            // software pipeline: neighbour k+1's records and neighbour k+2's index in flight during k
            for (int k = 0; k < lcnt; ++k) {
                const float4 q = qn, vj = vn, ja = an, jb = bn;
                if (k + 1 < lcnt) {
                    const float4* r = a.jrec + 4 * static_cast<int64_t>(jn);
                    qn = __ldg(r);
                    vn = __ldg(r + 1);
                    if (DO_A) {
                        an = __ldg(r + 2);
                        bn = __ldg(r + 3);
                    }
                }
                if (k + 2 < lcnt) jn = lst[(k + 2) * kGroup];
                const float dx = q.x - I.pi.x, dy = q.y - I.pi.y, dz = q.z - I.pi.z;
                const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                sph_neighbour<PASS, SOLIDS>(T, maxv, I, q.w, dx, dy, dz, r2, vj, ja, jb, p);
            }
            store_item<MASK>(cv.part + static_cast<int64_t>(w) * K * kGroup + threadIdx.x, T, maxv);
            continue;
        }
        int cnt = 0;
        // phase 2 over the lane lists collected so far
        auto drain = [&]() {
            int m = cnt;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
            // software pipeline: the records of neighbour k+1 are in flight while k is computed
            const float4 zero = make_float4(0, 0, 0, 0);
            int jn = cnt > 0 ? nb[lane] : 0;
            const float4* r0 = a.jrec + 4 * static_cast<int64_t>(jn);
            float4 qn = __ldg(r0), vn = __ldg(r0 + 1);
            float4 an = DO_A ? __ldg(r0 + 2) : zero, bn = DO_A ? __ldg(r0 + 3) : zero;
            for (int k = 0; k < m; ++k) {
                const float4 q = qn, vj = vn, ja = an, jb = bn;
                if (k + 1 < cnt) {
                    jn = nb[(k + 1) * 32 + lane];
                    const float4* r = a.jrec + 4 * static_cast<int64_t>(jn);
                    qn = __ldg(r);
                    vn = __ldg(r + 1);
                    if (DO_A) {
                        an = __ldg(r + 2);
                        bn = __ldg(r + 3);
                    }
                }
                if (k < cnt) {
                    const float dx = q.x - I.pi.x, dy = q.y - I.pi.y, dz = q.z - I.pi.z;
                    const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                    sph_neighbour<PASS, SOLIDS>(T, maxv, I, q.w, dx, dy, dz, r2, vj, ja, jb, p);
                }
            }
            cnt = 0;
            __syncwarp();
        };
        const int* chunks = cv.list + static_cast<int64_t>(g) * cv.nchunks + c0;
        int chunk_base = 0;  // position in `chunks` of the current stage
        if (!pipe.run(chunks, c1 - c0, [&](const float4* J, int nj) {
                for (int s0 = 0; s0 < nj; s0 += kChunk) {
                    const int jbase = chunks[chunk_base + s0 / kChunk] * kChunk;
                    // 64 independent tests into eight 8-bit masks (no serial chain), then the set bits
                    unsigned m8[8];
#pragma unroll
                    for (int b = 0; b < 8; ++b) {
                        unsigned m = 0;
#pragma unroll
                        for (int t = 0; t < 8; ++t) {
                            const float4 q = J[s0 + b * 8 + t];
                            const float dx = q.x - I.pi.x, dy = q.y - I.pi.y, dz = q.z - I.pi.z;
                            const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                            m |= static_cast<unsigned>(in_open_closed(r2, 0u, I.span)) << t;
                        }
                        m8[b] = m;
                    }
                    unsigned lo = m8[0] | (m8[1] << 8) | (m8[2] << 16) | (m8[3] << 24);
                    unsigned hi = m8[4] | (m8[5] << 8) | (m8[6] << 16) | (m8[7] << 24);
                    while (lo) {
                        nb[cnt * 32 + lane] = jbase + __ffs(lo) - 1;
                        ++cnt;
                        lo &= lo - 1u;
                    }
                    while (hi) {
                        nb[cnt * 32 + lane] = jbase + 32 + __ffs(hi) - 1;
                        ++cnt;
                        hi &= hi - 1u;
                    }
                    // a lane could overflow on the next chunk: process the lists now
                    if (__any_sync(0xffffffffu, cnt > kNbCap - kChunk)) drain();
                }
                chunk_base += nj / kChunk;
            }))
            return;
        drain();
        store_item<MASK>(cv.part + static_cast<int64_t>(w) * K * kGroup + threadIdx.x, T, maxv);
    }
}



// ---- the items of a particle, added in their order (compensated: in FP64) ----------------------------
template <bool COMP>
__global__ void k_fixed_density_finish(DevArrays a, DevParams p, CullView cv) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const int64_t g = i / kGroup, l = i % kGroup;
    float rho;
    if (COMP) {
        double s = 0.0;
        for (int k = cv.item_start[g]; k < cv.item_start[g + 1]; ++k)
            s += static_cast<double>(cv.part[static_cast<int64_t>(k) * 2 * kGroup + l]) +
                 static_cast<double>(cv.part[(static_cast<int64_t>(k) * 2 + 1) * kGroup + l]);
        rho = static_cast<float>(s * static_cast<double>(p.w_pref));
    } else {
        float s = 0.0f;
        for (int k = cv.item_start[g]; k < cv.item_start[g + 1]; ++k) s += cv.part[static_cast<int64_t>(k) * kGroup + l];
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
    float4* r = a.jrec + 4 * i;
    r[0] = a.posm[i]; r[1] = vr; r[2] = jA; r[3] = jB;
}

template <int PASS, bool SOLIDS, bool COMP>
__global__ void k_fixed_finish(DevArrays a, DevParams p, CullView cv, bool grav) {
    constexpr uint32_t MASK = field_mask<PASS, false, SOLIDS>();
    constexpr int K = popc_c(MASK);
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (PASS != PASS_VGRAD && has(p, GSPH_VARIABLE_TIMESTEP) && i == 0) a.dt_state[1] = p.max_dt;
    if (i >= a.n) return;
    float g[3] = {0.0f, 0.0f, 0.0f};
    grav = grav && PASS != PASS_VGRAD;
    if (grav)
        for (int c = 0; c < 3; ++c) g[c] = static_cast<float>(a.gfold[c * a.n_pad + i]);
    const int b = cv.item_start[i / kGroup], e = cv.item_start[i / kGroup + 1];
    auto at = [&](int k, int o) { return cv.part[(static_cast<int64_t>(k) * K + o) * kGroup + i % kGroup]; };
    sph_finish<PASS, SOLIDS>(a, p, i, [&](int f) {
        const int o = field_offset<MASK>(f);
        if (f == F_MAXV) {
            float m = 0.0f;
            for (int k = b; k < e; ++k) m = fmaxf(m, at(k, o));
            return m;
        }
        if (COMP) {
            double s = 0.0;
            for (int k = b; k < e; ++k) s += static_cast<double>(at(k, o));
            return static_cast<float>(s);
        }
        float s = 0.0f;
        for (int k = b; k < e; ++k) s += at(k, o);
        return s;
    }, grav, g);
}

// One block: chunks per item ic = ceil(total near chunks / target) so that items carry equal work,
// then the exclusive scan of the per-group item counts ceil(count / ic) in a fixed order.
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads) k_fixed_items(const int* __restrict__ count, int* __restrict__ start,
                                                             int ngroups, int target) {
    __shared__ int warp_sums[kScanThreads / 32];
    __shared__ int carry;
    __shared__ int ic_sh;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int part = 0;  // total near chunks
    for (int g = threadIdx.x; g < ngroups; g += kScanThreads) part += count[g];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) warp_sums[warp] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long total = 0;
        for (int w = 0; w < kScanThreads / 32; ++w) total += warp_sums[w];
        const long long ic = (total + target - 1) / target;
        ic_sh = static_cast<int>(ic < 1 ? 1 : ic);
        carry = 0;
    }
    __syncthreads();
    const int ic = ic_sh;
    for (int base = 0; base < ngroups; base += kScanThreads) {
        const int g = base + threadIdx.x;
        const int v = (g < ngroups) ? (count[g] + ic - 1) / ic : 0;
        int x = v;  // inclusive warp scan
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        __syncthreads();
        if (lane == 31) warp_sums[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int w = warp_sums[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            warp_sums[lane] = w;  // inclusive over warps
        }
        __syncthreads();
        const int before = carry + (warp ? warp_sums[warp - 1] : 0) + x - v;
        if (g < ngroups) start[g] = before;
        __syncthreads();
        if (threadIdx.x == kScanThreads - 1) carry = before + v;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        start[ngroups] = carry;
        start[ngroups + 1] = ic;
    }
}

// ================================================================================================
// symmetric all-pairs gravity (Newton's third law): every unordered pair evaluated once
// ================================================================================================
// The row-packed form of the kernel in pairs.cu: a thread's eight row particles in four f32x2 pairs, one column per
// round. Groups, tasks, slots and column rotation as there. Four CTAs per SM (128 registers); the FMA pipe is 72 % busy:
// N = 262,144 in 22.3 ms.
constexpr int kFixT = 128, kFixI = 8, kFixB = kFixT * kFixI, kFixJT = 256;
static_assert(kFixB % kFixJT == 0 && kFixJT % kFixT == 0 && kFixJT % 32 == 0, "symmetric gravity tiles");
constexpr int kFixCtas = 4;

__host__ __device__ __forceinline__ void fixed_sym_task(int t, int G, int& ga, int& gb) {
    const int noff = G * (G - 1) / 2;
    if (t >= noff) {
        ga = gb = t - noff;
        return;
    }
    int r = 0, rem = t;
    while (rem >= G - 1 - r) {
        rem -= G - 1 - r;
        ++r;
    }
    ga = r;
    gb = r + 1 + rem;
}

template <int GRAV, bool COMP>
__global__ void __launch_bounds__(kFixT, kFixCtas) k_fixed_gravity_sym(const float4* __restrict__ posm, float* __restrict__ part,
                                                       int64_t n_pad, int G, int gs, float eps2) {
    constexpr int P = kFixI / 2;
    constexpr int K = COMP ? 6 : 3;
    __shared__ float4 J[kFixJT];
    __shared__ float js[kFixT / 32][kFixJT][3];
    // the row particles' running sums (and, compensated, their rounding-error terms) stay in shared
    // memory, touched once per j-tile; the pair loop keeps only the tile's partials in registers
    __shared__ float2 rsh[3 * P][kFixT];
    __shared__ float2 csh[COMP ? 3 * P : 1][kFixT];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int ga, gb;
    fixed_sym_task(static_cast<int>(blockIdx.x), G, ga, gb);
    const int nb = static_cast<int>(n_pad / kFixB);
    const int ra0 = ga * gs, ra1 = min(nb, ra0 + gs);
    const int cg0 = gb * gs, cg1 = min(nb, cg0 + gs);
    const bool diag = ga == gb;
    // partials: G + 1 slots per particle, stored [slot][component][n_pad] so that a warp's 32 consecutive
    // particles write (and the fold kernel reads) 128 contiguous bytes; a particle of group g holds its row
    // sums from tasks (g, gb), gb = g .. G-1, in slots 0 .. G-1-g and its column sums from tasks (ga, g),
    // ga = 0 .. g, in slots G-g .. G, each slot written by exactly one task
    const int s_row = gb - ga, s_col = G - gb + ga;
    auto slot = [&](int64_t particle, int sl, int c) { return part + (static_cast<int64_t>(sl) * K + c) * n_pad + particle; };
    if (diag)  // the group's first block is never a column here: its column slot is zero
        for (int e = tid; e < kFixB; e += kFixT)
            for (int c = 0; c < K; ++c) *slot(static_cast<int64_t>(ra0) * kFixB + e, s_col, c) = 0.0f;
    const float2 E2 = make_float2(eps2, eps2);

    for (int a = ra0; a < ra1; ++a) {
        const int64_t base = static_cast<int64_t>(a) * kFixB + tid;
        float2 X[P], Y[P], Z[P], MI[P];
#pragma unroll
        for (int k = 0; k < P; ++k) {
            const float4 u = posm[base + static_cast<int64_t>(2 * k) * kFixT];
            const float4 w = posm[base + static_cast<int64_t>(2 * k + 1) * kFixT];
            X[k] = make_float2(u.x, w.x); Y[k] = make_float2(u.y, w.y); Z[k] = make_float2(u.z, w.z);
            MI[k] = make_float2(-u.w, -w.w);
            rsh[k][tid] = rsh[P + k][tid] = rsh[2 * P + k][tid] = make_float2(0.0f, 0.0f);
            if (COMP) csh[k][tid] = csh[P + k][tid] = csh[2 * P + k][tid] = make_float2(0.0f, 0.0f);
        }
        // tiles: the block's own (one-sided) when diagonal, then the columns
        const int64_t d0 = static_cast<int64_t>(a) * kFixB;
        const int nd = diag ? kFixB / kFixJT : 0;
        const int64_t c0 = static_cast<int64_t>(diag ? a + 1 : cg0) * kFixB, c1 = static_cast<int64_t>(cg1) * kFixB;
        const int nc = c1 > c0 ? static_cast<int>((c1 - c0) / kFixJT) : 0;
        const int total = nd + nc;
        const bool first = a == ra0;
        auto src = [&](int k) { return k < nd ? d0 + static_cast<int64_t>(k) * kFixJT : c0 + static_cast<int64_t>(k - nd) * kFixJT; };
        constexpr int kPf = kFixJT / kFixT;  // j-records each thread stages per tile
        float4 pf[kPf];
#pragma unroll
        for (int h = 0; h < kPf; ++h) pf[h] = make_float4(0, 0, 0, 0);
        if (total > 0) {
#pragma unroll
            for (int h = 0; h < kPf; ++h) pf[h] = posm[src(0) + h * kFixT + tid];
        }
        for (int k = 0; k < total; ++k) {
            __syncthreads();  // the previous tile's reads of J and js are done
#pragma unroll
            for (int h = 0; h < kPf; ++h) J[tid + h * kFixT] = pf[h];
            __syncthreads();
            if (k + 1 < total) {
#pragma unroll
                for (int h = 0; h < kPf; ++h) pf[h] = posm[src(k + 1) + h * kFixT + tid];
            }
            float2 TX[P], TY[P], TZ[P];
#pragma unroll
            for (int q = 0; q < P; ++q) TX[q] = TY[q] = TZ[q] = make_float2(0.0f, 0.0f);
            if (k < nd) {  // one-sided, as k_gravity_x2
#pragma unroll 4
                for (int j = 0; j < kFixJT; ++j) {
                    const float4 q = J[j];
                    const float2 qx = make_float2(q.x, q.x), qy = make_float2(q.y, q.y), qz = make_float2(q.z, q.z),
                                 qm = make_float2(q.w, q.w);
#pragma unroll
                    for (int m = 0; m < P; ++m) {
                        const float2 dx = sub2(qx, X[m]), dy = sub2(qy, Y[m]), dz = sub2(qz, Z[m]);
                        const float2 r2 = fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, E2)));
                        float2 inv = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
                        if (GRAV == 2) inv = make_float2(fminf(inv.x, 1e12f), fminf(inv.y, 1e12f));
                        const float2 sj = mul2(qm, mul2(mul2(inv, inv), inv));
                        TX[m] = fma2(dx, sj, TX[m]); TY[m] = fma2(dy, sj, TY[m]); TZ[m] = fma2(dz, sj, TZ[m]);
                    }
                }
            } else {
                // column sums by rotation: in round r of a block of 32 columns, lane l pairs its rows
                // with column (l + r) % 32, adds its share to that column's running sum and hands the sum
                // to lane l - 1, which takes the column in round r + 1; after 32 rounds lane l holds the
                // warp's sum for column l (no butterfly, no selects, 3 shuffles per column)
                const int next = (lane + 1) & 31;
#pragma unroll 1
                for (int j0 = 0; j0 < kFixJT; j0 += 32) {
                    float cx = 0.0f, cy = 0.0f, cz = 0.0f;
#pragma unroll 2
                    for (int r = 0; r < 32; ++r) {
                        const float4 q = J[j0 + ((lane + r) & 31)];
                        const float2 qx = make_float2(q.x, q.x), qy = make_float2(q.y, q.y),
                                     qz = make_float2(q.z, q.z), qm = make_float2(q.w, q.w);
                        float2 tx = make_float2(0.0f, 0.0f), ty = tx, tz = tx;
#pragma unroll
                        for (int m = 0; m < P; ++m) {
                            const float2 dx = sub2(qx, X[m]), dy = sub2(qy, Y[m]), dz = sub2(qz, Z[m]);
                            const float2 r2 = fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, E2)));
                            float2 inv = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
                            if (GRAV == 2) inv = make_float2(fminf(inv.x, 1e12f), fminf(inv.y, 1e12f));
                            const float2 i3 = mul2(mul2(inv, inv), inv);
                            const float2 sj = mul2(qm, i3), si = mul2(MI[m], i3);
                            TX[m] = fma2(dx, sj, TX[m]); TY[m] = fma2(dy, sj, TY[m]); TZ[m] = fma2(dz, sj, TZ[m]);
                            tx = fma2(dx, si, tx); ty = fma2(dy, si, ty); tz = fma2(dz, si, tz);
                        }
                        cx = __shfl_sync(0xffffffffu, cx + (tx.x + tx.y), next);
                        cy = __shfl_sync(0xffffffffu, cy + (ty.x + ty.y), next);
                        cz = __shfl_sync(0xffffffffu, cz + (tz.x + tz.y), next);
                    }
                    js[warp][j0 + lane][0] = cx;
                    js[warp][j0 + lane][1] = cy;
                    js[warp][j0 + lane][2] = cz;
                }
            }
            // the tile's row partials into the running sums: a two-sum fold (compensated), or one add
            // (plain: a sum of 256-term tile sums, not one running sum over the whole column group)
#pragma unroll
            for (int m = 0; m < P; ++m) {
                float2 ax = rsh[m][tid], ay = rsh[P + m][tid], az = rsh[2 * P + m][tid];
                if (COMP) {
                    float2 cx = csh[m][tid], cy = csh[P + m][tid], cz = csh[2 * P + m][tid];
                    fold(ax.x, cx.x, TX[m].x); fold(ax.y, cx.y, TX[m].y);
                    fold(ay.x, cy.x, TY[m].x); fold(ay.y, cy.y, TY[m].y);
                    fold(az.x, cz.x, TZ[m].x); fold(az.y, cz.y, TZ[m].y);
                    csh[m][tid] = cx; csh[P + m][tid] = cy; csh[2 * P + m][tid] = cz;
                } else {
                    ax = add2(ax, TX[m]); ay = add2(ay, TY[m]); az = add2(az, TZ[m]);
                }
                rsh[m][tid] = ax; rsh[P + m][tid] = ay; rsh[2 * P + m][tid] = az;
            }
            if (k >= nd) {  // this tile's column sums over the CTA's row block, into the column slot
                __syncthreads();
                const int64_t jb = c0 + static_cast<int64_t>(k - nd) * kFixJT;
#pragma unroll
                for (int h = 0; h < kFixJT / kFixT; ++h) {
                    const int j = tid + h * kFixT;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float v = (js[0][j][c] + js[1][j][c]) + (js[2][j][c] + js[3][j][c]);
                        float* dst = slot(jb + j, s_col, c);
                        if (COMP) {
                            float* cdst = slot(jb + j, s_col, 3 + c);
                            if (first) {
                                *dst = v;
                                *cdst = 0.0f;
                            } else {
                                float sv = *dst, cv = *cdst;
                                fold(sv, cv, v);
                                *dst = sv;
                                *cdst = cv;
                            }
                        } else {
                            *dst = first ? v : *dst + v;
                        }
                    }
                }
            }
        }
        // the row sums of block a into its row slot
#pragma unroll
        for (int m = 0; m < P; ++m) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t pr = base + static_cast<int64_t>(2 * m + h) * kFixT;
                *slot(pr, s_row, 0) = h ? rsh[m][tid].y : rsh[m][tid].x;
                *slot(pr, s_row, 1) = h ? rsh[P + m][tid].y : rsh[P + m][tid].x;
                *slot(pr, s_row, 2) = h ? rsh[2 * P + m][tid].y : rsh[2 * P + m][tid].x;
                if (COMP) {
                    *slot(pr, s_row, 3) = h ? csh[m][tid].y : csh[m][tid].x;
                    *slot(pr, s_row, 4) = h ? csh[P + m][tid].y : csh[P + m][tid].x;
                    *slot(pr, s_row, 5) = h ? csh[2 * P + m][tid].y : csh[2 * P + m][tid].x;
                }
            }
        }
    }
}


inline unsigned blocks_for(int64_t n, int t) { return static_cast<unsigned>((n + t - 1) / t); }

CullView view(const DevArrays& a, const SpatialArrays& sp, const FixedArrays& fx, bool lists) {
    CullView cv;
    cv.list = sp.list;
    cv.count = sp.count;
    cv.item_start = fx.item_start;
    cv.ngroups = static_cast<int>(a.n_pad / kGroup);
    cv.nchunks = a.n_pad / kChunk;
    cv.part = fx.part;
    cv.nb = lists ? fx.nb : nullptr;
    cv.nbcnt = lists ? fx.nbcnt : nullptr;
    cv.nbover = lists ? fx.nbover : nullptr;
    cv.box_lo = sp.box_lo;
    cv.box_hi = sp.box_hi;
    return cv;
}

template <int PASS, bool SOLIDS>
cudaError_t pass_t(const DevArrays& a, const DevParams& p, const CullView& cv, bool comp, bool grav, int sms, cudaEvent_t join,
                   cudaStream_t s) {
    const size_t smem = pipe_smem_bytes(1, kStageChunks * kChunk) + (kGroup / 32) * kNbCap * 32 * sizeof(int);
    k_fixed_pairs<PASS, SOLIDS><<<sms * 5, kGroup, smem, s>>>(a, p, cv);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && join) e = cudaStreamWaitEvent(s, join, 0);
    if (e != cudaSuccess) return e;
    if (comp) k_fixed_finish<PASS, SOLIDS, true><<<blocks_for(a.n, 256), 256, 0, s>>>(a, p, cv, grav);
    else k_fixed_finish<PASS, SOLIDS, false><<<blocks_for(a.n, 256), 256, 0, s>>>(a, p, cv, grav);
    return cudaGetLastError();
}
template <int PASS>
cudaError_t pass(const DevArrays& a, const DevParams& p, const CullView& cv, bool comp, bool grav, int sms, cudaEvent_t join,
                 cudaStream_t s) {
    return has(p, GSPH_SOLIDS) ? pass_t<PASS, true>(a, p, cv, comp, grav, sms, join, s)
                               : pass_t<PASS, false>(a, p, cv, comp, grav, sms, join, s);
}

template <int GRAV, bool COMP>
void gravity_sym(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s) {
    const int G = L.grav_sym_G;
    k_fixed_gravity_sym<GRAV, COMP><<<static_cast<unsigned>(G * (G + 1) / 2), kFixT, 0, s>>>(a.posm, a.gpart, a.n_pad, G,
                                                                                            L.grav_sym_gs, p.eps2);
}

}  // namespace

// sums of item partials at most `target` items in total plus one per group for rounding
size_t fixed_items(int64_t n_pad, int sms) {
    return static_cast<size_t>(30) * sms + static_cast<size_t>(n_pad / kGroup);
}
size_t fixed_part_floats() { return 2 * static_cast<size_t>(popc_c(field_mask<PASS_FUSED, false, true>())) * kGroup; }
size_t fixed_list_ints() { return static_cast<size_t>(kItemNb) * kGroup; }

cudaError_t launch_fixed_gravity(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s) {
    if (L.grav_sym_G == 0) return launch_gravity_partials(a, p, L, s);
    const bool comp = L.accum == GSPH_ACCUM_COMPENSATED;
    if (p.eps2 > 0.0f) comp ? gravity_sym<1, true>(a, p, L, s) : gravity_sym<1, false>(a, p, L, s);
    else comp ? gravity_sym<2, true>(a, p, L, s) : gravity_sym<2, false>(a, p, L, s);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? launch_gravity_fold(a, L, L.grav_sym_G + 1, s) : e;
}

cudaError_t launch_fixed_sph(const DevArrays& a, const DevParams& p, const Launch& L, const SpatialArrays& sp,
                             const FixedArrays& fx, int sms, bool grav, cudaEvent_t join, cudaStream_t s, int& launches) {
    const bool comp = L.accum == GSPH_ACCUM_COMPENSATED;
    const bool summed = !has(p, GSPH_INTEGRATE_DENSITY), bals = has(p, GSPH_BALSARA_SWITCH);
    const bool vgrad = has(p, GSPH_SOLIDS) || !summed || bals;
    k_fixed_items<<<1, kScanThreads, 0, s>>>(sp.count, fx.item_start, static_cast<int>(a.n_pad / kGroup), 30 * sms);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    ++launches;
    const CullView cv = view(a, sp, fx, summed);
    if (summed) {
        const size_t smem = pipe_smem_bytes(1, kStageChunks * kChunk);
        if (comp) {
            k_fixed_density<true><<<sms * 12, kGroup, smem, s>>>(a.posm, p, cv, a.status);
            k_fixed_density_finish<true><<<blocks_for(a.n, 256), 256, 0, s>>>(a, p, cv);
        } else {
            k_fixed_density<false><<<sms * 12, kGroup, smem, s>>>(a.posm, p, cv, a.status);
            k_fixed_density_finish<false><<<blocks_for(a.n, 256), 256, 0, s>>>(a, p, cv);
        }
        e = cudaGetLastError();
        launches += 2;
    } else {
        e = launch_prepare(a, p, s);
        launches += 1;
    }
    if (e != cudaSuccess) return e;
    launches += 2;
    if (vgrad && bals) {
        e = pass<PASS_VGRAD>(a, p, cv, comp, false, sms, nullptr, s);
        if (e != cudaSuccess) return e;
        launches += 2;
        return pass<PASS_ACC>(a, p, cv, comp, grav, sms, join, s);
    }
    return vgrad ? pass<PASS_FUSED>(a, p, cv, comp, grav, sms, join, s) : pass<PASS_ACC>(a, p, cv, comp, grav, sms, join, s);
}

}  // namespace gsph
