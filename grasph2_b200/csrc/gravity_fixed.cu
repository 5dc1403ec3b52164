// gravity_fixed.cu -- symmetric gravity in a kept order of summation.
//
// Two kinds of derivatives amplify a last-place change of the acceleration far beyond rounding. They keep this kernel, and
// the launch shapes that set the order of its sums as a context is made (autotuning may choose others):
//   * network proposals (surrogate_run.cu). The network takes its inputs and keeps its activations in BF16; a change
//     in the last place moves one of them across a rounding boundary every few thousand particles, and one such flip
//     moves a particle's proposed stress by up to 5 % of the stress rms, in the proposal after the one whose acceleration
//     changed. It is the network's own rounding noise, and the error against 64 bits is the same in either order: what is kept
//     is that a context made today proposes what it did when the model was judged;
//   * contexts that integrate the density (GSPH_INTEGRATE_DENSITY). The pressure, and with it the Mohr-Coulomb yield
//     stress, comes from the distance of an FP32 density from rest: in the first steps one last place of the density is
//     0.6 % of it.
// Everything else takes the column-packed kernel of pairs.cu, 1.16 (equal masses: 1.28) times as fast: that is the price,
// 5 of the 22.4 ms of a proposal with 262,144 particles. The results differ in the last places only.
// Both masses multiply 1/r^3 here, so separations must be within 1.5e-13 .. 4.3e12 (gravity_sym.cuh; a
// look-up of far tiles in this kernel cost every proposal 4.5 %).
#include "f32x2.cuh"
#include "gravity_sym.cuh"
#include "pairs.cuh"

namespace gsph {

namespace {

// ================================================================================================
// symmetric all-pairs gravity (Newton's third law): every unordered pair evaluated once
// ================================================================================================
// The row-packed form of the kernel in pairs.cu: a thread's eight row particles in four f32x2 pairs, one column per
// round. Groups, tasks, slots and column rotation as there. Four CTAs per SM (128 registers); the FMA pipe is 72 % busy:
// N = 262,144 in 22.3 ms.
constexpr int kFixT = 128, kFixI = 8, kFixB = kFixT * kFixI, kFixJT = 256;
static_assert(kFixB % kFixJT == 0 && kFixJT % kFixT == 0 && kFixJT % 32 == 0, "symmetric gravity tiles");
constexpr int kFixCtas = 4;

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
    sym_task(static_cast<int>(blockIdx.x), G, ga, gb);
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


template <int GRAV, bool COMP>
void gravity_sym(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s) {
    const int G = L.grav_sym_G;
    k_fixed_gravity_sym<GRAV, COMP><<<static_cast<unsigned>(G * (G + 1) / 2), kFixT, 0, s>>>(a.posm, a.gpart, a.n_pad, G,
                                                                                            L.grav_sym_gs, p.eps2);
}

}  // namespace

cudaError_t launch_fixed_gravity(const DevArrays& a, const DevParams& p, const Launch& L, cudaStream_t s,
                                 const KTimer* t) {
    if (L.grav_sym_G == 0) return launch_gravity_partials(a, p, L, s, t);
    const bool comp = L.accum == GSPH_ACCUM_COMPENSATED;
    cudaError_t e = t ? timer_record(t->start, s) : cudaSuccess;
    if (e != cudaSuccess) return e;
    if (p.eps2 > 0.0f) comp ? gravity_sym<1, true>(a, p, L, s) : gravity_sym<1, false>(a, p, L, s);
    else comp ? gravity_sym<2, true>(a, p, L, s) : gravity_sym<2, false>(a, p, L, s);
    e = cudaGetLastError();
    if (e == cudaSuccess && t) e = timer_record(t->stop, s);
    return e == cudaSuccess ? launch_gravity_fold(a, L, L.grav_sym_G + 1, s, !t) : e;
}


}  // namespace gsph
