// gravity_sym.cuh -- the inner parts of symmetric gravity: a block of rows in registers against a tile of columns in
// shared memory, every unordered pair once. Used by the all-pairs kernel (pairs.cu, which explains the layout) and the
// ensemble's (ensemble.cu); gravity_fixed.cu shares its tasks.
#pragma once

#include "common.cuh"
#include "f32x2.cuh"

namespace gsph {

template <int R_, int T_, int CTAS_>
struct SymShape {
    static constexpr int R = R_, T = T_, B = R_ * T_, CTAS = CTAS_;
    static constexpr int JT = B < 256 ? B : 256;  // columns per tile
    static constexpr int PF = JT / T_;            // records a thread stages
    static constexpr int W = T_ / 32;
    static_assert(JT % 64 == 0 && B % JT == 0 && JT % T_ == 0, "symmetric gravity tiles");
};

// the groups ga <= gb of task t: the G (G - 1) / 2 pairs of distinct groups first, then the G diagonal ones
__host__ __device__ __forceinline__ void sym_task(int t, int G, int& ga, int& gb) {
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

// T += d s, c += d s for the three components: each pair of multiply-adds with common factors back to back
__device__ __forceinline__ void add_both(float2& tx, float2& ty, float2& tz, float2& cx, float2& cy, float2& cz, float2 dx,
                                         float2 dy, float2 dz, float2 s) {
    uint64_t t0 = u64_of(tx), t1 = u64_of(ty), t2 = u64_of(tz), c0 = u64_of(cx), c1 = u64_of(cy), c2 = u64_of(cz);
    asm("fma.rn.f32x2 %0, %6, %9, %0;\n fma.rn.f32x2 %3, %6, %9, %3;\n"
        " fma.rn.f32x2 %1, %7, %9, %1;\n fma.rn.f32x2 %4, %7, %9, %4;\n"
        " fma.rn.f32x2 %2, %8, %9, %2;\n fma.rn.f32x2 %5, %8, %9, %5;\n"
        : "+l"(t0), "+l"(t1), "+l"(t2), "+l"(c0), "+l"(c1), "+l"(c2)
        : "l"(u64_of(dx)), "l"(u64_of(dy)), "l"(u64_of(dz)), "l"(u64_of(s)));
    tx = f2_of(t0); ty = f2_of(t1); tz = f2_of(t2);
    cx = f2_of(c0); cy = f2_of(c1); cz = f2_of(c2);
}

// a thread's rows, duplicated into both halves and negated (a difference is an addition, a column's share a product)
template <typename S>
struct SymRows {
    float2 X[S::R], Y[S::R], Z[S::R], M[S::R];
    float2 TX[S::R], TY[S::R], TZ[S::R];  // sums over the tile
    __device__ __forceinline__ void set(int k, float4 u) {
        X[k] = make_float2(-u.x, -u.x); Y[k] = make_float2(-u.y, -u.y);
        Z[k] = make_float2(-u.z, -u.z); M[k] = make_float2(-u.w, -u.w);
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int q = 0; q < S::R; ++q) TX[q] = TY[q] = TZ[q] = make_float2(0.0f, 0.0f);
    }
};

// record j of a tile into its column pair (j with j + 32 in blocks of 64): xy = (x x' y y'), zm = (z z' m m')
__device__ __forceinline__ void sym_stage(float4* XY, float4* ZM, int j, float4 r) {
    const int half = (j >> 5) & 1, q = (j >> 6) * 32 + (j & 31);
    float* xy = reinterpret_cast<float*>(&XY[q]);
    float* zm = reinterpret_cast<float*>(&ZM[q]);
    xy[half] = r.x; xy[2 + half] = r.y;
    zm[half] = r.z; zm[2 + half] = r.w;
}

// the separations of row m from a column pair, and 1/r
template <typename S, int GRAV>
__device__ __forceinline__ float2 sym_pair(const SymRows<S>& r, int m, float4 xy, float4 zm, float2 E2, float2& dx, float2& dy,
                                           float2& dz) {
    dx = add2(make_float2(xy.x, xy.y), r.X[m]);
    dy = add2(make_float2(xy.z, xy.w), r.Y[m]);
    dz = add2(make_float2(zm.x, zm.y), r.Z[m]);
    const float2 r2 = fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, E2)));
    float2 inv = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
    if (GRAV == 2) inv = make_float2(fminf(inv.x, 1e12f), fminf(inv.y, 1e12f));
    return inv;
}
__device__ __forceinline__ float2 cube2(float2 v) { return mul2(mul2(v, v), v); }

// the rows against every column pair of the tile: row sums into r, the warp's column sums into js[component][column].
// EQ: neither carries the masses (rows times the columns' mass, columns times minus the rows' are the caller's).
template <typename S, int GRAV, bool EQ>
__device__ __forceinline__ void sym_columns(SymRows<S>& rows, const float4* XY, const float4* ZM, float2 E2,
                                            float (*js)[S::JT]) {
    const int lane = threadIdx.x & 31, next = (lane + 1) & 31;
#pragma unroll 1
    for (int j0 = 0; j0 < S::JT / 2; j0 += 32) {
        float2 cx = make_float2(0.0f, 0.0f), cy = cx, cz = cx;
#pragma unroll 2
        for (int r = 0; r < 32; ++r) {
            const int j = j0 + ((lane + r) & 31);
            const float4 xy = XY[j], zm = ZM[j];
#pragma unroll
            for (int m = 0; m < S::R; ++m) {
                float2 dx, dy, dz;
                const float2 i3 = cube2(sym_pair<S, GRAV>(rows, m, xy, zm, E2, dx, dy, dz));
                if (EQ) {
                    add_both(rows.TX[m], rows.TY[m], rows.TZ[m], cx, cy, cz, dx, dy, dz, i3);
                } else {
                    const float2 sj = mul2(make_float2(zm.z, zm.w), i3), si = mul2(rows.M[m], i3);
                    rows.TX[m] = fma2(dx, sj, rows.TX[m]);
                    rows.TY[m] = fma2(dy, sj, rows.TY[m]);
                    rows.TZ[m] = fma2(dz, sj, rows.TZ[m]);
                    cx = fma2(dx, si, cx); cy = fma2(dy, si, cy); cz = fma2(dz, si, cz);
                }
            }
            cx.x = __shfl_sync(0xffffffffu, cx.x, next); cx.y = __shfl_sync(0xffffffffu, cx.y, next);
            cy.x = __shfl_sync(0xffffffffu, cy.x, next); cy.y = __shfl_sync(0xffffffffu, cy.y, next);
            cz.x = __shfl_sync(0xffffffffu, cz.x, next); cz.y = __shfl_sync(0xffffffffu, cz.y, next);
        }
        const int j = 2 * j0 + lane;
        js[0][j] = cx.x; js[0][j + 32] = cx.y;
        js[1][j] = cy.x; js[1][j + 32] = cy.y;
        js[2][j] = cz.x; js[2][j + 32] = cz.y;
    }
}

// one-sided: the rows' sums over the tile's columns, masses included (a block against itself). FAR: see below
template <typename S, int GRAV, bool FAR>
__device__ __forceinline__ void sym_own(SymRows<S>& rows, const float4* XY, const float4* ZM, float2 E2) {
#pragma unroll 2
    for (int j = 0; j < S::JT / 2; ++j) {
        const float4 xy = XY[j], zm = ZM[j];
#pragma unroll
        for (int m = 0; m < S::R; ++m) {
            float2 dx, dy, dz;
            const float2 inv = sym_pair<S, GRAV>(rows, m, xy, zm, E2, dx, dy, dz), mj = make_float2(zm.z, zm.w);
            const float2 sj = FAR ? mul2(mul2(mj, inv), mul2(inv, inv)) : mul2(mj, cube2(inv));
            rows.TX[m] = fma2(dx, sj, rows.TX[m]);
            rows.TY[m] = fma2(dy, sj, rows.TY[m]);
            rows.TZ[m] = fma2(dz, sj, rows.TZ[m]);
        }
    }
}

// ---- separations that 1/r^3 does not suit -----------------------------------------------------------
// The sums above form 1/r^3 before a mass enters. One FP32 number holds it for separations from 1.5e-13 to 4.3e12 (from 3e38
// down to the smallest normal number), not between stars in metres or atoms in metres. Particles are far when a coordinate of
// theirs reaches 2^40 (below, no two of them are more than sqrt(3) 2^41 = 3.8e12 apart), or by their softening. Far sums are
// one-sided, (m / r) (1 / r^2) as in the one-sided kernels, and hold as long as r^2 and the force do: in the ensemble a
// task's, looked up once before its sweep, in a context all of them, in the fold (pairs.cu).
__device__ __forceinline__ bool sym_far(float4 q) {  // NaN counts as far
    return !(fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fabsf(q.z)) < 0x1p40f);
}
template <int GRAV>
__device__ __forceinline__ bool sym_far_eps(float eps2) {  // 1/eps^3 above 1e38, or a larger reach
    return GRAV == 1 && !(eps2 >= 5e-26f && eps2 <= 4e24f);
}
// the sums of nr <= B rows over nc columns: component c of row o in out[c * stride + o], compensated the rounding errors in
// the three components behind
template <typename S, int GRAV, bool COMP>
__device__ __forceinline__ void sym_far_pass(const float4* row, int nr, const float4* col, int nc, float eps2, float4* XY, float4* ZM,
                                          float* out, int64_t stride) {
    const float4 none = make_float4(1e18f, 1e18f, 1e18f, 0.0f);
    SymRows<S> rows;
    float s[3][S::R], e[3][S::R];
#pragma unroll
    for (int k = 0; k < S::R; ++k) {
        const int o = threadIdx.x + k * S::T;
        rows.set(k, o < nr ? row[o] : none);
        for (int c = 0; c < 3; ++c) s[c][k] = e[c][k] = 0.0f;
    }
    for (int j0 = 0; j0 < nc; j0 += S::JT) {
        __syncthreads();  // the previous tile's reads are done
#pragma unroll
        for (int h = 0; h < S::PF; ++h) {
            const int j = threadIdx.x + h * S::T;
            sym_stage(XY, ZM, j, j0 + j < nc ? col[j0 + j] : none);
        }
        __syncthreads();
        rows.clear();
        sym_own<S, GRAV, true>(rows, XY, ZM, make_float2(eps2, eps2));
#pragma unroll
        for (int k = 0; k < S::R; ++k) {
            const float t[3] = {rows.TX[k].x + rows.TX[k].y, rows.TY[k].x + rows.TY[k].y, rows.TZ[k].x + rows.TZ[k].y};
            for (int c = 0; c < 3; ++c) {
                if (COMP) fold(s[c][k], e[c][k], t[c]);
                else s[c][k] += t[c];
            }
        }
    }
#pragma unroll
    for (int k = 0; k < S::R; ++k) {
        const int o = threadIdx.x + k * S::T;
        if (o >= nr) break;
        for (int c = 0; c < 3; ++c) {
            out[c * stride + o] = s[c][k];
            if (COMP) out[(3 + c) * stride + o] = e[c][k];
        }
    }
}

}  // namespace gsph
