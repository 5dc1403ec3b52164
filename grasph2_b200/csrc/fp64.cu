// fp64.cu -- the double-precision build of the hot path: GraSPH2's DOUBLE_PRECISION switch
// (settings/precisionSettings.h:16-17, src/types.h:32-43: f1_t = double, m3_t = Mat<double,3,3>).
//
// Same physics and pass sequence as the FP32 kernels, in FP64 throughout: symmetric all-pairs gravity in a kernel of
// its own, and the density and SPH sums over the particles within h (curve order, bounding boxes, neighbour lists).
// Very large contexts and no_cull sweep all pairs in one kernel per pass, each thread one i and every j: the
// reference's tile loop (src/particles/algorithms.h:270-309) without its remainder bug. B200 runs FP64 at half
// the FP32 rate, so this mode is the accuracy reference for trajectories the FP32 forms are measured
// against (energy drift), and the drop-in for callers of the reference's FP64 build.
#include "fp64.cuh"
#include "potential.cuh"
#include "rsqrt64.cuh"

namespace gsph {

namespace {

constexpr int kT64 = 128;  // threads per block = j-tile of the FP64 kernels

inline unsigned blocks_for(int64_t n, int t) { return static_cast<unsigned>((n + t - 1) / t); }

__host__ __device__ __forceinline__ bool has64(const DevParams64& p, uint32_t f) { return (p.flags & f) != 0; }

// ---- src/sph/kernel.h, eos.h, models.h in FP64 ----------------------------------------------------
__device__ __forceinline__ double w_poly64(double q) {  // kernel.h:130-136 without the prefactor
    if (q > 1.0) return 0.0;
    if (q < 0.5) return 6.0 * q * q * q - 6.0 * q * q + 1.0;
    const double a = 1.0 - q;
    return 2.0 * a * a * a;
}
__device__ __forceinline__ double dw_poly64(double q) {  // kernel.h:169-175
    if (q > 1.0) return 0.0;
    if (q < 0.5) return 3.0 * q * q - 2.0 * q;
    const double a = 1.0 - q;
    return -a * a;
}
__device__ __forceinline__ double pressure64(const DevParams64& p, double rho) {  // eos.h:88-96
    if (has64(p, GSPH_SOLIDS)) return p.bulk / p.dbulk * (pow(rho / p.rho0, p.dbulk) - 1.0);
    return p.c * p.c * (rho - p.rho0);
}
__device__ __forceinline__ double art64(double mateps, double s) { return s > 0.0 ? -mateps * s : 0.0; }

__device__ __forceinline__ void jrecord64(const DevParams64& p, double rho, double4 sA, double4 sB, double bal,
                                          double4& jA, double4& jB) {
    const double pres = pressure64(p, rho);
    const double r2 = rho * rho;
    if (has64(p, GSPH_SOLIDS)) {
        jA = make_double4((sA.x - pres) / r2, (sA.y - pres) / r2, (sA.z - pres) / r2, sA.w / r2);
        jB = make_double4(sB.x / r2, sB.y / r2, bal, 0.0);
    } else {
        const double s = -pres / r2;
        jA = make_double4(s, s, s, 0.0);
        jB = make_double4(0.0, 0.0, bal, 0.0);
    }
}

// ---- density ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kT64) k64_density(DevArrays64 a, DevParams64 p) {
    __shared__ double4 tile[kT64];
    const int64_t i = static_cast<int64_t>(blockIdx.x) * kT64 + threadIdx.x;
    const double4 pi = a.posm[i];
    double rho = 0.0;
    for (int64_t t0 = 0; t0 < a.n_pad; t0 += kT64) {
        __syncthreads();
        tile[threadIdx.x] = a.posm[t0 + threadIdx.x];
        __syncthreads();
        for (int j = 0; j < kT64; ++j) {
            const double4 q = tile[j];
            const double dx = q.x - pi.x, dy = q.y - pi.y, dz = q.z - pi.z;
            const double r2 = dx * dx + dy * dy + dz * dz;
            if (r2 <= p.H2 && r2 > 0.0) rho += q.w * w_poly64(sqrt(r2) / p.H);  // computeDerivatives.h:72
        }
    }
    if (i >= a.n) return;
    rho *= p.w_pref;
    if (has64(p, GSPH_DEAL_WITH_NO_PARTNERS) && rho < 0.001) rho = p.rho0 * 0.01;  // :85-88
    double4 vr = a.velrho[i];
    vr.w = rho;
    a.velrho[i] = vr;
    double4 jA, jB;
    jrecord64(p, rho, a.sA[i], a.sB[i], a.balsara[i], jA, jB);
    a.jA[i] = jA;
    a.jB[i] = jB;
}

__global__ void k64_prepare(DevArrays64 a, DevParams64 p) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    double4 jA, jB;
    jrecord64(p, a.velrho[i].w, a.sA[i], a.sB[i], a.balsara[i], jA, jB);
    a.jA[i] = jA;
    a.jB[i] = jB;
}

// ---- velocity gradient / acceleration passes ------------------------------------------------------
// PASS as in pairs.cuh: 0 velocity gradient (calcBalsaraDensityDTDStressDT), 1 acceleration
// (calcAcceleration), 2 both in one sweep.
struct I64 {  // particle i and the switches the pair body reads
    double4 pi, vi, jA, jB;
    double bi, ai[6];
    bool bals, av, xsph, arts, divv_on;
};
__device__ __forceinline__ I64 load_i64(const DevParams64& p, double4 pi, double4 vi, double4 jA, double4 jB) {
    I64 s;
    s.pi = pi; s.vi = vi; s.jA = jA; s.jB = jB;
    s.bals = has64(p, GSPH_BALSARA_SWITCH);
    s.av = has64(p, GSPH_ARTIFICIAL_VISCOSITY);
    s.xsph = has64(p, GSPH_XSPH);
    s.arts = has64(p, GSPH_ARTIFICIAL_STRESS);
    s.divv_on = s.bals || has64(p, GSPH_INTEGRATE_DENSITY);
    s.bi = s.bals ? jB.z : 1.0;
    s.ai[0] = art64(p.mateps, jA.x); s.ai[1] = art64(p.mateps, jA.y); s.ai[2] = art64(p.mateps, jA.z);
    s.ai[3] = art64(p.mateps, jA.w); s.ai[4] = art64(p.mateps, jB.x); s.ai[5] = art64(p.mateps, jB.y);
    return s;
}
// the sums of one particle: [0..2] a, [3..5] XSPH, [6..11] E, [12..14] W or the curl, [15] div v, [16] max v_sig
constexpr int kF64 = 17;
struct Acc64 {
    double f[kF64];
};
// which of them a pass sums (the others stay zero)
template <int PASS, bool SOLIDS>
__device__ __forceinline__ constexpr bool sums64(int f) {
    if (f < 6 || f == 16) return PASS != 0;
    if (f < 12) return PASS != 1 && SOLIDS;
    return PASS != 1;
}

// the SPH terms of one neighbour, 0 < r2 <= H2, (rx, ry, rz) = r_ij (computeDerivatives.h:118-141, :237-295)
template <int PASS, bool SOLIDS>
__device__ __forceinline__ void pair64(Acc64& T, const I64& I, double mj, double rx, double ry, double rz, double r2,
                                       double4 vj, double4 ja, double4 jb, const DevParams64& p) {
    constexpr bool DO_V = PASS != 1;
    constexpr bool DO_A = PASS != 0;
    double* f = T.f;
    const double r = sqrt(r2);
    const double qq = r / p.H;
    const double dwr = p.dw_pref * dw_poly64(qq) / r;
    const double g0 = dwr * rx, g1 = dwr * ry, g2 = dwr * rz;  // grad_i W
    const double vx = I.vi.x - vj.x, vy = I.vi.y - vj.y, vz = I.vi.z - vj.z;
    const double rhoj = vj.w;
    if (DO_V) {
        const double mr = mj / rhoj;
        if (SOLIDS) {  // models.h:225-248
            const double t = -0.5 * mr;
            f[6] += t * (vx * g0 + vx * g0); f[7] += t * (vy * g1 + vy * g1); f[8] += t * (vz * g2 + vz * g2);
            f[9] += t * (vx * g1 + vy * g0); f[10] += t * (vx * g2 + vz * g0); f[11] += t * (vy * g2 + vz * g1);
            f[12] += t * (vx * g1 - vy * g0); f[13] += t * (vx * g2 - vz * g0); f[14] += t * (vy * g2 - vz * g1);
        } else if (I.bals) {
            f[12] += mr * (vy * g2 - vz * g1); f[13] += mr * (vz * g0 - vx * g2); f[14] += mr * (vx * g1 - vy * g0);
        }
        if (I.divv_on) f[15] -= mr * (vx * g0 + vy * g1 + vz * g2);
    }
    if (DO_A) {
        double st[6] = {I.jA.x + ja.x, I.jA.y + ja.y, I.jA.z + ja.z, I.jA.w + ja.w, I.jB.x + jb.x, I.jB.y + jb.y};
        if (I.arts) {
            const double w = pow(p.w_pref * w_poly64(qq) * p.inv_w_normalsep, p.matexp);
            const double aj[6] = {art64(p.mateps, ja.x), art64(p.mateps, ja.y), art64(p.mateps, ja.z),
                                  art64(p.mateps, ja.w), art64(p.mateps, jb.x), art64(p.mateps, jb.y)};
#pragma unroll
            for (int k = 0; k < 6; ++k) st[k] += w * (I.ai[k] + aj[k]);
        }
        // (xx, yy, zz, xy, xz, yz) . grad W
        f[0] += mj * (st[0] * g0 + st[3] * g1 + st[4] * g2);
        f[1] += mj * (st[3] * g0 + st[1] * g1 + st[5] * g2);
        f[2] += mj * (st[4] * g0 + st[5] * g1 + st[2] * g2);
        if (I.av) {  // models.h:158-185
            const double w = (rx * vx + ry * vy + rz * vz) / r;
            if (w < 0.0) {
                const double vsig = p.c + p.c - p.beta * w;
                const double rhoij = (I.vi.w + rhoj) * 0.5;
                const double bj = I.bals ? jb.z : 1.0;
                const double II = -0.25 * (I.bi + bj) * p.alpha * w * vsig / rhoij;
                f[0] -= mj * II * g0; f[1] -= mj * II * g1; f[2] -= mj * II * g2;
                if (I.bals) f[16] = fmax(f[16], vsig);
            }
        }
        if (I.xsph) {
            const double w = 2.0 * mj / (I.vi.w + rhoj) * (p.w_pref * w_poly64(qq));
            f[3] -= w * vx; f[4] -= w * vy; f[5] -= w * vz;
        }
    }
}

// environmentAcceleration (:33-47)
__device__ __forceinline__ void environment64(const DevParams64& p, double4 x, double4 v, double& ax, double& ay,
                                              double& az) {
    if (has64(p, GSPH_CLOHESSY_WILTSHIRE)) {
        const double n = p.cw_n;
        const double s1 = 3 * n * n * x.x + 2 * n * v.y, s2 = -2 * n * v.x, s3 = -n * n * x.z;
        ax += s1 + s2 + s3; ay += s1 + s2 + s3; az += s1 + s2 + s3;
    }
    if (has64(p, GSPH_CONSTANT_ACCELERATION)) {
        ax += p.const_acc[0]; ay += p.const_acc[1]; az += p.const_acc[2];
    }
}

// do_after of the passes for particle i (its slot in `a`); jb_out (nullable): where the Balsara value also goes
template <int PASS, bool SOLIDS>
__device__ __forceinline__ void finish64(const DevArrays64& a, const DevParams64& p, int64_t i, const Acc64& T,
                                         const I64& I, double gx, double gy, double gz, double4* jb_out) {
    constexpr bool DO_V = PASS != 1;
    constexpr bool DO_A = PASS != 0;
    const double* f = T.f;
    if (DO_V) {  // calcBalsaraDensityDTDStressDT::do_after (:144-161)
        double c0 = f[12], c1 = f[13], c2 = f[14];
        if (SOLIDS) {
            const double Em[3][3] = {{f[6], f[9], f[10]}, {f[9], f[7], f[11]}, {f[10], f[11], f[8]}};
            const double R[3][3] = {{0.0, f[12], f[13]}, {-f[12], 0.0, f[14]}, {-f[13], -f[14], 0.0}};
            const double4 sa = a.sA[i], sb = a.sB[i];
            const double Sm[3][3] = {{sa.x, sa.w, sb.x}, {sa.w, sa.y, sb.y}, {sb.x, sb.y, sa.z}};
            const double tr = Em[0][0] + Em[1][1] + Em[2][2];
            double D[3][3];
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int e = 0; e < 3; ++e) {  // dstress_dt, models.h:250-268
                    double v = 2.0 * p.shear * Em[d][e];
                    if (d == e) v -= 2.0 * p.shear * tr / 3.0;
#pragma unroll
                    for (int k = 0; k < 3; ++k) v += Sm[d][k] * R[e][k] + Sm[e][k] * R[d][k];
                    D[d][e] = v;
                }
            a.dA[i] = make_double4(D[0][0], D[1][1], D[2][2], 0.5 * (D[0][1] + D[1][0]));
            a.dB[i] = make_double4(0.5 * (D[0][2] + D[2][0]), 0.5 * (D[1][2] + D[2][1]), 0.0, 0.0);
            c0 = -2.0 * R[1][2];
            c1 = -2.0 * R[2][0];
            c2 = -2.0 * R[0][1];
        }
        a.rhodot[i] = has64(p, GSPH_INTEGRATE_DENSITY) ? -I.vi.w * f[15] : 0.0;
        double bal = 0.0;
        if (I.bals) {  // models.h:187-192
            const double absdiv = fabs(f[15]);
            bal = absdiv / (absdiv + sqrt(c0 * c0 + c1 * c1 + c2 * c2) + 0.0001 * p.c / p.H);
            double4 jb = I.jB;
            jb.z = bal;
            a.jB[i] = jb;
            if (jb_out) *jb_out = jb;
        }
        a.balsara[i] = bal;
    }
    if (DO_A) {  // calcAcceleration::do_after (:301-312)
        double ax = f[0] + p.G * gx, ay = f[1] + p.G * gy, az = f[2] + p.G * gz;
        environment64(p, I.pi, I.vi, ax, ay, az);
        a.acc[i] = make_double4(ax, ay, az, f[16]);
        a.xvel[i] = make_double4(f[3], f[4], f[5], 0.0);
    }
}

// all pairs, gravity and SPH in one sweep, a thread per particle: the form of no_cull and of particle counts
// too large for the slots and neighbour lists of the kernels below
template <int PASS, bool SOLIDS>
__global__ void __launch_bounds__(kT64) k64_pairs(DevArrays64 a, DevParams64 p) {
    constexpr bool DO_A = PASS != 0;
    __shared__ double4 P[kT64], V[kT64], JA[kT64], JB[kT64];
    const int64_t i = static_cast<int64_t>(blockIdx.x) * kT64 + threadIdx.x;
    const I64 I = load_i64(p, a.posm[i], a.velrho[i], a.jA[i], a.jB[i]);
    const bool grav = DO_A && has64(p, GSPH_SELF_GRAVITY);
    const bool sph = has64(p, GSPH_SPH);
    double gx = 0, gy = 0, gz = 0;
    Acc64 T;
#pragma unroll
    for (int k = 0; k < kF64; ++k) T.f[k] = 0.0;
    for (int64_t t0 = 0; t0 < a.n_pad; t0 += kT64) {
        __syncthreads();
        P[threadIdx.x] = a.posm[t0 + threadIdx.x];
        V[threadIdx.x] = a.velrho[t0 + threadIdx.x];
        if (DO_A) {
            JA[threadIdx.x] = a.jA[t0 + threadIdx.x];
            JB[threadIdx.x] = a.jB[t0 + threadIdx.x];
        }
        __syncthreads();
        for (int j = 0; j < kT64; ++j) {
            const double4 q = P[j];
            const double rx = I.pi.x - q.x, ry = I.pi.y - q.y, rz = I.pi.z - q.z;  // r_ij
            const double r2 = rx * rx + ry * ry + rz * rz;
            if (!(r2 > 0.0)) continue;
            if (grav) {  // computeDerivatives.h:229-235
                const double inv = 1.0 / sqrt(r2 + p.eps2);
                const double s = q.w * inv * inv * inv;
                gx -= rx * s; gy -= ry * s; gz -= rz * s;
            }
            if (!sph || r2 > p.H2) continue;
            pair64<PASS, SOLIDS>(T, I, q.w, rx, ry, rz, r2, V[j], JA[j], JB[j], p);
        }
    }
    if (DO_A && has64(p, GSPH_VARIABLE_TIMESTEP) && i == 0) a.dt_state[1] = p.max_dt;  // :306-309
    if (i >= a.n) return;
    finish64<PASS, SOLIDS>(a, p, i, T, I, gx, gy, gz, nullptr);
}

// ================================================================================================
// symmetric all-pairs gravity and culled SPH passes
// ================================================================================================
// The sums of one step, instead of the two all-pairs sweeps above:
//   k64_stage        positions, velocities in curve order (P, J), bounding box of every 32 particles
//   k64_density      density over the boxes within h, recording each particle's neighbours
//   k64_sph          the SPH terms over those lists, then the epilogue
//   k64_gravity_sym  every unordered pair once, on its own stream beside them; k64_gravity_fold
// FP64 arithmetic throughout; every sum runs in a fixed order. Against the sweeps (one thread per particle, so 4,096
// particles filled 32 CTAs): a step of the 4,096-particle fluid 1.30 -> 0.07 ms, of the 30,011-particle impact
// 11.1 -> 1.4 ms.
constexpr int kC64 = 32;       // particles per bounding box, and per CTA of the culled kernels
constexpr int kW64 = 4;        // warps that share one CTA's 32 particles
constexpr int kNb64 = 64;      // neighbour-list slots per particle and warp

// Curve slot s holds particle o = order[s]. J packs a neighbour's 128 bytes (position/mass, velocity/density,
// sigma/rho^2, Balsara), so that a gather touches one line. The boxes are rounded outwards to FP32.
__global__ void __launch_bounds__(128) k64_stage(DevArrays64 a, DevParams64 p) {
    const int64_t s = static_cast<int64_t>(blockIdx.x) * 128 + threadIdx.x;
    const int64_t o = a.order[s];
    const double4 x = a.posm[o], v = a.velrho[o];
    a.P[s] = x;
    double4* J = a.J + 4 * s;
    J[0] = x;
    J[1] = v;
    if (has64(p, GSPH_INTEGRATE_DENSITY)) jrecord64(p, v.w, a.sA[o], a.sB[o], a.balsara[o], J[2], J[3]);
    const bool real = s < a.n;  // the curve order keeps the padding behind every particle
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    if (real) {
        lo[0] = __double2float_rd(x.x); lo[1] = __double2float_rd(x.y); lo[2] = __double2float_rd(x.z);
        hi[0] = __double2float_ru(x.x); hi[1] = __double2float_ru(x.y); hi[2] = __double2float_ru(x.z);
    }
#pragma unroll
    for (int w = 16; w > 0; w >>= 1)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], w));
            hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], w));
        }
    if ((threadIdx.x & 31) == 0) {
        a.box_lo[s / kC64] = make_float4(lo[0], lo[1], lo[2], 0.0f);
        a.box_hi[s / kC64] = make_float4(hi[0], hi[1], hi[2], 0.0f);
    }
}

// The neighbours of a CTA's 32 particles (lane l of every warp holds particle s = 32 blockIdx.x + l): warp w takes the
// boxes w, w + 4, w + 8, ... (near boxes come in runs along the curve, so the four warps get equal shares),
// skips those farther than h (1 + kMargin64) from the CTA's own box, stages the 32 positions of a near one in shared
// memory and calls hit(j, r_ij, |r_ij|^2, m_j) for every 0 < r2 <= H2, j ascending. The test is FP64 as in the
// all-pairs sweep; the box test only skips pairs that are farther apart than h in any rounding.
constexpr float kMargin64 = 1e-3f;
template <typename Hit>
__device__ __forceinline__ void near64(const DevArrays64& a, double H2, float hm2, double4 pi, double2 (*xy)[2], Hit&& hit) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nbox = static_cast<int>(a.n_pad / kC64);
    const float4 l = a.box_lo[blockIdx.x], u = a.box_hi[blockIdx.x];
    for (int b0 = 0; b0 < nbox; b0 += 32 * kW64) {
        const int b = b0 + kW64 * lane + warp;
        bool near = false;
        if (b < nbox) {
            const float4 bl = a.box_lo[b], bu = a.box_hi[b];
            const float gx = fmaxf(0.0f, fmaxf(bl.x - u.x, l.x - bu.x)), gy = fmaxf(0.0f, fmaxf(bl.y - u.y, l.y - bu.y)),
                        gz = fmaxf(0.0f, fmaxf(bl.z - u.z, l.z - bu.z));
            near = !(gx * gx + gy * gy + gz * gz > hm2);
        }
        unsigned todo = __ballot_sync(0xffffffffu, near);
        while (todo) {
            const int jb = kC64 * (b0 + kW64 * (__ffs(todo) - 1) + warp);
            todo &= todo - 1;
            const double4 q = a.P[jb + lane];
            __syncwarp();  // the previous box's reads are done
            xy[lane][0] = make_double2(q.x, q.y);
            xy[lane][1] = make_double2(q.z, q.w);
            __syncwarp();
            unsigned m = 0;
#pragma unroll 8
            for (int j = 0; j < kC64; ++j) {
                const double2 A = xy[j][0], B = xy[j][1];
                const double rx = pi.x - A.x, ry = pi.y - A.y, rz = pi.z - B.x;
                const double r2 = rx * rx + ry * ry + rz * rz;
                m |= static_cast<unsigned>(r2 <= H2 && r2 > 0.0) << j;
            }
            while (m) {
                const int j = __ffs(m) - 1;
                m &= m - 1;
                const double2 A = xy[j][0], B = xy[j][1];
                const double rx = pi.x - A.x, ry = pi.y - A.y, rz = pi.z - B.x;
                hit(jb + j, rx, ry, rz, rx * rx + ry * ry + rz * rz, B.y);
            }
        }
    }
}

__global__ void __launch_bounds__(kC64 * kW64) k64_density_near(DevArrays64 a, DevParams64 p, float hm2) {
    __shared__ double2 xy[kW64][kC64][2];
    __shared__ double red[kW64][kC64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t s = static_cast<int64_t>(blockIdx.x) * kC64 + lane;
    const double4 pi = a.P[s];
    double rho = 0.0;
    int cnt = 0;
    int* lst = a.nb + static_cast<int64_t>(warp) * kNb64 * a.n_pad + s;
    near64(a, p.H2, hm2, pi, xy[warp], [&](int j, double, double, double, double r2, double mj) {
        rho += mj * w_poly64(sqrt(r2) / p.H);  // computeDerivatives.h:72
        if (cnt < kNb64) lst[static_cast<int64_t>(cnt) * a.n_pad] = j;
        ++cnt;
    });
    a.nbcnt[static_cast<int64_t>(warp) * a.n_pad + s] = cnt;
    red[warp][lane] = rho;
    __syncthreads();
    if (warp != 0 || s >= a.n) return;
    rho = ((red[0][lane] + red[1][lane]) + (red[2][lane] + red[3][lane])) * p.w_pref;
    if (has64(p, GSPH_DEAL_WITH_NO_PARTNERS) && rho < 0.001) rho = p.rho0 * 0.01;  // :85-88
    const int64_t o = a.order[s];
    double4 vr = a.velrho[o];
    vr.w = rho;
    a.velrho[o] = vr;
    double4* J = a.J + 4 * s;
    J[1] = vr;
    jrecord64(p, rho, a.sA[o], a.sB[o], a.balsara[o], J[2], J[3]);
}

// LISTS: the neighbours come from the recorded lists (a particle with more than kNb64 in one warp's share sends that
// warp back to the boxes); otherwise from the boxes, recording the lists for a later pass.
template <int PASS, bool SOLIDS, bool LISTS>
__global__ void __launch_bounds__(kC64 * kW64) k64_sph(DevArrays64 a, DevParams64 p, float hm2) {
    __shared__ double2 xy[kW64][kC64][2];
    __shared__ double red[kW64 - 1][kF64][kC64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t s = static_cast<int64_t>(blockIdx.x) * kC64 + lane;
    const double4* Js = a.J + 4 * s;
    const I64 I = load_i64(p, Js[0], Js[1], Js[2], Js[3]);
    Acc64 T;
#pragma unroll
    for (int k = 0; k < kF64; ++k) T.f[k] = 0.0;
    int* lst = a.nb + static_cast<int64_t>(warp) * kNb64 * a.n_pad + s;
    int cnt = LISTS ? a.nbcnt[static_cast<int64_t>(warp) * a.n_pad + s] : 0;
    if (LISTS && !__any_sync(0xffffffffu, cnt > kNb64)) {
        for (int k = 0; k < cnt; ++k) {
            const double4* J = a.J + 4 * static_cast<int64_t>(lst[static_cast<int64_t>(k) * a.n_pad]);
            const double4 q = J[0];
            const double rx = I.pi.x - q.x, ry = I.pi.y - q.y, rz = I.pi.z - q.z;
            pair64<PASS, SOLIDS>(T, I, q.w, rx, ry, rz, rx * rx + ry * ry + rz * rz, J[1], J[2], J[3], p);
        }
    } else {
        cnt = 0;
        near64(a, p.H2, hm2, I.pi, xy[warp], [&](int j, double rx, double ry, double rz, double r2, double mj) {
            const double4* J = a.J + 4 * static_cast<int64_t>(j);
            pair64<PASS, SOLIDS>(T, I, mj, rx, ry, rz, r2, J[1], J[2], J[3], p);
            if (!LISTS && cnt < kNb64) lst[static_cast<int64_t>(cnt) * a.n_pad] = j;
            ++cnt;
        });
        if (!LISTS) a.nbcnt[static_cast<int64_t>(warp) * a.n_pad + s] = cnt;
    }
    if (warp > 0) {
#pragma unroll
        for (int k = 0; k < kF64; ++k)
            if (sums64<PASS, SOLIDS>(k)) red[warp - 1][k][lane] = T.f[k];
    }
    __syncthreads();
    if (PASS != 0 && has64(p, GSPH_VARIABLE_TIMESTEP) && blockIdx.x == 0 && threadIdx.x == 0)
        a.dt_state[1] = p.max_dt;  // :306-309
    if (warp > 0 || s >= a.n) return;
#pragma unroll
    for (int k = 0; k < kF64; ++k)
        if (sums64<PASS, SOLIDS>(k)) {
            if (k == 16) T.f[k] = fmax(fmax(T.f[k], red[0][k][lane]), fmax(red[1][k][lane], red[2][k][lane]));
            else T.f[k] = (T.f[k] + red[0][k][lane]) + (red[1][k][lane] + red[2][k][lane]);
        }
    const int64_t o = a.order[s];
    double g[3] = {0.0, 0.0, 0.0};
    if (PASS != 0 && has64(p, GSPH_SELF_GRAVITY))
        for (int c = 0; c < 3; ++c) g[c] = a.gfold[c * a.n_pad + o];
    finish64<PASS, SOLIDS>(a, p, o, T, I, g[0], g[1], g[2], PASS == 0 ? a.J + 4 * s + 3 : nullptr);
}

// Symmetric all-pairs gravity (Newton's third law), the scheme of the FP32 kernel (pairs.cu) in FP64. Blocks of
// 128 I particles form G groups of `gs` blocks; CTA t is the task (ga, gb), ga <= gb: every row block of ga against
// the column blocks of gb (the later ones when ga == gb) in tiles of 128 columns. One 1/r^3 serves both particles:
// row sums stay in registers, column sums pass round the warp by rotation and are added over the four warps in shared
// memory. Each particle has G + 1 slots [slot][component][n_pad], each written by one task.
//
// Bound: the FP64 pipe (64 lanes per SM and clock). 20 FP64 instructions per unordered pair (3 separation, 3 r^2 + eps^2,
// 6 x^(-3/2), 2 masses, 6 sums) plus 3 / I for the column sums; the all-pairs sweep needed about 75 per ordered one.
// `live` is false in a pair with a NaN separation and in the self pair, which the reference skips (r^2 > 0).
__device__ __forceinline__ double inv_cube_any64(double& dx, double& dy, double& dz, double eps2) {
    const double r2 = dx * dx + dy * dy + dz * dz;
    if (!(r2 > 0.0)) {
        dx = dy = dz = 0.0;
        return 0.0;
    }
    const double inv = 1.0 / sqrt(r2 + eps2);
    return inv * inv * inv;
}

template <int I>
__global__ void __launch_bounds__(kT64, I == 4 ? 3 : 4) k64_gravity_sym(const double4* __restrict__ pos, double* __restrict__ part,
                                                           int64_t n_pad, int G, int gs, double eps2) {
    constexpr int B = kT64 * I;
    __shared__ double2 Jxy[kT64], Jzm[kT64];
    __shared__ double js[kT64 / 32][3][kT64];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int ga, gb;
    {  // the G (G - 1) / 2 pairs of distinct groups first, then the diagonal ones
        const int t = static_cast<int>(blockIdx.x), noff = G * (G - 1) / 2;
        int r = 0, rem = t;
        if (t >= noff) {
            r = t - noff;
            rem = -1;
        } else {
            while (rem >= G - 1 - r) {
                rem -= G - 1 - r;
                ++r;
            }
        }
        ga = r;
        gb = r + 1 + rem;
    }
    const int nb = static_cast<int>(n_pad / B);
    const int ra0 = ga * gs, ra1 = min(nb, ra0 + gs), cg0 = gb * gs, cg1 = min(nb, cg0 + gs);
    const bool diag = ga == gb;
    const int s_row = gb - ga, s_col = G - gb + ga;
    auto slot = [&](int64_t particle, int sl, int c) { return part + (static_cast<int64_t>(sl) * 3 + c) * n_pad + particle; };
    if (diag)  // the group's first block is never a column here: its column slot is zero
        for (int e = tid; e < B; e += kT64)
            for (int c = 0; c < 3; ++c) *slot(static_cast<int64_t>(ra0) * B + e, s_col, c) = 0.0;
    for (int ab = ra0; ab < ra1; ++ab) {
        const int64_t base = static_cast<int64_t>(ab) * B + tid;
        double X[I], Y[I], Z[I], M[I], AX[I], AY[I], AZ[I];
#pragma unroll
        for (int k = 0; k < I; ++k) {
            const double4 q = pos[base + static_cast<int64_t>(k) * kT64];
            X[k] = q.x; Y[k] = q.y; Z[k] = q.z; M[k] = -q.w;
            AX[k] = AY[k] = AZ[k] = 0.0;
        }
        const int64_t d0 = static_cast<int64_t>(ab) * B;
        const int nd = diag ? I : 0;  // the block's own tiles, one-sided
        const int64_t c0 = static_cast<int64_t>(diag ? ab + 1 : cg0) * B, c1 = static_cast<int64_t>(cg1) * B;
        const int total = nd + (c1 > c0 ? static_cast<int>((c1 - c0) / kT64) : 0);
        auto src = [&](int k) { return (k < nd ? d0 + static_cast<int64_t>(k) * kT64 : c0 + static_cast<int64_t>(k - nd) * kT64) + tid; };
        double4 pf = make_double4(0, 0, 0, 0);
        if (total > 0) pf = pos[src(0)];
        for (int k = 0; k < total; ++k) {
            __syncthreads();  // the previous tile's reads of J and js are done
            Jxy[tid] = make_double2(pf.x, pf.y);
            Jzm[tid] = make_double2(pf.z, pf.w);
            __syncthreads();
            if (k + 1 < total) pf = pos[src(k + 1)];
            const bool own = k < nd;
            const int next = (lane + 1) & 31;
#pragma unroll 1
            for (int j0 = 0; j0 < kT64; j0 += 32) {
                double cx = 0.0, cy = 0.0, cz = 0.0;
#pragma unroll 1
                for (int r = 0; r < 32; ++r) {
                    const int j = j0 + ((lane + r) & 31);
                    const double2 A = Jxy[j], Bq = Jzm[j];
                    double dx[I], dy[I], dz[I], x[I], i3[I];
                    bool ok = true;
#pragma unroll
                    for (int m = 0; m < I; ++m) {
                        dx[m] = A.x - X[m]; dy[m] = A.y - Y[m]; dz[m] = Bq.x - Z[m];
                        x[m] = fma(dz[m], dz[m], fma(dy[m], dy[m], fma(dx[m], dx[m], eps2)));
                        ok = ok && series_range64(x[m]);
                    }
                    if (ok) {
#pragma unroll
                        for (int m = 0; m < I; ++m) i3[m] = inv_cube64(x[m]);
                    } else {
#pragma unroll
                        for (int m = 0; m < I; ++m) i3[m] = inv_cube_any64(dx[m], dy[m], dz[m], eps2);
                    }
#pragma unroll
                    for (int m = 0; m < I; ++m) {
                        const double sj = Bq.y * i3[m];
                        AX[m] = fma(dx[m], sj, AX[m]); AY[m] = fma(dy[m], sj, AY[m]); AZ[m] = fma(dz[m], sj, AZ[m]);
                    }
                    if (!own) {
#pragma unroll
                        for (int m = 0; m < I; ++m) {
                            const double si = M[m] * i3[m];
                            cx = fma(dx[m], si, cx); cy = fma(dy[m], si, cy); cz = fma(dz[m], si, cz);
                        }
                        // lane l hands column (l + r) % 32 to lane l - 1: after 32 rounds it holds column l
                        cx = __shfl_sync(0xffffffffu, cx, next);
                        cy = __shfl_sync(0xffffffffu, cy, next);
                        cz = __shfl_sync(0xffffffffu, cz, next);
                    }
                }
                js[warp][0][j0 + lane] = cx;
                js[warp][1][j0 + lane] = cy;
                js[warp][2][j0 + lane] = cz;
            }
            if (!own) {  // the tile's column sums over the CTA's row block, into the column slot
                __syncthreads();
                const int64_t j = c0 + static_cast<int64_t>(k - nd) * kT64 + tid;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const double v = (js[0][c][tid] + js[1][c][tid]) + (js[2][c][tid] + js[3][c][tid]);
                    double* dst = slot(j, s_col, c);
                    *dst = ab == ra0 ? v : *dst + v;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < I; ++k) {
            const int64_t pr = base + static_cast<int64_t>(k) * kT64;
            *slot(pr, s_row, 0) = AX[k];
            *slot(pr, s_row, 1) = AY[k];
            *slot(pr, s_row, 2) = AZ[k];
        }
    }
}

// a particle's G + 1 slots: four threads sum a run of them each, the runs are added in order. FINISH: the
// gravity-only epilogue; else the sums go to gfold for k64_sph.
template <bool FINISH>
__global__ void __launch_bounds__(256) k64_gravity_fold(DevArrays64 a, DevParams64 p, int S) {
    const int lane = threadIdx.x & 31, q = lane >> 3;
    const int64_t i = (static_cast<int64_t>(blockIdx.x) * 256 + (threadIdx.x & ~31)) / 4 + (lane & 7);
    if (FINISH && has64(p, GSPH_VARIABLE_TIMESTEP) && blockIdx.x == 0 && threadIdx.x == 0) a.dt_state[1] = p.max_dt;
    const int R = (S + 3) / 4, k0 = min(S, q * R), k1 = min(S, k0 + R);
    double t[3] = {0.0, 0.0, 0.0};
    if (i < a.n)
#pragma unroll 4
        for (int k = k0; k < k1; ++k)
#pragma unroll
            for (int c = 0; c < 3; ++c) t[c] += a.gpart[(static_cast<int64_t>(k) * 3 + c) * a.n_pad + i];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double b = __shfl_down_sync(0xffffffffu, t[c], 8), d = __shfl_down_sync(0xffffffffu, t[c], 16),
                     e = __shfl_down_sync(0xffffffffu, t[c], 24);
        t[c] = ((t[c] + b) + d) + e;
    }
    if (lane >= 8 || i >= a.n) return;
    if (!FINISH) {
        for (int c = 0; c < 3; ++c) a.gfold[c * a.n_pad + i] = t[c];
        return;
    }
    double ax = p.G * t[0], ay = p.G * t[1], az = p.G * t[2];
    environment64(p, a.posm[i], a.velrho[i], ax, ay, az);
    a.acc[i] = make_double4(ax, ay, az, 0.0);
    a.xvel[i] = make_double4(0.0, 0.0, 0.0, 0.0);
}

// FP32 copy of the positions, for the curve keys
__global__ void k64_to32(DevArrays64 a, float4* out) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n_pad) return;
    const double4 q = a.posm[i];
    out[i] = make_float4(static_cast<float>(q.x), static_cast<float>(q.y), static_cast<float>(q.z), 0.0f);
}

// ---- leapfrog (src/integration.h) ---------------------------------------------------------------------
__device__ __forceinline__ void plasticity64(double4& a, double4& b, double Y) {  // models.h:194-205
    const double J2 = 0.5 * (a.x * a.x + a.y * a.y + a.z * a.z + 2.0 * (a.w * a.w + b.x * b.x + b.y * b.y));
    const double f = Y * Y / (3.0 * J2);
    if (f < 1.0) {
        a.x *= f; a.y *= f; a.z *= f; a.w *= f;
        b.x *= f; b.y *= f;
    }
}

__device__ __forceinline__ void kick_drift64(const DevArrays64& a, const DevParams64& p, int64_t i, double kick_dt,
                                             double dt) {
    double4 vr = a.velrho[i];
    const double4 ac = a.acc[i];
    vr.x += ac.x * kick_dt; vr.y += ac.y * kick_dt; vr.z += ac.z * kick_dt;
    double4 x = a.posm[i];
    const bool sph = has64(p, GSPH_SPH);
    double ux = vr.x, uy = vr.y, uz = vr.z;
    if (sph && has64(p, GSPH_XSPH)) {
        const double4 xv = a.xvel[i];
        ux += p.xsph * xv.x; uy += p.xsph * xv.y; uz += p.xsph * xv.z;
    }
    x.x += ux * dt; x.y += uy * dt; x.z += uz * dt;
    if (sph) {
        if (has64(p, GSPH_INTEGRATE_DENSITY)) {
            double rho = vr.w + a.rhodot[i] * dt;
            if (rho < 0.0) rho = 0.0;
            vr.w = rho;
        }
        if (has64(p, GSPH_SOLIDS)) {
            double4 sa = a.sA[i], sb = a.sB[i];
            const double4 da = a.dA[i], db = a.dB[i];
            sa.x += da.x * dt; sa.y += da.y * dt; sa.z += da.z * dt; sa.w += da.w * dt;
            sb.x += db.x * dt; sb.y += db.y * dt;
            if (has64(p, GSPH_PLASTICITY_MC))
                plasticity64(sa, sb, p.tanfr * (p.bulk / p.dbulk * (pow(vr.w / p.rho0, p.dbulk) - 1.0)) + p.cohesion);
            else if (has64(p, GSPH_PLASTICITY_MIESE))
                plasticity64(sa, sb, p.Y);
            a.sA[i] = sa;
            a.sB[i] = sb;
        }
    }
    if (has64(p, GSPH_SIMPLE_BOX_BOUNDARY)) {
        const double m = 1.0 + p.box_refl;
        double* xc[3] = {&x.x, &x.y, &x.z};
        double* vc[3] = {&vr.x, &vr.y, &vr.z};
        for (int d = 0; d < 3; ++d) {
            if (d == 2 && p.dim != 3) break;
            if (*xc[d] > p.box_max[d]) { *xc[d] = p.box_max[d]; *vc[d] -= m * *vc[d]; }
            else if (*xc[d] < p.box_min[d]) { *xc[d] = p.box_min[d]; *vc[d] -= m * *vc[d]; }
        }
    }
    a.posm[i] = x;
    a.velrho[i] = vr;
}

__global__ void k64_leapfrog_fixed(DevArrays64 a, DevParams64 p, double kick_dt) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < a.n) kick_drift64(a, p, i, kick_dt, p.fixed_dt);
}

// variable step (integration.h:130-217); dt_state holds positive doubles, min-reduced as int64
__global__ void k64_dt_criteria(DevArrays64 a, DevParams64 p) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const double dt = a.dt_state[0];
    double mindt = p.max_dt;
    if (i < a.n) {
        double4 vr = a.velrho[i];
        const double4 ac = a.acc[i];
        vr.x += ac.x * dt * 0.5; vr.y += ac.y * dt * 0.5; vr.z += ac.z * dt * 0.5;
        a.velrho[i] = vr;
        if (has64(p, GSPH_ACCELERATION_CRITERION))
            mindt = fmin(mindt, sqrt(p.accel_acc * p.H / sqrt(ac.x * ac.x + ac.y * ac.y + ac.z * ac.z)));
        if (has64(p, GSPH_VELOCITY_CRITERION)) mindt = fmin(mindt, p.vel_acc * p.H / ac.w);
    }
    for (int o = 16; o > 0; o >>= 1) mindt = fmin(mindt, __shfl_xor_sync(0xffffffffu, mindt, o));
    if ((threadIdx.x & 31) == 0)
        atomicMin(reinterpret_cast<unsigned long long*>(a.dt_state + 1),
                  static_cast<unsigned long long>(__double_as_longlong(mindt)));
}
__global__ void k64_dt_first(DevArrays64 a, DevParams64 p) {
    if (threadIdx.x == 0 && blockIdx.x == 0) a.dt_state[1] = p.initial_dt;
}
__global__ void k64_leapfrog_variable(DevArrays64 a, DevParams64 p) {
    const double nxt = a.dt_state[1];
    const double dt = nxt < p.min_dt ? p.min_dt : nxt;
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < a.n) kick_drift64(a, p, i, dt * 0.5, dt);
}
__global__ void k64_dt_commit(DevArrays64 a, DevParams64 p) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        const double nxt = a.dt_state[1];
        a.dt_state[0] = nxt < p.min_dt ? p.min_dt : nxt;
    }
}

// ---- transfers: caller's float attributes (and FP64 positions) <-> device doubles --------------------
__global__ void k64_pack(DevArrays64 a, int attr, const float* __restrict__ src) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    switch (attr) {
        case 0: { double4 q = a.posm[i]; q.x = src[3 * i]; q.y = src[3 * i + 1]; q.z = src[3 * i + 2]; a.posm[i] = q; break; }
        case 1: { double4 q = a.posm[i]; q.w = src[i]; a.posm[i] = q; break; }
        case 2: { double4 q = a.velrho[i]; q.x = src[3 * i]; q.y = src[3 * i + 1]; q.z = src[3 * i + 2]; a.velrho[i] = q; break; }
        case 3: { double4 q = a.acc[i]; q.x = src[3 * i]; q.y = src[3 * i + 1]; q.z = src[3 * i + 2]; a.acc[i] = q; break; }
        case 4: a.balsara[i] = src[i]; break;
        case 5: a.xvel[i] = make_double4(src[3 * i], src[3 * i + 1], src[3 * i + 2], 0.0); break;
        case 6: { double4 q = a.velrho[i]; q.w = src[i]; a.velrho[i] = q; break; }
        case 7: a.rhodot[i] = src[i]; break;
        case 8:
        case 9: {
            const float* m = src + 9 * i;
            const double4 A = make_double4(m[0], m[4], m[8], 0.5 * (double(m[1]) + m[3]));
            const double4 B = make_double4(0.5 * (double(m[2]) + m[6]), 0.5 * (double(m[5]) + m[7]), 0.0, 0.0);
            if (attr == 8) { a.sA[i] = A; a.sB[i] = B; }
            else { a.dA[i] = A; a.dB[i] = B; }
            break;
        }
        case 10: { double4 q = a.acc[i]; q.w = src[i]; a.acc[i] = q; break; }
        default: break;
    }
}

__global__ void k64_unpack(DevArrays64 a, int attr, float* __restrict__ dst) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    auto f = [](double v) { return static_cast<float>(v); };
    switch (attr) {
        case 0: { const double4 q = a.posm[i]; dst[3 * i] = f(q.x); dst[3 * i + 1] = f(q.y); dst[3 * i + 2] = f(q.z); break; }
        case 1: dst[i] = f(a.posm[i].w); break;
        case 2: { const double4 q = a.velrho[i]; dst[3 * i] = f(q.x); dst[3 * i + 1] = f(q.y); dst[3 * i + 2] = f(q.z); break; }
        case 3: { const double4 q = a.acc[i]; dst[3 * i] = f(q.x); dst[3 * i + 1] = f(q.y); dst[3 * i + 2] = f(q.z); break; }
        case 4: dst[i] = f(a.balsara[i]); break;
        case 5: { const double4 q = a.xvel[i]; dst[3 * i] = f(q.x); dst[3 * i + 1] = f(q.y); dst[3 * i + 2] = f(q.z); break; }
        case 6: dst[i] = f(a.velrho[i].w); break;
        case 7: dst[i] = f(a.rhodot[i]); break;
        case 8:
        case 9: {
            const double4 A = (attr == 8) ? a.sA[i] : a.dA[i];
            const double4 B = (attr == 8) ? a.sB[i] : a.dB[i];
            float* m = dst + 9 * i;
            m[0] = f(A.x); m[1] = f(A.w); m[2] = f(B.x);
            m[3] = f(A.w); m[4] = f(A.y); m[5] = f(B.y);
            m[6] = f(B.x); m[7] = f(B.y); m[8] = f(A.z);
            break;
        }
        case 10: dst[i] = f(a.acc[i].w); break;
        default: break;
    }
}

// `acc64`: caller-side double output of one attribute (3 or 1 components) -- the FP64 download
__global__ void k64_unpack_d(DevArrays64 a, int attr, double* __restrict__ dst) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    double4 q;
    switch (attr) {
        case 0: q = a.posm[i]; break;
        case 2: q = a.velrho[i]; break;
        case 3: q = a.acc[i]; break;
        default: q = make_double4(a.velrho[i].w, 0, 0, 0);  // density
    }
    if (attr == 6) {
        dst[i] = q.x;
    } else {
        dst[3 * i] = q.x; dst[3 * i + 1] = q.y; dst[3 * i + 2] = q.z;
    }
}

// double host layout <-> device doubles, every attribute (the DOUBLE_PRECISION host buffers)
__global__ void k64_pack_f64(DevArrays64 a, int attr, const double* __restrict__ src) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    switch (attr) {
        case 0: { double4 q = a.posm[i]; q.x = src[3 * i]; q.y = src[3 * i + 1]; q.z = src[3 * i + 2]; a.posm[i] = q; break; }
        case 1: { double4 q = a.posm[i]; q.w = src[i]; a.posm[i] = q; break; }
        case 2: { double4 q = a.velrho[i]; q.x = src[3 * i]; q.y = src[3 * i + 1]; q.z = src[3 * i + 2]; a.velrho[i] = q; break; }
        case 3: { double4 q = a.acc[i]; q.x = src[3 * i]; q.y = src[3 * i + 1]; q.z = src[3 * i + 2]; a.acc[i] = q; break; }
        case 4: a.balsara[i] = src[i]; break;
        case 5: a.xvel[i] = make_double4(src[3 * i], src[3 * i + 1], src[3 * i + 2], 0.0); break;
        case 6: { double4 q = a.velrho[i]; q.w = src[i]; a.velrho[i] = q; break; }
        case 7: a.rhodot[i] = src[i]; break;
        case 8:
        case 9: {
            const double* m = src + 9 * i;
            const double4 A = make_double4(m[0], m[4], m[8], 0.5 * (m[1] + m[3]));
            const double4 B = make_double4(0.5 * (m[2] + m[6]), 0.5 * (m[5] + m[7]), 0.0, 0.0);
            if (attr == 8) { a.sA[i] = A; a.sB[i] = B; }
            else { a.dA[i] = A; a.dB[i] = B; }
            break;
        }
        case 10: { double4 q = a.acc[i]; q.w = src[i]; a.acc[i] = q; break; }
        default: break;
    }
}

__global__ void k64_unpack_f64(DevArrays64 a, int attr, double* __restrict__ dst) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    switch (attr) {
        case 0: { const double4 q = a.posm[i]; dst[3 * i] = q.x; dst[3 * i + 1] = q.y; dst[3 * i + 2] = q.z; break; }
        case 1: dst[i] = a.posm[i].w; break;
        case 2: { const double4 q = a.velrho[i]; dst[3 * i] = q.x; dst[3 * i + 1] = q.y; dst[3 * i + 2] = q.z; break; }
        case 3: { const double4 q = a.acc[i]; dst[3 * i] = q.x; dst[3 * i + 1] = q.y; dst[3 * i + 2] = q.z; break; }
        case 4: dst[i] = a.balsara[i]; break;
        case 5: { const double4 q = a.xvel[i]; dst[3 * i] = q.x; dst[3 * i + 1] = q.y; dst[3 * i + 2] = q.z; break; }
        case 6: dst[i] = a.velrho[i].w; break;
        case 7: dst[i] = a.rhodot[i]; break;
        case 8:
        case 9: {
            const double4 A = (attr == 8) ? a.sA[i] : a.dA[i];
            const double4 B = (attr == 8) ? a.sB[i] : a.dB[i];
            double* m = dst + 9 * i;
            m[0] = A.x; m[1] = A.w; m[2] = B.x;
            m[3] = A.w; m[4] = A.y; m[5] = B.y;
            m[6] = B.x; m[7] = B.y; m[8] = A.z;
            break;
        }
        case 10: dst[i] = a.acc[i].w; break;
        default: break;
    }
}

__global__ void k_narrow(const double* __restrict__ in, float* __restrict__ out, int64_t n) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) out[i] = static_cast<float>(in[i]);
}
__global__ void k_widen(const float* __restrict__ in, double* __restrict__ out, int64_t n) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) out[i] = in[i];
}

__global__ void k64_pack_pos(DevArrays64 a, const double* __restrict__ src) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    double4 q = a.posm[i];
    q.x = src[3 * i]; q.y = src[3 * i + 1]; q.z = src[3 * i + 2];
    a.posm[i] = q;
}

__global__ void k64_init(DevArrays64 a) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= a.n_pad) return;
    const double4 z = make_double4(0, 0, 0, 0);
    a.posm[i] = (i < a.n) ? z : make_double4(1e18, 1e18, 1e18, 0.0);
    a.velrho[i] = (i < a.n) ? z : make_double4(0, 0, 0, 1.0);
    a.acc[i] = z; a.xvel[i] = z; a.sA[i] = z; a.sB[i] = z; a.dA[i] = z; a.dB[i] = z; a.jA[i] = z; a.jB[i] = z;
    a.rhodot[i] = 0.0;
    a.balsara[i] = 0.0;
}

// ---- FP64 diagnostics (same quantities as the FP32 path) ---------------------------------------------
constexpr int kDiag64 = 12;
__global__ void __launch_bounds__(kT64) k64_diag(DevArrays64 a, DevParams64 p, double half_kick, double* blocks) {
    __shared__ double red[kT64 / 32][kDiag64];
    const int64_t i = static_cast<int64_t>(blockIdx.x) * kT64 + threadIdx.x;
    double f[kDiag64] = {};
    const double4 x = a.posm[i];
    if (i < a.n) {
        const double4 vr = a.velrho[i], ac = a.acc[i];
        const double m = x.w;
        const double vx = vr.x + half_kick * ac.x, vy = vr.y + half_kick * ac.y, vz = vr.z + half_kick * ac.z;
        f[0] = 0.5 * m * (vx * vx + vy * vy + vz * vz);
        f[4] = m * vx; f[5] = m * vy; f[6] = m * vz;
        f[7] = m * (x.y * vz - x.z * vy); f[8] = m * (x.z * vx - x.x * vz); f[9] = m * (x.x * vy - x.y * vx);
        f[10] = m;
        if (has64(p, GSPH_SPH)) {
            const double rho = vr.w, r0 = p.rho0;
            if (has64(p, GSPH_SOLIDS)) {
                const double K = p.bulk, nn = p.dbulk;
                f[2] = m * ((fabs(nn - 1.0) < 1e-12)
                                ? K / r0 * (log(rho / r0) + r0 / rho - 1.0)
                                : K / nn * ((pow(rho, nn - 1.0) - pow(r0, nn - 1.0)) / ((nn - 1.0) * pow(r0, nn)) +
                                            (1.0 / rho - 1.0 / r0)));
                const double4 sa = a.sA[i], sb = a.sB[i];
                const double ss = sa.x * sa.x + sa.y * sa.y + sa.z * sa.z + 2.0 * (sa.w * sa.w + sb.x * sb.x + sb.y * sb.y);
                f[3] = m * ss / (4.0 * p.shear * rho);
            } else {
                f[2] = m * p.c * p.c * (log(rho / r0) + r0 / rho - 1.0);
            }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = 0; k < kDiag64; ++k) {
        double v = f[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < kDiag64) {
        double s = 0.0;
        for (int w = 0; w < kT64 / 32; ++w) s += red[w][threadIdx.x];
        blocks[static_cast<int64_t>(blockIdx.x) * kDiag64 + threadIdx.x] = s;
    }
}
}  // namespace

DevParams64 make_dev_params64(const gsph_params& p, double w_pref, double dw_pref, double inv_w_normalsep) {
    DevParams64 d{};
    d.flags = p.flags;
    d.dim = p.dimension;
    d.H = p.H;
    d.H2 = p.H * p.H;
    d.eps2 = p.grav_eps * p.grav_eps;
    d.G = p.grav_G;
    d.w_pref = w_pref;
    d.dw_pref = dw_pref;
    d.rho0 = p.rho0;
    d.bulk = p.bulk;
    d.dbulk = p.dbulk_dp;
    d.c = p.soundspeed;
    d.shear = p.shear;
    d.Y = p.Y;
    d.tanfr = p.tanfr;
    d.cohesion = p.cohesion;
    d.alpha = p.av_alpha;
    d.beta = p.av_beta;
    d.mateps = p.mateps;
    d.matexp = p.matexp;
    d.inv_w_normalsep = inv_w_normalsep;
    d.xsph = p.xsph_factor;
    d.fixed_dt = p.fixed_dt;
    d.initial_dt = p.initial_dt;
    d.min_dt = p.min_dt;
    d.max_dt = p.max_dt;
    d.accel_acc = p.accel_accuracy;
    d.vel_acc = p.velocity_accuracy;
    d.cw_n = p.cw_n;
    for (int k = 0; k < 3; ++k) {
        d.const_acc[k] = p.const_acc[k];
        d.box_min[k] = p.box_min[k];
        d.box_max[k] = p.box_max[k];
    }
    d.box_refl = p.box_reflectiveness;
    return d;
}

cudaError_t launch64_init(const DevArrays64& a, cudaStream_t s) {
    k64_init<<<blocks_for(a.n_pad, 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}

// Row blocks of 128 I particles: the largest I that still gives the tasks of 48 blocks or more (1,176 for two waves
// of four CTAs per SM), at most 64 groups. N = 4,096: I = 1, 528 tasks; N = 30,011: I = 4, 60 groups.
void gravity64_shape(DevArrays64& a) {
    a.grav_I = a.n_pad / (kT64 * 4) >= 48 ? 4 : (a.n_pad / (kT64 * 2) >= 48 ? 2 : 1);
    const int64_t nb = a.n_pad / (kT64 * a.grav_I);
    a.grav_gs = static_cast<int>((nb + 63) / 64);
    a.grav_G = static_cast<int>((nb + a.grav_gs - 1) / a.grav_gs);
}
size_t gravity64_doubles(const DevArrays64& a) { return static_cast<size_t>(a.grav_G + 1) * 3 * a.n_pad; }
size_t lists64_ints(int64_t n_pad) { return static_cast<size_t>(kW64) * kNb64 * n_pad; }
size_t counts64_ints(int64_t n_pad) { return static_cast<size_t>(kW64) * n_pad; }
size_t boxes64(int64_t n_pad) { return static_cast<size_t>(n_pad / kC64); }
cudaError_t launch64_to32(const DevArrays64& a, float4* out, cudaStream_t s) {
    k64_to32<<<blocks_for(a.n_pad, 256), 256, 0, s>>>(a, out);
    return cudaGetLastError();
}

namespace {
cudaError_t gravity64(const DevArrays64& a, const DevParams64& p, bool finish, cudaStream_t s, int& launches) {
    const unsigned tasks = static_cast<unsigned>(a.grav_G * (a.grav_G + 1) / 2);
    switch (a.grav_I) {
        case 1: k64_gravity_sym<1><<<tasks, kT64, 0, s>>>(a.posm, a.gpart, a.n_pad, a.grav_G, a.grav_gs, p.eps2); break;
        case 2: k64_gravity_sym<2><<<tasks, kT64, 0, s>>>(a.posm, a.gpart, a.n_pad, a.grav_G, a.grav_gs, p.eps2); break;
        default: k64_gravity_sym<4><<<tasks, kT64, 0, s>>>(a.posm, a.gpart, a.n_pad, a.grav_G, a.grav_gs, p.eps2);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const unsigned nb = blocks_for(a.n * 4, 256);
    if (finish) k64_gravity_fold<true><<<nb, 256, 0, s>>>(a, p, a.grav_G + 1);
    else k64_gravity_fold<false><<<nb, 256, 0, s>>>(a, p, a.grav_G + 1);
    launches += 2;
    return cudaGetLastError();
}
template <int PASS>
cudaError_t sph64(const DevArrays64& a, const DevParams64& p, bool lists, cudaStream_t s) {
    const unsigned nb = static_cast<unsigned>(a.n_pad / kC64);
    const float hm = static_cast<float>(p.H) * (1.0f + kMargin64), hm2 = hm * hm;
    const int T = kC64 * kW64;
    if (has64(p, GSPH_SOLIDS)) {
        if (lists) k64_sph<PASS, true, true><<<nb, T, 0, s>>>(a, p, hm2);
        else k64_sph<PASS, true, false><<<nb, T, 0, s>>>(a, p, hm2);
    } else {
        if (lists) k64_sph<PASS, false, true><<<nb, T, 0, s>>>(a, p, hm2);
        else k64_sph<PASS, false, false><<<nb, T, 0, s>>>(a, p, hm2);
    }
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch64_derivatives(const DevArrays64& a, const DevParams64& p, cudaStream_t s, int& launches,
                                 const Fork64& f) {
    const unsigned nb = static_cast<unsigned>(a.n_pad / kT64);
    const bool sph = has64(p, GSPH_SPH), grav = has64(p, GSPH_SELF_GRAVITY);
    const bool solids = has64(p, GSPH_SOLIDS), summed = !has64(p, GSPH_INTEGRATE_DENSITY);
    const bool vgrad = sph && (solids || !summed || has64(p, GSPH_BALSARA_SWITCH));
    const bool two = vgrad && has64(p, GSPH_BALSARA_SWITCH);
    cudaError_t e = cudaSuccess;
    if (!sph && grav && a.gpart) return gravity64(a, p, true, s, launches);
    if (sph && a.order) {
        const bool forked = grav && f.side;
        if (forked) {
            e = cudaEventRecord(f.fork, s);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(f.side, f.fork, 0);
        }
        if (e == cudaSuccess && grav) e = gravity64(a, p, false, forked ? f.side : s, launches);
        if (e == cudaSuccess && forked) e = cudaEventRecord(f.join, f.side);
        if (e != cudaSuccess) return e;
        k64_stage<<<nb, kT64, 0, s>>>(a, p);
        if (summed) {
            const float hm = static_cast<float>(p.H) * (1.0f + kMargin64);
            k64_density_near<<<static_cast<unsigned>(a.n_pad / kC64), kC64 * kW64, 0, s>>>(a, p, hm * hm);
            ++launches;
        }
        ++launches;
        e = cudaGetLastError();
        if (e == cudaSuccess && two) {
            e = sph64<0>(a, p, summed, s);
            ++launches;
        }
        if (e == cudaSuccess && forked) e = cudaStreamWaitEvent(s, f.join, 0);
        if (e != cudaSuccess) return e;
        ++launches;
        if (two) return sph64<1>(a, p, true, s);
        return vgrad ? sph64<2>(a, p, summed, s) : sph64<1>(a, p, summed, s);
    }
    if (sph) {
        if (summed) k64_density<<<nb, kT64, 0, s>>>(a, p);
        else k64_prepare<<<blocks_for(a.n, 256), 256, 0, s>>>(a, p);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        ++launches;
    }
    if (two) {
        if (solids) k64_pairs<0, true><<<nb, kT64, 0, s>>>(a, p);
        else k64_pairs<0, false><<<nb, kT64, 0, s>>>(a, p);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        ++launches;
    }
    if (vgrad && !two) {
        if (solids) k64_pairs<2, true><<<nb, kT64, 0, s>>>(a, p);
        else k64_pairs<2, false><<<nb, kT64, 0, s>>>(a, p);
    } else {
        if (solids) k64_pairs<1, true><<<nb, kT64, 0, s>>>(a, p);
        else k64_pairs<1, false><<<nb, kT64, 0, s>>>(a, p);
    }
    ++launches;
    return cudaGetLastError();
}

cudaError_t launch64_leapfrog(const DevArrays64& a, const DevParams64& p, int not_first_step, cudaStream_t s,
                              int& launches) {
    const unsigned nb = blocks_for(a.n, 256);
    if (!has64(p, GSPH_VARIABLE_TIMESTEP)) {
        k64_leapfrog_fixed<<<nb, 256, 0, s>>>(a, p, p.fixed_dt * (not_first_step ? 1.0 : 0.5));
        ++launches;
        return cudaGetLastError();
    }
    if (not_first_step) k64_dt_criteria<<<nb, 256, 0, s>>>(a, p);
    else k64_dt_first<<<1, 32, 0, s>>>(a, p);
    k64_leapfrog_variable<<<nb, 256, 0, s>>>(a, p);
    k64_dt_commit<<<1, 32, 0, s>>>(a, p);
    launches += 3;
    return cudaGetLastError();
}

cudaError_t launch64_pack(const DevArrays64& a, int attr, const float* src, cudaStream_t s) {
    k64_pack<<<blocks_for(a.n, 256), 256, 0, s>>>(a, attr, src);
    return cudaGetLastError();
}
cudaError_t launch64_unpack(const DevArrays64& a, int attr, float* dst, cudaStream_t s) {
    k64_unpack<<<blocks_for(a.n, 256), 256, 0, s>>>(a, attr, dst);
    return cudaGetLastError();
}
cudaError_t launch64_unpack_d(const DevArrays64& a, int attr, double* dst, cudaStream_t s) {
    k64_unpack_d<<<blocks_for(a.n, 256), 256, 0, s>>>(a, attr, dst);
    return cudaGetLastError();
}
cudaError_t launch64_pack_f64(const DevArrays64& a, int attr, const double* src, cudaStream_t s) {
    k64_pack_f64<<<blocks_for(a.n, 256), 256, 0, s>>>(a, attr, src);
    return cudaGetLastError();
}
cudaError_t launch64_unpack_f64(const DevArrays64& a, int attr, double* dst, cudaStream_t s) {
    k64_unpack_f64<<<blocks_for(a.n, 256), 256, 0, s>>>(a, attr, dst);
    return cudaGetLastError();
}
cudaError_t launch_narrow(const double* in, float* out, int64_t n, cudaStream_t s) {
    k_narrow<<<blocks_for(n, 256), 256, 0, s>>>(in, out, n);
    return cudaGetLastError();
}
cudaError_t launch_widen(const float* in, double* out, int64_t n, cudaStream_t s) {
    k_widen<<<blocks_for(n, 256), 256, 0, s>>>(in, out, n);
    return cudaGetLastError();
}
cudaError_t launch64_pack_pos(const DevArrays64& a, const double* src, cudaStream_t s) {
    k64_pack_pos<<<blocks_for(a.n, 256), 256, 0, s>>>(a, src);
    return cudaGetLastError();
}
size_t diag64_scratch_doubles(int64_t n_pad) {
    return static_cast<size_t>(n_pad / kT64) * kDiag64 + kDiag64 + potential_partials();
}
cudaError_t launch64_diagnostics(const DevArrays64& a, const DevParams64& p, double half_kick, double* scratch,
                                 double* out, cudaStream_t s) {
    const int nb = static_cast<int>(a.n_pad / kT64);
    k64_diag<<<nb, kT64, 0, s>>>(a, p, half_kick, scratch);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    double* pot = scratch + static_cast<int64_t>(nb) * kDiag64;
    int npot = 0;
    if (has64(p, GSPH_SELF_GRAVITY)) {
        e = launch_pair_potential(PotSource64{a.posm}, a.n, p.eps2, pot, npot, s);
        if (e != cudaSuccess) return e;
    }
    k_sum_partials<kDiag64><<<1, 32 * kDiag64, 0, s>>>(scratch, nb, pot, npot, -p.G, out);
    return cudaGetLastError();
}

}  // namespace gsph
