// fp64.cuh -- the double-precision build of the hot path (fp64.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/grasph2_b200.h"

namespace gsph {

struct DevParams64 {
    uint32_t flags;
    int dim;
    double H, H2, eps2, G, w_pref, dw_pref;
    double rho0, bulk, dbulk, c, shear, Y, tanfr, cohesion, alpha, beta;
    double mateps, matexp, inv_w_normalsep, xsph;
    double fixed_dt, initial_dt, min_dt, max_dt, accel_acc, vel_acc, cw_n;
    double const_acc[3], box_min[3], box_max[3], box_refl;
};

// Same roles as DevArrays, all in double4 / double; positions live in posm (x, y, z, m).
struct DevArrays64 {
    int64_t n, n_pad;
    double4 *posm, *velrho, *acc, *xvel, *sA, *sB, *dA, *dB, *jA, *jB;
    double *rhodot, *balsara;
    double* dt_state;  // [0] current, [1] next
    // symmetric gravity (null: all pairs in one sweep): [G + 1][3][n_pad] slots and their sums [3][n_pad]
    double *gpart, *gfold;
    int grav_I, grav_G, grav_gs;
    // culled SPH passes (null: all pairs): curve order, positions and packed records in that order, boxes, lists
    int* order;
    double4 *P, *J;
    float4 *box_lo, *box_hi;
    int *nb, *nbcnt;
};
// stream and events that let the gravity kernel run beside the SPH passes (null: in order on one stream)
struct Fork64 {
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};
// Above this many particles the slots (1.6 KB a particle) and lists (1 KB) are not allocated and every pass
// sweeps all pairs: a step then takes a minute and more, and the contexts keep their size.
constexpr int64_t kMaxSlots64 = int64_t(1) << 22;
void gravity64_shape(DevArrays64& a);
size_t gravity64_doubles(const DevArrays64& a);
size_t lists64_ints(int64_t n_pad);    // nb
size_t counts64_ints(int64_t n_pad);   // nbcnt
size_t boxes64(int64_t n_pad);
// FP32 copy of the positions (curve keys)
cudaError_t launch64_to32(const DevArrays64& a, float4* out, cudaStream_t s);

DevParams64 make_dev_params64(const gsph_params& p, double w_pref, double dw_pref, double inv_w_normalsep);
cudaError_t launch64_init(const DevArrays64& a, cudaStream_t s);
cudaError_t launch64_derivatives(const DevArrays64& a, const DevParams64& p, cudaStream_t s, int& launches,
                                 const Fork64& f = Fork64());
cudaError_t launch64_leapfrog(const DevArrays64& a, const DevParams64& p, int not_first_step, cudaStream_t s,
                              int& launches);
cudaError_t launch64_pack(const DevArrays64& a, int attr, const float* src, cudaStream_t s);
cudaError_t launch64_unpack(const DevArrays64& a, int attr, float* dst, cudaStream_t s);
cudaError_t launch64_unpack_d(const DevArrays64& a, int attr, double* dst, cudaStream_t s);
cudaError_t launch64_pack_pos(const DevArrays64& a, const double* src, cudaStream_t s);
cudaError_t launch64_pack_f64(const DevArrays64& a, int attr, const double* src, cudaStream_t s);
cudaError_t launch64_unpack_f64(const DevArrays64& a, int attr, double* dst, cudaStream_t s);
cudaError_t launch_narrow(const double* in, float* out, int64_t n, cudaStream_t s);
cudaError_t launch_widen(const float* in, double* out, int64_t n, cudaStream_t s);
size_t diag64_scratch_doubles(int64_t n_pad);
cudaError_t launch64_diagnostics(const DevArrays64& a, const DevParams64& p, double half_kick, double* scratch,
                                 double* out, cudaStream_t s);

}  // namespace gsph
