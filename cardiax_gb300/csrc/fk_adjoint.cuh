// Adjoint (reverse-mode) Euler step: declarations.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "fk_math.cuh"

namespace fk {

constexpr int kAdjParams = 13;       // differentiable parameters (cardiax/params.py fields 0..12)
constexpr int kAdjParamStride = 16;  // doubles per gradient slot
constexpr int ADJ_BAND = 6;          // cells this close to an edge use the explicit transposes

struct AdjointArgs {
    const float *u, *v, *w, *D;        // state x_t and diffusivity
    const float *lu, *lv, *lw;         // cotangent of x_{t+1}
    float *olu, *olv, *olw;            // cotangent of x_t (separate buffers)
    float *gD;                         // += dL/dD (null: not accumulated)
    double *gtheta;                    // += per-block partial dL/dtheta (null: not accumulated)
    int H, W, pitch;
    float t, dt, rdx;
    int n_stim;
    Model m;
    Stim stim[kMaxStim];
    double theta_factor[12];           // constant factors of the parameter sums (set_theta_factors)
};

// dt and the model's constants in dL/dtheta, fields 0..11 of cardiax/params.py (field 12, V_v, enters
// only through a Heaviside gate: zero); from a.m and a.dt.
void set_theta_factors(AdjointArgs &a);

// Number of dL/dtheta slots (kAdjParamStride doubles each) written by launch_adjoint.
int64_t adjoint_slots(int H, int W);
// One reverse step.  chained: the launch before it on the stream is the reverse step before it, or waits
// for that one in full, so that the state and D may be read before it has ended.
cudaError_t launch_adjoint(const AdjointArgs &a, bool chained, cudaStream_t stream);
// Reverse step k of a segment for n_exp experiments of one grid that share D and the parameters:
// `first` (and, in device memory, exps[0]) describes step 0 of the first one's segment, the others' states
// lie exp_stride floats apart and their cotangents, dL/dD and slots one after the other; exps[e] has the
// stimuli of experiment e.  parity selects the cotangent buffer read.
cudaError_t launch_adjoint_batch(const AdjointArgs &first, const AdjointArgs *exps, int n_exp, int64_t exp_stride,
                                 int k, int parity, float t, bool chained, cudaStream_t stream);

// dL/dD of n_exp experiments summed to the dense H x W plane oD, dL/dtheta over them and the slots to oth
// (kAdjParams floats).  One launch: as a loop of library calls (62 launches for 16 experiments) the sums took
// some 130 us at the end of a gradient pass.
cudaError_t launch_adjoint_sum(const float *gD, const double *gtheta, int n_exp, int H, int W, int pitch, float *oD,
                               float *oth, cudaStream_t stream);

}  // namespace fk
