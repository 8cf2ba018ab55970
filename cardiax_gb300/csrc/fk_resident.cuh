// The resident stepper: many Euler steps of small and mid-sized tissues in one launch, the state
// held on chip for all of them.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "fk_pack.cuh"
#include "fk_step.cuh"

namespace fk {

constexpr int kResMaxOut = 32;       // states one launch can write out by list
constexpr int kResMaxSteps = 8192;   // steps of one launch: a launch ends within some 50 ms
constexpr int kResMinRows = 2, kResMaxRows = 5;  // rows per thread the kernel is built for

// How an H x W grid (n_exp copies of it) is cut into one tile per CTA.
struct ResPlan {
    int rows = 0;              // rows of 4 columns per thread
    int nr = 0, nc = 0;        // tile rows and columns per tissue
    int ng = 0, nq = 0;        // row groups (of `rows` rows) and quads of the grid
    int max_g = 0, max_q = 0;  // the largest tile's
    int threads = 0;
    int su_w = 0, su_h = 0;    // u tile in shared memory (floats per row, rows)
    size_t smem = 0;
    int64_t slot = 0;          // 64-bit words of one tile's outgoing strips (one parity)
    int64_t tiles = 0;         // of all tissues
    bool ok() const { return rows != 0; }
    size_t workspace() const { return (size_t)(tiles * 2 * slot) * 8; }
};

// The plan for n_exp tissues of an H x W grid on a device of n_sm SMs; not ok() when the tiles do
// not fit on chip (see fk_resident.cu for the sizes).
ResPlan resident_plan(int64_t H, int64_t W, int64_t n_exp, int n_sm);
// The same for the current device (n_sm looked up once per device; not ok() without one).
ResPlan resident_plan(int64_t H, int64_t W, int64_t n_exp);

struct ResidentArgs {
    int n;                     // steps of this launch
    int nr, nc, ng, nq;        // see ResPlan
    int max_q, max_g, su_w, su_h;
    int64_t slot;
    uint64_t *xchg;            // outgoing strips: [tile][parity][slot] words (value, tag)
    int64_t t0;                // step index of the launch's first step
    // states written out, after step out_step[k] of the launch to StepArgs::vo + out_off[k];
    // with `every`, after every step s (from 1) to vo + s * every instead
    int n_out;
    int64_t every;
    int out_step[kResMaxOut];
    int64_t out_off[kResMaxOut];
};

// Launches ra.n steps of n_exp tissues: `a` describes the one tissue, or with `exps` (device
// memory) the model, sizes, dt and dx that all share.  The workspace's words must be zero.
cudaError_t launch_resident(const ResPlan &p, const ResidentArgs &ra, const StepArgs &a,
                            const StepArgs *exps, cudaStream_t stream);

}  // namespace fk
