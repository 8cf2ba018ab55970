// The resident stepper: many Euler steps of small and mid-sized tissues in one launch, the state
// held on chip for all of them.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <vector>

#include "fk_pack.cuh"
#include "fk_step.cuh"

namespace fk {

constexpr int kResMaxOut = 32;       // states one launch can write out by list
constexpr int kResMaxSteps = 8192;   // steps of one launch: a launch ends within some 50 ms
constexpr int kResMinRows = 2, kResMaxRows = 5;  // rows per thread the kernel is built for

constexpr int kResClusterRows = 2;   // rows per thread where the tiles are one cluster
constexpr int kResMaxCtas = 160;     // blocks of one launch (at most one per SM)
constexpr int kResMaxClasses = 16;   // sets of constants one launch of several tissues holds
constexpr size_t kResMaxSmem = 224 * 1024;

// How an H x W grid is cut into one tile per CTA.
struct ResPlan {
    int rows = 0;              // rows of 4 columns per thread
    int nr = 0, nc = 0;        // tile rows and columns
    int ng = 0, nq = 0;        // row groups (of `rows` rows) and quads of the grid
    int max_g = 0, max_q = 0;  // the largest tile's
    int threads = 0;
    int su_w = 0, su_h = 0;    // u tile in shared memory (floats per row, rows)
    size_t smem = 0;
    int64_t slot = 0;          // 64-bit words of one tile's outgoing strips (one parity)
    int64_t tiles = 0;
    double cost = 0.0;         // estimated us per step
    bool cluster = false;      // the tiles are one thread-block cluster
    bool ok() const { return rows != 0; }
    size_t workspace() const { return (size_t)(tiles * 2 * slot) * 8; }
};
inline size_t resident_smem(int rows, int threads, int su_floats) {
    return sizeof(float) * 2 * (size_t)su_floats + (size_t)3 * rows * threads * 16;
}

// best[t], t = 0 .. most: the fastest plan of `rows` rows per thread and at most t tiles (of equal ones
// that of the fewest tiles); not ok() where there is none.
void resident_plans(int64_t H, int64_t W, int most, int rows, std::vector<ResPlan> &best);
// The fastest plan on a device of n_sm SMs that takes clusters of up to max_cluster blocks, and on the current device (not ok() without one).
ResPlan resident_plan(int64_t H, int64_t W, int n_sm, int max_cluster);
ResPlan resident_plan(int64_t H, int64_t W);
// The calling thread's next n resident launches are refused (self-test).
void refuse_resident_launches(int n);
// The most blocks a launch may use on the current device (0: no cooperative launches, no device).
int resident_ctas();

// A tissue of a launch of several: its arguments (reads `state`), its plan, the first block of its
// tiles and its number in the batch.
struct ResTissue {
    StepArgs args;
    int nr, nc, ng, nq, su_w, first, id, pad;
};
struct ResClass {
    Model m;
    float dt, rdx;
};

struct ResidentArgs {
    int n;                     // steps of this launch
    int nr, nc, ng, nq;        // see ResPlan (one tissue)
    int max_q, max_g;          // (several tissues: the largest of the launch)
    int su_w, su;              // floats per row of the u tile (one tissue), of one u buffer
    int64_t slot;
    uint64_t *xchg;            // outgoing strips: [tile][parity][slot] words (value, tag)
    int64_t t0;                // step index of the launch's first step
    // states written out, after step out_step[k] of the launch to StepArgs::vo + out_off[k];
    // with `every`, after every step s (from 1) to vo + s * every instead.  Several tissues with
    // `base`: base + id * tissue_stride in place of vo.
    int n_out;
    int64_t every;
    int out_step[kResMaxOut];
    int64_t out_off[kResMaxOut];
    // several tissues (tissues != nullptr; device memory): per block the tissue << 8 | class
    const ResTissue *tissues;
    float *base;
    int64_t tissue_stride;
    uint32_t cta[kResMaxCtas];
    ResClass cls[kResMaxClasses];
};

// Launches ra.n steps with `rows` rows per thread; `a` describes the one tissue (several: only its
// dt and dx constants are read, by the launch-wide stencil coefficients).  The words of the strips
// must be zero.
// kResRefused: the device does not run that many blocks at once at present (a context with fewer SMs than the
// device); nothing was launched, and one launch per step still runs.
constexpr cudaError_t kResRefused = cudaErrorCooperativeLaunchTooLarge;
constexpr int kRefused = -1;  // the same as a return code of the functions that call it (never of an entry point)
cudaError_t launch_resident(int rows, int ctas, int threads, size_t smem, bool cluster, const ResidentArgs &ra,
                            const StepArgs &a, cudaStream_t stream);

}  // namespace fk
