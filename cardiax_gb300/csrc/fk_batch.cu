// C ABI of the batched path: many tissues advanced by one persistent kernel per step, with
// runs of steps captured into a CUDA graph.  No reference counterpart (the reference loops over
// tissues in Python, deepx/generate.py:135-210); per tissue the arithmetic is exactly that of
// fk_forward_euler (cardiax/solve.py:92-100), bit for bit.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <new>
#include <numeric>
#include <vector>

#include "../../include/cardiax_gb300.h"
#include "fk_capi_internal.h"
#include "fk_resident.cuh"
#include "fk_step.cuh"
#include "fk_tb.cuh"

using namespace fk;

// The tile geometries the batched kernel is built for (fk_batch_rows32.cu, fk_batch_rows16.cu):
// rows x 64 columns, u loaded with a 4-cell halo (rows + 8 rows), D with a 2-row halo.
typedef cudaError_t (*BatchLaunchFn)(const void *, const void *, const void *, const int *, int,
                                     int, int, const int *, int, int, bool, int *, int,
                                     cudaStream_t);
cudaError_t fk_batch_launch_rows32(const void *, const void *, const void *, const int *, int, int,
                                   int, const int *, int, int, bool, int *, int, cudaStream_t);
cudaError_t fk_batch_launch_rows16(const void *, const void *, const void *, const int *, int, int,
                                   int, const int *, int, int, bool, int *, int, cudaStream_t);
namespace {
struct TileShape {
    int rows, cols, ctas_per_sm;
    BatchLaunchFn launch;
};
constexpr int kShapes = 2;
const TileShape kShape[kShapes] = {{32, 64, 2, fk_batch_launch_rows32},
                                   {16, 64, 2, fk_batch_launch_rows16}};
}  // namespace

// One launch of the resident kernel: some of the batch's tissues, for all steps of a call.
struct ResWave {
    int rows = 0, threads = 0, ctas = 0;
    size_t smem = 0;
    double cost = 0.0;           // estimated us per step
    int first = 0;               // its tissues' place in the device table
    std::vector<int> tissue;
    std::vector<ResPlan> plan;   // of each
    ResidentArgs args{};
};
struct ResWaves {
    std::vector<ResWave> w;
    double cost = 0.0;           // us per step of all tissues
    size_t xchg_bytes = 0;
    bool ok() const { return !w.empty(); }
};

struct fk_batch {
    // the resident kernel in place of one launch per step (fk_batch_set_resident; turned off by the
    // knobs of the stepping kernel)
    ResWaves res;
    int resident = 0;  // 2: whatever the estimate says
    ResTissue *d_res = nullptr;
    uint64_t *d_xchg = nullptr;
    std::vector<ResTissue> h_res;
    int64_t cells = 0;
    int n = 0, grid = 0, device = -1;
    int shape = 0;  // index into kShape of the tile geometry in use
    // work order (0: contiguous runs; k = 1, 2, 4, 8: round-robin in chunks of k items) and
    // arithmetic of the batched kernel
    int interleave = 1, packed = 0;
    int depth = 1;                   // Euler steps per launch: 1, or 2 (blocked kernel)
    bool tb_ok = false;              // every tissue can be blocked (and no activation tracking)
    BatchTbMaps *d_tbmaps = nullptr;
    int grid_tb = 0;                 // CTAs of the blocked kernel (one per SM)
    std::vector<BatchTbMaps> h_tbmaps;
    BatchTissue *d_tissues = nullptr;
    int *d_t = nullptr;
    int *status = nullptr;
    bool act = false;
    // per tile geometry: TMA maps (box heights differ), the work list and the CTAs' runs of it
    struct PerShape {
        BatchMaps *d_maps = nullptr;
        BatchItem *d_items = nullptr;
        int *d_ranges = nullptr;  // kBatchMaxGrid + 1 item offsets: CTA c runs [r[c], r[c+1])
        int n_items = 0;
        std::vector<BatchMaps> h_maps;
        std::vector<BatchItem> h_items;
        std::vector<uint8_t> h_edge;  // per item: an edge tile
        std::vector<int> h_ranges;
    } sp[kShapes];
    // host staging (kept alive until destroy: the uploads are asynchronous)
    std::vector<BatchTissue> h_tissues;
    std::vector<int> order;        // tissues, larger first
    std::vector<fk_grid> grids;    // per tissue
    // captured graph
    cudaStream_t capture_stream = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int graph_steps = 0, graph_grid = 0, graph_shape = 0, graph_opts = 0, graph_depth = 1;
};

namespace {

constexpr size_t kAlign = 128;
size_t align_up(size_t x) { return (x + kAlign - 1) / kAlign * kAlign; }

int64_t tiles_of(const fk_grid &g, int shape) {
    const TileShape &t = kShape[shape];
    return ((g.H + t.rows - 1) / t.rows) * ((g.W + t.cols - 1) / t.cols);
}

struct Layout {
    size_t maps[kShapes], tbmaps, tissues, items[kShapes], ranges[kShapes], t, res, xchg, total;
};

Layout layout(int n, const int64_t *n_items, const ResWaves &res) {
    Layout L;
    size_t at = 0;
    for (int k = 0; k < kShapes; ++k) {
        L.maps[k] = at;
        at = align_up(at + sizeof(BatchMaps) * n);
    }
    L.tbmaps = at;
    at = align_up(at + sizeof(BatchTbMaps) * n);
    L.tissues = at;
    at = align_up(at + sizeof(BatchTissue) * n);
    for (int k = 0; k < kShapes; ++k) {
        L.items[k] = at;
        at = align_up(at + sizeof(BatchItem) * n_items[k]);
        L.ranges[k] = at;
        at = align_up(at + sizeof(int) * (kBatchMaxGrid + 1));
    }
    L.t = at;
    at = align_up(at + 16);
    L.res = at;
    if (res.ok()) at = align_up(at + sizeof(ResTissue) * n);
    L.xchg = at;
    L.total = align_up(at + (res.ok() ? res.xchg_bytes : 0));
    return L;
}

// ---- the resident kernel's launches ------------------------------------------------------------------
// The tissues of a batch are independent, so any set of them that fits on chip together can run all
// steps of a call in one launch before the next set starts: 48 mixed tissues (5.9 M cells), 64 steps:
// 45.6 us per step in the batched kernel (143 GCUPS: 40 % of its items are edge tiles, each loaded and
// stored every step), 35.7 in such launches (33.6 over 256 steps; a launch also loads and stores all).
constexpr int kResMaxTissues = 4096, kResMaxWaves = 64;

ResClass res_class(const fk_tissue &t) {
    ResClass c;
    std::memset(&c, 0, sizeof c);
    c.m = make_model(t.params);
    c.dt = (float)t.dt;
    c.rdx = 1.0f / (float)t.dx;
    return c;
}

// By shape and rows per thread: the best plan of at most 0, 1, .. ctas tiles (the cost falls with the tiles).
struct ResPlans {
    struct Shape {
        std::vector<ResPlan> best;
        int least = 0;  // the fewest tiles that hold the tissue (ctas where all blocks do not)
    };
    int ctas;
    std::map<std::pair<int64_t, int64_t>, Shape> made[kResMaxRows + 1];
    const Shape &of(const fk_grid &g, int R) {
        Shape &p = made[R][{g.H, g.W}];
        if (p.best.empty()) {
            resident_plans(g.H, g.W, ctas, R, p.best);
            while (p.least < ctas && !p.best[p.least].ok()) ++p.least;
        }
        return p;
    }
    const ResPlan &least(const fk_grid &g, int R) {
        const Shape &p = of(g, R);
        return p.best[p.least];
    }
};

// The launch of wave x's tissues with R rows per thread (x.rows stays 0 where they do not fit).
void plan_wave(const fk_tissue *ts, ResPlans &plans, int R, const std::vector<int> &cls, ResWave &x) {
    const int n = (int)x.tissue.size();
    x.plan.resize(n);
    int left = plans.ctas;
    for (int i = 0; i < n; ++i) {
        x.plan[i] = plans.least(ts[x.tissue[i]].g, R);
        if (!x.plan[i].ok()) return;
        left -= (int)x.plan[i].tiles;
    }
    if (left < 0) return;
    // blocks left over go to the tissue that takes longest, while that helps
    while (left > 0) {
        int worst = 0;
        for (int i = 1; i < n; ++i)
            if (x.plan[i].cost > x.plan[worst].cost) worst = i;
        const std::vector<ResPlan> &p = plans.of(ts[x.tissue[worst]].g, R).best;
        const int tiles = (int)x.plan[worst].tiles;
        int t = tiles;
        while (t < tiles + left && !(p[t].cost < x.plan[worst].cost)) ++t;
        if (!(p[t].cost < x.plan[worst].cost)) break;
        left -= t - tiles;
        x.plan[worst] = p[t];
    }
    for (int i = 0; i < n; ++i) {
        const ResPlan &p = x.plan[i];
        for (int t = 0; t < p.tiles; ++t) x.args.cta[x.ctas + t] = (uint32_t)i << 8 | (uint32_t)cls[i];
        x.ctas += (int)p.tiles;
        x.threads = std::max(x.threads, p.threads);
        x.args.max_q = std::max(x.args.max_q, p.max_q);
        x.args.max_g = std::max(x.args.max_g, p.max_g);
        x.args.su = std::max(x.args.su, p.su_w * p.su_h);
        x.cost = std::max(x.cost, p.cost);
    }
    // (threads and u buffers may come from different tissues: their sum need not fit)
    x.smem = resident_smem(R, x.threads, x.args.su);
    if (x.smem > kResMaxSmem) return;
    x.args.slot = 2 * 16 * (int64_t)x.args.max_q + 2 * 4 * (int64_t)x.args.max_g * R;
    x.rows = R;
}

// Sets made with `R` rows per thread, largest tissues first, each into the first set with room; with `each` a
// set then takes the rows that are fastest for it (the last sets hold few tissues: 48 mixed ones, six sets of 4 rows,
// the last of two 512^2 tissues then of 2 rows: 37.2 -> 35.7 us per step).
ResWaves plan_waves_rows(const fk_tissue *ts, int n, ResPlans &plans, int R, bool each) {
    ResWaves out;
    std::vector<ResPlan> plan(n);
    for (int k = 0; k < n; ++k) {
        plan[k] = plans.least(ts[k].g, R);
        if (!plan[k].ok()) return out;
    }
    std::vector<int> order(n);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return plan[x].tiles > plan[y].tiles; });
    struct Set {
        int ctas = 0, n_cls = 0;
        std::vector<int> tissue, cls;
        ResClass c[kResMaxClasses];
    };
    std::vector<Set> sets;
    for (int k : order) {
        const ResClass c = res_class(ts[k]);
        for (size_t q = 0;; ++q) {
            if (q == sets.size()) {
                if ((int)q == kResMaxWaves) return out;
                sets.emplace_back();
            }
            Set &x = sets[q];
            if (x.ctas + plan[k].tiles > plans.ctas) continue;
            int id = 0;
            while (id < x.n_cls && std::memcmp(&x.c[id], &c, sizeof c) != 0) ++id;
            if (id == kResMaxClasses) continue;
            if (id == x.n_cls) x.c[x.n_cls++] = c;
            x.ctas += (int)plan[k].tiles;
            x.tissue.push_back(k);
            x.cls.push_back(id);
            break;
        }
    }
    int at = 0;
    for (const Set &x : sets) {
        ResWave best;
        for (int r = each ? kResMinRows : R; r <= (each ? kResMaxRows : R); ++r) {
            ResWave w;
            w.tissue = x.tissue;
            plan_wave(ts, plans, r, x.cls, w);
            if (w.rows && (!best.rows || w.cost < best.cost)) best = std::move(w);
        }
        if (!best.rows) return ResWaves();
        std::copy(x.c, x.c + x.n_cls, best.args.cls);
        best.first = at;
        at += (int)x.tissue.size();
        out.xchg_bytes = std::max(out.xchg_bytes, (size_t)(best.ctas * 2 * best.args.slot) * 8);
        out.cost += best.cost;
        out.w.push_back(std::move(best));
    }
    return out;
}

ResWaves plan_waves(const fk_tissue *ts, int n) {
    ResWaves best;
    ResPlans plans{resident_ctas(), {}};
    if (plans.ctas < 2 || n > kResMaxTissues) return best;
    int64_t cells = 0;
    for (int k = 0; k < n; ++k) {
        if (check_grid(ts[k].g) || ts[k].act.last || ts[k].n_stimuli > kMaxStim) return best;
        cells += ts[k].g.H * ts[k].g.W;
    }
    if (cells > (int64_t)kResMaxWaves * plans.ctas * 512 * 4 * kResMaxRows) return best;
    int rows = 0;
    for (int R = kResMinRows; R <= kResMaxRows; ++R) {
        ResWaves w = plan_waves_rows(ts, n, plans, R, false);
        if (w.ok() && (!best.ok() || w.cost < best.cost)) {
            best = std::move(w);
            rows = R;
        }
    }
    if (best.w.size() > 1) best = plan_waves_rows(ts, n, plans, rows, true);
    // the most blocks first: where the device refuses a launch, nothing has run yet (see run_resident)
    std::stable_sort(best.w.begin(), best.w.end(), [](const ResWave &x, const ResWave &y) { return x.ctas > y.ctas; });
    return best;
}

// us of n steps: the resident launches (a launch's fixed cost is 15 to 30 us), and one launch per
// step (4.4 us at least, about 140 GCUPS on mixed tissues).
double res_time(const ResWaves &r, int64_t n) { return (double)r.w.size() * 30.0 + r.cost * (double)n; }
double step_time(int64_t cells, int64_t n) { return std::max(4.4, (double)cells / 140e3) * (double)n; }
// Whether n steps take the resident launches; stepping them takes `more` us more than step_time, they
// `also` more than res_time.
bool takes_resident(const fk_batch *b, int64_t n, double more = 0.0, double also = 0.0) {
    return b->resident == 2 ||
           (b->resident && res_time(b->res, n) + also < step_time(b->cells, n) + more);
}

// Relative cost of an edge tile (clamped halo, one-sided rows, bounds checks) against an
// interior one, for balancing the CTAs' runs of the work list.
constexpr double kEdgeCost = 1.1;

bool interior_tile(const fk_grid &g, int shape, int64_t i0, int64_t j0) {
    const TileShape &t = kShape[shape];
    return i0 >= BAND && i0 + t.rows <= g.H - BAND && j0 >= BAND && j0 + t.cols <= g.W - BAND;
}

// Cuts the work list into `grid` contiguous runs of about equal cost: r[c] .. r[c+1] for CTA c.
void make_ranges(const std::vector<BatchItem> &items, const std::vector<uint8_t> &edge, int grid,
                 std::vector<int> &r) {
    const int n = (int)items.size();
    double total = 0.0;
    for (int k = 0; k < n; ++k) total += edge[k] ? kEdgeCost : 1.0;
    r.assign(grid + 1, n);
    r[0] = 0;
    double acc = 0.0;
    int c = 1;
    for (int k = 0; k < n && c < grid; ++k) {
        acc += edge[k] ? kEdgeCost : 1.0;
        while (c < grid && acc >= total * c / grid) r[c++] = k + 1;
    }
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// The work list of tile geometry `q` for the plan's work order, and the CTAs' runs of it.
// Interleaved order: every tissue's edge tiles (the costlier clamped-halo path) first, then the
// interior tiles, each group with the larger tissues first (CTAs take every G-th item).
// Contiguous runs: tissue by tissue (larger first), each tissue's tiles column by column, so
// that a CTA's run changes tissue rarely and its next item is usually the tile below the
// current one, whose top halo rows it has just loaded (they are still in L2).
// Round-robin in chunks of c: the kernel's CTA g of G takes items g, g + G, g + 2G, ...; the
// list is permuted so that those are c consecutive items of the natural order in turn
// (natural item x of chunk p = x / c goes to position (p / G) c G + (x % c) G + p % G), so a
// CTA steps through c neighbouring tiles, mostly of one tissue, before the next chunk.  A last
// partial block of chunks keeps the natural order.
void chunk_items(fk_batch::PerShape &P, int c, int G) {
    const int64_t n = (int64_t)P.h_items.size();
    if (c <= 1 || G < 1 || n == 0) return;
    const int64_t full = n / ((int64_t)c * G) * c * G;  // items in whole blocks
    std::vector<BatchItem> it(P.h_items);
    std::vector<uint8_t> ed(P.h_edge);
    for (int64_t x = 0; x < full; ++x) {
        const int64_t p = x / c, blk = p / G;
        const int64_t to = blk * c * G + (x % c) * G + p % G;
        P.h_items[to] = it[x];
        P.h_edge[to] = ed[x];
    }
}

void build_items(fk_batch *b, int q) {
    fk_batch::PerShape &P = b->sp[q];
    const TileShape &ts = kShape[q];
    P.h_items.clear();
    P.h_edge.clear();
    // want_edge: 1 edge only, 0 interior only, -1 both; by_column: column-major tile order
    auto add = [&](int k, int want_edge, bool by_column) {
        const fk_grid &g = b->grids[k];
        const int64_t nr = (g.H + ts.rows - 1) / ts.rows, nc = (g.W + ts.cols - 1) / ts.cols;
        for (int64_t a = 0; a < (by_column ? nc : nr); ++a)
            for (int64_t c = 0; c < (by_column ? nr : nc); ++c) {
                const int64_t i0 = (by_column ? c : a) * ts.rows, j0 = (by_column ? a : c) * ts.cols;
                const int edge = interior_tile(g, q, i0, j0) ? 0 : 1;
                if (want_edge >= 0 && edge != want_edge) continue;
                P.h_items.push_back(BatchItem{k, (int32_t)i0, (int32_t)j0, 0});
                P.h_edge.push_back((uint8_t)edge);
            }
    };
    if (b->interleave) {
        for (int k : b->order) add(k, 1, false);
        for (int k : b->order) add(k, 0, false);
        chunk_items(P, b->interleave, b->grid);
    } else {
        for (int k : b->order) add(k, -1, true);
    }
    make_ranges(P.h_items, P.h_edge, b->grid, P.h_ranges);
}

void release_graph(fk_batch *b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
    b->graph_steps = 0;
}

// The device table of the resident launches: per tissue its arguments (state to state), its plan and
// its place.
void fill_resident(fk_batch *b) {
    b->h_res.resize(b->n);
    for (const ResWave &w : b->res.w) {
        int block = 0;
        for (size_t i = 0; i < w.tissue.size(); ++i) {
            const int k = w.tissue[i];
            const ResPlan &p = w.plan[i];
            ResTissue &t = b->h_res[w.first + (int)i];
            std::memset(&t, 0, sizeof t);
            t.args = b->h_tissues[k].args[0];
            const int64_t plane = b->grids[k].H * b->grids[k].pitch;
            t.args.vo = const_cast<float *>(t.args.v);
            t.args.wo = t.args.vo + plane;
            t.args.uo = t.args.vo + 2 * plane;
            t.nr = p.nr;
            t.nc = p.nc;
            t.ng = p.ng;
            t.nq = p.nq;
            t.su_w = p.su_w;
            t.first = block;
            t.id = k;
            block += (int)p.tiles;
        }
    }
}

// n steps from t0 of every tissue through the resident launches: in place; or, n at most kResMaxSteps,
// leaving the tissues' own states as they were and writing those of tissue k to base + k * stride + an
// offset: every x_{t0+s}, s = 1 .. n, at offset s * every, or those of the steps steps[i] (n_outs of
// them, the last one t0 + n) at offset outs[i] - base.  kRefused: the first launch was, nothing ran.
struct ResOut {
    float *base = nullptr;
    int64_t stride = 0, every = 0;
    const int64_t *steps = nullptr;
    float *const *outs = nullptr;
    int n_outs = 0;
};
int run_resident(const fk_batch *b, int64_t t0, int64_t n, const ResOut &out, cudaStream_t s) {
    for (const ResWave &w : b->res.w) {
        ResidentArgs ra = w.args;
        ra.xchg = b->d_xchg;
        ra.tissues = b->d_res + w.first;
        ra.base = out.base;
        ra.tissue_stride = out.stride;
        ra.every = out.every;
        StepArgs a{};  // the constants of the launch come from its classes
        a.m = ra.cls[0].m;
        a.dt = ra.cls[0].dt;
        a.rdx = ra.cls[0].rdx;
        for (int64_t done = 0; done < n;) {
            const int64_t c = std::min<int64_t>(n - done, n - done == kResMaxSteps + 1 ? kResMaxSteps - 1
                                                                                      : kResMaxSteps);
            ra.t0 = t0 + done;
            ra.n = (int)c;
            ra.n_out = 1;
            ra.out_step[0] = (int)c;
            ra.out_off[0] = 0;
            if (out.outs) {
                ra.n_out = out.n_outs;
                for (int k = 0; k < out.n_outs; ++k) {
                    ra.out_step[k] = (int)(out.steps[k] - t0);
                    ra.out_off[k] = out.outs[k] - out.base;
                }
            }
            if (cudaMemsetAsync(b->d_xchg, 0, (size_t)(w.ctas * 2 * ra.slot) * 8, s) != cudaSuccess)
                return FK_ERR_CUDA;
            const cudaError_t e = launch_resident(w.rows, w.ctas, w.threads, w.smem, false, ra, a, s);
            if (e != cudaSuccess)
                return e == kResRefused && &w == b->res.w.data() && done == 0 ? kRefused : FK_ERR_CUDA;
            done += c;
        }
    }
    return FK_OK;
}

// Whether the tissues all lie on one grid; *ns: floats of a state.
bool one_grid(const fk_batch *b, int64_t *ns) {
    const StepArgs &a0 = b->h_tissues[0].args[0];
    for (int e = 1; e < b->n; ++e) {
        const StepArgs &a = b->h_tissues[e].args[0];
        if (a.H != a0.H || a.W != a0.W || a.pitch != a0.pitch) return false;
    }
    *ns = 3 * (int64_t)a0.H * a0.pitch;
    return true;
}

}  // namespace

extern "C" {

size_t fk_batch_workspace_bytes(const fk_tissue *tissues, int n) {
    if (!tissues || n <= 0) return 0;
    int64_t items[kShapes] = {};
    for (int k = 0; k < n; ++k)
        for (int q = 0; q < kShapes; ++q) items[q] += tiles_of(tissues[k].g, q);
    return layout(n, items, plan_waves(tissues, n)).total;
}

int fk_batch_create(const fk_tissue *tissues, int n, void *workspace, size_t bytes, void *stream,
                    fk_batch **out) {
    if (!tissues || !workspace || !out) return FK_ERR_NULL;
    if (n <= 0 || n > (1 << 20)) return FK_ERR_ARGUMENT;
    if ((reinterpret_cast<uintptr_t>(workspace) & (kAlign - 1)) != 0) return FK_ERR_ALIGN;
    int64_t n_items[kShapes] = {};
    bool any_act = false, all_act = true;
    for (int k = 0; k < n; ++k) {
        const fk_tissue &t = tissues[k];
        int rc = check_grid(t.g);
        if (rc) return rc;
        if (!t.state || !t.scratch || !t.D) return FK_ERR_NULL;
        if (!aligned16(t.state) || !aligned16(t.scratch) || !aligned16(t.D)) return FK_ERR_ALIGN;
        if (!(t.dx > 0.0) || !std::isfinite(t.dx) || !std::isfinite(t.dt)) return FK_ERR_ARGUMENT;
        const bool a = t.act.last != nullptr;
        if (a && (!t.act.first || !t.act.count)) return FK_ERR_NULL;
        any_act |= a;
        all_act &= a;
        for (int q = 0; q < kShapes; ++q) n_items[q] += tiles_of(t.g, q);
    }
    if (any_act && !all_act) return FK_ERR_ARGUMENT;  // tracking is all or nothing per batch
    for (int q = 0; q < kShapes; ++q)
        if (n_items[q] > (int64_t(1) << 30)) return FK_ERR_SHAPE;
    ResWaves res = plan_waves(tissues, n);
    Layout L = layout(n, n_items, res);
    if (bytes < L.total && res.ok()) {  // a workspace of the stepping kernel alone will do
        res = ResWaves();
        L = layout(n, n_items, res);
    }
    if (bytes < L.total) return FK_ERR_ARGUMENT;

    fk_batch *b = new (std::nothrow) fk_batch();
    if (!b) return FK_ERR_ARGUMENT;
    b->n = n;
    b->act = any_act;
    b->status = status_ptr();
    if (!b->status || cudaGetDevice(&b->device) != cudaSuccess) {
        delete b;
        return FK_ERR_CUDA;
    }
    int n_sm = 0;
    cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, b->device);
    b->grid = n_sm > 0 ? n_sm * kShape[0].ctas_per_sm : 1;
    b->grid_tb = n_sm > 0 ? n_sm : 1;
    if (b->grid > kBatchMaxGrid) b->grid = kBatchMaxGrid;
    char *ws = static_cast<char *>(workspace);
    b->d_tissues = reinterpret_cast<BatchTissue *>(ws + L.tissues);
    b->d_tbmaps = reinterpret_cast<BatchTbMaps *>(ws + L.tbmaps);
    b->h_tbmaps.resize(n);
    b->tb_ok = !any_act;
    for (int k = 0; k < n; ++k) b->tb_ok &= tb_batchable(tissues[k].g.H, tissues[k].g.W);
    b->d_t = reinterpret_cast<int *>(ws + L.t);
    b->res = std::move(res);
    b->resident = b->res.ok() ? 1 : 0;
    b->d_res = reinterpret_cast<ResTissue *>(ws + L.res);
    b->d_xchg = reinterpret_cast<uint64_t *>(ws + L.xchg);
    for (int k = 0; k < n; ++k) b->cells += tissues[k].g.H * tissues[k].g.W;
    b->h_tissues.resize(n);
    for (int q = 0; q < kShapes; ++q) {
        fk_batch::PerShape &P = b->sp[q];
        P.d_maps = reinterpret_cast<BatchMaps *>(ws + L.maps[q]);
        P.d_items = reinterpret_cast<BatchItem *>(ws + L.items[q]);
        P.d_ranges = reinterpret_cast<int *>(ws + L.ranges[q]);
        P.n_items = (int)n_items[q];
        P.h_maps.resize(n);
    }

    // tiles of the larger tissues first: the persistent CTAs then finish together
    std::vector<int> order(n);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
        return tiles_of(tissues[x].g, 0) > tiles_of(tissues[y].g, 0);
    });
    for (int k = 0; k < n; ++k) {
        const fk_tissue &t = tissues[k];
        const int64_t plane = t.g.H * t.g.pitch;
        Stim st[kMaxStim];
        int rc = make_stims(t.stimuli, t.n_stimuli, t.g, st);
        const Model m = make_model(t.params);
        // TMA maps per geometry: u with a 4-cell halo, D with a 2-row halo (columns: 4 cells)
        for (int q = 0; q < kShapes && !rc; ++q) {
            const TileShape &ts = kShape[q];
            const int sw = ts.cols + 8, su_h = ts.rows + 8, sd_h = ts.rows + 4;
            BatchMaps &bm = b->sp[q].h_maps[k];
            if ((rc = make_plane_map(&bm.maps[0].d, t.D, t.g.H, t.g.W, t.g.pitch, sw, sd_h))) break;
            for (int p = 0; p < 2 && !rc; ++p) {
                const float *in = p ? t.scratch : t.state;
                float *o = p ? t.state : t.scratch;
                StepMaps &sm = bm.maps[p];
                if (p) sm.d = bm.maps[0].d;
                if ((rc = make_plane_map(&sm.u, in + 2 * plane, t.g.H, t.g.W, t.g.pitch, sw, su_h)) ||
                    (rc = make_plane_map(&sm.ov, o, t.g.H, t.g.W, t.g.pitch, ts.cols, ts.rows)) ||
                    (rc = make_plane_map(&sm.ow, o + plane, t.g.H, t.g.W, t.g.pitch, ts.cols,
                                         ts.rows)) ||
                    (rc = make_plane_map(&sm.ou, o + 2 * plane, t.g.H, t.g.W, t.g.pitch, ts.cols,
                                         ts.rows)))
                    break;
            }
        }
        // the blocked kernel's maps (haloed boxes of the loaded planes, output-tile boxes)
        if (!rc && b->tb_ok) {
            int bw = 0, bh = 0, ow = 0, oh = 0;
            tb_box(kBatchTbDepth, &bw, &bh, &ow, &oh);
            const fk_grid &g = t.g;
            for (int p = 0; p < 2 && !rc; ++p) {
                const float *in = p ? t.scratch : t.state;
                float *o = p ? t.state : t.scratch;
                TbMaps &tm = b->h_tbmaps[k].maps[p];
                if ((rc = make_plane_map(&tm.d, t.D, g.H, g.W, g.pitch, bw, bh)) ||
                    (rc = make_plane_map(&tm.v, in, g.H, g.W, g.pitch, bw, bh)) ||
                    (rc = make_plane_map(&tm.w, in + plane, g.H, g.W, g.pitch, bw, bh)) ||
                    (rc = make_plane_map(&tm.u, in + 2 * plane, g.H, g.W, g.pitch, bw, bh)) ||
                    (rc = make_plane_map(&tm.ov, o, g.H, g.W, g.pitch, ow, oh)) ||
                    (rc = make_plane_map(&tm.ow, o + plane, g.H, g.W, g.pitch, ow, oh)) ||
                    (rc = make_plane_map(&tm.ou, o + 2 * plane, g.H, g.W, g.pitch, ow, oh)))
                    break;
            }
        }
        for (int p = 0; p < 2 && !rc; ++p) {
            const float *in = p ? t.scratch : t.state;
            float *o = p ? t.state : t.scratch;
            StepArgs &a = b->h_tissues[k].args[p];
            std::memset(&a, 0, sizeof(a));
            a.v = in;
            a.w = in + plane;
            a.u = in + 2 * plane;
            a.D = t.D;
            a.vo = o;
            a.wo = o + plane;
            a.uo = o + 2 * plane;
            a.H = (int)t.g.H;
            a.W = (int)t.g.W;
            a.pitch = (int)t.g.pitch;
            a.dt = (float)t.dt;
            a.rdx = 1.0f / (float)t.dx;
            a.n_stim = t.n_stimuli;
            a.m = m;
            for (int s = 0; s < t.n_stimuli; ++s) a.stim[s] = st[s];
            a.status = b->status;
            if (any_act) {
                a.act_first = t.act.first;
                a.act_last = t.act.last;
                a.act_count = t.act.count;
                a.act_threshold = t.act.threshold;
            }
        }
        if (rc) {
            delete b;
            return rc;
        }
    }
    b->order = order;
    b->grids.resize(n);
    for (int k = 0; k < n; ++k) b->grids[k] = tissues[k].g;
    for (int q = 0; q < kShapes; ++q) build_items(b, q);
    if (b->res.ok()) fill_resident(b);
    cudaStream_t s = (cudaStream_t)stream;
    bool ok = cudaMemcpyAsync(b->d_tissues, b->h_tissues.data(), sizeof(BatchTissue) * n,
                              cudaMemcpyHostToDevice, s) == cudaSuccess;
    if (ok && b->res.ok())
        ok = cudaMemcpyAsync(b->d_res, b->h_res.data(), sizeof(ResTissue) * n, cudaMemcpyHostToDevice,
                             s) == cudaSuccess;
    if (ok && b->tb_ok)
        ok = cudaMemcpyAsync(b->d_tbmaps, b->h_tbmaps.data(), sizeof(BatchTbMaps) * n,
                             cudaMemcpyHostToDevice, s) == cudaSuccess;
    for (int q = 0; q < kShapes && ok; ++q) {
        const fk_batch::PerShape &P = b->sp[q];
        ok = cudaMemcpyAsync(P.d_maps, P.h_maps.data(), sizeof(BatchMaps) * n,
                             cudaMemcpyHostToDevice, s) == cudaSuccess &&
             cudaMemcpyAsync(P.d_items, P.h_items.data(), sizeof(BatchItem) * P.n_items,
                             cudaMemcpyHostToDevice, s) == cudaSuccess &&
             cudaMemcpyAsync(P.d_ranges, P.h_ranges.data(), sizeof(int) * P.h_ranges.size(),
                             cudaMemcpyHostToDevice, s) == cudaSuccess;
    }
    if (!ok || cudaStreamSynchronize(s) != cudaSuccess) {
        delete b;
        return FK_ERR_CUDA;
    }
    *out = b;
    return FK_OK;
}

int fk_batch_set_resident(fk_batch *b, int on) {
    if (!b) return FK_ERR_NULL;
    if (on && !b->res.ok()) return FK_ERR_ARGUMENT;
    b->resident = on == 2 ? 2 : on != 0;
    return FK_OK;
}

int fk_batch_takes_resident(const fk_batch *b, int64_t steps) {
    return b && steps >= 2 && takes_resident(b, steps) ? 1 : 0;
}

int fk_batch_set_grid(fk_batch *b, int ctas) {
    if (!b) return FK_ERR_NULL;
    if (ctas < 1 || ctas > kBatchMaxGrid) return FK_ERR_ARGUMENT;
    b->resident = 0;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != b->device) return FK_ERR_CUDA;
    // ordered after the plan's earlier work; the host copies stay alive in the plan
    if (cudaDeviceSynchronize() != cudaSuccess) return FK_ERR_CUDA;
    b->grid = ctas;
    for (int q = 0; q < kShapes; ++q) {
        fk_batch::PerShape &P = b->sp[q];
        if (b->interleave > 1) {  // the chunk permutation depends on the CTA count
            build_items(b, q);
            if (cudaMemcpy(P.d_items, P.h_items.data(), sizeof(BatchItem) * P.n_items,
                           cudaMemcpyHostToDevice) != cudaSuccess)
                return FK_ERR_CUDA;
        }
        std::vector<int> r;
        make_ranges(P.h_items, P.h_edge, ctas, r);
        if (cudaMemcpy(P.d_ranges, r.data(), sizeof(int) * r.size(), cudaMemcpyHostToDevice) !=
            cudaSuccess)
            return FK_ERR_CUDA;
        P.h_ranges.swap(r);
    }
    release_graph(b);
    return FK_OK;
}

int fk_batch_set_options(fk_batch *b, int interleave, int packed) {
    if (!b) return FK_ERR_NULL;
    if (interleave != 0 && interleave != 1 && interleave != 2 && interleave != 4 &&
        interleave != 8)
        return FK_ERR_ARGUMENT;
    b->resident = 0;
    const int il = interleave, pk = packed ? 1 : 0;
    if (il != b->interleave || pk != b->packed) release_graph(b);
    b->packed = pk;
    if (il == b->interleave) return FK_OK;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != b->device) return FK_ERR_CUDA;
    b->interleave = il;
    // the work lists change order: rebuild and upload them after the plan's earlier work
    if (cudaDeviceSynchronize() != cudaSuccess) return FK_ERR_CUDA;
    for (int q = 0; q < kShapes; ++q) {
        build_items(b, q);
        const fk_batch::PerShape &P = b->sp[q];
        if (cudaMemcpy(P.d_items, P.h_items.data(), sizeof(BatchItem) * P.n_items,
                       cudaMemcpyHostToDevice) != cudaSuccess ||
            cudaMemcpy(P.d_ranges, P.h_ranges.data(), sizeof(int) * P.h_ranges.size(),
                       cudaMemcpyHostToDevice) != cudaSuccess)
            return FK_ERR_CUDA;
    }
    return FK_OK;
}

int fk_batch_set_depth(fk_batch *b, int depth) {
    if (!b) return FK_ERR_NULL;
    if (depth != 1 && depth != kBatchTbDepth) return FK_ERR_ARGUMENT;
    if (depth != 1 && !b->tb_ok) return FK_ERR_ARGUMENT;
    b->resident = 0;
    if (depth != b->depth) release_graph(b);
    b->depth = depth;
    return FK_OK;
}

int fk_batch_set_tile_rows(fk_batch *b, int rows) {
    if (!b) return FK_ERR_NULL;
    for (int q = 0; q < kShapes; ++q)
        if (kShape[q].rows == rows) {
            if (b->shape != q) release_graph(b);
            b->resident = 0;
            b->shape = q;
            return FK_OK;
        }
    return FK_ERR_ARGUMENT;
}

static cudaError_t launch_one(const fk_batch *b, int n_items, int t_offset, int parity, bool act,
                              cudaStream_t s) {
    const fk_batch::PerShape &P = b->sp[b->shape];
    return kShape[b->shape].launch(b->d_tissues, P.d_maps, P.d_items, P.d_ranges, n_items,
                                   b->interleave, b->packed, b->d_t, t_offset, parity, act,
                                   b->status, b->grid, s);
}

// Buffer flips of `count` steps (each launch reads one buffer and writes the other): one per
// step at depth 1; at depth 2 one per pair of steps plus one for an odd last step.
static int64_t flips(const fk_batch *b, int64_t count) {
    return b->depth == 1 ? count : count / 2 + (count & 1);
}

static int launch_steps(fk_batch *b, int count, cudaStream_t s) {
    if (b->depth == 1) {
        const int n_items = b->sp[b->shape].n_items;
        for (int k = 0; k < count; ++k)
            if (launch_one(b, n_items, k, k & 1, b->act, s) != cudaSuccess) return FK_ERR_CUDA;
    } else {  // two steps per launch of the blocked kernel (32 x 64 work items), then the odd one
        const fk_batch::PerShape &P = b->sp[0];
        int k = 0, f = 0;
        for (; k + 2 <= count; k += 2, ++f)
            if (launch_batch_tb(b->d_tissues, b->d_tbmaps, P.d_items, P.n_items, b->d_t, k, f & 1,
                                b->status, b->grid_tb, s) != cudaSuccess)
                return FK_ERR_CUDA;
        if (k < count &&
            launch_one(b, b->sp[b->shape].n_items, k, f & 1, b->act, s) != cudaSuccess)
            return FK_ERR_CUDA;
    }
    return launch_add_int(b->d_t, count, s) == cudaSuccess ? FK_OK : FK_ERR_CUDA;
}

static int ensure_graph(fk_batch *b, int steps) {
    const int opts = b->interleave * 2 + b->packed;
    if (b->exec && b->graph_steps == steps && b->graph_grid == b->grid &&
        b->graph_shape == b->shape && b->graph_opts == opts && b->graph_depth == b->depth)
        return FK_OK;
    release_graph(b);
    if (!b->capture_stream &&
        cudaStreamCreateWithFlags(&b->capture_stream, cudaStreamNonBlocking) != cudaSuccess)
        return FK_ERR_CUDA;
    // first launch of each kernel outside capture (sets function attributes)
    if (cudaStreamBeginCapture(b->capture_stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
        return FK_ERR_CUDA;
    int rc = launch_steps(b, steps, b->capture_stream);
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(b->capture_stream, &g);
    if (rc || e != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        return rc ? rc : FK_ERR_CUDA;
    }
    if (cudaGraphInstantiate(&b->exec, g, 0) != cudaSuccess) {
        cudaGraphDestroy(g);
        return FK_ERR_CUDA;
    }
    b->graph = g;
    b->graph_steps = steps;
    b->graph_grid = b->grid;
    b->graph_shape = b->shape;
    b->graph_opts = opts;
    b->graph_depth = b->depth;
    return FK_OK;
}

__global__ static void set_int_kernel(int *p, int v) { *p = v; }

int fk_batch_forward_euler(fk_batch *b, int64_t t0, int64_t t1, int graph_steps, void *stream) {
    if (!b) return FK_ERR_NULL;
    if (t1 < t0 || t1 > (int64_t(1) << 24) || t0 < -(int64_t(1) << 24) || graph_steps < 0)
        return FK_ERR_ARGUMENT;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != b->device) return FK_ERR_CUDA;
    cudaStream_t s = (cudaStream_t)stream;
    int64_t n = t1 - t0;
    if (n == 0) return FK_OK;
    // (two steps at least: in place, a block may write its cells only after its neighbours' first loads)
    if (n >= 2 && takes_resident(b, n)) {
        const int rc = run_resident(b, t0, n, ResOut{}, s);
        if (rc != kRefused) return rc;
    }
    set_int_kernel<<<1, 1, 0, s>>>(b->d_t, (int)t0);
    if (cudaGetLastError() != cudaSuccess) return FK_ERR_CUDA;
    // the smem attribute must be set outside any capture: one plain (empty-range) call does it
    int rc;
    if (graph_steps > 0) {
        // a replay must flip the buffers an even number of times: G steps, G even (depth 1) or
        // a multiple of 4 (depth 2: G / 2 launches)
        const int q = b->depth == 1 ? 2 : 4;
        const int G = (graph_steps + q - 1) / q * q;
        if (n >= G) {
            if (!b->exec || b->graph_steps != G || b->graph_grid != b->grid ||
                b->graph_shape != b->shape || b->graph_opts != b->interleave * 2 + b->packed ||
                b->graph_depth != b->depth) {
                if ((rc = launch_steps(b, 0, s))) return rc;
                if (launch_one(b, 0, 0, 0, b->act, s) != cudaSuccess)  // configures the kernel
                    return FK_ERR_CUDA;
                if (b->depth != 1 &&
                    launch_batch_tb(b->d_tissues, b->d_tbmaps, b->sp[0].d_items, 0, b->d_t, 0, 0,
                                    b->status, b->grid_tb, s) != cudaSuccess)
                    return FK_ERR_CUDA;
                if ((rc = ensure_graph(b, G))) return rc;
            }
            for (int64_t r = 0; r < n / G; ++r)
                if (cudaGraphLaunch(b->exec, s) != cudaSuccess) return FK_ERR_CUDA;
            n %= G;
        }
    }
    if ((rc = launch_steps(b, (int)n, s))) return rc;
    if (flips(b, n) & 1) {  // the replayed graphs flipped an even number of times
        if (launch_batch_copyback(b->d_tissues, b->n, s) != cudaSuccess) return FK_ERR_CUDA;
    }
    return FK_OK;
}

// Copies the state held by buffer `parity` of every tissue (0: state, 1: scratch; three
// consecutive planes) to dst + e * exp_stride (tissue e, all on one grid of `ns` floats).
__global__ static void batch_state_out_kernel(const BatchTissue *tissues, int parity, float *dst,
                                              int64_t exp_stride, int64_t ns) {
    const float4 *src = reinterpret_cast<const float4 *>(tissues[blockIdx.y].args[parity].v);
    float4 *out = reinterpret_cast<float4 *>(dst + (int64_t)blockIdx.y * exp_stride);
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < ns / 4;
         k += (int64_t)gridDim.x * blockDim.x)
        out[k] = __ldcg(src + k);
}

// The other way: tissue e's state from src + e * exp_stride.
__global__ static void batch_state_in_kernel(const BatchTissue *tissues, const float *src, int64_t exp_stride,
                                             int64_t ns) {
    float4 *dst = reinterpret_cast<float4 *>(const_cast<float *>(tissues[blockIdx.y].args[0].v));
    const float4 *in = reinterpret_cast<const float4 *>(src + (int64_t)blockIdx.y * exp_stride);
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < ns / 4;
         k += (int64_t)gridDim.x * blockDim.x)
        __stcg(dst + k, __ldcg(in + k));
}

int fk_batch_forward_states(fk_batch *b, int64_t t0, const int64_t *steps, float *const *outs, int n_steps,
                            int64_t exp_stride, void *stream) {
    if (!b || (n_steps > 0 && (!steps || !outs))) return FK_ERR_NULL;
    if (n_steps < 0 || t0 < -(int64_t(1) << 24)) return FK_ERR_ARGUMENT;
    int64_t ns = 0;
    if (!one_grid(b, &ns)) return FK_ERR_SHAPE;
    if ((exp_stride & 3) || exp_stride < ns) return FK_ERR_ALIGN;
    for (int k = 0; k < n_steps; ++k) {
        if (steps[k] < (k ? steps[k - 1] : t0) || steps[k] > (int64_t(1) << 24)) return FK_ERR_ARGUMENT;
        if (!outs[k]) return FK_ERR_NULL;
        if (reinterpret_cast<uintptr_t>(outs[k]) & 15u) return FK_ERR_ALIGN;
    }
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != b->device) return FK_ERR_CUDA;
    cudaStream_t s = (cudaStream_t)stream;
    const dim3 cgrid(64, b->n);
    int64_t t = t0;
    bool refused = false;
    for (int k = 0; k < n_steps;) {
        // as many states, of distinct steps, as one resident launch writes
        int m = 0;
        if (b->resident && !refused)
            while (k + m < n_steps && m < kResMaxOut && steps[k + m] > (m ? steps[k + m - 1] : t) &&
                   steps[k + m] - t <= kResMaxSteps)
                ++m;
        const int64_t n = m ? steps[k + m - 1] - t : 0;
        // (a stepped state is also copied out, and one more resident launch copies the last one back)
        const double copy = 2.0 + (double)b->cells / 170e3;
        if (m && takes_resident(b, n, m * copy, copy)) {
            int rc = run_resident(b, t, n, ResOut{outs[k], exp_stride, 0, steps + k, outs + k, m}, s);
            if (rc == kRefused) {
                refused = true;
                continue;
            }
            if (rc) return rc;
            k += m;
            batch_state_in_kernel<<<cgrid, 256, 0, s>>>(b->d_tissues, outs[k - 1], exp_stride, ns);
        } else {
            int rc = fk_batch_forward_euler(b, t, steps[k], 0, stream);
            if (rc) return rc;
            batch_state_out_kernel<<<cgrid, 256, 0, s>>>(b->d_tissues, 0, outs[k], exp_stride, ns);
            ++k;
        }
        if (cudaGetLastError() != cudaSuccess) return FK_ERR_CUDA;
        t = steps[k - 1];
    }
    return FK_OK;
}

int fk_batch_recompute(fk_batch *b, int64_t s, int64_t n, float *bufs, int64_t exp_stride,
                       void *stream) {
    if (!b || !bufs) return FK_ERR_NULL;
    if (n < 1 || s < -(int64_t(1) << 24) || s + n > (int64_t(1) << 24)) return FK_ERR_ARGUMENT;
    if (b->act) return FK_ERR_ARGUMENT;  // recomputed steps must not record activations again
    int64_t ns = 0;
    if (!one_grid(b, &ns)) return FK_ERR_SHAPE;
    if (exp_stride < n * ns || (reinterpret_cast<uintptr_t>(bufs) & 15u) || (exp_stride & 3))
        return FK_ERR_ALIGN;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != b->device) return FK_ERR_CUDA;
    cudaStream_t cs = (cudaStream_t)stream;
    const dim3 cgrid(64, b->n);
    // (a step outside the resident kernel also copies its states out: 12 bytes per cell read and
    // written, at about 4 TB/s from L2)
    if (n - 1 >= 2 && n - 1 <= kResMaxSteps &&
        takes_resident(b, n - 1, (double)(n - 1) * (2.0 + (double)b->cells / 170e3))) {
        batch_state_out_kernel<<<cgrid, 256, 0, cs>>>(b->d_tissues, 0, bufs, exp_stride, ns);
        if (cudaGetLastError() != cudaSuccess) return FK_ERR_CUDA;
        const int rc = run_resident(b, s, n - 1, ResOut{bufs, exp_stride, ns, nullptr, nullptr, 0}, cs);
        if (rc != kRefused) return rc;
    }
    set_int_kernel<<<1, 1, 0, cs>>>(b->d_t, (int)s);
    batch_state_out_kernel<<<cgrid, 256, 0, cs>>>(b->d_tissues, 0, bufs, exp_stride, ns);
    if (cudaGetLastError() != cudaSuccess) return FK_ERR_CUDA;
    for (int64_t k = 1; k < n; ++k) {
        // step s+k-1 reads buffer (k-1)&1 and leaves x_{s+k} in buffer k&1
        if (launch_one(b, b->sp[b->shape].n_items, (int)(k - 1), (int)((k - 1) & 1), false, cs) !=
            cudaSuccess)
            return FK_ERR_CUDA;
        batch_state_out_kernel<<<cgrid, 256, 0, cs>>>(b->d_tissues, (int)(k & 1), bufs + k * ns,
                                                      exp_stride, ns);
        if (cudaGetLastError() != cudaSuccess) return FK_ERR_CUDA;
    }
    return FK_OK;
}

int fk_batch_destroy(fk_batch *b) {
    if (!b) return FK_ERR_NULL;
    release_graph(b);
    if (b->capture_stream) cudaStreamDestroy(b->capture_stream);
    delete b;
    return FK_OK;
}

}  // extern "C"
