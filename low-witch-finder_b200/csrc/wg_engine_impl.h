// The engine object behind include/witchgpu.h (private to the library).
#pragma once

#include <cuda_runtime.h>

#include <cstdio>
#include <string>
#include <vector>

#include "../../include/witchgpu.h"
#include "wg_tiling.h"
#include "wg_phase1.cuh"

namespace wg {
struct P2Tables;
struct P2World;
struct P2Chunk;
struct P2Hut;
struct P2Result;
struct QueueRes;
}  // namespace wg

struct wg_engine {
    int device = 0;
    int sm_count = 148;
    int unit_per_sm[2] = {1, 1};   // unit_ctas_per_sm of the FP64 and the FP32 instance
    int fp32_core = 1;   // 1 FP32 core with FP64 rechecks, 3 also the cave samples, 0 FP64, 2 as 3 re-taking every gate
    int job_queue = 1;   // wg_seed_check_jobs through the device work queue (1) or the host batch loop (0)
    // autotuned job settings (wg_engine_tune): regions per unit per job class (0 = window_for's
    // rule) and (seed, region) checks per queue slice (0 = kWorkPerBatch)
    uint32_t tuned_win[4] = {0, 0, 0, 0};
    uint64_t tuned_budget = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaStream_t copy_stream = nullptr;   // host seed uploads of wg_seed_check, one batch ahead
    cudaEvent_t ev_up = nullptr;          // recorded after the last upload enqueued
    std::string err;

    uint32_t *rec_unit = nullptr, *rec_off = nullptr, *rec_cnt = nullptr, *surv = nullptr, *deep = nullptr;
    wg::Candidate *out = nullptr;
    uint32_t *counters = nullptr;
    unsigned long long *hist = nullptr;
    uint32_t *h_counters = nullptr;         // pinned; h_hist lies behind it
    unsigned long long *h_hist = nullptr;
    // pinned staging of large results (copy_result), kept at its largest size up to kStageBytes
    char *stage = nullptr;
    size_t stage_bytes = 0;
    cudaEvent_t stage_ev[8] = {};
    cudaEvent_t kev[4] = {nullptr, nullptr, nullptr, nullptr};   // around the three kernels of a batch
    int64_t *d_seed_list = nullptr;
    uint64_t d_seed_cap = 0;
    // breadth-first climate stage of one-region batches: two item lists and their counts
    wg::RegionList lists[2] = {};         // the list kernels' alternating lists, in one block
    void *list_block = nullptr;
    wg::SpotItem *spot_items[2] = {nullptr, nullptr};
    uint32_t *spot_counts = nullptr;

    // phase 2 (wg_p2engine.cu): device tables, grow-only work buffers
    wg::P2Tables *p2_tables = nullptr;
    std::vector<void *> p2_game;          // device copies of the game data tables
    wg::P2World *p2_worlds = nullptr;
    wg::P2Chunk *p2_jobs = nullptr;
    wg::P2Hut *p2_huts = nullptr;
    wg::P2Result *p2_results = nullptr;
    int32_t *p2_pts = nullptr;
    double *p2_vals = nullptr;
    // Deep Dive solver (wg_solve.cu): its device tables and work buffers
    struct SolveState *solve = nullptr;
    // Deep Dive region walk (wg_deep.cu): its grow-only work buffers
    struct WalkState *walk = nullptr;
    // device work queue of batched jobs (wg_queue.cu): its state and output buffer
    wg::QueueRes *queue = nullptr;
    // mineshaft finisher (wg_finish.cu): its grow-only buffers
    struct FinishState *finish = nullptr;

    int p2_world_cap = 0, p2_job_cap = 0, p2_hut_cap = 0, p2_result_cap = 0, p2_pt_cap = 0, p2_val_cap = 0;

    int fail(int code, const char *what, cudaError_t e = cudaSuccess) {
        char buf[512];
        if (e != cudaSuccess) std::snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
        else std::snprintf(buf, sizeof buf, "%s", what);
        err = buf;
        return code;
    }
};

// Frees the phase-2 state of an engine (called by wg_engine_close).
void p2_release(wg_engine *eng);
// Frees the Deep Dive solver state of an engine (called by wg_engine_close).
void solve_release(wg_engine *eng);
// Frees the region walk's buffers of an engine (called by wg_engine_close).
void walk_release(wg_engine *eng);
// Frees the finisher's buffers of an engine (called by wg_engine_close).
void finish_release(wg_engine *eng);

namespace wg {

// Phase-2 state of up to 512 chunks (wg_p2engine.cu): the seed-independent tables, the worlds of
// `seeds` (large biomes or not) and, per chunk i (world index world[i], chunk cx[i], cz[i]), its
// grid, aquifer, block states and carver result in eng->p2_worlds / eng->p2_jobs, chunk i at
// index i.  Asynchronous on eng->stream.
int p2_prepare_chunks(wg_engine *eng, const std::vector<uint64_t> &seeds, int large, const std::vector<int> &world,
                      const std::vector<int> &cx, const std::vector<int> &cz);

// The counters' and the funnel's block.
constexpr size_t kHistOffset = 128, kCountBytes = kHistOffset + sizeof(unsigned long long) * (P1_KINDS + kTiers);
static_assert(sizeof(uint32_t) * CNT_WORDS <= kHistOffset, "the funnel lies behind the counters");

// Copies a result from device memory, complete on eng->stream, to the caller's pageable memory.  From
// 1 MiB on through pinned staging in pieces, several threads copying pieces out (and taking the page
// faults of a fresh buffer) while later ones are on the bus.  A walk's 268k start chunks (10.7 MB) into
// a fresh buffer, whole call: 2.65-2.95 ms with one cudaMemcpy, 2.5 ms so; 8 threads 2.7 ms.
constexpr size_t kStageBytes = 16u << 20, kStagePiece = 2u << 20;
int copy_result(wg_engine *eng, void *dst, const void *src, size_t bytes);

// Per-batch work budget: (seed, region) checks per batch and units per batch, and the sizes of
// the engine's phase-1 work lists.
constexpr uint64_t kWorkPerBatch = 1ull << 27;
constexpr uint32_t kMaxUnits = 1u << 20;
constexpr uint32_t kCapRec = kMaxUnits + (1u << 16);
constexpr uint32_t kCapSurv = 1u << 23;
constexpr uint32_t kCapDeep = 1u << 20;
constexpr uint32_t kCapOut = 1u << 20;
// Units per batch of the breadth-first one-region climate stage (its item lists are this long;
// its climate survivors, ~1.7 %, stay far below the record capacity).
constexpr uint32_t kSpotUnits = 1u << 22;

// Whether a batch takes the breadth-first one-region climate stage.
inline bool spot_path(bool jobs, uint64_t win, bool codes, bool single_biome) {
    return !jobs && win == 1 && !codes && !single_biome;
}

// Regions per seed from which a unit takes the one-CTA kernel (launch_unit) however many seeds there
// are: 8,192 seeds x 2,025 regions take it 1.73 ms and the list kernels 1.41; 3,552 x 4,096 1.07 and 1.99.
constexpr uint64_t kUnitCtaRegions = 3072;
// The same for its FP64 instance, whose regions take twice as long: a rect of at most 4,096 regions, which the
// fused kernels walk as one unit (18,000 seeds x 3,249 regions 5.93 ms and 5.41 fused, x 3,364 5.83 and 5.59,
// 16,666 x 3,600 5.67 and 5.92, 14,648 x 4,096 5.11 and 6.25), and the regions per tile of a larger one (6e7
// regions in all, rects of tiles of 2,732 regions 6.83 and 5.11, 4,000 5.89 and 5.10, 4,098 5.59 and 5.11, 4,225
// 5.44 and 6.19, 4,500 5.32 and 5.53, 5,000 4.95 and 5.10, 16,384 4.1 and 6.0).
constexpr uint64_t kUnitCtaRegions64 = 3600, kUnitCtaTile64 = 4200;
// A strip of fewer regions across than this makes tiles of few regions (a tile is at most 1,023 long), so it
// takes the one-CTA kernel only for a few waves of them: 1,000 seeds x 20,000 x 1 3.11 ms and 1.66 fused, x
// 10,000 x 3 2.44 and 2.36, x 10,000 x 4 2.88 and 2.97; one seed x 1,000,000 x 1 0.21 and 0.54.
constexpr uint64_t kUnitCtaStrip = 4;
// Whether so few units are better off with one CTA each.  The fused kernels put 16 in a CTA, so their time goes up
// with every round of 16 units an SM (a second round shares the SM with the first, a third follows), the unit
// kernel's with every unit; the line of each round lies where they meet.  Measured, FP32, unit kernel's time in
// fused kernels' times at 444, 1,332, 2,331, 2,400, 4,620 and 4,842 units of 148 SMs: 81 regions 0.55, 0.93, 1.38, 1.32,
// 1.95, 1.81; 400 regions 0.43, 0.83, 1.26, 1.09, 1.72, 1.49; 1,600 regions 0.28, 0.61, 0.97, 0.79, 1.29, 0.97; 2,500
// regions 0.21, 0.49, 0.69, 0.61, 1.00, 0.77; FP64 0.54, 1.01, 1.45, 1.32, 2.08, 1.87; 0.47, 0.87, 1.32, 1.16, 1.77, 1.51;
// 0.30, 0.68, 1.10, 0.86, 1.45, 1.10; 0.23, 0.55, 0.83, 0.68, 1.13, 0.89.
bool few_units(double n_units, double n_regions, int sm_count, bool fp32);
// Whether seeds of a rw x rh rect take the one-CTA kernel however many they are (rects kUnitCtaStrip across
// and more); f32: its FP32 instance.
inline bool unit_rect(uint64_t rw, uint64_t rh, bool f32) {
    const uint64_t n = rw * rh;
    if (f32) return n >= kUnitCtaRegions;
    return n <= 4096 ? n >= kUnitCtaRegions64 : tile_rect(rw, rh, kUnitCtaMax).win() >= kUnitCtaTile64;
}

// Job classes of the autotuner by regions per seed: <= 16, <= 256, <= 4096, more.
constexpr uint64_t kJobClassMax[4] = {16, 256, 4096, ~0ull};
inline int job_class(uint64_t n_regions) {
    int c = 0;
    while (c < 3 && n_regions > kJobClassMax[c]) c++;
    return c;
}
// Regions per unit of a job: the engine's tuned value for its class, else the whole rect up to 4,096 regions, and
// above that tiles of 16,384 for the one-CTA kernel and of 2,048 for the fused kernels.
inline uint64_t job_window(const wg_engine *eng, uint64_t n_regions, bool unit) {
    const uint64_t w = eng ? eng->tuned_win[job_class(n_regions)] : 0u;
    if (!w) return n_regions <= 4096 ? n_regions : (unit ? 16384u : 2048u);
    return n_regions < w ? n_regions : w;
}
// Whether a job takes the one-CTA kernel, and its tiles.  A tuned window (the tuner tries 2,048 to 16,384) may make
// them smaller than that kernel pays for: 16 jobs of 256 seeds x 129 x 129 regions in windows of 512, 1,024 and
// 2,048 took it 14.0, 11.2 and 7.0 ms, the fused kernels 6.4, 5.7 and 5.6.
inline Tiling job_tiles(const wg_engine *eng, uint64_t rw, uint64_t rh, bool single_biome, bool f32, bool &unit) {
    const uint64_t n = rw * rh, least = f32 ? kUnitCtaRegions : n <= 4096 ? kUnitCtaRegions64 : kUnitCtaTile64;
    if (!single_biome && std::min(rw, rh) >= kUnitCtaStrip) {
        const Tiling t = tile_rect(rw, rh, std::min(job_window(eng, n, true), kUnitCtaMax));
        unit = t.win() >= least;
        if (unit) return t;
    }
    unit = false;
    return tile_rect(rw, rh, std::min<uint64_t>(job_window(eng, n, false), 4096));
}

// One phase-1 request over one rect (wg_engine.cu).
struct Request {
    const int64_t *d_seeds;   // device seeds or nullptr (generator)
    uint64_t gen_base;
    uint64_t n_seeds;
    wg_opts opts;
    int max_height, salt;
    int rx0, rx1, rz0, rz1;
    int8_t *d_codes, *d_tiers;   // optional per-region verdicts (device)
    const int64_t *d_spot_s48;   // optional spots mode (BatchArgs::spot_s48 and the spot regions)
    const int32_t *d_spot_rx, *d_spot_rz;
    const int64_t *h_seeds;      // optional host seeds: run_request uploads each batch's seeds into
                                 // d_seeds on the copy stream while the batch before it runs
};

struct Sink {            // where phase-1 survivors go after each batch
    std::vector<Candidate> *host = nullptr;
    Candidate *dev = nullptr;
    uint64_t dev_cap = 0;
    uint64_t found = 0;
};

// Units per batch from which the list kernels run the climate and first entrance stages.  Below, their
// seven builds in a row outweigh their higher rate (9 x 9 regions, fused and list kernels: 16,384 seeds
// 358 and 391 us, 24,576 482 and 467, 131,072 2,030 and 1,650; 1 x 2 regions: 228 and 270, 296 and 297,
// 1,048 and 679).
constexpr uint32_t kListUnits = 24576;
// Strips of one or two regions longer than this keep the fused kernels, whose samples do not need a lattice:
// 600,000 seeds x 200 x 1 13.8 ms and 14.9 fused, x 100 x 2 13.2 and 14.7; 60,000 x 1,000 x 1 5.17 and 4.58, x
// 1,000 x 2 8.84 and 8.24.
constexpr uint32_t kListStrip = 500;
static_assert(kListStrip < kTileSide, "only strips that stay out of the list kernels have longer tiles");
// The same for the cave gate of one-region units, 1.7 % of which reach it.
constexpr uint32_t kSpotListUnits = 1u << 19;
constexpr int kListKernels = 6;   // launches of launch_lists
// Allocates the list kernels' lists (228 MB) once per engine; false where there is no memory for them.
bool list_buffers(wg_engine *eng);
// Whether a batch of n_units units takes the list kernels.
inline bool list_path(const BatchArgs &a, uint32_t n_units) {
    const bool strip = !a.jobs && std::min(a.tw, a.th) <= 2 && std::max(a.tw, a.th) > kListStrip;
    return !a.unit_cta && a.fp32_core == 1 && a.small_coords && !a.single_biome && n_units >= kListUnits && !strip;
}
// The BatchArgs fields every batch of an engine shares (work lists, counters, rules, salt).
BatchArgs base_args(wg_engine *eng, const wg_opts &opts, int salt);
// Runs units [unit0, unit0 + n_units) of `proto` (three kernels, one sync), halving on overflow.
int run_batch(wg_engine *eng, const BatchArgs &proto, uint64_t unit0, uint32_t n_units, Sink &sink,
              wg_scan_stats &st);
int run_request(wg_engine *eng, const Request &rq, Sink &sink, wg_scan_stats &st);

}  // namespace wg
