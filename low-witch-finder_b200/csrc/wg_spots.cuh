// ------------------------------------------------------------------------------------
// Climate stage for one-region units (the Deep Dive terrain stage: 65,536 upper-bit variants of
// a spot, each a different world seed over one region).  The climate kernel builds all 18 climate
// tables of a unit because a 9 x 9 unit needs nearly all of them; a one-region unit needs the two
// tier-0 tables and then one more per erosion step it reaches (about 3.2 of 18 on average), and
// each step samples only its own octave.  So the stage runs breadth first over lists in HBM:
// tier 0 for every unit, then one kernel per erosion step over the survivors of the step before
// (one table per item, the partial sum carried in the item), then temperature and ridge for the
// erosion survivors; ridge survivors become unit records for the entrance kernel, or in batches of 2^19
// units and more go through the cave gates of wg_lists.cuh first.
// A lane owns one byte column of its warp's table area and builds one table at a time there; the warps
// of a block wait for no other (24 warps an SM).  Measured, 256 spots (1.7e7 world seeds), the whole
// stage: columns initialised byte by byte in 272-byte rows of a 256-thread block 20.4 ms, by the warp in
// 16-byte stores 20.1 ms; the cave gate's noises through the list kernels 19.7 ms.  The tier-0 kernel
// builds 3.3e9 tables/s at 65 % issue (7,376 instructions per 32 tables, 6,600 of them the shuffle): the
// table construction bounds the stage.
// ------------------------------------------------------------------------------------
#pragma once

constexpr int kSpotWarps = 4, kSpotThreads = 32 * kSpotWarps;

struct SpotSmem {
    alignas(16) uint8_t tab[kSpotWarps][kRows * 32];
    uint32_t grad[kGradWords];
};

// Builds, in every valid lane's column, the table of climate step k of its seed, and samples it at the
// unit's climate point (xc, zc).  Called by the whole warp.
__device__ __forceinline__ double spot_sample(uint8_t *tab, const uint32_t *grad, int large, int k, bool valid, uint64_t seed,
                                              double xc, double zc) {
    const ClimateStep &cs = c_steps[large][k];
    const int8_t *const sl = c_slot_a[large][cs.slot];
    const int lane = threadIdx.x & 31;
    Xr r{};
    if (valid) r = octave_rng(c_noise[sl[0]], seed_fork_of(seed), sl[1], sl[2]);
    double ox = 0.0, oy = 0.0, oz = 0.0;
    warp_build(tab, lane, valid, r, ox, oy, oz);
    if (!valid) return 0.0;
    const int jy = (int)floor(oy);
    const double hy = oy - jy;
    const ColTable<32> T{tab + lane, grad};
    return perlin_y0(T, ox, oz, jy, hy, fade(hy), keep_precision((xc * cs.sc) * cs.lac),
                     keep_precision((zc * cs.sc) * cs.lac));
}

// The unit's world seed and climate point (its only region's hut chunk middle).
__device__ __forceinline__ uint64_t spot_point(const BatchArgs &a, uint32_t u, double &xc, double &zc) {
    const UnitPos up = unit_pos(a, u);
    const uint64_t seed = seed_value(a, up.g);
    int cx, cz;
    hut_chunk(seed, up.rx, up.rz, a.salt, cx, cz);
    xc = (cx * 16 + 8) * 0.25;   // exact: an integer over 4
    zc = (cz * 16 + 8) * 0.25;
    return seed;
}

__device__ __forceinline__ void spot_append(SpotItem *out, uint32_t *out_n, uint32_t cap, bool keep, const SpotItem &it,
                                            uint32_t *overflow) {
    cg::coalesced_group grp = cg::coalesced_threads();
    const unsigned m = grp.ballot(keep);
    uint32_t base = 0;
    if (grp.thread_rank() == 0 && m) base = atomicAdd(out_n, (uint32_t)__popc(m));
    base = grp.shfl(base, 0);
    if (keep) {
        const uint32_t at = base + (uint32_t)__popc(m & ((1u << grp.thread_rank()) - 1u));
        if (at < cap) out[at] = it;
        else atomicOr(overflow, 1u);
    }
}

__device__ __forceinline__ void spot_count(unsigned long long *hist, int idx, uint32_t n) {
    const uint32_t tot = __reduce_add_sync(0xFFFFFFFFu, n);
    if ((threadIdx.x & 31) == 0 && tot) atomicAdd(&hist[idx], (unsigned long long)tot);
}

// Tier 0: lanes 2i and 2i+1 build octaves 0A and 0B of one unit; the even lane sums them in the
// reference's order and applies the tier-0 threshold.
__global__ void __launch_bounds__(kSpotThreads) spot_tier0_kernel(const __grid_constant__ BatchArgs a, SpotItem *out, uint32_t *out_n,
                                                                  uint32_t cap) {
    __shared__ SpotSmem S;
    fill_grad_table(S.grad, threadIdx.x);
    __syncthreads();
    uint8_t *const tab = S.tab[threadIdx.x >> 5];
    const int large = a.large_biomes ? 1 : 0;
    const ClimateStep &s0 = c_steps[large][0], &s1 = c_steps[large][1];
    uint32_t rejected = 0;
    const uint64_t tasks = 2ull * a.n_units;
    for (uint64_t base = (uint64_t)blockIdx.x * kSpotThreads; base < tasks; base += (uint64_t)gridDim.x * kSpotThreads) {
        const uint64_t task = base + threadIdx.x;
        const bool valid = task < tasks;
        const uint32_t u = (uint32_t)(task >> 1);
        double xc = 0.0, zc = 0.0;
        uint64_t seed = 0;
        if (valid) seed = spot_point(a, u, xc, zc);
        const double v = spot_sample(tab, S.grad, large, (int)(task & 1), valid, seed, xc, zc);
        const double v1 = __shfl_down_sync(0xFFFFFFFFu, v, 1);
        bool keep = false;
        SpotItem it{u, 0u, 0.0, 0.0};
        if (valid && !(task & 1)) {
            double sum = 0.0;
            sum += (s0.c1 * v) * s0.c2;
            sum += (s1.c1 * v1) * s1.c2;
            if (sum * s1.amp < s1.thr) rejected++;
            else {
                keep = true;
                it.sum = sum;
            }
        }
        spot_append(out, out_n, cap, keep, it, &a.counters[CNT_OVERFLOW]);
    }
    spot_count(a.hist, P1_KINDS + s1.tier, rejected);
    spot_count(a.hist, P1_EROSION, rejected);
}

// Climate steps [k0, k1) for every listed item, one table at a time per item, in the state
// machine's order (erosion tier checks, the A/B split, temperature, ridge).  Items that pass the
// last erosion tier or temperature go to `out` for the next stage; ridge survivors become unit
// records (CNT_RECORDS / CNT_SURVIVORS, one region each) for the entrance kernel.
__global__ void __launch_bounds__(kSpotThreads) spot_steps_kernel(const __grid_constant__ BatchArgs a, int k0, int k1, const SpotItem *in,
                                                                  const uint32_t *in_n, SpotItem *out, uint32_t *out_n,
                                                                  uint32_t cap) {
    __shared__ SpotSmem S;
    fill_grad_table(S.grad, threadIdx.x);
    __syncthreads();
    uint8_t *const tab = S.tab[threadIdx.x >> 5];
    const int large = a.large_biomes ? 1 : 0;
    const uint32_t n = min(*in_n, cap);
    uint32_t rej_tier = 0, rej_temp = 0, rej_ridge = 0;
    for (uint32_t base = blockIdx.x * kSpotThreads; base < n; base += gridDim.x * kSpotThreads) {
        const uint32_t e = base + threadIdx.x;
        bool keep = false;
        SpotItem it{0u, 0u, 0.0, 0.0};
        bool alive = e < n;
        double xc = 0.0, zc = 0.0, sum = 0.0, sum_a = 0.0;
        uint64_t seed = 0;
        if (alive) {
            it = in[e];
            seed = spot_point(a, it.unit, xc, zc);
            sum = it.sum;
            sum_a = it.sum_a;
        }
        for (int k = k0; k < k1 && __any_sync(0xFFFFFFFFu, alive); k++) {
            const ClimateStep &cs = c_steps[large][k];
            const double v = spot_sample(tab, S.grad, large, k, alive, seed, xc, zc);
            bool passed = false;
            if (alive) {
                sum += (cs.c1 * v) * cs.c2;
                switch (cs.act) {
                    case ACT_TIER:
                    case ACT_TIER_LAST:
                        if (sum * cs.amp < cs.thr) {
                            alive = false;
                            rej_tier++;
                        } else if (cs.act == ACT_TIER_LAST) {
                            sum = 0.0;
                        }
                        break;
                    case ACT_END_SUB_A:
                        sum_a = sum;
                        sum = 0.0;
                        break;
                    case ACT_TEMPERATURE: {
                        const double t = (sum_a + sum) * cs.amp;
                        const bool bad = a.mc_1_18_2 ? (t < -0.45) : (t > 0.2 || t < -0.45);
                        if (bad) {
                            alive = false;
                            rej_temp++;
                        }
                        sum = 0.0;
                        sum_a = 0.0;
                        break;
                    }
                    case ACT_RIDGE: {
                        const double rg = (sum_a + sum) * cs.amp;
                        if ((rg > 0.42 && rg < 0.91) || (rg < -0.42 && rg > -0.91) || (!a.pre_26_2 && rg <= -0.91)) {
                            alive = false;
                            rej_ridge++;
                        } else if (a.lists[0].surv) {
                            passed = true;
                        } else {
                            emit_single(a, it.unit, 0u);   // climate survivor: a record of one region
                        }
                        alive = false;   // ridge is the last climate step
                        break;
                    }
                    default:
                        break;
                }
            }
            if (k + 1 == kClimateSteps && a.lists[0].surv) {   // climate survivors of the warp, one region each
                const unsigned m = __ballot_sync(0xFFFFFFFFu, passed);
                const int src = (int)__fns(m, 0, (int)(threadIdx.x & 31) + 1) & 31;
                const uint32_t unit = __shfl_sync(0xFFFFFFFFu, it.unit, src);
                list_emit(a, a.lists[0], (int)(threadIdx.x & 31), (uint32_t)__popc(m), threadIdx.x & 31, unit, 0u, 0.0);
            }
        }
        if (alive) {
            keep = true;
            it.sum = sum;
            it.sum_a = sum_a;
        }
        spot_append(out, out_n, cap, keep, it, &a.counters[CNT_OVERFLOW]);
    }
    // a step kernel over erosion steps checks one tier (the caller runs one step per launch there)
    if (k1 <= 8) {
        spot_count(a.hist, P1_KINDS + (k1 - 2), rej_tier);
        spot_count(a.hist, P1_EROSION, rej_tier);
    }
    spot_count(a.hist, P1_TEMPERATURE, rej_temp);
    spot_count(a.hist, P1_RIDGE, rej_ridge);
}

static int g_spot_per_sm = 0;

void launch_spot_climate(const BatchArgs &a, SpotItem *list0, SpotItem *list1, uint32_t *counts, uint32_t cap,
                         int sm_count, cudaStream_t s) {
    if (!g_spot_per_sm) {
        int n0 = 0, n1 = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n0, spot_tier0_kernel, kSpotThreads, 0);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n1, spot_steps_kernel, kSpotThreads, 0);
        g_spot_per_sm = n0 < n1 ? n0 : n1;
        if (g_spot_per_sm < 1) g_spot_per_sm = 1;
    }
    const int grid = sm_count * g_spot_per_sm;   // the resident blocks: the kernels loop over their items
    SpotItem *lists[2] = {list0, list1};
    cudaMemsetAsync(counts, 0, sizeof(uint32_t) * 2, s);
    spot_tier0_kernel<<<grid, kSpotThreads, 0, s>>>(a, lists[0], &counts[0], cap);
    int cur = 0;
    // erosion steps 2..7, one launch each; then temperature (8..11) and ridge (12..17)
    const int bounds[][2] = {{2, 3}, {3, 4}, {4, 5}, {5, 6}, {6, 7}, {7, 8}, {8, 12}, {12, 18}};
    for (const auto &b : bounds) {
        cudaMemsetAsync(&counts[cur ^ 1], 0, sizeof(uint32_t), s);
        spot_steps_kernel<<<grid, kSpotThreads, 0, s>>>(a, b[0], b[1], lists[cur], &counts[cur], lists[cur ^ 1],
                                                        &counts[cur ^ 1], cap);
        cur ^= 1;
    }
    if (a.lists[0].surv) launch_cave_lists(a, s);
}
