// The unit kernel: all of phase 1 for one unit (a tile of one seed's regions) in one CTA.  Included by
// wg_phase1.cu (it uses its constant tables and cave formulas).
//
// (SINGLE_BIOME requests, whose every region passes the climate stage, take the fused kernels.)
// For units of many regions, and for calls too small to fill the GPU with 16-unit CTAs.  The seed's
// 18 climate tables and the entrance gate's 18 tables are built once per CTA, side by side (one
// thread each), so nothing is rebuilt per record or per candidate; the ladder's other 36 are built
// only when a region of the unit gets that far.
//
// Tier 0 and the next two erosion steps read octaves 1/512 and 1/256 of the quart coordinate: a
// region is a quarter or half of a lattice cell wide, and at y = 0 a lattice column's two corners
// blend into one linear function A x + B z + C (the y fraction is the table's).  So a 32 x 32 block of
// regions needs at most 11 x 11 and 19 x 19 such columns per table: they are formed once in shared
// memory, and a sample is four 16-byte loads and about 30 operations instead of 14 table lookups,
// 8 gradients and a 3-D blend (about 170).
//
// Coordinates are 8.56 fixed point (wg_fixed.h): base of the unit per table and axis, plus the hut's chunk
// offset times the table's step, which costs no FP64.
//
// A block costs two barriers: the next block's lattice bases are formed a block ahead, and the pool is
// looked at only when it is full.  (With six, and the lists packed after each of the erosion steps 4-7:
// 1.6e9 regions of one seed 55.9 -> 54.2 ms; barriers were 5 % of a CTA's time.)
//
// Measured against the three fused kernels, which rebuilt a seed's tables for every 2,048-region
// window, record and candidate (whole calls): one seed over the whole world (1.37e10 regions) 939 -> 425 ms, one
// seed x 24,964 regions 529 -> 105 us (13 windows in one CTA before), x 400 regions 170 -> 82 us.  Of a large unit's
// time the table builds take 2 %, the lattices 12 %, hut positions and tier 0 22 %, steps 2-3 16 %, the
// later gates 21 %, barriers 8 %, the entrance gate 12 % (its first test then in FP32; in FP64 a large unit takes
// 2 % longer), the ladder 6 %.
#pragma once

constexpr int kUThreads = 256;
constexpr int kUWarps = kUThreads / 32;
constexpr int kBlock = 32;                    // regions per side of a lattice block
constexpr int kUPitch = 516;                  // bytes between tables: 256 entries twice and one more
constexpr int kUTabs = kSlotsC;               // cave tables; the climate tables sit at 18..35 until the ladder
constexpr int kUClim = kSlotsB;               // first climate table (step order)
constexpr int kLat0 = 11, kLat1 = 19;         // lattice columns per axis of a block, octaves 1/512 and 1/256
constexpr int kLatTables = 4;                 // erosion steps 0..3
constexpr int kList = kBlock * kBlock / kUWarps;   // a warp's regions of a block: its tier-0 survivors fit
constexpr int kPoolFull = kUWarps * 64;       // pooled regions that start a drain: two full rounds a warp
constexpr int kPool = kPoolFull + kBlock * kBlock;
constexpr int kUSurv = kUThreads + kUWarps * kList;   // what waited and one drain's
constexpr int kWide = 2 * kUWarps;            // last survivors that take the entrance gate a warp each
constexpr int kUDeep = 256;                   // deep candidates finished here; more go to the ladder kernel's list
static_assert(kUClim + kSlotsA <= kUTabs, "climate tables overlay ladder tables");

// Smallest |value| of the two scaled spaghetti noises that settles spaghetti >= 0 whatever the other
// noises are.  spaghetti = clamp(max(|e l|, |e n|) - h, -1, 1) + q with h <= 0.065 + 0.023 (V + 1) / 2 and
// q >= -0.05 (1 + V)(V - 0.4), where V = 2 * 0.8334 * kPerlinMax bounds a one-octave DoublePerlin: at
// kPerlinMax = 1.0625 (a sample's largest value is 1.0364) h <= 0.0969, q >= -0.1900.
constexpr double kPerlinMax = 1.0625;
constexpr double kSpagSure = 0.29;

// Where a block lies in its lattice tables: its base in lattice coordinates of its first cell, that
// cell, and the columns per axis (and ceil(2^20 / nx)).
struct LatBase {
    uint64_t x[kLatTables], z[kLatTables];
    int cell_x[kLatTables], cell_z[kLatTables], nx[kLatTables], nz[kLatTables];
    uint32_t inv[kLatTables];
};

// What the kernel keeps of the tables' constants (err: bounds of the first entrance test's four noises in
// FP32), and each table's generator (climate tables in step order, then the cave tables).  In global
// memory: lanes that read different words of constant memory take turns, and in a call of one wave every
// turn is a miss (the 18 lanes' steps and generators: 10,000 of a CTA's 60,000 cycles, now 2,500).
struct UnitConst {
    ClimateSteps steps;
    uint64_t fstep[kSlotsA];
    double err[4];
};
struct TableRng {
    uint64_t name_lo, name_hi, oct_lo, oct_hi, sub;
};
struct UnitTables {
    alignas(16) UnitConst c;
    TableRng rng[kSlotsA + kSlotsC];
};
static_assert(sizeof(UnitConst) % 16 == 0, "copied in 16-byte words");
__device__ UnitTables g_unit_tables[2];        // [large_biomes]

static void upload_unit_tables(const NoiseSpec *specs, const ClimateStep *const steps[2], const int8_t (*slot_a)[kSlotsA][3],
                               const int8_t (*slot_c)[kSlotsC][3]) {
    UnitTables host[2];
    for (int l = 0; l < 2; l++) {
        UnitTables &u = host[l];
        auto rng = [&](const int8_t *s) {
            const NoiseSpec &n = specs[s[0]];
            return TableRng{n.name_lo, n.name_hi, n.oct_lo[s[2]], n.oct_hi[s[2]], (uint64_t)s[1]};
        };
        for (int k = 0; k < kClimateSteps; k++) {
            const ClimateStep &s = steps[l][k];
            ClimateSteps &t = u.c.steps;
            t.sc[k] = s.sc;
            t.lac[k] = s.lac;
            t.c1[k] = s.c1;
            t.c2[k] = s.c2;
            t.thr[k] = s.thr;
            t.amp[k] = s.amp;
            t.slot[k] = s.slot;
            t.act[k] = s.act;
            t.tier[k] = s.tier;
            t.cf[k] = s.cf;
            t.lo[k] = s.lo;
            t.hi[k] = s.hi;
            u.c.fstep[k] = s.fstep;
            u.rng[k] = rng(slot_a[l][s.slot]);
        }
        for (int t = 0; t < kSlotsC; t++) u.rng[kSlotsA + t] = rng(slot_c[l][t]);
        const int quick[4] = {N_SPAGHETTI_RARITY, N_SPAGHETTI_1, N_SPAGHETTI_2, N_CAVE_ENTRANCE};
        for (int q = 0; q < 4; q++) u.c.err[q] = dp_err_f32(specs[quick[q]]);
    }
    cudaMemcpyToSymbol(g_unit_tables, host, sizeof host);
}

// Regions along one side of a block of a tile that is `other` regions wide across it: kBlock, or in a thin
// tile as many as the lattices' columns hold (149 for one region: with 32 a block fed one warp of eight).
// n regions span at most 0.255 n cells of octave 1/512 and 0.51 n of 1/256, and 3 columns more.
__host__ __device__ constexpr uint32_t lattice_side(uint32_t columns, uint32_t other, uint32_t per_1000) {
    return ((columns / (other * per_1000 / 1000 + 3) - 2) * 1000 - 1) / per_1000;
}
__host__ __device__ constexpr uint32_t block_side(uint32_t other) {
    if (other >= (uint32_t)kBlock) return kBlock;
    const uint32_t a = lattice_side(kLat0 * kLat0, other, 255), b = lattice_side(kLat1 * kLat1, other, 510),
                   c = kBlock * kBlock / other;
    const uint32_t s = a < b ? a : b, t = s < c ? s : c;
    return t > (uint32_t)kBlock ? t : kBlock;
}

// What only the FP32 instance keeps: the climate tables' fixed-point constants, the lattice columns and
// where they lie.
template <bool F32>
struct UnitFixed {
    uint64_t fx[kSlotsA], fz[kSlotsA];
    float hyf[kSlotsA], fyf[kSlotsA];
    float w0[kLatTables], w1[kLatTables], c0[kLatTables], c1[kLatTables];
    LatBase lat_base[2];                       // this block's and the next one's
};
template <>
struct UnitFixed<false> {};
template <bool F32>
struct UnitLattice {
    float4 l0[2][kLat0 * kLat0];
    float4 l1[2][kLat1 * kLat1];
};
template <>
struct UnitLattice<false> {};

template <bool F32>
struct UnitSmem : UnitFixed<F32> {
    using Real = typename std::conditional<F32, float, double>::type;
    uint8_t tab[kUTabs * kUPitch];
    double org[3 * kUTabs];                    // cave tables' origins [slot][3]
    double cox[kSlotsA], coz[kSlotsA], chy[kSlotsA];   // climate tables, step order
    int jy[kSlotsA];
    union {
        UnitLattice<F32> lat;
        double mh[kUWarps][2 * kSlotsB];       // a warp's survivor at 50 and 60, or candidate at maxHeight
        LadderVals lad;
    };
    uint32_t wl[kUWarps][kList];               // a warp's list: survivor words and their erosion sums
    Real ws[kUWarps][kList];
    uint32_t pool[kPool];                      // the CTA's regions past erosion step 3
    Real pool_s[kPool];
    uint32_t surv[kUSurv];                     // climate survivors waiting for the entrance gate
    uint32_t und[2 * kUThreads];               // those its first test left open
    uint32_t deep[kUDeep];
    uint32_t n_pool, n_surv, n_und, n_deep, n_total;
    unsigned int hist[P1_KINDS + kTiers];
    uint32_t grad[kGradWords];
    GradF gf;
    alignas(16) UnitConst c;
};

// A survivor word of the unit kernel: the hut's chunk offset from the unit's first chunk, x | z << 16;
// its region is (x >> 5, z >> 5), since a hut lies in the first 24 chunks of its region.
__device__ __forceinline__ uint32_t region_word(uint32_t e) { return ((e & 0xFFFFu) >> 5) | ((e >> 21) << 16); }

struct UnitCtx {
    uint64_t seed, g;
    UnitPos up;
    int ucx, ucz;      // the unit's first chunk
};

__device__ __forceinline__ void unit_note(const BatchArgs &a, const UnitCtx &U, uint32_t e, int code, int tier) {
    if (a.codes) note_code(a, U.g, U.up.region(region_word(e)), code, tier);
}

// One y = 0 sample of climate step k in FP32 from the table itself (perlin_y0_f32's operations
// with the fixed-point coordinates: the fractions lie within u / 2 of the exact ones as there, so the
// bound above perlin_y0_f32 holds).
template <bool F32>
__device__ __forceinline__ float unit_sample_f32(const UnitSmem<F32> &S, int k, uint32_t dx, uint32_t dz) {
    const uint8_t *P = S.tab + (kUClim + k) * kUPitch;
    const uint64_t step = S.c.fstep[k];
    const uint64_t cx = fixed_at(S.fx[k], step, dx), cz = fixed_at(S.fz[k], step, dz);
    const float g = fixed_frac(cx), l = fixed_frac(cz);
    const F2 gl = f2(g, l);
    float g1, l1;
    f2_split(f2_add(gl, f2(-1.0f, -1.0f)), g1, l1);
    const float hyf = S.hyf[k], hy1 = __fsub_rn(hyf, 1.0f), fyf = S.fyf[k];
    const uint8_t *Pj = P + S.jy[k], *Pk = P + fixed_cell(cz);
    const uint32_t i = fixed_cell(cx);
    const uint32_t a = P[i], b = P[i + 1];
    const uint32_t c = Pj[a], d = Pj[a + 1], e = Pj[b], f = Pj[b + 1];
    auto grad = [&](uint32_t hash, float x, float y, float z) {
        const uint32_t h = hash & 15u;
        const float2 q = S.gf.xz[h];
        return __fmaf_rn(q.x, x, __fmaf_rn(S.gf.y[h], y, __fmul_rn(q.y, z)));
    };
    const F2 v00 = f2(grad(Pk[c], g, hyf, l), grad(Pk[c + 1], g, hyf, l1));
    const F2 v10 = f2(grad(Pk[e], g1, hyf, l), grad(Pk[e + 1], g1, hyf, l1));
    const F2 v01 = f2(grad(Pk[d], g, hy1, l), grad(Pk[d + 1], g, hy1, l1));
    const F2 v11 = f2(grad(Pk[f], g1, hy1, l), grad(Pk[f + 1], g1, hy1, l1));
    float fx, fz;
    f2_split(fade_f32x2(gl), fx, fz);
    const F2 x0 = lerp_f32x2(f2(fx, fx), v00, v10), x1 = lerp_f32x2(f2(fx, fx), v01, v11);
    float y0, y1;
    f2_split(lerp_f32x2(f2(fyf, fyf), x0, x1), y0, y1);
    return lerp_f32(fz, y0, y1);
}

// The same sample from the block's lattice columns (table k < 4): corner values A x + B z + C, then
// the x and z blends.  Bound, u = 2^-24: A, B, C within 1.5 u each (rounded weights, one rounded
// sum, magnitude <= 1); fractions, and those less 1, within u; two FMAs of values <= 2: corner 1.5 * 3 u + 2 u + 2 u = 8.5 u;
// x blend 8.5 u + 4 * 4 u + 2 u = 26.5 u; z blend 26.5 u + 4 * 4 u + 2 u = 44.5 u, under kPerlinF32ErrUlps.
__device__ __forceinline__ float lat_sample(const float4 *L, int nx, uint64_t cx, uint64_t cz) {
    const float g = fixed_frac(cx), l = fixed_frac(cz);
    const F2 gl = f2(g, l);
    float g1, l1;
    f2_split(f2_add(gl, f2(-1.0f, -1.0f)), g1, l1);
    const float4 *p = L + fixed_cell(cz) * (uint32_t)nx + fixed_cell(cx);
    const float4 q00 = p[0], q10 = p[1], q01 = p[nx], q11 = p[nx + 1];
    const float v00 = __fmaf_rn(q00.x, g, __fmaf_rn(q00.y, l, q00.z));
    const float v10 = __fmaf_rn(q10.x, g1, __fmaf_rn(q10.y, l, q10.z));
    const float v01 = __fmaf_rn(q01.x, g, __fmaf_rn(q01.y, l1, q01.z));
    const float v11 = __fmaf_rn(q11.x, g1, __fmaf_rn(q11.y, l1, q11.z));
    float fx, fz;
    f2_split(fade_f32x2(gl), fx, fz);
    float y0, y1;
    f2_split(lerp_f32x2(f2(fx, fx), f2(v00, v01), f2(v10, v11)), y0, y1);
    return lerp_f32(fz, y0, y1);
}

// The climate point of a survivor word, and step k's sample there in FP64 with the reference's
// operations.
__device__ __forceinline__ void unit_point(const UnitCtx &U, uint32_t e, double &xc, double &zc) {
    xc = ((U.ucx + (int)(e & 0xFFFFu)) * 16 + 8) * 0.25;   // exact: an integer over 4
    zc = ((U.ucz + (int)(e >> 16)) * 16 + 8) * 0.25;
}
template <bool F32>
__device__ __forceinline__ double unit_sample64(const UnitSmem<F32> &S, int k, double xc, double zc) {
    const ClimateSteps &st = S.c.steps;
    const ColTable<1> T{S.tab + (kUClim + k) * kUPitch, S.grad};
    const double sc = st.sc[k], lac = st.lac[k], hy = S.chy[k];
    return perlin_y0(T, S.cox[k], S.coz[k], S.jy[k], hy, fade(hy), keep_precision((xc * sc) * lac),
                     keep_precision((zc * sc) * lac));
}
// FP64 octave sum of erosion steps [0, k1] in the reference's order.
template <bool F32>
__device__ __noinline__ double unit_sum64(const UnitSmem<F32> &S, int k1, double xc, double zc) {
    const ClimateSteps &st = S.c.steps;
    double sum = 0.0;
    for (int k = 0; k <= k1; k++) sum += (st.c1[k] * unit_sample64(S, k, xc, zc)) * st.c2[k];
    return sum;
}
// FP64 DoublePerlin value of the temperature / ridge noise of steps k0 .. k0 + n - 1.
template <bool F32>
__device__ __noinline__ double unit_value64(const UnitSmem<F32> &S, int k0, int n, double xc, double zc) {
    const ClimateSteps &st = S.c.steps;
    double sum = 0.0, sum_a = 0.0;
    for (int k = k0; k < k0 + n; k++) {
        sum += (st.c1[k] * unit_sample64(S, k, xc, zc)) * st.c2[k];
        if (st.act[k] == ACT_END_SUB_A) {
            sum_a = sum;
            sum = 0.0;
        }
    }
    return (sum_a + sum) * st.amp[k0 + n - 1];
}

__device__ __forceinline__ bool temperature_bad(const BatchArgs &a, double t) {
    return a.mc_1_18_2 ? (t < -0.45) : (t > 0.2 || t < -0.45);
}
__device__ __forceinline__ bool ridge_bad(const BatchArgs &a, double rg) {
    return (rg > 0.42 && rg < 0.91) || (rg < -0.42 && rg > -0.91) || (!a.pre_26_2 && rg <= -0.91);
}

// What a warp carries through a unit.
struct WarpCounts {
    TierCounts tc;
    uint32_t temp = 0, ridge = 0, rechecks = 0;
};

// One erosion step over one round of 32 list entries: the sum after step k and whether the entry
// survives the step's tier.
template <bool F32, bool LAT>
__device__ __forceinline__ bool unit_step(UnitSmem<F32> &S, const BatchArgs &a, const UnitCtx &U, WarpCounts &W, int k,
                                          bool all_rechecks, uint32_t e, const LatBase *B, uint32_t ex, uint32_t ez,
                                          typename UnitSmem<F32>::Real prev, typename UnitSmem<F32>::Real &sum) {
    const ClimateSteps &st = S.c.steps;
    bool reject;
    if constexpr (F32) {
        float v;
        if constexpr (LAT) {
            const uint64_t step = S.c.fstep[k];
            v = lat_sample(S.lat.l1[k - 2], B->nx[k], fixed_at(B->x[k], step, ex), fixed_at(B->z[k], step, ez));
        } else {
            v = unit_sample_f32(S, k, e & 0xFFFFu, e >> 16);
        }
        sum = __fmaf_rn(st.cf[k], v, prev);
        if (!all_rechecks && sum < st.lo[k]) reject = true;
        else if (!all_rechecks && sum >= st.hi[k]) reject = false;
        else {   // inside the error band: the exact partial sum of steps 0..k
            W.rechecks++;
            double xc, zc;
            unit_point(U, e, xc, zc);
            reject = unit_sum64(S, k, xc, zc) * st.amp[k] < st.thr[k];
        }
    } else {
        double xc, zc;
        unit_point(U, e, xc, zc);
        sum = prev + (st.c1[k] * unit_sample64(S, k, xc, zc)) * st.c2[k];
        reject = sum * st.amp[k] < st.thr[k];
    }
    if (reject) {
        W.tc.add(st.tier[k]);
        unit_note(a, U, e, P1_EROSION, st.tier[k]);
    }
    return !reject;
}

// Erosion steps 4..7, temperature and ridge for n <= kList pooled regions (words, erosion sums); the
// survivors join the unit's list.  A region keeps its lane through the four steps: they pass 46 % of what
// comes in, so lists packed again after each step would take as many rounds for a warp's 64.
template <bool F32>
__device__ __forceinline__ void unit_drain(UnitSmem<F32> &S, const BatchArgs &a, const UnitCtx &U, WarpCounts &W,
                                           const uint32_t *words, const typename UnitSmem<F32>::Real *sums, uint32_t n,
                                           bool all_rechecks, int large) {
    using Real = typename UnitSmem<F32>::Real;
    const ClimateSteps &st = S.c.steps;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *const wl = S.wl[warp];
    const unsigned below = (1u << lane) - 1u;
    uint32_t n7 = 0;
    __syncwarp();
#pragma unroll 1
    for (uint32_t b = 0; b < n; b += 32) {
        const uint32_t q = b + (uint32_t)lane;
        bool keep = q < n;
        const uint32_t e = keep ? words[q] : 0u;
        Real sum = keep ? sums[q] : Real(0);
#pragma unroll 1
        for (int k = 4; k < 8; k++)
            if (keep) keep = unit_step<F32, false>(S, a, U, W, k, all_rechecks, e, nullptr, 0, 0, sum, sum);
        const unsigned m = __ballot_sync(0xFFFFFFFFu, keep);
        if (keep) wl[n7 + (uint32_t)__popc(m & below)] = e;
        n7 += (uint32_t)__popc(m);
    }
    __syncwarp();
    n = n7;
    // temperature: four lanes per region, summed in order by the first; then ridge with six
    constexpr int kT0 = 8, kR0 = 12;
    uint32_t nr = 0;
#pragma unroll 1
    for (uint32_t base = 0; base < n; base += 8) {
        const uint32_t i = base + (uint32_t)(lane >> 2);
        const int p = lane & 3;
        const bool have = i < n;
        const uint32_t e = have ? wl[i] : 0u;
        double xc, zc;
        unit_point(U, e, xc, zc);
        Real v = 0;
        if (have) {
            if constexpr (F32) v = unit_sample_f32(S, kT0 + p, e & 0xFFFFu, e >> 16);
            else v = unit_sample64(S, kT0 + p, xc, zc);
        }
        const Real vs[4] = {v, __shfl_down_sync(0xFFFFFFFFu, v, 1), __shfl_down_sync(0xFFFFFFFFu, v, 2),
                            __shfl_down_sync(0xFFFFFFFFu, v, 3)};
        bool keep = false;
        if (have && p == 0) {
            bool bad;
            if constexpr (F32) {
                float sum = 0.0f;
                for (int q = 0; q < 4; q++) sum = __fmaf_rn(st.cf[kT0 + q], vs[q], sum);
                const F32Bands &B = c_bands[large];
                if (all_rechecks || (sum >= B.t_lo[0] && sum < B.t_hi[0]) || (sum >= B.t_lo[1] && sum < B.t_hi[1])) {
                    W.rechecks++;
                    bad = temperature_bad(a, unit_value64(S, kT0, 4, xc, zc));
                } else {
                    bad = sum < B.t_lo[0] || (!a.mc_1_18_2 && sum >= B.t_hi[1]);
                }
            } else {
                double sum = 0.0, sum_a = 0.0;
                for (int q = 0; q < 4; q++) {
                    const int k = kT0 + q;
                    sum += (st.c1[k] * vs[q]) * st.c2[k];
                    if (st.act[k] == ACT_END_SUB_A) {
                        sum_a = sum;
                        sum = 0.0;
                    }
                }
                bad = temperature_bad(a, (sum_a + sum) * st.amp[kT0 + 3]);
            }
            if (bad) {
                W.temp++;
                unit_note(a, U, e, P1_TEMPERATURE, -1);
            } else {
                keep = true;
            }
        }
        const unsigned m = __ballot_sync(0xFFFFFFFFu, keep);
        __syncwarp();
        if (keep) wl[nr + (uint32_t)__popc(m & below)] = e;
        nr += (uint32_t)__popc(m);
    }
    __syncwarp();
#pragma unroll 1
    for (uint32_t base = 0; base < nr; base += 5) {
        const uint32_t i = base + (uint32_t)(lane / 6);
        const int p = lane % 6;
        const bool have = lane < 30 && i < nr;
        const uint32_t e = have ? wl[i] : 0u;
        double xc, zc;
        unit_point(U, e, xc, zc);
        Real v = 0;
        if (have) {
            if constexpr (F32) v = unit_sample_f32(S, kR0 + p, e & 0xFFFFu, e >> 16);
            else v = unit_sample64(S, kR0 + p, xc, zc);
        }
        const Real vs[6] = {v,
                            __shfl_down_sync(0xFFFFFFFFu, v, 1),
                            __shfl_down_sync(0xFFFFFFFFu, v, 2),
                            __shfl_down_sync(0xFFFFFFFFu, v, 3),
                            __shfl_down_sync(0xFFFFFFFFu, v, 4),
                            __shfl_down_sync(0xFFFFFFFFu, v, 5)};
        if (have && p == 0) {
            bool bad;
            if constexpr (F32) {
                float sum = 0.0f;
                for (int q = 0; q < 6; q++) sum = __fmaf_rn(st.cf[kR0 + q], vs[q], sum);
                const F32Bands &B = c_bands[large];
                bool inside = all_rechecks;
                for (int q = 0; q < 4; q++) inside |= sum >= B.r_lo[q] && sum < B.r_hi[q];
                if (inside) {
                    W.rechecks++;
                    bad = ridge_bad(a, unit_value64(S, kR0, 6, xc, zc));
                } else {
                    // above[q]: the ridge value lies above threshold q (-0.91, -0.42, 0.42, 0.91)
                    const bool a0 = sum >= B.r_hi[0], a1 = sum >= B.r_hi[1], a2 = sum >= B.r_hi[2],
                               a3 = sum >= B.r_hi[3];
                    bad = (a2 && !a3) || (!a1 && a0) || (!a.pre_26_2 && !a0);
                }
            } else {
                double sum = 0.0, sum_a = 0.0;
                for (int q = 0; q < 6; q++) {
                    const int k = kR0 + q;
                    sum += (st.c1[k] * vs[q]) * st.c2[k];
                    if (st.act[k] == ACT_END_SUB_A) {
                        sum_a = sum;
                        sum = 0.0;
                    }
                }
                bad = ridge_bad(a, (sum_a + sum) * st.amp[kR0 + 5]);
            }
            if (bad) {
                W.ridge++;
                unit_note(a, U, e, P1_RIDGE, -1);
            } else {
                S.surv[atomicAdd(&S.n_surv, 1u)] = e;   // room for a whole block (see the caller)
            }
        }
    }
    __syncwarp();
}

// Table t of the unit built by one thread in shared memory: the climate tables (step order) or cave
// table `slot`; the entries are stored twice and once more by unit_double_tables.
__device__ __forceinline__ Xr unit_table_rng(int large, bool climate, int idx, const Xr &fork) {
    const TableRng t = g_unit_tables[large].rng[climate ? idx : kSlotsA + idx];
    return octave_rng(t.name_lo, t.name_hi, t.oct_lo, t.oct_hi, fork, t.sub != 0);
}

// Identity in the first 256 bytes of n tables from table t0 (word by word, whole CTA).
__device__ __forceinline__ void unit_init_tables(uint8_t *tab, int t0, int n) {
    for (int q = threadIdx.x; q < n * 64; q += kUThreads) {
        const uint32_t w = (uint32_t)q & 63u;
        *reinterpret_cast<uint32_t *>(tab + (t0 + (q >> 6)) * kUPitch + 4 * w) = w * 0x04040404u + 0x03020100u;
    }
}
// Entries 256..511 = 0..255 and 512..515 = 0..3: a lookup at an unreduced sum of two bytes and one.
__device__ __forceinline__ void unit_double_tables(uint8_t *tab, int t0, int n) {
    for (int q = threadIdx.x; q < n * 64; q += kUThreads) {
        uint32_t *p = reinterpret_cast<uint32_t *>(tab + (t0 + (q >> 6)) * kUPitch);
        const uint32_t w = (uint32_t)q & 63u, v = p[w];
        p[64 + w] = v;
        if (w == 0) p[128] = v;
    }
}

// The entrance gate's cave tables as a sample source.
struct SrcUnit {
    const uint8_t *tab;
    const double *org;
    const uint32_t *gt;
    __device__ __forceinline__ double p3(int slot, double x, double y, double z) const {
        ColTable<1> T{tab + slot * kUPitch, gt};
        return perlin_3d(T, org[3 * slot], org[3 * slot + 1], org[3 * slot + 2], x, y, z);
    }
};

// dbl3d on the unit's tables, out of line: every cave noise goes through one copy of the sample.
__device__ __noinline__ double unit_dbl(const uint8_t *tab, const double *org, const uint32_t *gt, int noise, int base,
                                        double x, double y, double z) {
    return dbl3d(SrcUnit{tab, org, gt}, noise, base, x, y, z);
}
// Entrance at (x, y, z) through unit_dbl (caves.c's formula, as entrance() above).
template <bool F32>
__device__ __noinline__ double unit_entrance(const UnitSmem<F32> &S, int x, int y, int z) {
    auto dbl = [&](int noise, int base, double px, double py, double pz) {
        return unit_dbl(S.tab, S.org, S.grad, noise, base, px, py, pz);
    };
    const double ent = dbl(N_CAVE_ENTRANCE, kBaseEntrance, (double)x * 0.75, (double)y * 0.5, (double)z * 0.75);
    const double t = (10.0 + (double)y) / 40.0;
    const double cl = t < 0.0 ? 0.3 : (t > 1.0 ? 0.0 : lerp(t, 0.3, 0.0));
    const double cc = ent + 0.37 + cl;
    const double e = tunnel_scale(dbl(N_SPAGHETTI_RARITY, kBaseRarity, (double)(int)((uint32_t)x * 2u), (double)y,
                                      (double)(int)((uint32_t)z * 2u)));
    const double tv = dbl(N_SPAGHETTI_THICKNESS, kBaseThickness, (double)x, (double)y, (double)z);
    const double h = lerp((tv - -1.0) / (1.0 - -1.0), 0.065, 0.088);
    const double l = dbl(N_SPAGHETTI_1, kBaseSp1, (double)x / e, (double)y / e, (double)z / e);
    const double m = fabs(e * l) - h;
    const double n = dbl(N_SPAGHETTI_2, kBaseSp2, (double)x / e, (double)y / e, (double)z / e);
    const double o = fabs(e * n) - h;
    const double p = clampd(jmax(m, o), -1.0, 1.0);
    const double mod = dbl(N_ROUGHNESS_MODULATOR, kBaseRmod, (double)x, (double)y, (double)z);
    const double rgh = dbl(N_ROUGHNESS, kBaseRough, (double)x, (double)y, (double)z);
    const double q = (-0.05 + (-0.05 * mod)) * (-0.4 + fabs(rgh));
    return jmin(cc, p + q);
}
// A DoublePerlin of the first entrance test: the reference's, or where the caller chose FP32 cave samples
// (cave32) those summed in FP64 (within dp_err_f32 of the reference's value).
template <bool F32>
__device__ __noinline__ double unit_quick(const UnitSmem<F32> &S, bool cave32, int noise, int base, double x, double y,
                                          double z) {
    if (!F32 || !cave32) {
        return unit_dbl(S.tab, S.org, S.grad, noise, base, x, y, z);
    } else {
        const NoiseSpec &ns = c_noise[noise];
        const int np = ns.npresent;
        double v = 0.0;
#pragma unroll 1
        for (int q = 0; q < 2 * np; q++) {
            const int p = q < np ? q : q - np, slot = base + q;
            const double l = ns.lac[p];
            const double sx = q < np ? x : x * kDblScale, sy = q < np ? y : y * kDblScale, sz = q < np ? z : z * kDblScale;
            const ColTableF<1> T{S.tab + slot * kUPitch, &S.gf};
            const double *o = S.org + 3 * slot;
            v += ns.amp[p] * ns.per[p] * (double)perlin_3d_f32(T, o[0], o[1], o[2], keep_precision(sx * l),
                                                               keep_precision(sy * l), keep_precision(sz * l));
        }
        return v * ns.amplitude;
    }
}

// Entrance at 50 and 60 of one survivor by one warp, a sample a lane: the code that ends it, or -1.
// unit_entrance's operations; v holds 18 samples of each height.
template <bool F32>
__device__ __noinline__ int unit_entrance_warp(const UnitSmem<F32> &S, double *v, int hx, int hz) {
    const SrcUnit src{S.tab, S.org, S.grad};
    const int lane = threadIdx.x & 31, h = lane & 1, y = h ? 60 : 50;
    double *const vh = v + h * kSlotsB;
    auto sample = [&](int slot, double e) {
        const int noise = c_slot_c[0][slot][0], sub = c_slot_c[0][slot][1], p = c_slot_c[0][slot][2];
        double px, py, pz;
        cave_point(noise, hx, y, hz, e, px, py, pz);
        vh[slot] = slot_sample_call(src, slot, sub, c_noise[noise].lac[p], px, py, pz);
    };
    if (lane < 28) sample(lane < 20 ? lane >> 1 : (lane >> 1) + 4, 1.0);   // all but spaghetti_3d_1 and _2
    __syncwarp();
    const double e = tunnel_scale(combine_vals(N_SPAGHETTI_RARITY, vh + kBaseRarity, 1));
    if (lane < 8) sample(kBaseSp1 + (lane >> 1), e);
    __syncwarp();
    const double t = (10.0 + (double)y) / 40.0;
    const double cl = t < 0.0 ? 0.3 : (t > 1.0 ? 0.0 : lerp(t, 0.3, 0.0));
    const double cc = combine_vals(N_CAVE_ENTRANCE, vh + kBaseEntrance, 1) + 0.37 + cl;
    const double tv = combine_vals(N_SPAGHETTI_THICKNESS, vh + kBaseThickness, 1);
    const double w = lerp((tv - -1.0) / (1.0 - -1.0), 0.065, 0.088);
    const double m = fabs(e * combine_vals(N_SPAGHETTI_1, vh + kBaseSp1, 1)) - w;
    const double o = fabs(e * combine_vals(N_SPAGHETTI_2, vh + kBaseSp2, 1)) - w;
    const double p = clampd(jmax(m, o), -1.0, 1.0);
    const double mod = combine_vals(N_ROUGHNESS_MODULATOR, vh + kBaseRmod, 1);
    const double rgh = combine_vals(N_ROUGHNESS, vh + kBaseRough, 1);
    const double q = (-0.05 + (-0.05 * mod)) * (-0.4 + fabs(rgh));
    const bool out = jmin(cc, p + q) >= 0;
    const unsigned b = __ballot_sync(0xFFFFFFFFu, out);   // the barrier also frees v
    return (b & 1u) ? P1_ENTRANCE_50 : ((b & 2u) ? P1_ENTRANCE_60 : -1);
}

// One CTA per unit.  F32: the FP32 noise core with the block lattices (small coordinates only), else
// FP64 samples throughout, in the reference's order.
template <bool F32>
__global__ void __launch_bounds__(kUThreads, 3) unit_kernel(const __grid_constant__ BatchArgs a) {
    using Real = typename UnitSmem<F32>::Real;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    UnitSmem<F32> &S = *reinterpret_cast<UnitSmem<F32> *>(smem_raw);
    if (blockIdx.x >= batch_units(a)) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned below = (1u << lane) - 1u;
    const int large = a.large_biomes ? 1 : 0;
    const bool all_rechecks = F32 && a.fp32_core == 2;
    const bool cave32 = F32 && a.fp32_core >= 2;   // FP32 cave samples: WG_NOISE_FP32_CAVES and the check mode
    UnitCtx U;
    U.up = unit_pos(a, blockIdx.x);
    U.g = U.up.g;
    U.seed = seed_value(a, U.g);
    U.ucx = U.up.rx * 32;
    U.ucz = U.up.rz * 32;

    if (tid < P1_KINDS + kTiers) S.hist[tid] = 0;
    if (tid == 0) S.n_pool = S.n_surv = S.n_und = S.n_deep = S.n_total = 0;
    for (int q = kUThreads - 1 - tid; q < (int)(sizeof(UnitConst) / 16); q += kUThreads)   // warps that build nothing
        reinterpret_cast<uint4 *>(&S.c)[q] = reinterpret_cast<const uint4 *>(&g_unit_tables[large].c)[q];
    fill_grad_table(S.grad, tid);
    fill_grad_table_f32(&S.gf, tid);
    // warp 0 builds the climate tables, warp 1 the entrance gate's: one table's 256 dependent steps
    // take about 10 us whatever is beside them
    const bool clim = warp == 0, builds = warp < 2 && lane < kSlotsA;
    Xr r{};
    if (builds) r = unit_table_rng(large, clim, lane, seed_fork_of(U.seed));
    unit_init_tables(S.tab, 0, kSlotsB + kSlotsA);
    __syncthreads();
    if (builds) {
        const int t = clim ? kUClim + lane : lane;
        double ox, oy, oz;
        perlin_shuffle<1>(S.tab + t * kUPitch, r, ox, oy, oz);
        if (clim) {
            const int jy = (int)floor(oy);
            const double hy = oy - jy, fy = fade(hy);
            S.cox[lane] = ox;
            S.coz[lane] = oz;
            S.chy[lane] = hy;
            S.jy[lane] = jy;
            if constexpr (F32) {
                S.hyf[lane] = __double2float_rn(hy);
                S.fyf[lane] = __double2float_rn(fy);
                const double sc = S.c.steps.sc[lane], lac = S.c.steps.lac[lane];
                const double xc = (U.ucx * 16 + 8) * 0.25, zc = (U.ucz * 16 + 8) * 0.25;
                S.fx[lane] = to_fixed(keep_precision((xc * sc) * lac) + ox);
                S.fz[lane] = to_fixed(keep_precision((zc * sc) * lac) + oz);
                if (lane < kLatTables) {
                    S.w0[lane] = __double2float_rn(1.0 - fy);
                    S.w1[lane] = __double2float_rn(fy);
                    S.c0[lane] = __double2float_rn((1.0 - fy) * hy);
                    S.c1[lane] = __double2float_rn(fy * (hy - 1.0));
                }
            }
        } else {
            S.org[3 * lane] = ox;
            S.org[3 * lane + 1] = oy;
            S.org[3 * lane + 2] = oz;
        }
    }
    __syncthreads();
    const uint32_t side_x = block_side(U.up.th), side_z = block_side(U.up.tw);
    const uint32_t nbx = (U.up.tw + side_x - 1) / side_x, nbz = (U.up.th + side_z - 1) / side_z;
    const uint32_t bw = (U.up.tw + nbx - 1) / nbx, bh = (U.up.th + nbz - 1) / nbz;
    const uint32_t n_blocks = nbx * nbz;
    auto lattice_base = [&](uint32_t blk) {   // one thread per table and axis, a block ahead of its use
        if constexpr (F32) {
            if (tid >= 2 * kLatTables || blk >= n_blocks) return;
            LatBase &B = S.lat_base[blk & 1u];
            const int k = tid >> 1;
            const bool z = tid & 1;
            const uint32_t at = z ? (blk / nbx) * bh : (blk % nbx) * bw;   // first region of the block, in the unit
            const uint32_t side = z ? min(bh, U.up.th - at) : min(bw, U.up.tw - at);
            const uint64_t step = S.c.fstep[k];
            const uint64_t b = (z ? S.fz[k] : S.fx[k]) + (uint64_t)(at * 32u) * step;
            const uint64_t b0 = b & 0x00FFFFFFFFFFFFFFull;
            const int cols = (int)fixed_cell(fixed_at(b0, step, (side - 1) * 32u + 23u)) + 2;
            (z ? B.z : B.x)[k] = b0;
            (z ? B.cell_z : B.cell_x)[k] = (int)(b >> 56);
            (z ? B.nz : B.nx)[k] = cols;
            if (!z) B.inv[k] = ((1u << 20) + (uint32_t)cols - 1) / (uint32_t)cols;
        }
    };
    lattice_base(0);
    unit_double_tables(S.tab, 0, kSlotsB + kSlotsA);
    __syncthreads();

    const ClimateSteps &st = S.c.steps;
    WarpCounts W;
    for (uint32_t blk = 0; blk < n_blocks; blk++) {
        const uint32_t x0 = (blk % nbx) * bw, z0 = (blk / nbx) * bh;   // first region of the block, in the unit
        const uint32_t w = min(bw, U.up.tw - x0), h = min(bh, U.up.th - z0), n = w * h;
        const LatBase *Bp = nullptr;
        if constexpr (F32) {
            // ---- the block's lattice columns ----
            const LatBase &B = *(Bp = &S.lat_base[blk & 1u]);
            lattice_base(blk + 1);   // into the other half, which no thread reads before the next block
            const int m0 = B.nx[0] * B.nz[0], m1 = m0 + B.nx[1] * B.nz[1], m2 = m1 + B.nx[2] * B.nz[2],
                      m3 = m2 + B.nx[3] * B.nz[3];
            for (int q = tid; q < m3; q += kUThreads) {
                const int k = (q >= m0) + (q >= m1) + (q >= m2);
                const int r = q - (k == 0 ? 0 : k == 1 ? m0 : k == 2 ? m1 : m2);
                const int iz = (int)(((uint32_t)r * B.inv[k]) >> 20), ix = r - iz * B.nx[k];   // r < 361, nx <= 120
                const uint8_t *P = S.tab + (kUClim + k) * kUPitch;
                const uint8_t *Pj = P + S.jy[k], *Pk = P + ((B.cell_z[k] + iz) & 255);
                const uint32_t pa = P[(B.cell_x[k] + ix) & 255];
                const uint32_t h0 = Pk[Pj[pa]] & 15u, h1 = Pk[Pj[pa + 1]] & 15u;
                const float2 g0 = S.gf.xz[h0], g1 = S.gf.xz[h1];
                float4 c;
                c.x = __fmaf_rn(S.w1[k], g1.x, __fmul_rn(S.w0[k], g0.x));
                c.y = __fmaf_rn(S.w1[k], g1.y, __fmul_rn(S.w0[k], g0.y));
                c.z = __fmaf_rn(S.c1[k], S.gf.y[h1], __fmul_rn(S.c0[k], S.gf.y[h0]));
                c.w = 0.0f;
                (k < 2 ? S.lat.l0[k] : S.lat.l1[k - 2])[r] = c;
            }
        }
        // Both cores: the lattice is complete, and every thread has read the last block's pool count (below)
        // before a warp of this block adds to it.
        __syncthreads();
        // ---- tier 0: this warp's regions of the block, 32 at a time ----
        const uint32_t inv = ((1u << 20) + w - 1) / w;   // q / w = (q * inv) >> 20 for q < 1,024, w <= 149
        const uint64_t lcg0 = hut_lcg(U.seed, U.up.rx + (int)x0, U.up.rz + (int)z0, a.salt);
        uint32_t n1 = 0;
#pragma unroll 1
        for (uint32_t b = (uint32_t)warp * 32u; b < n; b += kUThreads) {
            const uint32_t q = b + (uint32_t)lane;
            const bool valid = q < n;
            uint32_t e = 0;
            Real sum = 0;
            bool pass = false;
            if (valid) {
                const uint32_t qz = (q * inv) >> 20, qx = q - qz * w;
                int j, k;
                hut_draws(lcg0 + qx * kHutX + qz * kHutZ, j, k);
                const uint32_t ex = qx * 32u + (uint32_t)j, ez = qz * 32u + (uint32_t)k;   // chunks from the block's first
                e = (x0 * 32u + ex) | ((z0 * 32u + ez) << 16);
                bool in_band = true;
                if constexpr (F32) {
                    const LatBase &B = *Bp;
                    const uint64_t s0 = S.c.fstep[0], s1 = S.c.fstep[1];
                    sum = __fmul_rn(st.cf[0],
                                    lat_sample(S.lat.l0[0], B.nx[0], fixed_at(B.x[0], s0, ex), fixed_at(B.z[0], s0, ez)));
                    sum = __fmaf_rn(st.cf[1],
                                    lat_sample(S.lat.l0[1], B.nx[1], fixed_at(B.x[1], s1, ex), fixed_at(B.z[1], s1, ez)),
                                    sum);
                    pass = sum >= st.hi[1];
                    in_band = all_rechecks || (!pass && !(sum < st.lo[1]));
                }
                if (in_band) {
                    double xc, zc;
                    unit_point(U, e, xc, zc);
                    const double s64 = unit_sum64(S, 1, xc, zc);
                    if constexpr (F32) W.rechecks++;
                    else sum = s64;
                    pass = !(s64 * st.amp[1] < st.thr[1]);
                }
                if (!pass) {
                    W.tc.add(st.tier[1]);
                    unit_note(a, U, e, P1_EROSION, st.tier[1]);
                }
            }
            const unsigned m = __ballot_sync(0xFFFFFFFFu, pass);
            if (pass) {
                const uint32_t at = n1 + (uint32_t)__popc(m & below);
                S.wl[warp][at] = e;
                S.ws[warp][at] = sum;
            }
            n1 += (uint32_t)__popc(m);
        }
        __syncwarp();
        // ---- erosion steps 2 and 3; their survivors join the pool ----
#pragma unroll 1
        for (int k = 2; k < 4; k++) {
            uint32_t nn = 0;
#pragma unroll 1
            for (uint32_t b = 0; b < n1; b += 32) {
                const uint32_t q = b + (uint32_t)lane;
                bool keep = false;
                uint32_t e = 0;
                Real sum = 0;
                if (q < n1) {
                    e = S.wl[warp][q];
                    keep = unit_step<F32, F32>(S, a, U, W, k, all_rechecks, e, Bp, (e & 0xFFFFu) - x0 * 32u,
                                               (e >> 16) - z0 * 32u, S.ws[warp][q], sum);
                }
                const unsigned m = __ballot_sync(0xFFFFFFFFu, keep);
                uint32_t at = nn + (uint32_t)__popc(m & below);
                if (k == 3) {
                    uint32_t base = 0;
                    if (lane == 0 && m) base = atomicAdd(&S.n_pool, (uint32_t)__popc(m));
                    at = __shfl_sync(0xFFFFFFFFu, base, 0) + (uint32_t)__popc(m & below);
                }
                __syncwarp();
                if (keep) {
                    (k == 3 ? S.pool : S.wl[warp])[at] = e;
                    (k == 3 ? S.pool_s : S.ws[warp])[at] = sum;
                }
                nn += (uint32_t)__popc(m);
            }
            __syncwarp();
            n1 = nn;
        }
        __syncthreads();   // the block's lattice and the pool are settled
        const bool last_blk = blk + 1 == n_blocks;
        // nothing to drain yet: the pool and the lists change again only past the barrier at the head of the next
        // block's tier 0, which both cores have
        if (!last_blk && S.n_pool < kPoolFull) continue;
        for (;;) {
            // ---- the rest of the climate gates for the pool, every warp an equal share of it, so
            // that none waits for another's ----
            const uint32_t np = S.n_pool;
            const bool drain = np >= kPoolFull || (last_blk && np > 0);
            const uint32_t take = drain ? min(np, (uint32_t)(kUWarps * kList)) : 0u;
            __syncthreads();   // every thread has read the count
            if (drain) {
                const uint32_t share = (take + kUWarps * 32 - 1) / (kUWarps * 32) * 32;
                const uint32_t from = min(take, (uint32_t)warp * share), cnt = min(take - from, share);
                if (tid == 0) S.n_pool = np - take;
                unit_drain<F32>(S, a, U, W, S.pool + (np - take + from), S.pool_s + (np - take + from), cnt, all_rechecks,
                                large);
                __syncthreads();
            }
            const bool last = last_blk && np == take;   // no more climate survivors will come
            // ---- entrance gate.  First test, one survivor per thread: at y = 50 the entrance noise
            // and the two scaled spaghetti noises settle 70 % of the survivors (both terms of the
            // minimum >= 0); the rest take the whole formula at 50 and 60.  Full rounds only. ----
            auto settle = [&](uint32_t e, int code) {   // ended by the entrance gate, or a candidate (-1)
                if (code >= 0) {
                    atomicAdd(&S.hist[code], 1u);
                    unit_note(a, U, e, code, -1);
                    return;
                }
                const uint32_t q = atomicAdd(&S.n_deep, 1u);
                if (q < kUDeep) {
                    S.deep[q] = e;
                    return;
                }
                const uint32_t di = atomicAdd(&a.counters[CNT_DEEP], 1u);
                if (di < a.cap_deep) {
                    a.deep[2 * di] = blockIdx.x;
                    a.deep[2 * di + 1] = region_word(e);
                } else {
                    atomicOr(&a.counters[CNT_OVERFLOW], 2u);
                }
            };
            for (;;) {
                const uint32_t ns = S.n_surv, nu = S.n_und;
                if (last && ns + nu <= kWide) {   // the unit's last few: a warp each
                    for (uint32_t q = (uint32_t)warp; q < ns + nu; q += kUWarps) {
                        const uint32_t e = q < ns ? S.surv[q] : S.und[q - ns];
                        const int code = unit_entrance_warp(S, S.mh[warp], (U.ucx + (int)(e & 0xFFFFu)) * 16 + 3,
                                                            (U.ucz + (int)(e >> 16)) * 16 + 3);
                        if (lane == 0) {
                            W.rechecks += all_rechecks;
                            settle(e, code);
                        }
                    }
                    __syncthreads();
                    if (tid == 0) {
                        S.n_total += ns;
                        S.n_surv = S.n_und = 0;
                    }
                    break;
                }
                const bool second = nu >= kUThreads || (last && ns == 0 && nu > 0);
                const bool first = !second && (ns >= kUThreads || (last && ns > 0));
                __syncthreads();   // every thread has read the counts
                if (!first && !second) break;
                const uint32_t cnt = first ? ns : nu, tk = min(cnt, (uint32_t)kUThreads);
                const bool have = (uint32_t)tid < tk;
                const uint32_t e = have ? (first ? S.surv : S.und)[cnt - tk + tid] : 0u;
                if (tid == 0) {
                    (first ? S.n_surv : S.n_und) = cnt - tk;
                    if (first) S.n_total += tk;
                }
                __syncthreads();
                if (have) {
                    const int hx = (U.ucx + (int)(e & 0xFFFFu)) * 16 + 3, hz = (U.ucz + (int)(e >> 16)) * 16 + 3;
                    if (first) {
                        int code = -1;
                        const double rar = unit_quick(S, cave32, N_SPAGHETTI_RARITY, kBaseRarity, (double)(int)((uint32_t)hx * 2u),
                                                      50.0, (double)(int)((uint32_t)hz * 2u));
                        const double er = cave32 ? S.c.err[0] : 0.0, sc = tunnel_scale(rar);
                        const double px = (double)hx / sc, py = 50.0 / sc, pz = (double)hz / sc;
                        const double l = unit_quick(S, cave32, N_SPAGHETTI_1, kBaseSp1, px, py, pz);
                        const double m = unit_quick(S, cave32, N_SPAGHETTI_2, kBaseSp2, px, py, pz);
                        const double sure = kSpagSure + (cave32 ? 2.0 * fmax(S.c.err[1], S.c.err[2]) : 0.0);
                        const bool edge = er > 0.0 && (fabs(rar + 0.5) <= er || fabs(rar) <= er || fabs(rar - 0.5) <= er);
                        if (!edge && fmax(fabs(sc * l), fabs(sc * m)) >= sure) {
                            // spaghetti(50) >= 0: the entrance term decides (its depth term is 0 at 50)
                            const double ent = unit_quick(S, cave32, N_CAVE_ENTRANCE, kBaseEntrance, (double)hx * 0.75, 25.0,
                                                          (double)hz * 0.75);
                            if (ent + 0.37 >= (cave32 ? S.c.err[3] : 0.0)) code = P1_ENTRANCE_50;
                        }
                        if (all_rechecks) code = -1;   // the check mode: the whole formula in FP64 for every survivor
                        if (code < 0) S.und[atomicAdd(&S.n_und, 1u)] = e;
                        else settle(e, code);
                    } else {
                        W.rechecks += all_rechecks;
                        settle(e, unit_entrance(S, hx, 50, hz) >= 0   ? P1_ENTRANCE_50
                                  : unit_entrance(S, hx, 60, hz) >= 0 ? P1_ENTRANCE_60
                                                                      : -1);
                    }
                }
                __syncthreads();
            }
            if (!drain || last || (!last_blk && np - take < kPoolFull)) break;
        }
    }

    // ---- the funnel of the climate stage ----
    {
        uint32_t total = 0;
        for (int t = 0; t < kTiers; t++) {
            const uint32_t v = __reduce_add_sync(0xFFFFFFFFu, W.tc.get(t));
            total += v;
            if (lane == 0 && v) atomicAdd(&S.hist[P1_KINDS + t], v);
        }
        const uint32_t nt = __reduce_add_sync(0xFFFFFFFFu, W.temp), nr = __reduce_add_sync(0xFFFFFFFFu, W.ridge),
                       nk = __reduce_add_sync(0xFFFFFFFFu, W.rechecks);
        if (lane == 0) {
            if (total) atomicAdd(&S.hist[P1_EROSION], total);
            if (nt) atomicAdd(&S.hist[P1_TEMPERATURE], nt);
            if (nr) atomicAdd(&S.hist[P1_RIDGE], nr);
            if (nk) atomicAdd(&a.counters[CNT_RECHECK], nk);
        }
    }
    if (tid == 0 && S.n_total) {
        atomicAdd(&a.counters[CNT_SURVIVORS], S.n_total);
        atomicAdd(&a.counters[CNT_RECORDS], 1u);
    }

    // ---- the ladder for the unit's deep candidates: the other 36 cave tables, over the climate ones ----
    const uint32_t n_deep = min(S.n_deep, (uint32_t)kUDeep);
    __syncthreads();
    if (n_deep) {
        unit_init_tables(S.tab, kSlotsB, kSlotsC - kSlotsB);
        __syncthreads();
        constexpr int kHalf = (kSlotsC - kSlotsB) / 2;
        if (warp < 2 && lane < kHalf) {
            const int t = kSlotsB + warp * kHalf + lane;
            Xr r = unit_table_rng(large, false, t, seed_fork_of(U.seed));
            double ox, oy, oz;
            perlin_shuffle<1>(S.tab + t * kUPitch, r, ox, oy, oz);
            S.org[3 * t] = ox;
            S.org[3 * t + 1] = oy;
            S.org[3 * t + 2] = oz;
        }
        __syncthreads();
        if (tid == 0) atomicAdd(&a.counters[CNT_DEEP_UNIT], n_deep);
        const SrcUnit src{S.tab, S.org, S.grad};
        for (uint32_t q = (uint32_t)warp; q < n_deep; q += kUWarps) {   // S.und is empty here
            const uint32_t e = S.deep[q];
            const bool cave = cave_at_max_height(src, S.mh[warp], (U.ucx + (int)(e & 0xFFFFu)) * 16 + 3,
                                           (U.ucz + (int)(e >> 16)) * 16 + 3, U.up.max_height, large);
            if (lane == 0) {
                if (cave) {
                    atomicAdd(&S.hist[P1_CAVE_AT_MAXH], 1u);
                    unit_note(a, U, e, P1_CAVE_AT_MAXH, -1);
                } else {
                    S.und[atomicAdd(&S.n_und, 1u)] = e;
                }
            }
        }
        __syncthreads();
        const uint32_t n_open = S.n_und;
        for (uint32_t q = 0; q < n_open; q++) {   // past it: the whole ladder, all threads on one candidate
            const uint32_t e = S.und[q];
            const uint32_t rw = region_word(e);
            ladder_candidate<kUThreads>(a, S.lad, src, U.seed, U.g, U.up.region(rw), U.up.rx + (int)(rw & 0xFFFFu),
                                        U.up.rz + (int)(rw >> 16), U.ucx + (int)(e & 0xFFFFu), U.ucz + (int)(e >> 16),
                                        U.up.max_height);
        }
    }
    if (tid < P1_KINDS + kTiers && S.hist[tid]) atomicAdd(&a.hist[tid], (unsigned long long)S.hist[tid]);
}

static unsigned long long g_smem_done_u32 = 0, g_smem_done_u64 = 0;

static void prepare_unit_launches() {
    allow_dynamic_smem(unit_kernel<true>, sizeof(UnitSmem<true>), g_smem_done_u32);
    allow_dynamic_smem(unit_kernel<false>, sizeof(UnitSmem<false>), g_smem_done_u64);
}

int unit_ctas_per_sm(bool f32) {
    prepare_unit_launches();
    int n = 0;
    if (f32) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, unit_kernel<true>, kUThreads, sizeof(UnitSmem<true>));
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, unit_kernel<false>, kUThreads, sizeof(UnitSmem<false>));
    return n < 1 ? 1 : n;
}

void launch_unit(const BatchArgs &a, cudaStream_t s) {
    prepare_unit_launches();
    if (a.fp32_core && a.small_coords) unit_kernel<true><<<a.n_units, kUThreads, sizeof(UnitSmem<true>), s>>>(a);
    else unit_kernel<false><<<a.n_units, kUThreads, sizeof(UnitSmem<false>), s>>>(a);
}
