// The list kernels: phase 1 of many units of few regions each (2^24 seeds x 9 x 9 regions), breadth
// first over lists in HBM.  Included by wg_phase1.cu.
//
// What bounds this work is building Perlin tables (256 dependent shuffle steps, about 26 warp
// instructions and 8 shared-memory wavefronts each), so the stages are cut where a seed drops out and
// each builds only its own tables, 32 at a time:
//
//   erosion      every unit                 8 tables, 4 units per warp
//   temperature  75 % of 9 x 9 units        4 tables, 8 units per warp
//   ridge        58 %                       6 tables, 5 units per warp
//   scaled caves 53 %                       6 tables (rarity, spaghetti_3d_1 and _2), 5 units per warp
//   entrance     nearly the same            6 tables, 5 units per warp
//   rough caves  half of those              6 tables (thickness, roughness and its modulator), 5 per warp
//
// and what the last three leave open (3 % of the climate survivors) goes to the entrance kernel,
// which decides at 50 and 60.  The cave stages sample in FP64, as the entrance kernel does (in FP32, as
// WG_NOISE_FP32_CAVES would have it, 2^24 seeds x 9 x 9 took 0.6 % less).  A warp owns its 32 tables (one byte column per lane, 32-byte
// rows) and waits for no other warp, so the warps of an SM drift apart and one's build fills the issue
// slots another's sampling leaves free.  Measured on 2^24 seeds x 9 x 9: these six kernels 175 ms and the
// entrance kernel's rest 6; the fused climate kernel 160 and the entrance kernel 74.
//
// Tier 0 takes its samples from lattice columns as the unit kernel does (wg_unit.cuh): a 9 x 9 block
// spans 2.2 cells of octave 1/512, so 25 columns per table replace 81 three-dimensional samples.
#pragma once

constexpr int kLWarps = 4, kLThreads = 32 * kLWarps;
constexpr int kRows = 257;                  // row 256 = row 0 (ColTableF)
constexpr int kLBlock = 9;                  // regions per side of a tier-0 block
constexpr int kLLat = 5;                    // its lattice columns per axis (2.2 cells)
constexpr int kLUnits = 4;                  // units of a warp in the erosion kernel
constexpr int kEWarps = 4, kEThreads = 32 * kEWarps;   // erosion CTAs: four on an SM, 16 warps at 128 registers
constexpr int kLList = 224;                 // tier-0 survivors a warp carries (a 9 x 9 group has 139 on average)

// Regions along one side of a tier-0 block of a tile `other` regions wide across it: kLBlock, or in a thin
// tile as many as the lattice's columns hold (23 for one region; 9 of them left 23 lanes idle).
__host__ __device__ constexpr uint32_t list_side(uint32_t other) {
    if (other >= (uint32_t)kLBlock) return kLBlock;
    const uint32_t s = lattice_side(kLLat * kLLat, other, 255);
    return s > (uint32_t)kLBlock ? s : kLBlock;
}

// unit_pos out of line: its divisions and table search would fill the instruction cache.
__device__ __noinline__ UnitPos unit_pos_call(const BatchArgs &a, uint32_t u) { return unit_pos(a, u); }

// Byte columns of a warp: initialised and shuffled by their lanes.
__device__ __forceinline__ void warp_build(uint8_t *tab, int lane, bool valid, Xr r, double &ox, double &oy, double &oz) {
    __syncwarp();   // the warp's last samples are taken
    uint4 *w = reinterpret_cast<uint4 *>(tab);
#pragma unroll 4
    for (int q = 0; q < 16; q++) {   // two 16-byte stores make a row
        const uint32_t v = (uint32_t)(q * 16 + (lane >> 1)) * 0x01010101u;
        w[q * 32 + lane] = make_uint4(v, v, v, v);
    }
    __syncwarp();
    if (valid) {
        perlin_shuffle<32>(tab + lane, r, ox, oy, oz);
        tab[256 * 32 + lane] = tab[lane];
    }
    __syncwarp();
}

// A climate table's constants, one per column.
struct ClimCols {
    uint64_t fx[32], fz[32];
    float hyf[32], fyf[32];
    int jy[32];
};
__device__ __forceinline__ void clim_col(ClimCols &C, int col, const ClimateStep &st, int ucx, int ucz, double ox,
                                         double oy, double oz) {
    const int jy = (int)floor(oy);
    const double hy = oy - jy;
    const double xc = (ucx * 16 + 8) * 0.25, zc = (ucz * 16 + 8) * 0.25;
    C.fx[col] = to_fixed((xc * st.sc) * st.lac + ox);
    C.fz[col] = to_fixed((zc * st.sc) * st.lac + oz);
    C.hyf[col] = __double2float_rn(hy);
    C.fyf[col] = __double2float_rn(fade(hy));
    C.jy[col] = jy;
}
// One y = 0 sample of a column at chunk offset (dx, dz) from its unit's first chunk.
__device__ __forceinline__ float col_sample(const uint8_t *tab, const ClimCols &C, const GradF &gf, int col, uint64_t step,
                                            uint32_t dx, uint32_t dz) {
    const uint64_t cx = fixed_at(C.fx[col], step, dx), cz = fixed_at(C.fz[col], step, dz);
    const ColTableF<32> T{tab + col, &gf};
    return perlin_y0_cell_f32(T, (int)fixed_cell(cx), C.jy[col], (int)fixed_cell(cz), fixed_frac(cx), fixed_frac(cz),
                              C.hyf[col], C.fyf[col]);
}

// The FP64 sample of climate step k of `seed`, for the decisions an FP32 sum leaves open: the origins
// are drawn again (they are not kept), the table is the column.
__device__ __noinline__ double col_sample64(const uint8_t *tab, int col, const uint32_t *gt, int large, int k, uint64_t seed, double xc,
                               double zc) {
    const ClimateStep &st = c_steps[large][k];
    const int8_t *s = c_slot_a[large][st.slot];
    Xr r = octave_rng(c_noise[s[0]], seed_fork_of(seed), s[1], s[2]);
    const double ox = xr_double(r) * 256.0, oy = xr_double(r) * 256.0, oz = xr_double(r) * 256.0;
    const int jy = (int)floor(oy);
    const double hy = oy - jy;
    const ColTable<32> T{tab + col, gt};
    return perlin_y0(T, ox, oz, jy, hy, fade(hy), keep_precision((xc * st.sc) * st.lac),
                     keep_precision((zc * st.sc) * st.lac));
}
// Octave sum of erosion steps [0, k1], columns col .. col + k1.
__device__ __forceinline__ double col_sum64(const uint8_t *tab, int col, const uint32_t *gt, int large, int k1, uint64_t seed,
                                         double xc, double zc) {
    double sum = 0.0;
    for (int k = 0; k <= k1; k++) {
        const ClimateStep &st = c_steps[large][k];
        sum += (st.c1 * col_sample64(tab, col + k, gt, large, k, seed, xc, zc)) * st.c2;
    }
    return sum;
}
// An erosion decision inside the FP32 sum's error band, or a verdict to note, for a list entry
// (unit << 30 | chunk offset z << 15 | x) of a warp whose first unit is u0: the rare paths, out of line.
__device__ __noinline__ bool erosion_recheck(const BatchArgs &a, const uint8_t *tab, const uint32_t *gt, int large, int k,
                                             uint32_t u0, uint32_t e) {
    const UnitPos p = unit_pos_call(a, u0 + (e >> 30));
    const double xc = ((p.rx * 32 + (int)(e & 0x7FFFu)) * 16 + 8) * 0.25;
    const double zc = ((p.rz * 32 + (int)((e >> 15) & 0x7FFFu)) * 16 + 8) * 0.25;
    const ClimateStep &st = c_steps[large][k];
    return !(col_sum64(tab, (int)(e >> 30) * 8, gt, large, k, seed_value(a, p.g), xc, zc) * st.amp < st.thr);
}
__device__ __forceinline__ uint32_t entry_word(uint32_t e) { return ((e & 0x7FFFu) >> 5) | (((e >> 15) & 0x7FFFu) >> 5) << 16; }
__device__ __noinline__ void erosion_note(const BatchArgs &a, uint32_t u0, uint32_t e, int tier) {
    const UnitPos p = unit_pos_call(a, u0 + (e >> 30));
    note_code(a, p.g, p.region(entry_word(e)), P1_EROSION, tier);
}
// DoublePerlin of steps k0 .. k0 + n - 1, columns col ...
__device__ __noinline__ double col_value64(const uint8_t *tab, int col, const uint32_t *gt, int large, int k0, int n,
                                           uint64_t seed, double xc, double zc) {
    double sum = 0.0, sum_a = 0.0;
    for (int p = 0; p < n; p++) {
        const ClimateStep &st = c_steps[large][k0 + p];
        sum += (st.c1 * col_sample64(tab, col + p, gt, large, k0 + p, seed, xc, zc)) * st.c2;
        if (st.act == ACT_END_SUB_A) {
            sum_a = sum;
            sum = 0.0;
        }
    }
    return (sum_a + sum) * c_steps[large][k0 + n - 1].amp;
}

// Appends n <= 32 regions (one per lane, of ascending record ids) to a list as records, one per run of
// equal ids.  On a full list only the overflow flag is set; every later kernel of the batch then ends.
__device__ __forceinline__ void list_emit(const BatchArgs &a, const RegionList &L, int lane, uint32_t n, uint32_t id,
                                          uint32_t unit, uint32_t word, double pay) {
    if (!n) return;
    const unsigned below = (1u << lane) - 1u;
    const uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, id, 1);
    const bool in = (uint32_t)lane < n, head = in && (lane == 0 || id != prev);
    const unsigned hm = __ballot_sync(0xFFFFFFFFu, head);
    const uint32_t nrec = (uint32_t)__popc(hm);
    uint32_t ri = 0, off = 0;
    if (lane == 0) {
        ri = atomicAdd(&a.counters[L.cnt], nrec);
        off = atomicAdd(&a.counters[L.cnt + 1], n);
    }
    ri = __shfl_sync(0xFFFFFFFFu, ri, 0);
    off = __shfl_sync(0xFFFFFFFFu, off, 0);
    if (ri + nrec > L.cap_rec || off + n > L.cap_surv) {
        if (lane == 0) atomicOr(&a.counters[CNT_OVERFLOW], 1u);
        return;
    }
    if (in) {
        L.surv[off + lane] = word;
        if (L.pay) L.pay[off + lane] = pay;
    }
    if (head) {
        const unsigned next = hm & ~below & ~(1u << lane);
        const uint32_t end = next ? (uint32_t)__ffs((int)next) - 1u : n, r = ri + (uint32_t)__popc(hm & below);
        L.unit[r] = unit;
        L.off[r] = off + lane;
        L.rcnt[r] = end - (uint32_t)lane;
    }
}

// ------------------------------------------------------------------------------------
// erosion
// ------------------------------------------------------------------------------------
struct ErosionWarp {
    alignas(16) uint8_t tab[kRows * 32];
    ClimCols col;
    float4 wy[2 * kLUnits];    // tier-0 tables: the y corners' weights (1 - fy, fy) and (1 - fy) hy, fy (hy - 1)
    uint64_t base[4];          // the block's lattice bases: table A x, z, table B x, z
    float4 lat[2][kLLat * kLLat];
    uint32_t wl[kLList];       // unit << 30 | chunk offset z << 15 | x
    float ws[kLList];
    uint32_t out[64];          // erosion survivors not yet in the list
};
static_assert(sizeof(ErosionWarp) % 16 == 0 && (kRows * 32) % 16 == 0, "warp_build writes 16 bytes at a time");
struct ErosionSmem {
    ErosionWarp w[kEWarps];
    GradF gf;
    uint32_t grad[kGradWords];
    unsigned int hist[P1_KINDS + kTiers];
};

__global__ void __launch_bounds__(kEThreads, 4) erosion_kernel(const __grid_constant__ BatchArgs a) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    ErosionSmem &S = *reinterpret_cast<ErosionSmem *>(smem_raw);
    const uint32_t n_units = batch_units(a);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned below = (1u << lane) - 1u;
    const int large = a.large_biomes ? 1 : 0;
    ErosionWarp &W = S.w[warp];
    fill_grad_table(S.grad, tid);
    fill_grad_table_f32(&S.gf, tid);
    if (tid < P1_KINDS + kTiers) S.hist[tid] = 0;
    __syncthreads();
    const ClimateStep *const st = c_steps[large];
    const int my_k = lane & 7;
    uint32_t tiers[2] = {0, 0};   // rejections of tiers 0 and 1; the others go straight to the histogram
    uint32_t rechecks = 0;
    const uint32_t groups = (n_units + kLUnits - 1) / kLUnits;
    for (uint32_t grp = blockIdx.x * kEWarps + (uint32_t)warp; grp < groups; grp += gridDim.x * kEWarps) {
        // ---- 8 tables of 4 units: lane = unit * 8 + step, so that a step's four columns lie in
        // different words of a row ----
        const uint32_t u0 = grp * kLUnits, my_u = u0 + (uint32_t)(lane >> 3);
        const bool valid = my_u < n_units;
        UnitPos up{};
        uint64_t seed = 0;
        if (valid) {
            up = unit_pos_call(a, my_u);
            seed = seed_value(a, up.g);
        }
        const int8_t *const slot = c_slot_a[large][st[my_k].slot];
        Xr r{};
        if (valid) r = octave_rng(c_noise[slot[0]], seed_fork_of(seed), slot[1], slot[2]);
        double ox = 0.0, oy = 0.0, oz = 0.0;
        warp_build(W.tab, lane, valid, r, ox, oy, oz);
        clim_col(W.col, lane, st[my_k], up.rx * 32, up.rz * 32, ox, oy, oz);
        if (my_k < 2) {
            const double hy = oy - floor(oy), fy = fade(hy);
            W.wy[(lane >> 3) * 2 + my_k] = make_float4(__double2float_rn(1.0 - fy), __double2float_rn(fy),
                                                       __double2float_rn((1.0 - fy) * hy), __double2float_rn(fy * (hy - 1.0)));
        }
        __syncwarp();

        uint32_t n1 = 0, n_out = 0;
        auto flush = [&](uint32_t n) {   // the first n <= 32 survivors to the list
            const uint32_t e = (uint32_t)lane < n ? W.out[lane] : 0u;
            list_emit(a, a.lists[0], lane, n, e >> 30, u0 + (e >> 30), entry_word(e), 0.0);
        };
        // erosion steps 2..7 breadth first over the warp's list
        auto drain = [&]() {
            __syncwarp();
            uint32_t n = n1;
#pragma unroll 1
            for (int k = 2; n && k < 8; k++) {
                const uint64_t step = st[k].fstep;
                const float cf = st[k].cf, lo = st[k].lo, hi = st[k].hi;
                uint32_t nn = 0;
#pragma unroll 1
                for (uint32_t b = 0; b < n; b += 32) {
                    const uint32_t q = b + (uint32_t)lane;
                    bool keep = false;
                    uint32_t e = 0;
                    float sum = 0.0f;
                    if (q < n) {
                        e = W.wl[q];
                        const int cu = (int)(e >> 30) * 8;
                        sum = __fmaf_rn(cf, col_sample(W.tab, W.col, S.gf, cu + k, step, e & 0x7FFFu, (e >> 15) & 0x7FFFu),
                                        W.ws[q]);
                        keep = sum >= hi;
                        if (!keep && !(sum < lo)) {   // inside the error band: the exact partial sum
                            rechecks++;
                            keep = erosion_recheck(a, W.tab, S.grad, large, k, u0, e);
                        }
                        if (a.codes && !keep) erosion_note(a, u0, e, st[k].tier);
                    }
                    const unsigned m = __ballot_sync(0xFFFFFFFFu, keep), mr = __ballot_sync(0xFFFFFFFFu, q < n && !keep);
                    if (k == 2) tiers[1] += (uint32_t)((mr >> lane) & 1u);
                    else if (lane == 0 && mr) atomicAdd(&S.hist[P1_KINDS + st[k].tier], (uint32_t)__popc(mr));
                    __syncwarp();
                    if (keep) {
                        const uint32_t at = (k == 7 ? n_out : nn) + (uint32_t)__popc(m & below);
                        if (k == 7) {
                            W.out[at] = e;
                        } else {
                            W.wl[at] = e;
                            W.ws[at] = sum;
                        }
                    }
                    __syncwarp();
                    if (k == 7) {
                        n_out += (uint32_t)__popc(m);
                        if (n_out >= 32) {
                            flush(32);
                            __syncwarp();
                            const uint32_t e2 = W.out[32 + lane];
                            __syncwarp();
                            W.out[lane] = e2;
                            n_out -= 32;
                            __syncwarp();
                        }
                    } else {
                        nn += (uint32_t)__popc(m);
                    }
                }
                n = nn;
            }
            n1 = 0;
        };

        // ---- tier 0, unit by unit, in blocks of at most 9 x 9 regions ----
        const int n_u = (int)min((uint32_t)kLUnits, n_units - u0);
#pragma unroll 1
        for (int u = 0; u < n_u; u++) {
            const int src = u * 8;
            const int rx = __shfl_sync(0xFFFFFFFFu, up.rx, src), rz = __shfl_sync(0xFFFFFFFFu, up.rz, src);
            const uint32_t tw = __shfl_sync(0xFFFFFFFFu, up.tw, src), th = __shfl_sync(0xFFFFFFFFu, up.th, src);
            const uint64_t sd = __shfl_sync(0xFFFFFFFFu, seed, src);
            const uint32_t side_x = list_side(th), side_z = list_side(tw);
            const uint32_t nbx = (tw + side_x - 1) / side_x, nbz = (th + side_z - 1) / side_z;
            const uint32_t bw = (tw + nbx - 1) / nbx, bh = (th + nbz - 1) / nbz;
            const uint64_t sa = st[0].fstep, sb = st[1].fstep;
#pragma unroll 1
            for (uint32_t bz = 0; bz < th; bz += bh) {
#pragma unroll 1
                for (uint32_t bx = 0; bx < tw; bx += bw) {
                    const uint32_t w = min(bw, tw - bx), h = min(bh, th - bz), n = w * h;
                    // the block's base per table and axis: lane 0-3 = table A x, z, table B x, z; its cells
                    constexpr uint64_t kFrac = 0x00FFFFFFFFFFFFFFull;
                    uint32_t cells = 0, cell0 = 0;   // lattice columns of this lane's axis, its first cell
                    __syncwarp();                    // the last block's samples are taken
                    if (lane < 4) {
                        const bool z = lane & 1;
                        const int c = src + (lane >> 1);
                        const uint64_t step = st[lane >> 1].fstep;
                        const uint64_t f = (z ? W.col.fz[c] : W.col.fx[c]) + (uint64_t)((z ? bz : bx) * 32u) * step;
                        W.base[lane] = f & kFrac;
                        cell0 = (uint32_t)(f >> 56);
                        cells = fixed_cell(fixed_at(f & kFrac, step, ((z ? h : w) - 1) * 32u + 23u)) + 2;
                    }
                    const int nax = (int)__shfl_sync(0xFFFFFFFFu, cells, 0), naz = (int)__shfl_sync(0xFFFFFFFFu, cells, 1),
                              nbx2 = (int)__shfl_sync(0xFFFFFFFFu, cells, 2), nbz2 = (int)__shfl_sync(0xFFFFFFFFu, cells, 3);
                    const int cax = (int)__shfl_sync(0xFFFFFFFFu, cell0, 0), caz = (int)__shfl_sync(0xFFFFFFFFu, cell0, 1),
                              cbx = (int)__shfl_sync(0xFFFFFFFFu, cell0, 2), cbz = (int)__shfl_sync(0xFFFFFFFFu, cell0, 3);
                    const int ma = nax * naz, mb = nbx2 * nbz2;
                    for (int q = lane; q < ma + mb; q += 32) {
                        const bool tb = q >= ma;
                        const int i = tb ? q - ma : q, nx = tb ? nbx2 : nax, iz = i / nx, ix = i - iz * nx;
                        const int c = src + (tb ? 1 : 0), jy = W.col.jy[c];
                        const int cx = (tb ? cbx : cax) + ix, cz = (tb ? cbz : caz) + iz;
                        const uint8_t *T = W.tab + c;
                        const int pa = T[(cx & 255) * 32];
                        const int p0 = T[((pa + jy) & 255) * 32], p1 = T[((pa + jy + 1) & 255) * 32];
                        const int h0 = T[((p0 + cz) & 255) * 32] & 15, h1 = T[((p1 + cz) & 255) * 32] & 15;
                        const float2 g0 = S.gf.xz[h0], g1 = S.gf.xz[h1];
                        const float4 wy = W.wy[u * 2 + (tb ? 1 : 0)];
                        float4 v;
                        v.x = __fmaf_rn(wy.y, g1.x, __fmul_rn(wy.x, g0.x));
                        v.y = __fmaf_rn(wy.y, g1.y, __fmul_rn(wy.x, g0.y));
                        v.z = __fmaf_rn(wy.w, S.gf.y[h1], __fmul_rn(wy.z, S.gf.y[h0]));
                        v.w = 0.0f;
                        W.lat[tb ? 1 : 0][i] = v;
                    }
                    __syncwarp();
                    const uint32_t inv = ((1u << 16) + w - 1) / w;   // q / w = (q * inv) >> 16 for q < 105, w <= 23
#pragma unroll 1
                    for (uint32_t b = 0; b < n; b += 32) {
                        const uint32_t q = b + (uint32_t)lane;
                        bool pass = false;
                        uint32_t e = 0;
                        float sum = 0.0f;
                        if (q < n) {
                            const uint32_t qz = (q * inv) >> 16, qx = q - qz * w;
                            int cx, cz;
                            hut_chunk(sd, rx + (int)(bx + qx), rz + (int)(bz + qz), a.salt, cx, cz);
                            const uint32_t dx = (uint32_t)(cx - rx * 32), dz = (uint32_t)(cz - rz * 32);
                            e = ((uint32_t)u << 30) | (dz << 15) | dx;
                            const uint32_t ex = dx - bx * 32u, ez = dz - bz * 32u;
                            sum = __fmul_rn(st[0].cf, lat_sample(W.lat[0], nax, fixed_at(W.base[0], sa, ex),
                                                                 fixed_at(W.base[1], sa, ez)));
                            sum = __fmaf_rn(st[1].cf, lat_sample(W.lat[1], nbx2, fixed_at(W.base[2], sb, ex),
                                                                 fixed_at(W.base[3], sb, ez)), sum);
                            pass = sum >= st[1].hi;
                            if (!pass && !(sum < st[1].lo)) {
                                rechecks++;
                                pass = erosion_recheck(a, W.tab, S.grad, large, 1, u0, e);
                            }
                            if (!pass) {
                                tiers[0]++;
                                if (a.codes) erosion_note(a, u0, e, st[1].tier);
                            }
                        }
                        const unsigned m = __ballot_sync(0xFFFFFFFFu, pass);
                        if (pass) {
                            const uint32_t at = n1 + (uint32_t)__popc(m & below);
                            W.wl[at] = e;
                            W.ws[at] = sum;
                        }
                        n1 += (uint32_t)__popc(m);
                        // the list is nearly full, or these were the last regions of the last unit
                        const bool last = u + 1 == n_u && bz + bh >= th && bx + bw >= tw && b + 32 >= n;
                        if (n1 > kLList - 32 || last) drain();
                    }
                }
            }
        }
        flush(n_out);
    }
    {
        for (int t = 0; t < 2; t++) {
            const uint32_t n = __reduce_add_sync(0xFFFFFFFFu, tiers[t]);
            if (lane == 0 && n) atomicAdd(&S.hist[P1_KINDS + st[1 + t].tier], n);
        }
        const uint32_t nk = __reduce_add_sync(0xFFFFFFFFu, rechecks);
        if (lane == 0) {
            if (nk) atomicAdd(&a.counters[CNT_RECHECK], nk);
        }
    }
    __syncthreads();
    if (tid < kTiers && S.hist[P1_KINDS + tid]) {
        atomicAdd(&a.hist[P1_KINDS + tid], (unsigned long long)S.hist[P1_KINDS + tid]);
        atomicAdd(&a.hist[P1_EROSION], (unsigned long long)S.hist[P1_KINDS + tid]);
    }
}

// ------------------------------------------------------------------------------------
// The stages after erosion: a warp takes 32 / K records, builds K tables for each (lane = record * K +
// table), and K lanes share a region, one sample each.
// ------------------------------------------------------------------------------------
enum : int { G_TEMPERATURE = 0, G_RIDGE, G_SCALED, G_ENTRANCE, G_ROUGH };
template <int G>
struct GateShape {
    static constexpr int K = G == G_TEMPERATURE ? 4 : 6;
    static constexpr int R = 32 / K;            // records per warp
    static constexpr bool climate = G <= G_RIDGE;
};

struct GateOrg {   // cave tables' origins, one per column
    double x[32], y[32], z[32];
};
struct GateWarp {
    alignas(16) uint8_t tab[kRows * 32];
    union {
        ClimCols col;
        GateOrg org;
    };
    uint64_t seed[8];
    int rx[8], rz[8];
    uint32_t unit[8], off[8], first[9];   // first: the records' prefix of region counts
    uint32_t out[2][64];                  // regions not yet in the lists: their record here, offset word and value
    uint32_t word[2][64];
    double pay[64];
};
static_assert(sizeof(GateWarp) % 16 == 0, "warp_build writes 16 bytes at a time");
struct GateSmem {
    GateWarp w[kLWarps];
    GradF gf;
    uint32_t grad[kGradWords];
    unsigned int hist[2];
};

template <int G>
__global__ void __launch_bounds__(kLThreads, 5) gate_kernel(const __grid_constant__ BatchArgs a, const __grid_constant__ RegionList in,
                                                               const __grid_constant__ RegionList out,
                                                               const __grid_constant__ RegionList open) {
    constexpr int K = GateShape<G>::K, R = GateShape<G>::R;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    GateSmem &S = *reinterpret_cast<GateSmem *>(smem_raw);
    if (a.counters[CNT_OVERFLOW]) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned below = (1u << lane) - 1u;
    const int large = a.large_biomes ? 1 : 0;
    GateWarp &W = S.w[warp];
    fill_grad_table(S.grad, tid);
    fill_grad_table_f32(&S.gf, tid);
    if (tid < 2) S.hist[tid] = 0;
    __syncthreads();
    const int my_r = min(lane / K, R - 1), my_p = lane % K;
    const bool lane_used = lane < R * K;
    constexpr int k0 = G == G_TEMPERATURE ? 8 : 12;
    // cave tables of the stage: column p of a record
    const int cslot = G == G_SCALED ? (my_p < 2 ? kBaseRarity + my_p : kBaseSp1 + my_p - 2)
                      : G == G_ENTRANCE ? kBaseEntrance + my_p
                                        : (my_p < 2 ? kBaseThickness + my_p : kBaseRmod + my_p - 2);
    const int8_t *const sl = GateShape<G>::climate ? c_slot_a[large][c_steps[large][k0 + (GateShape<G>::climate ? my_p : 0)].slot]
                                                   : c_slot_c[large][cslot];
    const NoiseSpec &ns = c_noise[sl[0]];
    const int sub = sl[1], oct = sl[2];
    const uint64_t step = GateShape<G>::climate ? c_steps[large][k0 + my_p].fstep : 0;
    uint32_t rechecks = 0, rejected = 0;
    const uint32_t n_rec = min(a.counters[in.cnt], in.cap_rec);
    const uint32_t groups = (n_rec + R - 1) / R;
    for (uint32_t grp = blockIdx.x * kLWarps + (uint32_t)warp; grp < groups; grp += gridDim.x * kLWarps) {
        const uint32_t rec = grp * R + (uint32_t)my_r;
        const bool valid = lane_used && rec < n_rec;
        UnitPos up{};
        uint64_t seed = 0;
        uint32_t unit = 0, cnt = 0, off = 0;
        if (rec < n_rec) {
            unit = in.unit[rec];
            off = in.off[rec];
            cnt = in.rcnt[rec];
            up = unit_pos_call(a, unit);
            seed = seed_value(a, up.g);
        }
        __syncwarp();
        if (my_p == 0 && lane_used) {
            W.seed[my_r] = seed;
            W.rx[my_r] = up.rx;
            W.rz[my_r] = up.rz;
            W.unit[my_r] = unit;
            W.off[my_r] = off;
        }
        Xr rng{};
        if (valid) rng = octave_rng(ns, seed_fork_of(seed), sub, oct);
        double ox = 0.0, oy = 0.0, oz = 0.0;
        warp_build(W.tab, lane, valid, rng, ox, oy, oz);
        if constexpr (GateShape<G>::climate) {
            clim_col(W.col, lane, c_steps[large][k0 + my_p], up.rx * 32, up.rz * 32, ox, oy, oz);
        } else {
            W.org.x[lane] = ox;
            W.org.y[lane] = oy;
            W.org.z[lane] = oz;
        }
        // prefix of the records' region counts
        uint32_t total = 0;
        for (int q = 0; q < R; q++) {
            const uint32_t c = __shfl_sync(0xFFFFFFFFu, cnt, q * K);
            if (lane == 0) W.first[q] = total;
            total += c;
        }
        if (lane == 0) W.first[R] = total;
        __syncwarp();
        uint32_t n_out[2] = {0, 0};
        auto flush = [&](int which, uint32_t n) {
            const uint32_t id = (uint32_t)lane < n ? W.out[which][lane] : 0u;
            const double pay = which == 0 && (uint32_t)lane < n ? W.pay[lane] : 0.0;
            list_emit(a, which ? open : out, lane, n, id, W.unit[id], W.word[which][lane], pay);
        };
#pragma unroll 1
        for (uint32_t base = 0; base < total; base += R) {
            const uint32_t i = base + (uint32_t)(lane / K);
            const bool have = lane_used && i < total;
            int r = 0;
            for (int q = 1; q < R; q++) r += i >= W.first[q] ? 1 : 0;
            uint32_t word = 0;
            int cx = 0, cz = 0;
            double in_pay = 0.0;
            if (have) {
                const uint32_t at = W.off[r] + (i - W.first[r]);
                word = in.surv[at];
                if (in.pay) in_pay = in.pay[at];
                hut_chunk(W.seed[r], W.rx[r] + (int)(word & 0xFFFFu), W.rz[r] + (int)(word >> 16), a.salt, cx, cz);
            }
            const int col = r * K + my_p;
            bool keep = false, is_open = false;
            double pay = 0.0;
            int code = -1;
            if constexpr (GateShape<G>::climate) {
                float v = 0.0f;
                if (have) v = col_sample(W.tab, W.col, S.gf, col, step, (uint32_t)(cx - W.rx[r] * 32), (uint32_t)(cz - W.rz[r] * 32));
                float sum = 0.0f;
#pragma unroll
                for (int q = 0; q < K; q++)
                    sum = __fmaf_rn(c_steps[large][k0 + q].cf, __shfl_down_sync(0xFFFFFFFFu, v, q), sum);
                if (have && my_p == 0) {
                    const F32Bands &B = c_bands[large];
                    bool bad, inside = false;
                    if constexpr (G == G_TEMPERATURE) {
                        inside = (sum >= B.t_lo[0] && sum < B.t_hi[0]) || (sum >= B.t_lo[1] && sum < B.t_hi[1]);
                        bad = sum < B.t_lo[0] || (!a.mc_1_18_2 && sum >= B.t_hi[1]);
                    } else {
                        for (int q = 0; q < 4; q++) inside |= sum >= B.r_lo[q] && sum < B.r_hi[q];
                        const bool a0 = sum >= B.r_hi[0], a1 = sum >= B.r_hi[1], a2 = sum >= B.r_hi[2], a3 = sum >= B.r_hi[3];
                        bad = (a2 && !a3) || (!a1 && a0) || (!a.pre_26_2 && !a0);
                    }
                    if (inside) {
                        rechecks++;
                        const double t = col_value64(W.tab, col, S.grad, large, k0, K, W.seed[r], (cx * 16 + 8) * 0.25,
                                                     (cz * 16 + 8) * 0.25);
                        bad = G == G_TEMPERATURE ? temperature_bad(a, t) : ridge_bad(a, t);
                    }
                    keep = !bad;
                    if (bad) code = G == G_TEMPERATURE ? P1_TEMPERATURE : P1_RIDGE;
                }
            } else {
                const int hx = cx * 16 + 3, hz = cz * 16 + 3;
                // FP64 samples in the reference's order, as everywhere in the default core's cave gates: what is
                // decided here is the reference's decision.
                const ColTable<32> T{W.tab + col, S.grad};
                const double scale = sub ? kDblScale : 1.0, lac = ns.lac[oct], amp = ns.amp[oct], per = ns.per[oct];
                auto sample = [&](double x, double y, double z) {
                    return (amp * perlin_3d(T, W.org.x[col], W.org.y[col], W.org.z[col], keep_precision((x * scale) * lac),
                                            keep_precision((y * scale) * lac), keep_precision((z * scale) * lac))) *
                           per;
                };
                // the DoublePerlin value of the noise whose 2 np tables are columns p, p + 1, .. of the region
                const int lead = lane - my_p;
                auto value = [&](int noise, double v, int p, int np) {
                    double s0 = 0.0, s1 = 0.0;
                    for (int q = 0; q < np; q++) s0 += __shfl_sync(0xFFFFFFFFu, v, (lead + p + q) & 31);
                    for (int q = 0; q < np; q++) s1 += __shfl_sync(0xFFFFFFFFu, v, (lead + p + np + q) & 31);
                    return (s0 + s1) * c_noise[noise].amplitude;
                };
                if constexpr (G == G_SCALED) {
                    double v = 0.0;
                    if (have && my_p < 2) v = sample((double)(int)((uint32_t)hx * 2u), 50.0, (double)(int)((uint32_t)hz * 2u));
                    const double sc = tunnel_scale(value(N_SPAGHETTI_RARITY, v, 0, 1));
                    if (have && my_p >= 2) v = sample((double)hx / sc, 50.0 / sc, (double)hz / sc);
                    const double l = value(N_SPAGHETTI_1, v, 2, 1), m = value(N_SPAGHETTI_2, v, 4, 1);
                    keep = have && my_p == 0;
                    pay = fmax(fabs(sc * l), fabs(sc * m));
                } else if constexpr (G == G_ENTRANCE) {
                    const double v = have ? sample((double)hx * 0.75, 25.0, (double)hz * 0.75) : 0.0;
                    const double ent = value(N_CAVE_ENTRANCE, v, 0, 3);
                    if (have && my_p == 0) {
                        // the entrance term's depth part is 0 at 50
                        if (ent + 0.37 < 0) is_open = true;
                        else if (in_pay >= kSpagSure) code = P1_ENTRANCE_50;
                        else keep = true;
                        pay = in_pay;
                    }
                } else {
                    const double v = have ? sample((double)hx, 50.0, (double)hz) : 0.0;
                    const double tv = value(N_SPAGHETTI_THICKNESS, v, 0, 1), mod = value(N_ROUGHNESS_MODULATOR, v, 2, 1),
                                 rgh = value(N_ROUGHNESS, v, 4, 1);
                    if (have && my_p == 0) {
                        const double h = lerp((tv - -1.0) / (1.0 - -1.0), 0.065, 0.088);
                        // the larger of the two differences is the larger term's: a rounded difference is monotone
                        const double p = clampd(in_pay - h, -1.0, 1.0);
                        const double q = (-0.05 + (-0.05 * mod)) * (-0.4 + fabs(rgh));
                        if (p + q >= 0) code = P1_ENTRANCE_50;
                        else is_open = true;
                    }
                }
            }
            if (code >= 0) {
                rejected++;
                if (a.codes) {
                    const UnitPos p = unit_pos_call(a, W.unit[r]);
                    note_code(a, p.g, p.region(word), code, -1);
                }
            }
            // what goes on keeps the records' order, so a list's runs of one record are its records
            const unsigned mk = __ballot_sync(0xFFFFFFFFu, keep), mo = __ballot_sync(0xFFFFFFFFu, is_open);
            if (keep) {
                const uint32_t at = n_out[0] + (uint32_t)__popc(mk & below);
                W.out[0][at] = (uint32_t)r;
                W.word[0][at] = word;
                W.pay[at] = pay;
            }
            if (is_open) {
                const uint32_t at = n_out[1] + (uint32_t)__popc(mo & below);
                W.out[1][at] = (uint32_t)r;
                W.word[1][at] = word;
            }
            n_out[0] += (uint32_t)__popc(mk);
            n_out[1] += (uint32_t)__popc(mo);
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 2; q++) {
                if (n_out[q] < 32) continue;
                flush(q, 32);
                __syncwarp();
                const uint32_t id = W.out[q][32 + lane], wd = W.word[q][32 + lane];
                const double py = q == 0 ? W.pay[32 + lane] : 0.0;
                __syncwarp();
                W.out[q][lane] = id;
                W.word[q][lane] = wd;
                if (q == 0) W.pay[lane] = py;
                n_out[q] -= 32;
                __syncwarp();
            }
        }
        flush(0, n_out[0]);
        flush(1, n_out[1]);
    }
    const uint32_t nr = __reduce_add_sync(0xFFFFFFFFu, rejected), nk = __reduce_add_sync(0xFFFFFFFFu, rechecks);
    if (lane == 0) {
        if (nr) atomicAdd(&S.hist[0], nr);
        if (nk) atomicAdd(&a.counters[CNT_RECHECK], nk);
    }
    __syncthreads();
    if (tid == 0 && S.hist[0])
        atomicAdd(&a.hist[G == G_TEMPERATURE ? P1_TEMPERATURE : G == G_RIDGE ? P1_RIDGE : P1_ENTRANCE_50],
                  (unsigned long long)S.hist[0]);
}

static unsigned long long g_smem_done_ero = 0, g_smem_done_gate[5] = {0, 0, 0, 0, 0};
static void prepare_list_launches() {
    allow_dynamic_smem(erosion_kernel, sizeof(ErosionSmem), g_smem_done_ero);
    allow_dynamic_smem(gate_kernel<G_TEMPERATURE>, sizeof(GateSmem), g_smem_done_gate[0]);
    allow_dynamic_smem(gate_kernel<G_RIDGE>, sizeof(GateSmem), g_smem_done_gate[1]);
    allow_dynamic_smem(gate_kernel<G_SCALED>, sizeof(GateSmem), g_smem_done_gate[2]);
    allow_dynamic_smem(gate_kernel<G_ENTRANCE>, sizeof(GateSmem), g_smem_done_gate[3]);
    allow_dynamic_smem(gate_kernel<G_ROUGH>, sizeof(GateSmem), g_smem_done_gate[4]);
}

// Grids of the resident CTAs; asked for once, by whichever thread comes first (after prepare_list_launches).
struct ListGrids {
    int erosion = 1, gate = 1;
    ListGrids() {
        int dev = 0, sms = 1, ero = 0, g = 8;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ero, erosion_kernel, kEThreads, sizeof(ErosionSmem));
        auto least = [&](auto kernel) {
            int n = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kLThreads, sizeof(GateSmem));
            if (n < g) g = n;
        };
        least(gate_kernel<G_TEMPERATURE>);
        least(gate_kernel<G_RIDGE>);
        least(gate_kernel<G_SCALED>);
        least(gate_kernel<G_ENTRANCE>);
        least(gate_kernel<G_ROUGH>);
        erosion = sms * (ero < 1 ? 1 : ero);
        gate = sms * (g < 1 ? 1 : g);
    }
};
static const ListGrids &list_grids() {
    prepare_list_launches();
    static const ListGrids grids;
    return grids;
}

static RegionList stage_list(const BatchArgs &a, int list, int cnt) {
    RegionList L = a.lists[list];
    L.cnt = cnt;
    return L;
}

// The first entrance tests for the climate survivors in lists[0].
static void launch_cave_lists(const BatchArgs &a, cudaStream_t s) {
    const int gate = list_grids().gate;
    const RegionList none{}, open = stage_list(a, 2, CNT_RECORDS);
    gate_kernel<G_SCALED><<<gate, kLThreads, sizeof(GateSmem), s>>>(a, stage_list(a, 0, CNT_CLIMATE_LIST),
                                                                    stage_list(a, 1, CNT_SCALED_LIST), open);
    gate_kernel<G_ENTRANCE><<<gate, kLThreads, sizeof(GateSmem), s>>>(a, stage_list(a, 1, CNT_SCALED_LIST),
                                                                      stage_list(a, 0, CNT_ENTRANCE_LIST), open);
    gate_kernel<G_ROUGH><<<gate, kLThreads, sizeof(GateSmem), s>>>(a, stage_list(a, 0, CNT_ENTRANCE_LIST), none, open);
}

// The climate and entrance stages of a batch: grids of the resident CTAs, whose warps take groups of
// units or records in turn.  lists[0], lists[1] alternate; lists[2] is the entrance kernel's input.
void launch_lists(const BatchArgs &a, cudaStream_t s) {
    const int gate = list_grids().gate;
    BatchArgs b = a;
    b.lists[0].cnt = CNT_EROSION_LIST;
    erosion_kernel<<<list_grids().erosion, kEThreads, sizeof(ErosionSmem), s>>>(b);
    const RegionList none{};
    gate_kernel<G_TEMPERATURE><<<gate, kLThreads, sizeof(GateSmem), s>>>(a, stage_list(a, 0, CNT_EROSION_LIST), stage_list(a, 1, CNT_TEMP_LIST), none);
    gate_kernel<G_RIDGE><<<gate, kLThreads, sizeof(GateSmem), s>>>(a, stage_list(a, 1, CNT_TEMP_LIST), stage_list(a, 0, CNT_CLIMATE_LIST), none);
    launch_cave_lists(a, s);
}
