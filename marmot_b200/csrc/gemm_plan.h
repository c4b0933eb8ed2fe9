// How the tcgen05 matmuls with weights in tensor memory (gemm_ts.cu, gemm_ti.cu) divide a call: the plan that the host makes, and what
// a CTA's share of it is.  Plain C++ apart from the qualifiers (block_formats.h), so that the CPU tests run this very code.
#pragma once

#include "block_formats.h"

#include <stddef.h>
#include <stdint.h>

namespace mcu {

constexpr int TS_ROWS = 128;     // weight rows per tile (TMEM lanes)
constexpr int TS_SLAB_K = 256;   // values of K per slab
constexpr int TS_MAX_JOBS = 4;
constexpr int TS_MAX_GROUPS = 256;
constexpr int TS_MAX_SPLIT = 8;
constexpr int TI_COLS = 16;      // tokens of a tile of the integer kernel
constexpr int I8_MAX_T = 16, I8_ROWS = 64, I8_COLS_PER_STAGE = 4;  // the mma.sync kernel (gemm_i8.cu): a stage is 64 rows x four blocks

MCU_HD int ts_min(int a, int b) { return a < b ? a : b; }

struct TsJob {
    const uint8_t *w;
    float *out;
    const float *bias;
    int F, ldo;
    int row_tile0;  // first row tile of the job
};
// (264 bytes: a kernel's parameters travel with each launch.  With eight bytes more, 912 with the tensor maps, calls made one by one took 0.1 to
// 0.2 us longer: 59 x 1536 x 256 Q6_K 9.46 us, 9.35 so, 8 x 4096 x 1024 Q4_K 8.55, 8.38, 40 x 1024 x 1024 Q8_0 7.98, 7.79.)
struct TsParams {
    TsJob jobs[TS_MAX_JOBS];
    const float *rowscale;  // fp16: per-token power-of-two factor undone in the epilogue
    float *partial;         // two slots of 128 x bn floats per CTA
    int *counters;          // one ticket per CTA, zero between launches
    int *err;
    const int *group_counts, *group_offsets;  // grouped launches (MoE experts), device memory
    long row_bytes;
    int n_jobs, T, bn, nb, slabs, raw_shift;  // raw_shift: log2 of the slab ring's depth
    short loose;            // weight rows that are not 16-byte multiples, or do not start on one
    short whole;            // the tiles are dealt to the CTAs whole, in turn
    int split;              // > 1: clusters of `split` CTAs (pairs) share a tile along K; otherwise ranges of units
    int tiles, t_tiles;     // output tiles in all; token tiles per row tile
    int groups, row_tiles;  // grouped launches: number of groups, row tiles per group
};
static_assert(sizeof(TsParams) <= 264, "see above");

// One output tile: which weights, which tokens, where the result goes.
struct TsTile {
    int job, f0, rows;       // rows that exist
    int w_row0;              // first weight row in the (stacked) matrix
    int t_row0, t_count;     // first activation / output row, and how many of the BN columns are tokens
};

// The units [u0, u1) of this CTA (one slab of one tile each), and what a tile is.
struct TsWork {
    const int *group_tile0;
    bool grouped;
    int bn, u0, u1, n_use;
    long long units;

    MCU_HD TsTile tile(const TsParams &p, int tile) const {
        TsTile t;
        int rt, tt, T_here, row_off, cols = bn;
        t.job = 0;
        if (grouped) {
            int g = 0;
            while (tile >= group_tile0[g + 1]) ++g;
            int in = tile - group_tile0[g];
            const int t_tiles = (group_tile0[g + 1] - group_tile0[g]) / p.row_tiles;
            rt = in / t_tiles;
            tt = in - rt * t_tiles;
            while (t.job + 1 < p.n_jobs && rt >= p.jobs[t.job + 1].row_tile0) ++t.job;
            rt -= p.jobs[t.job].row_tile0;
            T_here = p.group_counts[g];
            row_off = p.group_offsets[g];
            cols = ((T_here + t_tiles - 1) / t_tiles + 15) & ~15;  // the group's tokens dealt evenly to its tiles
            t.w_row0 = g * p.jobs[t.job].F;
        } else {
            rt = tile / p.t_tiles;
            tt = tile - rt * p.t_tiles;
            while (t.job + 1 < p.n_jobs && rt >= p.jobs[t.job + 1].row_tile0) ++t.job;
            rt -= p.jobs[t.job].row_tile0;
            T_here = p.T;
            row_off = 0;
            t.w_row0 = 0;
        }
        t.f0 = rt * TS_ROWS;
        t.w_row0 += t.f0;
        t.rows = ts_min(TS_ROWS, p.jobs[t.job].F - t.f0);
        t.t_row0 = row_off + tt * cols;
        t.t_count = ts_min(cols, T_here - tt * cols);
        return t;
    }
};
MCU_HD TsWork ts_work(const TsParams &p, bool grouped, const int *group_tile0, int bn, int cta, int n_cta) {
    TsWork w;
    const int KS = p.slabs;
    w.group_tile0 = group_tile0;
    w.grouped = grouped;
    w.bn = bn;
    w.units = (long long)(grouped ? group_tile0[p.groups] : p.tiles) * KS;
    w.n_use = (int)(w.units < n_cta ? w.units : n_cta);  // (a grouped launch may find fewer units than CTAs)
    if (p.split > 1) {
        const int t = cta / p.split, part = cta - t * p.split;
        w.u0 = t * KS + KS * part / p.split;
        w.u1 = t * KS + KS * (part + 1) / p.split;
        return w;
    }
    if (p.whole) {  // as many CTAs as tiles, or fewer: the first ones take one more
        const int each = p.tiles / n_cta, more = p.tiles - each * n_cta;
        w.u0 = KS * (cta * each + ts_min(cta, more));
        w.u1 = w.u0 + KS * (each + (cta < more ? 1 : 0));
        return w;
    }
    w.u0 = cta < w.n_use ? (int)(w.units * cta / w.n_use) : 0;
    w.u1 = cta < w.n_use ? (int)(w.units * (cta + 1) / w.n_use) : 0;
    return w;
}

// A tile cut between CTAs (ranges of units): the CTAs that hold a share of it, and the slot of each (0: its range starts inside the
// tile or at its start, 1: before it).
struct TsOwners {
    int first, last;
};
MCU_HD TsOwners ts_owners(const TsWork &w, int tile, int KS) {
    const long long lo = (long long)tile * KS, hi = lo + KS;
    return {(int)(((lo + 1) * w.n_use - 1) / w.units), (int)((hi * w.n_use - 1) / w.units)};
}
MCU_HD int ts_share_slot(const TsWork &w, int tile, int KS, int cta) { return w.units * cta / w.n_use >= (long long)tile * KS ? 0 : 1; }

// ---- host ----
struct TsPlan {
    int bn, t_tiles, split, n_cta;
    double cost;
    int whole = 0;
};

// How to spread `tiles` output tiles of KS slabs over `room` SMs, and what it costs in cycles, by measurements of all the forms at 70 to 512
// tokens and 2048 x 2048 to 4096 x 28672 weights.  A slab takes the longer of its conversion (less in tiles of up to 64 columns, whose
// stages hold 128 values of K) and its MMAs; a tile ends with its epilogue.
// - Whole tiles, one or several to a CTA: 2000 for a CTA's start, 2500 between two tiles of it.  (As a CTA of its own, a further tile cost its
//   start as well, and the kernels behind could not start early before the last wave: 20 x 2304 x 35840 Q4_K 25.4 -> 20.5 us, 39 x 1536 x 51200
//   Q8_0 34.5 -> 27.5, 512 x 4096 x 14336 Q8_0 80.1 -> 77.9.)
// - A tile over a cluster: the exchange of the shares through the CTAs' shared memories.
// - Equal ranges of slabs: cut tiles have their shares written to memory, and read again by the CTA that comes last; a tile of 256
//   columns costs 47000 so, which only many tiles per CTA are worth (512 x 4096 x 14336 Q8_0: 77 us in ranges, 65.5 in whole tiles).  The way
//   through memory and the tickets costs 6000 besides, 11000 in narrow tiles, by all forms at 9 to 2048 tokens and thirteen sizes
//   (9 x 2048 x 5632 Q8_0: 17.5 us in ranges, 9.8 in clusters of two; 17 x 2048 x 32000 Q4_K: 24.7, 17.7 in whole tiles; 2048 x 14336 x 4096
//   Q4_K: 266, 231 in whole tiles; 512 x 4096 x 28672 Q4_K: 115.7, 112 in whole tiles).
inline TsPlan ts_spread(int kind, int tiles, int KS, int bn, int t_tiles, int room) {
    const long U = (long)tiles * KS;
    const bool wide = bn > 64;
    const double conv = kind == KIND_Q4_K ? (wide ? 1500 : 1120) : kind == KIND_Q6_K ? (wide ? 2100 : 1700) : (wide ? 1750 : 1500);
    const double mma = 8.5 * bn, unit = mma > conv ? mma : conv, tile_end = 1000.0 + 8.0 * bn;
    TsPlan best{bn, t_tiles, 1, 0, 1e30};
    auto consider = [&](int split, long n, double cost, int whole = 0) {
        if (cost < best.cost) best = TsPlan{bn, t_tiles, split, (int)n, cost, whole};
    };
    const int waves = (tiles + room - 1) / room;
    consider(1, tiles < room ? tiles : room, waves * (KS * unit) + (waves - 1) * 2500.0 + tile_end + 2000.0, 1);
    for (int sp = 2; sp <= TS_MAX_SPLIT && sp <= KS; sp *= 2) {
        // A cluster is placed inside a GPC (16 to 20 SMs): sixteen clusters of eight did not run at once (2048 x 2048: 12.6 us,
        // 64 CTAs in clusters of four 7.5), fourteen do.
        const int usable = sp >= 8 ? room * 7 / 9 : room;
        const double exchange = sp == 2 ? 3500.0 + 30.0 * bn : 5000.0 + 20.0 * bn;
        if ((long)tiles * sp <= usable) consider(sp, (long)tiles * sp, (KS + sp - 1) / sp * unit + tile_end + 2000.0 + exchange);
    }
    const long n = U < room ? U : room;
    const long upc = (U + n - 1) / n;
    const bool cut = U % n != 0 || upc % KS != 0;
    const double shares = cut ? (double)KS / upc + 1.0 : 0.0;
    const double exchange = shares * 65.0 * bn + (!cut ? 0.0 : wide ? 6000.0 : 11000.0);
    consider(1, n, upc * unit + ((double)upc / KS + 1.0) * tile_end + 2000.0 + exchange);
    return best;
}

inline TsPlan ts_plan(int kind, int T, int K, const int *F, int n_jobs, int sms) {
    const int nb = (K + block_values(kind) - 1) / block_values(kind);
    const int KS = (nb * block_values(kind) + TS_SLAB_K - 1) / TS_SLAB_K;
    int rows = 0;
    for (int j = 0; j < n_jobs; ++j) rows += (F[j] + TS_ROWS - 1) / TS_ROWS;
    TsPlan best{};
    best.cost = 1e30;
    // as few token tiles as there can be, or a few more: narrower tiles fill the SMs better, but the weights are converted more often
    // (6 % for each: with all SMs at work the chip runs into its power limit)
    const int fewest = (T + 255) / 256, most = (T + 63) / 64;
    for (int tried = fewest; tried <= most && tried <= fewest + 3; ++tried) {
        const int bn = ((T + tried - 1) / tried + 15) / 16 * 16;
        const int t_tiles = (T + bn - 1) / bn;  // (not `tried`: widened to 16 columns, fewer tiles may hold all tokens, and the last would be empty)
        TsPlan pl = ts_spread(kind, rows * t_tiles, KS, bn, t_tiles, sms);
        pl.cost *= 1.0 + 0.06 * (t_tiles - fewest);
        if (pl.cost < best.cost) best = pl;
    }
    return best;
}

// The same for the integer kernel: whole tiles, one or several to a CTA, a tile over a cluster, or equal ranges, whichever ends
// first, by a sweep of all three at nine tokens: a slab takes about 900 cycles (Q6_K 2100), the start of a CTA 2700 and each of its tiles 800 (8 x 4096 x 28672
// Q4_K, 224 tiles: 27.0 us in ranges, 24.6 so), a cluster's exchange 1500; a tile cut between
// ranges costs 9000 and 700 for every share that the last CTA reads (13056 x 1792 Q4_K: 22 us in ranges of five slabs, 13 in
// clusters of eight).  Clusters of eight: as in ts_spread.  Of clusters of four 33 run at once (a GPC's SMs are not always a multiple of four);
// the rest were a second wave: 9 tokens x 2048 on 33, 34 row tiles 8.4, 14.1 us, the latter 8.8 in clusters of two; Q6_K x 14336 24.9, 43.5, 28.3.
inline TsPlan ti_plan(int kind, int tiles, int KS, int sms) {
    const long U = (long)tiles * KS, n_most = U < sms ? U : sms, upc = (U + n_most - 1) / n_most;
    const double unit = kind == KIND_Q4_K ? 900.0 : 2100.0;
    TsPlan best{TI_COLS, 1, 1, (int)n_most, 1e30};
    auto consider = [&](int split, long n, double cost, int whole = 0) {
        if (cost < best.cost) best = TsPlan{TI_COLS, 1, split, (int)n, cost, whole};
    };
    const int waves = (tiles + sms - 1) / sms;
    consider(1, tiles < sms ? tiles : sms, waves * (KS * unit + 800.0) + 2700.0, 1);
    for (int sp = 2; sp <= TS_MAX_SPLIT && sp <= KS; sp *= 2)
        if ((long)tiles * sp <= (sp >= 8 ? sms * 7 / 9 : sp >= 4 ? sms * 9 / 10 : sms)) consider(sp, (long)tiles * sp, (KS + sp - 1) / sp * unit + 5000.0);
    const bool cut = U % n_most != 0 || upc % KS != 0;
    consider(1, n_most, (double)upc * unit + 2000.0 + (cut ? 9000.0 + 700.0 * ((double)KS / upc + 1.0) : 0.0));
    return best;
}

// Microseconds of a call of 5 to 16 tokens on `row_tiles` tiles of 128 rows with the integer kernel, staging included, and on `groups`
// groups of 64 rows with the mma.sync one: fitted to both at 5, 8, 9, 12 and 16 tokens, K 1024 to 14336 and 512 to 32000 rows (within
// 10 % of all but a few).  A stage of the latter takes 2.35 or 2.45 us and its first ones are 8 to 10; the former's cycles are those
// of its plan, which clusters on less than half of the SMs beat, and single waves, with SMs to spare.
// Both are fits to the kernels as they were then, and the integer one has become the faster for more of Q6_K since (8 tokens, integer and mma.sync:
// 4096 x 1024 7.9, 9.2 us; 2048 x 4096 8.4, 8.4; 4096 x 28672 37.2, 41.3; 14336 x 4096 21.4, 26.7, with 16 tokens 25.5, 28.7).  Over 290 calls
// of Q6_K and of short Q4_K rows the choice is 4.4 % slower than the better of the two, at most 33 % (8 x 4096 x 5248 17.6, 13.3).
inline double ti_us(int kind, int T, int K, int row_tiles, int sms) {
    const TsPlan pl = ti_plan(kind, row_tiles, (K + QK_K - 1) / QK_K, sms);
    if (kind == KIND_Q6_K && pl.split > 1 && 2 * pl.n_cta <= sms) return (T <= 8 ? 2.5 : 1.35) + (T <= 8 ? 0.6 : 0.8) * 1e-3 * pl.cost;
    const bool wave = pl.split == 1 && pl.n_cta == row_tiles && row_tiles <= sms;
    return 4.6 + (T <= 8 ? (wave ? 0.47 : 0.57) : (wave ? 0.62 : 0.68)) * 1e-3 * pl.cost;
}
inline double i8_us(int kind, int T, int K, int groups, int sms) {
    if (kind == KIND_Q4_K) return T <= 8 ? 5.0 : 5.6;  // (where i8_pays: a stage to a CTA)
    const int stages = ((K + QK_K - 1) / QK_K + I8_COLS_PER_STAGE - 1) / I8_COLS_PER_STAGE;  // of a group of rows
    const double per_cta = (double)groups * stages / sms;
    if (per_cta <= 1.0) return T <= 8 ? 7.2 + 0.47 * stages : 8.0 + 0.52 * stages;
    return T <= 8 ? 10.4 + 2.35 * per_cta : 12.3 + 2.45 * per_cta;
}
// The mma.sync kernel's stage units: the first one of CTA c of C, and the CTA whose span holds unit x.
MCU_HD int i8_span_begin(int SU, int c, int C) { return (int)(((long long)SU * c) / C); }
MCU_HD int i8_owner(int SU, int x, int C) { return (int)((((long long)(x + 1) * C + SU - 1) / SU) - 1); }

// Does a matrix of F rows (two: `mats`) belong on the mma.sync kernel rather than the tcgen05 one?  Q4_K: rows of up to four blocks, a stage
// for every CTA (5 us, 7 there whatever the size); larger ones never by more than a few per cent.  Q6_K: by the times above.
inline bool i8_pays(int kind, int T, int K, int F, int mats, int sms) {
    const int groups = mats * ((F + I8_ROWS - 1) / I8_ROWS);
    if (kind == KIND_Q4_K) return K <= QK_K * I8_COLS_PER_STAGE && groups <= sms;
    return i8_us(kind, T, K, groups, sms) < ti_us(kind, T, K, mats * ((F + TS_ROWS - 1) / TS_ROWS), sms);
}

}  // namespace mcu
