// The work division of the tcgen05 matmuls (csrc/gemm_plan.h) checked tile by tile and unit by unit; driven by test_matmul_plan_cpu.py.
#include "../marmot_b200/csrc/gemm_plan.h"

#include <map>
#include <set>
#include <utility>
#include <vector>

using namespace mcu;

// 0, or which of the statements below does not hold.
static int check(const TsParams &p, int bn, int n_cta, int sms, const int *group_tile0, const std::vector<std::pair<int, int>> &want) {
    const bool grouped = group_tile0 != nullptr;
    const int KS = p.slabs, tiles = grouped ? group_tile0[p.groups] : p.tiles;
    if (bn < 16 || bn > 256 || bn % 16 != 0) return 1;
    // every output tile holds tokens and rows, and together they cover every (row, token) of every job once
    long long covered = 0, all = 0;
    std::set<std::pair<int, int>> seen;  // (job and first row, first token)
    for (int i = 0; i < tiles; ++i) {
        const TsWork w = ts_work(p, grouped, group_tile0, bn, 0, n_cta);
        const TsTile t = w.tile(p, i);
        if (t.t_count < 1 || t.t_count > bn) return 2;
        if (t.rows < 1 || t.rows > TS_ROWS || t.f0 + t.rows > p.jobs[t.job].F) return 3;
        if (t.t_row0 < 0 || t.t_row0 + t.t_count > p.T) return 4;
        if (!seen.insert({t.w_row0 * TS_MAX_JOBS + t.job, t.t_row0}).second) return 5;
        covered += (long long)t.rows * t.t_count;
    }
    for (const auto &rows_tokens : want) all += (long long)rows_tokens.first * rows_tokens.second;
    if (covered != all) return 6;
    // the CTAs' units are the tiles' slabs, each once
    const long long U = (long long)tiles * KS;
    if (p.split > 1) {
        if (n_cta != tiles * p.split || n_cta > sms || p.split > KS) return 7;
    } else if (n_cta > sms) {
        return 8;
    }
    long long at = 0;
    std::map<int, std::vector<int>> holders;  // tiles that are not whole in a CTA: its CTAs
    std::set<std::pair<int, int>> slots;
    const TsWork any = ts_work(p, grouped, group_tile0, bn, 0, n_cta);
    for (int c = 0; c < n_cta; ++c) {
        const TsWork w = ts_work(p, grouped, group_tile0, bn, c, n_cta);
        if (w.u0 == w.u1) {
            if (!grouped) return 9;
            continue;
        }
        if (w.u0 != at || w.u1 < w.u0 || w.u1 > U) return 10;
        at = w.u1;
        if (p.split > 1) continue;
        for (int u = w.u0; u < w.u1;) {
            const int tile = u / KS, e = ts_min((tile + 1) * KS, w.u1);
            if (e - u != KS) {
                if (p.whole) return 11;
                holders[tile].push_back(c);
                const int slot = ts_share_slot(any, tile, KS, c);
                if (slot != (u == w.u0 ? 0 : 1) || !slots.insert({c, slot}).second) return 12;
            }
            u = e;
        }
    }
    if (at != U) return 13;
    std::set<int> tickets;
    for (const auto &h : holders) {
        const TsOwners own = ts_owners(any, h.first, KS);
        for (int c : h.second)  // (the kernels ask for the first one's slot only)
            if (c != own.first && ts_share_slot(any, h.first, KS, c) != 0) return 17;
        if (own.first != h.second.front() || own.last != h.second.back() || own.last - own.first + 1 != (int)h.second.size()) return 14;
        if (!tickets.insert(own.first).second) return 15;
    }
    return 0;
}

extern "C" int check_plan(int integer, int kind, int T, int K, const int *F, int n_jobs, int sms) {
    TsParams p{};
    p.nb = (K + block_values(kind) - 1) / block_values(kind);
    p.slabs = (p.nb * block_values(kind) + TS_SLAB_K - 1) / TS_SLAB_K;
    p.n_jobs = n_jobs;
    p.T = T;
    int row_tiles = 0;
    std::vector<std::pair<int, int>> want;
    for (int j = 0; j < n_jobs; ++j) {
        p.jobs[j].F = F[j];
        p.jobs[j].row_tile0 = row_tiles;
        row_tiles += (F[j] + TS_ROWS - 1) / TS_ROWS;
        want.push_back({F[j], T});
    }
    p.t_tiles = (T + TI_COLS - 1) / TI_COLS;
    TsPlan pl;
    if (integer) {
        pl = ti_plan(kind, row_tiles * p.t_tiles, p.slabs, sms);
        if (sms == 148 && pl.n_cta > (pl.split == 8 ? 15 * 8 : pl.split == 4 ? 33 * 4 : sms)) return 16;  // all clusters at once (cudaOccupancyMaxActiveClusters)
    } else {
        pl = ts_plan(kind, T, K, F, n_jobs, sms);
        p.t_tiles = pl.t_tiles;
    }
    p.split = pl.split;
    p.whole = pl.whole;
    p.tiles = row_tiles * p.t_tiles;
    return check(p, pl.bn, pl.n_cta, sms, nullptr, want);
}

// the plans that deal the tiles whole: every CTA has tiles, the counts differ by one at most (-1: the plan is another one)
extern "C" int check_whole(int integer, int kind, int T, int K, const int *F, int n_jobs, int sms) {
    TsParams p{};
    p.nb = (K + block_values(kind) - 1) / block_values(kind);
    p.slabs = (p.nb * block_values(kind) + TS_SLAB_K - 1) / TS_SLAB_K;
    p.n_jobs = n_jobs;
    p.T = T;
    int row_tiles = 0;
    std::vector<std::pair<int, int>> want;
    for (int j = 0; j < n_jobs; ++j) {
        p.jobs[j].F = F[j];
        p.jobs[j].row_tile0 = row_tiles;
        row_tiles += (F[j] + TS_ROWS - 1) / TS_ROWS;
        want.push_back({F[j], T});
    }
    p.t_tiles = (T + TI_COLS - 1) / TI_COLS;
    const TsPlan pl = integer ? ti_plan(kind, row_tiles * p.t_tiles, p.slabs, sms) : ts_plan(kind, T, K, F, n_jobs, sms);
    if (!pl.whole) return -1;
    if (!integer) p.t_tiles = pl.t_tiles;
    p.split = pl.split;
    p.whole = 1;
    p.tiles = row_tiles * p.t_tiles;
    int least = 1 << 30, most = 0;
    for (int c = 0; c < pl.n_cta; ++c) {
        const TsWork w = ts_work(p, false, nullptr, pl.bn, c, pl.n_cta);
        if (w.u0 % p.slabs != 0 || w.u1 % p.slabs != 0) return 20;
        least = ts_min(least, w.u1 - w.u0);
        most = most > w.u1 - w.u0 ? most : w.u1 - w.u0;
    }
    if (pl.split != 1 || pl.n_cta > sms || least < p.slabs || most - least > p.slabs) return 21;
    return check(p, pl.bn, pl.n_cta, sms, nullptr, want);
}

// groups of `counts` tokens over stacked matrices of F rows each, as ts_group_table lays them out
extern "C" int check_groups(int slabs, const int *counts, int groups, const int *F, int n_jobs, int bn, int sms) {
    TsParams p{};
    p.slabs = slabs;
    p.n_jobs = n_jobs;
    p.split = 1;
    p.groups = groups;
    std::vector<int> offsets(groups), tile0(groups + 1, 0);
    std::vector<std::pair<int, int>> want;
    for (int j = 0; j < n_jobs; ++j) {
        p.jobs[j].F = F[j];
        p.jobs[j].row_tile0 = p.row_tiles;
        p.row_tiles += (F[j] + TS_ROWS - 1) / TS_ROWS;
    }
    for (int g = 0; g < groups; ++g) {
        offsets[g] = p.T;
        p.T += counts[g];
        tile0[g + 1] = tile0[g] + (counts[g] + bn - 1) / bn * p.row_tiles;
        for (int j = 0; j < n_jobs; ++j) want.push_back({F[j], counts[g]});
    }
    p.group_counts = counts;
    p.group_offsets = offsets.data();
    return check(p, bn, sms, sms, tile0.data(), want);
}

// the mma.sync kernel's division
extern "C" int i8_begin(int SU, int c, int C) { return i8_span_begin(SU, c, C); }
extern "C" int i8_holder(int SU, int x, int C) { return i8_owner(SU, x, C); }
