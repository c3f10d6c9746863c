// How the weight-gradient kernels' work is cut into CTAs: host arithmetic only, no CUDA.
//
// A work item is a block of weight rows; it sums over all token tiles.  Items may be whole (one CTA, which writes the bf16 result
// itself) or split over the tokens (fp32 partial sums, added by a reduction).  The hardware deals CTAs in launch order to the SM that
// frees up first, so the duration of a plan is that of a list schedule; a plan is the cheapest of a few families, by that duration.
#pragma once
#include <stdint.h>

#include "kernels.h"

namespace fmhf {
namespace {   // (a table shared by two builds of the library in one process would mix their plans)

struct DwPlan {
    int tiles_per_seq, tiles_total, nsplit, tiles_per_split;
    int n_direct;               // blocks that are not split at all
    int n_mixed, small_tiles;   // uneven split of the first n_mixed blocks (two-way splits only), else 0
    double tiles;               // predicted duration, in token tiles
};

// How the weight-gradient kernel of a head dimension cuts its work, and what a CTA costs besides its token tiles (weights in,
// first tile through the pipeline, accumulators out: the intercept of kernel time over tiles per CTA, about 7 us), a split's
// extra launch (4 us) and a byte of partial sums (written once, read once, about 4 TB/s), all in units of one token tile.
// (d_h = 128: measured on the kernel that worked with lane = token.  The present one takes 1.33 us a tile and 9.4 us a CTA besides, over one to
// six full waves of 4 to 128 tiles a CTA, so these figures split more than is best: with 1.33 and 9.4, 140 of 1495 drawn shapes get another
// plan, whose whole backward takes 8.4 % less, single ones between 14 % more and 1.6 times less.)
struct DwShape {
    int rows, tokens;
    double tile_us;
    double fixed() const { return 7.0 / tile_us; }
    double launch() const { return 4.0 / tile_us; }
    double sums(double bytes) const { return bytes / 4.0e6 / tile_us; }
};
inline DwShape dw_shape(int dh) { return dh == 128 ? DwShape{64, 128, 1.8} : DwShape{128, 64, dh == 64 ? 0.8 : 1.0}; }

// The times at which the SMs become free, as few (time, number of SMs) groups: jobs come in runs of equal length, so a run is dealt
// out by groups of SMs, and by whole rounds where every SM gets one, instead of job by job.  A run adds one group at most.
class SmTimes {
  public:
    explicit SmTimes(int num_sms) : sms_(num_sms), n_(1) { t_[0] = 0.0; c_[0] = num_sms; }
    void run(long long jobs, double len) {
        while (jobs > 0) {
            if (jobs >= sms_ && t_[n_ - 1] - t_[0] <= len) {
                const long long rounds = jobs / sms_;
                for (int i = 0; i < n_; ++i) t_[i] += (double)rounds * len;
                jobs -= rounds * sms_;
                continue;
            }
            const double end = t_[0] + len;
            const int take = jobs < c_[0] ? (int)jobs : c_[0];
            jobs -= take;
            int from = 0;
            if ((c_[0] -= take) == 0) from = 1;                    // the group moves as a whole
            int at = from;                                         // where (end, take) belongs among the groups that stay
            while (at < n_ && t_[at] < end) ++at;
            if (at < n_ && t_[at] == end) {
                c_[at] += take;
                if (from) drop_first();
            } else if (from) {
                for (int i = 1; i < at; ++i) { t_[i - 1] = t_[i]; c_[i - 1] = c_[i]; }
                t_[at - 1] = end; c_[at - 1] = take;
            } else {
                for (int i = n_; i > at; --i) { t_[i] = t_[i - 1]; c_[i] = c_[i - 1]; }
                t_[at] = end; c_[at] = take;
                ++n_;
            }
        }
    }
    double end() const { return t_[n_ - 1]; }

  private:
    void drop_first() {
        --n_;
        for (int i = 0; i < n_; ++i) { t_[i] = t_[i + 1]; c_[i] = c_[i + 1]; }
    }
    int sms_, n_;
    double t_[8];   // at most four runs a schedule
    int c_[8];
};

// First element of [Hkuv][I][DH] that belongs to a split block.
inline long long dw_first(const flashmhf_dims &d, const DwPlan &pl) {
    const int I = d.E * d.De, rows = dw_shape(d.Dh).rows, nblk_j = (I + rows - 1) / rows;
    return pl.nsplit > 1 ? ((long long)(pl.n_direct / nblk_j) * I + (long long)(pl.n_direct % nblk_j) * rows) * d.Dh : 0;
}
// Whole sets of partial sums, one at least.
inline size_t dw_workspace(const flashmhf_dims &d, const DwPlan &pl) {
    const size_t plane = (size_t)d.Hkuv * (size_t)d.E * d.De * d.Dh, need = (size_t)pl.nsplit * (plane - (size_t)dw_first(d, pl));
    return (need + plane - 1) / plane * 3 * plane * sizeof(float);
}

namespace dw_detail {

// With a two-way split the CTAs are equal and their last wave is partly empty (704 CTAs on 148 SMs: the fifth wave is
// 76 % full, 5 % of the kernel).  Splitting some blocks unevenly -- long parts launched first, short parts last, the
// equal halves of the other blocks in between -- lets the short parts fill the SMs the last wave would leave idle.
// The split point and the number of such blocks are found by simulating the launch order for a few candidates.
// The partial sums still number two per block, so the reduction and the workspace do not change.
// Returns the simulated duration (token tiles).
inline double plan_uneven(DwPlan &p, long long items, int num_sms, double fixed) {
    p.n_mixed = p.small_tiles = 0;
    const int T = p.tiles_total, half = p.tiles_per_split;
    auto makespan = [&](long long nmix, int small) {
        SmTimes sm(num_sms);
        sm.run(nmix, T - small + fixed);
        sm.run(items - nmix, half + fixed);
        sm.run(items - nmix, T - half + fixed);
        sm.run(nmix, small + fixed);
        return sm.end();
    };
    if (items > 2048 || T < 2) return (double)((2 * items + num_sms - 1) / num_sms) * (half + fixed);
    const double base = makespan(0, 0);
    // worth another launch order from 1.5 % on, which no cut can give where the SMs are as busy as that already
    const double busy = (double)items * (T + 2 * fixed) / num_sms;
    if (T < 32 || busy > 0.985 * base) return base;
    double best = base;
    const int step_small = T / 32 > 1 ? T / 32 : 1, step_mix = num_sms / 4 > 1 ? num_sms / 4 : 1;
    for (int small = step_small; small < half; small += step_small)
        for (int nmix = step_mix; nmix <= items; nmix += step_mix) {
            if ((double)((nmix + num_sms - 1) / num_sms) * (T - small + fixed) >= best - 1e-9) break;
            const double m = makespan(nmix, small);
            if (m < best - 1e-9) { best = m; p.n_mixed = nmix; p.small_tiles = small; }
        }
    if (best > 0.985 * base) {
        p.n_mixed = p.small_tiles = 0;
        best = base;
    }
    return best;
}

// Whole blocks for as many full waves as there are, and the rest split k ways to fill the last one: only the rest has partial sums.
// `sums`: the time to add one set of partial sums of all blocks.  `fits`: whether there is room for a plan's partial sums.  Returns the
// duration, addition included, of a plan that takes less than `best`, or `best`.
template <typename Fits>
double plan_rest(DwPlan &p, long long items, int num_sms, double fixed, double launch, double sums, double best, const Fits &fits) {
    const int T = p.tiles_total;
    DwPlan b = p;
    if (items > 2048 || T < 8) return best;
    for (int k = 2; k <= 6; ++k) {
        const int tiles = (T + k - 1) / k;
        if ((T + tiles - 1) / tiles != k) continue;
        for (int q = 2; q * (long long)num_sms / 4 < items; ++q) {   // quarter waves
            const long long nd = q * (long long)num_sms / 4, split = items - nd;
            const double add = launch + k * sums * (double)split / (double)items;
            const double busy = ((double)items * T + fixed * (double)(nd + k * split)) / num_sms;
            const double whole = (double)((nd + num_sms - 1) / num_sms) * (T + fixed);
            if ((busy > whole ? busy : whole) + add >= best - 1e-9) continue;   // not even with every SM busy to the end
            SmTimes sm(num_sms);
            sm.run(nd, T + fixed);
            sm.run((k - 1) * split, tiles + fixed);
            sm.run(split, T - (k - 1) * tiles + fixed);
            const double m = sm.end() + add;
            DwPlan c = p;
            c.n_direct = (int)nd;
            c.nsplit = k;
            c.tiles_per_split = tiles;
            if (m < best - 1e-9 && fits(c)) { best = m; b = c; }
        }
    }
    p = b;
    return best;
}

// `room`: bytes there are for partial sums.  (A plan without any always fits.)
inline DwPlan make_plan(const flashmhf_dims &d, int num_sms, bool followed, size_t room) {
    const DwShape sh = dw_shape(d.Dh);
    const long long items = (long long)d.Hkuv * (((long long)d.E * d.De + sh.rows - 1) / sh.rows);
    const double sums = sh.sums((double)d.Hkuv * d.E * d.De * 3 * d.Dh * 4);   // one set of partial sums
    DwPlan p0{};
    p0.tiles_per_seq = (d.S + sh.tokens - 1) / sh.tokens;
    p0.tiles_total = p0.tiles_per_seq * (d.H / d.Hkuv) * d.B;
    auto fits = [&](const DwPlan &p) { return room == SIZE_MAX || dw_workspace(d, p) <= room; };
    // whole, then the rest split, then equal (or two uneven) parts; each family only where it can still be the shortest
    DwPlan best = p0;
    best.nsplit = 1;
    best.tiles_per_split = p0.tiles_total;
    double best_cost = (double)((items + num_sms - 1) / num_sms) * (p0.tiles_total + sh.fixed());
    // The dQ/dR kernel fills the last wave.  (The whole backward of 16 shapes of each head dimension whose plan this factor decides, against
    // none: 1.5 % faster at d_h = 64, 5.8 % at 96, 3.0 % at 128, the latter with the kernel before; single shapes between 7 % slower and 31 %
    // faster.)
    if (followed) best_cost *= 0.9;
    DwPlan rest = p0;
    const double rest_cost = plan_rest(rest, items, num_sms, sh.fixed(), sh.launch(), sums, best_cost, fits);
    if (rest_cost < best_cost) { best = rest; best_cost = rest_cost; }
    for (int ns = 2; ns <= 16 && ns <= p0.tiles_total; ++ns) {
        DwPlan p = p0;
        p.tiles_per_split = (p.tiles_total + ns - 1) / ns;
        p.nsplit = (p.tiles_total + p.tiles_per_split - 1) / p.tiles_per_split;  // no empty split
        if (p.nsplit != ns || !fits(p)) continue;
        const double add = sh.launch() + ns * sums;
        if ((double)items * (p.tiles_total + ns * sh.fixed()) / num_sms + add >= best_cost - 1e-9) continue;   // as in plan_rest
        const double cost = add + (ns == 2 ? plan_uneven(p, items, num_sms, sh.fixed())
                                           : (double)((items * ns + num_sms - 1) / num_sms) * (p.tiles_per_split + sh.fixed()));
        if (cost < best_cost - 1e-9) { best_cost = cost; best = p; }
    }
    best.tiles = best_cost;
    return best;
}

}  // namespace dw_detail

// The plan of a call: a pure function of its arguments, kept in a small table per thread (no lock; a shape that comes back late is
// planned again).  `followed`: the dQ/dR kernel comes next and fills the last wave, so an unsplit plan loses less there.
inline DwPlan dw_plan(const flashmhf_dims &d, int num_sms, bool followed, size_t room = SIZE_MAX) {
    struct Entry {
        int32_t B, H, S, Dh, Hkuv, E, De, num_sms, followed;
        size_t room;
        DwPlan p;
    };
    constexpr int kEntries = 256;
    static thread_local Entry table[kEntries];   // (a plan for no SMs is nobody's: zeroed entries never match)
    uint32_t h = 2166136261u;
    for (int32_t v : {d.B, d.H, d.S, d.Dh, d.Hkuv, d.E, d.De, (int32_t)followed}) h = (h ^ (uint32_t)v) * 16777619u;
    Entry &e = table[(h ^ (h >> 15)) % kEntries];
    if (e.num_sms != num_sms || e.followed != (int32_t)followed || e.B != d.B || e.H != d.H || e.S != d.S || e.Dh != d.Dh || e.Hkuv != d.Hkuv ||
        e.E != d.E || e.De != d.De || e.room != room)
        e = Entry{d.B, d.H, d.S, d.Dh, d.Hkuv, d.E, d.De, num_sms, (int32_t)followed, room, dw_detail::make_plan(d, num_sms, followed, room)};
    return e.p;
}

}  // namespace
}  // namespace fmhf
