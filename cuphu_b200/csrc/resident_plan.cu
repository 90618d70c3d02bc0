/*
 * resident_plan.cu -- which tiles of a job run on the chip, in which groups
 * of blocks, and in which order.
 */
#include "resident_geom.cuh"

#include <algorithm>
#include <cmath>

namespace cuphu {

/* most items any block of a group of 2^g holds */
static int res_most(int nitems, int g)
{
    int most = 0;
    for (int m = 0; m < (1 << g); ++m) most = std::max(most, res_count(nitems, m, g));
    return most;
}

/* Choose the group sizes and the schedule.  An iteration of a tile costs about
 * c0 + c1 x (most items of one block): c0 the exchange, c1 one item (both
 * measured, in us).  Small groups spread the exchange over more work per block
 * and let many tiles run side by side; large ones shorten a tile's
 * iteration.  The bound k on the items of a block that gives the smallest
 * estimated makespan over the job's tiles is taken.  Tiles that no group holds
 * (above 1792 items in mixed precision, 1024 in FP64) are streamed. */
void plan_resident(const std::vector<TileDesc> &tiles, int nblk, bool fp64, ResidentPlan &R)
{
    const int cap = fp64 ? kResItems64 : kResItemsMixed;
    const double c0 = fp64 ? 5.0 : 3.8, c1 = 0.6;
    R = ResidentPlan();
    std::vector<int> fit;
    for (int t = 0; t < (int)tiles.size(); ++t)
        if (res_most(tiles[t].nitems, kResMaxG) <= cap && nblk >= (1 << kResMaxG)) fit.push_back(t);
        else R.streamed.push_back(t);
    if (fit.empty()) return;
    auto shape = [&](int nitems, int k, int &g, int &most) {
        for (g = 3; g < kResMaxG; ++g)
            if ((most = res_most(nitems, g)) <= k) return;
        most = res_most(nitems, g);
    };
    auto active = [&](int nitems, int g) {
        int a = 0;
        for (int m = 0; m < (1 << g); ++m) a += res_count(nitems, m, g) > 0;
        return a;
    };
    int best_k = cap;
    double best = 0.0;
    for (int k = 1; k <= cap; ++k) {
        double area = 0.0, longest = 0.0;
        for (int t : fit) {
            int g, most;
            shape(tiles[t].nitems, k, g, most);
            const int a = active(tiles[t].nitems, g);
            const double d = std::sqrt((double)tiles[t].nitems) * (c0 + c1 * most);
            /* groups that do not pack waste the blocks left over */
            area += d / (nblk / a);
            longest = std::max(longest, d);
        }
        const double est = std::max(area, longest);
        if (k == 1 || est < best) {
            best = est;
            best_k = k;
        }
    }
    struct Job { int t, g, a; double d; };
    std::vector<Job> jobs;
    for (int t : fit) {
        int g, most;
        shape(tiles[t].nitems, best_k, g, most);
        jobs.push_back({t, g, active(tiles[t].nitems, g),
                        std::sqrt((double)tiles[t].nitems) * (c0 + c1 * most)});
    }
    std::stable_sort(jobs.begin(), jobs.end(), [](const Job &a, const Job &b) { return a.d > b.d; });
    /* longest first onto the blocks that are free first; blocks process
     * their tiles in this order, so the first unfinished tile of the order
     * always has all its blocks */
    std::vector<double> load(nblk, 0.0);
    std::vector<std::vector<ResWork>> per(nblk);
    std::vector<int> idx(nblk);
    for (const Job &j : jobs) {
        for (int b = 0; b < nblk; ++b) idx[b] = b;
        std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return load[a] < load[b]; });
        const double start = load[idx[j.a - 1]];
        const int sched = (int)R.sched.size();
        R.sched.push_back({j.t, j.g, j.a, (int)R.phys.size()});
        int used = 0;
        for (int m = 0; m < (1 << j.g); ++m) {
            if (res_count(tiles[j.t].nitems, m, j.g) == 0) {
                R.phys.push_back(0xffff);
                continue;
            }
            const int b = idx[used++];
            R.phys.push_back((unsigned short)b);
            per[b].push_back({sched, m});
            load[b] = start + j.d;
        }
    }
    R.blk_off.push_back(0);
    for (int b = 0; b < nblk; ++b) {
        R.work.insert(R.work.end(), per[b].begin(), per[b].end());
        R.blk_off.push_back((int)R.work.size());
    }
    /* blocks without work at the end of the grid are not launched */
    R.nblk = nblk;
    while (R.nblk > 1 && per[R.nblk - 1].empty()) --R.nblk;
}

constexpr size_t kRimPx = 2 * kItemBx + 2 * kItemBy;   /* rim packets of an item, per buffer */
size_t resident_rim_bytes(int nblk, bool fp64)
{
    return fp64 ? (size_t)nblk * kResItems64 * 2 * kRimPx * 16
                : (size_t)nblk * kResItemsMixed * 2 * kRimPx * 8;
}
size_t resident_mail_bytes(int nblk)
{
    return (size_t)nblk * 2 * kNComp * kResMembers * sizeof(ulonglong2);
}

}  // namespace cuphu
