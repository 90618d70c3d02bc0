/*
 * resident_plan.cu -- which tiles of a job run on the chip, in which groups
 * of blocks, and in which order.
 */
#include "resident_geom.cuh"

#include <algorithm>
#include <cmath>

namespace cuphu {
namespace {

/* how a tile may be split: members (with items: nact) and the most items of
 * one of them */
struct Shape {
    int g = 0, a = 0, b = 0, rcols = 0;
    int nmem = 0, nact = 0, most = 0;
    bool ok() const { return nact > 0; }
};

/* FP64: the smallest group of 2^g members that keeps to k items per block */
Shape slots_shape(int nitems, int k, int nblk)
{
    Shape s;
    for (int g = 3; g <= kResMaxG; ++g) {
        int most = 0, nact = 0;
        for (int m = 0; m < (1 << g); ++m) {
            const int n = res_count(nitems, m, g);
            most = std::max(most, n);
            nact += n > 0;
        }
        if (most > k || nact > nblk) continue;
        s.g = g;
        s.nmem = 1 << g;
        s.nact = nact;
        s.most = most;
        break;
    }
    return s;
}

/* mixed: the region of at most k items that needs the fewest blocks, then the
 * one with the shortest rim */
Shape region_shape(const TileDesc &T, int k, int nblk)
{
    const int nby = T.nitems / T.nbx;
    Shape s;
    int best_rim = 0;
    for (int b = 1; b <= kResMaxB && b <= T.nbx; ++b)
        for (int a = 1; a * b <= k && a <= nby; ++a) {
            const int rrows = (nby + a - 1) / a, rcols = (T.nbx + b - 1) / b, n = rrows * rcols;
            if (n > std::min(nblk, kResMaxBlocks)) continue;
            const int rim = 16 * a + 64 * b;
            if (s.ok() && (n > s.nact || (n == s.nact && rim >= best_rim))) continue;
            s.a = a;
            s.b = b;
            s.rcols = rcols;
            s.nmem = s.nact = n;
            s.most = a * b;
            best_rim = rim;
        }
    return s;
}
}  // namespace

/* Choose the splits and the schedule.  An iteration of a tile costs about c0 +
 * c1 x (most items of one block): c0 the exchanges, c1 one item (measured, in
 * us).  Small groups spread the exchange over more work per block and let many
 * tiles run side by side; large ones shorten a tile's iteration.  The bound k
 * on the items of a block that gives the smallest estimated makespan over the
 * job's tiles is taken.  Tiles that no group holds (above 16 items for each
 * of the GPU's SMs in mixed precision, 1024 items in FP64) are streamed. */
void plan_resident(const std::vector<TileDesc> &tiles, int nblk, bool fp64, ResidentPlan &R)
{
    const int cap = fp64 ? kResItems64 : kResItemsMixed;
    const double c0 = fp64 ? 4.8 : 2.4, c1 = fp64 ? 0.78 : 0.42;
    R = ResidentPlan();
    /* the split of tile t under the bound k, or the nearest one above it */
    auto shape = [&](int t, int k) {
        Shape s;
        for (; k <= cap && !s.ok(); ++k)
            s = fp64 ? slots_shape(tiles[t].nitems, k, nblk) : region_shape(tiles[t], k, nblk);
        return s;
    };
    auto cost = [&](int t, const Shape &s) {
        return std::sqrt((double)tiles[t].nitems) * (c0 + c1 * s.most);
    };
    std::vector<int> fit;
    for (int t = 0; t < (int)tiles.size(); ++t)
        if (shape(t, cap).ok()) fit.push_back(t);
        else R.streamed.push_back(t);
    if (fit.empty()) return;
    int best_k = cap;
    double best = 0.0;
    for (int k = 1; k <= cap; ++k) {
        double area = 0.0, longest = 0.0;
        for (int t : fit) {
            const Shape s = shape(t, k);
            const double d = cost(t, s);
            area += d / (nblk / s.nact);   /* groups that do not pack waste what is left over */
            longest = std::max(longest, d);
        }
        const double est = std::max(area, longest);
        if (k == 1 || est < best) {
            best = est;
            best_k = k;
        }
    }
    struct Job { int t; Shape s; double d; };
    std::vector<Job> jobs;
    for (int t : fit) {
        const Shape s = shape(t, best_k);
        jobs.push_back({t, s, cost(t, s)});
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
        const double start = load[idx[j.s.nact - 1]];
        const int sched = (int)R.sched.size();
        R.sched.push_back({j.t, j.s.nmem, j.s.nact, (int)R.phys.size(), j.s.g, j.s.a, j.s.b,
                           j.s.rcols});
        int used = 0;
        for (int m = 0; m < j.s.nmem; ++m) {
            if (fp64 && res_count(tiles[j.t].nitems, m, j.s.g) == 0) {
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

/* rim packets: FP64 16 bytes for the ring of each item, mixed 8 bytes for the
 * four sides of a region (256 pixels each), two buffers */
size_t resident_rim_bytes(int nblk, bool fp64)
{
    return fp64 ? (size_t)nblk * kResItems64 * 2 * (2 * kItemBx + 2 * kItemBy) * 16
                : (size_t)nblk * 2 * 4 * 256 * 8;
}
size_t resident_mail_bytes(int nblk, bool fp64)
{
    return (size_t)nblk * 2 * (fp64 ? 4 * kResMembers : kNComp * kResMaxBlocks) * sizeof(ulonglong2);
}

}  // namespace cuphu
