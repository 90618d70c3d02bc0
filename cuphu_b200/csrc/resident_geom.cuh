/*
 * resident_geom.cuh -- how a tile's items are split over a group of blocks.
 */
#pragma once

#include "resident.cuh"

namespace cuphu {

/* ── geometry of a group ───────────────────────────────────────────────────
 * u = the slot's bits in the order the tree combines them (lane bits 4..0,
 * then warp bits 2..0); member = the low g bits of u, sub = the rest.  Local
 * items are numbered level by level (items 256 j + slot), and the last,
 * partial level is a prefix of the subs (res_last). */
__host__ __device__ __forceinline__ int res_slot(int u) { return ((u >> 3) & 31) | ((u & 7) << 5); }
__host__ __device__ __forceinline__ int res_u(int slot) { return ((slot & 31) << 3) | (slot >> 5); }
/* subs of member m that hold an item in a last level of `rem` items */
__host__ __device__ __forceinline__ int res_last(int rem, int m, int g)
{
    const int lanes = rem - 32 * (m & 7);          /* lanes of this warp in use */
    const int hi = m >> 3, step = g - 3;
    if (lanes <= hi) return 0;
    const int l = lanes < 32 ? lanes : 32;
    return (l - hi + (1 << step) - 1) >> step;
}
__host__ __device__ __forceinline__ int res_count(int nitems, int m, int g)
{
    return ((nitems >> 8) << (8 - g)) + res_last(nitems & 255, m, g);
}

}  // namespace cuphu
