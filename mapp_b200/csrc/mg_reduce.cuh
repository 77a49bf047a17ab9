// Warp / block reduction helpers shared by the force-field kernels.
#pragma once

#include "mg_internal.h"

namespace mg {

constexpr int kFFBlock = 256;           // threads per force-field block (8 warps)
constexpr int kFFWarps = kFFBlock / 32;

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float warp_sumf(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over an aligned group of G lanes (G = 8, 16 or 32) of one warp; every
// lane of the group must call it (other groups of the warp may be elsewhere).
template <int G>
__device__ __forceinline__ double group_sum(double v)
{
    const unsigned mask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31) & ~(G - 1)));
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
    return v;
}

// Lanes of a warp that hold the same key: pairs are sorted by their first
// site, so equal keys are contiguous lanes [first, last].
struct Seg {
    int first, last;
};

__device__ __forceinline__ Seg seg_of(int key)
{
    unsigned m = __match_any_sync(0xffffffffu, key);
    Seg s;
    s.first = __ffs(m) - 1;
    s.last = 31 - __clz(m);
    return s;
}

// Sum of v over the lanes of the caller's segment, returned in the segment's
// first lane (every lane of the warp must call it).
__device__ __forceinline__ double seg_sum(double v, const Seg& s)
{
    int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        double t = __shfl_down_sync(0xffffffffu, v, o);
        if (lane + o <= s.last) v += t;
    }
    return v;
}

// Segments of a warp whose keys are sorted (equal keys in contiguous lanes,
// padding lanes with key -1 at the end): boundaries from one shuffle and one
// ballot instead of a match instruction.
__device__ __forceinline__ Seg seg_sorted(int key)
{
    const int lane = threadIdx.x & 31;
    const int prev = __shfl_up_sync(0xffffffffu, key, 1);
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || prev != key);
    const unsigned upto = heads & (0xffffffffu >> (31 - lane));  // heads at or before this lane
    const unsigned after = heads & ~(0xffffffffu >> (31 - lane));
    Seg sg;
    sg.first = 31 - __clz(upto);
    sg.last = after ? __ffs(after) - 2 : 31;
    return sg;
}

// Sums of NV values per lane over a warp's pairs, through a shared-memory
// buffer of the warp's own (RowBuf<NV>): rows_put writes the values (and each
// lane's run key: the pairs' first site, equal keys in contiguous lanes, -1 for
// none; only for rows_runs) and rows_scatter / rows_runs add them up, calling
// put(row, q, x) for value q of row `row` (an atomic add).  One L1 data-stage
// cycle goes to every shuffle and to every distinct line of a reduction:
//  - rows_scatter: one row per lane.  NV reductions of 32 rows each would touch
//    32 NV lines; with consecutive lanes on consecutive values of a row they
//    touch about 32 + NV.
//  - rows_runs: the sums of the runs of equal keys.  NV segmented shuffle sums of
//    doubles take 10 NV shuffles; here a lane sums COLS consecutive pairs of one
//    value and only the runs' ends are shuffled.
template <int NV>
struct RowBuf {
    static constexpr int COLS = NV <= 2 ? 2 : (NV <= 4 ? 4 : 8);  // lanes side by side on a pair's values
    static constexpr int PITCH = NV | 1;                          // odd: no bank conflicts
    double v[32 * PITCH];
    int key[32];
};

template <int NV>
__device__ __forceinline__ void rows_put(RowBuf<NV>& b, const double (&v)[NV], int key)
{
    const int lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NV; q++) b.v[lane * RowBuf<NV>::PITCH + q] = v[q];
    b.key[lane] = key;
    __syncwarp();
}

template <int NV, typename Put>
__device__ __forceinline__ void rows_scatter(const RowBuf<NV>& b, int row, Put put)
{
    const int lane = threadIdx.x & 31;
    if (!__any_sync(0xffffffffu, row >= 0)) return;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        const int e = k * 32 + lane, src = e / NV, q = e - src * NV;
        const int r = __shfl_sync(0xffffffffu, row, src);
        const double x = b.v[src * RowBuf<NV>::PITCH + q];
        if (r >= 0 && x != 0.0) put(r, q, x);
    }
}

template <int NV, typename Put>
__device__ __forceinline__ void rows_runs(const RowBuf<NV>& b, Put put)
{
    constexpr int COLS = RowBuf<NV>::COLS;
    const int lane = threadIdx.x & 31, q = lane % COLS, p0 = (lane / COLS) * COLS;
    int cur = b.key[p0];
    double s = 0.0;
#pragma unroll
    for (int t = 0; t < COLS; t++) {
        const int k = b.key[p0 + t];
        if (k != cur) {
            if (q < NV && cur >= 0 && s != 0.0) put(cur, q, s);
            s = 0.0;
            cur = k;
        }
        if (q < NV) s += b.v[(p0 + t) * RowBuf<NV>::PITCH + q];
    }
    // the ends of the COLS-pair stretches, joined over stretches of one run
#pragma unroll
    for (int o = COLS; o < 32; o <<= 1) {
        const double t = __shfl_down_sync(0xffffffffu, s, o);
        const int k = __shfl_down_sync(0xffffffffu, cur, o);
        if (lane + o < 32 && k == cur) s += t;
    }
    const int prev = __shfl_up_sync(0xffffffffu, cur, COLS);
    if (q < NV && cur >= 0 && (lane < COLS || prev != cur) && s != 0.0) put(cur, q, s);
}

// Batched form: is the cell of owned site i still being evaluated?
__device__ __forceinline__ bool site_active(const Dev& d, int i)
{
    return d.cell_active == nullptr || d.cell_active[d.site_cell[i]] != 0;
}

// Batched form: adds e (this lane's energy term of owned site i; i < 0 for a
// lane without one) to the energy of i's cell, one atomic per run of equal
// cells in the warp (sites and pairs are numbered cell by cell).  Every lane
// of the warp must call it.
__device__ __forceinline__ void cell_energy_add(const Dev& d, int i, double e)
{
    const int cell = i >= 0 ? d.site_cell[i] : -1;
    const Seg s = seg_of(cell);
    const double t = seg_sum(e, s);
    if (cell >= 0 && (int)(threadIdx.x & 31) == s.first && t != 0.0) atomicAdd(&d.cell_E[cell], t);
}

// Persistent grid size for a force kernel: enough blocks to fill every SM at
// the kernel's resident-block count, never more than the work needs.
inline int persistent_grid(long long threads_needed, int blocks_per_sm)
{
    long long need = (threads_needed + kFFBlock - 1) / kFFBlock;
    long long cap = (long long)num_sms() * blocks_per_sm;
    return (int)(need < cap ? (need > 0 ? need : 1) : cap);
}

// Sums NV per-thread values over the block (up to 1024 threads) and writes them to
// partial[(row) * 8 + v] (row = blockIdx.x + row_offset).  Every thread of the
// block must call it.
template <int NV>
__device__ __forceinline__ void block_partials(const double (&vals)[NV], double* partial, int row)
{
    __shared__ double sh[32][8];  // up to 1024 threads
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int v = 0; v < NV; v++) {
        double s = warp_sum(vals[v]);
        if (lane == 0) sh[w][v] = s;
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double s = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) s += sh[k][threadIdx.x];
        partial[(size_t)row * 8 + threadIdx.x] = s;
    }
}

}  // namespace mg
