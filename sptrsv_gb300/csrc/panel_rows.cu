// panel_rows.cu -- exact FP64 products over dense panels, one warp per four rows (the batched path and
// the single-system supernodal path).
//
// Row r of a chunk is one dot product, x_r = G_r [b_own ; x_rect] (supernodal.cu), and the chunks of a
// path form a chain, so what a chunk costs is the way from the last x it waits for to the first of its
// own that the next chunk can read.  A warp therefore takes four rows whole and publishes them itself:
// no partial sums, counters or fences between SMs lie on that way.  Lanes take the columns 32 at a time
// -- the chunk's own right-hand side first, from the rows' diagonal on, then the solved columns from the
// farthest to the nearest, so that only the last few wait -- and hold the sums of four rows by up to four
// right-hand sides, added across the lanes at the end.  G is read straight into registers, coalesced, for
// U steps at once, with their right-hand sides; solved columns' indices one such group ahead.  A poll
// reads again all of the group's values that are pending, and a step is multiplied as soon as its own are
// there, so that a chunk's columns cost one latency of L2 (or of HBM, for its G) a group, not one each.
// The order of additions is fixed, so results do not depend on timing.
//
// Items are taken from a ticketed queue in an order in which every item waits on smaller tickets only; a
// warp draws its next ticket before it works on the one in hand, and works on them in order, so the
// smallest unfinished ticket is always being worked on.
//
// An FP64 operation holds its SM quarter's pipe for 64 cycles: a chunk of 256 rows after one of 256 costs
// a warp 8 steps of 4 products (one right-hand side) or 8 (two), ~1 or ~2 us.  U = 4 and 2 for them, 2 and 1
// where registers are few.  Bands of 64 / 128 / 181 / 256 with one right-hand side, against one step read
// ahead: 50 / 201 / 619 / 1994 -> 39 / 139 / 369 / 864 us (U = 2: 1071 at 256; own and solved columns in
// one group 63 / 213 / 541 / 1231, its first products held up by the wait), the 40^3 factor 183 -> 159 us.
// Four right-hand sides to a warp read G half as often, 2 % faster on the 40^3 factor with 32 columns and
// slower everywhere else (24^3 x 3 99 -> 154 us, 64 x 64 band x 3 79 -> 106 us); one to a warp 40 % slower
// there.  Five CTAs an SM (96 registers): 3 / 4 / 5 / 6 / 8 took 2.09 / 1.77 / 1.72 / 1.73 / 1.81 ms on 40^3 x 32.
//
// Measured on GB300 against column blocks of 64-row panels with partial sums in global memory: the 40^3
// dissection factor with 1 / 32 right-hand sides 538 / 4282 -> 156 / 1680 us (the last is 77 % of the FP64
// rate), the 64 x 64 band factor 99 -> 39 us (a chain of 16 steps of ~2 us).
#include <algorithm>
#include "common.cuh"
#include "batch.cuh"

namespace sptrsv {

constexpr int kRowsItem = kPanelRows;  // rows of an item

// Rows [r, r + nr) of the chunk by right-hand sides [c0, c0 + NC), U steps of 32 columns at a time.
template <int NC, int U>
__device__ __forceinline__ bool rows_item(const BChunk& C, int r, int nr, int m, int c0,
                                          const double* __restrict__ b, double* x, Ctl* ctl, int64_t budget) {
    constexpr int R = kRowsItem;
    const int lane = threadIdx.x & 31;
    const int w = C.w, M = C.m;
    const double* g[R];
#pragma unroll
    for (int i = 0; i < R; ++i) g[i] = C.g64 + (size_t)(r + min(i, nr - 1)) * C.ld;
    const int n_own = (w - r + 31) >> 5, n_all = n_own + ((M + 31) >> 5);
    double acc[R * NC];
#pragma unroll
    for (int q = 0; q < R * NC; ++q) acc[q] = 0.0;
    double gv[U][R], v[U][NC];
    int at[U];
    auto load_g = [&](int u, int k) {
#pragma unroll
        for (int i = 0; i < R; ++i) gv[u][i] = k >= 0 ? __ldg(g[i] + k) : 0.0;
    };
    auto multiply = [&](int u) {
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < NC; ++j) acc[i * NC + j] = fma(gv[u][i], v[u][j], acc[i * NC + j]);
    };
    // solved columns, from the farthest; the lane's column of step s (-1: none) and its row of x
    auto column = [&](int s) -> int {
        const int k = 32 * (n_all - 1 - s) + lane;
        return s < n_all && k < M ? w + k : -1;
    };
    auto row = [&](int s) -> int {
        const int k = column(s);
        return k < 0 ? -1 : C.rect[k - w];
    };
#pragma unroll
    for (int u = 0; u < U; ++u) at[u] = row(n_own + u);
    for (int s = 0; s < n_own; s += U) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = r + 32 * (s + u) + lane;
            load_g(u, k < w ? k : -1);
#pragma unroll
            for (int j = 0; j < NC; ++j) v[u][j] = k < w ? __ldg(b + (size_t)(C.a + k) * m + c0 + j) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (s + u < n_own) multiply(u);
    }
    for (int s = n_own; s < n_all; s += U) {
        int next[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            load_g(u, column(s + u));
#pragma unroll
            for (int j = 0; j < NC; ++j) v[u][j] = at[u] >= 0 ? ld_relaxed(x + (size_t)at[u] * m + c0 + j) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) next[u] = row(s + U + u);
        uint64_t t0 = 0;
        unsigned q = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (s + u >= n_all) break;
            for (;; ++q) {
                bool pend = false;
#pragma unroll
                for (int j = 0; j < NC; ++j) pend |= at[u] >= 0 && Pend<double>::is(v[u][j]);
                if (!__any_sync(0xffffffffu, pend)) break;
                if (q >= 4) __nanosleep(q < 256 ? 20 : 100);
                if ((q & 63u) == 63u) {
                    bool ok = !aborted(ctl);
                    if (t0 == 0) t0 = gtimer();
                    else if (ok && (int64_t)(gtimer() - t0) > budget) {
                        record_error(ctl, SPTRSV_ERR_TIMEOUT);
                        ok = false;
                    }
                    if (!__all_sync(0xffffffffu, ok)) return false;
                }
#pragma unroll
                for (int z = u; z < U; ++z)
#pragma unroll
                    for (int j = 0; j < NC; ++j)
                        if (at[z] >= 0 && Pend<double>::is(v[z][j])) v[z][j] = ld_relaxed(x + (size_t)at[z] * m + c0 + j);
            }
            multiply(u);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) at[u] = next[u];
    }
    // sums across the lanes: halves exchanged while a lane holds more than one, so R * NC + log2 additions
    // in all; lane l ends with sum (l >> shift)
    int off = 16;
#pragma unroll
    for (int half = R * NC / 2; half >= 1; half >>= 1) {
        const bool upper = lane & off;
#pragma unroll
        for (int q = 0; q < half; ++q) {
            const double give = upper ? acc[q] : acc[q + half];
            const double keep = upper ? acc[q + half] : acc[q];
            acc[q] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
        off >>= 1;
    }
    constexpr int kShift = R * NC == 8 ? 2 : 3;  // lanes per sum, as a shift
    for (; off >= 1; off >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], off);
    const int q = lane >> kShift, i = q / NC, j = q % NC;
    if ((lane & ((1 << kShift) - 1)) == 0 && i < nr)
        st_relaxed(x + (size_t)(C.a + r + i) * m + c0 + j, Pend<double>::fix(acc[0]));
    return true;
}

// kBeside: for running beside other kernels (the batch's refinement), whose CTAs need registers next to four
// of this one's: 64 a thread instead of 92 (512-system mix 109.9 -> 92.6 ms, 48 systems 1.92 -> 1.44 ms;
// alone 5 % slower).
//
// Batched (sys != nullptr): items[t] = {panel, rows / 4 | group << 8}, one per ticket.  One system
// (sys == nullptr, `rhs` columns): ticket t is group t % ncg of items[t / ncg].
template <bool kBeside>
__global__ void __launch_bounds__(128, kBeside ? 8 : 5) k_panel_rows(const BSys* __restrict__ sys, int rhs, int ncg,
                                                       const double* __restrict__ bbase, double* xbase, Ctl* ctl,
                                                       unsigned* ticket, int64_t budget,
                                                       const int2* __restrict__ items, unsigned ntickets,
                                                       const BChunk* __restrict__ panels) {
    const int lane = threadIdx.x & 31;
    unsigned next = 0;
    if (lane == 0) next = atomicAdd(ticket, 1u);
    for (;;) {
        const unsigned t = __shfl_sync(0xffffffffu, next, 0);
        if (t >= ntickets || aborted(ctl)) break;
        if (lane == 0) next = atomicAdd(ticket, 1u);
        int2 it;
        int cg;
        if (sys) {
            it = items[t];
            cg = it.y >> 8;
            it.y &= 0xFF;
        } else {
            it = items[t / ncg];
            cg = (int)(t % ncg);
        }
        const BChunk C = panels[it.x];
        const int m = sys ? sys[C.sys].rhs : rhs;
        const long long xb0 = sys ? sys[C.sys].xb0 : 0;
        const int c0 = cg * kPanelCols, nc = min(kPanelCols, m - c0);
        const int r = C.r0 + it.y * kRowsItem, nr = min(kRowsItem, C.r0 + C.pw - r);
        const double* b = bbase + xb0;
        double* x = xbase + xb0;
        bool ok;
        if (nc == 1) ok = rows_item<1, kBeside ? 2 : 4>(C, r, nr, m, c0, b, x, ctl, budget);
        else ok = rows_item<kPanelCols, kBeside ? 1 : 2>(C, r, nr, m, c0, b, x, ctl, budget);
        if (!ok) break;
    }
}

int launch_panel_rows(const BSys* sys, int rhs, const double* b, double* x, Ctl* ctl, unsigned* ticket, int64_t budget,
                      const int2* items, unsigned nitems, const BChunk* panels, int ctas_per_sm, int sm_count,
                      cudaStream_t st, int64_t* launches) {
    if (!nitems) return 0;
    const int ncg = sys ? 1 : panel_groups(rhs);
    const unsigned ntickets = nitems * (unsigned)ncg;
    // The kernel uses no shared memory, but kernels that do run beside it (the batch's refinement): an SM
    // that it has taken with an all-L1 split stays closed to them until it ends.
    const auto kernel = sys ? k_panel_rows<true> : k_panel_rows<false>;
    CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 50));
    int per_sm = 0;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 128, 0));
    per_sm = std::max(1, std::min(per_sm, ctas_per_sm));
    const int grid = (int)std::max<long long>(1, std::min<long long>((long long)per_sm * sm_count, (ntickets + 3ll) / 4));
    kernel<<<grid, 128, 0, st>>>(sys, rhs, ncg, b, x, ctl, ticket, budget, items, ntickets, panels);
    ++*launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

}  // namespace sptrsv
