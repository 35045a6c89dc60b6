// settle.cu -- the FP64 solve of a deep DAG by sweeps that run until the solution stands still.
//
// Substitution is the only fixed point of x_i <- (b_i - sum_j U_ij x_j) / U_ii: row n-1 has no other
// value, so row n-2 has none, and so on up.  Sweeping that rule over all rows at once therefore
// computes what the exact kernels compute, from any start and in any order, once the sweeps stand
// still; they do after a few dozen when U's off-diagonals are small against its diagonal, instead of
// after as many dependent hops as the DAG has levels.  A sweep reads U once at bandwidth, a hop costs
// 0.2 us on one CTA.  A matrix whose sweeps contract too slowly is given up after a few of them (see
// settle_verdict) and solved by the exact kernel launched behind this one, which returns at once
// when this one has finished (ctl->done).
//
// When it stands still: a sweep's record is the largest change of any row, relative to the largest of
// |x_i|, |b_i / U_ii| and the terms |U_ij x_j / U_ii| that row is formed from.  The change is not the
// error: with a rate rho a sweep, rho / (1 - rho) of it is left, as much as the change itself at one bit a
// sweep.  So the rate is read from the records where contraction rules them (2^-40; from 2^-48 on,
// rounding flips keep a few hundred rows of millions moving by a few ulps for as many sweeps again), and
// the sweeps go on until what is left at that rate is below 2^-54, half the rounding of one term.
// Emulated on the CPU against 80-bit solutions, 20,000 rows, error in norm as a multiple of
// substitution's: chains x_i = b_i + w x_i+1 with w = 0.3 / 0.5 / 0.6 / 0.7 / 0.8 1.01 / 1.00 / 1.12 / 1.08 /
// 1.14 with one right-hand side (stopped at a record of 2^-48: 1.0 / 1.1 / 1.4 / 1.7 / 5.1), 1.00 or left to
// the exact kernel with several (1.0 / 1.9 / 3.6 / 5.2 / 9.7); two entries of 0.35 0.93 (4.8 and 11), eight
// of 0.075 0.68 (1.2 and 2.9), the random recipe 0.71 (0.71: it gains four bits a sweep).
//
// Sweep order.  Each warp owns a contiguous run of rows and walks it upwards from its bottom, 32 rows
// a tile (lane per row; 32 / NC rows for NC right-hand sides): a row sees this sweep's values of
// everything below it in the run, so only columns inside the tile, across the run's lower edge and far
// away are one sweep old.  Those inside the tile are a quarter of a 64-column band
// and cost the most sweeps, so with one right-hand side a tile's changes are folded in once more
// before they are written (k_settle, "second look"): half the sweeps for a third more arithmetic.
//
// Repeatability.  With several right-hand sides the exact kernel (a warp per row) gives the same bits every
// time, and so do the sweeps: they go from one vector to another, and a row outside the run is always the
// last sweep's.  With one, the exact kernel's last bits follow its timing (the window kernel's rows split
// their sums where they have to wait), and x is swept in place: another run's row may be this sweep's or
// the last one's, a few sweeps fewer (2M rows 15, 20 with two vectors), and the result differs by roundings
// from solve to solve.  Two vectors cost, 8.8 entries a row: 2k rows x 8 233 -> 274 us, 10k x 2 307 -> 371,
// 50k x 8 542 -> 740, 200k x 8 1,288 -> 1,418 (of it about a sweep for the stop above).
//
// Bound by the FP64 pipe (57 % active by ncu at 500k rows; an operation holds its SM quarter's pipe for 64
// cycles, and a tile takes its longest row's count, 1.9 times the mean of 7.6 off-diagonals) and, below
// ~200k rows, by the chain of loads and FMAs through a tile.  Measured on GB300, 8.8 entries a row: 2M rows
// 68 -> 1.87 ms (16 sweeps of 116 us), 200k rows 6.9 -> 0.45 ms (20), 50k rows 1.7 -> 0.29 ms (20), 10k rows
// 0.37 -> 0.23 ms (34 of 6 us); 200k rows x 8 columns 70 -> 1.52 ms (27).  Tried and not kept: two FP32 corrections first (their sweeps are bound by instructions
// and L1, 90 us against 120 at 2M rows: 3.4 ms in all against 3.1 then), rows kept in shared memory for all
// sweeps (200k rows 0.40, but 200k x 8 1.69), 16-byte copies for the staging (no change).
//
// One cooperative launch runs all sweeps, with a grid barrier after each.
#include <algorithm>
#include <cmath>
#include "common.cuh"
#include "kernels.cuh"

namespace sptrsv {

constexpr int kSetWarps = 8;
constexpr size_t kSetSmem = 220 * 1024;
constexpr int kSetPending = 5000;  // offset of a sweep's record: 0 = nothing changed
constexpr int kSetRated = kSetPending - 40;  // the rate is read at the first record at or below
constexpr int kSetStill = kSetPending - 49;  // changes below 2^-48 (the exponents are floors)
constexpr float kSetLeft = -54.f;            // what may be left when the sweeps end

struct SettleArgs {
    int n, rhs;
    const int* rp;
    const int* col;
    const double* val;
    const double* invd;
    const double* b;
    double* x;
    double* y;   // several right-hand sides: the other vector
    Ctl* ctl;
    int* worst;  // kSettleSweeps records: the largest change of each sweep, as an exponent
    int64_t budget;
    int most;   // sweeps, up to kSettleSweeps
    int tiles;  // tiles per warp
    int cap;    // staged entries of a tile; a tile with more is read from global memory
};

template <int NC> struct SetShape {
    static constexpr int kRows = 32 / NC;  // rows of a tile
    static constexpr bool kPair = NC > 1;  // two vectors
    // One right-hand side: a tile's buffer at a time and three CTAs an SM (2M rows 1.81 ms; two buffers and
    // two CTAs 2.11, one and two 2.11, one and four 2.14).  Several: two buffers, two CTAs (200k rows x 8
    // 1.35 ms; one and three 1.42).
    static constexpr int kBufs = NC == 1 ? 1 : 2;
    static constexpr int kCtas = NC == 1 ? 3 : 2;
};

// Bytes of a warp's buffers: one or two tiles of `cap` staged entries (columns and values), one tile's x at
// every entry (cap * NC), the tile's changes.
__host__ __device__ __forceinline__ size_t set_warp_bytes(int cap, int nc, int bufs) {
    return (size_t)cap * (bufs * 12 + 8 * nc) + 32 * 8;
}

__device__ __forceinline__ int d_exp(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }

// Exponent of |a - b|, a != b, within one, from their bits (an FP64 subtraction would hold the pipe for 64
// cycles): bit patterns of one sign are ordered like the values and a unit in the last place apart; with
// the signs or the exponents further apart the larger value's exponent.
__device__ __forceinline__ int d_gap(double a, double b) {
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    const int ea = d_exp(a), eb = d_exp(b), hi = max(ea, eb), lo = min(ea, eb);
    if ((x ^ y) < 0 || hi - lo > 1) return hi;
    return lo - 52 + 63 - __clzll(x > y ? x - y : y - x);
}

// After sweep p (from 0), of at most `most`: 0 go on, 1 the solution stands still, 2 leave the matrix to
// the exact kernel.  `last`: the sweep after which what is left is small enough, -1 until the rate is read
// (over the last four and eight sweeps, the slower one).  Until then, from the ninth sweep on, the faster
// one has to get there within `most`.
__device__ __forceinline__ int settle_verdict(const int* worst, int p, int most, int& last) {
    const int now = ld_relaxed(worst + p);
    if (now <= 0) return 1;  // no row changed
    const float size = (float)(now - kSetPending);
    auto rate = [&](int back) { return (float)(ld_relaxed(worst + p - min(back, p)) - now) / (float)min(back, p); };
    if (last < 0 && now <= kSetRated) {
        const float g = p == 0 ? 1.f : fmaxf(0.05f, fminf(rate(4), rate(8)));  // bits a sweep
        last = p + max(0, (int)ceilf((size + 1.f - log2f(exp2f(g) - 1.f) - kSetLeft) / g));
    }
    if (last >= 0) {
        if (p >= last && now <= kSetStill) return 1;
        return last < most ? 0 : 2;
    }
    if (p < 8) return 0;
    const float g = fmaxf(rate(4), rate(8));
    return g > 0.f && (float)p + (size - kSetLeft) / g <= (float)most ? 0 : 2;
}

__device__ __forceinline__ void set_cp4(void* s, const void* g) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(s);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(a), "l"(g) : "memory");
}
__device__ __forceinline__ void set_cp8(void* s, const void* g) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(s);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(a), "l"(g) : "memory");
}

// x changes within the launch, so never the read-only path: rows that no other warp writes in this sweep
// through L1 (a warp's own stores update it), other rows from L2, where this sweep's values are.
__device__ __forceinline__ double set_ld(const double* p, bool still) {
    double v;
    if (still) asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    else asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}

template <int NC>
__global__ void __launch_bounds__(kSetWarps * 32, SetShape<NC>::kCtas) k_settle(SettleArgs A) {
    constexpr int R = SetShape<NC>::kRows, B = SetShape<NC>::kBufs;
    constexpr bool kPair = SetShape<NC>::kPair;
    extern __shared__ __align__(16) char set_smem[];
    __shared__ int s_worst;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = lane / NC, j0 = lane % NC;
    const int n = A.n, m = A.rhs, cap = A.cap;
    char* base = set_smem + warp * set_warp_bytes(cap, NC, B);
    double* sv = (double*)base;            // [B][cap] values
    double* sx = sv + B * cap;             // [cap][NC] x at the tile's entries
    double* dl = sx + cap * NC;            // [32] the tile's changes
    int* sc = (int*)(dl + 32);             // [B][cap] columns
    const int ntiles = (n + R - 1) / R;
    const int t0 = min((int)(blockIdx.x * kSetWarps + warp) * A.tiles, ntiles), t1 = min(t0 + A.tiles, ntiles);
    const int run_top = n - R * t0;

    // x = D^-1 b
    for (int t = t0; t < t1; ++t) {
        const int top = n - R * t, lo = max(0, top - R), i = lo + r;
        if (i < top)
            for (int j = j0; j < m; j += NC) A.x[(size_t)i * m + j] = A.b[(size_t)i * m + j] * A.invd[i];
    }
    if (!grid_barrier(A.ctl, gridDim.x, A.budget)) return;

    struct Rows { int e0, e1, s, e; };
    auto rows_of = [&](int t) {
        Rows q{0, 0, 0, 0};
        if (t < t1) {
            const int top = n - R * t, lo = max(0, top - R);
            q.e0 = A.rp[lo];
            q.e1 = A.rp[top];
            if (lo + r < top) {
                q.s = A.rp[lo + r] + 1;
                q.e = A.rp[lo + r + 1];
            }
        }
        return q;
    };
    auto stage = [&](const Rows& q, int buf) {
        const int cnt = q.e1 - q.e0;
        if (cnt <= cap)
            for (int k = lane; k < cnt; k += 32) {
                set_cp4(sc + buf * cap + k, A.col + q.e0 + k);
                set_cp8(sv + buf * cap + k, A.val + q.e0 + k);
            }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };

    int last = -1;
    for (int p = 0; p < A.most; ++p) {
        if (threadIdx.x == 0) s_worst = 0;
        __syncthreads();
        int worst = 0;
        const double* const src = kPair && (p & 1) ? A.y : A.x;
        double* const dst = kPair && !(p & 1) ? A.y : A.x;
        // x of a column of a tile that ends at row `top`: this sweep's in the rest of the run
        auto x_of = [&](int c, int top, int j) {
            const size_t k = (size_t)c * m + j;
            if constexpr (kPair) return set_ld((c >= top && c < run_top ? dst : src) + k, true);
            else return set_ld(src + k, c < run_top);
        };
        Rows cur = rows_of(t0);
        if (B == 2) stage(cur, 0);
        Rows nxt = rows_of(t0 + 1);
        for (int t = t0; t < t1; ++t) {
            const int buf = (t - t0) & (B - 1);
            const int top = n - R * t, lo = max(0, top - R), i = lo + r;
            if (B == 2) stage(nxt, buf ^ 1);
            else stage(cur, 0);
            const Rows after = rows_of(t + 2);
            const bool staged = cur.e1 - cur.e0 <= cap;
            const double* pv = sv + buf * cap - cur.e0;
            const int* pc = sc + buf * cap - cur.e0;
            const double di = i < top ? A.invd[i] : 0.0;
            for (int jb = 0; jb < m; jb += NC) {
                const int j = jb + j0;
                const bool mine = i < top && j < m;
                const size_t at = mine ? (size_t)i * m + j : 0;
                // the row's sum apart from b_i: its roundings are those of the smaller terms
                double acc = 0.0, bi = 0.0, old = 0.0;
                if (mine) {
                    bi = A.b[at];
                    old = set_ld(src + at, true);
                }
                const int eb = d_exp(bi);
                if (jb == 0) {
                    if (B == 2) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
                    else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
                    __syncwarp();
                }
                if (staged) {
                    // x at every entry, all of a lane's loads in flight together (a diagonal's is not used)
                    const int cnt = (cur.e1 - cur.e0) * NC;
                    for (int q0 = 0; q0 < cnt; q0 += 32 * 8) {
                        double xv[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            const int q = q0 + lane + 32 * u;
                            if (q < cnt) {
                                const int c = sc[buf * cap + q / NC];
                                if (jb + q % NC < m) xv[u] = x_of(c, top, jb + q % NC);
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            const int q = q0 + lane + 32 * u;
                            if (q < cnt) sx[q] = xv[u];
                        }
                    }
                    __syncwarp();
                }
                unsigned em = 0;  // largest sum of the exponents of a term's factors, in the exponent's place
                int inside = 0;   // entries with their column in this tile
                if (mine) {
                    const double* px = sx - (size_t)cur.e0 * NC + j0;
                    for (int k = cur.s; k < cur.e; ++k) {
                        const int c = staged ? pc[k] : __ldg(A.col + k);
                        const double v = staged ? pv[k] : __ldg(A.val + k);
                        const double xv = staged ? px[(size_t)k * NC] : x_of(c, top, j);
                        acc = fma(v, xv, acc);
                        em = max(em, ((unsigned)__double2hiint(v) & 0x7ff00000u) +
                                         ((unsigned)__double2hiint(xv) & 0x7ff00000u));
                        inside += c < top;
                    }
                }
                double y = (bi - acc) * di;
                if constexpr (NC == 1) {
                    // second look: the tile's own changes, once
                    // (no change is zero for infinities too)
                    dl[lane] = mine && __double_as_longlong(y) != __double_as_longlong(old) ? y - old : 0.0;
                    __syncwarp();
                    if (mine) {
                        double more = 0.0;
                        for (int k = cur.s; inside > 0; ++k) {
                            const int c = staged ? pc[k] : __ldg(A.col + k);
                            if (c < top) {
                                more = fma(staged ? pv[k] : __ldg(A.val + k), dl[c - lo], more);
                                --inside;
                            }
                        }
                        y = fma(-more, di, y);
                    }
                }
                if (mine && __double_as_longlong(y) != __double_as_longlong(old)) {
                    const int ei = d_exp(di) - 1023;
                    const int size = max(d_exp(y), max(eb, (int)(em >> 20) - 1023) + ei);
                    const int gap = d_gap(y, old) - size;
                    worst = max(worst, gap + kSetPending);
                    if (!kPair) st_relaxed(dst + at, y);
                }
                if (kPair && mine) dst[at] = y;
                __syncwarp();  // sx and dl are read before they are written again
            }
            __syncwarp();  // the staged entries are read, the tile's x written, before the next tile
            cur = nxt;
            nxt = after;
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        worst = __reduce_max_sync(0xffffffffu, worst);
        if (lane == 0 && worst > 0) atomicMax(&s_worst, worst);
        __syncthreads();
        if (threadIdx.x == 0 && s_worst > 0) atomicMax(A.worst + p, s_worst);
        if (!grid_barrier(A.ctl, gridDim.x, A.budget)) return;
        const int verdict = settle_verdict(A.worst, p, A.most, last);
        if (verdict == 1 && blockIdx.x == 0 && threadIdx.x == 0) {
            A.ctl->done = 1;
            A.ctl->steps = p + 1;
        }
        if (verdict == 1 && dst != A.x)  // the run's rows of the solution
            for (size_t k = (size_t)max(0, n - R * t1) * m + lane; k < (size_t)max(0, run_top) * m; k += 32) A.x[k] = dst[k];
        if (verdict) return;
    }
}

// Prepares the exact kernel behind k_settle: x pending when it has to run, no row left to claim when
// it has not.
__global__ void k_settle_gate(double* x, size_t count, Ctl* ctl) {
    if (*(volatile const int*)&ctl->done) {
        if (blockIdx.x == 0 && threadIdx.x == 0) ctl->ticket = 0xF0000000u;
        return;
    }
    const double v = Pend<double>::value();
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < count; k += (size_t)gridDim.x * blockDim.x) x[k] = v;
}

// Staged entries of a tile: the mean tile and four deviations of a Poisson count, if shared memory holds it.
template <int NC>
static int set_cap(int n, long long nnz) {
    const double mean = SetShape<NC>::kRows * (double)nnz / n;
    const int fit = (int)((kSetSmem / kSetWarps - 256) / (12 * SetShape<NC>::kBufs + 8 * NC));
    return std::min(fit, (int)(mean + 4.0 * std::sqrt(mean)) + 15) / 8 * 8;
}

template <int NC>
static double long_us_t(int n, long long nnz, int rhs, int longest) {
    if ((SetShape<NC>::kRows - 1) * (double)nnz / n + longest <= set_cap<NC>(n, nnz)) return 0.0;
    return (NC == 1 ? 0.2 : 0.46) * longest * ((rhs + NC - 1) / NC);
}

// What the longest row adds to a sweep, in microseconds: where its tile does not fit the staging buffer, a
// lane walks it through global memory, an entry after the other, while the other warps wait.  Measured on
// GB300, 40,000 rows with one row of 400 / 3,000 / 12,000 entries, 22 sweeps: 2.0 / 12.6 / 47.9 ms with one
// right-hand side (the exact kernel 1.4 / 2.0 / 4.2), 4.5 / 31.7 / 118.8 ms with eight (11.0 / 11.3 / 12.4).
double settle_long_us(int n, long long nnz, int rhs, int longest) {
    if (rhs == 1) return long_us_t<1>(n, nnz, rhs, longest);
    if (rhs == 2) return long_us_t<2>(n, nnz, rhs, longest);
    if (rhs <= 4) return long_us_t<4>(n, nnz, rhs, longest);
    if (rhs <= 8) return long_us_t<8>(n, nnz, rhs, longest);
    if (rhs <= 16) return long_us_t<16>(n, nnz, rhs, longest);
    return long_us_t<32>(n, nnz, rhs, longest);
}

template <int NC>
static int settle_t(const SolveArgs& a, int* worst, double* y, int most) {
    constexpr int R = SetShape<NC>::kRows;
    const int cap = set_cap<NC>(a.n, a.nnz);
    const size_t bytes = kSetWarps * set_warp_bytes(cap, NC, SetShape<NC>::kBufs);
    const void* fn = (const void*)k_settle<NC>;
    // the limit belongs to the kernel on the device: the largest any matrix asks for, so that no thread's
    // launch finds it lowered by another's
    CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSetSmem));
    int per_sm = 0;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kSetWarps * 32, bytes));
    if (per_sm < 1) return SPTRSV_ERR_UNSUPPORTED;
    const int ntiles = (a.n + R - 1) / R;
    // Tiles of the shortest run: longer runs take fewer sweeps (fewer rows see a neighbour's old values),
    // shorter ones spread further.  One right-hand side: 10k rows 207 / 278 / 291 us at 1 / 2 / 3 tiles, 50k
    // rows 290 / 282 / 283, 200k rows 489 / 496 / 435.  Several: 10k rows x 8 310 / 384 us at 2 / 4.
    const int shortest = NC > 1 ? 2 : ntiles <= a.sm_count * kSetWarps ? 1 : 3;
    const int warps = std::max(1, std::min(per_sm * a.sm_count * kSetWarps, ntiles / shortest));
    // a caller's budget is for waits on rows: a sweep over millions of rows keeps a barrier waiting longer
    const int64_t budget = std::max<int64_t>(a.budget, kDefaultBudgetNs);
    SettleArgs s{a.n, a.rhs, a.rp, a.col, (const double*)a.val, (const double*)a.invd, (const double*)a.b, (double*)a.x, y,
                 a.ctl, worst, budget, most, (ntiles + warps - 1) / warps, cap};
    const int grid = ((ntiles + s.tiles - 1) / s.tiles + kSetWarps - 1) / kSetWarps;
    void* args[] = {(void*)&s};
    CUDA_TRY(launch_cooperative(fn, grid, kSetWarps * 32, args, bytes, a.st));
    ++*a.launches;
    return 0;
}

// Bytes of `work`: the sweeps' records and the other vector.
size_t settle_work(int n, int rhs) {
    return sizeof(int) * kSettleSweeps + (rhs > 1 ? sizeof(double) * (size_t)n * rhs : 0);
}

int launch_settle(const SolveArgs& a, void* work, int most) {
    int* worst = (int*)work;
    double* y = a.rhs > 1 ? (double*)(worst + kSettleSweeps) : nullptr;
    CUDA_TRY(cudaMemsetAsync(worst, 0, sizeof(int) * kSettleSweeps, a.st));
    int rc;
    if (a.rhs == 1) rc = settle_t<1>(a, worst, y, most);
    else if (a.rhs == 2) rc = settle_t<2>(a, worst, y, most);
    else if (a.rhs <= 4) rc = settle_t<4>(a, worst, y, most);
    else if (a.rhs <= 8) rc = settle_t<8>(a, worst, y, most);
    else if (a.rhs <= 16) rc = settle_t<16>(a, worst, y, most);
    else rc = settle_t<32>(a, worst, y, most);
    if (rc) return rc;
    const size_t count = (size_t)a.n * a.rhs;
    k_settle_gate<<<(int)std::min<size_t>((count + 255) / 256, 2048), 256, 0, a.st>>>((double*)a.x, count, a.ctl);
    ++*a.launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

}  // namespace sptrsv
