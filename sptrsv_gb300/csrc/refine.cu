// refine.cu -- FP32 bulk solves with FP64 iterative refinement.
//
// One refinement step, all on the device (no host round trip, so the whole solve is one
// CUDA graph launch):
//   r   = b - U x               FP64 SpMV over the FP64 values (k_residual_*); ||r_c||^2 per
//                               column for the convergence test; r is also stored in FP32 as
//                               the inner right-hand side, and d0 = D^-1 r seeds the sweeps;
//   test                        rel = max_c ||r_c|| / ||b_c||; once rel <= tol the `done` flag
//                               is raised (flat graphs: every later kernel returns at once;
//                               conditional graphs: the outer WHILE node stops);
//   d  ~= U^{-1} r              FP32 inner solve, either
//                                 JACOBI: d <- D^-1 (r - N d) sweeps over an interleaved
//                                 (column, FP32 value) copy of the off-diagonals, until the
//                                 largest change is below max(10^-e, 0.1 tol / rel) of the
//                                 largest |d| (the inner WHILE node) -- fully parallel; it
//                                 converges for any triangular U because N is nilpotent, and
//                                 fast when U is diagonally dominant -- or
//                                 an exact FP32 sync-free / level-set solve (solve.cu);
//   x  += d                     FP64 update.
// x starts at 0, so the first residual is b itself.
//
// Short rows: the FP64 residual uses warp tiles of 32 consecutive rows (the warp copies the
// tile's entries into shared memory with coalesced loads, then each lane sums its own row in
// order: deterministic; tiles with more than kTileMax entries read straight from global memory);
// the default Jacobi sweep gives each lane a row of the paired layout, whose entries
// come by bulk copies, and runs a whole inner solve as one launch.  Long-row matrices use the warp-per-row kernels (LPR lanes per row).
#include "common.cuh"
#include "kernels.cuh"

namespace sptrsv {

constexpr int kTileMax = 512;   // staged entries per warp
constexpr int kJacWarps = 8;    // warps per block, Jacobi tile kernel (4 KiB stage per warp)
constexpr int kResWarps = 4;    // warps per block, residual tile kernel (6 KiB stage per warp)

__device__ __forceinline__ bool is_done(const Ctl* ctl) { return *(volatile const int*)&ctl->done != 0; }

// ||b_c||^2 for row-major b (rhs <= 1024).
__global__ void k_colnorm2(int n, int rhs, const double* __restrict__ b, double* __restrict__ out) {
    extern __shared__ double acc[];
    for (int c = threadIdx.x; c < rhs; c += blockDim.x) acc[c] = 0.0;
    __syncthreads();
    const int per_pass = (blockDim.x / rhs) > 0 ? (blockDim.x / rhs) : 0;
    if (rhs == 1) {
        double s = 0.0;
        for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
            const double v = b[i];
            s += v * v;
        }
        s = warp_sum(s);
        if ((threadIdx.x & 31) == 0) atomicAdd(&acc[0], s);
    } else if (per_pass > 0 && (int)threadIdx.x < per_pass * rhs) {
        const int c = threadIdx.x % rhs, r0 = threadIdx.x / rhs;
        double s = 0.0;
        for (long long i = (long long)blockIdx.x * per_pass + r0; i < n; i += (long long)gridDim.x * per_pass) {
            const double v = b[i * rhs + c];
            s += v * v;
        }
        atomicAdd(&acc[c], s);
    } else if (per_pass == 0) {
        for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < (long long)n * rhs;
             p += (long long)gridDim.x * blockDim.x) {
            const double v = b[p];
            atomicAdd(&acc[p % rhs], v * v);
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < rhs; c += blockDim.x) atomicAdd(out + c, acc[c]);
}

// Interleaved FP32 off-diagonals: entry k of row i (k > rp[i]) goes to slot k - i - 1, so the
// off-diagonals of row i occupy [rp[i] - i, rp[i+1] - i - 1).
__global__ void k_build_offdiag(int n, const int* __restrict__ rp, const int* __restrict__ col,
                                const double* __restrict__ val, int2* __restrict__ off) {
    const int lane = threadIdx.x & 31;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5)
        for (int k = rp[i] + 1 + lane; k < rp[i + 1]; k += 32)
            off[k - i - 1] = make_int2(col[k], __float_as_int((float)val[k]));
}

// roff[i] = first off-diagonal slot of row i = rp[i] - i, padded past n with its end value.
__global__ void k_build_roff(int n, int pad, const int* __restrict__ rp, int* __restrict__ roff) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n + pad; i += gridDim.x * blockDim.x)
        roff[i] = (i <= n) ? rp[i] - i : rp[n] - n;
}

__global__ void k_pair_len(int n, const int* __restrict__ rp, int* __restrict__ len2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int len = rp[i + 1] - rp[i] - 1;
        len2[i] = len + (len & 1);
    }
}

__global__ void k_pad_roff(int n, int pad, int* __restrict__ roff) {
    const int total = roff[n];
    for (int i = n + 1 + blockIdx.x * blockDim.x + threadIdx.x; i <= n + pad; i += gridDim.x * blockDim.x)
        roff[i] = total;
}

__global__ void k_build_offdiag_pairs(int n, const int* __restrict__ rp, const int* __restrict__ col,
                                      const double* __restrict__ val, const int* __restrict__ roff,
                                      int2* __restrict__ off) {
    const int lane = threadIdx.x & 31;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
        const int b = rp[i] + 1, len = rp[i + 1] - b, o = roff[i];
        for (int k = lane; k < len; k += 32) off[o + k] = make_int2(col[b + k], __float_as_int((float)val[b + k]));
        if (lane == 0 && (len & 1)) off[o + len] = make_int2(i, __float_as_int(0.f));
    }
}

// Group-jagged layout (32-row groups, jagged diagonals inside each group).  Group g holds rows
// 32g .. 32g+31; they are ranked by off-diagonal count, longest first (ties by row), and
// jmeta[32g + R] = (local row << 27) | count of the rank-R row.  Entry t of the rank-R row lives at
// jbase[g] + sum_{t' < t} c_g(t') + R, where c_g(t') = rows of the group with more than t' entries:
// the entries of one diagonal t are contiguous, so a warp whose lane R walks the rank-R row loads
// each diagonal with one coalesced request, and no slot is padding.  Rows past n count 0 entries.
// jbase[ngroups] = total entries, jbase[ngroups + 1] = 1 if some row has >= 2^27 entries.
constexpr int kJdsLenBits = 27;
constexpr int kJdsLenMask = (1 << kJdsLenBits) - 1;

__global__ void k_jds_sizes(int n, int ngroups, const int* __restrict__ rp, int* __restrict__ gsize,
                            int* __restrict__ overflow) {
    const int lane = threadIdx.x & 31;
    for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ngroups; g += (gridDim.x * blockDim.x) >> 5) {
        const int i = 32 * g + lane;
        const int len = (i < n) ? rp[i + 1] - rp[i] - 1 : 0;
        if (len > kJdsLenMask) atomicOr(overflow, 1);
        const int s = __reduce_add_sync(0xffffffffu, len);
        if (lane == 0) gsize[g] = s;
    }
}

__global__ void k_jds_fill(int n, int ngroups, const int* __restrict__ rp, const int* __restrict__ col,
                           const double* __restrict__ val, const int* __restrict__ jbase, int* __restrict__ jmeta,
                           int2* __restrict__ jent) {
    const int lane = threadIdx.x & 31;
    for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ngroups; g += (gridDim.x * blockDim.x) >> 5) {
        const int i = 32 * g + lane;
        const int first = (i < n) ? rp[i] + 1 : 0;
        const int len = (i < n) ? rp[i + 1] - first : 0;
        int rank = 0;
        for (int j = 0; j < 32; ++j) {
            const int lj = __shfl_sync(0xffffffffu, len, j);
            rank += (lj > len) || (lj == len && j < lane);
        }
        jmeta[32 * g + rank] = (lane << kJdsLenBits) | len;
        const int maxlen = __reduce_max_sync(0xffffffffu, len);
        int pos = jbase[g] + rank;
        for (int t = 0; t < maxlen; ++t) {
            const unsigned act = __ballot_sync(0xffffffffu, len > t);
            if (t < len) jent[pos] = make_int2(col[first + t], __float_as_int((float)val[first + t]));
            pos += __popc(act);
        }
    }
}

// Jacobi seed d0 = D^-1 r from the FP32 residual and FP32 reciprocal (FP32 pipe; the FP64 pipe
// is the residual kernels' bottleneck on this GPU), or the pending fill for an exact inner solve.
__device__ __forceinline__ void seed_out(int seed, float* d0, size_t p, float r32, float invd32) {
    if (seed == 1) d0[p] = r32 * invd32;
    else if (seed == 2) d0[p] = __uint_as_float(kPend32);
}

// r = b when x = 0 (the first correction of a solve): the matrix is not read.
__device__ __forceinline__ void residual_of_b(int n, const double* __restrict__ b, const float* __restrict__ invd,
                                              float* __restrict__ r32, float* __restrict__ d0, int seed,
                                              double* __restrict__ rn2, double* s_acc) {
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double r = b[i];
        const float rf = (float)r;
        r32[i] = rf;
        seed_out(seed, d0, i, rf, invd[i]);
        acc = fma(r, r, acc);
    }
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) atomicAdd(s_acc, acc);
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(rn2, *s_acc);
}

// r = b - U x (rhs == 1), warp tiles of 32 rows staged in shared memory.
__global__ void __launch_bounds__(kResWarps * 32) k_residual_tile(int n, const int* __restrict__ rp,
                                                                  const int* __restrict__ col,
                                                                  const double* __restrict__ val,
                                                                  const float* __restrict__ invd,
                                                                  const double* __restrict__ b,
                                                                  const double* __restrict__ x,
                                                                  double* __restrict__ x_out, float* __restrict__ r32,
                                                                  float* __restrict__ d0, int seed,
                                                                  double* __restrict__ rn2, const Ctl* ctl) {
    __shared__ int s_col[kResWarps][kTileMax];
    __shared__ double s_val[kResWarps][kTileMax];
    __shared__ double s_acc;
    if (is_done(ctl)) return;
    if (threadIdx.x == 0) s_acc = 0.0;
    __syncthreads();
    if (*(volatile const int*)&ctl->x_zero) {
        residual_of_b(n, b, invd, r32, d0, seed, rn2, &s_acc);
        return;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int* sc = s_col[w];
    double* sv = s_val[w];
    double acc = 0.0;
    for (int t = blockIdx.x * kResWarps + w; t * 32 < n; t += gridDim.x * kResWarps) {
        const int r0 = t * 32, i = r0 + lane;
        const int s = rp[min(i, n)];
        int e = __shfl_down_sync(0xffffffffu, s, 1);
        if (lane == 31) e = rp[min(r0 + 32, n)];
        const int E0 = __shfl_sync(0xffffffffu, s, 0), E1 = __shfl_sync(0xffffffffu, e, 31);
        double sum = 0.0;
        if (E1 - E0 <= kTileMax) {
            for (int q = lane; q < E1 - E0; q += 32) {
                sc[q] = __ldg(col + E0 + q);
                sv[q] = __ldg(val + E0 + q);
            }
            __syncwarp();
            if (i < n) {
#pragma unroll 4
                for (int k = s - E0; k < e - E0; ++k) sum = fma(sv[k], __ldg(x + sc[k]), sum);
            }
            __syncwarp();
        } else if (i < n) {
            for (int k = s; k < e; ++k) sum = fma(__ldg(val + k), __ldg(x + __ldg(col + k)), sum);
        }
        if (i < n) {
            const double r = b[i] - sum;
            const float rf = (float)r;
            r32[i] = rf;
            seed_out(seed, d0, i, rf, invd[i]);
            acc = fma(r, r, acc);
            if (x_out) x_out[i] = x[i];
        }
    }
    acc = warp_sum(acc);
    if (lane == 0) atomicAdd(&s_acc, acc);
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(rn2, s_acc);
}

// r = b - U x for several right-hand sides, short rows: as k_residual_tile, four columns of a row at a time.
__global__ void __launch_bounds__(kResWarps * 32) k_residual_tile_m(int n, int rhs, const int* __restrict__ rp,
                                                                    const int* __restrict__ col,
                                                                    const double* __restrict__ val,
                                                                    const float* __restrict__ invd,
                                                                    const double* __restrict__ b,
                                                                    const double* __restrict__ x,
                                                                    float* __restrict__ r32, float* __restrict__ d0,
                                                                    int seed, double* __restrict__ rn2, const Ctl* ctl) {
    constexpr int NC = 4;
    __shared__ int s_col[kResWarps][kTileMax];
    __shared__ double s_val[kResWarps][kTileMax];
    extern __shared__ double s_accm[];
    if (is_done(ctl)) return;
    const bool zero = *(volatile const int*)&ctl->x_zero;  // r = b, the matrix is not read
    for (int c = threadIdx.x; c < rhs; c += blockDim.x) s_accm[c] = 0.0;
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (long long t = blockIdx.x * kResWarps + w; t * 32 < n; t += gridDim.x * kResWarps) {
        const int r0 = (int)(t * 32), rows = min(32, n - r0), i = r0 + min(lane, rows - 1);
        const int s = rp[i], e = rp[i + 1];
        const int E0 = __shfl_sync(0xffffffffu, s, 0), E1 = __shfl_sync(0xffffffffu, e, rows - 1);
        const bool staged = !zero && E1 - E0 <= kTileMax;
        if (staged)
            for (int q = lane; q < E1 - E0; q += 32) {
                s_col[w][q] = __ldg(col + E0 + q);
                s_val[w][q] = __ldg(val + E0 + q);
            }
        __syncwarp();
        const float di = invd[i];
        for (int c0 = 0; c0 < rhs; c0 += NC) {
            double sum[NC], sq[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) sum[c] = sq[c] = 0.0;
            auto walk = [&](auto entry) {
#pragma unroll 4
                for (int k = s - E0; k < e - E0; ++k) {
                    double v;
                    const double* xj = x + (size_t)entry(k, v) * rhs + c0;
#pragma unroll
                    for (int c = 0; c < NC; ++c)
                        if (c0 + c < rhs) sum[c] = fma(v, xj[c], sum[c]);
                }
            };
            if (lane < rows) {
                if (zero) {
                } else if (staged) walk([&](int k, double& v) { v = s_val[w][k]; return s_col[w][k]; });
                else walk([&](int k, double& v) { v = __ldg(val + E0 + k); return __ldg(col + E0 + k); });
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    if (c0 + c < rhs) {
                        const size_t p = (size_t)i * rhs + c0 + c;
                        const double r = b[p] - sum[c];
                        const float rf = (float)r;
                        r32[p] = rf;
                        seed_out(seed, d0, p, rf, di);
                        sq[c] = r * r;
                    }
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                if (c0 + c >= rhs) break;
                const double v = warp_sum(sq[c]);
                if (lane == 0) atomicAdd(&s_accm[c0 + c], v);
            }
        }
        __syncwarp();
    }
    __syncthreads();
    for (int c = threadIdx.x; c < rhs; c += blockDim.x) atomicAdd(rn2 + c, s_accm[c]);
}

// r = b - U x (rhs == 1), LPR lanes per row (long rows).
template <int LPR>
__global__ void __launch_bounds__(256) k_residual_v(int n, const int* __restrict__ rp, const int* __restrict__ col,
                                                    const double* __restrict__ val, const float* __restrict__ invd,
                                                    const double* __restrict__ b, const double* __restrict__ x,
                                                    double* __restrict__ x_out, float* __restrict__ r32,
                                                    float* __restrict__ d0, int seed, double* __restrict__ rn2,
                                                    const Ctl* ctl) {
    if (is_done(ctl)) return;
    if (*(volatile const int*)&ctl->x_zero) x_out = nullptr;  // x is still the zero start vector
    __shared__ double s_acc;
    if (threadIdx.x == 0) s_acc = 0.0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int gl = lane % LPR;
    const unsigned gmask = (LPR == 32) ? 0xffffffffu : (((1u << LPR) - 1u) << ((lane / LPR) * LPR));
    const long long gid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LPR;
    const long long gstride = ((long long)gridDim.x * blockDim.x) / LPR;
    double acc = 0.0;
    for (long long i = gid; i < n; i += gstride) {
        const int s = rp[i], e = rp[i + 1];
        double sum = 0.0;
        for (int k = s + gl; k < e; k += LPR) sum = fma(val[k], x[col[k]], sum);
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(gmask, sum, o);
        if (gl == 0) {
            const double r = b[i] - sum;
            const float rf = (float)r;
            r32[i] = rf;
            seed_out(seed, d0, i, rf, invd[i]);
            acc = fma(r, r, acc);
            if (x_out) x_out[i] = x[i];
        }
    }
    acc = warp_sum(acc);
    if (lane == 0) atomicAdd(&s_acc, acc);
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(rn2, s_acc);
}

// rhs > 1: warp per row, lanes over RHS columns, entries sequential.
__global__ void __launch_bounds__(256) k_residual_m(int n, int rhs, const int* __restrict__ rp,
                                                    const int* __restrict__ col, const double* __restrict__ val,
                                                    const float* __restrict__ invd, const double* __restrict__ b,
                                                    const double* __restrict__ x, float* __restrict__ r32,
                                                    float* __restrict__ d0, int seed, double* __restrict__ rn2,
                                                    const Ctl* ctl) {
    if (is_done(ctl)) return;
    extern __shared__ double s_accm[];
    for (int c = threadIdx.x; c < rhs; c += blockDim.x) s_accm[c] = 0.0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long ws = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long i = w; i < n; i += ws) {
        const int s = rp[i], e = rp[i + 1];
        const float di = invd[i];
        for (int c = lane; c < rhs; c += 32) {
            double sum = 0.0;
            for (int k = s; k < e; ++k) sum = fma(val[k], x[(size_t)col[k] * rhs + c], sum);
            const size_t p = (size_t)i * rhs + c;
            const double r = b[p] - sum;
            const float rf = (float)r;
            r32[p] = rf;
            seed_out(seed, d0, p, rf, di);
            atomicAdd(&s_accm[c], r * r);
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < rhs; c += blockDim.x) atomicAdd(rn2 + c, s_accm[c]);
}

__device__ __forceinline__ double rel_of(int rhs, double* rn2, const double* bn2) {
    double rel = 0.0;
    for (int c = 0; c < rhs; ++c) {
        const double r = rn2[c], bb = bn2[c];
        const double q = (bb > 0.0) ? sqrt(r / bb) : (r > 0.0 ? INFINITY : 0.0);
        rel = fmax(rel, q);
        rn2[c] = 0.0;
    }
    return rel;
}

// Flat graphs: the convergence test of step `step`.
__global__ void k_check(int rhs, double* rn2, const double* bn2, Ctl* ctl, double tol, int step, int reset_ticket) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    ctl->x_zero = 0;
    if (ctl->done) return;
    const double rel = rel_of(rhs, rn2, bn2);
    ctl->rel_res = rel;
    ctl->steps = step;
    if (rel <= tol) ctl->done = 1;
    if (reset_ticket) ctl->ticket = 0u;
}

// Conditional graphs: the test at the top of every outer iteration.  Continues (and arms the
// inner loop) while rel > tol and fewer than max_refine corrections were applied.
// Relative accuracy asked of a correction: a tenth of what would just reach the tolerance.
constexpr double kInnerTarget = 0.1;

__global__ void k_check_outer(int rhs, double* rn2, const double* bn2, Ctl* ctl, double tol, int max_refine,
                              cudaGraphConditionalHandle h_outer, cudaGraphConditionalHandle h_inner) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double rel = rel_of(rhs, rn2, bn2);
    ctl->rel_res = rel;
    const int step = ctl->steps;
    const bool stop = rel <= tol || step >= max_refine;
    ctl->x_zero = 0;
    if (rel <= tol) ctl->done = 1;
    ctl->inner_count = 0;
    ctl->dmax_bits = ctl->dmax2_bits = 0u;
    ctl->dchg_bits = ctl->dchg2_bits = 0u;
    if (stop) {
        ctl->inner_eps = -1.f;
        cudaGraphSetConditional(h_outer, 0);
        if (h_inner) cudaGraphSetConditional(h_inner, 0);
    } else {
        ctl->steps = step + 1;
        // inexact correction: x + d has residual ~ rel * (relative error of d), so the next inner
        // solve only needs kInnerTarget * tol / rel (never tighter than its own floor, below)
        ctl->inner_eps = (float)fmin(1.0, kInnerTarget * tol / rel);
        if (h_inner) cudaGraphSetConditional(h_inner, 1);
    }
}

// Conditional graphs: after each pair of sweeps.  Stops the inner loop once the largest
// change is at most max(eps, ctl->inner_eps) times the largest |d|, or after max_sweeps sweeps:
// eps is the FP32 floor of the sweeps, ctl->inner_eps what the outer residual still asks for.
__global__ void k_check_inner(Ctl* ctl, float eps_floor, int max_sweeps, cudaGraphConditionalHandle h_inner) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const float eps = fmaxf(eps_floor, ctl->inner_eps);
    const float dmax = __uint_as_float(ctl->dmax_bits), dchg = __uint_as_float(ctl->dchg_bits);
    const int cnt = ctl->inner_count + 2;
    ctl->inner_count = cnt;
    ctl->inner_total += 2;
    ctl->dmax_bits = 0u;
    ctl->dchg_bits = 0u;
    if (!(dchg > eps * dmax) || cnt >= max_sweeps) cudaGraphSetConditional(h_inner, 0);
}

__device__ __forceinline__ void reduce_stats(float dmax, float dchg, Ctl* ctl, unsigned* s_max) {
    for (int o = 16; o > 0; o >>= 1) {
        dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
        dchg = fmaxf(dchg, __shfl_xor_sync(0xffffffffu, dchg, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&s_max[0], __float_as_uint(dmax));
        atomicMax(&s_max[1], __float_as_uint(dchg));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicMax(&ctl->dmax_bits, s_max[0]);
        atomicMax(&ctl->dchg_bits, s_max[1]);
    }
}

// One FP32 Jacobi sweep over warp tiles: dst = D^-1 (r - N src), or x += that when `last`.
// stats: accumulate max|d| and max|d - src| (non-negative floats order like their bits).
template <int TMAX, int MINB>
__global__ void __launch_bounds__(kJacWarps * 32, MINB) k_jacobi_tile(int n, const int* __restrict__ rp,
                                                                const int2* __restrict__ off,
                                                                const float* __restrict__ invd,
                                                                const float* __restrict__ r,
                                                                const float* __restrict__ src, float* __restrict__ dst,
                                                                double* __restrict__ x, int last, int stats, Ctl* ctl) {
    __shared__ __align__(16) int2 stage[kJacWarps][TMAX];
    __shared__ unsigned s_max[2];
    if (is_done(ctl)) return;
    if (threadIdx.x < 2) s_max[threadIdx.x] = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int2* sb = stage[w];
    float dmax = 0.f, dchg = 0.f;
    for (int t = blockIdx.x * kJacWarps + w; t * 32 < n; t += gridDim.x * kJacWarps) {
        const int r0 = t * 32, i = r0 + lane;
        const int ii = min(i, n);
        const int s = rp[ii] - ii;  // first off-diagonal slot of row i
        int e = __shfl_down_sync(0xffffffffu, s, 1);
        if (lane == 31) {
            const int j = min(r0 + 32, n);
            e = rp[j] - j;
        }
        const int E0 = __shfl_sync(0xffffffffu, s, 0), E1 = __shfl_sync(0xffffffffu, e, 31);
        float sum = 0.f;
        const int a0 = E0 & ~1;  // 16-byte aligned start (pairs of int2)
        if (E1 - a0 <= TMAX) {
            const int npair = (E1 - a0 + 1) >> 1;
            const int4* v4 = reinterpret_cast<const int4*>(off + a0);
            int4* s4 = reinterpret_cast<int4*>(sb);
            for (int q = lane; q < npair; q += 32) s4[q] = __ldg(v4 + q);
            __syncwarp();
            if (i < n) {
#pragma unroll 4
                for (int k = s - a0; k < e - a0; ++k) {
                    const int2 p = sb[k];
                    sum = fmaf(__int_as_float(p.y), __ldg(src + p.x), sum);
                }
            }
            __syncwarp();
        } else if (i < n) {
            for (int k = s; k < e; ++k) {
                const int2 p = __ldg(off + k);
                sum = fmaf(__int_as_float(p.y), __ldg(src + p.x), sum);
            }
        }
        if (i < n) {
            const float d = (r[i] - sum) * invd[i];
            if (stats) {
                dmax = fmaxf(dmax, fabsf(d));
                dchg = fmaxf(dchg, fabsf(d - src[i]));
            }
            if (last) x[i] += (double)d;
            else dst[i] = d;
        }
    }
    if (stats) reduce_stats(dmax, dchg, ctl, s_max);
}

// Lane-per-row sweep reading the interleaved off-diagonals straight from global memory (L1 keeps
// the lines a warp's 32 neighbouring rows share); bounded to 32 registers for full occupancy.
__global__ void __launch_bounds__(256, 8) k_jacobi_direct(int n, const int* __restrict__ roff,
                                                         const int2* __restrict__ off,
                                                         const float* __restrict__ invd,
                                                         const float* __restrict__ r, const float* __restrict__ src,
                                                         float* __restrict__ dst, double* __restrict__ x, int last,
                                                         int stats, Ctl* ctl) {
    __shared__ unsigned s_max[2];
    if (is_done(ctl)) return;
    if (threadIdx.x < 2) s_max[threadIdx.x] = 0u;
    __syncthreads();
    float dmax = 0.f, dchg = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int s = __ldg(roff + i), e = __ldg(roff + i + 1);
        float sum = 0.f;
#pragma unroll 4
        for (int k = s; k < e; ++k) {
            const int2 p = __ldg(off + k);
            sum = fmaf(__int_as_float(p.y), __ldg(src + p.x), sum);
        }
        const float d = (r[i] - sum) * invd[i];
        if (stats) {
            dmax = fmaxf(dmax, fabsf(d));
            dchg = fmaxf(dchg, fabsf(d - src[i]));
        }
        if (last) x[i] += (double)d;
        else dst[i] = d;
    }
    if (stats) reduce_stats(dmax, dchg, ctl, s_max);
}

// Lane-per-row sweep with explicit load batching: the next row's offsets are fetched while the
// current row is summed, and each batch of B entries issues all B entry loads, then all B
// gathers, then the B FMAs (in entry order, so the sum is the same as the sequential loop's).
template <int B, int MINB>
__global__ void __launch_bounds__(256, MINB) k_jacobi_batched(int n, const int* __restrict__ roff,
                                                             const int2* __restrict__ off,
                                                             const float* __restrict__ invd,
                                                             const float* __restrict__ r,
                                                             const float* __restrict__ src, float* __restrict__ dst,
                                                             double* __restrict__ x, int last, int stats, Ctl* ctl) {
    __shared__ unsigned s_max[2];
    if (is_done(ctl)) return;
    if (threadIdx.x < 2) s_max[threadIdx.x] = 0u;
    __syncthreads();
    float dmax = 0.f, dchg = 0.f;
    const int stride = gridDim.x * blockDim.x;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int s = 0, e = 0;
    if (i < n) { s = __ldg(roff + i); e = __ldg(roff + i + 1); }
    while (i < n) {
        const int inext = i + stride;
        int sn = 0, en = 0;
        if (inext < n) { sn = __ldg(roff + inext); en = __ldg(roff + inext + 1); }
        const float ri = r[i], di = invd[i];
        float sum = 0.f;
        for (int k0 = s; k0 < e; k0 += B) {
            int2 p[B];
            float g[B];
#pragma unroll
            for (int j = 0; j < B; ++j) p[j] = (k0 + j < e) ? __ldg(off + k0 + j) : make_int2(i, 0);
#pragma unroll
            for (int j = 0; j < B; ++j) g[j] = (k0 + j < e) ? __ldg(src + p[j].x) : 0.f;
#pragma unroll
            for (int j = 0; j < B; ++j) sum = fmaf(__int_as_float(p[j].y), g[j], sum);
        }
        const float d = (ri - sum) * di;
        if (stats) {
            dmax = fmaxf(dmax, fabsf(d));
            dchg = fmaxf(dchg, fabsf(d - src[i]));
        }
        if (last) x[i] += (double)d;
        else dst[i] = d;
        i = inext;
        s = sn;
        e = en;
    }
    if (stats) reduce_stats(dmax, dchg, ctl, s_max);
}

// The sweep over the group-jagged layout: a warp per 32-row group, lane R on the rank-R row.  One
// diagonal of the group is one contiguous run of entries, so every entry load of the warp is a
// single coalesced request (the lane-per-row layouts touch one cache line per lane instead).  B
// diagonals per batch: B loads, B gathers, B FMAs in entry order; the group's next metadata is
// fetched while the current group is summed.  Measured on GB300 against the paired lane-per-row
// sweep: L1 throughput 51 % instead of 76 %, 5 % fewer DRAM bytes, the same time (the sweep is
// bound by load latency, not by L1 wavefronts); issuing the next batch's loads ahead of the current
// gathers (register pipelining, also unrolled by two) made it slower.
template <int B, int MINB>
__global__ void __launch_bounds__(256, MINB) k_jacobi_jds(int n, int ngroups, const int* __restrict__ jmeta,
                                                         const int* __restrict__ jbase,
                                                         const int2* __restrict__ jent,
                                                         const float* __restrict__ invd,
                                                         const float* __restrict__ r,
                                                         const float* __restrict__ src, float* __restrict__ dst,
                                                         double* __restrict__ x, int last, int stats, Ctl* ctl) {
    __shared__ unsigned s_max[2];
    if (is_done(ctl)) return;
    if (threadIdx.x < 2) s_max[threadIdx.x] = 0u;
    __syncthreads();
    float dmax = 0.f, dchg = 0.f;
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int meta = 0, base = 0;
    if (g < ngroups) { meta = __ldg(jmeta + 32 * g + lane); base = __ldg(jbase + g); }
    while (g < ngroups) {
        const int gn = g + nwarps;
        int meta_n = 0, base_n = 0;
        if (gn < ngroups) { meta_n = __ldg(jmeta + 32 * gn + lane); base_n = __ldg(jbase + gn); }
        const int len = meta & kJdsLenMask;
        const int row = 32 * g + (int)((unsigned)meta >> kJdsLenBits);
        const bool valid = row < n;
        const int maxlen = __reduce_max_sync(0xffffffffu, len);
        float ri = 0.f, di = 0.f;
        if (valid) { ri = r[row]; di = invd[row]; }
        float sum = 0.f;
        int pos = base + lane;
        for (int t0 = 0; t0 < maxlen; t0 += B) {
            int2 e[B];
            float gv[B];
#pragma unroll
            for (int j = 0; j < B; ++j) {
                const unsigned act = __ballot_sync(0xffffffffu, len > t0 + j);
                e[j] = (t0 + j < len) ? __ldg(jent + pos) : make_int2(0, 0);
                pos += __popc(act);
            }
#pragma unroll
            for (int j = 0; j < B; ++j) gv[j] = (t0 + j < len) ? __ldg(src + e[j].x) : 0.f;
#pragma unroll
            for (int j = 0; j < B; ++j) sum = fmaf(__int_as_float(e[j].y), gv[j], sum);
        }
        if (valid) {
            const float d = (ri - sum) * di;
            if (stats) {
                dmax = fmaxf(dmax, fabsf(d));
                dchg = fmaxf(dchg, fabsf(d - src[row]));
            }
            if (last) x[row] += (double)d;
            else dst[row] = d;
        }
        g = gn;
        meta = meta_n;
        base = base_n;
    }
    if (stats) reduce_stats(dmax, dchg, ctl, s_max);
}

// Same, two rows per thread per iteration (i and i + half the grid): two independent load chains
// in flight per thread.
__global__ void __launch_bounds__(256, 8) k_jacobi_direct2(int n, const int* __restrict__ roff,
                                                          const int2* __restrict__ off,
                                                          const float* __restrict__ invd,
                                                          const float* __restrict__ r, const float* __restrict__ src,
                                                          float* __restrict__ dst, double* __restrict__ x, int last,
                                                          int stats, Ctl* ctl) {
    __shared__ unsigned s_max[2];
    if (is_done(ctl)) return;
    if (threadIdx.x < 2) s_max[threadIdx.x] = 0u;
    __syncthreads();
    float dmax = 0.f, dchg = 0.f;
    const int stride = gridDim.x * blockDim.x;
    for (int i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += 2 * stride) {
        const int i1 = i0 + stride;
        const bool has1 = i1 < n;
        const int s0 = __ldg(roff + i0), e0 = __ldg(roff + i0 + 1);
        const int s1 = has1 ? __ldg(roff + i1) : 0, e1 = has1 ? __ldg(roff + i1 + 1) : 0;
        float sum0 = 0.f, sum1 = 0.f;
        const int l0 = e0 - s0, l1 = e1 - s1;
        const int lmax = l0 > l1 ? l0 : l1;
#pragma unroll 2
        for (int q = 0; q < lmax; ++q) {
            if (q < l0) {
                const int2 p = __ldg(off + s0 + q);
                sum0 = fmaf(__int_as_float(p.y), __ldg(src + p.x), sum0);
            }
            if (q < l1) {
                const int2 p = __ldg(off + s1 + q);
                sum1 = fmaf(__int_as_float(p.y), __ldg(src + p.x), sum1);
            }
        }
        const float d0 = (r[i0] - sum0) * invd[i0];
        if (stats) {
            dmax = fmaxf(dmax, fabsf(d0));
            dchg = fmaxf(dchg, fabsf(d0 - src[i0]));
        }
        if (last) x[i0] += (double)d0;
        else dst[i0] = d0;
        if (has1) {
            const float d1 = (r[i1] - sum1) * invd[i1];
            if (stats) {
                dmax = fmaxf(dmax, fabsf(d1));
                dchg = fmaxf(dchg, fabsf(d1 - src[i1]));
            }
            if (last) x[i1] += (double)d1;
            else dst[i1] = d1;
        }
    }
    if (stats) reduce_stats(dmax, dchg, ctl, s_max);
}

// ---------------------------------------------------------------------------------------
// SELL-32-256 copy of the off-diagonals for the sweeps: rows are sorted by off-diagonal count
// (descending, stable) inside windows of 256 rows and grouped into slices of 32; a slice stores
// entry k of its 32 rows contiguously (column-major inside the slice) and is padded to its
// longest row with (column = the row itself, value 0).  A warp sweeps a slice with every load
// coalesced (256 bytes per instruction) and no divergence.
constexpr int kSellWin = 256;

// One block of 256 threads per window: bitonic sort of (count, row) by count descending, row
// ascending (stable order), then slice lengths.
__global__ void __launch_bounds__(kSellWin) k_sell_sort(int n, const int* __restrict__ rp, int* __restrict__ perm,
                                                        int* __restrict__ slen) {
    __shared__ int key[kSellWin], idx[kSellWin];
    const int w = blockIdx.x, t = threadIdx.x;
    const int row = w * kSellWin + t;
    key[t] = row < n ? rp[row + 1] - rp[row] - 1 : -1;  // padding rows sort last
    idx[t] = row;
    __syncthreads();
    for (int k = 2; k <= kSellWin; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            const int p = t ^ j;
            if (p > t) {
                const bool up = (t & k) == 0;  // this pair sorts "descending by key, ascending by row"
                const int ka = key[t], kb = key[p], ia = idx[t], ib = idx[p];
                const bool a_first = ka > kb || (ka == kb && ia < ib);
                if (a_first != up) {
                    key[t] = kb; key[p] = ka;
                    idx[t] = ib; idx[p] = ia;
                }
            }
            __syncthreads();
        }
    }
    perm[row] = idx[t] < n ? idx[t] : -1;
    if ((t & 31) == 0) slen[row >> 5] = key[t] > 0 ? key[t] : 0;  // first row of a slice is its longest
}

__global__ void k_sell_sizes(int nslices, const int* __restrict__ slen, int* __restrict__ sz) {
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nslices; s += gridDim.x * blockDim.x) sz[s] = 32 * slen[s];
}

__global__ void k_sell_fill(int nslices, const int* __restrict__ rp, const int* __restrict__ col,
                            const double* __restrict__ val, const int* __restrict__ perm, const int* __restrict__ slen,
                            const int* __restrict__ sptr, int2* __restrict__ sell) {
    const int lane = threadIdx.x & 31;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nslices; s += (gridDim.x * blockDim.x) >> 5) {
        const int row = perm[32 * s + lane];
        const int len = slen[s];
        const int base = sptr[s];
        const int b = row >= 0 ? rp[row] + 1 : 0, e = row >= 0 ? rp[row + 1] : 0;
        for (int k = 0; k < len; ++k) {
            int2 v = make_int2(row >= 0 ? row : 0, 0);  // padding: 0 * x[row]
            if (b + k < e) v = make_int2(col[b + k], __float_as_int((float)val[b + k]));
            sell[base + 32 * k + lane] = v;
        }
    }
}

__global__ void __launch_bounds__(256, 8) k_jacobi_sell(int nslices, const int* __restrict__ perm,
                                                       const int* __restrict__ slen, const int* __restrict__ sptr,
                                                       const int2* __restrict__ sell,
                                                       const float* __restrict__ invd, const float* __restrict__ r,
                                                       const float* __restrict__ src, float* __restrict__ dst,
                                                       double* __restrict__ x, int last, int stats, Ctl* ctl) {
    __shared__ unsigned s_max[2];
    if (is_done(ctl)) return;
    if (threadIdx.x < 2) s_max[threadIdx.x] = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    float dmax = 0.f, dchg = 0.f;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nslices; s += (gridDim.x * blockDim.x) >> 5) {
        const int row = __ldg(perm + 32 * s + lane);
        const int len = __ldg(slen + s);
        const int2* p = sell + __ldg(sptr + s) + lane;
        float sum = 0.f;
#pragma unroll 4
        for (int k = 0; k < len; ++k) {
            const int2 v = __ldg(p + 32 * k);
            sum = fmaf(__int_as_float(v.y), __ldg(src + v.x), sum);
        }
        if (row >= 0) {
            const float d = (r[row] - sum) * invd[row];
            if (stats) {
                dmax = fmaxf(dmax, fabsf(d));
                dchg = fmaxf(dchg, fabsf(d - src[row]));
            }
            if (last) x[row] += (double)d;
            else dst[row] = d;
        }
    }
    if (stats) reduce_stats(dmax, dchg, ctl, s_max);
}

// SELL build, first half: window sorts, slice lengths and slice offsets; returns the entry count.
int sell_prepare(int n, const int* rp, int* perm, int* slen, int* sptr, int* part, int sm_count, cudaStream_t st,
                 int64_t* launches, int* total) {
    const int nwin = (n + kSellWin - 1) / kSellWin;
    const int nslices = nwin * (kSellWin / 32);
    k_sell_sort<<<nwin, kSellWin, 0, st>>>(n, rp, perm, slen);
    k_sell_sizes<<<sm_count * 4, 256, 0, st>>>(nslices, slen, sptr);
    *launches += 2;
    int rc = scan_exclusive(sptr, sptr, nslices, part, st, launches);
    if (rc) return rc;
    CUDA_TRY(cudaMemcpyAsync(total, sptr + nslices, sizeof(int), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    return 0;
}

// SELL build, second half: the slices' column-major entries (`sell` holds `total` entries).
int sell_fill(int n, const int* rp, const int* col, const double* val, const int* perm, const int* slen,
              const int* sptr, int2* sell, int sm_count, cudaStream_t st, int64_t* launches) {
    const int nslices = ((n + kSellWin - 1) / kSellWin) * (kSellWin / 32);
    k_sell_fill<<<sm_count * 8, 256, 0, st>>>(nslices, rp, col, val, perm, slen, sptr, sell);
    ++*launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}
int sell_slices(int n) { return ((n + kSellWin - 1) / kSellWin) * (kSellWin / 32); }

// ---------------------------------------------------------------------------------------
// The default sweep of short rows with few right-hand sides, over the paired layout: every row's slots
// start on a 16-byte boundary and come in pairs, so one 16-byte load brings two entries; the pad entry of
// an odd row adds 0 * d_i.  A block takes tiles of R rows.  One more warp brings each tile's entries to
// shared memory by a bulk copy, S tiles deep, while a lane per row sums the tile before: B entries (B / 2
// pair loads, B gathers, B FMAs in entry order) at a time.  What is left to wait for is the gathers; with
// the entries loaded by the lanes as well (L1 76 % busy) a sweep took 38 us
// at 2M rows and 17.2M entries, 62 % of the measured copy bandwidth.
//
// kLoop: the whole inner solve in one cooperative launch.  A grid barrier follows each sweep and every
// block makes the test of k_check_inner after each second one; then x += d.  Launching the sweeps and the
// test from a WHILE node cost 4 us a sweep (9 us where the sweep itself is short).  The next sweep's
// first tiles are copied ahead of the barrier, and a block with no more than S tiles keeps them all in
// shared memory: up to 311k rows the entries are read once.  Three residuals and 28 sweeps: 2M rows
// 1.31 -> 1.06 ms, 1M 0.75 -> 0.63, 400k 0.46 -> 0.36, 100k 0.33 -> 0.20, 20k 0.28 -> 0.15, 2k 0.26 -> 0.14.
// R = 256, four blocks an SM: 128 x 8 spend the gain on a barrier of 1,216 blocks (1.53 ms at 2M rows),
// 512 x 2, 320 x 3 and three stages are within 4 %.  One sweep a launch: R = 128, eight blocks (1.16 ms,
// 256 x 4 1.22).
//
// Sweeps read 8 bytes an entry and 16 a row.  What does not fit L2 with the four vectors is read
// evict-first, so that the vectors and the first tiles stay from sweep to sweep: 60 MB in all, half of L2
// (lines of the other die are held twice).  2M rows: no policy 1.15 ms, everything evict-first 1.07,
// 28 MB kept 1.05.
//
// NC = 4: several right-hand sides, a lane on four columns of its row at a time, over the same copy of
// the entries (kBulkCols has the times).
//
// Every wait is bounded, and copies in flight land before a block ends.
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait for phase `parity` of *bar; false on timeout or abort (error recorded)
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity, Ctl* ctl, int64_t budget) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = gtimer();
    for (;;) {
        if (mbar_try_wait(bar, parity)) return true;
        if (aborted(ctl)) return false;
        if ((int64_t)(gtimer() - t0) > budget) { record_error(ctl, SPTRSV_ERR_TIMEOUT); return false; }
    }
}

// L2 policy of entries that no later sweep finds in L2 anyway: first to go, so that the vectors stay.
__device__ __forceinline__ uint64_t evict_first_policy() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void bulk_g2s_hint(void* dst, const void* src, unsigned bytes, uint64_t* bar, uint64_t policy) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar)), "l"(policy)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// The same without the abort flag: what is in flight lands whatever else went wrong.
__device__ __forceinline__ void mbar_drain(uint64_t* bar, unsigned parity, int64_t budget) {
    const uint64_t t0 = gtimer();
    while (!mbar_try_wait(bar, parity) && (int64_t)(gtimer() - t0) <= budget) {}
}

struct BulkArgs {
    int n, rhs, cap, keep;  // cap: pairs a stage holds; tiles before `keep` are read with no L2 policy
    const int* roff;
    const int4* off2;
    const float *invd, *r;
    float *d0, *d1;  // the first sweep reads d0
    double* x;
    int last, stats;  // one sweep: x += its result; measure its change
    float eps_floor;  // loop: as k_check_inner
    int max_sweeps;
    Ctl* ctl;
    int64_t budget;
};

template <int R, int S, int MINB, bool kLoop, int NC>
__global__ void __launch_bounds__(R + 32, MINB) k_jacobi_bulk(const BulkArgs A) {
    constexpr int B = NC == 1 ? 8 : 4;
    const int rhs = NC == 1 ? 1 : A.rhs;
    extern __shared__ __align__(128) int4 stage[];  // S x cap pairs
    __shared__ __align__(8) uint64_t full[S], empty[S];
    __shared__ int base[S];  // first pair of the stage's tile, -1: too large for a stage
    __shared__ unsigned s_max[2];
    Ctl* const ctl = A.ctl;
    if (is_done(ctl)) return;
    const int tid = threadIdx.x, n = A.n, cap = A.cap, grid = gridDim.x;
    const int tiles = (n + R - 1) / R, mine = (tiles - 1 - (int)blockIdx.x) / grid + 1;  // grid <= tiles
    const int* const roff = A.roff;
    const int4* const off2 = A.off2;
    const float eps = kLoop ? ctl->inner_eps : 0.f;
    const bool producer = tid >= R;
    if (tid == 0) {
        for (int q = 0; q < S; ++q) {
            mbar_init(&full[q], 1);
            mbar_init(&empty[q], R / 32);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (tid < 2) s_max[tid] = 0u;
    __syncthreads();
    // A loop whose tiles all have a stage of their own copies them once.
    const bool resident = kLoop && mine <= S;
    unsigned phase = 0u;      // bit q: parity of stage q's next wait (consumers: full, producer: empty)
    int q = 0, issued = 0;    // producer: stages in use while < S, and tiles copied ahead for the next sweep
    int ahead = 0, copies = 0, b0 = 0, b1 = 0;
    uint64_t policy = 0;
    bool ok = true;
    auto in = [&](int row) { return (unsigned)row < (unsigned)n; };
    auto bounds = [&](int j) {
        const long long t = blockIdx.x + (long long)(j < mine ? j : 0) * grid;
        b0 = __ldg(roff + t * R) >> 1;
        b1 = __ldg(roff + min((long long)n, (t + 1) * R)) >> 1;
    };
    auto issue = [&](int j) {  // tile j of this block; j + 1's bounds are loaded here
        const int e0 = b0, cnt = b1 - b0;
        bounds(j + 1);
        if (issued == S) {
            if (!(ok = mbar_wait(&empty[q], (phase >> q) & 1u, ctl, A.budget))) return;
            phase ^= 1u << q;
        } else {
            ++issued;
        }
        const bool fits = cnt <= cap;
        base[q] = fits ? e0 : -1;
        const unsigned bytes = fits ? (unsigned)cnt * 16u : 0u;
        mbar_expect_tx(&full[q], bytes);
        if (bytes) {
            if ((int)blockIdx.x + j * grid < A.keep) bulk_g2s(stage + (size_t)q * cap, off2 + e0, bytes, &full[q]);
            else bulk_g2s_hint(stage + (size_t)q * cap, off2 + e0, bytes, &full[q], policy);
        }
        ++copies;
        q = q + 1 == S ? 0 : q + 1;
    };
    if (tid == R) {
        policy = evict_first_policy();
        bounds(0);
    }
    int i = blockIdx.x * R + tid, s = 0, e = 0;
    float ri = 0.f, di = 0.f;
    if (!producer && in(i)) {
        s = __ldg(roff + i);
        e = __ldg(roff + i + 1);
        if (NC == 1) ri = A.r[i];
        di = A.invd[i];
    }
    int sweeps = 0;
    const bool any = !kLoop || eps >= 0.f;  // below: the last correction is d0 itself
    while (any) {
        const float* const src = sweeps & 1 ? A.d1 : A.d0;
        float* const dst = sweeps & 1 ? A.d0 : A.d1;
        const bool stats = kLoop ? (sweeps & 1) : A.stats;
        const bool last = !kLoop && A.last;
        float dmax = 0.f, dchg = 0.f;
        if (producer) {
            if (tid == R && !(resident && sweeps)) {
                for (int j = ahead; ok && j < mine; ++j) issue(j);
                ahead = 0;
                if (kLoop && !resident)
                    for (; ok && ahead < S; ++ahead) issue(ahead);  // the next sweep's, before the barrier
            }
            __syncwarp();
        } else {
            if (resident) q = 0;
            for (int j = 0; j < mine; ++j) {
                // the next tile's rows; after the last, the first tile's for the next sweep
                const int inext = j + 1 < mine ? i + grid * R : blockIdx.x * R + tid;
                int sn = 0, en = 0;
                float rn = 0.f, dn = 0.f;
                if (in(inext) && (kLoop || j + 1 < mine)) {
                    sn = __ldg(roff + inext);
                    en = __ldg(roff + inext + 1);
                    if (NC == 1) rn = A.r[inext];
                    dn = A.invd[inext];
                }
                ok = __all_sync(0xffffffffu, mbar_wait(&full[q], (phase >> q) & 1u, ctl, A.budget));
                if (!ok) break;
                if (!resident) phase ^= 1u << q;
                if constexpr (NC == 1) {
                    float sum = 0.f;
                    if (in(i)) {
                        const int e0 = base[q];
                        auto walk = [&](auto entry) {
                            for (int k0 = s; k0 < e; k0 += B) {
                                int4 p[B / 2];
                                float g[B];
#pragma unroll
                                for (int u = 0; u < B / 2; ++u)
                                    p[u] = (k0 + 2 * u < e) ? entry((k0 >> 1) + u) : make_int4(i, 0, i, 0);
#pragma unroll
                                for (int u = 0; u < B / 2; ++u) {
                                    g[2 * u] = (k0 + 2 * u < e) ? src[p[u].x] : 0.f;
                                    g[2 * u + 1] = (k0 + 2 * u < e) ? src[p[u].z] : 0.f;
                                }
#pragma unroll
                                for (int u = 0; u < B / 2; ++u) {
                                    sum = fmaf(__int_as_float(p[u].y), g[2 * u], sum);
                                    sum = fmaf(__int_as_float(p[u].w), g[2 * u + 1], sum);
                                }
                            }
                        };
                        if (e0 >= 0) walk([&](int k) { return stage[q * cap + (k - e0)]; });
                        else walk([&](int k) { return __ldg(off2 + k); });
                    }
                    if (!resident) {
                        __syncwarp();
                        if ((tid & 31) == 0) mbar_arrive(&empty[q]);
                    }
                    if (in(i)) {
                        const float d = (ri - sum) * di;
                        if (stats) {
                            dmax = fmaxf(dmax, fabsf(d));
                            dchg = fmaxf(dchg, fabsf(d - src[i]));
                        }
                        if (last) A.x[i] += (double)d;
                        else dst[i] = d;
                    }
                } else {
                    const int e0 = base[q];
                    for (int c0 = 0; c0 < rhs; c0 += NC) {
                        const size_t row = (size_t)i * rhs + c0;
                        float rc[NC], sum[NC];
#pragma unroll
                        for (int c = 0; c < NC; ++c) {
                            rc[c] = in(i) && c0 + c < rhs ? A.r[row + c] : 0.f;
                            sum[c] = 0.f;
                        }
                        auto walk = [&](auto entry, auto gather) {
                            for (int k0 = s; k0 < e; k0 += B) {
                                int4 p[B / 2];
                                float g[B][NC];
#pragma unroll
                                for (int u = 0; u < B / 2; ++u)
                                    p[u] = (k0 + 2 * u < e) ? entry((k0 >> 1) + u) : make_int4(i, 0, i, 0);
#pragma unroll
                                for (int u = 0; u < B / 2; ++u) {
                                    const bool here = k0 + 2 * u < e;
                                    gather(here, src + (size_t)p[u].x * rhs + c0, g[2 * u]);
                                    gather(here, src + (size_t)p[u].z * rhs + c0, g[2 * u + 1]);
                                }
#pragma unroll
                                for (int u = 0; u < B / 2; ++u)
#pragma unroll
                                    for (int c = 0; c < NC; ++c) {
                                        sum[c] = fmaf(__int_as_float(p[u].y), g[2 * u][c], sum[c]);
                                        sum[c] = fmaf(__int_as_float(p[u].w), g[2 * u + 1][c], sum[c]);
                                    }
                            }
                        };
                        auto staged = [&](int k) { return stage[q * cap + (k - e0)]; };
                        auto direct = [&](int k) { return __ldg(off2 + k); };
                        auto each = [&](bool here, const float* v, float* g) {
#pragma unroll
                            for (int c = 0; c < NC; ++c) g[c] = here && c0 + c < rhs ? v[c] : 0.f;
                        };
                        auto four = [&](bool here, const float* v, float* g) {
                            const float4 w = here ? *reinterpret_cast<const float4*>(v) : make_float4(0.f, 0.f, 0.f, 0.f);
                            g[0] = w.x;
                            g[1] = w.y;
                            g[2] = w.z;
                            g[3] = w.w;
                        };
                        if (rhs % 4 == 0) {
                            if (e0 >= 0) walk(staged, four);
                            else walk(direct, four);
                        } else {
                            if (e0 >= 0) walk(staged, each);
                            else walk(direct, each);
                        }
                        if (!resident && c0 + NC >= rhs) {  // the stage is free
                            __syncwarp();
                            if ((tid & 31) == 0) mbar_arrive(&empty[q]);
                        }
#pragma unroll
                        for (int c = 0; c < NC; ++c)
                            if (in(i) && c0 + c < rhs) {
                                const float d = (rc[c] - sum[c]) * di;
                                if (stats) {
                                    dmax = fmaxf(dmax, fabsf(d));
                                    dchg = fmaxf(dchg, fabsf(d - src[row + c]));
                                }
                                if (last) A.x[row + c] += (double)d;
                                else dst[row + c] = d;
                            }
                    }
                }
                q = q + 1 == S ? 0 : q + 1;
                i = inext;
                s = sn;
                e = en;
                ri = rn;
                di = dn;
            }
        }
        ++sweeps;
        unsigned* const top = !kLoop || (sweeps >> 1) & 1 ? &ctl->dmax_bits : &ctl->dmax2_bits;  // and its neighbour
        if (stats) {
            for (int o = 16; o > 0; o >>= 1) {
                dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
                dchg = fmaxf(dchg, __shfl_xor_sync(0xffffffffu, dchg, o));
            }
            if ((tid & 31) == 0) {
                atomicMax(&s_max[0], __float_as_uint(dmax));
                atomicMax(&s_max[1], __float_as_uint(dchg));
            }
            __syncthreads();
            if (tid < 2) {
                atomicMax(top + tid, s_max[tid]);
                s_max[tid] = 0u;
                // the other pair's maxima: every block has read them (before the first sweep's barrier)
                if (kLoop && blockIdx.x == 0)
                    st_relaxed((int*)(top == &ctl->dmax_bits ? &ctl->dmax2_bits : &ctl->dmax_bits) + tid, 0);
            }
        }
        if (!kLoop) break;
        if (!grid_barrier(ctl, grid, A.budget) || __syncthreads_or(!ok)) break;
        if (stats) {
            const float m = __int_as_float(ld_relaxed((const int*)top)), c = __int_as_float(ld_relaxed((const int*)top + 1));
            if (!(c > fmaxf(A.eps_floor, eps) * m) || sweeps >= A.max_sweeps) break;
        }
    }
    // copies that no sweep took (ahead of one that did not come, after a wait that was given up) land
    // before the block's memory is let go
    if (tid == R)
        for (int z = 0; z < S && z < copies; ++z)
            mbar_drain(&full[z], (unsigned)((copies - z + S - 1) / S - 1) & 1u, A.budget);
    if (!kLoop) return;
    if (!producer) {  // x += d, four loads of each in flight (one: 90 us of the 2M-row solve)
        constexpr int U = 4;
        const size_t total = (size_t)n * rhs, step = (size_t)grid * R;
        for (size_t p = blockIdx.x * (size_t)R + tid; p < total; p += U * step) {
            double xv[U];
            float dv[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (p + u * step < total) {
                    xv[u] = A.x[p + u * step];
                    dv[u] = A.d0[p + u * step];
                }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (p + u * step < total) A.x[p + u * step] = xv[u] + (double)dv[u];
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        ctl->inner_count = sweeps;
        ctl->inner_total += sweeps;
    }
}

// Same sweep, LPR lanes per row over the CSR FP32 values (long rows).
template <int LPR>
__global__ void __launch_bounds__(256) k_jacobi_v(int n, const int* __restrict__ rp, const int* __restrict__ col,
                                                  const float* __restrict__ val, const float* __restrict__ invd,
                                                  const float* __restrict__ r, const float* __restrict__ src,
                                                  float* __restrict__ dst, double* __restrict__ x, int last,
                                                  int stats, Ctl* ctl) {
    __shared__ unsigned s_max[2];
    if (is_done(ctl)) return;
    if (threadIdx.x < 2) s_max[threadIdx.x] = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int gl = lane % LPR;
    const unsigned gmask = (LPR == 32) ? 0xffffffffu : (((1u << LPR) - 1u) << ((lane / LPR) * LPR));
    const long long gid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LPR;
    const long long gstride = ((long long)gridDim.x * blockDim.x) / LPR;
    float dmax = 0.f, dchg = 0.f;
    for (long long i = gid; i < n; i += gstride) {
        const int s = rp[i], e = rp[i + 1];
        float sum = 0.f;
        for (int k = s + 1 + gl; k < e; k += LPR) sum = fmaf(val[k], src[col[k]], sum);
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(gmask, sum, o);
        if (gl == 0) {
            const float d = (r[i] - sum) * invd[i];
            if (stats) {
                dmax = fmaxf(dmax, fabsf(d));
                dchg = fmaxf(dchg, fabsf(d - src[i]));
            }
            if (last) x[i] += (double)d;
            else dst[i] = d;
        }
    }
    if (stats) reduce_stats(dmax, dchg, ctl, s_max);
}

__global__ void __launch_bounds__(256) k_jacobi_m(int n, int rhs, const int* __restrict__ rp,
                                                  const int* __restrict__ col, const float* __restrict__ val,
                                                  const float* __restrict__ invd, const float* __restrict__ r,
                                                  const float* __restrict__ src, float* __restrict__ dst,
                                                  double* __restrict__ x, int last, int stats, Ctl* ctl) {
    __shared__ unsigned s_max[2];
    if (is_done(ctl)) return;
    if (threadIdx.x < 2) s_max[threadIdx.x] = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long ws = ((long long)gridDim.x * blockDim.x) >> 5;
    float dmax = 0.f, dchg = 0.f;
    for (long long i = w; i < n; i += ws) {
        const int s = rp[i], e = rp[i + 1];
        const float di = invd[i];
        for (int c = lane; c < rhs; c += 32) {
            float sum = 0.f;
            for (int k = s + 1; k < e; ++k) sum = fmaf(val[k], src[(size_t)col[k] * rhs + c], sum);
            const size_t p = (size_t)i * rhs + c;
            const float d = (r[p] - sum) * di;
            if (stats) {
                dmax = fmaxf(dmax, fabsf(d));
                dchg = fmaxf(dchg, fabsf(d - src[p]));
            }
            if (last) x[p] += (double)d;
            else dst[p] = d;
        }
    }
    if (stats) reduce_stats(dmax, dchg, ctl, s_max);
}

__global__ void k_axpy_f32(size_t count, const float* __restrict__ d, double* __restrict__ x, const Ctl* ctl) {
    if (is_done(ctl)) return;
    for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < count; p += (size_t)gridDim.x * blockDim.x)
        x[p] += (double)d[p];
}

// Exact inner solves skip themselves once the refinement has converged.
__global__ void k_gate_ticket(Ctl* ctl) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && ctl->done) ctl->ticket = 0xF0000000u;  // no row left to claim
}

// ---------------------------------------------------------------------------------------
static int lpr_for(int n, int nnz) {
    const double mean = n > 0 ? (double)nnz / n : 1.0;
    if (mean <= 6.0) return 4;
    if (mean <= 12.0) return 8;
    if (mean <= 24.0) return 16;
    return 32;
}
// warp tiles pay off while a 32-row tile usually fits the stage
static bool short_rows(const RefineArgs& a) { return (double)a.nnz / a.n <= kShortRowLen; }
static bool use_tiles(const RefineArgs& a) { return short_rows(a) && a.off; }

static int stream_grid(int sm_count) { return sm_count * 8; }

// One resident wave: blocks per SM from the occupancy calculator, times the SM count, so that a
// grid-stride kernel never leaves a partial second wave.
static int resident_grid(const void* fn, int block, int sm_count) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, block, 0) != cudaSuccess || per_sm < 1) per_sm = 1;
    return per_sm * sm_count;
}

int launch_pair_offsets(int n, const int* rp, int* len2, int* roff, int roff_pad, int* part, int sm_count,
                        cudaStream_t st, int64_t* launches) {
    k_pair_len<<<sm_count * 4, 256, 0, st>>>(n, rp, len2);
    ++*launches;
    CUDA_TRY(cudaGetLastError());
    int rc = scan_exclusive(len2, roff, n, part, st, launches);
    if (rc) return rc;
    k_pad_roff<<<1, 64, 0, st>>>(n, roff_pad, roff);
    ++*launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int launch_build_offdiag_pairs(int n, const int* rp, const int* col, const double* val, const int* roff, int2* off,
                               int sm_count, cudaStream_t st, int64_t* launches) {
    k_build_offdiag_pairs<<<sm_count * 8, 256, 0, st>>>(n, rp, col, val, roff, off);
    ++*launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int launch_jds_sizes(int n, const int* rp, int* gsize, int* overflow, int sm_count, cudaStream_t st,
                     int64_t* launches) {
    const int ngroups = (n + 31) / 32;
    k_jds_sizes<<<sm_count * 8, 256, 0, st>>>(n, ngroups, rp, gsize, overflow);
    ++*launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int launch_jds_fill(int n, const int* rp, const int* col, const double* val, const int* jbase, int* jmeta, int2* jent,
                    int sm_count, cudaStream_t st, int64_t* launches) {
    const int ngroups = (n + 31) / 32;
    k_jds_fill<<<sm_count * 8, 256, 0, st>>>(n, ngroups, rp, col, val, jbase, jmeta, jent);
    ++*launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int launch_build_offdiag(int n, const int* rp, const int* col, const double* val, int2* off, int* roff,
                         int roff_pad, int sm_count, cudaStream_t st, int64_t* launches) {
    k_build_offdiag<<<sm_count * 8, 256, 0, st>>>(n, rp, col, val, off);
    k_build_roff<<<sm_count * 4, 256, 0, st>>>(n, roff_pad, rp, roff);
    *launches += 2;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

__global__ void k_mark_x_zero(Ctl* ctl) {
    if (threadIdx.x == 0 && blockIdx.x == 0) ctl->x_zero = 1;
}

// x = 0, ||b_c||^2; the device-looped graphs also mark x as zero so that their first residual
// is taken from b without reading the matrix.
int launch_refine_init(const RefineArgs& a, bool mark_zero) {
    CUDA_TRY(cudaMemsetAsync(a.x, 0, sizeof(double) * (size_t)a.n * a.rhs, a.st));
    if (mark_zero) {
        k_mark_x_zero<<<1, 32, 0, a.st>>>(a.ctl);
        ++*a.launches;
    }
    CUDA_TRY(cudaMemsetAsync(a.rn2, 0, sizeof(double) * a.rhs, a.st));
    CUDA_TRY(cudaMemsetAsync(a.bn2, 0, sizeof(double) * a.rhs, a.st));
    k_colnorm2<<<stream_grid(a.sm_count), 256, sizeof(double) * a.rhs, a.st>>>(a.n, a.rhs, a.b, a.bn2);
    ++*a.launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

// seed: 0 none, 1 Jacobi d0 = D^{-1} r into d32[0], 2 pending fill of d32[0].
int launch_residual(const RefineArgs& a, bool jacobi_seed, int final_check) {
    const int seed = final_check ? 0 : (jacobi_seed ? 1 : 2);
    const int grid = stream_grid(a.sm_count);
    if (short_rows(a) && a.rhs == 1) {
        static int grid_rt = 0;
        if (!grid_rt) grid_rt = resident_grid((const void*)k_residual_tile, kResWarps * 32, a.sm_count);
        k_residual_tile<<<grid_rt, kResWarps * 32, 0, a.st>>>(a.n, a.rp, a.col, a.val, a.invd32, a.b, a.x,
                                                                      a.x_out, a.r32, a.d32[0], seed, a.rn2, a.ctl);
    } else if (short_rows(a) && a.off) {
        const size_t smem = sizeof(double) * a.rhs;
        int per_sm = 0;
        CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_residual_tile_m, kResWarps * 32, smem));
        k_residual_tile_m<<<std::max(1, per_sm) * a.sm_count, kResWarps * 32, smem, a.st>>>(
            a.n, a.rhs, a.rp, a.col, a.val, a.invd32, a.b, a.x, a.r32, a.d32[0], seed, a.rn2, a.ctl);
    } else if (a.rhs == 1) {
        switch (lpr_for(a.n, a.nnz)) {
            case 4: k_residual_v<4><<<grid, 256, 0, a.st>>>(a.n, a.rp, a.col, a.val, a.invd32, a.b, a.x, a.x_out, a.r32, a.d32[0], seed, a.rn2, a.ctl); break;
            case 8: k_residual_v<8><<<grid, 256, 0, a.st>>>(a.n, a.rp, a.col, a.val, a.invd32, a.b, a.x, a.x_out, a.r32, a.d32[0], seed, a.rn2, a.ctl); break;
            case 16: k_residual_v<16><<<grid, 256, 0, a.st>>>(a.n, a.rp, a.col, a.val, a.invd32, a.b, a.x, a.x_out, a.r32, a.d32[0], seed, a.rn2, a.ctl); break;
            default: k_residual_v<32><<<grid, 256, 0, a.st>>>(a.n, a.rp, a.col, a.val, a.invd32, a.b, a.x, a.x_out, a.r32, a.d32[0], seed, a.rn2, a.ctl); break;
        }
    } else {
        k_residual_m<<<grid, 256, sizeof(double) * a.rhs, a.st>>>(a.n, a.rhs, a.rp, a.col, a.val, a.invd32, a.b, a.x,
                                                                  a.r32, a.d32[0], seed, a.rn2, a.ctl);
    }
    ++*a.launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int launch_check(const RefineArgs& a, int step, bool reset_ticket) {
    k_check<<<1, 32, 0, a.st>>>(a.rhs, a.rn2, a.bn2, a.ctl, a.tol, step, reset_ticket ? 1 : 0);
    ++*a.launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int launch_check_outer(const RefineArgs& a, int max_refine, cudaGraphConditionalHandle ho,
                       cudaGraphConditionalHandle hi) {
    k_check_outer<<<1, 32, 0, a.st>>>(a.rhs, a.rn2, a.bn2, a.ctl, a.tol, max_refine, ho, hi);
    ++*a.launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int launch_check_inner(const RefineArgs& a, float eps, int max_sweeps, cudaGraphConditionalHandle hi) {
    k_check_inner<<<1, 32, 0, a.st>>>(a.ctl, eps, max_sweeps, hi);
    ++*a.launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

// The launch shape of k_jacobi_bulk.
template <int R, int S>
struct BulkShape {
    int cap, tiles, keep;
    size_t smem;
    // a stage holds the mean tile (half a row's entries and pads) and a tenth more; larger tiles are
    // read from global memory.  At most 61 KB (kShortRowLen).
    static int pairs(double mean_len) { return (int)(R * 0.55 * (mean_len - 0.45)) + 16; }
    explicit BulkShape(const RefineArgs& a) {
        cap = pairs((double)a.nnz / a.n);
        smem = (size_t)cap * 16 * S;
        tiles = (int)(((long long)a.n + R - 1) / R);
        const double bytes = 8.0 * ((double)a.nnz - 0.5 * a.n), room = 60e6 - (4.0 + 12.0 * a.rhs) * a.n;
        keep = room >= bytes ? tiles : room <= 0.0 ? 0 : (int)(tiles * (room / bytes));
    }
    BulkArgs args(const RefineArgs& a) const {
        BulkArgs A{};
        A.n = a.n;
        A.rhs = a.rhs;
        A.cap = cap;
        A.keep = keep;
        A.roff = a.roff;
        A.off2 = reinterpret_cast<const int4*>(a.off);
        A.invd = a.invd32;
        A.r = a.r32;
        A.x = a.x;
        A.ctl = a.ctl;
        A.budget = std::max<int64_t>(a.budget, kDefaultBudgetNs);  // a caller's budget is for waits on rows
        return A;
    }
    int grid(const void* fn, const RefineArgs& a, int* blocks) const {
        int per_sm = 0;
        // (the limit belongs to the kernel on the device: the largest any matrix asks for, for every thread's
        // launches)
        CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, pairs(kShortRowLen) * 16 * S));
        CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, R + 32, smem));
        if (per_sm < 1) return SPTRSV_ERR_UNSUPPORTED;
        *blocks = std::min(tiles, per_sm * a.sm_count);
        return 0;
    }
};

// Whether the inner solve runs as one launch (launch_jacobi_loop).
bool refine_loops(const RefineArgs& a) { return use_tiles(a) && !a.jmeta && a.roff && a.pairs; }

int launch_jacobi_loop(const RefineArgs& a, float eps, int max_sweeps) {
    constexpr int R = 256, S = 2;
    const BulkShape<R, S> shape(a);
    BulkArgs A = shape.args(a);
    A.d0 = a.d32[0];
    A.d1 = a.d32[1];
    A.eps_floor = eps;
    A.max_sweeps = max_sweeps;
    const void* fn = a.rhs == 1 ? (const void*)k_jacobi_bulk<R, S, 4, true, 1> : (const void*)k_jacobi_bulk<R, S, 3, true, 4>;
    int blocks;
    int rc = shape.grid(fn, a, &blocks);
    if (rc) return rc;
    void* args[] = {(void*)&A};
    CUDA_TRY(launch_cooperative(fn, blocks, R + 32, args, shape.smem, a.st));
    ++*a.launches;
    return 0;
}

int launch_jacobi_sweep(const RefineArgs& a, int src, bool last, bool stats) {
    const int grid = stream_grid(a.sm_count);
    const float* s = a.d32[src];
    float* d = a.d32[src ^ 1];
    const int st_flag = stats ? 1 : 0;
    if (use_tiles(a) && a.jmeta) {  // (the layouts other than the paired one: one right-hand side)
        static int grid_j6 = 0;
        if (!grid_j6) grid_j6 = resident_grid((const void*)k_jacobi_jds<6, 6>, 256, a.sm_count);
        k_jacobi_jds<6, 6><<<grid_j6, 256, 0, a.st>>>(a.n, (a.n + 31) / 32, a.jmeta, a.jbase, a.off, a.invd32, a.r32, s,
                                                     d, a.x, last, st_flag, a.ctl);
    } else if (use_tiles(a) && a.roff && a.pairs) {
        constexpr int R = 128, S = 2;
        const BulkShape<R, S> shape(a);
        BulkArgs A = shape.args(a);
        A.d0 = a.d32[src];
        A.d1 = d;
        A.last = last;
        A.stats = st_flag;
        void (*fn)(BulkArgs) = a.rhs == 1 ? k_jacobi_bulk<R, S, 8, false, 1> : k_jacobi_bulk<R, S, 6, false, 4>;
        int blocks;
        int rc = shape.grid((const void*)fn, a, &blocks);
        if (rc) return rc;
        fn<<<blocks, R + 32, shape.smem, a.st>>>(A);
    } else if (use_tiles(a) && a.roff && (a.sweep_kernel == 7)) {
        static int grid_b4 = 0;
        if (!grid_b4) grid_b4 = resident_grid((const void*)k_jacobi_batched<4, 8>, 256, a.sm_count);
        k_jacobi_batched<4, 8><<<grid_b4, 256, 0, a.st>>>(a.n, a.roff, a.off, a.invd32, a.r32, s, d, a.x, last,
                                                         st_flag, a.ctl);
    } else if (use_tiles(a) && a.roff && (a.sweep_kernel == 8 || a.sweep_kernel == 0)) {
        static int grid_b8 = 0;
        if (!grid_b8) grid_b8 = resident_grid((const void*)k_jacobi_batched<8, 6>, 256, a.sm_count);
        k_jacobi_batched<8, 6><<<grid_b8, 256, 0, a.st>>>(a.n, a.roff, a.off, a.invd32, a.r32, s, d, a.x, last,
                                                         st_flag, a.ctl);
    } else if (a.rhs == 1 && a.sell && a.sweep_kernel == 6) {
        static int grid_s = 0;
        if (!grid_s) grid_s = resident_grid((const void*)k_jacobi_sell, 256, a.sm_count);
        k_jacobi_sell<<<grid_s, 256, 0, a.st>>>(a.nslices, a.sell_perm, a.sell_len, a.sell_ptr, a.sell, a.invd32, a.r32,
                                                s, d, a.x, last, st_flag, a.ctl);
    } else if (use_tiles(a) && a.roff && a.sweep_kernel == 4) {
        static int grid_d2 = 0;
        if (!grid_d2) grid_d2 = resident_grid((const void*)k_jacobi_direct2, 256, a.sm_count);
        k_jacobi_direct2<<<grid_d2, 256, 0, a.st>>>(a.n, a.roff, a.off, a.invd32, a.r32, s, d, a.x, last, st_flag,
                                                   a.ctl);
    } else if (use_tiles(a) && a.roff && a.sweep_kernel == 2) {
        static int grid_d = 0;
        if (!grid_d) grid_d = resident_grid((const void*)k_jacobi_direct, 256, a.sm_count);
        k_jacobi_direct<<<grid_d, 256, 0, a.st>>>(a.n, a.roff, a.off, a.invd32, a.r32, s, d, a.x, last, st_flag, a.ctl);
    } else if (use_tiles(a) && a.sweep_kernel == 3) {
        static int grid_t8 = 0;
        if (!grid_t8) grid_t8 = resident_grid((const void*)k_jacobi_tile<384, 8>, kJacWarps * 32, a.sm_count);
        k_jacobi_tile<384, 8><<<grid_t8, kJacWarps * 32, 0, a.st>>>(a.n, a.rp, a.off, a.invd32, a.r32, s, d, a.x,
                                                                   last, st_flag, a.ctl);
    } else if (use_tiles(a)) {
        static int grid_jt = 0;
        if (!grid_jt) grid_jt = resident_grid((const void*)k_jacobi_tile<kTileMax, 1>, kJacWarps * 32, a.sm_count);
        k_jacobi_tile<kTileMax, 1><<<grid_jt, kJacWarps * 32, 0, a.st>>>(a.n, a.rp, a.off, a.invd32, a.r32, s, d, a.x, last,
                                                                  st_flag, a.ctl);
    } else if (a.rhs == 1) {
        switch (lpr_for(a.n, a.nnz)) {
            case 4: k_jacobi_v<4><<<grid, 256, 0, a.st>>>(a.n, a.rp, a.col, a.val32, a.invd32, a.r32, s, d, a.x, last, st_flag, a.ctl); break;
            case 8: k_jacobi_v<8><<<grid, 256, 0, a.st>>>(a.n, a.rp, a.col, a.val32, a.invd32, a.r32, s, d, a.x, last, st_flag, a.ctl); break;
            case 16: k_jacobi_v<16><<<grid, 256, 0, a.st>>>(a.n, a.rp, a.col, a.val32, a.invd32, a.r32, s, d, a.x, last, st_flag, a.ctl); break;
            default: k_jacobi_v<32><<<grid, 256, 0, a.st>>>(a.n, a.rp, a.col, a.val32, a.invd32, a.r32, s, d, a.x, last, st_flag, a.ctl); break;
        }
    } else {
        k_jacobi_m<<<grid, 256, 0, a.st>>>(a.n, a.rhs, a.rp, a.col, a.val32, a.invd32, a.r32, s, d, a.x, last,
                                           st_flag, a.ctl);
    }
    ++*a.launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int launch_axpy_pending(const RefineArgs& a, int src) {
    const size_t count = (size_t)a.n * a.rhs;
    const int blocks = (int)std::min<size_t>((count + 255) / 256, (size_t)a.sm_count * 8);
    k_axpy_f32<<<blocks, 256, 0, a.st>>>(count, a.d32[src], a.x, a.ctl);
    ++*a.launches;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int launch_exact_inner(const RefineArgs& a, int schedule, int rows_per_warp, int dst, int max_level,
                       const int* lptr, const int* lrows, int warps) {
    SolveArgs s{};
    s.n = a.n;
    s.rp = a.rp;
    s.col = a.col;
    s.val = a.val32;
    s.invd = a.invd32;
    s.b = a.r32;
    s.x = a.d32[dst];
    s.rhs = a.rhs;
    s.ctl = a.ctl;
    s.budget = a.budget;
    s.sm_count = a.sm_count;
    s.warps = warps;
    s.nnz = a.nnz;
    s.st = a.st;
    s.launches = a.launches;
    if (schedule == SPTRSV_SCHED_LEVELSET) return launch_levelset(true, s, max_level, lptr, lrows);
    k_gate_ticket<<<1, 32, 0, a.st>>>(a.ctl);
    ++*a.launches;
    if (schedule == SPTRSV_SCHED_SYNCFREE_THREAD && a.rhs == 1) return launch_pull_thread(true, s);
    if (schedule == SPTRSV_SCHED_SYNCFREE_BLOCK && a.rhs == 1) return launch_bsf(true, s);
    if (schedule == SPTRSV_SCHED_SYNCFREE_WINDOW && a.rhs == 1) return launch_window(true, s);
    return launch_pull_warp(true, s, rows_per_warp, 0);
}

}  // namespace sptrsv
