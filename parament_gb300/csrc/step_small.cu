// Fused plain-path kernel for d <= 64: Hamiltonian assembly, Chebyshev
// (Clenshaw) exponential and the running product of a chunk of consecutive
// steps, all resident in shared memory.  One CTA owns one chunk; nothing but
// the samples is read from HBM per step (the expansion stack stays in L2) and
// one d x d product per chunk is written back.
//
// Replaces, for small d, the reference's expansion GEMMs and quadrature kernels
// (src/cuda/parament.cpp:486-563, src/cuda/control_expansion.cu:27-170), the
// batched Clenshaw GEMMs plus diagonal adds (src/cuda/parament.cpp:569-652,
// src/cuda/diagonal_add.cu:21-51) and the lower levels of the tree product
// (src/cuda/parament.cpp:657-718).
//
// For x = Hnorm h <= 1 and orders from 5 on the polynomial is evaluated by powers
// of X (as in step_group.cu, with the same coefficients),
//     Y = X^2,  r = c_M X Y + c_(M-1) Y + c_(M-2) X + c_(M-3),
//     r <- r Y + c_(k+1) X + c_k,
// (M + 1) / 2 products instead of M - 1; at order 3 both take two.  The products are
// what the kernel spends its time on (the FP64 pipe in complex128, shared-memory
// loads and FMAs in complex64): d = 16, K = 2, 4096 steps in complex128 (order 5),
// 777 -> 640 us.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "ctx.h"
#include "kernels.h"

namespace pgb {

template <class R>
struct SmallArgs {
    cplx_t<R> J[kMaxOrder + 1];
    R c[kMaxOrder + 1];  // by powers: c_n (odd n: times i); c_0 of E (complex128) or of U - J_0
    R low[2];            // complex64: what FP32 leaves of c_1 and c_2
    const cplx_t<R> *stack;
    const cplx_t<R> *carr;
    cplx_t<R> *chunks;
    long long P;
    int nchunks;
    int d, Ke, M;
    R s;
    WeightSpec w;
};

// Complex64 instances keep to 128 registers so that two CTAs share an SM.
template <class R, int TM, bool POWERS>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 2 : 1) k_small_steps(const __grid_constant__ SmallArgs<R> a) {
    using C = cplx_t<R>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int d = a.d, dd = d * d, ld = d + 1, sz = d * ld;
    C *Xs = reinterpret_cast<C *>(smem_raw);
    C *Bs = Xs + sz;
    C *Ps = Bs + sz;
    C *ws = Ps + sz;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const long long s0 = a.P * blockIdx.x / a.nchunks;
    const long long s1 = a.P * (blockIdx.x + 1) / a.nchunks;
    const int M = a.M;
    const R s = a.s;

    bool own[TM][TM];
    int eo[TM][TM];  // shared-memory index (stride ld); the global index is r*d+c
    bool diag[TM][TM];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TM; ++j) {
            int r = ty + 16 * i, c = tx + 16 * j;
            own[i][j] = (r < d) && (c < d);
            eo[i][j] = r * ld + c;
            diag[i][j] = (r == c);
        }

    C b2[TM][TM], acc[TM][TM];
    for (long long st = s0; st < s1; ++st) {
        for (int m = tid; m < a.Ke; m += blockDim.x) ws[m] = step_weight(a.carr, a.w, m, st);
        __syncthreads();
        if constexpr (POWERS) {
            // complex64 forms U, adding J_0 last, as the recurrence below does;
            // complex128 forms E = U - I.
            constexpr bool kHasU = sizeof(R) == 4;
            C x[TM][TM];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TM; ++j) {
                    if (!own[i][j]) continue;
                    const int ge = (ty + 16 * i) * d + tx + 16 * j;
                    C v = a.stack[ge];
                    for (int m = 0; m < a.Ke; ++m) cfma(v, ws[m], a.stack[(size_t)(m + 1) * dd + ge]);
                    x[i][j] = v;
                    Xs[eo[i][j]] = v;
                }
            __syncthreads();
            tile_gemm<C, TM>(acc, Xs, Xs, d, ld, ty, tx);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TM; ++j)
                    if (own[i][j]) Bs[eo[i][j]] = b2[i][j] = acc[i][j];  // Y
            __syncthreads();
            tile_gemm<C, TM>(acc, Xs, Bs, d, ld, ty, tx);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TM; ++j) {
                    if (!own[i][j]) continue;
                    const C q = acc[i][j], y = b2[i][j], v = x[i][j];
                    C r;
                    r.x = fma(a.c[M - 1], y.x, -a.c[M] * q.y) - a.c[M - 2] * v.y;
                    r.y = fma(a.c[M - 1], y.y, a.c[M] * q.x) + a.c[M - 2] * v.x;
                    if (diag[i][j]) r.x += a.c[M - 3];
                    acc[i][j] = r;
                }
            for (int k = M - 5; k >= 0; k -= 2) {
                __syncthreads();
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TM; ++j)
                        if (own[i][j]) Xs[eo[i][j]] = acc[i][j];
                __syncthreads();
                tile_gemm<C, TM>(acc, Xs, Bs, d, ld, ty, tx);
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TM; ++j) {
                        if (!own[i][j]) continue;
                        C r = acc[i][j];
                        if (kHasU && k == 0) {
                            const C y = Bs[eo[i][j]];
                            r.x = fma(a.low[1], y.x, fma(-a.low[0], x[i][j].y, r.x));
                            r.y = fma(a.low[1], y.y, fma(a.low[0], x[i][j].x, r.y));
                        }
                        r.x = fma(-a.c[k + 1], x[i][j].y, r.x);
                        r.y = fma(a.c[k + 1], x[i][j].x, r.y);
                        if (diag[i][j]) {
                            r.x += a.c[k];
                            if (kHasU && k == 0) r.x += a.J[0].x;
                            if (!kHasU && k == 0 && st == s0) r.x += (R)1;  // the first step's P
                        }
                        acc[i][j] = r;
                    }
            }
            __syncthreads();
        } else {
            // X = H0 + sum_m w_m H_m (own elements), straight from the L2-resident
            // stack; b_M = J[M] I and b_(M-1) = s J[M] X + J[M-1] I need only the
            // thread's own elements, so they are formed in the same pass.
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TM; ++j) {
                    if (!own[i][j]) continue;
                    const int e = eo[i][j];
                    const int ge = (ty + 16 * i) * d + tx + 16 * j;
                    C v = a.stack[ge];
                    for (int m = 0; m < a.Ke; ++m) cfma(v, ws[m], a.stack[(size_t)(m + 1) * dd + ge]);
                    Xs[e] = v;
                    C bm1 = cscale(cmul(a.J[M], v), s);
                    if (diag[i][j]) bm1 = cadd(bm1, a.J[M - 1]);
                    if (M == 1) {
                        acc[i][j] = bm1;  // U = s J[1] X + J[0] I, since b_2 = 0
                    } else {
                        b2[i][j] = diag[i][j] ? a.J[M] : mk<C>(0.0, 0.0);
                        Bs[e] = bm1;
                    }
                }
            if (M > 1) {
                __syncthreads();
                for (int k = M - 2; k >= 0; --k) {
                    tile_gemm<C, TM>(acc, Bs, Xs, d, ld, ty, tx);
                    __syncthreads();
                    const R beta = (k == 0) ? (R)-2 : (R)-1;
#pragma unroll
                    for (int i = 0; i < TM; ++i)
#pragma unroll
                        for (int j = 0; j < TM; ++j) {
                            if (!own[i][j]) continue;
                            C v = cscale(acc[i][j], s);
                            v.x += beta * b2[i][j].x;
                            v.y += beta * b2[i][j].y;
                            if (diag[i][j]) v = cadd(v, a.J[k]);
                            if (k > 0) {
                                b2[i][j] = Bs[eo[i][j]];
                                Bs[eo[i][j]] = v;
                            } else {
                                acc[i][j] = v;  // U_j
                            }
                        }
                    if (k > 0) __syncthreads();
                }
            }
        }
        // Chunk product P <- U_j P (later step on the left).
        if (st == s0) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TM; ++j)
                    if (own[i][j]) Ps[eo[i][j]] = acc[i][j];
            __syncthreads();
        } else {
            // U P = P + (U - I) P: the near-identity factor enters the sums
            // without its unit diagonal, so sequential accumulation does not
            // round small contributions against 1 (that bias adds up
            // coherently over thousands of steps in FP32).
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TM; ++j)
                    if (own[i][j]) {
                        C u = acc[i][j];
                        if (diag[i][j] && !(POWERS && sizeof(R) == 8)) u.x -= (R)1;
                        Bs[eo[i][j]] = u;
                    }
            __syncthreads();
            tile_gemm<C, TM>(acc, Bs, Ps, d, ld, ty, tx);
            __syncthreads();
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TM; ++j)
                    if (own[i][j]) Ps[eo[i][j]] = cadd(Ps[eo[i][j]], acc[i][j]);
            __syncthreads();
        }
    }
    if (s1 > s0) {
        C *dst = a.chunks + (size_t)blockIdx.x * dd;
        for (int e = tid; e < dd; e += blockDim.x) dst[e] = Ps[(e / d) * ld + e % d];
    }
}

size_t small_smem_bytes(bool fp64, int d, int Ke) {
    size_t c = fp64 ? 16 : 8;
    return c * (3 * (size_t)d * (d + 1) + (size_t)Ke);
}

template <class R, int TM>
static const void *small_kernel_ptr(bool powers) {
    return powers ? reinterpret_cast<const void *>(&k_small_steps<R, TM, true>)
                  : reinterpret_cast<const void *>(&k_small_steps<R, TM, false>);
}

static const void *pick_small(bool fp64, int d, bool powers) {
    int tm = (d + 15) / 16;
    if (fp64) {
        switch (tm) {
            case 1: return small_kernel_ptr<double, 1>(powers);
            case 2: return small_kernel_ptr<double, 2>(powers);
            case 3: return small_kernel_ptr<double, 3>(powers);
            default: return small_kernel_ptr<double, 4>(powers);
        }
    }
    switch (tm) {
        case 1: return small_kernel_ptr<float, 1>(powers);
        case 2: return small_kernel_ptr<float, 2>(powers);
        case 3: return small_kernel_ptr<float, 3>(powers);
        default: return small_kernel_ptr<float, 4>(powers);
    }
}

// The polynomial by powers of X: l.x is set, and it saves products.
static bool small_powers(const StepLaunch &l) { return l.x > 0.0 && l.x <= 1.0 && l.M >= 5; }

int small_chunk_count(bool fp64, int d, int Ke, long long P, int num_sms) {
    const void *fn = pick_small(fp64, d, true);
    size_t smem = small_smem_bytes(fp64, d, Ke);
    allow_smem(fn);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 256, smem) != cudaSuccess || per_sm < 1) per_sm = 1;
    long long n = (long long)per_sm * num_sms;
    return (int)std::max<long long>(1, std::min<long long>(n, P));
}

template <class R>
static cudaError_t launch_small_t(const StepLaunch &l) {
    using C = cplx_t<R>;
    SmallArgs<R> a;
    for (int k = 0; k <= l.M; ++k) a.J[k] = mk<C>(l.J[2 * k], l.J[2 * k + 1]);
    a.stack = static_cast<const C *>(l.stack);
    a.carr = static_cast<const C *>(l.carr);
    a.chunks = static_cast<C *>(l.chunks);
    a.P = l.P;
    a.nchunks = l.nchunks;
    a.d = l.d;
    a.Ke = l.Ke;
    a.M = l.M;
    a.s = (R)l.s;
    a.w = WeightSpec{l.w.pts, l.w.K, l.w.amps, l.w.mode, l.w.magnus, l.w.hfac};
    size_t smem = small_smem_bytes(l.fp64, l.d, l.Ke);
    const bool powers = small_powers(l);
    if (powers && l.fp64) {
        double c0[2];
        std::vector<double> mu;
        power_coefficients(l.M, l.x, 2.0 / l.s, c0, mu);
        a.c[0] = (R)c0[0];
        for (int n = 1; n <= l.M; ++n) a.c[n] = (R)mu[2 * n + (n & 1)];
    } else if (powers) {
        std::vector<double> c;
        plain_coefficients(l.M, l.x, 2.0 / l.s, c);
        for (int n = 0; n <= l.M; ++n) a.c[n] = (R)c[n];
        for (int n = 1; n <= 2; ++n) a.low[n - 1] = (R)low_part(c[n]);
    }
    const void *fn = pick_small(l.fp64, l.d, powers);
    cudaError_t e = allow_smem(fn);
    if (e != cudaSuccess) return e;
    void *args[] = {&a};
    return cudaLaunchKernel(fn, dim3(l.nchunks), dim3(256), args, smem, l.stream);
}

cudaError_t launch_small_steps(const StepLaunch &l) {
    if (l.d < 1 || l.d > kSmallMaxDim || l.M < 1 || l.M > kMaxOrder || l.nchunks < 1) return cudaErrorInvalidValue;
    return l.fp64 ? launch_small_t<double>(l) : launch_small_t<float>(l);
}

}  // namespace pgb
