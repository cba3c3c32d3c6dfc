// Whole propagations of small problems in one launch: d <= 8, x = Hnorm h <= 1.
//
// A group of 16 threads (half a warp) owns a chunk of consecutive steps; a thread
// keeps a TM x TM micro-tile (4 TM >= d) of every matrix, rows ty + 4 i and column
// pairs 2 tx + 8 j.  Groups share a CTA and the expansion stack in shared memory,
// and meet only within themselves.
//
// The scheme is that of k_small_steps (step_small.cu; src/cuda/parament.cpp:486-718)
// with the step's Chebyshev-Bessel polynomial regrouped by powers of X (as in
// fx.cu: no cancellation for x <= 1),
//     Y = X^2,  r = c_M X Y + c_(M-1) Y + c_(M-2) X + c_(M-3),
//     r <- r Y + c_(k+1) X + c_k,   E_j = U_j - I,
// (M + 1) / 2 products instead of M - 1, and the running product of the chunk as
// P <- P + E P.  complex128 keeps E_j and P - I (the unit diagonal never meets
// the small terms); complex64 forms U_j, with the coefficients that the Clenshaw
// kernels have, and rounds it as they do.
//
// The chunk products meet without another launch.  The group that finds the
// product beside its own finished goes on with the pair, the other one ends:
// nobody waits.  In double-float (complex64) or FP64, as k_tree_df and tree_product do:
// the nodes are products and not their distances from I, which would leave a propagator
// of size 1e-10 good to 1e-6 of itself.
//
// What bounds it: latency.  A qubit's 100 steps took 71 us with host buffers, ten
// launches (256 threads per chunk, a launch per level of the tree) between two
// copies; they take 40 us with one.  Above d = 8 the pair of a level takes one
// group longer than a launch over several SMs, and groups of 64 threads with 4 x
// 4 tiles (d = 27: 217 us against 195) or 2 x 2 in complex128 (d = 16: 833 against
// 775) were no faster than 256 threads per chunk.
#include <math.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "ctx.h"
#include "kernels.h"
#include "split_common.cuh"

namespace pgb {

constexpr int kGroupStackBytes = 96 << 10;  // largest stack kept in shared memory

template <class R>
struct GroupArgs {
    R c[kMaxOrder + 1];  // c_n, real for even n, imaginary for odd n; c_0 of E (complex128) or of U - J_0
    R low[2];            // complex64: what FP32 leaves of c_1 and c_2
    R j0;                // complex64: J_0, added last
    const cplx_t<R> *stack, *carr;
    void *nodes;         // nodes of the tree, float4 (double-float) or double2
    // A pair's first arrival leaves the launch's turn there, the second finds it and
    // leaves zero.  What launches that overlapped on one context may leave behind has
    // another turn and counts for nothing.
    unsigned *arrived, turn;
    cplx_t<R> *out;
    long long P;
    int nchunks, d, Ke, M, ld, stack_smem;
    WeightSpec w;
};

constexpr int kGroupSide = 4, kGroupThreads = 16;

__device__ __forceinline__ void group_sync(int g) { __syncwarp(0xFFFFu << (16 * (g & 1))); }

// Node of the tree: double-float for complex64, FP64 for complex128.
template <class R>
struct Node;
template <>
struct Node<float> {
    using T = float4;
    __device__ static T make(float2 v, bool) { return make_float4(v.x, 0.f, v.y, 0.f); }
    // a b as b + (a - I) b
    __device__ static T left(T a, bool diag) {
        const df r = diag ? df_add_f(df{a.x, a.y}, -1.0f) : df{a.x, a.y};
        return make_float4(r.hi, r.lo, a.z, a.w);
    }
    __device__ static T start(T b) { return b; }
    __device__ static void mac1(float &hi, float &lo, float xh, float xl, float yh, float yl) {
        const float p = __fmul_rn(xh, yh);
        float e = __fmaf_rn(xh, yh, -p);
        e = __fmaf_rn(xh, yl, e);
        e = __fmaf_rn(xl, yh, e);
        float s, t;
        two_sum(hi, p, s, t);
        hi = s;
        lo = __fadd_rn(lo, __fadd_rn(t, e));
    }
    __device__ static void mac(T &c, T a, T b) {
        mac1(c.x, c.y, a.x, a.y, b.x, b.y);
        mac1(c.x, c.y, -a.z, -a.w, b.z, b.w);
        mac1(c.z, c.w, a.x, a.y, b.z, b.w);
        mac1(c.z, c.w, a.z, a.w, b.x, b.y);
    }
    __device__ static T norm(T v) {
        const df r = df_norm(v.x, v.y), i = df_norm(v.z, v.w);
        return make_float4(r.hi, r.lo, i.hi, i.lo);
    }
    // Rounded once.
    __device__ static float2 out(T v) { return make_float2(__fadd_rn(v.x, v.y), __fadd_rn(v.z, v.w)); }
};
template <>
struct Node<double> {
    using T = double2;
    // The chunk product from it less I.
    __device__ static T make(double2 v, bool diag) {
        if (diag) v.x += 1.0;
        return v;
    }
    __device__ static T left(T a, bool) { return a; }
    __device__ static T start(T) { return make_double2(0.0, 0.0); }
    __device__ static void mac(T &c, T a, T b) { cfma(c, a, b); }
    __device__ static T norm(T v) { return v; }
    __device__ static double2 out(T v) { return v; }
};

template <class R, int TM>
__global__ void __launch_bounds__(384) k_group_steps(const __grid_constant__ GroupArgs<R> a) {
    using C = cplx_t<R>;
    constexpr int T = kGroupSide, NT = kGroupThreads;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int d = a.d, dd = d * d, ld = a.ld, sz = d * ld;
    const int g = threadIdx.x / NT, gt = threadIdx.x % NT, ngroups = blockDim.x / NT;
    const int ty = gt / T, tx = gt % T;
    C *Sm = reinterpret_cast<C *>(smem_raw);  // the stack, rows as they are
    const int per = 4 * sz + max(2, (a.Ke + 1) & ~1);
    C *Xs = Sm + (a.stack_smem ? ((1 + a.Ke) * dd + 1) / 2 * 2 : 0) + (size_t)g * per;
    C *Ys = Xs + sz, *Rs = Ys + sz, *Ps = Rs + sz, *ws = Ps + sz;
    if (a.stack_smem) {
        for (int i = threadIdx.x; i < (1 + a.Ke) * dd; i += blockDim.x) Sm[i] = a.stack[i];
        __syncthreads();
    }
    const C *stack = a.stack_smem ? Sm : a.stack;
    const long long chunk = (long long)blockIdx.x * ngroups + g;
    if (chunk >= a.nchunks) return;
    const long long s0 = a.P * chunk / a.nchunks, s1 = a.P * (chunk + 1) / a.nchunks;
    const int M = a.M;

    // Own elements: row(i), col(j); reads past d are clamped, their results dropped.
    auto row = [&](int i) { return ty + T * i; };
    auto col = [&](int j) { return TM == 1 ? tx : 2 * tx + (j & 1) + 2 * T * (j >> 1); };
    int ro[TM], co[TM];
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        ro[i] = min(row(i), d - 1) * ld;
        co[i] = min(col(i), d - 1);
    }
    auto own = [&](int i, int j) { return row(i) < d && col(j) < d; };
    // acc = A B
    auto gemm = [&](C(&acc)[TM][TM], const C *A, const C *B) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TM; ++j) acc[i][j] = mk<C>(0.0, 0.0);
#pragma unroll 2
        for (int k = 0; k < d; ++k) {
            C av[TM], bv[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = A[ro[i] + k];
            if (TM > 1 && sizeof(R) == 4) {
                // Pairs of columns; rows are padded to even lengths, so the
                // second of the last pair reads padding.
#pragma unroll
                for (int j = 0; j < TM; j += 2) {
                    const float4 v = *reinterpret_cast<const float4 *>(B + k * ld + min(col(j), (d - 1) & ~1));
                    bv[j] = mk<C>(v.x, v.y);
                    bv[(j + 1) % TM] = mk<C>(v.z, v.w);
                }
            } else {
#pragma unroll
                for (int j = 0; j < TM; ++j) bv[j] = B[k * ld + co[j]];
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TM; ++j) cfma(acc[i][j], av[i], bv[j]);
        }
    };
    auto put = [&](C *dst, const C(&v)[TM][TM]) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TM; ++j)
                if (own(i, j)) dst[row(i) * ld + col(j)] = v[i][j];
    };
    // v += c_n m: c_n real for even n, imaginary for odd n.
    auto add_even = [](C &v, R c, C m) {
        v.x = fma(c, m.x, v.x);
        v.y = fma(c, m.y, v.y);
    };
    auto add_odd = [](C &v, R c, C m) {
        v.x = fma(-c, m.y, v.x);
        v.y = fma(c, m.x, v.y);
    };

    // The step's propagator into dst as E = U - I; complex64 has U in v.
    constexpr bool kHasU = sizeof(R) == 4;
    auto put_e = [&](C *dst, const C(&v)[TM][TM]) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TM; ++j)
                if (own(i, j)) {
                    C e = v[i][j];
                    if (kHasU && row(i) == col(j)) e.x -= (R)1;
                    dst[row(i) * ld + col(j)] = e;
                }
    };

    C x[TM][TM], y[TM][TM], acc[TM][TM];
    C wnext = gt < a.Ke ? step_weight(a.carr, a.w, gt, s0) : mk<C>(0.0, 0.0);
    for (long long st = s0; st < s1; ++st) {
        // Weights (the first NT of them were fetched a step ahead) and X.
        if (gt < a.Ke) {
            ws[gt] = wnext;
            if (st + 1 < s1) wnext = step_weight(a.carr, a.w, gt, st + 1);
        }
        for (int m = gt + NT; m < a.Ke; m += NT) ws[m] = step_weight(a.carr, a.w, m, st);
        group_sync(g);
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TM; ++j) x[i][j] = stack[min(row(i), d - 1) * d + co[j]];
        for (int m = 0; m < a.Ke; ++m) {
            const C w = ws[m];
            const C *h = stack + (size_t)(m + 1) * dd;
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TM; ++j) cfma(x[i][j], w, h[min(row(i), d - 1) * d + co[j]]);
        }
        put(Xs, x);
        group_sync(g);
        gemm(y, Xs, Xs);
        put(Ys, y);
        group_sync(g);
        gemm(acc, Xs, Ys);
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TM; ++j) {
                C r = mk<C>(0.0, 0.0);
                if (row(i) == col(j)) r.x = a.c[M - 3];
                add_odd(r, a.c[M - 2], x[i][j]);
                add_even(r, a.c[M - 1], y[i][j]);
                add_odd(r, a.c[M], acc[i][j]);
                if (kHasU && M == 3) {
                    add_odd(r, a.low[0], x[i][j]);
                    add_even(r, a.low[1], y[i][j]);
                }
                if (kHasU && M == 3 && row(i) == col(j)) r.x += a.j0;
                acc[i][j] = r;
            }
        // Horner; the factor alternates between two buffers, X's being free now.
        C *cur = Rs, *other = Xs;
        if (M > 3)
            put(cur, acc);
        else
            put_e(cur, acc);
        group_sync(g);
        for (int k = M - 5; k >= 0; k -= 2) {
            gemm(acc, cur, Ys);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TM; ++j) {
                    if (kHasU && k == 0) {
                        add_odd(acc[i][j], a.low[0], x[i][j]);
                        add_even(acc[i][j], a.low[1], y[i][j]);
                    }
                    add_odd(acc[i][j], a.c[k + 1], x[i][j]);
                    if (row(i) == col(j)) {
                        acc[i][j].x += a.c[k];
                        if (kHasU && k == 0) acc[i][j].x += a.j0;
                    }
                }
            if (k > 0)
                put(other, acc);
            else
                put_e(other, acc);
            C *t = cur;
            cur = other;
            other = t;
            group_sync(g);
        }
        // P <- P + E P (complex128, on P - I: E P + E + P).
        if (st == s0) {
            put(Ps, acc);
        } else {
            C pr[TM][TM];
            gemm(pr, cur, Ps);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TM; ++j)
                    if (own(i, j)) {
                        if (!kHasU) pr[i][j] = cadd(acc[i][j], pr[i][j]);
                        pr[i][j] = cadd(Ps[row(i) * ld + col(j)], pr[i][j]);
                    }
            group_sync(g);
            put(Ps, pr);
        }
    }
    group_sync(g);
    // The tree: this group's node covers chunks first .. first + 2^l - 1.
    using N = Node<R>;
    using E = typename N::T;
    E *nodes = static_cast<E *>(a.nodes);
    E *As = reinterpret_cast<E *>(Xs);  // 2 dd nodes: at most 4 d (d + 1) C
    E *Bs = As + dd;
    volatile int *flag = reinterpret_cast<volatile int *>(ws);
    for (int e = gt; e < dd; e += NT) nodes[chunk * dd + e] = N::make(Ps[(e / d) * ld + e % d], e / d == e % d);
    long long first = chunk;
    for (int l = 0; (1ll << l) < a.nchunks; ++l) {
        const bool right = (first >> l) & 1;
        const long long lo = right ? first - (1ll << l) : first, hi = lo + (1ll << l);
        if (hi >= a.nchunks) continue;  // no partner on this level
        __threadfence();
        group_sync(g);
        if (gt == 0) {
            const bool second = atomicExch(&a.arrived[hi], a.turn) == a.turn;
            if (second) a.arrived[hi] = 0;
            *flag = second;
        }
        group_sync(g);
        if (*flag == 0) return;  // the partner's group takes the pair
        __threadfence();
        for (int e = gt; e < dd; e += NT) {
            As[e] = N::left(__ldcg(&nodes[hi * dd + e]), e / d == e % d);
            Bs[e] = __ldcg(&nodes[lo * dd + e]);
        }
        group_sync(g);
        for (int e = gt; e < dd; e += NT) {
            const int r = e / d, c = e % d;
            E v = N::start(Bs[e]);
            for (int k = 0; k < d; ++k) N::mac(v, As[r * d + k], Bs[k * d + c]);
            __stcg(&nodes[lo * dd + e], N::norm(v));
        }
        first = lo;
    }
    // The root, node 0.  Each element was written by the thread that reads it.
    for (int e = gt; e < dd; e += NT) a.out[e] = N::out(__ldcg(&nodes[e]));
}

// ------------------------------------------------------------------ host side

// In complex128 a group's product with d > 4 lasts longer than that of 256 threads
// (k_small_steps), which counts while there are hardly more steps than levels of the
// tree: d = 8, order 9, 51 us against 42 for one step, 72 against 67 for eight.
bool group_applies(bool fp64, int d, int M, double x, long long P) {
    return d <= 2 * kGroupSide && M >= 3 && x <= 1.0 && !(fp64 && d > kGroupSide && P <= 8);
}

// Groups per CTA and chunks: as many groups as shared memory and 384 threads
// hold (an SM's share if there are fewer), one chunk per resident group at most.
bool group_plan(bool fp64, int d, int Ke, long long P, int num_sms, GroupPlan &q) {
    if (fp64)
        q.fn = d <= 4 ? reinterpret_cast<const void *>(&k_group_steps<double, 1>)
                      : reinterpret_cast<const void *>(&k_group_steps<double, 2>);
    else
        q.fn = d <= 4 ? reinterpret_cast<const void *>(&k_group_steps<float, 1>)
                      : reinterpret_cast<const void *>(&k_group_steps<float, 2>);
    const size_t c = fp64 ? 16 : 8;
    q.ld = (d + 3) / 2 * 2;  // even, and rows a few banks apart
    const size_t per = c * (4 * (size_t)d * q.ld + std::max(2, (Ke + 1) & ~1));
    size_t stack = c * (((1 + (size_t)Ke) * d * d + 1) / 2 * 2);
    q.stack_smem = stack <= kGroupStackBytes;
    if (!q.stack_smem) stack = 0;
    const size_t room = 220 << 10;
    if (stack + per > room) return false;
    long long groups = std::min<long long>((long long)((room - stack) / per), 384 / kGroupThreads);
    groups = std::max<long long>(1, std::min<long long>(groups, (P + num_sms - 1) / num_sms));
    q.groups = (int)groups;
    q.smem = stack + per * groups;
    int per_sm = 0;
    if (allow_smem(q.fn) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, q.fn, kGroupThreads * q.groups, q.smem) !=
            cudaSuccess ||
        per_sm < 1) {
        cudaGetLastError();
        return false;
    }
    q.nchunks = (int)std::min<long long>(P, (long long)per_sm * groups * num_sms);
    q.grid = (q.nchunks + q.groups - 1) / q.groups;
    return true;
}

template <class R>
static cudaError_t launch_group_t(const StepLaunch &l, const GroupPlan &q, double x, double hnorm, void *nodes,
                                  unsigned *arrived, unsigned turn, void *out) {
    using C = cplx_t<R>;
    GroupArgs<R> a;
    a.j0 = a.low[0] = a.low[1] = (R)0;
    if (l.fp64) {
        double c0[2];
        std::vector<double> mu;
        power_coefficients(l.M, x, hnorm, c0, mu);
        a.c[0] = (R)c0[0];
        for (int n = 1; n <= l.M; ++n) a.c[n] = (R)(n % 2 ? mu[2 * n + 1] : mu[2 * n]);
    } else {
        std::vector<double> c;
        a.j0 = (R)plain_coefficients(l.M, x, hnorm, c);
        for (int n = 0; n <= l.M; ++n) a.c[n] = (R)c[n];
        for (int n = 1; n <= 2; ++n) a.low[n - 1] = (R)low_part(c[n]);
    }
    a.stack = static_cast<const C *>(l.stack);
    a.carr = static_cast<const C *>(l.carr);
    a.nodes = nodes;
    a.arrived = arrived;
    a.turn = turn;
    a.out = static_cast<C *>(out);
    a.P = l.P;
    a.nchunks = q.nchunks;
    a.d = l.d;
    a.Ke = l.Ke;
    a.M = l.M;
    a.ld = q.ld;
    a.stack_smem = q.stack_smem;
    a.w = WeightSpec{l.w.pts, l.w.K, l.w.amps, l.w.mode, l.w.magnus, l.w.hfac};
    void *args[] = {&a};
    return cudaLaunchKernel(q.fn, dim3(q.grid), dim3(kGroupThreads * q.groups), args, q.smem, l.stream);
}

cudaError_t launch_group_steps(const StepLaunch &l, const GroupPlan &q, double x, double hnorm, void *nodes,
                               unsigned *arrived, unsigned turn, void *out) {
    return l.fp64 ? launch_group_t<double>(l, q, x, hnorm, nodes, arrived, turn, out)
                  : launch_group_t<float>(l, q, x, hnorm, nodes, arrived, turn, out);
}

}  // namespace pgb
