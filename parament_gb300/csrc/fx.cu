// Propagation on fixed-point matrices and exact sliced products on the tensor cores
// (fx.cuh): complex128 from d = kFxMinDim on (seven digits), and complex64 with d >
// 64, where the 3xTF32 kernel does not serve, in the plain form (four digits) and
// the split form (five).  Few steps of a low order stay with the FP32 and FP64 kernels
// (fx_faster).
//
// The same X_j, Chebyshev order and Bessel coefficients as the FP64 kernels
// (step_small.cu, gemm.cu; src/cuda/parament.cpp:486-718).  What changes:
//
//   * The polynomial.  For x = Hnorm h <= 1 the Chebyshev-Bessel sum is
//     evaluated by powers of X (the same polynomial, regrouped as in split.cu;
//     sum |c_n| |X|^n <= e^x, so no cancellation): Y = X^2 and, for M >= 9,
//     W = X^3, then Horner's rule in Y or W with coefficients of degree 1 or 2,
//         M   3  5  7  9  11  13  15
//         products   2  3  4  4   5   6   6    (Clenshaw: M - 1).
//     Above x = 1 the Clenshaw recurrence runs as before.  Every coefficient
//     (-i)^n times a real number is real or imaginary, so an epilogue needs one
//     64-bit multiply per value and term.
//   * E_j = U_j - I is what is formed, and the running product of a chunk of steps is
//     U <- U + E_j U: the unit diagonal never meets the small terms, and a product
//     that decays keeps its digits (held as U - I, a lossy propagator of size 1e-10
//     came out good to 1e-5 of itself).  The pairwise tree holds both U and E = U - I
//     of its nodes and multiplies by the smaller of a left operand: b + E b or U b.
//   * The plain complex64 form keeps the FP32 coefficients of the other complex64
//     kernels and rounds 1 + the diagonal of E_j to FP32, so U_j is the one those
//     form (rounded otherwise, results drift apart by 1e-8 a step).
//   * X_j = sum_m w_jm S_m is itself a product, weights (steps x 1 + Ke) times
//     the stack (1 + Ke rows of 2 dp^2 numbers), on the same sliced kernel:
//     one row of weights per step, each with an exponent of its own.
//
// d <= 64: one CTA per chunk walks its steps through all products of a step,
// the matrices in global memory (L2), no launch per product (k_fx_steps).
// d > 64: the chunks advance together, one launch per product of a round
// (k_fx_gemm over the chunks' items and their 64 x 64 tiles).
#include <math.h>
#include <stdlib.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "ctx.h"
#include "fx.cuh"
#include "kernels.h"

namespace pgb {
namespace fx {

// ------------------------------------------------------------------ set-up of the stack

// Largest biased exponent of each stack matrix (emax zeroed before).
template <class C>
__global__ void k_fx_stack_max(const C *src, i64 dd, int *emax) {
    const C *m = src + (size_t)blockIdx.y * dd;
    int e = 0;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < dd; i += (i64)gridDim.x * blockDim.x) {
        const double2 v = make_double2(m[i].x, m[i].y);
        e = max(e, max((__double2hiint(v.x) >> 20) & 0x7FF, (__double2hiint(v.y) >> 20) & 0x7FF));
    }
    e = __reduce_max_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0) atomicMax(&emax[blockIdx.y], e);
}

// Exponent e with |v| < 2^e for a largest biased exponent.
__device__ __forceinline__ int exp_of(int biased) { return max(biased, 1) - 1022; }

// Row norm of each stack matrix in units of its 2^e (rnorm zeroed before): a warp a row.
template <class C>
__global__ void k_fx_stack_norms(const C *src, int d, const int *emax, float *rnorm) {
    const C *m = src + (size_t)blockIdx.y * d * d;
    const int s = -exp_of(emax[blockIdx.y]), lane = threadIdx.x & 31;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < d; i += (gridDim.x * blockDim.x) >> 5) {
        double t = 0.0;
        for (int j = lane; j < d; j += 32) {
            const C v = m[(size_t)i * d + j];
            t += hypot(scalbn((double)v.x, s), scalbn((double)v.y, s));
        }
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) atomicMax(reinterpret_cast<int *>(&rnorm[blockIdx.y]), __float_as_int((float)t * 1.0001f));
    }
}

// The stack as fixed-point items, every matrix at its own exponent.
template <class C>
__global__ void k_fx_stack(const C *src, int d, int dp, const int *emax, i64 *dst) {
    const int m = blockIdx.y, s = 62 - exp_of(emax[m]);
    const C *a = src + (size_t)m * d * d;
    i64 *o = dst + (size_t)m * 2 * dp * dp;
    const i64 n = (i64)dp * dp;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const int r = (int)(i / dp), c = (int)(i % dp);
        const i64 k = (i64)(c >> 2) * 4 * dp + 4 * r + (c & 3);
        double2 v = make_double2(0.0, 0.0);
        if (r < d && c < d) v = make_double2(a[(size_t)r * d + c].x, a[(size_t)r * d + c].y);
        o[k] = __double2ll_rn(scalbn(v.x, s));
        o[n + k] = __double2ll_rn(scalbn(v.y, s));
    }
}

// ------------------------------------------------------------------ weights and X

// P steps in nch chunks of consecutive steps: len + 1 in the first nlong, len in
// the others, so that the chunks with a step left are always the first ones.
struct Chunks {
    i64 len;
    int nlong, nch;
    __host__ __device__ __forceinline__ i64 start(i64 c) const { return c * len + (c < nlong ? c : nlong); }
    __host__ __device__ __forceinline__ i64 steps(i64 c) const { return len + (c < nlong ? 1 : 0); }
    __host__ __device__ __forceinline__ i64 longest() const { return len + (nlong > 0 ? 1 : 0); }
};

// Row j of a batch: step i0 + j % per of chunk j / per (none: a zero row).
struct Rows {
    Chunks ch;
    int per;
    i64 i0;
    __device__ __forceinline__ i64 step(i64 j) const {
        const i64 c = j / per, i = i0 + j % per;
        return (c < ch.nch && i < ch.steps(c)) ? ch.start(c) + i : -1;
    }
};

// One warp per row: the step's weights times the stack matrices' scales, as
// integers at the row's exponent; the exponent of X_j and its length (zero
// here, kPoison for weights that are not finite).
// A: the arithmetic of the weights (complex64 samples in FP64 for the split form).
template <class A, class C>
__global__ void __launch_bounds__(128) k_fx_weights(const C *carr, WeightSpec w, int Ke, const int *emax,
                                                    const float *rnorm, Rows rows, i64 nrows, int kpad, int lgk, i64 *W, i64 plane,
                                                    Info *info, Info *zero0, Info *zero1, i64 n0, i64 n1) {
    // The infos of the round's results start at zero.
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n0 + n1; i += (i64)gridDim.x * blockDim.x)
        (i < n0 ? zero0[i] : zero1[i - n0]) = Info{0, 0, 0.0f};
    const i64 j = (i64)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (j >= nrows) return;
    const i64 st = rows.step(j);
    i64 *re = W + j * kpad, *im = re + plane;
    if (st < 0) {
        for (int m = lane; m < kpad; m += 32) re[m] = im[m] = 0;
        if (lane == 0) info[j] = Info{0, 0, 0.0f};
        return;
    }
    auto weight = [&](int m) {
        const A q = m == 0 ? mk<A>(1.0, 0.0) : step_weight_as<A>(carr, w, m - 1, st);
        const double2 v = make_double2(q.x, q.y);
        const int e = exp_of(emax[m]);
        return make_double2(scalbn(v.x, e), scalbn(v.y, e));
    };
    int be = 0;
    for (int m = lane; m <= Ke; m += 32) {
        const double2 v = weight(m);
        be = max(be, max((__double2hiint(v.x) >> 20) & 0x7FF, (__double2hiint(v.y) >> 20) & 0x7FF));
    }
    be = __reduce_max_sync(0xffffffffu, be);
    const int e = exp_of(be);
    float r = 0.0f;  // the row norm of X_j, in units of 2^e
    for (int m = lane; m < kpad; m += 32) {
        double2 v = make_double2(0.0, 0.0);
        if (m <= Ke && be < 0x7FF) v = weight(m);
        const double2 u = make_double2(scalbn(v.x, -e), scalbn(v.y, -e));
        if (m <= Ke) r += ((float)fabs(u.x) + (float)fabs(u.y)) * rnorm[m];
        re[m] = __double2ll_rn(scalbn(u.x, 62));
        im[m] = __double2ll_rn(scalbn(u.y, 62));
    }
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if (lane == 0) info[j] = Info{e + lgk, be < 0x7FF ? 0 : kPoison, 1.0001f * r * pow2f(-lgk)};
}

struct AssembleArgs {
    const i64 *W, *stack;
    i64 wplane;
    i64 *X;
    Info *info;
    i64 nrows, item;  // item: 2 dp^2
    int kpad, kvalid, lgk;
    int *fault;
};

// Products a CTA of a grid runs of `units` dealt out in turn.
__device__ __forceinline__ i64 my_units(i64 units) { return (units - blockIdx.x + gridDim.x - 1) / gridDim.x; }

// Tile (64 rows, 64 numbers of a plane) of X = W S.
struct AssembleWork {
    using At = i64;
    const AssembleArgs &a;
    Shared &s;
    Thread &t;
    i64 rt, units, plane;
    __device__ __forceinline__ At first() const { return blockIdx.x; }
    __device__ __forceinline__ At next(At u) const { return u + gridDim.x; }
    __device__ __forceinline__ bool more(At u) const { return u < units; }
    __device__ __forceinline__ bool needs(At, At) const { return false; }
    __device__ __forceinline__ int head(At) const { return a.lgk; }
    __device__ __forceinline__ bool operands(At u, Operand &A, Operand &B) const {
        A = Operand{a.W + (u % rt) * 64 * a.kpad, a.kpad, 4, a.wplane, 0};
        B = Operand{a.stack + (u / rt) * 64, a.item, 4, plane, 0};
        return false;
    }
    __device__ __forceinline__ bool epilogue(At u, i64 (&v)[kCols], uint32_t n) const {
        const i64 r0 = (u % rt) * 64, row = r0 + t.r;
        int *rowmb = s.rowmb[n & 1];
        if (row < a.nrows) {
            u64 m = 0;
#pragma unroll
            for (int j = 0; j < kCols; ++j) m |= (u64)(v[j] ^ (v[j] >> 63));
            atomicMax(&rowmb[t.r], bits_of(m));
            i64 *dst = a.X + row * a.item + t.p * plane + (u / rt) * 64 + t.c0;
#pragma unroll
            for (int i = 0; i < kCols / 4; ++i) store4(dst + 4 * i, v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
        if (!(t.ok = fsync_and(t.ok))) return false;
        if (t.tid < 64) {
            if (r0 + t.tid < a.nrows) atomicMax(&a.info[r0 + t.tid].mb, rowmb[t.tid]);
            rowmb[t.tid] = 0;
        }
        return true;
    }
};

template <int S>
__global__ void __launch_bounds__(kThreads, 1) k_fx_assemble(const __grid_constant__ AssembleArgs a) {
    extern __shared__ unsigned char raw[];
    __shared__ Shared s;
    Thread t;
    setup(s, t, raw);
    const i64 plane = a.item / 2, rt = (a.nrows + 63) / 64, units = rt * (plane / 64);
    const int nst = a.kpad / kStageK;
    const AssembleWork w{a, s, t, rt, units, plane};
    run<S>(s, t, w, my_units(units), nst, a.kvalid);
    teardown(s, t, t.ok, a.fault);
}

// ------------------------------------------------------------------ d <= 64: whole steps in one launch

enum { kBufX, kBufY, kBufW, kBufR0, kBufR1, kBufE, kBufP, kBufs };
constexpr int kMaxOps = 64;
constexpr i64 kItem64 = 2 * 64 * 64;

struct StepsArgs {
    Op op[kMaxOps];  // a step's products, and the running product (into kBufX: its target)
    int nops;        // without the running product
    const i64 *X;
    const Info *xinfo;
    i64 *scratch;  // per chunk: Y, W, R0, R1, E
    i64 *pbuf;     // 2 x nch running products
    i64 *chunks;   // nch finished products
    Info *pinfo, *cinfo;
    Chunks ch;
    i64 i0;
    int per, d, nst;
    float cap;  // sqrt(2) d
    int *fault;
};

// A CTA walks chunks blockIdx.x and blockIdx.x + gridDim.x (if there is one)
// step by step, product by product, the two in turn: a product's operands come
// from the product before the last, so it is cut and multiplied while the last
// one is finished.  With one chunk every product waits for the one before.
struct StepsWork {
    struct At {
        int i, o, k;  // step of the batch, product, chunk slot
    };
    const StepsArgs &a;
    Shared &s;
    Thread &t;
    // Every finisher writes the same exponents and lengths after a product's
    // barrier, so each finds them without another one; the cutters after
    // `finished`.
    Info (*info)[kBufs];
    int nk, steps;  // chunk slots, steps of the batch

    __device__ __forceinline__ i64 chunk(int k) const { return blockIdx.x + k * gridDim.x; }
    // Steps of the batch that slot k has (the first slot's chunk is not the shorter one).
    __device__ __forceinline__ int end(int k) const { return (int)(min(a.ch.steps(chunk(k)), a.i0 + a.per) - a.i0); }
    __device__ __forceinline__ At first() const { return At{0, 0, 0}; }
    __device__ __forceinline__ bool more(const At &q) const { return q.i < steps; }
    __device__ __forceinline__ At next(At q) const {
        do {
            if (++q.k == nk) {
                q.k = 0;
                if (++q.o == a.nops + (a.i0 + q.i > 0 ? 1 : 0)) {
                    q.o = 0;
                    ++q.i;
                }
            }
        } while (q.i < steps && q.i >= end(q.k));
        return q;
    }
    __device__ __forceinline__ bool needs(const At &q, const At &before) const { return q.k == before.k; }
    __device__ __forceinline__ i64 *item(const At &q, int b, bool out) const {
        const i64 c = chunk(q.k), i = a.i0 + q.i;
        i64 *dst = i == a.ch.steps(c) - 1 ? a.chunks + c * kItem64 : a.pbuf + ((i & 1) * a.ch.nch + c) * kItem64;
        if (b == kBufX) return out ? dst : const_cast<i64 *>(a.X) + (c * a.per + q.i) * kItem64;
        if (b == kBufP) return out ? dst : a.pbuf + (((i - 1) & 1) * a.ch.nch + c) * kItem64;
        return a.scratch + (5 * c + b - kBufY) * kItem64;
    }
    __device__ __forceinline__ Info info_of(const At &q, int b) const {
        return b == kBufX ? a.xinfo[chunk(q.k) * a.per + q.i] : info[q.k][b];
    }
    __device__ __forceinline__ int head(const At &q) const { return product_of(info_of(q, a.op[q.o].a), a.cap).head; }
    __device__ __forceinline__ bool operands(const At &q, Operand &A, Operand &B) const {
        const Op &op = a.op[q.o];
        A = Operand{item(q, op.a, false), 4, 256, 4096, headroom(info_of(q, op.a))};
        B = Operand{item(q, op.b, false), 4, 256, 4096, headroom(info_of(q, op.b))};
        return op.imag != 0;
    }
    __device__ __forceinline__ bool epilogue(const At &q, i64 (&T)[kCols], uint32_t n) const {
        const Op &op = a.op[q.o];
        const Info ia = info_of(q, op.a), ib = info_of(q, op.b);
        const Product p = product_of(ia, a.cap);
        Sum S{ia.e - headroom(ia) + ib.e - headroom(ib) + p.head, p.head - p.bits,
              row_norm(ia, a.cap) * row_norm(ib, a.cap) * pow2f(-p.head)};
        const int off = t.c0 * 64 + 4 * t.r;
        const bool bad = ia.mb == kPoison || ib.mb == kPoison;
        auto view = [&](int b) { return View{item(q, b, false) + off, info_of(q, b)}; };
        Info r0{}, r1{};
#pragma unroll 1
        for (int o = 0; o < 2; ++o) {
            const Out &out = op.out[o];
            if (absent(q, out)) continue;
            bool poison = bad;
            Info r;
            r.e = out_exponent(out, S, a.cap, view, poison, r.r);
            r.mb = poison ? kPoison : 0;
            merge_or(s, t, n, o, put_out(out, t, T, S, r.e, view, 4096, 256, t.r, t.c0, a.d,
                                         item(q, out.buf, true) + t.p * 4096 + off));
            if (!out.plain) S = Sum{r.e, 0, r.r};
            if (o == 0)
                r0 = r;
            else
                r1 = r;
        }
        if (!(t.ok = fsync_and(t.ok))) return false;
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            const u64 m = read_or(s, t, n, o);
            if (absent(q, op.out[o])) continue;
            Info r = o == 0 ? r0 : r1;
            r.mb = max(r.mb, bits_of(m));
            // The running product stands in X's place as a result.
            info[q.k][op.out[o].buf == kBufX ? kBufP : op.out[o].buf] = r;
        }
        return true;
    }
    // A step's last product gives the running product too, I + E, in the first step.
    __device__ __forceinline__ bool absent(const At &q, const Out &o) const {
        return o.buf < 0 || (o.buf == kBufP && a.i0 + q.i > 0);
    }
};

__global__ void __launch_bounds__(kThreads, 1) k_fx_steps(const __grid_constant__ StepsArgs a) {
    extern __shared__ unsigned char raw[];
    __shared__ Shared s;
    __shared__ Info info[2][kBufs];
    Thread t;
    setup(s, t, raw);
    StepsWork w{a, s, t, info, blockIdx.x + gridDim.x < a.ch.nch ? 2 : 1, 0};
    w.steps = max(0, w.end(0));
    i64 products = 0;
    for (int k = 0; k < w.nk; ++k)
        if (w.end(k) > 0) products += (i64)w.end(k) * (a.nops + 1) - (a.i0 == 0 ? 1 : 0);
    if (a.i0 > 0 && t.tid < w.nk) info[t.tid][kBufP] = a.pinfo[w.chunk(t.tid)];
    __syncthreads();
    run<7>(s, t, w, products, a.nst, 64);
    if (t.tid == 0 && t.ok)
        for (int k = 0; k < w.nk; ++k) {
            const i64 c = w.chunk(k);
            if (w.end(k) > 0) (a.i0 + w.end(k) == a.ch.steps(c) ? a.cinfo : a.pinfo)[c] = info[k][kBufP];
        }
    teardown(s, t, t.ok, a.fault);
}

// ------------------------------------------------------------------ d > 64 and the tree: one product of many items

struct Buf {
    i64 *ptr;
    i64 stride;  // numbers from one item to the next
    Info *info;
    int istride;
};
struct GemmArgs {
    Op op;
    Op alt;      // instead of op where its left operand is the smaller one
    int tree;    // with alt, and the row norms of the results measured
    Buf buf[kBufs];
    int items, nt, dp, d, nst;
    float cap;  // sqrt(2) d
    int *fault;
};

struct GemmWork {
    using At = i64;
    const GemmArgs &a;
    Shared &s;
    Thread &t;
    int tiles;
    i64 units, plane, qs;
    __device__ __forceinline__ At first() const { return blockIdx.x; }
    __device__ __forceinline__ At next(At u) const { return u + gridDim.x; }
    __device__ __forceinline__ bool more(At u) const { return u < units; }
    __device__ __forceinline__ bool needs(At, At) const { return false; }
    __device__ __forceinline__ View view(int b, i64 it, i64 off) const {
        const Buf &q = a.buf[b];
        return View{q.ptr + it * q.stride + off, q.info[it * q.istride]};
    }
    __device__ __forceinline__ const Op &op_of(i64 it) const {
        if (!a.tree) return a.op;
        const Info x = view(a.op.a, it, 0).info, y = view(a.alt.a, it, 0).info;
        return y.e - headroom(y) < x.e - headroom(x) ? a.alt : a.op;
    }
    __device__ __forceinline__ int head(At u) const {
        const i64 it = u / tiles;
        return product_of(view(op_of(it).a, it, 0).info, a.cap).head;
    }
    __device__ __forceinline__ bool operands(At u, Operand &A, Operand &B) const {
        const i64 it = u / tiles;
        const int tile = (int)(u % tiles), I = tile / a.nt, J = tile % a.nt;
        const Op &op = op_of(it);
        const View va = view(op.a, it, I * 256), vb = view(op.b, it, (i64)J * 64 * a.dp);
        A = Operand{va.re, 4, qs, plane, headroom(va.info)};
        B = Operand{vb.re, 4, qs, plane, headroom(vb.info)};
        return op.imag != 0;
    }
    __device__ __forceinline__ bool epilogue(At u, i64 (&T)[kCols], uint32_t n) const {
        const i64 it = u / tiles;
        const int tile = (int)(u % tiles), I = tile / a.nt, J = tile % a.nt;
        const Op &op = op_of(it);
        const Info ia = view(op.a, it, 0).info, ib = view(op.b, it, 0).info;
        const Product p = product_of(ia, a.cap);
        Sum S{ia.e - headroom(ia) + ib.e - headroom(ib) + p.head, p.head - p.bits,
              row_norm(ia, a.cap) * row_norm(ib, a.cap) * pow2f(-p.head)};
        const bool bad = ia.mb == kPoison || ib.mb == kPoison;
        const int row = I * 64 + t.r, col0 = J * 64 + t.c0;
        const i64 off = (i64)col0 * a.dp + 4 * row;
        auto at = [&](int b) { return view(b, it, off); };
        Info r0{}, r1{};
#pragma unroll 1
        for (int o = 0; o < 2; ++o) {
            const Out &out = op.out[o];
            if (out.buf < 0) continue;
            bool poison = bad;
            Info r;
            r.e = out_exponent(out, S, a.cap, at, poison, r.r);
            r.mb = poison ? kPoison : 0;
            const Buf &q = a.buf[out.buf];
            merge_or(s, t, n, o, put_out(out, t, T, S, r.e, at, plane, qs, row, col0, a.d,
                                         q.ptr + it * q.stride + t.p * plane + off,
                                         a.tree ? &s.rows[n & 1][o][t.r] : nullptr));
            if (!out.plain) S = Sum{r.e, 0, r.r};
            if (o == 0)
                r0 = r;
            else
                r1 = r;
        }
        if (!(t.ok = fsync_and(t.ok))) return false;
        if (a.tree && t.tid < 64) {
            // The norm: as many tiles as a row has, times the largest sum over one (bounds
            // from the operands' norms grow from level to level; what the sums then
            // leave unused cost 6e-15 at d = 32, x = 0.5).
            for (int o = 0; o < 2; ++o) {
                if (op.out[o].buf < 0) continue;
                const uint32_t r = __reduce_max_sync(0xffffffffu, s.rows[n & 1][o][t.tid]);
                s.rows[n & 1][o][t.tid] = 0;
                const Buf &q = a.buf[op.out[o].buf];
                if (t.lane == 0)
                    atomicMax(reinterpret_cast<int *>(&q.info[it * q.istride].r),
                              __float_as_int(1.001f * (float)a.nt * (float)r * pow2f(-24)));
            }
        }
        if (t.tid == 0) {
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const u64 m = read_or(s, t, n, o);
                if (op.out[o].buf < 0) continue;
                const Buf &q = a.buf[op.out[o].buf];
                const Info r = o == 0 ? r0 : r1;
                Info *i = &q.info[it * q.istride];
                if (tile == 0) {
                    i->e = r.e;
                    if (!a.tree) i->r = r.r;
                }
                atomicMax(&i->mb, max(r.mb, bits_of(m)));
            }
        }
        return true;
    }
};

template <int S>
__global__ void __launch_bounds__(kThreads, 1) k_fx_gemm(const __grid_constant__ GemmArgs a) {
    extern __shared__ unsigned char raw[];
    __shared__ Shared s;
    Thread t;
    setup(s, t, raw);
    const int tiles = a.nt * a.nt;
    const i64 units = (i64)a.items * tiles;
    const GemmWork w{a, s, t, tiles, units, (i64)a.dp * a.dp, 4ll * a.dp};
    run<S>(s, t, w, my_units(units), a.nst, a.dp);
    teardown(s, t, t.ok, a.fault);
}

// E = U - I beside the chunk products U, and the row norms of both, for the tree (the
// infos zeroed before).  A warp takes 32 rows of an item, eight warps its columns.
__global__ void __launch_bounds__(256) k_fx_less_one(const i64 *U, const Info *in, i64 *E, Info *einfo, Info *uinfo,
                                                     int d, int dp) {
    __shared__ float sums[2][8][32];
    const Info u = in[blockIdx.y];
    const int h = headroom(u), lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = blockIdx.x * 32 + lane;
    const int e = max(u.e - h, 0) + 1, left = u.e - e;  // |E| <= 1 + 2^(u.e - h)
    const i64 plane = (i64)dp * dp, one = e <= 62 ? 1ll << (62 - e) : 0;
    const i64 *src = U + 2 * plane * blockIdx.y;
    i64 *dst = E + 2 * plane * blockIdx.y;
    auto scale = [&](i64 v) {
        if (left >= 0) return (i64)((u64)v << min(left, 63));
        return left < -62 ? 0ll : (v + (1ll << (-left - 1))) >> -left;
    };
    u64 bits = 0;
    float su = 0.0f, se = 0.0f;
    for (int q = warp; q < dp / 4; q += 8) {
        const i64 at = (i64)q * 4 * dp + 4 * row;
        i64 x[4], y[4];
        load4(src + at, x[0], x[1], x[2], x[3]);
        load4(src + plane + at, y[0], y[1], y[2], y[3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            su += hypotf((float)x[j], (float)y[j]);
            x[j] = scale(x[j]) - (4 * q + j == row && row < d ? one : 0);
            y[j] = scale(y[j]);
            se += hypotf((float)x[j], (float)y[j]);
            bits |= (u64)(x[j] ^ (x[j] >> 63)) | (u64)(y[j] ^ (y[j] >> 63));
        }
        store4(dst + at, x[0], x[1], x[2], x[3]);
        store4(dst + plane + at, y[0], y[1], y[2], y[3]);
    }
    sums[0][warp][lane] = su;
    sums[1][warp][lane] = se;
    const int mb = __reduce_max_sync(0xffffffffu, bits_of(bits));
    if (lane == 0) atomicMax(&einfo[blockIdx.y].mb, u.mb == kPoison ? kPoison : mb);
    __syncthreads();
    if (warp < 2) {
        float s = 0.0f;
        for (int k = 0; k < 8; ++k) s += sums[warp][k][lane];
        Info *o = &(warp == 0 ? uinfo : einfo)[blockIdx.y];
        atomicMax(reinterpret_cast<int *>(&o->r), __float_as_int(1.001f * s * pow2f(-62)));
        if (lane == 0 && blockIdx.x == 0) o->e = warp == 0 ? u.e : e;
        if (lane == 0 && warp == 0 && blockIdx.x == 0) o->mb = u.mb;
    }
}

// An odd leftover of a level: an item and its info, E and U.
__global__ void __launch_bounds__(256) k_fx_carry(const i64 *e0, const i64 *u0, i64 *e1, i64 *u1, const Info *ei0,
                                                  const Info *ui0, Info *ei1, Info *ui1, i64 n) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *ei1 = *ei0, *ui1 = *ui0;
    for (i64 i = 4 * ((i64)blockIdx.x * blockDim.x + threadIdx.x); i < n; i += 4ll * gridDim.x * blockDim.x) {
        i64 a, b, c, d;
        load4(e0 + i, a, b, c, d);
        store4(e1 + i, a, b, c, d);
        load4(u0 + i, a, b, c, d);
        store4(u1 + i, a, b, c, d);
    }
}

// The result in the context's precision, row-major d x d.
template <class C>
__global__ void k_fx_out(const i64 *U, const Info *info, int d, int dp, C *out) {
    const Info q = *info;
    const i64 plane = (i64)dp * dp, n = (i64)d * d;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const int r = (int)(i / d), c = (int)(i % d);
        const i64 k = (i64)(c >> 2) * 4 * dp + 4 * r + (c & 3);
        double2 v = make_double2(scalbn((double)U[k], q.e - 62), scalbn((double)U[plane + k], q.e - 62));
        if (q.mb == kPoison) v.x = v.y = __longlong_as_double(0x7FF8000000000000ll);
        out[i] = mk<C>(v.x, v.y);
    }
}

// ------------------------------------------------------------------ host side

static int ceil_log2(i64 n) {
    int l = 0;
    while ((1ll << l) < n) ++l;
    return l;
}

// A real or imaginary coefficient re + i im (one of them zero).
static Coef coef(long double re, long double im) {
    const long double v = im != 0.0L ? im : re;
    if (v == 0.0L) return Coef{0, 0, 0};
    int e = 0;
    const long double f = frexpl(v, &e);
    return Coef{(i64)ldexpl(f, 62), e, im != 0.0L ? 1 : 0};
}

static Out plain_out(int buf) {
    Out o{};
    o.buf = buf;
    o.plain = 1;
    return o;
}
static Out no_out() {
    Out o{};
    o.buf = -1;
    return o;
}

// The products of a step: E from X.  Powers of X for x <= 1, the Clenshaw
// recurrence above.
static void build_program(FxForm form, int M, double x, double hnorm, std::vector<Op> &ops) {
    ops.clear();
    auto add = [](Out &o, Coef c, int buf) {
        if (c.m) o.term[o.nterm++] = Term{c, buf};
    };
    if (x <= 1.0) {
        std::vector<Coef> cs(M + 1);
        if (form == FxForm::kPlain32) {
            std::vector<double> c;
            const double j0 = plain_coefficients(M, x, hnorm, c);
            cs[0] = coef((long double)j0 - 1.0L + c[0], 0.0L);
            for (int n = 1; n <= M; ++n) cs[n] = coef(n % 2 ? 0.0L : c[n], n % 2 ? c[n] : 0.0L);
        } else {
            double c0[2];
            std::vector<double> mu;
            power_coefficients(M, x, hnorm, c0, mu);
            cs[0] = coef(c0[0], c0[1]);
            for (int n = 1; n <= M; ++n) cs[n] = coef(mu[2 * n], mu[2 * n + 1]);
        }
        auto cf = [&](int n) { return cs[n]; };
        Op y{kBufX, kBufX, 0, {plain_out(kBufY), no_out()}};
        ops.push_back(y);
        // An imaginary factor of a product goes into its operand.
        // Horner in Y: r = c_M X Y + c_(M-1) Y + c_(M-2) X + c_(M-3), then r Y + c_(k+1) X + c_k.
        auto horner = [&](int a, int b, Coef tc, int k, int deg, bool fin) {
            Op o{a, b, tc.imag, {Out{}, no_out()}};
            tc.imag = 0;
            Out &r = o.out[0];
            r.buf = fin ? kBufE : (a == kBufR0 ? kBufR1 : kBufR0);
            r.grid = fin && form == FxForm::kPlain32;
            r.t = tc;
            const int powbuf[3] = {0, kBufX, kBufY};
            for (int n = 1; n <= deg; ++n) add(r, cf(k + n), powbuf[n]);
            r.diag = cf(k);
            ops.push_back(o);
            return r.buf;
        };
        const Coef one = coef(1.0, 0.0);
        if (M < 9) {
            int r = horner(kBufX, kBufY, cf(M), M - 3, 2, M == 3);
            for (int k = M - 5; k >= 0; k -= 2) r = horner(r, kBufY, one, k, 1, k == 0);
        } else {
            // W = X Y and, beside it, the top coefficient of the rule in W:
            // degree 3 (with W itself) where 3 divides M; its c_M is imaginary,
            // so the buffer then holds i W and r W = -(i r (i W)).
            const bool three = M % 3 == 0;
            const int top = three ? M - 3 : M - M % 3;
            Op w{kBufX, kBufY, three ? 1 : 0, {plain_out(kBufW), Out{}}};
            Out &r = w.out[1];
            r.buf = kBufR0;
            if (three) {
                r.t = cf(M);
                r.t.imag = 0;
            }
            add(r, cf(top + 1), kBufX);
            if (M - top >= 2) add(r, cf(top + 2), kBufY);
            r.diag = cf(top);
            ops.push_back(w);
            int cur = kBufR0;
            Coef f = one;
            if (three) {
                f.m = -f.m;
                f.imag = 1;
            }
            for (int k = top - 3; k >= 0; k -= 3) cur = horner(cur, kBufW, f, k, 2, k == 0);
        }
        return;
    }
    // b_M = J_M, b_(M-1) = s J_M X + J_(M-1), b_k = s b_(k+1) X - b_(k+2) + J_k
    // with s = 2 / Hnorm; E = s b_1 X - 2 b_2 + J_0 - 1.  b_(M-2) comes from X X
    // directly: s^2 J_M X^2 + s J_(M-1) X + J_(M-2) - J_M.  s is a coefficient of
    // 62 bits: rounded into X it would turn every step's phase alike.
    const long double sc = 2.0L / hnorm;
    std::vector<double> J(2 * (M + 1));
    bessel_coeffs(M, x, J.data());
    // J_0 - 1 from the even orders (power_coefficients says why); where x is large (a
    // manual order may be far below it) they do not end at M + 41, and J_0 is far from 1.
    long double j0m1 = (long double)jn(0, x) - 1.0L;
    if (x <= 8.0) {
        j0m1 = 0.0L;
        for (int k = M + 41; k >= 2; k -= 2) j0m1 -= 2.0L * jn(k, x);
    }
    auto j = [&](int k, long double f) { return coef(f * J[2 * k], f * J[2 * k + 1]); };
    int prev = -1, cur = -1, n = 0;  // buffers of b_(k+2) and b_(k+1); -1: from X
    const int rot[3] = {kBufY, kBufW, kBufR0};
    for (int k = M - 2; k >= 0; --k) {
        Op o{cur < 0 ? kBufX : cur, kBufX, 0, {Out{}, no_out()}};
        Out &r = o.out[0];
        const double beta = k == 0 ? -2.0 : -1.0;
        long double dr = k == 0 ? j0m1 : J[2 * k], di = J[2 * k + 1];
        if (cur < 0) {  // k = M - 2
            r.t = j(M, sc * sc);
            o.imag = r.t.imag;
            r.t.imag = 0;
            add(r, j(M - 1, sc), kBufX);
            dr += beta * J[2 * M];
            di += beta * J[2 * M + 1];
        } else {
            r.t = coef(sc, 0.0L);
            if (prev < 0) {  // k = M - 3: b_(M-1) = s J_M X + J_(M-1)
                add(r, j(M, sc * beta), kBufX);
                dr += beta * J[2 * (M - 1)];
                di += beta * J[2 * (M - 1) + 1];
            } else {
                add(r, coef(beta, 0.0), prev);
            }
        }
        r.diag = coef(dr, di);
        r.buf = k == 0 ? kBufE : rot[n++ % 3];
        prev = cur;
        cur = r.buf;
        ops.push_back(o);
    }
}

static bool disabled() {
    static const bool off = [] {
        const char *v = getenv("PARAMENT_DISABLE_TENSOR_CORES");
        return v && v[0] && v[0] != '0';
    }();
    return off;
}

template <int S>
static cudaError_t set_smem() {
    cudaError_t e = cudaSuccess;
    for (const void *fn : {reinterpret_cast<const void *>(&k_fx_assemble<S>),
                           reinterpret_cast<const void *>(&k_fx_gemm<S>),
                           S == 7 ? reinterpret_cast<const void *>(&k_fx_steps) : nullptr})
        if (e == cudaSuccess && fn)
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Digits<S>::smem);
    return e;
}

// The workspace of a propagation, carved from one allocation.
struct Plan {
    int d, dp, nt, kpad, kvalid, nch, per;
    Chunks ch;
    i64 item, rows;
    size_t off_w, off_x, off_s, off_p, off_c, off_t, off_info, bytes;
    size_t n_info;
};

static Plan make_plan(int d, int Ke, i64 P, int num_sms) {
    Plan q{};
    q.d = d;
    q.dp = (d + 63) / 64 * 64;
    q.nt = q.dp / 64;
    q.item = 2ll * q.dp * q.dp;
    q.kvalid = 1 + Ke;
    q.kpad = (q.kvalid + kStageK - 1) / kStageK * kStageK;
    const int tiles = q.nt * q.nt;
    if (tiles == 1) {
        // Two chunks per SM; X of up to 16 steps of every chunk at a time (320 MB).
        q.nch = (int)std::min<i64>(2ll * num_sms, P);
        q.per = (int)std::min<i64>(16, (P + q.nch - 1) / q.nch);
    } else {
        // About sixteen waves of tiles per product, in rounds of equal size (eight: 5 to
        // 10 % slower at d = 128 and 200, two: a quarter).
        const i64 g0 = std::min<i64>(P, std::max<i64>(1, (16ll * num_sms + tiles - 1) / tiles));
        const i64 L = (P + g0 - 1) / g0;
        q.nch = (int)((P + L - 1) / L);
        q.per = 1;
    }
    q.ch = Chunks{P / q.nch, (int)(P % q.nch), q.nch};
    q.rows = (i64)q.nch * q.per;
    const i64 rpad = (q.rows + 63) / 64 * 64;
    size_t o = 0;
    auto take = [&](size_t n) {
        const size_t at = o;
        o += (n + 255) / 256 * 256;
        return at;
    };
    const size_t m = sizeof(i64) * (size_t)q.item;
    q.off_w = take(sizeof(i64) * 2 * (size_t)rpad * q.kpad);
    q.off_x = take(m * (size_t)q.rows);
    q.off_s = take(m * 5 * (size_t)q.nch);
    q.off_p = take(m * 2 * (size_t)q.nch);
    q.off_c = take(m * (size_t)q.nch);
    // X rows; the results of a step's products (then the tree's); P0 P1; finished chunks.
    q.n_info = (size_t)q.rows + (kMaxOps + 4) * (size_t)q.nch;
    q.off_info = take(sizeof(Info) * q.n_info);
    q.bytes = o;
    return q;
}

// Bytes before the matrices of the fixed-point stack: the largest exponents and the row
// norms.
static size_t stack_head(int n) { return ((sizeof(int) + sizeof(float)) * (size_t)n + 255) / 256 * 256; }

template <int S>
static cudaError_t launch_gemm_op(const GemmArgs &a, int num_sms, cudaStream_t st, int *launches) {
    const i64 units = (i64)a.items * a.nt * a.nt;
    k_fx_gemm<S><<<(int)std::min<i64>(units, num_sms), kThreads, Digits<S>::smem, st>>>(a);
    ++*launches;
    return cudaGetLastError();
}

}  // namespace fx

using namespace fx;

// Whether these kernels are the faster ones for P steps of order M.  A product takes
// them about as long at any d up to 64 and has a latency of some 20 us; the other
// kernels' products are short at small d and take turns with fewer launches.  Measured
// against those, times here over times there:
//   complex64, plain   d = 96 M = 3  1.96 (16 steps) 1.31 (2048)   M = 7  1.62, 0.81
//                      d = 128       1.61, 0.95                           1.15, 0.60
//                      d = 200       1.13, 0.87                           0.74, 0.59
//                      d = 500       0.62 (1 step: 1.26)                  0.45 (0.71)
//   The line: the FP32 kernels' time per step goes as tiles d M, that of these as the
//   tiles; of 780 pairs from d = 65 to 500 and orders 3 to 9 it leaves 5 per cent at most
//   where they are the slower ones and 1 per cent of the time on the whole.
//   split form         d = 65 M = 7  1.66 (1 step) 1.12 (8) 0.90 (16)
//                      d = 128       1.63, 0.75, 0.50;  d = 300: 1.61, 0.57 (2 steps)
//   complex128         d = 17 M = 5  1.15 (16 steps) 1.25 (152) 0.97 (200) 0.62 (3000)
//                      d = 22        1.01, 1.17, 0.87, 0.50;  d = 32: 0.84, 0.99, 0.71, 0.35
//   (one step per SM at most is one product after the other in either kernel).
static bool fx_faster(FxForm form, int d, int M, long long P, int num_sms) {
    const long long nt = (d + 63) / 64, tiles = nt * nt;
    if (form == FxForm::kFp64) return P > num_sms || M > 7 || d > (M > 3 ? 20 : kFxSimtDim);
    if (form == FxForm::kSplit32) return P >= 2 && P * d * d >= 80000;
    return P * tiles * ((long long)d * M - 420) >= 155000;
}

bool fx_applies(const Ctx *c, FxForm form, int M, double x, long long P) {
    if (M < 3 || !isfinite(c->hnorm) || c->hnorm <= 0.0) return false;
    if (form != FxForm::kFp64 && x > 1.0) return false;
    return (form == FxForm::kSplit32 ? c->fx_split_ready : c->fx_ready) &&
           fx_faster(form, (int)c->dim, M, P, c->num_sms);
}

// Whether a context's Hamiltonian gets a fixed-point stack: complex64 from 65 on
// (below, the step kernels of one launch are faster: a product's epilogue takes
// longer here than its digits), and the plain form not where the 3xTF32 kernel runs: d
// = 512, 64 steps of order 7 take 2.45 ms there and 5.96 here, d = 256 0.62 and 1.01.
static bool fx_serves(FxForm form, int d) {
    if (disabled()) return false;
    if (form == FxForm::kFp64) return d >= kFxMinDim;
    return d > 64 && (form == FxForm::kSplit32 || d < 256 || d % 128 != 0);
}

static size_t fixed_bytes(unsigned dim, unsigned Ke) {
    const size_t dp = (dim + 63) / 64 * 64, n = 1 + (size_t)Ke;
    return stack_head((int)n) + sizeof(i64) * 2 * dp * dp * n;
}

// A stack in fixed point at dst, on the context's stream (the caller waits for it).
// More than 65535 matrices do not fit the launch grid and fail here: the other kernels
// then serve, and drain's shift (6 and the bits of twice as many) stays below 24.
template <class C>
static bool convert_stack(Ctx *c, const void *stack, void *dst) {
    const int d = (int)c->dim, dp = (d + 63) / 64 * 64, n = 1 + (int)c->Ke;
    int *emax = static_cast<int *>(dst);
    const C *src = static_cast<const C *>(stack);
    float *rnorm = reinterpret_cast<float *>(emax + n);
    if (cudaMemsetAsync(emax, 0, (sizeof(int) + sizeof(float)) * n, c->stream) != cudaSuccess) return false;
    k_fx_stack_max<C><<<dim3(std::max(1, std::min(256, d * d / 1024)), n), 256, 0, c->stream>>>(src, (i64)d * d, emax);
    k_fx_stack_norms<C><<<dim3(std::min(256, (d + 7) / 8), n), 256, 0, c->stream>>>(src, d, emax, rnorm);
    k_fx_stack<C><<<dim3(std::max(1, std::min(1024, dp * dp / 512)), n), 256, 0, c->stream>>>(
        src, d, dp, emax, reinterpret_cast<i64 *>(static_cast<char *>(dst) + stack_head(n)));
    return cudaGetLastError() == cudaSuccess;
}

size_t fx_stack_bytes(const Ctx *c, unsigned dim, unsigned Ke) {
    return fx_serves(c->fp64 ? FxForm::kFp64 : FxForm::kPlain32, (int)dim) ? fixed_bytes(dim, Ke) : 0;
}

// The plain form's stack, at c->fx_stack (null: the other kernels serve).
void fx_prepare(Ctx *c) {
    c->fx_ready = false;
    if (!c->fx_stack) return;
    c->fx_ready = c->fp64 ? convert_stack<double2>(c, c->stack.ptr, c->fx_stack)
                          : convert_stack<float2>(c, c->stack.ptr, c->fx_stack);
}

void fx_prepare_split(Ctx *c) {
    c->fx_split_ready = false;
    if (!fx_serves(FxForm::kSplit32, (int)c->dim)) return;
    // A set-up allocation, not counted by the allocation-failure injection.
    const size_t bytes = fixed_bytes(c->dim, c->Ke);
    c->fx_split.release();
    void *p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    c->fx_split.ptr = p;
    c->fx_split.cap = bytes;
    c->fx_split_ready = convert_stack<float2>(c, c->split_stack.ptr, p);
}

bool fx_ensure(Ctx *c, long long P, cudaStream_t stream) {
    const Plan q = make_plan((int)c->dim, (int)c->Ke, P, c->num_sms);
    if (c->fx_ws.cap < q.bytes && capturing(stream)) return false;
    return c->fx_ws.ensure(q.bytes) == cudaSuccess;
}

template <int S, class A, class C>
static cudaError_t run_fx_t(Ctx *c, FxForm form, const void *d_carr, const WeightSpecHost &wh, double x, int M,
                            long long P, void *d_out, cudaStream_t st) {
    const void *sb = form == FxForm::kSplit32 ? c->fx_split.ptr : c->fx_stack;
    const int d = (int)c->dim, Ke = (int)c->Ke, n = 1 + Ke;
    const Plan q = make_plan(d, Ke, P, c->num_sms);
    int launches = 0;
    cudaError_t e = set_smem<S>();
    if (e != cudaSuccess) return e;
    const size_t head = stack_head(n);
    const int *emax = static_cast<const int *>(sb);
    const float *rnorm = reinterpret_cast<const float *>(emax + n);
    const i64 *stack = reinterpret_cast<const i64 *>(static_cast<const char *>(sb) + head);
    char *ws = static_cast<char *>(c->fx_ws.ptr);
    i64 *W = reinterpret_cast<i64 *>(ws + q.off_w), *X = reinterpret_cast<i64 *>(ws + q.off_x);
    i64 *scr = reinterpret_cast<i64 *>(ws + q.off_s), *Pb = reinterpret_cast<i64 *>(ws + q.off_p);
    i64 *chunks = reinterpret_cast<i64 *>(ws + q.off_c);
    Info *xinfo = reinterpret_cast<Info *>(ws + q.off_info), *sinfo = xinfo + q.rows;
    Info *pinfo = sinfo + (kMaxOps + 1) * (size_t)q.nch, *cinfo = pinfo + 2 * (size_t)q.nch;
    std::vector<Op> ops;
    build_program(form, M, x, c->held_norm(), ops);
    if ((int)ops.size() >= kMaxOps) return cudaErrorInvalidValue;  // orders up to 63: 62 products
    const WeightSpec w{wh.pts, wh.K, wh.amps, wh.mode, wh.magnus, wh.hfac};
    const i64 rpad = (q.rows + 63) / 64 * 64;
    const int lgw = std::max(5, ceil_log2(2ll * q.kvalid));
    const float cap = 1.41422f * (float)d;
    const int nst = (d + kStageK - 1) / kStageK;
    auto assemble = [&](i64 i0, i64 rows, int per, Info *zero0 = nullptr, i64 n0 = 0, Info *zero1 = nullptr,
                        i64 n1 = 0) -> cudaError_t {
        const Rows r{q.ch, per, i0};
        k_fx_weights<A><<<(unsigned)((rows + 3) / 4), 128, 0, st>>>(static_cast<const C *>(d_carr), w, Ke, emax,
                                                                  rnorm, r, rows, q.kpad, lgw, W, rpad * q.kpad, xinfo, zero0,
                                                                  zero1, n0, n1);
        const AssembleArgs a{W, stack, rpad * q.kpad, X, xinfo, rows, q.item, q.kpad, q.kvalid, lgw, c->d_fault};
        const i64 units = ((rows + 63) / 64) * (q.item / 128);
        k_fx_assemble<S><<<(int)std::min<i64>(units, c->num_sms), kThreads, Digits<S>::smem, st>>>(a);
        launches += 2;
        return cudaGetLastError();
    };
    if (c->timing) cudaEventRecord(c->ev_start, st);
    // The running product of a chunk, U <- U + E U, into kBufX of its caller; in the
    // first step I + E, a second result of the step's last product.
    const Coef one = coef(1.0, 0.0), minus = coef(-1.0, 0.0);
    Op run{kBufE, kBufP, 0, {Out{}, no_out()}};
    run.out[0].buf = kBufX;
    run.out[0].t = one;
    run.out[0].nterm = 1;
    run.out[0].term[0] = Term{one, kBufP};
    Out first{};
    first.buf = kBufP;
    first.t = one;
    first.diag = one;
    ops.back().out[1] = first;
    if (q.nt == 1) {
        StepsArgs a;
        for (size_t k = 0; k < ops.size(); ++k) a.op[k] = ops[k];
        a.op[ops.size()] = run;
        a.nops = (int)ops.size();
        a.X = X;
        a.xinfo = xinfo;
        a.scratch = scr;
        a.pbuf = Pb;
        a.chunks = chunks;
        a.pinfo = pinfo;
        a.cinfo = cinfo;
        a.ch = q.ch;
        a.per = q.per;
        a.d = d;
        a.nst = nst;
        a.cap = cap;
        a.fault = c->d_fault;
        for (i64 i0 = 0; i0 < q.ch.longest(); i0 += q.per) {
            if ((e = assemble(i0, q.rows, q.per)) != cudaSuccess) return e;
            a.i0 = i0;
            k_fx_steps<<<std::min(q.nch, c->num_sms), kThreads, Digits<7>::smem, st>>>(a);
            ++launches;
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
    } else {
        const i64 longest = q.ch.longest(), mat = q.item, set = mat * q.nch;
        GemmArgs a{};
        a.nt = q.nt;
        a.dp = q.dp;
        a.d = d;
        a.nst = nst;
        a.cap = cap;
        a.fault = c->d_fault;
        for (i64 i = 0; i < longest; ++i) {
            const int active = i < q.ch.len ? q.nch : q.ch.nlong;
            for (int b = 0; b < kBufs; ++b) a.buf[b] = Buf{};
            a.buf[kBufX] = Buf{X, mat, xinfo, 1};
            for (int b = 0; b < 5; ++b) a.buf[kBufY + b] = Buf{scr + b * set, mat, nullptr, 1};
            Buf dst{Pb + (i & 1) * set, mat, pinfo + (i & 1) * q.nch, 1};
            a.buf[kBufP] = Buf{Pb + ((i - 1) & 1) * set, mat, pinfo + ((i - 1) & 1) * q.nch, 1};
            // A buffer may be written more than once in a round: the lengths, which
            // start at zero, are kept per result.
            const size_t results = ops.size() + 1;
            if ((e = assemble(i, active, 1, sinfo, (i64)results * q.nch, dst.info, q.nch)) != cudaSuccess) return e;
            size_t slot = 0;
            if (i == 0) a.buf[kBufP] = dst;
            a.items = active;
            for (const Op &o : ops) {
                a.op = o;
                if (i > 0 && o.out[1].buf == kBufP) a.op.out[1] = no_out();
                for (const Out &out : a.op.out)
                    if (out.buf >= 0 && out.buf != kBufP) a.buf[out.buf].info = sinfo + slot++ * q.nch;
                if ((e = launch_gemm_op<S>(a, c->num_sms, st, &launches)) != cudaSuccess) return e;
            }
            if (i > 0) {
                a.buf[kBufX] = dst;
                a.op = run;
                if ((e = launch_gemm_op<S>(a, c->num_sms, st, &launches)) != cudaSuccess) return e;
            }
            if (active < q.nch) {
                // The chunks without a step in this round keep their product.
                const Buf &prev = a.buf[kBufP];
                const size_t rest = (size_t)(q.nch - active);
                e = cudaMemcpyAsync(dst.ptr + active * mat, prev.ptr + active * mat, sizeof(i64) * mat * rest,
                                    cudaMemcpyDeviceToDevice, st);
                if (e == cudaSuccess)
                    e = cudaMemcpyAsync(dst.info + active, prev.info + active, sizeof(Info) * rest,
                                        cudaMemcpyDeviceToDevice, st);
                if (e != cudaSuccess) return e;
            }
        }
        chunks = Pb + ((longest - 1) & 1) * set;
        cinfo = pinfo + ((longest - 1) & 1) * q.nch;
    }
    if (c->timing) cudaEventRecord(c->ev_stop, st);
    // Pairwise tree over the chunk products, later chunks on the left: U_a U_b as U_b + E_a
    // U_b with E = U - I, or as U_a U_b where U_a is the smaller one (a dense unitary, or a
    // propagator that decays), both U and E for the next level.  The digits of an
    // operand are cut at a fixed distance below its largest entry: in U alone, 64 steps of
    // x = 0.05 at d = 64 were off by 1.5e-15 (FP64 2.7e-16), in E alone a propagator of
    // size 1e-10 by 1e-7 of itself.
    const i64 *res = chunks;
    const Info *rinfo = cinfo;
    if (q.nch > 1) {
        GemmArgs a{};
        a.nt = q.nt;
        a.dp = q.dp;
        a.d = d;
        a.nst = nst;
        a.cap = cap;
        a.fault = c->d_fault;
        // Left: X as E, W as U; right: Y as U, R0 as E.  Results: U to R1, E to E.
        auto result = [&](int buf, const Coef &dg, int term) {
            Out o{};
            o.buf = buf;
            o.t = one;
            o.diag = dg;
            if (term >= 0) o.term[o.nterm++] = Term{one, term};
            return o;
        };
        const Coef none{0, 0, 0};
        const size_t set = (size_t)q.item * q.nch;
        i64 *E[2] = {scr, scr + set}, *U[2] = {chunks, scr + 2 * set};
        // Infos of E and U of each level, behind each other, zeroed at once.
        size_t all = 0;
        for (i64 n2 = q.nch; n2 > 1; n2 = (n2 + 1) / 2) all += (size_t)n2;
        Info *ei = sinfo, *ui = ei + q.nch;
        if ((e = cudaMemsetAsync(sinfo, 0, sizeof(Info) * 2 * (all + 1), st)) != cudaSuccess) return e;
        k_fx_less_one<<<dim3(q.dp / 32, q.nch), 256, 0, st>>>(chunks, cinfo, E[0], ei, ui, d, q.dp);
        ++launches;
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        int k = 0;
        for (i64 n2 = q.nch; n2 > 1; k ^= 1) {
            const i64 pairs = n2 / 2;
            const bool last = n2 == 2;
            Info *en = ui + n2, *un = en + (n2 + 1) / 2;
            a.buf[kBufX] = Buf{E[k] + q.item, 2 * q.item, ei + 1, 2};
            a.buf[kBufR0] = Buf{E[k], 2 * q.item, ei, 2};
            a.buf[kBufW] = Buf{U[k] + q.item, 2 * q.item, ui + 1, 2};
            a.buf[kBufY] = Buf{U[k], 2 * q.item, ui, 2};
            a.buf[kBufR1] = Buf{U[k ^ 1], q.item, un, 1};
            a.buf[kBufE] = Buf{E[k ^ 1], q.item, en, 1};
            a.items = (int)pairs;
            a.tree = 1;
            if (last) {
                a.op = Op{kBufX, kBufY, 0, {result(kBufR1, none, kBufY), no_out()}};
                a.alt = Op{kBufW, kBufY, 0, {result(kBufR1, none, -1), no_out()}};
            } else {
                a.op = Op{kBufX, kBufY, 0, {result(kBufE, none, kBufR0), result(kBufR1, one, -1)}};
                a.alt = Op{kBufW, kBufY, 0, {result(kBufR1, none, -1), result(kBufE, minus, -1)}};
            }
            if ((e = launch_gemm_op<S>(a, c->num_sms, st, &launches)) != cudaSuccess) return e;
            if (n2 & 1) {
                const i64 o = n2 - 1;
                k_fx_carry<<<(int)std::min<i64>(512, (q.item + 1023) / 1024), 256, 0, st>>>(
                    E[k] + o * q.item, U[k] + o * q.item, E[k ^ 1] + pairs * q.item, U[k ^ 1] + pairs * q.item,
                    ei + o, ui + o, en + pairs, un + pairs, q.item);
                ++launches;
                if ((e = cudaGetLastError()) != cudaSuccess) return e;
            }
            n2 = pairs + (n2 & 1);
            ei = en;
            ui = un;
        }
        res = U[k];
        rinfo = ui;
    }
    const i64 total = (i64)d * d;
    k_fx_out<<<(int)std::min<i64>((total + 255) / 256, 1024), 256, 0, st>>>(res, rinfo, d, q.dp,
                                                                           static_cast<C *>(d_out));
    ++launches;
    c->launches = launches;
    return cudaGetLastError();
}

cudaError_t run_fx(Ctx *c, FxForm form, const void *d_carr, const WeightSpecHost &wh, double x, int M, long long P,
                   void *d_out, cudaStream_t st) {
    c->fx_ran = true;
    if (form == FxForm::kFp64) return run_fx_t<7, double2, double2>(c, form, d_carr, wh, x, M, P, d_out, st);
    if (form == FxForm::kPlain32) return run_fx_t<4, float2, float2>(c, form, d_carr, wh, x, M, P, d_out, st);
    return run_fx_t<5, double2, float2>(c, form, d_carr, wh, x, M, P, d_out, st);
}

}  // namespace pgb
