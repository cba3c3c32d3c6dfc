// Fixed-point complex matrices and their exact sliced products on the tcgen05
// tensor cores: the complex128 arithmetic of the kernels in fx.cu.
//
// Why: the FP64 pipe of this GPU does two fused multiply-adds per SM and clock
// (1.2 TFLOP/s in all), so a complex128 product of 64 x 64 matrices costs an SM
// half a million clocks there.  As integers cut into 8-bit digits the same
// product is 34 small bf16-rate products, about ten thousand clocks, and its
// error is smaller than that of 53-bit floating-point sums.
//
// A matrix is an item of two planes (re, im) of dp x dp 64-bit integers (dp: d
// rounded up to 64, padding zero) with an exponent e of its own:
//     value = v 2^(e - 62),  |v| <= 2^62,
// and the measured length mb of its largest |v| in bits.  An operand is
// shifted left by 62 - mb first, so a loose exponent costs no digits.  Adding
// 0x8080808080808080 turns the top seven bytes into the digits of
//     v = sum_s q_s 2^(8 (7 - s)),  q_s in [-128, 127], |q_0| <= 64,
// (rounded at the eighth byte): byte s minus 128, which fp16 holds exactly.
//
// Products of digits of level L = s + t <= 7 (34 of the 49) accumulate in their
// own FP32 accumulator of tensor memory, which never rounds: over 64 complex
// columns (128 real terms) a level is at most 128 (2 64 128 + 5 128 128) < 2^24.
// After every 64 columns the levels are read, shifted together as integers and
// added to the thread's 64-bit sums.  The dropped levels (6 digit pairs of
// level 8 and on) are below 2^-58 sqrt(d) of the product of the operands'
// maxima; with the levels up to 6 only (28 products) the error measured five
// times that of FP64 sums, with those up to 7 a third of it.
//
// Real formulation of one K stage of 16 complex columns (M = 128 rows, K = 32):
//     [C_r; C_i] = [[A_r, -A_i], [A_i, A_r]] [B_r; B_i].
// The A digits of one slice are a 128 x 32 K-major tile (64-byte swizzle), the
// B digits a 32 x 64 MN-major tile (128-byte swizzle) so that the slices of B
// stack along N (ozaki.cuh).  Two stages of 84 KB: the 512 threads cut stage
// k + 1 while the tensor core multiplies stage k.
#pragma once

#include "ozaki.cuh"

namespace pgb {
namespace fx {

constexpr int kThreads = 512;
constexpr int kSlices = 7;
constexpr int kLevels = 8;
constexpr int kStageK = 16;                                  // complex columns of a stage
constexpr int kGroup = 4;                                    // stages per exact accumulation
constexpr uint32_t kASliceB = 128 * 64;                      // 8 KB
constexpr uint32_t kBSliceB = 32 * 128;                      // 4 KB
constexpr uint32_t kStageB = kSlices * (kASliceB + kBSliceB);  // 84 KB
constexpr size_t kSmem = 2 * (size_t)kStageB + 1024;
constexpr uint32_t kWait = 1u << 24;
constexpr int kPoison = 127;  // measured length of an item that holds infinities or NaN
static_assert(kSmem <= 232448 - 4096, "shared memory of the fx kernels");

typedef long long i64;
typedef unsigned long long u64;

// e: exponent, mb: bits of the largest magnitude (kPoison: not finite).
struct Info {
    int e, mb;
};
__device__ __forceinline__ int headroom(Info i) { return i.mb >= 62 ? 0 : 62 - i.mb; }

struct Shared {
    uint64_t bar[2];
    uint32_t tmem_base;
    uint32_t orhi[2], orlo[2];  // running OR of the magnitudes of an item
    int rowmb[64];
};

// Where a thread sits: tensor-memory lane 32 (warp % 4) + lane, plane p, row r
// of the 64 x 64 tile, columns c0 .. c0 + 15.
struct Thread {
    int tid, lane, warp, p, r, c0;
    uint32_t tm;      // this thread's lane and first column in tensor memory
    unsigned char *smem;
    uint32_t ncommit[2];
    bool ok;
};

__device__ __forceinline__ uint32_t sw64(int row, int k) {
    return (uint32_t)((row >> 3) * 512 + (row & 7) * 64 + ((((k >> 3) ^ (row >> 1)) & 3) << 4) + ((k & 7) << 1));
}
// K-major operand with the 64-byte swizzle: 512 bytes between groups of eight rows.
__device__ __forceinline__ uint64_t desc_k_sw64(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}
// kind::f16 with FP16 operands, FP32 accumulators, A K-major, B MN-major, M = 128.
__host__ __device__ constexpr uint32_t idesc(int N) {
    return (1u << 4) | (1u << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// The MMAs of one stage (one thread).  The slices of B that a slice s of A
// meets (t <= 7 - s) stack along N, at most four at a time; level s + t sits at
// tensor-memory columns 64 (s + t).  `fresh` starts the levels: s = 0 starts
// levels 0 .. 6, the pair (1, 6) level 7.
__device__ __forceinline__ void issue_stage(uint32_t tmem, uint32_t sa, uint32_t sb, bool fresh) {
#pragma unroll
    for (int s = 0; s < kSlices; ++s) {
        const int nt = (kLevels - s) < kSlices ? kLevels - s : kSlices;
        for (int t0 = 0; t0 < nt;) {
            int n = nt - t0 < 4 ? nt - t0 : 4;
            uint32_t acc = (fresh && s == 0) ? 0u : 1u;
            if (fresh && s == 1 && t0 == 4) n = 2;
            if (fresh && s == 1 && t0 == 6) acc = 0u;
            const uint32_t d = tmem + 64u * (uint32_t)(s + t0), id = idesc(64 * n);
            const uint32_t a = sa + (uint32_t)s * kASliceB, b = sb + (uint32_t)t0 * kBSliceB;
            oz::mma_bf16(d, desc_k_sw64(a), oz::desc_mn_sw128(b, kBSliceB), id, acc);
            oz::mma_bf16(d, desc_k_sw64(a + 32), oz::desc_mn_sw128(b + 2048, kBSliceB), id, 1u);
            t0 += n;
        }
    }
}

// Eight 64-bit values from 32-byte aligned memory.
__device__ __forceinline__ void load8(const i64 *p, i64 (&v)[8]) {
    const longlong2 *q = reinterpret_cast<const longlong2 *>(p);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const longlong2 x = q[i];
        v[2 * i] = x.x;
        v[2 * i + 1] = x.y;
    }
}

// Digit s of eight shifted values as fp16: byte 7 - s minus 128, two at a time
// (0x6400 | byte is 1024 + byte in fp16).
template <int S>
__device__ __forceinline__ uint4 digits8(const u64 (&u)[8]) {
    constexpr uint32_t by = S < 4 ? 3 - S : 7 - S;
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t x = (uint32_t)(S < 4 ? u[2 * i] >> 32 : u[2 * i]);
        const uint32_t y = (uint32_t)(S < 4 ? u[2 * i + 1] >> 32 : u[2 * i + 1]);
        const uint32_t b = (__byte_perm(x, y, by | (4 + by) << 8) & 0x00FF00FFu) | 0x64006400u;
        asm("sub.f16x2 %0, %1, %2;" : "=r"(w[i]) : "r"(b), "r"(0x64806480u));
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// One operand of a product: element (row, col) of plane p at
// ptr + p * plane + row * ld + col, normalised by `shift` bits.
struct Operand {
    const i64 *ptr;
    i64 ld, plane;
    int shift;
};

// A thread's share of the cutting: eight columns of one row and plane, of A
// (threads 0 .. 255; the row of a lane is laid out so that the eight lanes of
// a store phase meet eight different 16-byte banks) or of B (threads 256 ..
// 511; rows k of the stage).
struct Cut {
    const i64 *src;   // stage 0
    i64 step;         // elements from one stage to the next
    int k, shift;     // B: row within the stage
    uint32_t o0, o1;  // byte offsets within a slice (A: the two copies)
    bool isA, n0, n1;  // A: the copies that are negated
};

// With `imag` the operand is i A: the product is i A B.
__device__ __forceinline__ Cut make_cut(const Thread &t, const Operand &A, const Operand &B, bool imag) {
    Cut c;
    c.isA = t.tid < 256;
    if (c.isA) {
        const int l = t.lane, w = t.warp, p = w >> 2;
        const int row = ((l >> 1) & 1) | ((l >> 2) & 2) | (l & 4) | ((l >> 1) & 8) | ((w & 3) << 4);
        const int k = 8 * (l & 1);
        c.src = A.ptr + p * A.plane + row * A.ld + k;
        c.step = kStageK;
        c.k = 0;
        c.shift = A.shift;
        // A_r: [A_r | .] of the real rows and [. | A_r] of the imaginary rows;
        // A_i: [A_i | .] of the imaginary rows and [. | -A_i] of the real rows.
        // (i A: the parts -A_i and A_r in their places.)
        const int q = imag ? 1 - p : p;
        c.o0 = sw64(q ? 64 + row : row, k);
        c.o1 = sw64(q ? row : 64 + row, kStageK + k);
        c.n0 = imag && p != 0;
        c.n1 = imag || p != 0;
    } else {
        const int w = t.warp - 8, p = w >> 2;
        c.k = ((w & 3) << 2) | (t.lane >> 3);
        const int col = 8 * (t.lane & 7);
        c.src = B.ptr + p * B.plane + c.k * B.ld + col;
        c.step = kStageK * B.ld;
        c.shift = B.shift;
        c.o0 = kSlices * kASliceB + oz::sw(kStageK * p + c.k, col);
        c.o1 = 0;
        c.n0 = c.n1 = false;
    }
    return c;
}

// Values of stage st; rows of B from kvalid on are zero.
__device__ __forceinline__ void cut_load(const Cut &c, int st, int kvalid, i64 (&v)[8]) {
    if (c.isA || st * kStageK + c.k < kvalid) {
        load8(c.src + st * c.step, v);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = 0;
    }
}

template <int S>
__device__ __forceinline__ void cut_store_slice(const Cut &c, unsigned char *stage, const u64 (&u)[8]) {
    const uint4 q = digits8<S>(u);
    if (c.isA) {
        unsigned char *b = stage + S * kASliceB;
        const uint4 m = oz::neg8(q);
        *reinterpret_cast<uint4 *>(b + c.o0) = c.n0 ? m : q;
        *reinterpret_cast<uint4 *>(b + c.o1) = c.n1 ? m : q;
    } else {
        *reinterpret_cast<uint4 *>(stage + S * kBSliceB + c.o0) = q;
    }
}

__device__ __forceinline__ void cut_store(const Cut &c, unsigned char *stage, const i64 (&v)[8]) {
    u64 u[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) u[j] = ((u64)v[j] << c.shift) + 0x8080808080808080ull;
    cut_store_slice<0>(c, stage, u);
    cut_store_slice<1>(c, stage, u);
    cut_store_slice<2>(c, stage, u);
    cut_store_slice<3>(c, stage, u);
    cut_store_slice<4>(c, stage, u);
    cut_store_slice<5>(c, stage, u);
    cut_store_slice<6>(c, stage, u);
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float (&v)[4]) {
    uint32_t r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}

// An integer of magnitude up to 2^22 held in a float, plus 0x4B400000: one add.
__device__ __forceinline__ int biased_int(float f) { return __float_as_int(__fadd_rn(f, 12582912.0f)); }

// Adds sum_L D_L 2^(8 (7 - L)) shifted right by `sh` (9 .. 32, rounded) to the
// thread's 16 sums.  Levels 0 .. 2 stay within 2^22; the others are converted.
__device__ __forceinline__ void drain(const Thread &t, int sh, i64 (&acc)[16]) {
    const int shl = 32 - sh;  // of the high part (levels 0 .. 3, units of 2^32)
    const int sl = sh - 8;    // of the low part (units of 2^8)
    const i64 half = 1ll << (sl - 1);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        float f[kLevels][4];
#pragma unroll
        for (int L = 0; L < kLevels; ++L) tmem_ld4(t.tm + 64u * L + 4u * g, f[L]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            constexpr uint32_t B = 0x4B400000u;
            const int h01 = (int)((uint32_t)biased_int(f[0][j]) * 256u + (uint32_t)biased_int(f[1][j]) - 257u * B);
            const int h23 = (int)((uint32_t)biased_int(f[2][j]) * 256u - 256u * B) + __float2int_rn(f[3][j]);
            const i64 hi = (i64)h01 * 65536 + h23;
            const int l67 = __float2int_rn(f[6][j]) + ((__float2int_rn(f[7][j]) + 128) >> 8);
            const i64 lo = (i64)__float2int_rn(f[4][j]) * 65536 + (i64)__float2int_rn(f[5][j]) * 256 + l67;
            acc[4 * g + j] += (hi << shl) + ((lo + half) >> sl);
        }
    }
}

// acc += A B 2^-sh (i A B with `imag`) over nst stages.  Every thread of the CTA calls it; returns
// false (in every thread) if a wait gave up.  Ends with all MMAs complete and
// all levels read, but no barrier.
__device__ __forceinline__ bool product(Shared &s, Thread &t, const Operand &A, const Operand &B, bool imag, int nst,
                                        int kvalid, int sh, i64 (&acc)[16]) {
    const Cut c = make_cut(t, A, B, imag);
    i64 v[8];
    cut_load(c, 0, kvalid, v);
    cut_store(c, t.smem, v);
    if (nst > 1) cut_load(c, 1, kvalid, v);
    for (int st = 0; st < nst; ++st) {
        const int b = st & 1;
        tc::fence_proxy_async();
        tc::fence_before_sync();
        const bool all = __syncthreads_and(t.ok) != 0;
        tc::fence_after_sync();
        if (!all) return false;
        if (t.tid == 0) {
            const uint32_t sa = tc::smem_addr(t.smem + b * kStageB);
            issue_stage(s.tmem_base, sa, sa + kSlices * kASliceB, (st & (kGroup - 1)) == 0);
            tc::mma_commit(&s.bar[b]);
        }
        ++t.ncommit[b];
        if (st + 1 < nst) {
            // The other buffer is free once stage st - 1 has been multiplied.
            if (st > 0) t.ok = tc::mbar_wait(&s.bar[b ^ 1], (t.ncommit[b ^ 1] - 1) & 1, kWait);
            cut_store(c, t.smem + (b ^ 1) * kStageB, v);
            if (st + 2 < nst) cut_load(c, st + 2, kvalid, v);
        }
        if ((st & (kGroup - 1)) == kGroup - 1 || st + 1 == nst) {
            t.ok = tc::mbar_wait(&s.bar[b], (t.ncommit[b] - 1) & 1, kWait) && t.ok;
            tc::fence_after_sync();
            drain(t, sh, acc);
        }
    }
    return true;
}

// ------------------------------------------------------------------ epilogue

// A real or imaginary coefficient m 2^(e - 62), 2^61 <= |m| < 2^62 (m = 0: none).
struct Coef {
    i64 m;
    int e, imag;
};
// coef * V, V an item: bufs[buf] of the kernel.
struct Term {
    Coef c;
    int buf;
};
constexpr int kTerms = 3;
// One result of a product T: T itself (plain), or t T + sum terms + diag I
// with t real (a thread holds one plane of T).
struct Out {
    int buf;  // -1: none
    int plain, nterm;
    Coef t;
    Term term[kTerms];
    Coef diag;
};
struct Op {
    int a, b;  // operands
    int imag;  // T = i A B, else A B
    Out out[2];
};

// An item as the epilogue sees it: this thread's row of the tile.
struct View {
    const i64 *re;  // plane 0; plane 1 at + plane
    i64 plane;
    Info info;
};

__device__ __forceinline__ void st4(i64 *p, i64 a, i64 b, i64 c, i64 d) {
    asm volatile("st.global.v4.b64 [%0], {%1,%2,%3,%4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
}

// Exponent of a result: two above the largest of up to four addends.
__device__ __forceinline__ int out_exponent(const Out &o, int eT, const View *views, bool &poison) {
    if (o.plain) return eT;
    int e = -1000000;
    if (o.t.m) e = eT + o.t.e;
#pragma unroll
    for (int k = 0; k < kTerms; ++k) {
        if (k >= o.nterm) break;
        const Info i = views[k].info;
        if (i.mb == kPoison) poison = true;
        e = max(e, i.e - headroom(i) + o.term[k].c.e);
    }
    if (o.diag.m) e = max(e, o.diag.e);
    return e + 2;
}

// The result's values for this thread (16 columns of its row and plane).
// r, c0: global row and first column; diagonal entries below d only.
__device__ __forceinline__ void out_values(const Out &o, const Thread &t, const i64 (&T)[16], int eT, int e,
                                           const View *views, int row, int col0, int d, i64 (&v)[16]) {
    if (o.plain) {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = T[j];
        return;
    }
    if (o.t.m) {
        const int sr = min(e - eT - o.t.e - 2, 63);
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __mul64hi(T[j], o.t.m) >> sr;
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = 0;
    }
    for (int k = 0; k < o.nterm; ++k) {
        const View &w = views[k];
        const Coef c = o.term[k].c;
        const int hr = headroom(w.info);
        const int sr = min(e - (w.info.e - hr) - c.e - 2, 63);
        const int p = c.imag ? 1 - t.p : t.p;
        const i64 m = (c.imag && t.p == 0) ? -c.m : c.m;
        const longlong2 *q = reinterpret_cast<const longlong2 *>(w.re + p * w.plane);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const longlong2 x = q[i];
            v[2 * i] += __mul64hi((i64)((u64)x.x << hr), m) >> sr;
            v[2 * i + 1] += __mul64hi((i64)((u64)x.y << hr), m) >> sr;
        }
    }
    if (o.diag.m && t.p == o.diag.imag && row < d && row >= col0 && row < col0 + 16) {
        const i64 x = o.diag.m >> min(e - o.diag.e, 63);
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (row == col0 + j) v[j] += x;
    }
}

__device__ __forceinline__ void store16(i64 *dst, const i64 (&v)[16]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) st4(dst + 4 * i, v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
}

// OR of the magnitudes (ones' complement for negative values) over the warp.
__device__ __forceinline__ u64 warp_or(const i64 (&v)[16]) {
    u64 m = 0;
#pragma unroll
    for (int j = 0; j < 16; ++j) m |= (u64)(v[j] ^ (v[j] >> 63));
    const uint32_t hi = __reduce_or_sync(0xffffffffu, (uint32_t)(m >> 32));
    const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)m);
    return (u64)hi << 32 | lo;
}

__device__ __forceinline__ int bits_of(u64 m) { return 64 - __clzll((i64)m); }

// Tensor memory, barriers and the thread's place; every thread calls these.
__device__ __forceinline__ void setup(Shared &s, Thread &t, unsigned char *raw) {
    t.tid = threadIdx.x;
    t.lane = t.tid & 31;
    t.warp = t.tid >> 5;
    const int q4 = t.warp & 3;
    t.p = q4 >> 1;
    t.r = 32 * (q4 & 1) + t.lane;
    t.c0 = 16 * (t.warp >> 2);
    t.smem = raw + ((1024u - (tc::smem_addr(raw) & 1023u)) & 1023u);
    t.ncommit[0] = t.ncommit[1] = 0;
    t.ok = true;
    if (t.warp == 0) {
        tc::tmem_alloc(&s.tmem_base, 512);
        tc::tmem_relinquish();
    }
    if (t.tid == 0) {
        tc::mbar_init(&s.bar[0], 1);
        tc::mbar_init(&s.bar[1], 1);
        tc::fence_mbar_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    t.tm = s.tmem_base + ((uint32_t)(32 * q4) << 16) + (uint32_t)t.c0;
}

__device__ __forceinline__ void teardown(Shared &s, Thread &t, int *fault) {
    const bool ok = __syncthreads_and(t.ok) != 0;
    if (!ok) {
        if (t.tid == 0 && fault) atomicAdd(fault, 1);
        // Products still in flight finish before tensor memory is freed.
        for (int b = 0; b < 2; ++b)
            if (t.ncommit[b] > 0) tc::mbar_wait(&s.bar[b], (t.ncommit[b] - 1) & 1, kWait);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (t.warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(s.tmem_base, 512);
    }
}

}  // namespace fx
}  // namespace pgb
