// Fixed-point complex matrices and their exact sliced products on the tcgen05
// tensor cores: the complex128 arithmetic of the kernels in fx.cu.
//
// Why: the FP64 pipe of this GPU does two fused multiply-adds per SM and clock
// (1.2 TFLOP/s in all), so a complex128 product of 64 x 64 matrices costs an SM
// half a million clocks there.  As integers cut into 8-bit digits the same
// product is 34 small bf16-rate products, about ten thousand clocks.
//
// A matrix is an item of two planes (re, im) of dp x dp 64-bit integers (dp: d
// rounded up to 64, padding zero) with an exponent e of its own:
//     value = v 2^(e - 62),  |v| <= 2^62,
// and the measured length mb of its largest |v| in bits.  An operand is
// shifted left by 62 - mb first, so a loose exponent costs no digits; what the sums'
// headroom costs is kept small by measured row norms (product_of).  Adding
// 0x8080808080808080 turns the top seven bytes into the digits of
//     v = sum_s q_s 2^(8 (7 - s)),  q_s in [-128, 127], |q_0| <= 64,
// (rounded at the eighth byte): byte s minus 128, which fp16 holds exactly.
// Four columns of a row are one 32-byte piece and the pieces of a column group
// follow each other row by row: the epilogue's lanes (one row each) and the
// lanes that cut operands (8 columns of a row each) both move whole lines
// (row-major items cost 32 passes of the load pipe per access).
//
// Products of digits of level L = s + t <= 7 (34 of the 49) accumulate in their
// own FP32 accumulator of tensor memory, which never rounds: over 64 complex
// columns (128 real terms) a level is at most 128 (2 64 128 + 5 128 128) < 2^24.
// After every 64 columns the levels are read, shifted together as integers and
// added to the thread's 64-bit sums.  The dropped levels (6 digit pairs of
// level 8 and on) are below 2^-58 sqrt(d) of the product of the operands'
// maxima; with the levels up to 6 only (28 products) the error measured 15 times
// as large.  Against 113-bit propagators whole calls are 0.2 to 1.5 times as far off
// as the FP64 kernels, 2.1 times in the worst case met (d = 64, 24 steps, x = 0.5,
// dense); a headroom of log2(2 d) bits for every sum instead took nearly diagonal
// Hamiltonians and large steps to 3 to 13 times.  All of this is of the maxima: an
// entry far below its matrix's largest loses relative accuracy that FP64 would keep
// (blocks coupled by 1e-8, d = 32: their amplitudes to 3e-9; exact zeros stay zero).
//
// Real formulation of one K stage of 16 complex columns (M = 128 rows, K = 32):
//     [C_r; C_i] = [[A_r, -A_i], [A_i, A_r]] [B_r; B_i].
// The A digits of one slice are a 128 x 32 K-major tile (64-byte swizzle), the
// B digits a 32 x 64 MN-major tile (128-byte swizzle) so that the slices of B
// stack along N (ozaki.cuh).
//
// Three kinds of warps walk the products of a launch, each at its own pace: eight
// cut operands into stages, one issues the digit products, eight read the levels
// and run the epilogues.  They meet on mbarriers only: `full` (a stage is cut),
// `done` (a stage is multiplied), `ready` (a group of stages is), `drained` (its
// levels are read), `finished` (a product is stored: two in turn, fx_turns.h).
//
// What bounds it: inside a long K with seven digits, 64 columns take 13 thousand
// clocks, 8 of them on the tensor core and 5 reading the levels, during which it
// stands still (its 512 columns hold one product's levels); cutting (4.5) and the
// operands' loads (6) lie underneath.  At d <= 128 the loads' latency and the
// epilogues (64-bit multiplies) weigh as much; with four or five digits they are
// all of it.  Measured: d = 64 Magnus, 4096 steps, 2.07 ms; d = 96, 512 steps, 1.70
// ms; d = 512, 16 steps, 3.24 ms a call; complex64, d = 128, 4096 steps, 8.05
// ms (FP32 kernel: 11.2).  With the finishers' sums spilled (136 registers) the
// first three took 2.36, 1.71 and 3.07; with eight warps that did all but the
// issuing 2.57, 1.80 and 3.13.  Accumulators for each half of the columns, one
// read while the other is filled, measured slower (2.84, 2.37, 4.49: the 32-column
// B tiles).
#pragma once

#include "fx_turns.h"
#include "ozaki.cuh"

namespace pgb {
namespace fx {

constexpr int kFinishers = 256, kCutters = 256;  // threads; warps 0 .. 7 and 8 .. 15
constexpr int kThreads = kFinishers + kCutters + 128;  // and a warpgroup of which one thread issues
constexpr int kIssuer = kFinishers + kCutters;
constexpr int kCols = 32;  // columns of a finisher
// Registers: 96 a thread at launch (61,440 in all), then by warpgroup.  The
// finishers must not spill: with this little L1 a spilled sum comes back from L2.
constexpr int kRegsFinish = 144, kRegsCut = 80, kRegsIssue = 24;
static_assert(kFinishers * kRegsFinish + kCutters * kRegsCut + 128 * kRegsIssue <= kThreads * 96, "register split");
constexpr int kStageK = 16;                       // complex columns of a stage
constexpr int kGroup = 4;                         // stages per exact accumulation
constexpr uint32_t kASliceB = 128 * 64;           // 8 KB
constexpr uint32_t kBSliceB = 32 * 128;           // 4 KB
constexpr int kMaxStages = 4;
// S digits per operand: 7 for complex128, 4 for the complex64 form, 5 for its split
// form.  The levels kept, the stages that fit and the accumulators: two sets where
// they fit into tensor memory, one read while the other is filled.
template <int S>
struct Digits {
    static constexpr int levels = S == 7 ? 8 : S;
    static constexpr uint32_t stage_bytes = S * (kASliceB + kBSliceB);  // 84, 48, 60 KB
    static constexpr int stages = S == 7 ? 2 : S == 5 ? 3 : 4;
    static constexpr int sets = levels <= 4 ? 2 : 1;
    static constexpr size_t smem = stages * (size_t)stage_bytes + 1024;
    static_assert(smem <= 232448 - 4096 && stages <= kMaxStages, "shared memory of the fx kernels");
};
constexpr uint32_t kWait = 1u << 24;
constexpr int kPoison = 127;  // measured length of an item that holds infinities or NaN

typedef long long i64;
typedef unsigned long long u64;

// e: exponent, mb: bits of the largest magnitude (kPoison: not finite), r: a bound of
// the row norms, max_i sum_k |a_ik|, in units of 2^e.
struct Info {
    int e, mb;
    float r;
};
__device__ __forceinline__ int headroom(Info i) { return i.mb >= 62 ? 0 : 62 - i.mb; }
// 2^k, within FP32.
__device__ __forceinline__ float pow2f(int k) { return __int_as_float((127 + min(max(k, -126), 127)) << 23); }
// The row norm of a normalised operand, sqrt(2) d (`cap`) at most.
__device__ __forceinline__ float row_norm(Info i, float cap) { return fminf(i.r * pow2f(headroom(i)), cap); }
__device__ __forceinline__ int ceil_log2f(float q) {
    const int b = __float_as_int(q);
    return ((b >> 23) & 255) - 127 + ((b & 0x7FFFFF) != 0);
}

// A product of two normalised items: its values stay below 2^bits in units of the
// operands' 2^(e - headroom), its sums are held with `head` bits above those units
// (drain wants five at least).  The bound is the left operand's row norm: with 2 d terms
// of the largest size instead, as for any two matrices, the sums of a nearly diagonal
// propagator would leave up to ten bits unused, and its products were 13 times (d = 96)
// as far off as those in FP64.
struct Product {
    int bits, head;
};
__device__ __forceinline__ Product product_of(Info a, float cap) {
    const int b = ceil_log2f(1.4143f * row_norm(a, cap));
    return Product{max(b, 0), max(b, 5)};
}

struct Shared {
    uint64_t full[kMaxStages], done[kMaxStages], ready[2], drained[2], finished[kFinishedBars], last;
    uint32_t tmem_base;
    uint32_t orhi[4][2], orlo[4][2];  // OR of the magnitudes of a product's results, four products in turn
    int rowmb[2][64];                 // lengths of a tile's rows, two tiles in turn
    uint32_t rows[2][2][64];          // sums over a tile's rows of two results, two tiles in turn
};

// Where a thread sits; finishers: tensor-memory lane 32 (warp % 4) + lane, plane
// p, row r of the 64 x 64 tile, columns c0 .. c0 + 31.
struct Thread {
    int tid, lane, warp, p, r, c0;
    uint32_t tm;      // this thread's lane and first column in tensor memory
    unsigned char *smem;
    bool ok;          // no wait gave up (then the remaining ones are skipped)
};

// Barrier of the finishers, with a vote.
__device__ __forceinline__ bool fsync_and(bool p) {
    int r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.and.pred q, 1, %2, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((int)p), "n"(kFinishers)
        : "memory");
    return r != 0;
}
template <int N>
__device__ __forceinline__ void regs_up() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void regs_down() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
__device__ __forceinline__ void arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_addr(bar)) : "memory");
}

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

// N = 64 n columns: slices t0 .. t0 + n - 1 of B against slice s of A, at
// tensor-memory columns 64 (s + t0) on.
__device__ __forceinline__ void issue_chain(uint32_t tmem, uint64_t da, uint64_t db, int s, int t0, int n,
                                            uint32_t acc) {
    const uint64_t a = da + (uint64_t)(s * (int)(kASliceB / 16)), b = db + (uint64_t)(t0 * (int)(kBSliceB / 16));
    oz::mma_bf16(tmem + 64u * (uint32_t)(s + t0), a, b, idesc(64 * n), acc);
    oz::mma_bf16(tmem + 64u * (uint32_t)(s + t0), a + 2, b + 128, idesc(64 * n), 1u);
}

// The MMAs of slice s of A (and, recursively, of the slices after it): the slices
// of B that it meets (level s + t kept) stacked along N in chains of at most four.
// FRESH starts the levels: s = 0 starts levels 0 .. S - 1; with one level more than
// slices the pair (1, S - 1) starts that one.
template <int S, bool FRESH, int s = 0>
__device__ __forceinline__ void issue_stage(uint32_t tmem, uint64_t da, uint64_t db) {
    constexpr int levels = Digits<S>::levels;
    constexpr int nt = levels - s < S ? levels - s : S;
    constexpr int first = nt <= 4 ? nt : nt == 7 ? 4 : 3;
    constexpr uint32_t acc = FRESH && s == 0 ? 0u : 1u;
    issue_chain(tmem, da, db, s, 0, first, acc);
    if constexpr (nt > first) {
        if constexpr (FRESH && s == 1 && (levels > S)) {
            issue_chain(tmem, da, db, s, first, nt - first - 1, 1u);
            issue_chain(tmem, da, db, s, nt - 1, 1, 0u);
        } else {
            issue_chain(tmem, da, db, s, first, nt - first, acc);
        }
    }
    if constexpr (s + 1 < S) issue_stage<S, FRESH, s + 1>(tmem, da, db);
}

// The issuing warp: `products` products of nst stages each.  Returns whether
// every wait ended.
template <int S>
__device__ __forceinline__ bool issue_products(Shared &s, const unsigned char *smem, i64 products, int nst) {
    using D = Digits<S>;
    const uint32_t base = tc::smem_addr(smem);
    uint32_t b = 0, round = 0, groups = 0;  // buffer, times round the buffers
    bool ok = true;
    for (i64 k = 0; k < products && ok; ++k)
        for (int st = 0; st < nst; ++st) {
            const bool fresh = (st & (kGroup - 1)) == 0;
            const uint32_t set = groups % D::sets, turn = groups / D::sets;
            ok = tc::mbar_wait(&s.full[b], round & 1, kWait);
            if (fresh && turn > 0) ok = ok && tc::mbar_wait(&s.drained[set], (turn - 1) & 1, kWait);
            if (!ok) break;
            tc::fence_after_sync();
            const uint64_t da = desc_k_sw64(base + b * D::stage_bytes);
            const uint64_t db = oz::desc_mn_sw128(base + b * D::stage_bytes + S * kASliceB, kBSliceB);
            const uint32_t tmem = s.tmem_base + set * 64u * D::levels;
            if (fresh)
                issue_stage<S, true>(tmem, da, db);
            else
                issue_stage<S, false>(tmem, da, db);
            tc::mma_commit(&s.done[b]);
            if (st + 1 == nst || (st & (kGroup - 1)) == kGroup - 1) {
                tc::mma_commit(&s.ready[set]);
                ++groups;
            }
            if (++b == D::stages) b = 0, ++round;
        }
    // What was issued finishes before tensor memory is freed.
    tc::mma_commit(&s.last);
    return tc::mbar_wait(&s.last, 0, kWait) && ok;
}

// Four 64-bit values of a 32-byte piece.
__device__ __forceinline__ void load4(const i64 *p, i64 &a, i64 &b, i64 &c, i64 &d) {
    asm volatile("ld.global.v4.b64 {%0,%1,%2,%3}, [%4];" : "=l"(a), "=l"(b), "=l"(c), "=l"(d) : "l"(p) : "memory");
}
__device__ __forceinline__ void store4(i64 *p, i64 a, i64 b, i64 c, i64 d) {
    asm volatile("st.global.v4.b64 [%0], {%1,%2,%3,%4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
}

// One operand of a product: element (row, col) of plane p at
// ptr + p * plane + row * rs + (col / 4) * qs + col % 4, normalised by `shift`
// bits.
struct Operand {
    const i64 *ptr;
    i64 rs, qs, plane;
    int shift;
};

// A thread's share of the cutting: eight columns of one row and plane of A (the
// row of a lane is laid out so that the eight lanes of a store phase meet eight
// different 16-byte banks) and of B (rows k of the stage).
struct Cut {
    const i64 *a, *b;    // stage 0
    i64 aqs, bqs, brs;   // from one piece to the next; from one row of B to the next
    int k, ash, bsh;     // B: row within the stage; shifts
    uint32_t o0, o1, ob;  // byte offsets within a slice (A: the two copies)
    bool n0, n1;         // A: the copies that are negated
};

// With `imag` the operand is i A: the product is i A B.
template <int S>
__device__ __forceinline__ Cut make_cut(const Thread &t, const Operand &A, const Operand &B, bool imag) {
    Cut c;
    const int l = t.lane, w = t.warp & 7, p = w >> 2;
    const int row = ((l >> 1) & 1) | ((l >> 2) & 2) | (l & 4) | ((l >> 1) & 8) | ((w & 3) << 4);
    const int k = 8 * (l & 1);
    c.a = A.ptr + p * A.plane + row * A.rs + (k / 4) * A.qs;
    c.aqs = A.qs;
    c.ash = A.shift;
    // A_r: [A_r | .] of the real rows and [. | A_r] of the imaginary rows;
    // A_i: [A_i | .] of the imaginary rows and [. | -A_i] of the real rows.
    // (i A: the parts -A_i and A_r in their places.)
    const int q = imag ? 1 - p : p;
    c.o0 = sw64(q ? 64 + row : row, k);
    c.o1 = sw64(q ? row : 64 + row, kStageK + k);
    c.n0 = imag && p != 0;
    c.n1 = imag || p != 0;
    c.k = ((w & 3) << 2) | (l >> 3);
    const int col = 8 * (l & 7);
    c.b = B.ptr + p * B.plane + c.k * B.rs + (col / 4) * B.qs;
    c.bqs = B.qs;
    c.brs = B.rs;
    c.bsh = B.shift;
    c.ob = S * kASliceB + oz::sw(kStageK * p + c.k, col);
    return c;
}

// Values of stage st; rows of B from kvalid on are zero.
__device__ __forceinline__ void load_a(const Cut &c, int st, i64 (&v)[8]) {
    const i64 *p = c.a + (i64)st * (kStageK / 4) * c.aqs;
    load4(p, v[0], v[1], v[2], v[3]);
    load4(p + c.aqs, v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void load_b(const Cut &c, int st, int kvalid, i64 (&v)[8]) {
    if (st * kStageK + c.k < kvalid) {
        const i64 *p = c.b + (i64)st * kStageK * c.brs;
        load4(p, v[0], v[1], v[2], v[3]);
        load4(p + c.bqs, v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = 0;
    }
}

// One slice (16 bytes: eight digits) from words that hold the digits of a pair
// of values in bytes 0 and 2 (LOW) or 1 and 3.  0x6400 | byte is 1024 + byte in
// fp16; 1152 less is the digit.
template <bool ISA, int K, bool LOW>
__device__ __forceinline__ void cut_slice(const Cut &c, unsigned char *stage, const uint32_t (&z)[4]) {
    uint32_t b[4], q[4], m[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        b[i] = LOW ? (z[i] & 0x00FF00FFu) | 0x64006400u : __byte_perm(z[i], 0x64646464u, 0x4341);
        asm("sub.f16x2 %0, %1, %2;" : "=r"(q[i]) : "r"(b[i]), "r"(0x64806480u));
    }
    const uint4 v = make_uint4(q[0], q[1], q[2], q[3]);
    if (ISA) {
        unsigned char *base = stage + K * kASliceB;
        if (c.n1) {  // (n0 only with n1)
#pragma unroll
            for (int i = 0; i < 4; ++i) asm("sub.f16x2 %0, %1, %2;" : "=r"(m[i]) : "r"(0x64806480u), "r"(b[i]));
            const uint4 n = make_uint4(m[0], m[1], m[2], m[3]);
            *reinterpret_cast<uint4 *>(base + c.o0) = c.n0 ? n : v;
            *reinterpret_cast<uint4 *>(base + c.o1) = n;
        } else {
            *reinterpret_cast<uint4 *>(base + c.o0) = v;
            *reinterpret_cast<uint4 *>(base + c.o1) = v;
        }
    } else {
        *reinterpret_cast<uint4 *>(stage + K * kBSliceB + c.ob) = v;
    }
}

// Digits of eight values into the stage's slices.  The shift and the digit bias
// are multiply-adds (the integer pipe for logic and shifts is the busier one);
// the bytes of a pair of values come together in four words.
template <int S, bool ISA>
__device__ __forceinline__ void cut_store(const Cut &c, unsigned char *stage, i64 (&v)[8]) {
    // The digit bias of the S bytes and half a unit of the next.
    constexpr u64 kBias = 0x8080808080808080ull << (8 * (7 - S));
    int h = ISA ? c.ash : c.bsh;
    if (h >= 32) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = (i64)((u64)v[j] << 32);
        h -= 32;
    }
    const uint32_t mul = 1u << h;
    uint32_t z[4][4];  // [bytes 0-1, 2-3 of the low words, of the high words][pair]
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t lo[2], hi[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const u64 x = (u64)v[2 * i + k];
            const u64 w = (u64)(uint32_t)x * mul + kBias;
            lo[k] = (uint32_t)w;
            hi[k] = (uint32_t)(w >> 32) + (uint32_t)(x >> 32) * mul;
        }
        if (S > 6) z[0][i] = __byte_perm(lo[0], lo[1], 0x5410);
        if (S > 4) z[1][i] = __byte_perm(lo[0], lo[1], 0x7632);
        z[2][i] = __byte_perm(hi[0], hi[1], 0x5410);
        z[3][i] = __byte_perm(hi[0], hi[1], 0x7632);
    }
    cut_slice<ISA, 0, false>(c, stage, z[3]);
    cut_slice<ISA, 1, true>(c, stage, z[3]);
    cut_slice<ISA, 2, false>(c, stage, z[2]);
    cut_slice<ISA, 3, true>(c, stage, z[2]);
    if constexpr (S > 4) cut_slice<ISA, 4, false>(c, stage, z[1]);
    if constexpr (S > 5) cut_slice<ISA, 5, true>(c, stage, z[1]);
    if constexpr (S > 6) cut_slice<ISA, 6, false>(c, stage, z[0]);
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

// Integers held in floats, |f| <= 2^22: f + 1.5 2^23 has f in its low bits.
constexpr float kMagic = 12582912.0f;
constexpr uint32_t kIntBias = 0x4B400000u;
__device__ __forceinline__ uint32_t biased_int(float f) { return __float_as_uint(__fadd_rn(f, kMagic)); }
// f = 256 q + r for an integer |f| < 2^24: biased q, and r (|r| <= 128).
__device__ __forceinline__ uint32_t split8(float f, float &r) {
    const float q = __fmaf_rn(f, 0.00390625f, kMagic);
    r = __fmaf_rn(__fsub_rn(q, kMagic), -256.0f, f);
    return __float_as_uint(q);
}

// Adds sum_L D_L 2^(-8 L) in the units of the thread's sums, of which a product of
// two items of scale 2^-62 has 2^(56 - sh) in level 0 (sh = 6 + the product's head, 11
// .. 24).
//
// Levels 0 .. 2 stay within 2^22 and convert by an addition; 3 .. 5 split into a
// multiple of 256 and a rest first (the conversion unit takes eight clocks a
// warp).  Of eight levels the rests of 4 and 5 and levels 6 and 7 are below 2^22 in
// the result's units and meet in FP32, good to 2^-2 of its last bit.
template <int S>
__device__ __forceinline__ void drain(const Thread &t, uint32_t set, int sh, i64 (&acc)[kCols]) {
    constexpr int levels = Digits<S>::levels;
    const uint32_t m3 = 1u << (32 - sh);                     // level 3
    const int m4 = 1 << (24 - sh);                           // level 4
    const float f4 = __int_as_float((127 + 24 - sh) << 23);  // the same
    const float f5 = __int_as_float((127 + 16 - sh) << 23);  // level 5
    const float f6 = __int_as_float((127 + 8 - sh) << 23);   // level 6
    const uint32_t tm = t.tm + set * 64u * levels;
#pragma unroll
    for (int g = 0; g < kCols / 4; ++g) {
        float f[8][4];
#pragma unroll
        for (int L = 0; L < levels; ++L) tmem_ld4(tm + 64u * L + 4u * g, f[L]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float r3;
            const uint32_t q3 = split8(f[3][j], r3);
            const int h01 = (int)(biased_int(f[0][j]) * 256u + biased_int(f[1][j]) - 257u * kIntBias);
            const int h23 = (int)((biased_int(f[2][j]) + q3) * 256u + biased_int(r3) - 513u * kIntBias);
            i64 v = acc[4 * g + j];
            if constexpr (levels == 8) {
                float r4, r5;
                const uint32_t q4 = split8(f[4][j], r4), q5 = split8(f[5][j], r5);
                const int q45 = (int)(q4 * 256u + q5 - 257u * kIntBias);
                float l = __fmaf_rn(__fmaf_rn(f[7][j], 0.00390625f, f[6][j]), f6, kMagic);
                l = __fadd_rn(__fmaf_rn(r4, f4, __fmul_rn(r5, f5)), l);
                v += (i64)q45 * m4 + (int)(__float_as_uint(l) - kIntBias);
            } else if constexpr (levels == 5) {
                v += (i64)__float2int_rn(f[4][j]) * m4;
            }
            acc[4 * g + j] = (i64)((u64)((i64)h01 * 65536 + h23) * (u64)m3 + (u64)v);
        }
    }
}

// Whether the wait ended for every lane (a warp leaves its loop as a whole).
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity) {
    return __all_sync(0xffffffffu, tc::mbar_wait(bar, parity, kWait)) != 0;
}

// The cutters' loop over the products of `w`, which deals out products (first,
// more, next) and gives their operands.  The values of the next stage are on
// their way while a stage is cut: those of A once A's are used, those of B once
// B's are.  Before product n is touched, product n - 2 has to be finished, and
// n - 1 too where `needs` says so.
template <int S, class W>
__device__ __forceinline__ void cutter(Shared &s, Thread &t, const W &w, int nst, int kvalid) {
    using D = Digits<S>;
    typename W::At at = w.first(), before = at;
    if (!w.more(at)) return;
    uint32_t b = 0, round = 0, n = 0, seen = 0;
    int st = 0;
    Cut c;
    i64 va[8], vb[8];
    auto begin = [&] {
        const uint32_t until = finished_before(n, w.needs(at, before));
        for (; seen < until; ++seen)
            if (t.ok) t.ok = warp_wait(&s.finished[finished_bar(seen)], finished_parity(seen));
        Operand A, B;
        const bool imag = w.operands(at, A, B);
        c = make_cut<S>(t, A, B, imag);
    };
    begin();
    load_a(c, 0, va);
    load_b(c, 0, kvalid, vb);
    while (t.ok) {
        if (round > 0) t.ok = warp_wait(&s.done[b], (round - 1) & 1);
        unsigned char *stage = t.smem + b * D::stage_bytes;
        const bool same = st + 1 < nst;  // the next stage is of this product
        cut_store<S, true>(c, stage, va);
        if (same) load_a(c, st + 1, va);
        cut_store<S, false>(c, stage, vb);
        if (same) load_b(c, st + 1, kvalid, vb);
        tc::fence_proxy_async();
        __syncwarp();
        if (t.lane == 0) arrive(&s.full[b]);
        if (++b == D::stages) b = 0, ++round;
        if (same) {
            ++st;
            continue;
        }
        st = 0;
        before = at;
        at = w.next(at);
        if (!w.more(at)) break;
        ++n;
        begin();
        load_a(c, 0, va);
        load_b(c, 0, kvalid, vb);
    }
}

// The finishers' loop: the levels of every group of stages into the sums, then
// w.epilogue (false ends).
template <int S, class W>
__device__ __forceinline__ void finisher(Shared &s, Thread &t, const W &w, int nst) {
    using D = Digits<S>;
    uint32_t groups = 0, n = 0;
    for (typename W::At at = w.first(); w.more(at); at = w.next(at), ++n) {
        i64 T[kCols];
        const int sh = 6 + w.head(at);
#pragma unroll
        for (int j = 0; j < kCols; ++j) T[j] = 0;
        for (int st = 0; st < nst; st += kGroup, ++groups) {
            const uint32_t set = groups % D::sets;
            if (t.ok) t.ok = tc::mbar_wait(&s.ready[set], (groups / D::sets) & 1, kWait);
            tc::fence_after_sync();
            drain<S>(t, set, sh, T);
            tc::fence_before_sync();
            __syncwarp();
            if (t.lane == 0) arrive(&s.drained[set]);
        }
        if (!w.epilogue(at, T, n)) break;
        __syncwarp();
        if (t.lane == 0) arrive(&s.finished[finished_bar(n)]);
    }
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
// with t real (a thread holds one plane of T).  A second result is one of T where the
// first is plain, else of the first result in T's place.
struct Out {
    int buf;  // -1: none
    int plain, nterm;
    int grid;  // E of complex64: 1 + the diagonal's real parts rounded to FP32
    Coef t;
    Term term[kTerms];
    Coef diag;
};
struct Op {
    int a, b;  // operands
    int imag;  // T = i A B, else A B
    Out out[2];
};

// An item as the epilogue sees it: this thread's row and first column.
struct View {
    const i64 *re;  // plane 0; plane 1 at + plane
    Info info;
};

// What is known of T: its units 2^eT, values below 2^(eT - h), row norms r in units of
// 2^eT.
struct Sum {
    int e, h;
    float r;
};
// Exponent and row norm (in its units) of a result: two above the largest of up to four
// addends.
template <class V>
__device__ __forceinline__ int out_exponent(const Out &o, Sum T, float cap, V view, bool &poison, float &norm) {
    if (o.plain) {
        norm = fminf(T.r, cap);
        return T.e;
    }
    auto size = [](const Coef &c) { return fabsf((float)(int)(c.m >> 32)) * 9.3132257e-10f; };  // 2^(32 - 62)
    int e = -1000000;
    const int ref = T.e + o.t.e;  // r in units of 2^ref
    float r = 0.0f;
    if (o.t.m) {
        e = ref - T.h;
        r = size(o.t) * T.r;
    }
#pragma unroll 1
    for (int k = 0; k < o.nterm; ++k) {
        const Info i = view(o.term[k].buf).info;
        const Coef c = o.term[k].c;
        if (i.mb == kPoison) poison = true;
        const int ek = i.e - headroom(i) + c.e;
        e = max(e, ek);
        r += size(c) * row_norm(i, cap) * pow2f(ek - ref);
    }
    if (o.diag.m) {
        e = max(e, o.diag.e);
        r += size(o.diag) * pow2f(o.diag.e - ref);
    }
    e += 2;
    norm = fminf(1.001f * r * pow2f(ref - e), cap);
    return e;
}

// A coefficient and the shift that its product needs, as one factor: the upper
// half of v * factor is the term in the result's units.  The upper and lower
// words of the factor are signed.  A coefficient of one is a shift alone.
struct Factor {
    int hi, lo, pre;  // pre: left shift of v first (a short item meets a large result)
    int sh;           // > 0: v >> sh, rounded
};
constexpr i64 kOne = 1ll << 61;
__device__ __forceinline__ Factor make_factor(i64 m, int sr, int headroom) {
    const int s = min(sr, 63) - headroom;
    Factor f;
    f.pre = s < 0 ? -s : 0;
    f.sh = m == kOne && s + 3 < 32 ? max(s, 0) + 3 : 0;
    if (s > 0) m = ((m >> (s - 1)) + 1) >> 1;
    f.lo = (int)(uint32_t)(u64)m;
    f.hi = (int)((m - f.lo) >> 32);
    return f;
}
// v * factor / 2^64, rounded (the product of the low words is left out, a
// quarter of a unit at most).  Rounding down instead would add the same sign to
// every element at every step.
__device__ __forceinline__ i64 scaled(i64 v, const Factor &f) {
    const int lo = (int)(uint32_t)(u64)v;
    const int hi = (int)(v >> 32) + (int)((uint32_t)lo >> 31);  // with the low word read as signed
    const i64 mid = (i64)lo * f.hi + ((i64)hi * f.lo + 0x80000000ll);
    return (i64)hi * f.hi + (int)(mid >> 32);
}
template <int N>
__device__ __forceinline__ void scale_add(const Factor &f, const i64 (&x)[N], i64 *acc, bool add) {
    if (f.sh) {
        const i64 half = 1ll << (f.sh - 1);
#pragma unroll
        for (int j = 0; j < N; ++j) acc[j] = ((x[j] + half) >> f.sh) + (add ? acc[j] : 0);
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) acc[j] = scaled(x[j], f) + (add ? acc[j] : 0);
    }
}

// One result, for this thread's columns of its row and plane: formed in place
// of T, stored at dst (pieces qs apart, as those of the terms); returns the OR of
// the magnitudes (ones' complement for negative values), and adds their sum in units
// of 2^38 to `sum` (below 2^29).  row, col0: global row
// and first column; diagonal entries below d only.  The loads of a term go out
// together: one wait per term, not one per piece.
template <class V>
__device__ __forceinline__ u64 put_out(const Out &o, const Thread &t, i64 (&T)[kCols], Sum S, int e, V view, i64 plane,
                                       i64 qs, int row, int col0, int d, i64 *dst,
                                       uint32_t *sum = nullptr) {
    if (!o.plain) {
        // T times its coefficient, then the terms, a quarter of the columns at a time;
        // the first loads go out before the multiplication.
        const Factor ft = o.t.m ? make_factor(o.t.m, e - (S.e - S.h) - o.t.e - 2, S.h) : Factor{0, 0, 0, 0};
        constexpr int H = kCols / 4;
#pragma unroll 1
        for (int k = 0; k < max(1, o.nterm); ++k) {
            Factor f{0, 0, 0, 0};
            const i64 *q = nullptr;
            if (k < o.nterm) {
                const View w = view(o.term[k].buf);
                const Coef c = o.term[k].c;
                q = w.re + (c.imag ? 1 - t.p : t.p) * plane;
                const int hr = headroom(w.info);
                f = make_factor((c.imag && t.p == 0) ? -c.m : c.m, e - (w.info.e - hr) - c.e - 2, hr);
            }
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                i64 x[H];
                if (q) {
#pragma unroll
                    for (int i = 0; i < H / 4; ++i)
                        load4(q + (h * H / 4 + i) * qs, x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]);
                }
                if (k == 0) {
                    i64 v[H];
#pragma unroll
                    for (int j = 0; j < H; ++j) v[j] = (i64)((u64)T[h * H + j] << ft.pre);
                    scale_add<H>(ft, v, T + h * H, false);
                }
                if (q) {
                    if (f.pre) {
#pragma unroll
                        for (int j = 0; j < H; ++j) x[j] = (i64)((u64)x[j] << f.pre);
                    }
                    scale_add<H>(f, x, T + h * H, true);
                }
            }
        }
        if (o.diag.m && t.p == o.diag.imag && row < d && row >= col0 && row < col0 + kCols) {
            const i64 x = o.diag.m >> min(e - o.diag.e, 63);
#pragma unroll
            for (int j = 0; j < kCols; ++j)
                if (row == col0 + j) T[j] += x;
        }
        if (o.grid && t.p == 0 && row < d && row >= col0 && row < col0 + kCols) {
#pragma unroll
            for (int j = 0; j < kCols; ++j)
                if (row == col0 + j) {
                    const float u = (float)(1.0 + scalbn((double)T[j], e - 62));
                    T[j] = __double2ll_rn(scalbn((double)u - 1.0, 62 - e));
                }
        }
    }
    u64 m = 0;
#pragma unroll
    for (int i = 0; i < kCols / 4; ++i) {
        store4(dst + i * qs, T[4 * i], T[4 * i + 1], T[4 * i + 2], T[4 * i + 3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) m |= (u64)(T[4 * i + j] ^ (T[4 * i + j] >> 63));
    }
    if (sum) {
        uint32_t u = 0;
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
            const int hi = (int)(T[j] >> 32);
            u += (uint32_t)(hi ^ (hi >> 31)) >> 6;
        }
        atomicAdd(sum, u + kCols);
    }
    return m;
}

// OR over the warp into the finishers' OR of result o of product n.
__device__ __forceinline__ void merge_or(Shared &s, const Thread &t, uint32_t n, int o, u64 m) {
    const uint32_t hi = __reduce_or_sync(0xffffffffu, (uint32_t)(m >> 32));
    const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)m);
    if (t.lane == 0) {
        atomicOr(&s.orhi[n & 3][o], hi);
        atomicOr(&s.orlo[n & 3][o], lo);
    }
}
// After the finishers' barrier of product n: its result o; clears the place of
// product n - 1, which every finisher has read by then and none fills before n + 3.
__device__ __forceinline__ u64 read_or(Shared &s, const Thread &t, uint32_t n, int o) {
    const u64 m = (u64)s.orhi[n & 3][o] << 32 | s.orlo[n & 3][o];
    if (t.tid == 0) s.orhi[(n - 1) & 3][o] = s.orlo[(n - 1) & 3][o] = 0;
    return m;
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
    t.c0 = kCols * (t.warp >> 2);
    t.smem = raw + ((1024u - (tc::smem_addr(raw) & 1023u)) & 1023u);
    t.ok = true;
    if (t.tid < 8) s.orhi[t.tid >> 1][t.tid & 1] = s.orlo[t.tid >> 1][t.tid & 1] = 0;
    if (t.tid < 128) s.rowmb[t.tid >> 6][t.tid & 63] = 0;
    if (t.tid < 256) s.rows[t.tid >> 7][(t.tid >> 6) & 1][t.tid & 63] = 0;
    if (t.warp == 0) {
        tc::tmem_alloc(&s.tmem_base, 512);
        tc::tmem_relinquish();
    }
    if (t.tid == 0) {
        for (int b = 0; b < kMaxStages; ++b) {
            tc::mbar_init(&s.full[b], kCutters / 32);
            tc::mbar_init(&s.done[b], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&s.ready[b], 1);
            tc::mbar_init(&s.drained[b], kFinishers / 32);
        }
        for (uint32_t b = 0; b < kFinishedBars; ++b) tc::mbar_init(&s.finished[b], kFinishers / 32);
        tc::mbar_init(&s.last, 1);
        tc::fence_mbar_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    t.tm = s.tmem_base + ((uint32_t)(32 * q4) << 16) + (uint32_t)t.c0;
}

// A launch: every role over the products of w (`products` of them for this CTA).
template <int S, class W>
__device__ __forceinline__ void run(Shared &s, Thread &t, const W &w, i64 products, int nst, int kvalid) {
    if (t.tid >= kIssuer) {
        regs_down<kRegsIssue>();
        if (t.tid == kIssuer) t.ok = issue_products<S>(s, t.smem, products, nst);
    } else if (t.tid >= kFinishers) {
        regs_down<kRegsCut>();
        cutter<S>(s, t, w, nst, kvalid);
    } else {
        regs_up<kRegsFinish>();
        finisher<S>(s, t, w, nst);
    }
}

// The CTA's end; ok: this thread's waits all ended.
__device__ __forceinline__ void teardown(Shared &s, const Thread &t, bool ok, int *fault) {
    tc::fence_before_sync();
    const bool all = __syncthreads_and(ok) != 0;
    if (!all && t.tid == 0 && fault) atomicAdd(fault, 1);
    if (t.warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(s.tmem_base, 512);
    }
}

}  // namespace fx
}  // namespace pgb
