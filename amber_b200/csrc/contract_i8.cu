// Mixed-precision triple-product lag accumulation on the int8 tensor cores: the
// lag-space GEMM of lagspace.cuh run as tcgen05 kind::i8 MMAs with exact int32
// accumulation in TMEM, FP64 recombination per pixel block and the compensated
// FP64 reduction of ls_reduce.  Replaces the float loop of 4_fbe/amber.c:247-279
// / amber_v2.c:243-283.
//
// Why not FP32 accumulation: on the B200 tensor cores a long FP32 accumulation
// chain of coherent (same-sign) products loses ~2^-24 of the running sum per
// step, which breaks the 1e-6-of-Σ|products| bound on the v2 sampling-mask
// sums; integer accumulation has no rounding at all.
//
// Representation.  Every block of 256 pixels of every ring map has one exponent
// E (maps.cu), shared by all channels.  Within block b the D2 operand is three
// base-254 digits of t = w·D2·127·2^−E2 (quantize_kernel), and the per-anchor
// product w·D1[p1]·w·D3[p3] is formed in FP32 on the CUDA cores (packed FP32x2),
// scaled by 127·2^−(E1+E3) and cut into three digits (the D maps) or four (the
// sampling-mask maps).  With Q_i the D2 digits and P_j the product digits:
//     Σ_x (w1D1)(w2D2)(w3D3) = 2^(E1+E2+E3)/127² · Σ_k 254^−k Σ_{i+j=k} Σ_x Q_i P_j.
// Class k accumulates in its own int32 TMEM accumulator.  Classes 0-2 (six
// MMAs per 32 pixels) bound the D-map error near 1e-7 of Σ|products|; the
// peaked sampling-mask maps also need class 3 (P3·Q0 + P2·Q1 + P1·Q2).  Up to
// N = 96 four accumulators and four-digit A buffers fit TMEM, and a mask block runs
// one sweep; at N = 128 it runs a second sweep that forms digits 1-3 of the product
// and accumulates class 3 alone.  The numbers behind this choice: a numpy
// emulation of these exact digit operations on the single-realisation
// workload's Ng1 = 354 and 740 maps gave 6–9e-8 (D, classes 0-2) and
// 4.5e-8 (mask, classes 0-3), against 5–8e-7 for the mask maps without class 3.
// A per-block exponent is what lets all anchors share one accumulator: the
// scale of a product no longer depends on its channels.  |class sum| ≤
// 3·127² per pixel and anchor, and a block holds at most 173 anchor groups of
// 256 pixels (44288 terms): the int32 accumulators cannot overflow.
//
// Operands.  A (TMEM, M = 128 rows Δ3, written by the formers with tcgen05.st)
// = the per-anchor product digits; B (shared memory, N ≤ 128 rows Δ2) = the D2
// digits of the anchor's window, read straight from the staged channel rows at
// the window's offset: TMA writes the D2 digits as [digit][16-pixel group]
// [channel][16 bytes], the K-major no-swizzle layout of 8-row core matrices,
// whose rows may start at any channel.  Per 32-pixel slice a unit stages, once,
// the fp32 D3 rows of its span (128B-swizzled, conflict-free row reads), the
// fp32 D1 rows of its anchor block and the D2 digits of its window span, and
// then runs every anchor group of the block against them.
//
// Warp roles (640 threads): warps 0-15 form the A digits (four sets of four
// warps, each set a whole anchor group, warp w the TMEM lanes 32·(w mod 4) .. +31)
// and run each block's epilogue; warp 16 streams the slices by TMA; warps 17 and
// 18 issue the MMAs, one elected thread each, into accumulators of their own;
// warp 19 scales the staged D1 rows.  Four to eight A buffers (as many as TMEM
// holds beside the accumulators; four are left at N = 96 and 48 of the four-digit
// modes, one for each set of formers) let the formers run ahead of the tensor
// pipe.  Every wait is bounded; on expiry the CTA raises an error flag the host
// turns into AMBER_ERR_TIMEOUT, drains its copies and MMAs after its last barrier
// and frees TMEM.  No cluster launch and no multicast.
//
// What bounds it, and what it measured (one CTA per SM, cycles per anchor group
// and 32-pixel slice on the Ng1 = 740 maps, 128 channels, nclen = 127; triangles
// of that size took 6.14 ms each before and 3.5 ms now):
//   * 932 before.  The six MMAs of a group need 384 cycles at N = 128 (N/2 each,
//     42 at least), 312 over the channel range alone.  The issuing warp was the
//     bound: an mbarrier wait per group, operands the compiler did not know to be
//     uniform (a register-to-uniform move each), and issue slots shared with the
//     formers.  Counts in place of barriers, one elected thread per issuing warp,
//     operands from a table and two issuing warps took it to 362 with the formers'
//     arithmetic switched off.
//   * 415 now, and the formers are the bound: ~240 instructions per warp and group at
//     62 % of the issue slots.  A packed FP32x2 op with three different 64-bit operands
//     costs 3.3 cycles against 1.0 for a scalar one and PRMT costs 2, so packed
//     ops save issue slots rather than pipe time: all-scalar digits were 8 % slower.
//   * Blocks of 8 rows outside the channel range are skipped (a quarter of them at
//     nc10 = nc/2 − 1, half at nc − 1).  12 or 20 former warps in place of 16
//     (128 or 80 registers each) were 8 % and 6 % slower.
#include <string.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <tuple>
#include <type_traits>
#include <vector>

#include "lagspace.cuh"
#include "tc_ptx.cuh"

namespace amber {

namespace {

using namespace tc;

constexpr int SLICE = 32;                    // pixels per K step (one kind::i8 MMA)
constexpr int NSLICE = LS_BLOCK / SLICE;     // slices per block
constexpr int NFORM = 16;                    // former / epilogue warps
constexpr int WARP_TMA = NFORM, WARP_MMA = NFORM + 1, WARP_MMA2 = NFORM + 2, WARP_SCALE = NFORM + 3;
constexpr int NMMA = 2;                      // MMA issuing warps
constexpr int NTHREADS = (NFORM + 4) * 32;
constexpr int TMEM_COLS = 512;
constexpr int NSET = NFORM / 4;              // former sets: each anchor group is formed by one set of 4 warps
constexpr int ABUF_COLS = 24;                // A buffer: 3 digits × 8 columns (32 int8 per row per digit)
constexpr int ABUF4_COLS = 32;               // with four digits
constexpr int NABUF_MAX = 8;                 // A buffers: as many as TMEM holds beside the accumulators
constexpr long MIN_GROUPS = 4;                // least work of a unit (lagspace.cuh): two blocks of a single anchor group
constexpr int NSTAGE_MAX = 8;                // stages: as many as shared memory holds
static_assert(3 * LS_ROWS + 5 * ABUF_COLS <= TMEM_COLS, "TMEM: five A buffers beside the widest accumulators");
static_assert(NSET <= 4, "a set may be one use of a buffer ahead of the tensor pipe, not two: sets ≤ buffers");

// Shared memory: barriers, hand-off counts and the unit's anchor groups, then the stages.
constexpr int SM_FLAGS = 512;                // [NABUF_MAX] hand-off counts of the A buffers
constexpr int SM_GROUPS = 768;               // [LS_SPAN + 1] anchor groups (uint4)
constexpr int SM_STAGES = 5 * 1024;
constexpr int SMEM_STAGES = 220 * 1024;      // bytes of all stages
static_assert(SM_GROUPS + 16 * (LS_SPAN + 1) <= SM_STAGES, "group table");
constexpr size_t SMEM_BYTES = 1024 + (size_t)SM_STAGES + SMEM_STAGES;

struct alignas(64) I8Desc {
    CUtensorMap t3;  // w·D3 fp32 {k, nc}, box {32, span3}, 128B swizzle
    CUtensorMap t1;  // w·D1 fp32 {k, nc}, box {32, AB}
    CUtensorMap t2;  // D2 digits {16, nc, kp/16, 3}, box {16, span2, 2, 3}
    CUtensorMap t2b; // a pair's second D2 (the other triangle with the same D1 and D3)
    const int *e1, *e2, *e2b, *e3;  // block exponents
    long tile2;                     // doubles from a unit's partial tile to the pair's second one
    const int *groups, *group_off;  // anchor groups of every anchor block
    long k;
    int nc, nc10, nclen, ks, rs, AB, ts;
    int span3, span2;
    int mask;                       // sampling-mask maps: class 3 as well
    uint32_t tx_bytes;              // bytes one slice's three TMA boxes deliver
    int nst, st_bytes, st_d1, st_d2, st_d2b;  // stages, bytes of one, offsets of its D1 rows and D2 digits (D3 first)
};

__device__ __forceinline__ float2 sub2(float2 a, float2 b)
{
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tsub.rn.f32x2 z, x, y;\n\t"
        "mov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

// Three or four base-254 digits of two products u·v at once (packed FP32x2): the product enters the
// first rounding unrounded (y0 = fma(u, v, M)), and round-to-nearest through the 1.5·2^23 magic number
// leaves each digit's two's-complement byte in the low mantissa bits.  M − y = −digit exactly; each
// residual s = 254·s − d is one fused op.  Only M and 254 are held in registers: a third 64-bit operand
// costs a packed op a third cycle of register reads, and more constants cost moves.
template <int ND>
__device__ __forceinline__ void digits254x2(float2 u, float2 v, float2 (&y)[4])
{
    const float2 M = make_float2(12582912.0f, 12582912.0f), K = make_float2(254.f, 254.f);
    y[0] = __ffma2_rn(u, v, M);                          // M + d0
    float2 s = __ffma2_rn(u, v, sub2(M, y[0]));          // u·v − d0
#pragma unroll
    for (int i = 1; i < ND; ++i) {
        y[i] = __ffma2_rn(s, K, M);                      // M + di
        s = __ffma2_rn(s, K, sub2(M, y[i]));             // 254·s − di
    }
}

__device__ __forceinline__ uint32_t pack_low_bytes(float a, float b, float c, float d)
{
    return __byte_perm(__byte_perm(__float_as_uint(a), __float_as_uint(b), 0x0040),
                       __byte_perm(__float_as_uint(c), __float_as_uint(d), 0x0040), 0x5410);
}

// 16 lanes × 8 columns: lane t/4 and t/4 + 8, column t%4 (v[0], v[1]) and 4 + t%4 (v[2], v[3]) of thread t
__device__ __forceinline__ void tmem_st16x8(uint32_t taddr, const uint32_t (&v)[4])
{
    asm volatile("tcgen05.st.sync.aligned.16x128b.x2.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3])
                 : "memory");
}
// 16 lanes × 16 columns: v, then w eight columns on
__device__ __forceinline__ void tmem_st16x16(uint32_t taddr, const uint32_t (&v)[4], const uint32_t (&w)[4])
{
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                 : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}

__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y, int z,
                                            int w)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
        : "memory");
}

// One kind::i8 MMA (A from TMEM) and one commit, issued by the MMA warps' elected thread.  The operands
// live in uniform registers there; the descriptor's upper half is the same for every window.  ADD 0
// overwrites the accumulator's columns.
template <int ADD>
__device__ __forceinline__ void umma_i8(uint32_t d, uint32_t a, uint32_t qlo, uint32_t qhi, uint32_t idesc)
{
    asm volatile("{\n\t.reg .b64 q;\n\tmov.b64 q, {%2, %3};\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], q, %4, %5;\n\t}" ::"r"(d),
                 "r"(a), "r"(qlo), "r"(qhi), "r"(idesc), "n"(ADD)
                 : "memory");
}
__device__ __forceinline__ void umma_commit_bar(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool elect_one()
{
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}

// Shared-memory descriptor of a K-major operand without swizzle: 8-row core matrices of
// 16-byte rows stacked every 128 bytes (SBO), the second 16-byte K chunk `lbo` bytes on.
__device__ __forceinline__ uint64_t smem_desc_plain(uint32_t saddr, uint32_t lbo)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);      // start address
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;  // leading byte offset: K-adjacent core matrices
    d |= (uint64_t)((128 >> 4) & 0x3FFF) << 32;  // stride byte offset: the next 8 rows
    d |= (uint64_t)1 << 46;                      // descriptor version (sm_100)
    return d;                                    // swizzle mode 0: none
}

__device__ __forceinline__ float4 lds128(uint32_t a)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}

// Hand-off count of an A buffer: its set's four former warps add one each per use.  Relaxed counts
// between the tcgen05 fences are the hand-off the tensor unit needs; an mbarrier wait or an acquire
// load here holds the queued MMAs back by ~70 cycles a group.
__device__ __forceinline__ uint32_t count_load(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.relaxed.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void count_add(uint32_t a)
{
    asm volatile("red.relaxed.cta.shared.add.u32 [%0], 1;" ::"r"(a) : "memory");
}
__device__ __noinline__ bool count_wait(uint32_t a, uint32_t need, volatile int *abort_flag, int *err, int code)
{
    const long long t0 = clock64();
    while (count_load(a) < need) {
        if (*abort_flag) return false;
        if (clock64() - t0 > WAIT_CYCLES) {
            *abort_flag = 1;
            atomicExch(err, code);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ uint4 lds_u128(uint32_t a)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}

// What one MMA issuing thread keeps between its items.
struct IssueState {
    uint32_t groups, ngr;          // table of anchor groups (shared address), its length
    uint32_t acc, nmma, a_first;   // TMEM: this thread's first accumulator, accumulator stride, A buffers
    uint32_t desc_lo, desc_hi, ddig, stage16;  // D2 descriptor of stage 0, next digit, next stage (16-byte units)
    uint32_t flags, bars, nabuf;   // hand-off counts and ab_empty barriers (shared addresses)
    uint32_t ab, need, seen;       // current A buffer, the count that means formed, the count last seen
    uint32_t s, ph, nst;           // current stage, its parity, stages
};

// Issues the MMAs of one item (a pixel block, one sweep): every slice's anchor groups in order.
// SECOND: which of the two issuing threads; class k = Σ_{i+j=k} Q_i·P_j.
//   SW_D: the A buffer holds P0, P1, P2; the first thread runs classes 0 and 1, the second class 2.
//   SW_CLASS3: P1, P2, P3; class 3 = P3·Q0 + P2·Q1 (first) + P1·Q2 (second, an accumulator of its own).
//   SW_MASK4: P0 .. P3; the first thread runs classes 0 and 3, the second classes 1 and 2.
//   SW_PAIR, SW_PAIR4: three or four digits; each thread runs every class of one of the pair's triangles.
// The loop is kept to few instructions beside the MMAs: they wait for issue slots behind the formers of
// the same SM partition.
enum { SW_D, SW_CLASS3, SW_MASK4, SW_PAIR, SW_PAIR4 };

template <bool SECOND, int SWEEP>
__device__ __forceinline__ bool issue_item(IssueState &t, int nsl, uint64_t *st_full, uint64_t *st_empty,
                                           volatile int *abort_flag, int *err)
{
    bool first = true;
    for (int sl = 0; sl < nsl; ++sl) {
        if (!mbar_wait(&st_full[t.s], t.ph, abort_flag, err, 33)) return false;
        const uint32_t sd = t.desc_lo + t.s * t.stage16;
        // the first group of an item sets every column of the accumulators: the table's last entry
        uint4 e = lds_u128(first ? t.groups + 16 * t.ngr : t.groups);
        uint32_t next = t.groups;
        for (uint32_t g = 0; g < t.ngr; ++g) {
            const uint32_t q0 = sd + e.x, q1 = q0 + t.ddig, q2 = q1 + t.ddig, qh = t.desc_hi;
            const uint32_t d = t.acc + e.y, idesc = e.z, a = t.a_first + t.ab * (SWEEP == SW_MASK4 || SWEEP == SW_PAIR4 ? ABUF4_COLS : ABUF_COLS);
            const uint32_t bar = t.bars + t.ab * 8;
            next += 16;
            e = lds_u128(next);
            if (t.seen < t.need && !count_wait(t.flags + t.ab * 4, t.need, abort_flag, err, 34)) return false;
            fence_after();
            if (++t.ab == t.nabuf) { t.ab = 0; t.need += 4; }
            t.seen = count_load(t.flags + t.ab * 4);
            // the MMAs that may be the first into their accumulator, then the rest
            auto leading = [&](auto addc) {
                constexpr int ADD = decltype(addc)::value;
                if constexpr (SWEEP == SW_PAIR || SWEEP == SW_PAIR4) {
#pragma unroll
                    for (int i = 0; i < (SWEEP == SW_PAIR4 ? 4 : 3); ++i)
                        umma_i8<ADD>(d + i * t.nmma, a + 8 * i, q0, qh, idesc);
                } else if constexpr (SWEEP == SW_D && !SECOND) {
                    umma_i8<ADD>(d, a, q0, qh, idesc);
                    umma_i8<ADD>(d + t.nmma, a + 8, q0, qh, idesc);
                } else if constexpr (SWEEP == SW_D) {
                    umma_i8<ADD>(d, a + 16, q0, qh, idesc);
                } else if constexpr (SWEEP == SW_CLASS3 && !SECOND) {
                    umma_i8<ADD>(d, a + 16, q0, qh, idesc);
                } else if constexpr (SWEEP == SW_CLASS3) {
                    umma_i8<ADD>(d, a, q2, qh, idesc);
                } else if constexpr (!SECOND) {
                    umma_i8<ADD>(d, a, q0, qh, idesc);
                    umma_i8<ADD>(d + 3 * t.nmma, a + 24, q0, qh, idesc);
                } else {
                    umma_i8<ADD>(d, a + 8, q0, qh, idesc);
                    umma_i8<ADD>(d + t.nmma, a + 16, q0, qh, idesc);
                }
            };
            if (first) leading(std::integral_constant<int, 0>());
            else leading(std::integral_constant<int, 1>());
            first = false;
            if constexpr (SWEEP == SW_PAIR || SWEEP == SW_PAIR4) {
                constexpr int NC = SWEEP == SW_PAIR4 ? 4 : 3;
#pragma unroll
                for (int i = 1; i < NC; ++i) umma_i8<1>(d + i * t.nmma, a + 8 * (i - 1), q1, qh, idesc);
#pragma unroll
                for (int i = 2; i < NC; ++i) umma_i8<1>(d + i * t.nmma, a + 8 * (i - 2), q2, qh, idesc);
            } else if constexpr (SWEEP == SW_D && !SECOND) {
                umma_i8<1>(d + t.nmma, a, q1, qh, idesc);
            } else if constexpr (SWEEP == SW_D) {
                umma_i8<1>(d, a + 8, q1, qh, idesc);
                umma_i8<1>(d, a, q2, qh, idesc);
            } else if constexpr (SWEEP == SW_CLASS3 && !SECOND) {
                umma_i8<1>(d, a + 8, q1, qh, idesc);
            } else if constexpr (SWEEP == SW_MASK4 && !SECOND) {
                umma_i8<1>(d + 3 * t.nmma, a + 16, q1, qh, idesc);
                umma_i8<1>(d + 3 * t.nmma, a + 8, q2, qh, idesc);
            } else if constexpr (SWEEP == SW_MASK4) {
                umma_i8<1>(d, a, q1, qh, idesc);
                umma_i8<1>(d + t.nmma, a + 8, q1, qh, idesc);
                umma_i8<1>(d + t.nmma, a, q2, qh, idesc);
            }
            umma_commit_bar(bar);
        }
        umma_commit_bar(smem_u32(&st_empty[t.s]));
        if (++t.s == t.nst) { t.s = 0; t.ph ^= 1; }
    }
    return true;
}

// Whether a mask job's four class accumulators and four four-digit A buffers fit TMEM at MMA width nmma (≤ 96).
__host__ __device__ constexpr bool mask4_fits(int nmma) { return 4 * nmma + NSET * ABUF4_COLS <= TMEM_COLS; }

// Whether two triangles' accumulators and the A buffers fit TMEM: N ≤ 64 (D maps) or 48 (mask maps).
__host__ __device__ constexpr bool pair_fits(bool mask, int nmma)
{
    return mask ? 8 * nmma + NSET * ABUF4_COLS <= TMEM_COLS : 6 * nmma + NSET * ABUF_COLS <= TMEM_COLS;
}

// MODE of a launch's jobs, each a kernel of its own (sharing one cost the three-digit sweeps 9 % in register spills):
//   JOB_D      D maps (SW_D), and mask maps too wide for the next (SW_D, SW_CLASS3);
//   JOB_MASK4  mask maps in one SW_MASK4 sweep;
//   JOB_PAIR, JOB_PAIR4  D or mask maps of two triangles with the same r1 and r3: they share the formed A
//              operand, whose digits are what bounds a small window's kernel, and differ in D2.
enum { JOB_D, JOB_MASK4, JOB_PAIR, JOB_PAIR4, JOB_MODES };

template <int MODE>
__global__ void __launch_bounds__(NTHREADS, 1)
    ls_i8_kernel(const I8Desc *__restrict__ jobs, const LsUnit *__restrict__ units, double *__restrict__ partial,
                 int *err)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
    uint64_t *st_full = bars, *st_ready = st_full + NSTAGE_MAX, *st_empty = st_ready + NSTAGE_MAX;
    uint64_t *ab_empty = st_empty + NSTAGE_MAX;
    uint64_t *acc_full = ab_empty + NABUF_MAX, *acc_empty = acc_full + 1, *drain = acc_empty + 1;
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(drain + NMMA);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    volatile int *issued = abort_flag + 1;  // slices whose copies the TMA warp has started
    int *ngroups_s = reinterpret_cast<int *>(smem + SM_FLAGS - 4);
    uint32_t *ab_flags = reinterpret_cast<uint32_t *>(smem + SM_FLAGS);
    uint4 *sgroups = reinterpret_cast<uint4 *>(smem + SM_GROUPS);
    unsigned char *stages = smem + SM_STAGES;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const LsUnit u = units[blockIdx.x];
    const I8Desc *jd = jobs + u.job;
    const int ks = jd->ks, nclen = jd->nclen, nc = jd->nc, nc10 = jd->nc10, rs = jd->rs;
    const int c0 = u.ab * jd->AB, c1 = min(nc, c0 + jd->AB);
    const int ts = jd->ts, toff3 = ks > 1 ? 0 : ts * u.t3, toff2 = ks > 1 ? 0 : ts * u.t2;
    const int mrows = ks > 1 ? ks * rs : min(ts, nclen - toff3);
    const int ncols = ks > 1 ? nclen : min(ts, nclen - toff2);  // lag columns
    const int nwin = ks > 1 ? nclen + ks - 1 : ncols;                // window rows of D2
    const int nmma = ((nwin + 15) / 16) * 16;                        // MMA N
    // Sweeps of an item: classes 0-2 alone (SW_D); for the mask maps all four classes at once where four
    // accumulators and four four-digit buffers fit TMEM (SW_MASK4: N ≤ 96), else classes 0-2 and then class 3
    // from digits formed again (SW_D, SW_CLASS3).  One sweep with four digits takes 1.25 times a sweep with three
    // where two took 2.2 times (realisations of 24-97 channels).
    constexpr bool FOUR = MODE == JOB_MASK4 || MODE == JOB_PAIR4, PAIR = MODE == JOB_PAIR || MODE == JOB_PAIR4;
    const int sweeps = MODE == JOB_D && jd->mask ? 2 : 1;
    constexpr int abuf_cols = FOUR ? ABUF4_COLS : ABUF_COLS, ncls = FOUR ? 4 : 3, nacc = PAIR ? 2 * ncls : ncls;
    const int nabuf = min(NABUF_MAX, (TMEM_COLS - nacc * nmma) / abuf_cols);
    const int nst = jd->nst, st_bytes = jd->st_bytes;
    double *out = partial + u.tile;

    // The unit's anchor groups {D2 descriptor offset, accumulator column, MMA instruction descriptor,
    // 16 × staged row of the first channel and mask of live 8-row blocks}.  Columns whose D2 channel lies outside [0, nc) add nothing, so a group's
    // MMAs run over its own channel range only (whole 16-column steps), and a group with no channel in
    // range at all (a corner tile of a wide window) is dropped.  The entry after the last is the first
    // group over all columns, which sets the accumulators.
    if (warp == 0) {
        // S32 accumulate, signed int8 A and B, both K-major, M = 128, N / 8 in bits 17-22
        const uint32_t idesc0 = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(LS_ROWS >> 4) << 24);
        const int g0 = jd->group_off[u.ab], g1 = jd->group_off[u.ab + 1];
        int n = 0;
        for (int gb = g0; gb < g1; gb += 32) {
            const int pb = gb + lane < g1 ? jd->groups[gb + lane] : 0;
            const int w2 = pb - nc10 + toff2, w3 = pb - nc10 + toff3;  // channels of the first column and row
            const int lo = max(0, -w2), hi = min(nwin, nc - w2);
            const bool keep = gb + lane < g1 && lo < hi && (ks > 1 || (w3 < nc && w3 + mrows > 0));
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            const int at = n + __popc(m & ((1u << lane) - 1u));
            const uint32_t row = (uint32_t)(pb - c0), col = (uint32_t)(lo / 16) * 16;
            // 8-row blocks of the tile with a row whose D3 channel (and anchor) is in range, bits 16-31
            uint32_t blocks = 0;
            for (int a = 0; a < ks && pb + a < c1; ++a) {
                const int ra = max(0, -(w3 + a)), rb = min(ks > 1 ? nclen : mrows, nc - (w3 + a));  // its lags in range
                if (ra < rb)
                    blocks |= (0xffffu << ((a * rs + ra) / 8)) & (0xffffu >> (15 - (a * rs + rb - 1) / 8));
            }
            if (keep)
                sgroups[at] = make_uint4(row + col, col, idesc0 | (((hi + 15) / 16) * 2u - col / 8) << 17,
                                         16 * row | blocks << 16);
            n += __popc(m);
        }
        __syncwarp();
        if (lane == 0) {
            *ngroups_s = n;
            const uint32_t row = n > 0 ? (sgroups[0].w & 0xffffu) / 16 : 0u;
            sgroups[n] = make_uint4(row, 0u, idesc0 | (uint32_t)(nmma / 8) << 17, 0u);
        }
    }
    if (tid < NABUF_MAX) ab_flags[tid] = 0u;
    if (tid == 0) {
        for (int s = 0; s < NSTAGE_MAX; ++s) {
            mbar_init(&st_full[s], 1);
            mbar_init(&st_ready[s], 1);
            mbar_init(&st_empty[s], NFORM + NMMA);
        }
        for (int s = 0; s < NABUF_MAX; ++s) mbar_init(&ab_empty[s], NMMA);
        mbar_init(acc_full, NMMA);
        mbar_init(acc_empty, NFORM);
        for (int s = 0; s < NMMA; ++s) mbar_init(&drain[s], 1);
        *abort_flag = 0;
        *issued = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == WARP_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32((const void *)tmem_slot)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t a_col0 = tmem + nacc * nmma;
    const int ngr = *ngroups_s;
    bool ok = true;
    const long k = jd->k;
    auto nslices = [&](long b) {
        const long n = (k - b * LS_BLOCK + SLICE - 1) / SLICE;
        return (int)(n < NSLICE ? n : NSLICE);
    };

    if (ngr == 0) {
        // no anchor of the block has a channel in range: the partial tile is zero
        for (int e = tid; e < LS_ROWS * ncols; e += NTHREADS) {
            out[e] = 0.0;
            if (PAIR) out[jd->tile2 + e] = 0.0;
        }
    } else if (warp == WARP_TMA) {
        if (lane == 0) {
            const int row0_3 = c0 - nc10 + toff3, row0_2 = c0 - nc10 + toff2;
            const int st_d1 = jd->st_d1, st_d2 = jd->st_d2;
            int ns = 0, s = 0, ph = 1;
            for (long b = u.b0; b < u.b1 && ok; ++b)
                for (int sw = 0; sw < sweeps && ok; ++sw)
                    for (int sl = 0; sl < nslices(b); ++sl, ++ns) {
                        if (!mbar_wait(&st_empty[s], ph, abort_flag, err, 31)) { ok = false; break; }
                        unsigned char *st = stages + s * st_bytes;
                        mbar_expect_tx(&st_full[s], jd->tx_bytes);
                        const int x = (int)(b * LS_BLOCK + sl * SLICE);
                        tma_load_2d(st, &jd->t3, &st_full[s], x, row0_3);
                        tma_load_2d(st + st_d1, &jd->t1, &st_full[s], x, c0);
                        tma_load_4d(st + st_d2, &jd->t2, &st_full[s], 0, row0_2, x / 16, 0);
                        if (PAIR) tma_load_4d(st + jd->st_d2b, &jd->t2b, &st_full[s], 0, row0_2, x / 16, 0);
                        if (++s == nst) { s = 0; ph ^= 1; }
                    }
            *issued = ns;
        }
    } else if (warp == WARP_SCALE) {
        // scales each stage's D1 rows by 127·2^−(E1+E3) once for every row that uses them
        const int n4 = (c1 - c0) * (SLICE / 4);
        int s = 0, ph = 0;
        for (long b = u.b0; b < u.b1 && ok; ++b) {
            const float sc = ldexpf(127.f, -(jd->e1[b] + jd->e3[b]));
            for (int i = 0; i < nslices(b) * sweeps; ++i) {
                if (!mbar_wait_warp(&st_full[s], ph, abort_flag, err, 38)) { ok = false; break; }
                float4 *d1 = reinterpret_cast<float4 *>(stages + s * st_bytes + jd->st_d1);
                for (int e = lane; e < n4; e += 32) {
                    float4 v = d1[e];
                    v.x *= sc;
                    v.y *= sc;
                    v.z *= sc;
                    v.w *= sc;
                    d1[e] = v;
                }
                // these generic writes precede the TMA write that reuses the stage
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&st_ready[s]);
                if (++s == nst) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == WARP_MMA || warp == WARP_MMA2) {
        // Two warps issue the MMAs, each into accumulators of its own, so no accumulator depends on the
        // order of the two issuing threads.  One elected thread of each runs the
        // whole loop: its operands are then uniform values for the compiler, which the shuffles say for
        // those that come from memory.  The B descriptors move with the start address alone (bits 0-13,
        // 16-byte units, no carry out for shared-memory addresses).
        const bool second = warp == WARP_MMA2;
        auto uni = [](int v) { return (uint32_t)__shfl_sync(0xffffffffu, v, 0); };
        IssueState t;
        t.ngr = uni(ngr);
        t.nmma = uni(nmma);
        t.nabuf = uni(nabuf);
        t.nst = uni(nst);
        const uint32_t lbo = uni(jd->span2) * 16;               // the second 16-pixel group of a digit
        const uint64_t desc0 = smem_desc_plain(smem_u32(stages + uni(PAIR && second ? jd->st_d2b : jd->st_d2)), lbo);
        t.ddig = (2 * lbo) >> 4;
        t.desc_lo = (uint32_t)desc0;
        t.desc_hi = (uint32_t)(desc0 >> 32);
        t.stage16 = uni(st_bytes) >> 4;
        t.groups = smem_u32(sgroups);
        t.flags = smem_u32(ab_flags);
        t.bars = smem_u32(ab_empty);
        const uint32_t tmem_u = uni((int)tmem);
        t.acc = tmem_u + (second ? (PAIR ? ncls : FOUR ? 1 : 2) * t.nmma : 0);
        t.a_first = tmem_u + nacc * t.nmma;
        t.ab = t.seen = t.s = t.ph = 0;
        t.need = 4;
        if (elect_one()) {
            int ni = 0;
            for (long b = u.b0; b < u.b1 && ok; ++b)
                for (int sw = 0; sw < sweeps && ok; ++sw, ++ni) {
                    // the epilogue of the previous item has read the accumulators out
                    ok = mbar_wait(acc_empty, (ni & 1) ^ 1, abort_flag, err, 32);
                    const int nsl = nslices(b);
                    if constexpr (PAIR) {
                        if (ok)
                            ok = issue_item<false, FOUR ? SW_PAIR4 : SW_PAIR>(t, nsl, st_full, st_empty, abort_flag, err);
                    } else if constexpr (FOUR) {
                        if (ok)
                            ok = second ? issue_item<true, SW_MASK4>(t, nsl, st_full, st_empty, abort_flag, err)
                                        : issue_item<false, SW_MASK4>(t, nsl, st_full, st_empty, abort_flag, err);
                    } else if (ok && sw == 0) {
                        ok = second ? issue_item<true, SW_D>(t, nsl, st_full, st_empty, abort_flag, err)
                                    : issue_item<false, SW_D>(t, nsl, st_full, st_empty, abort_flag, err);
                    } else if (ok) {
                        ok = second ? issue_item<true, SW_CLASS3>(t, nsl, st_full, st_empty, abort_flag, err)
                                    : issue_item<false, SW_CLASS3>(t, nsl, st_full, st_empty, abort_flag, err);
                    }
                    if (ok) umma_commit_bar(smem_u32(acc_full));
                }
        }
        __syncwarp();
    } else {
        // ---- warps 0-15: form the A digits, then each block's epilogue ----
        const int q = warp & 3, ps = warp >> 2;
        const uint32_t lane_field = (uint32_t)(32 * q) << 16;
        const uint32_t stage0 = smem_u32(stages), st_d1 = (uint32_t)jd->st_d1;
        const uint32_t flag0 = smem_u32(ab_flags), group0 = smem_u32(sgroups) + 12;
        // TMEM lane 32q + 8j + i holds accumulator row 8·(4j + q) + 4·(i & 1) + i / 2.  The 8-row blocks
        // go round the four quarters of the lanes, so that the blocks an anchor's window leaves empty (a
        // quarter to half of them) come off all four SM partitions alike; and the two lanes that one
        // eight-thread phase of a shared load reads (below) hold rows four apart, whose 128-byte swizzles
        // differ in the half of the row, so the phase is free of bank conflicts.
        auto row_of = [](int L) { return 8 * ((L >> 1 & 12) | L >> 5) + ((L & 1) << 2 | (L >> 1 & 3)); };
        // The 16 formers are four sets of four: set ps forms every fourth anchor group of the
        // item's sequence (slices, groups within a slice), and within a set warp q fills TMEM lanes
        // 32q .. 32q+31 of the group's A buffer with all 32 pixels, so the per-group work
        // (addresses, waits, TMEM hand-off) is spread over 32 pixels.  A thread forms four rows
        // (lanes t/4 + 8j, one 8-row block each) of two 4-pixel words each (words t%4 and 4 + t%4), so its
        // two D1 words serve every row of an anchor slot.  A block without a row in range stores zero
        // digits without the arithmetic.  The first lanes' digits are formed before the buffer is waited for.  Rows past a slot's lags hold digits of whatever was read: their
        // accumulator rows are never read out.  D3 channels outside [0, nc) arrive as zero rows from the TMA
        // bounds fill.
        const uint32_t c4 = (lane & 3) << 4;
        // 16 × (D3 row less the group's first row) and 16 × anchor slot of the thread's rows
        uint32_t roff[4], slot[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = row_of(32 * q + 8 * j + (lane >> 2));
            slot[j] = ks > 1 ? 16 * (r / rs) : 0;
            roff[j] = ks > 1 ? slot[j] + 16 * (r % rs) : 16 * r;
        }
        int s = 0, ph = 0, ni = 0, ab = ps % nabuf;
        int g = ps;               // next group of this set, counted from the current slice's first
        uint32_t abph = 1 ^ (ps / nabuf & 1);  // parity to wait for on ab_empty[ab]
        auto form_slice = [&](auto ndc, auto nsc, auto onec) {
            constexpr int ND = decltype(ndc)::value, NS = decltype(nsc)::value;
            constexpr int D0 = ND - NS;                   // ND digits formed, the last NS stored
            constexpr bool ONE = decltype(onec)::value;   // one anchor slot
            const uint32_t st = stage0 + (uint32_t)(s * st_bytes);
            for (; g < ngr; g += NSET) {
                uint32_t word;
                asm volatile("ld.shared.b32 %0, [%1];" : "=r"(word) : "r"(group0 + 16 * g));
                const uint32_t row = word & 0xffffu, blocks = word >> (16 + q);  // 16 × first row, live blocks
                const uint32_t col = a_col0 + lane_field + ab * (NS == 4 ? ABUF4_COLS : ABUF_COLS);
                // 16-byte chunk c of a 128-byte-swizzled row lies at chunk c ^ (row & 7)
                auto chunk_of = [&](uint32_t r16) { return st + 8 * r16 + ((r16 & 0x70u) ^ c4); };
                float4 v1[2];
                uint32_t a3[2] = {0, 0};  // words t%4 and 4 + t%4 of the D3 row
                if constexpr (ONE) {
                    a3[0] = chunk_of(row + roff[0]);
                    a3[1] = a3[0] ^ 64;
                    const uint32_t a1 = st_d1 + chunk_of(row);
                    v1[0] = lds128(a1);
                    v1[1] = lds128(a1 ^ 64);
                }
#pragma unroll
                for (int half = 0; half < 2; ++half) {  // TMEM lanes 16·half .. +15 of the warp's 32
                    uint32_t w[NS][4];  // zeros where a block is dead: one initialisation beats an else branch each
#pragma unroll
                    for (int dd = 0; dd < NS; ++dd)
#pragma unroll
                        for (int e = 0; e < 4; ++e) w[dd][e] = 0u;
#pragma unroll
                    for (int jj = 0; jj < 2; ++jj) {
                        const int j = 2 * half + jj;
                        if (blocks >> (4 * j) & 1) {
                            if constexpr (!ONE) {
                                a3[0] = chunk_of(row + roff[j]);
                                a3[1] = a3[0] ^ 64;
                                const uint32_t a1 = st_d1 + chunk_of(row + slot[j]);
                                v1[0] = lds128(a1);
                                v1[1] = lds128(a1 ^ 64);
                            }
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                const float4 x = lds128(a3[h] + (ONE ? 4096 * j : 0));
                                float2 ya[4], yb[4];
                                digits254x2<ND>(make_float2(v1[h].x, v1[h].y), make_float2(x.x, x.y), ya);
                                digits254x2<ND>(make_float2(v1[h].z, v1[h].w), make_float2(x.z, x.w), yb);
#pragma unroll
                                for (int dd = 0; dd < NS; ++dd)
                                    w[dd][2 * h + jj] =
                                        pack_low_bytes(ya[dd + D0].x, ya[dd + D0].y, yb[dd + D0].x, yb[dd + D0].y);
                            }
                        }
                    }
                    if (half == 0) {
                        if (!mbar_wait_conv(&ab_empty[ab], abph, abort_flag, err, 36)) { ok = false; return; }
                        fence_after();
                    }
                    const uint32_t tcol = col + ((uint32_t)(16 * half) << 16);
                    tmem_st16x16(tcol, w[0], w[1]);
                    if constexpr (NS == 4) tmem_st16x16(tcol + 16, w[2], w[3]);
                    else tmem_st16x8(tcol + 16, w[2]);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                fence_before();
                __syncwarp();
                if (lane == 0) count_add(flag0 + ab * 4);
                ab += NSET;
                while (ab >= nabuf) { ab -= nabuf; abph ^= 1; }
            }
            g -= ngr;
        };
        for (long b = u.b0; b < u.b1 && ok; ++b) {
            const int E13 = jd->e1[b] + jd->e3[b];
            for (int sw = 0; sw < sweeps && ok; ++sw, ++ni) {
                for (int sl = 0; sl < nslices(b); ++sl) {
                    if (!mbar_wait_conv(&st_ready[s], ph, abort_flag, err, 35)) { ok = false; break; }
                    auto form = [&](auto onec) {
                        using std::integral_constant;
                        if constexpr (FOUR) form_slice(integral_constant<int, 4>(), integral_constant<int, 4>(), onec);
                        else if (sw == 0) form_slice(integral_constant<int, 3>(), integral_constant<int, 3>(), onec);
                        else form_slice(integral_constant<int, 4>(), integral_constant<int, 3>(), onec);
                    };
                    if (ks == 1) form(std::true_type());
                    else form(std::false_type());
                    if (!ok) break;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&st_empty[s]);
                    if (++s == nst) { s = 0; ph ^= 1; }
                }
                if (!ok) break;
                // ---- epilogue: int32 class accumulators → FP64, added into the unit's partial tile ----
                if (!mbar_wait_warp(acc_full, ni & 1, abort_flag, err, 37)) { ok = false; break; }
                fence_after();
                const bool first = b == u.b0 && sw == 0;
                // this lane's accumulator row and anchor slot
                const int r = row_of(32 * q + lane), a = ks > 1 ? r / rs : 0;
                const bool row_ok = ks > 1 ? r < mrows && r - a * rs < nclen : r < mrows;
                for (int tri = 0; tri < (PAIR ? 2 : 1); ++tri) {
                    const int E = E13 + (tri ? jd->e2b : jd->e2)[b];
                    // one unit of the last class in the sums: 127^−2·254^−2 (classes 0-2) or 127^−2·254^−3
                    const double scale = ldexp(1.0, E) * (sw == 0 && !FOUR ? 1.0 / (16129.0 * 64516.0)
                                                                           : 1.0 / (16129.0 * 16387064.0));
                    const uint32_t acc = tmem + lane_field + tri * ncls * nmma;
                    double *outt = out + (tri ? jd->tile2 : 0);
                    for (int cb = 8 * ps; cb < nmma; cb += 8 * NSET) {
                        uint32_t v0[8], v1[8], v2[8], v3[8];
                        tmem_ld8(acc + cb, v0);
                        if (sw == 0) tmem_ld8(acc + nmma + cb, v1);
                        tmem_ld8(acc + 2 * nmma + cb, v2);
                        if (FOUR) tmem_ld8(acc + 3 * nmma + cb, v3);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        if (!row_ok) continue;
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const int colx = cb + e - a;  // slot a of a packed tile: lag column = column − a
                            if (colx < 0 || colx >= ncols) continue;
                            long long V = (long long)(int)v0[e] + (long long)(int)v2[e];  // class 3 alone, in two parts
                            if (sw == 0)
                                V = (long long)(int)v0[e] * 64516LL + (long long)(int)v1[e] * 254LL + (long long)(int)v2[e];
                            if (FOUR) V = V * 254LL + (long long)(int)v3[e];
                            double *o = outt + (long)colx * LS_ROWS + r;
                            const double val = (double)V * scale;
                            *o = first ? val : *o + val;
                        }
                    }
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty);
            }
        }
    }

    fence_before();
    __syncthreads();
    if (*abort_flag) {
        // A wait gave up.  Copies and MMAs still in flight, those of a role that had finished its own loop
        // included, have to end before the shared memory and TMEM that they use go away.
        if (warp == WARP_TMA && lane == 0) {
            const int n = *issued, ring = jd->nst;
            for (int q = max(0, n - ring); q < n; ++q)
                for (long long i = 0; i < WAIT_LIMIT && !mbar_try_wait(&st_full[q % ring], ((q / ring) & 1)); ++i)
                    __nanosleep(100);
        } else if ((warp == WARP_MMA || warp == WARP_MMA2) && elect_one()) {  // the thread that issued them
            uint64_t *dr = drain + (warp == WARP_MMA2 ? 1 : 0);
            umma_commit_bar(smem_u32(dr));
            for (long long i = 0; i < WAIT_LIMIT && !mbar_try_wait(dr, 0); ++i) __nanosleep(100);
        }
        __syncthreads();
    }
    if (warp == WARP_MMA) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

typedef CUresult (*EncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int encode(amber_cuda_ctx *c, CUtensorMap *m, CUtensorMapDataType dt, int rank, const void *base,
           const cuuint64_t *dims, const cuuint64_t *strides, const cuuint32_t *box, CUtensorMapSwizzle sw)
{
    static EncodeTiled enc = nullptr;
    if (!enc) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn)
            return fail(c, AMBER_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
        enc = (EncodeTiled)fn;
    }
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(m, dt, (cuuint32_t)rank, (void *)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(c, AMBER_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return AMBER_OK;
}

}  // namespace

size_t contract_partial_cap(const amber_cuda_ctx *c)
{
    return std::max<size_t>((size_t)512 << 20, std::min<size_t>((size_t)8 << 30, c->budget / 8));
}

int contract_i8_jobs(amber_cuda_ctx *c, const std::vector<I8Job> &jobs)
{
    int rc;
    if (jobs.empty()) return AMBER_OK;
    if ((rc = ensure(c, c->misc, 256, "error flag"))) return rc;
    int *d_err = (int *)c->misc.p;
    if (!c->i8_open && (rc = cuda_check(c, cudaMemsetAsync(d_err, 0, sizeof(int), c->stream), "error flag"))) return rc;
    c->i8_open = true;
    const size_t pcap = contract_partial_cap(c);
    const CUtensorMapDataType u8 = CU_TENSOR_MAP_DATA_TYPE_UINT8, f32 = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    static void (*const KERNELS[JOB_MODES])(const I8Desc *, const LsUnit *, double *, int *) = {
        ls_i8_kernel<JOB_D>, ls_i8_kernel<JOB_MASK4>, ls_i8_kernel<JOB_PAIR>, ls_i8_kernel<JOB_PAIR4>};
    for (auto kernel : KERNELS)
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
    // Items: a job, or two jobs that share D1 and D3 and fit a pair (how jobs are paired changes no result:
    // every sum of digits is exact).  A pair has half the units of its two jobs, each with 1.3 times the work, so
    // jobs are paired where they would make more than three units an SM apart: D maps of a 59-channel
    // realisation 10.4 → 8.7 ms, half of them in pairs.
    long apart = 0;
    for (const I8Job &jb : jobs) apart += ls_shape(jb.nc, jb.nc10, jb.k, c->num_sms, MIN_GROUPS).units();
    const bool pairing = apart > 3L * c->num_sms;
    struct Item {
        size_t a, b;  // b = a: no second job
        int mode;
    };
    std::vector<Item> items;
    {
        std::map<std::tuple<const float *, const float *, bool, const std::vector<int> *>, size_t> open;  // awaiting a partner
        for (size_t i = 0; i < jobs.size(); ++i) {
            const I8Job &jb = jobs[i];
            const int nmma = ls_shape(jb.nc, jb.nc10, jb.k, c->num_sms, MIN_GROUPS).cols(0);
            const int mode = jb.mask_pass && mask4_fits(nmma) ? JOB_MASK4 : JOB_D;
            if (pairing && pair_fits(jb.mask_pass, nmma)) {
                const auto key = std::make_tuple(jb.m1.f32, jb.m3.f32, jb.mask_pass, jb.weight);
                const auto it = open.find(key);
                if (it != open.end() && jobs[items[it->second].a].k == jb.k && jobs[items[it->second].a].nc10 == jb.nc10) {
                    items[it->second].b = i;
                    items[it->second].mode = jb.mask_pass ? JOB_PAIR4 : JOB_PAIR;
                    open.erase(it);
                    continue;
                }
                open[key] = items.size();
            }
            items.push_back(Item{i, i, mode});
        }
    }
    size_t j0 = 0;
    while (j0 < items.size()) {
        // plan as many items as their partial tiles allow in one upload
        std::vector<LsJobPlan> plans;
        long used = 0;  // doubles of partial tiles
        size_t j1 = j0;
        for (; j1 < items.size(); ++j1) {
            const I8Job &jb = jobs[items[j1].a];
            LsJobPlan p;
            ls_plan_job(p, jb.nc, jb.nc10, jb.k, *jb.weight, c->num_sms, MIN_GROUPS, ls_force_bpu(c->chunk_px));
            const long need = p.s.units() * p.s.tile() * (items[j1].b != items[j1].a ? 2 : 1);
            if (j1 > j0 && sizeof(double) * (size_t)(used + need) > pcap) break;
            p.unit_base = used;
            used += need;
            plans.push_back(std::move(p));
        }
        // the units of each mode: a launch each
        std::vector<LsUnit> units;
        size_t begin[JOB_MODES + 1];
        for (int mode = 0; mode < JOB_MODES; ++mode) {
            begin[mode] = units.size();
            for (size_t i = 0; i < plans.size(); ++i) {
                const size_t first = units.size();
                if (items[j0 + i].mode != mode) continue;
                ls_units(plans[i], (int)i, units);
                if (mode == JOB_D && jobs[items[j0 + i].a].mask_pass)
                    for (size_t q = first; q < units.size(); ++q) units[q].work *= 1.6;  // the class-3 sweep
            }
            // largest units first, so that the small ones fill the tail of the launch
            std::stable_sort(units.begin() + begin[mode], units.end(),
                             [](const LsUnit &a, const LsUnit &b) { return a.work > b.work; });
        }
        begin[JOB_MODES] = units.size();
        size_t ngroups = 0, noff = 0;
        for (const LsJobPlan &p : plans) {
            ngroups += p.groups.size();
            noff += p.group_off.size();
        }
        const size_t desc_b = sizeof(I8Desc) * plans.size(), unit_b = sizeof(LsUnit) * units.size();
        const size_t off_u = (desc_b + 255) / 256 * 256, off_g = off_u + (unit_b + 255) / 256 * 256;
        const size_t off_o = off_g + (sizeof(int) * ngroups + 255) / 256 * 256;
        const size_t stage_b = off_o + sizeof(int) * noff;
        if ((rc = ensure(c, c->partial, sizeof(double) * (size_t)used, "partial lag tiles"))) return rc;
        if ((rc = ensure(c, c->jobdesc, stage_b, "job list"))) return rc;
        void *staging;
        if ((rc = job_stage(c, stage_b, &staging))) return rc;
        char *h = (char *)staging, *d = (char *)c->jobdesc.p;
        I8Desc *hd = (I8Desc *)h;
        int *hg = (int *)(h + off_g), *ho = (int *)(h + off_o);
        std::vector<LsReduceJob> red;
        size_t gpos = 0, opos = 0;
        for (size_t i = 0; i < plans.size(); ++i) {
            const Item &item = items[j0 + i];
            const I8Job &jb = jobs[item.a], &jb2 = jobs[item.b];
            const bool pair = item.b != item.a;
            const LsJobPlan &p = plans[i];
            const LsShape &s = p.s;
            I8Desc &x = hd[i];
            memset(&x, 0, sizeof(x));
            x.span3 = s.AB + (s.k > 1 ? s.nclen : s.rows(0)) - 1;
            x.span2 = s.AB + s.cols(0) - 1;
            const cuuint64_t fdims[2] = {(cuuint64_t)jb.k, (cuuint64_t)jb.nc};
            const cuuint64_t fstr[1] = {(cuuint64_t)jb.kp * 4};
            const cuuint32_t box3[2] = {SLICE, (cuuint32_t)x.span3}, box1[2] = {SLICE, (cuuint32_t)s.AB};
            if ((rc = encode(c, &x.t3, f32, 2, jb.m3.f32, fdims, fstr, box3, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
            if ((rc = encode(c, &x.t1, f32, 2, jb.m1.f32, fdims, fstr, box1, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
            const cuuint64_t ddims[4] = {16, (cuuint64_t)jb.nc, (cuuint64_t)(jb.kp / 16), 3};
            const cuuint64_t dstr[3] = {16, (cuuint64_t)jb.nc * 16, (cuuint64_t)jb.nc * jb.kp};
            const cuuint32_t box2[4] = {16, (cuuint32_t)x.span2, 2, 3};
            if ((rc = encode(c, &x.t2, u8, 4, jb.m2.dig, ddims, dstr, box2, CU_TENSOR_MAP_SWIZZLE_NONE))) return rc;
            if (pair && (rc = encode(c, &x.t2b, u8, 4, jb2.m2.dig, ddims, dstr, box2, CU_TENSOR_MAP_SWIZZLE_NONE)))
                return rc;
            x.e1 = jb.m1.bexp;
            x.e2 = jb.m2.bexp;
            x.e2b = jb2.m2.bexp;
            x.tile2 = p.s.units() * p.s.tile();
            x.e3 = jb.m3.bexp;
            x.groups = (const int *)(d + off_g) + gpos;
            x.group_off = (const int *)(d + off_o) + opos;
            x.k = jb.k;
            x.nc = jb.nc;
            x.nc10 = jb.nc10;
            x.nclen = s.nclen;
            x.ks = s.k;
            x.rs = s.rs;
            x.AB = s.AB;
            x.ts = s.ts;
            x.mask = jb.mask_pass ? 1 : 0;
            const int d2_bytes = 3 * 2 * x.span2 * 16;
            x.tx_bytes = (uint32_t)(x.span3 * 128 + s.AB * 128 + (pair ? 2 : 1) * d2_bytes);
            // whole 8-row swizzle atoms for the fp32 rows; every part starts on a 1024-byte boundary.  The
            // formers read a slot's whole 8-row blocks (all LS_ROWS rows with one slot) from every anchor on,
            // past the tile's rows too.
            x.st_d1 = (s.AB - 1 + (s.k > 1 ? s.rs : LS_ROWS) + 7) / 8 * 1024;
            x.st_d2 = x.st_d1 + (s.AB + 7) / 8 * 1024;
            x.st_d2b = x.st_d2 + (d2_bytes + 1023) / 1024 * 1024;
            x.st_bytes = pair ? x.st_d2b + (d2_bytes + 1023) / 1024 * 1024 : x.st_d2b;
            x.nst = std::min(NSTAGE_MAX, SMEM_STAGES / x.st_bytes);
            std::copy(p.groups.begin(), p.groups.end(), hg + gpos);
            for (size_t q = 0; q < p.group_off.size(); ++q) ho[opos + q] = p.group_off[q];
            gpos += p.groups.size();
            opos += p.group_off.size();
            for (int q = 0; q < (pair ? 2 : 1); ++q)
                red.push_back(LsReduceJob{(const double *)c->partial.p + p.unit_base + q * x.tile2,
                                          q ? jb2.lag_out : jb.lag_out, s.nclen, s.k, s.rs, s.T, s.ts, s.nab, s.V,
                                          s.tile()});
        }
        std::copy(units.begin(), units.end(), (LsUnit *)(h + off_u));
        if ((rc = cuda_check(c, cudaMemcpyAsync(d, h, stage_b, cudaMemcpyHostToDevice, c->stream), "job list upload")))
            return rc;
        if ((rc = job_stage_sent(c))) return rc;
        phase_begin(c, 1);
        const LsUnit *du = (const LsUnit *)(d + off_u);
        for (int mode = 0; mode < JOB_MODES; ++mode) {
            const unsigned n = (unsigned)(begin[mode + 1] - begin[mode]);
            if (n == 0) continue;
            KERNELS[mode]<<<n, NTHREADS, SMEM_BYTES, c->stream>>>((const I8Desc *)d, du + begin[mode],
                                                                  (double *)c->partial.p, d_err);
            c->launches += 1;
            c->contractions += 1;
        }
        phase_end(c);
        if ((rc = cuda_check(c, cudaGetLastError(), "ls_i8_kernel launch"))) return rc;
        if ((rc = ls_reduce(c, red))) return rc;
        j0 = j1;
    }
    return AMBER_OK;
}

int contract_i8_finish(amber_cuda_ctx *c)
{
    if (!c->i8_open) return AMBER_OK;
    c->i8_open = false;
    int rc, herr = 0;
    if ((rc = cuda_check(c, cudaMemcpyAsync(&herr, c->misc.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream),
                         "error flag read")))
        return rc;
    if ((rc = cuda_check(c, cudaStreamSynchronize(c->stream), "contract_i8"))) return rc;
    if (herr) return fail(c, AMBER_ERR_TIMEOUT, "int8 tensor-core contraction: a pipeline wait gave up (site %d)", herr);
    return AMBER_OK;
}

}  // namespace amber
