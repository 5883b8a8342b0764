// Ring filter + unnormalised 2D c2r, fused and batched over (ring × channel).
//
// Replaces Dfg/Ifg + fill_s2d_float/fill_s2I (4_fbe/amber_funcs.c:573-621,
// 967-1010, 1109-1131) and the mask transform inside calCR (389-437).  For a
// ring [lo, hi) the reference scatters grid cell (ia mod N1, j) into bin
// (ia mod Ng1, j) of a zeroed Ng1 × (Ng1/2+1) half-plane for ia ∈ (−Ng1/2,
// Ng1/2], j < Ng1/3, lo ≤ √(ia²+j²) < hi, √ > 0, then runs
// fftw_plan_dft_c2r_2d.  Only |ia|, j < hi are ever non-zero, so instead of a
// full FFT of a mostly-empty plane we evaluate the transform directly on the
// non-zero support ("pruned DFT"), which is exact for any Ng1 — the map sides
// here have large prime factors (740 = 4·5·37, 1460 = 4·5·73):
//
//   pass 1 (axis 0, per column j < J):  Y[n0][j] = Σ_ia X[ia][j] · e^{+2πi·ia·n0/Ng1}
//   pass 2 (axis 1, c2r):               D[n0][n1] = Re Y[n0][0] + 2 Σ_{j≥1} Re(Y[n0][j] · e^{+2πi·j·n1/Ng1})
//
// The c2r convention — complex DFT along axis 0, then a 1D c2r along axis 1
// that ignores Im of bin 0 — is what a rank-2 c2r does with the non-Hermitian
// j = 0 column the ring scatter produces; the Nyquist bin j = Ng1/2 is never
// filled because j < Ng1/3.
//
// Both passes sum even and odd terms apart, so that one point of a quarter of the axis gives four (Ng1 is
// even), and take the twiddles e^{2πik/Ng1} from a table in shared memory at indices that advance
// incrementally (k += n mod Ng1).  Pass 1 stages one column of the spectrum for C channels and runs on the FP64
// cores, lanes over channels; pass 2 is a GEMM on the FP64 tensor cores over (pixel) × (row, channel).
// All arithmetic is FP64.
#include <cuda_bf16.h>
#include <limits.h>
#include <math.h>

#include <algorithm>
#include <vector>

#include "lagspace.cuh"

namespace amber {

namespace {

constexpr int kThreads = 256;

// Rows of column j that fall inside ring [lo, hi) for an ng-point output grid.
__device__ __forceinline__ bool in_ring(long ia, long j, double lo, double hi)
{
    double uu = sqrt(1.0 * (double)(ia * ia + j * j));
    return uu >= lo && uu < hi && uu > 0.0;
}

// Ring edges and column counts of the slots one launch builds, passed by value: no upload and no
// stream synchronisation before the launch, so the host can queue the next request's maps while
// these run.  A batch with more slots runs as several launches.
constexpr int RING_META_MAX = 96;
struct RingMeta {
    double lo[RING_META_MAX], hi[RING_META_MAX];
    int jc[RING_META_MAX];
};

template <int C>
__global__ void __launch_bounds__(kThreads) ring_cols_kernel(const void *__restrict__ src, int src_complex, long n1,
                                                              long nc, long chan_base, long nch, long ng,
                                                              const RingMeta meta, int jmax,
                                                              const double2 *__restrict__ tw_g,
                                                              double2 *__restrict__ Y, int rowcap)
{
    extern __shared__ double2 smem[];
    double2 *tw = smem;                        // ng
    double2 *xs = tw + ng;                     // rowcap × C
    int *ias = reinterpret_cast<int *>(xs + (size_t)rowcap * C);  // rowcap
    __shared__ int warp_cnt[kThreads / 32];
    __shared__ int nrows_s;

    const int j = blockIdx.x, s = blockIdx.y;
    const long q0 = (long)blockIdx.z * C;
    if (j >= meta.jc[s]) return;
    const double lo = meta.lo[s], hi = meta.hi[s];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long h1 = n1 / 2 + 1;

    for (long i = tid; i < ng; i += kThreads) tw[i] = tw_g[i];

    // Ordered compaction of the ring's rows in this column: the even ones, then the odd ones.
    const long A = (long)ceil(hi) - 1;
    const long ia_min = max(-A, -ng / 2 + 1), ia_max = min(A, ng / 2);
    if (tid == 0) nrows_s = 0;
    __syncthreads();
    int neven = 0;
    for (int p = 0; p < 2; ++p) {
        for (long base = ia_min + ((ia_min ^ p) & 1); base <= ia_max; base += 2 * kThreads) {
            long ia = base + 2 * tid;
            bool hit = ia <= ia_max && in_ring(ia, j, lo, hi);
            unsigned m = __ballot_sync(0xffffffffu, hit);
            if (lane == 0) warp_cnt[warp] = __popc(m);
            __syncthreads();
            int off = nrows_s;
            for (int w = 0; w < warp; ++w) off += warp_cnt[w];
            off += __popc(m & ((1u << lane) - 1u));
            if (hit && off < rowcap) ias[off] = (int)ia;
            __syncthreads();
            if (tid == 0) {
                int tot = 0;
                for (int w = 0; w < kThreads / 32; ++w) tot += warp_cnt[w];
                nrows_s += tot;
            }
            __syncthreads();
        }
        if (p == 0) neven = min(nrows_s, rowcap);
    }
    const int nrows = min(nrows_s, rowcap);

    // Gather the ring's cells for C channels (channel-innermost: coalesced).
    for (int e = tid; e < nrows * C; e += kThreads) {
        int r = e / C, q = e % C;
        long ia = ias[r];
        long iN = ia < 0 ? n1 + ia : ia;
        long cell = iN * h1 + j;
        double2 v = make_double2(0.0, 0.0);
        if (q0 + q < nch) {
            long ch = chan_base + q0 + q;
            if (src_complex)
                v = reinterpret_cast<const double2 *>(src)[cell * nc + ch];
            else
                v.x = reinterpret_cast<const double *>(src)[cell * nc + ch];
        }
        xs[r * C + q] = v;
    }
    __syncthreads();

    // Y[n0][j] for this thread's channel q, R rows n0 ≤ Ng/4 at a time.  With the sums of Re X·cos (a), Im X·sin
    // (b), Re X·sin (c) and Im X·cos (d) over the even and over the odd ia, one n0 gives four output rows (the
    // sines change sign at −n0 and h − n0, the odd terms at h ± n0; h = Ng/2, Ng even): one FMA per output row
    // and ia in place of four.  Bound by the shared twiddle loads beside the FP64 FMAs; fourteen rings of 128
    // channels on 740 × 740 pixels 2.9 → 0.65 ms, three of 354 × 354 (D and mask maps) 0.41 → 0.12 ms.
    constexpr int G = 32 / C;  // n0 groups per warp
    constexpr int R = 4;
    const int q = lane % C, g = lane / C;
    const int ngroups = (kThreads / 32) * G, h = (int)(ng / 2), nmax = h / 2;
    const int ngi = (int)ng;
    for (int nb = warp * G + g; nb * R <= nmax; nb += ngroups) {
        int n0[R];
        double4 sum[2][R];  // even, odd: (a, b, c, d)
#pragma unroll
        for (int r = 0; r < R; ++r) n0[r] = min(nb * R + r, nmax);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            int idx[R], step[R], prev = INT_MIN;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                sum[p][r] = make_double4(0.0, 0.0, 0.0, 0.0);
                step[r] = 2 * n0[r] >= ngi ? 2 * n0[r] - ngi : 2 * n0[r];
                idx[r] = 0;
            }
            for (int row = p ? neven : 0; row < (p ? nrows : neven); ++row) {
                const int ia = ias[row];
                if (ia != prev + 2) {
                    const long iam = ia < 0 ? ia + ngi : ia;
#pragma unroll
                    for (int r = 0; r < R; ++r) idx[r] = (int)((iam * n0[r]) % ngi);
                } else {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const int t = idx[r] + step[r];
                        idx[r] = t >= ngi ? t - ngi : t;
                    }
                }
                prev = ia;
                const double2 x = xs[row * C + q];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const double2 w = tw[idx[r]];
                    sum[p][r].x = fma(x.x, w.x, sum[p][r].x);
                    sum[p][r].y = fma(x.y, w.y, sum[p][r].y);
                    sum[p][r].z = fma(x.x, w.y, sum[p][r].z);
                    sum[p][r].w = fma(x.y, w.x, sum[p][r].w);
                }
            }
        }
        if (q0 + q < nch) {
            double2 *out = Y + ((long)s * ng * jmax + j) * nch + q0 + q;
            auto put = [&](int n, double re, double im) { out[(long)n * jmax * nch] = make_double2(re, im); };
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int n = nb * R + r;
                if (n > nmax) continue;
                const double4 e = sum[0][r], o = sum[1][r];
                const double a = e.x + o.x, b = e.y + o.y, c = e.z + o.z, d = e.w + o.w;
                const double am = e.x - o.x, bm = e.y - o.y, cm = e.z - o.z, dm = e.w - o.w;
                put(n, a - b, c + d);
                if (n > 0) put(ngi - n, a + b, d - c);
                if (2 * n < h) {
                    put(h - n, am + bm, dm - cm);
                    if (n > 0) put(h + n, am - bm, cm + dm);
                }
            }
        }
    }
}

__device__ __forceinline__ uint16_t bf16_bits(float f)
{
    __nv_bfloat16 b = __float2bfloat16_rn(f);
    return *reinterpret_cast<uint16_t *>(&b);
}

// D(16×8) += A(16×8) · B(8×8), FP64.  Fragments (g = lane / 4, t = lane % 4): A {(g, t), (g+8, t),
// (g, t+4), (g+8, t+4)}, B {(t, g), (t+4, g)}, C {(g, 2t), (g, 2t+1), (g+8, 2t), (g+8, 2t+1)}.
__device__ __forceinline__ void dmma(double (&c)[4], const double (&a)[4], double b0, double b1)
{
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                 : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

// Pass 2 as an FP64 GEMM over (pixel x ≤ Ng/4) × (column = output row n0, channel) with j as the
// contraction: with C_e, C_o the sums of Re Y·cos over even and odd j and S_e, S_o those of Im Y·sin, one
// quarter of the row gives the whole row (h = Ng/2; Ng is even):
//     D[x] = C_e + C_o − S_e − S_o,   D[Ng − x] = C_e + C_o + S_e + S_o,
//     D[h − x] = C_e − C_o + S_e − S_o,   D[h + x] = C_e − C_o − S_e + S_o,
// i.e. half an FMA per pixel and j.  A CTA holds RC columns' spectrum rows in shared memory; two warps share
// every fourth tile of 16 x, half the columns each.  The A fragments (cos, sin of j·x) come from the twiddle table, at indices that
// advance by 16·x mod Ng per step of 16 j, and serve RN column tiles.  Bound by the FP64 pipe for wide
// rings and by the map stores for narrow ones.  On the FP64 cores with two FMAs per pixel and j, each fed by a
// shared load of its own, fourteen rings of 128 channels on 740 × 740 pixels took 13.6 ms; now 3.8 ms.
constexpr int RC = 32;       // columns per CTA
constexpr int RS = RC + 1;   // their stride in shared memory: odd, so that a fragment load is conflict-free
constexpr int RN = RC / 16;  // column tiles (of 8) per warp
constexpr int RROWS_THREADS = 256;
constexpr int RX = 16 * (RROWS_THREADS / 64);  // x per round of the CTA's warps

__global__ void __launch_bounds__(RROWS_THREADS, 2) ring_rows_kernel(const double2 *__restrict__ Y, int ng, int jmax,
                                                                      const RingMeta meta, long nch,
                                                                      const double2 *__restrict__ tw_g, long kp, int jstage,
                                                                      double *__restrict__ out_f64,
                                                                      uint16_t *__restrict__ out_hi,
                                                                      uint16_t *__restrict__ out_lo,
                                                                      float *__restrict__ out_f32,
                                                                      const int *__restrict__ weight)
{
    extern __shared__ double2 smem[];
    double2 *tw = smem;       // ng
    double2 *ys = tw + ng;    // [jstage][RS]: all of the ring's J, or a run of them at a time
    const int s = blockIdx.y;
    const long col0 = (long)blockIdx.x * RC, ncol = (long)ng * nch;
    const int J = meta.jc[s], steps = (J + 15) / 16;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < ng; i += RROWS_THREADS) tw[i] = tw_g[i];
    // this thread's column of the staged spectrum (RROWS_THREADS is a multiple of RC)
    const int sc = tid % RC;
    const long scol = col0 + sc;
    const double2 *src = Y + (((long)s * ng + scol / nch) * jmax) * nch + scol % nch;
    auto stage = [&](int j0) {
        const int n = min(jstage, 16 * steps - j0);
        for (int j = tid / RC; j < n; j += RROWS_THREADS / RC) {
            double2 v = make_double2(0.0, 0.0);
            if (j0 + j < J && scol < ncol) v = src[(long)(j0 + j) * nch];
            if (j0 + j == 0) v.y = 0.0;  // c2r ignores Im of the DC bin
            else { v.x *= 2.0; v.y *= 2.0; }
            ys[j * RS + sc] = v;
        }
    };
    stage(0);
    __syncthreads();

    const int g = lane >> 2, t = lane & 3;
    const int h = ng / 2, xmax = h / 2, nb = (warp & 1) * 8 * RN;  // first column of this warp
    // the columns this thread stores: row origin (−1: past the last column) and channel multiplicity (the
    // mixed path's fp32 maps carry it, 0 for flagged channels)
    long at[2 * RN];
    double wq[2 * RN];
#pragma unroll
    for (int i = 0; i < 2 * RN; ++i) {
        const unsigned col = (unsigned)(col0 + nb + 8 * (i / 2) + 2 * t + i % 2);
        const unsigned n0 = col / (unsigned)nch, ch = col % (unsigned)nch;
        at[i] = col < (unsigned)ncol ? ((long)s * nch + ch) * kp + (long)n0 * ng : -1;
        wq[i] = weight && col < (unsigned)ncol ? (double)weight[ch] : 1.0;
    }
    for (int xg = 0; xg <= xmax; xg += RX) {
        const int x0 = xg + 16 * (warp >> 1);
        // twiddle indices of j = 2t and 2t + 8 for the lane's two x (clamped: rows past xmax are not stored)
        const int xa[2] = {min(x0 + g, xmax), min(x0 + g + 8, xmax)};
        int idx[2][2], d16[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            idx[i][0] = (2 * t * xa[i]) % ng;
            idx[i][1] = ((2 * t + 8) * xa[i]) % ng;
            d16[i] = (16 * xa[i]) % ng;
        }
        double ce[RN][4], co[RN][4], se[RN][4], so[RN][4];
#pragma unroll
        for (int n = 0; n < RN; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) ce[n][e] = co[n][e] = se[n][e] = so[n][e] = 0.0;
        const double2 *yj = ys + 2 * t * RS + nb + g;
        for (int st = 0, left = jstage / 16; st < steps; ++st, yj += 16 * RS) {
            if (left-- == 0) {  // a ring too wide for one stage: its next run of j
                __syncthreads();
                stage(16 * st);
                __syncthreads();
                left = jstage / 16 - 1;
                yj = ys + 2 * t * RS + nb + g;
            }
            double ac[4], as[4], bc[4], bs[4];  // cos, sin at even and at odd j
#pragma unroll
            for (int kk = 0; kk < 2; ++kk)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const double2 w = tw[idx[i][kk]];
                    int o = idx[i][kk] + xa[i];
                    o = o >= ng ? o - ng : o;
                    const double2 v = tw[o];
                    ac[2 * kk + i] = w.x;
                    as[2 * kk + i] = w.y;
                    bc[2 * kk + i] = v.x;
                    bs[2 * kk + i] = v.y;
                    o = idx[i][kk] + d16[i];
                    idx[i][kk] = o >= ng ? o - ng : o;
                }
#pragma unroll
            for (int n = 0; n < RN; ++n) {
                const double2 e0 = yj[8 * n], e1 = yj[8 * RS + 8 * n];
                const double2 o0 = yj[RS + 8 * n], o1 = yj[9 * RS + 8 * n];
                dmma(ce[n], ac, e0.x, e1.x);
                dmma(se[n], as, e0.y, e1.y);
                dmma(co[n], bc, o0.x, o1.x);
                dmma(so[n], bs, o0.y, o1.y);
            }
        }
#pragma unroll
        for (int n = 0; n < RN; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int x = x0 + g + 8 * (e >> 1), i = 2 * n + (e & 1);
                const long o = at[i];
                if (x > xmax || o < 0) continue;
                const double cp = ce[n][e] + co[n][e], cm = ce[n][e] - co[n][e];
                const double sp = se[n][e] + so[n][e], sm = se[n][e] - so[n][e];
                auto put = [&](int n1, double v) {
                    if (out_f64) out_f64[o + n1] = v;
                    if (out_f32) out_f32[o + n1] = (float)(v * wq[i]);
                    if (out_hi) {
                        // split: hi = bf16(v), lo = bf16(v − hi) (both round-to-nearest)
                        const uint16_t hb = bf16_bits((float)v);
                        out_hi[o + n1] = hb;
                        out_lo[o + n1] = bf16_bits((float)(v - (double)__uint_as_float((uint32_t)hb << 16)));
                    }
                };
                put(x, cp - sp);
                if (x > 0) put(ng - x, cp + sp);
                if (2 * x < h) {
                    put(h - x, cm + sm);
                    if (x > 0) put(h + x, cm - sm);
                }
            }
        if (16 * steps > jstage && xg + RX <= xmax) {
            __syncthreads();
            stage(0);
            __syncthreads();
        }
    }
}

// Fixed-point digits for the int8 tensor-core contraction.  Every block of
// LS_BLOCK pixels of a ring slot has one exponent E, shared by all channels:
// the smallest with max|v| < 2^E over the block (0 for an all-zero block).
// Then, with base 254,
//     v·2^−E·127 = d0 + d1/254 + d2/254² + r,   d0, d1, d2 ∈ [−127, 127],
// |r| ≤ 1/(2·254²): signed, balanced digits that use the whole int8 range.
// An exponent per pixel block (rather than per channel row) is what lets the
// contraction add every anchor into one accumulator (lagspace.cuh), and it
// follows the maps' spatial dynamic range: the sampling-mask maps are sharply
// peaked at the origin, so blocks far from it get a much finer digit scale.
__device__ __forceinline__ void digits254(float t, uint32_t &b0, uint32_t &b1, uint32_t &b2)
{
    // round-to-nearest via the 1.5·2^23 magic number: the integer sits in the
    // low mantissa bits, so its low byte is the two's-complement int8 digit
    const float M = 12582912.0f;
    float y0 = t + M;
    float r0 = (t - (y0 - M)) * 254.f;
    float y1 = r0 + M;
    float r1 = (r0 - (y1 - M)) * 254.f;
    float y2 = r1 + M;
    b0 = __float_as_uint(y0);
    b1 = __float_as_uint(y1);
    b2 = __float_as_uint(y2);
}

// bexp[s][b] for block b of slot s (one CTA of LS_BLOCK threads per block: a thread per pixel,
// looping over the channels, so every channel row is read coalesced).
__global__ void __launch_bounds__(LS_BLOCK) block_expo_kernel(const float *__restrict__ f32, long k, long kp,
                                                              long nch, long nblk, int *__restrict__ bexp)
{
    __shared__ float red[LS_BLOCK / 32];
    const long b = blockIdx.x;
    const int s = blockIdx.y;
    const long x = b * LS_BLOCK + threadIdx.x;
    float m = 0.f;
    if (x < k)
        for (long ch = 0; ch < nch; ++ch) m = fmaxf(m, fabsf(f32[((long)s * nch + ch) * kp + x]));
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < LS_BLOCK / 32; ++w) m = fmaxf(m, red[w]);
        bexp[(long)s * nblk + b] = m > 0.f ? ilogbf(m) + 1 : 0;
    }
}

// Slots of one quantize launch: the rings that stand second in a triangle of the batch (the contraction reads
// no other ring's digits), which of the rings of a batch is often a quarter.
struct SlotList {
    unsigned char s[256];
};

// Three digit planes per listed slot in the contraction's staging order,
// dig[s][digit][x/16][ch][16 pixels]: a TMA box of consecutive channels and two 16-pixel
// groups then lands in shared memory exactly as the MMA reads a K-major operand without
// swizzle (8-row core matrices of 16 bytes).  Pixels at or past k become zero digits.
__global__ void __launch_bounds__(256) quantize_kernel(const float *__restrict__ f32, const int *__restrict__ bexp,
                                                       long k, long kp, long nch, long nblk,
                                                       const SlotList slots, int8_t *__restrict__ dig)
{
    const long b = blockIdx.x;
    const int s = slots.s[blockIdx.y];
    const float sc = ldexpf(127.f, -bexp[(long)s * nblk + b]);
    const long kpg = kp / 16;
    for (long e = threadIdx.x; e < (LS_BLOCK / 16) * nch; e += blockDim.x) {
        const long g = e / nch, ch = e % nch;
        const long x0 = b * LS_BLOCK + g * 16;
        const float4 *src = reinterpret_cast<const float4 *>(f32 + ((long)s * nch + ch) * kp + x0);
        uint32_t w[3][4];
        float4 in[4];  // rows are kp ≡ 0 (mod 256) floats from a 256-byte boundary: 16-byte loads, and past k too
#pragma unroll
        for (int q = 0; q < 4; ++q) in[q] = src[q];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float v[4] = {in[q].x, in[q].y, in[q].z, in[q].w};
            uint32_t a[4], bb[4], cc[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) digits254(x0 + 4 * q + t < k ? v[t] * sc : 0.f, a[t], bb[t], cc[t]);
            w[0][q] = __byte_perm(__byte_perm(a[0], a[1], 0x0040), __byte_perm(a[2], a[3], 0x0040), 0x5410);
            w[1][q] = __byte_perm(__byte_perm(bb[0], bb[1], 0x0040), __byte_perm(bb[2], bb[3], 0x0040), 0x5410);
            w[2][q] = __byte_perm(__byte_perm(cc[0], cc[1], 0x0040), __byte_perm(cc[2], cc[3], 0x0040), 0x5410);
        }
#pragma unroll
        for (int d = 0; d < 3; ++d)
            *reinterpret_cast<uint4 *>(dig + (((long)s * 3 + d) * kpg + x0 / 16) * nch * 16 + ch * 16) =
                make_uint4(w[d][0], w[d][1], w[d][2], w[d][3]);
    }
}

// Host: exact per-slot column counts and the largest number of ring rows in
// any column (for the shared-memory staging size).
void ring_shape(long ng, double lo, double hi, int *jcols, int *rows_max)
{
    long J = std::min<long>(ng / 3, (long)ceil(hi));
    long A = (long)ceil(hi) - 1;
    long ia_min = std::max(-A, -ng / 2 + 1), ia_max = std::min(A, ng / 2);
    int best = 0;
    for (long j = 0; j < J; ++j) {
        int n = 0;
        for (long ia = ia_min; ia <= ia_max; ++ia) {
            double uu = sqrt(1.0 * (double)(ia * ia + j * j));
            if (uu >= lo && uu < hi && uu > 0.0) ++n;
        }
        best = std::max(best, n);
    }
    *jcols = (int)std::max<long>(J, 0);
    *rows_max = best;
}

}  // namespace

int build_maps(amber_cuda_ctx *c, const MapJob &job)
{
    const long ng = job.ng;
    std::vector<int> jc(job.nslots);
    int jmax = 1, rows_max = 1;
    for (int s = 0; s < job.nslots; ++s) {
        int rm;
        ring_shape(ng, job.lo[s], job.hi[s], &jc[s], &rm);
        jmax = std::max(jmax, jc[s]);
        rows_max = std::max(rows_max, rm);
    }
    const double2 *tw;
    int rc = twiddle_table(c, ng, &tw);
    if (rc) return rc;
    size_t ybytes = sizeof(double2) * (size_t)job.nslots * ng * jmax * job.nch;
    if ((rc = ensure(c, c->y, ybytes, "map intermediate"))) return rc;
    double2 *Y = reinterpret_cast<double2 *>(c->y.p);

    // pass 1: choose channels per block so the staged column fits
    const size_t smem_cap = 200 * 1024;
    auto p1_smem = [&](int C) { return sizeof(double2) * ng + (sizeof(double2) * C + sizeof(int)) * rows_max; };
    int C1 = 32;
    while (C1 > 1 && C1 / 2 >= job.nch) C1 /= 2;  // calCR's one channel: the lanes go to more rows
    while (C1 > 1 && p1_smem(C1) > smem_cap) C1 /= 2;
    if (p1_smem(C1) > smem_cap) return fail(c, AMBER_ERR_ARG, "ring too wide for the column stage (%d rows)", rows_max);
    const size_t s1 = p1_smem(C1);
    // pass 2: a stage of j that leaves room for two CTAs an SM where the widest ring fits it
    const size_t s2_cap = std::max((size_t)112 * 1024, sizeof(double2) * ((size_t)ng + 16 * RS));
    const int jstage = (int)std::min<size_t>((jmax + 15) / 16, (s2_cap / sizeof(double2) - ng) / (16 * RS)) * 16;
    const size_t s2 = sizeof(double2) * ((size_t)ng + (size_t)jstage * RS);
    // up to RING_META_MAX slots per launch pair, each launch's pointers offset to its first slot
    for (int sb = 0; sb < job.nslots; sb += RING_META_MAX) {
        const int ns = std::min(RING_META_MAX, job.nslots - sb);
        RingMeta meta;
        for (int i = 0; i < ns; ++i) {
            meta.lo[i] = job.lo[sb + i];
            meta.hi[i] = job.hi[sb + i];
            meta.jc[i] = jc[sb + i];
        }
        double2 *Ys = Y + (size_t)sb * ng * jmax * job.nch;
        const size_t so = (size_t)sb * job.nch * job.kp;
        double *of64 = job.out_f64 ? job.out_f64 + so : nullptr;
        uint16_t *ohi = job.out_hi ? job.out_hi + so : nullptr, *olo = job.out_lo ? job.out_lo + so : nullptr;
        float *of32 = job.out_f32 ? job.out_f32 + so : nullptr;
        dim3 g1(jmax, ns, (unsigned)((job.nch + C1 - 1) / C1));
#define LAUNCH_COLS(CC)                                                                                        \
    do {                                                                                                        \
        cudaFuncSetAttribute(ring_cols_kernel<CC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1);        \
        ring_cols_kernel<CC><<<g1, kThreads, s1, c->stream>>>(job.src, job.src_complex ? 1 : 0, job.n1, job.nc, \
                                                               job.chan_base, job.nch, ng, meta, jmax, tw, Ys,  \
                                                               rows_max);                                        \
    } while (0)
        switch (C1) {
            case 32: LAUNCH_COLS(32); break;
            case 16: LAUNCH_COLS(16); break;
            case 8: LAUNCH_COLS(8); break;
            case 4: LAUNCH_COLS(4); break;
            case 2: LAUNCH_COLS(2); break;
            default: LAUNCH_COLS(1); break;
        }
#undef LAUNCH_COLS
        c->launches += 1;
        if ((rc = cuda_check(c, cudaGetLastError(), "ring_cols_kernel launch"))) return rc;

        cudaFuncSetAttribute(ring_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s2);
        ring_rows_kernel<<<dim3((unsigned)((ng * job.nch + RC - 1) / RC), ns), RROWS_THREADS, s2, c->stream>>>(
            Ys, (int)ng, jmax, meta, job.nch, tw, job.kp, jstage, of64, ohi, olo, of32, job.weight);
        c->launches += 1;
        if ((rc = cuda_check(c, cudaGetLastError(), "ring_rows_kernel launch"))) return rc;
    }
    if (job.dig) {
        const long nblk = job.kp / LS_BLOCK;
        dim3 gq((unsigned)nblk, (unsigned)job.nslots);
        block_expo_kernel<<<gq, LS_BLOCK, 0, c->stream>>>(job.out_f32, ng * ng, job.kp, job.nch, nblk, job.bexp);
        SlotList list;
        unsigned n = 0;
        for (int s = 0; s < job.nslots; ++s)
            if (job.need_dig.empty() || job.need_dig[s]) list.s[n++] = (unsigned char)s;
        if (n > 0)
            quantize_kernel<<<dim3((unsigned)nblk, n), 256, 0, c->stream>>>(job.out_f32, job.bexp, ng * ng, job.kp,
                                                                            job.nch, nblk, list, job.dig);
        c->launches += n > 0 ? 2 : 1;
        rc = cuda_check(c, cudaGetLastError(), "quantize_kernel launch");
    }
    return rc;
}

}  // namespace amber
