// MAPS two-point function on the device: the multi-frequency angular power
// spectrum C_ℓ(Δν) of the normalised grid, as 4_fbe/maps.c:179-210 computes it
// by calling cl_dnu (4_fbe/amber_funcs.c:1418-1488) for every channel pair
// nn1 <= nn2.  Per log bin b of U = |(ia, j)|·Du in [umin, umax) and pair (p, q):
//   no_b[p]     = Σ_{cells in b} NTiG[p]
//   S_b[p][q]   = Σ_{cells in b} (Re_p·Re_q + Im_p·Im_q)·NTiG[p]
//   binps       = S_b[p][q] / no_b[p]                  (where no_b[p] != 0)
//   cldnu[b][Δ] = Σ_{p = 0 .. nc−1−Δ} binps(p, p + Δ)  (p ascending)
// and the printed binu / num are usum / no and no of the last pair (p = nc−1).
//
// Every sum runs in the reference's order with the reference's roundings
// (cells in index order, separate multiplies and adds — the reference build has
// no FMA contraction — then the division, then the Δ sums over p ascending), so
// the results are bit-identical to the reference's loops.  The bin of each cell
// (sqrt, log10, floor of the reference's expressions) is computed on the host
// with the C library, so no device-vs-host libm difference can move a cell.
//
// Kernels:
//   cldnu_pairs  one CTA per (bin, 16×16 tile of (p, q) with q-tile >= p-tile):
//                the bin's cells in chunks of 16 through four stages of shared memory,
//                two p of one q per thread, FP64, sums to P[b][p][q − p]; in a diagonal
//                tile one more warp adds no_b[p] and usum_b[p];
//   cldnu_reduce one warp per (bin, Δ): Σ_p P[b][p][Δ] / no_b[p].
// Work: 5 FP64 operations per (cell, pair); the bin's grid rows are read once
// per tile pair.  Bound by the largest bin's chain of cells.
#include <math.h>

#include <algorithm>
#include <vector>

#include "common.cuh"

namespace amber {

namespace {

constexpr int kTile = 16;    // (p, q) tile of a CTA
constexpr int kChunk = 16;   // cells per shared-memory stage
constexpr int kStages = 4;
constexpr int kPair = 128;   // threads that add pairs, two p of one q each
constexpr int kThreads = kPair + 32;  // and a warp that adds a diagonal tile's counts

// One stage: the chunk's cells for the tile's p channels (value and sampling weight) and q channels, and their U.
struct Stage {
    double2 g1[kChunk][kTile], g2[kChunk][kTile];
    double w1[kChunk][kTile];
    double u[kChunk];
};

// n bytes (16 or 8) from global to shared memory, or zeros when !in
template <int N>
__device__ __forceinline__ void copy_async(void *dst, const void *src, bool in)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(N), "r"(in ? N : 0)
                 : "memory");
}

// P[b][p][q − p] = Σ_{cells in b} (Re_p·Re_q + Im_p·Im_q)·NTiG[p] for one tile of pairs, and in a diagonal tile
// the bin's counts and ΣU of its channels.  The cells of a pair are added one after another, so a bin's chain is
// as long as its cells: the bins run largest first, in tiles small enough that the largest one's pairs lie on many
// SMs, a tile's warps on all four partitions of its SM, with three chunks of cells in flight.  256² cells, 128
// channels, 15 bins (the largest has 19004 cells): 5.2 ms in 32 × 32 tiles staged without overlap and with the counts
// in a launch of their own; 0.75 ms with the counts in CTAs of their own (a chain of mask loads of 75 cycles a
// cell), two warps a tile and two stages; 0.55-0.68 ms now, the call 1.40 → 1.20 ms.
__global__ void __launch_bounds__(kThreads) cldnu_pairs(const double2 *__restrict__ grid,
                                                        const double *__restrict__ mask,
                                                        const int *__restrict__ cells, const double *__restrict__ uu,
                                                        const int *__restrict__ bin_off, long nc, int ntile,
                                                        int *__restrict__ no, double *__restrict__ usum,
                                                        double *__restrict__ P)
{
    __shared__ Stage st[kStages];
    const int b = gridDim.y - 1 - blockIdx.y;  // log bins: the last holds the most cells
    const int k0 = bin_off[b], k1 = bin_off[b + 1];
    // t → (tp, tq), tq >= tp
    int t = blockIdx.x, tp = 0;
    while (t >= ntile - tp) {
        t -= ntile - tp;
        ++tp;
    }
    const int tq = tp + t;
    const long p0 = (long)tp * kTile, q0 = (long)tq * kTile;
    // pairs: q channel and first p channel; staging: channel and first cell of the chunk
    const int ch = threadIdx.x % kTile, row = threadIdx.x / kTile;
    constexpr int KR = kPair / kTile, KN = kChunk / KR;
    const bool pairs = threadIdx.x < kPair, pin = p0 + ch < nc, qin = q0 + ch < nc;
    const int lane = (int)threadIdx.x - kPair;  // of the counting warp
    double acc[2] = {0.0, 0.0}, u = 0.0;
    int n = 0, cell[KN];
    auto load_cells = [&](int kc) {
        if (!pairs) return;
#pragma unroll
        for (int i = 0; i < KN; ++i) cell[i] = kc + row + KR * i < k1 ? cells[kc + row + KR * i] : -1;
    };
    auto stage = [&](Stage &s, int kc) {
        if (pairs) {
#pragma unroll
            for (int i = 0; i < KN; ++i) {
                const int k = row + KR * i;
                const long at = (cell[i] >= 0 ? (long)cell[i] : 0) * nc;
                const long ap = at + (pin ? p0 + ch : 0), aq = at + (qin ? q0 + ch : 0);
                copy_async<16>(&s.g1[k][ch], grid + ap, cell[i] >= 0 && pin);
                copy_async<16>(&s.g2[k][ch], grid + aq, cell[i] >= 0 && qin);
                copy_async<8>(&s.w1[k][ch], mask + ap, cell[i] >= 0 && pin);
            }
        } else if (lane < kChunk) {
            const bool in = kc + lane < k1;
            copy_async<8>(&s.u[lane], uu + (in ? kc + lane : k0), in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (k0 < k1) {
#pragma unroll
        for (int i = 0; i < kStages - 1; ++i) {
            load_cells(k0 + kChunk * i);
            stage(st[i], k0 + kChunk * i);
        }
        load_cells(k0 + kChunk * (kStages - 1));
    }
    int cur = 0;
    for (int kc = k0; kc < k1; kc += kChunk, cur = (cur + 1) % kStages) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();  // this chunk is in; every reader of the stage filled next is done
        stage(st[(cur + kStages - 1) % kStages], kc + kChunk * (kStages - 1));
        load_cells(kc + kChunk * kStages);
        const int nk = min(kChunk, k1 - kc);
        const Stage &s = st[cur];
        if (pairs) {
#pragma unroll 4
            for (int k = 0; k < nk; ++k) {
                const double2 g2 = s.g2[k][ch];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    // numer = Re1·Re2 + Im1·Im2; numer *= NTiG; pksum += numer
                    const double2 g1 = s.g1[k][row + KR * i];
                    const double numer = __dmul_rn(__dadd_rn(__dmul_rn(g1.x, g2.x), __dmul_rn(g1.y, g2.y)),
                                                   s.w1[k][row + KR * i]);
                    acc[i] = __dadd_rn(acc[i], numer);
                }
            }
        } else if (tp == tq && lane < kTile) {
#pragma unroll 4
            for (int k = 0; k < nk; ++k) {
                // no[tmp] += NTiG (int += double); the mask is 0 or 1, for which the conversions drop out
                const double w = s.w1[k][lane];
                n = w == 0.0 || w == 1.0 ? n + (w == 1.0) : (int)((double)n + w);
                u = __dadd_rn(u, __dmul_rn(s.u[k], w));
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (pairs) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const long p = p0 + row + KR * i, q = q0 + ch;
            if (q >= p && q < nc) P[((long)b * nc + p) * nc + (q - p)] = acc[i];
        }
    } else if (tp == tq && lane < kTile && p0 + lane < nc) {
        no[(long)b * nc + p0 + lane] = n;
        usum[(long)b * nc + p0 + lane] = u;
    }
}

// cldnu[b][Δ] = Σ_p binps(p, p + Δ), p ascending, binps = P / no_b[p] where the count is not zero: one warp
// per (bin, Δ) divides 32 terms at a time, then adds them one after another.  Bound by the loads' latency:
// one thread per (bin, Δ) had a dependent load, divide and add for each p.  256² cells, 128 channels, 15 bins:
// 76 µs before, 7 µs now.
__global__ void __launch_bounds__(32) cldnu_reduce(const double *__restrict__ P, const int *__restrict__ no, long nc,
                                                   double *__restrict__ cldnu)
{
    const long b = blockIdx.y, d = blockIdx.x;
    double s = 0.0;
    for (long p0 = 0; p0 + d < nc; p0 += 32) {
        const long p = p0 + threadIdx.x;
        double v = 0.0;
        if (p + d < nc) {
            v = P[(b * nc + p) * nc + d];
            const int n = no[b * nc + p];
            if (n != 0) v = __ddiv_rn(v, (double)n);
        }
        const int m = (int)min(32L, nc - d - p0);
        for (int i = 0; i < m; ++i) s = __dadd_rn(s, __shfl_sync(0xffffffffu, v, i));
    }
    if (threadIdx.x == 0) cldnu[b * nc + d] = s;
}

}  // namespace

}  // namespace amber

using namespace amber;

extern "C" int amber_cuda_cl_dnu(amber_cuda_ctx *c, int NB, double umin, double umax, double *cldnu, double *numdnu,
                                 double *binu, int *num)
{
    if (!c || !cldnu) return AMBER_ERR_ARG;
    if (!c->grid.p || c->N1 <= 0 || c->nc <= 0) return fail(c, AMBER_ERR_STATE, "cl_dnu: no grid loaded");
    if (NB <= 0 || NB > 4096 || !(umin > 0) || !(umax > umin))
        return fail(c, AMBER_ERR_ARG, "cl_dnu: need 0 < NB <= 4096 and 0 < umin < umax");
    const long N1 = c->N1, H = N1 / 2 + 1, nc = c->nc;
    // bins of the cells, the reference's expressions (amber_funcs.c:1448-1462) on the host
    const double binsiz = log10(umax / umin) / (1. * NB);
    std::vector<std::vector<int>> by_bin(NB);
    std::vector<std::vector<double>> uu_bin(NB);
    for (long i = 0; i < N1; ++i)
        for (long j = 0; j < H; ++j) {
            const long ia = (i > N1 / 2) ? (N1 - i) : i;
            const double uu = sqrt(1. * (ia * ia + j * j)) * c->Du;
            if (!(uu >= umin && uu < umax)) continue;
            const int tmp = (int)floor(log10(uu / umin) / binsiz);
            if (tmp < 0 || tmp >= NB) continue;  // U rounding onto umax: the reference writes past its arrays
            by_bin[tmp].push_back((int)(i * H + j));
            uu_bin[tmp].push_back(uu);
        }
    std::vector<int> cells, off(NB + 1, 0);
    std::vector<double> uus;
    for (int b = 0; b < NB; ++b) {
        cells.insert(cells.end(), by_bin[b].begin(), by_bin[b].end());
        uus.insert(uus.end(), uu_bin[b].begin(), uu_bin[b].end());
        off[b + 1] = (int)cells.size();
    }
    const long ncell = std::max<long>(1, (long)cells.size());
    const int ntile = (int)((nc + kTile - 1) / kTile);
    // scratch: P [NB][nc][nc] + usum [NB][nc] + uu [cells] (doubles), then no [NB][nc] + cells + off (ints)
    auto up4 = [](size_t n) { return (n + 3) / 4 * 4; };
    const size_t nP = (size_t)NB * nc * nc, nU = (size_t)NB * nc;
    const size_t o_usum = up4(nP), o_uu = o_usum + up4(nU), o_int = o_uu + up4(ncell);
    const size_t n_int = (size_t)NB * nc + ncell + NB + 1;
    const size_t bytes = sizeof(double) * o_int + sizeof(int) * n_int;
    int rc;
    if ((rc = ensure(c, c->mixed_scratch, bytes, "cl_dnu scratch"))) return rc;
    cudaSetDevice(c->device);
    double *P = (double *)c->mixed_scratch.p;
    double *usum = P + o_usum, *d_uu = P + o_uu;
    int *no = (int *)(P + o_int), *d_cells = no + (size_t)NB * nc, *d_off = d_cells + ncell;
    cudaStream_t s = c->stream;
    if (!cells.empty()) {
        if ((rc = cuda_check(c, cudaMemcpyAsync(d_cells, cells.data(), sizeof(int) * cells.size(),
                                                cudaMemcpyHostToDevice, s), "cl_dnu cells")))
            return rc;
        if ((rc = cuda_check(c, cudaMemcpyAsync(d_uu, uus.data(), sizeof(double) * uus.size(), cudaMemcpyHostToDevice,
                                                s), "cl_dnu U")))
            return rc;
    }
    if ((rc = cuda_check(c, cudaMemcpyAsync(d_off, off.data(), sizeof(int) * (NB + 1), cudaMemcpyHostToDevice, s),
                         "cl_dnu bins")))
        return rc;
    const double2 *grid = (const double2 *)c->grid.p;
    const double *mask = (const double *)c->mask.p;
    const unsigned npair = (unsigned)(ntile * (ntile + 1) / 2);
    cldnu_pairs<<<dim3(npair, NB), kThreads, 0, s>>>(grid, mask, d_cells, d_uu, d_off, nc, ntile, no, usum, P);
    // no / usum come back first; the Δ sums then reuse the usum slot (same stream, in order)
    std::vector<int> h_no((size_t)NB * nc);
    std::vector<double> h_usum((size_t)NB * nc);
    if ((rc = cuda_check(c, cudaGetLastError(), "cl_dnu launch"))) return rc;
    if ((rc = cuda_check(c, cudaMemcpyAsync(h_no.data(), no, sizeof(int) * h_no.size(), cudaMemcpyDeviceToHost, s),
                         "cl_dnu counts")))
        return rc;
    if ((rc = cuda_check(c, cudaMemcpyAsync(h_usum.data(), usum, sizeof(double) * h_usum.size(), cudaMemcpyDeviceToHost,
                                            s), "cl_dnu U sums")))
        return rc;
    cldnu_reduce<<<dim3((unsigned)nc, NB), 32, 0, s>>>(P, no, nc, usum);
    c->launches += 2;
    if ((rc = cuda_check(c, cudaGetLastError(), "cl_dnu launch"))) return rc;
    if ((rc = cuda_check(c, cudaMemcpyAsync(cldnu, usum, sizeof(double) * nU, cudaMemcpyDeviceToHost, s),
                         "cl_dnu download")))
        return rc;
    if ((rc = cuda_check(c, cudaStreamSynchronize(s), "cl_dnu"))) return rc;
    // maps.c:187 (numdnu[nn2−nn1] += 1 per pair) and the last pair's binu / num (maps.c:197-205)
    if (numdnu)
        for (long d = 0; d < nc; ++d) {
            double v = 0.;
            for (long p = 0; p + d < nc; ++p) v += 1.;
            numdnu[d] = v;
        }
    for (int b = 0; b < NB; ++b) {
        const int n = h_no[(size_t)b * nc + nc - 1];
        const double u = h_usum[(size_t)b * nc + nc - 1];
        if (binu) binu[b] = n != 0 ? u / (1. * n) : u;
        if (num) num[b] = n;
    }
    return AMBER_OK;
}
