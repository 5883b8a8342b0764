// Lag-space contraction plan and the deterministic reduction of the units' partial
// tiles (see lagspace.cuh).
#include <algorithm>

#include "lagspace.cuh"

namespace amber {

namespace {

int round16(int n) { return (n + 15) / 16 * 16; }

// lag[Δ2·nclen + Δ3] = Σ over the job's units (anchor blocks, then units of the block, then
// slots) of the partial tiles, TwoSum-compensated, in a fixed order: RED_PARTS threads a cell each add an
// equal run of the terms, eight loads ahead of their sums, and the first adds the runs' sums in order.
// Partial tiles are [column][row] so that consecutive Δ3 read consecutive doubles.  Bound by the latency of
// a cell's chain of loads, not by bytes: 282 terms a cell (46 triangles of 32 channels, eight launches) took
// 0.79 ms with one thread a cell and 0.17 ms with eight.
constexpr int RED_PARTS = 8;

__global__ void __launch_bounds__(32 * RED_PARTS) ls_reduce_kernel(const LsReduceJob *__restrict__ jobs)
{
    __shared__ double ssum[RED_PARTS][32], scomp[RED_PARTS][32];
    const LsReduceJob j = jobs[blockIdx.y];
    const long ncsize = (long)j.nclen * j.nclen;
    const int lane = threadIdx.x, part = threadIdx.y;
    const long d = (long)blockIdx.x * 32 + lane;
    const long TILE = j.tile;
    double s = 0.0, comp = 0.0;
    auto add = [&](double v) {
        const double t = s + v, bp = t - s;
        comp += (s - (t - bp)) + (v - bp);
        s = t;
    };
    if (d < ncsize) {
        const int d2 = (int)(d / j.nclen), d3 = (int)(d % j.nclen);
        const int n = j.nab * j.V * j.k;
        const int i0 = (int)((long)n * part / RED_PARTS), i1 = (int)((long)n * (part + 1) / RED_PARTS);
        // term i: unit i / k, slot i % k (k = 1 for a wide window's tile pair)
        const double *p;
        if (j.k > 1) {
            p = j.partial + (long)d2 * LS_ROWS + d3;
        } else {
            const int t2 = d2 / j.ts, t3 = d3 / j.ts;
            p = j.partial + (long)(t3 * j.T + t2) * j.nab * j.V * TILE + (long)(d2 % j.ts) * LS_ROWS + d3 % j.ts;
        }
        p += (i0 / j.k) * TILE + (i0 % j.k) * j.rs;
        int slot = i0 % j.k;
        auto next = [&] {
            const double v = *p;
            p += j.rs;
            if (++slot == j.k) {
                slot = 0;
                p += TILE - (long)j.k * j.rs;
            }
            return v;
        };
        int i = i0;
        for (; i + 8 <= i1; i += 8) {
            double v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = next();
#pragma unroll
            for (int q = 0; q < 8; ++q) add(v[q]);
        }
        for (; i < i1; ++i) add(next());
    }
    ssum[part][lane] = s;
    scomp[part][lane] = comp;
    __syncthreads();
    if (part != 0 || d >= ncsize) return;
    for (int q = 1; q < RED_PARTS; ++q) {
        add(ssum[q][lane]);
        comp += scomp[q][lane];
    }
    j.lag[d] = s + comp;
}

}  // namespace

int LsShape::rows(int t3) const { return k > 1 ? k * rs : std::min(ts, nclen - ts * t3); }
int LsShape::cols(int t2) const
{
    return k > 1 ? round16(nclen + k - 1) : round16(std::min(ts, nclen - ts * t2));
}

LsShape ls_shape(int nc, int nc10, long k_px, int sms, long min_groups, long force_bpu)
{
    LsShape s;
    s.nc = nc;
    s.nc10 = nc10;
    s.nclen = 2 * nc10 + 1;
    s.rs = (s.nclen + 7) / 8 * 8;
    s.k = s.rs <= LS_ROWS / 2 ? LS_ROWS / s.rs : 1;
    s.T = s.k > 1 ? 1 : (s.nclen + LS_ROWS - 1) / LS_ROWS;
    // Near-equal tiles of whole 8-row blocks: an edge tile of a few lags costs nearly a whole one (an MMA at
    // least 42 cycles, the formers all its rows against one column), so 129 lags run as 72 + 57.
    s.ts = std::min(LS_ROWS, ((s.nclen + s.T - 1) / s.T + 7) / 8 * 8);
    // Staged rows of one unit: D3 spans AB + rows − 1 channels and the D2 window AB + N − 1;
    // both must fit one TMA box (LS_SPAN rows).  An anchor block also holds at most LS_GROUPS anchor
    // groups, so that they and LS_BLOCK pixels of int8 digit products cannot overflow the int32 accumulators
    // (|class sum| ≤ 3·127² per term, 2^31 / 48387 = 44381 terms).  The channels go into blocks of equal
    // size: a last block of a few anchors would pay a whole unit's staging.
    const int span_extra = std::max(s.rows(0), s.cols(0)) - 1;
    const int widest = std::max(1, std::min({nc, LS_SPAN - span_extra, LS_GROUPS * s.k}));
    s.nab = (nc + widest - 1) / widest;
    s.AB = std::min(widest, ((nc + s.nab - 1) / s.nab + s.k - 1) / s.k * s.k);
    s.nab = (nc + s.AB - 1) / s.AB;
    s.nblk = std::max<long>(1, (k_px + LS_BLOCK - 1) / LS_BLOCK);
    // Units: about six per SM for a large job, so the last wave is short; down to one block each (two where a block
    // is a single anchor group) for a small one, so that it still spreads over the SMs: at eight blocks a unit, the
    // kernel of one 2304-pixel triangle of 16 channels (9 blocks) took 104 µs on two SMs, and the eight
    // launches of a 32-channel realisation's 46 triangles 4.0 ms against 2.4 ms at one block a unit.
    const long per_block = std::max(1, s.AB / s.k) + 2;
    const long min_bpu = std::max<long>(1, (min_groups + per_block - 1) / per_block);
    const long combos = (long)s.T * s.T * s.nab;
    const long target = 6L * std::max(1, sms);
    s.bpu = force_bpu > 0 ? std::min(s.nblk, force_bpu)
                          : std::min(s.nblk, std::max(min_bpu, (s.nblk * combos + target - 1) / target));
    s.V = (int)((s.nblk + s.bpu - 1) / s.bpu);
    return s;
}

void ls_plan_job(LsJobPlan &p, int nc, int nc10, long k_px, const std::vector<int> &weight, int sms, long min_groups,
                 long force_bpu)
{
    p.s = ls_shape(nc, nc10, k_px, sms, min_groups, force_bpu);
    p.groups.clear();
    p.group_off.assign(1, 0);
    for (int ab = 0; ab < p.s.nab; ++ab) {
        const int c0 = ab * p.s.AB, c1 = std::min(nc, c0 + p.s.AB);
        for (int pb = c0; pb < c1; pb += p.s.k) {
            bool any = false;
            for (int a = 0; a < p.s.k && pb + a < c1; ++a) any = any || weight[pb + a] > 0;
            if (any) p.groups.push_back(pb);
        }
        p.group_off.push_back((int)p.groups.size());
    }
}

void ls_units(const LsJobPlan &p, int job, std::vector<LsUnit> &out)
{
    const LsShape &s = p.s;
    long local = 0;
    for (int t3 = 0; t3 < s.T; ++t3)
        for (int t2 = 0; t2 < s.T; ++t2)
            for (int ab = 0; ab < s.nab; ++ab)
                for (int v = 0; v < s.V; ++v) {
                    LsUnit u;
                    u.job = job;
                    u.t3 = (short)t3;
                    u.t2 = (short)t2;
                    u.ab = ab;
                    u.b0 = (int)(v * s.bpu);
                    u.b1 = (int)std::min(s.nblk, (v + 1) * s.bpu);
                    u.tile = p.unit_base + s.tile() * local++;
                    u.work = (double)(u.b1 - u.b0) * (p.group_off[ab + 1] - p.group_off[ab]);
                    out.push_back(u);
                }
}

int ls_reduce(amber_cuda_ctx *c, const std::vector<LsReduceJob> &jobs)
{
    if (jobs.empty()) return AMBER_OK;
    int rc;
    const size_t bytes = sizeof(LsReduceJob) * jobs.size();
    if ((rc = ensure(c, c->lsred, bytes, "lag reduction job list"))) return rc;
    if ((rc = cuda_check(c, cudaMemcpyAsync(c->lsred.p, jobs.data(), bytes, cudaMemcpyHostToDevice, c->stream),
                         "lag reduction job list")))
        return rc;
    long cells = 0;
    for (const LsReduceJob &j : jobs) cells = std::max<long>(cells, (long)j.nclen * j.nclen);
    phase_begin(c, 2);
    for (size_t j0 = 0; j0 < jobs.size(); j0 += 65535) {
        const unsigned nj = (unsigned)std::min<size_t>(65535, jobs.size() - j0);
        ls_reduce_kernel<<<dim3((unsigned)((cells + 31) / 32), nj), dim3(32, RED_PARTS), 0, c->stream>>>(
            (const LsReduceJob *)c->lsred.p + j0);
        c->launches += 1;
    }
    phase_end(c);
    return cuda_check(c, cudaGetLastError(), "ls_reduce launch");
}

}  // namespace amber
