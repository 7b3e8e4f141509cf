// sphg_pairs2.cuh — the FP32 pair passes with two particles per lane pair.
//
// Two neighbouring lanes take two consecutive particles of the cell-sorted
// list.  The particles lie in the same or the next cell, so their candidate
// runs overlap almost entirely: the lanes walk the union of the two sets once,
// one lane the even candidates and one the odd, and evaluate the pair terms of
// BOTH particles for each candidate in Blackwell's packed FP32 arithmetic
// (fma/mul/add.rn.f32x2), one particle in each half.  A candidate that is a
// neighbour of only one of the two gets the kernel values W = 0 and grad W = 0
// in the other half.  (0 times the infinity or NaN of a candidate is NaN, so a
// particle whose sums come out not finite visits its own neighbours once more,
// alone: visit_alone.)  At the end the lanes swap halves (one shuffle per sum)
// and each finishes its own particle.  The pair test stays the exact FP64 one.
//
// Why: the passes are bound by instruction issue (129 and 143 warp
// instructions per particle for water_pass_a and _b with one particle per
// lane, 60-75 % of the issue slots), not by memory or the FP32 pipe; one
// record load, one loop step and one packed instruction now serve two
// particles.  Giving a lane both particles and all candidates instead halves
// the number of warps: measured no faster, since the latency was no longer
// hidden (34-45 % of the issue slots at 12-16 warps per SM).
//
// Used in FP32 mode when every h is equal (SearchConst::uniform), for the
// two-phase water passes and the soil pass.  Contexts with several h, and
// FP64, run the one-particle forms, and so does the water-only step: its
// density is an FP32 sum every step, whose last bit the Tait equation turns into
// 3e-5 of the pressure, so its passes keep their rounding.
#pragma once
#include "sphg_device.cuh"

// ------------------------------------------------------- packed helpers
__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float2 rcp2(float2 a) { return make_float2(rcp_approx(a.x), rcp_approx(a.y)); }
__device__ __forceinline__ float2 sel2(bool a, bool b, float2 v) { return make_float2(a ? v.x : 0.0f, b ? v.y : 0.0f); }

// Constants of the pair terms, computed once on the host (h is the one
// smoothing length of the context): as kernel parameters they cost the
// passes no vector registers.
struct PairK {
    float h, nih;             // h, -1/h
    float sn1, sn0;           // cubic spline, q <= 1: s' = sn1 (-q) + sn0
    float ks, kw;             // grad W = ks s' dx, W = kw w'
    float nh, h2e, alpha, beta, alpha_c;   // -h, etq^2 h^2, alpha/2 and beta of art_visc, alpha c_soil
    float r0, dd, p1, p2;     // wall force; dd over ks
    float kb;                 // Forchheimer
    double dh;                // delta h of delta-SPH
    double thr;               // exact squared pair-test threshold
};

// The shapes w' and s' of two pairs (W = kw w', grad W = ks s' dx); the halves
// whose pair is no neighbour (hit false) get zero.  FU: 2 - q, whose powers the
// kernels are, in one multiply-add, so rounded once (water_pass_a and the
// soil-only pass; the momentum and cross sums of the two-phase passes were as close
// to FP64 with q rounded first, and keep that: a run held against the oracle there
// has a particle within a rounding of yielding).
template <int SKF, bool FU>
__device__ __forceinline__ void kernel_pair(const PairK& K, float2 r2, bool h0, bool h1, float2& w, float2& s) {
    if constexpr (SKF == 1 || SKF == 4) {
        const float2 rinv = make_float2(rsqrt_approx(fmaxf(r2.x, 1e-30f)), rsqrt_approx(fmaxf(r2.y, 1e-30f)));
        const float2 r = mul2(r2, rinv), nq = mul2(r, splat2(K.nih));   // -q
        const float2 u = FU ? fma2(r, splat2(K.nih), splat2(2.0f)) : add2(nq, splat2(2.0f));   // 2 - q
        if constexpr (SKF == 1) {   // W = fac/6 (4 - 6 q^2 + 3 q^3 | (2-q)^3), s = -fac/(2h) ((4 - 3q)/h | (2-q)^2 / r)
            const float2 wn = fma2(mul2(nq, nq), fma2(splat2(-3.0f), nq, splat2(-6.0f)), splat2(4.0f));
            const float2 sn = fma2(splat2(K.sn1), nq, splat2(K.sn0));
            const float2 uu = mul2(u, u);
            const float2 wf = mul2(uu, u), sf = mul2(uu, rinv);
            w = sel2(h0, h1, make_float2(nq.x >= -1.0f ? wn.x : wf.x, nq.y >= -1.0f ? wn.y : wf.y));
            s = sel2(h0, h1, make_float2(nq.x >= -1.0f ? sn.x : sf.x, nq.y >= -1.0f ? sn.y : sf.y));
        } else {   // the gradient polynomial -5 + 15q/2 - 15q^2/4 + 5q^3/8 is -5/8 (2 - q)^3
            const float2 uu = mul2(u, u);
            w = sel2(h0, h1, mul2(mul2(uu, uu), fma2(splat2(-2.0f), nq, splat2(1.0f))));
            s = sel2(h0, h1, mul2(uu, u));
        }
    } else {   // ks = kw = 1
        KernelConst<float, SKF> k;
        k.init(K.h);
        float w0, s0, w1, s1;
        k.eval(r2.x, w0, s0);
        k.eval(r2.y, w1, s1);
        w = sel2(h0, h1, make_float2(w0, w1));
        s = sel2(h0, h1, make_float2(s0, s1));
    }
}

// ---------------------------------------------------------- candidate runs
constexpr int PAIR_MASK = 126;   // candidates that the two lanes' 63-bit masks hold

// Three row runs of the cell-sorted list; candidate t = 0 .. tot - 1.
struct Runs3 {
    int b0, b1, b2, L0, L01, tot;
    __device__ __forceinline__ int at(int t) const { return t < L0 ? b0 + t : (t < L01 ? b1 + (t - L0) : b2 + (t - L01)); }
};

// rows cy-1 .. cy+1, cells xlo-kx .. xhi+kx
__device__ __forceinline__ Runs3 row_runs(const GridGeom& g, const int* __restrict__ cstart, int xlo, int xhi, int cy) {
    const int x0 = xlo > g.kx ? xlo - g.kx : 0;
    const int x1 = (xhi < g.ncx - 1 - g.kx ? xhi + g.kx : g.ncx - 1) + 1;
    Runs3 r{0, 0, 0, 0, 0, 0};
    if (cy > 0) { r.b0 = __ldg(cstart + (cy - 1) * g.ncx + x0); r.L0 = __ldg(cstart + (cy - 1) * g.ncx + x1) - r.b0; }
    r.b1 = __ldg(cstart + cy * g.ncx + x0);
    r.L01 = r.L0 + __ldg(cstart + cy * g.ncx + x1) - r.b1;
    r.tot = r.L01;
    if (cy + 1 < g.ncy) { r.b2 = __ldg(cstart + (cy + 1) * g.ncx + x0); r.tot += __ldg(cstart + (cy + 1) * g.ncx + x1) - r.b2; }
    return r;
}

// The lane pair's two particles: sorted slots k & ~1 (half 0) and k | 1 (half
// 1); this lane finishes slot k.  Slots beyond n repeat the last particle and
// are inactive.
struct LanePair {
    int k, k0, k1, lane;      // own slot, the two halves' slots, own half
    bool valid, v0, v1;
    double2 x0, x1;
    int cx, cy, ox, oy;       // own cell, the other lane's cell
    __device__ __forceinline__ LanePair(const GridGeom& g, const double2* __restrict__ xs, int n) {
        k = (int)(blockIdx.x * blockDim.x + threadIdx.x);
        lane = k & 1;
        valid = k < n;
        k0 = k & ~1;
        k1 = k | 1;
        v0 = k0 < n;
        v1 = k1 < n;
        if (!v0) k0 = n - 1;
        if (!v1) k1 = n - 1;
        x0 = xs[k0];
        x1 = xs[k1];
        bool cl;
        cell_coords(g, lane ? x1.x : x0.x, lane ? x1.y : x0.y, cx, cy, cl);
        ox = __shfl_xor_sync(0xffffffffu, cx, 1);
        oy = __shfl_xor_sync(0xffffffffu, cy, 1);
    }
    // this lane's particle's part of a sum over both lanes
    __device__ __forceinline__ float mine(float2 v) const {
        return (lane ? v.y : v.x) + __shfl_xor_sync(0xffffffffu, lane ? v.x : v.y, 1);
    }
    // this lane's particle's half alone
    __device__ __forceinline__ float own(float2 v) const { return lane ? v.y : v.x; }
    __device__ __forceinline__ int mine(int h0, int h1) const {
        return (lane ? h1 : h0) + __shfl_xor_sync(0xffffffffu, lane ? h0 : h1, 1);
    }
};

// The candidates of the two particles, in one part (the union of both
// particles' runs: same row, and few enough for the hit masks) or in two
// parts (each particle's own runs, the other inactive).  Both lanes of a pair
// agree.
struct PairRuns {
    Runs3 u;
    bool one;
    __device__ __forceinline__ void init(const GridGeom& g, const int* __restrict__ cstart, const LanePair& p) {
        one = !p.v1 || p.cy == p.oy;
        u = Runs3{0, 0, 0, 0, 0, 0};
        if (p.v0 && one) {
            u = row_runs(g, cstart, p.v1 ? min(p.cx, p.ox) : p.lane ? p.ox : p.cx, p.v1 ? max(p.cx, p.ox) : p.lane ? p.ox : p.cx,
                         p.lane ? p.oy : p.cy);
            if (p.v1 && u.tot > PAIR_MASK) one = false;
        }
    }
    __device__ __forceinline__ int parts() const { return __any_sync(0xffffffffu, !one) ? 2 : 1; }
    // runs of a part, and which of the two particles it covers
    __device__ __forceinline__ Runs3 part(const GridGeom& g, const int* __restrict__ cstart, const LanePair& p, int i,
                                          bool& a0, bool& a1) const {
        a0 = p.v0 && i == 0;
        a1 = p.v1 && (one ? i == 0 : i == 1);
        if (one) return i == 0 ? u : Runs3{0, 0, 0, 0, 0, 0};
        const bool own = p.lane == i;   // part i is particle i's
        return row_runs(g, cstart, own ? p.cx : p.ox, own ? p.cx : p.ox, own ? p.cy : p.oy);
    }
    // row of a part's particles
    __device__ __forceinline__ int row(const LanePair& p, int i) const { return p.lane == (one ? 0 : i) ? p.cy : p.oy; }
};

// Hit masks of one lane over its own candidates (bit i = candidate 2 i + lane):
// particle 0 in x, y, particle 1 in z, w.  The highest bit alone marks a
// particle with more candidates than the masks hold.
__device__ __forceinline__ bool pair_overflow(unsigned lo, unsigned hi) { return hi == 0x80000000u && lo == 0u; }

// This lane's half of the candidates against both particles: the exact FP64
// pair test (the reference's operations, m_particles.f90:972-973; thr is its
// exact squared threshold), then body(m, dx, dy, h0, h1) with the halves'
// hits.  s0, s1: the particles' own indices (skipped).  With REC the hits are
// also recorded.  Adds the hits up.
template <bool REC, class F>
__device__ __forceinline__ void pair_scan(const Runs3& r, int lane, double thr, const double2* xs, double2 x0, double2 x1,
                                          int s0, int s1, bool a0, bool a1, uint4& mask, int& hits0, int& hits1, F&& body) {
    unsigned w0 = 0u, w1 = 0u, bit = 1u;
    for (int t = lane; t < r.tot; t += 2) {
        const int m = r.at(t);
        const double2 xb = xs[m];
        const double dx0 = x0.x - xb.x, dy0 = x0.y - xb.y, dx1 = x1.x - xb.x, dy1 = x1.y - xb.y;
        const bool h0 = a0 && m != s0 && __dadd_rn(__dmul_rn(dx0, dx0), __dmul_rn(dy0, dy0)) < thr;
        const bool h1 = a1 && m != s1 && __dadd_rn(__dmul_rn(dx1, dx1), __dmul_rn(dy1, dy1)) < thr;
        body(m, make_float2((float)dx0, (float)dx1), make_float2((float)dy0, (float)dy1), h0, h1);
        if (REC) {
            if (h0) w0 |= bit;
            if (h1) w1 |= bit;
            bit <<= 1;
            if (bit == 0u) {   // 32 candidates of this lane
                hits0 += __popc(w0);
                hits1 += __popc(w1);
                if (t < 64) {
                    if (a0) mask.x = w0;
                    if (a1) mask.z = w1;
                } else if (t < 128) {
                    if (a0) mask.y = w0;
                    if (a1) mask.w = w1;
                }
                w0 = w1 = 0u;
                bit = 1u;
            }
        } else {
            hits0 += h0;
            hits1 += h1;
        }
    }
    if (REC) {
        hits0 += __popc(w0);
        hits1 += __popc(w1);
        if (r.tot <= 64) {   // (a whole word was stored above when the lane has 32 candidates)
            if (bit != 1u) {
                if (a0) mask.x = w0;
                if (a1) mask.z = w1;
            }
        } else if (r.tot <= PAIR_MASK) {
            if (a0) mask.y = w0;
            if (a1) mask.w = w1;
        } else {
            if (a0) { mask.x = 0u; mask.y = 0x80000000u; }
            if (a1) { mask.z = 0u; mask.w = 0x80000000u; }
        }
    }
}

// The same visit replayed from this lane's recorded masks: the same
// neighbours in the same order, without testing any candidate again.
template <class F>
__device__ __forceinline__ void pair_replay(const Runs3& r, int lane, double thr, const double2* xs, double2 x0, double2 x1,
                                            int s0, int s1, bool a0, bool a1, uint4 mask, F&& body) {
    if ((a0 && pair_overflow(mask.x, mask.y)) || (a1 && pair_overflow(mask.z, mask.w))) {   // only ever one active particle
        int h0 = 0, h1 = 0;
        pair_scan<false>(r, lane, thr, xs, x0, x1, s0, s1, a0, a1, mask, h0, h1, body);
        return;
    }
    if (!a0) mask.x = mask.y = 0u;
    if (!a1) mask.z = mask.w = 0u;
    int t0 = lane;
    unsigned cur = mask.x | mask.z;
    while (true) {
        if (cur == 0u) {   // the lane's second word (more than 64 candidates), if any
            if ((mask.y | mask.w) == 0u) break;
            mask.x = mask.y; mask.z = mask.w; mask.y = mask.w = 0u;
            cur = mask.x | mask.z;
            t0 = 64 + lane;
        }
        const unsigned bit = cur & (0u - cur);
        cur ^= bit;
        const int m = r.at(t0 + 2 * (31 - __clz((int)bit)));
        const double2 xb = xs[m];
        body(m, make_float2((float)(x0.x - xb.x), (float)(x1.x - xb.x)),
             make_float2((float)(x0.y - xb.y), (float)(x1.y - xb.y)), (mask.x & bit) != 0u, (mask.z & bit) != 0u);
    }
}

// The lane's own particle's neighbours, and no other candidate, by the lane alone
// (nothing of it is shared with other lanes): body as in pair_scan, with the
// other half inactive and its sums left to be ignored.
template <class F>
__device__ __forceinline__ void visit_alone(const GridGeom& g, const int* __restrict__ cstart, double thr, const double2* xs,
                                            const LanePair& p, int self, F&& body) {
    const Runs3 r = row_runs(g, cstart, p.cx, p.cx, p.cy);
    const double2 xa = p.lane ? p.x1 : p.x0;
#pragma unroll 1
    for (int t = 0; t < r.tot; ++t) {
        const int m = r.at(t);
        const double2 xb = xs[m];
        const double dx = xa.x - xb.x, dy = xa.y - xb.y;
        if (m != self && __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)) < thr)
            body(m, splat2((float)dx), splat2((float)dy), p.lane == 0, p.lane == 1);
    }
}
__device__ __forceinline__ bool all_finite() { return true; }
template <typename... R>
__device__ __forceinline__ bool all_finite(float v, R... rest) { return isfinite(v) && all_finite(rest...); }

// count_stats with the warp's integer reductions
__device__ __forceinline__ void count_stats_redux(DevCounters* cnt, int list, int phase_slot, int hits, bool valid) {
    const unsigned F = 0xffffffffu;
    const unsigned sum = __reduce_add_sync(F, valid ? (unsigned)hits : 0u);
    if (phase_slot < 0) {
        if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&cnt->pairs[list], (unsigned long long)sum);
        return;
    }
    const int hi = __reduce_max_sync(F, valid ? hits : 0);
    const int lo = __reduce_min_sync(F, valid ? hits : 0x7fffffff);
    const unsigned z = __reduce_add_sync(F, valid && hits == 0 ? 1u : 0u);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&cnt->pairs[list], (unsigned long long)sum);
        atomicMax(&cnt->maxiac[phase_slot], hi);
        atomicMin(&cnt->miniac[phase_slot], lo);
        if (z) atomicAdd(&cnt->noiac[phase_slot], (int)z);
    }
}

// ------------------------------------------------------ shared-memory staging
// The candidates of a block's particles in shared memory: positions and NB - 1
// record arrays (16-byte multiples), as stage_block, with one thread per copy.
template <int TPB, int NB>
__device__ __forceinline__ bool stage_pairs(StageHdr& H, const StageArrays<NB>& A, const GridGeom& g,
                                            const int* __restrict__ cstart, const double2* __restrict__ xs, int n, int cap,
                                            const LanePair& p, int* timeout) {
    const int tid = threadIdx.x;
    const int k0 = blockIdx.x * TPB;
    const int last = (k0 + TPB < n ? k0 + TPB : n) - 1 - k0;
    if (tid == 0) {
        H.row[0] = p.cy; H.xlo[0] = p.cx; H.xhi[0] = p.cx;
        H.bad = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&H.bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid == last) { H.row[1] = p.cy; H.xlo[1] = p.cx; H.xhi[1] = p.cx; }
    __syncthreads();
    if (p.valid) {
        const int row0 = H.row[0], row1 = H.row[1];
        if (p.cy == row0) atomicMax(&H.xhi[0], p.cx);
        else if (p.cy == row1) atomicMin(&H.xlo[1], p.cx);
        else H.bad = 1;
    }
    __syncthreads();
    if (tid < 32) {
        int gb = 0, len = 0;
        if (tid < 6) {
            const int part = tid / 3, y = H.row[part] + tid % 3 - 1;
            if ((part == 0 || H.row[1] != H.row[0]) && y >= 0 && y < g.ncy) {
                const int xl = H.xlo[part] - g.kx > 0 ? H.xlo[part] - g.kx : 0;
                const int xh = H.xhi[part] + g.kx < g.ncx - 1 ? H.xhi[part] + g.kx : g.ncx - 1;
                gb = cstart[y * g.ncx + xl];
                len = cstart[y * g.ncx + xh + 1] - gb;
            }
        }
        int off = len;   // inclusive scan over the six runs
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, off, d);
            if (tid >= d) off += v;
        }
        const int total = __shfl_sync(0xffffffffu, off, 5);
        off -= len;
        const int st = !H.bad && total <= cap;
        if (tid < 6) { H.gbeg[tid] = gb; H.len[tid] = len; H.soff[tid] = off; }
        if (tid == 0) {
            H.staged = st;
            if (st) {
                unsigned bytes = 0;
                for (int i = 0; i < NB; ++i) bytes += (unsigned)total * (unsigned)A.esize[i];
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&H.bar)), "r"(bytes)
                             : "memory");
            }
        }
        __syncwarp();
        if (st && tid < 6 && len > 0) {
#pragma unroll
            for (int i = 0; i < NB; ++i)
                bulk_copy_g2s((char*)A.dst[i] + (size_t)off * A.esize[i], (const char*)A.src[i] + (size_t)gb * A.esize[i],
                              (unsigned)len * (unsigned)A.esize[i], &H.bar);
        }
    }
    __syncthreads();
    if (!H.staged) return false;
    stage_wait(H, timeout);
    return true;
}

// runs in the staged arrays of particles in row cy, and the slot of the
// staged copy of sorted slot k in that row
__device__ __forceinline__ Runs3 staged_runs3(const StageHdr& H, Runs3 r, int cy) {
    const int j = cy == H.row[0] ? 0 : 3;
    r.b0 += H.soff[j] - H.gbeg[j];
    r.b1 += H.soff[j + 1] - H.gbeg[j + 1];
    r.b2 += H.soff[j + 2] - H.gbeg[j + 2];
    return r;
}
__device__ __forceinline__ int staged_slot(const StageHdr& H, int k, int cy) {
    const int j = cy == H.row[0] ? 1 : 4;
    return k + H.soff[j] - H.gbeg[j];
}
