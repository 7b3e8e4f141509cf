// sphg_kernels.cuh — the sm_100a kernels of libsphg.
//
// Per step (two-phase, declarations_sph.f90:525-791 with single_step :1131):
//   k_cell_count      cell key per particle, rank inside its cell         elementwise
//   k_cell_scatter    counting-sort scatter into cell order              elementwise
//   k_cell_sort       order each cell by original index (reorder steps; else in the gather)  per cell
//   k_gather          sorted copies: x, h, (v, m, rho) at the half step (the leapfrog predictor);
//                     soil: DP + stress pair pass inputs
//   k_water_sum       summation density (water-only step)                pair pass
//   k_water_pass_a    continuity / df2, delta-SPH(rho), strain rate, EOS  pair pass
//   k_water_pass_b    momentum, art. viscosity, delta-SPH(vof), wall force, XSPH  pair pass
//   k_soil_pass       every same-phase soil term + flow rule + Jaumann   pair pass
//   cross_soil_sums   Darcy drag + pore pressure on soil (in k_soil_pass) pair sums
//   cross_water_sums  Darcy drag, dvof, vof2 on water (in k_water_pass_b) pair sums
//   Corrector         leapfrog corrector / first step (+ DP on soil), in the last pass of each phase
// The FP32 passes of a step with soil and one h are in sphg_kernels2.cuh.
// Every pair pass is a gather: one thread per particle in cell order visits
// the 3 x 3 neighbouring cells (three contiguous row segments of the sorted
// list), evaluates the reference's pair test bit-exactly in FP64 and sums the
// particle's own side of each pair term.  The reference scatters each pair
// to both ends (e.g. m_particles.f90:2427-2428); the gather evaluates the pair
// once from each end, with the algebraically identical term, so the sums
// match the reference to rounding, and the pair set matches exactly.
#pragma once
#include "sphg_device.cuh"

struct SimConst {
    int skf, single_phase, summation_density, average_velocity, visc_artificial;
    int artificial_density, soil_artificial_stress, volume_fraction, water_artificial_volume;
    int volume_fraction_renorm, stress_integration, plasticity, yield_dp;
    int half;              // the step starts with the leapfrog predictor (not the first step or a right-hand side alone)
    int renorm_now;        // this step renormalises vof (itimestep % interval == 0)
    double gravity, numeric_gravity, alpha, beta, etq, dd, p1, p2, delta, epsilon, dt;
    double w_rho0, w_b, w_gamma, w_c, w_mu;
    double s_rho0, s_k, s_E, s_niu, s_c, s_perm, s_G, s_alpha1;
    double s_kb;           // permeability x Forchheimer b (0: linear Darcy)
    const SceneTab* tab;   // per-scene dt, water b and c, soil alpha1 (indexed by PhaseDev::sid)
};

#ifndef SPHG_TPB
#define SPHG_TPB 128
#endif
// Default x cells per neighbour cell (GridGeom::kx; sphg_tuning.x_split
// overrides it per context).  Step time on a B200 at 912,016 particles:
// 1: 0.596-0.603 ms, 2: 0.558-0.565, 3: 0.567, 4: 0.548 (the candidate
// strip narrows from 3 to 2.25 support radii; the pair set is the same).
#ifndef SPHG_X_SPLIT
#define SPHG_X_SPLIT 4
#endif
// minimum resident blocks per SM of each pair pass (register cap for the
// compiler: 65,536 / (SPHG_TPB * min blocks) registers per thread).  FP32: timed on a B200 at 912,016
// particles of one h, before those ran the paired passes; now for the water-only step and several h.
// water_pass_a (staged, recording the hit masks) 131 us at 8 blocks, 134 at
// 7, 138 at 10 (48 registers).  water_pass_b (replaying the masks, with the
// cross pairs) 176 us at 6 blocks, 164 at 7, 181 at 8 (spills).  soil_pass
// with the cross pairs: 86 us uncapped (128 registers), 91 at 5, 86 at 6.
#ifndef SPHG_MINB_A
#define SPHG_MINB_A 8
#endif
#ifndef SPHG_MINB_B
#define SPHG_MINB_B 7
#endif
// neighbours of one block of the two-phase water_pass_a (FP64 with one h) staged in shared
// memory (records; the sizes of 128 consecutive particles' candidate runs at
// dx = 0.002 m: mean 414, largest 544).  Each lane tests its candidates
// from there one at a time and runs the pair body on each hit at once
// (scan_direct): in FP32, which runs it paired now, 123.5 us per launch at 912,016 particles, against 130.7 us
// with the hit buffer that batches the bodies across the warp, and 130.4 us
// for the direct scan reading through L1.
#ifndef SPHG_STAGE_A
#define SPHG_STAGE_A 576
#endif
#ifndef SPHG_MINB_SOIL
#define SPHG_MINB_SOIL 1
#endif

// FP64, 912,016 particles: serial chains of FP64 operations, hidden by resident
// blocks.  water_pass_a 181 us uncapped, 184 at 5; water_pass_b 314 uncapped (166
// registers), 273 at 4; soil_pass 140 uncapped (214), 112 at 3.  One block more of
// either of the last two spills: 474 at 5 and 140 at 4, before the quotients'
// corrections.
#ifndef SPHG_MINB_A64
#define SPHG_MINB_A64 5
#endif
#ifndef SPHG_MINB_B64
#define SPHG_MINB_B64 4
#endif
#ifndef SPHG_MINB_S64
#define SPHG_MINB_S64 3
#endif

// launch the step's kernels with programmatic stream serialization (0: plain launches)
#ifndef SPHG_PDL
#define SPHG_PDL 1
#endif

__device__ __forceinline__ int gtid() { return blockIdx.x * blockDim.x + threadIdx.x; }

// Programmatic dependent launch: the step's kernels are launched so that the
// next one may start while this one finishes (Engine::launch_pdl).  A kernel
// lets its successor launch as soon as all of its own blocks have started,
// and waits for its predecessor's results before touching any memory.
// Launched without the attribute, both are no-ops.
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ----------------------------------------------------------------- cell list
// Cell key (row-major) of a particle at p and its rank inside its cell; the
// clamped and non-finite positions are counted into the step's counters, or
// into the next step's (next != 0).
__device__ __forceinline__ void cell_key(const GridGeom& g, double2 p, int a, int* __restrict__ cell_id,
                                         int* __restrict__ rank, int* __restrict__ counts, DevCounters* cnt, int next) {
    int cx, cy; bool clamped;
    cell_coords(g, p.x, p.y, cx, cy, clamped);
    if (clamped) atomicAdd(next ? &cnt->n_out_next : &cnt->n_out, 1);
    if (!(isfinite(p.x) && isfinite(p.y))) atomicAdd(next ? &cnt->nonfinite_next : &cnt->nonfinite, 1);
    const int c = cy * g.ncx + cx;
    cell_id[a] = c;
    rank[a] = atomicAdd(counts + c, 1);
}

static __global__ void __launch_bounds__(256) k_cell_count(const double2* __restrict__ x, int n, GridGeom g,
                                                    int* __restrict__ cell_id, int* __restrict__ rank,
                                                    int* __restrict__ counts, DevCounters* cnt, int next) {
    pdl_enter();
    int a = gtid();
    if (a >= n) return;
    cell_key(g, x[a], a, cell_id, rank, counts, cnt, next);
}

// Exclusive scan of the cells' counts, start[ncell] = the total: each block
// scans a chunk of kScanChunk counts on top of the sum of all counts before it,
// taken from the chunk sums of k_cell_sums or, for few cells, from the counts
// themselves (one launch instead of two).  us per step with and without the chunk
// sums: 3.5k cells 30.6, 30.2; 15k 22.1, 22.4; 28k 24.0, 25.2; 52k 26.3, 29.4;
// 100k 28.3, 34.3: the line is 16k.  Bound: launches and
// their latency.  With the cells ordered inside the gather and the counters
// reset by the step's check, us per step before and after: 7.4k particles 33.4,
// 28.4; 150k 95, 91; 190k 77, 70; 330k 172, 165; 912k 325, 316; the ensemble's
// dry group 121, 104.
// Above kSumsDirect chunks the blocks' reads of all sums before theirs, which grow
// with the square of the cells, cost more than a launch that scans the sums:
// us per step of 6.6k particles without and with it, 4M cells 34.0, 34.5; 8M 45.5,
// 45.5; 16M 71.0, 69.7; 69M 284, 238; 180M 1,020, 573.  Bound there: HBM, four
// passes over the cells (counts read twice and cleared, starts written).
constexpr int kScanChunk = 2048;
constexpr int kScanDirect = 16 * 1024;   // cells up to which a block adds up the counts before it
constexpr int kSumsDirect = 4096;        // chunks up to which a block adds up the chunk sums before it; above, one block scans them first
__device__ __forceinline__ int block_sum256(int v) {
    __shared__ int part[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    int t = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += part[w];
    return t;
}
static __global__ void __launch_bounds__(256) k_cell_sums(const int* __restrict__ counts, int ncell, int* __restrict__ sums) {
    pdl_enter();
    const int b = blockIdx.x * kScanChunk;
    int v = 0;
#pragma unroll
    for (int q = 0; q < kScanChunk / 256; ++q) {
        const int i = b + q * 256 + threadIdx.x;
        if (i < ncell) v += counts[i];
    }
    v = block_sum256(v);
    if (threadIdx.x == 0) sums[blockIdx.x] = v;
}
// The chunk sums replaced by the sum of all sums before each, by one block, 4,096 at a time.
static __global__ void __launch_bounds__(1024) k_sums_scan(int* __restrict__ sums, int n) {
    pdl_enter();
    __shared__ int warp_tot[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int carry = 0;
    for (int b = 0; b < n; b += 4096) {
        const int i0 = b + tid * 4;
        int v[4], own = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) { v[q] = i0 + q < n ? sums[i0 + q] : 0; own += v[q]; }
        int inc = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (lane == 31) warp_tot[warp] = inc;
        __syncthreads();
        int w = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += u;
        }
        int run = carry + inc - own + (warp ? __shfl_sync(0xffffffffu, w, warp - 1) : 0);
        carry += __shfl_sync(0xffffffffu, w, 31);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (i0 + q < n) sums[i0 + q] = run;
            run += v[q];
        }
        __syncthreads();   // warp_tot is read before the next tile's sums replace it
    }
}
// sums: null, or the chunk sums (scanned: already scanned by k_sums_scan)
static __global__ void __launch_bounds__(256) k_cell_scan(const int* __restrict__ counts, int ncell, int* __restrict__ start,
                                                          const int* __restrict__ sums, int scanned) {
    pdl_enter();
    const int b = blockIdx.x * kScanChunk, tid = threadIdx.x;
    int before = 0;
    if (sums && scanned) before = tid == 0 ? sums[blockIdx.x] : 0;
    else if (sums) for (int i = tid; i < (int)blockIdx.x; i += 256) before += sums[i];
    else {
#pragma unroll 4
        for (int i = tid; i < b / 4; i += 256) {
            const int4 u = reinterpret_cast<const int4*>(counts)[i];
            before += u.x + u.y + u.z + u.w;
        }
    }
    constexpr int PER = kScanChunk / 256;   // 8: two 16-byte accesses per thread
    const int i0 = b + tid * PER;
    int v[PER], own = 0;
    if (i0 + PER <= ncell) {
        const int4 u = reinterpret_cast<const int4*>(counts + i0)[0], w = reinterpret_cast<const int4*>(counts + i0)[1];
        v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w; v[4] = w.x; v[5] = w.y; v[6] = w.z; v[7] = w.w;
    } else {
#pragma unroll
        for (int q = 0; q < PER; ++q) v[q] = i0 + q < ncell ? counts[i0 + q] : 0;
    }
#pragma unroll
    for (int q = 0; q < PER; ++q) own += v[q];
    before = block_sum256(before);
    // inclusive scan of the threads' sums
    __shared__ int warp_tot[8];
    int inc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, inc, o);
        if ((tid & 31) >= o) inc += u;
    }
    if ((tid & 31) == 31) warp_tot[tid >> 5] = inc;
    __syncthreads();
    int run = before + inc - own;
    for (int w = 0; w < (tid >> 5); ++w) run += warp_tot[w];
    if (i0 + PER < ncell) {
        int o[PER];
#pragma unroll
        for (int q = 0; q < PER; ++q) { o[q] = run; run += v[q]; }
        reinterpret_cast<int4*>(start + i0)[0] = make_int4(o[0], o[1], o[2], o[3]);
        reinterpret_cast<int4*>(start + i0)[1] = make_int4(o[4], o[5], o[6], o[7]);
    } else {
        for (int q = 0; q < PER && i0 + q < ncell; ++q) {
            start[i0 + q] = run;
            run += v[q];
            if (i0 + q + 1 == ncell) start[ncell] = run;
        }
    }
}

// Also resets the cells' counts, consumed by the scan, for the corrector, which
// counts the next step's cells (counts may be null).  The grid has a thread per
// particle and, for grids of many more cells, one per 16 cells: cleared by the
// particles' blocks alone, a step of 6.6k particles took 28.8 us at 1M cells and
// 143 at 16M; with these, 26.4 and 69.7.  (One thread per 4 cells changes the
// small steps' block counts, and with them where the next passes' blocks land:
// 32.4 us for the FP32 step of 6.6k particles instead of 28.8.)
static __global__ void __launch_bounds__(256) k_cell_scatter(int n, const int* __restrict__ cell_id, const int* __restrict__ rank,
                                                      const int* __restrict__ cell_start, int* __restrict__ perm,
                                                      int* __restrict__ counts, int ncell) {
    pdl_enter();
    int a = gtid();
    if (a < n) perm[cell_start[cell_id[a]] + rank[a]] = a;
    if (counts)
        for (int c = a; c < ncell; c += gridDim.x * blockDim.x) counts[c] = 0;
}

// Insertion sort of each cell's (few) entries by original particle index, so
// the visiting order, and with it every sum, depends neither on atomic timing
// nor on the current state order (a download/upload restart is bit-identical).
// A step without a reorder leaves this to the gather (sorted_slot).
static __global__ void __launch_bounds__(256) k_cell_sort(int ncell, const int* __restrict__ cell_start,
                                                   const int* __restrict__ orig, int* __restrict__ perm) {
    pdl_enter();
    int c = gtid();
    if (c >= ncell) return;
    int b = cell_start[c], e = cell_start[c + 1];
    for (int i = b + 1; i < e; ++i) {
        int v = perm[i], ov = orig[v], j = i - 1;
        while (j >= b && orig[perm[j]] > ov) { perm[j + 1] = perm[j]; --j; }
        perm[j + 1] = v;
    }
}

// Sorted slot of the particle a, from the scattered cell list: its cell's first
// slot plus the number of the cell's particles with a lower original index.
__device__ __forceinline__ int sorted_slot(const int* __restrict__ scattered, const int* __restrict__ cell_id,
                                           const int* __restrict__ cell_start, const int* __restrict__ orig, int a) {
    const int c = cell_id[a], b = cell_start[c], e = cell_start[c + 1];
    if (e - b == 1) return b;
    const int o = orig[a];
    int t = b;
    for (int i = b; i < e; ++i) t += orig[scattered[i]] < o;
    return t;
}

// ------------------------------------------------------------- integrators
// What the last pass of a phase does after its sums: nothing (right-hand side
// only, sphg_single_step) or the leapfrog corrector of this step.
struct StepCtl {
    int update;      // run the corrector (first_step or second_half)
    int first;       // itimestep == 1: first_step
    int with_vof;    // integrate the water volume fraction (two-phase)
    int do_dp;       // Drucker-Prager after the corrector (soil)
    int* ncount;     // non-null: after the corrector, the cell key and rank of the new position, counted
                     // into this phase's per-cell counts for the next step's cell list
};

// first_half, declarations_sph.f90:643-684 (and :812-825, :998-1025).  The
// half-step rho, vof and v are r + dt/2 * rate of the state and the rates of the
// step before, which stay in place until the corrector; they are formed where
// they are needed (the gather, water_pass_a, soil_finish) and never stored, and
// the corrector keeps the full-step values as rho_min, vof_min and v_min.
template <typename T>
__device__ __forceinline__ double half_step(double r, double dt, T rate) { return r + (dt / 2.0) * (double)rate; }

// The stress part of first_half on soil (stress_integration 2) and the
// Drucker-Prager call that follows it (:559, :1027).  Returns its fail flag.
template <typename T>
__device__ __forceinline__ int first_half_stress(const PhaseDev<T>& P, int a, const SimConst& c, const SceneTab& st, int do_dp,
                                                 double& p, double& sxx, double& sxy, double& syy) {
    if (c.stress_integration == 2) {
        const T d0 = P.dsxx[a], d1 = P.dsxy[a], d2 = P.dsyy[a], d3 = P.dp[a];
        P.sxx_min[a] = sxx; P.sxy_min[a] = sxy; P.syy_min[a] = syy; P.p_min[a] = p;
        sxx = half_step(sxx, st.dt, d0);
        sxy = half_step(sxy, st.dt, d1);
        syy = half_step(syy, st.dt, d2);
        p = half_step(p, st.dt, d3);
    }
    return do_dp ? dp_return(p, sxx, sxy, syy, st.s_alpha1) : 0;
}

// The corrector: first_step (:686-723) when first != 0, else second_half
// (:725-762), plus the Drucker-Prager call after it on soil (:583, :601,
// :1069, :1107).  load() reads all of the particle's state it needs before any
// result of the pass is stored (the stores could alias the loads, so reading
// field by field between them made each load wait for the one before: the
// last passes spent half their time so); apply() integrates and stores.
template <typename T>
struct Corrector {
    typedef typename V2<T>::t T2;
    double dt, rho, vof, alpha1, p, sxx, sxy, syy;
    double2 v, x;
    T drho;
    bool real;
    __device__ __forceinline__ void load(const PhaseDev<T>& P, int a, const SimConst& c, const StepCtl& u, bool soil) {
        const int sid = P.sid[a];
        real = P.itype[a] >= 0;
        x = P.x[a];
        v = P.v[a];
        rho = c.single_phase && !soil && !u.first ? P.rho_min[a] : P.rho[a];   // the water-only sum has replaced rho
        if (!soil) {
            drho = P.drho[a];
            vof = P.vof[a];
        } else if (c.stress_integration == 2 && !u.first) {
            p = P.p_min[a]; sxx = P.sxx_min[a]; sxy = P.sxy_min[a]; syy = P.syy_min[a];
        } else {
            p = P.p[a]; sxx = P.sxx[a]; sxy = P.sxy[a]; syy = P.syy[a];
        }
        dt = c.tab[sid].dt;
        alpha1 = soil ? c.tab[sid].s_alpha1 : 0.0;
    }
    // rho and v, x; the new position
    __device__ __forceinline__ void move(const PhaseDev<T>& P, int a, const SimConst& c, int first, T2 d, T2 av) {
        const double h = first ? dt / 2.0 : dt;
        if (!c.summation_density) {
            if (!first) P.rho_min[a] = rho;
            P.rho[a] = rho + h * (double)drho;
        }
        if (real) {
            if (!first) P.v_min[a] = v;
            v.x = v.x + h * (double)d.x + (double)av.x;
            x.x = x.x + dt * v.x;
            v.y = v.y + h * (double)d.y + (double)av.y;
            x.y = x.y + dt * v.y;
            P.v[a] = v;
            P.x[a] = x;
        }
    }
    __device__ __forceinline__ int stress(const PhaseDev<T>& P, int a, const SimConst& c, int first, int do_dp, T dsxx, T dsxy,
                                          T dsyy, T dp) {
        const double h = c.stress_integration == 1 ? dt : first ? dt / 2.0 : dt;
        sxx = sxx + h * (double)dsxx;
        sxy = sxy + h * (double)dsxy;
        syy = syy + h * (double)dsyy;
        p = p + h * (double)dp;
        int fail = 0;
        if (do_dp) { fail = dp_return(p, sxx, sxy, syy, alpha1); P.fail[a] = fail; }
        P.p[a] = p; P.sxx[a] = sxx; P.sxy[a] = sxy; P.syy[a] = syy;
        return fail;
    }
};

__device__ __forceinline__ void count_fail(DevCounters* cnt, int slot, int fail) {
    int s = __syncthreads_count(fail);
    if (threadIdx.x == 0 && s) atomicAdd(&cnt->nfail[slot], s);
}

// ------------------------------------------------------------------ gathers
// Sorted copies of position, h (with_hs: not needed when every h is equal) and
// (v, vol, rho).  With fh != 0 the records carry the half-step state of the
// leapfrog predictor (first_half, + DP on soil).  For soil also the in-step
// Drucker-Prager return (declarations_sph.f90:1242-1247) on the state and the
// stress/pressure record of the soil pass.  Bound by DRAM: it reads and writes
// each field once, with every load before the first store.  scattered: the
// cell list before its cells are ordered; the gather then finds each
// particle's slot itself and writes perm, which saves the sort's launch and pass
// over the cells.  Storing the half
// step as well (and reading it back in the corrector) took 53 us for the two
// phases of 912,016 particles instead of 34, and the step 345 us instead of
// 322; 5, 6 and 8 resident blocks spill and take 33, 36 and 38 us.
template <typename T>
__global__ void __launch_bounds__(256, 4) k_gather(PhaseDev<T> P, SimConst c, int soil, int do_dp, int fh, int with_hs,
                                                int fh_dp, DevCounters* cnt, const int* __restrict__ scattered) {
    pdl_enter();
    int k = gtid();
    int fail0 = 0, fail = 0;
    if (k < P.n) {
        const int a = scattered ? k : P.perm[k];   // by particle, which reads the state in order, or by slot
        const double2 x = P.x[a];
        double2 v = P.v[a];
        double rho = P.rho[a];
        const double mass = P.mass[a], h = with_hs ? P.hsml[a] : 0.0;
        const int sid = soil || fh ? P.sid[a] : 0, itype = soil || fh ? P.itype[a] : 0;
        const SceneTab& st = c.tab[sid];
        if (scattered) k = sorted_slot(scattered, P.cell_id, P.cell_start, P.orig, a);
        double p = 0.0, sxx = 0.0, sxy = 0.0, syy = 0.0, cc = 0.0, vof = 0.0;
        if (soil) { p = P.p[a]; sxx = P.sxx[a]; sxy = P.sxy[a]; syy = P.syy[a]; cc = P.c[a]; vof = P.vof[a]; }
        if (fh) {
            const T drho = P.drho[a];
            const typename V2<T>::t d = P.dv[a];
            if (!c.summation_density) rho = half_step(rho, st.dt, drho);
            if (itype >= 0) { v.x = half_step(v.x, st.dt, d.x); v.y = half_step(v.y, st.dt, d.y); }
            if (soil) fail0 = first_half_stress(P, a, c, st, fh_dp, p, sxx, sxy, syy);
        }
        if (soil) {
            if (do_dp) fail = dp_return(p, sxx, sxy, syy, st.s_alpha1);
            if (fh || do_dp) { P.p[a] = p; P.sxx[a] = sxx; P.sxy[a] = sxy; P.syy[a] = syy; }
            if (do_dp) P.fail[a] = fail;
            else if (fh && fh_dp) P.fail[a] = fail0;
            RecB<T> rb;
            rb.p = (T)p; rb.c = (T)cc; rb.vof = (T)vof;
            rb.sxx = (T)sxx; rb.sxy = (T)sxy; rb.syy = (T)syy;
            rb.itype = (T)itype; rb.aux = T(0);
            P.recB[k] = rb;
        }
        if (scattered) P.perm[k] = a;
        P.xs[k] = x;
        if (with_hs) P.hs[k] = h;
        RecA<T> ra;
        ra.vx = (T)v.x; ra.vy = (T)v.y; ra.vol = (T)(mass / rho); ra.rho = (T)rho;
        P.recA[k] = ra;
    }
    if (fh && fh_dp) count_fail(cnt, 0, fail0);
    if (soil && do_dp) count_fail(cnt, 1, fail);
}

// Per-particle interaction statistics (interaction_statistics,
// m_particles.f90:555-597) and the pair count of the list.
__device__ __forceinline__ void count_stats(DevCounters* cnt, int list, int phase_slot, int hits, bool valid) {
    unsigned long long h = valid ? (unsigned long long)hits : 0ull;
    int hmax = valid ? hits : 0, hmin = valid ? hits : 0x7fffffff, hz = (valid && hits == 0) ? 1 : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        h += __shfl_xor_sync(0xffffffffu, h, o);
        hmax = max(hmax, __shfl_xor_sync(0xffffffffu, hmax, o));
        hmin = min(hmin, __shfl_xor_sync(0xffffffffu, hmin, o));
        hz += __shfl_xor_sync(0xffffffffu, hz, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&cnt->pairs[list], h);
        if (phase_slot >= 0) {
            atomicMax(&cnt->maxiac[phase_slot], hmax);
            atomicMin(&cnt->miniac[phase_slot], hmin);
            if (hz) atomicAdd(&cnt->noiac[phase_slot], hz);
        }
    }
}

// hit-buffer depth per thread: 24 covers the ~20 neighbours of a particle at
// support 2h = 2.4 dx in one drain (FP32); FP64 entries are larger.
template <typename T> struct Chunk { static const int value = sizeof(T) == 4 ? 24 : 16; };
#define SPHG_HITBUF(T) __shared__ HitBuf<T, SPHG_TPB, Chunk<T>::value> hb
// (one entry when the pass does not use it)
#define SPHG_HITBUF_G(T, G) __shared__ HitBuf<T, (G) == 1 ? SPHG_TPB : 1, (G) == 1 ? Chunk<T>::value : 1> hb

// Kernel constants for particle a: per particle when every h is equal, else
// per pair (mhsml = (h_a + h_b)/2).
template <typename T, int SKF>
__device__ __forceinline__ void pair_kernel(const KernelConst<T, SKF>& ka, const SearchConst& sc, double ha,
                                            const double* __restrict__ hs, int m, T dx, T dy, T& w, T& s, T& r2,
                                            T& mh) {
    r2 = sqsum<T>(dx, dy);
    if (sc.uniform) {
        ka.eval(r2, w, s);
        mh = ka.h;
    } else {
        KernelConst<T, SKF> kb;
        const double mhd = (ha + hs[m]) / 2.0;
        kb.init((T)mhd);
        kb.eval(r2, w, s);
        mh = (T)mhd;
    }
}

// ------------------------------------------------------ water: summation rho
// sum_density (m_particles.f90:2243-2298) and the df2 divergence of the
// water-only step, drho = -rho*(df2(vx,'x') + df2(vy,'y'))
// (declarations_sph.f90:1465-1466, df2 m_particles.f90:1802-1831).
template <typename T>
__device__ __forceinline__ void water_sum_finish(const PhaseDev<T>& P, const SimConst& c, int k, const RecA<T>& ra, T num, T wi,
                                                 T sx, T sy, int hits) {
    const int a = P.perm[k];
    const T rho = num / wi;
    const double mass = P.mass[a];
    if (c.half && !c.summation_density) P.rho_min[a] = P.rho[a];   // the corrector integrates from it
    P.rho[a] = (double)rho;
    P.drho[a] = -rho * (sx / rho + sy / rho);
    RecA<T> r2;
    r2.vx = ra.vx; r2.vy = ra.vy; r2.vol = (T)(mass / (double)rho); r2.rho = rho;
    P.recA2[k] = r2;
    P.countiac[a] = hits;
}

// G > 1: G lanes per particle (scan_lanes), no hit masks.
template <typename T, int SKF, int G = 1>
__global__ void __launch_bounds__(SPHG_TPB) k_water_sum(PhaseDev<T> P, GridGeom g, SearchConst sc, SimConst c, DevCounters* cnt) {
    pdl_enter();
    const int k = gtid() / G;
    const bool valid = k < P.n;
    const int kk = valid ? k : 0;
    const double2 xa = P.xs[kk];
    const double ha = P.hs[kk];
    const RecA<T> ra = P.recA[kk];
    KernelConst<T, SKF> ka;
    ka.init((T)ha);
    T w0, s0;
    ka.eval(T(0), w0, s0);
    const T ma = ra.vol * ra.rho;
    T wi = w0 * ma / ra.rho;
    T num = w0 * ma;
    T sx = T(0), sy = T(0);
    const RecA<T>* __restrict__ rec = P.recA;
    uint4 mask;
    auto body = [&](int m, T dx, T dy) {
        const RecA<T> rb = rec[m];
        T w, sr, r2, mh;
        pair_kernel<T, SKF>(ka, sc, ha, P.hs, m, dx, dy, w, sr, r2, mh);
        const T mb = rb.vol * rb.rho;
        wi += rb.vol * w;
        num += mb * w;
        sx += mb * ((rb.vx - ra.vx) * (sr * dx));
        sy += mb * ((rb.vy - ra.vy) * (sr * dy));
    };
    int hits;
    bool finish = valid;
    if constexpr (G == 1) {
        SPHG_HITBUF(T);
        hits = visit_batched_rec(hb, g, sc, P.cell_start, P.xs, P.hs, xa, ha, k, valid, mask, body);
        if (valid && P.hmask) P.hmask[k] = mask;
    } else {
        finish = valid && threadIdx.x % G == 0;
        if (threadIdx.x % G) { wi = T(0); num = T(0); }
        hits = scan_lanes<G, T>(sc, candidate_runs(g, P.cell_start, xa, valid), P.xs, P.hs, xa, ha, k, body);
        lanes_sum<G>(wi, num, sx, sy, hits);
    }
    if (finish) water_sum_finish(P, c, k, ra, num, wi, sx, sy, hits);
    count_stats(cnt, 0, 0, hits, finish);
}

// A particle's own density in the mean densities of the FP64 passes: an infinite
// one as 1e200, whose reciprocal is zero for every purpose and has a residual.
template <typename T> __device__ __forceinline__ T finite_rho(T rho) { return sizeof(T) == 8 && rho > T(1e200) ? T(1e200) : rho; }

// The powers of the Tait equation, r^gamma - 1, and of the sound speed, r^3.  FP64
// calls pow, as the reference does.  The single-precision mode (whose equation
// of state is in FP64 all the same) takes gamma = 7, the exponent of water, and the cube
// as products with their rounding errors carried along: no further from the
// exact value than pow, which took 250 instructions a call (an eighth of its
// water_pass_a's).  Infinite products stand alone (their errors are NaN).
template <typename T>
__device__ __forceinline__ double cube(double r) {
    if (sizeof(T) == 8) return pow(r, 3.0);
    const double r2 = r * r, r3 = r2 * r;
    if (isinf(r3)) return r3;
    return r3 + (fma(r2, r, -r3) + fma(r, r, -r2) * r);
}
template <typename T>
__device__ __forceinline__ double tait(double r, double gamma) {
    if (sizeof(T) == 8 || gamma != 7.0) return pow(r, gamma) - 1;
    const double r2 = r * r, e2 = fma(r, r, -r2);
    const double r3 = r2 * r, e3 = fma(r2, r, -r3) + e2 * r;
    const double r6 = r3 * r3, e6 = fma(r3, r3, -r6) + 2.0 * r3 * e3;
    const double r7 = r6 * r, e7 = fma(r6, r, -r7) + e6 * r;
    return isinf(r7) ? r7 : (r7 - 1.0) + e7;
}

// What water_pass_a does with a particle's sums: EOS, newtonian_fluid, the
// record of the next pass, the interaction count.
template <typename T, bool SINGLE>
__device__ __forceinline__ void water_a_finish(const PhaseDev<T>& P, const SimConst& c, int k, T con, T dl, T t0, T t1, T t2,
                                               T t3, int hits) {
    const T c23 = (T)SPHG_F32LIT(2.0f / 3.0f);
    const int a = P.perm[k];
    T txx, txy, tyy, drho;
    double p, cnew, vof;
    // every load before the first store
    double rho = P.rho[a];
    const int sid = P.sid[a], itype = P.itype[a];
    if (SINGLE) {
        const double pold = P.p[a];
        cnew = P.c[a];
        drho = P.drho[a] + dl;
        txx = c23 * (T(2) * t0 - t1);
        txy = t2 + t3;
        tyy = c23 * (T(2) * t1 - t0);
        p = rho > 0.0 ? c.tab[sid].w_b * tait<T>(rho / c.w_rho0, c.w_gamma) : pold;
        vof = 1.0;
    } else {
        drho = con + dl;
        txx = t0; txy = t1; tyy = t2;
        vof = P.vof[a];
        const T dold = c.half ? P.drho[a] : T(0), fold = c.half && c.volume_fraction ? P.dvof[a] : T(0);
        const SceneTab& st = c.tab[sid];
        if (c.half) {
            rho = half_step(rho, st.dt, dold);
            if (c.volume_fraction) vof = half_step(vof, st.dt, fold);
        }
        const double ratio = rho / (c.w_rho0 * vof);
        p = st.w_b * tait<T>(ratio, c.w_gamma);
        cnew = st.w_c * cube<T>(ratio);
        P.c[a] = cnew;
    }
    P.drho[a] = drho;
    P.p[a] = p;
    // newtonian_fluid: sxx = mu*txx in place (sxx and txx are one array)
    const double sxx = c.w_mu * (double)txx, sxy = c.w_mu * (double)txy, syy = c.w_mu * (double)tyy;
    P.sxx[a] = sxx; P.sxy[a] = sxy; P.syy[a] = syy;
    RecB<T> rb;
    rb.p = (T)p; rb.c = (T)cnew; rb.vof = (T)vof;
    rb.sxx = (T)sxx; rb.sxy = (T)sxy; rb.syy = (T)syy;
    rb.itype = (T)itype; rb.aux = T(0);
    P.recB[k] = rb;
    if (!SINGLE) P.countiac[a] = hits;
}

// ----------------------------------------------------------- water: pass A
// Two-phase (SINGLE = false), declarations_sph.f90:1195-1233:
//   con_density :2402, delta_sph(rho) :2658, shear_strain_rate :2855,
//   pressure :2133 (Tait with vof, c ~ (rho/rho0 vof)^3), newtonian_fluid :2484.
// Water-only (SINGLE = true), declarations_sph.f90:1471-1490:
//   delta_sph on the summation density, Tait without vof, t = df(v) form.
// delta_sph's (dx . grad W) 2 (f_a - f_b) / r^2 is evaluated as 2 s (f_a - f_b)
// since grad W = s dx.
// G as in k_water_sum.
template <typename T, int SKF, bool SINGLE, int G = 1>
__global__ void __launch_bounds__(SPHG_TPB, sizeof(T) == 4 ? SPHG_MINB_A : SPHG_MINB_A64) k_water_pass_a(PhaseDev<T> P, GridGeom g, SearchConst sc, SimConst c, DevCounters* cnt) {
    pdl_enter();
    const int k = gtid() / G;
    const bool valid = k < P.n;
    const int kk = valid ? k : 0;
    const int a = P.perm[kk];
    const double2 xa = P.xs[kk];
    const double ha = P.hs[kk];
    const RecA<T>* __restrict__ rec = SINGLE ? P.recA2 : P.recA;
    const RecA<T> ra = rec[kk];
    const T pref = (T)(c.delta * ha * P.c[a]);   // delta*hsml(i)*c(i), c of the previous EOS call
    const T c23 = (T)SPHG_F32LIT(2.0f / 3.0f);
    const bool dens = c.artificial_density;
    KernelConst<T, SKF> ka;
    ka.init((T)ha);
    T con = 0, dl = 0, t0 = 0, t1 = 0, t2 = 0, t3 = 0;
    uint4 mask = make_uint4(0u, 0u, 0u, 0u);
    if (SINGLE && G == 1 && valid) mask = P.hmask[k];   // recorded by k_water_sum
    auto body = [&](const RecA<T>* R, int m, T dx, T dy) {
        const RecA<T> rb = R[m];
        T w, sr, r2, mh;
        pair_kernel<T, SKF>(ka, sc, ha, P.hs, m, dx, dy, w, sr, r2, mh);
        const T gx = sr * dx, gy = sr * dy;
        if (!SINGLE) con += (rb.vol * rb.rho) * ((ra.vx - rb.vx) * gx + (ra.vy - rb.vy) * gy);
        if (dens) dl += pref * rb.vol * ((ra.rho - rb.rho) * (T(2) * sr));
        if (SINGLE) {   // df(vx,'x'), df(vy,'y'), df(vx,'y'), df(vy,'x')
            const T su = ra.vx + rb.vx, sv = ra.vy + rb.vy;
            t0 += rb.vol * (su * gx);
            t1 += rb.vol * (sv * gy);
            t2 += rb.vol * (su * gy);
            t3 += rb.vol * (sv * gx);
        } else {        // shear_strain_rate, dv = v_b - v_a
            const T du = rb.vx - ra.vx, dv = rb.vy - ra.vy;
            t0 += rb.vol * (c23 * (T(2) * du * gx - dv * gy));
            t1 += rb.vol * (du * gy + dv * gx);
            t2 += rb.vol * (c23 * (T(2) * dv * gy - du * gx));
        }
    };
    int hits;
    bool finish = valid;
    if constexpr (G > 1) {
        finish = valid && threadIdx.x % G == 0;
        hits = scan_lanes<G, T>(sc, candidate_runs(g, P.cell_start, xa, valid), P.xs, P.hs, xa, ha, k,
                                [&](int m, T dx, T dy) { body(rec, m, dx, dy); });
        lanes_sum<G>(con, dl, t0, t1, t2, t3, hits);
    } else if constexpr (SINGLE) {
        hits = visit_masked<T>(g, sc, P.cell_start, P.xs, P.hs, xa, ha, k, valid, mask,
                               [&](int m, T dx, T dy) { body(rec, m, dx, dy); });
    } else {
        // neighbours staged in shared memory when they fit (positions and records)
        extern __shared__ __align__(128) unsigned char stage_mem[];
        __shared__ StageHdr H;
        const int cap = stage_capacity(16 + (int)sizeof(RecA<T>));
        int cx, cy;
        bool cl;
        cell_coords(g, xa.x, xa.y, cx, cy, cl);
        const CandRuns cr = candidate_runs(g, P.cell_start, xa, valid);
        StageArrays<2> A;
        A.src[0] = P.xs; A.dst[0] = stage_mem; A.esize[0] = 16;
        A.src[1] = rec; A.dst[1] = stage_mem + (size_t)cap * 16; A.esize[1] = (int)sizeof(RecA<T>);
        if (cap > 0 && stage_block<SPHG_TPB, 2>(H, A, g, P.cell_start, P.xs, P.n, cap, sc.uniform, cx, cy, valid,
                                                 &cnt->timeout)) {
            int self_s;
            const CandRuns sr = staged_runs(H, cr, cy, k, self_s);
            const double2* sxs = (const double2*)stage_mem;
            const RecA<T>* sA = (const RecA<T>*)(stage_mem + (size_t)cap * 16);
            hits = scan_direct<true, T>(sc, sr, sxs, P.hs, xa, ha, self_s, mask,
                                        [&](int m, T dx, T dy) { body(sA, m, dx, dy); });
        } else {   // rare: the block's runs do not fit
            hits = scan_direct<true, T>(sc, cr, P.xs, P.hs, xa, ha, k, mask,
                                        [&](int m, T dx, T dy) { body(rec, m, dx, dy); });
        }
    }
    if (finish) {
        if (!SINGLE && G == 1) P.hmask[k] = mask;
        water_a_finish<T, SINGLE>(P, c, k, con, dl, t0, t1, t2, t3, hits);
    }
    if (!SINGLE) count_stats(cnt, 0, 0, hits, finish);
}

// ------------------------------------------------------------- cross phase
// Neighbour sums over the water x soil pairs (direct_find_2
// m_particles.f90:1004), run inside the last same-phase pass of each phase.
// Neighbours come from the other phase's records of this step.  FCH: the
// Forchheimer drag, each pair's Darcy term scaled by (1 + k b |v_w - v_s|).
//
// Soil side: darcy_law :3832 and pore_water_pressure :3877; the gradient is
// taken, as the reference does, with dx = x_water - x_soil.  With m =
// vol*rho, Darcy's m_w*cf*(v_w - v_s)*W/(rho_w rho_s) becomes
// vol_w*rho_w*vof_w*vof_s*(-g/k)*(v_w - v_s)*W/rho_s; the sums here are the
// pair parts, the particle factors are applied by the caller.  The pore
// pressure m_w p_w/(rho_w rho_s) becomes vol_w p_w / rho_s.
template <typename T, int SKF, bool FCH, class V>
__device__ __forceinline__ void cross_soil_sums(V&& visit, const PhaseDev<T>& W, const SearchConst& sc,
                                                const SimConst& c, const KernelConst<T, SKF>& ka, double ha,
                                                const RecA<T>& ra, T& ddx, T& ddy, T& dpx, T& dpy) {
    visit([&](int m, T dx, T dy) {
        const RecA<T> rb = W.recA[m];
        const RecB<T> qb = W.recB[m];
        T w, sr, rr, mh;
        pair_kernel<T, SKF>(ka, sc, ha, W.hs, m, dx, dy, w, sr, rr, mh);
        // x_water - x_soil = -(x_a - x_b)
        const T gx = -sr * dx, gy = -sr * dy;
        T q = rb.vol * rb.rho * qb.vof * w;
        const T ux = rb.vx - ra.vx, uy = rb.vy - ra.vy;
        if constexpr (FCH) q *= T(1) + (T)c.s_kb * sqrt(ux * ux + uy * uy);
        ddx += q * ux;
        ddy += q * uy;
        const T mp = rb.vol * qb.p;
        dpx += mp * gx;
        dpy += mp * gy;
    });
}

// Water side: darcy_law :3832, volume_fraction_water2 :3940 (dvof) and
// volume_fraction_water :3912 (vof2).  Returns the number of pairs.
template <typename T, int SKF, bool FCH, class V>
__device__ __forceinline__ int cross_water_sums(V&& visit, const PhaseDev<T>& S, const SearchConst& sc,
                                                const SimConst& c, const KernelConst<T, SKF>& ka, double ha,
                                                const RecA<T>& ra, T& ddx, T& ddy, T& dvof, T& v2) {
    return visit([&](int m, T dx, T dy) {
        const RecA<T> rb = S.recA[m];
        const T phis = S.recB[m].vof;
        T w, sr, rr, mh;
        pair_kernel<T, SKF>(ka, sc, ha, S.hs, m, dx, dy, w, sr, rr, mh);
        const T mb = rb.vol * rb.rho;
        const T ux = ra.vx - rb.vx, uy = ra.vy - rb.vy;
        T q = rb.vol * phis * w;
        if constexpr (FCH) q *= T(1) + (T)c.s_kb * sqrt(ux * ux + uy * uy);
        ddx -= q * ux;
        ddy -= q * uy;
        dvof -= mb * (sr * (ux * dx + uy * dy));
        v2 += mb * w;
    });
}

// A water particle's sums of water_pass_b: momentum (before the division by
// rho), artificial viscosity plus wall force, XSPH, delta-SPH on vof, and the
// cross pairs' sums.
template <typename T>
struct WaterB {
    T mx, my, fx, fy, xsx, xsy, dvf;
    T cdx, cdy, cdvof, cv2;
    int chits;
};

// What water_pass_b does with them: the rates, the renormalisation, the
// leapfrog corrector and the next step's cell key.
template <typename T, bool SINGLE>
__device__ __forceinline__ void water_b_finish(const PhaseDev<T>& P, const GridGeom& g, const SimConst& c, const StepCtl& u,
                                               DevCounters* cnt, int k, T rho_a, T phia, const WaterB<T>& w) {
    typedef typename V2<T>::t T2;
    const int a = P.perm[k];
    Corrector<T> q;
    T2 av;
    const int itype = P.itype[a];
    if (!c.average_velocity) av = P.av[a];
    if (u.update) q.load(P, a, c, u, false);
    const bool renorm = !SINGLE && c.volume_fraction && c.renorm_now;
    double rho = 0.0, vof = 0.0;
    if (renorm) { rho = P.rho[a]; vof = P.vof[a]; }
    T dvx = w.mx, dvy = w.my;
    if (rho_a > T(0)) { dvx = dvx / rho_a; dvy = dvy / rho_a; }
    dvx = dvx + w.fx;
    dvy = dvy + w.fy + (T)c.gravity;
    if (c.average_velocity) {
        const T eps = itype > 0 ? (T)c.epsilon : T(1);
        av.x = eps * w.xsx; av.y = eps * w.xsy;
        P.av[a] = av;
    }
    T2 o; o.x = dvx; o.y = dvy;
    if constexpr (!SINGLE) {
        const T fd = phia * (T)(-c.numeric_gravity / c.s_perm);
        o.x = dvx + fd * w.cdx; o.y = dvy + fd * w.cdy;
        T dvof = w.dvf;
        if (c.volume_fraction) {
            const T irho0 = (T)(1.0 / c.s_rho0);
            dvof = w.dvf + w.cdvof * irho0;
            const T vof2 = T(1) - w.cv2 * irho0;
            P.vof2[a] = vof2;
            if (renorm) {
                rho = rho / vof * (double)vof2;
                vof = (double)vof2;
                if (u.first) { q.rho = rho; q.vof = vof; }   // the first step integrates from them
                if (!u.update) { P.rho[a] = rho; P.vof[a] = vof; }
            }
        }
        P.dvof[a] = dvof;
        P.countiac[a] = w.chits;
        if (u.update && u.with_vof && c.volume_fraction) {
            if (!u.first) P.vof_min[a] = q.vof;
            P.vof[a] = q.vof + (u.first ? q.dt / 2.0 : q.dt) * (double)dvof;
        }
    }
    P.dv[a] = o;
    double2 xnew;
    if (u.update) { q.move(P, a, c, u.first, o, av); xnew = q.x; }   // last pass of the water phase
    else if (u.ncount) xnew = P.x[a];
    if (u.ncount) cell_key(g, xnew, a, P.cell_id, P.cell_fill, u.ncount, cnt, 1);
}

// ----------------------------------------------------------- water: pass B
// Momentum dv = (-vof*df(p) + df(vof*sxx) + df(vof*sxy)) / rho
// (declarations_sph.f90:1257-1265; df m_particles.f90:1711), art_visc :2504,
// delta_sph(vof) :2658, repulsive_force :1605, gravity, av_vel :2761.
// The water-only step (declarations_sph.f90:1494-1518) is the same with
// vof = 1 and neither wall force nor delta-SPH on vof.  The wall force takes
// dx = x_real - x_virtual, as the reference does with real particles
// numbered before virtual ones.
//
// Two-phase (SINGLE = false): the water side of the cross pairs follows in
// the same kernel (cross_water_sums), then the renormalisation rho <-
// rho/vof*vof2, vof <- vof2 every renorm_interval steps
// (declarations_sph.f90:1414-1421), then, as the last pass of the water
// phase, the leapfrog corrector.  FCH as in cross_water_sums.
template <typename T, int SKF, bool SINGLE, bool FCH, int G = 1>
__global__ void __launch_bounds__(SPHG_TPB, sizeof(T) == 4 ? SPHG_MINB_B : SPHG_MINB_B64) k_water_pass_b(PhaseDev<T> P, PhaseDev<T> S, GridGeom g, SearchConst sc,
                                                          SearchConst scx, SimConst c, StepCtl u, DevCounters* cnt) {
    pdl_enter();
    typedef typename V2<T>::t T2;
    const int k = gtid() / G;
    const bool valid = k < P.n;
    const int kk = valid ? k : 0;
    const int a = P.perm[kk];
    const double2 xa = P.xs[kk];
    const double ha = P.hs[kk];
    const RecA<T>* __restrict__ rec = SINGLE ? P.recA2 : P.recA;
    const RecA<T> ra = rec[kk];
    const RecB<T> qa = P.recB[kk];
    const bool real_a = P.itype[a] > 0;
    const T phia = qa.vof;
    const T fa_xx = phia * qa.sxx, fa_xy = phia * qa.sxy, fa_yy = phia * qa.syy;
    const T pref = (T)(c.delta * ha) * qa.c;
    const T alpha = (T)c.alpha, beta = (T)c.beta, etq2 = (T)(c.etq * c.etq);
    const T r0 = (T)P.dspp, dd = (T)c.dd, p1 = (T)c.p1, p2 = (T)c.p2;
    const bool do_rep = !SINGLE && real_a;
    const bool do_dvof = !SINGLE && c.water_artificial_volume;
    const bool visc = c.visc_artificial, xsph = c.average_velocity;
    KernelConst<T, SKF> ka;
    ka.init((T)ha);
    // x/y pairs: d1 = sum vb (pa+pb) gradW; d2 = sum vb (sxx, sxy) dW/dx;
    // d3 = sum vb (sxy, syy) dW/dy; av, rp, xv as art_visc, repulsive_force, av_vel
    T2 d1 = splat2(T(0)), d2 = splat2(T(0)), d3 = splat2(T(0)), av = splat2(T(0)), rp = splat2(T(0)), xv = splat2(T(0));
    T dvf = 0;
    T2 fa_a, fa_b, va;
    fa_a.x = fa_xx; fa_a.y = fa_xy; fa_b.x = fa_xy; fa_b.y = fa_yy;
    va.x = ra.vx; va.y = ra.vy;
    const uint4 mask = G == 1 && valid ? P.hmask[k] : make_uint4(0u, 0u, 0u, 0u);   // recorded by the step's first water pass
    const T rho_m = finite_rho(ra.rho);
    auto body = [&](const RecA<T>* RA, const RecB<T>* RB, int m, T dx, T dy) {
        const RecA<T> rb = RA[m];
        const RecB<T> qb = RB[m];
        T w, sr, rr, mh;
        pair_kernel<T, SKF>(ka, sc, ha, P.hs, m, dx, dy, w, sr, rr, mh);
        T2 d, vb2;
        d.x = dx; d.y = dy;
        vb2.x = rb.vx; vb2.y = rb.vy;
        const T2 gr = mul2(splat2(sr), d);                       // (gx, gy)
        const T vb = rb.vol;
        const T pp = qa.p + qb.p;
        d1 = fma2(splat2(vb), mul2(splat2(pp), gr), d1);
        T2 sb_a, sb_b;                                           // (sxx, sxy), (sxy, syy) of the neighbour
        sb_a.x = qb.sxx; sb_a.y = qb.sxy; sb_b.x = qb.sxy; sb_b.y = qb.syy;
        const T2 s_a = fma2(splat2(qb.vof), sb_a, fa_a);          // phi_a s_a + phi_b s_b
        const T2 s_b = fma2(splat2(qb.vof), sb_b, fa_b);
        d2 = fma2(splat2(vb), mul2(s_a, splat2(gr.x)), d2);
        d3 = fma2(splat2(vb), mul2(s_b, splat2(gr.y)), d3);
        const T2 dv = sub2(va, vb2);                              // v_a - v_b
        const T mb = vb * rb.rho;
        // 1 / mean density (art_visc and av_vel); in FP64 from one division with 1 / (r^2 + etq^2 h^2), then corrected
        T irho, iden = T(0), den = T(0);
        if constexpr (sizeof(T) == 8) {
            const T mr = T(0.5) * (rho_m + rb.rho);
            den = fmax(rr + mh * mh * etq2, T(1e-300));
            const T inv = T(1) / (mr * den);
            irho = rcp_near(mr, inv * den);
            iden = inv * mr;
        } else {
            irho = rcp_<T>(T(0.5) * (ra.rho + rb.rho));
        }
        if (visc) {
            const T vr = dv.x * dx + dv.y * dy;
            if (vr < T(0)) {
                T muv;
                if constexpr (sizeof(T) == 8) muv = quot_(mh * vr, den, iden);
                else muv = div_<T>(mh * vr, rr + mh * mh * etq2);
                const T mc = T(0.5) * (qa.c + qb.c);
                const T piv = ((beta * muv - alpha * mc) * muv) * irho;
                av = fma2(splat2(-mb), mul2(splat2(piv), gr), av);
            }
        }
        if (do_dvof) dvf += pref * vb * ((phia - qb.vof) * (T(2) * sr));
        if (do_rep && qb.itype < T(0)) {
            const T r = sqrt(rr);
            if (!(r > r0)) {
                const T f = (powr_<T>(r0 / r, p1) - powr_<T>(r0 / r, p2)) / (r * r);
                rp = fma2(mul2(splat2(dd), d), splat2(f), rp);
            }
        }
        if (xsph) {
            const T q = (mb * w) * irho;
            xv = fma2(splat2(-q), dv, xv);
        }
    };
    // Neighbours read through L1, not staged in shared memory: staging them
    // (positions and both records, up to 560 per block) cut the resident
    // blocks to 6 per SM and measured 179 us per launch at 912,016 particles
    // against 164 us for this form at 7 blocks.  Loading each lane's next
    // hit's records during the current one (16 more registers) measured 210
    // us at 6 blocks.
    auto each = [&](int m, T dx, T dy) { body(rec, P.recB, m, dx, dy); };
    if constexpr (G == 1) {
        visit_masked<T>(g, sc, P.cell_start, P.xs, P.hs, xa, ha, k, valid, mask, each);
    } else {
        scan_lanes<G, T>(sc, candidate_runs(g, P.cell_start, xa, valid), P.xs, P.hs, xa, ha, k, each);
        lanes_sum<G>(d1.x, d1.y, d2.x, d2.y, d3.x, d3.y, av.x, av.y, rp.x, rp.y, xv.x, xv.y, dvf);
    }
    const T d1x = d1.x, d1y = d1.y, d2x = d2.x, d2y = d2.y, d3x = d3.x, d3y = d3.y;
    const T avx = av.x, avy = av.y, rpx = rp.x, rpy = rp.y, xsx = xv.x, xsy = xv.y;
    WaterB<T> w;
    w.mx = -(phia * d1x) + d2x + d3x;
    w.my = -(phia * d1y) + d2y + d3y;
    w.fx = avx + rpx; w.fy = avy + rpy;
    w.xsx = xsx; w.xsy = xsy;
    w.dvf = dvf;
    w.cdx = w.cdy = w.cdvof = w.cv2 = T(0);
    w.chits = 0;
    const bool finish = valid && threadIdx.x % G == 0;
    if constexpr (!SINGLE && G == 1) {
        SPHG_HITBUF(T);
        w.chits = cross_water_sums<T, SKF, FCH>([&](auto&& f) { return visit_batched(hb, g, scx, S.cell_start, S.xs, S.hs, xa, ha, -1, valid, f); },
                                                S, scx, c, ka, ha, ra, w.cdx, w.cdy, w.cdvof, w.cv2);
    } else if constexpr (!SINGLE) {
        w.chits = cross_water_sums<T, SKF, FCH>([&](auto&& f) { return scan_lanes<G, T>(scx, candidate_runs(g, S.cell_start, xa, valid), S.xs, S.hs, xa, ha, -1, f); },
                                                S, scx, c, ka, ha, ra, w.cdx, w.cdy, w.cdvof, w.cv2);
        lanes_sum<G>(w.cdx, w.cdy, w.cdvof, w.cv2, w.chits);
    }
    if (finish) water_b_finish<T, SINGLE>(P, g, c, u, cnt, k, ra.rho, phia, w);
    if constexpr (!SINGLE) count_stats(cnt, 2, -1, w.chits, finish);
}

// A soil particle's sums of soil_pass: momentum (before the division by rho),
// artificial viscosity plus wall force, XSPH, the rates, and the cross pairs'
// sums.
template <typename T>
struct SoilSums {
    T mx, my, fx, fy, xsx, xsy;
    T drho, txx, txy, tyy, vcc, wxy, dp, dsx, dsxy, dsy;
    T cdx, cdy, cpx, cpy;
    int hits;
};

// What soil_pass does with them: plastic_or_not, plastic_flow_rule3 and
// Jaumann_rate on the post-DP state, the rates, the leapfrog corrector and
// the next step's cell key.
template <typename T, bool SINGLE>
__device__ __forceinline__ void soil_finish(const PhaseDev<T>& P, const GridGeom& g, const SimConst& c, const StepCtl& u,
                                            DevCounters* cnt, int k, T rho_a, T phis, const SoilSums<T>& w, int& fail,
                                            int& fail3) {
    typedef typename V2<T>::t T2;
    const int a = P.perm[k];
    // every load before the first store
    Corrector<T> cr;
    T2 av;
    const int itype = P.itype[a];
    const double alpha1 = c.tab[P.sid[a]].s_alpha1;
    const double p = P.p[a], sxx = P.sxx[a], sxy = P.sxy[a], syy = P.syy[a];
    double rho = P.rho[a];
    if (c.half) rho = half_step(rho, c.tab[P.sid[a]].dt, P.drho[a]);
    if (!c.average_velocity) av = P.av[a];
    if (u.update) cr.load(P, a, c, u, true);
    T dvx = w.mx, dvy = w.my;
    if (rho_a > T(0)) { dvx = dvx / rho_a; dvy = dvy / rho_a; }
    dvx = dvx + w.fx;
    dvy = dvy + w.fy + (T)c.gravity;
    if (c.average_velocity) {
        const T eps = itype > 0 ? (T)c.epsilon : T(1);
        av.x = eps * w.xsx; av.y = eps * w.xsy;
        P.av[a] = av;
    }
    P.drho[a] = w.drho;
    // plastic_or_not + plastic_flow_rule3 + Jaumann_rate on the post-DP state
    const double dtxx = (double)w.txx, dtxy = (double)w.txy, dtyy = (double)w.tyy, dvcc = (double)w.vcc;
    const double G = c.s_E / (2.0 * (1 + c.s_niu));
    double ds0 = 0.0, ds1 = 0.0, ds2 = 0.0, dp = 0.0;
    fail = 0;
    if (c.plasticity == 3) {
        const double J2a = sqrt((sxx * sxx + 2.0 * (sxy * sxy) + syy * syy + (sxx + syy) * (sxx + syy)) / 2.0) + 1.0e-6;
        if (fabs(J2a - alpha1 * (3.0 * p)) < SPHG_F32LIT(1.0e-5f)) fail = 1;
        P.fail[a] = fail;
        if (fail) {
            const double exx = dtxx / 2.0 + dvcc / 3.0, exy = dtxy / 2.0, eyy = dtyy / 2.0 + dvcc / 3.0;
            const double sde = sxx * exx + 2.0 * sxy * exy + syy * eyy;
            double J2 = (sxx * sxx + 2.0 * (sxy * sxy) + syy * syy + (sxx + syy) * (sxx + syy)) / 2.0;
            J2 = J2 + 1.0e-10;
            const double al = alpha1, K = c.s_k;
            const double dlambda = (3.0 * al * K * dvcc + G / sqrt(J2) * sde) / (9.0 * (al * al) * K + G);
            if (!(dlambda < 0)) {
                ds0 = ds0 - dlambda * (G / sqrt(J2) * sxx);
                ds1 = ds1 - dlambda * (G / sqrt(J2) * sxy);
                ds2 = ds2 - dlambda * (G / sqrt(J2) * syy);
                dp = dp + 3.0 * K * al * dlambda;
                P.eps_p[a] = P.eps_p[a] + dlambda * sxy / (2 * sqrt(J2)) * SPHG_F32LIT(0.000005f);
            }
        }
    }
    const double dwxy = (double)w.wxy;
    ds0 = ds0 + G * dtxx; ds1 = ds1 + G * dtxy; ds2 = ds2 + G * dtyy;
    dp = dp - c.s_k * dvcc;
    ds0 = ds0 + 2.0 * sxy * dwxy;
    ds1 = ds1 - (sxx - syy) * dwxy;
    ds2 = ds2 - 2.0 * sxy * dwxy;
    const T rxx = (T)(ds0 + (double)w.dsx), rxy = (T)(ds1 + (double)w.dsxy), ryy = (T)(ds2 + (double)w.dsy);
    const T rp = (T)(dp + (double)w.dp);
    P.dsxx[a] = rxx; P.dsxy[a] = rxy; P.dsyy[a] = ryy; P.dp[a] = rp;
    P.c[a] = c.s_c;
    P.txx[a] = w.txx; P.tyy[a] = w.tyy; P.txy[a] = w.wxy;   // wxy is txy (alias)
    P.vcc[a] = w.vcc;
    P.countiac[a] = w.hits;
    T2 o; o.x = dvx; o.y = dvy;
    if constexpr (!SINGLE) {
        const T irs = T(1) / rho_a;
        const T fd = phis * (T)(-c.numeric_gravity / c.s_perm) * irs, fp = irs * phis;
        o.x = dvx + (fd * w.cdx + fp * w.cpx); o.y = dvy + (fd * w.cdy + fp * w.cpy);
        if (c.volume_fraction) P.vof[a] = rho / c.s_rho0;
    }
    P.dv[a] = o;
    fail3 = 0;
    double2 xnew;
    if (u.update) {   // last pass of the soil phase
        cr.drho = w.drho;
        cr.move(P, a, c, u.first, o, av);
        fail3 = cr.stress(P, a, c, u.first, u.do_dp, rxx, rxy, ryy, rp);
        xnew = cr.x;
    } else if (u.ncount) {
        xnew = P.x[a];
    }
    if (u.ncount) cell_key(g, xnew, a, P.cell_id, P.cell_fill, u.ncount, cnt, 1);
}

// ------------------------------------------------------------------ soil
// Same-phase soil terms in one pass (declarations_sph.f90:1195-1373 for the
// two-phase step, :1546-1645 for the soil-only step): con_density,
// delta_sph(rho), shear_strain_rate, velocity_divergence, momentum (df3 of
// vof-weighted p and s two-phase, df soil-only), art_visc, delta_sph on p and
// s, repulsive_force (two-phase only), gravity, av_vel; then per particle
// plastic_or_not :3447, plastic_flow_rule3 :3700 and Jaumann_rate :3047,
// whose spin sum wxy comes from the same pass.
//
// Two-phase (SINGLE = false): the soil side of the cross pairs follows in the
// same kernel (cross_soil_sums), then volume_fraction_soil :3970 and, as the
// last pass of the soil phase, the leapfrog corrector.  FCH as in
// cross_soil_sums.
template <typename T, int SKF, bool SINGLE, bool FCH, int G = 1>
__global__ void __launch_bounds__(SPHG_TPB, sizeof(T) == 4 ? SPHG_MINB_SOIL : SPHG_MINB_S64) k_soil_pass(PhaseDev<T> P, PhaseDev<T> W, GridGeom g, SearchConst sc,
                                                       SearchConst scx, SimConst c, DevCounters* cnt, int slot, StepCtl u) {
    pdl_enter();
    const int k = gtid() / G;
    const bool valid = k < P.n;
    const int kk = valid ? k : 0;
    const int a = P.perm[kk];
    const double2 xa = P.xs[kk];
    const double ha = P.hs[kk];
    const RecA<T> ra = P.recA[kk];
    const RecB<T> qa = P.recB[kk];
    const bool real_a = P.itype[a] > 0;
    const T cs = (T)c.s_c;                          // pressure(): c = soil%c
    const T pref_old = (T)(c.delta * ha) * qa.c;    // delta_sph(rho) runs before pressure()
    const T pref = (T)(c.delta * ha) * cs;
    const T c23 = (T)SPHG_F32LIT(2.0f / 3.0f);
    const T alpha = (T)c.alpha, beta = (T)c.beta, etq2 = (T)(c.etq * c.etq);
    const T r0 = (T)P.dspp, dd = (T)c.dd, p1 = (T)c.p1, p2 = (T)c.p2;
    const T phia = SINGLE ? T(1) : qa.vof;
    const T fap = phia * qa.p, faxx = phia * qa.sxx, faxy = phia * qa.sxy, fayy = phia * qa.syy;
    const T ira2 = T(1) / (ra.rho * ra.rho);
    const bool dens = c.artificial_density, visc = c.visc_artificial, xsph = c.average_velocity;
    const bool dstress = c.soil_artificial_stress, do_rep = !SINGLE && real_a;
    KernelConst<T, SKF> ka;
    ka.init((T)ha);
    T con = 0, dl = 0, txx = 0, txy = 0, tyy = 0, vcc = 0, wxy = 0;
    T s1x = 0, s1y = 0, s2x = 0, s3x = 0, s2y = 0, s3y = 0;
    T avx = 0, avy = 0, rpx = 0, rpy = 0, xsx = 0, xsy = 0;
    T dpp = 0, dsx = 0, dsxy = 0, dsy = 0;
    const T rho_m = finite_rho(ra.rho);
    auto body = [&](int m, T dx, T dy) {
        const RecA<T> rb = P.recA[m];
        const RecB<T> qb = P.recB[m];
        T w, sr, rr, mh;
        pair_kernel<T, SKF>(ka, sc, ha, P.hs, m, dx, dy, w, sr, rr, mh);
        const T gx = sr * dx, gy = sr * dy;
        const T du = rb.vx - ra.vx, dv = rb.vy - ra.vy;   // v_b - v_a
        const T vb = rb.vol, mb = vb * rb.rho;
        const T e = T(2) * sr;                            // 2 (dx . grad W) / r^2
        // in FP64, 1 / mean density, 1 / (r^2 + etq^2 h^2) and 1 / rho_b from one division (corrected where they are used)
        T irho64 = T(0), iden64 = T(0), irb64 = T(0), den = T(0);
        const T mr = T(0.5) * (rho_m + rb.rho);
        if constexpr (sizeof(T) == 8) {
            den = fmax(rr + mh * mh * etq2, T(1e-300));
            const T md = mr * den, inv = T(1) / (md * rb.rho);
            irb64 = inv * md;
            irho64 = inv * (den * rb.rho);
            iden64 = inv * (mr * rb.rho);
        }
        // a / mean density
        auto over_mr = [&](T a) {
            if constexpr (sizeof(T) == 8) return quot_(a, mr, irho64);
            else return div_<T>(a, mr);
        };
        con -= mb * (du * gx + dv * gy);
        if (dens) dl += pref_old * vb * ((ra.rho - rb.rho) * e);
        txx += vb * (c23 * (T(2) * du * gx - dv * gy));
        txy += vb * (du * gy + dv * gx);
        tyy += vb * (c23 * (T(2) * dv * gy - du * gx));
        vcc += vb * (du * gx + dv * gy);
        wxy += vb * (T(0.5) * (du * gy - dv * gx));
        if (SINGLE) {       // df: m_b/rho_b (f_a + f_b) gradW
            const T pp = fap + qb.p;
            s1x += vb * (pp * gx); s1y += vb * (pp * gy);
            s2x += vb * ((faxx + qb.sxx) * gx);
            s3x += vb * ((faxy + qb.sxy) * gy);
            s2y += vb * ((faxy + qb.sxy) * gx);
            s3y += vb * ((fayy + qb.syy) * gy);
        } else {            // df3: m_b (f_a/rho_a^2 + f_b/rho_b^2) gradW
            T irb;
            if constexpr (sizeof(T) == 8) irb = rcp_near(rb.rho, irb64);
            else irb = rcp_<T>(rb.rho);
            const T ib = qb.vof * irb * irb;
            const T pp = fap * ira2 + qb.p * ib;
            s1x += mb * (pp * gx); s1y += mb * (pp * gy);
            const T xx = faxx * ira2 + qb.sxx * ib;
            const T xy = faxy * ira2 + qb.sxy * ib;
            const T yy = fayy * ira2 + qb.syy * ib;
            s2x += mb * (xx * gx);
            s3x += mb * (xy * gy);
            s2y += mb * (xy * gx);
            s3y += mb * (yy * gy);
        }
        if (visc) {
            const T vr = -(du * dx + dv * dy);
            if (vr < T(0)) {
                T muv;
                if constexpr (sizeof(T) == 8) muv = quot_(mh * vr, den, iden64);
                else muv = div_<T>(mh * vr, rr + mh * mh * etq2);
                const T piv = over_mr((beta * muv - alpha * cs) * muv);
                avx -= mb * (piv * gx);
                avy -= mb * (piv * gy);
            }
        }
        if (dstress) {
            const T q = pref * vb * e;
            dpp += q * (qa.p - qb.p);
            dsx += q * (qa.sxx - qb.sxx);
            dsxy += q * (qa.sxy - qb.sxy);
            dsy += q * (qa.syy - qb.syy);
        }
        if (do_rep && qb.itype < T(0)) {
            const T r = sqrt(rr);
            if (!(r > r0)) {
                const T f = (powr_<T>(r0 / r, p1) - powr_<T>(r0 / r, p2)) / (r * r);
                rpx += dd * dx * f;
                rpy += dd * dy * f;
            }
        }
        if (xsph) {
            const T q = over_mr(mb * w);
            xsx += q * du;
            xsy += q * dv;
        }
    };
    int hits;
    const bool finish = valid && threadIdx.x % G == 0;
    SPHG_HITBUF_G(T, G);
    if constexpr (G == 1) {
        hits = visit_batched(hb, g, sc, P.cell_start, P.xs, P.hs, xa, ha, k, valid, body);
    } else {
        hits = scan_lanes<G, T>(sc, candidate_runs(g, P.cell_start, xa, valid), P.xs, P.hs, xa, ha, k, body);
        lanes_sum<G>(con, dl, txx, txy, tyy, vcc, wxy, s1x, s1y, s2x, s3x, s2y, s3y);
        lanes_sum<G>(avx, avy, rpx, rpy, xsx, xsy, dpp, dsx, dsxy, dsy, hits);
    }
    SoilSums<T> w;
    if (SINGLE) { w.mx = -s1x + s2x + s3x; w.my = -s1y + s2y + s3y; }
    else {
        w.mx = -(s1x * ra.rho) + s2x * ra.rho + s3x * ra.rho;
        w.my = -(s1y * ra.rho) + s2y * ra.rho + s3y * ra.rho;
    }
    w.fx = avx + rpx; w.fy = avy + rpy;
    w.xsx = xsx; w.xsy = xsy;
    w.drho = con + dl;
    w.txx = txx; w.txy = txy; w.tyy = tyy; w.vcc = vcc; w.wxy = wxy;
    w.dp = dpp; w.dsx = dsx; w.dsxy = dsxy; w.dsy = dsy;
    w.cdx = w.cdy = w.cpx = w.cpy = T(0);
    w.hits = hits;
    if constexpr (!SINGLE && G == 1) {
        cross_soil_sums<T, SKF, FCH>([&](auto&& f) { return visit_batched(hb, g, scx, W.cell_start, W.xs, W.hs, xa, ha, -1, valid, f); },
                                     W, scx, c, ka, ha, ra, w.cdx, w.cdy, w.cpx, w.cpy);
    } else if constexpr (!SINGLE) {
        cross_soil_sums<T, SKF, FCH>([&](auto&& f) { return scan_lanes<G, T>(scx, candidate_runs(g, W.cell_start, xa, valid), W.xs, W.hs, xa, ha, -1, f); },
                                     W, scx, c, ka, ha, ra, w.cdx, w.cdy, w.cpx, w.cpy);
        lanes_sum<G>(w.cdx, w.cdy, w.cpx, w.cpy);
    }
    int fail = 0, fail3 = 0;
    if (finish) soil_finish<T, SINGLE>(P, g, c, u, cnt, k, ra.rho, qa.vof, w, fail, fail3);
    count_stats(cnt, slot, slot, hits, finish);
    if (c.plasticity == 3) count_fail(cnt, 2, fail);
    if (u.update && u.do_dp) count_fail(cnt, 3, fail3);
}

// The step's counters and the batch's sticky flags as the host reads them.
struct CounterMirror { DevCounters c; int sticky[4]; };

// The counters' values at the start of a step.  take_next: the step's cell keys
// were counted by the corrector of the step before, with its clamped and
// non-finite positions.
__device__ __forceinline__ void reset_counters(DevCounters* c, int take_next) {
    const int i = threadIdx.x;
    if (i < 3) c->pairs[i] = 0ull;
    if (i < 2) { c->maxiac[i] = 0; c->miniac[i] = 0x7fffffff; c->noiac[i] = 0; }
    if (i < 4) c->nfail[i] = 0;
    if (i == 0) {
        c->n_out = take_next ? c->n_out_next : 0;
        c->nonfinite = take_next ? c->nonfinite_next : 0;
        c->n_out_next = 0; c->nonfinite_next = 0;
        c->overflow = 0; c->timeout = 0;
    }
}
static __global__ void k_reset_counters(DevCounters* c, int take_next) {
    pdl_enter();
    reset_counters(c, take_next);
}

// Sticky per-batch flags: a pair list above max_interaction (the reference
// stops there, m_particles.f90:992-993) and non-finite positions.  With a
// mirror (mapped pinned host memory) the step's counters and the flags are
// also written there, so the host reads them after its synchronisation with
// no copy of its own, and (next != 0) the counters are reset for the next step,
// whose cells the corrector has counted.  One warp, a word per lane.
static __global__ void k_check(DevCounters* __restrict__ c, int* __restrict__ sticky, unsigned long long cap,
                               CounterMirror* __restrict__ mirror, int next) {
    pdl_enter();
    const int i = threadIdx.x;
    constexpr int W = (int)(sizeof(DevCounters) / sizeof(int));
    static_assert(sizeof(DevCounters) % sizeof(int) == 0 && W <= 32, "a counter word per lane");
    int word = 0;
    if (mirror && i < W) word = reinterpret_cast<const int*>(c)[i];
    bool flag = false;
    if (i == 0) flag = c->pairs[0] / 2 > cap || c->pairs[1] / 2 > cap || c->pairs[2] > cap;
    if (i == 1) flag = c->nonfinite != 0;
    if (i == 2) flag = c->timeout != 0;
    if (flag) {
        sticky[i] = 1;
        if (mirror) mirror->sticky[i] = 1;
    }
    if (mirror) {
        if (i < W) reinterpret_cast<int*>(&mirror->c)[i] = word;
        __syncwarp();
        if (next) reset_counters(c, 1);
    }
}

// ------------------------------------------------------- layout transforms
// Every persistent field of a phase permuted into the current cell order in
// one launch: dst_i[k] = src_i[perm[k]].
struct PermField { const void* src; void* dst; int bytes; int pad; };
struct PermList { int count; int pad; PermField f[44]; };
static __global__ void __launch_bounds__(256) k_permute_all(int n, const int* __restrict__ perm, PermList L) {
    pdl_enter();
    int k = gtid();
    if (k >= n) return;
    const int a = perm[k];
    for (int i = 0; i < L.count; ++i) {
        const PermField& f = L.f[i];
        if (f.bytes == 4) ((int*)f.dst)[k] = ((const int*)f.src)[a];
        else if (f.bytes == 8) ((long long*)f.dst)[k] = ((const long long*)f.src)[a];
        else ((int4*)f.dst)[k] = ((const int4*)f.src)[a];
    }
}

// Morton (Z-order) state order: the key of the particle in sorted slot k is
// the interleaved bits of its support-radius cell (x cell / kx, row); the
// stable sort of the slots by key keeps the cell list's order inside a cell.
__device__ __forceinline__ unsigned spread_bits16(unsigned v) {
    v &= 0xffffu;
    v = (v | (v << 8)) & 0x00ff00ffu;
    v = (v | (v << 4)) & 0x0f0f0f0fu;
    v = (v | (v << 2)) & 0x33333333u;
    v = (v | (v << 1)) & 0x55555555u;
    return v;
}
static __global__ void __launch_bounds__(256) k_morton_keys(int n, const int* __restrict__ perm,
                                                            const int* __restrict__ cell_id, GridGeom g,
                                                            unsigned* __restrict__ key, int* __restrict__ val) {
    pdl_enter();
    const int k = gtid();
    if (k >= n) return;
    const int a = perm[k];
    const int c = cell_id[a];
    key[k] = spread_bits16((unsigned)((c % g.ncx) / g.kx)) | (spread_bits16((unsigned)(c / g.ncx)) << 1);
    val[k] = a;
}
// new state index of each old one (inv[order[j]] = j), then the cell list's
// slots renumbered to the new state indices
static __global__ void __launch_bounds__(256) k_invert(int n, const int* __restrict__ order, int* __restrict__ inv) {
    pdl_enter();
    const int j = gtid();
    if (j < n) inv[order[j]] = j;
}
static __global__ void __launch_bounds__(256) k_renumber(int n, const int* __restrict__ inv, int* __restrict__ perm) {
    pdl_enter();
    const int k = gtid();
    if (k < n) perm[k] = inv[perm[k]];
}

template <typename S>
__global__ void __launch_bounds__(256) k_permute(int n, const int* __restrict__ perm, const S* __restrict__ src, S* __restrict__ dst) {
    int k = gtid();
    if (k < n) dst[k] = src[perm[k]];
}
static __global__ void __launch_bounds__(256) k_iota(int n, int* __restrict__ v) {
    pdl_enter();
    int k = gtid();
    if (k < n) v[k] = k;
}
// state order -> original (Fortran) order, widening to double
template <typename S>
__global__ void __launch_bounds__(256) k_to_original(int n, const int* __restrict__ orig, const S* __restrict__ src,
                                                     double* __restrict__ dst, int comps) {
    int a = gtid();
    if (a >= n) return;
    const S* s = src + (size_t)a * comps;
    double* d = dst + (size_t)orig[a] * comps;
    for (int t = 0; t < comps; ++t) d[t] = (double)s[t];
}
// original order -> state order, narrowing from double
template <typename S>
__global__ void __launch_bounds__(256) k_from_original(int n, const int* __restrict__ orig, const double* __restrict__ src,
                                                       S* __restrict__ dst, int comps) {
    int a = gtid();
    if (a >= n) return;
    const double* s = src + (size_t)orig[a] * comps;
    S* d = dst + (size_t)a * comps;
    for (int t = 0; t < comps; ++t) d[t] = (S)s[t];
}
static __global__ void __launch_bounds__(256) k_from_original_i(int n, const int* __restrict__ orig, const int* __restrict__ src,
                                                         int* __restrict__ dst) {
    int a = gtid();
    if (a < n) dst[a] = src[orig[a]];
}

// Several fields of a phase at once between the state order and the caller's
// original order, through one staging area in which field i occupies
// stage[off, off + n*comps) in original order.  wide: 1 the device field is
// FP64, 0 of the precision's type S, 2 int32 (and int32 in the staging area).  One launch per group of fields lets
// the host copies of the group run back to back on the copy engine; each
// field has its own row of blocks (blockIdx.y), so that the fields' loads do
// not wait on one another.
struct XferField { void* dev; long long off; int comps; int wide; };
struct XferList { int count; int pad; XferField f[40]; };
template <typename S>
__global__ void __launch_bounds__(256) k_to_original_all(int n, const int* __restrict__ orig, const __grid_constant__ XferList L,
                                                         double* __restrict__ stage) {
    const int a = gtid();
    if (a >= n || (int)blockIdx.y >= L.count) return;
    const XferField& f = L.f[blockIdx.y];
    if (f.wide == 2) { ((int*)(stage + f.off))[orig[a]] = ((const int*)f.dev)[a]; return; }
    double* d = stage + f.off + (size_t)orig[a] * f.comps;
    if (f.wide) {
        const double* s = (const double*)f.dev + (size_t)a * f.comps;
        for (int t = 0; t < f.comps; ++t) d[t] = s[t];
    } else {
        const S* s = (const S*)f.dev + (size_t)a * f.comps;
        for (int t = 0; t < f.comps; ++t) d[t] = (double)s[t];
    }
}
// The water's shared working arrays after a two-phase step (sxx => txx,
// syy => tyy, sxy => txy; declarations_sph.f90:371-377, 414-415): the soil
// pass has written the first n_soil entries with soil values, indexed by the
// soil's original order, and txy holds zero beyond them (Jaumann_rate,
// m_particles.f90:3077).  stage: the water field staged in the water's
// original order (nw entries).
template <typename S>
__global__ void __launch_bounds__(256) k_alias_soil(int ns, int nw, const int* __restrict__ sorig, const S* __restrict__ src,
                                                    double* __restrict__ stage, int zero_tail) {
    const int i = gtid();
    if (i < ns) {
        const int o = sorig[i];
        if (o < nw) stage[o] = (double)src[i];
    } else if (zero_tail && i < nw) {
        stage[i] = 0.0;
    }
}
template <typename S>
__global__ void __launch_bounds__(256) k_from_original_all(int n, const int* __restrict__ orig, const __grid_constant__ XferList L,
                                                           const double* __restrict__ stage) {
    const int a = gtid();
    if (a >= n || (int)blockIdx.y >= L.count) return;
    const XferField& f = L.f[blockIdx.y];
    if (f.wide == 2) { ((int*)f.dev)[a] = ((const int*)(stage + f.off))[orig[a]]; return; }
    const double* s = stage + f.off + (size_t)orig[a] * f.comps;
    if (f.wide) {
        double* d = (double*)f.dev + (size_t)a * f.comps;
        for (int t = 0; t < f.comps; ++t) d[t] = s[t];
    } else {
        S* d = (S*)f.dev + (size_t)a * f.comps;
        for (int t = 0; t < f.comps; ++t) d[t] = (S)s[t];
    }
}

// Pair export: per particle (original index i), the neighbours j > i (or, for
// the cross list, every neighbour), sorted, written at offset[i].
static __global__ void __launch_bounds__(SPHG_TPB) k_pairs_count(int n, const int* __restrict__ perm, const int* __restrict__ orig,
                                                          const double2* __restrict__ xs, const double* __restrict__ hs,
                                                          GridGeom g, SearchConst sc, const int* __restrict__ cstart_o,
                                                          const double2* __restrict__ xs_o, const double* __restrict__ hs_o,
                                                          const int* __restrict__ perm_o, const int* __restrict__ orig_o,
                                                          int cross, int* __restrict__ count, int pass, const long long* __restrict__ offset,
                                                          int* __restrict__ out_i, int* __restrict__ out_j, long long cap) {
    int k = gtid();
    if (k >= n) return;
    const int oi = orig[perm[k]];
    const double2 xa = xs[k];
    const double ha = hs[k];
    int cnt = 0;
    long long base = pass ? offset[oi] : 0;
    visit_neighbours(g, sc, cstart_o, xs_o, hs_o, xa, ha, cross ? -1 : k,
        [&](int m, double, double, double, double) {
            const int oj = orig_o[perm_o[m]];
            if (!cross && oj <= oi) return;
            if (pass) {
                long long pos = base + cnt;
                if (pos < cap) { out_i[pos] = oi + 1; out_j[pos] = oj + 1; }
            }
            ++cnt;
        });
    if (!pass) { count[oi] = cnt; return; }
    // sort this particle's j's (few) in place
    long long b = base, e = base + cnt;
    if (e > cap) e = cap;
    for (long long i = b + 1; i < e; ++i) {
        int v = out_j[i];
        long long j = i - 1;
        while (j >= b && out_j[j] > v) { out_j[j + 1] = out_j[j]; --j; }
        out_j[j + 1] = v;
    }
}
