// lanczos.cu — kernel (c): persistent, batched, fused Lanczos.
//
// One cooperative launch runs every step of many independent Lanczos runs
// ("jobs": sectors of the ground-state search, the eigenvector pass of the
// winning sector, c / c^+ excitation runs of the Green's function).
//
// The recurrence is the reference's (src/lanczos_solver.f90:92-173):
//   v_1 = v_init,  v_k = y_{k-1} - a_{k-1} w_{k-1}  (k >= 2),
//   b_k = ||v_k||,  w_k = v_k / b_k,
//   y_k = H w_k - b_k w_{k-1},  a_k = <w_k, y_k>,
// with a(1..), b(1) = 0, b(k) = ||v_k|| (k >= 2) stored as they are accepted.
//
// A step is two phases; H.v is split as in hv_plane.cuh:
//   column phase  each CTA stages slabs of whole columns of
//                 v_k = y_{k-1} - a_{k-1} w_{k-1}, stores v_k, sums
//                 ||v_k||^2 exactly and writes D = the down-hop part of
//                 H v_k over y_{k-1} (its own columns);
//   row phase     with b_k known from those sums, each CTA stages tiles of
//                 whole rows of v_k, adds the diagonal, up-hop and exchange
//                 parts to D, scales by 1 / b_k, subtracts b_k w_{k-1},
//                 stores y_k over D (its own rows) and sums <w_k, y_k>.
// Vectors are stored unnormalised (w_k = v_k / b_k is formed where it is
// read), in the internal string order of hv_plane.cuh, as 4 x 4 blocks of
// 128 bytes (lz_index), so that both phases move whole lines.  A run holds y
// and the last two v: 24 bytes a state.  Every neighbour value comes from
// shared memory, every global access is a stream, and both reductions are
// exact sums, as in the reference.
//
// What bounds it: the load/store pipe (hop values from shared memory, 2 x 8
// bytes a hop and state, 1.1-1.2 times the conflict-free wavefronts) and the
// latency of staging and of the arrivals, then DRAM (64 bytes a state and
// step once the vectors exceed L2).  Registers decide the rest: all 128 of a
// thread are in use, and the largest tiles spill a little (8 x 8 columns by
// rows, 512 threads: 116 bytes stored and 148 loaded; 256 threads 20 and 20; with
// exchange terms 76 to 152 and 124 to 252 for tiles of eight columns or rows;
// others 0 to 28); 80 registers for half as many threads again lost a sixth, tile
// functions called instead of inlined a third.  Measured per step against slabs of the reference's string order
// staged as (y, w) pairs under grid-wide barriers: 9 sectors of nsite 12
// 146 -> 124 us, 4 sectors of nsite 13 280 -> 196 us, one sector of nsite 14
// 279 -> 212 us, of nsite 15 1,092 -> 930 us, of nsite 8 13.6 -> 9.4 us.  With
// the hop lists of the row phase loaded ahead, a CTA serving one run where that
// comes out even (lz_cut) and no look-up of its range left in a phase: 100, 185,
// 202, 809 and 8.9 us, 9 sectors of nsite 10 30 -> 15.
//
// The tiles of all jobs of a phase form one list, cut into one contiguous
// range per CTA at equal modelled cost (lz_plan); within a job the column
// slabs are numbered by round, so the CTAs stage neighbouring slabs at the
// same time.  A job's participants in a phase are the CTAs whose range meets
// its list positions.  Jobs are synchronised one by one: a participant that has
// finished its tiles of a phase writes its partial sum into its slot and
// arrives on the job's counter; a participant of the next phase waits for
// all arrivals of the earlier ones and derives the run's scalars from the
// slots in a fixed order, so all get the same bits.  Runs do not wait for
// one another, and a small run's phases are synchronised over its own few
// CTAs.
//
// The v_k of a run are ping-pong buffers, or (LzJob::keep) one slot for each
// of its first steps, so that the eigenvector can be summed from them
// afterwards.  The eigenvector pass (LZ_EIGVEC) reruns the recurrence with the
// stored a, b (src/lanczos_solver.f90:213-300) and accumulates
// sum_k coeff_k w_k: all of it, or (LzJob::resume) from the last kept step on,
// whose column phase stages the kept v_k, so every later vector has the bits
// of the scan's.  It runs in the kernel that the scan ran in (JobSpec::form):
// in another one's summation order the fixed coefficients lose the vectors'
// norm once they have converged.
//
// A launch may be a slice of longer runs (LzBatch::slice): when its phase
// budget runs out, a closing pass opens every unfinished run's next step
// (derives a(k-1) and the finish test) and stores the state marked opened,
// so a later launch, with any mix of other runs, resumes it.
#include <algorithm>
#include <cmath>
#include <queue>
#include <cuda_runtime.h>
#include "edzt_internal.h"
#include "hv_plane.cuh"

static constexpr unsigned long long kBarrierTimeoutNs = 5ull * 1000ull * 1000ull * 1000ull;
static constexpr int kMaxPlanes = 4;                    // planes of a tile
static constexpr int kMaxRows = 8;                      // rows of a row tile
static constexpr int kLzThreads = 512;                  // threads per SM: one CTA, or two of half as many
static constexpr unsigned kDone = 0x80000000u;          // a job's counter word: the run has finished

size_t lz_sync_bytes(int njobs) { return sizeof(unsigned) * 32 * (size_t)njobs; }   // one 128-byte line per job

static size_t lz_row_smem(int nup, int R) { return (size_t)nup * R * sizeof(double); }
static size_t lz_col_smem(int ndn, int WC) { return (size_t)lz_pad(ndn) * WC * sizeof(double); }

__device__ __forceinline__ unsigned long long globaltimer_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void red_release_add(unsigned* p, unsigned v)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ int find_job(const long long* __restrict__ prefix, int njobs, long long t)
{
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(prefix + mid) <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// x / d from r = 1 / d, rounded as a division is: one correction of x * r by
// its remainder (P. Markstein, IBM J. Res. Dev. 34 (1990) 111-119).
__device__ __forceinline__ double div_by(double x, double d, double r)
{
    const double q = x * r;
    return fma(fma(-q, d, x), r, q);
}

// Element (jd, ju) (internal order) of the start vector of a job.
__device__ __forceinline__ double init_value(const LzJob& J, int jd, int ju)
{
    if (J.init == LZ_INIT_APPLYC) return apply_c_at(J.ac, J.src, __ldg(J.S.up.str + ju), __ldg(J.S.dn.str + jd));
    const long long e = (long long)__ldg(J.S.dn.nat + jd) * J.S.up.count + __ldg(J.S.up.nat + ju);
    return (J.init == LZ_INIT_HASH) ? edzt_u01(J.key, (uint64_t)e) : __ldg(J.src + e);
}

// ---------------------------------------------------------------------------
// the persistent kernel
// ---------------------------------------------------------------------------
// A CTA's shared memory: this, the model tables, the staged tile.
struct LzShared {
    double red[32];                          // reduction scratch
    double* wint;                            // [P * P] interaction energies by impurity patterns
    double* amp_up;                          // [namp] hop amplitudes by slot
    double* amp_dn;
    double* dg;                              // [kMaxRows * P] a row tile's diagonal by row and up impurity pattern, less e1 of the column
    double* chunk;                           // the staged tile
    LzJob J;                                 // the current run
    LzState S;                               // its state in the current phase
    const LzJob* jobs;                       // the launch
    const long long* slab_of;
    double* slots;
    unsigned* sync;
    int* status;
    unsigned long long wait_ns;
    double sum;                              // this CTA's partial sum of the last phase
    double *vk, *vp;                         // v_k, v_{k-1}
    long long vsize;                         // doubles of a vector
    double rb, rp;                           // 1 / S.b_cur, 1 / S.b_prev (0 before the second step)
    int job, phase;                          // what J and S hold
    int ok;
    int pd[kMaxRows];                        // a row tile's down impurity patterns
    int c0[kMaxPlanes];                      // first column of a column tile's planes
};

// Doubles of the tables of a model: P impurity patterns a spin, namp amplitude slots.
static int table_doubles(int P, int namp) { return P * P + 2 * namp + kMaxRows * P; }
static size_t fixed_bytes(int tables) { return (sizeof(LzShared) + sizeof(double) * tables + 127) / 128 * 128; }

extern __shared__ __align__(128) unsigned char lz_smem[];
__device__ __forceinline__ LzShared& lz_shared() { return *reinterpret_cast<LzShared*>(lz_smem); }

// Wait until a job's counter word reaches `need` arrivals or is marked done
// (bounded: on a timeout, or when another CTA reported an error, false).
__device__ __forceinline__ bool wait_arrivals(const unsigned* sw, unsigned need, LzShared& C, bool& done)
{
    unsigned w = ld_acquire_u32(sw);
    if (!(w & kDone) && w < need) {
        const unsigned long long t0 = globaltimer_ns();
        unsigned it = 0;
        while (w = ld_acquire_u32(sw), !(w & kDone) && w < need) {
            if ((++it & 63u) == 0u) {
                if (ld_acquire_s32(C.status) != EDZT_DEV_OK) return false;
                if (globaltimer_ns() - t0 > C.wait_ns) {
                    atomicCAS(C.status, EDZT_DEV_OK, EDZT_DEV_BARRIER_TIMEOUT);
                    return false;
                }
            }
        }
    }
    done = (w & kDone) != 0u;
    return true;
}

// Enter job j in phase p: wait for the earlier phases' arrivals and derive
// the run's state (one warp; the rest of the CTA waits at the barrier).
// The closing pass of a slice (closing) opens the next step only: it derives
// a(k-1) and the finish test of a column phase and stores the state, marked
// opened, under both parities for the launch that resumes it.  False: an
// error, leave the kernel.
__device__ __forceinline__ bool begin_job(int j, int p, bool closing)
{
    LzShared& C = lz_shared();
    __syncthreads();                                     // nobody reads the previous job's state any more
    const bool same = (j == C.job);
    if (!same) {
        const int* src = reinterpret_cast<const int*>(C.jobs + j);
        int* dst = reinterpret_cast<int*>(&C.J);
        for (int i = threadIdx.x; i < (int)(sizeof(LzJob) / sizeof(int)); i += blockDim.x) dst[i] = __ldg(src + i);
        __syncthreads();
        if (threadIdx.x == 0) {
            C.wint = reinterpret_cast<double*>(&C + 1);
            C.amp_up = C.wint + C.J.S.P * C.J.S.P;
            C.amp_dn = C.amp_up + C.J.S.up.namp;
            C.dg = C.amp_dn + C.J.S.dn.namp;
            C.vsize = lz_vec_size(C.J.S.up.count, C.J.S.dn.count);
        }
        __syncthreads();
        stage_table(C.J.S.wint, C.J.S.P * C.J.S.P, C.wint);
        stage_table(C.J.S.up.amp, C.J.S.up.namp, C.amp_up);
        stage_table(C.J.S.dn.amp, C.J.S.dn.namp, C.amp_dn);
    }
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x, ph = p & 1;
        const LzPhase& O = C.J.ph[ph ^ 1];
        unsigned* word = C.sync + 32 * (size_t)j;
        int ok = 1, done = 0;
        // a run that only this CTA takes part in: nothing to wait for, its sum is here
        const bool alone = same && C.phase == p - 1 && C.J.ph[0].npart == 1 && C.J.ph[1].npart == 1 &&
                           C.J.ph[0].part0 == C.J.ph[1].part0;
        if (lane == 0 && p > 0 && !alone) {
            bool d = false;
            const unsigned need = (unsigned)((p + 1) / 2) * C.J.ph[0].npart + (unsigned)(p / 2) * C.J.ph[1].npart;
            ok = wait_arrivals(word, need, C, d);
            done = d;
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        done = __shfl_sync(0xffffffffu, done, 0);
        // the partial sums of the previous phase, in participant order
        double sum = 0.0;
        if (alone) sum = (lane == 0) ? C.sum : 0.0;
        else if (ok && !done && p > 0)
            for (int i = lane; i < O.npart; i += 32) sum += __ldcg(C.slots + O.slot0 + i);
        sum = warp_sum(sum);
        if (lane == 0) {
            if (!(same && C.phase == p - 1)) {           // else derived here in the previous phase
                const int* ss = reinterpret_cast<const int*>(C.J.st + ((p + 1) & 1));
                int* sd = reinterpret_cast<int*>(&C.S);
                for (int i = 0; i < (int)(sizeof(LzState) / sizeof(int)); i++) sd[i] = __ldcg(ss + i);
            }
            LzState& n = C.S;
            const bool out = ((int)blockIdx.x == C.J.ph[ph].part0);   // the job's first participant
            const bool coeff = (C.J.mode == LZ_COEFF);
            const bool resumed = (ph == 0 && n.opened);  // step already opened by a closing pass
            if (ph == 0 && !n.opened) n.k += 1;          // the column phase opens the next step
            n.opened = 0;
            const int k = n.k;
            if (done) n.active = 0;
            auto finish = [&](int nstep) {
                n.active = 0;
                n.nstep = nstep;
            };
            if (n.active && !resumed) {
                if (ph == 0) {
                    if (k >= 2) {                        // a(k-1) = <w, y> of the last row phase (:134,159)
                        const double a = coeff ? sum : C.J.a[k - 2];
                        if (out && coeff) C.J.a[k - 2] = a;
                        n.a_prev = a;
                        if (k - 1 >= C.J.maxnstep) finish(k - 1);             // :137-141, :161-164
                    } else {
                        n.a_prev = 0.0;
                    }
                } else {
                    n.b_prev = n.b_cur;
                    if (k == 1) {                        // ||v_init|| (:128-130); b(1) = 0 (:135)
                        const double nrm = sqrt(sum);
                        n.norm0 = nrm;
                        n.b_cur = nrm;
                        if (out && coeff) C.J.b[0] = 0.0;
                        if (!(nrm > 0.0)) finish(0);     // zero start vector
                    } else {                             // b(k) = ||v_k|| (:144,167), breakdown (:161)
                        const double bk = coeff ? sqrt(sum) : C.J.b[k - 1];
                        if (coeff && bk < 1.0e-16) {
                            if (out) C.J.b[k - 1] = 0.0;
                            finish(k - 1);
                        } else {
                            if (out && coeff) C.J.b[k - 1] = bk;
                            n.b_cur = bk;
                        }
                    }
                }
                if (closing && n.active) n.opened = 1;
            }
            if (out && !done) {                          // published by the arrival (or the launch's end)
                C.J.st[p & 1] = n;
                if (closing) C.J.st[(p + 1) & 1] = n;
                if (!n.active) {
                    __threadfence();
                    atomicOr(word, kDone);
                }
            }
            C.vk = lz_v(C.J, k, C.vsize);
            C.vp = lz_v(C.J, k - 1, C.vsize);
            C.rb = 1.0 / n.b_cur;
            C.rp = (k >= 2 && ph == 1) ? 1.0 / n.b_prev : 0.0;
            C.job = j;
            C.phase = p;
            C.ok = ok;
        }
    }
    __syncthreads();
    return C.ok != 0;
}

// Leave the current job in phase ph with this thread's share acc of the sum.
__device__ __forceinline__ void end_job(int ph, double acc)
{
    LzShared& C = lz_shared();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    acc = warp_sum(acc);
    if (lane == 0) C.red[wid] = acc;
    __syncthreads();                                     // this CTA's stores of the phase are before it
    if (wid == 0) {
        double s = (lane < (int)(blockDim.x >> 5)) ? C.red[lane] : 0.0;
        s = warp_sum(s);
        if (lane == 0) {
            const int q = (int)blockIdx.x - C.J.ph[ph].part0;
            EDZT_OK_OR(q >= 0 && q < C.J.ph[ph].npart, 24, blockIdx.x, C.J.ph[ph].tile0, C.J.ph[ph].npart, return)
            __stcg(C.slots + C.J.ph[ph].slot0 + q, s);
            red_release_add(C.sync + 32 * (size_t)C.job, 1u);
            C.sum = s;
        }
    }
}

// Column phase of step k on the NP slabs of PW columns at list positions
// t, t + 1, ...: stage v_k on their columns of every row, store it, sum v^2,
// write the down-hop part of H v_k over y.  Returns this thread's share of
// the sum.
// col_init: step 1 from the start vector, or a resumed step from its kept v_k.
template <int PW>
__device__ __noinline__ double col_init(int np)
{
    constexpr int H = PW / 2;
    LzShared& C = lz_shared();
    const int nup = C.J.S.up.count, ndn = C.J.S.dn.count, ndp = lz_pad(ndn), ps = ndp * PW, n = ndp * H;
    double* ws = C.chunk;
    double* vk = C.vk;
    const bool kept = C.S.k > 1;
    double acc = 0.0;
    for (int q = 0; q < np; q++)
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const int id = i / (4 * H) * 4 + 2 * (i & 1), cc = (i >> 1) & (PW - 1), c = C.c0[q] + cc;
            double2 v = make_double2(0.0, 0.0);
            const unsigned o = (unsigned)(C.c0[q] / 4 * 4 * ndp) + (H == 2 ? 2u * i : (unsigned)(i / 4 * 16 + (C.c0[q] & 2) * 4 + i % 4 * 2));
            if (kept) {
                v = __ldcg(reinterpret_cast<const double2*>(vk + o));
            } else {
                if (c < nup && id < ndn) v.x = init_value(C.J, id, c);
                if (c < nup && id + 1 < ndn) v.y = init_value(C.J, id + 1, c);
                __stcg(reinterpret_cast<double2*>(vk + o), v);
            }
            double* d = ws + q * ps + id * PW + cc;
            d[0] = v.x;
            d[PW] = v.y;
            acc = fma(v.x, v.x, acc);
            acc = fma(v.y, v.y, acc);
        }
    return acc;
}

template <int NP, int PW, int T>
__device__ __forceinline__ double col_tile(int np, int t_next)
{
    constexpr int H = PW / 2;
    LzShared& C = lz_shared();
    
    double acc = 0.0;
    const DevSpin& dn = C.J.S.dn;
    const int nup = C.J.S.up.count, ndn = dn.count, k = C.S.k, ndp = lz_pad(ndn), ps = ndp * PW;
    double* ws = C.chunk;                              // [NP][ndp][PW]
    double* __restrict__ vk = C.vk;
    double* __restrict__ yd = C.J.Y;
    // Staged item i of plane q: 16 bytes, two rows of one column.  A slab of
    // four columns is one contiguous run of blocks (a slab of two the halves
    // of its blocks), read and written in storage order: whole lines per warp.
    const int n = ndp * H;
    auto off = [&](int q, int i) {
        return (unsigned)(C.c0[q] / 4 * 4 * ndp) + (H == 2 ? 2u * i : (unsigned)(i / 4 * 16 + (C.c0[q] & 2) * 4 + i % 4 * 2));
    };
    auto put = [&](int q, int i, unsigned o, double2 v) {
        const int id = i / (4 * H) * 4 + 2 * (i & 1), cc = (i >> 1) & (PW - 1), c = C.c0[q] + cc;
        if (c >= nup) v = make_double2(0.0, 0.0);        // the padding holds nothing
        if (id + 1 >= ndn) {
            v.y = 0.0;
            if (id >= ndn) v.x = 0.0;
        }
        double* d = ws + q * ps + id * PW + cc;
        d[0] = v.x;
        d[PW] = v.y;
        __stcg(reinterpret_cast<double2*>(vk + o), v);
        acc = fma(v.x, v.x, acc);
        acc = fma(v.y, v.y, acc);
    };
    if (k == 1 || k == C.J.resume) {
        acc = col_init<PW>(np);
    } else {
        const double* __restrict__ vp = C.vp;
        const double am = -C.S.a_prev, bp = C.S.b_cur, rp = C.rb;
        constexpr int U = T > 256 ? 4 : 3;       // pairs of y and of v_{k-1} in flight per thread
#pragma unroll 1
        for (int q = 0; q < np; q++)
            for (int i0 = threadIdx.x; i0 < n; i0 += U * T) {
                double2 yy[U], vv[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int i = i0 + u * T;
                    if (i < n) {
                        yy[u] = __ldcg(reinterpret_cast<const double2*>(yd + off(q, i)));
                        vv[u] = __ldcg(reinterpret_cast<const double2*>(vp + off(q, i)));
                    }
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int i = i0 + u * T;
                    if (i < n)
                        put(q, i, off(q, i), make_double2(fma(am, div_by(vv[u].x, bp, rp), yy[u].x),
                                                          fma(am, div_by(vv[u].y, bp, rp), yy[u].y)));
                }
            }
    }
    __syncthreads();
    // the next tile's slabs, on their way during this one's hop sums
    const int c_next = ((int)threadIdx.x < NP) ? (int)__ldg(C.slab_of + t_next + threadIdx.x) * PW : 0;
    HopList nxt{};
    const int m = ndn * H;
    if ((int)threadIdx.x < m) nxt = hop_list(dn, threadIdx.x / H);
    for (int i = threadIdx.x; i < m; i += T) {
        const HopList cur = nxt;                     // this row's hop list; the next one's in flight
        const int id = i / H;
        if (i + T < m) nxt = hop_list(dn, (i + T) / H);
        double2 d[NP];
#pragma unroll
        for (int q = 0; q < NP; q++) d[q] = make_double2(0.0, 0.0);
        plane_hops<NP, PW>(dn, id, cur, C.amp_dn, ws + 2 * (i % H), ps, d, 72);
#pragma unroll
        for (int q = 0; q < NP; q++) {
            if (q < np) {
                double* o = yd + lz_index(id, C.c0[q] + 2 * (i % H), ndp);
                __stcg(o, d[q].x);
                __stcg(o + 4, d[q].y);
            }
        }
    }
    __syncthreads();
    if ((int)threadIdx.x < NP) C.c0[threadIdx.x] = c_next;
    __syncthreads();
    return acc;
}

// Row phase of step k on rows [r0, r0 + NP * PW): stage v_k, finish
// y_k = H w_k - b_k w_{k-1}, store it over D (or also accumulate the
// eigenvector).  Returns this thread's share of <w_k, y_k>.  X: the model has
// exchange terms.
template <int NP, int PW, bool X, int T>
__device__ __forceinline__ double row_tile(int r0, int np)
{
    constexpr int W = NP * PW, H = PW / 2;
    LzShared& C = lz_shared();
    
    double acc = 0.0;
    const DevSpin& up = C.J.S.up;
    const int nup = up.count, ndn = C.J.S.dn.count, k = C.S.k, ndp = lz_pad(ndn), P = C.J.S.P;
    const double* __restrict__ vk = C.vk;
    const double* __restrict__ vp = C.vp;
    double* __restrict__ yd = C.J.Y;
    const double bk = C.S.b_cur, rb = C.rb, bp = C.S.b_prev, rp = C.rp;
    const bool first = (k == 1);
    const int nr = min(W, ndn - r0), ps = nup * PW;
    double* xs = C.chunk;                              // [NP][nup][PW]
    const int m = nup * H;
    for (int i = threadIdx.x; i < W * P; i += T) {
        const int r = i / P, pu = i - r * P;
        const bool in = r < nr;
        const int pd = in ? __ldg(C.J.S.dn.imp + r0 + r) : 0;
        C.dg[i] = in ? __ldg(C.J.S.dn.e1 + r0 + r) + C.wint[pu * P + pd] : 0.0;
        if (pu == 0) C.pd[r] = pd;
    }
    // item i: column i / H, rows r0 + 2 * (i % H) and the next of every plane
    auto at = [&](int i) { return lz_index(r0 + 2 * (i % H), i / H, ndp); };
    for (int i = threadIdx.x; i < m; i += T) {       // the whole tile in flight at once
        const unsigned o = at(i);
#pragma unroll
        for (int p = 0; p < NP; p++)
            if (p < np) copy_async16(xs + (size_t)p * ps + 2 * i, vk + o + 16 * p);
    }
    HopList nxt{};
    double2 sn[NP], wn[NP];                          // D and v_{k-1} of the next item
    auto load_next = [&](int i) {
        const unsigned o = at(i);
#pragma unroll
        for (int p = 0; p < NP; p++) {
            sn[p] = wn[p] = make_double2(0.0, 0.0);
            if (p >= np) break;
            sn[p] = __ldcg(reinterpret_cast<const double2*>(yd + o + 16 * p));
            wn[p] = first ? make_double2(0.0, 0.0) : __ldcg(reinterpret_cast<const double2*>(vp + o + 16 * p));
        }
    };
    if ((int)threadIdx.x < m) nxt = hop_list(up, threadIdx.x / H);
    copy_async_wait_all();
    __syncthreads();
    if (C.J.mode != LZ_COEFF) {                       // eigenvector pass: += coeff_k w_k
        const double ck = C.J.coeff[k - 1];
        for (int i = threadIdx.x; i < m; i += T) {
#pragma unroll
            for (int p = 0; p < NP; p++) {
                if (p >= np) break;
                const double2 v = *reinterpret_cast<const double2*>(xs + (size_t)p * ps + 2 * i);
                double2* e = reinterpret_cast<double2*>(C.J.eig + at(i) + 16 * p);
                double2 z = first ? make_double2(0.0, 0.0) : __ldcg(e);
                z.x = fma(ck, div_by(v.x, bk, rb), z.x);
                z.y = fma(ck, div_by(v.y, bk, rb), z.y);
                __stcg(e, z);
            }
        }
    }
    auto fetch = [&](int id2, int iu2) { return __ldcg(vk + lz_index(id2, iu2, ndp)); };
    for (int i = threadIdx.x; i < m; i += T) {
        const HopList cur = nxt;
        load_next(i);
        if (i + T < m) nxt = hop_list(up, (i + T) / H);
        double2 s[NP];
#pragma unroll
        for (int p = 0; p < NP; p++) s[p] = make_double2(0.0, 0.0);
        const int iu = i / H, h = i - iu * H;
        const double e1u = __ldg(up.e1 + iu);
        const int pu = __ldg(up.imp + iu);

        plane_hops<NP, PW>(up, iu, cur, C.amp_up, xs + 2 * h, ps, s, 71);
        double* out = yd + at(i);
#pragma unroll
        for (int p = 0; p < NP; p++) {
            if (p >= np) break;
            const int r = p * PW + 2 * h;
            const double2 v = *reinterpret_cast<const double2*>(xs + (size_t)p * ps + 2 * i);
            auto row = [&](int rr, double sum, double vv, double dd, double ww) {
                double y = fma(e1u + C.dg[rr * P + pu], vv, sum);
                if constexpr (X) { if (C.J.S.has_j && rr < nr) y = exchange_part(C.J.S, r0 + rr, iu, pu, C.pd[rr], y, fetch); }
                y = fma(-bk, div_by(ww, bp, rp), div_by(y + dd, bk, rb));
                if (rr < nr) acc = fma(div_by(vv, bk, rb), y, acc);
                return y;
            };
            double2 y;
            y.x = row(r, s[p].x, v.x, sn[p].x, wn[p].x);
            y.y = row(r + 1, s[p].y, v.y, sn[p].y, wn[p].y);
            __stcg(reinterpret_cast<double2*>(out + 16 * p), y);
        }
    }
    __syncthreads();
    return acc;
}

// Row phase of one row, for lines so long that two do not fit (13,400 up
// strings or more: nsite 17 and beyond).  It sums in row_tile's order: the
// eigenvector pass of a shorter sector of the same scan runs there.
template <bool X, int T>
__device__ __forceinline__ double long_row(int r0)
{
    LzShared& C = lz_shared();
    const DevSpin& up = C.J.S.up;
    const int nup = up.count, k = C.S.k, ndp = lz_pad(C.J.S.dn.count), P = C.J.S.P;
    const double* __restrict__ vk = C.vk;
    const double* __restrict__ vp = C.vp;
    const double bk = C.S.b_cur, rb = C.rb, bp = C.S.b_prev, rp = C.rp;
    double* xs = C.chunk;                                // [nup]
    double acc = 0.0;
    for (int iu = threadIdx.x; iu < nup; iu += T) copy_async8(xs + iu, vk + lz_index(r0, iu, ndp), true);
    const int pd = __ldg(C.J.S.dn.imp + r0);
    const double e1d = __ldg(C.J.S.dn.e1 + r0);
    copy_async_wait_all();
    __syncthreads();
    auto fetch = [&](int id2, int iu2) { return __ldcg(vk + lz_index(id2, iu2, ndp)); };
    for (int iu = threadIdx.x; iu < nup; iu += T) {
        const unsigned o = lz_index(r0, iu, ndp);
        const int hc = __ldg(up.hcnt + iu), pu = __ldg(up.imp + iu);
        const double v = xs[iu];
        double y = 0.0;
        for (int h = 0; h < hc; h++) {
            const uint32_t e = __ldg(reinterpret_cast<const uint32_t*>(up.hpk) + ((size_t)(h >> 2) * nup + iu) * 4 + (h & 3));
            y = fma(C.amp_up[edzt_hop_slot(e)], xs[edzt_hop_rank(e)], y);
        }
        y = fma(__ldg(up.e1 + iu) + (e1d + C.wint[pu * P + pd]), v, y);
        if constexpr (X) { if (C.J.S.has_j) y = exchange_part(C.J.S, r0, iu, pu, pd, y, fetch); }
        const double w = div_by(v, bk, rb);
        y = fma(-bk, k == 1 ? 0.0 : div_by(__ldcg(vp + o), bp, rp), div_by(y + __ldcg(C.J.Y + o), bk, rb));
        __stcg(C.J.Y + o, y);
        acc = fma(w, y, acc);
        if (C.J.mode != LZ_COEFF) {
            const double z = (k == 1) ? 0.0 : __ldcg(C.J.eig + o);
            __stcg(C.J.eig + o, fma(C.J.coeff[k - 1], w, z));
        }
    }
    __syncthreads();
    return acc;
}

// NC planes of PW columns of a column tile; NR planes of PR rows of a row
// tile (PR 1: one row); X: a model of the launch has exchange terms.
template <int NC, int NR, int PW, int PR, bool X, int T>
__global__ void __launch_bounds__(T, kLzThreads / T) k_lanczos(LzBatch B, const LzJob* __restrict__ jobs,
                                                           const long long* __restrict__ prefix, double* slots,
                                                           unsigned* sync, int* status)
{
    LzShared& C = lz_shared();
    const int G = gridDim.x;
    if (threadIdx.x == 0) {
        C.jobs = jobs;
        C.slab_of = prefix + 2 * (size_t)(B.njobs + 1) + 2 * (size_t)(G + 1);
        C.slots = slots;
        C.sync = sync;
        C.status = status;
        C.wait_ns = B.wait_ns ? B.wait_ns : kBarrierTimeoutNs;
        C.job = C.phase = -1;
        C.chunk = reinterpret_cast<double*>(lz_smem + B.fixed);
    }
    __syncthreads();
    // This CTA's positions of each phase, [t0, t1), and the job of the first:
    // looked up once, since every arrival that is waited for empties the L1.
    const long long* range = prefix + 2 * (size_t)(B.njobs + 1);
    const int t0c = (int)__ldg(range + blockIdx.x), t1c = (int)__ldg(range + blockIdx.x + 1);
    const int t0r = (int)__ldg(range + G + 1 + blockIdx.x), t1r = (int)__ldg(range + G + 2 + blockIdx.x);
    const int j0c = find_job(prefix, B.njobs, t0c), j0r = find_job(prefix + B.njobs + 1, B.njobs, t0r);
    const int e0c = min(t1c, (int)__ldg(prefix + j0c + 1)), e0r = min(t1r, (int)__ldg(prefix + B.njobs + 2 + j0r));
    if (threadIdx.x < NC && t0c < t1c) C.c0[threadIdx.x] = (int)__ldg(C.slab_of + t0c + threadIdx.x) * PW;
    const bool stalled = (int)blockIdx.x == B.stall_cta;
    int p = 0, idle = 0;
    for (; p < B.max_phases; p++) {
        const int ph = p & 1;
        const int t_end = ph ? t1r : t1c;
        int t = ph ? t0r : t0c, j = ph ? j0r : j0c, j_end = ph ? e0r : e0c;
        bool alive = false;
        while (t < t_end) {
            if (!begin_job(j, p, false)) return;
            if (C.S.active) {
                alive = true;
                double acc = 0.0;
                // a tile: the job's next list positions, one per plane
                if (ph == 0) {
#pragma unroll 1
                    while (t < j_end) {
                        const int np = min(NC, j_end - t);
                        t += np;
                        acc += col_tile<NC, PW, T>(np, t < t_end ? t : t0c);
                    }
                } else {
#pragma unroll 1
                    for (; t < j_end; t += NR) {
                        const int r0 = (t - (int)C.J.ph[1].tile0) * PR;
                        if constexpr (PR == 1) acc += long_row<X, T>(r0);
                        else acc += row_tile<NR, PR, X, T>(r0, min(NR, j_end - t));
                    }
                }
                if (stalled) return;                     // fault test: leave without arriving
                end_job(ph, acc);
            } else if (ph == 0) {                        // a finished run's slabs are passed over
                __syncthreads();
                const int tn = j_end < t_end ? j_end : t0c;
                if (threadIdx.x < NC) C.c0[threadIdx.x] = (int)__ldg(C.slab_of + tn + threadIdx.x) * PW;
            }
            t = j_end;
            j++;
            if (t < t_end) j_end = min(t_end, (int)__ldg(prefix + (ph ? B.njobs + 1 : 0) + j + 1));
        }
        // every run of both phases' lists has finished
        idle = alive ? 0 : idle + 1;
        if (idle >= 2) return;
    }
    if (B.slice) {                                       // budget spent: open every run's next step
        int j = j0c, j_end = e0c;
        for (int t = t0c; t < t1c; t = j_end, j++) {
            j_end = min(t1c, (int)__ldg(prefix + j + 1));
            if (!begin_job(j, p, true)) return;
        }
    }
}

#ifdef EDZT_DEVICE_CHECKS
int lz_debug_bad(long long* out4)
{
    return cudaMemcpyFromSymbol(out4, g_edzt_bad, 4 * sizeof(long long)) == cudaSuccess ? 0 : 2;
}
#endif

using LzKernel = void (*)(LzBatch, const LzJob*, const long long*, double*, unsigned*, int*);

// The kernel of a tile shape: wc columns by r rows (two CTAs of half the
// threads only of shapes that have a use for them).
static LzKernel lz_kernel(const LzPlan& P)
{
#define EDZT_LZ(c, w, nc, nr, pw, pr)                                                                    \
    if (P.wc == c && P.r == w && P.block == kLzThreads)                                                  \
        return P.exchange ? k_lanczos<nc, nr, pw, pr, true, kLzThreads>                                  \
                          : k_lanczos<nc, nr, pw, pr, false, kLzThreads>;
#define EDZT_LZ2(c, w, nc, nr, pw, pr)                                                                   \
    EDZT_LZ(c, w, nc, nr, pw, pr)                                                                        \
    if (P.wc == c && P.r == w && P.block == kLzThreads / 2)                                              \
        return P.exchange ? k_lanczos<nc, nr, pw, pr, true, kLzThreads / 2>                              \
                          : k_lanczos<nc, nr, pw, pr, false, kLzThreads / 2>;
    EDZT_LZ2(16, 8, 4, 2, 4, 4)
    EDZT_LZ2(8, 8, 2, 2, 4, 4)
    EDZT_LZ2(8, 4, 2, 1, 4, 4)
    EDZT_LZ(8, 2, 2, 1, 4, 2)
    EDZT_LZ(8, 1, 2, 1, 4, 1)
    EDZT_LZ(4, 8, 1, 2, 4, 4)
    EDZT_LZ2(4, 4, 1, 1, 4, 4)
    EDZT_LZ(4, 2, 1, 1, 4, 2)
    EDZT_LZ(4, 1, 1, 1, 4, 1)
    EDZT_LZ(2, 8, 1, 2, 2, 4)
    EDZT_LZ(2, 4, 1, 1, 2, 4)
    EDZT_LZ2(2, 2, 1, 1, 2, 2)
    EDZT_LZ2(2, 1, 1, 1, 2, 1)
#undef EDZT_LZ2
#undef EDZT_LZ
    return nullptr;
}

int lz_grid_size(int device, const LzPlan& P)
{
    int per_sm = 0, nsm = 0;
    const LzKernel k = lz_kernel(P);
    cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLzSmemMax);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)k, P.block, P.smem);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
    return per_sm * nsm;
}

cudaError_t launch_lanczos_persistent(const LzPlan& P, const LzBatch& B, const LzJob* jobs, const long long* prefix,
                                      double* slots, unsigned* sync_words, int* status, cudaStream_t s)
{
    LzBatch b = B;
    b.fixed = P.fixed;
    void* args[] = {(void*)&b, (void*)&jobs, (void*)&prefix, (void*)&slots, (void*)&sync_words, (void*)&status};
    return cudaLaunchCooperativeKernel((const void*)lz_kernel(P), dim3(P.grid), dim3(P.block), args,
                                       P.smem, s);
}

// ---------------------------------------------------------------------------
// small runs: one CTA a run, everything in shared memory
// ---------------------------------------------------------------------------
// Small runs spend their steps in the persistent kernel on latency: staging,
// arrivals, the tables' way through L2, 4.5 us a phase even for a few hundred
// states.  Here the last two v, y, the hop lists and the tables of a run stay
// in the shared memory of one CTA, and a step is two sums over it.  Four rows
// of a column share the decode of an up hop; 768 threads, since 512 left the
// issue slots idle half of the time and 1,024 run out of columns.  Bound by
// the instructions and wavefronts of the hop sums.  A step of a lone run, in
// us (persistent kernel): 400 states 1.9 (8.7), 1,225 3.3 (8.7), 4,900 6.5
// (8.8), 7,056 9.8 (8.9), with the v_k kept up to a fifth more.  The line lies
// where a step still takes less than half: with larger runs in the same call
// these come in a launch of their own, before the others'.
constexpr long long kLzSmallStates = 2000;
constexpr size_t kLzSmallSmemMax = kLzSmemMax - 4096;   // besides the descriptor and the sums

// Where a run's parts lie in shared memory, in bytes.
struct LzSmall {
    int hu, hd;                   // hop lists
    int v, wint, amp_up, amp_dn, e1u, e1d;   // v: v0, v1 and y
    int cu, cd, pu, pd;           // hop counts, impurity patterns
    int size;
};

__host__ __device__ inline LzSmall lz_small_layout(const DevSector& S)
{
    LzSmall L;
    int o = 0;
    auto part = [&o](long long bytes) {
        const int at = o;
        o += (int)((bytes + 15) / 16 * 16);
        return at;
    };
    L.hu = part(4LL * S.up.hw * S.up.count);
    L.hd = part(4LL * S.dn.hw * S.dn.count);
    L.v = part(24LL * S.dim);
    L.wint = part(8LL * S.P * S.P);
    L.amp_up = part(8LL * S.up.namp);
    L.amp_dn = part(8LL * S.dn.namp);
    L.e1u = part(8LL * S.up.count);
    L.e1d = part(8LL * S.dn.count);
    L.cu = part(S.up.count);
    L.cd = part(S.dn.count);
    L.pu = part(S.up.count);
    L.pd = part(S.dn.count);
    L.size = o;
    return L;
}

// Sum over the CTA, the same in every thread.  Alternating buffers: the next
// sum's writes need no barrier behind this one's reads.
template <int T>
__device__ __forceinline__ double cta_sum(double v, double* red)
{
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = ((int)(threadIdx.x & 31) < T / 32) ? red[threadIdx.x & 31] : 0.0;
    return __shfl_sync(0xffffffffu, warp_sum(v), 0);
}

// T threads; R: rows of one column that a thread sums at a time.
template <int T, int R, bool X>
__global__ void __launch_bounds__(T) k_lanczos_small(const LzJob* __restrict__ jobs)
{
    __shared__ LzJob J;
    __shared__ double red[2][32];
    {
        const int* src = reinterpret_cast<const int*>(jobs + blockIdx.x);
        int* dst = reinterpret_cast<int*>(&J);
        for (int i = threadIdx.x; i < (int)(sizeof(LzJob) / sizeof(int)); i += T) dst[i] = __ldg(src + i);
    }
    __syncthreads();
    const DevSpin &up = J.S.up, &dn = J.S.dn;
    const int nup = up.count, ndn = dn.count, n = nup * ndn, P = J.S.P, ndp = lz_pad(ndn);
    const LzSmall L = lz_small_layout(J.S);
    uint4* hu = reinterpret_cast<uint4*>(lz_smem + L.hu);
    uint4* hd = reinterpret_cast<uint4*>(lz_smem + L.hd);
    double* v = reinterpret_cast<double*>(lz_smem + L.v);
    double* vp = v + n;
    double* y = vp + n;
    double* wint = reinterpret_cast<double*>(lz_smem + L.wint);
    double* amp_up = reinterpret_cast<double*>(lz_smem + L.amp_up);
    double* amp_dn = reinterpret_cast<double*>(lz_smem + L.amp_dn);
    double* e1u = reinterpret_cast<double*>(lz_smem + L.e1u);
    double* e1d = reinterpret_cast<double*>(lz_smem + L.e1d);
    unsigned char *cu = lz_smem + L.cu, *cd = lz_smem + L.cd, *pu = lz_smem + L.pu, *pd = lz_smem + L.pd;
    for (int i = threadIdx.x; i < up.hw / 4 * nup; i += T) hu[i] = __ldg(up.hpk + i);
    for (int i = threadIdx.x; i < dn.hw / 4 * ndn; i += T) hd[i] = __ldg(dn.hpk + i);
    stage_table(J.S.wint, P * P, wint);
    stage_table(up.amp, up.namp, amp_up);
    stage_table(dn.amp, dn.namp, amp_dn);
    stage_table(up.e1, nup, e1u);
    stage_table(dn.e1, ndn, e1d);
    for (int i = threadIdx.x; i < nup; i += T) { cu[i] = __ldg(up.hcnt + i); pu[i] = __ldg(up.imp + i); }
    for (int i = threadIdx.x; i < ndn; i += T) { cd[i] = __ldg(dn.hcnt + i); pd[i] = __ldg(dn.imp + i); }
    // e / nup = umulhi(e, magic) for e < n: the error e * nup / 2^32 stays below 1 / nup
    const unsigned magic = nup > 1 ? 0xffffffffu / nup + 1 : 0;
    auto row_of = [&](int e) { return nup > 1 ? (int)__umulhi((unsigned)e, magic) : e; };
    const long long vsize = lz_vec_size(nup, ndn);
    const int items = (ndn + R - 1) / R * nup;
    // The eigenvector pass takes the scan's steps again, all of them in this
    // form of the kernel: a, b and every vector have the scan's bits.
    const bool coeff = J.mode == LZ_COEFF;
    double a = 0.0, bk = 1.0, rb = 1.0, bp = 1.0, rp = 0.0, norm0 = 0.0;   // a_{k-1}; b_k, b_{k-1} and their reciprocals
    int nstep = 0;
    for (int k = 1;; k++) {
        double* kept = J.keep ? lz_v(J, k, vsize) : nullptr;
        double acc = 0.0;
        auto put = [&](int e, double x) {
            v[e] = x;
            acc = fma(x, x, acc);
            if (kept) {
                const int id = row_of(e);
                __stcg(kept + lz_index(id, e - id * nup, ndp), x);
            }
        };
        if (k == 1) {
            for (int e = threadIdx.x; e < n; e += T) {
                const int id = row_of(e);
                put(e, init_value(J, id, e - id * nup));
            }
        } else {                                         // v_k = y - a_{k-1} w_{k-1}
            for (int e0 = threadIdx.x; e0 < n; e0 += R * T) {
                double x[R];
#pragma unroll
                for (int u = 0; u < R; u++) {
                    const int e = e0 + u * T;
                    if (e < n) x[u] = fma(-a, div_by(vp[e], bk, rb), y[e]);
                }
#pragma unroll
                for (int u = 0; u < R; u++) {
                    const int e = e0 + u * T;
                    if (e < n) put(e, x[u]);
                }
            }
        }
        const double nrm = sqrt(cta_sum<T>(acc, red[0]));
        bp = bk;
        rp = rb;
        if (k == 1) {                                    // ||v_init|| (:128-130); b(1) = 0 (:135)
            norm0 = nrm;
            if (coeff && threadIdx.x == 0) J.b[0] = 0.0;
            if (!(nrm > 0.0)) break;                     // zero start vector
        } else if (nrm < 1.0e-16) {                      // breakdown (:161)
            if (coeff && threadIdx.x == 0) J.b[k - 1] = 0.0;
            break;
        } else if (coeff && threadIdx.x == 0) {
            J.b[k - 1] = nrm;                            // b(k) = ||v_k|| (:144,167)
        }
        bk = nrm;
        rb = 1.0 / bk;
        acc = 0.0;
        for (int i = threadIdx.x; i < items; i += T) {   // y = H w_k - b_k w_{k-1}
            const int blk = row_of(i), iu = i - blk * nup, r0 = blk * R;
            const double* line[R];                       // rows past the last one repeat it
            double s[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int id = min(r0 + r, ndn - 1);
                line[r] = v + id * nup;
                s[r] = (e1u[iu] + e1d[id] + wint[pu[iu] * P + pd[id]]) * line[r][iu];
            }
            const int hcu = cu[iu];
            for (int h0 = 0; h0 < hcu; h0 += 4) {
                const uint4 q = hu[(h0 >> 2) * nup + iu];
                const uint32_t f[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int h = 0; h < 4; h++)
                    if (h0 + h < hcu) {
                        const double am = amp_up[edzt_hop_slot(f[h])];
                        const int t = edzt_hop_rank(f[h]);
#pragma unroll
                        for (int r = 0; r < R; r++) s[r] = fma(am, line[r][t], s[r]);
                    }
            }
            int hcd[R], most = 0;
#pragma unroll
            for (int r = 0; r < R; r++) {
                hcd[r] = cd[min(r0 + r, ndn - 1)];
                most = max(most, hcd[r]);
            }
            for (int h0 = 0; h0 < most; h0 += 4)
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if (h0 >= hcd[r]) continue;
                    const uint4 q = hd[(h0 >> 2) * ndn + min(r0 + r, ndn - 1)];
                    const uint32_t f[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                    for (int h = 0; h < 4; h++)
                        if (h0 + h < hcd[r]) s[r] = fma(amp_dn[edzt_hop_slot(f[h])], v[edzt_hop_rank(f[h]) * nup + iu], s[r]);
                }
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int id = r0 + r;
                if (id >= ndn) break;
                if constexpr (X) {
                    if (J.S.has_j)
                        s[r] = exchange_part(J.S, id, iu, pu[iu], pd[id], s[r],
                                             [&](int id2, int iu2) { return v[id2 * nup + iu2]; });
                }
                double z = div_by(s[r], bk, rb);
                if (k > 1) z = fma(-bk, div_by(vp[id * nup + iu], bp, rp), z);
                y[id * nup + iu] = z;
                const double w = div_by(line[r][iu], bk, rb);
                acc = fma(w, z, acc);
                if (!coeff) {                            // += coeff_k w_k, this thread's element in every step
                    double* e = J.eig + lz_index(id, iu, ndp);
                    __stcg(e, fma(__ldg(J.coeff + k - 1), w, k == 1 ? 0.0 : __ldcg(e)));
                }
            }
        }
        a = cta_sum<T>(acc, red[1]);                        // a(k) = <w_k, y_k> (:134,159)
        if (coeff && threadIdx.x == 0) J.a[k - 1] = a;
        nstep = k;
        if (k >= J.maxnstep) break;                      // :137-141, :161-164
        double* t = v;
        v = vp;
        vp = t;
    }
    if (threadIdx.x == 0) {
        LzState f;
        f.k = nstep + 1;
        f.active = f.opened = 0;
        f.nstep = nstep;
        f.a_prev = a;
        f.b_cur = bk;
        f.b_prev = bp;
        f.norm0 = norm0;
        J.st[0] = f;
        J.st[1] = f;
    }
}

size_t lz_small_smem(const DevSector& S)
{
    if (S.dim > kLzSmallStates) return 0;
    const size_t size = (size_t)lz_small_layout(S).size;
    return size <= kLzSmallSmemMax ? size : 0;
}

// Forms 1, 3: up to 512 states, a thread an element; 2, 4: more, four rows of a
// column a thread; 3, 4 with exchange terms.  Chosen by a model's runs alone,
// not by what else is in the launch: the forms differ in the last bits.
int lz_small_form(const DevSector& S) { return 1 + (S.dim > 512 ? 1 : 0) + (S.has_j ? 2 : 0); }

cudaError_t launch_lanczos_small(const LzJob* jobs, int nj, size_t smem, int form, cudaStream_t s)
{
    using Kernel = void (*)(const LzJob*);
    static const Kernel kernels[kSmallForms] = {k_lanczos_small<512, 1, false>, k_lanczos_small<768, 4, false>,
                                                k_lanczos_small<512, 1, true>, k_lanczos_small<768, 4, true>};
    static OnceEach done;
    edzt_once_per_device(done, [&] {                      // where it fails the launch does
        for (const Kernel k : kernels)
            cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLzSmallSmemMax);
    });
    kernels[form - 1]<<<nj, form % 2 ? 512 : 768, smem, s>>>(jobs);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// launch plan
// ---------------------------------------------------------------------------
// Most dynamic shared memory of a CTA of 256 threads, two of which share an SM.
static constexpr size_t kLzSmemTwoPerSm = 113 * 1024;
// Fixed cost of a list position in states, for cutting the list into CTA ranges
static constexpr double kLzTileCost = 256.0;
// A CTA that serves two jobs in a phase reloads tables and waits twice: worth
// this much work in states, or an uneven share of the whole, where the loads of
// both cuts are this close
static constexpr double kLzSwitchCost = 2000.0;
static constexpr double kLzUneven = 1.15;
static constexpr double kLzClose = 1.1;
// Lines of which a few are taken two at a time
static constexpr int kLzLongLine = 500;
// Time of a tile's lines with two CTAs on the SM over their time with one
static constexpr double kLzPairSlowdown = 2.037;
// What a pass over a tile takes besides its lines (staging round, barriers), and
// a job besides its passes (tables, the wait for its arrivals), in lines of 6 ns.
// Fitted to 111 launches of 1 to 169 runs of nsite 6 to 13, timed with one and
// with two CTAs per SM.  The line is drawn between two that lie close: 9 runs of
// nsite 12 (99.8 us a step with two, 105 with one) and two runs of 924 and 495 by
// 792 strings (32.8 and 30.9).  96 of the 111 are taken right to 1%, four are
// missed by 5 to 17% (the c / c^+ runs of ten models of nsite 6 to 9: 12.6 instead
// of 10.8); lines alone at 1.75 miss 28 by more than 5%, one by 145%.
static constexpr double kLzPassLines = 200.0, kLzJobLines = 600.0;

// Load of the busiest CTA of a phase whose CTAs take the ranges `range`, in
// lines: those of its passes (a partly filled tile 0.8 of a pass), `slow` times
// as long as for a CTA that has the SM to itself, its passes and its jobs.
static double phase_load(const LzJob* jobs, int nj, int G, int ph, const long long* range, double slow)
{
    double most = 0.0;
    int j = 0;
    for (int b = 0; b < G; b++) {
        double load = 0.0;
        for (long long t = range[b]; t < range[b + 1];) {
            while (jobs[j].ph[ph].tile0 + jobs[j].ph[ph].ntiles <= t) j++;
            const LzPhase& Q = jobs[j].ph[ph];
            const int lines = (ph == 0) ? jobs[j].S.dn.count : jobs[j].S.up.count, planes = std::max(1, Q.planes);
            const int n = (int)(std::min(range[b + 1], Q.tile0 + Q.ntiles) - t);
            const double full = n / planes, rest = n % planes ? 1.0 : 0.0;
            load += slow * lines * (full + 0.8 * rest) + kLzPassLines * (full + rest) + kLzJobLines;
            t += n;
        }
        most = std::max(most, load);
    }
    return most;
}

// Both phases of a plan.
static double lz_load(const LzJob* jobs, int nj, int G, const std::vector<long long>& prefix, double slow)
{
    const long long* range = prefix.data() + 2 * (size_t)(nj + 1);
    return phase_load(jobs, nj, G, 0, range, slow) + phase_load(jobs, nj, G, 1, range + G + 1, slow);
}

LzPlan lz_plan(int device, LzJob* jobs, int nj, std::vector<long long>& prefix, const LzShape* force)
{
    LzPlan P;
    int tables = 0, lines_up = 0, lines_dn = 0, nsm = 0;
    long long columns = 0, rows = 0;                     // in groups of four
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
    for (int j = 0; j < nj; j++) {
        const DevSector& S = jobs[j].S;
        columns += (S.up.count + 3) / 4;
        rows += (S.dn.count + 3) / 4;
        lines_up = std::max(lines_up, S.up.count);
        lines_dn = std::max(lines_dn, S.dn.count);
        tables = std::max(tables, table_doubles(S.P, std::max(S.up.namp, S.dn.namp)));
        P.exchange = P.exchange || S.has_j;
    }
    P.fixed = fixed_bytes(tables);
    auto chunk = [&](int wc, int r) { return std::max(lz_col_smem(lines_dn, wc), lz_row_smem(lines_up, r)); };
    auto shape = [&](LzPlan& Q, int wc, int r, int block) {
        Q.wc = wc;
        Q.r = r;
        Q.block = block;
        Q.smem = Q.fixed + chunk(wc, r);
        return Q.smem <= (block < kLzThreads ? kLzSmemTwoPerSm : kLzSmemMax);
    };
    auto cut = [&](LzPlan& Q, std::vector<long long>& pre) {
        for (int j = 0; j < nj; j++) {
            jobs[j].ph[0].width = std::min(Q.wc, 4);
            jobs[j].ph[1].width = std::min(Q.r, 4);
            jobs[j].ph[0].planes = Q.wc / jobs[j].ph[0].width;
            jobs[j].ph[1].planes = Q.r / jobs[j].ph[1].width;
        }
        Q.grid = lz_grid_size(device, Q);
        if (Q.grid <= 0) return;
        Q.slots = lz_cut(jobs, nj, Q.grid, pre, Q.total, Q.block < kLzThreads ? kLzPairSlowdown : 1.0);
        lz_group_slabs(jobs, nj, Q.grid, pre);
        pre.resize(pre.size() + kMaxPlanes, 0);          // the kernel reads whole tiles of slab numbers
    };
    LzPlan F = P;
    if (force && shape(F, force->wc, force->r, force->block)) {
        cut(F, prefix);
        return F;
    }
    // The widest tiles that fit one CTA per SM: a hop is decoded once for the
    // lines of a tile (nsite 14: eight lines 202 us a step, four 250).  Columns
    // and rows each by the length of their own lines: rows of 12,870 strings
    // leave tiles of two, but columns of 16 strings are best taken eight at a
    // time (us a step, 2 x 2 and 8 x 2: (8,1) of nsite 16 111 and 68, (8,2) 120
    // and 76; 2 x 2 and 2 x 8: (0,8) 101 and 60, (2,6) of nsite 17 113 and 70).
    // Where fours of long rows, or columns, occupy half of the SMs at most, they
    // are taken two at a time, by twice as many CTAs (8 x 8 and 8 x 2: (7,1) of
    // nsite 14 36 and 27, (7,2) 36 and 28, (6,3) of nsite 12 20.1 and 17.5; 2 x 8:
    // (2,7) of nsite 14 35 and 26); lines of 252 strings gain nothing from it.
    // Tiles of eight lines may also run two CTAs per SM, which overlap one's staging
    // with the other's hop sums but halve what a CTA gets through: taken when
    // the busiest CTA's load (lz_load) is less then than with one CTA per SM (us
    // a step, one / two CTAs: 9 sectors of
    // nsite 12 106 / 99, of nsite 10 18.2 / 15.5; one sector of nsite 12
    // 23 / 31; 2 sectors of nsite 13 92 / 110).
    int wc = 8, r = 8;
    while (wc > 2 && P.fixed + lz_col_smem(lines_dn, wc) > kLzSmemMax) wc /= 2;
    while (r > 1 && P.fixed + lz_row_smem(lines_up, r) > kLzSmemMax) r /= 2;
    if (lines_dn >= kLzLongLine && 2 * columns <= nsm) wc = std::min(wc, 2);
    if (lines_up >= kLzLongLine && 2 * rows <= nsm) r = std::min(r, 2);
    shape(P, wc, r, kLzThreads);
    cut(P, prefix);
    LzPlan Q = P;
    if (P.wc == 8 && P.r == 8 && shape(Q, 8, 8, kLzThreads / 2)) {
        const double one = lz_load(jobs, nj, P.grid, prefix, 1.0);
        std::vector<long long> pre;
        std::vector<LzPhase> mine;                       // the jobs' phases of P
        for (int j = 0; j < nj; j++) mine.insert(mine.end(), jobs[j].ph, jobs[j].ph + 2);
        cut(Q, pre);
        if (Q.grid > P.grid && lz_load(jobs, nj, Q.grid, pre, kLzPairSlowdown) < one) {
            prefix.swap(pre);
            return Q;
        }
        for (int j = 0; j < nj; j++) std::copy_n(mine.data() + 2 * j, 2, jobs[j].ph);
    }
    return P;
}

bool lz_shape_fits(const DevSector& S, const LzShape& q)
{
    const size_t need = fixed_bytes(table_doubles(S.P, std::max(S.up.namp, S.dn.namp))) +
                        std::max(lz_col_smem(S.dn.count, q.wc), lz_row_smem(S.up.count, q.r));
    return need <= (q.block < kLzThreads ? kLzSmemTwoPerSm : kLzSmemMax);
}

// lz_cut numbers a job's slabs by round (the r-th list position of every
// participant side by side).  A tile of n planes takes n positions at once:
// in every group of n full rounds the slabs are renumbered so that a
// participant's n slabs are neighbours, and the participants' groups still
// follow one another.
void lz_group_slabs(const LzJob* jobs, int nj, int G, std::vector<long long>& prefix)
{
    const long long* range = prefix.data() + 2 * (size_t)(nj + 1);
    long long* slab = prefix.data() + 2 * (size_t)(nj + 1) + 2 * (size_t)(G + 1);
    for (int j = 0; j < nj; j++) {
        const LzPhase& Q = jobs[j].ph[0];
        const int n = Q.planes;
        if (n <= 1) continue;
        const long long lo = Q.tile0, hi = Q.tile0 + Q.ntiles;
        long long full = hi - lo;                        // rounds that every participant takes part in
        for (int q = 0; q < Q.npart; q++)
            full = std::min(full, std::min(range[Q.part0 + q + 1], hi) - std::max(range[Q.part0 + q], lo));
        for (long long r = 0; r < full / n * n; r++)
            for (int q = 0; q < Q.npart; q++)
                slab[std::max(range[Q.part0 + q], lo) + r] = r / n * n * Q.npart + (long long)q * n + r % n;
    }
}

long long lz_cut(LzJob* jobs, int nj, int G, std::vector<long long>& prefix, long long total[2], double slow)
{
    long long slots = 0;
    prefix.assign(2 * (size_t)(nj + 1) + 2 * (size_t)(G + 1), 0);
    std::vector<long long> slab_order;
    for (int ph = 0; ph < 2; ph++) {
        long long* pre = prefix.data() + (size_t)ph * (nj + 1);
        for (int j = 0; j < nj; j++) {
            LzPhase& Q = jobs[j].ph[ph];
            const int count = (ph == 0) ? jobs[j].S.up.count : jobs[j].S.dn.count;
            Q.ntiles = (count + Q.width - 1) / Q.width;
            Q.tile0 = pre[j];
            pre[j + 1] = pre[j] + Q.ntiles;
        }
        const long long T = pre[nj];
        total[ph] = T;
        // CTA ranges: with no more tiles than CTAs, CTA b takes tile b; else
        // either the list is cut where the running cost (a tile costs its
        // states plus a fixed amount) crosses b/G of the total, every CTA
        // keeping at least one tile, or (with no more jobs than CTAs) each job
        // gets CTAs in proportion to its cost, so that a CTA serves one job and
        // need not reload its tables or wait for two: whichever leaves the
        // busiest CTA less to do (phase_load), and where that is close the
        // latter, unless its costliest CTA has much more than its share (two
        // runs of nsite 12, 924 and 495 by 792 strings: 30.8 us a step instead
        // of 29.8; kLzClose from 1.1 to 1.25 the same, 1.05 too narrow).  All sectors of a model at once
        // show it, as do batches of uneven sizes (us a step when that went by
        // the states alone, and by phase_load: nsite 11 341 and 156, nsite 12 928
        // and 440, nsite 10 48 both; 40 batches and served sets of 3 to 16 models
        // of 6 to 12 sites 9% less kernel time, none more than 1.3% more).
        long long* range = prefix.data() + 2 * (size_t)(nj + 1) + (size_t)ph * (G + 1);
        if (T <= G) {
            for (int b = 0; b <= G; b++) range[b] = std::min<long long>(b, T);
        } else {
            // a job's positions cost the same but for a last one of fewer lines
            std::vector<double> cost((size_t)nj, 0.0), each((size_t)nj, 0.0), cum((size_t)nj + 1, 0.0);
            for (int j = 0; j < nj; j++) {
                const LzPhase& Q = jobs[j].ph[ph];
                const double lines = (ph == 0) ? jobs[j].S.dn.count : jobs[j].S.up.count;
                const double count = (ph == 0) ? jobs[j].S.up.count : jobs[j].S.dn.count;
                each[j] = lines * Q.width + kLzTileCost;
                cost[j] = lines * count + kLzTileCost * Q.ntiles;
                cum[j + 1] = cum[j] + cost[j];
            }
            std::vector<int> share;
            range[0] = 0;
            range[G] = T;
            for (int b = 1, j = 0; b < G; b++) {
                const double target = cum[nj] * b / G;
                while (j + 1 < nj && cum[j + 1] <= target) j++;
                const LzPhase& Q = jobs[j].ph[ph];
                const long long t = Q.tile0 + std::min<long long>(Q.ntiles - 1, (long long)((target - cum[j]) / each[j]));
                range[b] = std::min(std::max(t, range[b - 1] + 1), T - (G - b));
            }
            if (nj <= G) {                               // CTAs one by one to the job whose CTAs have the most to do
                share.assign((size_t)nj, 1);
                std::priority_queue<std::pair<double, int>> load;
                for (int j = 0; j < nj; j++) load.push({cost[j], j});
                for (int left = G - nj; left > 0; left--) {
                    int j = -1;
                    std::vector<std::pair<double, int>> full;   // jobs with a CTA for every tile
                    while (!load.empty()) {
                        j = load.top().second;
                        if (share[j] < jobs[j].ph[ph].ntiles) break;
                        full.push_back(load.top());
                        load.pop();
                        j = -1;
                    }
                    if (j >= 0) {
                        load.pop();
                        share[j]++;
                        load.push({cost[j] / share[j], j});
                    }
                    for (const auto& f : full) load.push(f);
                    if (j < 0) break;
                }
                std::vector<long long> own((size_t)G + 1);
                int b = 0;
                for (int j = 0; j < nj; j++)
                    for (int q = 0; q < share[j]; q++)
                        own[b++] = jobs[j].ph[ph].tile0 + (long long)jobs[j].ph[ph].ntiles * q / share[j];
                own[G] = T;
                const double one = phase_load(jobs, nj, G, ph, own.data(), slow);
                const double even = phase_load(jobs, nj, G, ph, range, slow);
                double worst = 0.0;
                for (int j = 0; j < nj; j++) {
                    const int nt = jobs[j].ph[ph].ntiles;
                    worst = std::max(worst, cost[j] / nt * ((nt + share[j] - 1) / share[j]));
                }
                const bool close = one < kLzClose * even && even < kLzClose * one;
                if (close ? worst <= kLzUneven * cum[nj] / G + kLzSwitchCost : one < even)
                    std::copy(own.begin(), own.end(), range);
            }
        }
        // participants of a job: the CTAs whose range meets its tiles (a contiguous run)
        auto owner = [&](long long tile) {
            return (int)(std::upper_bound(range, range + G + 1, tile) - range) - 1;
        };
        for (int j = 0; j < nj; j++) {
            LzPhase& Q = jobs[j].ph[ph];
            Q.part0 = owner(Q.tile0);
            Q.npart = owner(Q.tile0 + Q.ntiles - 1) - Q.part0 + 1;
            Q.slot0 = slots;
            slots += Q.npart;
        }
        // Column phase: the slab each tile position stages.  A participant
        // takes its positions in order; numbering the slabs by round (the
        // r-th tile of every participant, participants in order) makes the
        // participants stage neighbouring slabs at the same time, so the
        // rows they read sit side by side in DRAM.
        if (ph == 0) {
            slab_order.assign((size_t)T, 0);
            for (int j = 0; j < nj; j++) {
                const LzPhase& Q = jobs[j].ph[0];
                const long long lo = Q.tile0, hi = Q.tile0 + Q.ntiles;
                long long next = 0;
                for (long long r = 0; next < Q.ntiles; r++)
                    for (int q = 0; q < Q.npart; q++) {
                        const long long s0 = std::max(range[Q.part0 + q], lo), s1 = std::min(range[Q.part0 + q + 1], hi);
                        if (s0 + r < s1) slab_order[(size_t)(s0 + r)] = next++;
                    }
            }
        }
    }
    prefix.insert(prefix.end(), slab_order.begin(), slab_order.end());
    return slots;
}
