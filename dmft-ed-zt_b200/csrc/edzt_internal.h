// edzt_internal.h — host-side declarations shared by the CUDA translation
// units of libedzt (not part of the public C ABI; see include/edzt.h).
#pragma once
#include <cstdint>
#include <vector>
#include <cuda_runtime.h>
#include "edzt_device.cuh"
#include "host_threads.h"

// Impurity model as the kernels see it.  Shapes follow the reference's
// Fortran arrays em(norb,2), ek(nbath,2), vmk(norb,nbath,2)
// (src/impurity_hamiltonian.f90:80-84), stored here with the spin index last.
struct DevModel {
    int norb, nbath, nsite;
    double em[EDZT_MAX_NORB][2];
    double ek[EDZT_MAX_NSITE][2];
    double vmk[EDZT_MAX_NORB][EDZT_MAX_NSITE][2];
    double U, Up, Jex, Jp, mu;
};

// Set-up of the current device such as a kernel's shared-memory attribute, which
// cudaFuncSetAttribute sets for that device only: f() the first time, done
// before any thread's call returns.
template <class F>
inline void edzt_once_per_device(OnceEach& done, F&& f)
{
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
    done.run(dev, f);
}

// ---- tables.cu -------------------------------------------------------------
void edzt_init_binomials(int device);
uint64_t edzt_binom(int n, int k);
// Fills str[C(nsite,n)] (ascending) and rank[2^nsite] on the device.  With
// norb > 0 the strings come in internal order instead: ascending with the
// norb impurity bits moved above the bath bits (hv_plane.cuh), and nat
// (nullable) gets each string's rank in the plain order.
void launch_build_strings(int nsite, int n, uint32_t* str, int32_t* rank, cudaStream_t s, int norb = 0,
                          int32_t* nat = nullptr);
// Per-string tables of one spin species (sigma = 0 up, 1 down) for a model.
// hpk: [hw/4][count] uint4 (packed hop entries, see edzt_hop_pack); amp:
// [2*norb*nbath] (at least 2) amplitude slots.
// One spin table to build: operators of `count` strings of spin sigma of a
// model (on the device).  Returns the launches made.
struct SpinBuild {
    const DevModel* m;
    const uint32_t* str;
    const int32_t* rank;
    double* e1;
    uint8_t* hcnt;
    uint32_t* hpk;
    double* amp;
    uint8_t* imp;
    int32_t* sub;
    int sigma, count, hw;
};
constexpr int kSpinBuilds = 40;            // per launch: they travel as its argument (4 KB)
int launch_build_spin_ops(const SpinBuild* t, int n, cudaStream_t s);
// Largest number of allowed hops of any string with n electrons of spin sigma.
int edzt_max_hops(const DevModel& m, int sigma, int n);

// ---- kernels.cu: standalone (non-persistent) kernels ------------------------
// Sums of a run's vectors in step order, as the eigenvector pass adds them:
// out = sum_k coeff[k] v_k (coeff null: v_1 itself).
struct VecSum {
    const double* v;          // v_1; one vector after the other
    const double* coeff;      // [nstep] on the device
    double* out;              // the reference's order (natural) or storage order
    const int32_t *natu, *natd;
    int nup, ndn, nstep, natural;
    double* part;             // [kVecSumBlocks] scratch for the norm (natural)
};
constexpr int kVecSums = 48;               // per launch: they travel as its argument (4 KB)
constexpr int kVecSumBlocks = 1184;
int launch_vec_sum(const VecSum* r, int n, cudaStream_t s);
// The same and out / ||out|| (natural only).
int launch_vec_sum_normalised(const VecSum* r, int n, cudaStream_t s);
// y = H x, or y += H x (accumulate), of a sector in the reference's string order.
void launch_hx(const DevSector& S, const double* x, double* y, int accumulate, cudaStream_t s);
// Whether a sector's staged row and column slab fit in shared memory.
bool hx_fits(int nup, int ndn);
// Deterministic dot product: result written to *out (device).  partials needs
// dot_partials_size() doubles.
int dot_partials_size();
void launch_dot(const double* a, const double* b, long long n, double* partials, double* out, cudaStream_t s);
// Scalars come from *p when p is non-null, else from the value argument.
void launch_swap_scale(double* w, double* v, long long n, const double* bk_p, double bk, cudaStream_t s);
void launch_axpy(double* y, const double* x, long long n, const double* alpha_p, double alpha, double sign,
                 cudaStream_t s);
void launch_scale_inv_sqrt(double* x, long long n, const double* nrm2, cudaStream_t s);
void launch_fill_start(double* v, long long n, uint64_t key, cudaStream_t s);
void launch_copy(double* dst, const double* src, long long n, cudaStream_t s);

void launch_apply_c(const ApplyCArgs& A, const double* in, double* out, cudaStream_t s);
// Per-block partial sums [occ_partials_size()] = [block][12]: occupation of
// orbital a by up (q = a), down (q = 4 + a) and both spins (q = 8 + a).
int occ_partials_size();
void launch_gs_occ(const double* x, const uint32_t* up, const uint32_t* dn, int nup, long long dim, int norb,
                   double* part, cudaStream_t s);

// Continued fractions (src/numeric_utils.f90:11-44) for many runs at once.
struct CFJob {
    const double* a;      // [levels]
    const double* b;      // [levels], b[0] unused
    double b1;            // b(1) = ||c^(+)|gs>|| (dmft_green.f90:219,249)
    int levels;           // number of CF levels (0: contributes nothing)
    double zr_shift;      // real part of z: +E0 for c^+, -E0 for c
    double sign;          // -1: z - a (continued_fraction_p), +1: z + a (continued_fraction_m)
    double* g;            // [nw] complex interleaved, written (levels >= 1)
};
// omega: Matsubara frequencies, or real frequencies with real_axis (z = w + i eta).
void launch_cf(const CFJob* jobs_dev, int njobs, const double* omega, int nw, cudaStream_t s, int real_axis = 0,
               double eta = 0.0);

// ---- arpack.cu: vector kernels of the restarted Lanczos (diag_arpack) ------
#define EDZT_RL_MAXV 8
struct RlVecs { const double* p[EDZT_RL_MAXV]; };
struct RlOut { double* p[EDZT_RL_MAXV]; };
int rl_partials_size();
// out[q] = <V_q, w> for q < nv (device, deterministic); partials: rl_partials_size() doubles.
void launch_rl_mdot(const RlVecs& V, int nv, const double* w, long long n, double* partials, double* out,
                    cudaStream_t s);
// w -= sum_q h[q] V_q (h on the device).
void launch_rl_project_out(double* w, const RlVecs& V, int nv, const double* h, long long n, cudaStream_t s);
// O_i = sum_{j<m} Y[j*k + i] V_j for i < k (Y on the device, m, k <= EDZT_RL_MAXV).
void launch_rl_combine(const RlOut& O, int k, const RlVecs& V, int m, const double* Y, long long n, cudaStream_t s);
void launch_rl_div(double* out, const double* w, double beta, long long n, cudaStream_t s);

// ---- lanczos.cu: persistent fused Lanczos over a batch of jobs ------------
enum LzMode { LZ_COEFF = 0, LZ_EIGVEC = 1 };
enum LzInit { LZ_INIT_HASH = 0, LZ_INIT_APPLYC = 1, LZ_INIT_COPY = 2 };

// The list positions of one job in one phase (0: column phase, slabs of
// `width` columns; 1: row phase, groups of `width` rows): [tile0, tile0 +
// ntiles) of that phase's list.  Its participants are the CTAs part0, part0 +
// 1, ... (npart of them); participant q owns partial-sum slot slot0 + q.
struct LzPhase {
    long long tile0;      // first position in the launch's list of the phase
    long long slot0;      // first partial-sum slot
    int ntiles;
    int npart;            // participating CTAs: part0, part0 + 1, ..., one slot each
    int width;            // columns (column phase) or rows (row phase) of a list position
    int part0;
    int planes;           // list positions staged together as one tile
};

// Recurrence state of one run between phases (every participating CTA
// derives the same value; the first participant also stores it).
struct LzState {
    int k;                // the step in progress: opened by a column phase, finished by the row phase
    int active;           // 1 while the run is going
    int nstep;            // result: number of valid Lanczos steps
    int opened;           // step k already opened (a_{k-1} derived) by the closing pass of a slice
    double a_prev;        // a_{k-1}
    double b_cur;         // the last norm known: b_{k-1} in a column phase, b_k in a row phase (||v_init|| for k = 1)
    double b_prev;        // b_{k-1} in a row phase
    double norm0;         // ||v_init||
};

// A run's vectors, in the internal string order (S.up.nat, S.dn.nat), are
// stored as 4 x 4 blocks of 128 bytes, the four rows of a column adjacent:
// slab of four columns, then group of four rows, column, row (lz_index).  A
// slab of columns is one contiguous stream, a group of rows is a 128-byte
// line per slab, and two rows of a column are one 16-byte access.  Rows and
// columns are padded to whole blocks; the padding is never read as values.
struct LzJob {
    DevSector S;          // spin tables in internal order
    double* Y;            // y_k; between a step's phases D, the down-hop part of H v_k
    double* V[2];         // v_k, unnormalised, by lz_v
    double* eig;          // EIGVEC: output eigenvector (unnormalised)
    const double* coeff;  // EIGVEC: ground eigenvector of the tridiagonal [nstep]
    double* a;            // [maxnstep] a(1..), written as steps are accepted
    double* b;            // [maxnstep] b(1..)
    int maxnstep;         // COEFF: LanczosSteps; EIGVEC: nstep of the coefficient pass
    int mode;
    int init;
    int keep;             // first steps whose v is kept, in lz_keep_slots vectors at V[0] (0: none)
    int resume;           // EIGVEC: the first step, its v and the one before given (0: step 1, from the start vector)
    LzPhase ph[2];
    LzState* st;          // [2] the run's state by phase parity (kept across launches of a sliced run)
    uint64_t key;         // LZ_INIT_HASH
    ApplyCArgs ac;        // LZ_INIT_APPLYC
    const double* src;    // LZ_INIT_APPLYC: the ground state; LZ_INIT_COPY: the start vector (the reference's order)
};

__host__ __device__ constexpr int lz_pad(int count) { return (count + 3) / 4 * 4; }

// Where element (id, iu) of a run's vector lies; ndp = lz_pad(down strings).
__host__ __device__ inline unsigned lz_index(int id, int iu, int ndp)
{
    return (unsigned)(((iu >> 2) * ndp + (id & ~3)) * 4 + (iu & 3) * 4 + (id & 3));
}

// Doubles of one vector of a run.
__host__ __device__ inline long long lz_vec_size(int nup, int ndn) { return (long long)lz_pad(nup) * lz_pad(ndn); }

// v_k of a run (k = 0: never read): two buffers in turn, or one slot for each
// of the first `keep` steps and two behind them in turn for the others.
__host__ __device__ inline double* lz_v(const LzJob& J, int k, long long size)
{
    if (!J.keep) return J.V[k & 1];
    const int i = k > 0 ? k - 1 : 0;
    return J.V[0] + (i < J.keep ? i : J.keep + ((i - J.keep) & 1)) * size;
}
__host__ __device__ constexpr int lz_keep_slots(int keep, int maxnstep) { return keep < maxnstep ? keep + 2 : maxnstep; }

struct LzBatch {
    int njobs;
    size_t fixed;                 // shared memory before the staged tile; set by the launch
    int max_phases;               // phase budget of the launch (even for a slice)
    unsigned long long wait_ns;   // wait limit of a job's arrivals (0: the default 5 s)
    int stall_cta;                // fault test: this CTA leaves without arriving (-1: none)
    int slice;                    // 1: a slice of longer runs; at the end of the budget every run
                                  // still going opens its next step, so a later launch resumes it
};

// Largest dynamic shared memory of one persistent CTA.
constexpr size_t kLzSmemMax = 227 * 1024;
// A tile shape of the persistent kernel: columns per slab tile, rows per row
// tile, threads per CTA.
struct LzShape {
    int wc, r, block;
};
// Plan of a launch: its kernel (tile shape, exchange terms), block, grid and
// shared memory; the jobs' phases are filled in.  prefix receives, per phase,
// the jobs' first list positions [njobs + 1], then per phase every CTA's first
// position [grid + 1] (CTA b takes the contiguous positions [range[b],
// range[b + 1]), cut by cost so the CTAs finish together), then the slab of
// each column-phase position [total[0]] and padding.  force: use this shape when every job
// fits it.
struct LzPlan {
    int wc = 0, r = 0;
    bool exchange = false;
    int block = 0;
    int grid = 0;
    size_t smem = 0;
    size_t fixed = 0;             // shared memory before the staged tile
    long long total[2] = {0, 0};
    long long slots = 0;
};
LzPlan lz_plan(int device, LzJob* jobs, int njobs, std::vector<long long>& prefix, const LzShape* force = nullptr);
// CTAs of a plan's kernel that can be resident.
int lz_grid_size(int device, const LzPlan& P);
bool lz_shape_fits(const DevSector& S, const LzShape& q);
// jobs[j].st: the job's state by phase parity; prefix: as lz_plan fills it;
// slots: [P.slots] partial sums; sync_words: lz_sync_bytes(njobs), zeroed.
cudaError_t launch_lanczos_persistent(const LzPlan& P, const LzBatch& B, const LzJob* jobs, const long long* prefix,
                                      double* slots, unsigned* sync_words, int* status, cudaStream_t s);
// Small runs from start to finish, one CTA each: the shared memory that a run
// takes (0: it is not of that kind), its form of the kernel (the
// forms sum in different orders: a model's runs all take the largest of
// theirs), and a launch with the most shared memory that any of its runs takes.
constexpr int kSmallForms = 4;
size_t lz_small_smem(const DevSector& S);
int lz_small_form(const DevSector& S);
cudaError_t launch_lanczos_small(const LzJob* jobs, int njobs, size_t smem, int form, cudaStream_t s);
// Sync-word buffer size (bytes) for a launch of njobs runs.
size_t lz_sync_bytes(int njobs);
// The device-free part of lz_plan: given every job's widths (ph[].width) and
// the grid G, the phases' tile lists, CTA ranges, participants and the column
// phase's slab order (prefix as lz_plan describes it), the tiles per phase
// (total) and the number of partial-sum slots (returned).  slow: time of a
// tile's lines over what they take a CTA that has the SM to itself.
long long lz_cut(LzJob* jobs, int njobs, int G, std::vector<long long>& prefix, long long total[2], double slow = 1.0);
// The slab order regrouped so that the slabs of a tile of several planes are neighbours.
void lz_group_slabs(const LzJob* jobs, int njobs, int G, std::vector<long long>& prefix);

// ---- edzt_host.cu: context accessors (no table building, no allocation) -----
struct edzt_ctx;
int edzt_ctx_device(const edzt_ctx* c);
cudaStream_t edzt_ctx_stream(const edzt_ctx* c);
void edzt_ctx_set_error(edzt_ctx* c, const char* msg);
void edzt_count_launches(edzt_ctx* c, long long n);
// The sector of (nu, nd) when its tables already exist; else an error code
// with the reason in *why.
int edzt_ctx_ready_sector(edzt_ctx* c, int nu, int nd, DevSector* S, const char** why);

#ifdef EDZT_DEVICE_CHECKS
int lz_debug_bad(long long* out4);
int kernels_debug_bad(long long* out4);
int tables_debug_bad(long long* out4);
#endif
