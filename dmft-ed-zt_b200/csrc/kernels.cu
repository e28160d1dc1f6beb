// kernels.cu — standalone (one launch per operation) sm_100a kernels:
// H.v, the BLAS-1 steps of the plain Lanczos drop-in, apply_c and the
// continued fractions.  The fused persistent Lanczos lives in lanczos.cu.
#include <algorithm>
#include <cuda_runtime.h>
#include "edzt_internal.h"
#include "hv_tile.cuh"

static constexpr int kWintDoubles = EDZT_MAX_P * EDZT_MAX_P;
static constexpr int kAmpDoubles = EDZT_MAX_AMP;

#ifdef EDZT_DEVICE_CHECKS
int kernels_debug_bad(long long* out4)
{
    return cudaMemcpyFromSymbol(out4, g_edzt_bad, 4 * sizeof(long long)) == cudaSuccess ? 0 : 2;
}
#endif

// ---------------------------------------------------------------------------
// H.v: y = H x (accumulate = 0) or y = y + H x (accumulate = 1), the `py`
// flag of src/impurity_hamiltonian.f90:241-245, in one pass over row tiles
// (hv_tile.cuh): CTA b of G takes rows [b ndn / G, (b + 1) ndn / G), at most
// R of them.  Bounded by the load/store pipe (hop values and gathers, 2.7
// wavefronts a state, the pipe 74% busy at nsite 14) and, from nsite 16, by
// L2.  Measured against the two launches of a column and a row phase that
// this replaces (nsite <= 13) and the single pass by element (from nsite 14):
// (7,5) of nsite 13 56.7 -> 48.6 us, nsite 12 38.2 -> 30.4, nsite 14
// 209 -> 162, nsite 15 798 -> 610, nsite 16 2,870 -> 2,680, nsite 8
// 24.4 -> 20.9 (device and launch, events around the call).
// ---------------------------------------------------------------------------
template <bool ACC, int R, int PL, int T, int NB>
__global__ void __launch_bounds__(T, NB) k_hx_tile(DevSector S, const double* __restrict__ x, double* __restrict__ y)
{
    extern __shared__ __align__(16) double smem[];
    double* wint = smem;
    double* amp = smem + kWintDoubles;
    const int nup = S.up.count, ndn = S.dn.count;
    const RowTile t = tile_layout(amp + kAmpDoubles, R, S.dn.hw);
    const int r0 = (int)((long long)blockIdx.x * ndn / gridDim.x);
    const int nr = (int)((long long)(blockIdx.x + 1) * ndn / gridDim.x) - r0;
    const double* __restrict__ x0 = x + (size_t)r0 * nup;
    for (int iu = threadIdx.x; iu < nup; iu += T) {        // the whole tile in flight at once
#pragma unroll
        for (int r = 0; r < (R + PL - 1) / PL * PL; r++)
            copy_async8(t.xs + ((size_t)(r / PL) * nup + iu) * PL + r % PL, x0 + (r < nr ? (size_t)r * nup + iu : 0), r < nr);
    }
    stage_row_tables<R>(S.dn, t, r0, nr, nup, x);
    stage_table(S.wint, S.P * S.P, wint);
    stage_table(S.up.amp, S.up.namp, amp);
    UpCol nxt{};
    if ((int)threadIdx.x < nup) nxt = up_col(S.up, threadIdx.x);
    copy_async_wait_all();
    __syncthreads();
    auto fetch = [&](int id2, int iu2) { return __ldg(x + (long long)id2 * nup + iu2); };
    for (int iu = threadIdx.x; iu < nup; iu += T) {
        const UpCol cur = nxt;                             // this column's up string; the next one's in flight
        if (iu + T < nup) nxt = up_col(S.up, iu + T);
        double acc[R];
        tile_col<R, PL>(S, t, wint, amp, iu, nr, cur, acc, [](const double* p) { return __ldg(p); });
        double* __restrict__ yo = y + (size_t)r0 * nup + iu;
#pragma unroll
        for (int r = 0; r < R; r++) {
            if (r < nr) {
                double v = acc[r];
                if (S.has_j) v = exchange_part(S, r0 + r, iu, cur.pu, t.pd[r], v, fetch);
                yo[(size_t)r * nup] = ACC ? yo[(size_t)r * nup] + v : v;
            }
        }
    }
}

static constexpr size_t kTileSmemMax = 227 * 1024 - 64;
static constexpr size_t kHxSmemLimit = 210 * 1024;      // of a sector's staged lines (hx_fits)

// Dynamic shared memory of a tile of R rows.
static size_t hx_tile_smem(const DevSector& S, int R, int PL)
{
    return (kWintDoubles + kAmpDoubles + (size_t)S.up.count * ((R + PL - 1) / PL * PL)) * sizeof(double) +
           tile_fixed_bytes(R, S.dn.hw);
}

template <int R, int PL, int T, int NB>
static void launch_hx_tile(const DevSector& S, const double* x, double* y, int accumulate, int grid, cudaStream_t s)
{
    static OnceEach attr_set;
    edzt_once_per_device(attr_set, [] {
        cudaFuncSetAttribute(k_hx_tile<false, R, PL, T, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmemMax);
        cudaFuncSetAttribute(k_hx_tile<true, R, PL, T, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmemMax);
    });
    const size_t sm = hx_tile_smem(S, R, PL);
    if (accumulate) k_hx_tile<true, R, PL, T, NB><<<grid, T, sm, s>>>(S, x, y);
    else k_hx_tile<false, R, PL, T, NB><<<grid, T, sm, s>>>(S, x, y);
}
bool hx_fits(int nup, int ndn)
{
    return (kWintDoubles + kAmpDoubles + (size_t)nup) * sizeof(double) <= kHxSmemLimit &&
           (kAmpDoubles + 2 * (size_t)ndn) * sizeof(double) <= kHxSmemLimit;
}

// Rows per tile: as many of 4, 2, 1 as leave every SM a tile and two CTAs (one
// from 8,000 strings) room in shared memory: the hop decode is shared by the
// tile's rows, but wide tiles of long rows leave too few warps (us at nsite 13
// with 4 / 2 / 1 rows 48.6 / 50.4 / 50.3, nsite 14 166 / 162 / 174, nsite 15
// 859 / 610 / 594).  Threads: 512, two CTAs per SM; four rows of 1,500 strings
// or more run 256 threads three times (80 registers: 48.6 against 53.1), rows
// of 8,000 or more 1,024 (2,677 against 2,732).  Rows of up to 200 strings take
// 128 threads, of up to 32 a warp, for as many CTAs as an SM holds: 512 threads
// are then mostly idle, and many rows come in many waves (us a call, 512 threads
// and now: (2,8) of nsite 16 67 and 36, (2,6) of nsite 17 71 and 45, (1,8) of
// nsite 16 64 and 22, (0,8) 53 and 20; with 220 strings, (3,6) of nsite 12, 128
// threads take 21.7 where 512 take 20.2).
void launch_hx(const DevSector& S, const double* x, double* y, int accumulate, cudaStream_t s)
{
    const int nup = S.up.count, ndn = S.dn.count;
    if (nup <= 0 || ndn <= 0) return;
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    int R = std::min(nup >= 8000 ? 1 : nup >= 3000 ? 2 : 4, std::max(1, ndn / nsm));
    if (R == 3) R = 2;
    const int grid = (ndn + R - 1) / R;
    if (R == 4 && nup <= 32) launch_hx_tile<4, 2, 32, 32>(S, x, y, accumulate, grid, s);
    else if (R == 4 && nup <= 200) launch_hx_tile<4, 2, 128, 8>(S, x, y, accumulate, grid, s);
    else if (R == 4 && nup >= 1500) launch_hx_tile<4, 2, 256, 3>(S, x, y, accumulate, grid, s);
    else if (R == 4) launch_hx_tile<4, 2, 512, 2>(S, x, y, accumulate, grid, s);
    else if (R == 2) launch_hx_tile<2, 2, 512, 2>(S, x, y, accumulate, grid, s);
    else if (nup >= 8000) launch_hx_tile<1, 1, 1024, 1>(S, x, y, accumulate, grid, s);
    else launch_hx_tile<1, 1, 512, 2>(S, x, y, accumulate, grid, s);
}

// ---------------------------------------------------------------------------
// Ground-state vector from kept Lanczos vectors (the eigenvector pass's sum,
// src/lanczos_solver.f90:213-300, without rerunning the recurrence).
// ---------------------------------------------------------------------------
// A run's vectors are read in storage order (lz_index), coalesced, eight of
// them in flight per thread; the results go to the reference's order, or stay
// in storage order where the recurrence goes on from them.
// Storage position e of a run's vector as its place in the reference's order (-1: padding).
__device__ __forceinline__ long long natural_of(unsigned e, int nup, int ndn, const int32_t* __restrict__ natu,
                                                const int32_t* __restrict__ natd)
{
    const unsigned ndp = (unsigned)lz_pad(ndn);
    const unsigned slab = e / (4 * ndp), rem = e - slab * 4 * ndp;
    const int iu = (int)(slab * 4 + ((rem >> 2) & 3)), id = (int)((rem >> 4) * 4 + (rem & 3));
    return (iu < nup && id < ndn) ? (long long)__ldg(natd + id) * nup + __ldg(natu + iu) : -1;
}

struct VecSumArgs { VecSum r[kVecSums]; };

// Blocks of a sum: one per 256 pairs of elements, at most eight per SM.
__host__ __device__ inline int vec_sum_blocks(const VecSum& r)
{
    const long long b = (lz_vec_size(r.nup, r.ndn) / 2 + 255) / 256;
    return b < kVecSumBlocks ? (int)b : kVecSumBlocks;
}

// blockIdx.y: the sum.  Bound by the read of the kept vectors: eight loads of 16
// bytes in flight per thread (of 8 bytes: 285 steps of nsite 15, 94 GB, took 6
// ms more).  The sums of a batch share a launch, as one alone fills the chip
// only from nsite 11 on (16 sums of nsite 8 to 11: 820 us apart).
__global__ void __launch_bounds__(256) k_vec_sum(const __grid_constant__ VecSumArgs A)
{
    __shared__ double scratch[32];
    const VecSum& R = A.r[blockIdx.y];
    const int nb = vec_sum_blocks(R);
    if ((int)blockIdx.x >= nb) return;
    const int nup = R.nup, ndn = R.ndn, nstep = R.nstep;
    const double* __restrict__ coeff = R.coeff;
    const long long pairs = lz_vec_size(nup, ndn) / 2;   // two rows of a column
    double sq[1] = {0.0};
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < pairs; i += (long long)nb * 256) {
        const double2* v = reinterpret_cast<const double2*>(R.v) + i;   // of v_1
        double2 acc = make_double2(0.0, 0.0);
        if (coeff) {
#pragma unroll 8
            for (int k = 0; k < nstep; k++) {
                const double2 x = __ldcs(v + k * pairs);
                const double c = __ldg(coeff + k);
                acc.x = fma(c, x.x, acc.x);
                acc.y = fma(c, x.y, acc.y);
            }
        } else {
            acc = __ldcs(v);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const unsigned e = (unsigned)(2 * i + h);
            const long long o = R.natural ? natural_of(e, nup, ndn, R.natu, R.natd) : e;
            if (o < 0) continue;
            const double z = h ? acc.y : acc.x;
            R.out[o] = z;
            sq[0] = fma(z, z, sq[0]);
        }
    }
    if (R.natural) {
        block_sum<1>(sq, scratch);
        if (threadIdx.x == 0) R.part[blockIdx.x] = sq[0];
    }
}

// out / ||out||: every block adds up the partial sums itself, in the same order.
__global__ void __launch_bounds__(256) k_vec_norm(const __grid_constant__ VecSumArgs A)
{
    __shared__ double scratch[32], norm;
    const VecSum& R = A.r[blockIdx.y];
    const int nb = vec_sum_blocks(R);
    if ((int)blockIdx.x >= nb) return;
    double sum[1] = {0.0};
    for (int i = threadIdx.x; i < nb; i += 256) sum[0] += R.part[i];
    block_sum<1>(sum, scratch);
    if (threadIdx.x == 0) norm = sqrt(sum[0]);
    __syncthreads();
    const double nrm = norm;
    const long long n = (long long)R.nup * R.ndn;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)nb * 256) R.out[i] /= nrm;
}

static int vec_sums(const VecSum* r, int n, bool norm, cudaStream_t s)
{
    int launches = 0;
    for (int i = 0; i < n; i += kVecSums) {
        VecSumArgs A;
        const int k = std::min(kVecSums, n - i);
        int blocks = 1;
        for (int q = 0; q < k; q++) {
            A.r[q] = r[i + q];
            blocks = std::max(blocks, vec_sum_blocks(A.r[q]));
        }
        const dim3 grid((unsigned)blocks, (unsigned)k);
        k_vec_sum<<<grid, 256, 0, s>>>(A);
        if (norm) k_vec_norm<<<grid, 256, 0, s>>>(A);
        launches += norm ? 2 : 1;
    }
    return launches;
}

int launch_vec_sum(const VecSum* r, int n, cudaStream_t s) { return vec_sums(r, n, false, s); }
int launch_vec_sum_normalised(const VecSum* r, int n, cudaStream_t s) { return vec_sums(r, n, true, s); }

// ---------------------------------------------------------------------------
// Deterministic dot product (mpi_dot_product, src/numeric_utils.f90:159-170):
// fixed grid of partial sums, then one block sums the partials in order.
// ---------------------------------------------------------------------------
static constexpr int kDotBlocks = 592;
static constexpr int kDotThreads = 256;

int dot_partials_size() { return kDotBlocks; }

__global__ void __launch_bounds__(kDotThreads) k_dot_partial(const double* __restrict__ a,
                                                             const double* __restrict__ b, long long n,
                                                             double* __restrict__ partials)
{
    __shared__ double scratch[32];
    double v[1] = {0.0};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        v[0] = fma(a[i], b[i], v[0]);
    block_sum<1>(v, scratch);
    if (threadIdx.x == 0) partials[blockIdx.x] = v[0];
}

__global__ void __launch_bounds__(kDotThreads) k_dot_final(const double* __restrict__ partials, int np,
                                                           double* __restrict__ out)
{
    __shared__ double scratch[32];
    double v[1] = {0.0};
    for (int i = threadIdx.x; i < np; i += blockDim.x) v[0] += partials[i];
    block_sum<1>(v, scratch);
    if (threadIdx.x == 0) *out = v[0];
}

void launch_dot(const double* a, const double* b, long long n, double* partials, double* out, cudaStream_t s)
{
    k_dot_partial<<<kDotBlocks, kDotThreads, 0, s>>>(a, b, n, partials);
    k_dot_final<<<1, kDotThreads, 0, s>>>(partials, kDotBlocks, out);
}

// w = v / b_k ; v = -b_k * w_old  (src/lanczos_solver.f90:152-156); *bk holds b_k.
__global__ void k_swap_scale(double* __restrict__ w, double* __restrict__ v, long long n,
                             const double* __restrict__ bk_p, double bk)
{
    const double b = bk_p ? *bk_p : bk;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const double t = w[i];
        w[i] = v[i] / b;
        v[i] = -b * t;
    }
}

void launch_swap_scale(double* w, double* v, long long n, const double* bk_p, double bk, cudaStream_t s)
{
    k_swap_scale<<<592, 256, 0, s>>>(w, v, n, bk_p, bk);
}

// y = y + (sign * alpha) * x  (daxpy with a device scalar)
__global__ void k_axpy(double* __restrict__ y, const double* __restrict__ x, long long n,
                       const double* __restrict__ alpha_p, double alpha, double sign)
{
    const double al = sign * (alpha_p ? *alpha_p : alpha);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        y[i] = fma(al, x[i], y[i]);
}

void launch_axpy(double* y, const double* x, long long n, const double* alpha_p, double alpha, double sign,
                 cudaStream_t s)
{
    k_axpy<<<592, 256, 0, s>>>(y, x, n, alpha_p, alpha, sign);
}

// x = x / sqrt(*nrm2)
__global__ void k_scale_inv_sqrt(double* __restrict__ x, long long n, const double* __restrict__ nrm2)
{
    const double nrm = sqrt(*nrm2);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        x[i] = x[i] / nrm;
}

void launch_scale_inv_sqrt(double* x, long long n, const double* nrm2, cudaStream_t s)
{
    k_scale_inv_sqrt<<<592, 256, 0, s>>>(x, n, nrm2);
}

__global__ void k_fill_start(double* __restrict__ v, long long n, uint64_t key)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        v[i] = edzt_u01(key, (uint64_t)i);
}

void launch_fill_start(double* v, long long n, uint64_t key, cudaStream_t s)
{
    k_fill_start<<<592, 256, 0, s>>>(v, n, key);
}

void launch_copy(double* dst, const double* src, long long n, cudaStream_t s)
{
    cudaMemcpyAsync(dst, src, (size_t)n * sizeof(double), cudaMemcpyDeviceToDevice, s);
}

// ---------------------------------------------------------------------------
// apply_c (src/ed_operator.f90:13-57), row-wise over the output sector.
// ---------------------------------------------------------------------------
__global__ void k_apply_c(ApplyCArgs A, const double* __restrict__ in, double* __restrict__ out)
{
    const long long n = (long long)A.out_nup * A.out_ndn;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = apply_c_value(A, in, i);
}

void launch_apply_c(const ApplyCArgs& A, const double* in, double* out, cudaStream_t s)
{
    const long long n = (long long)A.out_nup * A.out_ndn;
    if (n <= 0) return;
    long long blocks = (n + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    k_apply_c<<<(int)blocks, 256, 0, s>>>(A, in, out);
}

// ---------------------------------------------------------------------------
// Continued fractions (src/numeric_utils.f90:11-44): one thread per (run, w).
//   f = b_n^2/(z -/+ a_n);  f = b_i^2/(z -/+ a_i - f), i = n-1..1
// Complex division by Smith's method.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cdiv_real(double num, double br, double bi, double* cr, double* ci)
{
    if (fabs(br) >= fabs(bi)) {
        const double r = bi / br, den = br + bi * r;
        *cr = num / den;
        *ci = (-num * r) / den;
    } else {
        const double r = br / bi, den = bi + br * r;
        *cr = (num * r) / den;
        *ci = (-num) / den;
    }
}

__global__ void k_cf(const CFJob* __restrict__ jobs, int njobs, const double* __restrict__ omega, int nw,
                     int real_axis, double eta)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= njobs * nw) return;
    const int jb = t / nw, iw = t - jb * nw;
    const CFJob J = jobs[jb];
    const int n = J.levels;
    if (n < 1) return;
    // z = (+-E0) + i w_n on the Matsubara axis, (+-E0) + w + i eta on the real axis
    const double zr = J.zr_shift + (real_axis ? omega[iw] : 0.0), zi = real_axis ? eta : omega[iw];
    auto bk = [&](int i) { return i == 0 ? J.b1 : J.b[i]; };   // b(1) = ||c^(+)|gs>|
    // the reference's recursion literally (numeric_utils.f90:18-22 / :39-43),
    // including its final level with b(1) when n == 1
    double xr, xi;
    cdiv_real(bk(n - 1) * bk(n - 1), zr + J.sign * J.a[n - 1], zi, &xr, &xi);
    for (int i = n - 1; i >= 2; i--)
        cdiv_real(bk(i - 1) * bk(i - 1), zr + J.sign * J.a[i - 1] - xr, zi - xi, &xr, &xi);
    cdiv_real(J.b1 * J.b1, zr + J.sign * J.a[0] - xr, zi - xi, &xr, &xi);
    J.g[2 * iw] = xr;
    J.g[2 * iw + 1] = xi;
}

void launch_cf(const CFJob* jobs_dev, int njobs, const double* omega, int nw, cudaStream_t s, int real_axis,
               double eta)
{
    const int n = njobs * nw;
    if (n <= 0) return;
    k_cf<<<(n + 127) / 128, 128, 0, s>>>(jobs_dev, njobs, omega, nw, real_axis, eta);
}

// ---------------------------------------------------------------------------
// Occupancies of the ground state (post_process.f90:62-112):
// occ(iorb, ispin) = sum |x_i|^2 over states with orbital iorb of spin ispin
// filled, docc(iorb) = sum |x_i|^2 over states with both spins filled.
// Fixed grid of per-block partial sums, summed in block order by the host.
// ---------------------------------------------------------------------------
static constexpr int kOccBlocks = 592;

__global__ void __launch_bounds__(256) k_gs_occ(const double* __restrict__ x, const uint32_t* __restrict__ up,
                                                const uint32_t* __restrict__ dn, int nup, long long dim, int norb,
                                                double* __restrict__ part)
{
    __shared__ double scratch[12 * 32];
    double acc[12];
#pragma unroll
    for (int q = 0; q < 12; q++) acc[q] = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += (long long)gridDim.x * blockDim.x) {
        const long long id = i / nup;
        const int iu = (int)(i - id * nup);
        const double w = x[i] * x[i];
        const uint32_t u = __ldg(up + iu), d = __ldg(dn + id);
#pragma unroll
        for (int a = 0; a < EDZT_MAX_NORB; a++) {
            if (a < norb) {
                const bool bu = (u >> a) & 1u, bd = (d >> a) & 1u;
                acc[a] += bu ? w : 0.0;
                acc[4 + a] += bd ? w : 0.0;
                acc[8 + a] += (bu && bd) ? w : 0.0;
            }
        }
    }
    block_sum<12>(acc, scratch);
    if (threadIdx.x == 0)
        for (int q = 0; q < 12; q++) part[(size_t)blockIdx.x * 12 + q] = acc[q];
}

int occ_partials_size() { return kOccBlocks * 12; }

void launch_gs_occ(const double* x, const uint32_t* up, const uint32_t* dn, int nup, long long dim, int norb,
                   double* part, cudaStream_t s)
{
    k_gs_occ<<<kOccBlocks, 256, 0, s>>>(x, up, dn, nup, dim, norb, part);
}
