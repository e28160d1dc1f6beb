// hv_plane.cuh — staged lines and hop sums of the two-phase H.v.
//
// H.v (src/impurity_hamiltonian.f90:98-246) is split by the spin whose
// string a term changes: with the sector vector as the matrix X[ndn][nup], a
// whole column is closed under the down hops and a whole row under the up
// hops.  A column tile is W whole columns, a row tile W whole rows; both are
// staged in shared memory as *lines* of the closed index t (t = down string
// of a column tile, up string of a row tile), W values per line, and the hop
// sum of line t is sum_h a_h * line(rank_h(t)), the same list for all W
// values.
//
// Layout: planes of PW = 4 values, [W / 4][count][4] (or one plane of 2).  A
// thread owns two adjacent values of a line in every plane, so two lanes
// read a line's 32 bytes and a quarter warp four lines.  Within a warp the
// lines are consecutive strings; their targets are nearly consecutive too
// when strings are ordered with the impurity bits on top (spin tables in
// *internal* order): the 16-byte loads then take 1.1-1.2 times the
// conflict-free number of wavefronts, where strings in the reference's order
// (impurity bit lowest, so that neighbours alternate between filled and
// empty impurity) take 1.7-1.9.  The hop decode is shared by the thread's
// W / 2 values.
#pragma once
#include "edzt_device.cuh"

__device__ __forceinline__ void stage_table(const double* __restrict__ src, int n, double* dst)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = __ldg(src + i);
}

// Asynchronous 8-byte copy global -> shared (cp.async, no register holds the
// value in flight, so a thread can have its whole share of a tile in flight
// at once); when `valid` is false nothing is read and the destination gets 0.
__device__ __forceinline__ void copy_async8(double* dst, const double* src, bool valid)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int bytes = valid ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

// Asynchronous 16-byte copy global -> shared through L2 (no register holds the data in flight).
__device__ __forceinline__ void copy_async16(double* dst, const double* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// Wait for every asynchronous copy this thread issued (the caller then syncs the CTA).
__device__ __forceinline__ void copy_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The packed hop list of string t (table [hw/4][count] of uint4): its count
// and first eight entries, loaded as one byte and two 16-byte words.  A
// loop over strings loads the next string's list before it uses the current
// one, so the table's latency overlaps the current string's arithmetic.
struct HopList {
    int hc;
    uint4 q0, q1;
};

__device__ __forceinline__ HopList hop_list(const DevSpin& sp, int t)
{
    HopList L;
    const uint4* __restrict__ hp = sp.hpk + t;
    L.hc = __ldg(sp.hcnt + t);
    L.q0 = (sp.hw > 0) ? __ldg(hp) : make_uint4(0u, 0u, 0u, 0u);
    L.q1 = (sp.hw > 4) ? __ldg(hp + sp.count) : make_uint4(0u, 0u, 0u, 0u);
    return L;
}

// acc[p] += a * (two values at l of plane p), planes ps doubles apart.
template <int NP>
__device__ __forceinline__ void plane_axpy(double a, const double* __restrict__ l, int ps, double2 (&acc)[NP])
{
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const double2 v = *reinterpret_cast<const double2*>(l + (size_t)p * ps);
        acc[p].x = fma(a, v.x, acc[p].x);
        acc[p].y = fma(a, v.y, acc[p].y);
    }
}

// Hop sum of string t: acc[p] += amp(h) * line(rank(h)) over its hops, in
// table order.  lines: the staged tile at this thread's pair of values.
template <int NP, int PW>
__device__ __forceinline__ void plane_hops(const DevSpin& sp, int t, const HopList& L, const double* __restrict__ amp,
                                           const double* __restrict__ lines, int ps, double2 (&acc)[NP], int code)
{
    const int hc = L.hc;
    const uint32_t e[8] = {L.q0.x, L.q0.y, L.q0.z, L.q0.w, L.q1.x, L.q1.y, L.q1.z, L.q1.w};
#pragma unroll
    for (int h = 0; h < 8; h++) {
        if (h < hc) {
            EDZT_OK_OR(edzt_hop_rank(e[h]) < sp.count && edzt_hop_slot(e[h]) < sp.namp, code, t, h, (long long)e[h],
                       continue)
            plane_axpy<NP>(amp[edzt_hop_slot(e[h])], lines + edzt_hop_rank(e[h]) * PW, ps, acc);
        }
    }
    for (int h0 = 8; h0 < hc; h0 += 4) {
        const uint4 q = __ldg(sp.hpk + t + (size_t)(h0 >> 2) * sp.count);
        const uint32_t f[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int h = 0; h < 4; h++) {
            if (h0 + h < hc) {
                EDZT_OK_OR(edzt_hop_rank(f[h]) < sp.count && edzt_hop_slot(f[h]) < sp.namp, code, t, h0 + h,
                           (long long)f[h], continue)
                plane_axpy<NP>(amp[edzt_hop_slot(f[h])], lines + edzt_hop_rank(f[h]) * PW, ps, acc);
            }
        }
    }
}

// Spin-flip and pair-hopping terms (impurity_hamiltonian.f90:179-226) of
// element (id, iu) with up impurity pattern pu and down pattern pd;
// fetch(id2, iu2) returns the vector at another element.
template <class Fetch>
__device__ __forceinline__ double exchange_part(const DevSector& S, int id, int iu, int pu, int pd, double acc,
                                                Fetch fetch)
{
    const int P = S.P;
    const int pp = pu * P + pd;
    const int nj = __ldg(S.jcnt + pp);
    for (int t = 0; t < nj; t++) {
        const JTrans tr = S.jt[pp * EDZT_MAX_JT + t];
        const int iu2 = __ldg(S.up.sub + iu * P + tr.pu2);
        const int id2 = __ldg(S.dn.sub + id * P + tr.pd2);
        EDZT_OK_OR(iu2 >= 0 && iu2 < S.up.count && id2 >= 0 && id2 < S.dn.count, 73, iu2, id2, pp, continue)
        acc = fma(tr.c, fetch(id2, iu2), acc);
    }
    return acc;
}
