// hv_tile.cuh — the matrix-free Fock-space H.v in one pass over row tiles.
//
// Restates the row sum of src/impurity_hamiltonian.f90:98-246.  A sector
// vector is the matrix X[ndn][nup] (up rank fast); element (id, iu) of H x:
//   diagonal    (e1_up[iu] + e1_dn[id] + wint[imp_up, imp_dn]) x(id, iu)
//   up hops     sum_h a_h x(id, iu')   same row: from shared memory
//   down hops   sum_h a_h x(id', iu)   same column of other rows
//   exchange    sum_t c_t x(id', iu')  (norb > 1)
// A CTA takes a tile of up to R consecutive rows, staged whole in shared
// memory, and a thread takes a column of all of them.  The up string's hop
// list is decoded once for the R rows; the rows lie in pairs, xs[p][iu][2],
// so a hop's two values are one 16-byte load.  The down hops of a row are
// the same for every thread (16-byte records in shared memory: amplitude,
// address of the target row), so each is one coalesced 8-byte load per
// thread straight into a register.  The terms are the reference's; only the
// summation order differs (diagonal, up hops, down hops, exchange).
#pragma once
#include "hv_plane.cuh"

// A down hop of a row: signed amplitude and the target row's address.
struct __align__(16) DnHop {
    double amp;
    const double* row;
};

// Shared memory of a tile, after the model tables.
struct RowTile {
    DnHop* dh;        // [R][hw]     down hops of each row
    double* e1d;      // [R]         down-string energies
    int* pd;          // [R]         down impurity patterns
    int* hd;          // [R]         down-hop counts
    double* xs;       // [ceil(R/PL)][nup][PL] the staged rows
};

__host__ __device__ constexpr size_t tile_fixed_bytes(int R, int hw)
{
    return (size_t)R * hw * sizeof(DnHop) + (size_t)((R + 1) / 2 * 2) * (sizeof(double) + 2 * sizeof(int));
}

__device__ __forceinline__ RowTile tile_layout(void* base, int R, int hw)
{
    const int Re = (R + 1) / 2 * 2;
    RowTile t;
    t.dh = reinterpret_cast<DnHop*>(base);
    t.e1d = reinterpret_cast<double*>(t.dh + (size_t)R * hw);
    t.pd = reinterpret_cast<int*>(t.e1d + Re);
    t.hd = t.pd + Re;
    t.xs = reinterpret_cast<double*>(t.hd + Re);
    return t;
}

// The down-hop records and energies of rows [r0, r0 + nr) of vector x.
template <int R>
__device__ __forceinline__ void stage_row_tables(const DevSpin& dn, const RowTile& t, int r0, int nr, int nup,
                                                 const double* __restrict__ x)
{
    const int hw = dn.hw, ndn = dn.count;
    const uint32_t* __restrict__ hp = reinterpret_cast<const uint32_t*>(dn.hpk);
    for (int i = threadIdx.x; i < nr * hw; i += blockDim.x) {
        const int r = i / hw, h = i - r * hw;
        const uint32_t e = __ldg(hp + ((size_t)(h >> 2) * ndn + r0 + r) * 4 + (h & 3));
        EDZT_OK_OR(edzt_hop_rank(e) < ndn && edzt_hop_slot(e) < dn.namp, 33, r0 + r, h, (long long)e, continue)
        t.dh[i].amp = __ldg(dn.amp + edzt_hop_slot(e));
        t.dh[i].row = x + (size_t)edzt_hop_rank(e) * nup;
    }
    for (int r = threadIdx.x; r < R; r += blockDim.x) {   // rows past the tile's end: zeros, as their staged values
        const bool in = r < nr;
        t.e1d[r] = in ? __ldg(dn.e1 + r0 + r) : 0.0;
        t.pd[r] = in ? __ldg(dn.imp + r0 + r) : 0;
        t.hd[r] = in ? __ldg(dn.hcnt + r0 + r) : 0;
    }
}

// The up string of a column: energy, impurity bits, hop count and first
// eight hops; loaded one column ahead of its use.
struct UpCol {
    double e1u;
    int pu;
    HopList L;
};

__device__ __forceinline__ UpCol up_col(const DevSpin& up, int iu)
{
    UpCol c;
    c.e1u = __ldg(up.e1 + iu);
    c.pu = __ldg(up.imp + iu);
    c.L = hop_list(up, iu);
    return c;
}

// acc[r] += a * (row r of the tile at column j)
template <int R, int PL>
__device__ __forceinline__ void tile_axpy(double a, const double* __restrict__ xs, int nup, int j, double (&acc)[R])
{
#pragma unroll
    for (int p = 0; p < (R + PL - 1) / PL; p++) {
        const double* l = xs + ((size_t)p * nup + j) * PL;
        if constexpr (PL == 2) {
            const double2 v = *reinterpret_cast<const double2*>(l);
            acc[2 * p] = fma(a, v.x, acc[2 * p]);
            if (2 * p + 1 < R) acc[2 * p + 1] = fma(a, v.y, acc[2 * p + 1]);
        } else {
            acc[p] = fma(a, *l, acc[p]);
        }
    }
}

// Column iu of the tile: (H x)(r0 + r, iu) without the exchange terms into
// acc[r]; ld(p) reads a down-hop neighbour.
template <int R, int PL, class Load>
__device__ __forceinline__ void tile_col(const DevSector& S, const RowTile& t, const double* __restrict__ wint,
                                         const double* __restrict__ amp, int iu, int nr, const UpCol& c,
                                         double (&acc)[R], Load ld)
{
    const int nup = S.up.count, hw = S.dn.hw;
    const int pu = c.pu * S.P;
#pragma unroll
    for (int p = 0; p < (R + PL - 1) / PL; p++) {
        const double* l = t.xs + ((size_t)p * nup + iu) * PL;
#pragma unroll
        for (int q = 0; q < PL; q++)
            if (p * PL + q < R)
                acc[p * PL + q] = (c.e1u + t.e1d[p * PL + q] + wint[pu + t.pd[p * PL + q]]) * l[q];
    }
    // down hops: eight loads of a row in flight at once
#pragma unroll
    for (int r = 0; r < R; r++) {
        if (r < nr) {
            const int hd = t.hd[r];
            const DnHop* __restrict__ dh = t.dh + r * hw;
            double g[8];
#pragma unroll
            for (int q = 0; q < 8; q++) g[q] = (q < hd) ? ld(dh[q].row + iu) : 0.0;
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (q < hd) acc[r] = fma(dh[q].amp, g[q], acc[r]);
            for (int q = 8; q < hd; q++) acc[r] = fma(dh[q].amp, ld(dh[q].row + iu), acc[r]);
        }
    }
    // up hops
    const int hc = c.L.hc;
    const uint32_t e[8] = {c.L.q0.x, c.L.q0.y, c.L.q0.z, c.L.q0.w, c.L.q1.x, c.L.q1.y, c.L.q1.z, c.L.q1.w};
#pragma unroll
    for (int h = 0; h < 8; h++) {
        if (h < hc) {
            EDZT_OK_OR(edzt_hop_rank(e[h]) < nup && edzt_hop_slot(e[h]) < S.up.namp, 71, iu, h, (long long)e[h],
                       continue)
            tile_axpy<R, PL>(amp[edzt_hop_slot(e[h])], t.xs, nup, edzt_hop_rank(e[h]), acc);
        }
    }
    for (int h0 = 8; h0 < hc; h0 += 4) {
        const uint4 q = __ldg(S.up.hpk + iu + (size_t)(h0 >> 2) * nup);
        const uint32_t f[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int h = 0; h < 4; h++)
            if (h0 + h < hc) tile_axpy<R, PL>(amp[edzt_hop_slot(f[h])], t.xs, nup, edzt_hop_rank(f[h]), acc);
    }
}
