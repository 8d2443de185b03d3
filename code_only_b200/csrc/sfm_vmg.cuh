// sfm_vmg.cuh -- the AMR-level V-cycle (vmg_fas, vmg.F90:116-243) on its
// 2^3-cell blocks, eight lanes per block.
//
// vmg_fas works level by level on the coarsest fmg level, where a block has 8
// cells and 56 ghost cells.  Refreshing the ghosts by three directional
// passes before every colour, and one launch per elementary operation, makes
// it about 61 dependent launches per level, each a few microseconds long
// whatever the level's size.  Here a lane holds one cell: its neighbours
// inside the block come by shuffle, those across a same-level face straight
// from the neighbouring block (a colour reads only the other colour, so the
// update is in place), and the operations between two dependencies share a
// launch: about 16 launches per level.
//
// Ghost cells that stay: the ones on coarse-fine faces (k_vmg_cf), which the
// reference sets once per leg and keeps through the sweeps (vmg_gridboundary,
// vmg.F90:710-725), and the full shells before the cubic restriction.  The
// coarse-fine formula reads the coarse block's own transverse ghost cells as
// the last fill before its last colour left them; k_vmg_margin takes that
// snapshot.  Every value and expression is the reference's: bit-identical.
//
// Used where Solver::facesOk holds: every coarse-fine margin has a plain
// source, and so (a refined block's faces are same-level or physical, and
// the chains across its edges and corners are among the margins) every
// neighbour of a refined block that the prolongation reads exists.
#pragma once
#include "sfm_device.cuh"
#include "sfm_fast.cuh"
#include "sfm_faces.cuh"

namespace sfm {

constexpr int kVB = 64;   // values of a block of 2^3 cells with its ghost shell (4^3)
__device__ __forceinline__ int vmg_off(int i, int j, int k) { return ((k + 1) * 4 + (j + 1)) * 4 + (i + 1); }
// stride of axis d in a block
__device__ __forceinline__ int vmg_stride(int d) { return d == 0 ? 1 : (d == 1 ? 4 : 16); }

// the value across the block face next to cell (offset off, side s of axis
// d): the neighbour's cell, the stored coarse-fine ghost, or 0 at the
// physical boundary (boundary_fill0)
template <class T>
__device__ __forceinline__ T vmg_outer(const T *u, const T *ghosts, const GFace *gf, int64_t b, int off, int s, int d) {
    const GFace g = gf[6 * b + s + 2 * d];
    const int st = vmg_stride(d);
    if (g.type == 0) return u[(int64_t)g.src * kVB + off + (s ? -st : st)];
    if (g.type == 1) return ghosts[b * kVB + off + (s ? st : -st)];
    return (T)0;
}

// div F in the reference's order (Flux::div) at a lane's cell: inner
// neighbours px, py, pz, outer ones ox, oy, oz
template <class T>
__device__ __forceinline__ T vmg_div(T uc, int i, int j, int k, T px, T py, T pz, T ox, T oy, T oz, T hi) {
    const T xp = i ? ox : px, xm = i ? px : ox, yp = j ? oy : py, ym = j ? py : oy, zp = k ? oz : pz, zm = k ? pz : oz;
    T t = (xp - uc) * hi - (uc - xm) * hi;
    t = t + (yp - uc) * hi;
    t = t - (uc - ym) * hi;
    t = t + (zp - uc) * hi;
    t = t - (uc - zm) * hi;
    return t;
}

// vmg_poisson_relax (vmg_poisson.F90:98-145) on blocks first .. first + nblk - 1.
// sw = 0: the colour ipass, in place (uo == u).  sw > 0 (a mixed-schedule
// choice): sw full sweeps with the outer values of before the launch, from u
// into uo (another array: neighbours still read u); coarse-fine ghosts from
// `ghosts`.
template <class T>
__global__ void __launch_bounds__(256) k_vmg_relax(const T *u, T *uo, const T *ghosts, const T *__restrict__ rhs,
                                                   const GFace *__restrict__ gf, int first, int nblk, T hh, T hi,
                                                   int ipass, int sw) {
    pdl_enter();
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int64_t q = t >> 3;
    const bool on = q < nblk;
    const int64_t b = first + (on ? q : nblk - 1);
    const int i = (int)t & 1, j = ((int)t >> 1) & 1, k = ((int)t >> 2) & 1, off = vmg_off(i, j, k);
    const bool red = i == ((j + k + 1) & 1);   // a colour-1 cell
    T uc = u[b * kVB + off], ox = (T)0, oy = (T)0, oz = (T)0, rr = (T)0;
    if (sw > 0 || red == (ipass == 1)) {
        ox = vmg_outer(u, ghosts, gf, b, off, i, 0);
        oy = vmg_outer(u, ghosts, gf, b, off, j, 1);
        oz = vmg_outer(u, ghosts, gf, b, off, k, 2);
        rr = rhs[b * kVB + off];
    }
    auto colour = [&](bool mine) {
        const T px = __shfl_xor_sync(0xffffffffu, uc, 1), py = __shfl_xor_sync(0xffffffffu, uc, 2),
                pz = __shfl_xor_sync(0xffffffffu, uc, 4);
        if (mine) {
            const T resh2 = (vmg_div(uc, i, j, k, px, py, pz, ox, oy, oz, hi) - rr * hh) * hh;
            uc = uc + (T)(1.0 / 6.0) * resh2;
        }
    };
    if (sw == 0) {
        const bool mine = red == (ipass == 1);
        colour(mine);
        if (on && mine) uo[b * kVB + off] = uc;
        return;
    }
    for (int r = 0; r < sw; r++) {
        colour(red);
        colour(!red);
    }
    if (on) uo[b * kVB + off] = uc;
}

// the cells of blocks first .. first + nblk - 1
template <class T>
__global__ void __launch_bounds__(256) k_vmg_copy(T *__restrict__ o, const T *__restrict__ a, int first, int nblk) {
    pdl_enter();
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if ((t >> 3) >= nblk) return;
    const int64_t c = (first + (t >> 3)) * kVB + vmg_off((int)t & 1, ((int)t >> 1) & 1, ((int)t >> 2) & 1);
    o[c] = a[c];
}

// vmg_gridboundary (vmg.F90:710-725): the face ghosts of the level's
// coarse-fine faces, a lane per ghost cell.  margin: the snapshot of
// k_vmg_margin, or null where the coarse level is still zero.
template <class T>
__global__ void __launch_bounds__(128) k_vmg_cf(T *u, const CFItem *__restrict__ items, int nitems,
                                                const T *__restrict__ margin) {
    pdl_enter();
    const int t = blockIdx.x * 128 + threadIdx.x, e = t >> 2;
    if (e >= nitems) return;
    const CFItem it = items[e];
    const int p = t & 1, q = (t >> 1) & 1;
    const int xc = it.lr == 0 ? 1 : 0;
    auto B = [&](int pb, int qb) -> T {
        const int a = pb + it.oa, b = qb + it.ob;
        const bool ia = a >= 0 && a < 2, ib = b >= 0 && b < 2;
        if (ia && ib) {
            int i, j, k;
            put3(it.dir, xc, a, b, i, j, k);
            return u[(int64_t)it.coarse * kVB + vmg_off(i, j, k)];
        }
        if (!margin) return (T)0;
        return margin[5 * (int64_t)e + (!ia ? (!ib ? 4 : b) : 2 + a)];
    };
    const int p1 = p ? 1 : -1, q1 = q ? 1 : -1;
    const T uH = ((T)9 * B(0, 0) + B(p1, q1) + (T)3 * B(0, q1) + (T)3 * B(p1, 0)) / (T)16;
    T *ub = u + (int64_t)it.fine * kVB;
    int i, j, k;
    put3(it.dir, it.lr ? 1 : 0, p, q, i, j, k);
    const int o = vmg_off(i, j, k), st = (it.lr ? 1 : -1) * vmg_stride(it.dir);   // towards the ghost
    const T u0 = ub[o], uN = ub[o - st];
    ub[o + st] = ((T)10 * u0 + (T)8 * uH - (T)3 * uN) / (T)15;
}

// the transverse ghost cells of the coarse planes under the level's
// coarse-fine faces, as a fill of the coarse level's same-level faces would
// leave them now: per face two cells across side a, two across side b, the edge
template <class T>
__global__ void __launch_bounds__(128) k_vmg_margin(const T *__restrict__ u, const CFItem *__restrict__ items, int nitems,
                                                    T *__restrict__ margin) {
    pdl_enter();
    const int e = blockIdx.x * 128 + threadIdx.x;
    if (e >= nitems) return;
    const CFItem it = items[e];
    const int xc = it.lr == 0 ? 1 : 0;
    auto val = [&](int s, int a, int b) -> T {
        if (s == kFaceZero) return (T)0;
        int i, j, k;
        put3(it.dir, xc, a, b, i, j, k);
        return u[(int64_t)(s >= 0 ? s : -2 - s) * kVB + vmg_off(i, j, k)];
    };
    const T v0 = val(it.ma, 1 - it.oa, 0), v1 = val(it.ma, 1 - it.oa, 1), v2 = val(it.mb, 0, 1 - it.ob),
            v3 = val(it.mb, 1, 1 - it.ob), v4 = val(it.mab, 1 - it.oa, 1 - it.ob);
    T *m = margin + 5 * (int64_t)e;
    m[0] = v0; m[1] = v1; m[2] = v2; m[3] = v3; m[4] = v4;
}

// Restriction of level v onto its refined parents (vmg.F90:170-200), a
// thread per child: U by rstrct_cubic (the child's full shell), RHS and the
// child's part of tau, -(div F)/h (OpTauFine), by rstrct_linear.
template <class T>
__global__ void __launch_bounds__(128) k_vmg_restrict(T *u, T *rhs, T *tau, const int32_t *__restrict__ parents,
                                                      int nparents, const int32_t *__restrict__ child, T hi) {
    pdl_enter();
    const int t = blockIdx.x * 128 + threadIdx.x;
    if (t >= 8 * nparents) return;
    const int p = parents[t >> 3], c8 = t & 7;
    const int64_t ch = child[8 * (int64_t)p + c8];
    const T *uf = u + ch * kVB;
    T a[kVB];
#pragma unroll
    for (int r = 0; r < kVB / 2; r++) {
        T v[2];
        vec_load<T, 2>(uf + 2 * r, v);
        a[2 * r] = v[0];
        a[2 * r + 1] = v[1];
    }
    T s = (T)0;
#pragma unroll
    for (int r = 0; r < kVB; r++) {
        const T w = a[r] * (T)((rstrct_w(r & 3) * rstrct_w((r >> 2) & 3)) * rstrct_w(r >> 4));
        s = r ? s + w : w;
    }
    auto F = [&](int o, int st) { return (a[o + st] - a[o]) * hi; };   // flux between o and o + st
    auto tf = [&](int i, int j, int k) -> T {
        const int o = ((k + 1) * 4 + (j + 1)) * 4 + (i + 1);
        T d = F(o, 1) - F(o - 1, 1);
        d = d + F(o, 4);
        d = d - F(o - 4, 4);
        d = d + F(o, 16);
        d = d - F(o - 16, 16);
        return -(d * hi);
    };
    T g = tf(0, 0, 0) + tf(1, 0, 0);
    g = g + tf(0, 1, 0);
    g = g + tf(0, 0, 1);
    g = g + tf(1, 1, 0);
    g = g + tf(1, 0, 1);
    g = g + tf(0, 1, 1);
    g = g + tf(1, 1, 1);
    const int64_t o = (int64_t)p * kVB + vmg_off(c8 & 1, (c8 >> 1) & 1, c8 >> 2);
    u[o] = s;
    rhs[o] = rstrct_linear(rhs + ch * kVB, 4, 0, 0, 0);
    tau[o] = g * (T)(1.0 / 8.0);
}

// The parents' level after the restriction, eight lanes per block: RUF = U
// on every block; on refined blocks tau += (div F)/h (OpTauParent), zeroed on
// the planes behind coarse-fine faces (vmg_tau_crop, vmg.F90:463-505; crop:
// bit f per block), and added to RHS.
template <class T>
__global__ void __launch_bounds__(256) k_vmg_tau(const T *__restrict__ u, T *__restrict__ ruf, T *__restrict__ rhs,
                                                 const T *__restrict__ tau, const GFace *__restrict__ gf,
                                                 const int8_t *__restrict__ skip, const uint8_t *__restrict__ crop,
                                                 int first, int nblk, T hi) {
    pdl_enter();
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int64_t q = t >> 3;
    const bool on = q < nblk;
    const int64_t b = first + (on ? q : nblk - 1);
    const int i = (int)t & 1, j = ((int)t >> 1) & 1, k = ((int)t >> 2) & 1, off = vmg_off(i, j, k);
    const T uc = u[b * kVB + off];
    const T px = __shfl_xor_sync(0xffffffffu, uc, 1), py = __shfl_xor_sync(0xffffffffu, uc, 2),
            pz = __shfl_xor_sync(0xffffffffu, uc, 4);
    if (!on) return;
    ruf[b * kVB + off] = uc;
    if (!skip[b]) return;
    const T ox = vmg_outer(u, u, gf, b, off, i, 0), oy = vmg_outer(u, u, gf, b, off, j, 1),
            oz = vmg_outer(u, u, gf, b, off, k, 2);
    T v = tau[b * kVB + off] + vmg_div(uc, i, j, k, px, py, pz, ox, oy, oz, hi) * hi;
    const int m = crop[b];
    if ((m >> i) & 1 || (m >> (2 + j)) & 1 || (m >> (4 + k)) & 1) v = (T)0;
    rhs[b * kVB + off] = rhs[b * kVB + off] + v;
}

// The correction of a level (vmg.F90:215-240), eight lanes per block: U +=
// the trilinear prolongation (vmg_interp_p2c_lev) of the parent level's
// U - RUF.  Beyond the parent: its same-level neighbours, highest dimension
// first; minus the boundary cell at the physical boundary
// (boundary_extrap).
template <class T>
__global__ void __launch_bounds__(256) k_vmg_correct(T *u, const T *__restrict__ ruf, const GFace *__restrict__ gf,
                                                     const int32_t *__restrict__ parent, const int8_t *__restrict__ oct,
                                                     int first, int nblk) {
    pdl_enter();
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int64_t q = t >> 3;
    if (q >= nblk) return;
    const int64_t b = first + q;
    const int i = (int)t & 1, j = ((int)t >> 1) & 1, k = ((int)t >> 2) & 1;
    const int D = parent[b], o[3] = {oct[3 * b], oct[3 * b + 1], oct[3 * b + 2]};
    const int s[3] = {i, j, k};
    // per axis: the near neighbour lies beyond the parent when the cell is on the outer side of its octant
    const bool out[3] = {s[0] == o[0], s[1] == o[1], s[2] == o[2]};
    auto R = [&](bool nx, bool ny, bool nz) -> T {   // coarse cell, near in the axes that are set
        const bool near[3] = {nx, ny, nz};
        int blk = D, c[3] = {o[0], o[1], o[2]};
        bool neg = false;
#pragma unroll
        for (int d = 2; d >= 0; d--) {
            if (!near[d]) continue;
            c[d] = 1 - o[d];
            if (!out[d]) continue;   // the parent's other cell
            const GFace g = gf[6 * (int64_t)blk + s[d] + 2 * d];
            if (g.type == 0) blk = g.src;
            else {
                c[d] = o[d];
                neg = !neg;
            }
        }
        const int64_t a = (int64_t)blk * kVB + vmg_off(c[0], c[1], c[2]);
        const T v = u[a] - ruf[a];
        return neg ? -v : v;
    };
    const T v = ((T)27 * R(false, false, false) +
                 (T)9 * (R(true, false, false) + R(false, true, false) + R(false, false, true)) +
                 (T)3 * (R(false, true, true) + R(true, false, true) + R(true, true, false)) + R(true, true, true)) /
                (T)64;
    const int64_t a = b * kVB + vmg_off(i, j, k);
    u[a] = u[a] + v;
}

// vmg_zeroAverage (vmg.F90:900-916) on base blocks 0 .. nblk - 1 in one CTA:
// block sums in Fortran SUM order, their running sum in block order by one
// thread (the other warps stage the next chunk), the mean subtracted
constexpr int kAveChunk = 992;
template <class T>
__global__ void __launch_bounds__(1024) k_vmg_zero_average(T *a, int nblk) {
    pdl_enter();
    __shared__ double ts[2][kAveChunk];
    __shared__ double mean;
    const int tid = threadIdx.x, nch = (nblk + kAveChunk - 1) / kAveChunk;
    auto stage = [&](int c) {
        const int b = c * kAveChunk + tid - 32;
        if (b >= nblk) return;
        double s = 0.0;
#pragma unroll
        for (int r = 0; r < 8; r++) s = s + (double)a[(int64_t)b * kVB + vmg_off(r & 1, (r >> 1) & 1, r >> 2)];
        ts[c & 1][tid - 32] = s;
    };
    double ave = 0.0;
    if (tid >= 32) stage(0);
    __syncthreads();
    for (int c = 0; c < nch; c++) {
        if (tid >= 32) {
            if (c + 1 < nch) stage(c + 1);
        } else if (tid == 0) {
            const int cnt = nblk - c * kAveChunk < kAveChunk ? nblk - c * kAveChunk : kAveChunk;
            for (int q = 0; q < cnt; q++) ave = ave + ts[c & 1][q];
        }
        __syncthreads();
    }
    if (tid == 0) mean = ave / (double)(8 * nblk);
    __syncthreads();
    const T m = (T)mean;
    for (int e = tid; e < 8 * nblk; e += 1024) {
        const int64_t c = (int64_t)(e >> 3) * kVB + vmg_off(e & 1, (e >> 1) & 1, (e >> 2) & 1);
        a[c] = a[c] - m;
    }
}

}  // namespace sfm
