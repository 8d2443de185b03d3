// sfm_faces.cuh -- sweeps and residuals of fmg_lin whose blocks exchange
// whole boundary planes instead of ghost cells.
//
// fmg_poisson_relax refreshes every ghost cell before each colour
// (fmg_poisson.F90:160-165): restriction onto covered blocks, three
// directional passes per AMR level and the flux correction, 20 to 25
// dependent launches that move several times the sweep's own bytes (a pass
// in x touches one 32-byte sector per value).  But the operator on a leaf
// block reads only the face part of the ghost layer, and each face has one
// of four sources:
//   - a leaf of the same level: that block's boundary plane;
//   - a block of the same level that is refined: the flux through the face
//     comes from the finer blocks (reflux), its ghost cell is not read;
//   - a coarser leaf: the parentlev formula (fmg_ghostcell.F90:312-496);
//   - the physical boundary: zero (boundary_fill0; the fields of fmg_lin are
//     corrections).
// So each sweep leaves its blocks' six boundary planes in a buffer of dense
// n x n planes, from which the neighbours' next sweep takes them in whole
// sectors, and the coarse-fine ghosts and the flux correction come from one
// kernel over the coarse-fine faces of all levels.  A colour is two launches
// (one without refinement).  Two plane buffers take turns, so a sweep never
// writes what a concurrent block reads.  Every value is the one the ghost
// passes would have put there, every expression unchanged: the fields are
// bit-identical.
//
// Where a ghost layer itself is read later -- the cubic restriction before
// a cubic prolongation, and the field after the last sweep of fmg_lin --
// Solver::relax runs the ghost passes before that sweep as well.
#pragma once
#include "sfm_device.cuh"
#include "sfm_fast.cuh"

namespace sfm {

// Where a block's face gets its ghost plane (Solver::d_fsrc): 6 * leaf + face
// for a leaf of the same level (its opposite plane), kFaceZero for the
// physical boundary and for a refined neighbour (never read), -2 - k for
// coarse-fine face k.
constexpr int kFaceZero = -1;
__host__ __device__ constexpr int face_cf(int k) { return -2 - k; }

// one coarse-fine face, with the sources of the coarse plane's margin (the
// transverse ghost cells the bilinear formula reads beyond the coarse
// block): across the coarse block's side a, side b, and both; a leaf, a
// refined block (-2 - id: the restriction of its child), or kFaceZero
struct CFItem {
    int32_t fine, coarse, slot;
    int32_t ma, mb, mab;
    int8_t dir, lr, oa, ob;
};

template <class T>
struct FaceArgs {
    const T *in;             // boundary planes [6 nb][n^2] of the current field
    T *out;                  // boundary planes the sweep leaves
    const T *cf;             // ghost planes of the coarse-fine faces [ncf][n^2]
    const T *zeros;          // a plane of zeros
    const int32_t *src;      // [6 nb]
    int zero;                // 1: the field is zero (a correction's first sweep): every ghost and flux is 0
};

// ---------------------------------------------------------------------------
// coarse-fine ghosts (fmg_ghfix_parentlev, bilinear) and flux correction
// (fmg_reflux_do) of all levels: a thread per coarse face cell writes the
// 2 x 2 fine ghosts over it and the mean of their fluxes.
// Bound by latency (a few hundred kilobytes to tens of megabytes, read once).
// ---------------------------------------------------------------------------
template <class T, int N>
__global__ void __launch_bounds__(128) k_cf_reflux(const T *__restrict__ u, const T *__restrict__ in,
                                                   T *__restrict__ cf, double *__restrict__ rbuf,
                                                   const CFItem *__restrict__ items, int nitems,
                                                   const int32_t *__restrict__ child, const double *__restrict__ h0,
                                                   const int32_t *__restrict__ level, int f) {
    pdl_enter();
    constexpr int G = N + 2, H = N / 2, NN = N * N;
    constexpr int64_t V = (int64_t)G * G * G;
    const int64_t idx = (int64_t)blockIdx.x * 128 + threadIdx.x;
    const int k = (int)(idx / (H * H)), r = (int)(idx - (int64_t)k * (H * H));
    if (k >= nitems) return;
    const CFItem it = items[k];
    const int pc = r % H, qc = r / H;
    const int fc = (1 - it.lr) + 2 * it.dir;       // the coarse block's face towards the fine one
    const int xc = it.lr == 0 ? N - 1 : 0;         // its plane
    auto coarse = [&](int pa, int qb) -> T {       // coarse cell (pa, qb) of the quadrant, margins included
        int a = pa + it.oa * H, b = qb + it.ob * H;
        const bool ia = a >= 0 && a < N, ib = b >= 0 && b < N;
        int s = it.coarse;
        if (!ia || !ib) s = !ia ? (!ib ? it.mab : it.ma) : it.mb;
        if (s == kFaceZero) return (T)0;
        a = a < 0 ? N - 1 : (a >= N ? 0 : a);
        b = b < 0 ? N - 1 : (b >= N ? 0 : b);
        if (s >= 0) return in[((int64_t)6 * s + fc) * NN + b * N + a];
        int ic, jc, kc;                            // a refined block: its value is the restriction of the child
        put3(it.dir, xc, a, b, ic, jc, kc);
        const int c = child[8 * (int64_t)(-2 - s) + ic / H + 2 * (jc / H) + 4 * (kc / H)];
        return rstrct_linear(u + (int64_t)c * V, G, 2 * (ic % H), 2 * (jc % H), 2 * (kc % H));
    };
    T B[3][3];
#pragma unroll
    for (int q = 0; q < 3; q++)
#pragma unroll
        for (int p = 0; p < 3; p++) B[q][p] = coarse(pc + p - 1, qc + q - 1);
    const T hi = (T)(1.0 / hlev(h0, level[it.fine], f));
    const int ff = it.lr + 2 * it.dir;
    const T *u0p = in + ((int64_t)6 * it.fine + ff) * NN;
    const T *ub = u + (int64_t)it.fine * V;
    const int x2 = it.lr == 0 ? 1 : N - 2;         // the fine block's second layer
    double flux[2][2];
#pragma unroll
    for (int dq = 0; dq < 2; dq++) {
        T g[2];
#pragma unroll
        for (int dp = 0; dp < 2; dp++) {
            const int p = 2 * pc + dp, q = 2 * qc + dq, p1 = 2 * dp, q1 = 2 * dq;   // near cells: pc -+ 1, qc -+ 1
            const T uH = ((T)9 * B[1][1] + B[q1][p1] + (T)3 * B[q1][1] + (T)3 * B[1][p1]) / (T)16;
            int i, j, l;
            put3(it.dir, x2, p, q, i, j, l);
            const T u0 = u0p[q * N + p], uN = ub[cidx(G, i, j, l)];
            g[dp] = ((T)10 * u0 + (T)8 * uH - (T)3 * uN) / (T)15;
            flux[dq][dp] = (double)((it.lr == 0 ? u0 - g[dp] : g[dp] - u0) * hi);
        }
        vec_store<T, 2>(cf + (int64_t)k * NN + (2 * qc + dq) * N + 2 * pc, g);
    }
    const double v = (flux[0][0] + flux[1][0] + flux[0][1] + flux[1][1]) * 0.25;
    rbuf[(int64_t)it.slot * NN + (qc + it.ob * H) * N + (pc + it.oa * H)] = v;
}

// ---------------------------------------------------------------------------
// the boundary planes of the listed blocks from their cells (first sweep
// after a field was set otherwise than by a sweep or a prolongation)
// ---------------------------------------------------------------------------
template <class T, int N>
__global__ void __launch_bounds__(256) k_faces_of(const T *__restrict__ u, T *__restrict__ out,
                                                  const int32_t *__restrict__ blocks, int nblk) {
    pdl_enter();
    constexpr int G = N + 2, NN = N * N;
    constexpr int64_t V = (int64_t)G * G * G;
    for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < (int64_t)nblk * 6 * NN; e += (int64_t)gridDim.x * 256) {
        const int q = (int)(e / (6 * NN)), r = (int)(e - (int64_t)q * (6 * NN));
        const int fc = r / NN, t = r - fc * NN, b = blocks[q];
        int i, j, k;
        put3(fc >> 1, (fc & 1) ? N - 1 : 0, t % N, t / N, i, j, k);
        out[(int64_t)b * 6 * NN + r] = u[b * V + cidx(G, i, j, k)];
    }
}
// ---------------------------------------------------------------------------
// red-black sweep of the listed blocks with the ghost planes from FaceArgs:
// k_relax_bulk's pipeline, but warp 0 also brings the block's six ghost
// planes (dense, 16-byte aligned 1D bulk copies) into the stage, beside the
// interior spans of u and rhs.  A thread owns a cell pair -- the colour-1
// cell and its x neighbour of colour 2 -- reads its outer neighbours from the
// staged block or plane by offsets computed once, and leaves the pair in the
// boundary planes it lies on.  SW = 0: colour `ipass`; SW > 0: SW full sweeps
// on the staged block (the mixed schedule's fused sweeps, with k_relax_bulk's
// expressions).  Waits are bounded as there.  (Planes read straight from
// global memory into registers left their latency on the consumers' path:
// 751 us against 370 us for k_relax_bulk's two fused sweeps on jeans6.)
// Bound by issue slots and the waits between colours.  56 registers a thread,
// so that nothing spills: two fused sweeps of 8^3 FP32 blocks at 5 CTAs per
// SM and 40 registers made the six-level cloud's mixed solve 74.5 ms, at 4
// CTAs 73.2; with places, planes and stages found by division per tile 75.8.
// ---------------------------------------------------------------------------
template <class T, int N>
struct FacePlan {
    using Bulk = BulkPlan<T, N>;
    static constexpr int LO = Bulk::LO, SPAN = Bulk::SPAN, NN = N * N;
    static constexpr int BPC = Tile<N>::BPC;
    static constexpr int BLK = 2 * SPAN + 6 * NN;   // values of a staged block: u span, rhs span, planes
    static constexpr int STAGE_BYTES = BPC * BLK * (int)sizeof(T);
    static constexpr int S0 = 49152 / STAGE_BYTES;
    static constexpr int S = S0 >= 3 ? 3 : 2;
    static constexpr int SMEM = S * STAGE_BYTES;
    static_assert((SPAN * sizeof(T)) % 16 == 0 && (NN * sizeof(T)) % 16 == 0, "copies are whole 16-byte units");
};
template <class T, int N, int NT>
__host__ __device__ constexpr int relax_faces_min_ctas() {
    constexpr int bySmem = (228 * 1024) / (FacePlan<T, N>::SMEM + 4 * 1024);
    constexpr int byRegs = 65536 / (NT * 56);
    constexpr int m = bySmem < byRegs ? bySmem : byRegs;
    return m < 1 ? 1 : (m > 2048 / NT ? 2048 / NT : m);
}
template <class T, int N, int NT, int SW>
__global__ void __launch_bounds__(NT, relax_faces_min_ctas<T, N, NT>())
    k_relax_faces(T *__restrict__ u, const T *__restrict__ rhs, const int32_t *__restrict__ blocks, int nblk,
                  const double *__restrict__ h0, const int32_t *__restrict__ level, const int32_t *__restrict__ rslot,
                  const double *__restrict__ rbuf, FaceArgs<T> fa, int f, int ipass, unsigned long long *out, int *err,
                  uint32_t cpolls) {
    pdl_enter();
    using Pl = FacePlan<T, N>;
    constexpr int G = N + 2, NN = N * N, BPC = Pl::BPC, HALF = N * N * N / 2, S = Pl::S, HN = N / 2;
    constexpr int64_t V = (int64_t)G * G * G;
    constexpr int NCW = NT / 32 - 1, NCT = 32 * NCW;   // consumer warps / threads
    constexpr int LO = Pl::LO, SPAN = Pl::SPAN, BLK = Pl::BLK;
    constexpr uint32_t SB = (uint32_t)(SPAN * sizeof(T)), FB = (uint32_t)(NN * sizeof(T));
    constexpr int ITER = (BPC * HALF + NCT - 1) / NCT;   // cell pairs per thread and tile
    extern __shared__ __align__(128) unsigned char bulk_smem[];
    T *const ring = reinterpret_cast<T *>(bulk_smem);    // [S][BPC][BLK]
    __shared__ __align__(8) uint64_t full[S], empty[S];
    __shared__ int issued[S], consumed[S], pab, cab;   // pab / cab: the producer / a consumer warp gave up
    // per-block data of the tiles: two windows of R steps (see k_relax_bulk)
    constexpr int R = (32 / BPC) > 2 * S ? 32 / BPC : 2 * S;
    __shared__ int bid[2 * R][BPC];
    __shared__ int fs[2 * R][BPC][6];
    __shared__ int ssl[2 * R][BPC][6];
    __shared__ int8_t hasr[2 * R][BPC];
    __shared__ T shh[2 * R][BPC], shi[2 * R][BPC];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ntiles = (nblk + BPC - 1) / BPC;
    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], NCW);
            issued[s] = 0;
            consumed[s] = 0;
        }
        pab = 0;
        cab = 0;
        mbar_init_fence();
    }
    __syncthreads();
    double m = 0.0;
    const int nsteps = ntiles > (int)blockIdx.x ? (ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    auto fill_window = [&](int w) {   // warp 0: a lane per (step, block) of the window
        for (int e = lane; e < R * BPC; e += 32) {
            const int step = w * R + e / BPC, q = e % BPC, slot = step % (2 * R);
            const int first = ((int)blockIdx.x + step * (int)gridDim.x) * BPC;
            if (step < nsteps && first + q < nblk) {
                const int b = blocks[first + q];
                bid[slot][q] = b;
                int any = 0;
                for (int fc = 0; fc < 6; fc++) {
                    const int v = rslot[6 * (int64_t)b + fc];
                    ssl[slot][q][fc] = v;
                    any |= v >= 0;
                    fs[slot][q][fc] = fa.zero ? kFaceZero : fa.src[6 * (int64_t)b + fc];
                }
                hasr[slot][q] = (int8_t)any;
                const double hd = hlev(h0, level[b], f);
                shh[slot][q] = (T)hd;
                shi[slot][q] = (T)(1.0 / hd);
            } else {
                hasr[slot][q] = 0;
            }
        }
        __syncwarp();
    };
    if (warp == 0) {
        fill_window(0);
        int it = 0;
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
            const int s = it % S;
            if (it >= S) {
                const bool ok = __all_sync(
                    0xffffffffu, mbar_wait_bounded_abort(&empty[s], (uint32_t)((it / S - 1) & 1), kWaitPolls, &cab));
                if (!ok) {
                    if (lane == 0) pab = 1;
                    break;
                }
            }
            if (__any_sync(0xffffffffu, *(volatile int *)&cab)) break;
            if (it % R == S && (it / R + 1) * R < nsteps) fill_window(it / R + 1);
            const int first = tile * BPC;
            const int cnt = nblk - first < BPC ? nblk - first : BPC;
            const int slot = it % (2 * R);
            if (lane == 0) {
                issued[s]++;
                mbar_expect_tx(&full[s], (uint32_t)cnt * (2 * SB + 6 * FB));   // releases the per-block data
            }
            __syncwarp();
            for (int e = lane; e < 8 * cnt; e += 32) {   // eight copies per block, a lane each
                const int q = e >> 3, w = e & 7;
                const int64_t b = bid[slot][q];
                T *st = ring + (s * BPC + q) * BLK;
                if (w < 6) {
                    const int v = fs[slot][q][w];
                    const T *p = v >= 0 ? fa.in + (int64_t)v * NN : (v == kFaceZero ? fa.zeros : fa.cf + (int64_t)(-2 - v) * NN);
                    bulk_load(st + 2 * SPAN + w * NN, p, FB, &full[s]);
                } else if (w == 6) {
                    bulk_load(st, u + b * V + LO, SB, &full[s]);
                } else {
                    bulk_load(st + SPAN, rhs + b * V + LO, SB, &full[s]);
                }
            }
        }
    } else {
        const int ct = tid - 32;   // consumer thread 0..NCT-1
        T mt = (T)0;               // max |resh2| (exact in T; widened once)
        // pair t = ct + x NCT of a tile: block q, cells (2 i2, j, k) and (2 i2 + 1, j, k)
        auto pair_of = [&](int x, int &q, int &i2, int &j, int &k) {
            const int t = ct + x * NCT;
            q = t / HALF;
            const int r = t - q * HALF;
            i2 = r % HN;
            j = (r / HN) % N;
            k = r / (HN * N);
        };
        // the pair's cell a (even or odd i) and its neighbours but the
        // partner, as offsets into the staged block
        struct Nb { int c, x, ym, yp, zm, zp; };
        auto around = [&](int i2, int j, int k, int a) {
            Nb o;
            o.c = cidx(G, 2 * i2 + a, j, k) - LO;
            const int i = 2 * i2 + a, F0 = 2 * SPAN;
            o.x = (a ? i2 == HN - 1 : i2 == 0) ? F0 + a * NN + k * N + j : o.c + (a ? 1 : -1);
            o.ym = j == 0 ? F0 + 2 * NN + k * N + i : o.c - G;
            o.yp = j == N - 1 ? F0 + 3 * NN + k * N + i : o.c + G;
            o.zm = k == 0 ? F0 + 4 * NN + j * N + i : o.c - G * G;
            o.zp = k == N - 1 ? F0 + 5 * NN + j * N + i : o.c + G * G;
            return o;
        };
        int q0, i20, j0, k0;   // one pair per thread: its place never changes
        pair_of(0, q0, i20, j0, k0);
        const int par0 = (j0 + k0 + 1) & 1;   // colour 1's cell of the pair
        Nb n1 = around(i20, j0, k0, par0), n2 = around(i20, j0, k0, 1 - par0);
        // where the pair goes in the block's planes (-1: not on that axis' planes); one cell in x, both in y and z
        struct Pl3 { int x, y, z; };
        auto planes_of = [&](int i2, int j, int k) {
            Pl3 o;
            o.x = i2 == 0 ? k * N + j : (i2 == HN - 1 ? NN + k * N + j : -1);
            o.y = j == 0 ? 2 * NN + k * N + 2 * i2 : (j == N - 1 ? 3 * NN + k * N + 2 * i2 : -1);
            o.z = k == 0 ? 4 * NN + j * N + 2 * i2 : (k == N - 1 ? 5 * NN + j * N + 2 * i2 : -1);
            return o;
        };
        const Pl3 pl0 = planes_of(i20, j0, k0);
        uint32_t phase = 0;   // stage s, its phase and the data slot by counting: no divisions per tile
        int s = -1, slot = -1;
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            if (++s == S) {
                s = 0;
                phase ^= 1;
            }
            if (++slot == 2 * R) slot = 0;
            const bool got = __all_sync(0xffffffffu, mbar_wait_bounded(&full[s], phase, cpolls));
            if constexpr (SW == 0) {
                if (!got) {
                    if (lane == 0) atomicExch(&cab, 1);
                    break;
                }
            }
            const int first = tile * BPC;
            T *const st = ring + s * BPC * BLK;
            auto live = [&](int x) {
                const int t = ct + x * NCT;
                return t < BPC * HALF && first + t / HALF < nblk;
            };
            // the pair's current values by colour, held by this thread alone; its right-hand sides and widths
            T own1[ITER], own2[ITER], rr1[ITER], rr2[ITER], th[ITER], ti[ITER];
            bool flux[ITER];
            if (got) {
#pragma unroll
                for (int x = 0; x < ITER; x++) {
                    if (!live(x)) continue;
                    int q, i2, j, k;
                    pair_of(x, q, i2, j, k);
                    const int a1 = (j + k + 1) & 1;
                    const T *p = st + q * BLK + cidx(G, 2 * i2, j, k) - LO;
                    own1[x] = p[a1];
                    own2[x] = p[1 - a1];
                    if (SW > 0 || ipass == 1) rr1[x] = p[SPAN + a1];
                    if (SW > 0 || ipass == 2) rr2[x] = p[SPAN + 1 - a1];
                    th[x] = shh[slot][q];
                    ti[x] = shi[slot][q];
                    flux[x] = hasr[slot][q] != 0;
                }
            }
            auto colour = [&](bool one, bool keep, bool store) {   // colour 1 (one) or 2
#pragma unroll
                for (int x = 0; x < ITER; x++) {
                    if (!live(x)) continue;
                    int q, i2, j, k;
                    pair_of(x, q, i2, j, k);
                    const int a1 = (j + k + 1) & 1, a = one ? a1 : 1 - a1;
                    const Nb o = ITER == 1 ? (one ? n1 : n2) : around(i2, j, k, a);
                    T *const ub = st + q * BLK;
                    const T uc = one ? own1[x] : own2[x], partner = one ? own2[x] : own1[x];
                    const T other = ub[o.x], ym = ub[o.ym], yp = ub[o.yp], zm = ub[o.zm], zp = ub[o.zp];
                    const T hh = th[x], hi = ti[x], rr = one ? rr1[x] : rr2[x];
                    T resh2;
                    if (SW == 0 || flux[x]) {   // the reference's flux form (fmg_poisson.F90:160-211)
                        const T xp = a ? other : partner, xm = a ? partner : other;
                        T fxp = (xp - uc) * hi, fxm = (uc - xm) * hi, fyp = (yp - uc) * hi, fym = (uc - ym) * hi,
                          fzp = (zp - uc) * hi, fzm = (uc - zm) * hi;
                        if (flux[x]) {   // faces covered by finer blocks take the corrected flux
                            auto corrected = [&](int fc, int p, int r, T &fl) {
                                const int sl = ssl[slot][q][fc];
                                if (sl >= 0) fl = fa.zero ? (T)0 : (T)rbuf[(int64_t)sl * NN + r * N + p];
                            };
                            const int i = 2 * i2 + a;
                            if (i == N - 1) corrected(1, j, k, fxp);
                            if (i == 0) corrected(0, j, k, fxm);
                            if (j == N - 1) corrected(3, i, k, fyp);
                            if (j == 0) corrected(2, i, k, fym);
                            if (k == N - 1) corrected(5, i, j, fzp);
                            if (k == 0) corrected(4, i, j, fzm);
                        }
                        T t = fxp - fxm;
                        t = t + fyp;
                        t = t - fym;
                        t = t + fzp;
                        t = t - fzm;
                        resh2 = (t - rr * hh) * hh;
                    } else {   // the mixed preconditioner's cheaper form (k_relax_bulk)
                        const T sx = (partner - uc) + (other - uc);
                        const T sy = (yp - uc) + (ym - uc);
                        const T sz = (zp - uc) + (zm - uc);
                        resh2 = fma((sx + sy) + sz, hi * hh, -(rr * (hh * hh)));
                    }
                    T v;
                    if constexpr (SW == 0) v = uc + (T)(1.0 / 6.0) * resh2;
                    else v = fma((T)(1.0 / 6.0), resh2, uc);
                    if (one) own1[x] = v;
                    else own2[x] = v;
                    if (store) u[(int64_t)bid[slot][q] * V + (o.c + LO)] = v;
                    if (keep) ub[o.c] = v;
                    if constexpr (sizeof(T) == 4) {
                        mt = fmaxf(fabsf(resh2), mt);   // one instruction; a NaN leaves mt, as the comparison does
                    } else {
                        const T ar = resh2 < (T)0 ? -resh2 : resh2;
                        mt = ar > mt ? ar : mt;
                    }
                }
            };
            if constexpr (SW > 0) {
                if (got) colour(true, true, SW == 1);
                // the consumers meet between colours; the first time they
                // also OR the failed waits, so every warp decides alike
                if (consumers_sync_or(1, NCT, !got)) {
                    if (ct == 0) atomicExch(&cab, 1);
                    break;
                }
#pragma unroll
                for (int r = 0; r < SW; r++) {
                    const bool last = r == SW - 1;
                    if (r > 0) {
                        colour(true, true, last);
                        asm volatile("bar.sync 1, %0;" ::"r"(NCT) : "memory");
                    }
                    colour(false, !last, last);
                    if (!last) asm volatile("bar.sync 1, %0;" ::"r"(NCT) : "memory");
                }
                // the stage held ordinary stores; the next bulk copy into it
                // goes through the async proxy
                fence_async_shared();
            } else {
                colour(ipass == 1, false, true);
            }
            __syncwarp();
            if (lane == 0) {
                if (warp == 1) consumed[s]++;
                mbar_arrive(&empty[s]);   // this warp is done with stage s
            }
#pragma unroll
            for (int x = 0; x < ITER; x++) {   // the pair into the planes it lies on
                if (!live(x)) continue;
                int q, i2, j, k;
                pair_of(x, q, i2, j, k);
                const bool one = (j + k) & 1;   // colour 1's cell is the even one
                const Pl3 pl = ITER == 1 ? pl0 : planes_of(i2, j, k);
                T *o = fa.out + (int64_t)bid[slot][q] * (6 * NN);
                const T pr[2] = {one ? own1[x] : own2[x], one ? own2[x] : own1[x]};
                if (pl.x >= 0) o[pl.x] = i2 == 0 ? pr[0] : pr[1];
                if (pl.y >= 0) vec_store<T, 2>(o + pl.y, pr);
                if (pl.z >= 0) vec_store<T, 2>(o + pl.z, pr);
            }
        }
        m = (double)mt;
    }
    __syncthreads();
    if (tid == 0 && (pab || cab)) {   // loads still in flight: wait for them (bounded), then report
        for (int s = 0; s < S; s++)
            for (int ph = consumed[s]; ph < issued[s]; ph++) mbar_wait_bounded(&full[s], (uint32_t)(ph & 1), kWaitPolls);
        atomicExch(err, 1);
    }
    cta_max_atomic(m, out);
}

// ---------------------------------------------------------------------------
// the descent step of fmg_lin (fmg.F90:296-311) in one launch: residual of
// level f (fmg_poisson_resid, ghosts from FaceArgs), its restriction into
// the next level's right-hand side (fmg_rstrct) and that level's correction
// zeroed (whole blocks, as fmg_fill0).  The residual itself stays in shared
// memory: nothing reads it afterwards.
// ---------------------------------------------------------------------------
// blocks per CTA: up to 256 coarse cells, a thread each, within 48 KB of staged blocks
template <int N>
__host__ __device__ constexpr int resid_faces_bpc() { return N >= 16 ? 1 : (N == 8 ? 4 : 16); }
template <class T, int N>
__global__ void __launch_bounds__(256) k_resid_faces(const T *__restrict__ u, const T *__restrict__ rhs,
                                                     T *__restrict__ rhsc, T *__restrict__ uc,
                                                     const int32_t *__restrict__ blocks, int nblk,
                                                     const double *__restrict__ h0, const int32_t *__restrict__ level,
                                                     const int32_t *__restrict__ rslot, const double *__restrict__ rbuf,
                                                     FaceArgs<T> fa, int f) {
    pdl_enter();
    constexpr int G = N + 2, NN = N * N, V = G * G * G, BPC = resid_faces_bpc<N>();
    constexpr int H = N / 2, GC = H + 2, VC = GC * GC * GC, HC = H * H * H;
    constexpr int LO = 1 + G + G * G, LEN = (N - 1) * LO + 1;   // interior span of a block
    __shared__ T sh[BPC * V];
    __shared__ int ssl[BPC][6], fs[BPC][6], sbid[BPC];
    __shared__ T shi[BPC];
    __shared__ int8_t hasr[BPC];
    const int first = blockIdx.x * BPC;
    const int nq = nblk - first < BPC ? nblk - first : BPC;
    for (int t = threadIdx.x; t < nq * LEN; t += 256) {
        const int q = t / LEN, r = t - q * LEN;
        sh[q * V + LO + r] = u[(int64_t)blocks[first + q] * V + LO + r];
    }
    if ((int)threadIdx.x < nq) {
        const int q = threadIdx.x, b = blocks[first + q];
        int any = 0;
        for (int fc = 0; fc < 6; fc++) {
            const int v = rslot[6 * (int64_t)b + fc];
            ssl[q][fc] = v;
            any |= v >= 0;
            fs[q][fc] = fa.src[6 * (int64_t)b + fc];
        }
        sbid[q] = b;
        hasr[q] = (int8_t)any;
        shi[q] = (T)(1.0 / hlev(h0, level[b], f));
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nq * 6 * NN; t += 256) {   // the ghost planes
        const int q = t / (6 * NN), r = t - q * (6 * NN), fc = r / NN, e = r - fc * NN;
        const int v = fs[q][fc];
        int i, j, k;
        put3(fc >> 1, (fc & 1) ? N : -1, e % N, e / N, i, j, k);
        sh[q * V + cidx(G, i, j, k)] =
            v >= 0 ? fa.in[(int64_t)v * NN + e] : (v == kFaceZero ? (T)0 : fa.cf[(int64_t)(-2 - v) * NN + e]);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nq * HC; t += 256) {
        const int q = t / HC, r = t - q * HC;
        const int i = r % H, j = (r / H) % H, k = r / (H * H);
        const T hi = shi[q];
        const T *rb = rhs + (int64_t)sbid[q] * V;
        const TileFlux<T, N> F{sh + q * V, hi, hasr[q] ? ssl[q] : nullptr, rbuf};
        auto res = [&](int di, int dj, int dk) -> T {
            const int a = 2 * i + di, b = 2 * j + dj, c = 2 * k + dk;
            return rb[cidx(G, a, b, c)] - F.div(a, b, c) * hi;
        };
        T s = res(0, 0, 0) + res(1, 0, 0);   // rstrct_linear's order
        s = s + res(0, 1, 0);
        s = s + res(0, 0, 1);
        s = s + res(1, 1, 0);
        s = s + res(1, 0, 1);
        s = s + res(0, 1, 1);
        s = s + res(1, 1, 1);
        rhsc[(int64_t)sbid[q] * VC + cidx(GC, i, j, k)] = s * (T)(1.0 / 8.0);
    }
    for (int t = threadIdx.x; t < nq * VC; t += 256) uc[(int64_t)sbid[t / VC] * VC + t % VC] = (T)0;
}

// ---------------------------------------------------------------------------
// the outer FP64 residual (fmg.F90:183, fmg_poisson_resid at level 0) with
// planes, and the correction's addition that leaves them.  Only on boxes
// without physical-boundary faces: there the ghosts of psi are not zero.
// ---------------------------------------------------------------------------
template <int N>
__host__ __device__ constexpr int resid_planes_bpc() { return N >= 16 ? 1 : (N == 8 ? 2 : 8); }
template <class TO, int N>
__global__ void __launch_bounds__(256) k_resid_planes(TO *__restrict__ res, const double *__restrict__ u,
                                                      const double *__restrict__ rhs,
                                                      const int32_t *__restrict__ blocks, int nblk,
                                                      const double *__restrict__ h0, const int32_t *__restrict__ level,
                                                      const int32_t *__restrict__ rslot,
                                                      const double *__restrict__ rbuf, FaceArgs<double> fa) {
    pdl_enter();
    constexpr int G = N + 2, NN = N * N, V = G * G * G, CELLS = N * N * N, BPC = resid_planes_bpc<N>();
    constexpr int LO = 1 + G + G * G, LEN = (N - 1) * LO + 1;   // interior span of a block
    __shared__ double sh[BPC * V];
    __shared__ int ssl[BPC][6], sbid[BPC];
    __shared__ double shi[BPC];
    __shared__ int8_t hasr[BPC];
    const int first = blockIdx.x * BPC;
    const int nq = nblk - first < BPC ? nblk - first : BPC;
    // the span's cells but its ghost positions (interior ones only), and the
    // ghost planes: disjoint, so one barrier
    for (int t = threadIdx.x; t < nq * LEN; t += 256) {
        const int q = t / LEN, r = t - q * LEN + LO;
        const int i = r % G, j = (r / G) % G;
        const double v = u[(int64_t)blocks[first + q] * V + r];
        if (i >= 1 && i <= N && j >= 1 && j <= N) sh[q * V + r] = v;
    }
    for (int t = threadIdx.x; t < nq * 6 * NN; t += 256) {
        const int q = t / (6 * NN), r = t - q * (6 * NN), fc = r / NN, e = r - fc * NN;
        const int v = fa.src[6 * (int64_t)blocks[first + q] + fc];
        int i, j, k;
        put3(fc >> 1, (fc & 1) ? N : -1, e % N, e / N, i, j, k);
        sh[q * V + cidx(G, i, j, k)] =
            v >= 0 ? fa.in[(int64_t)v * NN + e] : (v == kFaceZero ? 0.0 : fa.cf[(int64_t)(-2 - v) * NN + e]);
    }
    if ((int)threadIdx.x < nq) {
        const int q = threadIdx.x, b = blocks[first + q];
        int any = 0;
        for (int fc = 0; fc < 6; fc++) {
            const int v = rslot[6 * (int64_t)b + fc];
            ssl[q][fc] = v;
            any |= v >= 0;
        }
        sbid[q] = b;
        hasr[q] = (int8_t)any;
        shi[q] = 1.0 / hlev(h0, level[b], 0);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nq * CELLS; t += 256) {
        const int q = t / CELLS, r = t - q * CELLS;
        const int i = r % N, j = (r / N) % N, k = r / NN;
        const double hi = shi[q];
        const TileFlux<double, N> F{sh + q * V, hi, hasr[q] ? ssl[q] : nullptr, rbuf};
        const int64_t c = (int64_t)sbid[q] * V + cidx(G, i, j, k);
        res[c] = (TO)(rhs[c] - F.div(i, j, k) * hi);
    }
}
template <class T, int N>
__global__ void __launch_bounds__(256) k_add_planes(double *__restrict__ a, const T *__restrict__ d,
                                                    const int32_t *__restrict__ blocks, int nblk,
                                                    double *__restrict__ planes) {
    pdl_enter();
    constexpr int G = N + 2, CELLS = N * N * N, PER = CELLS / 256 > 0 ? CELLS / 256 : 1;
    constexpr int BPC = CELLS >= 256 ? 1 : 256 / CELLS;   // blocks per step of a CTA
    constexpr int64_t V = (int64_t)G * G * G;
    for (int b0 = blockIdx.x * BPC; b0 < nblk; b0 += gridDim.x * BPC) {
        const int q = b0 + (int)threadIdx.x / CELLS;
        if (q >= nblk) continue;
        const int64_t b = blocks[q];
        double v[PER];
#pragma unroll
        for (int x = 0; x < PER; x++) {
            const int r = (int)threadIdx.x % CELLS + 256 * x;
            const int64_t c = b * V + cidx(G, r % N, (r / N) % N, r / (N * N));
            v[x] = a[c] + (double)d[c];
        }
#pragma unroll
        for (int x = 0; x < PER; x++) {
            const int r = (int)threadIdx.x % CELLS + 256 * x;
            const int i = r % N, j = (r / N) % N, k = r / (N * N);
            a[b * V + cidx(G, i, j, k)] = v[x];
            faces_put<double, N>(planes, b, i, j, k, v[x]);
        }
    }
}

}  // namespace sfm
