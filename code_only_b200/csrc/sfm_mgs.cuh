// sfm_mgs.cuh -- the base-grid multigrid (mg.F90:42-218) with every level in
// shared memory: one CTA for base grids of up to 16^3 cells, a cluster of 8
// CTAs with the large levels cut into z slabs for 32^3.
//
// A solve is a few hundred dependent steps (colour sweeps, residuals,
// transfers), most of them on levels of 1 to 512 cells: its time is the time
// of a step.  k_mg_cycle spends a step on L2 latency (large levels), on level
// pointers and widths looked up at run time, on integer division into cell
// coordinates and on barriers of 16 warps.  Here the level is a template
// argument (extents, offsets and widths are constants or one shared load),
// levels of at most 4^3 cells run on one warp with __syncwarp, the slabs of
// neighbouring CTAs are read through distributed shared memory, and ghost
// cells do not exist: each access resolves its boundary itself (periodic
// image, zero, minus or plus the boundary cell), which is the value the
// reference's boundary steps store, so those steps and their barriers are
// gone.  Every other expression is k_mg_cycle's, in its order: bit-identical.
#pragma once
#include "sfm_device.cuh"
#include "sfm_mg.cuh"

namespace sfm {

// boundary of the base grid: what lies beyond its faces
enum MgMode {
    kMgPeriodic = 0,   // periodic images
    kMgIsolated = 1,   // zero for the operator, minus the boundary cell for prolongations
    kMgZMirror = 2,    // isolated, but the z-min face mirrors
    kMgZPeriodic = 3   // isolated in x and y, periodic in z
};

struct MgsArgs {
    const int32_t *baseIdx;   // base block of each position
    int ngb;                  // base blocks per edge
    int n, G;                 // cells per block edge, with ghosts
    int64_t V;
    double hbase;
    int nmax;                 // cap on the defect corrections
};

// TOP: log2 of the base grid's cells per edge; C: CTAs of the cluster
template <int TOP, int C, int MODE>
struct Mgs {
    static constexpr int kWideMin = 4;   // levels of at least 2^4 cells per edge are cut into slabs
    static __host__ __device__ constexpr bool wide(int ln) { return C > 1 && ln >= kWideMin; }
    static __host__ __device__ constexpr int planes(int ln) { return wide(ln) ? (1 << ln) / C : (1 << ln); }
    static __host__ __device__ constexpr int vol(int ln) { return (1 << (2 * ln)) * planes(ln); }
    // shared memory, in doubles: per level U, RHO and RHS (the finest: U, RHO, PSI, SRC)
    static __host__ __device__ constexpr int base(int ln) {
        int o = 0;
        for (int l = TOP; l > ln; l--) o += (l == TOP ? 4 : 3) * vol(l);
        return o;
    }
    static __host__ __device__ constexpr int U(int ln) { return base(ln); }
    static __host__ __device__ constexpr int RHO(int ln) { return base(ln) + vol(ln); }
    static __host__ __device__ constexpr int RHS(int ln) { return base(ln) + 2 * vol(ln); }   // ln < TOP
    static constexpr int PSI = 2 * vol(TOP), SRC = 3 * vol(TOP);
    static __host__ __device__ constexpr int total() { return base(-1); }
    static constexpr bool perXY = MODE == kMgPeriodic, perZ = MODE == kMgPeriodic || MODE == kMgZPeriodic;
    static constexpr bool mirZ = MODE == kMgZMirror;

    struct Tables {            // per kernel: cubic nodes and weights of levels 2.. (index n + i), widths
        int c[2 << TOP][4];
        double w[2 << TOP][4];
        double h2[TOP + 1], h2i[TOP + 1];
    };
    struct Ctx {
        const Tables *t;
        int rank;              // CTA in the cluster
    };
    static __device__ __forceinline__ void fill_tables(Tables &t, double hbase) {
        for (int e = threadIdx.x; e < (2 << TOP); e += blockDim.x) {   // entry n + i of level n >= 4
            int n = 4;
            while (2 * n <= e) n *= 2;
            if (e >= 4) cubic_weights(e - n, -1, n / 2, t.c[e], t.w[e]);
        }
        if ((int)threadIdx.x <= TOP) {
            const double hh = hbase * (double)(1 << (TOP - (int)threadIdx.x));
            t.h2[threadIdx.x] = hh * hh;
            t.h2i[threadIdx.x] = 1.0 / (hh * hh);
        }
    }
    static __device__ __forceinline__ void meet() {   // everyone who holds a part of the finest level
        if (C > 1) mg_cluster_sync();
        else __syncthreads();
    }
    // maximum over the cluster; red (32 values) and slot in shared memory
    static __device__ __forceinline__ double vmax(double v, double *red, double *slot) {
        v = mg_block_max(v, red);
        if (C > 1) {
            if (threadIdx.x == 0) *slot = v;
            mg_cluster_sync();
            for (int q = 0; q < C; q++) {
                const double t = *mg_map_rank(slot, q);
                v = t > v ? t : v;
            }
            mg_cluster_sync();
        }
        return v;
    }
    // residual of PSI into the finest RHO; this thread's maximum
    static __device__ __forceinline__ double defect(const Ctx &x) {
        constexpr int N = 1 << TOP;
        double v = 0.0;
        for (int c = threadIdx.x; c < vol(TOP); c += blockDim.x) {
            const double r = resid<TOP>(x, PSI, SRC, c & (N - 1), (c >> TOP) & (N - 1), c >> (2 * TOP));
            sm()[RHO(TOP) + c] = r;
            const double q = fabs(r);
            v = q > v ? q : v;
        }
        return v;
    }
    // mg_lin (mg.F90:106-218) for the residual in RHO, its correction added
    // to PSI; this thread's max |resh2| of the last sweep
    static __device__ __forceinline__ double correct(const Ctx &x) {
        double rm = 0.0;
        if (TOP >= 3 || threadIdx.x < 32) {   // base grids of at most 4^3 cells: one warp
            rstrct_rho<TOP>(x);
            rm = fmg<TOP>(x);
        }
        if (TOP < 3) __syncthreads();
        for (int c = threadIdx.x; c < vol(TOP); c += blockDim.x) sm()[PSI + c] = sm()[PSI + c] + sm()[U(TOP) + c];
        return rm;
    }
    // this CTA's arrays (the symbol itself, so that accesses are shared loads and not generic ones)
    static __device__ __forceinline__ double *sm() {
        extern __shared__ double mgs_smem[];
        return mgs_smem;
    }

    // who works on a level: the cluster, the CTA (8^3 and up), or one warp
    template <int LN>
    static __device__ __forceinline__ int team_size() {
        return LN >= 3 ? (int)blockDim.x : 32;
    }
    template <int LN>
    static __device__ __forceinline__ void sync() {
        if constexpr (wide(LN)) mg_cluster_sync();
        else if constexpr (LN >= 3) __syncthreads();
        else __syncwarp();
    }
    // cell (i, j, k) of an array of level LN, on whichever CTA holds the plane
    template <int LN, bool REMOTE>
    static __device__ __forceinline__ double get(const Ctx &x, int off, int i, int j, int k) {
        constexpr int n = 1 << LN, P = planes(LN);
        if constexpr (wide(LN)) {
            const int r = k / P, o = off + ((k - r * P) * n + j) * n + i;
            return r == x.rank ? sm()[o] : mg_map_rank(sm(), r)[o];
        } else {
            const int o = off + (k * n + j) * n + i;
            return REMOTE ? mg_map_rank(sm(), 0)[o] : sm()[o];
        }
    }
    // the seven-point sum of mg_poisson.F90 in its order; (i, j, kl) a cell of this CTA's slab
    template <int LN>
    static __device__ __forceinline__ double lap(const Ctx &x, int u, int i, int j, int kl, double uc) {
        constexpr int n = 1 << LN, P = planes(LN);
        const double *c = sm() + u + (kl * n + j) * n;
        auto X = [&](int a) -> double {
            if (perXY) return c[a & (n - 1)];
            return a >= 0 && a < n ? c[a] : 0.0;
        };
        auto Y = [&](int b) -> double {
            if (perXY) return sm()[u + (kl * n + (b & (n - 1))) * n + i];
            return b >= 0 && b < n ? sm()[u + (kl * n + b) * n + i] : 0.0;
        };
        auto Z = [&](int d) -> double {   // d: plane relative to the slab
            if constexpr (wide(LN)) {
                if (d >= 0 && d < P) return sm()[u + (d * n + j) * n + i];
                int k = d + x.rank * P;
                if (k < 0 || k >= n) {
                    if (!perZ) return mirZ && k < 0 ? uc : 0.0;
                    k &= n - 1;
                }
                return mg_map_rank(sm(), k / P)[u + ((k & (P - 1)) * n + j) * n + i];
            } else {
                if (perZ) return sm()[u + ((d & (n - 1)) * n + j) * n + i];
                if (d >= 0 && d < n) return sm()[u + (d * n + j) * n + i];
                return mirZ && d < 0 ? uc : 0.0;
            }
        };
        double s = X(i + 1) + X(i - 1);
        s = s + Y(j + 1);
        s = s + Y(j - 1);
        s = s + Z(kl + 1);
        s = s + Z(kl - 1);
        s = s - 6.0 * uc;
        return s;
    }
    // value of a coarse level for a prolongation, one cell beyond the box included
    template <int LN, bool REMOTE>
    static __device__ __forceinline__ double beyond(const Ctx &x, int u, int i, int j, int k) {
        constexpr int n = 1 << LN;
        bool neg = false;
        auto fix = [&](int a, bool per, bool mirror) {
            if (a >= 0 && a < n) return a;
            if (per) return a & (n - 1);
            if (!(mirror && a < 0)) neg = !neg;
            return a < 0 ? 0 : n - 1;
        };
        i = fix(i, perXY, false);
        j = fix(j, perXY, false);
        k = fix(k, perZ, mirZ);
        const double v = get<LN, REMOTE>(x, u, i, j, k);
        return neg ? -v : v;
    }
    // one sweep, both colours; this thread's max |resh2|
    template <int LN>
    static __device__ __forceinline__ double relax(const Ctx &x, int rhs) {
        constexpr int n = 1 << LN, u = U(LN), P = planes(LN);
        double rm = 0.0;
        const double h2 = x.t->h2[LN];
#pragma unroll 1
        for (int ipass = 1; ipass <= 2; ipass++) {
            if constexpr (LN == 0) {
                if (ipass == 2 && threadIdx.x == 0) {
                    const double uc = sm()[u];
                    const double resh2 = lap<0>(x, u, 0, 0, 0, uc) - h2 * sm()[rhs];
                    sm()[u] = uc + (1.0 / 6.0) * resh2;
                    rm = fabs(resh2);
                }
            } else {
                constexpr int half = n * n * P / 2;
                for (int c = threadIdx.x; c < half; c += team_size<LN>()) {
                    const int i2 = c & (n / 2 - 1), j = (c >> (LN - 1)) & (n - 1), kl = c >> (2 * LN - 1);
                    const int k = kl + (wide(LN) ? x.rank * P : 0);
                    const int i = 2 * i2 + ((j + k + ipass) & 1);
                    const int o = (kl * n + j) * n + i;
                    const double uc = sm()[u + o];
                    const double resh2 = lap<LN>(x, u, i, j, kl, uc) - h2 * sm()[rhs + o];
                    sm()[u + o] = uc + (1.0 / 6.0) * resh2;
                    const double a = fabs(resh2);
                    rm = a > rm ? a : rm;
                }
            }
            sync<LN>();
        }
        return rm;
    }
    // residual of one cell (mg_poisson.F90:5-28)
    template <int LN>
    static __device__ __forceinline__ double resid(const Ctx &x, int u, int rhs, int i, int j, int kl) {
        constexpr int n = 1 << LN;
        const int o = (kl * n + j) * n + i;
        const double l = lap<LN>(x, u, i, j, kl, sm()[u + o]);
        return -x.t->h2i[LN] * l + sm()[rhs + o];
    }
    // fn(i, j, kl) summed over the eight children of coarse cell (i, j, kl) in rstrct_linear's order
    template <class F>
    static __device__ __forceinline__ double rstrct(F &&fn, int i, int j, int k) {
        double s = fn(2 * i, 2 * j, 2 * k) + fn(2 * i + 1, 2 * j, 2 * k);
        s = s + fn(2 * i, 2 * j + 1, 2 * k);
        s = s + fn(2 * i, 2 * j, 2 * k + 1);
        s = s + fn(2 * i + 1, 2 * j + 1, 2 * k);
        s = s + fn(2 * i + 1, 2 * j, 2 * k + 1);
        s = s + fn(2 * i, 2 * j + 1, 2 * k + 1);
        s = s + fn(2 * i + 1, 2 * j + 1, 2 * k + 1);
        return s * (1.0 / 8.0);
    }
    // over the coarse cells under this team's part of level LN: fine planes
    // 2 kc, 2 kc + 1 are in one CTA, the coarse one where its level keeps it
    template <int LN, class F>
    static __device__ __forceinline__ void to_coarse(const Ctx &x, int dst, int zero, F &&fn) {
        constexpr int nc = 1 << (LN - 1), PC = planes(LN) / 2;
        for (int c = threadIdx.x; c < nc * nc * PC; c += team_size<LN>()) {
            const int i = c & (nc - 1), j = (c >> (LN - 1)) & (nc - 1), kl = c >> (2 * (LN - 1));
            const double v = rstrct(fn, i, j, kl);
            if constexpr (wide(LN) && !wide(LN - 1)) {   // the small level lives on CTA 0
                double *b = mg_map_rank(sm(), 0);
                const int o = c + x.rank * (nc * nc * PC);
                b[dst + o] = v;
                if (zero >= 0) b[zero + o] = 0.0;
            } else {
                sm()[dst + c] = v;
                if (zero >= 0) sm()[zero + c] = 0.0;
            }
        }
        sync<LN>();
    }
    // prolongation of level LN - 1 onto level LN: stored, or added
    template <int LN>
    static __device__ __forceinline__ void interp(const Ctx &x, bool cubic) {
        constexpr int n = 1 << LN, P = planes(LN), LC = LN - 1;
        constexpr bool REM = wide(LN) && !wide(LC);   // the coarse level is CTA 0's
        for (int c = threadIdx.x; c < n * n * P; c += team_size<LN>()) {
            const int i = c & (n - 1), j = (c >> LN) & (n - 1), kl = c >> (2 * LN);
            const int k = kl + (wide(LN) ? x.rank * P : 0);
            auto B = [&](int a, int b, int d) { return beyond<LC, REM>(x, U(LC), a, b, d); };
            double v;
            if (cubic && LN >= 2) {
                const int *ci = x.t->c[n + i], *cj = x.t->c[n + j], *ck = x.t->c[n + k];
                const double *wi = x.t->w[n + i], *wj = x.t->w[n + j], *wk = x.t->w[n + k];
                double bxy[4];
#pragma unroll 1
                for (int mk = 0; mk < 4; mk++) {
                    double bx[4];
#pragma unroll
                    for (int mj = 0; mj < 4; mj++)
                        bx[mj] = wi[0] * B(ci[0], cj[mj], ck[mk]) + wi[1] * B(ci[1], cj[mj], ck[mk]) +
                                 wi[2] * B(ci[2], cj[mj], ck[mk]) + wi[3] * B(ci[3], cj[mj], ck[mk]);
                    const double t = wj[0] * bx[0] + wj[1] * bx[1] + wj[2] * bx[2] + wj[3] * bx[3];
                    if (mk == 0) bxy[0] = t;
                    else if (mk == 1) bxy[1] = t;
                    else if (mk == 2) bxy[2] = t;
                    else bxy[3] = t;
                }
                v = wk[0] * bxy[0] + wk[1] * bxy[1] + wk[2] * bxy[2] + wk[3] * bxy[3];
            } else {   // trilinear_cell
                const int ic = i / 2, jc = j / 2, kc = k / 2;
                const int ic1 = ic + 2 * (i & 1) - 1, jc1 = jc + 2 * (j & 1) - 1, kc1 = kc + 2 * (k & 1) - 1;
                v = (27.0 * B(ic, jc, kc) + 9.0 * (B(ic1, jc, kc) + B(ic, jc1, kc) + B(ic, jc, kc1)) +
                     3.0 * (B(ic, jc1, kc1) + B(ic1, jc, kc1) + B(ic1, jc1, kc)) + B(ic1, jc1, kc1)) / 64.0;
            }
            sm()[U(LN) + c] = cubic ? v : sm()[U(LN) + c] + v;
        }
        sync<LN>();
    }
    // runs fn on the team of level LN - 1 from code the team of level LN runs
    template <int LN, class F>
    static __device__ __forceinline__ void on_coarser(const Ctx &x, F &&fn) {
        if constexpr (wide(LN) && !wide(LN - 1)) {
            if (x.rank == 0) fn();
            mg_cluster_sync();
        } else if constexpr (LN == 3) {
            if (threadIdx.x < 32) fn();
            __syncthreads();
        } else {
            fn();
        }
    }
    // the V-cycle from level LN (mg.F90:170-215): right-hand side RHO where it
    // starts, RHS below; returns this thread's max |resh2| of the last sweep
    template <int LN, bool FIRST>
    static __device__ __noinline__ double vcycle(const Ctx x) {
        constexpr int rhs = FIRST ? RHO(LN) : RHS(LN);
        double rm = 0.0;
#pragma unroll 1
        for (int q = 0; q < 2; q++) rm = relax<LN>(x, rhs);
        if constexpr (LN > 0) {
            to_coarse<LN>(x, RHS(LN - 1), U(LN - 1),
                          [&](int i, int j, int kl) { return resid<LN>(x, U(LN), rhs, i, j, kl); });
            on_coarser<LN>(x, [&] { vcycle<LN - 1, false>(x); });
            interp<LN>(x, false);
#pragma unroll 1
            for (int q = 0; q < 2; q++) rm = relax<LN>(x, rhs);
        }
        return rm;
    }
    // the FMG up to level LN (mg.F90:106-218)
    template <int LN>
    static __device__ __forceinline__ double fmg(const Ctx &x) {
        if constexpr (LN == 0) {
            if (threadIdx.x == 0) sm()[U(0)] = 0.0;
            __syncwarp();
            return vcycle<0, true>(x);
        } else {
            on_coarser<LN>(x, [&] { fmg<LN - 1>(x); });
            interp<LN>(x, true);
            double rm = 0.0;
#pragma unroll 1
            for (int jc = 0; jc < 2; jc++) rm = vcycle<LN, true>(x);
            return rm;
        }
    }
    // RHO of every coarser level
    template <int LN>
    static __device__ __forceinline__ void rstrct_rho(const Ctx &x) {
        if constexpr (LN > 0) {
            constexpr int n = 1 << LN;
            to_coarse<LN>(x, RHO(LN - 1), -1, [&](int i, int j, int kl) { return sm()[RHO(LN) + (kl * n + j) * n + i]; });
            on_coarser<LN>(x, [&] { rstrct_rho<LN - 1>(x); });
        }
    }
};

// mg_cycle (mg.F90:42-94) on the base blocks of u and rhs: gather
// (mg_data.F90:179-253), corrections, and the potential back into u.
template <class T, int TOP, int C, int MODE>
__global__ void __launch_bounds__(512, 1) k_mgs_cycle(T *__restrict__ ub, const T *__restrict__ rhsb, MgsArgs a) {
    pdl_enter();
    using M = Mgs<TOP, C, MODE>;
    double *const mgs_smem = M::sm();
    __shared__ typename M::Tables tab;
    __shared__ double red[32], slot;
    constexpr int N = 1 << TOP, P = M::planes(TOP), VOL = M::vol(TOP);
    const int tid = threadIdx.x, rank = C > 1 ? mg_cluster_rank() : 0;
    const typename M::Ctx x{&tab, rank};
    M::fill_tables(tab, a.hbase);
    auto cell = [&](int c) -> int64_t {   // the block cell of this CTA's base cell c
        const int I = c & (N - 1), J = (c >> TOP) & (N - 1), K = (c >> (2 * TOP)) + rank * P;
        const int ib = I / a.n, jb = J / a.n, kb = K / a.n;
        return (int64_t)a.baseIdx[(kb * a.ngb + jb) * a.ngb + ib] * a.V + cidx(a.G, I - ib * a.n, J - jb * a.n, K - kb * a.n);
    };
    for (int c = tid; c < VOL; c += 512) {
        const int64_t b = cell(c);
        mgs_smem[M::SRC + c] = (double)rhsb[b];
        mgs_smem[M::PSI + c] = (double)ub[b];
    }
    M::meet();
    const double errmax = (double)1.e-2f;   // default-real literal (mg.F90:50)
    double rhomax = 0.0;
    for (int it = 1; it <= a.nmax; it++) {
        const double v = M::defect(x);
        M::meet();
        if (it == 1) rhomax = M::vmax(v, red, &slot);
        const double rm = M::correct(x);
        const double hh = a.hbase;
        const double res = M::vmax(rm, red, &slot) / (hh * hh);   // PSI is complete after it
        if (res / rhomax < errmax) break;
    }
    for (int c = tid; c < VOL; c += 512) ub[cell(c)] = (T)mgs_smem[M::PSI + c];
    if (C > 1) mg_cluster_sync();   // no CTA leaves while another may still read its shared memory
}

}  // namespace sfm
