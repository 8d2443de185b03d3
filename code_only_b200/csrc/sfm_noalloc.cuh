// sfm_noalloc.cuh -- a uniform periodic base-grid solve that allocates
// nothing (exported as sfm_uniform_solve_noalloc).
//
// Some callers cannot allocate device memory at the point where they need a
// solve: code running inside a fixed memory pool or an arena handed out at
// start-up, a real-time step whose allocator calls would synchronise the
// device, or a host library that has promised its user a fixed device
// footprint.  For them this entry point runs the base-grid multigrid
// (mg_lin as repeated defect corrections, mg.F90:42-94) on the caller's
// device buffers, with every working array in shared memory (sfm_mgs.cuh):
// one CTA up to 16^3 cells, a cluster of 8 CTAs for 32^3.  Nothing is
// allocated: no cudaMalloc, no cudaFree, no allocating library call.  The
// only set-up is, once per device, the lookup of the two result words'
// address and the kernels' shared-memory opt-in.
//
// Limits and contract:
//   - n (cells per edge) is a power of two, 2 <= n <= SFM_NOALLOC_MAX_N (32);
//   - no state carries over from one call to the next;
//   - the two result words (residual, cycle count) are one pair per device
//     and loaded library, written only by calls that ask for host outputs: of
//     two such calls on the same device whose executions overlap, the host
//     outputs and the status of either may be the other's.  Order calls that
//     ask for host outputs on one stream or with events;
//   - the first call on each device does the set-up; make that first call
//     before any stream capture on that device.
//
// Bound by the serial chain of colour sweeps and transfers (about 400
// dependent steps a cycle).  n = 32, rel_tol 1e-10: 2.1 ms with the level
// arrays in global memory on one CTA of 1024 threads, 0.55 ms here.
#pragma once
#include "sfm_mgs.cuh"

namespace sfm {

constexpr int NOALLOC_MAX_N = 32;
static __device__ double g_noalloc_out[2];   // relative residual and cycle count

template <int TOP>
__host__ __device__ constexpr int noalloc_ctas() { return TOP >= 5 ? 8 : 1; }

// rho and psi are dense n^3 arrays, x fastest, n = 2^TOP.  Solves
// lap(psi) = four_pi_G * (rho - mean rho) on the periodic grid of cell width
// h: psi starts at zero; each cycle forms the residual (mg_poisson.F90:5-28),
// solves for the correction with mg_lin and adds it (mg.F90:62-90), until
// max|residual| <= rel_tol * max|four_pi_G (rho - mean)| or max_cycles.
// out: the result words, or null where the call asks for none.
template <int TOP>
__global__ void __launch_bounds__(512, 1) k_mgs_uniform_noalloc(const double *__restrict__ rho, double *__restrict__ psi,
                                                                double h, double four_pi_G, double rel_tol,
                                                                int max_cycles, double *out) {
    constexpr int C = noalloc_ctas<TOP>();
    using M = Mgs<TOP, C, kMgPeriodic>;
    __shared__ typename M::Tables tab;
    __shared__ double red[32], slot, wsum[32];
    constexpr int N3 = 1 << (3 * TOP), VOL = M::vol(TOP);
    double *const sm = M::sm();
    const int tid = threadIdx.x, rank = C > 1 ? mg_cluster_rank() : 0, first = rank * VOL;
    const typename M::Ctx x{&tab, rank};
    M::fill_tables(tab, h);
    // Mean of rho, in every CTA (rho is at most 256 KB, from L2): 1024 partial
    // sums in cell order, two per thread, then a fixed tree over each 32 and
    // the 32 results in order.
    //
    // A NaN or Inf density would make the mean and every source value NaN;
    // max|source| would then stay 0 (NaN fails every comparison) and the
    // loop would stop at once with psi = 0 reported as converged.  Refuse
    // it instead: psi is set to NaN everywhere and the result words carry a
    // cycle count of -1, which the host turns into SFM_ENONFINITE.
    int bad = 0;
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
        double s = 0.0;
        for (int c = tid + 512 * half; c < N3; c += 1024) {
            const double v = rho[c];
            bad |= !isfinite(v);
            s = s + v;
        }
        for (int o = 16; o > 0; o >>= 1) s = s + __shfl_down_sync(0xffffffffu, s, o);
        if ((tid & 31) == 0) wsum[16 * half + (tid >> 5)] = s;
    }
    if (__syncthreads_or(bad)) {
        for (int c = tid; c < VOL; c += 512) psi[first + c] = __longlong_as_double(0x7ff8000000000000LL);
        if (out && rank == 0 && tid == 0) {
            out[0] = __longlong_as_double(0x7ff8000000000000LL);
            out[1] = -1.0;
        }
        return;
    }
    double tot = 0.0;
    for (int w = 0; w < 32; w++) tot = tot + wsum[w];
    const double mean = tot / (double)N3;
    double smax = 0.0;
    for (int c = tid; c < VOL; c += 512) {
        const double v = four_pi_G * (rho[first + c] - mean);
        sm[M::SRC + c] = v;
        sm[M::PSI + c] = 0.0;
        const double a = fabs(v);
        smax = a > smax ? a : smax;
    }
    M::meet();   // every CTA has started before any reads another's shared memory
    smax = M::vmax(smax, red, &slot);
    int it = 0;
    double rrel = 0.0;
    for (;;) {
        const double rmax = M::vmax(M::defect(x), red, &slot);
        rrel = smax > 0.0 ? rmax / smax : 0.0;
        if (rrel <= rel_tol || it >= max_cycles) break;
        M::correct(x);
        M::meet();
        it++;
    }
    for (int c = tid; c < VOL; c += 512) psi[first + c] = sm[M::PSI + c];
    if (out && rank == 0 && tid == 0) {
        out[0] = rrel;
        out[1] = (double)it;
    }
}

// go(kernel, CTAs of the cluster, shared bytes) for n = 2^top
template <class F>
inline void noalloc_with(int top, F &&go) {
    auto one = [&](auto t) {
        constexpr int TOP = decltype(t)::value, C = noalloc_ctas<TOP>();
        go(k_mgs_uniform_noalloc<TOP>, C, (int)(Mgs<TOP, C, kMgPeriodic>::total() * sizeof(double)));
    };
    switch (top) {
        case 1: one(std::integral_constant<int, 1>{}); break;
        case 2: one(std::integral_constant<int, 2>{}); break;
        case 3: one(std::integral_constant<int, 3>{}); break;
        case 4: one(std::integral_constant<int, 4>{}); break;
        default: one(std::integral_constant<int, 5>{}); break;
    }
}

}  // namespace sfm
