// sfm_link.cu -- the block links of an AMR hierarchy built on the device.
//
// After each refinement the reference derives every new block's links from
// its parent's: ParentGid, ChildGid(lri,lrj,lrk) and NeighborGid(lr,dir),
// the neighbours being children of the parent or of the parent's neighbours
// (update_neighbor, update_neighbor_linklist, update_parent_linklist;
// grid.F90:587-731), and fmg_make_linklist copies them into the solver's
// structure (fmg_data_if.F90:298-411).  sfm_link_blocks computes the same
// links from the blocks' levels and integer positions alone, so a hierarchy
// regridded on the device needs no round trip through the host: one hash
// table keyed by (level, i, j, k) in device memory, one lookup per parent
// and neighbour; the children are the inverse of the parents.
//
//   parent    the block at level L - 1 holding (i/2, j/2, k/2)
//   child c   the block at level L + 1 at (2i + c&1, 2j + (c>>1)&1, 2k + (c>>2)&1)
//   nbr f     f = lr + 2 dir: the block at level L one step left (lr = 0) or
//             right along dir; a periodic direction wraps at the level's
//             extent ngb[dir] << L, another one gives -1 and touch = 1 there
//
// The table is open-addressed (linear probing, twice as many slots as
// blocks, so every probe sequence ends at an empty slot within the table);
// the result does not depend on insertion order.  A duplicated block, a
// block above the base level without a parent, or a block with some but
// not all of its 8 children is reported as SFM_EHIER.
#include <cuda_runtime.h>
#include <stdint.h>

#include <condition_variable>
#include <mutex>

#include "../../include/sfmg.h"

namespace {

constexpr int kCoordBits = 20;   // i, j, k < 2^20 on every level
constexpr int kMaxLevels = 16;   // level < 2^4 above the three coordinates
constexpr int32_t kEmpty = -1;   // a free slot

// A slot holds a block's index; its key is the block's own level and
// position, so the table is 4 bytes a slot and one fill clears it.
struct LinkTable {
    int32_t *slot;
    const int32_t *level, *ijk;
    uint64_t mask;   // slots - 1 (slots a power of two)
};

__host__ __device__ __forceinline__ uint64_t link_key(int L, int64_t i, int64_t j, int64_t k) {
    return ((uint64_t)L << (3 * kCoordBits)) | ((uint64_t)k << (2 * kCoordBits)) | ((uint64_t)j << kCoordBits) |
           (uint64_t)i;
}
__device__ __forceinline__ uint64_t link_hash(uint64_t x) {   // 64-bit finaliser (murmur3 fmix64)
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdULL;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ULL;
    x ^= x >> 33;
    return x;
}
__device__ __forceinline__ bool link_is(const LinkTable &t, int32_t b, int L, int64_t i, int64_t j, int64_t k) {
    return t.level[b] == L && t.ijk[3 * (int64_t)b] == i && t.ijk[3 * (int64_t)b + 1] == j && t.ijk[3 * (int64_t)b + 2] == k;
}

__global__ void k_link_insert(LinkTable t, int nb, int nlev, int3 ngb, int *err) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
        const int L = t.level[b];
        const int64_t i = t.ijk[3 * (int64_t)b], j = t.ijk[3 * (int64_t)b + 1], k = t.ijk[3 * (int64_t)b + 2];
        if (L < 0 || L >= nlev || i < 0 || j < 0 || k < 0 || i >= ((int64_t)ngb.x << L) ||
            j >= ((int64_t)ngb.y << L) || k >= ((int64_t)ngb.z << L)) {   // outside its level's box
            atomicExch(err, 1);
            continue;
        }
        uint64_t s = link_hash(link_key(L, i, j, k)) & t.mask;
        for (uint64_t probe = 0; probe <= t.mask; probe++, s = (s + 1) & t.mask) {
            const int32_t prev = atomicCAS(t.slot + s, kEmpty, b);
            if (prev == kEmpty) break;
            if (link_is(t, prev, L, i, j, k)) {   // the same block twice
                atomicExch(err, 1);
                break;
            }
        }
    }
}

// the block at (L, i, j, k), or -1; the table was filled by a completed launch
__device__ int32_t link_find(const LinkTable &t, int L, int64_t i, int64_t j, int64_t k) {
    uint64_t s = link_hash(link_key(L, i, j, k)) & t.mask;
    for (uint64_t probe = 0; probe <= t.mask; probe++, s = (s + 1) & t.mask) {
        const int32_t v = t.slot[s];
        if (v == kEmpty) return -1;
        if (link_is(t, v, L, i, j, k)) return v;
    }
    return -1;
}

// Eight lanes per block, a link each (6 neighbours, the parent): a lookup is
// a chain of two or three dependent loads, which the lanes wait for together.
__global__ void __launch_bounds__(256) k_link_lookup(LinkTable t, int nb, int nlev, int3 ngb, int3 per, int32_t *parent,
                                                     int32_t *nbr, int8_t *touch, int *err) {
    const int w = threadIdx.x & 7;
    for (int64_t b = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 3; b < nb; b += (int64_t)gridDim.x * 32) {
        const int L = t.level[b];
        const int64_t q[3] = {t.ijk[3 * b], t.ijk[3 * b + 1], t.ijk[3 * b + 2]};
        if (L < 0 || L >= nlev) continue;   // reported by k_link_insert
        if (w < 6) {
            const int dir = w >> 1;
            const int64_t ext = (int64_t)(dir == 0 ? ngb.x : (dir == 1 ? ngb.y : ngb.z)) << L;
            const bool pd = (dir == 0 ? per.x : (dir == 1 ? per.y : per.z)) != 0;
            int64_t r = (dir == 0 ? q[0] : (dir == 1 ? q[1] : q[2])) + ((w & 1) ? 1 : -1);
            const bool out = r < 0 || r >= ext;
            if (out && pd) r = (r + ext) % ext;
            int32_t n = -1;
            if (!out || pd) n = link_find(t, L, dir == 0 ? r : q[0], dir == 1 ? r : q[1], dir == 2 ? r : q[2]);
            nbr[6 * b + w] = n;
            touch[6 * b + w] = (int8_t)(out && !pd);
        } else if (w == 6) {
            int32_t p = -1;
            if (L > 0) {
                p = link_find(t, L - 1, q[0] >> 1, q[1] >> 1, q[2] >> 1);
                if (p < 0) atomicExch(err, 1);
            }
            parent[b] = p;
        }
    }
}

// every block into its parent's list (child filled with -1 before)
__global__ void k_link_children(int nb, int nlev, const int32_t *level, const int32_t *ijk, const int32_t *parent,
                                int32_t *child) {
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += (int64_t)gridDim.x * blockDim.x) {
        const int L = level[b];
        if (L < 1 || L >= nlev) continue;
        const int32_t p = parent[b];
        if (p >= 0) child[8 * (int64_t)p + (ijk[3 * b] & 1) + 2 * (ijk[3 * b + 1] & 1) + 4 * (ijk[3 * b + 2] & 1)] = (int32_t)b;
    }
}

// a block has all of its 8 children or none
__global__ void k_link_check(int nb, const int32_t *child, int *err) {
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += (int64_t)gridDim.x * blockDim.x) {
        int found = 0;
        for (int c = 0; c < 8; c++) found += child[8 * b + c] >= 0;
        if (found != 0 && found != 8) atomicExch(err, 1);
    }
}

// Error words: a call owns one from its first launch until it has waited for
// its stream, so calls on several threads and streams never share one.
constexpr int kErrWords = 64;
__device__ int g_link_err[kErrWords];
std::mutex g_link_mu;
std::condition_variable g_link_cv;
uint64_t g_link_busy = 0;
struct ErrWord {
    int at = 0;
    ErrWord() {
        std::unique_lock<std::mutex> lk(g_link_mu);
        g_link_cv.wait(lk, [] { return g_link_busy != ~(uint64_t)0; });
        while (g_link_busy >> at & 1) at++;
        g_link_busy |= (uint64_t)1 << at;
    }
    ~ErrWord() {
        {
            std::lock_guard<std::mutex> lk(g_link_mu);
            g_link_busy &= ~((uint64_t)1 << at);
        }
        g_link_cv.notify_one();
    }
};

bool on_device(const void *p, int dev) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) && a.device == dev;
}

}  // namespace

extern "C" int sfm_link_blocks(int32_t nblocks, int32_t nlev, const int32_t *d_level, const int32_t *d_ijk,
                               const int32_t ngb[3], const int32_t periodic[3], int32_t *d_parent,
                               int32_t *d_child, int32_t *d_nbr, int8_t *d_touch, void *stream) {
    if (nblocks <= 0 || nlev <= 0 || nlev > kMaxLevels || !d_level || !d_ijk || !ngb || !periodic || !d_parent ||
        !d_child || !d_nbr || !d_touch)
        return SFM_EINVAL;
    for (int d = 0; d < 3; d++)
        if (ngb[d] <= 0 || ((int64_t)ngb[d] << (nlev - 1)) > ((int64_t)1 << kCoordBits)) return SFM_EINVAL;
    int dev = 0, ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
        cudaGetLastError();
        return SFM_EDEVICE;
    }
    if (cudaGetDevice(&dev) != cudaSuccess) return SFM_ECUDA;
    for (const void *p : {(const void *)d_level, (const void *)d_ijk, (const void *)d_parent, (const void *)d_child,
                          (const void *)d_nbr, (const void *)d_touch})
        if (!on_device(p, dev)) return SFM_EINVAL;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) return SFM_EINVAL;
    if (cap != cudaStreamCaptureStatusNone) return SFM_EINVAL;   // the call waits for the stream
    uint64_t slots = 1;
    while (slots < 2 * (uint64_t)nblocks) slots <<= 1;
    // The table lies in d_child (8 ints per block, the table at most 4) until
    // the children are written, so that the call allocates nothing: a stream
    // pool gives its memory back at every synchronisation, and mapping it
    // anew was 420 of a call's 520 us (133,856 blocks; 100 us without).
    const LinkTable t{d_child, d_level, d_ijk, slots - 1};
    const ErrWord word;
    int *err = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void **>(&err), g_link_err) != cudaSuccess) {
        cudaGetLastError();
        return SFM_ECUDA;
    }
    err += word.at;
    int herr = 1;
    cudaMemsetAsync(err, 0, sizeof(int), s);
    cudaMemsetAsync(d_child, 0xff, slots * sizeof(int32_t), s);
    const int3 box = make_int3(ngb[0], ngb[1], ngb[2]);
    const unsigned full = 148 * 8;
    auto ctas = [&](int64_t threads) { return (unsigned)((threads + 255) / 256 < full ? (threads + 255) / 256 : full); };
    k_link_insert<<<ctas(nblocks), 256, 0, s>>>(t, nblocks, nlev, box, err);
    k_link_lookup<<<ctas(8 * (int64_t)nblocks), 256, 0, s>>>(t, nblocks, nlev, box,
                                                             make_int3(periodic[0] != 0, periodic[1] != 0, periodic[2] != 0),
                                                             d_parent, d_nbr, d_touch, err);
    cudaMemsetAsync(d_child, 0xff, 8 * (size_t)nblocks * sizeof(int32_t), s);
    k_link_children<<<ctas(nblocks), 256, 0, s>>>(nblocks, nlev, d_level, d_ijk, d_parent, d_child);
    k_link_check<<<ctas(nblocks), 256, 0, s>>>(nblocks, d_child, err);
    const cudaError_t launched = cudaGetLastError();
    cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s);
    // the wait comes first: what was queued still writes the error word and the caller's arrays
    const cudaError_t ran = cudaStreamSynchronize(s);
    if (launched != cudaSuccess || ran != cudaSuccess) return SFM_ECUDA;
    return herr == 0 ? SFM_OK : SFM_EHIER;
}
