/*
 * LOQUAT-B200 neighbour grid (replaces the closed LoquatGrid of the
 * reference, src/loquat_grid.h:28-66).
 *
 * A stable counting sort by cell key instead of a full radix sort: the key
 * range is the cell count, so one histogram + one scan place every particle.
 *   1. k_hash_count  key per particle, warp-aggregated atomic count per cell,
 *                    the atomic's return value is the particle's rank
 *   2. scan          exclusive sum of the counts -> cell start table
 *   3. k_scatter     slot = start[key] + rank
 *   4. k_cell_order  ranks from atomics are not ordered across warps, so each
 *                    cell's slot range is put back in ascending previous-slot
 *                    order; the result equals a stable sort by key, bit for
 *                    bit.  The same pass writes what follows from the order:
 *                    the sorted keys, the per-cell begin/end (-1 when empty)
 *                    for callers of the reference interface (the native
 *                    driver reads the start table directly) and the slots'
 *                    particle identities.
 * HBM traffic per particle: 16 B position read, 8 B key+rank written and read
 * back, 8 B sorted outputs; plus 12 B per cell for count, start and bounds.
 */
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <unordered_map>
#include <utility>

#include <cooperative_groups.h>
#include <cub/device/device_scan.cuh>

#include "lq_internal.cuh"
#include "lq_device.cuh"
#include <loquat_grid.h>

namespace lqb {

namespace {

constexpr int kBlock = 256;

inline int blocks_for(long long n, int b = kBlock) { return (int)((n + b - 1) / b); }

__global__ void __launch_bounds__(kBlock) k_hash_count(const Parameters* __restrict__ P, int np, int npb,
                                                       const float4* __restrict__ pos, int* __restrict__ key,
                                                       int* __restrict__ rank, int* __restrict__ count,
                                                       int* __restrict__ health, const float4* __restrict__ idep,
                                                       Frames fr)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = i < np;
    int k = 0;
    if (active) {
        const float ih = __ldg(&P->i_h);
        const int nx = __ldg(&P->cell_num_x), ny = __ldg(&P->cell_num_y), nz = __ldg(&P->cell_num_z);
        const float4 p = __ldg(pos + i);
        int cy = cell_axis(p.y, ih, ny);
        if (fr.rows) {
            /* local cell, then the object's row block */
            const float s = floorf(0.5f * p.y * ih);
            const int local = (s >= 0.0f && s < 1.0e9f) ? (int)s : -1;
            cy = local < 0 ? -1 : frame_row(fr, __ldg(&idep[i].x), local);
        }
        const int cx = cell_axis(p.x, ih, nx), cz = cell_axis(p.z, ih, nz);
        if (cx < 0 || cy < 0 || cz < 0) {
            k = __ldg(&P->ncell_delete);
            if (health) atomicAdd(health + (i < npb ? HEALTH_BND_OUT : HEALTH_MAT_OUT), 1);
        } else {
            k = (i < npb ? 0 : __ldg(&P->ncell_one_layer)) + (cx * ny + cy) * nz + cz;
        }
    }
    const unsigned act = __ballot_sync(0xffffffffu, active);
    if (!active) return;
    const unsigned peers = __match_any_sync(act, k);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(count + k, __popc(peers));
    base = __shfl_sync(peers, base, leader);
    key[i] = k;
    rank[i] = base + __popc(peers & ((1u << lane) - 1u));
}

__global__ void __launch_bounds__(kBlock) k_fill_int(int* __restrict__ p, int n, int v)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

__global__ void k_add_int(int* __restrict__ p, int v) { *p += v; }

__global__ void __launch_bounds__(kBlock) k_scatter(int np, const int* __restrict__ key, const int* __restrict__ rank,
                                                    const int* __restrict__ start, int* __restrict__ part_idx)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    const int d = __ldg(start + key[i]) + rank[i];
    if (lq_in_range(d, np)) part_idx[d] = i;
}

/* What a search writes of its order besides part_idx: the sorted keys, the
 * per-cell bounds and the identities of the slots' particles (each may be
 * null; ident_out[slot] = ident_in[previous slot], or the previous slot
 * itself without ident_in: identities that start here). */
struct OrderOutputs {
    int* part_cel;
    int* beg;
    int* end;
    const int* ident_in;
    int* ident_out;
};

/* A warp orders kCells cells: lanes load the cells' slots (the next ones'
 * meanwhile), a vote tells whether they are in order, and if not each lane
 * finds its particle's place by counting the smaller ones.  The lanes that a
 * cell gets follow the fullest of the warp's cells: with up to 16 particles
 * each, 4, 8 or 16, so two to eight cells at a time; else all 32, and a cell
 * of up to 128 in four loads.  A cell of more is ordered by its own lane,
 * beside the warp's other such cells.  Bound by the chain of cells; a search
 * over 2.3 M particles, 18 a cell, a few percent of which changed theirs, takes
 * 84 us, of which bounds and identities (23 us as kernels of their own) are
 * written here.
 *
 * Measured against one thread per cell that inserts (and against one cell at a
 * time whatever its size), us a search over 2.0 M particles with 0.9, 1.9, 3.8,
 * 16 and 128 a cell on average: 121, 82, 64, 54, 712; one thread per cell 125,
 * 89, 74, 91, 1030; one cell at a time 182, 131, 88, 54, 2739. */
template <int kCells>
__global__ void __launch_bounds__(kBlock) k_cell_order(int ncell, int np, const int* __restrict__ start, int* part_idx,
                                                       OrderOutputs out)
{
    __shared__ unsigned char full[kBlock / 32][32];     /* the warp's cells that hold particles */
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int first = (blockIdx.x * kBlock + threadIdx.x) / 32 * kCells;
    const int c = first + lane;
    int s = 0, n = 0;
    if (lane < kCells && c < ncell) {
        s = __ldg(start + c);
        n = __ldg(start + c + 1) - s;
        if (out.beg) {
            out.beg[c] = n > 0 ? s : -1;
            out.end[c] = n > 0 ? s + n : -1;
        }
    }
    auto place = [&](int d, int v, int cell) {      /* slot d holds previous slot v's particle */
        if (out.part_cel) out.part_cel[d] = cell;
        if (out.ident_out) out.ident_out[d] = !lq_in_range(v, np) ? -1 : out.ident_in ? __ldg(out.ident_in + v) : v;
    };
    unsigned todo = __ballot_sync(FULL, n > 0);
    unsigned big = 0;
    if (!__any_sync(FULL, n > 16)) {
        if (n > 0) full[w][__popc(todo & ((1u << lane) - 1u))] = (unsigned char)lane;
        __syncwarp();
        const int cells = __popc(todo);
        const int most = __reduce_max_sync(FULL, n);
        const int W = most <= 4 ? 4 : most <= 8 ? 8 : 16;
        const int sub = lane & (W - 1), per = 32 / W;
        int q = lane / W, at = 0, cs = 0, cn = 0, v = INT_MAX;
        auto take = [&]() {
            at = q < cells ? full[w][q] : 0;
            cs = __shfl_sync(FULL, s, at);
            cn = __shfl_sync(FULL, n, at);
            if (q >= cells) cn = 0;
            v = sub < cn ? part_idx[cs + sub] : INT_MAX;
            q += per;
        };
        take();
        for (int base = 0; base < cells; base += per) {
            const int at0 = at, cs0 = cs, cn0 = cn, v0 = v;
            take();
            const int after = __shfl_down_sync(FULL, v0, 1, W);
            int r = sub;
            if (__any_sync(FULL, sub + 1 < cn0 && v0 > after)) {
                r = 0;
                for (int o = 0; o < W; ++o) r += __shfl_sync(FULL, v0, o, W) < v0;
                if (sub < cn0) part_idx[cs0 + r] = v0;
            }
            if (sub < cn0) place(cs0 + r, v0, first + at0);
        }
    } else {
        big = __ballot_sync(FULL, n > 128);
        todo &= ~big;
        int k = __ffs((int)todo) - 1;
        int cs = __shfl_sync(FULL, s, k & 31), cn = __shfl_sync(FULL, n, k & 31);
        int v = todo && lane < cn ? part_idx[cs + lane] : INT_MAX;
        while (todo) {
            todo &= todo - 1;
            const int k2 = __ffs((int)todo) - 1;
            const int s2 = __shfl_sync(FULL, s, k2 & 31), n2 = __shfl_sync(FULL, n, k2 & 31);
            const int v2 = todo && lane < n2 ? part_idx[s2 + lane] : INT_MAX;
            const int cell = first + k;
            if (cn <= 32) {
                const int after = __shfl_down_sync(FULL, v, 1);
                int r = lane;
                if (__any_sync(FULL, lane + 1 < cn && v > after)) {
                    r = 0;
                    for (int o = 0; o < cn; ++o) r += __shfl_sync(FULL, v, o) < v;
                    if (lane < cn) part_idx[cs + r] = v;
                }
                if (lane < cn) place(cs + r, v, cell);
            } else {
                int u4[4], r[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    u4[u] = 32 * u + lane < cn ? part_idx[cs + 32 * u + lane] : INT_MAX;
                    r[u] = 0;
                }
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    for (int o = 0; o < 32; ++o) {
                        const int x = __shfl_sync(FULL, u4[b], o);
#pragma unroll
                        for (int u = 0; u < 4; ++u) r[u] += x < u4[u];
                    }
                __syncwarp();
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (32 * u + lane < cn) {
                        part_idx[cs + r[u]] = u4[u];
                        place(cs + r[u], u4[u], cell);
                    }
            }
            k = k2;
            cs = s2;
            cn = n2;
            v = v2;
        }
    }
    if (!big) return;
    if (n > 128) {
        bool sorted = true;     /* most arrive in order: a read-only pass leaves them alone */
        for (int a = s + 1; a < s + n && sorted; ++a) sorted = part_idx[a - 1] < part_idx[a];
        for (int a = s + 1; a < s + n && !sorted; ++a) {
            const int x = part_idx[a];
            int b = a - 1;
            while (b >= s && part_idx[b] > x) {
                part_idx[b + 1] = part_idx[b];
                --b;
            }
            part_idx[b + 1] = x;
        }
    }
    __syncwarp();
    for (unsigned m = big; m; m &= m - 1) {
        const int k = __ffs((int)m) - 1, cs = __shfl_sync(FULL, s, k), cn = __shfl_sync(FULL, n, k);
        for (int d = cs + lane; d < cs + cn; d += 32) place(d, part_idx[d], first + k);
    }
}

__device__ __forceinline__ float4 element(const float4* p, int i) { return p[i]; }
__device__ __forceinline__ tensor2d element(const tensor2d* p, int i) { return load_t2_rw(p, i); }
__device__ __forceinline__ void put(float4* p, int i, const float4& v) { p[i] = v; }
__device__ __forceinline__ void put(tensor2d* p, int i, const tensor2d& v) { store_t2(p, i, v); }

/* One array permuted in place through its cache: gathered into the cache,
 * then copied back, where the cache is still in L2.  Each thread takes
 * kSortItems elements, a block's apart by its threads, with all loads issued
 * before the first store.
 *
 * Two plain launches: a sort goes on beside another stream's sorts and
 * beside a resident kernel of the caller's, where a cooperative launch
 * with a grid barrier waits until all its blocks fit on the device at once.
 * The copy is launched while the gather runs (its blocks come onto the
 * device once every block of the gather has, and then wait for the gather's
 * end), which takes the gap between the two out: 3.3 us a call in a graph
 * for 11 k to 150 k float4 elements, 16.2 for 2.3 M and 69 for 6.6 M
 * (tensor2d 35 and 104), where the cooperative launch took 3.7 to 5.1, 18.7
 * and 73 (37 and 112); called one by one 6.4 us against 6.1 below 150 k. */
constexpr int kSortItems = 4;

template <class T>
__device__ __forceinline__ void gather_items(int n, long long first, const int* idx, const T* data, T* cache)
{
    int j[kSortItems];
    T v[kSortItems];
#pragma unroll
    for (int u = 0; u < kSortItems; ++u) j[u] = first + u * kBlock < n ? __ldg(idx + first + u * kBlock) : -1;
#pragma unroll
    for (int u = 0; u < kSortItems; ++u)
        if (j[u] >= 0 && lq_in_range(j[u], n)) v[u] = element(data, j[u]);
#pragma unroll
    for (int u = 0; u < kSortItems; ++u)
        if (j[u] >= 0 && lq_in_range(j[u], n)) put(cache, (int)(first + u * kBlock), v[u]);
}

template <class W>
__device__ __forceinline__ void copy_items(long long words, long long first, const W* from, W* to)
{
    W v[kSortItems];
#pragma unroll
    for (int u = 0; u < kSortItems; ++u)
        if (first + u * kBlock < words) v[u] = from[first + u * kBlock];
#pragma unroll
    for (int u = 0; u < kSortItems; ++u)
        if (first + u * kBlock < words) to[first + u * kBlock] = v[u];
}

template <class T>
__global__ void __launch_bounds__(kBlock) k_sort_gather(int n, const int* __restrict__ idx, const T* data, T* cache)
{
    cudaTriggerProgrammaticLaunchCompletion();
    gather_items(n, (long long)blockIdx.x * (kSortItems * kBlock) + threadIdx.x, idx, data, cache);
}

template <class W>
__global__ void __launch_bounds__(kBlock) k_sort_copy_back(long long words, const W* from, W* to)
{
    cudaGridDependencySynchronize();
    copy_items(words, (long long)blockIdx.x * (kSortItems * kBlock) + threadIdx.x, from, to);
}

/* Few elements: both steps by one cluster of blocks in one launch, which
 * needs room for eight blocks in one part of the device only.  Up to the
 * elements that its threads take at once: 2.9 us a call in a graph for 4.5 k
 * float4 elements and 3.8 for tensor2d (3.0 and 3.3 with two launches), but
 * 5.7 us called one by one instead of 9.7, since a caller with so few
 * elements waits for the host; for 11 k tensor2d elements 5.7 us, 3.8 with two
 * launches. */
constexpr int kSortCluster = 8;
constexpr int kSortSmall = kSortCluster * kSortItems * kBlock;
template <class W, class T>
__global__ void __cluster_dims__(kSortCluster, 1, 1) __launch_bounds__(kBlock)
    k_sort_small(int n, const int* __restrict__ idx, T* data, T* cache)
{
    const int first = blockIdx.x * (kSortItems * kBlock) + threadIdx.x;
    gather_items(n, first, idx, data, cache);
    cooperative_groups::this_cluster().sync();
    const int words = n * (int)(sizeof(T) / sizeof(W));
    for (int at = first; at < words; at += kSortSmall)
        copy_items(words, at, reinterpret_cast<const W*>(cache), reinterpret_cast<W*>(data));
}

__global__ void __launch_bounds__(kBlock) k_gather_state(int n, const int* __restrict__ idx, State in, State out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int j = __ldg(idx + i);
    if (!lq_in_range(j, n)) return;
    out.pos[i] = __ldg(in.pos + j);
    out.vel[i] = __ldg(in.vel + j);
    out.idep[i] = __ldg(in.idep + j);
    store_t2(out.str, i, load_t2(in.str, j));
    store_t2(out.stn, i, load_t2(in.stn, j));
    if (in.xlo) {
        out.xlo[i] = in.xlo[j];
        out.vlo[i] = in.vlo[j];
    }
}

}  // namespace

int fill_int(int* p, int n, int v, cudaStream_t s)
{
    if (n <= 0) return LQ_OK;
    k_fill_int<<<blocks_for(n), kBlock, 0, s>>>(p, n, v);
    LQ_TRY_CUDA(cudaGetLastError(), "k_fill_int");
    return LQ_OK;
}

int add_int(int* p, int v, cudaStream_t s)
{
    k_add_int<<<1, 1, 0, s>>>(p, v);
    LQ_TRY_CUDA(cudaGetLastError(), "k_add_int");
    return LQ_OK;
}

int scan_scratch_bytes(int ncell, size_t* bytes)
{
    *bytes = 0;
    LQ_TRY_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, *bytes, (const int*)nullptr, (int*)nullptr, ncell + 1),
                "scan scratch query");
    return LQ_OK;
}

/* --------------------------------------------- identities of the grids */
namespace {

/* `started`: ident holds the identity of each of np slots.  Not so after a
 * search over another particle count, which does not follow the other slots'
 * particles: the next search over np particles then starts them again. */
struct IdentityRecord {
    int* ident = nullptr;
    int* tmp = nullptr;
    int np = 0;
    long long gen = 0;
    bool started = false;
};
std::mutex g_id_mu;
std::unordered_map<const int*, IdentityRecord> g_ids;
long long g_id_gen = 0;

/* The record that a search over np particles updates (null: none); the
 * caller holds g_id_mu. */
IdentityRecord* identity_for_search(const int* key, int np)
{
    auto it = g_ids.find(key);
    if (it == g_ids.end()) return nullptr;
    IdentityRecord& r = it->second;
    if (np == r.np) return np > 0 ? &r : nullptr;
    r.started = false;
    r.gen = ++g_id_gen;
    return nullptr;
}

}  // namespace

int grid_search(const Parameters* ph, const Parameters* pd, const float4* pos, GridBuffers& g, bool bounds,
                int* health, cudaStream_t s, const float4* idep, const Frames& fr, const int* identity_key)
{
    const int np = ph->np, npb = ph->npb, ncell = ph->ncell;
    if (np < 0 || npb < 0 || npb > np || ncell < 1)
        return set_error(LQ_ERR_ARG, "grid_search: bad sizes np=%d npb=%d ncell=%d", np, npb, ncell);
    if (np > g.np_cap || ncell > g.ncell_cap)
        return set_error(LQ_ERR_ARG, "grid_search: np=%d ncell=%d exceed grid capacity np=%d ncell=%d", np, ncell,
                         g.np_cap, g.ncell_cap);
    if (ph->ncell != 2 * ph->ncell_one_layer + 1 || ph->ncell_delete != ncell - 1)
        return set_error(LQ_ERR_ARG, "grid_search: Parameters cell counts are not initialised");
    LQ_TRY_CUDA(cudaMemsetAsync(g.count, 0, sizeof(int) * ((size_t)ncell + 1), s), "cell counts");
    if (np > 0) {
        if (fr.rows && !idep) return set_error(LQ_ERR_ARG, "grid_search: frames need the idep array");
        k_hash_count<<<blocks_for(np), kBlock, 0, s>>>(pd, np, npb, pos, g.key, g.rank, g.count, health, idep, fr);
        LQ_TRY_CUDA(cudaGetLastError(), "k_hash_count");
    }
    size_t bytes = g.scan_bytes;
    LQ_TRY_CUDA(cub::DeviceScan::ExclusiveSum(g.scan_tmp, bytes, g.count, g.start, ncell + 1, s), "cell scan");
    OrderOutputs out{g.part_cel, bounds ? g.beg : nullptr, bounds ? g.end : nullptr, nullptr, nullptr};
    if (np > 0) {
        k_scatter<<<blocks_for(np), kBlock, 0, s>>>(np, g.key, g.rank, g.start, g.part_idx);
        LQ_TRY_CUDA(cudaGetLastError(), "k_scatter");
    }
    if (np > 0 || bounds) {
        std::unique_lock<std::mutex> lock(g_id_mu, std::defer_lock);
        IdentityRecord* id = nullptr;
        if (identity_key) {
            lock.lock();    /* until the launch that follows the identities is queued */
            id = identity_for_search(identity_key, np);
        }
        if (id) {
            out.ident_in = id->started ? id->ident : nullptr;
            out.ident_out = id->tmp;
        }
        /* few cells: fewer per warp, whose chain of cells is the time
         * (15 k cells: 6.0 us a launch with 8, 12.3 with 32; 2.1 M cells:
         * 83 us a search with 16, 86 with 8, 90 with 32) */
        if (ncell <= 1 << 18)
            k_cell_order<8><<<blocks_for(ncell, kBlock / 4), kBlock, 0, s>>>(ncell, np, g.start, g.part_idx, out);
        else
            k_cell_order<16><<<blocks_for(ncell, kBlock / 2), kBlock, 0, s>>>(ncell, np, g.start, g.part_idx, out);
        LQ_TRY_CUDA(cudaGetLastError(), "k_cell_order");
        if (id) {
            std::swap(id->ident, id->tmp);
            id->started = true;
        }
    }
    return LQ_OK;
}

template <class W, class T>
static int sort_array(int n, const int* idx, T* data, T* cache, cudaStream_t s)
{
    if (n <= 0) return LQ_OK;
    if (n <= kSortSmall) {
        k_sort_small<W><<<kSortCluster, kBlock, 0, s>>>(n, idx, data, cache);
        LQ_TRY_CUDA(cudaGetLastError(), "k_sort_small");
        return LQ_OK;
    }
    k_sort_gather<<<blocks_for(n, kSortItems * kBlock), kBlock, 0, s>>>(n, idx, data, cache);
    LQ_TRY_CUDA(cudaGetLastError(), "k_sort_gather");
    const long long words = (long long)n * (int)(sizeof(T) / sizeof(W));
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(blocks_for(words, kSortItems * kBlock));
    c.blockDim = dim3(kBlock);
    c.stream = s;
    c.attrs = &early;
    c.numAttrs = 1;
    LQ_TRY_CUDA(cudaLaunchKernelEx(&c, k_sort_copy_back<W>, words, reinterpret_cast<const W*>(cache),
                                   reinterpret_cast<W*>(data)),
                "k_sort_copy_back");
    return LQ_OK;
}

int sort_float4(int n, const int* idx, float4* data, float4* cache, cudaStream_t s)
{
    return sort_array<float4>(n, idx, data, cache, s);
}

int sort_tensor2d(int n, const int* idx, tensor2d* data, tensor2d* cache, cudaStream_t s)
{
    return sort_array<float2>(n, idx, data, cache, s);
}

/* This translation unit's count of bounds violations (always 0 without
 * LQ_CHECKED). */
int bounds_count_grid(unsigned long long* v)
{
#ifdef LQ_CHECKED
    LQ_TRY_CUDA(cudaMemcpyFromSymbol(v, lq_bounds_count, sizeof(*v)), "bounds counter");
#else
    *v = 0;
#endif
    return LQ_OK;
}

namespace {

__global__ void __launch_bounds__(kBlock) k_iota(int n, int* __restrict__ p)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = i;
}

/* p[i] = i, there when the call returns, whatever stream reads it next. */
int fill_identities(int n, int* p)
{
    if (n <= 0) return LQ_OK;
    cudaStream_t s = nullptr;
    LQ_TRY_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "grid identities");
    k_iota<<<blocks_for(n), kBlock, 0, s>>>(n, p);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaStreamDestroy(s);
    LQ_TRY_CUDA(e, "grid identities");
    return LQ_OK;
}

}  // namespace

int identity_reset(const int* key, int np)
{
    std::lock_guard<std::mutex> lock(g_id_mu);
    IdentityRecord& r = g_ids[key];
    if (r.np != np || !r.ident) {
        cudaFree(r.ident);
        cudaFree(r.tmp);
        r = IdentityRecord{};
        const size_t b = sizeof(int) * (size_t)(np > 0 ? np : 1);
        cudaError_t e = cudaMalloc((void**)&r.ident, b);
        if (e == cudaSuccess) e = cudaMalloc((void**)&r.tmp, b);
        if (e != cudaSuccess) {
            cudaFree(r.ident);
            cudaFree(r.tmp);
            g_ids.erase(key);
            return set_error(LQ_ERR_ALLOC, "grid identities: %s", cudaGetErrorString(e));
        }
        r.np = np;
    }
    r.gen = ++g_id_gen;
    r.started = false;
    LQ_TRY(fill_identities(np, r.ident));
    r.started = true;
    return LQ_OK;
}

void identity_release(const int* key)
{
    std::lock_guard<std::mutex> lock(g_id_mu);
    auto it = g_ids.find(key);
    if (it == g_ids.end()) return;
    cudaFree(it->second.ident);
    cudaFree(it->second.tmp);
    g_ids.erase(it);
}

bool identity_find(const int* key, GridIdentity* out)
{
    std::lock_guard<std::mutex> lock(g_id_mu);
    auto it = g_ids.find(key);
    if (it == g_ids.end() || !it->second.started) return false;
    out->ident = it->second.ident;
    out->np = it->second.np;
    out->gen = it->second.gen;
    return true;
}

int gather_state(int n, const int* idx, const State& in, const State& out, cudaStream_t s)
{
    if (n <= 0) return LQ_OK;
    k_gather_state<<<blocks_for(n), kBlock, 0, s>>>(n, idx, in, out);
    LQ_TRY_CUDA(cudaGetLastError(), "k_gather_state");
    return LQ_OK;
}

}  // namespace lqb

/* ------------------------------------------------------------------ C ABI */

namespace {

struct LqGrid {
    lqb::GridBuffers g;
};

void free_grid_buffers(lqb::GridBuffers& g)
{
    if (g.beg) lqb::identity_release(g.beg);
    cudaFree(g.key);
    cudaFree(g.rank);
    cudaFree(g.count);
    cudaFree(g.start);
    cudaFree(g.part_idx);
    cudaFree(g.part_cel);
    cudaFree(g.beg);
    cudaFree(g.end);
    cudaFree(g.scan_tmp);
    g = lqb::GridBuffers();
}

int alloc_grid_buffers(lqb::GridBuffers& g, int np, int ncell)
{
    if (np < 0 || ncell < 1) return lqb::set_error(LQ_ERR_ARG, "grid: bad sizes np=%d ncell=%d", np, ncell);
    free_grid_buffers(g);
    size_t npb = sizeof(int) * (size_t)(np > 0 ? np : 1);
    size_t ncb = sizeof(int) * (size_t)(ncell + 1);
    LQ_TRY(lqb::scan_scratch_bytes(ncell, &g.scan_bytes));
    cudaError_t e = cudaSuccess;
    e = e ? e : cudaMalloc(&g.key, npb);
    e = e ? e : cudaMalloc(&g.rank, npb);
    e = e ? e : cudaMalloc(&g.part_idx, npb);
    e = e ? e : cudaMalloc(&g.part_cel, npb);
    e = e ? e : cudaMalloc(&g.count, ncb);
    e = e ? e : cudaMalloc(&g.start, ncb);
    e = e ? e : cudaMalloc(&g.beg, ncb);
    e = e ? e : cudaMalloc(&g.end, ncb);
    e = e ? e : cudaMalloc(&g.scan_tmp, g.scan_bytes > 0 ? g.scan_bytes : 16);
    if (e != cudaSuccess) {
        free_grid_buffers(g);
        return lqb::set_error(LQ_ERR_ALLOC, "grid: device allocation failed: %s", cudaGetErrorString(e));
    }
    g.np_cap = np;
    g.ncell_cap = ncell;
    return lqb::identity_reset(g.beg, np);
}

}  // namespace

extern "C" int lq_grid_create(int np, int ncell, void** grid)
{
    if (!grid) return lqb::set_error(LQ_ERR_ARG, "lq_grid_create: null output");
    *grid = nullptr;
    LqGrid* G = new LqGrid();
    int st = alloc_grid_buffers(G->g, np, ncell);
    if (st != LQ_OK) {
        delete G;
        return st;
    }
    *grid = G;
    return LQ_OK;
}

extern "C" int lq_grid_resize(void* grid, int np, int ncell)
{
    if (!grid) return lqb::set_error(LQ_ERR_ARG, "lq_grid_resize: null grid");
    return alloc_grid_buffers(static_cast<LqGrid*>(grid)->g, np, ncell);
}

extern "C" int lq_grid_destroy(void* grid)
{
    if (!grid) return LQ_OK;
    LqGrid* G = static_cast<LqGrid*>(grid);
    free_grid_buffers(G->g);
    delete G;
    return LQ_OK;
}

extern "C" int lq_grid_neighbor_search(void* grid, const void* par_host, const void* par_device,
                                       const float* pospres, const float* idep, void* stream)
{
    (void)idep;
    if (!grid || !par_host || !par_device || (!pospres && static_cast<const Parameters*>(par_host)->np > 0))
        return lqb::set_error(LQ_ERR_ARG, "lq_grid_neighbor_search: null argument");
    LqGrid* G = static_cast<LqGrid*>(grid);
    const Parameters* ph = static_cast<const Parameters*>(par_host);
    LQ_TRY(lqb::grid_search(ph, static_cast<const Parameters*>(par_device), reinterpret_cast<const float4*>(pospres),
                            G->g, true, nullptr, static_cast<cudaStream_t>(stream), nullptr, lqb::Frames(),
                            G->g.beg));
    return LQ_OK;
}

extern "C" int lq_grid_arrays(void* grid, const int** part_cel, const int** part_idx, const int** cell_beg,
                              const int** cell_end, const int** cell_start)
{
    if (!grid) return lqb::set_error(LQ_ERR_ARG, "lq_grid_arrays: null grid");
    LqGrid* G = static_cast<LqGrid*>(grid);
    if (part_cel) *part_cel = G->g.part_cel;
    if (part_idx) *part_idx = G->g.part_idx;
    if (cell_beg) *cell_beg = G->g.beg;
    if (cell_end) *cell_end = G->g.end;
    if (cell_start) *cell_start = G->g.start;
    return LQ_OK;
}

extern "C" int lq_grid_sort_float4(void* grid, int np, float* data, float* cache, void* stream)
{
    if (!grid || (np > 0 && (!data || !cache))) return lqb::set_error(LQ_ERR_ARG, "lq_grid_sort_float4: null argument");
    LqGrid* G = static_cast<LqGrid*>(grid);
    if (np > G->g.np_cap) return lqb::set_error(LQ_ERR_ARG, "lq_grid_sort_float4: np exceeds grid capacity");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return lqb::sort_float4(np, G->g.part_idx, reinterpret_cast<float4*>(data), reinterpret_cast<float4*>(cache), s);
}

extern "C" int lq_grid_sort_tensor2d(void* grid, int np, float* data, float* cache, void* stream)
{
    if (!grid || (np > 0 && (!data || !cache)))
        return lqb::set_error(LQ_ERR_ARG, "lq_grid_sort_tensor2d: null argument");
    LqGrid* G = static_cast<LqGrid*>(grid);
    if (np > G->g.np_cap) return lqb::set_error(LQ_ERR_ARG, "lq_grid_sort_tensor2d: np exceeds grid capacity");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return lqb::sort_tensor2d(np, G->g.part_idx, reinterpret_cast<tensor2d*>(data), reinterpret_cast<tensor2d*>(cache),
                              s);
}

/* ------------------------------------------------- C++ drop-in LoquatGrid */
/* The eight private members keep the reference layout (src/loquat_grid.h:32-41).
 * buffer holds [count | start | scan scratch], each 256-byte aligned. */

namespace {

[[noreturn]] void die(const char* what)
{
    fprintf(stderr, "LoquatGrid::%s failed: %s\n", what, lq_last_error());
    exit(EXIT_FAILURE);
}

inline size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

}  // namespace

LoquatGrid::LoquatGrid()
    : part_cel(nullptr), part_idx(nullptr), cell_beg(nullptr), cell_end(nullptr), part_cel_cache(nullptr),
      part_idx_cache(nullptr), buffer(nullptr), buffer_storage_bytes(0)
{
}

LoquatGrid::~LoquatGrid()
{
    if (cell_beg) lqb::identity_release(cell_beg);
    cudaFree(part_cel);
    cudaFree(part_idx);
    cudaFree(cell_beg);
    cudaFree(cell_end);
    cudaFree(part_cel_cache);
    cudaFree(part_idx_cache);
    cudaFree(buffer);
}

void LoquatGrid::GridConfig(Parameters* par_host)
{
    ResizeArrayLength(par_host->np, par_host->ncell);
    /* ParticleInteraction's working arrays too, at set-up as the reference
     * allocates its own, so the step loop allocates nothing */
    if (lq_interaction_reserve(par_host) != LQ_OK) die("GridConfig");
}

void LoquatGrid::ResizeArrayLength(int np_new, int ncell_new)
{
    if (np_new < 0 || ncell_new < 1) {
        lqb::set_error(LQ_ERR_ARG, "bad sizes np=%d ncell=%d", np_new, ncell_new);
        die("ResizeArrayLength");
    }
    if (cell_beg) lqb::identity_release(cell_beg);
    cudaFree(part_cel);
    cudaFree(part_idx);
    cudaFree(cell_beg);
    cudaFree(cell_end);
    cudaFree(part_cel_cache);
    cudaFree(part_idx_cache);
    cudaFree(buffer);
    size_t scan = 0;
    if (lqb::scan_scratch_bytes(ncell_new, &scan) != LQ_OK) die("ResizeArrayLength");
    const size_t npb = sizeof(int) * (size_t)(np_new > 0 ? np_new : 1);
    const size_t ncb = sizeof(int) * (size_t)ncell_new;
    const size_t tab = align256(sizeof(int) * (size_t)(ncell_new + 1));
    buffer_storage_bytes = 2 * tab + align256(scan > 0 ? scan : 16);
    cudaError_t e = cudaSuccess;
    e = e ? e : cudaMalloc(&part_cel, npb);
    e = e ? e : cudaMalloc(&part_idx, npb);
    e = e ? e : cudaMalloc(&cell_beg, ncb);
    e = e ? e : cudaMalloc(&cell_end, ncb);
    e = e ? e : cudaMalloc(&part_cel_cache, npb);
    e = e ? e : cudaMalloc(&part_idx_cache, npb);
    e = e ? e : cudaMalloc(&buffer, buffer_storage_bytes);
    if (e != cudaSuccess) {
        lqb::set_error(LQ_ERR_ALLOC, "%s", cudaGetErrorString(e));
        die("ResizeArrayLength");
    }
    /* particle identities through the searches (ParticleInteraction keeps
     * its neighbour lists across searches with them) */
    if (lqb::identity_reset(cell_beg, np_new) != LQ_OK) die("ResizeArrayLength");
}

void LoquatGrid::SortParticleByCellIndex(Parameters* par_host)
{
    (void)par_host; /* the sort runs inside NeighborSearch */
}

void LoquatGrid::NeighborSearch(Parameters* par_host, Parameters* par_device, float4* pospres, float4* idep)
{
    (void)idep;
    const int ncell = par_host->ncell;
    const size_t tab = align256(sizeof(int) * (size_t)(ncell + 1));
    lqb::GridBuffers g;
    g.np_cap = par_host->np;
    g.ncell_cap = ncell;
    g.key = part_cel_cache;
    g.rank = part_idx_cache;
    g.count = static_cast<int*>(buffer);
    g.start = reinterpret_cast<int*>(static_cast<char*>(buffer) + tab);
    g.scan_tmp = static_cast<char*>(buffer) + 2 * tab;
    g.scan_bytes = buffer_storage_bytes - 2 * tab;
    g.part_idx = part_idx;
    g.part_cel = part_cel;
    g.beg = cell_beg;
    g.end = cell_end;
    if (lqb::grid_search(par_host, par_device, pospres, g, true, nullptr, 0, nullptr, lqb::Frames(), cell_beg) !=
        LQ_OK)
        die("NeighborSearch");
}

void LoquatGrid::SortArrayFloat4(int np, float4* data, float4* data_cache)
{
    if (lqb::sort_float4(np, part_idx, data, data_cache, 0) != LQ_OK) die("SortArrayFloat4");
}

void LoquatGrid::SortArrayTensor2d(int np, tensor2d* data, tensor2d* data_cache)
{
    if (lqb::sort_tensor2d(np, part_idx, data, data_cache, 0) != LQ_OK) die("SortArrayTensor2d");
}
