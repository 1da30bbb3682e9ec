// pa_post.cu -- passes over a generated edge list: row canonicalisation and
// undirected degrees (the device side of src/PA/cuPPA/cuPPA.cu:103-165, which
// copies the whole graph to the host and counts there).
#include <algorithm>

#include "pa_device.cuh"
#include "pa_internal.h"
#include "pa_wide.h"

namespace pa {
namespace {

constexpr uint32_t kFull = 0xffffffffu;

// Sort each generated node's d pairs by dst.  A group of d lanes holds one row;
// lane i's rank is the number of smaller values in its group (values in a row
// are distinct), and it stores its pair at that rank.  All loads of a warp
// iteration happen before its stores, so in == out is safe.
template <typename Id>
__global__ void canon_kernel(const Id *in, Id *out, uint64_t n, uint32_t d, uint64_t seed_edges)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t G = 32u / d;
    const uint32_t g = lane / d, i = lane - g * d;
    const bool used = lane < G * d;
    const uint64_t rows = n - (d + 1);
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    const uint64_t w0 = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);

    // seed edges are already canonical
    if (in != out)
        for (uint64_t e = w0 * 32 + lane; e < seed_edges; e += warps * 32) {
            out[2 * e] = in[2 * e];
            out[2 * e + 1] = in[2 * e + 1];
        }

    for (uint64_t r0 = w0 * G; r0 < rows; r0 += warps * G) {
        const uint64_t row = r0 + g;
        const bool act = used && row < rows;
        const uint64_t e = seed_edges + row * d + i;
        Id src = 0, dst = 0;
        if (act) {
            src = in[2 * e];
            dst = in[2 * e + 1];
        }
        uint32_t rank = 0;
        for (uint32_t j = 0; j < d; ++j) {
            const Id o = __shfl_sync(kFull, dst, g * d + j);
            rank += (o < dst) ? 1u : 0u;
        }
        __syncwarp();
        if (act) {
            const uint64_t eo = seed_edges + row * d + rank;
            out[2 * eo] = src;
            out[2 * eo + 1] = dst;
        }
    }
}

// ---------------------------------------------------------------------------
// Undirected degrees.
//
// A generated pair's source is known from its place (pair seed_edges + r*d + j
// belongs to node u_first + r), so the counts start at d for every generated node
// and a pair costs one atomic, for its target; a pair whose source is another
// (a list in some other order) moves one count from the expected node to its own.
//
// What bounds it: the target atomics, spread over the whole count array.  They
// run at L2 speed only while the array stays in L2, so the counts are 32 bits
// wide, in the front half of the output, and widened in place at the end
// (64-bit counts for lists of 2^31 pairs and more, and below kDegNarrow nodes,
// whose 64-bit counts are in L2 too and need no widening launches).  Early nodes hold the
// hubs: ids below kLowIds are counted in shared memory, one flush per block.
//
// Seed edges: SLOTS lists hold none, and the counts start with them; those of PAIRS
// lists are spread over the grid like the rest.  A clique's source repeats through its
// row, so a warp counts equal sources with one atomic (d = 8,192, n = 2 d, 3.4 * 10^7
// seed edges: 36.4 ms by one block, 0.45 so).
// n = 2^24, d = 8, p = 0.3, 32-bit ids: 5.63 -> 0.97 ms (138 G targets/s; two
// atomics a pair combined by __match_any_sync before); p = 0.1, 64-bit ids:
// 15.9 -> 0.82 ms; n = 10^6: 0.309 -> 0.062 ms.
// ---------------------------------------------------------------------------
constexpr uint32_t kDegThreads = 512;
constexpr uint32_t kDegChunk = 8192;   // pairs per block step at most
constexpr uint64_t kDegNarrow = 1ull << 22;   // nodes above which 32-bit counts pay
constexpr uint32_t kLowIds = 8192;     // 32 KB of shared counters

// The counts before any pair is read: d from node `from` on, `low` below.
template <typename Cnt>
__global__ void __launch_bounds__(kDegThreads) degree_init_kernel(Cnt *deg, uint64_t n, uint64_t from,
                                                                  uint32_t d, uint32_t low)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n; u += stride)
        deg[u] = u >= from ? (Cnt)d : (Cnt)low;
}

// Pairs (or, with Slots, targets) of the generated nodes: `count` of them from E
// + (Slots ? 0 : 2) * seed_edges, `chunk` (<= kDegChunk) a block step; with pairs the
// seed edges too.
template <typename Id, bool Slots, typename Cnt>
__global__ void __launch_bounds__(kDegThreads) degree_kernel(const Id *E, uint64_t count,
                                                             uint32_t chunk, uint32_t d,
                                                             uint32_t d_inv, uint64_t u_first,
                                                             uint64_t seed_edges,
                                                             uint64_t n, bool vec, Cnt *deg)
{
    __shared__ uint32_t low[kLowIds];
    for (uint32_t i = threadIdx.x; i < kLowIds; i += kDegThreads) low[i] = 0;
    __syncthreads();
    if constexpr (!Slots) {
        const uint64_t step = (uint64_t)gridDim.x * kDegThreads;
        const uint32_t lane = threadIdx.x & 31u;
        for (uint64_t e0 = (uint64_t)blockIdx.x * kDegThreads + (threadIdx.x - lane); e0 < seed_edges;
             e0 += step) {
            const uint64_t e = e0 + lane;
            uint64_t s = ~0ull, t = ~0ull;
            if (e < seed_edges) {
                s = (uint64_t)(int64_t)E[2 * e];
                t = (uint64_t)(int64_t)E[2 * e + 1];
            }
            const bool in = s < n && t < n;   // ids are used as addresses: never trust them
            const uint32_t same = __match_any_sync(kFull, in ? s : ~0ull);
            if (in && (uint32_t)__ffs(same) - 1u == lane) {
                if (s < kLowIds) atomicAdd(low + s, (uint32_t)__popc(same));
                else atomicAdd(deg + s, (Cnt)__popc(same));
            }
            if (in) {
                if (t < kLowIds) atomicAdd(low + t, 1u);
                else atomicAdd(deg + t, (Cnt)1);
            }
        }
    }
    const Id *G = E + (Slots ? 0 : 2 * seed_edges);
    constexpr uint32_t U = 4;   // loads in flight per thread
    for (uint64_t c0 = (uint64_t)blockIdx.x * chunk; c0 < count; c0 += (uint64_t)gridDim.x * chunk) {
        const uint64_t row0 = c0 / d;
        const uint32_t x0 = (uint32_t)(c0 - row0 * d);   // the chunk starts at slot x0 of row row0
        const uint32_t len = (uint32_t)min((uint64_t)chunk, count - c0);
        for (uint32_t b = threadIdx.x; b < len; b += U * kDegThreads) {
            uint64_t s[U], t[U];
#pragma unroll
            for (uint32_t q = 0; q < U; ++q) {
                const uint32_t x = b + q * kDegThreads;
                t[q] = ~0ull;
                s[q] = ~0ull;
                if (x < len) {
                    if constexpr (Slots) {
                        t[q] = (uint64_t)__ldcs(G + c0 + x);
                    } else if (!vec) {
                        s[q] = (uint64_t)(int64_t)G[2 * (c0 + x)];
                        t[q] = (uint64_t)(int64_t)G[2 * (c0 + x) + 1];
                    } else if constexpr (sizeof(Id) == 4) {
                        const int2 w = __ldcs(reinterpret_cast<const int2 *>(G) + c0 + x);
                        s[q] = (uint64_t)(int64_t)w.x;
                        t[q] = (uint64_t)(int64_t)w.y;
                    } else {
                        const longlong2 w = __ldcs(reinterpret_cast<const longlong2 *>(G) + c0 + x);
                        s[q] = (uint64_t)w.x;
                        t[q] = (uint64_t)w.y;
                    }
                }
            }
#pragma unroll
            for (uint32_t q = 0; q < U; ++q) {
                const uint32_t x = b + q * kDegThreads;
                if (x >= len) continue;
                if (Slots ? t[q] < n : (t[q] < n && s[q] < n)) {
                    if (t[q] < kLowIds) atomicAdd(low + t[q], 1u);
                    else atomicAdd(deg + t[q], (Cnt)1);
                } else {
                    t[q] = ~0ull;   // not counted at either end
                }
                if constexpr (!Slots) {
                    const uint64_t u = u_first + row0 + (d == 1 ? x : __umulhi(x0 + x, d_inv));
                    if (s[q] != u || t[q] == ~0ull) {
                        atomicAdd(deg + u, (Cnt)-1);
                        if (t[q] != ~0ull) atomicAdd(deg + s[q], (Cnt)1);
                    }
                }
            }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kLowIds; i += kDegThreads)
        if (low[i]) atomicAdd(deg + i, (Cnt)low[i]);   // ids below n only were counted
}

// 32-bit counts [lo, hi) of the array's front to 64 bits in place: 8 lo >= 4 hi,
// so no count of the range is overwritten before it is read.
__global__ void __launch_bounds__(256) widen_kernel(uint32_t *c, uint64_t lo, uint64_t hi)
{
    unsigned long long *w = reinterpret_cast<unsigned long long *>(c);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += stride)
        w[i] = c[i];
}

// The first `count` (at most kLowIds) of them, through shared memory (one block).
__global__ void __launch_bounds__(1024) widen_low_kernel(uint32_t *c, uint32_t count)
{
    __shared__ uint32_t v[kLowIds];
    for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) v[i] = c[i];
    __syncthreads();
    unsigned long long *w = reinterpret_cast<unsigned long long *>(c);
    for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) w[i] = v[i];
}

// MurmurHash3's 64-bit finalizer (Appleby, public domain): a bijective mix.
__device__ __forceinline__ uint64_t fmix64(uint64_t k)
{
    k ^= k >> 33;
    k *= 0xFF51AFD7ED558CCDull;
    k ^= k >> 33;
    k *= 0xC4CEB9FE1A85EC53ull;
    k ^= k >> 33;
    return k;
}

// Digest term of id x at position pos (the position is mixed in first, so two
// elements that trade places change the digest).
__device__ __forceinline__ uint64_t digest_term(uint64_t pos, uint64_t x)
{
    return fmix64(fmix64(pos * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull) ^ x);
}

// Sum and xor of the digest terms of x[0..count), positions from `base`.  A
// thread takes 16-byte vectors (two int64 or four int32 ids) with streaming
// loads when x is 16-byte aligned; a warp and then the block reduce, and one
// thread per block adds to acc (sum) and xors into acc + 1.
template <typename Id>
__global__ void __launch_bounds__(256) digest_kernel(const Id *x, uint64_t count, uint64_t base,
                                                     bool vec, unsigned long long *acc)
{
    constexpr uint32_t V = 16 / sizeof(Id);
    uint64_t sum = 0, xr = 0;
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t nvec = vec ? count / V : 0;
    const uint4 *xv = reinterpret_cast<const uint4 *>(x);
    for (uint64_t i = tid; i < nvec; i += stride) {
        const uint4 w = __ldcs(xv + i);
        Id vals[V];
        memcpy(vals, &w, sizeof(w));
#pragma unroll
        for (uint32_t j = 0; j < V; ++j) {
            const uint64_t h = digest_term(base + i * V + j, (uint64_t)(int64_t)vals[j]);
            sum += h;
            xr ^= h;
        }
    }
    for (uint64_t i = nvec * V + tid; i < count; i += stride) {
        const uint64_t h = digest_term(base + i, (uint64_t)(int64_t)x[i]);
        sum += h;
        xr ^= h;
    }
    for (int off = 16; off > 0; off >>= 1) {
        sum += __shfl_xor_sync(kFull, sum, off);
        xr ^= __shfl_xor_sync(kFull, xr, off);
    }
    __shared__ uint64_t ssum[8], sxr[8];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (lane == 0) {
        ssum[warp] = sum;
        sxr[warp] = xr;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (uint32_t w = 1; w < (blockDim.x >> 5); ++w) {
            sum += ssum[w];
            xr ^= sxr[w];
        }
        atomicAdd(acc, (unsigned long long)sum);
        atomicXor(acc + 1, (unsigned long long)xr);
    }
}

int grid_for(uint64_t work_items, uint32_t threads, uint32_t per_sm = 8)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    uint64_t want = (work_items + threads - 1) / threads;
    const uint64_t cap = (uint64_t)sms * per_sm;
    if (want > cap) want = cap;
    return (int)(want ? want : 1);
}

template <typename Id, bool Slots, typename Cnt>
void degrees_launch(const pa_params *prm, const GenPlan &p, const Id *E, Cnt *deg, cudaStream_t s)
{
    const uint64_t n = prm->n, count = (n - p.u_first) * prm->d;
    // the generated nodes' out-edges; with SLOTS the seed edges too, both ends (CLIQUE:
    // every seed node has d; STAR_REF: node d has d, the others 1)
    const uint64_t from = !Slots ? p.u_first : (prm->seed_mode == PA_SEED_CLIQUE ? 0 : prm->d);
    degree_init_kernel<Cnt><<<grid_for(n, kDegThreads), kDegThreads, 0, s>>>(deg, n, from, prm->d,
                                                                             Slots ? 1u : 0u);
    // floor(x / d) = umulhi(x, d_inv) for x below 2^16: d_inv = ceil(2^32 / d) is off
    // by less than 1 / x (d = 1: 2^32 does not fit)
    // one load per pair when the pairs are aligned to their size
    const bool vec = (reinterpret_cast<uintptr_t>(E) & (2 * sizeof(Id) - 1)) == 0;
    const uint32_t d_inv = (uint32_t)(((1ull << 32) + prm->d - 1) / prm->d);
    // whole chunks, four blocks per SM; less per block step where that leaves SMs idle
    uint32_t chunk = kDegChunk;
    while (chunk > 1024 && count < 600ull * chunk) chunk /= 2;
    const uint64_t blocks = std::max<uint64_t>((count + chunk - 1) / chunk,
                                               Slots ? 0 : p.seed_edges / (4 * kDegThreads));
    degree_kernel<Id, Slots, Cnt><<<grid_for(blocks, 1, 4), kDegThreads, 0, s>>>(
        E, count, chunk, prm->d, d_inv, p.u_first, p.seed_edges, n, vec, deg);
}

template <typename Id>
void degrees_any(const pa_params *prm, const GenPlan &p, const Id *E, int64_t *d_deg, cudaStream_t s)
{
    if (p.n_edges >= (1ull << 31) || prm->n <= kDegNarrow) {
        unsigned long long *deg = reinterpret_cast<unsigned long long *>(d_deg);
        if (p.slots) degrees_launch<Id, true>(prm, p, E, deg, s);
        else degrees_launch<Id, false>(prm, p, E, deg, s);
        return;
    }
    uint32_t *deg = reinterpret_cast<uint32_t *>(d_deg);
    if (p.slots) degrees_launch<Id, true>(prm, p, E, deg, s);
    else degrees_launch<Id, false>(prm, p, E, deg, s);
    uint64_t hi = prm->n;
    while (hi > kLowIds) {
        const uint64_t lo = (hi + 1) / 2;
        widen_kernel<<<grid_for(hi - lo, 256), 256, 0, s>>>(deg, lo, hi);
        hi = lo;
    }
    widen_low_kernel<<<1, 1024, 0, s>>>(deg, (uint32_t)hi);
}

}  // namespace
}  // namespace pa

using namespace pa;

extern "C" {

int pa_canonicalize(const pa_params *prm, const void *d_edges, void *d_out, void *stream)
{
    GenPlan p;
    const int rc = make_plan(prm, &p);
    if (rc != PA_OK) return rc;
    if (!d_edges || !d_out) return PA_ERR_INVALID;
    if (p.slots) return PA_ERR_NOT_SUPPORTED;
    const uint64_t rows = prm->n - p.u_first;
    const uint32_t threads = 256;
    const int grid = grid_for(rows * prm->d, threads);
    cudaStream_t s = (cudaStream_t)stream;
    if (p.wide) return gen::canon_wide(p.id_bytes, d_edges, d_out, prm->n, prm->d, p.seed_edges, s);
    if (p.id_bytes == 8)
        canon_kernel<int64_t><<<grid, threads, 0, s>>>((const int64_t *)d_edges, (int64_t *)d_out,
                                                       prm->n, prm->d, p.seed_edges);
    else
        canon_kernel<int32_t><<<grid, threads, 0, s>>>((const int32_t *)d_edges, (int32_t *)d_out,
                                                       prm->n, prm->d, p.seed_edges);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PA_OK : set_cuda_error(e);
}

int pa_degrees(const pa_params *prm, const void *d_edges, int64_t *d_deg, void *stream)
{
    GenPlan p;
    const int rc = make_plan(prm, &p);
    if (rc != PA_OK) return rc;
    if (!d_edges || !d_deg) return PA_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    if (p.id_bytes == 8) degrees_any<int64_t>(prm, p, (const int64_t *)d_edges, d_deg, s);
    else degrees_any<int32_t>(prm, p, (const int32_t *)d_edges, d_deg, s);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PA_OK : set_cuda_error(e);
}

int pa_digest(const void *d_ids, uint64_t count, uint32_t id_bits, uint64_t index_base,
              uint64_t *d_acc, void *stream)
{
    if (!d_acc || (id_bits != 32 && id_bits != 64) || (count && !d_ids)) return PA_ERR_INVALID;
    if (reinterpret_cast<uintptr_t>(d_acc) & 7u) return PA_ERR_INVALID;
    if (!count) return PA_OK;
    const uint32_t threads = 256;
    const bool vec = (reinterpret_cast<uintptr_t>(d_ids) & 15u) == 0;
    // Up to eight blocks of 256 threads per SM (grid_for): enough 16-byte loads
    // in flight to stream at HBM speed; the grid never exceeds the work.
    const int grid = grid_for(count / (vec ? 16u / (id_bits / 8u) : 1u) + 1, threads);
    cudaStream_t s = (cudaStream_t)stream;
    if (id_bits == 64)
        digest_kernel<int64_t><<<grid, threads, 0, s>>>((const int64_t *)d_ids, count, index_base,
                                                        vec, (unsigned long long *)d_acc);
    else
        digest_kernel<int32_t><<<grid, threads, 0, s>>>((const int32_t *)d_ids, count, index_base,
                                                        vec, (unsigned long long *)d_acc);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? PA_OK : set_cuda_error(e);
}

}  // extern "C"
