// pa_start.cu -- graphs generated with waits on single slots.
//
// Early in a graph most copy reads land on nodes that are still being
// generated.  The persistent kernel publishes completion per tile, and a tile
// is complete only once the sources of all of its nodes are, so a dependency
// chain counted in tiles is far longer than the same chain counted in nodes:
// the longest chain of a random recursive graph grows like c*ln(u) in nodes,
// while a tile takes the maximum over the chains of all its ~2*tile_nodes copy
// sources at every step (a simulation of d = 4, p = 1/2 gives 28 node steps but
// 136 tile steps at 8192 nodes, 49 against 365 at 2^18).  With each step a
// poll round trip, the first few million nodes of a graph cost milliseconds.
//
// This kernel takes the tile out of the chain.  Before it runs, every pair of
// its region is set to all-ones (by the set-up kernel, a memset above 32 MB), which is
// never a node id.  A lane
// stores its slot's pair the moment the slot is final -- every lower slot of
// its node final and its candidate distinct from theirs -- and a copy read of
// slot (v, k) re-reads that pair's target field until it is not all-ones.  The
// datum is its own completion flag: it is written once, with its final value,
// so a gpu-scope relaxed load returns either the fill or that value, and no
// fence, flag or watermark is involved.  Copy sources inside the lane's own
// warp pass are taken from the source lane by shuffle once it is final, as in
// the persistent kernel.  (Filling inside the kernel instead -- each warp
// filling the tile it claims, with per-tile opened flags and a watermark for
// readers -- measured slower on B200 than the fill it saves: 88.7 against
// 68.0 ms for n = 2^30, d = 4.)
//
// Work is claimed one start tile at a time: P warp passes (1, 2 or kStartPasses,
// start_variant says which and why) of G = 32/d nodes each (lane = node-in-pass
// * d + slot), resolved together, so a wait in one pass does not hold back the
// others.  Claims of several tiles at once were tried for one-pass tiles: a tile
// behind an unfinished one of its warp holds up every chain through it (n =
// 10^6, d = 4, eight a claim: 379 against 107 us).  Warp w of a block claims
// from counter w (of kStartCounters), which hands out tiles w, w + 8, ... in
// increasing order: eight counter lines instead of one, since a single counter
// saturates at one atomic every few nanoseconds.  Several graphs share one
// launch in level order (pa_gen_core.cuh).
//
// Draws, the slot order and the rejection rule are the persistent kernel's, so
// the output is bit-identical to it and to the sequential definition
// (src/PA/SPA/SerialCopyModel3.cpp:50-92 of the reference, with Philox draws).
#include <algorithm>

#include "pa_gen_core.cuh"

namespace pa {
namespace gen {
namespace {

template <typename Id>
struct Sentinel {
    static constexpr uint64_t value = sizeof(Id) == 8 ? ~0ull : 0xffffffffull;
};

// Read slot (v, k) into s: true with its value, or false (s.val = v) while it
// still holds the fill.
template <typename Id, bool Slots>
__device__ __forceinline__ bool read_slot(Slot<uint32_t> &s, const GenArgs &a, const Id *E,
                                          uint32_t v, uint32_t k)
{
    const uint64_t x = ld_slot(slot_addr<Id, uint32_t, Slots>(E, a, v, k));
    if (x != Sentinel<Id>::value) {
        s.val = (uint32_t)x;
        return true;
    }
    s.val = v;
    return false;
}

// Where the candidate of a fresh draw comes from (32-bit node arithmetic: the
// start region ends below 2^31); true if slot (s.val, k) is to be read for it.
__device__ __forceinline__ bool place_start(Slot<uint32_t> &s, const DrawT<uint32_t> &dr, uint32_t r,
                                            const GenArgs &a, uint32_t pbase)
{
    uint32_t st = ST_KNOWN;
    s.val = dr.v;
    bool read = false;
    if (!dr.direct) {
        if (dr.v <= a.d) {
            s.val = (uint32_t)seed_slot(dr.v, dr.k, a.d, a.seed_mode);
        } else if (dr.v < pbase) {
            read = true;
        } else {
            st = ST_PEND_TILE;   // an earlier node of this same pass
        }
    }
    s.meta = st | (dr.k << 2) | (r << 8);
    return read;
}

template <typename Id, bool Slots>
__device__ __forceinline__ void classify_start(Slot<uint32_t> &s, const DrawT<uint32_t> &dr,
                                               uint32_t r, const GenArgs &a, const Id *E,
                                               uint32_t pbase, uint32_t &n_pend)
{
    if (place_start(s, dr, r, a, pbase) &&
        !read_slot<Id, Slots>(s, a, E, s.val, meta_k(s.meta))) {
        s.meta |= ST_PEND_GLOBAL;
        ++n_pend;
    }
}

// The lower lanes of this lane's node whose key equals this lane's.  Latency: the
// launch is bound by the rounds of its chains, where up to three shuffles answer
// sooner than a match over 32 distinct keys (n = 10^5, d = 4: 51.2 -> 46.4 us); they
// take more instructions, which bind larger graphs (n = 2^24, p = 0: 3.83 against
// 4.58 ms with shuffles).
template <bool Latency>
__device__ __forceinline__ uint32_t lower_equal(uint32_t key, const Lane &L, uint32_t d)
{
    if (Latency && d <= 4) {
        uint32_t low = 0;
#pragma unroll
        for (uint32_t j = 1; j < 4; ++j) {
            const uint32_t o = __shfl_up_sync(kFull, key, j);
            if (L.slot >= j && o == key) low |= (1u << L.lane) >> j;
        }
        return L.used ? low : 0u;
    }
    return __match_any_sync(kFull, key) & L.lt & L.gmask;
}

// The bit of slot (v, k) in the filter of rejected slots (start_kernel).
__device__ __forceinline__ uint32_t hop_bit(uint32_t v, uint32_t k, uint32_t d)
{
    return ((v * d + k) * 0x9E3779B1u) >> (32u - kHopLog2);
}

// Resolve the P warp passes of one start tile together; every slot is
// stored as soon as it is final.  Copy sources in the lane's own pass come from
// the source lane by shuffle; sources in an earlier pass of the tile are polled
// in memory like any other.  Returns false when the warp must stop (wait limit,
// or another warp failed).  Hop: slots that end on a later draw than their first are
// entered in the filter `rejected`.
template <typename Id, bool Slots, int P, bool Latency, bool Hop>
__device__ __forceinline__ bool resolve_start(Slot<uint32_t> (&s)[P], const GenArgs &a,
                                              Id *E, uint32_t tb, bool withhold, const Lane &L,
                                              uint32_t done, uint32_t *rejected,
                                              uint32_t &n_retry, uint32_t &n_wait,
                                              uint32_t &n_pend, uint32_t &n_poll)
{
    const uint32_t d = a.d, G = a.groups;
    // this lane's slot of pass 0: a pair (PAIRS) or an id (SLOTS, seed_edges = 0)
    const uint64_t e_lane = a.seed_edges + (uint64_t)(tb - (uint32_t)a.u_first) * d + L.lane;
    Id *pair0 = Slots ? E + e_lane : E + 2 * e_lane;
    uint32_t stored = 0;   // bit j: pass j's slot is stored (or inactive)
#pragma unroll
    for (int j = 0; j < P; ++j)
        if (!(L.used && tb + j * G + L.g < a.start_end)) stored |= 1u << j;
    const uint32_t max_sleep = min(a.max_sleep_ns, 512u);
    uint64_t spin_t0 = 0;
    uint32_t sleep_ns = 32;
    // done, bit j: every active slot of pass j is final and stored (warp-uniform);
    // a finished pass costs no more match or ballot while the others wait
    // bit j: this lane's slot of pass j changed after the pass's last match; a
    // pass in which no lane changed would match and vote exactly as before, so
    // only its pending reads are polled (one vote per pass and round)
    uint32_t dirty = (1u << P) - 1u;
    for (;;) {
        bool changed = false;
#pragma unroll
        for (int j = 0; j < P; ++j) {
            if ((done >> j) & 1u) continue;
            const uint32_t pbase = tb + j * G;
            const uint32_t u = pbase + L.g;
            const bool active = L.used && u < a.start_end;
            bool ch = (dirty >> j) & 1u;
            if (active && meta_st(s[j].meta) == ST_PEND_GLOBAL) {
                if (read_slot<Id, Slots>(s[j], a, E, s[j].val, meta_k(s[j].meta))) {
                    s[j].meta &= ~3u;
                    ch = true;
                    changed = true;
                } else {
                    ++n_poll;
                }
            }
            if (!__any_sync(kFull, ch)) continue;
            dirty &= ~(1u << j);
            const bool known = active && meta_st(s[j].meta) == ST_KNOWN;
            // node values are < 2^31: the lane-unique keys of unknown lanes never collide
            const uint32_t low =
                lower_equal<Latency>(known ? s[j].val : (0xffffffe0u | L.lane), L, d);
            const bool bad = active && (!known || low != 0u);
            const uint32_t badm = __ballot_sync(kFull, bad);
            const bool fin = active && (badm & L.gmask & L.le) == 0u;
            if (fin && !((stored >> j) & 1u)) {
                if (!withhold) {
                    if constexpr (Slots) st_relaxed_id(pair0 + (uint64_t)(j * G * d), s[j].val);
                    else st_relaxed_pair(pair0 + 2 * (uint64_t)(j * G * d), u, s[j].val);
                }
                stored |= 1u << j;
                if (Hop && meta_r(s[j].meta) != 0u) {
                    const uint32_t h = hop_bit(u, L.slot, d);
                    atomicOr(rejected + (h >> 5), 1u << (h & 31u));
                }
            }
            const uint32_t finm = __ballot_sync(kFull, fin || !active);
            if (finm == kFull) {
                done |= 1u << j;
                continue;
            }

            // copy sources in this pass: the source lane's value once it is final
            const bool same = active && meta_st(s[j].meta) == ST_PEND_TILE;
            const uint32_t src = same ? (s[j].val - pbase) * d + meta_k(s[j].meta) : L.lane;
            const uint32_t sv = __shfl_sync(kFull, s[j].val, src);
            if (same && ((finm >> src) & 1u)) {
                s[j].val = sv;
                s[j].meta &= ~3u;
                dirty |= 1u << j;
                changed = true;
            }

            // a candidate equal to a final lower slot of the node is rejected
            if (known && !fin && (low & finm) != 0u) {
                const uint32_t r = meta_r(s[j].meta) + 1u;
                classify_start<Id, Slots>(s[j], draw<uint32_t>(u, L.slot, r, a), r, a, E, pbase,
                                          n_pend);
                dirty |= 1u << j;
                changed = true;
                ++n_retry;
            }
        }
        if (done == (1u << P) - 1u) return true;

        if (!__any_sync(kFull, changed)) {
            unsigned long long now = 0;
            uint32_t err = 0;
            if (L.lane == 0) {
                now = globaltimer_ns();
                err = ld_relaxed_u32(&my_rep(a)->error);
                ++n_wait;
            }
            now = __shfl_sync(kFull, now, 0);
            err = __shfl_sync(kFull, err, 0);
            if (err != 0) return false;
            if (spin_t0 == 0) spin_t0 = now;
            if (now - spin_t0 > a.spin_limit_ns) {
                if (L.lane == 0) raise_error(a, (uint32_t)PA_ERR_SPIN_TIMEOUT);
                return false;
            }
            __nanosleep(sleep_ns);
            sleep_ns = min(sleep_ns * 2u, max_sleep);
        } else {
            spin_t0 = 0;
            sleep_ns = 32;
        }
    }
}

// Store the passes of a tile that are settled as drawn: every slot known, no value
// twice in a node.  Nearly all are, late in a large graph, and the rounds of
// resolve_start, made for slots that wait, take several times the instructions
// and a match each, which bound the launch where copies are few or in L2 (85 % of
// the match unit, 65 % of the issue slots at n = 2^24, d = 4, p = 1).  Up to d = 8 equal
// values are looked for by d - 1 shuffles.  Returns the stored passes.
// n = 2^24, d = 4: p = 1 667 -> 492 us, p = 0.5 851 -> 805; n = 10^7 536 -> 494; n = 2^28,
// p = 0.9 12.6 -> 10.3 ms.
template <typename Id, bool Slots, int P>
__device__ __forceinline__ uint32_t store_settled(const Slot<uint32_t> (&s)[P], const GenArgs &a,
                                                  Id *E, uint32_t tb, bool withhold, const Lane &L)
{
    const uint32_t d = a.d, pd = a.groups * d;
    const uint64_t e_lane = a.seed_edges + (uint64_t)(tb - (uint32_t)a.u_first) * d + L.lane;
    Id *to = Slots ? E + e_lane : E + 2 * e_lane;
    uint32_t done = 0;
#pragma unroll
    for (int j = 0; j < P; ++j) {
        const uint32_t u = tb + j * a.groups + L.g;
        const bool active = L.used && u < a.start_end;
        const uint32_t x = s[j].val;
        Id *const at = to;
        to += Slots ? pd : 2 * pd;
        if (!__all_sync(kFull, !active || meta_st(s[j].meta) == ST_KNOWN)) continue;
        bool dup = false;
        if (d <= 4) {
#pragma unroll
            for (uint32_t q = 1; q < 4; ++q) {
                const uint32_t o = __shfl_up_sync(kFull, x, q);
                dup |= L.slot >= q && o == x;
            }
        } else if (d <= 8) {
#pragma unroll
            for (uint32_t q = 1; q < 8; ++q) {
                const uint32_t o = __shfl_up_sync(kFull, x, q);
                dup |= L.slot >= q && o == x;
            }
        } else {
            // node values are < 2^31: the keys of other lanes never collide
            const uint32_t eq = __match_any_sync(kFull, active ? x : (0xffffffe0u | L.lane));
            dup = (eq & L.lt & L.gmask) != 0u;
        }
        if (__any_sync(kFull, active && dup)) continue;
        if (active && !withhold) {
            if constexpr (Slots) st_relaxed_id(at, x);
            else st_relaxed_pair(at, u, x);
        }
        done |= 1u << j;
    }
    return done;
}

__device__ __forceinline__ void set_lane(Lane &L, const GenArgs &a)
{
    L.g = L.lane / a.d;
    L.slot = L.lane - L.g * a.d;
    L.used = L.lane < a.groups * a.d;
    L.gmask = L.used ? (a.d == 32 ? kFull : (((1u << a.d) - 1u) << (L.g * a.d))) : 0u;
}

// Hop.  The copies of a large graph are bound by DRAM, which moves 128 bytes for a
// slot's 4 to 16 (n = 2^28, d = 4, p = 0.5: 69 GB for half as many slots of 16).  But slot
// (v, k) holds what its own first draw gave, unless that was rejected: was the draw
// direct, its value is known without a read, and was it a copy, that one's slot is
// read instead.  So such a graph is launched in growing ranges of nodes; every slot
// that ends on a later draw leaves a hashed bit in a filter (false hits cost a read);
// and copies of earlier launches' slots (below hop_end: final, their bits set) that
// the filter, held in shared memory, does not hold are drawn again.  One draw of the
// warp serves each lane's first such copy of the tile's four passes: draws take
// instructions, which bind the launch next (a draw per copy of two passes 14.31 ms,
// of all four 16.13, two draws as here 14.27, one 13.92; none 15.82).
template <typename Id, bool Slots, uint32_t MinBlocks, int P, bool Hop>
__global__ void __launch_bounds__(kThreads, MinBlocks) start_kernel(const StartArgs b)
{
    __shared__ uint32_t s_rejected[Hop ? kHopFilterBytes / 4 : 1];
    __shared__ GenArgs s_args[kThreads / 32];
    // per warp: the (level, graph) segment of its last claim, [lo, hi) and the
    // local unit of lo -- a warp's claims T, T + 8, ... mostly stay inside one,
    // and the two searches of map_unit cost as much as a tile's own work
    __shared__ unsigned long long s_seg[kThreads / 32][3];
    const uint32_t warp = threadIdx.x >> 5;
    GenArgs &a = s_args[warp];
    cudaGridDependencySynchronize();
    if ((threadIdx.x & 31u) == 0) {
        s_seg[warp][0] = 1;   // empty segment
        s_seg[warp][1] = 0;
    }
    __syncwarp();
    if constexpr (Hop) {
        for (uint32_t i = threadIdx.x; i < kHopFilterBytes / 16; i += kThreads)
            reinterpret_cast<uint4 *>(s_rejected)[i] =
                reinterpret_cast<const uint4 *>(b.rejected)[i];
        __syncthreads();
    }

    Lane L;
    L.lane = threadIdx.x & 31u;
    L.lt = lanemask_lt();
    L.le = L.lt | (1u << L.lane);
    uint32_t cur = 0xffffffffu;
    if (b.count == 1) {
        if (L.lane == 0) a = b.one;
        __syncwarp();
        set_lane(L, a);
        cur = 0;
    }

    if (!Slots && b.write_seeds) {
        // closed forms; nothing reads them back (SLOTS does not store them)
        const uint32_t gw = blockIdx.x * (kThreads / 32) + warp;
        const uint32_t nw = gridDim.x * (kThreads / 32);
        for (uint32_t i = gw; i < b.count; i += nw) {
            const GenArgs *ai = b.count == 1 ? &a : b.inst + i;
            Id *Ei = reinterpret_cast<Id *>(ai->edges);
            const uint32_t di = ai->d, mode = ai->seed_mode;
            const uint64_t se = ai->seed_edges;
            for (uint64_t e = L.lane; e < se; e += 32) {
                uint64_t src, dst;
                seed_edge(e, di, mode, src, dst);
                st_pair(Ei + 2 * e, src, dst);
            }
        }
    }

    uint32_t n_retry = 0, n_wait = 0, n_pend = 0, n_poll = 0;
    bool ok = true;
    // Counter `warp` hands out tiles warp, warp + 8, ... in increasing order.
    // Let T* be the lowest unfinished tile.  If it is claimed, its warp is
    // working on it (a warp holds one tile at a time) and every tile it reads
    // is lower, hence finished: it progresses.  If not, every tile its counter has handed out is lower,
    // hence finished, so the warps of that counter are free and the next of
    // them to claim takes T*.  Any resident block has a warp on every counter,
    // so this holds for any grid.
    unsigned long long *my_ticket = b.ticket + 16 * warp;
    while (ok) {
        unsigned long long c = 0;
        if (L.lane == 0) c = atomicAdd(my_ticket, 1ull);
        c = __shfl_sync(kFull, c, 0);
        const unsigned long long T = b.t_begin + c * kStartCounters + warp;
        if (T >= b.t_end) break;
        uint32_t i = 0;
        uint64_t t = T;
        if (b.count != 1) {
            const unsigned long long lo = s_seg[warp][0], hi = s_seg[warp][1];
            if (T >= lo && T < hi) {
                i = cur;   // the segment's graph is the one loaded
                t = s_seg[warp][2] + (T - lo);
            } else {
                unsigned long long nlo, nhi, t0;
                map_unit_seg(b.tab, b.count, T, i, nlo, nhi, t0);
                t = t0 + (T - nlo);
                __syncwarp();
                if (L.lane == 0) {
                    s_seg[warp][0] = nlo;
                    s_seg[warp][1] = nhi;
                    s_seg[warp][2] = t0;
                }
                __syncwarp();
            }
        }
        if (i != cur) {
            __syncwarp();
            const uint32_t *src = reinterpret_cast<const uint32_t *>(b.inst + i);
            uint32_t *dst = reinterpret_cast<uint32_t *>(&a);
            for (uint32_t w = L.lane; w < sizeof(GenArgs) / 4; w += 32) dst[w] = __ldg(src + w);
            __syncwarp();
            cur = i;
            set_lane(L, a);
        }
        Id *E = reinterpret_cast<Id *>(a.edges);
        const uint32_t tb = (uint32_t)(a.u_first + t * (P * a.groups));
        Slot<uint32_t> s[P];
        if constexpr (P == 1 || (P == kStartPasses && MinBlocks == kStartMinBlocks)) {
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const uint32_t pbase = tb + j * a.groups;
                const uint32_t u = pbase + L.g;
                s[j].val = 0;
                s[j].meta = ST_KNOWN;
                if (L.used && u < a.start_end)
                    classify_start<Id, Slots>(s[j], draw<uint32_t>(u, L.slot, 0u, a), 0u, a, E,
                                              pbase, n_pend);
            }
        } else {
            // the passes' first reads go out together, so that a tile waits for one
            // memory latency and not for one per pass
            uint32_t x[P];
            uint32_t reads = 0;   // bit j: pass j's slot of this lane is read
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const uint32_t pbase = tb + j * a.groups;
                const uint32_t u = pbase + L.g;
                s[j].val = 0;
                s[j].meta = ST_KNOWN;
                if (L.used && u < a.start_end &&
                    place_start(s[j], draw<uint32_t>(u, L.slot, 0u, a), 0u, a, pbase))
                    reads |= 1u << j;
            }
            if constexpr (Hop) {
                uint32_t cand = 0;   // bit j: pass j's copy is of an earlier launch's slot
#pragma unroll
                for (int j = 0; j < P; ++j)
                    if (((reads >> j) & 1u) && s[j].val < b.hop_end) cand |= 1u << j;
                const uint32_t bit = cand & (0u - cand);
                Slot<uint32_t> q = s[0];
#pragma unroll
                for (int j = 1; j < P; ++j)
                    if (bit == 1u << j) q = s[j];
                const uint32_t h = hop_bit(q.val, meta_k(q.meta), a.d);
                const DrawT<uint32_t> dr = draw<uint32_t>(q.val, meta_k(q.meta), 0u, a);
                if (bit != 0u && ((s_rejected[h >> 5] >> (h & 31u)) & 1u) == 0u) {
                    if (!place_start(q, dr, 0u, a, b.hop_end)) reads ^= bit;
#pragma unroll
                    for (int j = 0; j < P; ++j)
                        if (bit == 1u << j) s[j] = q;
                }
            }
#pragma unroll
            for (int j = 0; j < P; ++j)
                if ((reads >> j) & 1u)
                    x[j] = (uint32_t)ld_slot(
                        slot_addr<Id, uint32_t, Slots>(E, a, s[j].val, meta_k(s[j].meta)));
#pragma unroll
            for (int j = 0; j < P; ++j)
                if ((reads >> j) & 1u) {
                    // values are below 2^31: the low word tells the fill
                    if (x[j] != 0xffffffffu) {
                        s[j].val = x[j];
                    } else {
                        s[j].meta |= ST_PEND_GLOBAL;
                        ++n_pend;
                    }
                }
        }
        constexpr bool kLatency = P == 1 && MinBlocks == kStartMinBlocksMid;
        const bool withhold = a.withhold_first && t == 0;
        const uint32_t done = store_settled<Id, Slots, P>(s, a, E, tb, withhold, L);
        if (done != (1u << P) - 1u)
            ok = resolve_start<Id, Slots, P, kLatency, Hop>(s, a, E, tb, withhold, L, done,
                                                            b.rejected, n_retry, n_wait,
                                                            n_pend, n_poll);
    }

#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        n_retry += __shfl_down_sync(kFull, n_retry, o);
        n_pend += __shfl_down_sync(kFull, n_pend, o);
        n_poll += __shfl_down_sync(kFull, n_poll, o);
    }
    if (L.lane == 0) {
        if (n_pend) atomicAdd(&b.ctl->pending_reads, (unsigned long long)n_pend);
        if (n_poll) atomicAdd(&b.ctl->pending_polls, (unsigned long long)n_poll);
        if (n_retry) atomicAdd(&b.ctl->retries, (unsigned long long)n_retry);
        if (n_wait) atomicAdd(&b.ctl->waits, (unsigned long long)n_wait);
    }
}

// All-ones over the start-region pairs of graph blockIdx.y (+ y0), 16 bytes per
// store.  Pair regions start 16-byte aligned for 64-bit ids; for 32-bit ids the
// region's ragged 8-byte ends are written separately.
__global__ void fill_start_kernel(const GenArgs *inst, uint32_t y0, uint32_t id_bytes)
{
    const GenArgs &a = inst[y0 + blockIdx.y];
    const uint64_t pair_bytes = 2ull * id_bytes;
    const uint64_t n_pairs = (a.start_end - a.u_first) * a.d;
    unsigned char *base = reinterpret_cast<unsigned char *>(a.edges) + a.seed_edges * pair_bytes;
    uint64_t lo = 0, hi = n_pairs * pair_bytes;
    if (hi == 0) return;
    const uint64_t mis = reinterpret_cast<uintptr_t>(base) & 15u;   // 0 or 8
    if (mis) {
        if (blockIdx.x == 0 && threadIdx.x == 0)
            *reinterpret_cast<unsigned long long *>(base) = ~0ull;
        lo = 16 - mis;
    }
    if ((hi - lo) & 15u) {
        if (blockIdx.x == 0 && threadIdx.x == 0)
            *reinterpret_cast<unsigned long long *>(base + hi - 8) = ~0ull;
        hi -= 8;
    }
    uint4 *p = reinterpret_cast<uint4 *>(base + lo);
    const uint64_t n16 = (hi - lo) >> 4;
    const uint4 ones = make_uint4(~0u, ~0u, ~0u, ~0u);
    for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n16;
         x += (uint64_t)gridDim.x * blockDim.x)
        p[x] = ones;
}

template <typename Id, bool Slots, uint32_t MinBlocks, int P, bool Hop>
int launch_start_t(const StartArgs &b, uint32_t blocks, cudaStream_t s)
{
    auto kern = start_kernel<Id, Slots, MinBlocks, P, Hop>;
    if (blocks == 0) {
        int dev = 0, sms = 0, per_sm = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, (int)kThreads, 0);
        if (e != cudaSuccess) return set_cuda_error(e);
        uint64_t g = (uint64_t)sms * (uint64_t)(per_sm > 0 ? per_sm : 1);
        // no more warps than start tiles (but one block at least, for the seed edges)
        const uint64_t need = (b.t_end - b.t_begin + kThreads / 32 - 1) / (kThreads / 32);
        if (need < g) g = need > 0 ? need : 1;
        blocks = (uint32_t)g;
    }
    // launched while the kernel before it (the control block's and the fill's, of a
    // small graph) still runs; start_kernel waits for its end
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, b);
    return e == cudaSuccess ? PA_OK : set_cuda_error(e);
}

}  // namespace

template <uint32_t MinBlocks, int P, bool Hop = false>
int launch_start_m(uint32_t id_bytes, const StartArgs &b, uint32_t blocks, cudaStream_t s,
                   bool slots)
{
    if (slots)
        return id_bytes == 8 ? launch_start_t<int64_t, true, MinBlocks, P, Hop>(b, blocks, s)
                             : launch_start_t<int32_t, true, MinBlocks, P, Hop>(b, blocks, s);
    return id_bytes == 8 ? launch_start_t<int64_t, false, MinBlocks, P, Hop>(b, blocks, s)
                         : launch_start_t<int32_t, false, MinBlocks, P, Hop>(b, blocks, s);
}

int launch_start(uint32_t id_bytes, const StartArgs &b, uint32_t blocks, cudaStream_t s,
                 bool slots, StartVariant v)
{
    if (v.passes == 1)
        return v.min_blocks == kStartMinBlocksMany
                   ? launch_start_m<kStartMinBlocksMany, 1>(id_bytes, b, blocks, s, slots)
                   : launch_start_m<kStartMinBlocksMid, 1>(id_bytes, b, blocks, s, slots);
    if (v.hop)
        return launch_start_m<kStartMinBlocksMid, kStartPasses, true>(id_bytes, b, blocks, s, slots);
    if (v.passes == 2) return launch_start_m<kStartMinBlocks, 2>(id_bytes, b, blocks, s, slots);
    if (v.min_blocks == kStartMinBlocksMid)
        return launch_start_m<kStartMinBlocksMid, kStartPasses>(id_bytes, b, blocks, s, slots);
    return launch_start_m<kStartMinBlocks, kStartPasses>(id_bytes, b, blocks, s, slots);
}

int fill_start(uint32_t id_bytes, const GenArgs *d_inst, uint32_t count, uint64_t max_pairs,
               cudaStream_t s)
{
    if (count == 0 || max_pairs == 0) return PA_OK;
    const uint64_t n16 = max_pairs * 2ull * id_bytes / 16 + 1;
    // 16 stores a thread for the largest graph: with one, the blocks of many small
    // graphs, most of them with nothing to do, took longer than the stores (a call
    // of 512 graphs of 10^3..10^5 nodes 6.7 -> 5.5 ms)
    const uint32_t gx = (uint32_t)std::min<uint64_t>(4096, (n16 + 4095) / 4096);
    for (uint32_t y0 = 0; y0 < count; y0 += 65535) {
        const uint32_t gy = std::min<uint32_t>(65535, count - y0);
        fill_start_kernel<<<dim3(gx, gy), 256, 0, s>>>(d_inst, y0, id_bytes);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return set_cuda_error(e);
    }
    return PA_OK;
}

}  // namespace gen
}  // namespace pa
