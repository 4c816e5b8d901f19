// Batched visibility lookups against resident DAGs.
//
// Replaces CompressedShadow::traverse (src/CompressedShadow.cpp:394-463) and
// the per-pixel descent of shader/traverse.cs:41-133.  One thread per query:
// quantise the NDC point with the reference's float32 order
// (src/CompressedShadowUtil.h:70-75: +1, *0.5, *(R-1), truncate), descend
// from the root choosing child x|y<<1|z<<2 from bit `level` of the path,
// stop at a lit or shadowed child, and finish in the 64-bit leafmask.  The
// answer of 32 consecutive queries is packed by one ballot into one word.
//
// The descent is a chain of dependent L1/L2 hits (an 8192^2 map's DAG is
// 9.4 MB), so every hop is kept short -- 32-bit offsets, one bounds check
// per node (DAG buffers carry a zeroed tail of kDagPad words, so both reads
// of a node stay inside the buffer once its offset is), and the child's
// 2-bit class and rank from one shift and one popcount.  The first `depth`
// levels below the root are replaced by a dense 3-D "top grid" of
// (2^depth)^3 words, indexed by the top `depth` bits of the quantised x, y,
// z: the node offset the descent reaches after those levels, or a lit /
// shadow sentinel.  It lives in global memory (L2-resident; up to 8 levels,
// at most 8x the DAG's size or, for a large first batch, a cell per two of its
// points), so one load replaces up to 8 dependent hops --
// and each thread carries Q independent queries (one, or for batches of
// several waves picked per levels below the grid and input kind, device or host
// memory, by timing Q = 1, 2, 4 on the first of them).  A leafmask DAG with a top grid and few levels below it takes
// k_lookup_fixed (the levels unrolled, 32-bit indices); any other DAG
// k_lookup.  Query points and answer words are touched once, so they go
// through the caches evict-first (ld/st .cs): a batch streams hundreds of MB
// past L2 and would otherwise push the DAG and its top grid out of it.  The
// grid lookups and evaluate (k_grid_lookup, k_grid_evaluate) route through
// the grid's cells and a grid index the same way.
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace cpvs {
namespace {

constexpr int kThreads = 256;
constexpr uint32_t kCellShadow = 0xFFFFFFFFu, kCellLit = 0xFFFFFFFEu;

__device__ __forceinline__ int32_t quantise(float v, float scale) {
    const float t = __fmul_rn(__fadd_rn(v, 1.0f), 0.5f);
    return __float2int_rz(__fmul_rn(t, scale));
}

// 2 * child index at `level`: bit `level` of x, y, z at weights 2, 4, 8.
__device__ __forceinline__ uint32_t child2(int32_t px, int32_t py, int32_t pz, int level) {
    return (((uint32_t)px >> level) & 1u) * 2u + (((uint32_t)py >> level) & 1u) * 4u +
           (((uint32_t)pz >> level) & 1u) * 8u;
}

// Descent from node `off` at `level` down to the leafmask, pointers relative
// to `base` (the DAG's first word).  Returns true when the voxel is lit.  A
// node offset outside the DAG (a malformed buffer) answers "shadow".
__device__ __forceinline__ bool descend(const uint32_t* __restrict__ dag, uint32_t words, uint32_t base,
                                        uint32_t off, int level, int min_level, bool leafmasks, int32_t px,
                                        int32_t py, int32_t pz) {
    for (; level >= min_level; --level) {
        if (off >= words) return false;
        const uint32_t c2 = child2(px, py, pz, level);
        const uint32_t m = __ldg(dag + off);
        const uint32_t v = (m >> c2) & 3u;
        if (v != kPartial) return v == kVisible;
        // rank among partial children = popcount of the partial bits below c2
        const uint32_t rank = __popc(m & 0xAAAAu & ((1u << c2) - 1u));
        off = base + __ldg(dag + off + 1u + rank);
    }
    if (!leafmasks) return true;  // unreachable: level 0 has no partial children
    if (off >= words) return false;
    const uint32_t c2 = ((uint32_t)pz & 7u) * 2u;
    const uint32_t m = __ldg(dag + off);
    const uint32_t v = (m >> c2) & 3u;
    if (v != kPartial) return v == kVisible;
    const uint32_t rank = __popc(m & 0xAAAAu & ((1u << c2) - 1u));
    const uint32_t b = ((uint32_t)px & 7u) + 8u * ((uint32_t)py & 7u);
    const uint32_t w = __ldg(dag + off + 1u + 2u * rank + (b >> 5));
    return (w >> (b & 31u)) & 1u;
}

// descend() for a leafmask DAG whose NL inner levels above the leaves are
// known at compile time (the levels below a grid index): the same reads and
// checks, unrolled, with constant shifts.
template <int NL>
__device__ __forceinline__ bool descend_fixed(const uint32_t* __restrict__ dag, uint32_t words, uint32_t base,
                                              uint32_t off, int32_t px, int32_t py, int32_t pz) {
#pragma unroll
    for (int s = 0; s < NL; ++s) {
        const int level = 3 + NL - 1 - s;
        if (off >= words) return false;
        const uint32_t c2 = child2(px, py, pz, level);
        const uint32_t m = __ldg(dag + off);
        const uint32_t v = (m >> c2) & 3u;
        if (v != kPartial) return v == kVisible;
        off = base + __ldg(dag + off + 1u + __popc(m & 0xAAAAu & ((1u << c2) - 1u)));
    }
    if (off >= words) return false;
    const uint32_t c2 = ((uint32_t)pz & 7u) * 2u;
    const uint32_t m = __ldg(dag + off);
    const uint32_t v = (m >> c2) & 3u;
    if (v != kPartial) return v == kVisible;
    const uint32_t rank = __popc(m & 0xAAAAu & ((1u << c2) - 1u));
    const uint32_t b = ((uint32_t)px & 7u) + 8u * ((uint32_t)py & 7u);
    const uint32_t w = __ldg(dag + off + 1u + 2u * rank + (b >> 5));
    return (w >> (b & 31u)) & 1u;
}

// The 64 voxels of leaf slice `pz` & 7 under the node at `off`: bit x + 8 y
// set where the voxel is lit (a whole lit or shadowed node or slice: all or
// none).  The same reads and checks as descend() and descend_fixed(); NL as
// there, -1 for a descent from `level`.
template <int NL>
__device__ __forceinline__ uint64_t leaf_slice(const uint32_t* __restrict__ dag, uint32_t words, uint32_t base,
                                               uint32_t off, int level, int32_t px, int32_t py, int32_t pz) {
    if constexpr (NL > 0) level = 3 + NL - 1;
    if constexpr (NL != 0) {
#pragma unroll
        for (; level >= 3; --level) {
            if (off >= words) return 0ull;
            const uint32_t c2 = child2(px, py, pz, level);
            const uint32_t m = __ldg(dag + off);
            const uint32_t v = (m >> c2) & 3u;
            if (v != kPartial) return v == kVisible ? ~0ull : 0ull;
            off = base + __ldg(dag + off + 1u + __popc(m & 0xAAAAu & ((1u << c2) - 1u)));
        }
    }
    if (off >= words) return 0ull;
    const uint32_t c2 = ((uint32_t)pz & 7u) * 2u;
    const uint32_t m = __ldg(dag + off);
    const uint32_t v = (m >> c2) & 3u;
    if (v != kPartial) return v == kVisible ? ~0ull : 0ull;
    const uint32_t* w = dag + off + 1u + 2u * __popc(m & 0xAAAAu & ((1u << c2) - 1u));
    return __ldg(w) | ((uint64_t)__ldg(w + 1) << 32);
}

// Top grid: cell (cx, cy, cz) at index (cz << 2 depth) | (cy << depth) | cx
// holds the node offset the descent reaches after the `depth` levels below
// the root whose child bits are those of cx, cy, cz (most significant
// first), or a sentinel when it ended in a lit or shadowed child on the way.
__device__ __forceinline__ uint32_t top_cell(int32_t px, int32_t py, int32_t pz, int shift, int depth) {
    const uint32_t m = (1u << depth) - 1u;
    return ((((uint32_t)pz >> shift) & m) << (2 * depth)) | ((((uint32_t)py >> shift) & m) << depth) |
           (((uint32_t)px >> shift) & m);
}

// One thread per cell of depth `depth` - 1: its descent, then the eight
// cells below it from one mask load and up to eight independent pointer
// loads (neighbouring cells share all but their last level, so walking
// each cell alone would repeat the same chain eight times).
//
// A launch takes the top grids of up to kTopBatch DAGs, entry e's from block
// `first` on: a small DAG's grid is one descent's latency on a few SMs (6 to 7
// us of a chain of 2 * depth dependent loads, 16 of them one after the other
// 105 us), so the grids of a batch of lights are made side by side.
constexpr int kTopBatch = 64;
struct TopJob {
    const uint32_t* dag;
    uint32_t* out;
    uint32_t words, first;
    int depth;
};
struct TopJobs {
    TopJob j[kTopBatch];
    uint32_t count;
};

__global__ void __launch_bounds__(kThreads) k_top_index(const __grid_constant__ TopJobs tab) {
    uint32_t lo = 0, hi = tab.count;  // the last entry whose first block is <= blockIdx.x
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (tab.j[mid].first <= blockIdx.x) lo = mid; else hi = mid;
    }
    const uint32_t* __restrict__ dag = tab.j[lo].dag;
    uint32_t* __restrict__ out = tab.j[lo].out;
    const uint32_t words = tab.j[lo].words;
    const int depth = tab.j[lo].depth, dp = depth - 1;
    const uint32_t pc = (blockIdx.x - tab.j[lo].first) * kThreads + threadIdx.x;
    if (pc >= 1u << (3 * dp)) return;
    const uint32_t pm = (1u << dp) - 1u;
    const uint32_t px = pc & pm, py = (pc >> dp) & pm, pz = pc >> (2 * dp);
    uint32_t off = 0, entry = 0;
    bool done = false;
    for (int d = 0; d < dp; ++d) {
        const int b = dp - 1 - d;
        const uint32_t c = ((px >> b) & 1u) | (((py >> b) & 1u) << 1) | (((pz >> b) & 1u) << 2);
        if (off >= words) {
            entry = kCellShadow;
            done = true;
            break;
        }
        const uint32_t m = dag[off];
        const uint32_t v = (m >> (2u * c)) & 3u;
        if (v != kPartial) {
            entry = (v == kVisible) ? kCellLit : kCellShadow;
            done = true;
            break;
        }
        off = dag[off + 1u + __popc(m & 0xAAAAu & ((1u << (2u * c)) - 1u))];
    }
    uint32_t m = 0;
    if (!done) {
        if (off >= words) {
            entry = kCellShadow;
            done = true;
        } else {
            m = dag[off];
        }
    }
    // x neighbours as one 8-byte store (the grid is 256-byte aligned, 2 px even)
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
        uint32_t e[2];
#pragma unroll
        for (uint32_t x = 0; x < 2; ++x) {
            const uint32_t c = 2u * r + x;
            e[x] = entry;
            if (!done) {
                const uint32_t v = (m >> (2u * c)) & 3u;
                e[x] = v == kPartial ? dag[off + 1u + __popc(m & 0xAAAAu & ((1u << (2u * c)) - 1u))]
                                     : (v == kVisible ? kCellLit : kCellShadow);
            }
        }
        const uint32_t cy = 2u * py + (r & 1u), cz = 2u * pz + (r >> 1);
        *reinterpret_cast<uint2*>(out + ((cz << (2 * depth)) | (cy << depth) | (2u * px))) = make_uint2(e[0], e[1]);
    }
}

// Q queries per thread, carried through the levels in lockstep so that each
// level issues Q independent loads (the descent is a chain of dependent
// L1/L2 hits, so memory-level parallelism per thread sets the rate).  Query
// q of a thread is i = (w*Q + q)*32 + lane: each of the Q ballots packs 32
// consecutive queries into one output word.
template <bool NDC, int Q>
__global__ void __launch_bounds__(kThreads)
    k_lookup(const uint32_t* __restrict__ dag, uint32_t words, int num_levels, bool leafmasks,
             const uint32_t* __restrict__ top, int depth, const void* __restrict__ q, uint64_t n,
             uint32_t* __restrict__ bits) {
    const int lane = threadIdx.x & 31;
    const int root = num_levels - 2, min_level = leafmasks ? 3 : 0;
    const int shift = root - depth + 1;  // the top grid takes bits root .. shift of each coordinate
    const uint64_t nwords = (n + 31) / 32;
    const uint64_t ngroups = (nwords + Q - 1) / Q;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const float scale = (float)((1u << (num_levels - 1)) - 1u);
    if (Q == 1) {
        // one query per thread, each descending on its own; the point of the
        // thread's next query is requested before the current one descends
        uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        uint32_t nx = 0, ny = 0, nz = 0;
        auto fetch = [&](uint64_t wq) {
            const uint64_t iq = wq * 32 + (uint64_t)lane;
            if (wq < nwords && iq < n) {
                const uint32_t* p = static_cast<const uint32_t*>(q) + 3 * iq;
                nx = __ldcs(p);
                ny = __ldcs(p + 1);
                nz = __ldcs(p + 2);
            }
        };
        fetch(w);
        for (; w < nwords; w += nw) {
            const uint64_t i = w * 32 + (uint64_t)lane;
            const uint32_t rx = nx, ry = ny, rz = nz;
            fetch(w + nw);
            bool lit = false;
            if (i < n) {
                int32_t px, py, pz;
                if (NDC) {
                    px = quantise(__uint_as_float(rx), scale);
                    py = quantise(__uint_as_float(ry), scale);
                    pz = quantise(__uint_as_float(rz), scale);
                } else {
                    px = (int32_t)rx;
                    py = (int32_t)ry;
                    pz = (int32_t)rz;
                }
                uint32_t off = 0;
                int level = root;
                bool done = false;
                if (depth > 0) {
                    const uint32_t e = __ldg(top + top_cell(px, py, pz, shift, depth));
                    if (e >= kCellLit) {
                        lit = (e == kCellLit);
                        done = true;
                    } else {
                        off = e;
                        level = root - depth;
                    }
                }
                if (!done) lit = descend(dag, words, 0u, off, level, min_level, leafmasks, px, py, pz);
            }
            const uint32_t word = __ballot_sync(0xffffffffu, lit);
            if (lane == 0) __stcs(bits + w, word);
        }
        return;
    }
    for (uint64_t gidx = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; gidx < ngroups; gidx += nw) {
        int32_t px[Q], py[Q], pz[Q];
        uint32_t off[Q];
        bool done[Q], lit[Q];
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const uint64_t i = (gidx * Q + k) * 32 + (uint64_t)lane;
            done[k] = true;
            lit[k] = false;
            off[k] = 0;
            px[k] = py[k] = pz[k] = 0;
            if (i < n) {
                if (NDC) {
                    const float* p = static_cast<const float*>(q) + 3 * i;
                    px[k] = quantise(__ldcs(p), scale);
                    py[k] = quantise(__ldcs(p + 1), scale);
                    pz[k] = quantise(__ldcs(p + 2), scale);
                } else {
                    const int32_t* p = static_cast<const int32_t*>(q) + 3 * i;
                    px[k] = __ldcs(p);
                    py[k] = __ldcs(p + 1);
                    pz[k] = __ldcs(p + 2);
                }
                done[k] = false;
            }
        }
        int level = root;
        if (depth > 0) {
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                if (done[k]) continue;
                const uint32_t e = __ldg(top + top_cell(px[k], py[k], pz[k], shift, depth));
                if (e >= kCellLit) {
                    lit[k] = (e == kCellLit);
                    done[k] = true;
                } else {
                    off[k] = e;
                }
            }
            level = root - depth;
        }
        for (; level >= min_level; --level) {
            uint32_t m[Q];
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                if (!done[k] && off[k] >= words) {
                    done[k] = true;  // malformed DAG: shadow
                    lit[k] = false;
                }
                m[k] = done[k] ? 0u : __ldg(dag + off[k]);
            }
            uint32_t slot[Q];
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                slot[k] = 0;
                if (done[k]) continue;
                const uint32_t c2 = child2(px[k], py[k], pz[k], level);
                const uint32_t v = (m[k] >> c2) & 3u;
                if (v != kPartial) {
                    lit[k] = (v == kVisible);
                    done[k] = true;
                } else {
                    slot[k] = off[k] + 1u + __popc(m[k] & 0xAAAAu & ((1u << c2) - 1u));
                }
            }
            bool any = false;
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                if (!done[k]) off[k] = __ldg(dag + slot[k]);
                any |= !done[k];
            }
            if (!__any_sync(0xffffffffu, any)) break;
        }
        if (leafmasks) {
            uint32_t m[Q];
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                if (!done[k] && off[k] >= words) {
                    done[k] = true;
                    lit[k] = false;
                }
                m[k] = done[k] ? 0u : __ldg(dag + off[k]);
            }
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                if (done[k]) continue;
                const uint32_t c2 = ((uint32_t)pz[k] & 7u) * 2u;
                const uint32_t v = (m[k] >> c2) & 3u;
                if (v != kPartial) {
                    lit[k] = (v == kVisible);
                } else {
                    const uint32_t rank = __popc(m[k] & 0xAAAAu & ((1u << c2) - 1u));
                    const uint32_t b = ((uint32_t)px[k] & 7u) + 8u * ((uint32_t)py[k] & 7u);
                    const uint32_t w = __ldg(dag + off[k] + 1u + 2u * rank + (b >> 5));
                    lit[k] = (w >> (b & 31u)) & 1u;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const uint32_t word = __ballot_sync(0xffffffffu, lit[k]);
            const uint64_t wi = gidx * Q + k;
            if (lane == 0 && wi < nwords) __stcs(bits + wi, word);
        }
    }
}

// The common case in straight-line code: a leafmask DAG with a top grid
// and NL inner levels below it (the c1 workload: levels 4 and 3), fewer
// than 2^31 queries.  The levels are unrolled, each query carries an
// `alive` flag instead of leaving a loop, and indices are 32-bit, so a
// query costs fewer instructions than in k_lookup; Q queries per thread are
// interleaved level by level, so each level issues Q independent loads with
// no lockstep loop around them.  The next group's points are requested
// before the current group descends.  Same answers as k_lookup: every node
// offset is checked against `words` before its mask is read, and the zeroed
// tail keeps a node's pointer and leaf words inside the buffer.
template <bool NDC, int Q, int NL>
__global__ void __launch_bounds__(kThreads)
    k_lookup_fixed(const uint32_t* __restrict__ dag, uint32_t words, int num_levels, const uint32_t* __restrict__ top,
                   int depth, const void* __restrict__ q, uint32_t n, uint32_t* __restrict__ bits) {
    const uint32_t lane = threadIdx.x & 31u;
    const int root = num_levels - 2;
    const int shift = root - depth + 1;  // the top grid takes bits root .. shift of each coordinate
    const int low = shift - NL;          // bit of the last inner level (3)
    const uint32_t nwords = (n + 31u) / 32u;
    const uint32_t ngroups = (nwords + Q - 1u) / Q;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const float scale = (float)((1u << (num_levels - 1)) - 1u);
    uint32_t nx[Q] = {}, ny[Q] = {}, nz[Q] = {};
    auto fetch = [&](uint32_t g) {
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const uint32_t i = (g * Q + k) * 32u + lane;
            if (g < ngroups && i < n) {
                const uint32_t* p = static_cast<const uint32_t*>(q) + 3u * (size_t)i;
                nx[k] = __ldcs(p);
                ny[k] = __ldcs(p + 1);
                nz[k] = __ldcs(p + 2);
            }
        }
    };
    uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    fetch(g);
    for (; g < ngroups; g += nw) {
        // this group's points, then the next group's requested before these
        // are used (two groups' reads in flight while a point arrives)
        uint32_t rx[Q], ry[Q], rz[Q];
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            rx[k] = nx[k];
            ry[k] = ny[k];
            rz[k] = nz[k];
        }
        fetch(g + nw);
        int32_t px[Q], py[Q], pz[Q];
        uint32_t off[Q];
        bool alive[Q], lit[Q];
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const uint32_t i = (g * Q + k) * 32u + lane;
            if (NDC) {
                px[k] = quantise(__uint_as_float(rx[k]), scale);
                py[k] = quantise(__uint_as_float(ry[k]), scale);
                pz[k] = quantise(__uint_as_float(rz[k]), scale);
            } else {
                px[k] = (int32_t)rx[k];
                py[k] = (int32_t)ry[k];
                pz[k] = (int32_t)rz[k];
            }
            alive[k] = i < n;
            lit[k] = false;
            off[k] = 0;
        }
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const uint32_t e = alive[k] ? __ldg(top + top_cell(px[k], py[k], pz[k], shift, depth)) : kCellShadow;
            if (e >= kCellLit) {
                lit[k] = alive[k] && e == kCellLit;
                alive[k] = false;
            } else {
                off[k] = e;
            }
        }
#pragma unroll
        for (int s = 0; s < NL; ++s) {
            const int b = NL - 1 - s;  // this level's bit above `low`
            uint32_t m[Q];
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                if (alive[k] && off[k] >= words) alive[k] = false;  // malformed DAG: shadow
                m[k] = alive[k] ? __ldg(dag + off[k]) : 0u;
            }
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                if (!alive[k]) continue;
                const uint32_t c2 = child2(px[k] >> low, py[k] >> low, pz[k] >> low, b);
                const uint32_t v = (m[k] >> c2) & 3u;
                if (v != kPartial) {
                    lit[k] = v == kVisible;
                    alive[k] = false;
                } else {
                    off[k] = __ldg(dag + off[k] + 1u + __popc(m[k] & 0xAAAAu & ((1u << c2) - 1u)));
                }
            }
        }
        // the leaf: slice z & 7, bit (x & 7) + 8 (y & 7) of its mask pair
        uint32_t m[Q];
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            if (alive[k] && off[k] >= words) alive[k] = false;
            m[k] = alive[k] ? __ldg(dag + off[k]) : 0u;
        }
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            if (alive[k]) {
                const uint32_t c2 = ((uint32_t)pz[k] & 7u) * 2u;
                const uint32_t v = (m[k] >> c2) & 3u;
                if (v != kPartial) {
                    lit[k] = v == kVisible;
                } else {
                    const uint32_t rank = __popc(m[k] & 0xAAAAu & ((1u << c2) - 1u));
                    const uint32_t bb = ((uint32_t)px[k] & 7u) + 8u * ((uint32_t)py[k] & 7u);
                    lit[k] = (__ldg(dag + off[k] + 1u + 2u * rank + (bb >> 5)) >> (bb & 31u)) & 1u;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const uint32_t word = __ballot_sync(0xffffffffu, lit[k]);
            const uint32_t wi = g * Q + k;
            if (lane == 0 && wi < nwords) __stcs(bits + wi, word);
        }
    }
}

// Grid routing at an integer path (shader/traverse.cs:75-88): outside the
// grid answers lit, a uniform cell its class, else the descent of the cell's
// DAG with pointers relative to its first word.  With a grid top index
// (`top`, `depth` levels of every cell DAG; see k_grid_top_index) the first
// levels are one load.  The path is kept in 32 bits: a side has at most 2^24
// voxels, and a coordinate outside, seen unsigned, has a bit above the side's.
struct GridRoute {
    const uint32_t* dag;
    const uint32_t* cells;
    const uint32_t* top;  // null: none
    uint32_t words;
    int gl;          // log2(length)
    int sh;          // path bits within a cell: dag_levels - 1
    int depth;       // levels of each cell DAG that `top` resolves (0: none)
    bool leafmasks;
};

// Where the descent of a path inside the grid begins: false when the path
// ends above it in a class (`lit`), else the node and the cell's first word.
template <int NL>
__device__ __forceinline__ bool grid_enter(const GridRoute& G, uint32_t px, uint32_t py, uint32_t pz, bool& lit,
                                           uint32_t& base, uint32_t& off, int& level) {
    base = __ldg(G.cells + (((pz >> G.sh) << (2 * G.gl)) | ((py >> G.sh) << G.gl) | (px >> G.sh)));
    off = base;
    level = G.sh - 1 - G.depth;
    if (NL >= 0 || G.top) {
        const int s = G.sh - G.depth, bits = G.gl + G.depth;
        off = __ldg(G.top + (((pz >> s) << (2 * bits)) | ((py >> s) << bits) | (px >> s)));
    }
    lit = off == kCellLit;
    return off < kCellLit;  // else a uniform cell, or the descent ended in the top levels
}

// NL >= 0: a leafmask grid with an index, NL inner levels below it
// (descend_fixed); -1: any grid.
template <int NL>
__device__ __forceinline__ bool grid_sample(const GridRoute& G, int32_t px, int32_t py, int32_t pz) {
    if (((uint32_t)px | (uint32_t)py | (uint32_t)pz) >> (G.sh + G.gl)) return true;
    bool lit;
    uint32_t base, off;
    int level;
    if (!grid_enter<NL>(G, (uint32_t)px, (uint32_t)py, (uint32_t)pz, lit, base, off, level)) return lit;
    if constexpr (NL >= 0) return descend_fixed<NL>(G.dag, G.words, base, off, px, py, pz);
    return descend(G.dag, G.words, base, off, level, G.leafmasks ? 3 : 0, G.leafmasks, px, py, pz);
}

// Lit samples of the footprint [px + lo, px + hi] x [py + lo, py + hi] at
// depth voxel pz; samples outside the grid are lit.  In a leafmask grid the
// footprint is taken leaf by leaf: its samples in one 8x8 leaf column share
// the descent and the slice, so they are one mask and one popcount (3x3: 1.6
// descents on average instead of 9).
template <int NL>
__device__ __forceinline__ uint32_t grid_footprint(const GridRoute& G, int32_t px, int32_t py, int32_t pz, int lo,
                                                   int hi) {
    const int f = hi - lo + 1;
    const int32_t lim = 1 << (G.sh + G.gl);
    if ((uint32_t)pz >= (uint32_t)lim) return (uint32_t)(f * f);
    // a far coordinate's whole footprint (offsets within 16) stays outside
    px = min(max(px, -64), lim + 64);
    py = min(max(py, -64), lim + 64);
    const int32_t x0 = max(px + lo, 0), x1 = min(px + hi, lim - 1), y0 = max(py + lo, 0), y1 = min(py + hi, lim - 1);
    if (x0 > x1 || y0 > y1) return (uint32_t)(f * f);
    uint32_t cnt = (uint32_t)(f * f - (x1 - x0 + 1) * (y1 - y0 + 1));
    if (NL < 0 && !G.leafmasks) {
        for (int32_t y = y0; y <= y1; ++y)
            for (int32_t x = x0; x <= x1; ++x) cnt += grid_sample<NL>(G, x, y, pz) ? 1u : 0u;
        return cnt;
    }
    for (int32_t ly = y0 >> 3; ly <= y1 >> 3; ++ly) {
        // the footprint's rows and columns in this leaf
        const int ra = max(y0 - 8 * ly, 0), rb = min(y1 - 8 * ly, 7);
        const uint64_t rows = (~0ull >> (8 * (7 - rb + ra))) << (8 * ra);
        for (int32_t lx = x0 >> 3; lx <= x1 >> 3; ++lx) {
            const int ca = max(x0 - 8 * lx, 0), cb = min(x1 - 8 * lx, 7);
            const uint32_t cols = (0xFFu >> (7 - cb + ca) << ca) * 0x01010101u;
            const uint64_t want = rows & (cols | ((uint64_t)cols << 32));
            bool lit;
            uint32_t base, off;
            int level;
            uint64_t s;
            if (grid_enter<NL>(G, (uint32_t)(8 * lx), (uint32_t)(8 * ly), (uint32_t)pz, lit, base, off, level))
                s = leaf_slice<NL>(G.dag, G.words, base, off, level, 8 * lx, 8 * ly, pz);
            else
                s = lit ? ~0ull : 0ull;
            cnt += (uint32_t)__popcll(s & want);
        }
    }
    return cnt;
}

// Grid top index: entry (gx, gy, gz) at index (gz << 2 bits) | (gy << bits) | gx,
// bits = log2(length) + depth, is the absolute DAG offset of the node that
// the cell's descent reaches after `depth` levels, or a lit / shadow sentinel
// (a uniform cell, or a lit / shadowed child on the way).
__global__ void k_grid_top_index(const uint32_t* __restrict__ dag, uint32_t words,
                                 const uint32_t* __restrict__ cells, uint32_t length, int dag_levels, int depth,
                                 int bits, uint32_t* __restrict__ out) {
    const uint64_t total = 1ull << (3 * bits);
    const uint32_t m = (1u << bits) - 1u;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t gx = (uint32_t)t & m, gy = (uint32_t)(t >> bits) & m, gz = (uint32_t)(t >> (2 * bits));
        const uint32_t cell = cells[((size_t)(gz >> depth) * length + (gy >> depth)) * length + (gx >> depth)];
        uint32_t entry;
        if (cell >= kCellLit) {
            entry = cell;
        } else {
            uint32_t off = cell;
            entry = 0;
            bool done = false;
            for (int d = 0; d < depth; ++d) {
                const int b = depth - 1 - d;
                const uint32_t c = ((gx >> b) & 1u) | (((gy >> b) & 1u) << 1) | (((gz >> b) & 1u) << 2);
                if (off >= words) {
                    entry = kCellShadow;
                    done = true;
                    break;
                }
                const uint32_t mk = dag[off];
                const uint32_t v = (mk >> (2u * c)) & 3u;
                if (v != kPartial) {
                    entry = (v == kVisible) ? kCellLit : kCellShadow;
                    done = true;
                    break;
                }
                off = cell + dag[off + 1u + __popc(mk & 0xAAAAu & ((1u << (2u * c)) - 1u))];
            }
            if (!done) entry = off;
        }
        out[t] = entry;
    }
}

// The same index from one thread per entry of resolution bits - 1 (depth
// >= 1): the descent to its node, then its eight entries from one mask load
// and up to eight independent pointer loads.
__global__ void k_grid_top_index_parents(const uint32_t* __restrict__ dag, uint32_t words,
                                         const uint32_t* __restrict__ cells, uint32_t length, int depth, int bits,
                                         uint32_t* __restrict__ out) {
    const int pb = bits - 1, dp = depth - 1;
    const uint64_t total = 1ull << (3 * pb);
    const uint32_t m = (1u << pb) - 1u;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t px = (uint32_t)t & m, py = (uint32_t)(t >> pb) & m, pz = (uint32_t)(t >> (2 * pb));
        const uint32_t cell = cells[((size_t)(pz >> dp) * length + (py >> dp)) * length + (px >> dp)];
        uint32_t entry = cell, off = cell, mk = 0;
        bool done = cell >= kCellLit;  // a uniform cell: every entry is its sentinel
        for (int d = 0; d < dp && !done; ++d) {
            const int b = dp - 1 - d;
            const uint32_t c = ((px >> b) & 1u) | (((py >> b) & 1u) << 1) | (((pz >> b) & 1u) << 2);
            if (off >= words) {
                entry = kCellShadow;
                done = true;
                break;
            }
            const uint32_t w = dag[off];
            const uint32_t v = (w >> (2u * c)) & 3u;
            if (v != kPartial) {
                entry = (v == kVisible) ? kCellLit : kCellShadow;
                done = true;
                break;
            }
            off = cell + dag[off + 1u + __popc(w & 0xAAAAu & ((1u << (2u * c)) - 1u))];
        }
        if (!done) {
            if (off >= words) {
                entry = kCellShadow;
                done = true;
            } else {
                mk = dag[off];
            }
        }
#pragma unroll
        for (uint32_t c = 0; c < 8; ++c) {
            uint32_t e = entry;
            if (!done) {
                const uint32_t v = (mk >> (2u * c)) & 3u;
                e = v == kPartial ? cell + dag[off + 1u + __popc(mk & 0xAAAAu & ((1u << (2u * c)) - 1u))]
                                  : (v == kVisible ? kCellLit : kCellShadow);
            }
            const uint64_t gx = 2ull * px + (c & 1u), gy = 2ull * py + ((c >> 1) & 1u), gz = 2ull * pz + (c >> 2);
            out[(gz << (2 * bits)) | (gy << bits) | gx] = e;
        }
    }
}

// Grid routing (shader/traverse.cs:75-88): the path at resolution
// 2^(dag_levels+grid_levels-1), its top bits select the cell, the cell word
// holds the DAG offset or a uniform-cell sentinel; then the cell's descent
// (grid_sample, with the grid top index when there is one).
template <int NL>
__global__ void __launch_bounds__(kThreads)
    k_grid_lookup(GridRoute G, const float* __restrict__ q, uint64_t n, uint32_t* __restrict__ bits) {
    const int lane = threadIdx.x & 31;
    const uint64_t nwords = (n + 31) / 32;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const float scale = (float)((1u << (G.sh + G.gl)) - 1u);
    for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nwords; w += nw) {
        const uint64_t i = w * 32 + (uint64_t)lane;
        bool lit = false;
        if (i < n) {
            const float* p = q + 3 * i;
            const int32_t px = quantise(__ldcs(p), scale), py = quantise(__ldcs(p + 1), scale), pz = quantise(__ldcs(p + 2), scale);
            lit = grid_sample<NL>(G, px, py, pz);
        }
        const uint32_t word = __ballot_sync(0xffffffffu, lit);
        if (lane == 0) __stcs(bits + w, word);
    }
}

// World-space evaluation (src/CompressedShadowContainer.cpp:93-124,
// shader/traverse.cs:134-148): pixel i's position p (the first three of its
// `fpp` floats) goes through the column-major light view-projection m as
// c_r = ((m[r]*x + m[4+r]*y) + m[8+r]*z) + m[12+r] (the shader's
// lightViewProj * vec4(p, 1), no contraction), ndc = c.xyz / c.w, then the
// grid lookup.  With filter f > 1, the f x f texel footprint around the
// path (offsets -(f-1)/2 .. f/2 in x and y, same depth voxel) is sampled and
// the lit fraction written as round(255 * lit / f^2) -- percentage-closer
// filtering, which the reference declares (setFilterSize) but never
// implements.  U8: one byte per pixel (0 / 255 when f <= 1, as an r8 image
// stores 0.0 / 1.0); else one bit per pixel, 32 per word.
struct EvalMatrix {
    float m[16];
};

//
// A G-buffer's neighbouring pixels see neighbouring voxels, so the descents
// mostly hit in L1 and the kernel is bound by instructions (180 a warp and
// pixel, 0.66 issued a cycle and scheduler): the path and the routing are in
// 32 bits, a position whose w is exactly 1 (every light with an orthographic
// projection) is not divided (x / 1 is x), and a filter's footprint is sampled
// leaf by leaf (grid_footprint; PCF).  A 3840x2160 G-buffer of an 8192^2
// light: 64 us against 99; 1920x1080 filtered 3x3: 50 us a call against 100.
//
// One pixel per thread and as many blocks as that takes (at most 2^30 pixels a
// launch), so a slow SM takes fewer blocks; a loop over one wave of blocks
// with the next position requested ahead cost 25 more instructions a pixel
// and left a quarter of the warps idle at its end.  The kernel alone against that
// loop, maps of 512^2 to 8192^2: 320x240 2.6 -> 2.1 us to 6.3 -> 5.9, 800x418
// 4.7 -> 3.5 to 10.6 -> 9.3, 1920x1080 19.9 -> 11.7 to 43.4 -> 32.3; a call takes
// 10 to 12 us of the host's time, which a frame below a million pixels hides in.
template <bool U8, int NL, bool PCF>
__global__ void __launch_bounds__(kThreads)
    k_grid_evaluate(GridRoute G, const float* __restrict__ pos, uint32_t fpp, uint32_t n, EvalMatrix M, int filter,
                    void* __restrict__ out) {
    const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    const float scale = (float)((1u << (G.sh + G.gl)) - 1u);
    bool lit = false;
    uint32_t cnt = 0;
    if (i < n) {
        float x, y, z;
        // four floats per pixel on a 16-byte boundary: one load per position
        if (fpp == 4 && (reinterpret_cast<uintptr_t>(pos) & 15u) == 0) {
            const float4 v = __ldcs(reinterpret_cast<const float4*>(pos) + i);
            x = v.x;
            y = v.y;
            z = v.z;
        } else {
            const float* p = pos + (size_t)fpp * i;
            x = __ldcs(p);
            y = __ldcs(p + 1);
            z = __ldcs(p + 2);
        }
        float c[4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
            c[r] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(M.m[r], x), __fmul_rn(M.m[4 + r], y)),
                                       __fmul_rn(M.m[8 + r], z)),
                             M.m[12 + r]);
        if (c[3] != 1.0f) {
            c[0] = __fdiv_rn(c[0], c[3]);
            c[1] = __fdiv_rn(c[1], c[3]);
            c[2] = __fdiv_rn(c[2], c[3]);
        }
        const int32_t px = quantise(c[0], scale), py = quantise(c[1], scale), pz = quantise(c[2], scale);
        if (PCF)
            cnt = grid_footprint<NL>(G, px, py, pz, -((filter - 1) / 2), filter / 2);
        else
            lit = grid_sample<NL>(G, px, py, pz);
    }
    if (U8) {
        if (i < n) {
            const uint32_t f2 = (uint32_t)(filter * filter);
            __stcs(static_cast<uint8_t*>(out) + i,
                   PCF ? (uint8_t)((255u * cnt + f2 / 2u) / f2) : (uint8_t)(lit ? 255u : 0u));
        }
    } else {
        const uint32_t word = __ballot_sync(0xffffffffu, lit);
        if ((threadIdx.x & 31u) == 0 && i < n) __stcs(static_cast<uint32_t*>(out) + (i >> 5), word);
    }
}

// One query against a table entry: its top grid first when it has one.
__device__ __forceinline__ bool multi_descend(const MultiDag& D, int32_t px, int32_t py, int32_t pz) {
    const int root = (int)D.num_levels - 2, min_level = D.leafmasks ? 3 : 0;
    int level = root;
    uint32_t off = 0;
    if (D.top) {
        const int depth = (int)D.top_depth;
        const uint32_t e = __ldg(D.top + top_cell(px, py, pz, root - depth + 1, depth));
        if (e >= kCellLit) return e == kCellLit;
        off = e;
        level = root - depth;
    }
    return descend(D.dag, D.words, 0u, off, level, min_level, D.leafmasks != 0, px, py, pz);
}

// Many resident DAGs at once: query i descends DAG dags[ids[i]] (its own
// depth and leafmask mode); ids outside the table answer "shadow".  The first
// kMultiHeld entries of the table are in shared memory (neighbouring queries
// name different DAGs, and an entry is five loads), from the launch's
// parameters when they are the whole table, and the id and point of a
// thread's next query are requested before the current one descends.
constexpr uint32_t kMultiHeld = 64;
struct MultiTable {
    MultiDag d[kMultiHeld];
};

// Entries of a table into memory from a launch's parameters.
__global__ void k_put_table(const __grid_constant__ MultiTable tab, MultiDag* __restrict__ out, uint32_t count) {
    if (threadIdx.x < count) out[threadIdx.x] = tab.d[threadIdx.x];
}

template <bool PARAM>
__global__ void __launch_bounds__(kThreads)
    k_multi_lookup(const __grid_constant__ MultiTable tab, const MultiDag* __restrict__ dags, uint32_t ndags,
                   const uint32_t* __restrict__ ids, const float* __restrict__ q, uint64_t n,
                   uint32_t* __restrict__ bits) {
    __shared__ MultiDag s_dag[kMultiHeld];
    __shared__ float s_scale[kMultiHeld];
    const uint32_t held = min(ndags, kMultiHeld);
    for (uint32_t t = threadIdx.x; t < held; t += kThreads) {
        s_dag[t] = PARAM ? tab.d[t] : dags[t];
        s_scale[t] = (float)((1u << (s_dag[t].num_levels - 1)) - 1u);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint64_t nwords = (n + 31) / 32;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    uint32_t id_n = 0;
    float x_n = 0.f, y_n = 0.f, z_n = 0.f;
    auto fetch = [&](uint64_t wq) {
        const uint64_t i = wq * 32 + (uint64_t)lane;
        if (i < n) {
            id_n = __ldcs(ids + i);
            const float* p = q + 3 * i;
            x_n = __ldcs(p);
            y_n = __ldcs(p + 1);
            z_n = __ldcs(p + 2);
        }
    };
    uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    fetch(w);
    for (; w < nwords; w += nw) {
        const uint64_t i = w * 32 + (uint64_t)lane;
        const uint32_t id = id_n;
        const float x = x_n, y = y_n, z = z_n;
        fetch(w + nw);
        bool lit = false;
        if (i < n && id < ndags) {
            if (id < held) {
                const float scale = s_scale[id];
                lit = multi_descend(s_dag[id], quantise(x, scale), quantise(y, scale), quantise(z, scale));
            } else {
                const MultiDag D = dags[id];
                const float scale = (float)((1u << (D.num_levels - 1)) - 1u);
                lit = multi_descend(D, quantise(x, scale), quantise(y, scale), quantise(z, scale));
            }
        }
        const uint32_t word = __ballot_sync(0xffffffffu, lit);
        if (lane == 0) __stcs(bits + w, word);
    }
}

// Segmented multi-DAG lookup: many independent requests in one launch.
// Segment s owns output words [word_start, word_start + ceil(n/32)); warp w
// finds its segment by binary search and answers 32 of its queries, reading
// the request's points and writing its bits where they lie (device memory,
// or host memory the GPU reads in place).
__global__ void __launch_bounds__(kThreads)
    k_segment_lookup(const MultiDag* __restrict__ dags, uint32_t ndags, const LookupSegment* __restrict__ segs,
                     uint32_t nsegs, uint64_t total_words) {
    const int lane = threadIdx.x & 31;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < total_words; w += nw) {
        uint32_t lo = 0, hi = nsegs;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (segs[mid].word_start <= w) lo = mid; else hi = mid;
        }
        const LookupSegment sg = segs[lo];
        const uint64_t lw = w - sg.word_start;
        const uint64_t i = lw * 32 + (uint64_t)lane;
        bool lit = false;
        if (i < sg.n && sg.dag < ndags) {
            const MultiDag D = dags[sg.dag];
            const float scale = (float)((1u << (D.num_levels - 1)) - 1u);
            const float* p = sg.xyz + 3 * i;
            const int32_t px = quantise(__ldcs(p), scale), py = quantise(__ldcs(p + 1), scale), pz = quantise(__ldcs(p + 2), scale);
            lit = multi_descend(D, px, py, pz);
        }
        const uint32_t word = __ballot_sync(0xffffffffu, lit);
        if (lane == 0) __stcs(sg.bits + lw, word);
    }
}

uint32_t lookup_grid(int num_sms, uint64_t n) {
    const uint64_t warps = (n + 31) / 32;
    const uint64_t blocks = (warps * 32 + kThreads - 1) / kThreads;
    const uint64_t cap = (uint64_t)(num_sms > 0 ? num_sms : 152) * 8;
    return (uint32_t)(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}

int device_sms() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

}  // namespace

int top_index_depth(uint32_t num_levels, bool leafmasks, uint64_t words, uint32_t max_factor, uint64_t cells) {
    const int root = (int)num_levels - 2, min_level = leafmasks ? 3 : 0;
    int d = root - min_level + 1;
    if (d > kTopIndexDepth) d = kTopIndexDepth;
    // no larger than max_factor times the DAG (at least 64 KiB), or `cells`
    uint64_t limit = words * 4 * max_factor > 65536 ? words * 4 * max_factor : 65536;
    if (cells * 4 > limit) limit = cells * 4;
    while (d > 0 && (uint64_t(4) << (3 * d)) > limit) --d;
    return d < 0 ? 0 : d;
}

cpvs_status launch_top_index(const TopGrid* grids, size_t count, cudaStream_t st) {
    for (size_t g0 = 0; g0 < count; g0 += kTopBatch) {
        TopJobs tab{};
        uint32_t blocks = 0;
        for (size_t g = g0; g < std::min(count, g0 + (size_t)kTopBatch); ++g) {
            const uint32_t parents = 1u << (3 * (grids[g].depth - 1));  // one thread per cell of depth - 1
            tab.j[tab.count++] = TopJob{grids[g].dag, grids[g].out, (uint32_t)grids[g].words, blocks, grids[g].depth};
            blocks += (parents + kThreads - 1) / kThreads;
        }
        k_top_index<<<blocks, kThreads, 0, st>>>(tab);
        CPVS_CUDA(cudaGetLastError());
    }
    return CPVS_OK;
}

// Inner levels below the top grid that k_lookup_fixed unrolls (0 ..
// kFixedLevels); other DAGs take k_lookup.
constexpr int kFixedLevels = 6;

template <bool NDC, int Q, int NL>
bool launch_fixed_nl(int nl, uint32_t g, cudaStream_t st, const uint32_t* dag, uint64_t words, uint32_t num_levels,
                     const uint32_t* top, int depth, const void* xyz, uint64_t n, uint32_t* bits) {
    if (nl == NL) {
        k_lookup_fixed<NDC, Q, NL><<<g, kThreads, 0, st>>>(dag, (uint32_t)words, (int)num_levels, top, depth, xyz,
                                                           (uint32_t)n, bits);
        return true;
    }
    if constexpr (NL < kFixedLevels) {
        return launch_fixed_nl<NDC, Q, NL + 1>(nl, g, st, dag, words, num_levels, top, depth, xyz, n, bits);
    } else {
        return false;
    }
}

template <bool NDC, int Q>
void launch_lookup_q(uint32_t g, cudaStream_t st, const uint32_t* dag, uint64_t words, uint32_t num_levels,
                     bool leafmasks, const uint32_t* top, int depth, const void* xyz, uint64_t n, uint32_t* bits) {
    // the straight-line kernel where it applies: leafmasks, a top grid, at
    // most kFixedLevels inner levels below it, fewer than 2^31 queries
    const int nl = (int)num_levels - 2 - depth - 3 + 1;
    if (Q <= 2 && leafmasks && top && depth > 0 && nl >= 0 && n < (1ull << 31) &&
        launch_fixed_nl<NDC, (Q <= 2 ? Q : 2), 0>(nl, g, st, dag, words, num_levels, top, depth, xyz, n, bits))
        return;
    k_lookup<NDC, Q><<<g, kThreads, 0, st>>>(dag, (uint32_t)words, (int)num_levels, leafmasks, top, depth, xyz, n,
                                             bits);
}

cpvs_status launch_lookup(const uint32_t* dag, uint64_t words, uint32_t num_levels, bool leafmasks,
                          const uint32_t* top, int top_depth, const void* xyz, bool ndc, uint64_t n, uint32_t* bits,
                          cudaStream_t st, Timing* timing, int queries_per_thread) {
    if (n == 0) return CPVS_OK;
    KernelTimer kt(timing, K_LOOKUP, st);
    const int Q = (queries_per_thread == 1 || queries_per_thread == 2) ? queries_per_thread : 4;
    const uint32_t g = lookup_grid(device_sms(), (n + Q - 1) / Q);
    const int depth = top ? top_depth : 0;
    if (ndc) {
        if (Q == 1) launch_lookup_q<true, 1>(g, st, dag, words, num_levels, leafmasks, top, depth, xyz, n, bits);
        else if (Q == 2) launch_lookup_q<true, 2>(g, st, dag, words, num_levels, leafmasks, top, depth, xyz, n, bits);
        else launch_lookup_q<true, 4>(g, st, dag, words, num_levels, leafmasks, top, depth, xyz, n, bits);
    } else {
        if (Q == 1) launch_lookup_q<false, 1>(g, st, dag, words, num_levels, leafmasks, top, depth, xyz, n, bits);
        else if (Q == 2) launch_lookup_q<false, 2>(g, st, dag, words, num_levels, leafmasks, top, depth, xyz, n, bits);
        else launch_lookup_q<false, 4>(g, st, dag, words, num_levels, leafmasks, top, depth, xyz, n, bits);
    }
    CPVS_CUDA(cudaGetLastError());
    return CPVS_OK;
}

int tune_lookup(const uint32_t* dag, uint64_t words, uint32_t num_levels, bool leafmasks, const uint32_t* top,
                int top_depth, const void* xyz, bool ndc, uint64_t n, uint32_t* bits, cudaStream_t st) {
    // up to 2^24 queries (~0.1 ms per launch), best of three timed runs
    // after a warm-up, so that launch-to-launch noise does not pick the
    // variant.  The sample's 201 MB of points exceed L2 as a large batch's do:
    // a sample that stays in L2 after the warm-up favours the variants that
    // hide latency over the one that streams best.  A batch may be ordered
    // (surface points first, say), so a large one is sampled in four chunks
    // spread over it: chunk c starts at c*n/4 rounded down to a whole answer
    // word; chunks of sample/4 (a multiple of 32, at most n/4) end inside the
    // batch and its answer words.
    const uint64_t sample = n < (1ull << 24) ? n : (1ull << 24);
    const int chunks = n > sample ? 4 : 1;
    const uint64_t per = chunks == 1 ? sample : (sample / chunks) & ~31ull;
    const size_t qbytes = 12;  // three floats or three int32 per query
    cudaEvent_t a = nullptr, b = nullptr;
    if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) {
        cudaGetLastError();
        return 4;
    }
    int best = 4;
    float best_ms = 1e30f;
    for (int q : {1, 2, 4}) {
        float ms = 1e30f;
        for (int rep = 0; rep < 4; ++rep) {  // the first run warms the caches
            float t = 0.f;
            cudaEventRecord(a, st);
            for (int c = 0; c < chunks; ++c) {
                const uint64_t off = (n / chunks * c) & ~31ull;
                launch_lookup(dag, words, num_levels, leafmasks, top, top_depth,
                              static_cast<const char*>(xyz) + off * qbytes, ndc, per, bits + off / 32, st, nullptr, q);
            }
            cudaEventRecord(b, st);
            cudaEventSynchronize(b);
            cudaEventElapsedTime(&t, a, b);
            if (rep > 0 && t < ms) ms = t;
        }
        if (ms < best_ms) {
            best_ms = ms;
            best = q;
        }
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaGetLastError();
    return best;
}

bool multi_table_fits(uint32_t ndags) { return ndags <= kMultiHeld; }

cpvs_status put_multi_table(const MultiDag* host, MultiDag* dags, uint32_t ndags, cudaStream_t st) {
    // a recorded copy would read the caller's table when the graph runs
    if (!capturing(st)) {
        CPVS_CUDA(cudaMemcpyAsync(dags, host, ndags * sizeof(MultiDag), cudaMemcpyHostToDevice, st));
        return CPVS_OK;
    }
    for (uint32_t at = 0; at < ndags; at += kMultiHeld) {
        MultiTable tab{};
        const uint32_t count = std::min(ndags - at, kMultiHeld);
        std::copy(host + at, host + at + count, tab.d);
        k_put_table<<<1, kMultiHeld, 0, st>>>(tab, dags + at, count);
        CPVS_CUDA(cudaGetLastError());
    }
    return CPVS_OK;
}

cpvs_status launch_multi_lookup(const MultiDag* host, const MultiDag* dags, uint32_t ndags, const uint32_t* ids,
                                const float* xyz, uint64_t n, uint32_t* bits, cudaStream_t st, Timing* timing) {
    if (n == 0) return CPVS_OK;
    KernelTimer kt(timing, K_MULTI_LOOKUP, st);
    const uint32_t g = lookup_grid(device_sms(), n);
    MultiTable tab{};
    if (multi_table_fits(ndags)) {
        std::copy(host, host + ndags, tab.d);
        k_multi_lookup<true><<<g, kThreads, 0, st>>>(tab, nullptr, ndags, ids, xyz, n, bits);
    } else {
        k_multi_lookup<false><<<g, kThreads, 0, st>>>(tab, dags, ndags, ids, xyz, n, bits);
    }
    CPVS_CUDA(cudaGetLastError());
    return CPVS_OK;
}

cpvs_status launch_segment_lookup(const MultiDag* dags, uint32_t ndags, const LookupSegment* segs, uint32_t nsegs,
                                  uint64_t total_words, cudaStream_t st, Timing* timing) {
    if (total_words == 0 || nsegs == 0) return CPVS_OK;
    KernelTimer kt(timing, K_MULTI_LOOKUP, st);
    k_segment_lookup<<<lookup_grid(device_sms(), total_words * 32), kThreads, 0, st>>>(dags, ndags, segs, nsegs,
                                                                                     total_words);
    CPVS_CUDA(cudaGetLastError());
    return CPVS_OK;
}

int grid_top_depth(uint32_t length, uint32_t dag_levels, bool leafmasks, uint64_t words) {
    const int root = (int)dag_levels - 2, min_level = leafmasks ? 3 : 0;
    const int gl = log2_u32(length);
    int d = root - min_level + 1;
    if (d > kTopIndexDepth) d = kTopIndexDepth;
    // no larger than 8x the combined DAG (at least 64 KiB, at most 64 MiB),
    // as a shadow's own top grid: one more level in the index (8 instead of
    // 7 for an 8192^2 map's 9.4 MB DAG) took a 4K frame's evaluate from
    // 0.147 to 0.126 ms
    uint64_t limit = words * 32 > 65536 ? words * 32 : 65536;
    if (limit > (64ull << 20)) limit = 64ull << 20;
    while (d > 0 && (uint64_t(4) << (3 * (gl + d))) > limit) --d;
    return d < 0 ? 0 : d;
}

GridRoute grid_route(const uint32_t* dag, uint64_t words, const uint32_t* cells, uint32_t length, uint32_t dag_levels,
                     bool leafmasks, const uint32_t* gtop, int gdepth) {
    return GridRoute{dag, cells, gtop, (uint32_t)words, log2_u32(length), (int)dag_levels - 1, gtop ? gdepth : 0,
                     leafmasks};
}

// Inner levels below a grid index that the grid kernels unroll (0 ..
// kFixedLevels), or -1: leafmask cell DAGs with an index only.
int grid_fixed_levels(const GridRoute& G) {
    if (!G.leafmasks || !G.top || G.depth <= 0) return -1;
    const int nl = G.sh - 1 - G.depth - 3 + 1;
    return nl >= 0 && nl <= kFixedLevels ? nl : -1;
}

// Calls f(std::integral_constant<int, nl>) for nl in [NL, kFixedLevels];
// false when nl is outside.
template <int NL, typename F>
bool dispatch_levels(int nl, F&& f) {
    if (nl == NL) {
        f(std::integral_constant<int, NL>());
        return true;
    }
    if constexpr (NL < kFixedLevels) {
        return dispatch_levels<NL + 1>(nl, f);
    } else {
        return false;
    }
}

cpvs_status launch_grid_top_index(const uint32_t* dag, uint64_t words, const uint32_t* cells, uint32_t length,
                                  uint32_t dag_levels, int depth, uint32_t* out, cudaStream_t st) {
    const int bits = log2_u32(length) + depth;
    if (depth >= 1) {
        const uint64_t parents = 1ull << (3 * (bits - 1));
        const uint32_t g = (uint32_t)std::min<uint64_t>((parents + 255) / 256, 152ull * 32);
        k_grid_top_index_parents<<<g, 256, 0, st>>>(dag, (uint32_t)words, cells, length, depth, bits, out);
    } else {
        const uint64_t total = 1ull << (3 * bits);
        const uint32_t g = (uint32_t)std::min<uint64_t>((total + 255) / 256, 152ull * 32);
        k_grid_top_index<<<g, 256, 0, st>>>(dag, (uint32_t)words, cells, length, (int)dag_levels, depth, bits, out);
    }
    CPVS_CUDA(cudaGetLastError());
    return CPVS_OK;
}

cpvs_status launch_grid_evaluate(const uint32_t* dag, uint64_t words, const uint32_t* cells, uint32_t length,
                                 uint32_t dag_levels, bool leafmasks, const uint32_t* gtop, int gdepth,
                                 const float* positions, uint32_t fpp, uint64_t n, const float* light_view_proj,
                                 uint32_t filter, bool u8, void* out, cudaStream_t st, Timing* timing) {
    if (n == 0) return CPVS_OK;
    KernelTimer kt(timing, K_EVALUATE, st);
    const GridRoute G = grid_route(dag, words, cells, length, dag_levels, leafmasks, gtop, gdepth);
    EvalMatrix M;
    for (int k = 0; k < 16; ++k) M.m[k] = light_view_proj[k];
    auto launch = [&](auto nlc) {
        constexpr int NLv = decltype(nlc)::value;
        auto* kernel = !u8          ? k_grid_evaluate<false, NLv, false>
                       : filter > 1 ? k_grid_evaluate<true, NLv, true>
                                    : k_grid_evaluate<true, NLv, false>;
        constexpr uint64_t kMost = 1ull << 30;
        for (uint64_t at = 0; at < n; at += kMost) {
            const uint32_t m = (uint32_t)std::min<uint64_t>(n - at, kMost);
            kernel<<<(m + kThreads - 1) / kThreads, kThreads, 0, st>>>(
                G, positions + at * fpp, fpp, m, M, (int)filter,
                static_cast<char*>(out) + (u8 ? at : at / 8));
        }
    };
    if (!dispatch_levels<0>(grid_fixed_levels(G), launch)) launch(std::integral_constant<int, -1>());
    CPVS_CUDA(cudaGetLastError());
    return CPVS_OK;
}

cpvs_status launch_grid_lookup(const uint32_t* dag, uint64_t words, const uint32_t* cells, uint32_t length,
                               uint32_t dag_levels, bool leafmasks, const uint32_t* gtop, int gdepth, const float* xyz,
                               uint64_t n, uint32_t* bits, cudaStream_t st, Timing* timing) {
    if (n == 0) return CPVS_OK;
    KernelTimer kt(timing, K_GRID_LOOKUP, st);
    const GridRoute G = grid_route(dag, words, cells, length, dag_levels, leafmasks, gtop, gdepth);
    const uint32_t g = lookup_grid(device_sms(), n);
    auto launch = [&](auto nlc) { k_grid_lookup<decltype(nlc)::value><<<g, kThreads, 0, st>>>(G, xyz, n, bits); };
    if (!dispatch_levels<0>(grid_fixed_levels(G), launch)) launch(std::integral_constant<int, -1>());
    CPVS_CUDA(cudaGetLastError());
    return CPVS_OK;
}

}  // namespace cpvs
