// CAPT construction on the GPU, with the same layout as the host builder (vg_capt.cpp, which
// follows collision/capt.hh:104-365 bit for bit, the capt.hh:226-233 scan included).
//
// The host builder splits recursively; this one goes level by level.  At level d every node
// holds N >> d consecutive entries of the point order: a bitonic network sorts each node's
// entries by (coordinate on axis d mod 3, current position), which is exactly the host's stable
// sort.  Each node's split value and the two scans of its sorted halves (capt.hh:226-233) follow
// from the sorted keys.  Its affordance list (the points of other nodes within r_max of its cell)
// is filtered into its children's lists in order, one thread block per node (ordered compaction),
// and the scanned ranges are appended, as the host builder does.  At the leaves, each leaf's
// representative and its afforded points that pass the cell test become its 8-point blocks, its
// box and its block range.
//
// What bounds a build of a few thousand points is launches and waits, not work: a launch per step
// and level, and a host wait per level for the size of its lists, made 5,271 points 1.54 ms.  So
// the levels whose nodes fit a tile sort in one launch (a block takes a subtree down to its
// leaves, keeping each level's order), a node's lists take their room from a counter instead of a
// scan, within room guessed before (a level that runs out is done again in a larger buffer), and
// the host waits once, for the size of the blocks, and once for each level that ran out.
#include "vg_capt_gpu.h"
#include "vg_capt_room.h"

#include "../../include/vamp_gb300.h"
#include "vg_internal.h"
#include "vg_pool.h"
#include "vg_sort.cuh"

#include <algorithm>
#include <type_traits>
#include <string>
#include <vector>

namespace vg
{
    namespace
    {
        constexpr float kInf = __builtin_huge_valf();
        constexpr int kListBlock = 128;  // threads per node in the list passes
        constexpr long long kOrdersMax = 1ll << 24;  // entries up to which the subtrees' orders are kept

        __global__ void init_points(const float *xyz, long long n, long long N, float *px, float *py, float *pz,
                                    uint32_t *ord)
        {
            const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (i >= N)
                return;
            px[i] = i < n ? xyz[3 * i + 0] : kInf;
            py[i] = i < n ? xyz[3 * i + 1] : kInf;
            pz[i] = i < n ? xyz[3 * i + 2] : kInf;
            ord[i] = static_cast<uint32_t>(i);
        }

        // `full` (here and below): not zero once a level's lists ran out of room (its number + 1).  What is
        // queued for the levels below then does nothing, so that the build can go on from that level.
        __global__ void load_keys(const uint32_t *ord, const float *axis, long long N, const int *full, float *key, uint32_t *pos)
        {
            const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (i >= N || *full)
                return;
            key[i] = axis[ord[i]];
            pos[i] = static_cast<uint32_t>(i);
        }

        // One compare-exchange stage of a bitonic network that sorts every aligned segment of S
        // entries ascending by (key, pos).
        __global__ void bitonic_stage(float *key, uint32_t *pos, uint32_t *ord, long long N, long long k, long long j,
                                      long long S, const int *full)
        {
            const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
            const long long p = i ^ j;
            if (i >= N || p <= i || *full)
                return;
            const bool up = k == S || (i & k) == 0;
            const float ki = key[i], kp = key[p];
            const bool greater = ki > kp || (ki == kp && pos[i] > pos[p]);
            if (greater == up)
            {
                key[i] = kp;
                key[p] = ki;
                const uint32_t a = pos[i];
                pos[i] = pos[p];
                pos[p] = a;
                const uint32_t o = ord[i];
                ord[i] = ord[p];
                ord[p] = o;
            }
        }

        constexpr int kSortTile = 2048;  // entries per shared-memory tile of the sort
        constexpr int kSmallTile = 512;

        // An entry under sort: its key, its position before the level's sort (breaks ties), its point.
        struct Entry
        {
            float key;
            uint32_t pos, ord;
        };

        __device__ __forceinline__ Entry shuffle_xor(Entry v, int lanes)
        {
            return {__shfl_xor_sync(0xffffffffu, v.key, lanes), __shfl_xor_sync(0xffffffffu, v.pos, lanes),
                    __shfl_xor_sync(0xffffffffu, v.ord, lanes)};
        }

        struct After
        {
            __device__ __forceinline__ bool operator()(const Entry &a, const Entry &b) const
            {
                return a.key > b.key || (a.key == b.key && a.pos > b.pos);
            }
        };

        // All compare-exchange stages of sizes k in [k0, k1] and strides below the tile, on tiles
        // of T = min(S, 2048) entries (S: the sorted segment size, a power of two).
        __global__ void __launch_bounds__(kSortTile / 2) bitonic_tile(float *key, uint32_t *pos, uint32_t *ord, long long S,
                                                                      long long k0, long long k1, const int *full)
        {
            __shared__ Entry sm[kSortTile];
            if (*full)
                return;
            const int T = static_cast<int>(S < kSortTile ? S : kSortTile), t = threadIdx.x;
            const long long base = static_cast<long long>(blockIdx.x) * T;
            Entry v[2] = {};
#pragma unroll
            for (int e = 0; e < 2; ++e)
            {
                const long long i = base + 2 * t + e;
                if (2 * t + e < T)
                    v[e] = {key[i], pos[i], ord[i]};
            }
            const unsigned b = static_cast<unsigned>(base), all = static_cast<unsigned>(S);
            sort_steps(v, sm, T, static_cast<unsigned>(k0), static_cast<unsigned>(k1), After{},
                       [&](unsigned i, unsigned k) { return k == all || ((b + i) & k) == 0; });
#pragma unroll
            for (int e = 0; e < 2; ++e)
            {
                const long long i = base + 2 * t + e;
                if (2 * t + e < T)
                {
                    key[i] = v[e].key;
                    pos[i] = v[e].pos;
                    ord[i] = v[e].ord;
                }
            }
        }

        struct NodeInfo
        {
            float up, down;
            long long h, l;  // ends of the two scanned ranges (capt.hh:226-233)
        };

        // first index in [lo, hi) whose key is > v (keys ascending)
        __device__ long long upper_bound(const float *key, long long lo, long long hi, float v)
        {
            while (lo < hi)
            {
                const long long m = lo + ((hi - lo) >> 1);
                if (key[m] > v)
                    hi = m;
                else
                    lo = m + 1;
            }
            return lo;
        }

        // A node's split value (returned) and scan ends from its S sorted keys at key[begin ..]; the ends
        // are shifted by `base`, the tile's place in the whole order.
        __device__ float split_node(const float *key, long long begin, long long S, long long base, float r_max, NodeInfo &ni)
        {
            const long long half = S >> 1;
            const float test = __fmul_rn(__fadd_rn(key[begin + half - 1], key[begin + half]), 0.5f);
            ni.up = __fadd_rn(test, r_max);
            ni.down = __fsub_rn(test, r_max);
            // lower half, from its smallest key: while key >= down and finite
            if (key[begin] >= ni.down && key[begin] < kInf && key[begin] > -kInf)
                ni.h = upper_bound(key, begin, begin + half, __int_as_float(0x7f7fffff));  // up to the first +inf
            else
                ni.h = begin;
            // upper half: while key <= up and finite
            ni.l = key[begin + half] > -kInf ? upper_bound(key, begin + half, begin + S, ni.up) : begin + half;
            {
                const long long f = upper_bound(key, begin + half, begin + S, __int_as_float(0x7f7fffff));
                ni.l = ni.l < f ? ni.l : f;
            }
            ni.h += base;
            ni.l += base;
            return test;
        }

        // split_node for every node of level d (heap order)
        __global__ void split_nodes(const float *key, long long N, int d, float r_max, const int *full, float *tests, NodeInfo *info)
        {
            const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (t < (1ll << d) && !*full)
            {
                const long long S = N >> d, at = (1ll << d) - 1 + t;
                tests[at] = split_node(key, t * S, S, 0, r_max, info[at]);
            }
        }

        // Levels d0 .. d1 - 1 of subtrees whose nodes at level d0 hold at most T entries: a block of T / 2
        // threads per tile of T entries sorts every level, splits its nodes and leaves each level's
        // order in orders[(d - d0) N ..], the last one in ord.  The network of each level is
        // bitonic_tile's.
        __global__ void __launch_bounds__(kSortTile / 2) sort_subtrees(const float *px, const float *py, const float *pz, long long N,
                                                                       int d0, int d1, int T, float r_max, const int *full,
                                                                       uint32_t *ord, uint32_t *orders, float *tests, NodeInfo *info)
        {
            __shared__ Entry sm[kSortTile];
            __shared__ float sk[kSortTile];
            if (*full)
                return;
            const long long base = static_cast<long long>(blockIdx.x) * T;
            const int t = threadIdx.x;
            Entry v[2] = {};
#pragma unroll
            for (int e = 0; e < 2; ++e)
            {
                if (2 * t + e < T)
                    v[e].ord = ord[base + 2 * t + e];
            }
            for (int d = d0; d < d1; ++d)
            {
                const long long S = N >> d;
                const float *axis = d % 3 == 0 ? px : d % 3 == 1 ? py : pz;
#pragma unroll
                for (int e = 0; e < 2; ++e)
                {
                    v[e].pos = static_cast<uint32_t>(base + 2 * t + e);
                    if (2 * t + e < T)
                        v[e].key = axis[v[e].ord];
                }
                const unsigned b = static_cast<unsigned>(base), all = static_cast<unsigned>(S);
                sort_steps(v, sm, all, 2u, all, After{}, [&](unsigned i, unsigned k) { return k == all || ((b + i) & k) == 0; });
                uint32_t *order = orders + static_cast<long long>(d - d0) * N + base;
#pragma unroll
                for (int e = 0; e < 2; ++e)
                {
                    if (2 * t + e < T)
                    {
                        sk[2 * t + e] = v[e].key;
                        order[2 * t + e] = v[e].ord;
                    }
                }
                __syncthreads();
                for (int n = t; n < T / S; n += blockDim.x)
                {
                    const long long at = (1ll << d) - 1 + base / S + n;
                    tests[at] = split_node(sk, static_cast<long long>(n) * S, S, base, r_max, info[at]);
                }
                __syncthreads();
            }
#pragma unroll
            for (int e = 0; e < 2; ++e)
            {
                if (2 * t + e < T)
                    ord[base + 2 * t + e] = v[e].ord;
            }
        }

        // block-wide exclusive scan of one flag per thread; returns the thread's offset, *total
        // the block's count
        __device__ unsigned block_scan(unsigned flag, unsigned *total)
        {
            __shared__ unsigned warp_sums[kListBlock / 32];
            const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            unsigned v = flag;
            for (int o = 1; o < 32; o <<= 1)
            {
                const unsigned y = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o)
                    v += y;
            }
            if (lane == 31)
                warp_sums[warp] = v;
            __syncthreads();
            unsigned base = 0, all = 0;
            for (int w = 0; w < kListBlock / 32; ++w)
            {
                base += w < warp ? warp_sums[w] : 0u;
                all += warp_sums[w];
            }
            __syncthreads();
            *total = all;
            return base + v - flag;
        }

        __device__ unsigned long long block_sum(unsigned long long v)
        {
            __shared__ unsigned long long part[kListBlock / 32];
            for (int o = 16; o > 0; o >>= 1)
                v += __shfl_xor_sync(0xffffffffu, v, o);
            if ((threadIdx.x & 31) == 0)
                part[threadIdx.x >> 5] = v;
            __syncthreads();
            unsigned long long all = 0;
            for (int w = 0; w < kListBlock / 32; ++w)
                all += part[w];
            __syncthreads();
            return all;
        }

        // The children's lists of each node of level d (one block per node): the node's list filtered in
        // order, then the scanned range.  A node's two lists take their room in `out` from the level's
        // counter, in any order; range[n] is node n's list.  Past the room `cap` nothing is written (the
        // counter still says what the level needs) and *full is set to d + 1.
        __global__ void child_lists(const ulonglong2 *range, const uint32_t *items, const float *axis, long long N, int d,
                                    const NodeInfo *info, const uint32_t *ord, unsigned long long cap, unsigned long long *used,
                                    int *full, ulonglong2 *child_range, uint32_t *out)
        {
            __shared__ unsigned long long room;
            const int ran_out = *static_cast<volatile int *>(full);
            if (__syncthreads_or(ran_out != 0 && ran_out != d + 1))
                return;  // a level above
            const long long t = blockIdx.x;
            const NodeInfo ni = info[(1ll << d) - 1 + t];
            const unsigned long long a0 = range[t].x, a1 = range[t].y;
            const long long S = N >> d, begin = t * S, half = S / 2;
            const unsigned long long s_lo = static_cast<unsigned long long>(ni.l - (begin + half)),
                                     s_hi = static_cast<unsigned long long>(ni.h - begin);
            // lists of one pass are read once
            const bool once = a1 - a0 <= kListBlock;
            uint32_t it = 0;
            bool lo = false, hi = false;
            auto load = [&](unsigned long long i) {
                lo = hi = false;
                if (i < a1)
                {
                    it = items[i];
                    const float v = axis[it];
                    lo = v <= ni.up;
                    hi = v >= ni.down;
                }
            };
            unsigned long long n_lo = 0, n_hi = 0;
            unsigned p_lo = 0, p_hi = 0, tot_lo = 0, tot_hi = 0;
            if (once)
            {
                load(a0 + threadIdx.x);
                p_lo = block_scan(lo ? 1u : 0u, &tot_lo);
                p_hi = block_scan(hi ? 1u : 0u, &tot_hi);
                n_lo = tot_lo;
                n_hi = tot_hi;
            }
            else
            {
                for (unsigned long long i = a0 + threadIdx.x; i < a1; i += blockDim.x)
                {
                    load(i);
                    n_lo += lo;
                    n_hi += hi;
                }
                n_lo = block_sum(n_lo);
                n_hi = block_sum(n_hi);
            }
            const unsigned long long need = n_lo + s_lo + n_hi + s_hi;
            if (threadIdx.x == 0)
                room = need ? atomicAdd(used + d, need) : 0ull;
            __syncthreads();
            unsigned long long w_lo = room, w_hi = room + n_lo + s_lo;
            const bool fits = room + need <= cap;
            if (threadIdx.x == 0)
            {
                child_range[2 * t] = fits ? make_ulonglong2(w_lo, w_hi) : make_ulonglong2(0, 0);
                child_range[2 * t + 1] = fits ? make_ulonglong2(w_hi, room + need) : make_ulonglong2(0, 0);
                if (!fits)
                    *full = d + 1;
            }
            if (!fits)
                return;
            if (once)
            {
                if (lo)
                    out[w_lo + p_lo] = it;
                if (hi)
                    out[w_hi + p_hi] = it;
            }
            else
            {
                for (unsigned long long c = a0; c < a1; c += blockDim.x)
                {
                    load(c + threadIdx.x);
                    p_lo = block_scan(lo ? 1u : 0u, &tot_lo);
                    p_hi = block_scan(hi ? 1u : 0u, &tot_hi);
                    if (lo)
                        out[w_lo + p_lo] = it;
                    if (hi)
                        out[w_hi + p_hi] = it;
                    w_lo += tot_lo;
                    w_hi += tot_hi;
                }
                n_lo = n_hi = 0;
            }
            for (long long i = begin + half + threadIdx.x; i < ni.l; i += blockDim.x)
                out[w_lo + n_lo + (i - begin - half)] = ord[i];
            for (long long i = begin + threadIdx.x; i < ni.h; i += blockDim.x)
                out[w_hi + n_hi + (i - begin)] = ord[i];
        }

        // each leaf's cell: the split planes along its path (right child: coordinate >= test)
        __global__ void leaf_cells(const float *tests, int nlog2, const int *full, float *cell)
        {
            const long long leaf = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (leaf >= 1ll << nlog2 || *full)
                return;
            float lo[3] = {-kInf, -kInf, -kInf}, hi[3] = {kInf, kInf, kInf};
            long long idx = 0;
            for (int d = 0; d < nlog2; ++d)
            {
                const bool right = (leaf >> (nlog2 - 1 - d)) & 1;
                const float t = tests[idx];
                for (int k = 0; k < 3; ++k)
                {
                    if (k == d % 3)
                    {
                        lo[k] = right ? t : lo[k];
                        hi[k] = right ? hi[k] : t;
                    }
                }
                idx = 2 * idx + 1 + right;
            }
            for (int k = 0; k < 3; ++k)
            {
                cell[6 * leaf + k] = lo[k];
                cell[6 * leaf + 3 + k] = hi[k];
            }
        }

        __device__ float cell_distsq(const float *c, float x, float y, float z)
        {
            const float p[3] = {x, y, z};
            float d[3];
            for (int k = 0; k < 3; ++k)
            {
                const float m = c[k] > p[k] ? c[k] : p[k];
                const float cl = c[3 + k] < m ? c[3 + k] : m;
                d[k] = __fsub_rn(p[k], cl);
            }
            return __fmaf_rn(d[2], d[2], __fmaf_rn(d[0], d[0], __fmul_rn(d[1], d[1])));
        }

        __device__ bool cell_inside_ball(const float *c, float x, float y, float z, float r2)
        {
            const float p[3] = {x, y, z};
            float d[3];
            for (int k = 0; k < 3; ++k)
            {
                const float a = __fsub_rn(p[k], c[k]), b = __fsub_rn(c[3 + k], p[k]);
                d[k] = a < b ? b : a;
            }
            return __fmaf_rn(d[2], d[2], __fmaf_rn(d[0], d[0], __fmul_rn(d[1], d[1]))) <= r2;
        }

        struct LeafParams
        {
            const ulonglong2 *range;
            const uint32_t *items;
            const float *px, *py, *pz;
            const uint32_t *ord;
            const float *cell;
            float max_l2, min_l2;
        };

        // number of 8-point blocks of each leaf (one block of threads per leaf)
        __global__ void count_leaves(const LeafParams p, const int *full, uint32_t *blocks)
        {
            if (*full)
                return;
            const long long t = blockIdx.x;
            const uint32_t rep = p.ord[t];
            const float rx = p.px[rep], ry = p.py[rep], rz = p.pz[rep];
            const float *c = p.cell + 6 * t;
            unsigned long long acc = 0;
            const bool finite = rx < kInf && rx > -kInf;
            if (finite && !cell_inside_ball(c, rx, ry, rz, p.min_l2))
            {
                const ulonglong2 list = p.range[t];
                for (unsigned long long i = list.x + threadIdx.x; i < list.y; i += blockDim.x)
                {
                    const uint32_t it = p.items[i];
                    acc += cell_distsq(c, p.px[it], p.py[it], p.pz[it]) <= p.max_l2;
                }
            }
            acc = block_sum(acc);
            if (threadIdx.x == 0)
                blocks[t] = static_cast<uint32_t>(finite ? (acc + 1 + 7) / 8 : 0);
        }

        __device__ float block_min(float v)
        {
            __shared__ float part[kListBlock / 32];
            for (int o = 16; o > 0; o >>= 1)
                v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
            if ((threadIdx.x & 31) == 0)
                part[threadIdx.x >> 5] = v;
            __syncthreads();
            float all = part[0];
            for (int w = 1; w < kListBlock / 32; ++w)
                all = fminf(all, part[w]);
            __syncthreads();
            return all;
        }

        // each leaf's blocks (its representative, then its accepted points in list order, padded
        // with +inf) and its box
        __global__ void write_leaves(const LeafParams p, const uint32_t *starts, float *aff, float *aabbs)
        {
            const long long t = blockIdx.x;
            const uint32_t rep = p.ord[t];
            const float rx = p.px[rep], ry = p.py[rep], rz = p.pz[rep];
            const float *c = p.cell + 6 * t;
            const bool finite = rx < kInf && rx > -kInf;
            float bmin[3] = {rx, ry, rz}, bmax[3] = {rx, ry, rz};
            if (finite)
            {
                const unsigned long long b0 = starts[t], nb = starts[t + 1] - b0;
                float *blk = aff + 24 * b0;
                auto put = [&](unsigned long long m, float x, float y, float z) {
                    float *b = blk + 24 * (m >> 3);
                    const unsigned l = static_cast<unsigned>(m & 7);
                    b[l] = x;
                    b[8 + l] = y;
                    b[16 + l] = z;
                };
                if (threadIdx.x == 0)
                    put(0, rx, ry, rz);
                unsigned long long w = 1;
                if (!cell_inside_ball(c, rx, ry, rz, p.min_l2))
                {
                    const ulonglong2 list = p.range[t];
                    for (unsigned long long s = list.x; s < list.y; s += blockDim.x)
                    {
                        const unsigned long long i = s + threadIdx.x;
                        bool ok = false;
                        float x = 0, y = 0, z = 0;
                        if (i < list.y)
                        {
                            const uint32_t it = p.items[i];
                            x = p.px[it];
                            y = p.py[it];
                            z = p.pz[it];
                            ok = cell_distsq(c, x, y, z) <= p.max_l2;
                        }
                        unsigned tot;
                        const unsigned at = block_scan(ok ? 1u : 0u, &tot);
                        if (ok)
                        {
                            put(w + at, x, y, z);
                            bmin[0] = fminf(bmin[0], x);
                            bmin[1] = fminf(bmin[1], y);
                            bmin[2] = fminf(bmin[2], z);
                            bmax[0] = fmaxf(bmax[0], x);
                            bmax[1] = fmaxf(bmax[1], y);
                            bmax[2] = fmaxf(bmax[2], z);
                        }
                        w += tot;
                    }
                }
                for (unsigned long long m = w + threadIdx.x; m < 8 * nb; m += blockDim.x)
                    put(m, kInf, kInf, kInf);
                for (int k = 0; k < 3; ++k)
                {
                    bmin[k] = block_min(bmin[k]);
                    bmax[k] = -block_min(-bmax[k]);
                }
            }
            if (threadIdx.x == 0)
            {
                for (int k = 0; k < 3; ++k)
                {
                    aabbs[6 * t + k] = bmin[k];
                    aabbs[6 * t + 3 + k] = bmax[k];
                }
            }
        }

        // what the host needs of a finished tree
        struct Summary
        {
            unsigned long long blocks;
            float top[6];        // box of every finite representative
            float top_tests[3];  // the first split values
            int full;            // a level that ran out of room + 1 (0: none; only then is the rest filled in)
        };

        // The leaves' first blocks (exclusive sums of their counts, starts[N] the total) by block 0, the
        // box of the finite representatives by block 1.
        __global__ void __launch_bounds__(1024) finish_tree(const uint32_t *blocks, long long N, uint32_t *starts, const uint32_t *ord,
                                                            const float *px, const float *py, const float *pz,
                                                            const float *tests, const int *full, Summary *sum)
        {
            const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
            if (*full)
            {
                if (blockIdx.x == 0 && t == 0)
                    sum->full = *full;
                return;
            }
            if (blockIdx.x == 0)
            {
                __shared__ unsigned long long wsum[32];
                // 1024 consecutive counts a round, the sums of the rounds before carried
                __shared__ unsigned long long carry;
                if (t == 0)
                    carry = 0;
                for (long long c = 0; c < N; c += 1024 * 8)
                {
                    // eight consecutive counts a thread
                    uint32_t v[8];
                    unsigned long long mine = 0;
                    const long long i0 = c + 8 * t;
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                    {
                        v[k] = i0 + k < N ? blocks[i0 + k] : 0u;
                        mine += v[k];
                    }
                    unsigned long long x = mine;
                    for (int o = 1; o < 32; o <<= 1)
                    {
                        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
                        if (lane >= o)
                            x += y;
                    }
                    if (lane == 31)
                        wsum[warp] = x;
                    __syncthreads();
                    unsigned long long at = carry + x - mine;
                    for (int w = 0; w < warp; ++w)
                        at += wsum[w];
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                    {
                        if (i0 + k < N)
                            starts[i0 + k] = static_cast<uint32_t>(at);
                        at += v[k];
                    }
                    __syncthreads();
                    if (t == 1023)
                        carry = at;
                    __syncthreads();
                }
                if (t == 0)
                {
                    starts[N] = static_cast<uint32_t>(carry);
                    sum->blocks = carry;
                    sum->full = 0;
                    for (int k = 0; k < 3; ++k)
                        sum->top_tests[k] = k < N - 1 ? tests[k] : 0.0f;
                }
                return;
            }
            float mn[3] = {kInf, kInf, kInf}, mx[3] = {-kInf, -kInf, -kInf};
            for (long long i = t; i < N; i += 1024)
            {
                const uint32_t r = ord[i];
                const float v[3] = {px[r], py[r], pz[r]};
                if (v[0] < kInf && v[0] > -kInf)
                {
                    for (int k = 0; k < 3; ++k)
                    {
                        mn[k] = fminf(mn[k], v[k]);
                        mx[k] = fmaxf(mx[k], v[k]);
                    }
                }
            }
            __shared__ float part[6][32];
            for (int k = 0; k < 3; ++k)
            {
                for (int o = 16; o > 0; o >>= 1)
                {
                    mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
                    mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
                }
                if (lane == 0)
                {
                    part[k][warp] = mn[k];
                    part[3 + k][warp] = mx[k];
                }
            }
            __syncthreads();
            if (t < 6)
            {
                float v = part[t][0];
                for (int w = 1; w < 32; ++w)
                    v = t < 3 ? fminf(v, part[t][w]) : fmaxf(v, part[t][w]);
                sum->top[t] = v;
            }
        }

        unsigned grid_of(long long n, int block)
        {
            return static_cast<unsigned>((n + block - 1) / block);
        }
    }  // namespace

    int capt_build_device(const float *xyz, size_t n, float r_min, float r_max, float r_point, cudaStream_t s,
                          DeviceCapt &out)
    {
        if (n < 2)
            return set_error(VG_ERR_ARG, "CAPT build: need at least 2 points");
        int nlog2 = 0;
        while ((size_t{1} << nlog2) < n)
            ++nlog2;
        const long long N = 1ll << nlog2;
        out = DeviceCapt{};
        out.nlog2 = nlog2;
        out.r_min = r_min;
        out.r_max = r_max;
        out.r_point = r_point;
        // the first level whose nodes fit a tile: its subtrees sort in one launch, where their levels'
        // orders (4 bytes an entry and level) are no burden
        int d0 = 0;
        while ((N >> d0) > kSortTile)
            ++d0;
        int d1 = d0;  // the first level of nodes of kSmallTile entries (d0 in smaller trees)
        while ((N >> d1) > kSmallTile)
            ++d1;
        bool subtrees = N <= kOrdersMax;
        const int T = static_cast<int>(std::min<long long>(N, kSortTile));
        ListRoom room(N);
        cudaError_t e = cudaSuccess;
        // results: split values, boxes, starts and the points, in one allocation
        {
            const size_t tests = (static_cast<size_t>(N) * sizeof(float) + 255) & ~size_t(255);
            const size_t boxes = (6 * static_cast<size_t>(N) * sizeof(float) + 255) & ~size_t(255);
            const size_t starts = ((static_cast<size_t>(N) + 1) * sizeof(uint32_t) + 255) & ~size_t(255);
            char *base = nullptr;
            e = pool_take(reinterpret_cast<void **>(&base), tests + boxes + starts + 3 * n * sizeof(float), s);
            if (e == cudaSuccess)
            {
                out.tests = reinterpret_cast<float *>(base);
                out.aabbs = reinterpret_cast<float *>(base + tests);
                out.starts = reinterpret_cast<uint32_t *>(base + tests + boxes);
                out.points = reinterpret_cast<float *>(base + tests + boxes + starts);
                e = cudaMemcpyAsync(out.points, xyz, 3 * n * sizeof(float), cudaMemcpyDeviceToDevice, s);
            }
        }
        // scratch of fixed size, and the lists' two buffers: level d's lists lie in the one, its
        // children's go to the other
        float *px = nullptr, *py = nullptr, *pz = nullptr, *key = nullptr, *cell = nullptr;
        uint32_t *ord = nullptr, *pos = nullptr, *orders = nullptr, *blocks = nullptr, *items[2] = {nullptr, nullptr};
        ulonglong2 *range[2] = {nullptr, nullptr};
        unsigned long long *used = nullptr, cap[2] = {0, 0};
        NodeInfo *info = nullptr;
        Summary *d_sum = nullptr;
        int *full = nullptr;
        char *scratch = nullptr;
        while (e == cudaSuccess)
        {
            size_t bytes = 0;
            auto carve = [&](auto **p, size_t count) {
                const size_t at = bytes;
                bytes += (std::max<size_t>(count, 1) * sizeof(**p) + 255) & ~size_t(255);
                *p = scratch ? reinterpret_cast<std::remove_reference_t<decltype(*p)>>(scratch + at) : nullptr;
            };
            auto carve_all = [&]() {
                bytes = 0;
                carve(&used, 32);
                carve(&full, 1);
                carve(&d_sum, 1);
                carve(&px, N);
                carve(&py, N);
                carve(&pz, N);
                carve(&key, N);
                carve(&ord, N);
                carve(&pos, N);
                carve(&orders, subtrees ? N * (nlog2 - d0) : 1);
                carve(&cell, 6 * N);
                carve(&range[0], N);
                carve(&range[1], N);
                carve(&info, N);
                carve(&blocks, N);
            };
            carve_all();
            e = pool_take(reinterpret_cast<void **>(&scratch), bytes, s);
            for (int k = 0; k < 2 && e == cudaSuccess; ++k)
            {
                cap[k] = room.entries();
                e = pool_take(reinterpret_cast<void **>(&items[k]), cap[k] * sizeof(uint32_t), s);
            }
            if (e == cudaSuccess)
            {
                carve_all();
                break;
            }
            for (void *p : {static_cast<void *>(scratch), static_cast<void *>(items[0]), static_cast<void *>(items[1])})
                pool_give(p, s);
            scratch = nullptr;
            items[0] = items[1] = nullptr;
            const unsigned long long tried = room.entries();
            if (e == cudaErrorMemoryAllocation && (room.shrink() || subtrees))
            {
                // with less, then; at the least without the subtrees' orders
                cudaGetLastError();
                subtrees = subtrees && room.entries() < tried;
                e = cudaSuccess;
            }
        }
        const float *axis[3] = {px, py, pz};
        // counters, *full and the root's empty list are zeros
        if (e == cudaSuccess)
            e = cudaMemsetAsync(used, 0, reinterpret_cast<char *>(d_sum) - reinterpret_cast<char *>(used), s);
        if (e == cudaSuccess)
            e = cudaMemsetAsync(range[0], 0, sizeof(ulonglong2), s);
        if (e == cudaSuccess)
            init_points<<<grid_of(N, 256), 256, 0, s>>>(xyz, static_cast<long long>(n), N, px, py, pz, ord);
        Summary sum{};
        // Every level is queued without a look at its lists.  If one ran out of room the levels below did
        // nothing: it gets a buffer of what the counter says and the build goes on from there.
        int from = 0;
        while (e == cudaSuccess)
        {
            for (int d = from; d < nlog2 && e == cudaSuccess; ++d)
            {
                const long long nodes = 1ll << d, S = N >> d;
                const bool tree = subtrees && d >= d0, sorted = d == from && sum.full;
                const uint32_t *order = tree ? orders + static_cast<long long>(d - d0) * N : ord;
                if (tree && !sorted && (d == d0 || d == d1))
                {
                    // full tiles down to nodes of kSmallTile entries, which then sort on more SMs
                    // (2,048 entries on one: 94 us for all eleven levels)
                    const int tile = d == d1 ? static_cast<int>(S) : T;
                    sort_subtrees<<<static_cast<unsigned>(N / tile), std::max(tile / 2, 32), 0, s>>>(
                        px, py, pz, N, d, d < d1 ? d1 : nlog2, tile, r_max, full, ord, orders + static_cast<long long>(d - d0) * N,
                        out.tests, info);
                }
                else if (!tree && !sorted)
                {
                    load_keys<<<grid_of(N, 256), 256, 0, s>>>(ord, axis[d % 3], N, full, key, pos);
                    // strides below the tile in shared memory, the longer ones one launch each
                    const long long st = std::min<long long>(S, kSortTile);
                    const unsigned tiles = static_cast<unsigned>(N / st),
                                   threads = static_cast<unsigned>(std::max<long long>(st / 2, 32));
                    bitonic_tile<<<tiles, threads, 0, s>>>(key, pos, ord, S, 2, st, full);
                    for (long long k = 2 * st; k <= S; k <<= 1)
                    {
                        for (long long j = k >> 1; j >= st; j >>= 1)
                            bitonic_stage<<<grid_of(N, 256), 256, 0, s>>>(key, pos, ord, N, k, j, S, full);
                        bitonic_tile<<<tiles, threads, 0, s>>>(key, pos, ord, S, k, k, full);
                    }
                    split_nodes<<<grid_of(nodes, 128), 128, 0, s>>>(key, N, d, r_max, full, out.tests, info);
                }
                const int p = d & 1, c = 1 - p;
                child_lists<<<static_cast<unsigned>(nodes), kListBlock, 0, s>>>(range[p], items[p], axis[d % 3], N, d, info, order, cap[c],
                                                                               used, full, range[c], items[c]);
                e = cudaGetLastError();
            }
            LeafParams lp{range[nlog2 & 1], items[nlog2 & 1], px, py, pz, ord, cell, 0.0f, 0.0f};
            {
                const float l1 = r_max + r_point, l0 = r_min + r_point;
                lp.max_l2 = l1 * l1;
                lp.min_l2 = l0 * l0;
            }
            unsigned long long h_used[32] = {};
            if (e == cudaSuccess)
            {
                leaf_cells<<<grid_of(N, 256), 256, 0, s>>>(out.tests, nlog2, full, cell);
                count_leaves<<<static_cast<unsigned>(N), kListBlock, 0, s>>>(lp, full, blocks);
                finish_tree<<<2, 1024, 0, s>>>(blocks, N, out.starts, ord, px, py, pz, out.tests, full, d_sum);
                e = cudaGetLastError();
            }
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(&sum, d_sum, sizeof(sum), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(h_used, used, sizeof(h_used), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess)
                e = cudaStreamSynchronize(s);
            if (e != cudaSuccess)
                break;
            if (!sum.full)
            {
                e = pool_take(reinterpret_cast<void **>(&out.aff), std::max<size_t>(24 * sum.blocks, 4) * sizeof(float), s);
                if (e == cudaSuccess)
                {
                    write_leaves<<<static_cast<unsigned>(N), kListBlock, 0, s>>>(lp, out.starts, out.aff, out.aabbs);
                    e = cudaGetLastError();
                }
                break;
            }
            // what the buffer holds, the lists of the level above, has been read
            from = sum.full - 1;
            const int c = 1 - (from & 1);
            pool_give(items[c], s);
            items[c] = nullptr;
            cap[c] = h_used[from];
            e = pool_take(reinterpret_cast<void **>(&items[c]), cap[c] * sizeof(uint32_t), s);
            if (e == cudaSuccess)
                e = cudaMemsetAsync(used + from, 0, sizeof(*used), s);
            if (e == cudaSuccess)
                e = cudaMemsetAsync(full, 0, sizeof(*full), s);
        }
        for (void *p : {static_cast<void *>(scratch), static_cast<void *>(items[0]), static_cast<void *>(items[1])})
            pool_give(p, s);
        if (e == cudaSuccess)
        {
            out.blocks = sum.blocks;
            for (int k = 0; k < 6; ++k)
                out.top[k] = sum.top[k];
            for (int k = 0; k < 3; ++k)
                out.top_tests[k] = sum.top_tests[k];
            return VG_OK;
        }
        cudaStreamSynchronize(s);
        out.release();
        return set_error(VG_ERR_CUDA, std::string("CAPT build on the GPU: ") + cudaGetErrorString(e));
    }

    void DeviceCapt::release()
    {
        // tests is the start of one allocation with aabbs, starts and points
        pool_give(tests, 0);
        pool_give(aff, 0);
        tests = aabbs = aff = points = nullptr;
        starts = nullptr;
    }
}  // namespace vg
