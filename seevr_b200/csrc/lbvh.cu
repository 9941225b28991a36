// lbvh.cu — linear BVH over AABBs, following the LBVH of bvh.comp:
// centroids (bvh.comp:69-79), centroid bounds (101-165), 30-bit Morton codes
// (32-46, 169-183), a stable LSD radix sort (185-295), the Karras 2012
// hierarchy with the index tiebreak for equal codes (59-65, 299-348), leaf
// boxes (352-368) and the boxes of the inner nodes, bottom-up (372-397).
//
// The sort is a onesweep radix sort: 8-bit digits (4 passes for 32-bit
// keys), a histogram of all digits counted where the keys are made, and per
// pass one kernel in which every tile ranks its keys stably (warp match_any
// multisplit), publishes its per-digit counts and resolves its global
// offsets by decoupled look-back.  A stable LSD sort of the same keys gives
// one permutation, so the order equals bvh.comp's 4-bit, 8-pass sort.
//
// The body broadphase traverses the tree once per body to count and once
// to write, emitting pairs (i, j>i) in canonical lexicographic order: the
// same set as the all-pairs test of physics.comp:451-472 (node boxes are
// exact unions of leaf boxes, so every overlapping leaf is reached).  Rows
// of static bodies, which can hold thousands of partners (a ground box), are
// traversed by whole blocks instead of one thread.
#include <algorithm>

#include "common.cuh"
#include "lbvh.cuh"

namespace seevr {

// ---- Morton codes (bvh.comp:32-46) ---------------------------------------
__device__ __forceinline__ uint32_t expand_bits(uint32_t v) {
    v &= 0x3FFu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}
__device__ __forceinline__ uint32_t quantize10(float x) {
    float t = x * 1024.0f;
    t = t < 0.0f ? 0.0f : (t > 1023.0f ? 1023.0f : t);
    return uint32_t(t);
}
__device__ __forceinline__ uint32_t morton3d(float x, float y, float z) {
    return (expand_bits(quantize10(x)) << 2) | (expand_bits(quantize10(y)) << 1) |
           expand_bits(quantize10(z));
}

// float <-> order-preserving uint (for exact atomic min/max of floats)
__device__ __forceinline__ uint32_t f2o(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o);
}

// ---- centroids + bounds ----------------------------------------------------
// bounds_o[0..2] = ordered min, [3..5] = complement of the ordered max (both by
// atomicMin), initialised to 0xFFFFFFFF by the caller.  Both kernels also clear the
// sort's histogram and look-back words.
struct SortState {
    uint32_t* hist;
    uint32_t* status;
    uint32_t words;  // of status
    __device__ __forceinline__ void clear() const {
        const uint32_t stride = gridDim.x * blockDim.x;
        for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < words; t += stride) status[t] = 0;
        for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < 4 * 256; t += stride) hist[t] = 0;
    }
};
__global__ void k_body_centroids(const float* __restrict__ aabb_min,
                                 const float* __restrict__ aabb_max, uint32_t n,
                                 float* __restrict__ centroid, uint32_t* bounds_o, SortState sort) {
    __shared__ uint32_t smn[3], smx[3];
    sort.clear();
    if (threadIdx.x < 3) {
        smn[threadIdx.x] = 0xFFFFFFFFu;
        smx[threadIdx.x] = 0xFFFFFFFFu;
    }
    __syncthreads();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        // body centroid = AABB centre
        const f3 c = scale(0.5f, add(ld3(aabb_min, i), ld3(aabb_max, i)));
        st3(centroid, i, c);
        atomicMin(&smn[0], f2o(c.x));
        atomicMin(&smn[1], f2o(c.y));
        atomicMin(&smn[2], f2o(c.z));
        atomicMin(&smx[0], ~f2o(c.x));
        atomicMin(&smx[1], ~f2o(c.y));
        atomicMin(&smx[2], ~f2o(c.z));
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        atomicMin(&bounds_o[threadIdx.x], smn[threadIdx.x]);
        atomicMin(&bounds_o[3 + threadIdx.x], smx[threadIdx.x]);
    }
}

// triangle centroids (bvh.comp:69-79)
__global__ void k_tri_centroids(const float* __restrict__ verts, const uint32_t* __restrict__ idx,
                                uint32_t n, float* __restrict__ centroid, uint32_t* bounds_o,
                                SortState sort) {
    __shared__ uint32_t smn[3], smx[3];
    sort.clear();
    if (threadIdx.x < 3) {
        smn[threadIdx.x] = 0xFFFFFFFFu;
        smx[threadIdx.x] = 0xFFFFFFFFu;
    }
    __syncthreads();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const uint32_t i0 = idx[size_t(i) * 3], i1 = idx[size_t(i) * 3 + 1], i2 = idx[size_t(i) * 3 + 2];
        f3 c;
        c.x = (verts[size_t(i0) * 3] + verts[size_t(i1) * 3] + verts[size_t(i2) * 3]) / 3.0f;
        c.y = (verts[size_t(i0) * 3 + 1] + verts[size_t(i1) * 3 + 1] + verts[size_t(i2) * 3 + 1]) / 3.0f;
        c.z = (verts[size_t(i0) * 3 + 2] + verts[size_t(i1) * 3 + 2] + verts[size_t(i2) * 3 + 2]) / 3.0f;
        st3(centroid, i, c);
        atomicMin(&smn[0], f2o(c.x));
        atomicMin(&smn[1], f2o(c.y));
        atomicMin(&smn[2], f2o(c.z));
        atomicMin(&smx[0], ~f2o(c.x));
        atomicMin(&smx[1], ~f2o(c.y));
        atomicMin(&smx[2], ~f2o(c.z));
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        atomicMin(&bounds_o[threadIdx.x], smn[threadIdx.x]);
        atomicMin(&bounds_o[3 + threadIdx.x], smx[threadIdx.x]);
    }
}

// ---- onesweep radix sort ---------------------------------------------------
constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 4;  // keys per thread, ranked one after the other
constexpr int kSortTile = kSortThreads * kSortItems;  // 2048
constexpr uint32_t kRadix = 256;

// Digits of a block's keys, counted in shared memory and added to the global
// histogram [4][256].
struct DigitCounts {
    uint32_t* sh;  // [4 * kRadix]
    __device__ __forceinline__ void clear() const {
        for (uint32_t t = threadIdx.x; t < 4 * kRadix; t += blockDim.x) sh[t] = 0;
    }
    __device__ __forceinline__ void add(uint32_t key) const {
#pragma unroll
        for (uint32_t p = 0; p < 4; ++p) atomicAdd(&sh[p * kRadix + ((key >> (8 * p)) & 0xFFu)], 1u);
    }
    __device__ __forceinline__ void flush(uint32_t* hist) const {
        for (uint32_t t = threadIdx.x; t < 4 * kRadix; t += blockDim.x)
            if (sh[t]) atomicAdd(&hist[t], sh[t]);
    }
};

__global__ void k_sort_counts(const uint32_t* __restrict__ keys, const uint32_t* n_dev, uint32_t n_cap,
                              uint32_t* __restrict__ hist) {
    __shared__ uint32_t sh[4 * kRadix];
    const DigitCounts counts{sh};
    wait_for_previous();
    const uint32_t n = n_dev ? min(*n_dev, n_cap) : n_cap;
    if (blockIdx.x * blockDim.x >= n) return;
    counts.clear();
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        counts.add(keys[i]);
    __syncthreads();
    counts.flush(hist);
}

// One LSD pass on digit `pass`.  status: [1 + tiles*256] u32, zero before the first
// pass; status[0] is the tile ticket, which goes on from pass to pass.  A word's bits
// 30-31 tell its state, bits 0-29 hold a value (n < 2^30).  A pass ends with every
// word an inclusive prefix, so that state is the next pass's "not yet", and the even
// and the odd passes' states differ: no clear between them.  The time is latency: the
// keys' loads, a warp's ranking and the look-back.  With eight keys per thread, each
// loaded when it is ranked, loads and ranking took 10,300 cycles of a tile; with all
// loads issued first 5,700, and a thread now ranks four keys.  A look-back reads four
// tiles ahead (1, 8 and 32: 1, 0 and 13% slower builds).
constexpr uint32_t kAhead = 4;
__global__ void __launch_bounds__(kSortThreads)
    k_sort_onesweep(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                    uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
                    const uint32_t* n_dev, uint32_t n_cap, uint32_t pass,
                    const uint32_t* __restrict__ hist, uint32_t* status, uint32_t* err,
                    uint32_t wait_limit) {
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_warp_hist[kSortWarps][kRadix];
    __shared__ uint32_t s_bin_off[kRadix], s_bins[kRadix / 32];
    wait_for_previous();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, shift = 8 * pass;
    const uint32_t n = n_dev ? min(*n_dev, n_cap) : n_cap;
    if (threadIdx.x == 0) {
        const uint32_t ticket = atomicAdd(status, 1u) - pass * gridDim.x;
        // no pass after one that gave up: slots it left unwritten hold keys that the
        // histogram does not count, and their digits' places run past the end
        s_tile = halted(err) ? kNone : ticket;
    }
    // the digit's first slot: exclusive scan of the histogram (a digit per thread)
    const uint32_t digits = threadIdx.x < kRadix ? hist[pass * kRadix + threadIdx.x] : 0u;
    uint32_t bin = digits;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, bin, off);
        if (lane >= uint32_t(off)) bin += y;
    }
    if (lane == 31 && warp < kRadix / 32) s_bins[warp] = bin;
    for (uint32_t t = threadIdx.x; t < kSortWarps * kRadix; t += blockDim.x)
        (&s_warp_hist[0][0])[t] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint32_t tiles = (n + kSortTile - 1) / kSortTile;
    if (tile >= tiles) return;
    // warp w owns keys [base_w, base_w + 32*kSortItems), processed in order
    const uint32_t base_w = tile * kSortTile + warp * 32 * kSortItems;
    uint32_t key[kSortItems], val[kSortItems], rank[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {  // all on their way before the first is ranked
        const uint32_t i = base_w + k * 32 + lane;
        key[k] = i < n ? keys_in[i] : 0xFFFFFFFFu;
        val[k] = i < n ? vals_in[i] : 0u;
    }
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const bool valid = base_w + k * 32 + lane < n;
        const uint32_t d = (key[k] >> shift) & 0xFFu;
        const unsigned active = __ballot_sync(0xFFFFFFFFu, valid);
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, valid ? d : 0x100u) & active;
        uint32_t before = 0;
        if (valid) {
            const uint32_t leader = __ffs(peers) - 1;
            const uint32_t cnt = __popc(peers);
            const uint32_t lt = __popc(peers & ((1u << lane) - 1u));
            if (lane == leader) {
                before = s_warp_hist[warp][d];
                s_warp_hist[warp][d] = before + cnt;
            }
            before = __shfl_sync(peers, before, leader);
            rank[k] = before + lt;
        } else {
            rank[k] = 0;
        }
        __syncwarp();
    }
    __syncthreads();
    // per digit: exclusive offsets over warps and the tile aggregate
    if (threadIdx.x < kRadix) {
        uint32_t agg = 0;
        const uint32_t d = threadIdx.x;
        for (uint32_t w = 0; w < kSortWarps; ++w) {
            const uint32_t c = s_warp_hist[w][d];
            s_warp_hist[w][d] = agg;
            agg += c;
        }
        // decoupled look-back for digit d
        const uint32_t aggregate = pass & 1u ? 3u : 1u, prefix = pass & 1u ? 0u : 2u;
        uint32_t* st = status + 1;
        uint32_t excl = 0;
        if (tile > 0) {
            atomicExch(&st[size_t(tile) * kRadix + d], (aggregate << 30) | agg);
            uint32_t spins = 0;
            bool found = false;
            for (int p = int(tile) - 1; p >= 0 && !found;) {
                uint32_t word[kAhead];
#pragma unroll
                for (uint32_t q = 0; q < kAhead; ++q)
                    word[q] = *reinterpret_cast<volatile uint32_t*>(&st[size_t(max(p - int(q), 0)) * kRadix + d]);
                bool waits = false;
#pragma unroll
                for (uint32_t q = 0; q < kAhead; ++q) {
                    const uint32_t f = word[q] >> 30;
                    if (found || waits || p < 0) continue;
                    waits = f != aggregate && f != prefix;
                    if (waits) continue;
                    excl += word[q] & 0x3FFFFFFFu;
                    found = f == prefix;
                    --p;
                }
                if (waits && ++spins > wait_limit) {
                    atomicOr(err, kFlagTimeout);
                    break;
                }
            }
        }
        atomicExch(&st[size_t(tile) * kRadix + d], (prefix << 30) | (excl + agg));
        uint32_t before = 0;
        for (uint32_t q = 0; q < warp; ++q) before += s_bins[q];
        s_bin_off[d] = before + bin - digits + excl;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t i = base_w + k * 32 + lane;
        if (i < n) {
            const uint32_t d = (key[k] >> shift) & 0xFFu;
            const uint32_t dst = s_bin_off[d] + s_warp_hist[warp][d] + rank[k];
            keys_out[dst] = key[k];
            vals_out[dst] = val[k];
        }
    }
}

// ---- hierarchy, leaves and boxes (bvh.comp:59-65, 299-397) --------------------
// The Karras hierarchy and its boxes in one bottom-up pass (the merge order of
// Apetrei 2014).  Between the sorted positions p and p + 1 lies one split of the
// tree.  A subtree over positions [lo, hi] is a child of the split at hi when its
// first and last keys differ from their outer neighbours' the way a left child's do
// (delta below), else of the split at lo - 1; both children meet there, and the
// second one to arrive goes on as their parent.  Karras numbers a left child by its
// last position, a right child by its first, so the links are known at the merge
// as well.
//
// The time is that of the longest path, a merge after the other.  A thread per leaf
// that met its siblings in global memory took up to 32 merges of 2,400 cycles each (a
// fence, an atomic and two dependent reads), after a kernel for the links and one for
// the leaves.  Here a block first merges what lies within its 1,024 leaves, in shared
// memory, and writes those nodes in their order; about a dozen subtrees stay and meet
// those of other blocks in global memory.  They post their box without a fence: no
// box holds kUnset, which every node's box is filled with beforehand, so the sibling,
// told by the atomic that it is second, reads the box until it has arrived.
// 134,156 triangles: 39 us (19 us of them in shared memory), 82 us for the three
// kernels; with the sort, the whole build 110 us, 198 us before.  (One block that merges
// all blocks' subtrees in its shared memory instead: a build of 141 us.)
constexpr uint32_t kTreeThreads = 1024;
constexpr uint32_t kUnset = 0xFFA5C3E1u;  // a NaN that no arithmetic makes
__device__ __forceinline__ bool arrived(float x) { return __float_as_uint(x) != kUnset; }
__device__ __forceinline__ float read_now(const float* p) { return *reinterpret_cast<const volatile float*>(p); }

// A caller's vertex may hold any bits: kUnset becomes the quiet NaN of its payload, so
// that no box is taken for one that has not arrived.
__device__ __forceinline__ float unmark(float x) {
    return arrived(x) ? x : __uint_as_float(kUnset | 0x00400000u);
}
__device__ __forceinline__ f3 unmark(f3 v) {
    return mk(unmark(v.x), unmark(v.y), unmark(v.z));
}

// Length of the common prefix of the codes at positions i < n - 1 and i + 1, ties by
// position.
__device__ __forceinline__ int delta(uint32_t a, uint32_t b, uint32_t i) {
    return a == b ? 32 + __clz(i ^ (i + 1u)) : __clz(a ^ b);
}

struct Box {
    f3 mn, mx;
};

// Where a build leaves its nodes: internal node p at p, the leaf at position i at
// n - 1 + i.
struct TriTree {
    TriOut o;
    const float* verts;
    const uint32_t* idx;
    const uint32_t* vals;
    __device__ __forceinline__ Box leaf_box(uint32_t i) const {
        const uint32_t pi = vals[i];
        const f3 v0 = ld3(verts, idx[size_t(pi) * 3]), v1 = ld3(verts, idx[size_t(pi) * 3 + 1]),
                 v2 = ld3(verts, idx[size_t(pi) * 3 + 2]);
        return Box{unmark(vmin(vmin(v0, v1), v2)), unmark(vmax(vmax(v0, v1), v2))};
    }
    __device__ __forceinline__ void leaf(uint32_t i, uint32_t node, const Box& b) const {
        if (o.prim_idx) o.prim_idx[i] = vals[i];
        o.left[node] = i;
        if (o.count) o.count[node] = 1;
        box(node, b);
    }
    __device__ __forceinline__ void box(uint32_t node, const Box& b) const {
        st3(o.node_min, node, b.mn);
        st3(o.node_max, node, b.mx);
    }
    __device__ __forceinline__ void inner(uint32_t node, uint32_t l, uint32_t r, const Box& b) const {
        o.left[node] = l;
        o.right[node] = r;
        o.parent[l] = node;
        o.parent[r] = node;
        if (o.count) o.count[node] = 0;
        box(node, b);
    }
    __device__ __forceinline__ Box read(uint32_t node) const {
        const float *a = o.node_min + size_t(node) * 3, *b = o.node_max + size_t(node) * 3;
        return Box{mk(read_now(a), read_now(a + 1), read_now(a + 2)),
                   mk(read_now(b), read_now(b + 1), read_now(b + 2))};
    }
    __device__ __forceinline__ void unset(uint32_t node) const {
        const float u = __uint_as_float(kUnset);
        box(node, Box{mk(u, u, u), mk(u, u, u)});
    }
    __device__ __forceinline__ void root() const { o.parent[0] = kNone; }
};

// The body tree: one 32-byte record per node, lo = (min, left child or, for a leaf,
// its body), hi = (max, right child or kLeafBit).  A traversal step reads one sector.
constexpr uint32_t kLeafBit = 0x80000000u;
struct BodyTree {
    const float* aabb_min;
    const float* aabb_max;
    const uint32_t* vals;
    float4* packed;
    __device__ __forceinline__ void put(uint32_t node, uint32_t l, uint32_t r, const Box& b) const {
        packed[2 * size_t(node)] = make_float4(b.mn.x, b.mn.y, b.mn.z, __uint_as_float(l));
        packed[2 * size_t(node) + 1] = make_float4(b.mx.x, b.mx.y, b.mx.z, __uint_as_float(r));
    }
    __device__ __forceinline__ Box leaf_box(uint32_t i) const {
        return Box{ld3(aabb_min, vals[i]), ld3(aabb_max, vals[i])};
    }
    __device__ __forceinline__ void leaf(uint32_t i, uint32_t node, const Box& b) const {
        put(node, vals[i], kLeafBit, b);
    }
    __device__ __forceinline__ void inner(uint32_t node, uint32_t l, uint32_t r, const Box& b) const {
        put(node, l, r, b);
    }
    __device__ __forceinline__ Box read(uint32_t node) const {
        const float* p = reinterpret_cast<const float*>(packed + 2 * size_t(node));
        return Box{mk(read_now(p), read_now(p + 1), read_now(p + 2)),
                   mk(read_now(p + 4), read_now(p + 5), read_now(p + 6))};
    }
    __device__ __forceinline__ void unset(uint32_t node) const {
        const float u = __uint_as_float(kUnset);
        put(node, 0, 0, Box{mk(u, u, u), mk(u, u, u)});
    }
    __device__ __forceinline__ void root() const {}
};

// step_morton (bvh.comp:169-183); also writes identity values, the decoded bounds
// (bounds_f) and the codes' digit counts.  One block of many threads per SM at most,
// so that few blocks add to the histogram.
constexpr uint32_t kMortonThreads = 512;
template <class Tree>
__global__ void k_morton(const float* __restrict__ centroid, uint32_t n,
                         const uint32_t* __restrict__ bounds_o, uint32_t* __restrict__ keys,
                         uint32_t* __restrict__ vals, float* bounds_f, uint32_t* __restrict__ flags, Tree tree,
                         uint32_t* __restrict__ hist) {
    __shared__ uint32_t sh[4 * kRadix];
    const DigitCounts counts{sh};
    wait_for_previous();
    counts.clear();
    __syncthreads();
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x;
    const f3 bmin = mk(o2f(bounds_o[0]), o2f(bounds_o[1]), o2f(bounds_o[2]));
    const f3 bmax = mk(o2f(~bounds_o[3]), o2f(~bounds_o[4]), o2f(~bounds_o[5]));
    if (first == 0 && bounds_f) {
        st3(bounds_f, 0, bmin);
        st3(bounds_f, 1, bmax);
    }
    const f3 ext = sub(bmax, bmin);
    const f3 inv = mk(ext.x > 1e-6f ? 1.0f / ext.x : 0.0f, ext.y > 1e-6f ? 1.0f / ext.y : 0.0f,
                      ext.z > 1e-6f ? 1.0f / ext.z : 0.0f);
    for (uint32_t i = first; i < n; i += gridDim.x * blockDim.x) {
        const f3 c = hadamard(sub(ld3(centroid, i), bmin), inv);
        const uint32_t key = morton3d(c.x, c.y, c.z);
        keys[i] = key;
        vals[i] = i;
        counts.add(key);
        if (i + 1 < n) {  // for the tree: no arrivals, no boxes
            flags[i] = 0;
            tree.unset(i);
        }
        tree.unset(n - 1 + i);
    }
    __syncthreads();
    counts.flush(hist);
}

// Node of the subtree over positions [lo, hi], given the prefix lengths at its ends.
__device__ __forceinline__ uint32_t node_of(uint32_t lo, uint32_t hi, int dl, int dr, uint32_t n) {
    return lo == hi ? n - 1 + lo : dl < 0 && dr < 0 ? 0u : dl > dr ? lo : hi;
}
// The children at a split of the subtree over [lo, hi].
__device__ __forceinline__ uint32_t left_of(uint32_t lo, uint32_t split, uint32_t n) {
    return lo == split ? n - 1 + split : split;
}
__device__ __forceinline__ uint32_t right_of(uint32_t hi, uint32_t split, uint32_t n) {
    return hi == split + 1 ? n + split : split + 1;
}

__device__ __forceinline__ void block_fence() { asm volatile("fence.acq_rel.cta;" ::: "memory"); }

// ---- subtrees of a list, merged in shared memory ----
// The list's subtrees cover neighbouring ranges of positions.  Between subtrees k and
// k + 1 lies the split at the last position of k; its prefix length is delta[k + 1]
// (delta[0] and delta[m]: the list's edges, -1 at the ends of the tree).  Nothing is
// written to global memory meanwhile: the fences would wait for it.
struct Merges {
    uint32_t m;
    const signed char* delta;  // [m + 1]
    uint32_t* met;             // [m] 2 (other end + 1) + side, zero before; kNone: merged
    float* box;                // [6][m] of subtrees that wait, at the end next to the split
    __device__ __forceinline__ void put(uint32_t at, const Box& b) const {
        volatile float* p = box + at;
        p[0] = b.mn.x;
        p[m] = b.mn.y;
        p[2 * m] = b.mn.z;
        p[3 * m] = b.mx.x;
        p[4 * m] = b.mx.y;
        p[5 * m] = b.mx.z;
    }
    __device__ __forceinline__ Box get(uint32_t at) const {
        const volatile float* p = box + at;
        return Box{mk(p[0], p[m], p[2 * m]), mk(p[3 * m], p[4 * m], p[5 * m])};
    }
    // Subtree k, box b, merged upwards for as long as it is the second one at its
    // splits.  done(s, a, z, right, box): the subtree [a, z], merged at the split after
    // s, a right child or not.  left(a, z): the subtree's sibling reaches over the
    // list's edge (its box waits at the end next to the split).
    template <class Done, class Left>
    __device__ __forceinline__ void climb(uint32_t k, Box b, Done done, Left left) const {
        uint32_t a = k, z = k, s = 0;
        for (bool leaf = true;; leaf = false) {
            const int dl = delta[a], dr = delta[z + 1];
            const bool right = dl > dr;
            if (!leaf) done(s, a, z, right, b);
            if (dl < 0 && dr < 0) return;  // the root
            put(right ? a : z, b);
            if (right ? a == 0 : z + 1 == m) {
                left(a, z);
                return;
            }
            s = right ? a - 1 : z;
            block_fence();
            const uint32_t other = atomicExch(&met[s], 2u * ((right ? z : a) + 1u) + (right ? 1u : 0u));
            if (other == 0u) return;  // the sibling will come here
            block_fence();
            met[s] = kNone;
            const uint32_t end = (other >> 1) - 1u;
            const Box o = get(right ? s : s + 1);
            b = right ? Box{vmin(o.mn, b.mn), vmax(o.mx, b.mx)} : Box{vmin(b.mn, o.mn), vmax(b.mx, o.mx)};
            if (right) a = end; else z = end;
        }
    }
    // The subtrees that wait for one over the edge: that at the split after s, if any.
    __device__ __forceinline__ bool waits(uint32_t s, uint32_t& a, uint32_t& z) const {
        const uint32_t v = met[s];
        if (v == 0u || v == kNone) return false;
        const uint32_t end = (v >> 1) - 1u;
        a = (v & 1u) ? s + 1 : end;
        z = (v & 1u) ? end : s;
        return true;
    }
};

// What a merge leaves for the write afterwards: range, split and box.
struct Merged {
    uint2* range;  // first and last subtree | split << 16
    float* box;    // [6][stride]
    uint32_t stride;
    __device__ __forceinline__ void put(uint32_t at, uint32_t s, uint32_t a, uint32_t z, const Box& b) const {
        range[at] = make_uint2(a, z | s << 16);
        float* p = box + at;
        p[0] = b.mn.x;
        p[stride] = b.mn.y;
        p[2 * stride] = b.mn.z;
        p[3 * stride] = b.mx.x;
        p[4 * stride] = b.mx.y;
        p[5 * stride] = b.mx.z;
    }
    __device__ __forceinline__ Box get(uint32_t at) const {
        const float* p = box + at;
        return Box{mk(p[0], p[stride], p[2 * stride]), mk(p[3 * stride], p[4 * stride], p[5 * stride])};
    }
};

// (At most 120 subtrees stay: they hang off the paths from the block's two edges to the
// root, and a path has at most 60 nodes, one per prefix length.)  A merged subtree's node lies in the block's range of
// positions, so the nodes are kept and written in their order.
constexpr uint32_t kMostLeft = 128;
constexpr uint32_t kTreeSmem = kTreeThreads * (4 + 4 + 8 + 24 + 24);
template <class Tree>
__global__ void __launch_bounds__(kTreeThreads)
    k_tree(const uint32_t* __restrict__ keys, uint32_t n, Tree tree, uint32_t* flags, uint32_t* err,
           uint32_t wait_limit) {
    extern __shared__ uint32_t tsm[];
    __shared__ signed char s_delta[kTreeThreads + 1];
    __shared__ uint2 s_left[kMostLeft];
    __shared__ uint32_t s_nleft;
    wait_for_previous();
    const uint32_t t = threadIdx.x, first = blockIdx.x * kTreeThreads, i = first + t;
    const uint32_t here = min(kTreeThreads, n - first);
    const bool stop = halted(err);  // the sort gave up: the keys are not ordered
    uint32_t *s_key = tsm, *s_met = tsm + kTreeThreads;
    const Merged merged{reinterpret_cast<uint2*>(tsm + 2 * kTreeThreads),
                        reinterpret_cast<float*>(tsm + 10 * kTreeThreads), kTreeThreads};
    Box b{};
    uint32_t key = 0;
    if (i < n && !stop) {
        s_key[t] = key = keys[i];
        b = tree.leaf_box(i);
    }
    s_met[t] = 0;
    merged.range[t] = make_uint2(kNone, 0);
    if (t == 0) s_nleft = 0;
    // (One answer for the block: another block's wait below may give up meanwhile, and
    // what a part of the block left out the rest would read.)
    if (__syncthreads_or(stop ? 1 : 0)) return;
    if (i < n) {
        const uint32_t after = t + 1 < here ? s_key[t + 1] : i + 1 < n ? keys[i + 1] : 0u;
        s_delta[t + 1] = i + 1 < n ? delta(key, after, i) : -1;
        if (t == 0) s_delta[0] = i > 0 ? delta(keys[i - 1], key, i - 1) : -1;
    }
    __syncthreads();
    const Merges list{here, s_delta, s_met, reinterpret_cast<float*>(tsm + 4 * kTreeThreads)};
    auto stays = [&](uint32_t a, uint32_t z) {
        const uint32_t e = atomicAdd(&s_nleft, 1u);
        if (e < kMostLeft) s_left[e] = make_uint2(a, z);
    };
    if (i < n)
        list.climb(t, b,
                   [&](uint32_t s, uint32_t a, uint32_t z, bool right, const Box& x) {
                       const bool root = z + 1 - a == n;
                       merged.put(root ? 0u : right ? a : z, s, a, z, x);
                   },
                   stays);
    __syncthreads();
    if (i < n) {
        tree.leaf(i, n - 1 + i, b);
        const uint2 r = merged.range[t];
        if (r.x != kNone) {
            const uint32_t a = first + r.x, z = first + (r.y & 0xFFFFu), split = first + (r.y >> 16);
            tree.inner(i, left_of(a, split, n), right_of(z, split, n), merged.get(t));
        }
        if (t + 1 < here && s_met[t] == kNone) flags[i] = 2;  // as two arrivals
        uint32_t a, z;
        if (t + 1 < here && list.waits(t, a, z)) stays(a, z);
    }
    if (n == here && t == 0) tree.root();
    __syncthreads();
    if (t >= min(s_nleft, kMostLeft)) return;
    uint32_t lo = s_left[t].x, hi = s_left[t].y;
    int dl = s_delta[lo], dr = s_delta[hi + 1];
    b = list.get(dl > dr ? lo : hi);
    lo += first;
    hi += first;
    auto split_delta = [&](uint32_t p) { return delta(keys[p], keys[p + 1], p); };
    while (dl >= 0 || dr >= 0) {
        const bool right = dl > dr;
        const uint32_t split = right ? lo - 1 : hi;
        const uint32_t other = atomicExch(&flags[split], 2u * ((right ? hi : lo) + 1u) + (right ? 1u : 0u));
        if (other == 0u) return;  // the sibling will come here
        const uint32_t end = (other >> 1) - 1u;
        const uint32_t node = right ? left_of(end, split, n) : right_of(end, split, n);
        Box o = tree.read(node);
        if (right) lo = end; else hi = end;
        dl = lo > 0 ? split_delta(lo - 1) : -1;
        dr = hi + 1 < n ? split_delta(hi) : -1;
        for (uint32_t polls = 0; !(arrived(o.mn.x) && arrived(o.mn.y) && arrived(o.mn.z) &&
                                   arrived(o.mx.x) && arrived(o.mx.y) && arrived(o.mx.z));
             o = tree.read(node))
            if (++polls > wait_limit) {
                atomicOr(err, kFlagTimeout);
                break;
            }
        b = right ? Box{vmin(o.mn, b.mn), vmax(o.mx, b.mx)} : Box{vmin(b.mn, o.mn), vmax(b.mx, o.mx)};
        tree.inner(node_of(lo, hi, dl, dr, n), left_of(lo, split, n), right_of(hi, split, n), b);
        flags[split] = 2;
    }
    tree.root();
}

cudaError_t init_lbvh() {
    const cudaError_t e = cudaFuncSetAttribute(k_tree<TriTree>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               int(kTreeSmem));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_tree<BodyTree>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTreeSmem));
}

// (In stream order: set up while the sort's last pass runs, its blocks of 1,024 threads
// make the build 126 instead of 118 us.)
template <class Tree>
int launch_tree(const Tree& tree, const uint32_t* keys, uint32_t n, uint32_t* flags, const LbvhScratch& s,
                uint32_t* err, cudaStream_t st) {
    k_tree<Tree><<<(n + kTreeThreads - 1) / kTreeThreads, kTreeThreads, kTreeSmem, st>>>(
        keys, n, tree, flags, err, s.wait_limit);
    return 1;
}

// ---- body pairs by traversal ------------------------------------------------
constexpr int kStack = 64;
constexpr int kRowBuf = 32;

__device__ __forceinline__ bool overlap_box(f3 mna, f3 mxa, f3 mnb, f3 mxb) {
    return !(mxa.x < mnb.x || mxb.x < mna.x || mxa.y < mnb.y || mxb.y < mna.y || mxa.z < mnb.z ||
             mxb.z < mna.z);
}

// Visit every leaf j (original index) with j > lo_j whose box overlaps
// body i's box, excluding static-static; `emit(j)` is called for each.
template <class F>
__device__ __forceinline__ void traverse(const World& w, const LbvhView& t, uint32_t i,
                                         uint32_t lo_j, uint32_t* err, F emit) {
    const f3 mna = ld3(w.aabb_min, i), mxa = ld3(w.aabb_max, i);
    const bool static_i = w.inv_mass[i] <= 0.0f;
    uint32_t stack[kStack];
    int sp = 0;
    stack[sp++] = 0;  // root (n >= 2)
    while (sp > 0) {
        const uint32_t node = stack[--sp];
        const float4 lo = __ldg(&t.packed[2 * size_t(node)]), hi = __ldg(&t.packed[2 * size_t(node) + 1]);
        if (!overlap_box(mna, mxa, mk(lo.x, lo.y, lo.z), mk(hi.x, hi.y, hi.z))) continue;
        const uint32_t a = __float_as_uint(lo.w), b = __float_as_uint(hi.w);
        if (b == kLeafBit) {
            const uint32_t j = a;
            if (j > lo_j && !(static_i && w.inv_mass[j] <= 0.0f)) emit(j);
        } else {
            if (sp + 2 > kStack) {
                atomicOr(err, kFlagTimeout);
                return;
            }
            stack[sp++] = b;
            stack[sp++] = a;
        }
    }
}

// Rows of dynamic bodies, one thread each; static bodies' rows (a ground
// box overlapping thousands of bodies) are left to k_lbvh_static_rows and
// listed here.  A row of at most kRowCache partners is kept, sorted, in
// row_cache, so the write pass copies it instead of traversing again.
// Threads take bodies in Morton order (the tree's leaf order), so a warp's
// bodies are neighbours whose traversals visit the same nodes.
__global__ void k_lbvh_count(World w, LbvhView t, uint32_t* __restrict__ row_count, uint32_t* err,
                             uint32_t* static_list, uint32_t* static_count,
                             uint32_t* __restrict__ row_cache) {
    if (halted(err)) return;  // the tree was not built
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= w.nb) return;
    const uint32_t i = w.nb >= 2 ? t.vals[q] : q;
    if (w.inv_mass[i] <= 0.0f) {
        static_list[atomicAdd(static_count, 1u)] = i;
        if (w.nb < 2) row_count[i] = 0;  // no tree for k_lbvh_static_rows to count by
        return;
    }
    uint32_t c = 0;
    uint32_t buf[kRowCache];
    if (w.nb >= 2)
        traverse(w, t, i, i, err, [&](uint32_t j) {
            if (c < kRowCache) {  // insertion into the ascending buffer
                uint32_t pos = c;
                while (pos > 0 && buf[pos - 1] > j) {
                    buf[pos] = buf[pos - 1];
                    --pos;
                }
                buf[pos] = j;
            }
            ++c;
        });
    row_count[i] = c;
    if (c <= kRowCache)
        for (uint32_t k = 0; k < c; ++k) row_cache[size_t(i) * kRowCache + k] = buf[k];
}

// Rows of static bodies, one block each: a breadth-first traversal whose
// frontier the block's threads expand together.  The partners are marked in a
// bitmap of the bodies in shared memory (up to kBitmapBodies bodies) and read
// out in ascending order.  The count pass leaves them in `found`, which the
// write pass copies when every static body had a block of its own (else it
// traverses again).  1,024 partners among 262,145 bodies: the write pass 4 us;
// 66 us with a second traversal and every partner's rank counted among the others,
// as larger scenes still do.
constexpr uint32_t kBitmapBodies = 360000;
template <bool kWrite>
__global__ void __launch_bounds__(256)
    k_lbvh_static_rows(World w, LbvhView t, uint32_t* row_count, const uint32_t* row_off,
                       const uint32_t* static_list, const uint32_t* static_count, uint32_t* bfs) {
    extern __shared__ uint32_t bits[];
    __shared__ uint32_t sh_next, sh_found, sh_cur, sh_warp[8];
    wait_for_previous();
    if (halted(w.status)) return;  // the tree (or the row offsets) are not valid
    const uint32_t n = w.nb;
    if (n < 2) return;
    uint32_t* fa = bfs + size_t(blockIdx.x) * 3 * 2 * n;
    uint32_t* fb = fa + 2 * n;
    uint32_t* found = fb + 2 * n;
    const uint32_t ns = *static_count, lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t words = n <= kBitmapBodies ? (n + 31) / 32 : 0u;
    if (kWrite && words && ns <= gridDim.x) {  // as the count pass left them
        if (blockIdx.x >= ns) return;
        const uint32_t i = static_list[blockIdx.x], base = row_off[i], cnt = row_count[i];
        for (uint32_t e = threadIdx.x; e < cnt && base + e < w.max_pairs; e += blockDim.x) {
            w.pairs[size_t(base + e) * 2] = i;
            w.pairs[size_t(base + e) * 2 + 1] = found[e];
        }
        return;
    }
    for (uint32_t r = blockIdx.x; r < ns; r += gridDim.x) {
        const uint32_t i = static_list[r];
        const f3 mna = ld3(w.aabb_min, i), mxa = ld3(w.aabb_max, i);
        for (uint32_t k = threadIdx.x; k < words; k += blockDim.x) bits[k] = 0;
        if (threadIdx.x == 0) {
            fa[0] = 0;  // root
            sh_cur = 1;
            sh_found = 0;
        }
        __syncthreads();
        uint32_t* in = fa;
        uint32_t* out = fb;
        while (sh_cur > 0) {
            const uint32_t cur = sh_cur;
            if (threadIdx.x == 0) sh_next = 0;
            __syncthreads();
            for (uint32_t k = threadIdx.x; k < cur; k += blockDim.x) {
                const uint32_t node = in[k];
                const float4 lo = __ldg(&t.packed[2 * size_t(node)]);
                const float4 hi = __ldg(&t.packed[2 * size_t(node) + 1]);
                if (!overlap_box(mna, mxa, mk(lo.x, lo.y, lo.z), mk(hi.x, hi.y, hi.z))) continue;
                const uint32_t a = __float_as_uint(lo.w), b = __float_as_uint(hi.w);
                if (b == kLeafBit) {
                    const uint32_t j = a;
                    // the row owner is static: only dynamic partners count
                    if (j > i && w.inv_mass[j] > 0.0f) {
                        if (words)
                            atomicOr(&bits[j >> 5], 1u << (j & 31u));
                        else
                            found[atomicAdd(&sh_found, 1u)] = j;
                    }
                } else {
                    const uint32_t o = atomicAdd(&sh_next, 2u);
                    out[o] = a;
                    out[o + 1] = b;
                }
            }
            __syncthreads();
            if (threadIdx.x == 0) sh_cur = sh_next;
            uint32_t* tmp = in;
            in = out;
            out = tmp;
            __syncthreads();
        }
        if (words) {  // a run of words per thread
            const uint32_t per = (words + blockDim.x - 1) / blockDim.x;
            const uint32_t k0 = min(threadIdx.x * per, words), k1 = min(k0 + per, words);
            uint32_t sum = 0;
            for (uint32_t k = k0; k < k1; ++k) sum += __popc(bits[k]);
            uint32_t at = sum;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, at, off);
                if (lane >= uint32_t(off)) at += y;
            }
            if (lane == 31) sh_warp[wid] = at;
            __syncthreads();
            for (uint32_t q = 0; q < wid; ++q) at += sh_warp[q];
            if (threadIdx.x == blockDim.x - 1) sh_found = at;
            at -= sum;
            for (uint32_t k = k0; k < k1; ++k)
                for (uint32_t m = bits[k]; m; m &= m - 1) found[at++] = 32 * k + uint32_t(__ffs(int(m))) - 1u;
            __syncthreads();
        }
        const uint32_t cnt = sh_found;
        if (!kWrite) {
            if (threadIdx.x == 0) row_count[i] = cnt;
        } else {
            const uint32_t base = row_off[i];
            for (uint32_t e = threadIdx.x; e < cnt; e += blockDim.x) {
                const uint32_t j = found[e];
                uint32_t rank = words ? e : 0u;
                if (!words)
                    for (uint32_t q = 0; q < cnt; ++q) rank += found[q] < j ? 1u : 0u;
                const uint32_t slot = base + rank;
                if (slot < w.max_pairs) {
                    w.pairs[size_t(slot) * 2] = i;
                    w.pairs[size_t(slot) * 2 + 1] = j;
                }
            }
        }
        __syncthreads();
    }
}

// Writes row i's pairs at row_off[i] in ascending j: a row the count pass
// kept is copied; longer rows are emitted in chunks of up to kRowBuf
// smallest remaining j, one traversal per chunk.
__global__ void k_lbvh_write(World w, LbvhView t, const uint32_t* __restrict__ row_count,
                             const uint32_t* __restrict__ row_off, uint32_t* err,
                             const uint32_t* __restrict__ row_cache) {
    if (halted(err)) return;  // the tree or the row offsets are not valid
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;  // Morton order, as the count
    if (q >= w.nb) return;
    const uint32_t i = w.nb >= 2 ? t.vals[q] : q;
    if (w.inv_mass[i] <= 0.0f) return;  // static rows: k_lbvh_static_rows
    uint32_t remaining = row_count[i];
    uint32_t slot = row_off[i];
    if (remaining <= kRowCache) {
        for (uint32_t k = 0; k < remaining && slot < w.max_pairs; ++k, ++slot) {
            w.pairs[size_t(slot) * 2] = i;
            w.pairs[size_t(slot) * 2 + 1] = row_cache[size_t(i) * kRowCache + k];
        }
        return;
    }
    uint32_t lo = i;
    while (remaining > 0 && slot < w.max_pairs) {
        uint32_t buf[kRowBuf];
        uint32_t nbuf = 0;
        // keep the kRowBuf smallest j > lo, sorted ascending (buf[kRowBuf - 1]
        // is read only once nbuf == kRowBuf, i.e. after every entry is set)
        traverse(w, t, i, lo, err, [&](uint32_t j) {
            if (nbuf == kRowBuf && j >= buf[kRowBuf - 1]) return;
            uint32_t pos = nbuf < kRowBuf ? nbuf++ : kRowBuf - 1;
            while (pos > 0 && buf[pos - 1] > j) {
                buf[pos] = buf[pos - 1];
                --pos;
            }
            buf[pos] = j;
        });
        if (nbuf == 0) break;
        for (uint32_t k = 0; k < nbuf && slot < w.max_pairs; ++k, ++slot) {
            w.pairs[size_t(slot) * 2] = i;
            w.pairs[size_t(slot) * 2 + 1] = buf[k];
        }
        remaining = remaining > nbuf ? remaining - nbuf : 0;
        lo = buf[nbuf - 1];
    }
}

// ---- launchers ---------------------------------------------------------------
static inline uint32_t blocks_for(uint32_t n, uint32_t t) {
    const uint32_t b = (n + t - 1) / t;
    return b ? b : 1;
}

int lbvh_sort(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_tmp,
              uint32_t* vals_tmp, uint32_t* keys_out, uint32_t* vals_out, const uint32_t* n_dev,
              uint32_t n, uint32_t passes, bool counted, const LbvhScratch& s, uint32_t* err,
              cudaStream_t st) {
    int launches = 0;
    if (!counted) {
        launch_after(k_sort_counts, std::min(blocks_for(n, 256), 148u * 4u), 256, 0, st, keys_in, n_dev, n,
                     s.hist);
        ++launches;
    }
    const uint32_t tiles = blocks_for(n, kSortTile);
    const uint32_t* ki = keys_in;
    const uint32_t* vi = vals_in;
    for (uint32_t p = 0; p < passes; ++p) {  // ping-pong, the last pass into out
        const bool tmp = (passes - 1 - p) & 1u;
        uint32_t *ko = tmp ? keys_tmp : keys_out, *vo = tmp ? vals_tmp : vals_out;
        launch_after(k_sort_onesweep, tiles, kSortThreads, 0, st, ki, vi, ko, vo, n_dev, n, p,
                     static_cast<const uint32_t*>(s.hist), s.status, err, s.wait_limit);
        ki = ko;
        vi = vo;
        ++launches;
    }
    return launches;
}

int lbvh_build_bodies(const World& w, const LbvhScratch& s, uint32_t* err, cudaStream_t st) {
    const uint32_t n = w.nb;
    if (n < 2) return 0;
    const BodyTree tree{w.aabb_min, w.aabb_max, s.vals_sorted, s.packed};
    cudaMemsetAsync(s.bounds_o, 0xFF, sizeof(uint32_t) * 6, st);
    const SortState sort{s.hist, s.status, lbvh_status_words(n)};
    k_body_centroids<<<blocks_for(n, 256), 256, 0, st>>>(w.aabb_min, w.aabb_max, n, s.centroid,
                                                         s.bounds_o, sort);
    launch_after(k_morton<BodyTree>, std::min(blocks_for(n, kMortonThreads), 148u), kMortonThreads, 0, st,
                 static_cast<const float*>(s.centroid), n, static_cast<const uint32_t*>(s.bounds_o), s.keys_a,
                 s.vals_a, s.bounds_f, s.flags, tree, s.hist);
    const int k = 2 + lbvh_sort(s.keys_a, s.vals_a, s.keys_b, s.vals_b, s.keys_sorted, s.vals_sorted,
                                nullptr, n, 4, true, s, err, st);
    return k + launch_tree(tree, s.keys_sorted, n, s.flags, s, err, st);
}

int launch_broadphase_lbvh(const World& w, const Scratch& sc, const LbvhScratch& s,
                           cudaStream_t st) {
    const uint32_t n = w.nb;
    if (n == 0) return 0;
    const int k = lbvh_build_bodies(w, s, &sc.status[0], st);
    const LbvhView t{s.vals_sorted, s.packed};
    cudaMemsetAsync(s.static_count, 0, sizeof(uint32_t), st);
    k_lbvh_count<<<blocks_for(n, 128), 128, 0, st>>>(w, t, sc.row_count, &sc.status[0],
                                                     s.static_list, s.static_count, s.row_cache);
    const uint32_t bitmap = n <= kBitmapBodies ? (n + 31) / 32 * 4 : 0u;
    k_lbvh_static_rows<false><<<kStaticBlocks, 256, bitmap, st>>>(w, t, sc.row_count, nullptr,
                                                                 s.static_list, s.static_count, s.bfs);
    launch_exclusive_scan(sc.row_count, sc.row_off, nullptr, n, &w.counters[0], w.max_pairs,
                          kFlagPairOverflow, sc, st);
    k_lbvh_write<<<blocks_for(n, 128), 128, 0, st>>>(w, t, sc.row_count, sc.row_off, &sc.status[0],
                                                     s.row_cache);
    launch_after(k_lbvh_static_rows<true>, kStaticBlocks, 256, bitmap, st, w, t, sc.row_count,
                 static_cast<const uint32_t*>(sc.row_off), static_cast<const uint32_t*>(s.static_list),
                 static_cast<const uint32_t*>(s.static_count), s.bfs);
    return k + 5;
}

int lbvh_build_triangles(const float* verts, const uint32_t* idx, uint32_t n, const LbvhScratch& s,
                         const TriOut& o, uint32_t* err, cudaStream_t st) {
    if (n == 0) return 0;
    const TriTree tree{o, verts, idx, o.sort_idx};
    cudaMemsetAsync(s.bounds_o, 0xFF, sizeof(uint32_t) * 6, st);
    const SortState sort{s.hist, s.status, lbvh_status_words(n)};
    k_tri_centroids<<<blocks_for(n, 256), 256, 0, st>>>(verts, idx, n, o.centroids, s.bounds_o, sort);
    launch_after(k_morton<TriTree>, std::min(blocks_for(n, kMortonThreads), 148u), kMortonThreads, 0, st,
                 static_cast<const float*>(o.centroids), n, static_cast<const uint32_t*>(s.bounds_o), s.keys_a,
                 s.vals_a, o.scene_bounds, o.flags, tree, s.hist);
    const int k = 2 + lbvh_sort(s.keys_a, s.vals_a, s.keys_b, s.vals_b, o.morton, o.sort_idx, nullptr, n, 4,
                                true, s, err, st);
    return k + launch_tree(tree, o.morton, n, o.flags, s, err, st);
}

}  // namespace seevr
