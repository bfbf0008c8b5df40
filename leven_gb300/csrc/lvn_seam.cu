// lvn_seam.cu -- the clipmap's seam meshes on the GPU: GenerateClipmapSeamMesh
// (leven/src/clipmap.cpp:573-610) for a batch of host chunks.  The reference
// gathers the seam nodes of a host and of the active nodes next to it
// (SelectSeamNodes / FilterSeamNode, clipmap.cpp:508-570), builds a pointer
// octree from them (Octree_ConstructUpwards, octree.cpp:90-148), numbers its
// leaves depth first (GenerateVertexIndices, octree.cpp:197-232) and contours
// it recursively (ContourCellProc / ContourFaceProc / ContourEdgeProc /
// ContourProcessEdge, octree.cpp:236-474) on the CPU.
//
// Here the neighbour search, which walks the clipmap's node tree, stays on the
// host; everything that touches seam nodes runs on the device, without building
// the tree:
//   * the depth-first leaf order is the Morton order of the leaves' minimum
//     corners (children are visited x << 2 | y << 1 | z), so the leaves are
//     sorted by Morton key (in parts that fit shared memory) and numbered by rank;
//   * the recursion emits one quad per final edge segment: an edge of the
//     smallest of the four leaves around it, all four present, not all four
//     in one CLIPMAP_LEAF_SIZE block (the straddle test of ContourEdgeProc /
//     ContourFaceProc prunes exactly those), with a sign change on that
//     leaf's edge.  Each leaf tests its 12 edges; the other three leaves come
//     from binary searches of the sorted keys.  This runs over blocks of 256
//     leaves, so a large host spreads over many CTAs;
//   * the recursion's order is restored by a key spelling the path the
//     recursion takes to the segment (cell: child 0-7, face 8-19, edge 20-25
//     in 5 bits; face: sub-face 0-3, edge 4-7 in 3 bits; edge: half in 1 bit),
//     by which the quads are sorted.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <vector>

#include "../../include/lvn.h"
#include "lvn_types.h"

namespace lvn {
namespace {

constexpr int kMaxLeaves = LVN_SEAM_MAX_LEAVES;  // per host
constexpr int kSlotBits = 15;                    // leaf sort entry: (morton << 4 | size log2) << 15 | slot
constexpr int kRankBits = 15;                    // quad payload: 4 ranks of 15 bits, flip at bit 60
static_assert(kMaxLeaves <= (1 << kRankBits) && kMaxLeaves <= (1 << kSlotBits), "rank bits");
constexpr int kMaxLevels = 12;    // log2(2 host size / smallest leaf): path keys of 5 bits per level fit 64 bits
constexpr int kQuadBlock = 256;     // leaves per CTA of the quad enumeration
constexpr int kSmallLeaves = 2048;  // leaf sorts up to this size run several CTAs per SM
constexpr int kBucketBits = 6;      // leaves of larger hosts are sorted in 64 Morton-prefix buckets
constexpr int kBuckets = 1 << kBucketBits;
constexpr int kSmallQuads = 2048;   // as do quad sorts up to this size; larger sorts are split in kParts
constexpr int kParts = 256;
static_assert(kSmallLeaves == kSmallQuads, "k_seam_parts' shared memory");
constexpr size_t kSmallLeafSmem = (size_t)kSmallLeaves * 8;
constexpr size_t kSmallSortSmem = (size_t)kSmallQuads * 16;

// the dual-contouring tables of contour_constants.h, as the reference's
// recursion uses them (its output order depends on them)
__constant__ int8_t cEdgeVMap[12][2] = {{0, 4}, {1, 5}, {2, 6}, {3, 7}, {0, 2}, {1, 3},
                                        {4, 6}, {5, 7}, {0, 1}, {2, 3}, {4, 5}, {6, 7}};
__constant__ int8_t cCellProcFaceMask[12][3] = {{0, 4, 0}, {1, 5, 0}, {2, 6, 0}, {3, 7, 0}, {0, 2, 1}, {4, 6, 1},
                                                {1, 3, 1}, {5, 7, 1}, {0, 1, 2}, {2, 3, 2}, {4, 5, 2}, {6, 7, 2}};
__constant__ int8_t cCellProcEdgeMask[6][5] = {{0, 1, 2, 3, 0}, {4, 5, 6, 7, 0}, {0, 4, 1, 5, 1},
                                               {2, 6, 3, 7, 1}, {0, 2, 4, 6, 2}, {1, 3, 5, 7, 2}};
__constant__ int8_t cFaceProcFaceMask[3][4][3] = {{{4, 0, 0}, {5, 1, 0}, {6, 2, 0}, {7, 3, 0}},
                                                  {{2, 0, 1}, {6, 4, 1}, {3, 1, 1}, {7, 5, 1}},
                                                  {{1, 0, 2}, {3, 2, 2}, {5, 4, 2}, {7, 6, 2}}};
__constant__ int8_t cFaceProcEdgeMask[3][4][6] = {
    {{1, 4, 0, 5, 1, 1}, {1, 6, 2, 7, 3, 1}, {0, 4, 6, 0, 2, 2}, {0, 5, 7, 1, 3, 2}},
    {{0, 2, 3, 0, 1, 0}, {0, 6, 7, 4, 5, 0}, {1, 2, 0, 6, 4, 2}, {1, 3, 1, 7, 5, 2}},
    {{1, 1, 0, 3, 2, 0}, {1, 5, 4, 7, 6, 0}, {0, 1, 5, 0, 4, 1}, {0, 3, 7, 2, 6, 1}}};
__constant__ int8_t cProcessEdgeMask[3][4] = {{3, 2, 1, 0}, {7, 5, 6, 4}, {11, 10, 9, 8}};

__device__ __forceinline__ int cbit(int child, int axis) { return (child >> (2 - axis)) & 1; }


struct SeamHost {
    int32_t min[3];
    int32_t size;
    int32_t unit;        // smallest leaf size among the gathered chunks
    int32_t lev;         // log2(2 size / unit)
    int32_t inside;      // 1: no gathered leaf reaches out of its CLIPMAP_LEAF_SIZE block
    int32_t pair_begin;  // gathered (chunk, neighbour mask) pairs
    int32_t pair_end;
    int64_t sel_off;     // the host's selected seam nodes (room for every node of its pairs)
    int64_t leaf_off;    // the host's leaves in the leaf arrays
    int64_t quad_off;    // the host's quads (12 per leaf at most) in the quad arrays
};

struct SeamArgs {
    const SeamHost* hosts;
    const int4* pairs;            // (chunk, mask of neighbour indices 0-7, host, -)
    const int4* chunks;           // (min xyz, size)
    const int32_t* seam_offsets;  // [num_chunks + 1]
    const lvn_seam_node* seams;
    int vpc;
    int32_t* counts;    // leaves per host
    int32_t* qcounts;   // quads per host
    uint64_t* sel;      // selected leaves' sort entries, per host at sel_off, by bucket
    uint32_t* slots;    // their seam indices, by the slot in the entry
    int32_t* bcount;    // leaves per (host, Morton-prefix bucket)
    const int32_t* bstart;  // the bucket's first slot in the host's region
    int32_t* cursor;    // next slot in the bucket
    const int4* lsort;  // leaf sorts: (host, first slot, count, -)
    uint64_t* ent;      // sorted leaf entries
    uint32_t* leaves;   // seam index per rank
    uint64_t* qkey;     // quad path keys
    uint64_t* qval;     // quad payloads (sorted by key after the sort kernel)
    const int2* items;  // quad enumeration: (host, first leaf)
    int4* parts;        // split sorts' parts: (host, first, count, dealt)
    int32_t* n_parts;
    // emit
    const int64_t* vout_off;
    const int64_t* tout_off;
    lvn_mesh_vertex* vout;
    lvn_mesh_triangle* tout;
    float colour[3];
};

// FilterSeamNode (clipmap.cpp:508-538)
__device__ __forceinline__ bool filter_seam_node(int child, const int32_t b[3], const int32_t mn[3],
                                                 const int32_t mx[3]) {
    switch (child) {
        case 0: return mx[0] == b[0] || mx[1] == b[1] || mx[2] == b[2];
        case 1: return mn[2] == b[2];
        case 2: return mn[1] == b[1];
        case 3: return mn[1] == b[1] || mn[2] == b[2];
        case 4: return mn[0] == b[0];
        case 5: return mn[0] == b[0] || mn[2] == b[2];
        case 6: return mn[0] == b[0] || mn[1] == b[1];
        default: return mn[0] == b[0] && mn[1] == b[1] && mn[2] == b[2];
    }
}

// SelectSeamNodes (clipmap.cpp:542-570): is seam node k of `chunk` one of the
// host's, for any of the neighbour indices in `mask`?  A chunk reached through
// several neighbour indices is tested once with all of them (the reference
// may list such a node twice; the octree it builds holds it once).
__device__ __forceinline__ bool seam_selected(const SeamHost& h, int4 chunk, int mask, const lvn_seam_node& s,
                                              int vpc, int32_t mn[3]) {
    const int node_size = chunk.w / vpc;
    const int extent = (chunk.w / (vpc * 4)) * 4;  // size * LEAF_SIZE_SCALE (clipmap.cpp:553-560)
    mn[0] = s.localspace_min[0] * node_size + chunk.x;
    mn[1] = s.localspace_min[1] * node_size + chunk.y;
    mn[2] = s.localspace_min[2] * node_size + chunk.z;
    for (int a = 0; a < 3; a++)
        if (mn[a] < h.min[a] || mn[a] >= h.min[a] + 2 * h.size) return false;  // AABB::pointIsInside
    const int32_t b[3] = {h.min[0] + h.size, h.min[1] + h.size, h.min[2] + h.size};
    const int32_t mx[3] = {mn[0] + extent, mn[1] + extent, mn[2] + extent};
    for (int i = 0; i < 8; i++)
        if (((mask >> i) & 1) && filter_seam_node(i, b, mn, mx)) return true;
    return false;
}

// bit interleaving by shifts and masks (bit i of v to bit 3i), and back
__device__ __forceinline__ uint64_t part1by2(uint64_t v) {
    v &= 0x1fffffull;
    v = (v | v << 32) & 0x1f00000000ffffull;
    v = (v | v << 16) & 0x1f0000ff0000ffull;
    v = (v | v << 8) & 0x100f00f00f00f00full;
    v = (v | v << 4) & 0x10c30c30c30c30c3ull;
    v = (v | v << 2) & 0x1249249249249249ull;
    return v;
}

__device__ __forceinline__ uint32_t compact1by2(uint64_t v) {
    v &= 0x1249249249249249ull;
    v = (v ^ (v >> 2)) & 0x10c30c30c30c30c3ull;
    v = (v ^ (v >> 4)) & 0x100f00f00f00f00full;
    v = (v ^ (v >> 8)) & 0x1f0000ff0000ffull;
    v = (v ^ (v >> 16)) & 0x1f00000000ffffull;
    v = (v ^ (v >> 32)) & 0x1fffffull;
    return (uint32_t)v;
}

// Morton code of a host-relative position in units of 1 << unit_log: x in
// the highest bit of each triple, as the octree's children are numbered
__device__ __forceinline__ uint64_t morton(const int32_t rel[3], int unit_log, int lev) {
    (void)lev;
    return (part1by2((uint32_t)rel[0] >> unit_log) << 2) | (part1by2((uint32_t)rel[1] >> unit_log) << 1) |
           part1by2((uint32_t)rel[2] >> unit_log);
}

__device__ __forceinline__ void unmorton(uint64_t code, int lev, int unit_log, int32_t rel[3]) {
    (void)lev;
    rel[0] = (int32_t)(compact1by2(code >> 2) << unit_log);
    rel[1] = (int32_t)(compact1by2(code >> 1) << unit_log);
    rel[2] = (int32_t)(compact1by2(code) << unit_log);
}

// SelectSeamNodes for every (host, gathered chunk) pair.  The counting pass
// (Place = false) counts the selected seam nodes per host and per bucket of
// the top kBucketBits bits of their host-relative Morton code (units of the
// host's smallest leaf); the placing pass writes each one's sort entry
// ((morton << 4 | size log2) << 15 | slot) and seam index at a slot of its
// bucket, so that each host's region holds its buckets in Morton order.
template <bool Place>
__global__ void __launch_bounds__(128) k_seam_select(SeamArgs A) {
    const int4 pr = A.pairs[blockIdx.x];
    const SeamHost h = A.hosts[pr.z];
    const int4 ch = A.chunks[pr.x];
    int unit_log = 0;
    while ((1 << unit_log) < h.unit) unit_log++;
    int size_log = 0;
    while ((h.unit << size_log) < ch.w / A.vpc) size_log++;
    const int s0 = A.seam_offsets[pr.x], s1 = A.seam_offsets[pr.x + 1];
    const int lane = threadIdx.x & 31;
    const int shift = 3 * h.lev - kBucketBits;  // lev >= 4: 2 host size / smallest leaf >= 16
    for (int base = s0; base < s1; base += blockDim.x) {
        const int k = base + threadIdx.x;
        int32_t mn[3];
        const bool take = k < s1 && seam_selected(h, ch, pr.y, A.seams[k], A.vpc, mn);
        if (!Place) {
            const unsigned ballot = __ballot_sync(0xffffffffu, take);
            if (lane == 0 && ballot) atomicAdd(&A.counts[pr.z], __popc(ballot));
        }
        if (!take) continue;
        const int32_t rel[3] = {mn[0] - h.min[0], mn[1] - h.min[1], mn[2] - h.min[2]};
        const uint64_t code = morton(rel, unit_log, h.lev);
        const int b = pr.z * kBuckets + (int)(code >> shift);
        if (!Place) {
            atomicAdd(&A.bcount[b], 1);
            continue;
        }
        const int slot = A.bstart[b] + atomicAdd(&A.cursor[b], 1);
        if (slot >= kMaxLeaves) continue;  // the host reported the count; nothing past its region is written
        A.sel[h.sel_off + slot] = ((code << 4 | (uint64_t)size_log) << kSlotBits) | (uint64_t)slot;
        A.slots[h.sel_off + slot] = (uint32_t)k;
    }
}

// Ascending sort of n entries in place (a bitonic network whose first step of
// each merge compares mirrored positions, so every comparator is ascending and
// entries past n never move: any n, no padding), keys with an optional payload.
template <bool Pair>
__device__ void block_sort(uint64_t* key, uint64_t* val, int n) {
    for (int k = 2; k < 2 * n; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            const int mask = j == (k >> 1) ? k - 1 : j;
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                const int l = i ^ mask;
                if (l > i && l < n) {
                    const uint64_t a = key[i], b = key[l];
                    if (a > b) {
                        key[i] = b;
                        key[l] = a;
                        if (Pair) {
                            const uint64_t t = val[i];
                            val[i] = val[l];
                            val[l] = t;
                        }
                    }
                }
            }
            __syncthreads();
        }
    }
}

struct LeafView {
    const uint64_t* ent;  // sorted entries
    int n;
    int lev, unit_log;
    int32_t root;  // 2 host size
};

__device__ __forceinline__ uint64_t ent_code(uint64_t e) { return e >> (kSlotBits + 4); }
__device__ __forceinline__ int ent_size_log(uint64_t e) { return (int)((e >> kSlotBits) & 15); }

// The leaf covering the region (min rel, size 1 << size_log units): its rank,
// -1 when nothing is there (a null child in the reference's tree), -2 when the
// region is subdivided (smaller leaves inside).
__device__ int find_leaf(const LeafView& v, const int32_t rel[3], int size_log) {
    for (int a = 0; a < 3; a++)
        if (rel[a] < 0 || rel[a] >= v.root) return -1;
    const uint64_t k = morton(rel, v.unit_log, v.lev);
    const uint64_t vol = 1ull << (3 * size_log);
    int lo = 0, hi = v.n;  // first entry with code >= k
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ent_code(v.ent[mid]) < k)
            lo = mid + 1;
        else
            hi = mid;
    }
    if (lo < v.n && ent_code(v.ent[lo]) < k + vol) {
        if (ent_code(v.ent[lo]) == k && ent_size_log(v.ent[lo]) >= size_log) return lo;
        return -2;
    }
    if (lo > 0) {  // a larger leaf before it in Morton order may contain the region
        const uint64_t e = v.ent[lo - 1];
        const int sl = ent_size_log(e);
        if (sl > size_log && (k >> (3 * sl)) == (ent_code(e) >> (3 * sl))) return lo - 1;
    }
    return -1;
}

__device__ __forceinline__ int log2_units(int32_t size, int32_t unit) {
    int l = 0;
    while ((unit << l) < size) l++;
    return l;
}

// The path of the reference's recursion (ContourCellProc from the seam
// octree's root) to the final segment along `dir` at line coordinates line[]
// (host-relative), starting at t0 along dir, `len` long.
__device__ uint64_t path_key(int32_t root, int dir, const int32_t line[3], int32_t t0, int32_t len) {
    uint64_t key = 0;
    int nbits = 0;
    auto put = [&](int digit, int width) {
        nbits += width;
        key |= (uint64_t)digit << (64 - nbits);
    };
    const int a1 = dir == 0 ? 1 : 0, a2 = dir == 2 ? 1 : 2;
    int32_t m[3] = {0, 0, 0};
    int32_t S = root;
    int32_t e0 = 0, es = 0;  // edge state: start along dir, length
    for (;;) {  // cell
        const int32_t h = S >> 1;
        const int32_t mid[3] = {m[0] + h, m[1] + h, m[2] + h};
        const bool on1 = line[a1] == mid[a1], on2 = line[a2] == mid[a2];
        const int hd = t0 >= mid[dir];
        if (!on1 && !on2) {
            int c = hd << (2 - dir);
            c |= (line[a1] > mid[a1]) << (2 - a1);
            c |= (line[a2] > mid[a2]) << (2 - a2);
            put(c, 5);
            for (int a = 0; a < 3; a++) m[a] += cbit(c, a) * h;
            S = h;
            continue;
        }
        if (on1 && on2) {
            int e = 0;
            for (int i = 0; i < 6; i++)
                if (cCellProcEdgeMask[i][4] == dir && cbit(cCellProcEdgeMask[i][0], dir) == hd) e = i;
            put(20 + e, 5);
            e0 = m[dir] + hd * h;
            es = h;
            break;
        }
        const int a = on1 ? a1 : a2, b = on1 ? a2 : a1;
        const int bs = line[b] > mid[b];
        const int c0 = (bs << (2 - b)) | (hd << (2 - dir)), c1 = c0 | (1 << (2 - a));
        int f = 0;
        for (int i = 0; i < 12; i++)
            if (cCellProcFaceMask[i][0] == c0 && cCellProcFaceMask[i][1] == c1) f = i;
        put(8 + f, 5);
        int32_t fb = m[b] + bs * h, fd = m[dir] + hd * h, fs = h;
        for (;;) {  // face, plane perpendicular to a
            const int32_t hh = fs >> 1;
            const int fhd = t0 >= fd + hh;
            if (line[b] != fb + hh) {
                const int fbs = line[b] > fb + hh;
                int i4 = 0;
                for (int i = 0; i < 4; i++) {
                    const int c = cFaceProcFaceMask[a][i][1];
                    if (cbit(c, b) == fbs && cbit(c, dir) == fhd) i4 = i;
                }
                put(i4, 3);
                fb += fbs * hh;
                fd += fhd * hh;
                fs = hh;
                continue;
            }
            int i4 = 0;
            for (int i = 0; i < 4; i++)
                if (cFaceProcEdgeMask[a][i][5] == dir && cbit(cFaceProcEdgeMask[a][i][1], dir) == fhd) i4 = i;
            put(4 + i4, 3);
            e0 = fd + fhd * hh;
            es = hh;
            break;
        }
        break;
    }
    while (es > len) {  // edge: halves along dir
        const int32_t eh = es >> 1;
        const int hf = t0 >= e0 + eh;
        put(hf, 1);
        e0 += hf * eh;
        es = eh;
    }
    return key;
}

// Leaf sort lsort[blockIdx.x] = (host, first, count <= kSmallLeaves): the host's
// slots [first, first + count) sorted in shared memory to A.ent and A.leaves at
// the same positions of the host's leaf range.  A small host is one sort; a larger
// one a sort per Morton-prefix bucket, which together order the whole host.
__global__ void __launch_bounds__(256) k_seam_leaves(SeamArgs A) {
    extern __shared__ uint64_t smem[];
    const int4 it = A.lsort[blockIdx.x];
    const SeamHost h = A.hosts[it.x];
    const int n = it.z;
    const uint64_t* ent = A.sel + h.sel_off + it.y;
    for (int i = threadIdx.x; i < n; i += blockDim.x) smem[i] = ent[i];
    __syncthreads();
    block_sort<false>(smem, nullptr, n);
    for (int r = threadIdx.x; r < n; r += blockDim.x) {
        const uint64_t e = smem[r];
        A.ent[h.leaf_off + it.y + r] = e;
        A.leaves[h.leaf_off + it.y + r] = A.slots[h.sel_off + (e & ((1u << kSlotBits) - 1))];
    }
}

// Sorts too large for that are split first: one CTA deals a sort's entries into
// 256 parts by the eight bits below their common prefix, and lists the parts that
// are not empty for k_seam_parts.  (In one CTA a frame's largest leaf and quad
// sorts, 10 to 20 thousand entries, took 172 and 143 us, on the call's critical
// path.)  Leaves (Quads = false): sort lsort[blockIdx.x], dealt to A.ent.  Quads:
// those of host list[blockIdx.x] when they are more than kSmallQuads, dealt to the
// unused half of the host's quad range; without one (2 quads > 12 leaves) the
// host is a single part where it lies.
template <bool Quads>
__global__ void __launch_bounds__(1024) k_seam_split(SeamArgs A, const int32_t* list) {
    __shared__ unsigned long long lo, hi;
    __shared__ int cursor[kParts], warp_sum[kParts / 32];
    int host, first = 0, n;
    if (Quads) {
        host = list[blockIdx.x];
        n = A.qcounts[host];
        if (n <= kSmallQuads) return;
    } else {
        const int4 it = A.lsort[blockIdx.x];
        host = it.x, first = it.y, n = it.z;
    }
    const SeamHost h = A.hosts[host];
    const uint64_t* key = Quads ? A.qkey + h.quad_off : A.sel + h.sel_off + first;
    const int t = threadIdx.x;
    if (Quads && 2 * (int64_t)n > 12 * (int64_t)A.counts[host]) {
        if (t == 0) A.parts[atomicAdd(A.n_parts, 1)] = make_int4(host, 0, n, 0);
        return;
    }
    if (t == 0) lo = ~0ull, hi = 0ull;
    if (t < kParts) cursor[t] = 0;
    __syncthreads();
    unsigned long long mn = ~0ull, mx = 0ull;
    for (int i = t; i < n; i += blockDim.x) {
        mn = min(mn, (unsigned long long)key[i]);
        mx = max(mx, (unsigned long long)key[i]);
    }
    atomicMin(&lo, mn);
    atomicMax(&hi, mx);
    __syncthreads();
    const int top = lo == hi ? 0 : 63 - __clzll((long long)(lo ^ hi));  // highest bit that differs
    const int shift = max(0, top - 7);
    for (int i = t; i < n; i += blockDim.x) atomicAdd(&cursor[(key[i] >> shift) & (kParts - 1)], 1);
    __syncthreads();
    int count = 0, inc = 0;
    if (t < kParts) {
        count = inc = cursor[t];
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, o);
            if ((t & 31) >= o) inc += v;
        }
        if ((t & 31) == 31) warp_sum[t >> 5] = inc;
    }
    __syncthreads();
    if (t < kParts) {
        int start = inc - count;
        for (int w = 0; w < (t >> 5); w++) start += warp_sum[w];
        cursor[t] = start;
        if (count) A.parts[atomicAdd(A.n_parts, 1)] = make_int4(host, first + start, count, 1);
    }
    __syncthreads();
    for (int i = t; i < n; i += blockDim.x) {
        const uint64_t k = key[i];
        const int at = atomicAdd(&cursor[(k >> shift) & (kParts - 1)], 1);
        if (Quads) {
            A.qkey[h.quad_off + n + at] = k;
            A.qval[h.quad_off + n + at] = A.qval[h.quad_off + i];
        } else {
            A.ent[h.leaf_off + first + at] = k;
        }
    }
}

// The listed parts (host, first, count, dealt), each sorted to its place: leaf
// entries and seam indices, or quad payloads.  A part that does not fit shared
// memory (keys that crowd below a long common prefix more than once) is sorted
// where it lies.
template <bool Quads>
__global__ void __launch_bounds__(256) k_seam_parts(SeamArgs A) {
    extern __shared__ uint64_t smem[];
    const int parts = *A.n_parts;
    for (int p = blockIdx.x; p < parts; p += gridDim.x) {
        const int4 it = A.parts[p];
        const SeamHost h = A.hosts[it.x];
        const int n = it.z;
        const int64_t dealt = Quads && it.w ? A.qcounts[it.x] : 0;
        uint64_t* key = Quads ? A.qkey + h.quad_off + dealt + it.y : A.ent + h.leaf_off + it.y;
        uint64_t* val = Quads ? A.qval + h.quad_off + dealt + it.y : nullptr;
        uint64_t *sk = key, *sv = val;
        if (n <= kSmallLeaves) {
            sk = smem;
            sv = smem + kSmallLeaves;
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                sk[i] = key[i];
                if (Quads) sv[i] = val[i];
            }
            __syncthreads();
        }
        block_sort<Quads>(sk, sv, n);
        for (int r = threadIdx.x; r < n; r += blockDim.x) {
            if (Quads) {
                A.qval[h.quad_off + it.y + r] = sv[r];
            } else {
                const uint64_t e = sk[r];
                key[r] = e;
                A.leaves[h.leaf_off + it.y + r] = A.slots[h.sel_off + (e & ((1u << kSlotBits) - 1))];
            }
        }
        __syncthreads();  // shared memory is reused
    }
}

// The 12 edges of a leaf that may carry a quad: those with a sign change and,
// where `inside` says that no gathered leaf reaches out of its CLIPMAP_LEAF_SIZE
// block, those around which the four regions of the leaf's size do not all lie
// in one block.  (A leaf found for a region contains it, so it lies in the
// region's block, and the straddle test below would drop the segment.)
__device__ __forceinline__ uint32_t open_edges(int corners, const int32_t pos[3], int32_t s, bool inside) {
    uint32_t cross = inside ? 0u : 0x3fu;  // bit 2 a + side: blocks change at that face of axis a
    for (int a = 0; a < 3; a++)
        for (int side = 0; side < 2; side++) {
            const uint32_t line = (uint32_t)(pos[a] + side * s);
            if ((line - (uint32_t)s) / CLIPMAP_LEAF_SIZE != line / CLIPMAP_LEAF_SIZE) cross |= 1u << (2 * a + side);
        }
    uint32_t out = 0;
#pragma unroll
    for (int e = 0; e < 12; e++) {
        const int dir = e >> 2, a1 = dir == 0 ? 1 : 0, a2 = dir == 2 ? 1 : 2;
        const int c0 = (int)((0x642054103210ull >> (4 * e)) & 15), c1 = c0 | (4 >> dir);
        const bool sign = ((corners >> c0) ^ (corners >> c1)) & 1;
        const bool reach = (cross >> (2 * a1 + cbit(c0, a1)) | cross >> (2 * a2 + cbit(c0, a2))) & 1;
        if (sign && reach) out |= 1u << e;
    }
    return out;
}

// The quads of the leaves [first, first + kQuadBlock) of one host, unsorted,
// with their recursion path keys.  One thread a leaf lists the edges that may
// carry a quad, a small part of the twelve (of a 428-chunk frame's 6.5 M about 1
// in 10); the searches then run over the list with every lane busy (0.62 ms when
// each edge was searched in place).  So few searches do not pay for a copy of the
// host's entries in shared memory (0.09 ms for the hosts up to 8192 leaves beside
// 0.09 for the others, against 0.13 for all).
__global__ void __launch_bounds__(kQuadBlock) k_seam_quads(SeamArgs A) {
    __shared__ uint16_t open[kQuadBlock * 12];  // leaf of the block * 12 + edge
    __shared__ int s_open;
    const int2 it = A.items[blockIdx.x];
    const SeamHost h = A.hosts[it.x];
    const int n = A.counts[it.x];
    const uint64_t* ent = A.ent + h.leaf_off;
    const int unit_log = log2_units(h.unit, 1);
    const int r_end = min(n, it.y + kQuadBlock);
    if (threadIdx.x == 0) s_open = 0;
    __syncthreads();
    for (int r0 = it.y + (threadIdx.x & ~31); r0 < r_end; r0 += blockDim.x) {
        const int r = r0 + (threadIdx.x & 31);
        uint32_t edges = 0;
        if (r < r_end) {
            const uint64_t me = ent[r];
            int32_t pos[3];
            unmorton(ent_code(me), h.lev, unit_log, pos);
            for (int a = 0; a < 3; a++) pos[a] += h.min[a];
            edges = open_edges(A.seams[A.leaves[h.leaf_off + r]].localspace_min[3] & 0xff, pos,
                               h.unit << ent_size_log(me), h.inside != 0);
        }
        int inc = __popc(edges);
        const int own = inc;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if ((threadIdx.x & 31) >= o) inc += t;
        }
        int at = 0;
        if ((threadIdx.x & 31) == 31 && inc) at = atomicAdd(&s_open, inc);
        at = __shfl_sync(0xffffffffu, at, 31) + inc - own;
        for (; edges; edges &= edges - 1) open[at++] = (uint16_t)((r - it.y) * 12 + __ffs(edges) - 1);
    }
    __syncthreads();
    const int n_open = s_open;
    LeafView v;
    v.ent = ent;
    v.n = n;
    v.lev = h.lev;
    v.unit_log = unit_log;
    v.root = 2 * h.size;
    for (int k = threadIdx.x; k < n_open; k += blockDim.x) {
        const int item = open[k];
        const int r = it.y + item / 12, e = item % 12;
        const uint64_t me = ent[r];
        const int c0 = cEdgeVMap[e][0], c1 = cEdgeVMap[e][1];
        const int corners = A.seams[A.leaves[h.leaf_off + r]].localspace_min[3] & 0xff;
        const int m1 = (corners >> c1) & 1;
        const int dir = e >> 2;
        int j = 0;
        for (int q = 0; q < 4; q++)
            if (cProcessEdgeMask[dir][q] == e) j = q;
        const int sl = ent_size_log(me);
        const int32_t s = h.unit << sl;
        int32_t lmin[3];
        unmorton(ent_code(me), h.lev, unit_log, lmin);
        int32_t line[3];
        for (int a = 0; a < 3; a++) line[a] = lmin[a] + cbit(c0, a) * s;
        // the four leaves around the edge, in the order ContourEdgeProc passes
        // them (the children of cellProcEdgeMask's first entry along dir)
        int rank[4];
        bool ok = true;
        for (int q = 0; q < 4 && ok; q++) {
            if (q == j) {
                rank[q] = r;
                continue;
            }
            const int child = cCellProcEdgeMask[2 * dir][q];
            int32_t rel[3];
            for (int a = 0; a < 3; a++) rel[a] = a == dir ? lmin[a] : line[a] - s + cbit(child, a) * s;
            rank[q] = find_leaf(v, rel, sl);
            ok = rank[q] >= 0;
        }
        if (!ok) continue;
        int min_index = 0, min_log = 64;  // ContourProcessEdge: the first of the smallest leaves
        for (int q = 0; q < 4; q++) {
            const int lq = ent_size_log(ent[rank[q]]);
            if (lq < min_log) {
                min_log = lq;
                min_index = q;
            }
        }
        if (min_index != j) continue;  // that leaf's edge is this segment: it emits the quad
        // the straddle test: not all four leaves in one CLIPMAP_LEAF_SIZE block
        bool one_block = true;
        int32_t b0[3];
        for (int q = 0; q < 4; q++) {
            int32_t rel[3];
            unmorton(ent_code(ent[rank[q]]), h.lev, unit_log, rel);
            for (int a = 0; a < 3; a++) {
                const int32_t blk = (int32_t)((uint32_t)(rel[a] + h.min[a]) & ~(uint32_t)(CLIPMAP_LEAF_SIZE - 1));
                if (q == 0)
                    b0[a] = blk;
                else
                    one_block &= blk == b0[a];
            }
        }
        if (one_block) continue;
        const int qi = atomicAdd(&A.qcounts[it.x], 1);  // < 12 n: every leaf edge emits at most once
        A.qkey[h.quad_off + qi] = path_key(2 * h.size, dir, line, lmin[dir], s);
        A.qval[h.quad_off + qi] = (uint64_t)rank[0] | ((uint64_t)rank[1] << kRankBits) |
                                  ((uint64_t)rank[2] << (2 * kRankBits)) | ((uint64_t)rank[3] << (3 * kRankBits)) |
                                  ((uint64_t)(m1 != 1) << (4 * kRankBits));
    }
}

// The quads of host list[blockIdx.x], at most kSmallQuads, in the recursion's
// order: payloads sorted in place.
__global__ void __launch_bounds__(256) k_seam_qsort(SeamArgs A, const int32_t* list) {
    extern __shared__ uint64_t smem[];
    const int hi = list[blockIdx.x];
    const SeamHost h = A.hosts[hi];
    const int nq = A.qcounts[hi];
    if (nq > kSmallQuads) return;
    uint64_t* key = A.qkey + h.quad_off;
    uint64_t* val = A.qval + h.quad_off;
    uint64_t* sk = smem;
    uint64_t* sv = smem + kSmallQuads;
    for (int i = threadIdx.x; i < nq; i += blockDim.x) {
        sk[i] = key[i];
        sv[i] = val[i];
    }
    __syncthreads();
    block_sort<true>(sk, sv, nq);
    for (int i = threadIdx.x; i < nq; i += blockDim.x) val[i] = sv[i];
}

// vertices (hosts with triangles only) and triangles, back to back by host;
// blockIdx.y splits a host's ranges over gridDim.y CTAs
__global__ void __launch_bounds__(256) k_seam_emit(SeamArgs A) {
    const SeamHost h = A.hosts[blockIdx.x];
    const int nq = A.qcounts[blockIdx.x];
    if (nq <= 0) return;
    const int n = A.counts[blockIdx.x];
    const int64_t vo = A.vout_off[blockIdx.x], to = A.tout_off[blockIdx.x];
    // a warp at a time, its 32 vertices or quads through shared memory, so that
    // every store instruction writes 128 bytes in a row (a thread storing its own
    // 48 or 24 bytes word by word kept the store queue full: 50 us for 442 hosts,
    // 23 so); word stores, as the outputs may be aligned to words only
    __shared__ float4 stage[8][96];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t* words = reinterpret_cast<const uint32_t*>(stage[warp]);
    const int first = 32 * (blockIdx.y * 8 + warp), step = 256 * gridDim.y;
    for (int r0 = first; r0 < n; r0 += step) {
        if (r0 + lane < n) {
            const lvn_seam_node s = A.seams[A.leaves[h.leaf_off + r0 + lane]];
            stage[warp][3 * lane] = make_float4(s.position[0], s.position[1], s.position[2], 0.f);
            stage[warp][3 * lane + 1] = make_float4(s.normal[0], s.normal[1], s.normal[2], 0.f);
            stage[warp][3 * lane + 2] =
                make_float4(A.colour[0], A.colour[1], A.colour[2], (float)(s.localspace_min[3] >> 8));
        }
        __syncwarp();
        uint32_t* out = reinterpret_cast<uint32_t*>(A.vout + vo + r0);
        for (int k = lane; k < 12 * min(32, n - r0); k += 32) out[k] = words[k];
        __syncwarp();
    }
    const uint64_t mask = (1ull << kRankBits) - 1;
    int2* const tri = reinterpret_cast<int2*>(stage[warp]);
    for (int q0 = first; q0 < nq; q0 += step) {
        if (q0 + lane < nq) {
            const uint64_t q = A.qval[h.quad_off + q0 + lane];
            const int i0 = (int)(q & mask), i1 = (int)((q >> kRankBits) & mask),
                      i2 = (int)((q >> (2 * kRankBits)) & mask), i3 = (int)((q >> (3 * kRankBits)) & mask);
            const bool flip = (q >> (4 * kRankBits)) & 1;  // (i0 i1 i3) (i0 i3 i2), or (i0 i3 i1) (i0 i2 i3)
            tri[3 * lane] = make_int2(i0, flip ? i3 : i1);
            tri[3 * lane + 1] = make_int2(flip ? i1 : i3, i0);
            tri[3 * lane + 2] = make_int2(flip ? i2 : i3, flip ? i3 : i2);
        }
        __syncwarp();
        uint32_t* out = reinterpret_cast<uint32_t*>(A.tout + to + 2 * q0);
        for (int k = lane; k < 6 * min(32, nq - q0); k += 32) out[k] = words[k];
        __syncwarp();
    }
}

// ---- host side -----------------------------------------------------------

template <class T, bool Host = false>
struct Grow {
    T* p = nullptr;
    size_t cap = 0;
    cudaError_t fit(size_t need) {
        if (need <= cap) return cudaSuccess;
        cudaError_t e = cudaDeviceSynchronize();
        if (e != cudaSuccess) return e;
        need = std::max(need, 2 * cap);
        if (p) Host ? cudaFreeHost(p) : cudaFree(p);
        p = nullptr;
        cap = 0;
        e = Host ? cudaMallocHost(&p, sizeof(T) * need) : cudaMalloc(&p, sizeof(T) * need);
        if (e == cudaSuccess) cap = need;
        return e;
    }
};

struct SeamWork {
    std::mutex mu;
    int device = -1, num_sms = 0;
    cudaStream_t stream = nullptr, side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr, ev_join2 = nullptr, ev_sorted = nullptr;
    Grow<SeamHost> hosts;
    Grow<int4> pairs;
    Grow<int4> chunks;
    Grow<int32_t> seam_offsets, counts, qcounts;
    Grow<lvn_seam_node> seams;
    Grow<uint64_t> sel, ent, qkey, qval;
    Grow<uint32_t> slots, leaves;
    Grow<int2> items;
    Grow<int32_t> lists, bcount, bstart, cursor;
    Grow<int4> lsort, parts;
    Grow<int32_t> n_parts;  // leaf parts, quad parts
    Grow<int32_t, true> hbuckets;  // pinned
    Grow<int64_t> offs;  // vertex offsets, triangle offsets
    Grow<lvn_mesh_vertex> vstage;
    Grow<lvn_mesh_triangle> tstage;
    Grow<int32_t, true> hcounts;  // pinned: counts, qcounts
};
SeamWork& seam_work() {
    static SeamWork w;
    return w;
}

int cuda_rc(cudaError_t e) {
    if (e == cudaSuccess) return LVN_OK;
    cudaGetLastError();
    return e == cudaErrorMemoryAllocation ? LVN_ERR_OUT_OF_MEMORY : LVN_ERR_CUDA;
}

#define SM_TRY(x)                        \
    do {                                 \
        const int rc__ = cuda_rc(x);     \
        if (rc__ != LVN_OK) return rc__; \
    } while (0)

// The clipmap's active nodes (the chunks) and the nodes above them;
// FindNode / FindActiveNodes (clipmap.cpp:982-1013, 1449-1479) over the
// complete octree rooted at (root_min, root_size).  A node is its level
// log2(size / CLIPMAP_LEAF_SIZE) and its root-relative position in units of its
// size (19 bits per axis: roots up to 2^27); one open-addressing table maps both
// kinds, so that a lookup tells an active node, a node above active ones and
// nothing apart (two tables and a division per axis and level took 0.33 ms for
// the 442 hosts of a frame).
class ActiveSet {
   public:
    static constexpr int32_t kNone = -1, kAbove = -2;

    ActiveSet(const int32_t rmin[3], int32_t rsize, int32_t num_chunks) : root_size_(rsize) {
        for (int a = 0; a < 3; a++) root_min_[a] = rmin[a];
        root_level_ = level(rsize);
        size_t cap = 64;
        while (cap < 8 * (size_t)num_chunks) cap <<= 1;
        slots_.assign(cap, Slot{kEmpty, kNone});
    }
    static int level(int32_t size) {
        int l = 0;
        while ((CLIPMAP_LEAF_SIZE << l) < size) l++;
        return l;
    }
    bool in_root(const int32_t mn[3], int32_t size) const {
        for (int a = 0; a < 3; a++) {
            const int64_t rel = (int64_t)mn[a] - root_min_[a];
            if (rel < 0 || rel + size > root_size_ || (rel & (size - 1))) return false;
        }
        return true;
    }
    // adds chunk c; false when it is listed twice
    bool add_active(const lvn_chunk_desc& d, int32_t c) {
        const int l = level(d.size);
        uint32_t u[3];
        cell(d.min, l, u);
        return insert(key(l, u[0], u[1], u[2]), c) == kNone;
    }
    // marks the nodes above an active one; false when one of them is active itself
    bool add_above(const lvn_chunk_desc& d) {
        int l = level(d.size);
        uint32_t u[3];
        cell(d.min, l, u);
        for (l++; l <= root_level_; l++) {
            for (uint32_t& x : u) x >>= 1;
            const int32_t was = insert(key(l, u[0], u[1], u[2]), kAbove);
            if (was >= 0) return false;
            if (was == kAbove) break;
        }
        return true;
    }
    // visits the active nodes FindActiveNodes lists for the node (mn, size)
    template <class F>
    void find_active(const int32_t mn[3], int32_t size, F&& visit) const {
        int l = level(size);
        uint32_t u[3];
        cell(mn, l, u);
        int32_t v = find(key(l, u[0], u[1], u[2]));
        if (v == kAbove) return descend(l, u[0], u[1], u[2], visit);
        // else an active node containing it, where there is one
        while (v == kNone && l < root_level_) {
            l++;
            for (uint32_t& x : u) x >>= 1;
            v = find(key(l, u[0], u[1], u[2]));
        }
        if (v >= 0) visit(v);
    }

   private:
    struct Slot {
        uint64_t key;
        int32_t val;
    };
    static constexpr uint64_t kEmpty = ~0ull;

    void cell(const int32_t mn[3], int l, uint32_t u[3]) const {
        for (int a = 0; a < 3; a++) u[a] = (uint32_t)(((int64_t)mn[a] - root_min_[a]) / CLIPMAP_LEAF_SIZE) >> l;
    }
    static uint64_t key(int l, uint32_t x, uint32_t y, uint32_t z) {
        return (((((uint64_t)x << 19) | y) << 19) | z) << 5 | (uint64_t)l;
    }
    size_t slot(uint64_t k) const { return (size_t)((k * 0x9e3779b97f4a7c15ull) >> 20) & (slots_.size() - 1); }
    int32_t find(uint64_t k) const {
        for (size_t i = slot(k);; i = (i + 1) & (slots_.size() - 1)) {
            if (slots_[i].key == k) return slots_[i].val;
            if (slots_[i].key == kEmpty) return kNone;
        }
    }
    // inserts (k, val) unless k is present; returns what was there
    int32_t insert(uint64_t k, int32_t val) {
        for (size_t i = slot(k);; i = (i + 1) & (slots_.size() - 1)) {
            if (slots_[i].key == k) return slots_[i].val;
            if (slots_[i].key == kEmpty) {
                slots_[i] = Slot{k, val};
                if (2 * ++used_ > slots_.size()) grow();
                return kNone;
            }
        }
    }
    void grow() {
        std::vector<Slot> old(2 * slots_.size(), Slot{kEmpty, kNone});
        old.swap(slots_);
        for (const Slot& s : old) {
            if (s.key == kEmpty) continue;
            size_t i = slot(s.key);
            while (slots_[i].key != kEmpty) i = (i + 1) & (slots_.size() - 1);
            slots_[i] = s;
        }
    }
    template <class F>
    void descend(int l, uint32_t x, uint32_t y, uint32_t z, F&& visit) const {
        if (l == 0) return;
        for (int i = 0; i < 8; i++) {
            const uint32_t cx = 2 * x + ((i >> 2) & 1), cy = 2 * y + ((i >> 1) & 1), cz = 2 * z + (i & 1);
            const int32_t v = find(key(l - 1, cx, cy, cz));
            if (v >= 0) visit(v);
            else if (v == kAbove) descend(l - 1, cx, cy, cz, visit);
        }
    }

    int32_t root_min_[3];
    int32_t root_size_;
    int root_level_;
    size_t used_ = 0;
    std::vector<Slot> slots_;
};

}  // namespace
}  // namespace lvn

using namespace lvn;

extern "C" {

int lvn_seam_generate(const lvn_chunk_desc* chunks, const int32_t* seam_offsets, int32_t num_chunks,
                      const lvn_seam_node* seams, int32_t seams_memory, int32_t voxels_per_chunk,
                      const int32_t root_min[3], int32_t root_size, const int32_t* hosts, int32_t num_hosts,
                      const float colour[3], lvn_batch_out* out) {
    if (!out || !root_min || !colour || num_chunks < 0 || num_hosts < 0 || (num_chunks > 0 && (!chunks || !seam_offsets)) ||
        (num_hosts > 0 && !hosts) || voxels_per_chunk < 8 || voxels_per_chunk > 64 ||
        (voxels_per_chunk & (voxels_per_chunk - 1)) || (seams_memory != LVN_MEMORY_HOST && seams_memory != LVN_MEMORY_DEVICE) ||
        (out->memory != LVN_MEMORY_HOST && out->memory != LVN_MEMORY_DEVICE) || (num_hosts > 0 && !out->chunks))
        return LVN_ERR_INVALID;
    if (root_size < CLIPMAP_LEAF_SIZE || (root_size & (root_size - 1))) return LVN_ERR_INVALID;
    const int vpc = voxels_per_chunk;
    if (root_size > (1 << 27)) return LVN_ERR_INVALID;
    ActiveSet act(root_min, root_size, num_chunks);
    for (int c = 0; c < num_chunks; c++) {
        const lvn_chunk_desc& d = chunks[c];
        if (d.size < CLIPMAP_LEAF_SIZE || (d.size & (d.size - 1)) || !act.in_root(d.min, d.size) ||
            seam_offsets[c + 1] < seam_offsets[c])
            return LVN_ERR_INVALID;
        if (!act.add_active(d, c)) return LVN_ERR_INVALID;  // listed twice
    }
    // the clipmap's active nodes never overlap: an active node above an active node is an error
    for (int c = 0; c < num_chunks; c++)
        if (!act.add_above(chunks[c])) return LVN_ERR_INVALID;
    const int64_t num_seams = num_chunks ? seam_offsets[num_chunks] : 0;
    if (seam_offsets && num_chunks && seam_offsets[0] != 0) return LVN_ERR_INVALID;
    // the gathered (chunk, neighbour mask) pairs of every host
    std::vector<SeamHost> hv(num_hosts);
    std::vector<int4> pairs;
    std::vector<uint8_t> mask_of((size_t)num_chunks, 0);  // neighbour indices a chunk was reached through
    std::vector<int32_t> touched;
    for (int hi = 0; hi < num_hosts; hi++) {
        if (hosts[hi] < 0 || hosts[hi] >= num_chunks) return LVN_ERR_INVALID;
        const lvn_chunk_desc& d = chunks[hosts[hi]];
        SeamHost& h = hv[hi];
        for (int a = 0; a < 3; a++) h.min[a] = d.min[a];
        h.size = d.size;
        h.pair_begin = (int32_t)pairs.size();
        touched.clear();
        for (int i = 0; i < 8; i++) {
            const int32_t nmin[3] = {d.min[0] + ((i >> 2) & 1) * d.size, d.min[1] + ((i >> 1) & 1) * d.size,
                                     d.min[2] + (i & 1) * d.size};
            if (!act.in_root(nmin, d.size)) continue;  // Clipmap::findNode finds no node there
            act.find_active(nmin, d.size, [&](int32_t c) {
                if (!mask_of[c]) touched.push_back(c);
                mask_of[c] |= (uint8_t)(1 << i);
            });
        }
        int unit = d.size / vpc;
        // blocks are counted from world 0: a leaf of up to their size lies in one when the root is aligned to them
        bool inside = true;
        for (int a = 0; a < 3; a++) inside &= root_min[a] % CLIPMAP_LEAF_SIZE == 0;
        for (const int32_t c : touched) {
            pairs.push_back(make_int4(c, mask_of[c], hi, 0));
            mask_of[c] = 0;
            unit = std::min(unit, chunks[c].size / vpc);
            inside &= chunks[c].size / vpc <= CLIPMAP_LEAF_SIZE;
        }
        h.pair_end = (int32_t)pairs.size();
        h.unit = unit;
        h.inside = inside ? 1 : 0;
        h.lev = 0;
        while ((unit << h.lev) < 2 * d.size) h.lev++;
        if (h.lev > kMaxLevels) return LVN_ERR_INVALID;
    }
    SeamWork& w = seam_work();
    std::lock_guard<std::mutex> lock(w.mu);
    int dev = 0;
    SM_TRY(cudaGetDevice(&dev));
    if (w.device != dev) {
        if (w.device >= 0) return LVN_ERR_INVALID;  // the scratch lives on the first device used
        SM_TRY(cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking));
        SM_TRY(cudaStreamCreateWithFlags(&w.side, cudaStreamNonBlocking));
        SM_TRY(cudaEventCreateWithFlags(&w.ev_fork, cudaEventDisableTiming));
        SM_TRY(cudaEventCreateWithFlags(&w.ev_join, cudaEventDisableTiming));
        SM_TRY(cudaEventCreateWithFlags(&w.ev_join2, cudaEventDisableTiming));
        SM_TRY(cudaEventCreateWithFlags(&w.ev_sorted, cudaEventDisableTiming));
        SM_TRY(cudaDeviceGetAttribute(&w.num_sms, cudaDevAttrMultiProcessorCount, dev));
        w.device = dev;
    }
    if (num_hosts == 0) {
        out->total_vertices = out->total_triangles = out->total_seams = 0;
        return LVN_OK;
    }
    const size_t nh = (size_t)num_hosts;
    SM_TRY(w.hosts.fit(nh));
    SM_TRY(w.pairs.fit(std::max<size_t>(pairs.size(), 1)));
    int64_t sel_total = 0;
    for (size_t i = 0; i < nh; i++) {
        hv[i].sel_off = sel_total;
        for (int p = hv[i].pair_begin; p < hv[i].pair_end; p++)
            sel_total += seam_offsets[pairs[p].x + 1] - seam_offsets[pairs[p].x];
    }
    SM_TRY(w.sel.fit(std::max<int64_t>(sel_total, 1)));
    SM_TRY(w.slots.fit(std::max<int64_t>(sel_total, 1)));
    SM_TRY(w.chunks.fit(std::max(num_chunks, 1)));
    SM_TRY(w.seam_offsets.fit((size_t)num_chunks + 1));
    SM_TRY(w.counts.fit(nh));
    SM_TRY(w.qcounts.fit(nh));
    SM_TRY(w.offs.fit(2 * nh));
    SM_TRY(w.hcounts.fit(2 * nh));
    std::vector<int4> c4(std::max(num_chunks, 1));
    for (int c = 0; c < num_chunks; c++)
        c4[c] = make_int4(chunks[c].min[0], chunks[c].min[1], chunks[c].min[2], chunks[c].size);
    cudaStream_t st = w.stream;
    SM_TRY(cudaMemcpyAsync(w.pairs.p, pairs.data(), sizeof(int4) * pairs.size(), cudaMemcpyHostToDevice, st));
    SM_TRY(cudaMemcpyAsync(w.chunks.p, c4.data(), sizeof(int4) * num_chunks, cudaMemcpyHostToDevice, st));
    SM_TRY(cudaMemcpyAsync(w.seam_offsets.p, seam_offsets, sizeof(int32_t) * (num_chunks + 1), cudaMemcpyHostToDevice,
                           st));
    const lvn_seam_node* dseams = seams;
    if (seams_memory == LVN_MEMORY_HOST && num_seams > 0) {
        SM_TRY(w.seams.fit((size_t)num_seams));
        SM_TRY(cudaMemcpyAsync(w.seams.p, seams, sizeof(lvn_seam_node) * num_seams, cudaMemcpyHostToDevice, st));
        dseams = w.seams.p;
    }
    SeamArgs A;
    std::memset(&A, 0, sizeof(A));
    A.hosts = w.hosts.p;
    A.pairs = w.pairs.p;
    A.chunks = w.chunks.p;
    A.seam_offsets = w.seam_offsets.p;
    A.seams = dseams;
    A.vpc = vpc;
    A.counts = w.counts.p;
    A.qcounts = w.qcounts.p;
    for (int a = 0; a < 3; a++) A.colour[a] = colour[a];
    A.sel = w.sel.p;
    A.slots = w.slots.p;
    const size_t nb = nh * kBuckets;
    SM_TRY(w.bcount.fit(nb));
    SM_TRY(w.bstart.fit(nb));
    SM_TRY(w.cursor.fit(nb));
    SM_TRY(w.hbuckets.fit(nb));
    A.bcount = w.bcount.p;
    A.bstart = w.bstart.p;
    A.cursor = w.cursor.p;
    // 1: the selected seam nodes of every host, counted by bucket
    SM_TRY(cudaMemcpyAsync(w.hosts.p, hv.data(), sizeof(SeamHost) * nh, cudaMemcpyHostToDevice, st));
    SM_TRY(cudaMemsetAsync(w.counts.p, 0, sizeof(int32_t) * nh, st));
    SM_TRY(cudaMemsetAsync(w.bcount.p, 0, sizeof(int32_t) * nb, st));
    SM_TRY(cudaMemsetAsync(w.cursor.p, 0, sizeof(int32_t) * nb, st));
    if (!pairs.empty()) {
        k_seam_select<false><<<(int)pairs.size(), 128, 0, st>>>(A);
        SM_TRY(cudaGetLastError());
    }
    SM_TRY(cudaMemcpyAsync(w.hcounts.p, w.counts.p, sizeof(int32_t) * nh, cudaMemcpyDeviceToHost, st));
    SM_TRY(cudaMemcpyAsync(w.hbuckets.p, w.bcount.p, sizeof(int32_t) * nb, cudaMemcpyDeviceToHost, st));
    SM_TRY(cudaStreamSynchronize(st));
    // bucket starts, and the leaf sorts: one per small host, one per non-empty bucket of a larger one
    std::vector<int32_t> bstart(nb);
    std::vector<int4> small_sorts, big_sorts;
    for (size_t i = 0; i < nh; i++) {
        int run = 0;
        for (int b = 0; b < kBuckets; b++) {
            bstart[i * kBuckets + b] = run;
            run += w.hbuckets.p[i * kBuckets + b];
        }
        const int n = w.hcounts.p[i];
        if (n == 0) continue;
        if (n <= kSmallLeaves) {
            small_sorts.push_back(make_int4((int)i, 0, n, 0));
            continue;
        }
        for (int b = 0; b < kBuckets; b++) {
            const int c = w.hbuckets.p[i * kBuckets + b];
            if (c) (c <= kSmallLeaves ? small_sorts : big_sorts).push_back(make_int4((int)i, bstart[i * kBuckets + b], c, 0));
        }
    }
    SM_TRY(cudaMemcpyAsync(w.bstart.p, bstart.data(), sizeof(int32_t) * nb, cudaMemcpyHostToDevice, st));
    if (!pairs.empty()) {
        k_seam_select<true><<<(int)pairs.size(), 128, 0, st>>>(A);
        SM_TRY(cudaGetLastError());
    }
    int64_t leaf_total = 0, quad_total = 0;
    bool limit = false;
    std::vector<int2> items;  // (host, first leaf) of the quad enumeration's CTAs
    for (size_t i = 0; i < nh; i++) {
        const int n = w.hcounts.p[i];
        limit |= n > kMaxLeaves;
        hv[i].leaf_off = leaf_total;
        hv[i].quad_off = quad_total;
        leaf_total += n;
        quad_total += 12 * (int64_t)n;
        for (int r = 0; r < n; r += kQuadBlock) items.push_back(make_int2((int)i, r));
    }
    if (limit) return LVN_ERR_DEVICE_STATUS;
    // 2: sorted leaves, quads, quads in order
    SM_TRY(w.ent.fit(std::max<int64_t>(leaf_total, 1)));
    SM_TRY(w.leaves.fit(std::max<int64_t>(leaf_total, 1)));
    SM_TRY(w.qkey.fit(std::max<int64_t>(quad_total, 1)));
    SM_TRY(w.qval.fit(std::max<int64_t>(quad_total, 1)));
    SM_TRY(w.items.fit(std::max<size_t>(items.size(), 1)));
    SM_TRY(w.lists.fit(nh));
    std::vector<int32_t> lists(nh);
    for (size_t i = 0; i < nh; i++) lists[i] = (int32_t)i;
    SM_TRY(cudaMemcpyAsync(w.lists.p, lists.data(), sizeof(int32_t) * nh, cudaMemcpyHostToDevice, st));
    const size_t n_sorts = small_sorts.size() + big_sorts.size();
    SM_TRY(w.lsort.fit(std::max<size_t>(n_sorts, 1)));
    std::vector<int4> sorts(small_sorts);
    sorts.insert(sorts.end(), big_sorts.begin(), big_sorts.end());
    SM_TRY(cudaMemcpyAsync(w.lsort.p, sorts.data(), sizeof(int4) * n_sorts, cudaMemcpyHostToDevice, st));
    A.ent = w.ent.p;
    A.leaves = w.leaves.p;
    A.qkey = w.qkey.p;
    A.qval = w.qval.p;
    A.items = w.items.p;
    SM_TRY(cudaMemcpyAsync(w.hosts.p, hv.data(), sizeof(SeamHost) * nh, cudaMemcpyHostToDevice, st));
    SM_TRY(cudaMemcpyAsync(w.items.p, items.data(), sizeof(int2) * items.size(), cudaMemcpyHostToDevice, st));
    SM_TRY(cudaMemsetAsync(w.qcounts.p, 0, sizeof(int32_t) * nh, st));
    // a host has at most one split sort of quads; the quads' parts reuse the list of the leaves'
    SM_TRY(w.parts.fit(kParts * std::max<size_t>(big_sorts.size(), nh)));
    SM_TRY(w.n_parts.fit(2));
    SM_TRY(cudaMemsetAsync(w.n_parts.p, 0, sizeof(int32_t) * 2, st));
    A.parts = w.parts.p;
    A.n_parts = w.n_parts.p;
    // the large sorts beside the small ones, on the second stream
    SM_TRY(cudaEventRecord(w.ev_fork, st));
    SM_TRY(cudaStreamWaitEvent(w.side, w.ev_fork, 0));
    SeamArgs B = A;
    B.lsort = w.lsort.p + small_sorts.size();
    const int part_ctas = 4 * w.num_sms;
    if (!big_sorts.empty()) {
        k_seam_split<false><<<(int)big_sorts.size(), 1024, 0, w.side>>>(B, nullptr);
        k_seam_parts<false><<<part_ctas, 256, kSmallSortSmem, w.side>>>(B);
        SM_TRY(cudaGetLastError());
        SM_TRY(cudaEventRecord(w.ev_sorted, w.side));
    }
    if (!small_sorts.empty()) {
        A.lsort = w.lsort.p;
        k_seam_leaves<<<(int)small_sorts.size(), 256, kSmallLeafSmem, st>>>(A);
        SM_TRY(cudaGetLastError());
    }
    if (!big_sorts.empty()) SM_TRY(cudaStreamWaitEvent(st, w.ev_sorted, 0));
    if (!items.empty()) {
        k_seam_quads<<<(int)items.size(), kQuadBlock, 0, st>>>(A);
        SM_TRY(cudaGetLastError());
    }
    SM_TRY(cudaEventRecord(w.ev_join, st));
    SM_TRY(cudaStreamWaitEvent(w.side, w.ev_join, 0));
    // quad sorts: hosts of up to kSmallQuads quads here, the others in parts on the side stream
    k_seam_qsort<<<num_hosts, 256, kSmallSortSmem, st>>>(A, w.lists.p);
    SM_TRY(cudaGetLastError());
    B.n_parts = w.n_parts.p + 1;
    k_seam_split<true><<<num_hosts, 1024, 0, w.side>>>(B, w.lists.p);
    k_seam_parts<true><<<part_ctas, 256, kSmallSortSmem, w.side>>>(B);
    SM_TRY(cudaGetLastError());
    SM_TRY(cudaEventRecord(w.ev_join2, w.side));
    SM_TRY(cudaStreamWaitEvent(st, w.ev_join2, 0));
    SM_TRY(cudaMemcpyAsync(w.hcounts.p + nh, w.qcounts.p, sizeof(int32_t) * nh, cudaMemcpyDeviceToHost, st));
    SM_TRY(cudaStreamSynchronize(st));
    // 3: output layout: hosts with triangles, back to back
    std::vector<int64_t> offs(2 * nh);
    int64_t tv = 0, tt = 0;
    for (size_t i = 0; i < nh; i++) {
        const int nq = w.hcounts.p[nh + i];
        const int nv = nq > 0 ? w.hcounts.p[i] : 0;
        lvn_chunk_result& r = out->chunks[i];
        std::memset(&r, 0, sizeof(r));
        r.vertex_offset = (int32_t)tv;
        r.num_vertices = nv;
        r.triangle_offset = (int32_t)tt;
        r.num_triangles = 2 * nq;
        r.num_nodes = w.hcounts.p[i];
        offs[i] = tv;
        offs[nh + i] = tt;
        tv += nv;
        tt += 2 * nq;
    }
    out->total_vertices = tv;
    out->total_triangles = tt;
    out->total_seams = 0;
    if (tv > out->vertex_capacity || tt > out->triangle_capacity) return LVN_ERR_CAPACITY;
    if (tt == 0) return LVN_OK;
    if ((tv && !out->vertices) || (tt && !out->triangles)) return LVN_ERR_INVALID;
    SM_TRY(cudaMemcpyAsync(w.offs.p, offs.data(), sizeof(int64_t) * 2 * nh, cudaMemcpyHostToDevice, st));
    A.vout_off = w.offs.p;
    A.tout_off = w.offs.p + nh;
    if (out->memory == LVN_MEMORY_DEVICE) {
        A.vout = out->vertices;
        A.tout = out->triangles;
    } else {
        SM_TRY(w.vstage.fit((size_t)tv));
        SM_TRY(w.tstage.fit((size_t)tt));
        A.vout = w.vstage.p;
        A.tout = w.tstage.p;
    }
    k_seam_emit<<<dim3(num_hosts, 16), 256, 0, st>>>(A);
    SM_TRY(cudaGetLastError());
    if (out->memory == LVN_MEMORY_HOST) {
        SM_TRY(cudaMemcpyAsync(out->vertices, w.vstage.p, sizeof(lvn_mesh_vertex) * tv, cudaMemcpyDeviceToHost, st));
        SM_TRY(cudaMemcpyAsync(out->triangles, w.tstage.p, sizeof(lvn_mesh_triangle) * tt, cudaMemcpyDeviceToHost, st));
    }
    SM_TRY(cudaStreamSynchronize(st));
    return LVN_OK;
}

}  // extern "C"
