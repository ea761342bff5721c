// rt_build.cu — BLAS / TLAS construction, TLAS refit and AS copies.
//
// Build = a binary hierarchy over Morton-ordered primitives, collapsed to
// 8-wide nodes:
//   1. primitive boxes (triangles, or instance world boxes) + centroid bounds
//   2. 30-bit Morton codes of the centroids, in the sort's first step
//   3. stable LSD radix sort, 8-bit digits, 4 passes: one block for up to
//      kSortBlockMax keys, else onesweep (one upfront histogram of all digits,
//      then one kernel per digit with decoupled look-back across partitions)
//   4. the binary hierarchy: PLOC clustering (RT_BUILD_PREFER_FAST_TRACE;
//      boxes and subtree sizes come with each merge), or the Karras LBVH
//      (index-augmented for ties) with bottom-up boxes from one arrival
//      counter per internal node
//   5. collapse to 8-wide nodes in one launch, a queue of tasks: a node takes
//      its binary children and repeatedly opens the child of largest surface
//      area until it has 8 children or none can open; a subtree of <=
//      leaf_max primitives is a leaf.  Each task carries the first position
//      of its primitives in the final order; its children's primitives
//      follow each other in slot order, and a leaf child writes its
//      primitives' positions (perm).
//   6. primitive records written in that final order.
// A TLAS of up to kTlasSmall instances goes through all of it in one block
// (k_tlas_small), whatever the build flags.
// Everything runs on the caller's stream; no host synchronisation.
//
// Replaces vkCmdBuildAccelerationStructuresKHR as called by
// AccelerationStructure::build_blas / new (src/util_structs.rs:140-283),
// build_tlas (src/util_functions.rs:453-510) and update_tlas
// (src/util_structs.rs:285-357), and vkCmdCopyAccelerationStructureKHR CLONE
// (src/util_structs.rs:359-405).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>

#include "rt_internal.h"

namespace rt {

namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kLeafBit = 0x80000000u;
constexpr uint32_t kSortThreads = 1024;
constexpr uint32_t kSortBlockMax = 8 * kSortThreads;  // keys that one block sorts
constexpr int kDopTriples = 14 * 13 * 12 / 6;  // 364 plane triples of the 14-DOP
constexpr int kPlocMaxRounds = 64;  // grid-wide PLOC rounds (ploc_grid_rounds stays below it for 2^28 primitives)

struct BuildState {
    uint32_t cb[6];   // centroid bounds, ordered-uint encoding: min xyz, max xyz
    uint32_t bb[6];   // primitive box bounds
    uint32_t error;
    uint32_t depth;
    uint32_t blas_kinds;  // TLAS: kBlasKind* bits of the BLASes its instances enter
    uint32_t merge_counter;  // PLOC merges so far (internal node ids count down from n - 2)
    uint32_t pair_merges;    // and those of k_ploc_pairs
    uint32_t radius_bits;    // BLAS: largest vertex distance from the bounds centre (float bits, rounded up)
    uint32_t dop_hi[7], dop_lo[7];  // BLAS: largest / smallest vertex projection on each 14-DOP axis (ordered uint)
    uint32_t ploc_round[kPlocMaxRounds + 2];  // PLOC clusters entering each round, k_ploc_pairs, the tail | kPloc* bits
    uint32_t ploc_ticket[kPlocMaxRounds];     // next tile of each round
    // collapse: one cache line each for the two counters that every warp adds
    // to and the flag that waiting warps read
    uint32_t _line0[32];
    unsigned long long progress;  // primitives placed in leaves << 32 | wide nodes allocated
    uint32_t _line1[30];
    uint32_t collapse_ticket;     // next wide-node slot to work on
    uint32_t _line2[31];
    uint32_t collapse_done;       // 1: every primitive has its leaf
    uint32_t _line3[31];
    uint32_t node_count;  // wide nodes in use
};
// The state's share of the build scratch.  It is more than the state needs:
// the scratch sizes that callers query, and the limit of the static-scratch
// build that follows from them, stay as they are.
constexpr uint64_t kBuildStateBytes = 10496;
static_assert(sizeof(BuildState) <= kBuildStateBytes, "build state size");

// The seven 14-DOP axes (unnormalised): x, y, z and the four diagonals.
__device__ __constant__ const int8_t kDopAxis[7][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {1, 1, 1},
                                                       {1, 1, -1}, {1, -1, 1}, {-1, 1, 1}};

__device__ __forceinline__ uint32_t f2o(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// Centre of the primitive bounds, computed the same way wherever it is used.
__device__ __forceinline__ float bounds_center(const BuildState* st, int k) {
    return 0.5f * (o2f(st->bb[k]) + o2f(st->bb[3 + k]));
}

// Distance of v from c, rounded up (every operation rounds towards +inf).
__device__ __forceinline__ float distance_ru(const float v[3], const float c[3]) {
    float s = 0.0f;
    for (int k = 0; k < 3; k++) {
        float d = fmaxf(__fsub_ru(v[k], c[k]), __fsub_ru(c[k], v[k]));
        s = __fadd_ru(s, __fmul_ru(d, d));
    }
    return __fsqrt_ru(s);
}

__device__ __forceinline__ void pad_box(float lo[3], float hi[3]) {
    for (int k = 0; k < 3; k++) {
        float m = fmaxf(fabsf(lo[k]), fabsf(hi[k]));
        float pad = m * 9.5367431640625e-07f + 1e-30f;  // 2^-20 relative
        lo[k] -= pad;
        hi[k] += pad;
    }
}

__device__ __forceinline__ bool finite3(const float v[3]) {
    return fabsf(v[0]) <= FLT_MAX && fabsf(v[1]) <= FLT_MAX && fabsf(v[2]) <= FLT_MAX;
}

// Block-wide min/max reduction of 12 ordered-uint values, then atomics.
__device__ void reduce_bounds(BuildState* st, const float cmin[3], const float cmax[3], const float bmin[3],
                              const float bmax[3]) {
    uint32_t v[12];
    for (int k = 0; k < 3; k++) {
        v[k] = f2o(cmin[k]);
        v[3 + k] = f2o(cmax[k]);
        v[6 + k] = f2o(bmin[k]);
        v[9 + k] = f2o(bmax[k]);
    }
    for (int off = 16; off > 0; off >>= 1) {
        for (int k = 0; k < 12; k++) {
            uint32_t o = __shfl_xor_sync(0xFFFFFFFFu, v[k], off);
            bool is_min = (k < 3) || (k >= 6 && k < 9);
            v[k] = is_min ? min(v[k], o) : max(v[k], o);
        }
    }
    // then over the block's warps, so that each block makes one atomic per
    // bound (one per warp serialised ~82k same-address atomics per bound on a
    // 2.6M-triangle build); every thread of the block must call this
    __shared__ uint32_t s[32][12];
    const uint32_t w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 12; k++) s[w][k] = v[k];
    __syncthreads();
    if (threadIdx.x < 12) {
        const int k = threadIdx.x;
        const bool is_min = (k < 3) || (k >= 6 && k < 9);
        uint32_t r = s[0][k];
        for (uint32_t j = 1; j < nw; j++) r = is_min ? min(r, s[j][k]) : max(r, s[j][k]);
        uint32_t* dst = k < 6 ? &st->cb[k] : &st->bb[k - 6];
        if (is_min) atomicMin(dst, r);
        else atomicMax(dst, r);
    }
}

__device__ __forceinline__ void init_state(BuildState* st, uint32_t n) {
    for (uint32_t i = threadIdx.x; i < kPlocMaxRounds; i += blockDim.x) st->ploc_ticket[i] = 0;
    if (threadIdx.x == 0) {
        st->ploc_round[0] = n;
        for (int k = 0; k < 3; k++) {
            st->cb[k] = 0xFFFFFFFFu;
            st->cb[3 + k] = 0u;
            st->bb[k] = 0xFFFFFFFFu;
            st->bb[3 + k] = 0u;
        }
        st->progress = 1;
        st->collapse_ticket = 0;
        st->collapse_done = 0;
        st->node_count = 1;
        st->error = 0;
        st->depth = 1;
        st->blas_kinds = 0;
        st->merge_counter = 0;
        st->pair_merges = 0;
        st->radius_bits = 0;
        for (int k = 0; k < 7; k++) {
            st->dop_hi[k] = 0u;
            st->dop_lo[k] = 0xFFFFFFFFu;
        }
    }
}
__global__ void k_init_state(BuildState* st, uint32_t n) {
    after_previous();
    init_state(st, n);
}

__device__ __forceinline__ int find_geometry(const BlasInput& in, uint32_t i) {
    int lo = 0, hi = (int)in.geometry_count - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (in.g[mid].prefix <= i) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Fetches triangle i's vertices; false for an invalid index or an inactive
// (NaN) triangle.
__device__ bool fetch_triangle(const BlasInput& in, uint32_t i, int* geom, uint32_t* prim, float v[3][3]) {
    int g = find_geometry(in, i);
    const BuildGeom& G = in.g[g];
    uint32_t p = i - G.prefix;
    *geom = g;
    *prim = p;
    uint32_t vi[3];
    if (G.idx) {
        vi[0] = G.idx[3 * (size_t)p];
        vi[1] = G.idx[3 * (size_t)p + 1];
        vi[2] = G.idx[3 * (size_t)p + 2];
    } else {
        vi[0] = 3 * p;
        vi[1] = 3 * p + 1;
        vi[2] = 3 * p + 2;
    }
    bool ok = true;
    for (int c = 0; c < 3; c++) {
        if (vi[c] > G.max_vertex) {
            ok = false;
            v[c][0] = v[c][1] = v[c][2] = __int_as_float(0x7FC00000);
            continue;
        }
        const float* src = G.pos + (size_t)vi[c] * G.stride_floats;
        v[c][0] = src[0];
        v[c][1] = src[1];
        v[c][2] = src[2];
        if (!finite3(v[c])) ok = false;
    }
    return ok;
}

// What a later kernel of the build finds zeroed: the PLOC look-back
// descriptors, the collapse's tasks, and the state of a onesweep sort.
struct ZeroedWords {
    unsigned long long* desc;
    unsigned long long* tasks;
    unsigned long long* sort;
    uint32_t descs, task_count, sort_words;
};
__device__ __forceinline__ void zero_words(const ZeroedWords& z, uint32_t i, uint32_t stride) {
    for (uint32_t k = i; k < z.sort_words; k += stride) z.sort[k] = 0ull;
    for (uint32_t k = i; k < z.descs; k += stride) z.desc[k] = 0ull;
    for (uint32_t k = i; k < z.task_count; k += stride) z.tasks[k] = 0ull;
}

// At most kPrimBlocks blocks, each thread over several triangles: every block
// ends with 12 atomics on the same two cache lines, and one block per 256
// triangles spent most of its time there (10.5M triangles, with k_write_tris: 57 us less).
constexpr uint32_t kPrimBlocks = 152 * 8;
__global__ void k_blas_prims(const __grid_constant__ BlasInput in, float4* boxes, BuildState* st, ZeroedWords z) {
    after_previous();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    zero_words(z, i, gridDim.x * blockDim.x);
    float cmin[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, cmax[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    float bmin[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, bmax[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (; i < in.n; i += gridDim.x * blockDim.x) {
        int g;
        uint32_t p;
        float v[3][3];
        float lo[3], hi[3];
        bool ok = fetch_triangle(in, i, &g, &p, v);
        if (ok) {
            for (int k = 0; k < 3; k++) {
                lo[k] = fminf(fminf(v[0][k], v[1][k]), v[2][k]);
                hi[k] = fmaxf(fmaxf(v[0][k], v[1][k]), v[2][k]);
            }
            pad_box(lo, hi);
            for (int k = 0; k < 3; k++) {
                float c = 0.5f * (lo[k] + hi[k]);
                cmin[k] = fminf(cmin[k], c);
                cmax[k] = fmaxf(cmax[k], c);
                bmin[k] = fminf(bmin[k], lo[k]);
                bmax[k] = fmaxf(bmax[k], hi[k]);
            }
        } else {
            for (int k = 0; k < 3; k++) {
                lo[k] = INFINITY;
                hi[k] = -INFINITY;
            }
            bool bad_index = false;
            const BuildGeom& G = in.g[g];
            if (G.idx) {
                for (int c = 0; c < 3; c++) bad_index |= G.idx[3 * (size_t)p + c] > G.max_vertex;
            } else {
                bad_index = 3 * p + 2 > G.max_vertex;
            }
            if (bad_index) atomicOr(&st->error, 1u << RT_ERR_INVALID);
        }
        boxes[2 * (size_t)i] = make_float4(lo[0], lo[1], lo[2], 0.0f);
        boxes[2 * (size_t)i + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
    }
    reduce_bounds(st, cmin, cmax, bmin, bmax);
}

// Fills a TLAS instance record from the caller's instance `r` (index id):
// world-to-object inverse, BLAS fields for the traversal, and the world box
// = the 8 transformed corners of the BLAS bounds, padded so the box stays
// conservative for the rounded object-space ray.  Returns false (empty box,
// tri_count 0) for a singular transform or a null / empty BLAS.
__device__ bool fill_instance(const RtAccelerationStructureInstance& r, uint32_t id, InstRecord* rec, float lo[3],
                              float hi[3], uint32_t* err) {
    const float* m = &r.transform[0][0];
    for (int k = 0; k < 12; k++) rec->o2w[k] = m[k];
    bool valid = affine_inverse(m, rec->w2o);
    rec->blas = r.acceleration_structure_reference;
    rec->instance_id = id;
    rec->custom_mask = r.instance_custom_index_and_mask;
    rec->sbt_flags = r.instance_shader_binding_table_record_offset_and_flags;
    rec->tri_count = 0;
    rec->node_count = 0;
    rec->prims_off256 = 0;
    for (int k = 0; k < 3; k++) {
        lo[k] = INFINITY;
        hi[k] = -INFINITY;
    }
    if (rec->blas == 0) valid = false;
    if (valid) {
        const AsHeader* bh = reinterpret_cast<const AsHeader*>(rec->blas);
        if (bh->magic != kAsMagic || bh->type != kAsTypeBottom) {
            valid = false;
            atomicOr(err, 1u << RT_ERR_BAD_AS);
        } else if (bh->prim_count == 0) {
            valid = false;
        } else {
            float blo[3] = {bh->bounds_lo[0], bh->bounds_lo[1], bh->bounds_lo[2]};
            float bhi[3] = {bh->bounds_hi[0], bh->bounds_hi[1], bh->bounds_hi[2]};
            for (int c = 0; c < 8; c++) {
                V3 p = mk3((c & 1) ? bhi[0] : blo[0], (c & 2) ? bhi[1] : blo[1], (c & 4) ? bhi[2] : blo[2]);
                V3 q = xform_point(rec->o2w, p);
                lo[0] = fminf(lo[0], q.x);
                lo[1] = fminf(lo[1], q.y);
                lo[2] = fminf(lo[2], q.z);
                hi[0] = fmaxf(hi[0], q.x);
                hi[1] = fmaxf(hi[1], q.y);
                hi[2] = fmaxf(hi[2], q.z);
            }
            // Cut to the box of the transformed bounding sphere: the ellipsoid
            // M S + t has half-extent r |row_k(M)| along world axis k.  The
            // transformed centre is widened by its rounding error (a few ulps
            // of |M c| + |t|); the padding below adds more.
            const float rad = bh->sphere_radius;
            if (rad > 0.0f && rad <= FLT_MAX) {
                const float* M = rec->o2w;
                V3 cw = xform_point(M, mk3(bh->sphere_center[0], bh->sphere_center[1], bh->sphere_center[2]));
                const float cwv[3] = {cw.x, cw.y, cw.z};
                for (int k = 0; k < 3; k++) {
                    const float a = M[4 * k], b = M[4 * k + 1], d = M[4 * k + 2];
                    const float row = __fsqrt_ru(__fadd_ru(__fadd_ru(__fmul_ru(a, a), __fmul_ru(b, b)), __fmul_ru(d, d)));
                    const float mc = __fadd_ru(__fadd_ru(__fmul_ru(fabsf(a), fabsf(bh->sphere_center[0])),
                                                         __fmul_ru(fabsf(b), fabsf(bh->sphere_center[1]))),
                                               __fadd_ru(__fmul_ru(fabsf(d), fabsf(bh->sphere_center[2])),
                                                         fabsf(M[4 * k + 3])));
                    const float e = __fadd_ru(__fmul_ru(rad, row), __fmul_ru(mc, 4.8e-7f));  // + 4 ulps of |M c| + |t|
                    lo[k] = fmaxf(lo[k], __fsub_rd(cwv[k], e));
                    hi[k] = fminf(hi[k], __fadd_ru(cwv[k], e));
                }
            }
            // and to the box of the transformed 14-DOP vertices
            const uint32_t nd = bh->dop_count;
            if (nd >= 4u && nd <= kDopMaxVertices) {
                float dlo[3] = {INFINITY, INFINITY, INFINITY}, dhi[3] = {-INFINITY, -INFINITY, -INFINITY};
                for (uint32_t v = 0; v < nd; v++) {
                    const V3 q = xform_point(rec->o2w, mk3(bh->dop_vertex[v][0], bh->dop_vertex[v][1],
                                                          bh->dop_vertex[v][2]));
                    dlo[0] = fminf(dlo[0], q.x); dlo[1] = fminf(dlo[1], q.y); dlo[2] = fminf(dlo[2], q.z);
                    dhi[0] = fmaxf(dhi[0], q.x); dhi[1] = fmaxf(dhi[1], q.y); dhi[2] = fmaxf(dhi[2], q.z);
                }
                for (int k = 0; k < 3; k++) {
                    lo[k] = fmaxf(lo[k], dlo[k]);
                    hi[k] = fminf(hi[k], dhi[k]);
                }
            }
            float ext = fmaxf(fmaxf(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]);
            for (int k = 0; k < 3; k++) {
                float pad = (fmaxf(fabsf(lo[k]), fabsf(hi[k])) + ext) * 1e-5f + 1e-20f;
                lo[k] -= pad;
                hi[k] += pad;
            }
            if (!finite3(lo) || !finite3(hi)) valid = false;
            if (valid) {
                rec->tri_count = bh->prim_count;
                rec->node_count = bh->node_count | (bh->node_bytes == kQNodeBytes ? kQuantizedBlasBit : 0u);
                rec->prims_off256 = (uint32_t)(bh->prims_offset / 256);
            }
        }
    }
    if (!valid) {
        rec->tri_count = 0;
        for (int k = 0; k < 3; k++) {
            lo[k] = INFINITY;
            hi[k] = -INFINITY;
        }
    }
    return valid;
}

// Instance i's record and box; every thread of the block takes part in the bounds.
__device__ __forceinline__ void tlas_prim(const RtAccelerationStructureInstance* inst, uint32_t i, uint32_t n,
                                          InstRecord* temp, BuildState* st, float4& blo, float4& bhi) {
    float cmin[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, cmax[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    float bmin[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, bmax[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    uint32_t kinds = 0;
    if (i < n) {
        RtAccelerationStructureInstance r = inst[i];
        InstRecord rec;
        float lo[3], hi[3];
        if (fill_instance(r, i, &rec, lo, hi, &st->error)) {
            for (int k = 0; k < 3; k++) {
                float c = 0.5f * (lo[k] + hi[k]);
                cmin[k] = cmax[k] = c;
                bmin[k] = lo[k];
                bmax[k] = hi[k];
            }
            kinds = blas_kind(rec.node_count);
        }
        temp[i] = rec;
        blo = make_float4(lo[0], lo[1], lo[2], 0.0f);
        bhi = make_float4(hi[0], hi[1], hi[2], 0.0f);
    }
    kinds = __reduce_or_sync(0xFFFFFFFFu, kinds);
    if ((threadIdx.x & 31u) == 0 && kinds) atomicOr(&st->blas_kinds, kinds);
    reduce_bounds(st, cmin, cmax, bmin, bmax);
}

__global__ void k_tlas_prims(const RtAccelerationStructureInstance* inst, uint32_t n, float4* boxes,
                             InstRecord* temp, BuildState* st, ZeroedWords z) {
    after_previous();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    zero_words(z, i, gridDim.x * blockDim.x);
    float4 lo, hi;
    tlas_prim(inst, i, n, temp, st, lo, hi);
    if (i < n) {
        boxes[2 * (size_t)i] = lo;
        boxes[2 * (size_t)i + 1] = hi;
    }
}

__device__ __forceinline__ uint32_t expand_bits10(uint32_t x) {
    x = (x * 0x00010001u) & 0xFF0000FFu;
    x = (x * 0x00000101u) & 0x0F00F00Fu;
    x = (x * 0x00000011u) & 0xC30C30C3u;
    x = (x * 0x00000005u) & 0x49249249u;
    return x;
}

// 30-bit Morton code of a box's centroid.
__device__ __forceinline__ uint32_t morton_code(float4 lo, float4 hi, const BuildState* st) {
    const float c[3] = {0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z)};
    uint32_t q[3] = {0, 0, 0};
    if (finite3(c)) {
        for (int k = 0; k < 3; k++) {
            float mn = o2f(st->cb[k]), mx = o2f(st->cb[3 + k]);
            float ext = mx - mn;
            float x = ext > 0.0f ? (c[k] - mn) / ext : 0.0f;
            float s = fminf(fmaxf(x * 1024.0f, 0.0f), 1023.0f);
            q[k] = (uint32_t)s;
        }
    }
    return (expand_bits10(q[0]) << 2) | (expand_bits10(q[1]) << 1) | expand_bits10(q[2]);
}

// Lanes of the (converged) warp whose 8-bit digit equals this lane's: one
// ballot per bit.  (__match_any_sync takes several times as long.)
__device__ __forceinline__ uint32_t digit_peers(uint32_t d) {
    uint32_t peers = 0xFFFFFFFFu;
#pragma unroll
    for (int b = 0; b < 8; b++) {
        const uint32_t bit = (d >> b) & 1u;
        peers &= __ballot_sync(0xFFFFFFFFu, bit) ^ (bit - 1u);
    }
    return peers;
}

// The whole sort in one block, for up to ITEMS * 1024 keys.  A pass ranks each
// warp's keys by digit in order (so it is stable), scans the counts of all
// (digit, warp) pairs, and moves the pairs through shared memory.  Keys past n
// are 2^32 - 1 and come last of equals, so they stay behind the n pairs.
// MORTON: the keys are the Morton codes of the boxes, the values their
// indices; otherwise the pairs are in k / v.  The result goes to k / v.
// Bound: latency and issue of one SM, 3 us and 0.9 us per item and pass (1,024
// keys 7 us, 4,096 keys 17 us with the codes); at 16 items onesweep's five
// launches are as fast.
constexpr uint32_t kSortRow = kSortThreads / 32 + 1;  // counts of one digit by warp, padded against bank conflicts
constexpr size_t sort_block_smem(int items) { return (256 * kSortRow + 2 * (size_t)items * kSortThreads) * 4; }
// The calling block (kSortThreads threads) sorts the pairs it holds: item r of
// a thread is number warp * ITEMS * 32 + 32 r + lane, before and after.
template <int ITEMS>
__device__ __forceinline__ void block_sort(uint32_t (&key)[ITEMS], uint32_t (&val)[ITEMS], uint32_t* sort_smem,
                                           uint32_t* warp_sums) {
    uint32_t* cnt = sort_smem;
    uint32_t* skeys = cnt + 256 * kSortRow;
    uint32_t* svals = skeys + ITEMS * kSortThreads;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, lt = (1u << lane) - 1u;
    const uint32_t first = warp * ITEMS * 32u + lane;
    for (int shift = 0; shift < 32; shift += 8) {
        for (uint32_t i = tid; i < 256 * kSortRow; i += kSortThreads) cnt[i] = 0;
        __syncthreads();
        uint32_t rank[ITEMS];
#pragma unroll
        for (int r = 0; r < ITEMS; r++) {
            const uint32_t d = (key[r] >> shift) & 255u, peers = digit_peers(d);
            uint32_t* c = &cnt[d * kSortRow + warp];
            const uint32_t before = *c;
            __syncwarp();
            if ((peers & lt) == 0u) *c = before + (uint32_t)__popc(peers);
            __syncwarp();
            rank[r] = before + (uint32_t)__popc(peers & lt);
        }
        __syncthreads();
        // exclusive scan over (digit, warp): eight counts per thread
        uint32_t* row = &cnt[(tid >> 2) * kSortRow + (tid & 3u) * 8u];
        uint32_t part[8], sum = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            part[j] = sum;
            sum += row[j];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, off);
            if (lane >= (uint32_t)off) incl += o;
        }
        if (lane == 31u) warp_sums[warp] = incl;
        __syncthreads();
        const uint32_t before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? warp_sums[lane] : 0u) + incl - sum;
#pragma unroll
        for (int j = 0; j < 8; j++) row[j] = before + part[j];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ITEMS; r++) {
            const uint32_t pos = cnt[((key[r] >> shift) & 255u) * kSortRow + warp] + rank[r];
            skeys[pos] = key[r];
            svals[pos] = val[r];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ITEMS; r++) {
            key[r] = skeys[first + 32u * r];
            val[r] = svals[first + 32u * r];
        }
    }
}

template <bool MORTON, int ITEMS>
__global__ void __launch_bounds__(kSortThreads) k_sort_block(uint32_t* k, uint32_t* v, uint32_t n, const float4* boxes,
                                                             const BuildState* st) {
    after_previous();
    extern __shared__ uint32_t sort_smem[];
    __shared__ uint32_t warp_sums[kSortThreads / 32];
    const uint32_t first = (threadIdx.x >> 5) * ITEMS * 32u + (threadIdx.x & 31u);  // item r of this thread: first + 32 r
    uint32_t key[ITEMS], val[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const uint32_t i = first + 32u * r;
        key[r] = 0xFFFFFFFFu;
        val[r] = 0u;
        if (i < n) {
            key[r] = MORTON ? morton_code(boxes[2 * (size_t)i], boxes[2 * (size_t)i + 1], st) : k[i];
            val[r] = MORTON ? i : v[i];
        }
    }
    block_sort<ITEMS>(key, val, sort_smem, warp_sums);
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const uint32_t i = first + 32u * r;
        if (i < n) {
            k[i] = key[r];
            v[i] = val[r];
        }
    }
}

// ---- onesweep radix sort ------------------------------------------------------
// Keys of more than one sort tile are sorted by the single-pass LSD scheme of
// Adinets & Merrill ("Onesweep", 2022): one upfront histogram of all four
// 8-bit digits, then one kernel per digit.  In a digit pass each block takes
// the next partition of kOsTile keys from a counter (so every earlier
// partition belongs to a block that is already running), ranks its keys
// stably per digit (one ballot per bit, warps over consecutive chunks), publishes
// its per-digit counts, and finds the keys of each digit in all earlier
// partitions by decoupled look-back: it walks back over their descriptors,
// adding aggregates until one carries the inclusive prefix.  The tile is then
// staged in shared memory in digit order and written out so that consecutive
// threads write consecutive positions.  Each look-back wait is bounded: after
// kOsSpinLimit polls the build records RT_ERR_TIMEOUT and goes on.
constexpr int kOsThreads = 256;
constexpr int kOsItems = 15;
constexpr uint32_t kOsTile = kOsThreads * kOsItems;  // 3840 keys per partition
constexpr int kOsWarps = kOsThreads / 32;
constexpr uint32_t kOsHistBlocks = 152 * 8;  // of the histogram: a full load of the SMs
constexpr uint32_t kOsAggregate = 1u << 30, kOsPrefix = 2u << 30, kOsValue = (1u << 30) - 1u;
constexpr uint32_t kOsSpinLimit = 1u << 22;
constexpr int kOsLook = 8;  // descriptors read at once in a look-back

// The sort's scratch header: digit counts of the four passes and each pass's
// partition counter.  The partition descriptors follow: [pass][partition][digit].
struct OnesweepState {
    uint32_t count[4][256];
    uint32_t next_partition[4];
};

__host__ __device__ inline uint32_t onesweep_partitions(uint32_t n) { return (n + kOsTile - 1) / kOsTile; }

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Digit counts of all four passes.  MORTON: the keys are the Morton codes of
// the boxes, written here with their indices as values.
template <bool MORTON>
__global__ void __launch_bounds__(kOsThreads) k_onesweep_hist(uint32_t* keys, uint32_t* vals, uint32_t n,
                                                              OnesweepState* os, const float4* boxes,
                                                              const BuildState* st) {
    after_previous();
    __shared__ uint32_t h[4][256];
    for (int i = threadIdx.x; i < 1024; i += blockDim.x) (&h[0][0])[i] = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t k;
        if (MORTON) {
            k = morton_code(boxes[2 * (size_t)i], boxes[2 * (size_t)i + 1], st);
            keys[i] = k;
            vals[i] = i;
        } else {
            k = keys[i];
        }
        atomicAdd(&h[0][k & 255u], 1u);
        atomicAdd(&h[1][(k >> 8) & 255u], 1u);
        atomicAdd(&h[2][(k >> 16) & 255u], 1u);
        atomicAdd(&h[3][k >> 24], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 1024; i += blockDim.x) {
        const uint32_t c = (&h[0][0])[i];
        if (c) atomicAdd(&(&os->count[0][0])[i], c);
    }
}

// Exclusive scan of 256 values by 256 threads (one value each).
__device__ __forceinline__ uint32_t block_scan256(uint32_t c, uint32_t* warp_sums) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t incl = c;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, off);
        if (lane >= (uint32_t)off) incl += o;
    }
    if (lane == 31u) warp_sums[warp] = incl;
    __syncthreads();
    uint32_t before = 0;
    for (uint32_t w = 0; w < warp; w++) before += warp_sums[w];
    return before + incl - c;
}

struct OnesweepShared {
    uint32_t keys[kOsTile];
    uint32_t vals[kOsTile];
    uint32_t warp_cnt[kOsWarps][256];  // keys of each digit per warp, then each warp's offset among them
    uint32_t tile_start[256];          // first position of each digit in the staged tile
    uint32_t out_start[256];           // first output position of the tile's keys of each digit
    uint32_t warp_sums[8];
    uint32_t partition;
};

// One digit pass (bits pass*8 .. pass*8+7) over n keys: kin / vin -> kout / vout.
// desc: this pass's descriptors, 256 per partition, zeroed.
__global__ void __launch_bounds__(kOsThreads, 3) k_onesweep_pass(const uint32_t* kin, const uint32_t* vin,
                                                               uint32_t* kout, uint32_t* vout, uint32_t n, int pass,
                                                               OnesweepState* os, uint32_t* desc,
                                                               uint32_t* error) {
    after_previous();
    __shared__ OnesweepShared sm;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const int shift = pass * 8;
    if (tid == 0) sm.partition = atomicAdd(&os->next_partition[pass], 1u);
    for (uint32_t i = tid; i < kOsWarps * 256; i += kOsThreads) (&sm.warp_cnt[0][0])[i] = 0;
    __syncthreads();
    const uint32_t p = sm.partition;
    const uint32_t base = p * kOsTile;
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t key[kOsItems], val[kOsItems], rank[kOsItems];
    // warp w ranks keys base + w*32*kOsItems .. in rounds of 32, in order: stable within the tile
    const uint32_t first = base + (uint32_t)warp * kOsItems * 32u + lane;
#pragma unroll
    for (int r = 0; r < kOsItems; r++) key[r] = first + r * 32u < n ? kin[first + r * 32u] : 0u;
#pragma unroll
    for (int r = 0; r < kOsItems; r++) val[r] = first + r * 32u < n ? vin[first + r * 32u] : 0u;
    const uint32_t digit_total = os->count[pass][tid];
#pragma unroll
    for (int r = 0; r < kOsItems; r++) {
        const bool valid = first + r * 32u < n;
        const uint32_t d = (key[r] >> shift) & 255u;
        const uint32_t peers = digit_peers(d) & __ballot_sync(0xFFFFFFFFu, valid);
        const uint32_t before = valid ? sm.warp_cnt[warp][d] : 0u;
        __syncwarp();
        if (valid && (peers & lt) == 0u) sm.warp_cnt[warp][d] = before + (uint32_t)__popc(peers);
        __syncwarp();
        rank[r] = valid ? before + (uint32_t)__popc(peers & lt) : 0xFFFFFFFFu;
    }
    __syncthreads();
    // thread d: the tile's keys of digit d, and each warp's offset among them
    const uint32_t d = tid;
    uint32_t total = 0;
    for (int w = 0; w < kOsWarps; w++) {
        const uint32_t c = sm.warp_cnt[w][d];
        sm.warp_cnt[w][d] = total;
        total += c;
    }
    // publish, then look back for the keys of digit d in the earlier partitions
    uint32_t* mine = desc + (size_t)p * 256u + d;
    uint32_t excl = 0;
    if (p == 0) {
        st_relaxed(mine, kOsPrefix | total);
    } else {
        st_relaxed(mine, kOsAggregate | total);
        // kOsLook descriptors at a time: when all partitions run at once, none
        // has a prefix yet and one read per step would take p round trips to L2
        uint32_t q = p, spins = 0;  // the partitions before q are still to be added
        for (bool more = true; more;) {
            uint32_t v[kOsLook];
#pragma unroll
            for (int j = 0; j < kOsLook; j++)
                v[j] = q > (uint32_t)j ? ld_relaxed(desc + (size_t)(q - 1u - j) * 256u + d) : kOsPrefix;
            uint32_t taken = 0;
#pragma unroll
            for (int j = 0; j < kOsLook; j++) {
                const uint32_t flag = v[j] & ~kOsValue;
                if (!more || taken != (uint32_t)j || flag == 0u) continue;
                excl += v[j] & kOsValue;
                taken++;
                if (flag == kOsPrefix) more = false;
            }
            q -= min(taken, q);
            if (more && taken < (uint32_t)kOsLook) {  // the next one is not published yet
                if (++spins > kOsSpinLimit) {  // bounded: report and go on with what was found
                    atomicOr(error, 1u << RT_ERR_TIMEOUT);
                    break;
                }
                __nanosleep(32);
            }
        }
        st_relaxed(mine, kOsPrefix | (excl + total));
    }
    sm.tile_start[d] = block_scan256(total, sm.warp_sums);
    __syncthreads();  // warp_sums is used again
    sm.out_start[d] = block_scan256(digit_total, sm.warp_sums) + excl;  // every key of a smaller digit comes before
    __syncthreads();
    // stage the tile in digit order, then write it out in that order
#pragma unroll
    for (int r = 0; r < kOsItems; r++) {
        if (rank[r] == 0xFFFFFFFFu) continue;
        const uint32_t dg = (key[r] >> shift) & 255u;
        const uint32_t local = sm.tile_start[dg] + sm.warp_cnt[warp][dg] + rank[r];
        sm.keys[local] = key[r];
        sm.vals[local] = val[r];
    }
    __syncthreads();
    const uint32_t cnt = min(kOsTile, n - base);
    for (uint32_t i = tid; i < cnt; i += kOsThreads) {
        const uint32_t k = sm.keys[i];
        const uint32_t dg = (k >> shift) & 255u;
        const uint32_t pos = sm.out_start[dg] + (i - sm.tile_start[dg]);
        if (pos < n) {
            kout[pos] = k;
            vout[pos] = sm.vals[i];
        }
    }
}

}  // namespace

uint64_t key_sort_state_bytes(uint32_t n) {
    return sizeof(OnesweepState) + (uint64_t)4 * onesweep_partitions(n ? n : 1) * 256u * 4u;
}

namespace {
template <bool MORTON, int ITEMS>
cudaError_t launch_sort_block(uint32_t* k, uint32_t* v, uint32_t n, const float4* boxes, const BuildState* st,
                              cudaStream_t stream) {
    const size_t smem = sort_block_smem(ITEMS);
    // a per-device attribute: set on every sort (a host-side call, no device work)
    const cudaError_t e =
        cudaFuncSetAttribute(k_sort_block<MORTON, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    launch(k_sort_block<MORTON, ITEMS>, 1, kSortThreads, smem, stream, k, v, n, boxes, st);
    return cudaGetLastError();
}

// Sorts n pairs (MORTON: the boxes' Morton codes and indices) into k0 / v0.
template <bool MORTON>
cudaError_t launch_sort(uint32_t* k0, uint32_t* v0, uint32_t* k1, uint32_t* v1, uint32_t n, uint8_t* state,
                        uint32_t* error, const float4* boxes, const BuildState* st, cudaStream_t stream) {
    if (n <= kSortThreads) return launch_sort_block<MORTON, 1>(k0, v0, n, boxes, st, stream);
    if (n <= 2 * kSortThreads) return launch_sort_block<MORTON, 2>(k0, v0, n, boxes, st, stream);
    if (n <= 4 * kSortThreads) return launch_sort_block<MORTON, 4>(k0, v0, n, boxes, st, stream);
    if (n <= kSortBlockMax) return launch_sort_block<MORTON, 8>(k0, v0, n, boxes, st, stream);
    OnesweepState* os = reinterpret_cast<OnesweepState*>(state);
    uint32_t* desc = reinterpret_cast<uint32_t*>(state + sizeof(OnesweepState));
    const uint32_t parts = onesweep_partitions(n);
    if (!MORTON) {  // a build's first kernel has zeroed it
        const cudaError_t e = cudaMemsetAsync(state, 0, key_sort_state_bytes(n), stream);
        if (e != cudaSuccess) return e;
    }
    launch(k_onesweep_hist<MORTON>, std::min<uint32_t>((n + kOsThreads - 1) / kOsThreads, kOsHistBlocks), kOsThreads, 0, stream, k0, v0, n, os, boxes, st);
    uint32_t* kin = k0;
    uint32_t* vin = v0;
    uint32_t* kout = k1;
    uint32_t* vout = v1;
    for (int pass = 0; pass < 4; pass++) {
        launch(k_onesweep_pass, parts, kOsThreads, 0, stream, kin, vin, kout, vout, n, pass, os, desc + (size_t)pass * parts * 256u, error);
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_key_sort(uint32_t* k0, uint32_t* v0, uint32_t* k1, uint32_t* v1, uint32_t n, uint8_t* state,
                            uint32_t* error, cudaStream_t stream) {
    if (n <= 1) return cudaSuccess;
    return launch_sort<false>(k0, v0, k1, v1, n, state, error, nullptr, nullptr, stream);
}

namespace {

__global__ void k_gather_boxes(const float4* boxes, const uint32_t* vals, uint32_t n, float4* sboxes) {
    after_previous();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t p = vals[i];
    sboxes[2 * (size_t)i] = boxes[2 * (size_t)p];
    sboxes[2 * (size_t)i + 1] = boxes[2 * (size_t)p + 1];
}

// ---- Karras hierarchy -------------------------------------------------------
__device__ __forceinline__ int kdelta(const uint32_t* k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    uint32_t a = k[i], b = k[j];
    if (a == b) return 32 + __clz((uint32_t)i ^ (uint32_t)j);
    return __clz(a ^ b);
}

__global__ void k_karras(const uint32_t* keys, uint32_t n_u, uint4* inodes, uint32_t* iparent, uint32_t* lparent,
                         uint32_t* flags, ZeroedWords z) {
    after_previous();
    int n = (int)n_u;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    zero_words(z, (uint32_t)i, gridDim.x * blockDim.x);
    if (i >= n - 1) return;
    flags[i] = 0;  // arrivals at the node, for k_bottom_up
    int d = (kdelta(keys, n, i, i + 1) - kdelta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = kdelta(keys, n, i, i - d);
    int lmax = 2;
    while (kdelta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (kdelta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = kdelta(keys, n, i, j);
    int s = 0;
    int t = l;
    do {
        t = (t + 1) >> 1;
        if (kdelta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    int gamma = i + s * d + min(d, 0);
    int first = min(i, j), last = max(i, j);
    uint32_t left = (first == gamma) ? (kLeafBit | (uint32_t)gamma) : (uint32_t)gamma;
    uint32_t right = (last == gamma + 1) ? (kLeafBit | (uint32_t)(gamma + 1)) : (uint32_t)(gamma + 1);
    inodes[i] = make_uint4(left, right, (uint32_t)first, (uint32_t)last);
    if (left & kLeafBit) lparent[gamma] = (uint32_t)i;
    else iparent[gamma] = (uint32_t)i;
    if (right & kLeafBit) lparent[gamma + 1] = (uint32_t)i;
    else iparent[gamma + 1] = (uint32_t)i;
    if (i == 0) iparent[0] = kNone;
}

__device__ __forceinline__ void load_box_cg(const float4* b, size_t i, float lo[3], float hi[3]) {
    float4 l = __ldcg(&b[2 * i]), h = __ldcg(&b[2 * i + 1]);
    lo[0] = l.x; lo[1] = l.y; lo[2] = l.z;
    hi[0] = h.x; hi[1] = h.y; hi[2] = h.z;
}

// Adds 1 to a node's arrivals and returns how many came before.  What the
// caller wrote is visible to whoever arrives later, and what those before it
// wrote is visible to the caller.
__device__ __forceinline__ uint32_t arrive(uint32_t* arrivals) {
    uint32_t before;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(arrivals) : "memory");
    return before;
}

// Boxes from the leaves up: a thread climbs until it is the first at a node;
// the second carries the box of its own child in registers, reads the
// other's, and goes on.  What the next step needs of the hierarchy is read
// beside the arrival, so a step waits for the arrival and one box.
// (4,096 leaves: 29 -> 22 us.)
__global__ void k_bottom_up(const uint4* inodes, const uint32_t* lparent, const uint32_t* iparent,
                            const float4* sboxes, float4* iboxes, uint32_t* flags, uint32_t n, uint32_t* err) {
    after_previous();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t p = lparent[i], self = kLeafBit | i;
    float lo[3], hi[3];
    load_box_cg(sboxes, i, lo, hi);
    for (int guard = 0; p != kNone; guard++) {
        if (guard >= 160 || p >= n - 1) {  // deeper than any Karras tree of 2^28 keys
            atomicOr(err, 1u << RT_ERR_BAD_AS);
            return;
        }
        const uint4 nd = inodes[p];
        const uint32_t above = iparent[p];
        if (arrive(&flags[p]) == 0u) return;
        const uint32_t other = nd.x == self ? nd.y : nd.x;
        float olo[3], ohi[3];
        if (other & kLeafBit) load_box_cg(sboxes, other & ~kLeafBit, olo, ohi);
        else load_box_cg(iboxes, other, olo, ohi);
        for (int k = 0; k < 3; k++) {
            lo[k] = fminf(lo[k], olo[k]);
            hi[k] = fmaxf(hi[k], ohi[k]);
        }
        iboxes[2 * (size_t)p] = make_float4(lo[0], lo[1], lo[2], __uint_as_float(nd.w - nd.z + 1u));  // primitives below
        iboxes[2 * (size_t)p + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
        self = p;
        p = above;
    }
}

// ---- PLOC hierarchy (RT_BUILD_PREFER_FAST_TRACE) --------------------------------
// Parallel locally-ordered clustering (Meister & Bittner, "Parallel
// Locally-Ordered Clustering for Bounding Volume Hierarchy Construction",
// IEEE TVCG 2018).  The clusters start as the Morton-ordered primitives.
// Each round every cluster finds, among the kPlocRadius clusters on either
// side of it, the one whose merged box has the smallest surface area; mutual
// nearest neighbours merge into a new internal node at the lower position,
// and the surviving clusters are compacted in order.  Internal node ids are
// handed out from n - 2 down, so the last merge (the root) is node 0, where
// the collapse starts.  A cluster is two float4: (lo, binary reference) and
// (hi, primitives below it).
//
// Mutual pairs alone leave 0.81 of the clusters per round, and in fans of
// slivers (the poles of a sphere), where each cluster's nearest is the next
// one of a chain, 0.98.  So a cluster at an odd position that has no mutual
// neighbour also merges with its nearest neighbour j when j is at an even
// position, has no mutual neighbour either, and its own nearest is hardly
// nearer (kPlocNear): j takes the best of those that ask.  That leaves 0.75
// per round (2.6M-triangle sphere: 26 rounds to 1024 clusters instead of 134).
// Nodes visited a ray, random rays, mutual pairs only -> now: spheres of 164k /
// 1M / 10.5M triangles 8.75 / 9.91 / 13.98 -> 8.70 / 9.66 / 12.24, 300k
// scattered triangles 91.2 -> 85.2, hair 25.5 -> 24.1, a torus 9.28 -> 9.53,
// 200k triangles of very different sizes 82.4 -> 83.9.
//
// Rounds over more than kPlocSmall clusters are one grid-wide launch each
// (k_ploc_round; the cluster count stays on the device), and k_ploc_pairs
// takes a mesh that needs more rounds than were launched.  One CTA with every
// cluster in shared memory finishes (k_ploc_tail).  When a round leaves more
// than 31/32 of its clusters (many equal or NaN areas), the next one merges
// neighbour pairs (i, i ^ 1) instead.
constexpr int kPlocRadius = 16;
constexpr uint32_t kPlocSmall = 1024;  // clusters the one-CTA tail holds, one per thread
constexpr float kPlocNear = 1.25f;
constexpr double kPlocFirstRate = 0.62, kPlocRate = 0.765;  // survivors of the first and of later rounds of closed meshes
constexpr uint32_t kPlocThreads = 512;
constexpr uint32_t kPlocTile = kPlocThreads - 6 * kPlocRadius;  // clusters a block owns per tile
constexpr uint32_t kPlocMaxBlocks = 152 * 4;
constexpr uint32_t kPlocParity = 1u << 31, kPlocForced = 1u << 30, kPlocCount = (1u << 28) - 1u;
constexpr uint32_t kPlocSpinLimit = 1u << 22;

struct PlocArgs {
    const float4* boxes;     // primitive boxes in caller order
    const uint32_t* vals;    // Morton order -> primitive
    float4* sboxes;          // primitive boxes in Morton order (written by the first round)
    float4* cbox[2];         // clusters, double-buffered
    uint4* inodes;
    float4* iboxes;
    BuildState* st;
    unsigned long long* desc;  // look-back descriptors: (round + 1) << 34 | state << 32 | survivors
    uint32_t n;
};

__device__ __forceinline__ float merged_half_area(float ax, float ay, float az, float bx, float by, float bz,
                                                  float cx, float cy, float cz, float dx, float dy, float dz) {
    // boxes (a, b) and (c, d) as lo, hi corners
    float ex = fmaxf(bx, dx) - fminf(ax, cx), ey = fmaxf(by, dy) - fminf(ay, cy), ez = fmaxf(bz, dz) - fminf(az, cz);
    return fmaf(ex, ey + ez, ey * ez);
}

// The internal node of a merge: children a and b, the merged box, the primitives below.
__device__ __forceinline__ void ploc_write_node(const PlocArgs& a, uint32_t id, uint32_t ra, uint32_t rb, float4 lo,
                                                float4 hi, uint32_t size) {
    a.inodes[id] = make_uint4(ra, rb, 0u, 0u);
    a.iboxes[2 * (size_t)id] = make_float4(lo.x, lo.y, lo.z, __uint_as_float(size));
    a.iboxes[2 * (size_t)id + 1] = make_float4(hi.x, hi.y, hi.z, 0.0f);
}

__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Survivors of the tiles before `tile` in this round, by decoupled look-back:
// the calling warp reads 32 descriptors at a time, waits until each is
// published, and stops at the first that carries an inclusive prefix.
// Bounded: after kPlocSpinLimit polls the build records RT_ERR_TIMEOUT.
__device__ uint32_t ploc_look_back(const unsigned long long* desc, uint32_t round, uint32_t tile, uint32_t* error) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t sum = 0, spins = 0;
    for (int64_t at = (int64_t)tile - 1;; at -= 32) {
        const int64_t q = at - lane;
        uint32_t state = 2u, value = 0u;  // before the first tile: a prefix of 0
        if (q >= 0) {
            for (;;) {
                const unsigned long long v = ld_relaxed64(&desc[q]);
                if ((uint32_t)(v >> 34) == round + 1u) {
                    state = (uint32_t)(v >> 32) & 3u;
                    value = (uint32_t)v;
                    break;
                }
                if (++spins > kPlocSpinLimit) {
                    atomicOr(error, 1u << RT_ERR_TIMEOUT);
                    break;  // go on with what was found
                }
                __nanosleep(20);
            }
        }
        __syncwarp();
        const unsigned prefix = __ballot_sync(0xFFFFFFFFu, state == 2u);
        const int stop = prefix ? __ffs(prefix) - 1 : 31;  // nearest tile with an inclusive prefix
        sum += __reduce_add_sync(0xFFFFFFFFu, (int)lane <= stop ? value : 0u);
        if (prefix) return sum;
    }
}

// The best of the neighbours looked at so far: the area of the merge with it
// (float bits) and its offset.  Areas are compared whole; the lower position
// wins ties.  Areas from kPlocNoArea on (infinity and NaN) are no neighbour.
constexpr uint32_t kPlocNoArea = 0x7F800000u;
struct PlocBest {
    uint32_t area = 0xFFFFFFFFu;
    int offset = 0;
    // neighbours in ascending position above all seen so far
    __device__ __forceinline__ void higher(uint32_t a, int o) {
        bool keep;
        area = __vibmin_u32(area, a, &keep);
        offset = keep ? offset : o;
    }
    // neighbours in descending position below all seen so far
    __device__ __forceinline__ void lower(uint32_t a, int o) {
        bool take;
        area = __vibmin_u32(a, area, &take);
        offset = take ? o : offset;
    }
};
// The nearest neighbours of a round: `area` of the merge, `offset` of its place (0: none).
struct PlocNear {
    const uint32_t* area;
    const int8_t* offset;
    __device__ __forceinline__ int operator()(int x) const { return x + offset[x]; }  // x itself if it has none
};
// The neighbours below place x, whose areas are in area[o - 1][place of the
// lower].  FIRST: place 0 is the first position; otherwise there are R places
// before x.
template <bool FIRST, int STRIDE>
__device__ __forceinline__ void ploc_below(const uint32_t (*area)[STRIDE], int x, int from, int to, PlocBest& best) {
#pragma unroll
    for (int o = from; o <= to; o++) best.lower(!FIRST || x >= o ? area[o - 1][x - o] : 0xFFFFFFFFu, -o);
}
// The nearest of all neighbours (of the tail's clusters).  Four runs at once:
// the comparisons of one wait for each other.
template <int STRIDE>
__device__ __forceinline__ PlocBest ploc_nearest(const uint32_t (*area)[STRIDE], int x) {
    constexpr int R = kPlocRadius, H = R / 2;
    PlocBest best, far, below, far_below;
#pragma unroll
    for (int o = 1; o <= H; o++) {
        best.higher(area[o - 1][x], o);
        far.higher(area[o + H - 1][x], o + H);
    }
    ploc_below<true>(area, x, 1, H, below);
    ploc_below<true>(area, x, H + 1, R, far_below);
    best.higher(far.area, far.offset);
    best.lower(below.area, below.offset);
    best.lower(far_below.area, far_below.offset);
    return best;
}
__device__ __forceinline__ void ploc_store(uint32_t* area, int8_t* offset, int x, const PlocBest& best) {
    area[x] = best.area;
    offset[x] = (int8_t)(best.area < kPlocNoArea ? best.offset : 0);
}
// An asker in one word, the best the smallest (PLOC++, Benthin et al., 2022,
// packs a distance and an offset so, but drops bits of the distance): how much
// its area is above the asked place's own nearest, in units in the last place,
// and in the low five bits its offset from there (-R..-1 as 0..15, 1..R as
// 16..31), so that the lower position wins ties.  The difference is not
// negative, since the asker is among the asked place's neighbours, and
// kPlocNear keeps it below 2^22.
__device__ __forceinline__ uint32_t ploc_asker(const PlocNear& near, int x, int y) {
    const int o = x - y;
    return (near.area[x] - near.area[y]) << 5 | (uint32_t)(o < 0 ? o + kPlocRadius : o + kPlocRadius - 1);
}
// Place x (its neighbour at y, odd position, not mutual) asks y when y's
// position is even, it has no mutual neighbour either and its own nearest is
// hardly nearer.
__device__ __forceinline__ void ploc_ask(const PlocNear& near, uint32_t* take, int x, int y) {
    const int z = near(y);
    if (z != y && near(z) == y) return;
    if (__uint_as_float(near.area[x]) <= __uint_as_float(near.area[y]) * kPlocNear)
        atomicMin(&take[y], ploc_asker(near, x, y));
}
// The place that place x merges with (x itself: none).  y: its nearest (x
// itself if it has none); odd: of its position.
__device__ __forceinline__ int ploc_partner(const PlocNear& near, const uint32_t* take, int x, int y, bool mutual,
                                            bool odd) {
    if (mutual) return y;
    if (odd) return y != x && take[y] == ploc_asker(near, x, y) ? y : x;
    const uint32_t k = take[x];
    const int o = (int)(k & 31u);
    return k == 0xFFFFFFFFu ? x : x + (o < kPlocRadius ? o - kPlocRadius : o - kPlocRadius + 1);
}

// One round over more than kPlocSmall clusters.  A block takes tiles in
// ticket order.  Of its 512 threads' positions the middle 416 are its own and
// 3 R on each side a halo: boxes for all 512, the areas of the pairs
// (p, p + 1..R) once each (they do not depend on the order of the boxes) in
// shared memory, the nearest neighbour (smallest area, the lower position on
// ties) of the positions within 2 R of an own one, which ask those within R,
// then the merges of the own positions: the lower of a pair keeps the new
// node, the higher drops out.  A position keeps its minimum over those above
// it in a register and reads back only the areas below (0.3 % of a pass at
// 163,840 triangles and 0.5 % at 10.5M against reading all 32).  The tile
// claims its merges' node ids with one atomic (counting down from n - 2) and
// finds its survivors' output position by look-back over the earlier tiles, so
// one launch reads each cluster once and writes each survivor once: 32 + 0.8 x
// 32 bytes per cluster.  (Neighbour
// search, merge and compaction as three launches moved about 200 bytes per
// cluster: PLOC of 10.5M triangles 3.6 ms; of 164k triangles 410 us.)  Bound:
// the barriers between a tile's phases (first round of 2.6M triangles, 132 us:
// 22.5 of the warps' 38 cycles per issue at a barrier, 28 of 32 lanes, issue 40
// %, L1 and shared memory 57 %, DRAM 21 %); for small counts the latency of one
// tile.
// The first round gathers the Morton-ordered primitive boxes itself.
// PER_SM: resident blocks, 4 (32 registers) where there are tiles for them
// all, which overlaps one tile's gathers with more others' arithmetic (10.5M
// triangles: pass 3.86 -> 3.64 ms), 3 (39 registers) for rounds bound by
// the latency of one tile (163,840 triangles 0.5 % faster so).
template <int PER_SM>
__global__ void __launch_bounds__(kPlocThreads, PER_SM) k_ploc_round(const __grid_constant__ PlocArgs a, int round) {
    after_previous();
    BuildState* st = a.st;
    const uint32_t word = st->ploc_round[round], count = word & kPlocCount;
    if (count <= kPlocSmall) {
        if (blockIdx.x == 0 && threadIdx.x == 0) st->ploc_round[round + 1] = word;
        return;
    }
    constexpr int R = kPlocRadius, T = (int)kPlocThreads;
    const bool forced = (word & kPlocForced) != 0u;
    const float4* cin = a.cbox[(word & kPlocParity) ? 1 : 0];
    float4* cout = a.cbox[(word & kPlocParity) ? 0 : 1];
    __shared__ float4 s0[T];          // lo, hi.x
    __shared__ float2 s1[T];          // hi.y, hi.z
    __shared__ uint32_t area[R][T - R];  // area[o - 1][t] = area of the pair (t, t + o), its bits
    __shared__ uint32_t near_area[T];    // nearest neighbours
    __shared__ int8_t near_offset[T];
    __shared__ uint32_t take[T];         // the asker a place takes
    const PlocNear nearest{near_area, near_offset};
    __shared__ uint32_t warp_sums[2 * T / 32];  // each warp's total, then the totals before it
    __shared__ uint32_t s_tile, s_claim, s_prefix;
    const int t = (int)threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t tiles = (count + kPlocTile - 1u) / kPlocTile;
    if (blockIdx.x >= tiles) return;  // the others are enough: each takes tiles until none is left
    for (;;) {
        if (t == 0) s_tile = atomicAdd(&st->ploc_ticket[round], 1u);
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= tiles) return;
        const int i = (int)(tile * kPlocTile) - 3 * R + t;  // this thread's position
        const bool inside = i >= 0 && i < (int)count;
        const bool own = inside && t >= 3 * R && t < T - 3 * R;
        // outside the round: a box whose merges have infinite area
        float4 lo = make_float4(INFINITY, INFINITY, INFINITY, 0.f), hi = lo;
        if (inside) {
            if (round == 0) {
                const size_t p = a.vals[i];
                lo = a.boxes[2 * p];
                hi = a.boxes[2 * p + 1];
                if (own) {
                    a.sboxes[2 * (size_t)i] = lo;
                    a.sboxes[2 * (size_t)i + 1] = hi;
                }
                lo.w = __uint_as_float(kLeafBit | (uint32_t)i);
                hi.w = __uint_as_float(1u);
            } else {
                lo = __ldcg(&cin[2 * (size_t)i]);
                hi = __ldcg(&cin[2 * (size_t)i + 1]);
            }
        }
        s0[t] = make_float4(lo.x, lo.y, lo.z, hi.x);
        s1[t] = make_float2(hi.y, hi.z);
        __syncthreads();
        PlocBest best;  // first of the positions above
        if (t < T - R) {
#pragma unroll
            for (int o = 1; o <= R; o++) {
                const float4 c = s0[t + o];
                const float2 d = s1[t + o];
                const uint32_t bits = __float_as_uint(
                    merged_half_area(lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, c.x, c.y, c.z, c.w, d.x, d.y));
                area[o - 1][t] = bits;
                best.higher(bits, o);
            }
        }
        __syncthreads();
        if (t >= R && t < T - R) {
            if (!forced) ploc_below<false>(area, t, 1, R, best);
            else best.area = 0u, best.offset = (i ^ 1) < (int)count ? (i ^ 1) - i : 0;
            if (!inside) best.offset = 0;
            ploc_store(near_area, near_offset, t, best);
        }
        take[t] = 0xFFFFFFFFu;
        __syncthreads();
        if (t >= R && t < T - R && inside && (i & 1)) {
            const int near = nearest(t);
            if (near >= 2 * R && near < T - 2 * R &&  // the neighbours that an own place can have
                ((near - t) & 1) && nearest(near) != t)
                ploc_ask(nearest, take, t, near);
        }
        __syncthreads();
        uint32_t k = 0u;
        bool merging = false;
        int tj = t;
        if (own) {
            const int near = nearest(t);
            tj = ploc_partner(nearest, take, t, near, near != t && nearest(near) == t, (i & 1) != 0);  // t itself: no merge
            merging = tj > t;
            k = tj < t ? 0u : 1u;
        }
        // one scan counts survivors (low 16 bits) and merges (high 16 bits)
        const uint32_t v = k | (merging ? 1u << 16 : 0u);
        uint32_t incl = v;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, off);
            if (lane >= (uint32_t)off) incl += o;
        }
        if (lane == 31u) warp_sums[warp] = incl;
        __syncthreads();
        if (warp == 1) {  // beside the look-back: both wait on L2
            const uint32_t m = __reduce_add_sync(0xFFFFFFFFu, lane < T / 32 ? warp_sums[lane] >> 16 : 0u);
            if (lane == 0) s_claim = m ? atomicAdd(&st->merge_counter, m) : 0u;
        }
        if (warp == 0) {
            const uint32_t w = lane < T / 32 ? warp_sums[lane] : 0u;
            uint32_t wi = w;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, wi, off);
                if (lane >= (uint32_t)off) wi += o;
            }
            const uint32_t total = __shfl_sync(0xFFFFFFFFu, wi, 31);
            const unsigned long long tag = (unsigned long long)(round + 1) << 34;
            if (lane == 0) st_relaxed64(&a.desc[tile], tag | (1ull << 32) | (total & 0xFFFFu));
            if (lane < T / 32) warp_sums[T / 32 + lane] = wi - w;
            const uint32_t before = ploc_look_back(a.desc, (uint32_t)round, tile, &st->error);
            if (lane == 0) {
                const uint32_t after = before + (total & 0xFFFFu);
                st_relaxed64(&a.desc[tile], tag | (2ull << 32) | after);
                s_prefix = before;
                if (tile == tiles - 1u)
                    st->ploc_round[round + 1] = (after & kPlocCount) | ((word & kPlocParity) ^ kPlocParity) |
                                                (after > count - count / 32u ? kPlocForced : 0u);
            }
        }
        __syncthreads();
        if (k) {
            const uint32_t excl = warp_sums[T / 32 + warp] + incl - v;
            const size_t pos = s_prefix + (excl & 0xFFFFu);
            if (merging) {
                const uint32_t claim = s_claim + (excl >> 16);
                if (claim + 2u > a.n) {  // more merges than a binary tree over n primitives has
                    atomicOr(&st->error, 1u << RT_ERR_BAD_AS);
                } else {
                    const uint32_t id = a.n - 2u - claim;
                    const float4 c = s0[tj];
                    const float2 d = s1[tj];
                    const size_t j = (size_t)(i + (tj - t));
                    const uint32_t rj = round == 0 ? kLeafBit | (uint32_t)j : __float_as_uint(__ldcg(&cin[2 * j]).w);
                    const uint32_t sj = round == 0 ? 1u : __float_as_uint(__ldcg(&cin[2 * j + 1]).w);
                    const uint32_t ri = __float_as_uint(lo.w), size = __float_as_uint(hi.w) + sj;
                    lo = make_float4(fminf(lo.x, c.x), fminf(lo.y, c.y), fminf(lo.z, c.z), __uint_as_float(id));
                    hi = make_float4(fmaxf(hi.x, c.w), fmaxf(hi.y, d.x), fmaxf(hi.z, d.y), __uint_as_float(size));
                    ploc_write_node(a, id, ri, rj, lo, hi, size);
                }
            }
            if (pos < count) {  // always, unless a look-back gave up
                cout[2 * pos] = lo;
                cout[2 * pos + 1] = hi;
            }
        }
        if (gridDim.x >= tiles) return;  // a block for each tile: no further one to ask for
        __syncthreads();                 // the next tile reuses the shared arrays
    }
}

// What the grid-wide rounds have left above kPlocSmall clusters: neighbour
// pairs, pairs of pairs and so on until kPlocSmall remain, in one grid-wide
// launch.  A block takes 2^k consecutive clusters, 2^k the least that leaves
// kPlocSmall groups, and merges them level by level in their own places; a
// merge's node id follows from its level and position, so the tree is the one
// that whole levels would give.  Almost always there is nothing to do: the
// rounds are enough for any mesh whose clusters merge at about the rates below,
// and a mesh for which they are not (every cluster's nearest neighbour has a
// nearer one, round after round: nested shells, each around the last) still
// takes one pass over its clusters instead of many by one block.
constexpr uint32_t kPlocPairThreads = 256;
constexpr uint32_t kPlocPairBlocks = 152 * 2;
__global__ void __launch_bounds__(kPlocPairThreads) k_ploc_pairs(const __grid_constant__ PlocArgs a, int round) {
    after_previous();
    BuildState* st = a.st;
    const uint32_t word = st->ploc_round[round], count = word & kPlocCount;
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    if (count <= kPlocSmall) {
        if (first) st->ploc_round[round + 1] = word;
        return;
    }
    float4* cin = a.cbox[(word & kPlocParity) ? 1 : 0];
    float4* cout = a.cbox[(word & kPlocParity) ? 0 : 1];
    const uint32_t levels = 32u - (uint32_t)__clz((count - 1u) / kPlocSmall);
    const uint32_t groups = (uint32_t)(((unsigned long long)count + (1ull << levels) - 1ull) >> levels);
    const uint32_t merges = st->merge_counter;
    if (first) {
        st->ploc_round[round + 1] = groups | ((word & kPlocParity) ^ kPlocParity);
        st->pair_merges = count - groups;
    }
    for (uint32_t g = blockIdx.x; g < groups; g += gridDim.x) {
        float4* c = cin + 2 * ((size_t)g << levels);  // the group's clusters
        uint32_t left = min(count - (g << levels), 1u << levels);
        for (uint32_t level = 0; level < levels; level++) {
            const uint32_t all = (count + (1u << level) - 1u) >> level;  // clusters of every group at this level
            const uint32_t claimed = merges + (count - all) + (g << (levels - 1u - level));
            const uint32_t pairs = (left + 1u) / 2u;  // the last may be one cluster alone
            float4* out = level + 1u == levels ? cout + 2 * (size_t)g : c;
            for (uint32_t base = 0; base < pairs; base += blockDim.x) {  // q is stored behind every later read
                const uint32_t q = base + threadIdx.x;
                const bool on = q < pairs, two = on && 2u * q + 1u < left;
                float4 lo, hi, l2, h2;
                if (on) {
                    lo = c[4 * (size_t)q];
                    hi = c[4 * (size_t)q + 1];
                }
                if (two) {
                    l2 = c[4 * (size_t)q + 2];
                    h2 = c[4 * (size_t)q + 3];
                }
                __syncthreads();
                if (two) {
                    const uint32_t claim = claimed + q;
                    const uint32_t ra = __float_as_uint(lo.w), rb = __float_as_uint(l2.w);
                    const uint32_t size = __float_as_uint(hi.w) + __float_as_uint(h2.w);
                    if (claim + 2u <= a.n) {
                        const uint32_t id = a.n - 2u - claim;
                        lo = make_float4(fminf(lo.x, l2.x), fminf(lo.y, l2.y), fminf(lo.z, l2.z), __uint_as_float(id));
                        hi = make_float4(fmaxf(hi.x, h2.x), fmaxf(hi.y, h2.y), fmaxf(hi.z, h2.z), __uint_as_float(size));
                        ploc_write_node(a, id, ra, rb, lo, hi, size);
                    } else {  // more merges than a binary tree over n primitives has
                        atomicOr(&st->error, 1u << RT_ERR_BAD_AS);
                    }
                }
                if (on) {
                    out[2 * (size_t)q] = lo;
                    out[2 * (size_t)q + 1] = hi;
                }
                __syncthreads();
            }
            left = pairs;
        }
    }
}

// The last rounds, in one CTA with every cluster (at most kPlocSmall, one
// per thread) in shared memory; node ids follow from the round's prefix sums.
// The areas of the pairs (i, i + 1..R) are computed once each: warp w takes
// 32 clusters and every S-th offset, S = 1..16 the warps there are per 32
// clusters, and the other warps only meet at the barriers.  Bound: issue of
// one SM for the first rounds, then four barriers and the shared-memory
// latency between them, about 1 us a round.  Meshes with fans of slivers (the
// poles of a sphere) take many rounds: 163,840 triangles 75, 4,096 triangles
// 40.  (With both directions evaluated by every thread of the block in each
// round, the tail of those took 535 and 290 us.)  A tail of 51 us: issue 46 %,
// 7.9 of the warps' 16 cycles per issue at a barrier.
struct PlocTailShared {
    float4 s0[kPlocSmall + kPlocRadius];  // lo, hi.x; behind the last cluster, boxes of infinite area
    float2 s1[kPlocSmall + kPlocRadius];  // hi.y, hi.z
    uint2 ref[kPlocSmall];                // binary reference, primitives below
    uint32_t near_area[kPlocSmall];       // nearest neighbours
    int8_t near_offset[kPlocSmall];
    uint32_t take[kPlocSmall];            // the asker a position takes
    uint32_t area[kPlocRadius][kPlocSmall];  // area[o - 1][i] = area of the pair (i, i + o), its bits
    uint32_t warp_sums[32];
};
// Rounds until one of the `count` clusters in s is left; returns the merges
// so far.  write_node(id, a, b, lo, hi, size) stores an internal node.
template <class W>
__device__ __forceinline__ uint32_t ploc_tail_rounds(PlocTailShared& s, uint32_t count, uint32_t merges, uint32_t n,
                                                     uint32_t* error, W write_node) {
    constexpr int R = kPlocRadius;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const PlocNear nearest{s.near_area, s.near_offset};
    bool forced = false;
    const float inf = INFINITY;
    if (tid < (uint32_t)R) {
        s.s0[count + tid] = make_float4(inf, inf, inf, inf);
        s.s1[count + tid] = make_float2(inf, inf);
    }
    __syncthreads();
    while (count > 1u) {  // a round after one with next to no merges merges pairs: it ends
        const uint32_t blocks = (count + 31u) >> 5;  // of 32 clusters
        if (!forced) {
            const int lg = min(4, 31 - __clz(32u / blocks));  // log2 S
            const uint32_t b = warp >> lg;
            if (b < blocks) {
                const uint32_t i = b * 32u + lane;
                const float4 p = s.s0[i];
                const float2 q = s.s1[i];
                const uint32_t step = 1u << lg;
#pragma unroll 4
                for (uint32_t o = 1u + (warp & (step - 1u)); o <= (uint32_t)R; o += step) {
                    const float4 u = s.s0[i + o];
                    const float2 v = s.s1[i + o];
                    s.area[o - 1u][i] =
                        __float_as_uint(merged_half_area(p.x, p.y, p.z, p.w, q.x, q.y, u.x, u.y, u.z, u.w, v.x, v.y));
                }
            }
        }
        __syncthreads();
        const bool here = tid < count;
        if (here) {
            PlocBest best;
            if (!forced) best = ploc_nearest(s.area, (int)tid);
            else best.area = 0u, best.offset = (tid ^ 1u) < count ? (int)(tid ^ 1u) - (int)tid : 0;
            ploc_store(s.near_area, s.near_offset, (int)tid, best);
            s.take[tid] = 0xFFFFFFFFu;
        }
        __syncthreads();
        int near = (int)tid;
        bool mutual = false;
        if (here) {
            near = nearest((int)tid);
            mutual = near != (int)tid && nearest(near) == (int)tid;
            if (near != (int)tid && !mutual && (tid & 1u) && !(near & 1)) ploc_ask(nearest, s.take, (int)tid, near);
        }
        __syncthreads();
        bool keep = false, merge = false;
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
        float2 q = make_float2(0.f, 0.f);
        uint2 r = make_uint2(0u, 0u);
        uint32_t partner = 0u;
        if (here) {
            const uint32_t j = (uint32_t)ploc_partner(nearest, s.take, (int)tid, near, mutual, (tid & 1u) != 0u);
            merge = j > tid;  // tid itself: no merge
            keep = j >= tid;
            p = s.s0[tid];
            q = s.s1[tid];
            r = s.ref[tid];
            if (merge) {
                const float4 u = s.s0[j];
                const float2 v = s.s1[j];
                const uint2 o = s.ref[j];
                p = make_float4(fminf(p.x, u.x), fminf(p.y, u.y), fminf(p.z, u.z), fmaxf(p.w, u.w));
                q = make_float2(fmaxf(q.x, v.x), fmaxf(q.y, v.y));
                r.y += o.y;
                partner = o.x;
            }
        }
        const unsigned kb = __ballot_sync(0xFFFFFFFFu, keep), mb = __ballot_sync(0xFFFFFFFFu, merge);
        if (lane == 0) s.warp_sums[warp] = (uint32_t)__popc(kb) | ((uint32_t)__popc(mb) << 16);
        __syncthreads();  // every old cluster has been read
        const uint32_t sum = s.warp_sums[lane];
        const uint32_t total = __reduce_add_sync(0xFFFFFFFFu, sum);
        if (tid < blocks * 32u) {
            const uint32_t before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? sum : 0u);
            const uint32_t lt = (1u << lane) - 1u;
            if (merge) {
                const uint32_t claim = merges + (before >> 16) + (uint32_t)__popc(mb & lt);
                if (claim + 2u <= n) {
                    const uint32_t id = n - 2u - claim;
                    write_node(id, r.x, partner, make_float4(p.x, p.y, p.z, 0.f),
                               make_float4(p.w, q.x, q.y, 0.f), r.y);
                    r.x = id;
                } else {
                    atomicOr(error, 1u << RT_ERR_BAD_AS);
                }
            }
            if (keep) {
                const uint32_t pos = (before & 0xFFFFu) + (uint32_t)__popc(kb & lt);
                s.s0[pos] = p;
                s.s1[pos] = q;
                s.ref[pos] = r;
            }
        }
        merges += total >> 16;
        forced = (total & 0xFFFFu) > count - 1u - count / 32u;
        count = total & 0xFFFFu;
        if (tid < (uint32_t)R) {
            s.s0[count + tid] = make_float4(inf, inf, inf, inf);
            s.s1[count + tid] = make_float2(inf, inf);
        }
        __syncthreads();
    }
    return merges;
}
__global__ void __launch_bounds__(kPlocSmall) k_ploc_tail(const __grid_constant__ PlocArgs a, int round) {
    after_previous();
    extern __shared__ float4 ploc_smem[];
    PlocTailShared& s = *reinterpret_cast<PlocTailShared*>(ploc_smem);
    BuildState* st = a.st;
    const uint32_t tid = threadIdx.x;
    const uint32_t word = st->ploc_round[round];
    const uint32_t count = word & kPlocCount;
    uint32_t merges = st->merge_counter + st->pair_merges;
    const float4* c = a.cbox[(word & kPlocParity) ? 1 : 0];
    if (count == 0u || count > kPlocSmall) {  // neither ever leaves the rounds and k_ploc_pairs
        if (tid == 0) atomicOr(&st->error, 1u << RT_ERR_BAD_AS);
        return;
    }
    if (tid < count) {
        float4 lo, hi;
        if (round == 0) {  // no grid-wide round: gather the primitives here
            const size_t p = a.vals[tid];
            lo = a.boxes[2 * p];
            hi = a.boxes[2 * p + 1];
            a.sboxes[2 * (size_t)tid] = lo;
            a.sboxes[2 * (size_t)tid + 1] = hi;
            lo.w = __uint_as_float(kLeafBit | tid);
            hi.w = __uint_as_float(1u);
        } else {
            lo = __ldcg(&c[2 * (size_t)tid]);
            hi = __ldcg(&c[2 * (size_t)tid + 1]);
        }
        s.s0[tid] = make_float4(lo.x, lo.y, lo.z, hi.x);
        s.s1[tid] = make_float2(hi.y, hi.z);
        s.ref[tid] = make_uint2(__float_as_uint(lo.w), __float_as_uint(hi.w));
    }
    __syncthreads();
    merges = ploc_tail_rounds(s, count, merges, a.n, &st->error, [&](uint32_t id, uint32_t ra, uint32_t rb, float4 lo,
                                                                     float4 hi, uint32_t size) {
        ploc_write_node(a, id, ra, rb, lo, hi, size);
    });
    if (tid == 0) st->merge_counter = merges;
}

// ---- collapse to 8-wide -------------------------------------------------------
// One launch.  A task is a binary node that becomes a wide node: it takes its
// binary children and repeatedly opens the child of largest surface area
// until it has `width` children or none can open; a subtree of <= leaf_max
// primitives is a leaf.  Tasks are queued by wide-node slot: eight lanes (one
// per child) take the next slot from a ticket counter, wait until its task
// has been written, and write the tasks of their internal children to slots
// they claim from the node counter, so the children of a node are neighbours.
// A task is one 64-bit word (binary node, first primitive position, depth),
// so nothing else has to be ordered between the lanes that write and read it.
// A slot is only ever waited for by running warps and written by the owner of
// a lower slot, which is running too; the launch ends when every primitive is
// in a leaf (the count travels with the node counter), and every wait is
// bounded.  Bound: latency, about seven dependent loads per level for small
// structures; gathers of binary nodes for large ones (2.6M triangles, 215 us:
// 20.6 cycles per issue on global loads, L2 hits 30 %, DRAM 16 %, issue 28 %).  (One launch per level
// with one thread per task, 15-40 us a level: 163,840 triangles 340 -> 80 us,
// 10,485,760 triangles 1.3 -> 0.92 ms.)
struct CollapseCtx {
    const uint4* inodes;
    const float4* iboxes;  // (lo, primitives below as bits), (hi, -) of each internal node
    const float4* sboxes;
    WideNode* nodes;
    uint32_t* parents;   // may be null
    BuildState* st;
    unsigned long long* tasks;  // one word per wide node, zeroed
    uint32_t* perm;          // final primitive order: position -> Morton-sorted position
    uint32_t leaf_max;
    uint32_t width;      // children per node: 8, or 4 (RT_BUILD_EXT_NODE_WIDTH_4)
    uint32_t max_nodes;
    uint32_t n;          // primitives
};
static_assert(kBlasLeafMax <= 2 && kTlasLeafMax <= 2, "a leaf child is one primitive or a pair");
constexpr int kCollapseThreads = 128;
constexpr uint32_t kCollapseBlocks = 152 * 8;
constexpr uint32_t kCollapseSpinLimit = 1u << 22;

__device__ __forceinline__ float half_area(float4 lo, float4 hi) {
    float dx = fmaxf(hi.x - lo.x, 0.0f), dy = fmaxf(hi.y - lo.y, 0.0f), dz = fmaxf(hi.z - lo.z, 0.0f);
    return dx * dy + dy * dz + dz * dx;
}
// A binary reference is in range: leaf < n, internal < n - 1.
__device__ __forceinline__ bool ref_ok(const CollapseCtx& c, uint32_t r) {
    return (r & kLeafBit) ? ((r & ~kLeafBit) < c.n) : (r + 1u < c.n);
}
__device__ __forceinline__ unsigned long long collapse_task(uint32_t bref, uint32_t first, uint32_t depth) {
    return (unsigned long long)bref | ((unsigned long long)first << 28) | ((unsigned long long)(min(depth, 254u) + 1u) << 56);
}

// Child slot `k` of a wide node.  r = its traversal entry, meta = its kind.
__device__ __forceinline__ void write_child(WideNode* nd, uint32_t k, float4 lo, float4 hi, uint32_t entry, bool used) {
    const float z = 0.0f;
    nd->lox[k] = used ? lo.x : z;
    nd->hix[k] = used ? hi.x : z;
    nd->loy[k] = used ? lo.y : z;
    nd->hiy[k] = used ? hi.y : z;
    nd->loz[k] = used ? lo.z : z;
    nd->hiz[k] = used ? hi.z : z;
    nd->child_ref[k] = used ? entry : kChildEmpty;
}

// The root of a structure of n <= leaf_max primitives (n may be 0): one leaf, or no child.
__device__ void write_single_leaf(const CollapseCtx& c) {
    if (c.parents) c.parents[0] = kNone;
    const float4 lo = make_float4(o2f(c.st->bb[0]), o2f(c.st->bb[1]), o2f(c.st->bb[2]), 0.0f);
    const float4 hi = make_float4(o2f(c.st->bb[3]), o2f(c.st->bb[4]), o2f(c.st->bb[5]), 0.0f);
    for (uint32_t k = 0; k < 8; k++)
        write_child(&c.nodes[0], k, lo, hi, kChildLeaf | ((c.n - 1u) << 28), k == 0 && c.n > 0);
    c.nodes[0].meta[0] = c.n;
    c.nodes[0].meta[1] = 0;
    for (int k = 0; k < 6; k++) c.nodes[0]._pad[k] = 0;
    for (uint32_t i = 0; i < c.n; i++) c.perm[i] = i;
}

// Words that other lanes write while this one waits: in the memory of the GPU,
// or (SHARED) in the shared memory of a build that one block does alone.
template <bool SHARED, class T>
__device__ __forceinline__ T queue_load(const T* p) {
    if constexpr (SHARED) return *const_cast<const volatile T*>(p);
    else if constexpr (sizeof(T) == 8) return ld_relaxed64(p);
    else return ld_relaxed(p);
}
template <bool SHARED, class T>
__device__ __forceinline__ void queue_store(T* p, T v) {
    if constexpr (SHARED) *const_cast<volatile T*>(p) = v;
    else if constexpr (sizeof(T) == 8) st_relaxed64(p, v);
    else st_relaxed(p, v);
}

// Works on tasks until every primitive is in a leaf (n > leaf_max; all lanes of the warp).
template <bool SHARED>
__device__ __forceinline__ void collapse_loop(const CollapseCtx& c) {
    const uint32_t lane = threadIdx.x & 31u, sub = lane & 7u, group = lane & 24u;
    const uint32_t lt = (1u << lane) - 1u;
    BuildState* st = c.st;
    uint32_t slot = kNone, depth_seen = 0, spins = 0, unreported = 0;  // primitives this warp has placed
    for (;;) {
        // groups without a slot take the next ones
        const unsigned want = __ballot_sync(0xFFFFFFFFu, slot == kNone && sub == 0u);
        if (want) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&st->collapse_ticket, (uint32_t)__popc(want));
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            if (slot == kNone) slot = base + (uint32_t)__popc(want & ((1u << group) - 1u));
        }
        unsigned long long task = 0;
        if (slot == 0u) task = collapse_task(0u, 0u, 0u);
        else if (slot < c.max_nodes) task = queue_load<SHARED>(&c.tasks[slot]);
        const bool ready = task != 0;
        if (!__any_sync(0xFFFFFFFFu, ready)) {
            if (unreported) {  // before waiting: the warp that reports the last ones ends the launch
                if (lane == 0) {
                    const unsigned long long before = atomicAdd(&st->progress, (unsigned long long)unreported << 32);
                    if ((uint32_t)(before >> 32) + unreported >= c.n) {
                        st->node_count = (uint32_t)before;
                        queue_store<SHARED>(&st->collapse_done, 1u);
                    }
                }
                unreported = 0;
                __syncwarp();
            }
            if (queue_load<SHARED>(&st->collapse_done)) break;
            if (++spins > kCollapseSpinLimit) {
                if (lane == 0) atomicOr(&st->error, 1u << RT_ERR_TIMEOUT);
                break;
            }
            __nanosleep(40);
            continue;
        }
        spins = 0;
        const uint32_t bref = (uint32_t)task & 0x0FFFFFFFu, first = (uint32_t)(task >> 28) & 0x0FFFFFFFu;
        const uint32_t depth = (uint32_t)(task >> 56) - 1u;
        bool bad = ready && bref + 1u >= c.n;
        uint4 top = make_uint4(0u, 0u, 0u, 0u);
        if (ready && !bad) {
            top = c.inodes[bref];
            bad = !ref_ok(c, top.x) || !ref_ok(c, top.y);
        }
        bool open = ready && !bad;  // the group may still open a child
        uint32_t cnt = open ? 2u : 0u, r = sub == 0u ? top.x : top.y, size = 0, key = 0;
        uint2 kids = make_uint2(0u, 0u);
        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
        bool load = sub < cnt;  // the lane has a new child
        for (uint32_t it = 2;; it++) {
            if (load) {
                const size_t x = r & ~kLeafBit;
                if (r & kLeafBit) {
                    lo = c.sboxes[2 * x];
                    hi = c.sboxes[2 * x + 1];
                    size = 1u;
                    key = 0u;
                } else {
                    lo = c.iboxes[2 * x];
                    hi = c.iboxes[2 * x + 1];
                    const uint4 nd = c.inodes[x];
                    kids = make_uint2(nd.x, nd.y);
                    size = __float_as_uint(lo.w);
                    const float a = half_area(lo, hi);
                    // 0: cannot be opened (small enough for a leaf, or a NaN area)
                    key = size > c.leaf_max && a >= 0.0f ? __float_as_uint(a) + 1u : 0u;
                }
            }
            if (it >= c.width) break;
            // open the child of largest area, the first of equals
            uint32_t m = open ? key : 0u;
            m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, 1));
            m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, 2));
            m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, 4));
            open = open && m != 0u;
            const unsigned at = __ballot_sync(0xFFFFFFFFu, open && key == m);
            if (!at) break;
            const uint32_t best = open ? (uint32_t)__ffs((at >> group) & 0xFFu) - 1u : 0u;
            const uint32_t kx = __shfl_sync(0xFFFFFFFFu, kids.x, (int)best, 8);
            const uint32_t ky = __shfl_sync(0xFFFFFFFFu, kids.y, (int)best, 8);
            load = false;
            if (open) {
                if (!ref_ok(c, kx) || !ref_ok(c, ky)) {
                    bad = true;
                    open = false;
                } else {
                    load = sub == best || sub == cnt;
                    if (sub == best) r = kx;
                    if (sub == cnt) r = ky;
                    cnt++;
                }
            }
        }
        if (bad) {  // malformed hierarchy: an empty node, its primitives given up
            cnt = 0;
            if (sub == 0u) atomicOr(&st->error, 1u << RT_ERR_BAD_AS);
        }
        // the children's primitives follow each other in slot order
        const bool child = sub < cnt;
        uint32_t at = child ? size : 0u;
        for (uint32_t off = 1; off < 8; off <<= 1) {
            const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, at, off, 8);
            if (sub >= off) at += o;
        }
        at += first - (child ? size : 0u);
        const bool leaf = child && ((r & kLeafBit) || size <= c.leaf_max), inner = child && !leaf;
        const unsigned inners = __ballot_sync(0xFFFFFFFFu, inner);
        uint32_t placed = leaf ? size : 0u;
        if (bad && sub == 0u) placed = bref + 1u < c.n ? __float_as_uint(c.iboxes[2 * (size_t)bref].w) : c.n;
        // Every warp adds to one counter: placed primitives are kept until the
        // warp has nothing to do, and an iteration without internal children
        // (most of them: the lowest nodes) leaves it alone.
        unreported += __reduce_add_sync(0xFFFFFFFFu, placed);
        uint32_t cs = 0;
        if (inners) {
            if (lane == 0) cs = (uint32_t)atomicAdd(&st->progress, (unsigned long long)__popc(inners));
            cs = __shfl_sync(0xFFFFFFFFu, cs, 0) + (uint32_t)__popc(inners & lt);
        }
        bool used = child;
        uint32_t meta = 0, entry = 0;
        if (inner) {
            meta = kMetaInternal;
            entry = cs;
            if (cs >= c.max_nodes) {  // more nodes than any hierarchy of n primitives has: give up
                atomicOr(&st->error, 1u << RT_ERR_TOO_LARGE);
                queue_store<SHARED>(&st->collapse_done, 1u);
                used = false;
            } else {
                if (c.parents) c.parents[cs] = slot;
                queue_store<SHARED>(&c.tasks[cs], collapse_task(r, at, depth + 1u));
            }
        } else if (leaf) {
            meta = size;
            entry = kChildLeaf | ((size - 1u) << 28) | at;
            if (at + size > c.n || size == 0u) {
                atomicOr(&st->error, 1u << RT_ERR_BAD_AS);
                used = false;
            } else if (r & kLeafBit) {
                c.perm[at] = r & ~kLeafBit;
            } else if ((kids.x & kids.y & kLeafBit) && size == 2u) {
                c.perm[at] = kids.x & ~kLeafBit;
                c.perm[at + 1u] = kids.y & ~kLeafBit;
            } else {
                atomicOr(&st->error, 1u << RT_ERR_BAD_AS);
                used = false;
            }
        }
        // meta bytes of children 0-3 and 4-7
        uint32_t mw = (used ? meta : 0u) << (8u * (sub & 3u));
        mw |= __shfl_xor_sync(0xFFFFFFFFu, mw, 1);
        mw |= __shfl_xor_sync(0xFFFFFFFFu, mw, 2);
        const uint32_t m1 = __shfl_sync(0xFFFFFFFFu, mw, 4, 8);
        if (ready) {
            WideNode* nd = &c.nodes[slot];
            write_child(nd, sub, lo, hi, entry, used);
            // the words after child_ref: meta[0], meta[1], six of padding
            reinterpret_cast<uint32_t*>(nd)[56 + sub] = sub == 0u ? mw : (sub == 1u ? m1 : 0u);
            if (slot == 0u && sub == 0u && c.parents) c.parents[0] = kNone;
            depth_seen = max(depth_seen, depth + 1u);
            slot = kNone;
        }
    }
    depth_seen = __reduce_max_sync(0xFFFFFFFFu, depth_seen);
    if (lane == 0 && depth_seen > 1u) atomicMax(&st->depth, depth_seen);
}

__global__ void __launch_bounds__(kCollapseThreads, 8) k_collapse(const __grid_constant__ CollapseCtx c) {
    after_previous();
    if (c.n > c.leaf_max) collapse_loop<false>(c);
    else if (blockIdx.x == 0 && threadIdx.x == 0) write_single_leaf(c);
}

// ---- primitive records ----------------------------------------------------------
// As k_blas_prims, at most kPrimBlocks blocks: each ends with 15 atomics on
// the same lines (615,000 of them for 10.5M triangles before).
__global__ void k_write_tris(const __grid_constant__ BlasInput in, const uint32_t* vals, const uint32_t* perm,
                             TriRecord* tris, BuildState* st) {
    after_previous();
    // the bounding sphere's radius and the 14-DOP's extreme projections (sums of
    // +-coordinates, rounded up for the maxima and down for the minima) over
    // the triangles that have a box (finite vertices)
    uint32_t rb = 0, dh[7], dl[7];
#pragma unroll
    for (int k = 0; k < 7; k++) {
        dh[k] = 0u;
        dl[k] = 0xFFFFFFFFu;
    }
    const float centre[3] = {bounds_center(st, 0), bounds_center(st, 1), bounds_center(st, 2)};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < in.n; i += gridDim.x * blockDim.x) {
        const uint32_t p = vals[min(perm[i], in.n - 1u)];
        int g = 0;
        uint32_t prim = 0;
        float v[3][3];
        if (fetch_triangle(in, p, &g, &prim, v)) {
            // an overflow (+inf) turns the sphere off
            rb = max(rb, __float_as_uint(fmaxf(fmaxf(distance_ru(v[0], centre), distance_ru(v[1], centre)),
                                               distance_ru(v[2], centre))));
#pragma unroll
            for (int k = 0; k < 7; k++) {
                float ph = -INFINITY, pl = INFINITY;
                for (int c = 0; c < 3; c++) {
                    float u = 0.0f, d = 0.0f;
                    for (int a = 0; a < 3; a++) {
                        const float x = kDopAxis[k][a] > 0 ? v[c][a] : (kDopAxis[k][a] < 0 ? -v[c][a] : 0.0f);
                        u = __fadd_ru(u, x);
                        d = __fadd_rd(d, x);
                    }
                    ph = fmaxf(ph, u);
                    pl = fminf(pl, d);
                }
                dh[k] = max(dh[k], f2o(ph));
                dl[k] = min(dl[k], f2o(pl));
            }
        } else {
            float qn = __int_as_float(0x7FC00000);
            for (int c = 0; c < 3; c++) v[c][0] = v[c][1] = v[c][2] = qn;
        }
        uint32_t flags = (in.g[g].flags & RT_GEOMETRY_OPAQUE) ? 1u : 0u;
        TriRecord r;
        r.v0 = make_float4(v[0][0], v[0][1], v[0][2], __uint_as_float(prim));
        r.v1 = make_float4(v[1][0], v[1][1], v[1][2], __uint_as_float((uint32_t)g));
        r.v2 = make_float4(v[2][0], v[2][1], v[2][2], __uint_as_float(flags));
        tris[i] = r;
    }
    // reduced over the warp, then over the block, and each block makes one atomic per value
    __shared__ uint32_t red[32][15];  // [warp][radius, 7 maxima, 7 minima]
    const uint32_t w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    const bool leader = (threadIdx.x & 31u) == 0u;
    rb = __reduce_max_sync(0xFFFFFFFFu, rb);
    if (leader) red[w][0] = rb;
#pragma unroll
    for (int k = 0; k < 7; k++) {
        const uint32_t hi = __reduce_max_sync(0xFFFFFFFFu, dh[k]), lo = __reduce_min_sync(0xFFFFFFFFu, dl[k]);
        if (leader) {
            red[w][1 + k] = hi;
            red[w][8 + k] = lo;
        }
    }
    __syncthreads();
    if (threadIdx.x < 15) {
        const int k = threadIdx.x;
        uint32_t r = red[0][k];
        for (uint32_t j = 1; j < nw; j++) r = k < 8 ? max(r, red[j][k]) : min(r, red[j][k]);
        if (k == 0) {
            if (r) atomicMax(&st->radius_bits, r);
        } else if (k < 8) {
            if (r != 0u) atomicMax(&st->dop_hi[k - 1], r);  // 0: no valid triangle in the block
        } else if (r != 0xFFFFFFFFu) {
            atomicMin(&st->dop_lo[k - 8], r);
        }
    }
}

__global__ void k_write_insts(const InstRecord* temp, const uint32_t* vals, const uint32_t* perm, uint32_t n,
                              InstRecord* out) {
    after_previous();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = temp[vals[min(perm[i], n - 1u)]];
}

// ---- 8-bit quantised nodes ----------------------------------------------------
// Smallest biased exponent e (quantum s = 2^(e-127)) with ext <= 252 s and
// |floor(L / s)| + 512 < 2^24, so that the grid origin (floor(L/s) - 1) s and
// every decoded plane origin + q s (q <= 255) are exact floats.
// e_floor keeps a thin axis's quantum at least 2^-24 of the node's largest
// extent: a flat node (a ground plane's, zero extent on one axis) would
// otherwise get the smallest quantum there, whose scale times any ray's
// inverse direction falls below the fast test's range, and every ray would
// take the exact decode.  The box grows by a quarter of that quantum at most.
__device__ uint32_t quantum_exponent(float L, float ext, uint32_t e_floor) {
    uint32_t e = (__float_as_uint(ext / 252.0f) >> 23) & 0xFFu;
    uint32_t el = (__float_as_uint(fabsf(L)) >> 23) & 0xFFu;
    e = max(e, el > 23u ? el - 23u : 1u);
    e = max(e, e_floor);
    if (e < 1u) e = 1u;
    for (; e < 254u; e++) {
        float s = __uint_as_float(e << 23);
        if (ext > 252.0f * s) continue;
        float k = floorf(L / s);
        if (!(fabsf(k) < 16776704.0f)) continue;
        return e;
    }
    return 254u;
}

__global__ void k_quantize_nodes(const WideNode* in, const BuildState* st, uint32_t max_nodes, QNode* out) {
    after_previous();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t count = min(st->node_count, max_nodes);
    if (i >= count) return;
    const WideNode& nd = in[i];
    QNode q;
    float lo[3][8], hi[3][8];
    bool valid[8];
    float L[3] = {INFINITY, INFINITY, INFINITY}, H[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int k = 0; k < 8; k++) {
        q.child_ref[k] = nd.child_ref[k];
        lo[0][k] = nd.lox[k]; lo[1][k] = nd.loy[k]; lo[2][k] = nd.loz[k];
        hi[0][k] = nd.hix[k]; hi[1][k] = nd.hiy[k]; hi[2][k] = nd.hiz[k];
        valid[k] = nd.child_ref[k] != kChildEmpty;
        for (int a = 0; a < 3; a++) valid[k] = valid[k] && lo[a][k] <= hi[a][k] && fabsf(lo[a][k]) <= FLT_MAX &&
                                               fabsf(hi[a][k]) <= FLT_MAX;
        if (!valid[k]) continue;
        for (int a = 0; a < 3; a++) {
            L[a] = fminf(L[a], lo[a][k]);
            H[a] = fmaxf(H[a], hi[a][k]);
        }
    }
    uint8_t* qlo[3] = {q.qlo_x, q.qlo_y, q.qlo_z};
    uint8_t* qhi[3] = {q.qhi_x, q.qhi_y, q.qhi_z};
    float mext = 0.0f;  // the node's largest extent
    for (int a = 0; a < 3; a++)
        if (L[a] <= H[a]) mext = fmaxf(mext, __fsub_ru(H[a], L[a]));
    const uint32_t em = (__float_as_uint(mext) >> 23) & 0xFFu;
    const uint32_t e_floor = em > 24u ? em - 24u : 1u;
    for (int a = 0; a < 3; a++) {
        if (!(L[a] <= H[a])) {  // no valid child: any grid, every child empty
            q.origin[a] = 0.0f;
            q.exp[a] = 127u;
            for (int k = 0; k < 8; k++) { qlo[a][k] = 255u; qhi[a][k] = 0u; }
            continue;
        }
        float ext = __fsub_ru(H[a], L[a]);
        uint32_t e = quantum_exponent(L[a], ext, e_floor);
        float s = __uint_as_float(e << 23);
        float origin = (floorf(L[a] / s) - 1.0f) * s;
        q.origin[a] = origin;
        q.exp[a] = (uint8_t)e;
        for (int k = 0; k < 8; k++) {
            if (!valid[k]) { qlo[a][k] = 255u; qhi[a][k] = 0u; continue; }
            // outward to the grid with at least kQuantSlack of a quantum to
            // spare on each side (origin + ql s <= lo - slack s); the
            // division by the power of two s is exact
            float ql = floorf(__fsub_rd(__fsub_rd(lo[a][k], origin) / s, kQuantSlack));
            float qh = ceilf(__fadd_ru(__fsub_ru(hi[a][k], origin) / s, kQuantSlack));
            qlo[a][k] = (uint8_t)fminf(fmaxf(ql, 0.0f), 255.0f);
            qhi[a][k] = (uint8_t)fminf(fmaxf(qh, 0.0f), 255.0f);
        }
    }
    q._pad = 0;
    const uint4* src = reinterpret_cast<const uint4*>(&q);
    uint4* dst = reinterpret_cast<uint4*>(&out[i]);
    for (int w = 0; w < 6; w++) dst[w] = src[w];
}

// ---- header ---------------------------------------------------------------------
struct HeaderStatic {
    uint32_t type, build_flags, prim_count, max_nodes, geometry_count, leaf_max, node_bytes;
    uint64_t total_size, nodes_offset, prims_offset, parents_offset;
    uint64_t prim_bytes;
};

// The header of a finished build, without a 14-DOP (one thread).
__device__ void write_header(AsHeader* h, const BuildState* st, const HeaderStatic& hs) {
    h->magic = kAsMagic;
    h->type = hs.type;
    h->build_flags = hs.build_flags;
    uint32_t err = st->error;
    h->status = err >> 1 ? (uint32_t)__ffs(err >> 1) : (uint32_t)RT_OK;  // the lowest RT_ERR_* bit
    uint32_t nc = st->node_count;
    if (nc > hs.max_nodes) nc = hs.max_nodes;
    h->node_count = nc;
    h->prim_count = hs.prim_count;
    h->max_nodes = hs.max_nodes;
    h->node_bytes = hs.node_bytes;
    h->total_size = hs.total_size;
    h->nodes_offset = hs.nodes_offset;
    h->prims_offset = hs.prims_offset;
    h->parents_offset = hs.parents_offset;
    for (int k = 0; k < 3; k++) {
        float lo = o2f(st->bb[k]), hi = o2f(st->bb[3 + k]);
        if (hs.prim_count == 0 || !(lo <= hi)) {
            lo = INFINITY;
            hi = -INFINITY;
        }
        h->bounds_lo[k] = lo;
        h->bounds_hi[k] = hi;
    }
    h->geometry_count = hs.geometry_count;
    h->depth = st->depth;
    h->leaf_max = hs.leaf_max;
    h->blas_kinds = hs.type == kAsTypeTop ? st->blas_kinds : 0u;
    // the sphere is written only where every triangle's distance was taken
    const float rad = __uint_as_float(st->radius_bits);
    const bool sphere = hs.type == kAsTypeBottom && hs.prim_count > 0 && st->radius_bits != 0u && rad <= FLT_MAX;
    for (int k = 0; k < 3; k++) h->sphere_center[k] = sphere ? bounds_center(st, k) : 0.0f;
    h->sphere_radius = sphere ? __fmul_ru(rad, 1.0000010f) : 0.0f;
    h->dop_count = 0;
    uint64_t nodes_end = hs.nodes_offset + (uint64_t)nc * hs.node_bytes;
    uint64_t par = hs.parents_offset ? align_up(nodes_end, 256) : 0;
    uint64_t par_end = par ? par + (uint64_t)nc * 4 : nodes_end;
    h->compacted_size = align_up(align_up(par_end, 256) + hs.prim_count * hs.prim_bytes, 256);
}

// The plane triples a < b < c of the 14-DOP in lexicographic order.
struct DopTriples {
    uint8_t t[kDopTriples][4];
};
constexpr DopTriples make_dop_triples() {
    DopTriples d{};
    int n = 0;
    for (int a = 0; a < 14; a++)
        for (int b = a + 1; b < 14; b++)
            for (int c = b + 1; c < 14; c++, n++) {
                d.t[n][0] = (uint8_t)a;
                d.t[n][1] = (uint8_t)b;
                d.t[n][2] = (uint8_t)c;
            }
    return d;
}
__device__ const DopTriples kDopTriple = make_dop_triples();

// Plane j of the 14-DOP: +axis (even) or -axis (odd), and n . p <= its height.
__device__ __forceinline__ float dop_dot(int j, float x, float y, float z) {
    const int8_t* a = kDopAxis[j >> 1];
    const float d = (float)a[0] * x + (float)a[1] * y + (float)a[2] * z;
    return (j & 1) ? -d : d;
}

// The header, and for a BLAS its 14-DOP's vertices (0: none), in one block.
// Every triple of the 14 planes is solved: first in float with a tolerance of
// 1e-5 of the scale (float rounding moves the point and its projections by a
// few 1e-6 of it), which leaves the vertices and few others; those are solved
// in double and kept when the point satisfies all 14 planes (1e-9 relative).
// Points within 1e-7 of an earlier one (in triple order) are dropped, again
// screened in float.  This part's double precision runs at two operations per
// clock and SM: with all 364 triples in double over three blocks the vertices
// took 28 us and the header another launch of 4 us; together 11.5 us now.  More than kDopMaxVertices
// distinct points (only through rounding) or a non-finite projection leave
// the header's dop_count at 0.  The vertices' float rounding (a few 1e-8
// relative) is covered by the instance box padding (1e-5 relative).
constexpr int kFinishThreads = 384;
static_assert(kFinishThreads >= kDopTriples, "one thread per triple");
__global__ void __launch_bounds__(kFinishThreads) k_finish(AsHeader* h, const BuildState* st,
                                                           const __grid_constant__ HeaderStatic hs) {
    after_previous();
    __shared__ float phf[14];
    __shared__ uint16_t list[kDopTriples];   // triples that pass the float screen, in order
    __shared__ double cand[kDopTriples][3];  // the points found, by place in the list
    __shared__ float candf[kDopTriples][3];
    __shared__ uint8_t found[kDopTriples];   // 1: a point of the 14-DOP; 2: and no earlier one is within the tolerance
    __shared__ uint32_t warp_sums[kFinishThreads / 32];
    __shared__ bool ok;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    const unsigned lt = (1u << lane) - 1u;
    if (t == kFinishThreads - 1) write_header(h, st, hs);
    if (hs.type != kAsTypeBottom || hs.prim_count == 0u) return;
    if (t == 0) {
        bool good = true;
        for (int k = 0; k < 7; k++) {
            const float hi = o2f(st->dop_hi[k]), lo = o2f(st->dop_lo[k]);
            if (!(lo <= hi) || !(fabsf(hi) <= FLT_MAX) || !(fabsf(lo) <= FLT_MAX)) good = false;
            phf[2 * k] = hi;
            phf[2 * k + 1] = -lo;
        }
        ok = good;
    }
    __syncthreads();  // and the header is written: its dop_count can be set below
    if (!ok) return;
    float scale_f = 0.0f;
    for (int j = 0; j < 14; j++) scale_f = fmaxf(scale_f, fabsf(phf[j]));
    const double scale = fmax(1e-30, (double)scale_f);
    bool pass = false;
    if (t < (uint32_t)kDopTriples) {
        const int a = kDopTriple.t[t][0], b = kDopTriple.t[t][1], c = kDopTriple.t[t][2];
        int A[3], B[3], C[3];
        for (int k = 0; k < 3; k++) {
            A[k] = (a & 1) ? -kDopAxis[a >> 1][k] : kDopAxis[a >> 1][k];
            B[k] = (b & 1) ? -kDopAxis[b >> 1][k] : kDopAxis[b >> 1][k];
            C[k] = (c & 1) ? -kDopAxis[c >> 1][k] : kDopAxis[c >> 1][k];
        }
        // rows of the adjugate: point = (ha (B x C) + hb (C x A) + hc (A x B)) / det
        const int bc[3] = {B[1] * C[2] - B[2] * C[1], B[2] * C[0] - B[0] * C[2], B[0] * C[1] - B[1] * C[0]};
        const int ca[3] = {C[1] * A[2] - C[2] * A[1], C[2] * A[0] - C[0] * A[2], C[0] * A[1] - C[1] * A[0]};
        const int ab[3] = {A[1] * B[2] - A[2] * B[1], A[2] * B[0] - A[0] * B[2], A[0] * B[1] - A[1] * B[0]};
        const int det = A[0] * bc[0] + A[1] * bc[1] + A[2] * bc[2];
        if (det != 0) {
            // heights / 32: no sum below can overflow, and every comparison is relative
            const float ha = phf[a] / 32.0f, hb = phf[b] / 32.0f, hc = phf[c] / 32.0f, r = 1.0f / (float)det;
            const float x = (ha * (float)bc[0] + hb * (float)ca[0] + hc * (float)ab[0]) * r;
            const float y = (ha * (float)bc[1] + hb * (float)ca[1] + hc * (float)ab[1]) * r;
            const float z = (ha * (float)bc[2] + hb * (float)ca[2] + hc * (float)ab[2]) * r;
            pass = true;
            for (int j = 0; j < 14; j++)
                pass = pass && !(dop_dot(j, x, y, z) > phf[j] / 32.0f + 3.125e-7f * scale_f + 1e-37f);
        }
    }
    // the triples that pass, in order
    const unsigned pb = __ballot_sync(0xFFFFFFFFu, pass);
    if (lane == 0) warp_sums[warp] = (uint32_t)__popc(pb);
    __syncthreads();
    uint32_t before = 0, npts = 0;
    for (uint32_t w = 0; w < kFinishThreads / 32; w++) {
        if (w < warp) before += warp_sums[w];
        npts += warp_sums[w];
    }
    if (pass) list[before + (uint32_t)__popc(pb & lt)] = (uint16_t)t;
    __syncthreads();
    for (uint32_t i = t; i < npts; i += kFinishThreads) {
        const int id = list[i];
        int P[3][3];
        double H[3];
        for (int q = 0; q < 3; q++) {
            const int a = kDopTriple.t[id][q];
            for (int k = 0; k < 3; k++) P[q][k] = (a & 1) ? -kDopAxis[a >> 1][k] : kDopAxis[a >> 1][k];
            H[q] = (double)phf[a];
        }
        // Cramer's rule on the rows A, B, C.  Their entries are 0 or +-1 and the
        // determinant is +-1, +-2 or +-4, so its reciprocal is exact and only the
        // sums below round.
        const int *A = P[0], *B = P[1], *C = P[2];
        const int det = A[0] * (B[1] * C[2] - B[2] * C[1]) - A[1] * (B[0] * C[2] - B[2] * C[0]) +
                        A[2] * (B[0] * C[1] - B[1] * C[0]);
        const double r = (double)(1.0f / (float)det);
        const double x = (H[0] * (B[1] * C[2] - B[2] * C[1]) - A[1] * (H[1] * C[2] - B[2] * H[2]) +
                          A[2] * (H[1] * C[1] - B[1] * H[2])) * r;
        const double y = (A[0] * (H[1] * C[2] - B[2] * H[2]) - H[0] * (B[0] * C[2] - B[2] * C[0]) +
                          A[2] * (B[0] * H[2] - H[1] * C[0])) * r;
        const double z = (A[0] * (B[1] * H[2] - H[1] * C[1]) - A[1] * (B[0] * H[2] - H[1] * C[0]) +
                          H[0] * (B[0] * C[1] - B[1] * C[0])) * r;
        const double slack = 1e-9 * scale;
        const double along[7] = {x, y, z, x + y + z, x + y - z, x - y + z, y - x + z};  // kDopAxis
        bool inside = true;
        for (int k = 0; k < 7; k++)
            inside = inside && along[k] <= (double)phf[2 * k] + slack && -along[k] <= (double)phf[2 * k + 1] + slack;
        cand[i][0] = x;
        cand[i][1] = y;
        cand[i][2] = z;
        candf[i][0] = (float)x;
        candf[i][1] = (float)y;
        candf[i][2] = (float)z;
        found[i] = inside ? 1 : 0;
    }
    __syncthreads();
    // A pair is a duplicate when every coordinate differs by at most 1e-7
    // scale (in double).  The float copies screen the pairs first: every
    // coordinate is within scale (1 + 1e-9) (the axis planes bound it), so
    // rounding to float moves a difference by at most 2^-23 scale, and a
    // pair whose float difference exceeds 4e-7 scale cannot pass the double
    // test.
    const double tol = 1e-7 * scale;
    const float tolf = 4e-7f * (float)scale;
    bool keep = t < npts && found[t] != 0;
    for (uint32_t j = 0; j < t && keep; j++) {
        if (!found[j] || fabsf(candf[t][0] - candf[j][0]) > tolf || fabsf(candf[t][1] - candf[j][1]) > tolf ||
            fabsf(candf[t][2] - candf[j][2]) > tolf)
            continue;
        keep = !(fabs(cand[t][0] - cand[j][0]) <= tol && fabs(cand[t][1] - cand[j][1]) <= tol &&
                 fabs(cand[t][2] - cand[j][2]) <= tol);
    }
    const unsigned kb = __ballot_sync(0xFFFFFFFFu, keep);
    if (lane == 0) warp_sums[warp] = (uint32_t)__popc(kb);
    __syncthreads();
    before = 0;
    uint32_t nv = 0;
    for (uint32_t w = 0; w < kFinishThreads / 32; w++) {
        if (w < warp) before += warp_sums[w];
        nv += warp_sums[w];
    }
    if (nv < 4u || nv > kDopMaxVertices) return;  // more points than a 14-DOP has, or too few: leave it off
    if (keep)
        for (int a = 0; a < 3; a++) h->dop_vertex[before + (uint32_t)__popc(kb & lt)][a] = candf[t][a];
    if (t == 0) h->dop_count = nv;
}

// ---- small TLAS in one block ----------------------------------------------------------
// A TLAS of 1 to 1,024 instances, one thread each: records and boxes, Morton
// sort, PLOC and the collapse in shared memory, one launch.  A frame rebuilds
// such a TLAS before it traces, and eight launches that each work on a few
// hundred instances were mostly launch and L2 latency.  Bound: latency, the
// rounds of the clustering first.  (17 instances 117 -> 33 us,
// 256 instances 190 -> 66 us.)  Above 1,024 the grid-wide path takes over, with
// its first round on more than one SM.  The block needs an SM of its own; behind
// a query of another stream that fills the GPU it is done 1,019 us (256
// instances 1,045) after it was queued, the eight launches were after 1,105
// (1,170): they waited for the same SMs to drain.
constexpr uint32_t kTlasSmall = 1024;
static_assert(kTlasSmall == kPlocSmall && kTlasSmall == kSortThreads, "one thread per instance");
struct TlasSmallArgs {
    const RtAccelerationStructureInstance* inst;
    InstRecord* temp;      // records in caller order (scratch)
    AsHeader* header;
    WideNode* nodes;
    uint32_t* parents;
    InstRecord* out;
    uint32_t n, width, max_nodes;
};
struct TlasSmallShared {
    BuildState st;
    union {
        struct {
            uint32_t sort[(256 * kSortRow + 2 * kTlasSmall)];
            float4 boxes[2 * kTlasSmall];  // in caller order
        };
        PlocTailShared ploc;
        unsigned long long tasks[kTlasSmall + 2];
    };
    uint32_t vals[kTlasSmall], perm[kTlasSmall];
    float4 sboxes[2 * kTlasSmall], iboxes[2 * kTlasSmall];
    uint4 inodes[kTlasSmall];
    uint32_t warp_sums[32];
};
__global__ void __launch_bounds__(kTlasSmall) k_tlas_small(const __grid_constant__ TlasSmallArgs a,
                                                           const __grid_constant__ HeaderStatic hs) {
    after_previous();
    extern __shared__ float4 tlas_smem[];
    TlasSmallShared& s = *reinterpret_cast<TlasSmallShared*>(tlas_smem);
    const uint32_t tid = threadIdx.x, n = a.n;
    init_state(&s.st, n);
    __syncthreads();
    float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
    tlas_prim(a.inst, tid, n, a.temp, &s.st, lo, hi);
    s.boxes[2 * tid] = lo;
    s.boxes[2 * tid + 1] = hi;
    __syncthreads();
    uint32_t key[1] = {tid < n ? morton_code(lo, hi, &s.st) : 0xFFFFFFFFu}, val[1] = {tid};
    block_sort<1>(key, val, s.sort, s.warp_sums);  // threads past n keep the last places
    if (tid < n) {
        lo = s.boxes[2 * val[0]];
        hi = s.boxes[2 * val[0] + 1];
        s.vals[tid] = val[0];
        s.sboxes[2 * tid] = lo;
        s.sboxes[2 * tid + 1] = hi;
    }
    __syncthreads();  // the boxes have been read: their place is the clusters' now
    if (tid < n) {
        s.ploc.s0[tid] = make_float4(lo.x, lo.y, lo.z, hi.x);
        s.ploc.s1[tid] = make_float2(hi.y, hi.z);
        s.ploc.ref[tid] = make_uint2(kLeafBit | tid, 1u);
    }
    __syncthreads();
    ploc_tail_rounds(s.ploc, n, 0u, n, &s.st.error, [&](uint32_t id, uint32_t ra, uint32_t rb, float4 l, float4 h,
                                                        uint32_t size) {
        s.inodes[id] = make_uint4(ra, rb, 0u, 0u);
        s.iboxes[2 * id] = make_float4(l.x, l.y, l.z, __uint_as_float(size));
        s.iboxes[2 * id + 1] = h;
    });
    for (uint32_t i = tid; i < a.max_nodes; i += kTlasSmall) s.tasks[i] = 0ull;
    __syncthreads();
    CollapseCtx c;
    c.inodes = s.inodes;
    c.iboxes = s.iboxes;
    c.sboxes = s.sboxes;
    c.nodes = a.nodes;
    c.parents = a.parents;
    c.st = &s.st;
    c.tasks = s.tasks;
    c.perm = s.perm;
    c.leaf_max = kTlasLeafMax;
    c.width = a.width;
    c.max_nodes = a.max_nodes;
    c.n = n;
    if (n <= kTlasLeafMax) {
        if (tid == 0) write_single_leaf(c);
    } else if ((tid >> 5) * 4u < a.max_nodes) {  // a warp works on four nodes
        collapse_loop<true>(c);
    }
    __syncthreads();
    if (tid == 0) write_header(a.header, &s.st, hs);
    // eight lanes copy a record (temp was written by this block)
    for (uint32_t i = tid >> 3; i < n; i += kTlasSmall / 8u) {
        const uint32_t from = s.vals[min(s.perm[i], n - 1u)];
        reinterpret_cast<uint4*>(&a.out[i])[tid & 7u] = __ldcg(reinterpret_cast<const uint4*>(&a.temp[from]) + (tid & 7u));
    }
}

// ---- TLAS refit ---------------------------------------------------------------------
__global__ void k_refit_insts(const RtAccelerationStructureInstance* inst, uint32_t n, AsHeader* h,
                              float4* sboxes, uint32_t* err) {
    after_previous();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    InstRecord* recs = reinterpret_cast<InstRecord*>(reinterpret_cast<uint8_t*>(h) + h->prims_offset);
    InstRecord rec = recs[i];
    uint32_t id = rec.instance_id;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    uint32_t kinds = 0;
    if (id < n) {
        RtAccelerationStructureInstance r = inst[id];
        if (fill_instance(r, id, &rec, lo, hi, err)) kinds = blas_kind(rec.node_count);
    } else {
        rec.tri_count = 0;
        atomicOr(err, 1u << RT_ERR_INVALID);
    }
    // the kinds only grow here: a refit may add a BLAS kind, never drop one
    const uint32_t active = __activemask();
    kinds = __reduce_or_sync(active, kinds);
    if ((threadIdx.x & 31u) == (uint32_t)(__ffs(active) - 1) && kinds) atomicOr(&h->blas_kinds, kinds);
    recs[i] = rec;
    sboxes[2 * (size_t)i] = make_float4(lo[0], lo[1], lo[2], 0.0f);
    sboxes[2 * (size_t)i + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
}

// Refit of a TLAS of up to 512 instances in one block: the records, then the
// nodes from the leaves up, eight lanes (one per child) to a node, with the
// instance boxes, the node boxes and the arrival counts in shared memory.  A
// node is done by the group that brings the last of its internal children.
// (105 instances: 48 us as a memset and three launches, 12 us now; bound
// by the latency of the instance transforms and of about four levels.)
constexpr uint32_t kRefitSmall = 512;
constexpr uint32_t kRefitNodes = kRefitSmall + 2;  // max_wide_nodes(n, 4)
__global__ void __launch_bounds__(kRefitSmall) k_refit_small(const RtAccelerationStructureInstance* inst, uint32_t n,
                                                             AsHeader* h) {
    after_previous();
    __shared__ float4 ibox[2 * kRefitSmall];
    __shared__ float nbox[kRefitNodes][6];
    __shared__ uint32_t arrived[kRefitNodes];
    __shared__ uint32_t err, kinds_seen;
    const uint32_t tid = threadIdx.x, sub = tid & 7u, group = tid & 24u;
    const unsigned gmask = 0xFFu << group;
    const uint32_t count = h->node_count, prims = h->prim_count;
    if (tid == 0) err = kinds_seen = 0u;
    for (uint32_t i = tid; i < kRefitNodes; i += kRefitSmall) arrived[i] = 0u;
    __syncthreads();
    uint8_t* base = reinterpret_cast<uint8_t*>(h);
    WideNode* nodes = reinterpret_cast<WideNode*>(base + h->nodes_offset);
    const uint32_t* parents = reinterpret_cast<const uint32_t*>(base + h->parents_offset);
    if (tid < n) {
        InstRecord* recs = reinterpret_cast<InstRecord*>(base + h->prims_offset);
        InstRecord rec;
        const uint32_t id = recs[tid].instance_id;
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        if (id < n) {
            const RtAccelerationStructureInstance r = inst[id];
            if (fill_instance(r, id, &rec, lo, hi, &err)) atomicOr(&kinds_seen, blas_kind(rec.node_count));
        } else {
            rec = recs[tid];
            rec.tri_count = 0;
            atomicOr(&err, 1u << RT_ERR_INVALID);
        }
        recs[tid] = rec;
        ibox[2 * tid] = make_float4(lo[0], lo[1], lo[2], 0.0f);
        ibox[2 * tid + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
    }
    __syncthreads();
    if (count > min(n + 2u, kRefitNodes)) {  // a TLAS of more instances than this update was given
        if (tid == 0) atomicOr(&err, 1u << RT_ERR_INVALID);
    } else {
        for (uint32_t first = tid >> 3; first < count; first += kRefitSmall / 8u) {
            uint32_t slot = first;
            bool leaf_node = true;  // climbs start at the nodes without internal children
            for (int guard = 0; guard < 64; guard++) {
                WideNode* nd = &nodes[slot];
                const uint32_t m = node_meta(nd->meta[0], nd->meta[1], (int)sub);
                const bool inner = m == kMetaInternal;
                if (leaf_node && __any_sync(gmask, inner)) break;
                leaf_node = false;
                uint32_t r = nd->child_ref[sub];
                if (m != 0u && !inner) r &= 0x0FFFFFFFu;  // leaf: first primitive
                float b[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
                if (m != 0u) {
                    if (inner ? r >= count : (m > 8u || r + m > prims || r + m > n)) {
                        atomicOr(&err, 1u << RT_ERR_BAD_AS);  // malformed child: leave its box empty
                    } else if (inner) {
                        for (int k = 0; k < 6; k++) b[k] = *const_cast<volatile float*>(&nbox[r][k]);
                    } else {
                        for (uint32_t q = 0; q < m; q++) {
                            const float4 l = ibox[2 * (r + q)], u = ibox[2 * (r + q) + 1];
                            b[0] = fminf(b[0], l.x); b[1] = fminf(b[1], l.y); b[2] = fminf(b[2], l.z);
                            b[3] = fmaxf(b[3], u.x); b[4] = fmaxf(b[4], u.y); b[5] = fmaxf(b[5], u.z);
                        }
                    }
                    nd->lox[sub] = b[0]; nd->loy[sub] = b[1]; nd->loz[sub] = b[2];
                    nd->hix[sub] = b[3]; nd->hiy[sub] = b[4]; nd->hiz[sub] = b[5];
                }
                for (int off = 1; off < 8; off <<= 1)
                    for (int k = 0; k < 6; k++) {
                        const float o = __shfl_xor_sync(gmask, b[k], off);
                        b[k] = k < 3 ? fminf(b[k], o) : fmaxf(b[k], o);
                    }
                const uint32_t p = parents[slot];
                const bool root = p == kNone || p >= count;
                uint32_t last = 0;
                if (sub == 0u) {
                    if (root) {
                        for (int k = 0; k < 3; k++) {
                            h->bounds_lo[k] = b[k];
                            h->bounds_hi[k] = b[3 + k];
                        }
                    } else {
                        for (int k = 0; k < 6; k++) *const_cast<volatile float*>(&nbox[slot][k]) = b[k];
                        __threadfence_block();
                        uint32_t need = 0;
                        for (int k = 0; k < 8; k++) need += node_meta(nodes[p].meta[0], nodes[p].meta[1], k) == kMetaInternal;
                        last = atomicAdd(&arrived[p], 1u) + 1u >= need ? 1u : 0u;
                        __threadfence_block();
                    }
                }
                last = __shfl_sync(gmask, last, (int)group);
                __syncwarp(gmask);  // the first lane has seen the children's boxes: so do the others
                if (root || !last) break;
                slot = p;
                if (guard == 63 && sub == 0u) atomicOr(&err, 1u << RT_ERR_STACK_OVERFLOW);
            }
        }
    }
    __syncthreads();
    if (tid == 0) {
        if (kinds_seen) h->blas_kinds |= kinds_seen;  // a refit may add a BLAS kind, never drop one
        if (err >> 1) h->status = (uint32_t)__ffs(err >> 1);  // the lowest RT_ERR_* bit
    }
}

__device__ __forceinline__ int internal_children(const WideNode* nd) {
    uint32_t m0 = __ldcg(&nd->meta[0]), m1 = __ldcg(&nd->meta[1]);
    int c = 0;
    for (int k = 0; k < 8; k++) c += node_meta(m0, m1, k) == kMetaInternal;
    return c;
}

__global__ void k_refit_nodes(AsHeader* h, const float4* sboxes, uint32_t* counters, uint32_t cap, uint32_t* err) {
    after_previous();
    uint32_t count = h->node_count;
    uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (count > cap) {  // a TLAS of more instances than this update was given
        if (slot == 0) atomicOr(err, 1u << RT_ERR_INVALID);
        return;
    }
    if (slot >= count) return;
    uint8_t* base = reinterpret_cast<uint8_t*>(h);
    WideNode* nodes = reinterpret_cast<WideNode*>(base + h->nodes_offset);
    const uint32_t* parents = reinterpret_cast<const uint32_t*>(base + h->parents_offset);
    if (internal_children(&nodes[slot]) != 0) return;
    for (int guard = 0; guard < 64; guard++) {
        WideNode* nd = &nodes[slot];
        uint32_t m0 = __ldcg(&nd->meta[0]), m1 = __ldcg(&nd->meta[1]);
        float ulo[3] = {INFINITY, INFINITY, INFINITY}, uhi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (int k = 0; k < 8; k++) {
            uint32_t m = node_meta(m0, m1, k);
            if (m == 0) continue;
            uint32_t r = __ldcg(&nd->child_ref[k]);
            if (m != kMetaInternal) r &= 0x0FFFFFFFu;  // leaf: first primitive
            float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
            if (m == kMetaInternal ? r >= count : (m > 8u || r + m > h->prim_count)) {
                atomicOr(err, 1u << RT_ERR_BAD_AS);  // malformed child: leave its box empty
            } else if (m == kMetaInternal) {
                const WideNode* cn = &nodes[r];
                uint32_t c0 = __ldcg(&cn->meta[0]), c1 = __ldcg(&cn->meta[1]);
                for (int q = 0; q < 8; q++) {
                    if (node_meta(c0, c1, q) == 0) continue;
                    lo[0] = fminf(lo[0], __ldcg(&cn->lox[q]));
                    lo[1] = fminf(lo[1], __ldcg(&cn->loy[q]));
                    lo[2] = fminf(lo[2], __ldcg(&cn->loz[q]));
                    hi[0] = fmaxf(hi[0], __ldcg(&cn->hix[q]));
                    hi[1] = fmaxf(hi[1], __ldcg(&cn->hiy[q]));
                    hi[2] = fmaxf(hi[2], __ldcg(&cn->hiz[q]));
                }
            } else {
                for (uint32_t q = 0; q < m; q++) {
                    float4 l = sboxes[2 * (size_t)(r + q)], u = sboxes[2 * (size_t)(r + q) + 1];
                    lo[0] = fminf(lo[0], l.x);
                    lo[1] = fminf(lo[1], l.y);
                    lo[2] = fminf(lo[2], l.z);
                    hi[0] = fmaxf(hi[0], u.x);
                    hi[1] = fmaxf(hi[1], u.y);
                    hi[2] = fmaxf(hi[2], u.z);
                }
            }
            nd->lox[k] = lo[0];
            nd->loy[k] = lo[1];
            nd->loz[k] = lo[2];
            nd->hix[k] = hi[0];
            nd->hiy[k] = hi[1];
            nd->hiz[k] = hi[2];
            for (int a = 0; a < 3; a++) {
                ulo[a] = fminf(ulo[a], lo[a]);
                uhi[a] = fmaxf(uhi[a], hi[a]);
            }
        }
        uint32_t p = __ldcg(&parents[slot]);
        if (p == kNone || p >= count) {
            for (int a = 0; a < 3; a++) {
                h->bounds_lo[a] = ulo[a];
                h->bounds_hi[a] = uhi[a];
            }
            return;
        }
        int need = internal_children(&nodes[p]);
        if ((int)arrive(&counters[p]) + 1 < need) return;
        slot = p;
    }
    atomicOr(err, 1u << RT_ERR_STACK_OVERFLOW);
}

__global__ void k_refit_status(AsHeader* h, const uint32_t* err) {
    after_previous();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    uint32_t e = *err;
    for (uint32_t b = 1; b < 32; b++)
        if (e & (1u << b)) {
            h->status = b;
            return;
        }
}

// ---- AS copy (CLONE / COMPACT) ------------------------------------------------------
__global__ void k_as_copy(const uint8_t* src, uint8_t* dst, uint64_t dst_size, uint32_t mode) {
    after_previous();
    const AsHeader* h = reinterpret_cast<const AsHeader*>(src);
    if (h->magic != kAsMagic) {
        if (blockIdx.x == 0 && threadIdx.x == 0 && dst_size >= kHeaderBytes)
            reinterpret_cast<AsHeader*>(dst)->status = RT_ERR_BAD_AS;
        return;
    }
    uint64_t nodes_bytes = (uint64_t)h->node_count * h->node_bytes;
    uint64_t prim_bytes = (uint64_t)h->prim_count * (h->type == kAsTypeTop ? kInstBytes : kTriBytes);
    uint64_t par_bytes = h->parents_offset ? (uint64_t)h->node_count * 4 : 0;
    uint64_t need = mode == RT_COPY_MODE_COMPACT ? h->compacted_size : h->total_size;
    if (need > dst_size) {
        if (blockIdx.x == 0 && threadIdx.x == 0 && dst_size >= kHeaderBytes) {
            AsHeader* d = reinterpret_cast<AsHeader*>(dst);
            d->magic = 0;
            d->status = RT_ERR_INVALID;
        }
        return;
    }
    uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    if (mode != RT_COPY_MODE_COMPACT) {
        // CLONE: the whole blob, position independent (offsets only).
        const uint4* s = reinterpret_cast<const uint4*>(src);
        uint4* d = reinterpret_cast<uint4*>(dst);
        uint64_t n16 = h->total_size / 16;
        for (uint64_t i = tid; i < n16; i += stride) d[i] = s[i];
        return;
    }
    // COMPACT: header | nodes[node_count] | parents[node_count] | prims
    uint64_t c_nodes = h->nodes_offset;
    uint64_t c_par = h->parents_offset ? align_up(c_nodes + nodes_bytes, 256) : 0;
    uint64_t c_prims = align_up(c_par ? c_par + par_bytes : c_nodes + nodes_bytes, 256);
    auto copy = [&](uint64_t so, uint64_t dof, uint64_t bytes) {
        const uint32_t* s = reinterpret_cast<const uint32_t*>(src + so);
        uint32_t* d = reinterpret_cast<uint32_t*>(dst + dof);
        for (uint64_t i = tid; i < bytes / 4; i += stride) d[i] = s[i];
    };
    copy(h->nodes_offset, c_nodes, nodes_bytes);
    if (par_bytes) copy(h->parents_offset, c_par, par_bytes);
    copy(h->prims_offset, c_prims, prim_bytes);
    if (tid == 0) {
        AsHeader hd = *h;
        hd.max_nodes = h->node_count;
        hd.parents_offset = c_par;
        hd.prims_offset = c_prims;
        hd.total_size = h->compacted_size;
        *reinterpret_cast<AsHeader*>(dst) = hd;
    }
}

inline uint32_t blocks_for(uint64_t n, uint32_t t) { return (uint32_t)((n + t - 1) / t); }
// PLOC hierarchy for builds that prefer trace speed (the reference's BLAS and
// TLAS flags); the Karras LBVH for PREFER_FAST_BUILD or no preference, and
// whenever one leaf holds everything.
inline bool uses_ploc(uint32_t n, bool top, uint32_t build_flags) {
    return (build_flags & RT_BUILD_PREFER_FAST_TRACE) && !(build_flags & RT_BUILD_PREFER_FAST_BUILD) &&
           n > (top ? kTlasLeafMax : kBlasLeafMax);
}

// Grid-wide PLOC rounds for n > kPlocSmall primitives: enough to reach
// kPlocSmall clusters at the measured survival rates, and 6 more.  A round
// that finds kPlocSmall or fewer does nothing (1 us); k_ploc_pairs takes
// what is above it after the last.  Spheres of up to 1M triangles need 8 rounds
// fewer, the one of 10.5M 3; with 2 more instead of 6, scattered triangles, hair
// and the 10.5M-triangle sphere were left to the pairs, whose trees are worse:
// 300,000 scattered triangles 89.8 nodes a ray instead of 84.5, 3,000,000 of
// them (many overlapping) deeper than the traversal's stack then was.
inline int ploc_grid_rounds(uint32_t n) {
    if (n <= kPlocSmall) return 0;
    const double x = kPlocFirstRate * (double)n / (double)kPlocSmall;
    const int rounds = 1 + (x > 1.0 ? (int)std::ceil(std::log(x) / -std::log(kPlocRate)) : 0) + 6;
    return std::min(rounds, kPlocMaxRounds);
}
// Whether round r is expected to fill the SMs with four blocks each (k_ploc_round<4>).
inline bool ploc_round_fills(uint32_t n, int r) {
    const double c = r == 0 ? (double)n : 1.35 * kPlocFirstRate * std::pow(kPlocRate, r - 1) * (double)n;
    return c / kPlocTile + 2.0 >= (double)kPlocMaxBlocks;
}

}  // namespace

// ---------------------------------------------------------------------------
// Layouts
// ---------------------------------------------------------------------------
AsLayout AsLayout::make(uint32_t n, bool top, uint32_t build_flags) {
    const bool quantized = !top && (build_flags & RT_BUILD_QUANTIZED_NODES) != 0;
    AsLayout l;
    l.max_nodes = (uint32_t)max_wide_nodes(n, node_width(build_flags));
    l.node_bytes = (quantized && !top) ? kQNodeBytes : kNodeBytes;
    l.nodes = kHeaderBytes;
    uint64_t end = l.nodes + (uint64_t)l.max_nodes * l.node_bytes;
    if (top) {
        l.parents = align_up(end, 256);
        end = l.parents + (uint64_t)l.max_nodes * 4;
    } else {
        l.parents = 0;
    }
    l.prims = align_up(end, 256);
    l.total = align_up(l.prims + (uint64_t)n * (top ? kInstBytes : kTriBytes), 256);
    return l;
}

// The look-back descriptors of a PLOC build, 8 bytes for each tile of its first
// round, in a region of about 24 bytes a primitive: what a build with several
// launches a round once needed.  The scratch sizes that callers query, and the
// triangle limit of the static-scratch build that follows from them, stay so.
static uint64_t ploc_desc_bytes(uint64_t n) {
    return 5 * align_up(n * 4, 256) + align_up((n + 1023) / 1024 * 4, 256) + align_up((n - 1) * 4, 256);
}

ScratchLayout ScratchLayout::make(uint32_t n, bool top, uint32_t build_flags) {
    const bool quantized = !top && (build_flags & RT_BUILD_QUANTIZED_NODES) != 0;
    const uint64_t cap = max_wide_nodes(n, node_width(build_flags));
    ScratchLayout s{};
    uint64_t nn = n ? n : 1;
    uint64_t ni = n > 1 ? n - 1 : 1;
    uint64_t o = 0;
    auto take = [&](uint64_t bytes) {
        uint64_t r = o;
        o = align_up(o + bytes, 256);
        return r;
    };
    s.state = take(kBuildStateBytes);
    s.boxes = take(nn * 32);
    s.sboxes = take(nn * 32);
    s.keys0 = take(nn * 4);
    s.keys1 = take(nn * 4);
    s.vals0 = take(nn * 4);
    s.vals1 = take(nn * 4);
    s.hist = take(key_sort_state_bytes((uint32_t)nn));  // onesweep state + partition descriptors
    s.inodes = take(ni * 16);
    s.iboxes = take(ni * 32);
    s.iparent = take(ni * 4);
    s.lparent = take(nn * 4);
    s.flags = take(ni * 4);
    s.temp_inst = top ? take(nn * kInstBytes) : 0;
    s.fp32_nodes = quantized ? take(cap * kNodeBytes) : 0;
    s.perm = take(nn * 4);
    s.ploc = uses_ploc(n, top, build_flags);
    if (s.ploc) {
        s.ploc_box0 = take(nn * 32);
        s.ploc_box1 = take(nn * 32);
        s.ploc_desc = take(ploc_desc_bytes(nn));
    }
    s.refit_counters = 0;
    s.build_total = o;
    // update (refit) scratch: sorted boxes + one counter per node, sized for
    // either node width (the refit does not know which one the TLAS was built with)
    uint64_t u = 0;
    u = align_up(u + nn * 32, 256);
    s.refit_counters = u;
    u = align_up(u + max_wide_nodes(n, 4) * 4 + 4, 256);  // + error word
    s.update_total = u;
    return s;
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
namespace {

cudaError_t build_common(uint32_t n, bool top, uint32_t build_flags, uint32_t geometry_count, uint8_t* dst,
                         uint8_t* scratch, cudaStream_t stream, const BlasInput* blas,
                         const RtAccelerationStructureInstance* inst) {
    const bool quantized = !top && (build_flags & RT_BUILD_QUANTIZED_NODES) != 0;
    ScratchLayout sl = ScratchLayout::make(n, top, build_flags);
    AsLayout al = AsLayout::make(n, top, build_flags);
    // quantised builds collapse into FP32 nodes in scratch, then quantise
    WideNode* fp32_nodes = quantized ? reinterpret_cast<WideNode*>(scratch + sl.fp32_nodes)
                                     : reinterpret_cast<WideNode*>(dst + al.nodes);
    BuildState* st = reinterpret_cast<BuildState*>(scratch + sl.state);
    float4* boxes = reinterpret_cast<float4*>(scratch + sl.boxes);
    float4* sboxes = reinterpret_cast<float4*>(scratch + sl.sboxes);
    uint32_t* keys[2] = {reinterpret_cast<uint32_t*>(scratch + sl.keys0), reinterpret_cast<uint32_t*>(scratch + sl.keys1)};
    uint32_t* vals[2] = {reinterpret_cast<uint32_t*>(scratch + sl.vals0), reinterpret_cast<uint32_t*>(scratch + sl.vals1)};
    uint32_t* hist = reinterpret_cast<uint32_t*>(scratch + sl.hist);
    uint4* inodes = reinterpret_cast<uint4*>(scratch + sl.inodes);
    float4* iboxes = reinterpret_cast<float4*>(scratch + sl.iboxes);
    uint32_t* iparent = reinterpret_cast<uint32_t*>(scratch + sl.iparent);
    uint32_t* lparent = reinterpret_cast<uint32_t*>(scratch + sl.lparent);
    uint32_t* flags = reinterpret_cast<uint32_t*>(scratch + sl.flags);
    InstRecord* temp = top ? reinterpret_cast<InstRecord*>(scratch + sl.temp_inst) : nullptr;
    const uint32_t T = 256;
    // PLOC: one look-back descriptor per tile of the first round.  The collapse's
    // tasks (8 bytes per possible wide node) take the Karras hierarchy's parent
    // arrays (12 n bytes) in PLOC builds and the unsorted boxes (32 n bytes, dead
    // once gathered) in Karras builds, so the scratch holds nothing more for them.
    unsigned long long* tasks = reinterpret_cast<unsigned long long*>(sl.ploc ? scratch + sl.iparent : scratch + sl.boxes);
    const uint32_t task_count = n > (top ? kTlasLeafMax : kBlasLeafMax) ? al.max_nodes : 0u;
    const ZeroedWords zero_ploc = {reinterpret_cast<unsigned long long*>(scratch + sl.ploc_desc), tasks,
                                   reinterpret_cast<unsigned long long*>(hist), sl.ploc ? blocks_for(n, kPlocTile) : 0u,
                                   sl.ploc ? task_count : 0u,
                                   n > kSortBlockMax ? (uint32_t)(key_sort_state_bytes(n) / 8u) : 0u};
    const ZeroedWords zero_karras = {nullptr, tasks, nullptr, 0u, task_count, 0u};

    HeaderStatic hs;
    hs.node_bytes = al.node_bytes;
    hs.type = top ? kAsTypeTop : kAsTypeBottom;
    hs.build_flags = build_flags;
    hs.prim_count = n;
    hs.max_nodes = al.max_nodes;
    hs.geometry_count = geometry_count;
    hs.leaf_max = top ? kTlasLeafMax : kBlasLeafMax;
    hs.total_size = al.total;
    hs.nodes_offset = al.nodes;
    hs.prims_offset = al.prims;
    hs.parents_offset = al.parents;
    hs.prim_bytes = top ? kInstBytes : kTriBytes;

    if (top && n > 0 && n <= kTlasSmall) {
        // a per-device attribute: set on every build (a host-side call, no device work)
        const cudaError_t smem_ok = cudaFuncSetAttribute(k_tlas_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                         (int)sizeof(TlasSmallShared));
        if (smem_ok != cudaSuccess) return smem_ok;
        TlasSmallArgs ta;
        ta.inst = inst;
        ta.temp = temp;
        ta.header = reinterpret_cast<AsHeader*>(dst);
        ta.nodes = fp32_nodes;
        ta.parents = reinterpret_cast<uint32_t*>(dst + al.parents);
        ta.out = reinterpret_cast<InstRecord*>(dst + al.prims);
        ta.n = n;
        ta.width = node_width(build_flags);
        ta.max_nodes = al.max_nodes;
        launch(k_tlas_small, 1, kTlasSmall, sizeof(TlasSmallShared), stream, ta, hs);
        return cudaGetLastError();
    }
    launch(k_init_state, 1, 32, 0, stream, st, n);
    if (n > 0) {
        if (top) launch(k_tlas_prims, blocks_for(n, T), T, 0, stream, inst, n, boxes, temp, st, zero_ploc);
        else launch(k_blas_prims, std::min(blocks_for(n, T), kPrimBlocks), T, 0, stream, *blas, boxes, st, zero_ploc);
        // Morton codes and their stable order: the sorted pairs land in keys[0] / vals[0]
        const int cur = 0;
        if (cudaError_t e = launch_sort<true>(keys[0], vals[0], keys[1], vals[1], n, reinterpret_cast<uint8_t*>(hist),
                                              &st->error, boxes, st, stream);
            e != cudaSuccess)
            return e;
        if (sl.ploc) {
            PlocArgs pa;
            pa.boxes = boxes;
            pa.vals = vals[cur];
            pa.sboxes = sboxes;
            pa.cbox[0] = reinterpret_cast<float4*>(scratch + sl.ploc_box0);
            pa.cbox[1] = reinterpret_cast<float4*>(scratch + sl.ploc_box1);
            pa.inodes = inodes;
            pa.iboxes = iboxes;
            pa.st = st;
            pa.desc = zero_ploc.desc;
            pa.n = n;
            const int rounds = ploc_grid_rounds(n);
            // every round has a block for each tile of the first: the clusters that a round finds
            // are known on the device only, and where they merge slowly a grid of the expected
            // size takes them a few tiles at a time (1.4M triangles in nested shells 4.9 -> 1.6 ms,
            // 200,000 of very different sizes 791 -> 450 us; the spheres of 163,840 and 10.5M
            // triangles, most of whose blocks find no tile in the later rounds, 0.8 and 0.4 % faster)
            const uint32_t g = std::min<uint32_t>(blocks_for(n, kPlocTile), kPlocMaxBlocks);
            for (int r = 0; r < rounds; r++) {
                if (ploc_round_fills(n, r)) launch(k_ploc_round<4>, g, kPlocThreads, 0, stream, pa, r);
                else launch(k_ploc_round<3>, g, kPlocThreads, 0, stream, pa, r);
            }
            // a per-device attribute: set on every build (a host-side call, no device work)
            const cudaError_t smem_ok =
                cudaFuncSetAttribute(k_ploc_tail, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(PlocTailShared));
            if (smem_ok != cudaSuccess) return smem_ok;
            if (rounds > 0) launch(k_ploc_pairs, kPlocPairBlocks, kPlocPairThreads, 0, stream, pa, rounds);
            launch(k_ploc_tail, 1, kPlocSmall, sizeof(PlocTailShared), stream, pa, rounds > 0 ? rounds + 1 : 0);
        } else {
            launch(k_gather_boxes, blocks_for(n, T), T, 0, stream, boxes, vals[cur], n, sboxes);
        }
        if (!sl.ploc && n > 1) {
            launch(k_karras, blocks_for(n - 1, T), T, 0, stream, keys[cur], n, inodes, iparent, lparent, flags, zero_karras);
            launch(k_bottom_up, blocks_for(n, T), T, 0, stream, inodes, lparent, iparent, sboxes, iboxes, flags, n, &st->error);
        }
        uint32_t* perm = reinterpret_cast<uint32_t*>(scratch + sl.perm);
        CollapseCtx cc;
        cc.inodes = inodes;
        cc.iboxes = iboxes;
        cc.sboxes = sboxes;
        cc.perm = perm;
        cc.nodes = fp32_nodes;
        cc.parents = top ? reinterpret_cast<uint32_t*>(dst + al.parents) : nullptr;
        cc.st = st;
        cc.tasks = tasks;
        cc.leaf_max = top ? kTlasLeafMax : kBlasLeafMax;
        cc.width = node_width(build_flags);
        cc.max_nodes = al.max_nodes;
        cc.n = n;
        // a group of 8 lanes per possible wide node, up to a full load of the SMs
        const uint32_t g = std::min<uint32_t>(blocks_for(al.max_nodes, kCollapseThreads / 8), kCollapseBlocks);
        launch(k_collapse, g, kCollapseThreads, 0, stream, cc);
        if (top) {
            launch(k_write_insts, blocks_for(n, T), T, 0, stream, temp, vals[cur], perm, n, reinterpret_cast<InstRecord*>(dst + al.prims));
        } else {
            launch(k_write_tris, std::min(blocks_for(n, T), kPrimBlocks), T, 0, stream, *blas, vals[cur], perm, reinterpret_cast<TriRecord*>(dst + al.prims), st);
        }
    } else {
        CollapseCtx cc{};
        cc.nodes = fp32_nodes;
        cc.parents = top ? reinterpret_cast<uint32_t*>(dst + al.parents) : nullptr;
        cc.st = st;
        cc.leaf_max = 1;
        cc.width = node_width(build_flags);
        cc.max_nodes = al.max_nodes;
        cc.n = n;
        launch(k_collapse, 1, kCollapseThreads, 0, stream, cc);
    }
    if (quantized) {
        uint32_t g = blocks_for(al.max_nodes, 128);
        launch(k_quantize_nodes, g, 128, 0, stream, fp32_nodes, st, al.max_nodes, reinterpret_cast<QNode*>(dst + al.nodes));
    }
    launch(k_finish, 1, kFinishThreads, 0, stream, reinterpret_cast<AsHeader*>(dst), st, hs);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_blas_build(const BlasInput& in, uint32_t build_flags, uint8_t* dst, uint8_t* scratch,
                              cudaStream_t stream) {
    return build_common(in.n, false, build_flags, in.geometry_count, dst, scratch, stream, &in, nullptr);
}

cudaError_t launch_tlas_build(const RtAccelerationStructureInstance* instances, uint32_t n, uint32_t build_flags,
                              uint8_t* dst, uint8_t* scratch, cudaStream_t stream) {
    return build_common(n, true, build_flags, 1, dst, scratch, stream, nullptr, instances);
}

cudaError_t launch_as_copy(const uint8_t* src, uint8_t* dst, uint64_t dst_size, uint32_t mode, cudaStream_t stream) {
    launch(k_as_copy, 1024, 256, 0, stream, src, dst, dst_size, mode);
    return cudaGetLastError();
}

cudaError_t launch_tlas_update(const RtAccelerationStructureInstance* instances, uint32_t n, const uint8_t* src,
                               uint8_t* dst, uint64_t dst_size, uint8_t* scratch, cudaStream_t stream) {
    ScratchLayout sl = ScratchLayout::make(n, true);
    // node capacity of either node width: the grid and the counters cover any TLAS of n instances
    const uint32_t cap = (uint32_t)max_wide_nodes(n, 4);
    if (src != dst) {
        launch(k_as_copy, 1024, 256, 0, stream, src, dst, dst_size, RT_COPY_MODE_CLONE);
    }
    if (n > 0 && n <= kRefitSmall) {
        launch(k_refit_small, 1, kRefitSmall, 0, stream, instances, n, reinterpret_cast<AsHeader*>(dst));
        return cudaGetLastError();
    }
    float4* sboxes = reinterpret_cast<float4*>(scratch);
    uint32_t* counters = reinterpret_cast<uint32_t*>(scratch + sl.refit_counters);
    // the error word lives after the counters
    uint32_t* err = counters + cap;
    cudaMemsetAsync(counters, 0, (size_t)cap * 4 + 4, stream);
    AsHeader* h = reinterpret_cast<AsHeader*>(dst);
    if (n > 0) launch(k_refit_insts, blocks_for(n, 256), 256, 0, stream, instances, n, h, sboxes, err);
    launch(k_refit_nodes, blocks_for(cap, 128), 128, 0, stream, h, sboxes, counters, cap, err);
    launch(k_refit_status, 1, 32, 0, stream, h, err);
    return cudaGetLastError();
}

}  // namespace rt
