// batch.cu -- Part 2 of gravcuda.h: every sink group of a step evaluated
// by persistent kernels from length-sorted work queues, on index lists into
// device-resident point and cell tables.
//
// Mixed precision (none of this exists in the reference, whose lists carry
// absolute FP32 copies, nln/mac.c:1421-1561):
//   * each sink is held as an FP32 offset from its group's FP64 centre;
//   * each source record is re-centred on the same FP64 centre (with its
//     periodic image shift) as a lane takes it up, so the inner loops subtract
//     two small FP32 numbers;
//   * partial sums of one tile are plain FP32, folded into FP64 sums per tile;
//   * work-item partials are combined per group in FP64, in a fixed order.
// Work decomposition: a work item is (group, kind, range of its list);
// long lists are split so that small problems still fill the GPU; every
// warp pulls items (costliest first) from its kind's queue until it is
// empty.  One warp owns one item: lane = source records, a tile of 64 to 256
// records in the lanes' registers, walked by the group's sinks (below).
// Cell tiles are staged by TMA row gathers (cp.async.bulk.tensor
// tile::gather4 over a 2-D tensor map of the table, one instruction per 4
// records) signalled by per-warp mbarriers, points by per-lane cp.async.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <chrono>
#include <mutex>
#include <numeric>
#include <type_traits>
#include <vector>

#include "build.cuh"
#include "common.cuh"
#include "gravcuda.h"
#include "ewald.cuh"
#define NLN_EWALD_NO_EXPORT
#include "host/ewald_table.cpp"
#include "interact.cuh"

namespace {

enum { KP = 0, KQ = 1, KH = 2 };
constexpr int kListWarps = 4;     // warps per block of the list kernels at most
constexpr int kPointTile = 256;   // records of a staged tile: points
constexpr int kQuadTile = 128;    // quadrupole cells
constexpr int kHexaTile = 64;     // order-4 cells
constexpr int kTile[3] = {kPointTile, kQuadTile, kHexaTile};

// Resident blocks the list kernels' registers are held to (-D to rebuild
// with others).
#ifndef GRAV_H_MINB
#define GRAV_H_MINB 3
#endif
#ifndef GRAV_Q_MINB
#define GRAV_Q_MINB 4
#endif
#ifndef GRAV_P_MINB
#define GRAV_P_MINB 4
#endif

// One group's correction moments as k_ewald_moments stores them (EwMoments).
struct EwStored {
    double lo[10];
    float hi[25];
    float pad[3];
};

struct DevProblem {
    const float4 *points;
    const nln_qcell *qcells;
    const nln_hcell *hcells;
    const nln_group *groups;
    const uint32_t *list[3];   // idx | shift << 27
    int64_t ntab[3];           // table sizes for bounds checks
    const Item *items[3];
    int nitems[3];
    int *counters;             // 4 queue heads: zero before an evaluation, zeroed by its k_finish
    int first;                 // first kernel of the evaluation: wait for what came before
    float4 *part;              // nslots x 32 lanes x 2 (hi, lo)
    const int64_t *gslot;      // ngroups + 1: slots of group g
    float4 *out;               // nbodies
    int64_t ngroups;           // k_finish covers groups gbegin .. ngroups-1
    int64_t gbegin;
    int64_t ncells;
    float eps2;
    float qsh;
    double box;
    unsigned *err;
    // periodic correction
    const int64_t *cptr;       // per-group offsets of the correction list
    const uint32_t *clist;     // correction list: point-table record | image << 27
    int ewald;
    EwTab ew;
    float ew_self;             // C(0) - pi/(alpha^2 L^3): the self term ewald() leaves out
    EwStored *ewm;             // per-group moments from k_ewald_moments
    EwStored *ewpart;          // its units' moments where a group's list is split (ewsplit > 1)
    int *ewdone;               // finished units per group, zero between evaluations
    int ewsplit;               // units per group
    // FP64 centres of the cells for the point table's monopole records (the
    // mixed form re-centres them like every other source): a cell table (the
    // centre is a record's first 24 bytes, one record every cstride bytes),
    // or null, where the FP32 point record is used
    const unsigned char *ccen;
    int cstride;
    // length_scale of the groups' span: the value, or the span on the device
    float hscale;
    const double *hscale_dev;
};

// Image code (0..26) to the image's shift: (code / 9 - 1, code / 3 % 3 - 1,
// code % 3 - 1) box.
__device__ __forceinline__ void decode_shift(uint32_t code, double box, double &sx, double &sy,
                                             double &sz) {
    const uint32_t third = code * 171u >> 9, x = code * 57u >> 9;  // code / 3, code / 9
    const uint32_t y = third - 3u * x, z = code - 3u * third;
    sx = x == 0 ? -box : x == 2 ? box : 0.0;
    sy = y == 0 ? -box : y == 2 ? box : 0.0;
    sz = z == 0 ? -box : z == 2 ? box : 0.0;
}

// Unpack the run-packed lists (format in nlnlists.h) of groups g0..g1-1,
// one warp per group.  Per 32-word block: a warp scan of the words' entry
// counts places each word's entries (an entry word stands for itself, a run
// word for the n entries after the word before it); then the warp writes
// the block's entries 32 consecutive ones at a time, each lane finding the
// word its entry comes from by a binary search over the scan.  Stores stay
// inside the group's plain range [ptr[g], ptr[g+1]); a group that does not
// fill it exactly, a run word that starts a group or follows a run word, or
// a run that would carry into the image code sets GC_DEV_BAD_RUNS.
__global__ void k_unpack(const uint32_t *__restrict__ z, const int64_t *__restrict__ zptr,
                         const int64_t *__restrict__ ptr, int64_t g0, int64_t g1,
                         uint32_t *__restrict__ out, unsigned *err) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t g = g0 + (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); g < g1;
         g += nwarps) {
        const int64_t zb = zptr[g], ze = zptr[g + 1], oe = ptr[g + 1];
        int64_t pos = ptr[g];
        uint32_t prev = 0;  // last word of the previous block
        bool have_prev = false, bad = false;
        for (int64_t b = zb; b < ze; b += 32) {
            const bool valid = b + lane < ze;
            const uint32_t w = valid ? z[b + lane] : 0u;
            const bool run = valid && (w >> NLN_IDX_BITS) == NLN_RUN_CODE;
            uint32_t before = __shfl_up_sync(FULL, w, 1);
            bool before_ok = true;
            if (lane == 0) {
                before = prev;
                before_ok = have_prev;
            }
            uint32_t cnt = !valid ? 0u : (run ? (w & NLN_IDX_MASK) : 1u);
            if (run && (!before_ok || (before >> NLN_IDX_BITS) == NLN_RUN_CODE || cnt == 0 ||
                        (before & NLN_IDX_MASK) + cnt > NLN_IDX_MASK)) {
                bad = true;
                cnt = 0;
            }
            const uint32_t first = run ? before + 1u : w;  // entry j of this word: first + j
            // block totals stay below 2^32: at most 32 words of 2^27 - 1
            uint32_t inc = cnt;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(FULL, inc, o);
                if (lane >= o)
                    inc += v;
            }
            const uint32_t total = __shfl_sync(FULL, inc, 31);
            if (pos + (int64_t)total > oe)
                bad = true;
            const int64_t room = oe - pos;
            const uint32_t lim = room <= 0 ? 0u : (room < (int64_t)total ? (uint32_t)room : total);
            for (uint32_t j0 = 0; j0 < lim; j0 += 32) {
                const uint32_t j = j0 + lane;
                // owner = number of words whose entries all lie before j
                int owner = 0;
#pragma unroll
                for (int step = 16; step >= 1; step >>= 1) {
                    const uint32_t v = __shfl_sync(FULL, inc, owner + step - 1);
                    if (v <= j)
                        owner += step;
                }
                owner = min(owner, 31);
                const uint32_t f = __shfl_sync(FULL, first, owner);
                const uint32_t s0 = __shfl_sync(FULL, inc - cnt, owner);
                if (j < lim)
                    out[pos + j] = f + (j - s0);
            }
            pos += total;
            prev = __shfl_sync(FULL, w, 31);
            have_prev = true;
        }
        if (pos != oe)
            bad = true;
        if (__any_sync(FULL, bad) && lane == 0)
            atomicOr(err, GC_DEV_BAD_RUNS);
    }
}

// Device-side check of an uploaded list, one warp per work item (or per
// group for the correction list): every entry's index inside its table and
// its image code in 0..26.  For the point list it also counts body and cell
// entries, weighted by the group's sinks.  acc: [0] error flag, [1] body
// interactions, [2] monopole-cell interactions.
__global__ void k_check_lists(const uint32_t *__restrict__ list, const Item *__restrict__ items,
                              int nitems, const int64_t *__restrict__ gptr, int64_t ngroups,
                              const nln_group *__restrict__ groups, uint32_t ntab, uint32_t nb,
                              int count_bodies, unsigned long long *acc) {
    const int lane = threadIdx.x & 31;
    const int64_t nwork = items ? nitems : ngroups;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nwork;
         w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        int64_t b, e;
        int32_t g;
        if (items) {
            const Item it = items[w];
            b = it.begin;
            e = it.end;
            g = it.group;
        } else {
            b = gptr[w];
            e = gptr[w + 1];
            g = (int32_t)w;
        }
        unsigned bad = 0;
        long long nbody = 0;
        for (int64_t k = b + lane; k < e; k += 32) {
            const uint32_t v = list[k];
            const uint32_t idx = v & NLN_IDX_MASK;
            bad |= (idx >= ntab || (v >> NLN_IDX_BITS) > 26u) ? 1u : 0u;
            nbody += idx < nb ? 1 : 0;
        }
        bad = __reduce_or_sync(0xffffffffu, bad);
        for (int d = 16; d > 0; d >>= 1) nbody += __shfl_xor_sync(0xffffffffu, nbody, d);
        if (lane == 0) {
            if (bad)
                atomicOr(&acc[0], 1ull);
            if (count_bodies) {
                const long long c = groups[g].count;
                atomicAdd(&acc[1], (unsigned long long)(nbody * c));
                atomicAdd(&acc[2], (unsigned long long)((e - b - nbody) * c));
            }
        }
    }
}

// ------------------------------------------------------------ list kernels
//
// A warp owns one work item: a range of one group's list.  Its lanes hold
// the source records, R each in registers, and the warp walks the group's
// sinks one by one: a sink's offsets are broadcast from shared memory, every
// lane evaluates its own records, and the 32 lanes' sums are added by a
// transposing butterfly that leaves sink s's sum in lane s.  So a group of c
// sinks costs c steps and not 32 (22.5 sinks a group on spheres, 24 to 32 in
// boxes), a record is read from shared memory once per tile and not once per
// sink, and its image shift, FP64 re-centring and moment scaling are done
// once for all sinks.  The butterfly costs about 10 FMA-pipe cycles a sink.
// Against lanes as sinks (32 records broadcast from shared memory), 160^3
// periodic box, MAC 2.5e-6: order 4 90.5 -> 65.5 ms, quadrupole 37.0 -> 30.0,
// points 43.2 -> 34.0; Plummer 64k, points 0.418 -> 0.338 ms.  The order-4
// kernel keeps the FMA pipe 73 % busy, where its operand reads allow 77 %.

// A sink as splat pairs of its negated offsets from the group centre.
struct __align__(16) Sink {
    float4 xy;
    float2 z, pad;
};
struct SinkTable {
    Sink s[32];
};

// Inside the order-4 kernel lengths are in units of the power of two below the
// span of the groups: its largest terms, R^4 r^4 m, would leave FP32 in systems
// that span some 1e5 lengths (unit masses), and its inverse powers in those of
// 1e-7.  A power of two changes no other bits.  1 over that unit:
__host__ __device__ inline float length_scale(double span) {
    if (!(span > 1e-18 && span < 1e18))
        return 1.f;
    float s = 1.f;
    for (; span >= 2.0; span *= 0.5) s *= 0.5f;
    for (; span < 1.0; span *= 2.0) s *= 2.f;
    return s;
}

// The span as the largest distance along an axis of a group's edge from `from`.
__host__ __device__ inline double group_span(const nln_group &G, const nln_group &from) {
    double s = 0;
    for (int d = 0; d < 3; d++) s = fmax(s, fabs(G.cen[d] - from.cen[d]));
    return s + G.radius;
}

// This lane's sink offset from the group centre c, into the table; `scale`: 1
// over the kernel's unit of length.
__device__ __forceinline__ void stage_sinks(SinkTable &T, const DevProblem &P, const nln_group &G,
                                            const double *c, int lane, float scale = 1.f) {
    __syncwarp();  // the previous item's sinks are no longer read
    if (lane < G.count) {
        const float4 s = P.points[G.first + lane];
        const float nx = -scale * (float)((double)s.x - c[0]),
                    ny = -scale * (float)((double)s.y - c[1]),
                    nz = -scale * (float)((double)s.z - c[2]);
        T.s[lane].xy = make_float4(nx, nx, ny, ny);
        T.s[lane].z = make_float2(nz, nz);
    }
    __syncwarp();
}

__device__ __forceinline__ float4 add4(float4 a, float4 b) {
    const float2 u = add2(f2(a.x, a.y), f2(b.x, b.y)), v = add2(f2(a.z, a.w), f2(b.z, b.w));
    return make_float4(u.x, u.y, v.x, v.y);
}
__device__ __forceinline__ float4 shfl_xor4(float4 v, int m) {
    return make_float4(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m),
                       __shfl_xor_sync(0xffffffffu, v.z, m), __shfl_xor_sync(0xffffffffu, v.w, m));
}
// A sink's running sum over the tiles of an item, in FP64: its conversions and
// adds take fewer issue slots than two-sum compensation in FP32 (1M bodies
// 6.53 -> 6.50 ms).
struct Total {
    double v[4] = {0, 0, 0, 0};
    __device__ __forceinline__ void add(float4 t) {
        v[0] += t.x;
        v[1] += t.y;
        v[2] += t.z;
        v[3] += t.w;
    }
};

// Partial sums of a warp's sinks: row b holds sinks 4 b .. 4 b + 3, lane l's
// entry a part of sink 4 b + (l & 3).  The pitch keeps two rows' reads on
// different banks.
struct SinkSums {
    float4 row[8][36];
};

// Every sink's sum over the warp's records, added to lane s's acc for
// sink s; eval(sink) gives this lane's part.  In a full block of four sinks lane l starts with
// sink l & 3, so that the two exchange levels need no selects: what it keeps
// is always its own sink's.  The last three levels are summed from shared
// memory once a tile.  The four evaluations of a block are one basic block
// (a test per sink kept them from overlapping: 19.4 against 20.1 cycles per
// point interaction, 18.5 with the registers to hold four of them).
template <int FOLDS, class Eval>
__device__ __forceinline__ void sum_sinks(const SinkTable &T, int nsink, int lane, SinkSums &buf,
                                          Total &acc, Eval eval) {
    const int sw = lane & 3, nb = nsink >> 2, rem = nsink & 3;
    const Sink *p0 = T.s + sw, *p1 = T.s + (sw ^ 1), *p2 = T.s + (sw ^ 2), *p3 = T.s + (sw ^ 3);
    float4 *out = &buf.row[0][lane];
#pragma unroll 1
    for (int b = 0; b < nb; b++) {
        float4 r0 = eval(*p0), r1 = eval(*p1);
        r0 = add4(r0, shfl_xor4(r1, 1));
        float4 r2 = eval(*p2), r3 = eval(*p3);
        r2 = add4(r2, shfl_xor4(r3, 1));
        *out = add4(r0, shfl_xor4(r2, 2));
        out += 36;
        p0 += 4;
        p1 += 4;
        p2 += 4;
        p3 += 4;
    }
    if (rem) {
        float4 keep = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (int i = 0; i < rem; i++) {
            float4 r = eval(T.s[4 * nb + i]);
            r = add4(r, shfl_xor4(r, 1));
            r = add4(r, shfl_xor4(r, 2));
            if (sw == i)
                keep = r;
        }
        *out = keep;
    }
    __syncwarp();
    if (lane < nsink) {
        const float4 *row = buf.row[lane >> 2] + sw;
#pragma unroll
        for (int f = 0; f < FOLDS; f++) {
            float4 v = row[4 * f];
#pragma unroll
            for (int k = FOLDS; k < 8; k += FOLDS) v = add4(v, row[4 * (f + k)]);
            acc.add(v);
        }
    }
    __syncwarp();  // read: the next tile may write
}

__device__ __forceinline__ void store_part(const DevProblem &P, const Item &item, int lane,
                                           const Total &acc) {
    float hi[4], lo[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        hi[q] = (float)acc.v[q];
        lo[q] = (float)(acc.v[q] - (double)hi[q]);
    }
    float4 *dst = P.part + ((size_t)item.slot * 32 + lane) * 2;
    dst[0] = make_float4(hi[0], hi[1], hi[2], hi[3]);
    dst[1] = make_float4(lo[0], lo[1], lo[2], lo[3]);
}

// Coordinate of an absent record, beyond any sink: with zero mass and
// moments it adds exactly zero.
constexpr float kFar = 1.0e18f;

// A record's FP64 position in image `code` as an FP32 offset from c;
// `shifted` (the same in every lane): some lane's image is not the box's own.
__device__ __forceinline__ void recentre(double x, double y, double z, uint32_t code, bool shifted,
                                         double box, const double *c, float *o) {
    if (shifted) {
        double sx, sy, sz;
        decode_shift(code, box, sx, sy, sz);
        x += sx;
        y += sy;
        z += sz;
    }
    o[0] = (float)(x - c[0]);
    o[1] = (float)(y - c[1]);
    o[2] = (float)(z - c[2]);
}

template <int KIND>
struct CellKind {
    using Rec = std::conditional_t<KIND == KH, nln_hcell, nln_qcell>;
    using Pair = std::conditional_t<KIND == KH, HexaPair, QuadPair>;
    static constexpr int rec_bytes = (int)sizeof(Rec);
    static constexpr int pairs = kTile[KIND] / 64;  // record pairs per lane
    static constexpr int stage_bytes = kTile[KIND] * rec_bytes;
    // per warp: the stage (its swizzle pattern repeats every 1024 bytes), the
    // sinks, their sums, the mbarrier
    static constexpr int warp_bytes =
        (stage_bytes + (int)(sizeof(SinkTable) + sizeof(SinkSums)) + 8 + 1023) / 1024 * 1024;
    // 16-byte chunk k of row r: the TMA swizzle of the row's width spreads
    // the lanes' own-row reads over all banks
    static __device__ __forceinline__ int chunk(int r, int k) {
        const int sw = KIND == KH ? r & 7 : (r >> 1) & 3;
        return r * rec_bytes + ((k ^ sw) << 4);
    }
};

// Half h (0: .x, 1: .y) of this lane's record pair from row r of the stage.
__device__ __forceinline__ void set_half(float2 &p, int h, float v) {
    if (h)
        p.y = v;
    else
        p.x = v;
}

template <int KIND>
__device__ __forceinline__ void load_cell(const unsigned char *stage, int r, bool valid,
                                          uint32_t code, double box, const double *c, float scale,
                                          typename CellKind<KIND>::Pair &p, int h) {
    using K = CellKind<KIND>;
    constexpr int NC = KIND == KH ? 8 : 4;
    const bool shifted = __any_sync(0xffffffffu, code != NLN_SHIFT_NONE);
    float f[4 * NC];
#pragma unroll
    for (int k = 0; k < NC; k++) {
        // the last chunk of a quadrupole record holds one field, of an order-4 record two
        const float4 v = *reinterpret_cast<const float4 *>(stage + K::chunk(r, k));
        f[4 * k] = v.x;
        f[4 * k + 1] = v.y;
        f[4 * k + 2] = v.z;
        f[4 * k + 3] = v.w;
    }
    // floats 0-5 the FP64 centre, 6 mass, 7 R, then q2[5] (order 4: q3[7], q4[9])
    auto d = [&](int k) { return __hiloint2double(__float_as_int(f[k + 1]), __float_as_int(f[k])); };
    float o[3];
    recentre(d(0), d(2), d(4), code, shifted, box, c, o);
#pragma unroll
    for (int k = 0; k < (KIND == KH ? 3 : 0); k++) o[k] *= scale;
    auto put = [&](float2 &dst, float v) { set_half(dst, h, valid ? v : 0.f); };
    set_half(p.x, h, valid ? o[0] : kFar);
    set_half(p.y, h, valid ? o[1] : kFar);
    set_half(p.z, h, valid ? o[2] : kFar);
    put(p.m, f[6]);
    const float R = KIND == KH ? scale * f[7] : f[7], c2 = -3.0f * R * R;
#pragma unroll
    for (int k = 0; k < 5; k++) put(p.q[k], c2 * f[8 + k]);
    if constexpr (KIND == KQ) {
        put(p.q[5], -(c2 * f[8] + c2 * f[10]));
    } else {
        const float c3 = 7.5f * R * R * R, c4 = -17.5f * R * R * R * R;
        const float *q3 = f + 13, *q4 = f + 20;
#pragma unroll
        for (int k = 0; k < 7; k++) put(p.o[k], c3 * q3[k]);
        put(p.o[7], -(c3 * q3[0] + c3 * q3[2]));
        put(p.o[8], -(c3 * q3[1] + c3 * q3[3]));
#pragma unroll
        for (int k = 0; k < 9; k++) put(p.h[k], c4 * q4[k]);
        put(p.h[9], -(c4 * q4[0] + c4 * q4[2]));
        put(p.h[10], -(c4 * q4[4] + c4 * q4[2]));
        put(p.h[11], -(c4 * q4[1] + c4 * q4[3]));
    }
}

// Quadrupole and order-4 lists: tiles of 128 or 64 cells, two or one record
// pairs per lane (a tile that ends short leaves out the second), gathered
// from the cell table by TMA (row gathers of four records, issued by lane 0)
// into one stage per warp, which is free for the next tile's copies as soon
// as the lanes hold their records.
// PLAIN: the plain FP32 form the reference's lists compute in (absolute FP32
// coordinates, nln/mac.c:1421-1561 copies cell centres as floats): sinks and
// sources are not re-centred on the group centre.  It exists to be compared
// with the mixed form.
template <int KIND, bool PLAIN>
__global__ void __launch_bounds__(32 * kListWarps, KIND == KH ? GRAV_H_MINB : GRAV_Q_MINB)
    k_cells(const __grid_constant__ CUtensorMap tmap, DevProblem P) {
    using K = CellKind<KIND>;
    constexpr int NP = K::pairs, NE = 2 * NP, CT = kTile[KIND];
    extern __shared__ __align__(1024) unsigned char smem[];
    if (P.first)
        pdl_wait();  // before the trigger: the kernels after this one rely on it
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    unsigned char *stage = smem + (size_t)(threadIdx.x >> 5) * K::warp_bytes;
    SinkTable &sinks = *reinterpret_cast<SinkTable *>(stage + K::stage_bytes);
    SinkSums &sums = *reinterpret_cast<SinkSums *>(&sinks + 1);
    uint64_t *bar = reinterpret_cast<uint64_t *>(&sums + 1);
    if (lane == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    __syncwarp();
    const uint32_t *list = P.list[KIND];
    const uint32_t ntab = (uint32_t)P.ntab[KIND];
    const float scale = KIND == KH ? (P.hscale_dev ? length_scale(*P.hscale_dev) : P.hscale) : 1.f;
    const float2 e2 = splat2(P.eps2 * (scale * scale));
    uint32_t phase = 0;
    for (;;) {
        int it = 0;
        if (lane == 0)
            it = atomicAdd(&P.counters[KIND], 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= P.nitems[KIND])
            break;
        const Item item = P.items[KIND][it];
        const nln_group G = P.groups[item.group];
        const double c[3] = {PLAIN ? 0.0 : G.cen[0], PLAIN ? 0.0 : G.cen[1],
                             PLAIN ? 0.0 : G.cen[2]};
        const int64_t nent = item.end - item.begin;
        const int ntile = (int)((nent + CT - 1) / CT);
        // this lane's entries of tile t
        auto fetch = [&](int t, uint32_t *e) {
#pragma unroll
            for (int h = 0; h < NE; h++) {
                const int64_t k = item.begin + (int64_t)t * CT + 32 * h + lane;
                e[h] = t < ntile && k < item.end ? __ldg(list + k) : 0u;
            }
        };
        // Start the copies of tile t: the row indices are gathered to lane 0;
        // unused rows of the last gather repeat row 0.  code: the image codes
        // of this lane's records.
        auto issue = [&](int t, const uint32_t *e, uint32_t *code) {
            const int nt = (int)min((int64_t)CT, nent - (int64_t)t * CT);
            const int ng4 = (nt + 3) >> 2;
            if (lane == 0)
                mbar_arrive_expect_tx(bar, (uint32_t)(ng4 * 4 * K::rec_bytes));
#pragma unroll
            for (int h = 0; h < NE; h++) {
                uint32_t idx = e[h] & NLN_IDX_MASK;
                const bool live = 32 * h + lane < nt;
                code[h] = live ? e[h] >> NLN_IDX_BITS : NLN_SHIFT_NONE;
                // entries are checked at upload, except in the pipelined end-to-end call
                if (live && (idx >= ntab || code[h] > 26u)) {
                    atomicOr(P.err, GC_DEV_BAD_INDEX);
                    idx = 0;
                    code[h] = NLN_SHIFT_NONE;
                }
                if (!live)
                    idx = 0;
                if (8 * h >= ng4)
                    continue;
#pragma unroll
                for (int g = 0; g < 8; g++) {
                    const int r0 = __shfl_sync(0xffffffffu, (int)idx, 4 * g);
                    const int r1 = __shfl_sync(0xffffffffu, (int)idx, 4 * g + 1);
                    const int r2 = __shfl_sync(0xffffffffu, (int)idx, 4 * g + 2);
                    const int r3 = __shfl_sync(0xffffffffu, (int)idx, 4 * g + 3);
                    if (lane == 0 && 8 * h + g < ng4)
                        tma_gather4(stage + (8 * h + g) * 4 * K::rec_bytes, &tmap, r0, r1, r2, r3,
                                    bar);
                }
            }
        };
        uint32_t ent[NE], code[NE];
#pragma unroll
        for (int h = 0; h < NE; h++) code[h] = NLN_SHIFT_NONE;
        fetch(0, ent);
        if (ntile > 0)
            issue(0, ent, code);
        fetch(1, ent);
        stage_sinks(sinks, P, G, c, lane, scale);
        Total acc;
        for (int t = 0; t < ntile; t++) {
            const int nt = (int)min((int64_t)CT, nent - (int64_t)t * CT);
            const bool ok = mbar_wait_bounded(bar, phase, P.err);
            if (!__all_sync(0xffffffffu, ok)) {
                pdl_wait();
                return;  // a lost copy: the error word is set, nothing else is in flight
            }
            phase ^= 1;
            typename K::Pair rec[NP];
#pragma unroll
            for (int h = 0; h < NE; h++)
                if (h < 2 || nt > 64 * (h >> 1))
                    load_cell<KIND>(stage, 32 * h + lane, 32 * h + lane < nt, code[h], P.box, c,
                                    scale, rec[h >> 1], h & 1);
            __syncwarp();  // the stage is free: start the next copies, then compute
            if (t + 1 < ntile)
                issue(t + 1, ent, code);
            fetch(t + 2, ent);
            // the forms of a tile are told apart outside the sink loop
            auto sums_of = [&](auto form) {
                constexpr bool F = decltype(form)::value;
                sum_sinks<KIND == KH ? 2 : 4>(sinks, G.count, lane, sums, acc, [&](const Sink &k) {
                    const float2 nx = f2(k.xy.x, k.xy.y), ny = f2(k.xy.z, k.xy.w), nz = k.z;
                    Sum2 A;
                    if constexpr (KIND == KH) {
                        cell_pair<F>(rec[0], nx, ny, nz, e2, P.qsh, A);
                    } else {
                        cell_pair<true>(rec[0], nx, ny, nz, e2, P.qsh, A);
                        if (F)
                            cell_pair<false>(rec[1], nx, ny, nz, e2, P.qsh, A);
                    }
                    return A.total();
                });
            };
            const bool form = KIND == KH ? P.qsh == 0.5f : nt > 64;
            if (form)
                sums_of(std::true_type());
            else
                sums_of(std::false_type());
        }
        if constexpr (KIND == KH) {
            for (int k = 0; k < 3; k++) acc.v[k] *= (double)scale * scale;
            acc.v[3] *= scale;
        }
        store_part(P, item, lane, acc);
    }
    pdl_wait();
}

// Point lists (bodies and cell monopoles): tiles of 256 records, eight per
// lane in four pairs.  Every lane copies its own next records (a body's 16
// bytes, a cell's FP64 centre and mass: 32) to its own slots of the warp's
// stage by cp.async while the warp computes the current tile, with the list
// words one tile further ahead; the registers that hold four evaluations at
// once leave 16 warps on an SM, too few to cover the loads otherwise.
struct PointStage {
    float4 chunk[kPointTile / 32][2][32];  // [record of the lane][half][lane]
};
constexpr int kPointWarpBytes = (int)(sizeof(PointStage) + sizeof(SinkTable) + sizeof(SinkSums));

template <bool PLAIN>
__global__ void __launch_bounds__(32 * kListWarps, GRAV_P_MINB) k_points(DevProblem P) {
    extern __shared__ __align__(16) unsigned char psm[];
    if (P.first)
        pdl_wait();  // before the trigger: the kernels after this one rely on it
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    PointStage &stage = *reinterpret_cast<PointStage *>(psm + (size_t)(threadIdx.x >> 5) * kPointWarpBytes);
    SinkTable &sinks = *reinterpret_cast<SinkTable *>(&stage + 1);
    SinkSums &sums = *reinterpret_cast<SinkSums *>(&sinks + 1);
    const uint32_t *list = P.list[KP];
    const uint32_t ntab = (uint32_t)P.ntab[KP];
    const uint32_t nb = PLAIN || !P.ccen ? ntab : ntab - (uint32_t)P.ncells;  // cells from here on
    const float2 e2 = splat2(P.eps2);
    constexpr int NP = kPointTile / 64, NE = 2 * NP;  // record pairs, records per lane
    // the word of an absent entry, told by its place and not by the word
    constexpr uint32_t kBody0 = NLN_SHIFT_NONE << NLN_IDX_BITS;
    for (;;) {
        int it = 0;
        if (lane == 0)
            it = atomicAdd(&P.counters[KP], 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= P.nitems[KP])
            break;
        const Item item = P.items[KP][it];
        const nln_group G = P.groups[item.group];
        const double c[3] = {PLAIN ? 0.0 : G.cen[0], PLAIN ? 0.0 : G.cen[1],
                             PLAIN ? 0.0 : G.cen[2]};
        auto fetch = [&](int64_t k0, uint32_t *e) {
#pragma unroll
            for (int j = 0; j < NE; j++) {
                const int64_t k = k0 + 32 * j + lane;
                e[j] = k < item.end ? __ldg(list + k) : kBody0;
            }
        };
        // Start this lane's copies of its entries' records.  Entries are
        // checked at upload, except in the pipelined end-to-end call: a bad
        // one becomes body 0 in the box's own image.
        auto copy = [&](int64_t k0, uint32_t *e) {
            const int n = (int)min((int64_t)kPointTile, item.end - k0);
            bool bad = false;
#pragma unroll
            for (int j = 0; j < NE; j++) {
                if (32 * j >= n)
                    break;
                if ((e[j] & NLN_IDX_MASK) >= ntab || (e[j] >> NLN_IDX_BITS) > 26u) {
                    bad = true;
                    e[j] = kBody0;
                }
                const uint32_t idx = e[j] & NLN_IDX_MASK;
                if (idx < nb) {
                    cp_async16(&stage.chunk[j][0][lane], P.points + idx);
                } else {
                    const unsigned char *r = P.ccen + (size_t)(idx - nb) * P.cstride;
                    cp_async16(&stage.chunk[j][0][lane], r);
                    cp_async16(&stage.chunk[j][1][lane], r + 16);
                }
            }
            cp_async_commit();
            if (bad)
                atomicOr(P.err, GC_DEV_BAD_INDEX);
        };
        uint32_t cur[NE], nxt[NE];
        fetch(item.begin, cur);
        copy(item.begin, cur);
        fetch(item.begin + kPointTile, nxt);
        stage_sinks(sinks, P, G, c, lane);
        Total acc;
        for (int64_t k0 = item.begin; k0 < item.end; k0 += kPointTile) {
            const int nt = (int)min((int64_t)kPointTile, item.end - k0);
            const int np = (nt + 63) >> 6;  // pairs in use
            MonoPair rec[NP];
            cp_async_wait<0>();  // this lane's records have landed
#pragma unroll
            for (int j = 0; j < NE; j++) {
                if ((j >> 2) > (np - 1) >> 1)
                    break;
                const bool live = 32 * j + lane < nt;
                const uint32_t idx = cur[j] & NLN_IDX_MASK;
                const uint32_t code = cur[j] >> NLN_IDX_BITS;
                const float4 u = stage.chunk[j][0][lane];
                double x = u.x, y = u.y, z = u.z;
                float m = u.w;
                if (idx >= nb) {
                    const float4 w = stage.chunk[j][1][lane];
                    x = __hiloint2double(__float_as_int(u.y), __float_as_int(u.x));
                    y = __hiloint2double(__float_as_int(u.w), __float_as_int(u.z));
                    z = __hiloint2double(__float_as_int(w.y), __float_as_int(w.x));
                    m = w.z;
                }
                float o[3];
                recentre(x, y, z, code, __any_sync(0xffffffffu, code != NLN_SHIFT_NONE), P.box, c,
                         o);
                set_half(rec[j >> 1].x, j & 1, live ? o[0] : kFar);
                set_half(rec[j >> 1].y, j & 1, live ? o[1] : kFar);
                set_half(rec[j >> 1].z, j & 1, live ? o[2] : kFar);
                set_half(rec[j >> 1].m, j & 1, live ? m : 0.f);
            }
            copy(k0 + kPointTile, nxt);
#pragma unroll
            for (int j = 0; j < NE; j++) cur[j] = nxt[j];
            fetch(k0 + 2 * kPointTile, nxt);
            // a tile of at most 128 records leaves out the other two pairs
            auto sums_of = [&](auto n) {
                sum_sinks<8>(sinks, G.count, lane, sums, acc, [&](const Sink &k) {
                    const float2 nx = f2(k.xy.x, k.xy.y), ny = f2(k.xy.z, k.xy.w), nz = k.z;
                    Sum2 A;
                    mono_pair<true>(rec[0], nx, ny, nz, e2, A);
#pragma unroll
                    for (int q = 1; q < decltype(n)::value; q++)
                        mono_pair<false>(rec[q], nx, ny, nz, e2, A);
                    return A.total();
                });
            };
            if (np > 2)
                sums_of(std::integral_constant<int, 4>());
            else
                sums_of(std::integral_constant<int, 2>());
        }
        store_part(P, item, lane, acc);
    }
    pdl_wait();
}

// Periodic correction moments (ewald.cuh) of groups gbegin..ngroups-1, one
// warp per unit from a queue (counter 3), lanes striding the unit's part of
// its group's correction list; a group has ewsplit units.  Bodies count as
// masses; a cell adds its traceless second to fourth moments (the list's cells
// include coarse ones standing for whole subtrees, and cells a tenth of the
// box wide near the half-box, where C varies on the scale of the cell), and
// its second-moment trace B2/3 against the constant Laplacian of C.

// Unit u of the moments' queue: group and tile range [t0, t1) of its list.
struct EwUnit {
    int64_t g, cb, ce;
    int t0, t1;
};

__device__ __forceinline__ EwUnit ew_unit(const DevProblem &P, int64_t u) {
    EwUnit r;
    const int part = (int)(u % P.ewsplit);
    r.g = P.gbegin + u / P.ewsplit;
    if (r.g >= P.ngroups)
        return r;
    r.cb = P.cptr[r.g];
    r.ce = P.cptr[r.g + 1];
    const int64_t nt = (r.ce - r.cb + 31) / 32;
    r.t0 = (int)(nt * part / P.ewsplit);
    r.t1 = (int)(nt * (part + 1) / P.ewsplit);
    return r;
}

// Store a unit's moments (already summed over the warp) as its group's, or,
// where the list is split, as a part: the warp that finishes the group's
// last unit adds the parts in order.
__device__ __forceinline__ void ew_store(const DevProblem &P, int64_t u, int64_t g, int lane,
                                         const EwSums &T) {
    EwStored *E = P.ewsplit > 1 ? P.ewpart + (g * P.ewsplit + u % P.ewsplit) : P.ewm + g;
    if (lane == 0) {
        const EwMoments M = T.full(P.ew.trace);
#pragma unroll
        for (int q = 0; q < 10; q++) E->lo[q] = M.lo[q];
#pragma unroll
        for (int q = 0; q < 25; q++) E->hi[q] = M.hi[q];
    }
    if (P.ewsplit == 1)
        return;
    __threadfence();
    int before = 0;
    if (lane == 0)
        before = atomicAdd(&P.ewdone[g], 1);
    if (__shfl_sync(0xffffffffu, before, 0) != P.ewsplit - 1)
        return;
    __threadfence();
    const EwStored *S = P.ewpart + g * P.ewsplit;
    EwStored &D = P.ewm[g];
    if (lane < 10) {
        double v = __ldcg(&S[0].lo[lane]);
        for (int k = 1; k < P.ewsplit; k++) v += __ldcg(&S[k].lo[lane]);
        D.lo[lane] = v;
    }
    if (lane < 25) {
        float v = __ldcg(&S[0].hi[lane]);
        for (int k = 1; k < P.ewsplit; k++) v += __ldcg(&S[k].hi[lane]);
        D.hi[lane] = v;
    }
    if (lane == 0)
        P.ewdone[g] = 0;
}

// Every entry needs its table node (144 B) and its cell record (112 of 128 B)
// from scattered addresses, and the node depends on the record's centre: list
// word three tiles ahead, the source's FP64 centre (plain loads) two tiles
// ahead, and one tile ahead the tile's 32 nodes and records by cp.async into
// one of two stages of the warp.  The warp copies them row by row, neighbour
// lanes neighbour chunks of a row: with each lane copying its own rows every
// instruction touched 32 cache lines and the L1's rate held the kernel (160^3
// box: 30.7 ms with the finish pass); TMA row gathers, the other way, cost 270
// of 1,500 instructions a tile to start (24.7 ms; now 13.9).  Rows of 9 and 7 chunks
// are read back without bank conflicts.
constexpr int kEwNodeChunks = ew::kNode / 4;   // 9
constexpr int kEwRecChunks = 7;                // floats 4..31 of nln_hcell
struct EwStage {
    float4 node[32 * kEwNodeChunks];
    float4 rec[32 * kEwRecChunks];
};
constexpr int kEwWarpBytes = 2 * (int)sizeof(EwStage);  // 16 KB

__global__ void __launch_bounds__(128) k_ewald_moments(DevProblem P) {
    extern __shared__ __align__(16) unsigned char ewsm[];
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    EwStage *stg = reinterpret_cast<EwStage *>(ewsm + (size_t)(threadIdx.x >> 5) * kEwWarpBytes);
    const uint32_t ntab = (uint32_t)P.ntab[0];
    const uint32_t nb = ntab - (uint32_t)P.ncells;
    constexpr uint32_t kNone = 0xffffffffu;
    // one source of the pipeline: list word (kNone: no entry in this lane)
    // and its position (FP64) with, for a body, its mass
    struct Src {
        uint32_t e;
        double x, y, z;
        float m;
    };
    // the entry whose rows are staged: its node and what kind it is
    struct Staged {
        EwNode N;
        bool live, cell;
        float m;
    };
    for (;;) {
        int it = 0;
        if (lane == 0)
            it = atomicAdd(&P.counters[3], 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        const EwUnit U = ew_unit(P, it);
        if (U.g >= P.ngroups)
            break;
        const nln_group G = P.groups[U.g];
        const double c[3] = {G.cen[0], G.cen[1], G.cen[2]};
        const int ntile = U.t1 - U.t0;
        // the list word is checked where it is used, a tile after its load
        auto entry = [&](int t) -> uint32_t {
            const int64_t k = U.cb + (int64_t)(U.t0 + t) * 32 + lane;
            return (t < ntile && k < U.ce) ? __ldg(P.clist + k) : kNone;
        };
        auto source = [&](uint32_t e, int t) -> Src {
            Src r{kNone, 0.0, 0.0, 0.0, 0.f};
            if (e == kNone) {
                if (t < ntile && U.cb + (int64_t)(U.t0 + t) * 32 + lane < U.ce)
                    atomicOr(P.err, GC_DEV_BAD_INDEX);
                return r;
            }
            const uint32_t idx = e & NLN_IDX_MASK;
            if (idx >= ntab || (e >> NLN_IDX_BITS) > 26u) {  // as in the list kernels
                atomicOr(P.err, GC_DEV_BAD_INDEX);
                return r;
            }
            r.e = e;
            if (idx < nb) {
                const float4 p = __ldg(P.points + idx);
                r.x = p.x;
                r.y = p.y;
                r.z = p.z;
                r.m = p.w;
            } else {
                const double *cen = P.hcells[idx - nb].cen;
                const double2 a = __ldg(reinterpret_cast<const double2 *>(cen));
                r.x = a.x;
                r.y = a.y;
                r.z = __ldg(cen + 2);
            }
            return r;
        };
        // Start the copies of a tile: chunk i of its 32 rows is chunk i % 9 (or
        // i % 7) of row i / 9 (or 7), whose lane names it.
        auto issue = [&](const Src &q, EwStage &S) -> Staged {
            Staged r;
            r.live = q.e != kNone;
            r.m = q.m;
            const uint32_t idx = q.e & NLN_IDX_MASK;
            r.cell = r.live && idx >= nb;
            int node = 0;
            if (r.live) {
                double sx, sy, sz;
                decode_shift(q.e >> NLN_IDX_BITS, P.box, sx, sy, sz);
                r.N = ew_node(P.ew, (float)(q.x + sx - c[0]), (float)(q.y + sy - c[1]),
                              (float)(q.z + sz - c[2]));
                node = r.N.node;
            }
            const unsigned live = __ballot_sync(0xffffffffu, r.live);
            const unsigned cells = __ballot_sync(0xffffffffu, r.cell);
            const int rec = r.cell ? (int)(idx - nb) : 0;
#pragma unroll
            for (int k = 0; k < kEwNodeChunks; k++) {
                const int i = 32 * k + lane, row = i / kEwNodeChunks;
                const int from = __shfl_sync(0xffffffffu, node, row);
                if (live >> row & 1u)
                    cp_async16(&S.node[i], P.ew.t + (size_t)from * ew::kNode + 4 * (i - row * kEwNodeChunks));
            }
            if (cells) {
#pragma unroll
                for (int k = 0; k < kEwRecChunks; k++) {
                    const int i = 32 * k + lane, row = i / kEwRecChunks;
                    const int from = __shfl_sync(0xffffffffu, rec, row);
                    if (cells >> row & 1u)
                        cp_async16(&S.rec[i], reinterpret_cast<const float4 *>(P.hcells + from) + 1 +
                                                  (i - row * kEwRecChunks));
                }
            }
            cp_async_commit();
            return r;
        };
        EwSums M;
        M.zero();
        Staged now = issue(source(entry(0), 0), stg[0]), next;
        Src s1 = source(entry(1), 1);
        uint32_t e2 = entry(2);
        for (int t = 0; t < ntile; t++) {
            __syncwarp();  // the other stage is no longer read
            next = issue(s1, stg[(t + 1) & 1]);
            s1 = source(e2, t + 2);  // consumed by the next tile's issue
            e2 = entry(t + 3);
            cp_async_wait<1>();  // this lane's copies for tile t have landed
            __syncwarp();        // and the other lanes'
            if (now.live) {
                const float4 *node = stg[t & 1].node + lane * kEwNodeChunks;
                const float4 *rec = stg[t & 1].rec + lane * kEwRecChunks - 1;
                ew_entry(M, P.ew.trace, now.N, now.cell, now.m, [&](int k) { return node[k]; },
                         [&](int k) { return rec[k]; });
            }
            now = next;
        }
        cp_async_wait<0>();
        __syncwarp();
        M.warp_sum();
        ew_store(P, it, U.g, lane, M);
    }
    pdl_wait();
}

// The same moments by a plain loop over the list, every load on demand: no
// shared memory, which suits a kernel that shares the SMs with the list
// kernels (the side stream).  The arithmetic and its order are
// k_ewald_moments', so the two store identical moments.
__global__ void __launch_bounds__(64) k_ewald_side(DevProblem P) {
    const int lane = threadIdx.x & 31;
    const uint32_t ntab = (uint32_t)P.ntab[0];
    const uint32_t nb = ntab - (uint32_t)P.ncells;
    for (;;) {
        int it = 0;
        if (lane == 0)
            it = atomicAdd(&P.counters[3], 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        const EwUnit U = ew_unit(P, it);
        if (U.g >= P.ngroups)
            break;
        const nln_group G = P.groups[U.g];
        EwSums M;
        M.zero();
        const int64_t end = min(U.ce, U.cb + (int64_t)U.t1 * 32);
        for (int64_t k = U.cb + (int64_t)U.t0 * 32 + lane; k < end; k += 32) {
            const uint32_t ent = P.clist[k];
            const uint32_t idx = ent & NLN_IDX_MASK;
            if (idx >= ntab || (ent >> NLN_IDX_BITS) > 26u) {  // as in the list kernels
                atomicOr(P.err, GC_DEV_BAD_INDEX);
                continue;
            }
            const bool cell = idx >= nb;
            double x, y, z;
            float m = 0.f;
            const float4 *rec = nullptr;
            if (cell) {
                const nln_hcell &h = P.hcells[idx - nb];
                x = h.cen[0];
                y = h.cen[1];
                z = h.cen[2];
                rec = reinterpret_cast<const float4 *>(&h);
            } else {
                const float4 p = P.points[idx];
                x = p.x;
                y = p.y;
                z = p.z;
                m = p.w;
            }
            double sx, sy, sz;
            decode_shift(ent >> NLN_IDX_BITS, P.box, sx, sy, sz);
            const EwNode N = ew_node(P.ew, (float)(x + sx - G.cen[0]), (float)(y + sy - G.cen[1]),
                                     (float)(z + sz - G.cen[2]));
            const float4 *node = reinterpret_cast<const float4 *>(P.ew.t + (size_t)N.node * ew::kNode);
            ew_entry(M, P.ew.trace, N, cell, m, [&](int q) { return __ldg(node + q); },
                     [&](int q) { return __ldg(rec + q); });
        }
        M.warp_sum();
        ew_store(P, it, U.g, lane, M);
    }
}

// Per group, in slot order: sum the partials of its work items in FP64,
// add the periodic correction, and write (ax, ay, az, phi) of each sink.
__global__ void k_finish(DevProblem P) {
    pdl_trigger();
    pdl_wait();
    if (blockIdx.x == 0 && threadIdx.x < 4)
        P.counters[threadIdx.x] = 0;  // the queues are done: the next evaluation starts at zero
    const int64_t g = P.gbegin + (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (g >= P.ngroups)
        return;
    const nln_group G = P.groups[g];
    double s[4] = {0, 0, 0, 0};
    for (int64_t k = P.gslot[g]; k < P.gslot[g + 1]; k++) {
        const float4 *src = P.part + ((size_t)k * 32 + lane) * 2;
        float4 h = src[0], l = src[1];
        s[0] += (double)h.x + (double)l.x;
        s[1] += (double)h.y + (double)l.y;
        s[2] += (double)h.z + (double)l.z;
        s[3] += (double)h.w + (double)l.w;
    }
    if (P.ewald) {
        const double c[3] = {G.cen[0], G.cen[1], G.cen[2]};
        EwMoments M;
        const EwStored &E = P.ewm[g];  // k_ewald_moments
#pragma unroll
        for (int q = 0; q < 10; q++) M.lo[q] = E.lo[q];
#pragma unroll
        for (int q = 0; q < 25; q++) M.hi[q] = E.hi[q];
        if (lane < G.count) {
            const float4 p = P.points[G.first + lane];
            double phi, ax, ay, az;
            ew_apply(M, (double)p.x - c[0], (double)p.y - c[1], (double)p.z - c[2], phi, ax, ay,
                     az);
            s[0] += ax;
            s[1] += ay;
            s[2] += az;
            s[3] += phi - (double)p.w * P.ew_self;
        }
    }
    if (lane < G.count)
        P.out[G.first + lane] = make_float4((float)s[0], (float)s[1], (float)s[2], (float)s[3]);
}

}  // namespace

// ------------------------------------------------------------ plan
struct grav_step_state;  // time-step state (step.cuh)
void step_state_free(grav_step_state *S);
void step_graph_reset(grav_step_state *S);
struct grav_adjoint_state;  // adjoint scratch (adjoint.cuh)
void adjoint_state_free(grav_adjoint_state *A);

struct grav_plan {
    grav_problem hp{};      // sizes and parameters (host pointers cleared)
    grav_tuning tune{};
    DevProblem dp{};
    std::vector<void *> allocs;
    int64_t counts[4] = {0, 0, 0, 0};
    int nsm = 148;
    int launches = 0;
    int64_t nslots = 0;
    CUtensorMap tmap[3];    // row-gather views of the quadrupole and order-4 tables
    int timing = 0;         // record events around each kernel of an evaluation
    cudaEvent_t ev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    std::vector<int64_t> lists_ptr[4];  // host copies of the P, Q, H (queue rebuilds) and
                                        // correction list offsets
    int64_t *order = nullptr;           // device-built plans: tree position -> input index
    bool plain = false;                 // plain FP32 kernels (grav_problem.precision = 1)
    int integrator = 0;                 // 0: Integrate, 1: CosmoIntegrate (step.cuh)
    bool queues_clear = false;          // dp.counters are zero once the enqueued work is done
    bool elsewhere = false;             // used on a stream that is not the default one
    bool evaluated = false;             // grav_groups_eval_CUDA has been enqueued (the
                                        // correction moments the adjoint reads are set)
    grav_step_state *step = nullptr;  // tree links, refit scratch and the step graph
    grav_adjoint_state *adj = nullptr;  // adjoint scratch
    // periodic: the side stream of k_ewald_moments, its fork/join events and
    // the per-group correction moments
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    EwStored *ewm = nullptr;
    // a table of cell centres of the plan's own (own_centres), filled from the cell table
    float4 *centres = nullptr;
    const unsigned char *centres_from = nullptr;
    int centres_stride = 0;
    void used_on(cudaStream_t st) { elsewhere = elsewhere || (st && st != cudaStreamLegacy); }
    // Group ranges of the work queue: items are sorted by cost within each
    // range, and chunk_item[k][c] is the first item of kind k in range c.
    // One range [0, ngroups) except in the pipelined end-to-end call.
    std::vector<int64_t> chunk_group;
    std::vector<int> chunk_item[3];
    cudaMemPool_t pool = nullptr;  // device buffers from this pool (the end-to-end call)
    // run-packed lists of the end-to-end call (P, Q, H, correction): device
    // words, their offsets and the plain offsets they unpack to
    uint32_t *zdev[4] = {nullptr, nullptr, nullptr, nullptr};
    const int64_t *zptr_dev[4] = {nullptr, nullptr, nullptr, nullptr};
    const int64_t *lptr_dev[4] = {nullptr, nullptr, nullptr, nullptr};
};

namespace {

// The row-gather view of a cell table: box = one full record (one row high,
// as the row gather requires), swizzled over the record's width
// (CellKind::chunk).
template <int KIND>
int encode_cells(CUtensorMap *m, const void *base, int64_t rows) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        GC_CHECK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
        if (!fn || q != cudaDriverEntryPointSuccess)
            return gc::set_status(-1, "cuTensorMapEncodeTiled unavailable");
        encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    constexpr uint32_t bytes = CellKind<KIND>::rec_bytes, w = bytes / 4;
    cuuint64_t dims[2] = {w, (cuuint64_t)rows};
    cuuint64_t strides[1] = {bytes};
    cuuint32_t box[2] = {w, 1};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void *>(base), dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        KIND == KH ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return gc::set_status(-1, "cuTensorMapEncodeTiled failed (%d) for %lld rows of %u bytes",
                              (int)r, (long long)rows, bytes);
    return 0;
}

// The table k_points reads FP64 cell centres and masses from, and its record size.
const unsigned char *cell_centres(const DevProblem &d, bool quad, int &stride) {
    stride = quad ? (int)sizeof(nln_qcell) : (int)sizeof(nln_hcell);
    return quad ? reinterpret_cast<const unsigned char *>(d.qcells)
                : reinterpret_cast<const unsigned char *>(d.hcells);
}

// A monopole's mass is the point table's.  The cell tables carry the same one
// in every problem that this library's builders make; where a caller's differ,
// k_points gets a table of its own (centre, mass, pad: 32 bytes a cell).
__global__ void k_masses_differ(const float4 *__restrict__ cells, const unsigned char *__restrict__ cen,
                                int stride, int64_t n, unsigned *differ) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool d = c < n && __float_as_uint(cells[c].w) !=
                                __float_as_uint(reinterpret_cast<const float *>(cen + c * stride)[6]);
    if (__any_sync(0xffffffffu, d) && (threadIdx.x & 31) == 0)
        atomicOr(differ, 1u);
}

__global__ void k_centre_table(const float4 *__restrict__ cells, const unsigned char *__restrict__ cen,
                               int stride, int64_t n, float4 *out) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n)
        return;
    const float4 *r = reinterpret_cast<const float4 *>(cen + c * stride);
    const float4 b = r[1];
    out[2 * c] = r[0];
    out[2 * c + 1] = make_float4(b.x, b.y, cells[c].w, 0.f);
}

template <typename T>
int dev_copy(grav_plan *pl, const T *src, size_t n, T **dst);

// dev_copy whose copy is asynchronous on the default stream when `async`
// (the end-to-end call's pool allocations are ordered on that stream).
template <typename T>
int dev_copy(grav_plan *pl, bool async, const T *src, size_t n, T **dst) {
    if (!async || !pl->pool)
        return dev_copy(pl, src, n, dst);
    if (int rc = dev_copy<T>(pl, nullptr, n, dst))
        return rc;
    if (src && n)
        GC_CHECK(cudaMemcpyAsync(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice, 0));
    return 0;
}

template <typename T>
int dev_copy(grav_plan *pl, const T *src, size_t n, T **dst) {
    *dst = nullptr;
    if (n == 0)
        return 0;
    if (pl->pool)
        GC_CHECK(gc::pool_malloc((void **)dst, n * sizeof(T), pl->pool, 0));
    else
        GC_CHECK(cudaMalloc((void **)dst, n * sizeof(T)));
    pl->allocs.push_back(*dst);
    if (src)
        GC_CHECK(cudaMemcpy(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice));
    return 0;
}

// After a refit too (its cell masses are the point table's own).
int fill_centres(grav_plan *pl, cudaStream_t st) {
    const int64_t nc = pl->dp.ncells;
    k_centre_table<<<(unsigned)((nc + 255) / 256), 256, 0, st>>>(
        pl->dp.points + pl->hp.nbodies, pl->centres_from, pl->centres_stride, nc, pl->centres);
    GC_CHECK(cudaGetLastError());
    return 0;
}

// d.ccen set: where its masses are not the point table's, a table of the
// plan's own takes its place.  The error word, still unused, carries the answer.
int own_centres(grav_plan *pl, int64_t nc) {
    DevProblem &d = pl->dp;
    unsigned differ = 0;
    k_masses_differ<<<(unsigned)((nc + 255) / 256), 256>>>(d.points + pl->hp.nbodies, d.ccen, d.cstride,
                                                           nc, d.err);
    GC_CHECK(cudaGetLastError());
    GC_CHECK(cudaMemcpy(&differ, d.err, sizeof(differ), cudaMemcpyDeviceToHost));
    if (!differ)
        return 0;
    GC_CHECK(cudaMemset(d.err, 0, sizeof(unsigned)));
    if (int rc = dev_copy<float4>(pl, nullptr, (size_t)nc * 2, &pl->centres))
        return rc;
    pl->centres_from = d.ccen;
    pl->centres_stride = d.cstride;
    d.ncells = nc;
    d.ccen = reinterpret_cast<const unsigned char *>(pl->centres);
    d.cstride = 2 * (int)sizeof(float4);
    return fill_centres(pl, 0);
}

// Defaults: 8 warps per block, which the list kernels run as blocks of four,
// as many resident as registers and shared memory allow (blocks_per_sm = 0),
// list chunks sized automatically
// (chunk_* = 0) from the totals once the lists are known.
grav_tuning default_tuning() {
    grav_tuning t;
    t.warps_per_block = 8;
    t.blocks_per_sm = 0;
    t.chunk_p = t.chunk_q = t.chunk_h = 0;
    t.ewald_n = 0;
    t.ewald_side = 0;
    return t;
}

// Split lists so that there are at least ~8 work items per resident warp
// (about 148 SMs x 16 warps), in whole tiles: shorter items spend more on
// their start than the idle warps are worth (8,000 bodies: 43 us a point
// kernel in items of 64 or 128, 33 us in tiles of 256).
int auto_chunk(int64_t total, int64_t ngroups, int nsm, int kind) {
    const int64_t warps = (int64_t)nsm * 16;
    int64_t ng = std::max<int64_t>(ngroups, 1);
    int64_t per = std::max<int64_t>(1, (8 * warps + ng - 1) / ng);
    int64_t avg = std::max<int64_t>(1, total / ng);
    const int64_t tile = kTile[kind];
    const int64_t c = (std::max<int64_t>(tile, avg / per) + tile - 1) / tile * tile;
    return (int)std::min<int64_t>(1 << 24, c);
}

// Work items of a plan from its kept list offsets and tuning: created group
// by group (slot order: a group's point items, then quadrupole, then order 4),
// then ordered per kind by cost, longest first, within each of the plan's
// group ranges (chunk_group; the whole set when empty).  Every item but a
// group's last of a kind is a full chunk, so the order is the full chunks in
// creation order, then the remainders by length (both stable).
int64_t make_queue(grav_plan *pl, std::vector<Item> items[3], std::vector<int64_t> &gslot) {
    const int64_t ng = pl->hp.ngroups;
    const int64_t chunk[3] = {pl->tune.chunk_p, pl->tune.chunk_q, pl->tune.chunk_h};
    if (pl->chunk_group.size() < 2)
        pl->chunk_group = {0, ng};
    const int nc = (int)pl->chunk_group.size() - 1;
    const int64_t *ptr[3];
    for (int k = 0; k < 3; k++) ptr[k] = pl->lists_ptr[k].empty() ? nullptr : pl->lists_ptr[k].data();
    // items per group and kind, then their first index and slot by prefix sums
    std::vector<int64_t> first[3];
    for (int k = 0; k < 3; k++) first[k].assign(ng + 1, 0);
    gslot.assign(ng + 1, 0);
#pragma omp parallel for schedule(static)
    for (int64_t g = 0; g < ng; g++) {
        int64_t all = 0;
        for (int k = 0; k < 3; k++) {
            const int64_t n = ptr[k] ? (ptr[k][g + 1] - ptr[k][g] + chunk[k] - 1) / chunk[k] : 0;
            first[k][g + 1] = n;
            all += n;
        }
        gslot[g + 1] = all;
    }
    for (int64_t g = 0; g < ng; g++) {
        for (int k = 0; k < 3; k++) first[k][g + 1] += first[k][g];
        gslot[g + 1] += gslot[g];
    }
    for (int k = 0; k < 3; k++) items[k].resize((size_t)first[k][ng]);
#pragma omp parallel for schedule(static)
    for (int64_t g = 0; g < ng; g++) {
        int32_t slot = (int32_t)gslot[g];
        for (int k = 0; k < 3; k++) {
            if (!ptr[k])
                continue;
            Item *out = items[k].data() + first[k][g];
            for (int64_t b = ptr[k][g]; b < ptr[k][g + 1]; b += chunk[k])
                *out++ = Item{(int32_t)g, slot++, b, std::min(ptr[k][g + 1], b + chunk[k])};
        }
    }
    for (int k = 0; k < 3; k++) {
        pl->chunk_item[k].resize(nc + 1);
        for (int c = 0; c <= nc; c++) pl->chunk_item[k][c] = (int)first[k][pl->chunk_group[c]];
    }
#pragma omp parallel for schedule(dynamic, 1)
    for (int task = 0; task < 3 * nc; task++) {
        const int k = task % 3, c = task / 3;
        auto b = items[k].begin() + pl->chunk_item[k][c], e = items[k].begin() + pl->chunk_item[k][c + 1];
        const int64_t full = chunk[k];
        auto mid = std::stable_partition(b, e, [full](const Item &x) { return x.end - x.begin == full; });
        std::stable_sort(mid, e, [](const Item &x, const Item &y) {
            return (x.end - x.begin) > (y.end - y.begin);
        });
    }
    return gslot[ng];
}

// The device address of page-locked host memory (lists read in place over
// PCIe), or null when `p` is not page-locked host memory.
const uint32_t *mapped_host(const uint32_t *p) {
    cudaPointerAttributes a{};
    if (!p || cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return a.type == cudaMemoryTypeHost ? static_cast<const uint32_t *>(a.devicePointer) : nullptr;
}

}  // namespace

namespace {
// The upload.  With nchunks > 0 (the pipelined end-to-end call) the list
// buffers are allocated but not filled: the caller copies each group range's
// lists while the kernels evaluate the previous range, and the kernels'
// own index checks stand in for the upload-time list check.
thread_local double t_phase[5];  // grav_groups_CUDA_phases
thread_local double t_build = 0, t_build_phase[6] = {0, 0, 0, 0, 0, 0};  // grav_plan_build_phases
thread_local double t_phase_be[4] = {0, 0, 0, 0};  // grav_build_eval_phases

// The end-to-end call's device buffers come from a pool per device that
// keeps freed memory reserved (until grav_groups_release_CUDA): mapping and
// unmapping tens of gigabytes in every call costs as much as the
// evaluation's tail.
constexpr int kMaxPoolDevices = 64;
std::mutex g_pool_mu;
cudaMemPool_t g_pool[kMaxPoolDevices] = {};

double now_s() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch())
        .count();
}

int e2e_pool(cudaMemPool_t *out) {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    int dev = 0;
    GC_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxPoolDevices)
        return gc::set_status(-1, "grav_groups_CUDA: device %d beyond %d", dev, kMaxPoolDevices);
    if (!g_pool[dev]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        GC_CHECK(cudaMemPoolCreate(&g_pool[dev], &props));
        uint64_t keep = UINT64_MAX;
        GC_CHECK(cudaMemPoolSetAttribute(g_pool[dev], cudaMemPoolAttrReleaseThreshold, &keep));
    }
    *out = g_pool[dev];
    return 0;
}

// adopt: a tree built on the device (gpu_tree_build) whose tables and lists
// the plan takes over instead of copying; hp then holds its host copies of
// the groups and offsets and device pointers to everything else.
int upload_impl(const grav_problem *hp, const grav_tuning *tuning, grav_plan **plan_out,
                int nchunks, const DevTree *adopt = nullptr) {
    *plan_out = nullptr;
    const double t_start = now_s();
    if (!hp || hp->nbodies <= 0 || hp->ngroups <= 0 || !hp->points || !hp->groups ||
        !hp->pptr || (!hp->plist && !(nchunks > 0 && hp->zlist[0])))
        return gc::set_status(-1, "grav_groups_upload_CUDA: incomplete problem");
    if (hp->nbodies + hp->ncells >= (int64_t)NLN_IDX_MASK)
        return gc::set_status(-1, "grav_groups_upload_CUDA: point table exceeds 27-bit indices");
    if (hp->precision != 0 && hp->precision != 1)
        return gc::set_status(-1, "grav_groups_upload_CUDA: precision must be 0 (mixed) or 1 "
                                  "(plain FP32)");
    grav_plan *pl = new grav_plan();
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&pl->nsm, cudaDevAttrMultiProcessorCount, dev);
    pl->hp = *hp;
    pl->plain = hp->precision == 1;
    if (adopt) {
        pl->pool = adopt->pool;  // freed the way they were allocated
        // the plan owns every buffer of the device-built tree from here on,
        // failures included (grav_plan_free releases them)
        void *own[] = {adopt->points, adopt->qcells, adopt->hcells, adopt->groups,
                       adopt->list[0], adopt->list[1], adopt->list[2], adopt->list[3],
                       adopt->order, adopt->ptr[0], adopt->ptr[1], adopt->ptr[2], adopt->ptr[3]};
        for (void *q : own)
            if (q)
                pl->allocs.push_back(q);
        pl->order = adopt->order;
    }
    pl->tune = tuning ? *tuning : default_tuning();
    const int64_t ng = hp->ngroups, nb = hp->nbodies, np = hp->nbodies + hp->ncells;
    const bool deferred = nchunks > 0;
    if (deferred && hp->lists_in_host) {
        grav_plan_free(pl);
        return gc::set_status(-1, "upload: deferred lists and lists_in_host exclude each other");
    }
    if (deferred) {
        if (int e = e2e_pool(&pl->pool)) {
            grav_plan_free(pl);
            return e;
        }
    }

    // validate everything the kernels will index
    int bad_group = 0;
    double span = 0;
#pragma omp parallel for schedule(static) reduction(| : bad_group) reduction(max : span)
    for (int64_t g = 0; g < ng; g++) {
        const nln_group &G = hp->groups[g];
        span = std::max(span, group_span(G, hp->groups[0]));
        if (G.count < 1 || G.count > 32 || G.first < 0 || G.first + G.count > nb)
            bad_group |= 1;
        if (hp->pptr[g + 1] < hp->pptr[g] || (hp->qptr && hp->qptr[g + 1] < hp->qptr[g]) ||
            (hp->hptr && hp->hptr[g + 1] < hp->hptr[g]))
            bad_group |= 1;
    }
    if (hp->pptr[0] != 0 || (hp->qptr && hp->qptr[0] != 0) || (hp->hptr && hp->hptr[0] != 0))
        bad_group |= 1;
    if (bad_group) {
        grav_plan_free(pl);
        return gc::set_status(-1, "a group has 0 or more than 32 sinks, lies outside the bodies, "
                                  "or has list offsets that decrease or do not start at 0");
    }
    // Every list entry is checked on the device: after the upload (k_check_lists),
    // or by the kernels as they read it (deferred lists, lists_in_host).  A host
    // pass over tens of gigabytes of lists would dominate an end-to-end call.
    const int64_t *eptr = hp->pptr;
    if ((hp->qptr && hp->qptr[ng] && (!hp->qcells || hp->ncells <= 0)) ||
        (hp->hptr && hp->hptr[ng] && (!hp->hcells || hp->ncells <= 0))) {
        grav_plan_free(pl);
        return gc::set_status(-1, "a cell list without its cell table");
    }
    const bool want_ewald = hp->box > 0 && hp->ewald;
    if (want_ewald) {
        if (!hp->cptr || (!hp->clist && !(deferred && hp->zlist[3])) ||
            (hp->ncells > 0 && !hp->hcells)) {
            grav_plan_free(pl);
            return gc::set_status(-1, "the Ewald correction needs the correction list and the "
                                      "order-4 cell table");
        }
        int bad = 0;
#pragma omp parallel for schedule(static) reduction(| : bad)
        for (int64_t g = 0; g < ng; g++)
            if (hp->cptr[g + 1] < hp->cptr[g])
                bad |= 1;
        if (bad || hp->cptr[0] != 0) {
            grav_plan_free(pl);
            return gc::set_status(-1, "bad correction list offsets");
        }
    }
    // run-packed lists (the end-to-end call): offsets from 0, never decreasing
    const int64_t *plain_ptr[4] = {hp->pptr, hp->qptr, hp->hptr, want_ewald ? hp->cptr : nullptr};
    bool packed[4] = {false, false, false, false};
    if (deferred) {
        for (int k = 0; k < 4; k++) {
            if (!hp->zlist[k] || !plain_ptr[k] || plain_ptr[k][ng] == 0)
                continue;
            const int64_t *z = hp->zptr[k];
            int bad = !z || z[0] != 0;
            if (!bad) {
#pragma omp parallel for schedule(static) reduction(| : bad)
                for (int64_t g = 0; g < ng; g++)
                    if (z[g + 1] < z[g])
                        bad |= 1;
            }
            if (bad) {
                grav_plan_free(pl);
                return gc::set_status(-1, "bad run-packed list offsets (kind %d)", k);
            }
            packed[k] = true;
        }
        if (!hp->plist && !packed[0]) {
            grav_plan_free(pl);
            return gc::set_status(-1, "grav_groups_CUDA: no point list");
        }
    }

    // The tables go first: in the end-to-end call (pool allocations, stream
    // ordered) their copies are asynchronous and overlap the work queue's
    // host build below; the upload's later copies and its final
    // synchronisation order everything before the kernels start.
    DevProblem &d = pl->dp;
    int rc = 0;
    float4 *pts = nullptr;
    nln_qcell *qc = nullptr;
    nln_hcell *hc = nullptr;
    nln_group *gr = nullptr;
    const bool want_q = hp->qptr && hp->qptr[ng];
    const bool want_h = (hp->hptr && hp->hptr[ng]) || (want_ewald && hp->ncells > 0);
    if (adopt) {
        pts = adopt->points;
        qc = want_q ? adopt->qcells : nullptr;
        hc = want_h ? adopt->hcells : nullptr;
        gr = adopt->groups;
    } else {
        rc |= dev_copy(pl, deferred, reinterpret_cast<const float4 *>(hp->points), (size_t)np,
                       &pts);
        if (want_q)
            rc |= dev_copy(pl, deferred, hp->qcells, (size_t)hp->ncells, &qc);
        if (want_h)
            rc |= dev_copy(pl, deferred, hp->hcells, (size_t)hp->ncells, &hc);
        rc |= dev_copy(pl, deferred, hp->groups, (size_t)ng, &gr);
    }
    d.points = pts;
    d.qcells = qc;
    d.hcells = hc;
    d.groups = gr;
    if (pl->tune.warps_per_block < 1 || pl->tune.warps_per_block > 8)
        pl->tune.warps_per_block = 8;
    if (pl->tune.chunk_p <= 0)
        pl->tune.chunk_p = auto_chunk(eptr[ng], ng, pl->nsm, KP);
    if (pl->tune.chunk_q <= 0)
        pl->tune.chunk_q = auto_chunk(hp->qptr ? hp->qptr[ng] : 0, ng, pl->nsm, KQ);
    if (pl->tune.chunk_h <= 0)
        pl->tune.chunk_h = auto_chunk(hp->hptr ? hp->hptr[ng] : 0, ng, pl->nsm, KH);

    // work items, created group by group (slot order), then sorted per kind by cost
    std::vector<Item> items[3];
    std::vector<int64_t> gslot;
    const int64_t *ptrs[4] = {eptr, hp->qptr, hp->hptr, want_ewald ? hp->cptr : nullptr};
    for (int k = 0; k < 4; k++)
        if (ptrs[k])
            pl->lists_ptr[k].assign(ptrs[k], ptrs[k] + ng + 1);
    if (deferred) {
        // group ranges holding about equal list bytes
        auto bytes_to = [&](int64_t g) {
            int64_t b = eptr[g];
            if (hp->qptr)
                b += hp->qptr[g];
            if (hp->hptr)
                b += hp->hptr[g];
            if (want_ewald)
                b += hp->cptr[g];
            return b;
        };
        // The first range's copy is not overlapped: split it further into
        // 1/8, 1/8, 1/4 and 1/2 of an equal share.
        const int64_t total = std::max<int64_t>(1, bytes_to(ng));
        std::vector<int64_t> wants;
        if (nchunks > 1)
            for (int d : {8, 4, 2}) wants.push_back(total / ((int64_t)nchunks * d));
        for (int c = 1; c < nchunks; c++) wants.push_back(total * c / nchunks);
        pl->chunk_group.assign(1, 0);
        int64_t g = 0;
        for (const int64_t want : wants) {
            int64_t lo = g, hi = ng;  // first group whose prefix reaches `want`
            while (lo < hi) {
                const int64_t mid = (lo + hi) / 2;
                if (bytes_to(mid) < want)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            g = lo;
            if (g > pl->chunk_group.back() && g < ng)
                pl->chunk_group.push_back(g);
        }
        pl->chunk_group.push_back(ng);
    }
    if (!adopt)
        pl->nslots = make_queue(pl, items, gslot);
    else
        pl->chunk_group = {0, ng};

    // interaction counts (sinks x sources); the point list's split into
    // bodies and cell monopoles is counted on the device (k_check_lists)
    for (int64_t g = 0; g < ng; g++) {
        const int64_t c = hp->groups[g].count;
        if (hp->qptr)
            pl->counts[2] += c * (hp->qptr[g + 1] - hp->qptr[g]);
        if (hp->hptr)
            pl->counts[3] += c * (hp->hptr[g + 1] - hp->hptr[g]);
    }

    t_phase[0] = now_s() - t_start;
    const double t_dev = now_s();
    uint32_t *l0 = nullptr, *l1 = nullptr, *l2 = nullptr, *all_clist = nullptr;
    if (deferred) {
        // one buffer for the four lists, filled range by range by the caller
        const size_t n[4] = {(size_t)hp->pptr[ng], hp->qptr ? (size_t)hp->qptr[ng] : 0,
                             hp->hptr ? (size_t)hp->hptr[ng] : 0,
                             want_ewald ? (size_t)std::max<int64_t>(1, hp->cptr[ng]) : 0};
        size_t off[4], words = 0;
        for (int k = 0; k < 4; k++) {
            off[k] = words;
            words += (n[k] + 63) / 64 * 64;
        }
        uint32_t *all = nullptr;
        rc |= dev_copy<uint32_t>(pl, nullptr, words, &all);
        if (all) {
            l0 = n[0] ? all + off[0] : nullptr;
            l1 = n[1] ? all + off[1] : nullptr;
            l2 = n[2] ? all + off[2] : nullptr;
            all_clist = n[3] ? all + off[3] : nullptr;
        }
        // packed kinds: device words (filled range by range) and both offset arrays
        for (int k = 0; k < 4; k++) {
            if (!packed[k])
                continue;
            uint32_t *zw = nullptr;
            int64_t *zp = nullptr, *lp = nullptr;
            rc |= dev_copy<uint32_t>(pl, nullptr, (size_t)std::max<int64_t>(1, hp->zptr[k][ng]), &zw);
            rc |= dev_copy(pl, hp->zptr[k], (size_t)ng + 1, &zp);
            rc |= dev_copy(pl, plain_ptr[k], (size_t)ng + 1, &lp);
            pl->zdev[k] = zw;
            pl->zptr_dev[k] = zp;
            pl->lptr_dev[k] = lp;
        }
    } else if (adopt) {
        l0 = adopt->list[0];
        l1 = hp->qptr ? adopt->list[1] : nullptr;
        l2 = hp->hptr ? adopt->list[2] : nullptr;
    } else if (hp->lists_in_host) {
        // the kernels read the lists in place from page-locked host memory
        const uint32_t *m0 = mapped_host(hp->plist);
        const uint32_t *m1 = hp->qptr ? mapped_host(hp->qlist) : nullptr;
        const uint32_t *m2 = hp->hptr ? mapped_host(hp->hlist) : nullptr;
        if (!m0 || (hp->qptr && !m1) || (hp->hptr && !m2)) {
            grav_plan_free(pl);
            return gc::set_status(-1, "grav_groups_upload_CUDA: lists_in_host needs the lists in "
                                      "page-locked host memory (cudaHostAlloc)");
        }
        l0 = const_cast<uint32_t *>(m0);
        l1 = const_cast<uint32_t *>(m1);
        l2 = const_cast<uint32_t *>(m2);
    } else {
        rc |= dev_copy(pl, hp->plist, (size_t)hp->pptr[ng], &l0);
        if (hp->qptr)
            rc |= dev_copy(pl, hp->qlist, (size_t)hp->qptr[ng], &l1);
        if (hp->hptr)
            rc |= dev_copy(pl, hp->hlist, (size_t)hp->hptr[ng], &l2);
    }
    d.list[0] = l0;
    d.list[1] = l1;
    d.list[2] = l2;
    d.ntab[0] = np;
    d.ntab[1] = d.ntab[2] = hp->ncells;
    int64_t *gs = nullptr;
    if (adopt) {
        // the offsets are on the device: so is the queue made there (96^3 box: 3.9 ms on the
        // host with its copies, 0.3 ms)
        const int64_t *const dptr[3] = {adopt->ptr[0], adopt->ptr[1], adopt->ptr[2]};
        const int64_t chunk[3] = {pl->tune.chunk_p, pl->tune.chunk_q, pl->tune.chunk_h};
        Item *it[3];
        rc |= gpu_make_queue(dptr, ng, chunk, 0, pl->pool, it, d.nitems, &gs, &pl->nslots);
        for (int k = 0; k < 3; k++) {
            d.items[k] = it[k];
            if (it[k])
                pl->allocs.push_back(it[k]);
            pl->chunk_item[k] = {0, d.nitems[k]};
        }
        if (gs)
            pl->allocs.push_back(gs);
    } else {
        for (int k = 0; k < 3; k++) {
            Item *it = nullptr;
            rc |= dev_copy(pl, items[k].data(), items[k].size(), &it);
            d.items[k] = it;
            d.nitems[k] = (int)items[k].size();
        }
        rc |= dev_copy(pl, gslot.data(), gslot.size(), &gs);
    }
    int *ctr = nullptr;  // 4 queue heads per group range
    rc |= dev_copy<int>(pl, nullptr, 4 * (pl->chunk_group.size() - 1), &ctr);
    d.counters = ctr;
    float4 *part = nullptr;
    rc |= dev_copy<float4>(pl, nullptr, (size_t)std::max<int64_t>(1, pl->nslots) * 64, &part);
    d.part = part;
    d.gslot = gs;
    d.cptr = nullptr;
    d.clist = nullptr;
    if (want_ewald) {
        int64_t *cp = nullptr;
        uint32_t *cl = nullptr;
        if (adopt)
            cp = adopt->ptr[3];
        else
            rc |= dev_copy(pl, hp->cptr, (size_t)ng + 1, &cp);
        if (hp->lists_in_host) {
            cl = const_cast<uint32_t *>(mapped_host(hp->clist));
            if (!cl) {
                grav_plan_free(pl);
                return gc::set_status(-1, "grav_groups_upload_CUDA: lists_in_host needs the "
                                          "correction list in page-locked host memory");
            }
        } else if (deferred) {
            cl = all_clist;
        } else if (adopt) {
            cl = adopt->list[3];
        } else {
            rc |= dev_copy(pl, hp->clist, (size_t)std::max<int64_t>(1, hp->cptr[ng]), &cl);
        }
        d.cptr = cp;
        d.clist = cl;
    }
    d.ewald = 0;
    if (want_ewald) {
        // FP64 table on the host, FP32 copy on the device
        const int n = pl->tune.ewald_n > 1 ? pl->tune.ewald_n : 32;
        // the table depends only on (box, n): build it once per process, with its FP32 values
        static std::mutex cache_mu;
        static double cache_box = 0, cache_c0 = 0;
        static int cache_n = 0;
        static std::vector<float> t32;
        float *tab = nullptr;
        double c0 = 0;
        {
            std::lock_guard<std::mutex> lk(cache_mu);
            if (cache_box != hp->box || cache_n != n) {
                std::vector<double> t64((size_t)n * n * n * NLN_EWALD_NQ, 0.0);
                if (ewald_table(hp->box, n, NLN_EWALD_REACH, t64.data())) {
                    grav_plan_free(pl);
                    return gc::set_status(-1, "Ewald table build failed");
                }
                t32.resize((size_t)n * n * n * ew::kNode);
                for (size_t node = 0; node < (size_t)n * n * n; node++)
                    for (int l = 0; l <= 5; l++)
                        for (int az = 0; az <= (l ? 1 : 0); az++)
                            for (int ay = 0; ay <= l - az; ay++)
                                t32[node * ew::kNode + ew::hidx(l - az - ay, ay, az)] =
                                    (float)t64[node * NLN_EWALD_NQ + ew::idx(l - az - ay, ay, az)];
                cache_c0 = t64[0];
                cache_box = hp->box;
                cache_n = n;
            }
            c0 = cache_c0;
            rc |= dev_copy(pl, t32.data(), t32.size(), &tab);
        }
        const double h = NLN_EWALD_REACH * hp->box / (n - 1);
        d.ew = EwTab{tab, n, (float)h, (float)(1.0 / h),
                     (float)(-4.0 * M_PI / (hp->box * hp->box * hp->box))};
        const double alpha = 2.0 / hp->box;
        d.ew_self = (float)(c0 - M_PI / (alpha * alpha * hp->box * hp->box * hp->box));
        d.ewald = 1;
        rc |= dev_copy<EwStored>(pl, nullptr, (size_t)ng, &pl->ewm);
        // Lists are split until there are 40 units per SM, more than three for
        // each of its 12 resident warps, but not below 8 tiles a unit: a 16^3 box
        // has 130 groups for 1,776 warps (moments 0.16 -> 0.07 ms), a 64^3 box
        // enough as it is.
        const int64_t tiles = hp->cptr[ng] / (32 * ng);
        d.ewsplit = (int)std::max<int64_t>(1, std::min<int64_t>((40 * (int64_t)pl->nsm + ng - 1) / ng,
                                                                tiles / 8));
        if (d.ewsplit > 1) {
            rc |= dev_copy<EwStored>(pl, nullptr, (size_t)(ng * d.ewsplit), &d.ewpart);
            rc |= dev_copy<int>(pl, nullptr, (size_t)ng, &d.ewdone);
            if (d.ewdone)
                cudaMemset(d.ewdone, 0, (size_t)ng * sizeof(int));
        }
        cudaError_t e = cudaStreamCreateWithFlags(&pl->side, cudaStreamNonBlocking);
        if (e == cudaSuccess)
            e = cudaEventCreateWithFlags(&pl->fork, cudaEventDisableTiming);
        if (e == cudaSuccess)
            e = cudaEventCreateWithFlags(&pl->join, cudaEventDisableTiming);
        if (e != cudaSuccess)
            rc |= gc::cuda_status(e, "upload: side stream");
    }
    float4 *out = nullptr;
    rc |= dev_copy<float4>(pl, nullptr, (size_t)nb, &out);
    d.out = out;
    unsigned *err = nullptr;
    rc |= dev_copy<unsigned>(pl, nullptr, 1, &err);
    d.err = err;
    if (rc) {
        grav_plan_free(pl);
        return rc;
    }
    cudaMemset(err, 0, sizeof(unsigned));
    if (adopt) {
        // lists from the device builder, which sized and checked them itself
        for (int k = 0; k < 4; k++) pl->counts[k] = adopt->counts[k];
    } else if (hp->lists_in_host || deferred) {
        // entries are checked by the kernels as they read them (bad ones set
        // the error word); the point list's body/cell split is not counted
        int64_t tot = 0;
        for (int64_t g = 0; g < ng; g++) tot += (int64_t)hp->groups[g].count * (hp->pptr[g + 1] - hp->pptr[g]);
        pl->counts[0] = tot;
        pl->counts[1] = 0;
    } else {
        // check every list entry on the device and count the point list's split
        unsigned long long *acc = nullptr;
        rc |= dev_copy<unsigned long long>(pl, nullptr, 3, &acc);
        if (rc) {
            grav_plan_free(pl);
            return rc;
        }
        cudaMemset(acc, 0, 3 * sizeof(unsigned long long));
        const unsigned blocks = (unsigned)pl->nsm * 8;
        const uint32_t ntabs[3] = {(uint32_t)np, (uint32_t)hp->ncells, (uint32_t)hp->ncells};
        for (int k = 0; k < 3; k++)
            if (d.nitems[k] > 0)
                k_check_lists<<<blocks, 256>>>(d.list[k], d.items[k], d.nitems[k], nullptr, 0,
                                                d.groups, ntabs[k], (uint32_t)nb, k == KP, acc);
        if (d.cptr)
            k_check_lists<<<blocks, 256>>>(d.clist, nullptr, 0, d.cptr, ng, d.groups, (uint32_t)np,
                                            (uint32_t)nb, 0, acc);
        unsigned long long h[3] = {0, 0, 0};
        const cudaError_t e = cudaMemcpy(h, acc, sizeof(h), cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) {
            grav_plan_free(pl);
            return gc::cuda_status(e, "grav_groups_upload_CUDA: list check");
        }
        if (h[0]) {
            grav_plan_free(pl);
            return gc::set_status(-1, "a list entry lies outside its table or has an image code "
                                      "beyond 26");
        }
        pl->counts[0] = (int64_t)h[1];
        pl->counts[1] = (int64_t)h[2];
    }
    memset(pl->tmap, 0, sizeof(pl->tmap));
    const bool has_q = d.qcells && hp->qptr && hp->qptr[ng];
    const bool has_h = d.hcells && hp->hptr && hp->hptr[ng];
    d.ccen = has_q || has_h ? cell_centres(d, has_q, d.cstride) : nullptr;
    if (d.ccen && !adopt && !pl->plain)
        rc |= own_centres(pl, np - nb);
    if (has_q)
        rc |= encode_cells<KQ>(&pl->tmap[KQ], d.qcells, hp->ncells);
    if (has_h)
        rc |= encode_cells<KH>(&pl->tmap[KH], d.hcells, hp->ncells);
    if (rc) {
        grav_plan_free(pl);
        return rc;
    }
    d.ngroups = ng;
    d.ncells = hp->ncells;
    d.eps2 = (float)hp->eps2;
    d.qsh = 0.5f * (hp->quad_phi_sign == 0.0f ? 1.0f : hp->quad_phi_sign);
    d.box = hp->box;
    d.hscale = length_scale(span);
    pl->hp.points = nullptr;
    pl->hp.qcells = nullptr;
    pl->hp.hcells = nullptr;
    pl->hp.groups = nullptr;
    pl->hp.pptr = pl->hp.qptr = pl->hp.hptr = nullptr;
    pl->hp.plist = nullptr;
    pl->hp.qlist = pl->hp.hlist = nullptr;
    // pool allocations, cleared words and copies on the default stream: complete
    // before other streams, which do not wait for it, use them
    if (const cudaError_t e = cudaStreamSynchronize(0); e != cudaSuccess) {
        grav_plan_free(pl);
        return gc::cuda_status(e, "upload: default stream");
    }
    *plan_out = pl;
    t_phase[1] = now_s() - t_dev;
    return 0;
}
}  // namespace

extern "C" int grav_groups_upload_CUDA(const grav_problem *hp, const grav_tuning *tuning,
                                       grav_plan **plan_out) {
    return upload_impl(hp, tuning, plan_out, 0);
}

namespace {
// The kernels of one evaluation do not read one another's results, but for
// the finish pass: with `after` a kernel may start as soon as every block of
// the one before it on the stream has, and fill the SMs that one's last wave
// leaves (2,000 bodies: 26.5 -> 16.5 us an evaluation).  Each waits for its
// predecessor before it ends, so the last one's end is the end of all.
int launch_after(const void *kern, unsigned blocks, unsigned threads, size_t smem, cudaStream_t st,
                 bool after, void **args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = after ? 1 : 0;
    GC_CHECK(cudaLaunchKernelExC(&cfg, kern, args));
    return 0;
}

// Where an evaluation's next kernel stands: alone (ordinary launch), first
// after whatever is on the stream (it may start early and waits for that
// itself), or after another of the evaluation's (launch_after).
enum Chain { kAlone, kFirst, kAfter };

// chain: set to kAfter once a kernel has been launched.
template <int KIND>
int launch_kind(grav_plan *pl, const DevProblem &dp, cudaStream_t st, Chain *chain = nullptr) {
    if (dp.nitems[KIND] == 0)
        return 0;
    const int wpb = std::min(pl->tune.warps_per_block, kListWarps);
    size_t warp;
    const void *kern;
    if constexpr (KIND == KP) {
        warp = kPointWarpBytes;
        kern = pl->plain ? (const void *)k_points<true> : (const void *)k_points<false>;
    } else {
        warp = CellKind<KIND>::warp_bytes;
        kern = pl->plain ? (const void *)k_cells<KIND, true> : (const void *)k_cells<KIND, false>;
    }
    // the limit belongs to the kernel, not to this plan: the most that any plan needs, so that
    // no other thread's launch finds it lowered
    GC_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(kListWarps * warp)));
    const size_t smem = wpb * warp;
    int fit = 0;
    GC_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, wpb * 32, smem));
    // a cap counts the caller's blocks, of warps_per_block warps each
    const int64_t cap = ((int64_t)pl->tune.blocks_per_sm * pl->tune.warps_per_block + wpb - 1) / wpb;
    const int per_sm = cap > 0 ? (int)std::min<int64_t>(cap, fit) : fit;
    const int blocks = std::min(std::max(1, per_sm) * pl->nsm, (dp.nitems[KIND] + wpb - 1) / wpb);
    CUtensorMap tm = pl->tmap[KIND];
    DevProblem d = dp;
    d.first = chain && *chain == kFirst;
    void *pargs[] = {&d}, *cargs[] = {&tm, &d};
    if (int rc = launch_after(kern, blocks, wpb * 32, smem, st, chain && *chain != kAlone,
                              KIND == KP ? pargs : cargs))
        return rc;
    if (chain)
        *chain = kAfter;
    pl->launches++;
    return 0;
}

// k_ewald_moments: `warps` warps per block, blocks_per_sm x SM count blocks
// (0: as many as fit), at most one warp per unit; over dp's groups, on
// stream s.
int launch_moments(grav_plan *pl, const DevProblem &dp, cudaStream_t s, int per_sm, int warps,
                   bool after) {
    const int64_t n = (dp.ngroups - dp.gbegin) * dp.ewsplit;
    if (n <= 0)
        return 0;
    const size_t smem = (size_t)warps * kEwWarpBytes;
    GC_CHECK(cudaFuncSetAttribute(k_ewald_moments, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  4 * kEwWarpBytes));
    if (per_sm <= 0) {
        int fit = 0;
        GC_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_ewald_moments, warps * 32,
                                                               smem));
        per_sm = std::max(1, fit);
    }
    DevProblem d = dp;
    d.ewm = pl->ewm;
    const unsigned blocks = (unsigned)std::max<int64_t>(
        1, std::min<int64_t>((n + warps - 1) / warps, (int64_t)per_sm * pl->nsm));
    void *args[] = {&d};
    if (int rc = launch_after((const void *)k_ewald_moments, blocks, warps * 32, smem, s, after, args))
        return rc;
    pl->launches++;
    return 0;
}

// Placement of the periodic correction moments: ewald_side > 0 runs them on
// a side stream beside the list kernels (k_ewald_side) in that many two-warp
// blocks per SM, sharing the SMs with them; ewald_side = -k runs them
// (k_ewald_moments) on the evaluation's stream between the list kernels and
// the finish pass, with the SMs to themselves, in blocks of k warps (k = 1,
// 2 or 4) as many as fit.  Automatic (0): the evaluation's stream, two-warp
// blocks.  Since k_ewald_moments stages its rows it is the faster place at
// every size (ms an evaluation on it, and beside the lists with 2 and 3 side
// blocks per SM): 64^3 at MAC 1e-5 4.56, 5.19, 4.65; 128^3 at 2.5e-6 63.8,
// 69.7, 66.2; 256^3 at 1.5e-6, where the correction list is 1.2 % of the
// order-4 interactions, 680, 748, 703.  One, two or four warps a block differ
// by less than 0.1 %.
int main_moments_warps(const grav_plan *pl) {
    const int k = -pl->tune.ewald_side;
    return (k == 1 || k == 2 || k == 4) ? k : 2;
}

int side_blocks(const grav_plan *pl) {
    return pl->dp.ewald && pl->side && pl->ewm ? std::max(0, pl->tune.ewald_side) : 0;
}

// Fork: k_ewald_moments over dp's groups on the side stream, after the work
// already on st; returns whether it forked (join with side_join).
int side_fork(grav_plan *pl, const DevProblem &dp, cudaStream_t st, bool &forked) {
    forked = false;
    const int per_sm = side_blocks(pl);
    if (per_sm <= 0 || dp.ngroups - dp.gbegin <= 0)
        return 0;
    GC_CHECK(cudaEventRecord(pl->fork, st));
    GC_CHECK(cudaStreamWaitEvent(pl->side, pl->fork, 0));
    DevProblem d = dp;
    d.ewm = pl->ewm;
    const int64_t n = (dp.ngroups - dp.gbegin) * dp.ewsplit;
    const unsigned blocks =
        (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 1) / 2, (int64_t)per_sm * pl->nsm));
    k_ewald_side<<<blocks, 64, 0, pl->side>>>(d);
    GC_CHECK(cudaGetLastError());
    pl->launches++;
    GC_CHECK(cudaEventRecord(pl->join, pl->side));
    forked = true;
    return 0;
}

int side_join(grav_plan *pl, cudaStream_t st) {
    GC_CHECK(cudaStreamWaitEvent(st, pl->join, 0));
    return 0;
}

// The finish pass, after the correction moments when they did not run on
// the side stream (forked).
int launch_finish(grav_plan *pl, const DevProblem &dp, cudaStream_t st, bool forked,
                  bool after = false) {
    if (dp.ewald && !forked)
        if (int rc = launch_moments(pl, dp, st, 0, main_moments_warps(pl), after))
            return rc;
    const int wpb = 2;
    const int64_t n = dp.ngroups - dp.gbegin;
    if (n <= 0)
        return 0;
    DevProblem d = dp;
    void *args[] = {&d};
    if (int rc = launch_after((const void *)k_finish, (unsigned)((n + wpb - 1) / wpb), wpb * 32, 0, st,
                              after && !forked, args))
        return rc;
    pl->launches++;
    return 0;
}
}  // namespace

namespace {
// A retune that ran out of memory leaves a plan without its work queue.
bool has_queue(const grav_plan *pl) {
    const DevProblem &d = pl->dp;
    for (int k = 0; k < 3; k++)
        if (d.nitems[k] > 0 && !d.items[k])
            return false;
    return d.part && d.gslot;
}
}  // namespace

extern "C" int grav_groups_eval_CUDA(grav_plan *pl, void *stream) {
    if (!pl)
        return gc::set_status(-1, "grav_groups_eval_CUDA: no plan");
    if (!has_queue(pl))
        return gc::set_status(-1, "grav_groups_eval_CUDA: the plan lost its work queue in a failed "
                                  "retune; retune it again");
    cudaStream_t st = (cudaStream_t)stream;
    pl->used_on(st);
    pl->launches = 0;
    auto mark = [&](int k) -> int {
        if (pl->timing)
            GC_CHECK(cudaEventRecord(pl->ev[k], st));
        return 0;
    };
    // The queues are at zero when the last evaluation's finish pass left them
    // so, which saves a memset node in front of each evaluation and lets its
    // first kernel start early (2k bodies: 16.5 -> 14.0 us, 64k 387 -> 385 us);
    // a captured evaluation clears them itself, whatever it is replayed after.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) {
        cudaGetLastError();
        cap = cudaStreamCaptureStatusActive;
    }
    const bool capturing = cap != cudaStreamCaptureStatusNone;
    const bool clear = capturing || !pl->queues_clear;
    if (!capturing)
        pl->queues_clear = false;
    if (clear)
        GC_CHECK(cudaMemsetAsync(pl->dp.counters, 0, 4 * sizeof(int), st));
    if (int rc = mark(0))
        return rc;
    bool forked = false;
    Chain state = clear ? kAlone : kFirst;
    Chain *chain = pl->timing ? nullptr : &state;  // events between them time whole kernels
    if (int rc = side_fork(pl, pl->dp, st, forked))
        return rc;
    if (int rc = launch_kind<KH>(pl, pl->dp, st, chain))
        return rc;
    if (int rc = mark(1))
        return rc;
    if (int rc = launch_kind<KQ>(pl, pl->dp, st, chain))
        return rc;
    if (int rc = mark(2))
        return rc;
    if (int rc = launch_kind<KP>(pl, pl->dp, st, chain))
        return rc;
    if (int rc = mark(3))
        return rc;
    DevProblem df = pl->dp;
    df.ewm = pl->ewm;
    if (forked)
        if (int rc = side_join(pl, st))
            return rc;
    if (int rc = launch_finish(pl, df, st, forked, chain && state == kAfter))
        return rc;
    if (!capturing)
        pl->queues_clear = true;
    pl->evaluated = true;
    return mark(4);
}

extern "C" int grav_plan_retune_CUDA(grav_plan *pl, const grav_tuning *tuning) {
    if (!pl || !tuning)
        return gc::set_status(-1, "grav_plan_retune_CUDA: bad arguments");
    const int64_t ng = pl->hp.ngroups;
    grav_tuning t = *tuning;
    if (t.warps_per_block < 1 || t.warps_per_block > 8)
        t.warps_per_block = 8;
    const int64_t tot[3] = {pl->lists_ptr[0].empty() ? 0 : pl->lists_ptr[0][ng],
                            pl->lists_ptr[1].empty() ? 0 : pl->lists_ptr[1][ng],
                            pl->lists_ptr[2].empty() ? 0 : pl->lists_ptr[2][ng]};
    if (t.chunk_p <= 0)
        t.chunk_p = auto_chunk(tot[0], ng, pl->nsm, KP);
    if (t.chunk_q <= 0)
        t.chunk_q = auto_chunk(tot[1], ng, pl->nsm, KQ);
    if (t.chunk_h <= 0)
        t.chunk_h = auto_chunk(tot[2], ng, pl->nsm, KH);
    t.ewald_n = pl->tune.ewald_n;  // the correction table is not rebuilt
    pl->tune = t;
    std::vector<Item> items[3];
    std::vector<int64_t> gslot;
    pl->nslots = make_queue(pl, items, gslot);
    // replace the queue's device buffers
    GC_CHECK(cudaDeviceSynchronize());
    auto drop = [&](const void *p) {
        if (!p)
            return;
        auto it = std::find(pl->allocs.begin(), pl->allocs.end(), p);
        if (it != pl->allocs.end()) {
            if (pl->pool)
                cudaFreeAsync(*it, 0);
            else
                cudaFree(*it);
            pl->allocs.erase(it);
        }
    };
    DevProblem &d = pl->dp;
    for (int k = 0; k < 3; k++) drop(d.items[k]);
    drop(d.part);
    drop(d.gslot);
    int rc = 0;
    for (int k = 0; k < 3; k++) {
        Item *it = nullptr;
        rc |= dev_copy(pl, items[k].data(), items[k].size(), &it);
        d.items[k] = it;
        d.nitems[k] = (int)items[k].size();
    }
    float4 *part = nullptr;
    rc |= dev_copy<float4>(pl, nullptr, (size_t)std::max<int64_t>(1, pl->nslots) * 64, &part);
    d.part = part;
    int64_t *gs = nullptr;
    rc |= dev_copy(pl, gslot.data(), gslot.size(), &gs);
    d.gslot = gs;
    if (pl->step)
        step_graph_reset(pl->step);  // a captured step holds the old queue
    GC_CHECK(cudaStreamSynchronize(0));  // as at the end of the upload
    return rc;
}

extern "C" int grav_plan_get_tuning(const grav_plan *pl, grav_tuning *out) {
    if (!pl || !out)
        return gc::set_status(-1, "grav_plan_get_tuning: bad arguments");
    *out = pl->tune;
    return 0;
}

extern "C" int grav_plan_set_timing(grav_plan *pl, int on) {
    if (!pl)
        return gc::set_status(-1, "grav_plan_set_timing: no plan");
    if (on && !pl->ev[0])
        for (int k = 0; k < 5; k++) GC_CHECK(cudaEventCreate(&pl->ev[k]));
    pl->timing = on ? 1 : 0;
    return 0;
}

extern "C" int grav_plan_kernel_ms(grav_plan *pl, float ms[4]) {
    if (!pl || !pl->timing)
        return gc::set_status(-1, "grav_plan_kernel_ms: timing is off");
    GC_CHECK(cudaEventSynchronize(pl->ev[4]));
    for (int k = 0; k < 4; k++) GC_CHECK(cudaEventElapsedTime(&ms[k], pl->ev[k], pl->ev[k + 1]));
    return 0;
}

extern "C" int grav_groups_download_CUDA(grav_plan *pl, float *acc_phi) {
    if (!pl || !acc_phi)
        return gc::set_status(-1, "grav_groups_download_CUDA: bad arguments");
    GC_CHECK(cudaMemcpy(acc_phi, pl->dp.out, (size_t)pl->hp.nbodies * sizeof(float4),
                        cudaMemcpyDeviceToHost));
    unsigned h = 0;
    GC_CHECK(cudaMemcpy(&h, pl->dp.err, sizeof(h), cudaMemcpyDeviceToHost));
    if (h) {
        cudaMemset(pl->dp.err, 0, sizeof(unsigned));
        return gc::set_status(-2, "batched kernels: device error word 0x%x", h);
    }
    return 0;
}

extern "C" float *grav_plan_output(grav_plan *pl) {
    return pl ? reinterpret_cast<float *>(pl->dp.out) : nullptr;
}

extern "C" void grav_plan_counts(const grav_plan *pl, int64_t out[4]) {
    for (int k = 0; k < 4; k++) out[k] = pl ? pl->counts[k] : 0;
}

extern "C" int grav_plan_launches(const grav_plan *pl) { return pl ? pl->launches : 0; }

extern "C" void grav_plan_free(grav_plan *pl) {
    if (!pl)
        return;
    // buffers go back to the pool in the default stream's order: work on another stream may
    // still use them (cudaFree waits by itself)
    if (pl->pool && pl->elsewhere)
        cudaDeviceSynchronize();
    if (pl->step)
        step_state_free(pl->step);
    if (pl->adj)
        adjoint_state_free(pl->adj);
    for (void *p : pl->allocs) {
        if (pl->pool)
            cudaFreeAsync(p, 0);  // back to the pool, reserved for the next call
        else
            cudaFree(p);
    }
    for (cudaEvent_t e : pl->ev)
        if (e)
            cudaEventDestroy(e);
    if (pl->side) {
        cudaStreamSynchronize(pl->side);
        cudaStreamDestroy(pl->side);
    }
    if (pl->fork)
        cudaEventDestroy(pl->fork);
    if (pl->join)
        cudaEventDestroy(pl->join);
    delete pl;
}

// step.cuh: the plan's step state adopts a device-built tree's links
int set_tree_adopt(grav_plan *pl, const DevTree &T, cudaMemPool_t pool);

namespace {
// The device build and the plan that adopts it; buffers from the device's
// pool (grav_groups_release_CUDA returns the memory it keeps reserved).
int build_plan(const nln_params *params, const float4 *bodies, int64_t n, double eps2,
               float quad_phi_sign, int ewald, const grav_tuning *tuning, grav_plan **plan) {
    *plan = nullptr;
    cudaMemPool_t pool = nullptr;
    if (int rc = e2e_pool(&pool))
        return rc;
    DevTree T;
    const double t0 = now_s();
    if (int rc = gpu_tree_build(*params, bodies, n, 0, T, pool))
        return rc;
    grav_problem hp{};
    hp.nbodies = T.n;
    hp.ncells = T.ncells;
    hp.ngroups = T.ngroups;
    hp.points = reinterpret_cast<const float *>(T.points);
    hp.qcells = T.qcells;
    hp.hcells = T.hcells;
    hp.groups = T.groups_h.data();
    hp.pptr = T.ptr_h[0].data();
    hp.qptr = T.ptr_h[1].data();
    hp.hptr = T.ptr_h[2].data();
    hp.plist = T.list[0];
    hp.qlist = T.list[1];
    hp.hlist = T.list[2];
    hp.eps2 = eps2;
    hp.box = params->box;
    hp.quad_phi_sign = quad_phi_sign;
    hp.ewald = params->box > 0 && ewald;
    hp.cptr = T.ptr_h[3].data();
    hp.clist = T.list[3];
    grav_plan *pl = nullptr;
    if (int rc = upload_impl(&hp, tuning, &pl, 0, &T)) {
        // upload_impl took the tree's buffers over and released them, but for its links
        for (void *q : {(void *)T.cell_first, (void *)T.cell_count, (void *)T.cell_child,
                        (void *)T.cell_nchild})
            cudaFreeAsync(q, 0);
        return rc;
    }
    // the tree's links (for the device refit and the adjoint) stay on the
    // device: the plan's step state adopts them
    if (int rc = set_tree_adopt(pl, T, pool)) {
        grav_plan_free(pl);
        return rc;
    }
    t_build = now_s() - t0;
    for (int k = 0; k < 6; k++) t_build_phase[k] = T.seconds[k];
    *plan = pl;
    return 0;
}

// out[order[i]] = in[i]: results from tree order back to the input order.
__global__ void k_unorder(const float4 *__restrict__ in, const int64_t *__restrict__ order,
                          int64_t n, float4 *out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const int64_t j = order[i];
        if (j >= 0 && j < n)
            out[j] = in[i];
    }
}
}  // namespace

extern "C" int grav_plan_build_CUDA(const nln_params *params, const float *bodies, int64_t n,
                                    double eps2, float quad_phi_sign, int ewald,
                                    const grav_tuning *tuning, grav_plan **plan) {
    if (!params || !bodies || !plan || n <= 0)
        return gc::set_status(-1, "grav_plan_build_CUDA: bad arguments");
    *plan = nullptr;
    if (((uintptr_t)bodies & 15u) != 0)
        return gc::set_status(-1, "grav_plan_build_CUDA: bodies must be 16-byte aligned");
    return build_plan(params, reinterpret_cast<const float4 *>(bodies), n, eps2, quad_phi_sign,
                      ewald, tuning, plan);
}

extern "C" int grav_build_eval_CUDA(const nln_params *params, const float *bodies, int64_t n,
                                    double eps2, float quad_phi_sign, int ewald,
                                    float *acc_phi) {
    if (!params || !bodies || !acc_phi || n <= 0)
        return gc::set_status(-1, "grav_build_eval_CUDA: bad arguments");
    const double t_start = now_s();
    cudaMemPool_t pool = nullptr;
    if (int rc = e2e_pool(&pool))
        return rc;
    float4 *dev = nullptr, *out = nullptr;
    const size_t bytes = (size_t)n * sizeof(float4);
    GC_CHECK(gc::pool_malloc((void **)&dev, bytes, pool, 0));
    cudaError_t e = gc::pool_malloc((void **)&out, bytes, pool, 0);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(dev, bodies, bytes, cudaMemcpyHostToDevice, 0);
    if (e != cudaSuccess) {
        cudaFreeAsync(dev, 0);
        if (out)
            cudaFreeAsync(out, 0);
        return gc::cuda_status(e, "grav_build_eval_CUDA: bodies");
    }
    const double t_h2d = now_s();
    grav_plan *pl = nullptr;
    int rc = build_plan(params, dev, n, eps2, quad_phi_sign, ewald, nullptr, &pl);
    const double t_built = now_s();
    if (!rc)
        rc = grav_groups_eval_CUDA(pl, nullptr);
    if (!rc) {
        k_unorder<<<(unsigned)((n + 255) / 256), 256>>>(pl->dp.out, pl->order, n, out);
        e = cudaGetLastError();
        if (e == cudaSuccess)
            e = cudaMemcpy(acc_phi, out, bytes, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess)
            rc = gc::cuda_status(e, "grav_build_eval_CUDA: results");
    }
    const double t_eval = now_s();
    if (!rc) {
        unsigned h = 0;
        e = cudaMemcpy(&h, pl->dp.err, sizeof(h), cudaMemcpyDeviceToHost);
        if (e != cudaSuccess)
            rc = gc::cuda_status(e, "grav_build_eval_CUDA: error word");
        else if (h)
            rc = gc::set_status(-2, "grav_build_eval_CUDA: device error word 0x%x", h);
    }
    if (pl)
        grav_plan_free(pl);
    cudaFreeAsync(dev, 0);
    cudaFreeAsync(out, 0);
    cudaStreamSynchronize(0);
    t_phase_be[0] = t_h2d - t_start;
    t_phase_be[1] = t_built - t_h2d;
    t_phase_be[2] = t_eval - t_built;
    t_phase_be[3] = now_s() - t_eval;
    return rc;
}

extern "C" void grav_build_eval_phases(double seconds[4]) {
    for (int k = 0; k < 4; k++) seconds[k] = t_phase_be[k];
}

extern "C" const int64_t *grav_plan_order(const grav_plan *pl) { return pl ? pl->order : nullptr; }

extern "C" void grav_plan_build_phases(double seconds[7]) {
    for (int k = 0; k < 6; k++) seconds[k] = t_build_phase[k];
    seconds[6] = t_build;
}

extern "C" int grav_plan_problem(const grav_plan *pl, grav_problem *out) {
    if (!pl || !out)
        return gc::set_status(-1, "grav_plan_problem: bad arguments");
    *out = pl->hp;
    const DevProblem &d = pl->dp;
    out->points = reinterpret_cast<const float *>(d.points);
    out->qcells = d.qcells;
    out->hcells = d.hcells;
    out->groups = d.groups;
    out->plist = d.list[0];
    out->qlist = d.list[1];
    out->hlist = d.list[2];
    out->clist = d.clist;
    auto host = [&](int k) { return pl->lists_ptr[k].empty() ? nullptr : pl->lists_ptr[k].data(); };
    out->pptr = host(0);
    out->qptr = host(1);
    out->hptr = host(2);
    out->cptr = host(3);
    for (int k = 0; k < 4; k++) {
        out->zptr[k] = nullptr;
        out->zlist[k] = nullptr;
    }
    return 0;
}

namespace {
// Group ranges of the pipelined end-to-end call: one per 2 GiB of list
// words copied (packed words where a kind is run-packed), at most 16, the
// first one split further; GRAV_E2E_CHUNKS overrides the count.
int e2e_chunks(const grav_problem *hp) {
    if (const char *e = getenv("GRAV_E2E_CHUNKS"))
        return std::max(1, std::min(64, atoi(e)));
    const int64_t ng = hp->ngroups;
    const int64_t *plain[4] = {hp->pptr, hp->qptr, hp->hptr,
                               hp->box > 0 && hp->ewald ? hp->cptr : nullptr};
    int64_t words = 0;
    for (int k = 0; k < 4; k++) {
        if (!plain[k])
            continue;
        words += (hp->zlist[k] && hp->zptr[k]) ? hp->zptr[k][ng] : plain[k][ng];
    }
    return (int)std::max<int64_t>(1, std::min<int64_t>(16, (words * 4 + (2ll << 30) - 1) >> 31));
}

// Copy group range c's slice of every list on `cs`, then make `st` wait for it.
int copy_range(grav_plan *pl, const grav_problem *hp, size_t c, cudaStream_t cs, cudaStream_t st,
               cudaEvent_t ev) {
    const int64_t g0 = pl->chunk_group[c], g1 = pl->chunk_group[c + 1];
    const DevProblem &d = pl->dp;
    const int64_t *ptr[4] = {hp->pptr, hp->qptr, hp->hptr, d.clist ? hp->cptr : nullptr};
    const uint32_t *src[4] = {hp->plist, hp->qlist, hp->hlist, hp->clist};
    const uint32_t *dst[4] = {d.list[0], d.list[1], d.list[2], d.clist};
    for (int k = 0; k < 4; k++) {
        if (pl->zdev[k]) {  // run-packed: copy the words, k_unpack fills dst
            ptr[k] = hp->zptr[k];
            src[k] = hp->zlist[k];
            dst[k] = pl->zdev[k];
        }
        if (!ptr[k] || !dst[k] || ptr[k][g1] <= ptr[k][g0])
            continue;
        GC_CHECK(cudaMemcpyAsync(const_cast<uint32_t *>(dst[k]) + ptr[k][g0], src[k] + ptr[k][g0],
                                 (size_t)(ptr[k][g1] - ptr[k][g0]) * sizeof(uint32_t),
                                 cudaMemcpyHostToDevice, cs));
    }
    GC_CHECK(cudaEventRecord(ev, cs));
    GC_CHECK(cudaStreamWaitEvent(st, ev, 0));
    return 0;
}

// Evaluate group range c: its work items, then its groups' finish pass.
int eval_range(grav_plan *pl, size_t c, cudaStream_t st) {
    DevProblem dp = pl->dp;
    for (int k = 0; k < 3; k++) {
        const int b = pl->chunk_item[k][c], e = pl->chunk_item[k][c + 1];
        dp.items[k] = pl->dp.items[k] ? pl->dp.items[k] + b : nullptr;
        dp.nitems[k] = e - b;
    }
    dp.counters = pl->dp.counters + 4 * c;
    dp.gbegin = pl->chunk_group[c];
    dp.ngroups = pl->chunk_group[c + 1];
    for (int k = 0; k < 4; k++) {
        if (!pl->zdev[k])
            continue;
        uint32_t *dst = const_cast<uint32_t *>(k < 3 ? pl->dp.list[k] : pl->dp.clist);
        const int64_t n = dp.ngroups - dp.gbegin;
        const unsigned blocks = (unsigned)std::max<int64_t>(
            1, std::min<int64_t>((n + 7) / 8, (int64_t)pl->nsm * 16));
        k_unpack<<<blocks, 256, 0, st>>>(pl->zdev[k], pl->zptr_dev[k], pl->lptr_dev[k], dp.gbegin,
                                         dp.ngroups, dst, pl->dp.err);
        GC_CHECK(cudaGetLastError());
        pl->launches++;
    }
    bool forked = false;
    int rc = side_fork(pl, dp, st, forked);
    if (!rc)
        rc = launch_kind<KH>(pl, dp, st);
    if (!rc)
        rc = launch_kind<KQ>(pl, dp, st);
    if (!rc)
        rc = launch_kind<KP>(pl, dp, st);
    dp.ewm = pl->ewm;
    if (!rc && forked)
        rc = side_join(pl, st);
    if (!rc)
        rc = launch_finish(pl, dp, st, forked);
    return rc;
}
}  // namespace

// The end-to-end call: upload the tables, then copy the lists range by range
// on a copy stream while the kernels evaluate the ranges already copied, and
// download.  Lists in page-locked host memory overlap best; pageable lists
// still overlap each copy with the previous range's kernels.
extern "C" int grav_groups_CUDA(const grav_problem *hp, float *acc_phi) {
    if (!hp || hp->ngroups <= 0 || !hp->pptr || !acc_phi)
        return gc::set_status(-1, "grav_groups_CUDA: incomplete problem");
    grav_plan *pl = nullptr;
    if (hp->lists_in_host) {
        if (int rc = grav_groups_upload_CUDA(hp, nullptr, &pl))
            return rc;
        double t0 = now_s();
        int rc = grav_groups_eval_CUDA(pl, nullptr);
        const cudaError_t e = rc ? cudaSuccess : cudaDeviceSynchronize();
        if (e != cudaSuccess)
            rc = gc::cuda_status(e, "grav_groups_CUDA: evaluation");
        t_phase[2] = now_s() - t0;
        t0 = now_s();
        if (!rc)
            rc = grav_groups_download_CUDA(pl, acc_phi);
        t_phase[3] = now_s() - t0;
        t0 = now_s();
        grav_plan_free(pl);
        t_phase[4] = now_s() - t0;
        return rc;
    }
    if (int rc = upload_impl(hp, nullptr, &pl, e2e_chunks(hp)))
        return rc;
    const size_t nc = pl->chunk_group.size() - 1;
    double t0 = now_s();
    auto chk = [](cudaError_t e, const char *what) {
        return e == cudaSuccess ? 0 : gc::cuda_status(e, what);
    };
    // one copy stream and one compute stream (ranges alternating over two
    // compute streams measured no faster: their kernels compete for the SMs)
    cudaStream_t cs = nullptr, st = nullptr;
    std::vector<cudaEvent_t> ev(nc, nullptr);
    int rc = 0;
    cudaError_t e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
    if (e == cudaSuccess)
        e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    for (size_t c = 0; c < nc && e == cudaSuccess; c++)
        e = cudaEventCreateWithFlags(&ev[c], cudaEventDisableTiming);
    rc = chk(e, "grav_groups_CUDA: streams");
    pl->queues_clear = false;
    if (!rc)
        rc = chk(cudaMemsetAsync(pl->dp.counters, 0, 4 * nc * sizeof(int), st),
                 "grav_groups_CUDA: queue heads");
    pl->launches = 0;
    for (size_t c = 0; c < nc && !rc; c++) {
        rc = copy_range(pl, hp, c, cs, st, ev[c]);
        if (!rc)
            rc = eval_range(pl, c, st);
    }
    if (!rc)
        rc = chk(cudaStreamSynchronize(st), "grav_groups_CUDA: evaluation");
    t_phase[2] = now_s() - t0;
    t0 = now_s();
    if (!rc)
        rc = grav_groups_download_CUDA(pl, acc_phi);
    t_phase[3] = now_s() - t0;
    t0 = now_s();
    if (cs)
        cudaStreamSynchronize(cs);
    if (st)
        cudaStreamSynchronize(st);
    for (cudaEvent_t x : ev)
        if (x)
            cudaEventDestroy(x);
    if (cs)
        cudaStreamDestroy(cs);
    if (st)
        cudaStreamDestroy(st);
    grav_plan_free(pl);
    t_phase[4] = now_s() - t0;
    return rc;
}

void dropin_release();  // dropin.cu: the sink buffers kept between walks

extern "C" void grav_groups_release_CUDA(void) {
    dropin_release();
    std::lock_guard<std::mutex> lk(g_pool_mu);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    if (dev >= 0 && dev < kMaxPoolDevices && g_pool[dev]) {
        cudaDeviceSynchronize();
        cudaMemPoolTrimTo(g_pool[dev], 0);
    }
}

extern "C" void grav_groups_CUDA_phases(double seconds[5]) {
    for (int k = 0; k < 5; k++) seconds[k] = t_phase[k];
}

// ------------------------------------------------------------ no-allocation evaluation
//
// grav_groups_eval_dev_CUDA runs the batched kernels above on a problem that
// is already on the device, with every byte of scratch taken from this one
// file-scope array: queue counters and the error word, one work item per
// (group, list kind), a checked copy of the groups, the slot offsets and
// the per-item partial sums.  Its address is looked up once per device.
static __device__ __align__(256) unsigned char g_dev_scratch[GRAV_DEV_SCRATCH_BYTES];

namespace {

constexpr int kMaxDevices = 64;

struct DevScratch {
    int *counters;      // 4 queue heads: must be 0 when the kernels start
    unsigned *err;      // device error word: must be 0 when the kernels start
    double *span;       // of the groups: must be 0 when the setup starts
    Item *items[3];
    nln_group *groups;  // checked copy of the caller's groups
    int64_t *gslot;
    float4 *part;
};

size_t round256(size_t b) { return (b + 255) / 256 * 256; }

// Scratch bytes for ng groups with nk list kinds.
size_t dev_scratch_bytes(int64_t ng, int nk) {
    return 256 + 3 * round256((size_t)ng * sizeof(Item)) + round256((size_t)ng * sizeof(nln_group)) +
           round256((size_t)(ng + 1) * sizeof(int64_t)) + (size_t)nk * ng * 64 * sizeof(float4);
}

// Once per device, with that device current: the scratch's address, the
// device's SM count and the shared-memory attribute of the list kernels this
// entry launches.
int dev_scratch_base(void **out, int *nsm) {
    static std::mutex mu;
    static void *base[kMaxDevices] = {};
    static int sms[kMaxDevices] = {};
    int dev = 0;
    GC_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices)
        return gc::set_status(-1, "grav_groups_eval_dev_CUDA: device %d beyond %d", dev, kMaxDevices);
    std::lock_guard<std::mutex> lk(mu);
    if (!base[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_dev_scratch);
        if (e != cudaSuccess)
            return gc::cuda_status(e, "grav_groups_eval_dev_CUDA: cudaGetSymbolAddress of the scratch");
        if (!p)
            return gc::set_status(-1, "grav_groups_eval_dev_CUDA: the scratch has no device address");
        int n = 0;
        e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess)
            return gc::cuda_status(e, "grav_groups_eval_dev_CUDA: SM count");
        if (n <= 0)
            return gc::set_status(-1, "grav_groups_eval_dev_CUDA: device %d reports no SMs", dev);
        GC_CHECK(cudaFuncSetAttribute(k_points<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kListWarps * kPointWarpBytes));
        GC_CHECK(cudaFuncSetAttribute(k_cells<KQ, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kListWarps * CellKind<KQ>::warp_bytes));
        GC_CHECK(cudaFuncSetAttribute(k_cells<KH, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kListWarps * CellKind<KH>::warp_bytes));
        sms[dev] = n;
        base[dev] = p;
    }
    *out = base[dev];
    *nsm = sms[dev];
    return 0;
}

// One thread per group: check the group and its list offsets, copy it, and
// write its work items (slot nk*g + kind rank) and slot offset.  A group
// that fails the checks flags GC_DEV_BAD_INDEX and becomes one sink (body
// 0) with empty lists, so no kernel leaves the tables.
__global__ void k_dev_setup(const nln_group *__restrict__ groups, const int64_t *p0,
                            const int64_t *p1, const int64_t *p2, int64_t ng, int64_t nbodies,
                            int nk, DevScratch S) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g == 0)
        S.gslot[ng] = (int64_t)nk * ng;
    if (g >= ng)
        return;
    nln_group G = groups[g];
    const int64_t *ptr[3] = {p0, p1, p2};
    bool ok = G.count >= 1 && G.count <= 32 && G.first >= 0 && G.first + G.count <= nbodies;
    for (int k = 0; k < 3; k++)
        if (ptr[k] && (ptr[k][g] < 0 || ptr[k][g + 1] < ptr[k][g]))
            ok = false;
    if (!ok) {
        atomicOr(S.err, GC_DEV_BAD_INDEX);
        G.first = 0;
        G.count = 1;
    }
    S.groups[g] = G;
    // not negative: their bits are in their order
    const double span = group_span(G, groups[0]);
    if (span > 0)
        atomicMax(reinterpret_cast<unsigned long long *>(S.span),
                  (unsigned long long)__double_as_longlong(span));
    int rank = 0;
    for (int k = 0; k < 3; k++) {
        if (!ptr[k])
            continue;
        const int64_t b = ok ? ptr[k][g] : 0, e = ok ? ptr[k][g + 1] : 0;
        S.items[k][g] = Item{(int32_t)g, (int32_t)((int64_t)nk * g + rank), b, e};
        rank++;
    }
    S.gslot[g] = (int64_t)nk * g;
}

}  // namespace

extern "C" int grav_groups_eval_dev_CUDA(const grav_problem *dp, float *acc_phi, void *stream) {
    if (!dp || !acc_phi || dp->nbodies <= 0 || dp->ngroups <= 0 || !dp->points || !dp->groups ||
        !dp->pptr || !dp->plist)
        return gc::set_status(-1, "grav_groups_eval_dev_CUDA: incomplete problem");
    if (dp->box > 0 && dp->ewald)
        return gc::set_status(-1, "grav_groups_eval_dev_CUDA: no Ewald correction here (its table "
                                  "is a per-plan allocation); use grav_groups_upload_CUDA");
    if (dp->nbodies + dp->ncells >= (int64_t)NLN_IDX_MASK)
        return gc::set_status(-1, "grav_groups_eval_dev_CUDA: point table exceeds 27-bit indices");
    if ((dp->qptr && (!dp->qlist || !dp->qcells)) || (dp->hptr && (!dp->hlist || !dp->hcells)))
        return gc::set_status(-1, "grav_groups_eval_dev_CUDA: a cell list without its table");
    auto misaligned = [](const void *p) { return ((uintptr_t)p & 15u) != 0; };
    if (misaligned(dp->points) || misaligned(dp->qcells) || misaligned(dp->hcells) ||
        misaligned(acc_phi))
        return gc::set_status(-1, "grav_groups_eval_dev_CUDA: tables and output must be "
                                  "16-byte aligned");
    const int64_t ng = dp->ngroups, np = dp->nbodies + dp->ncells;
    const int nk = 1 + (dp->qptr ? 1 : 0) + (dp->hptr ? 1 : 0);
    const size_t need = dev_scratch_bytes(ng, nk);
    if (need > (size_t)GRAV_DEV_SCRATCH_BYTES) {
        int64_t fit = 0;
        while (dev_scratch_bytes(fit + 1, nk) <= (size_t)GRAV_DEV_SCRATCH_BYTES) fit += 1;
        return gc::set_status(-1, "grav_groups_eval_dev_CUDA: %lld groups need %zu bytes of "
                                  "scratch; the static scratch holds %zu (at most %lld groups with "
                                  "%d list kinds)",
                              (long long)ng, need, (size_t)GRAV_DEV_SCRATCH_BYTES, (long long)fit, nk);
    }
    void *basev = nullptr;
    int nsm = 0;
    if (int rc = dev_scratch_base(&basev, &nsm))
        return rc;
    unsigned char *base = static_cast<unsigned char *>(basev);
    DevScratch S{};
    size_t off = 0;
    S.counters = reinterpret_cast<int *>(base);
    S.err = reinterpret_cast<unsigned *>(base + 4 * sizeof(int));
    S.span = reinterpret_cast<double *>(base + 8 * sizeof(int));
    off = 256;
    for (int k = 0; k < 3; k++) {
        S.items[k] = reinterpret_cast<Item *>(base + off);
        off += round256((size_t)ng * sizeof(Item));
    }
    S.groups = reinterpret_cast<nln_group *>(base + off);
    off += round256((size_t)ng * sizeof(nln_group));
    S.gslot = reinterpret_cast<int64_t *>(base + off);
    off += round256((size_t)(ng + 1) * sizeof(int64_t));
    S.part = reinterpret_cast<float4 *>(base + off);

    // a plan on the stack: device pointers only, nothing owned
    grav_plan pl;
    pl.nsm = nsm;
    pl.tune = default_tuning();
    DevProblem &d = pl.dp;
    d.points = reinterpret_cast<const float4 *>(dp->points);
    d.qcells = dp->qptr ? dp->qcells : nullptr;
    d.hcells = dp->hptr ? dp->hcells : nullptr;
    d.groups = S.groups;
    const int64_t *ptrs[3] = {dp->pptr, dp->qptr, dp->hptr};
    const uint32_t *lists[3] = {dp->plist, dp->qlist, dp->hlist};
    for (int k = 0; k < 3; k++) {
        d.list[k] = ptrs[k] ? lists[k] : nullptr;
        d.items[k] = ptrs[k] ? S.items[k] : nullptr;
        d.nitems[k] = ptrs[k] ? (int)ng : 0;
    }
    d.ntab[0] = np;
    d.ntab[1] = d.ntab[2] = dp->ncells;
    d.counters = S.counters;
    d.part = S.part;
    d.gslot = S.gslot;
    d.out = reinterpret_cast<float4 *>(acc_phi);
    d.ngroups = ng;
    d.ncells = dp->ncells;
    d.eps2 = (float)dp->eps2;
    d.qsh = 0.5f * (dp->quad_phi_sign == 0.0f ? 1.0f : dp->quad_phi_sign);
    d.box = dp->box;
    d.hscale_dev = S.span;
    d.err = S.err;
    d.cptr = nullptr;
    d.clist = nullptr;
    d.ewald = 0;
    memset(pl.tmap, 0, sizeof(pl.tmap));
    int rc = 0;
    if (d.qcells)
        rc = encode_cells<KQ>(&pl.tmap[KQ], d.qcells, dp->ncells);
    if (!rc && d.hcells)
        rc = encode_cells<KH>(&pl.tmap[KH], d.hcells, dp->ncells);
    if (rc)
        return rc;

    cudaStream_t st = (cudaStream_t)stream;
    GC_CHECK(cudaMemsetAsync(base, 0, 256, st));  // queue counters and error word
    // From here on work is queued on the shared scratch: every return waits
    // for the stream first, so that no call leaves kernels behind that could
    // still write the scratch when the next call starts.
    auto finish = [&](int status) {
        const cudaError_t e = cudaStreamSynchronize(st);
        if (status)
            return status;
        return e == cudaSuccess ? 0 : gc::cuda_status(e, "grav_groups_eval_dev_CUDA: evaluation");
    };
    k_dev_setup<<<(unsigned)((ng + 255) / 256), 256, 0, st>>>(dp->groups, dp->pptr, dp->qptr,
                                                               dp->hptr, ng, dp->nbodies, nk, S);
    if (cudaError_t e = cudaGetLastError(); e != cudaSuccess)
        return finish(gc::cuda_status(e, "grav_groups_eval_dev_CUDA: setup launch"));
    if ((rc = launch_kind<KH>(&pl, pl.dp, st)) || (rc = launch_kind<KQ>(&pl, pl.dp, st)) ||
        (rc = launch_kind<KP>(&pl, pl.dp, st)))
        return finish(rc);
    k_finish<<<(unsigned)((ng + 7) / 8), 256, 0, st>>>(pl.dp);
    if (cudaError_t e = cudaGetLastError(); e != cudaSuccess)
        return finish(gc::cuda_status(e, "grav_groups_eval_dev_CUDA: finish launch"));
    unsigned h = 0;
    if (cudaError_t e = cudaMemcpyAsync(&h, S.err, sizeof(h), cudaMemcpyDeviceToHost, st);
        e != cudaSuccess)
        return finish(gc::cuda_status(e, "grav_groups_eval_dev_CUDA: reading the error word"));
    if (int r = finish(0))
        return r;
    if (h)
        return gc::set_status(-2, "grav_groups_eval_dev_CUDA: device error word 0x%x", h);
    return 0;
}

#include "step.cuh"
#include "adjoint.cuh"
