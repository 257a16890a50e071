// build.cu -- the tree build and the MAC walk on the GPU: the producer side
// of the batched lists (nlnhost.h's nln_tree_build + nln_tree_walk) without
// leaving the device.
//
// Every step follows the host builder and shares its arithmetic
// (host/tree_math.h), and this file is compiled without fused
// multiply-adds (-fmad=false) as the host library is without contraction,
// so the tables and lists are bit-identical to the host's:
//   bounding cube     exact min / max of the FP32 positions, enlarged on the host as nlnhost.cpp
//   Morton keys       21 bits per axis, stable radix sort of (key, input index)
//   cells             level-synchronous octant splits of the sorted keys, two kernels a level
//   moments           FP64 sums over each cell's bodies in the canonical blocked order of
//                     nlnhost.cpp (64 bodies, 64 partials, then in order): one thread per
//                     block at each of the three levels
//   tables, rcrit     nln_cell_tables, nln_cell_rcrit (tree_math.h), one thread per cell
//   sink groups       the runs of nlnhost.cpp's collect_groups: small children of every
//                     large cell merged in order, sorted by first body
//   walk              nln_walk_cell (tree_math.h), one warp per group: a counting pass,
//                     offsets, a filling pass in nln_walk_group's order
// Algorithms restated from the reference: nln/cofm.c:96-231,247-574 (moments,
// critical radii), nln/mac.c:1774-1844 (DLRcritMAC), nln/mac.c:91-111 (images).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cub/cub.cuh>
#include <vector>

#include "build.cuh"
#include "common.cuh"
#include "host/tree_math.h"

namespace {

constexpr int KEY_LEVELS = 21;
constexpr int kSumBlock = 64;  // the canonical sum's block (nlnhost.cpp)
constexpr int kThreads = 256;

double now_s() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch())
        .count();
}

__host__ __device__ inline uint64_t spread3(uint32_t v) {
    uint64_t x = v & 0x1fffff;
    x = (x | x << 32) & 0x1f00000000ffffULL;
    x = (x | x << 16) & 0x1f0000ff0000ffULL;
    x = (x | x << 8) & 0x100f00f00f00f00fULL;
    x = (x | x << 4) & 0x10c30c30c30c30c3ULL;
    x = (x | x << 2) & 0x1249249249249249ULL;
    return x;
}

unsigned grid_of(int64_t n, int threads = kThreads) {
    return (unsigned)std::max<int64_t>(1, (n + threads - 1) / threads);
}

// device buffers freed at the end of the build unless released to the
// caller; from a memory pool (stream-ordered on st) when one is given
struct Bufs {
    cudaMemPool_t pool = nullptr;
    cudaStream_t st = nullptr;
    std::vector<void *> held;
    ~Bufs() {
        for (void *p : held) free_one(p);
    }
    void free_one(void *p) {
        if (pool)
            cudaFreeAsync(p, st);
        else
            cudaFree(p);
    }
    template <typename T>
    cudaError_t get(T **p, size_t n) {
        *p = nullptr;
        const size_t bytes = std::max<size_t>(1, n) * sizeof(T);
        cudaError_t e = pool ? gc::pool_malloc((void **)p, bytes, pool, st)
                             : cudaMalloc((void **)p, bytes);
        if (e == cudaSuccess)
            held.push_back(*p);
        return e;
    }
    template <typename T>
    void release(T *p) {  // ownership passes on
        auto it = std::find(held.begin(), held.end(), (void *)p);
        if (it != held.end())
            held.erase(it);
    }
    template <typename T>
    void drop(T *p) {
        auto it = std::find(held.begin(), held.end(), (void *)p);
        if (it != held.end()) {
            free_one(*it);
            held.erase(it);
        }
    }
};

#define BC(call)                                                       \
    do {                                                               \
        cudaError_t _e = (call);                                       \
        if (_e != cudaSuccess)                                         \
            return gc::cuda_status(_e, "GPU tree build: " #call);     \
    } while (0)

// ------------------------------------------------------------ bounding cube
// Per-block min / max of the positions; a non-finite position, or with
// box > 0 one outside [0, box), sets *bad.
__global__ void k_bbox(const float4 *__restrict__ b, int64_t n, double box, float *blo, float *bhi,
                       unsigned *bad) {
    __shared__ float slo[3][kThreads], shi[3][kThreads];
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    unsigned flag = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float4 p = b[i];
        const float x[3] = {p.x, p.y, p.z};
        for (int d = 0; d < 3; d++) {
            if (!isfinite(x[d]) || (box > 0 && !(x[d] >= 0.0f && (double)x[d] < box)))
                flag = 1;
            lo[d] = fminf(lo[d], x[d]);
            hi[d] = fmaxf(hi[d], x[d]);
        }
    }
    if (flag)
        atomicOr(bad, 1u);
    for (int d = 0; d < 3; d++) {
        slo[d][threadIdx.x] = lo[d];
        shi[d][threadIdx.x] = hi[d];
    }
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w)
            for (int d = 0; d < 3; d++) {
                slo[d][threadIdx.x] = fminf(slo[d][threadIdx.x], slo[d][threadIdx.x + w]);
                shi[d][threadIdx.x] = fmaxf(shi[d][threadIdx.x], shi[d][threadIdx.x + w]);
            }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int d = 0; d < 3; d++) {
            blo[3 * blockIdx.x + d] = slo[d][0];
            bhi[3 * blockIdx.x + d] = shi[d][0];
        }
}

// ------------------------------------------------------------ keys, sort, permute
__global__ void k_keys(const float4 *__restrict__ b, int64_t n, double ox, double oy, double oz,
                       double scale, uint64_t *key, int64_t *idx) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const float4 p = b[i];
    const double x[3] = {p.x, p.y, p.z}, o[3] = {ox, oy, oz};
    uint32_t c[3];
    for (int d = 0; d < 3; d++) {
        const double u = (x[d] - o[d]) * scale;
        int64_t v = (int64_t)floor(u);
        v = v < 0 ? 0 : (v > (1 << KEY_LEVELS) - 1 ? (1 << KEY_LEVELS) - 1 : v);
        c[d] = (uint32_t)v;
    }
    key[i] = spread3(c[0]) << 2 | spread3(c[1]) << 1 | spread3(c[2]);
    idx[i] = i;
}

__global__ void k_permute(const float4 *__restrict__ b, const int64_t *__restrict__ order,
                          int64_t n, float *spos, float *smass, float4 *points) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const float4 p = b[order[i]];
    spos[3 * i] = p.x;
    spos[3 * i + 1] = p.y;
    spos[3 * i + 2] = p.z;
    smass[i] = p.w;
    points[i] = p;
}

// ------------------------------------------------------------ cells
struct Cells {
    int64_t *first;
    int32_t *count, *child, *nchild;
    double *gc;    // 3 per cell
    double *side;
};

// One level of the tree, two kernels, with the level's cells [lo, hi) in
// device memory (state[2 l], state[2 l + 1]): the host launches every level
// without waiting for the one before (100k-body sphere: 0.76 -> 0.25 ms; its
// 20 levels had waited for two copies each).  A block takes a contiguous part
// of the level, so that the children, appended in order, land as
// nlnhost.cpp's build_cells puts them.
constexpr int kSplitBlocks = 296;
constexpr int kSplitThreads = 256;
constexpr int kMaxLevels = KEY_LEVELS + 2;

__device__ inline void split_part(const int64_t *state, int level, int64_t &lo, int64_t &hi,
                                  int64_t &b, int64_t &e) {
    lo = state[2 * level];
    hi = state[2 * level + 1];
    const int64_t per = (hi - lo + kSplitBlocks - 1) / kSplitBlocks;
    b = min(hi, lo + blockIdx.x * per);
    e = min(hi, b + per);
}

// Children per octant by binary search of the sorted keys, a thread per cell
// and octant: bounds[8 c + o] the end of octant o, relative to the cell's first
// body; sums[block] the part's children.
__global__ void __launch_bounds__(kSplitThreads)
    k_split_count(Cells C, const int64_t *__restrict__ state, int level,
                  const uint64_t *__restrict__ keys, int leaf_max, int32_t *bounds, int32_t *sums) {
    int64_t lo, hi, b, e;
    split_part(state, level, lo, hi, b, e);
    const int o = threadIdx.x & 7;
    int kids = 0;
    for (int64_t c = b + threadIdx.x / 8; c < e; c += kSplitThreads / 8) {
        const int32_t cnt = C.count[c];
        const bool open = cnt > leaf_max && level < KEY_LEVELS;
        const int64_t first = C.first[c];
        int64_t a = first;
        if (open) {
            const int shift = 3 * (KEY_LEVELS - 1 - level);
            int64_t bb = first + cnt;
            while (a < bb) {
                const int64_t mid = (a + bb) / 2;
                if ((int)((keys[mid] >> shift) & 7) <= o)
                    a = mid + 1;
                else
                    bb = mid;
            }
        }
        const int32_t end = (int32_t)(a - first);
        // a cell's eight threads are neighbours of one warp and take this turn together
        const unsigned eight = 0xffu << (threadIdx.x & 24);
        const int32_t before = __shfl_up_sync(eight, end, 1, 8);
        bounds[8 * c + o] = open ? end : 0;
        kids += open && end > (o ? before : 0) ? 1 : 0;
    }
    typedef cub::BlockReduce<int, kSplitThreads> Reduce;
    __shared__ typename Reduce::TempStorage tmp;
    const int total = Reduce(tmp).Sum(kids);
    if (threadIdx.x == 0)
        sums[blockIdx.x] = total;
}

// The children, in order behind the level; state gets the next level's cells.
// Beyond cap cells nothing is written and *over set.
__global__ void __launch_bounds__(kSplitThreads)
    k_split_write(Cells C, int64_t *state, int level, const int32_t *__restrict__ bounds,
                  const int32_t *__restrict__ sums, int64_t cap, unsigned *over) {
    int64_t lo, hi, b, e;
    split_part(state, level, lo, hi, b, e);
    typedef cub::BlockReduce<int64_t, kSplitThreads> Reduce;
    typedef cub::BlockScan<int, kSplitThreads> Scan;
    __shared__ union {
        typename Reduce::TempStorage r;
        typename Scan::TempStorage s;
    } tmp;
    __shared__ int64_t sh[2];
    int64_t before = 0, all = 0;  // children of the parts before this one, and of the level
    for (int k = threadIdx.x; k < kSplitBlocks; k += kSplitThreads) {
        all += sums[k];
        before += k < (int)blockIdx.x ? sums[k] : 0;
    }
    before = Reduce(tmp.r).Sum(before);
    __syncthreads();
    all = Reduce(tmp.r).Sum(all);
    if (threadIdx.x == 0) {
        sh[0] = before;
        sh[1] = all;
    }
    __syncthreads();
    int64_t base = hi + sh[0];
    const bool fits = hi + sh[1] <= cap;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        state[2 * level + 2] = hi;
        state[2 * level + 3] = fits ? hi + sh[1] : hi;
        if (!fits)
            *over = 1;
    }
    if (!fits)
        return;
    for (int64_t c0 = b; c0 < e; c0 += kSplitThreads) {
        const int64_t c = c0 + threadIdx.x;
        int nk = 0;
        if (c < e)
            for (int o = 0; o < 8; o++) nk += bounds[8 * c + o] > (o ? bounds[8 * c + o - 1] : 0);
        int off, total;
        __syncthreads();
        Scan(tmp.s).ExclusiveSum(nk, off, total);
        if (nk > 0) {
            C.child[c] = (int32_t)(base + off);
            C.nchild[c] = (int32_t)nk;
            const double side = C.side[c];
            const int64_t first = C.first[c];
            int64_t d = base + off;
            for (int o = 0; o < 8; o++) {
                const int32_t x = o ? bounds[8 * c + o - 1] : 0, y = bounds[8 * c + o];
                if (y <= x)
                    continue;
                C.first[d] = first + x;
                C.count[d] = y - x;
                C.child[d] = -1;
                C.nchild[d] = 0;
                C.side[d] = 0.5 * side;
                C.gc[3 * d] = C.gc[3 * c] + ((o >> 2) & 1 ? 0.25 : -0.25) * side;
                C.gc[3 * d + 1] = C.gc[3 * c + 1] + ((o >> 1) & 1 ? 0.25 : -0.25) * side;
                C.gc[3 * d + 2] = C.gc[3 * c + 2] + ((o >> 0) & 1 ? 0.25 : -0.25) * side;
                d++;
            }
        }
        base += total;
    }
}

__global__ void k_split_root(Cells C, int32_t n, double g0, double g1, double g2, double side,
                             int64_t *state) {
    C.first[0] = 0;
    C.count[0] = n;
    C.child[0] = -1;
    C.nchild[0] = 0;
    C.gc[0] = g0;
    C.gc[1] = g1;
    C.gc[2] = g2;
    C.side[0] = side;
    state[0] = 0;
    state[1] = 1;
}

// ------------------------------------------------------------ canonical sums
// Pass 1 (K = 4): mass and offset sums about the geometric centre; pass 2
// (K = NLN_NMOM, + 1 max): raw moments about the centre of mass.  Level 0:
// one thread per block of 64 bodies of a cell; level 1: per block of 64
// level-0 partials; level 2: per cell, its level-1 partials in order.
__global__ void k_sum_blocks(const Cells C, int64_t ncells, int64_t *b0, int64_t *b1) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c > ncells)
        return;
    const int64_t n = c < ncells ? (C.count[c] + kSumBlock - 1) / kSumBlock : 0;
    b0[c] = n;
    b1[c] = (n + kSumBlock - 1) / kSumBlock;
}

template <int K>
__device__ inline void body_terms(const float *spos, const float *smass, int64_t b,
                                  const double *ctr, double *a, double &mx) {
    if (K == 4)
        nln_mass_terms(spos + 3 * b, smass[b], ctr, a);
    else
        mx = fmax(mx, nln_moment_terms(spos + 3 * b, smass[b], ctr, a));
}

__device__ inline int64_t owner(const int64_t *off, int64_t ncells, int64_t j) {
    int64_t a = 0, b = ncells;  // the last cell c with off[c] <= j
    while (b - a > 1) {
        const int64_t mid = (a + b) / 2;
        if (off[mid] <= j)
            a = mid;
        else
            b = mid;
    }
    return a;
}

template <int K>
__global__ void k_sum0(const Cells C, int64_t ncells, const int64_t *__restrict__ o0,
                       int64_t total, const float *spos, const float *smass, const double *ctr,
                       double *p0) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= total)
        return;
    const int64_t c = owner(o0, ncells, j);
    const int64_t blk = j - o0[c];
    const int64_t first = C.first[c], cnt = C.count[c];
    const double cc[3] = {ctr[3 * c], ctr[3 * c + 1], ctr[3 * c + 2]};
    double a[K + 1];
    for (int q = 0; q <= K; q++) a[q] = 0.0;
    double mx = 0.0;
    const int64_t k1 = cnt < (blk + 1) * kSumBlock ? cnt : (blk + 1) * kSumBlock;
    for (int64_t k = blk * kSumBlock; k < k1; k++) body_terms<K>(spos, smass, first + k, cc, a, mx);
    a[K] = mx;
    for (int q = 0; q <= K; q++) p0[j * (K + 1) + q] = a[q];
}

// A thread per block and component: each component's partials in their order.
template <int K>
__global__ void k_sum1(const Cells C, int64_t ncells, const int64_t *__restrict__ o0,
                       const int64_t *__restrict__ o1, int64_t total, const double *p0,
                       double *p1) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t j = i / (K + 1);
    const int q = (int)(i - j * (K + 1));
    if (j >= total)
        return;
    const int64_t c = owner(o1, ncells, j);
    const int64_t blk = j - o1[c];
    const int64_t nb0 = o0[c + 1] - o0[c];
    double a = 0.0;
    const int64_t k1 = nb0 < (blk + 1) * kSumBlock ? nb0 : (blk + 1) * kSumBlock;
    for (int64_t k = blk * kSumBlock; k < k1; k++) {
        const double s = p0[(o0[c] + k) * (K + 1) + q];
        a = q < K ? a + s : fmax(a, s);
    }
    p1[j * (K + 1) + q] = a;
}

// Level 2 of pass 1: the centre of mass (nlnhost.cpp compute_moments).
__global__ void k_sum2_mass(const Cells C, int64_t ncells, const int64_t *__restrict__ o1,
                            const double *p1, double *cen, double *mass) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells)
        return;
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    for (int64_t k = o1[c]; k < o1[c + 1]; k++)
        for (int q = 0; q < 4; q++) a[q] += p1[k * 5 + q];
    const double m = a[0];
    for (int d = 0; d < 3; d++) cen[3 * c + d] = C.gc[3 * c + d] + (m > 0 ? a[1 + d] / m : 0.0);
    mass[c] = m;
}

// Level 2 of pass 2, then the cell's table records and critical radii and
// its walk record.
__global__ void k_sum2_tables(const Cells C, int64_t ncells, int64_t n,
                              const int64_t *__restrict__ o1, const double *p1, const double *cen,
                              const double *mass, nln_mac P, float4 *points, nln_qcell *qc,
                              nln_hcell *hc, nln_wcell *wc) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells)
        return;
    constexpr int K = NLN_NMOM;
    double mo[K];
    for (int q = 0; q < K; q++) mo[q] = 0.0;
    double bmax2 = 0.0;
    for (int64_t k = o1[c]; k < o1[c + 1]; k++) {
        for (int q = 0; q < K; q++) mo[q] += p1[k * (K + 1) + q];
        bmax2 = fmax(bmax2, p1[k * (K + 1) + K]);
    }
    const double cc[3] = {cen[3 * c], cen[3 * c + 1], cen[3 * c + 2]};
    const double m = mass[c], bmax = sqrt(bmax2);
    nln_qcell q;
    nln_hcell h;
    float pt[4];
    nln_cell_tables(cc, m, bmax, mo, pt, &q, &h);
    points[n + c] = make_float4(pt[0], pt[1], pt[2], pt[3]);
    qc[c] = q;
    hc[c] = h;
    double rc[3];
    nln_cell_rcrit(P, C.count[c], m, bmax, mo[31], mo[32], mo[33], rc);
    nln_wcell w;
    for (int d = 0; d < 3; d++) w.cen[d] = cc[d];
    w.bmax = bmax;
    for (int d = 0; d < 3; d++) w.rc[d] = rc[d];
    w.first = C.first[c];
    w.count = C.count[c];
    w.child = C.child[c];
    w.nchild = C.nchild[c];
    w.pad = 0;
    wc[c] = w;
}

// ------------------------------------------------------------ sink groups
// The runs of nlnhost.cpp collect_groups: the root alone when it is small
// (<= gmax bodies, or a leaf); for every large cell, its small children in
// order, adjacent ones merged while the run stays within gmax.
__global__ void k_runs(const Cells C, int64_t ncells, int gmax, int64_t *nruns, int64_t *rfirst,
                       int32_t *rcount) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells)
        return;
    const bool small = C.count[c] <= gmax || C.child[c] < 0;
    int nr = 0;
    if (small) {
        if (c == 0) {
            rfirst[0] = C.first[0];
            rcount[0] = C.count[0];
            nr = 1;
        }
    } else {
        int64_t mf = -1;
        int32_t mc = 0;
        for (int k = 0; k < C.nchild[c]; k++) {
            const int64_t d = C.child[c] + k;
            if (C.count[d] > gmax && C.child[d] >= 0)
                continue;
            if (mf >= 0 && mf + mc == C.first[d] && mc + C.count[d] <= gmax) {
                mc += C.count[d];
            } else {
                if (mf >= 0) {
                    rfirst[8 * c + nr] = mf;
                    rcount[8 * c + nr] = mc;
                    nr++;
                }
                mf = C.first[d];
                mc = C.count[d];
            }
        }
        if (mf >= 0) {
            rfirst[8 * c + nr] = mf;
            rcount[8 * c + nr] = mc;
            nr++;
        }
    }
    nruns[c] = nr;
}

__global__ void k_runs_compact(int64_t ncells, const int64_t *nruns, const int64_t *roff,
                               const int64_t *rfirst, const int32_t *rcount, int64_t *first,
                               int32_t *count) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells)
        return;
    for (int r = 0; r < nruns[c]; r++) {
        first[roff[c] + r] = rfirst[8 * c + r];
        count[roff[c] + r] = rcount[8 * c + r];
    }
}

// Runs longer than gmax (a leaf of coincident bodies that cannot split) as
// consecutive pieces of gmax bodies, the last one the remainder, as
// nlnhost.cpp splits them: pieces of run r start at poff[r].
__global__ void k_run_pieces(int64_t nr, const int64_t *rfirst, const int32_t *rcount,
                             const int64_t *poff, int gmax, int64_t *first, int32_t *count) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nr)
        return;
    int64_t o = poff[r];
    for (int32_t k = 0; k < rcount[r]; k += gmax) {
        first[o] = rfirst[r] + k;
        count[o] = rcount[r] - k < gmax ? rcount[r] - k : gmax;
        o++;
    }
}

__global__ void k_piece_count(int64_t nr, const int32_t *rcount, int gmax, int64_t *np) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r < nr)
        np[r] = (rcount[r] + gmax - 1) / gmax;
}

// Group records: FP64 centre of mass of its sinks in order, radius.
__global__ void k_groups(int64_t ng, const int64_t *first, const int32_t *count,
                         const float *spos, const float *smass, nln_group *groups) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ng)
        return;
    const int64_t f = first[g];
    const int32_t cnt = count[g];
    const float *P = spos + 3 * f;
    const float *M = smass + f;
    double m = 0, s[3] = {0, 0, 0};
    for (int32_t k = 0; k < cnt; k++) {
        m += M[k];
        for (int d = 0; d < 3; d++) s[d] += M[k] * (double)P[3 * k + d];
    }
    nln_group G;
    double r2max = 0;
    for (int d = 0; d < 3; d++) G.cen[d] = m > 0 ? s[d] / m : (double)P[d];
    for (int32_t k = 0; k < cnt; k++) {
        double r2 = 0;
        for (int d = 0; d < 3; d++) {
            const double x = (double)P[3 * k + d] - G.cen[d];
            r2 += x * x;
        }
        r2max = fmax(r2max, r2);
    }
    G.first = f;
    G.count = cnt;
    G.radius = (float)(sqrt(r2max) * (1.0 + 1e-6));
    groups[g] = G;
}

// ------------------------------------------------------------ walk
// One warp per group.  A warp keeps the group's pending cells on a stack in
// shared memory, first in walk order on top, and every round takes the top
// 32 of them, one per lane (nln_walk_cell, the host walk's own decision).
// The counting pass needs no order: opened cells put their children back,
// the rest is counted.  The filling pass must write the host walk's order:
// the leading lanes that opened nothing are final and written at once,
// coalesced, and the lanes behind the first opened cell go back in place, an
// opened cell as its children, a decided one marked with its decision, so no
// cell is decided twice.  Bounded by the FP64 decision and the scattered
// 80-byte cell records, with the walk's parallelism 32 times the group count;
// one thread per group had too few threads below a million bodies and wrote
// every entry uncoalesced (both passes, 100k-body sphere 50.6 -> 1.65 ms, 96^3
// box 71 -> 16 ms, 160^3 238 -> 117 ms).  Issue slots are 62 to 71 % busy;
// single-precision bounds in place of the FP64 square roots changed nothing.
constexpr int kWalkWarps = 4;
// Stack entries per warp, of which the last NLN_WALK_STACK are kept for an
// ordinary depth-first walk: lanes whose children would reach into them go
// back undecided, all but the first, so a round always gets on and the stack
// never fills.
constexpr int kWalkStack = 768;

enum { W_OPEN = 0, W_MARK = 5 };  // 1..4: NLN_MONO..NLN_LEAF, decided; 5: a correction entry alone
constexpr uint32_t kWalkCell = NLN_IDX_MASK;
constexpr int kWalkType = 27;     // bits 27-29: W_OPEN, NLN_*, W_MARK
constexpr int kWalkFlag = 30;     // undecided: bit 30 covered; decided: 1 cell, 2 bodies to the
                                  // correction list
constexpr uint8_t kOwnImages = 31;  // image code of a leaf whose bodies take their own images

__device__ __forceinline__ nln_wcell load_wcell(const nln_wcell *wc, uint32_t i) {
    static_assert(sizeof(nln_wcell) == 80, "five 16-byte loads");
    union {
        double2 d[5];
        nln_wcell c;
    } u;
    const double2 *s = reinterpret_cast<const double2 *>(wc + i);
#pragma unroll
    for (int k = 0; k < 5; k++) u.d[k] = __ldg(s + k);
    return u.c;
}

// inclusive warp scan
__device__ __forceinline__ int warp_scan(int v, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d)
            v += u;
    }
    return v;
}

__device__ __forceinline__ int64_t warp_sum(int64_t v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

// The runs (first[l], n[l] entries) of the lanes, one after another, at
// out[pos..end): entry j of a run is first + j with the run's image code, or
// with kOwnImages the body's own image.  Returns the new position; writes
// stay below end.
__device__ __forceinline__ int64_t emit_runs(uint32_t *out, int64_t pos, int64_t end,
                                             uint32_t first, int n, uint32_t code, int lane,
                                             const float *spos, const nln_group &G, double box) {
    const unsigned FULL = 0xffffffffu;
    if (!__any_sync(FULL, n > 1)) {  // cells only: one entry per lane at most
        const unsigned m = __ballot_sync(FULL, n == 1);
        const int64_t k = pos + __popc(m & ((1u << lane) - 1u));
        if (n == 1 && code != kOwnImages && k < end)
            out[k] = first | code << NLN_IDX_BITS;
        if (!__any_sync(FULL, n == 1 && code == kOwnImages))
            return pos + __popc(m);
    }
    const int inc = warp_scan(n, lane);
    const int total = __shfl_sync(FULL, inc, 31);
    constexpr int U = 4;  // searches in flight
    for (int j0 = 0; j0 < total; j0 += 32 * U) {
        int owner[U];  // lanes whose runs all lie before entry j0 + 32 u + lane
#pragma unroll
        for (int u = 0; u < U; u++) owner[u] = 0;
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1)
#pragma unroll
            for (int u = 0; u < U; u++)
                if (__shfl_sync(FULL, inc, owner[u] + step - 1) <= j0 + 32 * u + lane)
                    owner[u] += step;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int j = j0 + 32 * u + lane, o = min(owner[u], 31);
            const uint32_t f = __shfl_sync(FULL, first, o);
            const int b = __shfl_sync(FULL, inc - n, o);
            uint32_t c = __shfl_sync(FULL, code, o);
            if (j < total && pos + j < end) {
                const uint32_t e = f + (uint32_t)(j - b);
                if (c == kOwnImages) {
                    const float *x = spos + 3 * (int64_t)e;
                    int sb[3];
                    for (int d = 0; d < 3; d++) sb[d] = nln_image(x[d] - G.cen[d], box);
                    c = nln_shift_code(sb);
                }
                out[pos + j] = e | c << NLN_IDX_BITS;
            }
        }
    }
    return pos + total;
}

// The walk's units in order: first the groups whose radius is a sixteenth of
// the cube or more (a sphere's sparse outskirts, any group of a small
// problem), which open most of the tree and would end last alone: eight units
// each, one per child of the root.  Then the others, a unit each.  Both as the
// groups lie in space.
constexpr int kWalkParts = 8;

__global__ void k_wide_groups(const nln_group *__restrict__ groups, int64_t ng, double wide,
                              int64_t *flag) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g <= ng)
        flag[g] = g < ng && groups[g].radius >= wide ? 1 : 0;
}

__global__ void k_walk_order(const nln_group *__restrict__ groups, int64_t ng, double wide,
                             const int64_t *__restrict__ before, int32_t *order) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g < ng)
        order[groups[g].radius >= wide ? before[g] : before[ng] + g - before[g]] = (int32_t)g;
}

// FILL false: cnt[6 g ..] = point, quadrupole, order-4 and correction
// entries, bodies among the points, bodies covered; ucnt[5 u ..] the first five
// of unit u of the wide groups.  FILL true: the entries, at the offsets pp, qp,
// hp, cp (ngroups + 1 each) of the four lists.
// PARTS: there are wide groups (nwide > 0); without them the kernel keeps to
// fewer registers.
template <bool FILL, bool PARTS>
__global__ void __launch_bounds__(32 * kWalkWarps)
    k_walk(const nln_wcell *__restrict__ wc, const float *__restrict__ spos, int64_t n,
           const nln_group *__restrict__ groups, const int32_t *__restrict__ order, int64_t ng,
           int64_t nwide, nln_mac P, int64_t *cnt, int64_t *ucnt, const int64_t *pp, const int64_t *qp, const int64_t *hp, const int64_t *cp,
           uint32_t *pl, uint32_t *ql, uint32_t *hl, uint32_t *cl, unsigned *err) {
    __shared__ uint32_t s_item[kWalkWarps][kWalkStack];
    __shared__ uint8_t s_code[kWalkWarps][FILL ? kWalkStack : 1];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t u = (int64_t)blockIdx.x * kWalkWarps + wib;
    const bool parts = PARTS && u < kWalkParts * nwide;
    const int64_t slot = parts ? u / kWalkParts : PARTS ? u - (kWalkParts - 1) * nwide : u;
    if (slot >= ng)
        return;
    const int part = (int)(u % kWalkParts);
    const int64_t g = PARTS ? order[slot] : slot;
    uint32_t *item = s_item[wib];
    uint8_t *codes = s_code[wib];
    const nln_group G = groups[g];
    const uint32_t nb = (uint32_t)n;
    const bool periodic = P.box > 0;
    int64_t covered = 0;               // this lane's
    int64_t np = 0, nbod = 0, nc = 0;  // counting: this lane's; filling: the warp's positions
    int64_t nq = 0, nh = 0;
    int64_t ep = 0, eq = 0, eh = 0, ec = 0;
    if (FILL) {
        np = pp[g], nq = qp[g], nh = hp[g], nc = cp[g];
        ep = pp[g + 1], eq = qp[g + 1], eh = hp[g + 1], ec = cp[g + 1];
        if (parts) {  // this part's range follows the parts before it
            const int64_t *c = ucnt + 5 * (u - part);
            for (int k = 0; k < part; k++)
                np += c[5 * k], nq += c[5 * k + 1], nh += c[5 * k + 2], nc += c[5 * k + 3];
        }
    }
    int sp = 1;
    if (lane == 0)
        item[0] = 0;
    if (parts) {
        // the root decides alike in every part: opened, part k walks its child
        // k; else part 0 walks the root itself
        const nln_wcell root = load_wcell(wc, 0);
        const nln_visit v = nln_walk_cell(root, G, P, false);
        if (v.what == NLN_OPEN) {
            sp = part < root.nchild ? 1 : 0;
            if (lane == 0)
                item[0] = (uint32_t)(root.child + part) | (v.covers ? 1u << kWalkFlag : 0u);
            if (v.covers && part == 0) {  // the root's own correction entry
                if (FILL) {
                    if (lane == 0 && nc < ec)
                        cl[nc] = nb | v.sc << NLN_IDX_BITS;
                    nc++;
                } else if (lane == 0) {
                    nc = 1;
                }
            }
        } else if (part > 0) {
            sp = 0;
        }
    }
    __syncwarp();
    bool overflow = false;
    while (sp > 0) {
        int w = min(32, sp);
        const bool mine = lane < w;
        uint32_t it = 0;
        uint32_t code = NLN_SHIFT_NONE;
        if (mine) {
            it = item[sp - 1 - lane];
            if (FILL)
                code = codes[sp - 1 - lane];
        }
        const uint32_t ci = it & kWalkCell;
        int type = mine ? (int)(it >> kWalkType & 7u) : W_MARK;
        int cflag = FILL && mine ? (int)(it >> kWalkFlag) : 0;
        int kids = 0, child = 0;
        int32_t bodies = 0;
        uint32_t first = 0;
        bool covers = false, ccov = false, opened = false, decided = false;
        if (mine && type == W_OPEN) {
            const nln_wcell c = load_wcell(wc, ci);
            ccov = (it >> kWalkFlag & 1u) != 0;
            const nln_visit v = nln_walk_cell(c, G, P, ccov);
            covers = v.covers;
            code = v.sc;
            ccov |= covers;
            first = (uint32_t)c.first;
            bodies = c.count;
            if (v.what == NLN_OPEN) {
                opened = true;
                child = c.child;
                kids = c.nchild;
            } else {
                decided = true;
                type = v.what;
                // the correction list gets the cell, or an uncovered leaf's bodies
                cflag = !periodic ? 0 : covers ? 1 : ccov ? 0 : type == NLN_LEAF ? 2 : 1;
                if (type == NLN_LEAF && !v.inside)
                    code = kOwnImages;
            }
        } else if (FILL && mine && type == NLN_LEAF) {
            first = (uint32_t)wc[ci].first;
            bodies = wc[ci].count;
        }
        __syncwarp();  // the window is read: its entries may be overwritten
        // entries each lane puts back, and the lanes whose entries fit with one
        // for each lane behind them: the others stay as they were
        const int slots0 = !mine ? 0 : FILL ? (opened ? kids + (covers ? 1 : 0) : 1) : kids;
        const int inc0 = warp_scan(slots0, lane);
        const bool fits = sp - w + inc0 + (w - 1 - lane) <= kWalkStack - NLN_WALK_STACK;
        const unsigned fit = __ballot_sync(FULL, mine && (fits || lane == 0));
        const int keep = fit == FULL ? 32 : __ffs(~fit) - 1;  // lanes that go through
        w = keep;
        const bool through = lane < w;
        if (through && decided)
            covered += bodies;
        if (!FILL) {
            if (through && mine) {
                np += type == NLN_LEAF ? bodies : type == NLN_MONO ? 1 : 0;
                nbod += type == NLN_LEAF ? bodies : 0;
                nq += type == NLN_QUAD;
                nh += type == NLN_HEXA;
                nc += covers ? 1 : opened ? 0 : cflag == 2 ? bodies : cflag;
            }
            const int total = __shfl_sync(FULL, inc0, w - 1);
            const int base = sp - w;
            if (base + total > kWalkStack) {
                overflow = true;
                break;
            }
            const uint32_t flag = ccov ? 1u << kWalkFlag : 0u;
            if (through)
                for (int k = 0; k < kids; k++)
                    item[base + inc0 - kids + k] = (uint32_t)(child + k) | flag;
            sp = base + total;
            __syncwarp();
            continue;
        }
        const unsigned open = __ballot_sync(FULL, opened && through);
        const int f = open ? __ffs(open) - 1 : w;
        // lanes before f are final: write them in order
        if (f > 0) {
            const bool fin = lane < f;
            const uint32_t self = nb + ci;
            const int t = fin ? type : W_MARK;
            const bool leaf = t == NLN_LEAF;
            np = emit_runs(pl, np, ep, leaf ? first : self, leaf ? bodies : t == NLN_MONO ? 1 : 0,
                           code, lane, spos, G, P.box);
            const unsigned lt = (1u << lane) - 1u;
            const unsigned mq = __ballot_sync(FULL, t == NLN_QUAD);
            const unsigned mh = __ballot_sync(FULL, t == NLN_HEXA);
            const uint32_t entry = ci | code << NLN_IDX_BITS;
            if (t == NLN_QUAD && nq + __popc(mq & lt) < eq)
                ql[nq + __popc(mq & lt)] = entry;
            if (t == NLN_HEXA && nh + __popc(mh & lt) < eh)
                hl[nh + __popc(mh & lt)] = entry;
            nq += __popc(mq);
            nh += __popc(mh);
            if (periodic) {
                const int cf = fin ? cflag : 0;
                // a leaf that enters whole keeps the cell's own image code
                uint32_t cc = code;
                if (cf == 1 && code == kOwnImages)
                    cc = nln_walk_cell(load_wcell(wc, ci), G, P, false).sc;
                nc = emit_runs(cl, nc, ec, cf == 2 ? first : self, cf == 2 ? bodies : cf, cc, lane,
                               spos, G, P.box);
            }
        }
        // lanes f .. w-1 go back on the stack in place
        const bool mark = opened && covers;
        const int slots = lane < f || !through ? 0 : slots0;
        const int gone = f > 0 ? __shfl_sync(FULL, inc0, f - 1) : 0;  // the final lanes' entries
        const int inc = inc0 - gone;
        const int top = sp - w + __shfl_sync(FULL, inc, w - 1);
        if (top > kWalkStack) {
            overflow = true;
            break;
        }
        if (slots) {
            int at = top - (inc - slots) - 1;  // this lane's first entry, downwards
            if (opened) {
                if (mark) {
                    item[at] = ci | (uint32_t)W_MARK << kWalkType | 1u << kWalkFlag;
                    codes[at] = (uint8_t)code;
                    at--;
                }
                const uint32_t flag = ccov ? 1u << kWalkFlag : 0u;
                for (int k = 0; k < kids; k++) item[at - k] = (uint32_t)(child + k) | flag;
            } else {
                item[at] = ci | (uint32_t)type << kWalkType | (uint32_t)cflag << kWalkFlag;
                codes[at] = (uint8_t)code;
            }
        }
        sp = top;
        __syncwarp();
    }
    covered = warp_sum(covered);
    if ((overflow || (!parts && covered != n)) && lane == 0)
        atomicOr(err, 1u);
    if (!FILL) {
        np = warp_sum(np);
        nq = warp_sum(nq);
        nh = warp_sum(nh);
        nc = warp_sum(nc);
        nbod = warp_sum(nbod);
        if (lane == 0) {
            const int64_t v[6] = {np, nq, nh, nc, nbod, covered};
            for (int k = 0; k < 6; k++) {
                if (!parts)
                    cnt[6 * g + k] = v[k];
                else
                    atomicAdd(reinterpret_cast<unsigned long long *>(cnt + 6 * g + k),
                              (unsigned long long)v[k]);
                if (parts && k < 5)
                    ucnt[5 * u + k] = v[k];
            }
        }
    } else if (lane == 0) {
        // the count pass sized every list: a walk that writes more or less is an error
        if (parts) {  // where the next part starts
            const int64_t *c = ucnt + 5 * (u - part);
            ep = pp[g], eq = qp[g], eh = hp[g], ec = cp[g];
            for (int k = 0; k <= part; k++)
                ep += c[5 * k], eq += c[5 * k + 1], eh += c[5 * k + 2], ec += c[5 * k + 3];
        }
        if (np != ep || nq != eq || nh != eh || nc != ec)
            atomicOr(err, 2u);
    }
}

template <typename T>
int exclusive_scan(Bufs &B, const T *in, T *out, int64_t n, cudaStream_t st) {
    size_t bytes = 0;
    BC(cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, (int)n, st));
    void *tmp = nullptr;
    BC(B.get((unsigned char **)&tmp, bytes));
    BC(cub::DeviceScan::ExclusiveSum(tmp, bytes, in, out, (int)n, st));
    B.drop(tmp);
    return 0;
}

// The build; on failure every buffer is freed and out's pointers are stale.
int build_tree(const nln_params &p, const float4 *bodies, int64_t n, cudaStream_t st, DevTree &out,
               cudaMemPool_t pool) {
    if (!bodies || n <= 0)
        return gc::set_status(-1, "GPU tree build: no bodies");
    if (p.leaf_max < 1 || p.leaf_max > 65535 || p.group_max < 1 || p.group_max > 64 ||
        p.tol <= 0.0 || p.p2cut < 0 || p.p4cut < 0)
        return gc::set_status(-1, "GPU tree build: bad parameters (leaf_max 1..65535, group_max "
                                  "1..64, tol > 0)");
    if (n + 1 >= (int64_t)NLN_IDX_MASK || n >= (int64_t)INT32_MAX)
        return gc::set_status(-1, "GPU tree build: too many bodies for 27-bit list indices");
    Bufs B;
    B.pool = pool;
    B.st = st;
    out.pool = pool;
    double t0 = now_s();
    // ---- bounding cube (the host arithmetic of nln_tree_build)
    const unsigned bb = 592;
    float *blo = nullptr, *bhi = nullptr;
    unsigned *flag = nullptr;
    BC(B.get(&blo, 3 * bb));
    BC(B.get(&bhi, 3 * bb));
    BC(B.get(&flag, 4));
    BC(cudaMemsetAsync(flag, 0, 4 * sizeof(unsigned), st));
    k_bbox<<<bb, kThreads, 0, st>>>(bodies, n, p.box, blo, bhi, flag);
    BC(cudaGetLastError());
    std::vector<float> hlo(3 * bb), hhi(3 * bb);
    unsigned hbad = 0;
    BC(cudaMemcpyAsync(hlo.data(), blo, 3 * bb * sizeof(float), cudaMemcpyDeviceToHost, st));
    BC(cudaMemcpyAsync(hhi.data(), bhi, 3 * bb * sizeof(float), cudaMemcpyDeviceToHost, st));
    BC(cudaMemcpyAsync(&hbad, flag, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    BC(cudaStreamSynchronize(st));
    if (hbad)
        return gc::set_status(-1, p.box > 0 ? "GPU tree build: periodic body outside [0, box)"
                                            : "GPU tree build: non-finite position");
    double origin[3] = {0, 0, 0}, side = 0;
    if (p.box > 0) {
        side = p.box;
    } else {
        double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (unsigned k = 0; k < bb; k++)
            for (int d = 0; d < 3; d++) {
                lo[d] = std::min(lo[d], (double)hlo[3 * k + d]);
                hi[d] = std::max(hi[d], (double)hhi[3 * k + d]);
            }
        double ext = 0;
        for (int d = 0; d < 3; d++) ext = std::max(ext, hi[d] - lo[d]);
        ext = ext > 0 ? ext * (1.0 + 1e-5) : 1.0;
        for (int d = 0; d < 3; d++) origin[d] = 0.5 * (lo[d] + hi[d]) - 0.5 * ext;
        side = ext;
    }
    // ---- keys, stable sort by (key, index), bodies in tree order
    const double scale = (double)(1u << KEY_LEVELS) / side;
    uint64_t *k_in = nullptr, *k_out = nullptr;
    int64_t *i_in = nullptr;
    BC(B.get(&k_in, n));
    BC(B.get(&k_out, n));
    BC(B.get(&i_in, n));
    BC(B.get(&out.order, n));
    k_keys<<<grid_of(n), kThreads, 0, st>>>(bodies, n, origin[0], origin[1], origin[2], scale,
                                             k_in, i_in);
    BC(cudaGetLastError());
    {
        size_t bytes = 0;
        BC(cub::DeviceRadixSort::SortPairs(nullptr, bytes, k_in, k_out, i_in, out.order, (int)n, 0,
                                           64, st));
        unsigned char *tmp = nullptr;
        BC(B.get(&tmp, bytes));
        BC(cub::DeviceRadixSort::SortPairs(tmp, bytes, k_in, k_out, i_in, out.order, (int)n, 0, 64,
                                           st));
        B.drop(tmp);
    }
    B.drop(k_in);
    B.drop(i_in);
    float *spos = nullptr, *smass = nullptr;
    BC(B.get(&spos, 3 * n));
    BC(B.get(&smass, n));
    // the point table is sized once the cells are known: bodies go to a
    // temporary float4 array first
    float4 *bpts = nullptr;
    BC(B.get(&bpts, n));
    k_permute<<<grid_of(n), kThreads, 0, st>>>(bodies, out.order, n, spos, smass, bpts);
    BC(cudaGetLastError());
    BC(cudaStreamSynchronize(st));
    out.seconds[0] = now_s() - t0;
    t0 = now_s();

    // ---- cells, level by level, in room for 7 n / leaf_max cells (2 n at most): a level whose
    // cells hold just over leaf_max bodies splits them into eight, which makes 6.5 n / leaf_max
    // cells in the worst grids and uniform boxes tried (0.37 n with leaves of 16, 0.20 with 32;
    // spheres 0.25 and 0.15; leaves of one body 1.5).  The plan keeps 20 of the 52 bytes a cell,
    // room included: cutting the arrays to the count costs a build of 64k bodies 0.03 of 2.2 ms.
    // Four times as many where that is too few (tight pairs make long chains), and never more
    // than the list indices could name.
    Cells C{};
    auto too_many = [] {
        return gc::set_status(-1, "GPU tree build: bodies plus cells exceed 27-bit list indices");
    };
    int64_t hstate[2 * (kMaxLevels + 1)];
    const int64_t most = (int64_t)NLN_IDX_MASK - n;
    for (int64_t cap = std::min(most, 1024 + std::min(2 * n, 7 * n / p.leaf_max));;
         cap = std::min(most, 4 * cap)) {
        int32_t *bounds = nullptr, *sums = nullptr;
        int64_t *state = nullptr;
        BC(B.get(&C.first, cap));
        BC(B.get(&C.count, cap));
        BC(B.get(&C.child, cap));
        BC(B.get(&C.nchild, cap));
        BC(B.get(&C.gc, 3 * cap));
        BC(B.get(&C.side, cap));
        BC(B.get(&bounds, 8 * cap));
        BC(B.get(&sums, kSplitBlocks));
        BC(B.get(&state, 2 * (kMaxLevels + 1)));
        BC(cudaMemsetAsync(state, 0, 2 * (kMaxLevels + 1) * sizeof(int64_t), st));
        BC(cudaMemsetAsync(flag, 0, sizeof(unsigned), st));
        k_split_root<<<1, 1, 0, st>>>(C, (int32_t)n, origin[0] + 0.5 * side, origin[1] + 0.5 * side,
                                       origin[2] + 0.5 * side, side, state);
        BC(cudaGetLastError());
        for (int level = 0; level < kMaxLevels; level++) {
            k_split_count<<<kSplitBlocks, kSplitThreads, 0, st>>>(C, state, level, k_out, p.leaf_max,
                                                                   bounds, sums);
            BC(cudaGetLastError());
            k_split_write<<<kSplitBlocks, kSplitThreads, 0, st>>>(C, state, level, bounds, sums, cap,
                                                                   flag);
            BC(cudaGetLastError());
        }
        BC(cudaMemcpyAsync(hstate, state, sizeof(hstate), cudaMemcpyDeviceToHost, st));
        BC(cudaMemcpyAsync(&hbad, flag, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
        BC(cudaStreamSynchronize(st));
        B.drop(bounds);
        B.drop(sums);
        B.drop(state);
        if (!hbad)
            break;
        if (cap == most)
            return too_many();
        B.drop(C.first);
        B.drop(C.count);
        B.drop(C.child);
        B.drop(C.nchild);
        B.drop(C.gc);
        B.drop(C.side);
    }
    int64_t nc = 0;
    for (int level = 0; level < kMaxLevels && hstate[2 * level + 1] > hstate[2 * level]; level++) {
        out.level_start.push_back(hstate[2 * level]);
        nc = hstate[2 * level + 1];
    }
    out.level_start.push_back(nc);
    if (n + nc + 1 >= (int64_t)NLN_IDX_MASK)
        return too_many();
    out.n = n;
    out.ncells = nc;
    out.box = p.box;
    BC(cudaStreamSynchronize(st));
    out.seconds[1] = now_s() - t0;
    t0 = now_s();

    // ---- moments: block offsets of the canonical sums
    int64_t *o0 = nullptr, *o1 = nullptr, *nb = nullptr, *nb1 = nullptr;
    BC(B.get(&o0, nc + 1));
    BC(B.get(&o1, nc + 1));
    BC(B.get(&nb, nc + 1));
    BC(B.get(&nb1, nc + 1));
    k_sum_blocks<<<grid_of(nc + 1), kThreads, 0, st>>>(C, nc, nb, nb1);
    BC(cudaGetLastError());
    if (int rc = exclusive_scan(B, nb, o0, nc + 1, st))
        return rc;
    if (int rc = exclusive_scan(B, nb1, o1, nc + 1, st))
        return rc;
    int64_t B0 = 0, B1 = 0;
    BC(cudaMemcpyAsync(&B0, o0 + nc, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    BC(cudaMemcpyAsync(&B1, o1 + nc, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    BC(cudaStreamSynchronize(st));
    double *cen = nullptr, *mass = nullptr, *p0 = nullptr, *p1 = nullptr;
    BC(B.get(&cen, 3 * nc));
    BC(B.get(&mass, nc));
    // pass 1: centre of mass
    BC(B.get(&p0, B0 * 5));
    BC(B.get(&p1, B1 * 5));
    k_sum0<4><<<grid_of(B0), kThreads, 0, st>>>(C, nc, o0, B0, spos, smass, C.gc, p0);
    BC(cudaGetLastError());
    k_sum1<4><<<grid_of(5 * B1), kThreads, 0, st>>>(C, nc, o0, o1, B1, p0, p1);
    BC(cudaGetLastError());
    k_sum2_mass<<<grid_of(nc), kThreads, 0, st>>>(C, nc, o1, p1, cen, mass);
    BC(cudaGetLastError());
    BC(cudaStreamSynchronize(st));
    B.drop(p0);
    B.drop(p1);
    // pass 2: raw moments, tables, critical radii, walk records
    constexpr int K2 = NLN_NMOM + 1;
    BC(B.get(&p0, B0 * K2));
    BC(B.get(&p1, B1 * K2));
    k_sum0<NLN_NMOM><<<grid_of(B0), kThreads, 0, st>>>(C, nc, o0, B0, spos, smass, cen, p0);
    BC(cudaGetLastError());
    k_sum1<NLN_NMOM><<<grid_of(K2 * B1), kThreads, 0, st>>>(C, nc, o0, o1, B1, p0, p1);
    BC(cudaGetLastError());
    BC(B.get(&out.points, n + nc));
    BC(B.get(&out.qcells, nc));
    BC(B.get(&out.hcells, nc));
    nln_wcell *wc = nullptr;
    BC(B.get(&wc, nc));
    BC(cudaMemcpyAsync(out.points, bpts, n * sizeof(float4), cudaMemcpyDeviceToDevice, st));
    nln_mac P;
    P.tol = p.tol;
    P.rel_tol = p.rel_tol;
    P.rel_tol0 = p.rel_tol0;
    P.ptol_boost = p.ptol_boost;
    P.bmax0 = 0.5 * side;
    P.p2cut = p.p2cut;
    P.p4cut = p.p4cut;
    P.box = p.box;
    P.ewald_theta = p.ewald_theta;
    k_sum2_tables<<<grid_of(nc), kThreads, 0, st>>>(C, nc, n, o1, p1, cen, mass, P, out.points,
                                                     out.qcells, out.hcells, wc);
    BC(cudaGetLastError());
    BC(cudaStreamSynchronize(st));
    B.drop(p0);
    B.drop(p1);
    B.drop(bpts);
    B.drop(cen);
    B.drop(mass);
    B.drop(o0);
    B.drop(o1);
    B.drop(nb);
    B.drop(nb1);
    out.seconds[2] = now_s() - t0;
    t0 = now_s();

    // ---- sink groups
    int32_t *rcount = nullptr, *gcount = nullptr;
    int64_t *nruns = nullptr, *rfirst = nullptr, *roff = nullptr, *gfirst = nullptr;
    BC(B.get(&nruns, nc + 1));
    BC(B.get(&rcount, 8 * nc));
    BC(B.get(&rfirst, 8 * nc));
    BC(B.get(&roff, nc + 1));
    BC(cudaMemsetAsync(nruns, 0, (nc + 1) * sizeof(int64_t), st));
    k_runs<<<grid_of(nc), kThreads, 0, st>>>(C, nc, p.group_max, nruns, rfirst, rcount);
    BC(cudaGetLastError());
    if (int rc = exclusive_scan(B, nruns, roff, nc + 1, st))  // roff[nc] = the run count
        return rc;
    int64_t ng = 0;
    BC(cudaMemcpyAsync(&ng, roff + nc, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    BC(cudaStreamSynchronize(st));
    if (ng <= 0)
        return gc::set_status(-1, "GPU tree build: no sink groups");
    int64_t *ufirst = nullptr;
    int32_t *ucount = nullptr;
    BC(B.get(&ufirst, ng));
    BC(B.get(&ucount, ng));
    BC(B.get(&gfirst, ng));
    BC(B.get(&gcount, ng));
    k_runs_compact<<<grid_of(nc), kThreads, 0, st>>>(nc, nruns, roff, rfirst, rcount, ufirst,
                                                      ucount);
    BC(cudaGetLastError());
    {
        size_t bytes = 0;
        BC(cub::DeviceRadixSort::SortPairs(nullptr, bytes, ufirst, gfirst, ucount, gcount, (int)ng,
                                           0, 64, st));
        unsigned char *tmp = nullptr;
        BC(B.get(&tmp, bytes));
        BC(cub::DeviceRadixSort::SortPairs(tmp, bytes, ufirst, gfirst, ucount, gcount, (int)ng, 0,
                                           64, st));
        B.drop(tmp);
    }
    // split runs longer than group_max
    {
        int64_t *np = nullptr, *poff = nullptr;
        BC(B.get(&np, ng + 1));
        BC(B.get(&poff, ng + 1));
        BC(cudaMemsetAsync(np, 0, (ng + 1) * sizeof(int64_t), st));
        k_piece_count<<<grid_of(ng), kThreads, 0, st>>>(ng, gcount, p.group_max, np);
        BC(cudaGetLastError());
        if (int rc = exclusive_scan(B, np, poff, ng + 1, st))
            return rc;
        int64_t npieces = 0;
        BC(cudaMemcpyAsync(&npieces, poff + ng, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        BC(cudaStreamSynchronize(st));
        if (npieces != ng) {
            int64_t *pf = nullptr;
            int32_t *pc = nullptr;
            BC(B.get(&pf, npieces));
            BC(B.get(&pc, npieces));
            k_run_pieces<<<grid_of(ng), kThreads, 0, st>>>(ng, gfirst, gcount, poff, p.group_max,
                                                            pf, pc);
            BC(cudaGetLastError());
            gfirst = pf;
            gcount = pc;
            ng = npieces;
        }
    }
    BC(B.get(&out.groups, ng));
    k_groups<<<grid_of(ng), kThreads, 0, st>>>(ng, gfirst, gcount, spos, smass, out.groups);
    BC(cudaGetLastError());
    out.ngroups = ng;
    BC(cudaStreamSynchronize(st));
    out.seconds[3] = now_s() - t0;
    t0 = now_s();

    // ---- walk: count, offsets, fill
    int64_t *cnt = nullptr, *ucnt = nullptr;
    BC(B.get(&cnt, 6 * ng));
    BC(cudaMemsetAsync(cnt, 0, 6 * ng * sizeof(int64_t), st));
    BC(cudaMemsetAsync(flag, 0, sizeof(unsigned), st));
    int32_t *worder = nullptr;
    int64_t nwide = 0;
    {
        int64_t *wide = nullptr, *before = nullptr;
        BC(B.get(&wide, ng + 1));
        BC(B.get(&before, ng + 1));
        BC(B.get(&worder, ng));
        k_wide_groups<<<grid_of(ng + 1), kThreads, 0, st>>>(out.groups, ng, side / 16, wide);
        BC(cudaGetLastError());
        if (int rc = exclusive_scan(B, wide, before, ng + 1, st))
            return rc;
        k_walk_order<<<grid_of(ng), kThreads, 0, st>>>(out.groups, ng, side / 16, before, worder);
        BC(cudaGetLastError());
        BC(cudaMemcpyAsync(&nwide, before + ng, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        BC(cudaStreamSynchronize(st));
    }
    // Parts only where at most a quarter of the groups are wide.  Both passes, groups whole and
    // in parts, ms: 30k sphere (60 of 1,350 wide) 0.75, 0.63; 100k (117 of 4,422) 1.60, 1.67; 2k
    // (26 of 96) 0.151, 0.155; but 16^3 box (128 of 130) 0.21, 0.17 and 32^3 (all of 1,024) 0.59,
    // 0.40: a few groups for all the SMs, which would gain from parts and are kept whole here.
    if (4 * nwide > ng)
        nwide = 0;
    const int64_t units = ng + (kWalkParts - 1) * nwide;
    BC(B.get(&ucnt, 5 * kWalkParts * nwide));
    const auto count_pass = nwide ? k_walk<false, true> : k_walk<false, false>;
    const auto fill_pass = nwide ? k_walk<true, true> : k_walk<true, false>;
    count_pass<<<grid_of(units, kWalkWarps), 32 * kWalkWarps, 0, st>>>(
        wc, spos, n, out.groups, worder, ng, nwide, P, cnt, ucnt, nullptr, nullptr, nullptr, nullptr,
        nullptr, nullptr, nullptr, nullptr, flag);
    BC(cudaGetLastError());
    std::vector<int64_t> hc(6 * ng);
    BC(cudaMemcpyAsync(hc.data(), cnt, 6 * ng * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    BC(cudaMemcpyAsync(&hbad, flag, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    out.groups_h.resize(ng);
    BC(cudaMemcpyAsync(out.groups_h.data(), out.groups, ng * sizeof(nln_group),
                       cudaMemcpyDeviceToHost, st));
    BC(cudaStreamSynchronize(st));
    for (int64_t g = 0; g < ng; g++)
        if (hc[6 * g + 5] != n)
            hbad |= 1u;
    if (hbad)
        return gc::set_status(-1, "GPU tree build: a group's walk did not cover every body "
                                  "exactly once, or overflowed its stack");
    const double t_count = now_s() - t0;
    t0 = now_s();
    for (int k = 0; k < 4; k++) out.ptr_h[k].assign(ng + 1, 0);
    for (int64_t g = 0; g < ng; g++) {
        // a group's lists cover every body once: no kind can exceed the point table
        for (int k = 0; k < 5; k++)
            if (hc[6 * g + k] < 0 || hc[6 * g + k] > n + nc)
                return gc::set_status(-1, "GPU tree build: group %lld counted %lld entries",
                                      (long long)g, (long long)hc[6 * g + k]);
        for (int k = 0; k < 4; k++) out.ptr_h[k][g + 1] = out.ptr_h[k][g] + hc[6 * g + k];
        const int64_t c = out.groups_h[g].count, nbod = hc[6 * g + 4];
        out.counts[0] += c * nbod;
        out.counts[1] += c * (hc[6 * g] - nbod);
        out.counts[2] += c * hc[6 * g + 1];
        out.counts[3] += c * hc[6 * g + 2];
    }
    int64_t *dptr[4];
    for (int k = 0; k < 4; k++) {
        out.len[k] = out.ptr_h[k][ng];
        BC(B.get(&out.list[k], out.len[k]));
        BC(B.get(&dptr[k], ng + 1));
        BC(cudaMemcpyAsync(dptr[k], out.ptr_h[k].data(), (ng + 1) * sizeof(int64_t),
                           cudaMemcpyHostToDevice, st));
    }
    out.seconds[5] = now_s() - t0;  // offsets and list allocation
    t0 = now_s();
    BC(cudaMemsetAsync(flag, 0, sizeof(unsigned), st));
    fill_pass<<<grid_of(units, kWalkWarps), 32 * kWalkWarps, 0, st>>>(
        wc, spos, n, out.groups, worder, ng, nwide, P, nullptr, ucnt, dptr[0], dptr[1], dptr[2],
        dptr[3], out.list[0], out.list[1], out.list[2], out.list[3], flag);
    BC(cudaGetLastError());
    BC(cudaMemcpyAsync(&hbad, flag, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    BC(cudaStreamSynchronize(st));
    if (hbad)
        return gc::set_status(-1, "GPU tree build: the filling walk differs from the counting "
                                  "walk (0x%x)", hbad);
    out.seconds[4] = t_count + (now_s() - t0);
    // ---- the tree links and list offsets, handed on
    out.cell_first = C.first;
    out.cell_count = C.count;
    out.cell_child = C.child;
    out.cell_nchild = C.nchild;
    for (int k = 0; k < 4; k++) out.ptr[k] = dptr[k];
    void *keep[] = {out.points, out.qcells, out.hcells, out.groups, out.list[0], out.list[1],
                    out.list[2], out.list[3], out.order, C.first, C.count, C.child, C.nchild,
                    dptr[0], dptr[1], dptr[2], dptr[3]};
    for (void *q : keep) B.release(q);
    return 0;
}

}  // namespace

int gpu_tree_build(const nln_params &p, const float4 *bodies, int64_t n, cudaStream_t st,
                   DevTree &out, cudaMemPool_t pool) {
    out = DevTree{};
    const int rc = build_tree(p, bodies, n, st, out, pool);
    if (rc)
        out = DevTree{};
    return rc;
}

// ------------------------------------------------------------ work queue
namespace {

struct QueueIn {
    const int64_t *ptr[3];
    int64_t chunk[3];
};

// Per group: full chunks of each kind (nfull[k (ng + 1) + g]), the length of
// its remainder (0: none) with the group itself for the sort, and all its
// items (its slots).
__global__ void k_queue_count(QueueIn Q, int64_t ng, int64_t *nfull, uint32_t *rem, int32_t *gid,
                              int64_t *nall) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g > ng)
        return;
    int64_t all = 0;
    for (int k = 0; k < 3; k++) {
        const int64_t len = g < ng && Q.ptr[k] ? Q.ptr[k][g + 1] - Q.ptr[k][g] : 0;
        const int64_t f = len / Q.chunk[k], r = len % Q.chunk[k];
        nfull[k * (ng + 1) + g] = f;
        all += f + (r ? 1 : 0);
        if (g < ng) {
            rem[k * ng + g] = (uint32_t)r;
            gid[k * ng + g] = (int32_t)g;
        }
    }
    nall[g] = all;
}

// Group g's first slot of kind k: after its items of the kinds before.
__device__ inline int64_t kind_slot(const QueueIn &Q, int64_t g, int k, const int64_t *gslot) {
    int64_t s = gslot[g];
    for (int j = 0; j < k; j++)
        if (Q.ptr[j])
            s += (Q.ptr[j][g + 1] - Q.ptr[j][g] + Q.chunk[j] - 1) / Q.chunk[j];
    return s;
}

// Remainders per kind, one atomic per warp.
__global__ void k_queue_nrem(const uint32_t *__restrict__ rem, int64_t ng, unsigned long long *n) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int k = 0; k < 3; k++) {
        const unsigned m = __ballot_sync(0xffffffffu, g < ng && rem[k * ng + g] != 0);
        if ((threadIdx.x & 31) == 0 && m)
            atomicAdd(&n[k], (unsigned long long)__popc(m));
    }
}

__global__ void k_queue_full(QueueIn Q, int k, int64_t ng, const int64_t *__restrict__ off,
                             const int64_t *__restrict__ gslot, Item *items) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ng)
        return;
    const int64_t b = Q.ptr[k][g];
    int64_t slot = kind_slot(Q, g, k, gslot);
    Item *out = items + off[g];
    for (int64_t j = 0; j < off[g + 1] - off[g]; j++)
        out[j] = Item{(int32_t)g, (int32_t)slot++, b + j * Q.chunk[k], b + (j + 1) * Q.chunk[k]};
}

__global__ void k_queue_rem(QueueIn Q, int k, int64_t nrem, const int32_t *__restrict__ gid,
                            const int64_t *__restrict__ gslot, Item *items) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrem)
        return;
    const int32_t g = gid[i];
    const int64_t b = Q.ptr[k][g], e = Q.ptr[k][g + 1], f = (e - b) / Q.chunk[k];
    items[i] = Item{g, (int32_t)(kind_slot(Q, g, k, gslot) + f), b + f * Q.chunk[k], e};
}

}  // namespace

int gpu_make_queue(const int64_t *const ptr[3], int64_t ng, const int64_t chunk[3], cudaStream_t st,
                   cudaMemPool_t pool, Item *items[3], int nitems[3], int64_t **gslot,
                   int64_t *nslots) {
    Bufs B;
    B.pool = pool;
    B.st = st;
    QueueIn Q;
    int64_t most = 1;
    for (int k = 0; k < 3; k++) {
        Q.ptr[k] = ptr[k];
        Q.chunk[k] = chunk[k];
        most = std::max(most, chunk[k]);
        items[k] = nullptr;
        nitems[k] = 0;
    }
    Item *made[3] = {nullptr, nullptr, nullptr};  // the caller's once nothing can fail any more
    int64_t *nfull = nullptr, *off = nullptr, *nall = nullptr, *slots = nullptr;
    uint32_t *rem = nullptr, *rem_s = nullptr;
    int32_t *gid = nullptr, *gid_s = nullptr;
    BC(B.get(&nfull, 3 * (ng + 1)));
    BC(B.get(&off, 3 * (ng + 1)));
    BC(B.get(&nall, ng + 1));
    BC(B.get(&slots, ng + 1));
    BC(B.get(&rem, 3 * ng));
    BC(B.get(&rem_s, 3 * ng));
    BC(B.get(&gid, 3 * ng));
    BC(B.get(&gid_s, 3 * ng));
    k_queue_count<<<grid_of(ng + 1), kThreads, 0, st>>>(Q, ng, nfull, rem, gid, nall);
    BC(cudaGetLastError());
    if (int rc = exclusive_scan(B, nall, slots, ng + 1, st))
        return rc;
    int bits = 1;
    while (bits < 32 && (int64_t)1 << bits < most) bits++;
    int64_t tot[4] = {0, 0, 0, 0};
    for (int k = 0; k < 3; k++) {
        if (!ptr[k])
            continue;
        if (int rc = exclusive_scan(B, nfull + k * (ng + 1), off + k * (ng + 1), ng + 1, st))
            return rc;
        size_t bytes = 0;
        BC(cub::DeviceRadixSort::SortPairsDescending(nullptr, bytes, rem + k * ng, rem_s + k * ng,
                                                     gid + k * ng, gid_s + k * ng, (int)ng, 0, bits, st));
        unsigned char *tmp = nullptr;
        BC(B.get(&tmp, bytes));
        BC(cub::DeviceRadixSort::SortPairsDescending(tmp, bytes, rem + k * ng, rem_s + k * ng,
                                                     gid + k * ng, gid_s + k * ng, (int)ng, 0, bits, st));
        B.drop(tmp);
        BC(cudaMemcpyAsync(&tot[k], off + k * (ng + 1) + ng, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    }
    BC(cudaMemcpyAsync(&tot[3], slots + ng, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    int64_t *nrem_d = nullptr;  // remainders per kind
    BC(B.get(&nrem_d, 3));
    BC(cudaMemsetAsync(nrem_d, 0, 3 * sizeof(int64_t), st));
    k_queue_nrem<<<grid_of(ng), kThreads, 0, st>>>(rem, ng, reinterpret_cast<unsigned long long *>(nrem_d));
    BC(cudaGetLastError());
    int64_t nrem[3];
    BC(cudaMemcpyAsync(nrem, nrem_d, sizeof(nrem), cudaMemcpyDeviceToHost, st));
    BC(cudaStreamSynchronize(st));
    for (int k = 0; k < 3; k++) {
        if (!ptr[k] || tot[k] + nrem[k] == 0)
            continue;
        BC(B.get(&made[k], tot[k] + nrem[k]));
        k_queue_full<<<grid_of(ng), kThreads, 0, st>>>(Q, k, ng, off + k * (ng + 1), slots, made[k]);
        BC(cudaGetLastError());
        if (nrem[k] > 0) {
            k_queue_rem<<<grid_of(nrem[k]), kThreads, 0, st>>>(Q, k, nrem[k], gid_s + k * ng, slots,
                                                                made[k] + tot[k]);
            BC(cudaGetLastError());
        }
    }
    BC(cudaStreamSynchronize(st));
    *gslot = slots;
    *nslots = tot[3];
    for (int k = 0; k < 3; k++) {
        items[k] = made[k];
        nitems[k] = made[k] ? (int)(tot[k] + nrem[k]) : 0;
        B.release(made[k]);
    }
    B.release(slots);
    return 0;
}
