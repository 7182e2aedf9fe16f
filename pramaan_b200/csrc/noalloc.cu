// noalloc.cu — y = A x over a caller-owned device CSR without allocating.
//
// Some callers cannot call cudaMalloc at the point where they need a sparse
// product: a branch-and-bound or rolling-horizon driver that has sized all of
// its device memory up front and runs under a fixed budget, code that runs
// while a stream is being captured into a CUDA graph (cudaMalloc is not a
// stream operation and cudaFree synchronises the device), and hosts that own
// the device memory pool and hand the library only pointers.  For them this
// file provides one entry point, pramaan_spmv_noalloc, that launches work on
// the caller's stream and allocates nothing: no cudaMalloc, no cudaFree, no
// allocating library routine.
//
// The product splits the non-zeros evenly over warps: warp k owns the rows
// that start in entries [k T, (k + 1) T) and streams their entries in tiles of
// 256 (coalesced loads, 8 gathers of x in flight per lane, products through
// shared memory, then the rows of the tile summed by 1 to 8 lanes each, or by
// the whole warp where a row is long).  Owning whole rows leaves nothing to
// combine between warps, except for giant rows (more than 2 T entries): those
// are cut at the range boundaries, every range leaves the sum of its piece, and
// the pieces of a row are added in a fixed order afterwards.  A product that
// fits one thread-block cluster (nnz <= 16,384) does so in the same launch and
// keeps the pieces in the shared memory of the cluster's first block.  A larger
// one keeps them in the scratch array below and adds them in a second,
// dependent launch.  The scratch is a file-scope array: every GPU that loads
// the library holds it (512 KiB) until the process exits, one call is limited
// to nnz <= 134,217,728, and all larger products share it, so when two of them
// overlap on the GPU (on different streams) the sums of their giant rows race;
// calls on one stream are ordered.  What a call reads there it has written
// itself, so nothing needs clearing between calls; a row number that another
// call left there is checked against the call's own row_ptr before it is used.
//
// What bounds it: the gathers.  B200 serves random 4-byte gathers at about one
// sector per SM per clock (ceiling.cu), 14 us for 4 M entries and 97 us for
// 27 M, and the stream's own sectors share that path.  Small products are
// bound by the chain search - row pointers - entries - gather - sums, five L2
// round trips.  Measured per call in a captured graph (before: tiles of 2,048
// entries per block, serial searches by one thread, a completion kernel that
// searched again):
//   1,000 x 3,000, 12 K entries              4.9 us   (10.2 us)
//   200,000 x 500,000, 4 M, uniform         24.8 us   (45.0 us)
//   500,000 x 1,250,000, 27 M, power law     134 us   (228 us)
//   the same size, 25.5 M, banded             54 us   (166 us; 0.59 of the HBM copy rate)
// Tiles of 512 entries (64 registers, 32 warps per SM instead of 48) cost
// 65 us on the banded and 18 against 16.5 us on a 1 M-entry product, when the
// shipped tiles took 61 us there.
#include <algorithm>
#include <atomic>
#include <climits>
#include <mutex>
#include <string>

#include "common.cuh"

namespace pb {
namespace {

constexpr int kNaWarps = 8;                          // warps per block
constexpr int kNaTile = 256;                         // entries per warp tile
constexpr int kNaChunks = kNaTile / 128;             // 16-byte loads per lane and array
constexpr int kNoAllocMaxNnz = 134217728;
constexpr int kNaSlots = 3;                          // scratch words per range
constexpr int kNaMaxRanges = 32768;
constexpr int kNaClusterBlocks = 8;                  // largest portable cluster
constexpr int kNaLaneRow = 32;                       // entries of a row one lane sums at most
constexpr int kNaLanePieces = 16;                    // pieces of a giant row one lane adds at most
constexpr int kNaLocalSpan = 16384;                  // columns: a tile within this span gathers through L1

// Scratch: range k has words 3k (its piece of a giant row that began earlier),
// 3k + 1 (its piece of a giant row that begins here) and 3k + 2 (that row, or -1).
__device__ __align__(256) float g_noalloc_carry[131072];
static_assert(kNaSlots * kNaMaxRanges <= 131072, "scratch words");

// Per device ordinal: the array's device address, looked up
// once with that device current.  The address belongs to the runtime's primary
// context of the device, the one every call of this entry point uses.
std::atomic<float*> g_carry_addr[64];
std::mutex g_setup_mutex;

struct NaArgs {
    const int* __restrict__ row_ptr;
    const int* __restrict__ col;
    const float* __restrict__ val;
    const float* __restrict__ x;
    float* __restrict__ y;
    float* carry;
    int m, n, nnz, T, ranges;
};

__device__ __forceinline__ int4 ld_stream(const int4* p) {
    int4 v;
    asm("ld.global.nc.L1::no_allocate.v4.s32 {%0, %1, %2, %3}, [%4];"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_stream(const float4* p) {
    float4 v;
    asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// First row r in [0, m] with row_ptr[r] >= lo_target (r_lo) and hi_target
// (r_hi), m when there is none, by the whole warp: 32 probes per step, so
// about log32(m) dependent loads.  Each step shrinks its interval whatever
// row_ptr holds.
__device__ __forceinline__ void first_rows(const int* __restrict__ rp, int m, int lo_target, int hi_target, int lane,
                                           int& r_lo, int& r_hi) {
    int lo[2] = {0, 0}, width[2] = {m, m};   // the answers lie in [lo, lo + width]
    const int target[2] = {lo_target, hi_target};
    while ((width[0] | width[1]) > 0) {
        int stride[2], probe[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            stride[q] = (width[q] >> 5) + 1;
            const int at = lane * stride[q];
            probe[q] = at < width[q] ? __ldg(rp + lo[q] + at) : INT_MAX;   // beyond the interval: at or above
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const unsigned yes = __ballot_sync(0xffffffffu, probe[q] >= target[q]);
            if (width[q] == 0) continue;
            const int j = yes ? __ffs(int(yes)) - 1 : 32;   // first probe at or above the target
            const int end = int(min(unsigned(j) * unsigned(stride[q]), unsigned(width[q])));   // 32 strides: up to 2^31
            const int begin = j > 0 ? (j - 1) * stride[q] + 1 : 0;
            lo[q] += begin;
            width[q] = end - begin;
        }
    }
    r_lo = lo[0];
    r_hi = lo[1];
}

__device__ __forceinline__ float warp_total(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum of entries [b, e) by the whole warp (a piece of a giant row).
__device__ __forceinline__ float piece_sum(const NaArgs& a, int b, int e, unsigned last_col, int lane) {
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k = b + lane; k < e; k += 128) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int q = k + 32 * u;
            if (q < e) {
                const unsigned c = min(static_cast<unsigned>(__ldg(a.col + q)), last_col);
                s[u] = fmaf(__ldg(a.val + q), __ldcg(a.x + c), s[u]);
            }
        }
    }
    return warp_total((s[0] + s[1]) + (s[2] + s[3]));
}

// Products of entries [base, base + kNaTile) into p.  kVec: col and val are
// 16-byte aligned, so lane l takes 4 consecutive entries per load.  kEdge: the
// tile holds entries outside [e0, e1) (other ranges' or none), which cost no
// gather; the others skip those tests.
template <bool kVec, bool kEdge>
__device__ __forceinline__ void tile_products(const NaArgs& a, int base, int e0, int e1, unsigned last_col, int lane,
                                              float* __restrict__ p) {
    unsigned c[4 * kNaChunks];
    float v[4 * kNaChunks];
    bool own[4 * kNaChunks];
#pragma unroll
    for (int u = 0; u < kNaChunks; ++u) {
        if (kVec && (!kEdge || base + u * 128 + lane * 4 + 3 < a.nnz)) {
            const int q = base + u * 128 + lane * 4;
            const int4 c4 = ld_stream(reinterpret_cast<const int4*>(a.col + q));
            const float4 v4 = ld_stream(reinterpret_cast<const float4*>(a.val + q));
            c[4 * u] = c4.x; c[4 * u + 1] = c4.y; c[4 * u + 2] = c4.z; c[4 * u + 3] = c4.w;
            v[4 * u] = v4.x; v[4 * u + 1] = v4.y; v[4 * u + 2] = v4.z; v[4 * u + 3] = v4.w;
        } else {
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int q = kVec ? base + u * 128 + lane * 4 + t : base + (4 * u + t) * 32 + lane;
                const bool in = !kEdge || q < a.nnz;
                c[4 * u + t] = in ? static_cast<unsigned>(__ldg(a.col + q)) : 0u;
                v[4 * u + t] = in ? __ldg(a.val + q) : 0.f;
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 4 * kNaChunks; ++k) {
        const int q = kVec ? base + (k / 4) * 128 + lane * 4 + k % 4 : base + k * 32 + lane;
        own[k] = !kEdge || (q >= e0 && q < e1);
        c[k] = min(c[k], last_col);   // malformed input never reads out of bounds
    }
    // Local columns (banded, multi-period; judged by one column per lane):
    // neighbouring rows share lines in L1.  Spread ones would only evict what
    // other warps wait for.
    const bool local = __reduce_max_sync(0xffffffffu, c[0]) - __reduce_min_sync(0xffffffffu, c[0]) < kNaLocalSpan;
    float g[4 * kNaChunks];
    if (local) {
#pragma unroll
        for (int k = 0; k < 4 * kNaChunks; ++k) g[k] = own[k] ? __ldca(a.x + c[k]) : 0.f;
    } else {
#pragma unroll
        for (int k = 0; k < 4 * kNaChunks; ++k) g[k] = own[k] ? __ldcg(a.x + c[k]) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kNaChunks; ++u) {
        if (kVec) {
            reinterpret_cast<float4*>(p)[u * 32 + lane] =
                make_float4(v[4 * u] * g[4 * u], v[4 * u + 1] * g[4 * u + 1], v[4 * u + 2] * g[4 * u + 2],
                            v[4 * u + 3] * g[4 * u + 3]);
        } else {
#pragma unroll
            for (int t = 0; t < 4; ++t) p[(4 * u + t) * 32 + lane] = v[4 * u + t] * g[4 * u + t];
        }
    }
}

// Sum of p[from, to) for each lane's own [from, to); `rows` lanes at most hold
// a non-empty one, the lowest ones.  1 << kLog lanes share a row: few long
// rows use the whole warp, many short ones a lane each; a row that would take
// a lane more than kNaLaneRow steps is summed by the whole warp.
template <int kLog>
__device__ __forceinline__ float row_sums(const float* __restrict__ p, int from, int to, int lane) {
    constexpr int G = 1 << kLog;
    const int f = kLog ? __shfl_sync(0xffffffffu, from, lane >> kLog) : from;
    const int t = kLog ? __shfl_sync(0xffffffffu, to, lane >> kLog) : to;
    const bool mine = t - f <= kNaLaneRow * G;
    const int end = mine ? t : f;
    const int longest = __reduce_max_sync(0xffffffffu, end - f);
    float part[4] = {0.f, 0.f, 0.f, 0.f};
    const int first = f + (lane & (G - 1));
    for (int q = 0; q < longest; q += 4 * G) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = first + q + u * G;
            if (k < end) part[u] += p[k];
        }
    }
    float sum = (part[0] + part[1]) + (part[2] + part[3]);
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (kLog) sum = __shfl_sync(0xffffffffu, sum, (lane << kLog) & 31);
    unsigned wide = __ballot_sync(0xffffffffu, to - from > kNaLaneRow * G);
    while (wide) {
        const int src = __ffs(int(wide)) - 1;
        wide &= wide - 1;
        const int wf = __shfl_sync(0xffffffffu, from, src), wt = __shfl_sync(0xffffffffu, to, src);
        float w = 0.f;
        for (int q = wf + lane; q < wt; q += 32) w += p[q];
        w = warp_total(w);
        if (lane == src) sum = w;
    }
    return sum;
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Where the ranges leave their words: the scratch array, or the shared memory
// of the cluster's first block.  ready() comes before put(), by the whole warp.
struct GlobalWords {
    float* at;
    __device__ __forceinline__ void ready() const {}
    __device__ __forceinline__ void put(int i, float v) const { at[i] = v; }
    // range k's giant row, or -1 (what is there may be another call's)
    __device__ __forceinline__ void mark(int k, int row, int lane) const {
        if (lane == 0) at[kNaSlots * k + 2] = __int_as_float(row);
    }
    __device__ __forceinline__ float get(int i) const { return __ldcg(at + i); }
};
struct ClusterWords {
    float* own;                // this block's array (the first block's is the one in use)
    mutable bool waited = false;
    // The first block's marks start as -1, so a range without a giant row stores nothing.
    __device__ explicit ClusterWords(float* shared) : own(shared) {
        if (threadIdx.x < kNaWarps * kNaClusterBlocks) own[kNaSlots * threadIdx.x + 2] = __int_as_float(-1);
        cluster_arrive();
    }
    __device__ __forceinline__ void ready() const {   // the first block runs and its marks are set
        if (!waited) cluster_wait();
        waited = true;
    }
    __device__ __forceinline__ void put(int i, float v) const {
        uint32_t first;
        asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(first) : "r"(smem_u32(own)));
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(first + 4u * unsigned(i)), "f"(v) : "memory");
    }
    __device__ __forceinline__ void mark(int k, int row, int lane) const {
        if (row >= 0 && lane == 0) put(kNaSlots * k + 2, __int_as_float(row));
    }
    __device__ __forceinline__ float get(int i) const { return own[i]; }
};

// Writes zeros to the empty rows at the front of [r, r1), whose row pointer is v
// (so is that of the row before): found 32, then 1,024, 32,768, ... rows to a lane
// and load.  Row by row the warp that owns a long run would read all its pointers
// 32 at a time.  Returns the first row left; runs shorter than 32 are left too.
template <class RowPtr>
__device__ __forceinline__ int skip_empty(const NaArgs& a, const RowPtr& rp, int v, int r, int r1, int lane) {
    int stride = 32;
    while (stride <= r1 - r) {
        const unsigned ahead = unsigned(stride) * unsigned(lane + 1);   // at most 2^30
        const bool empty = ahead <= unsigned(r1 - r) && rp(r + int(ahead)) == v;
        const int strides = __popc(__ballot_sync(0xffffffffu, empty));
        const int end = r + stride * strides;
        for (unsigned i = unsigned(r) + unsigned(lane); i < unsigned(end); i += 32) a.y[i] = 0.f;
        r = end;
        if (strides < 32 && stride == 32) break;
        stride = strides < 32 ? 32 : min(stride * 32, 1 << 25);
    }
    return r;
}

// One range by one warp.
template <bool kVec, class Words>
__device__ __forceinline__ void range_product(const NaArgs& a, const Words& words, int k, int lane, float* __restrict__ p) {
    const unsigned last_col = static_cast<unsigned>(a.n - 1);
    const bool last = k == a.ranges - 1;
    const int lo = k * a.T, hi = last ? a.nnz : lo + a.T;
    int r, r1;
    first_rows(a.row_ptr, a.m, lo, hi, lane, r, r1);
    if (last) r1 = a.m;   // with the empty rows after the last entry
    auto rp = [&](int i) { return min(max(__ldg(a.row_ptr + i), 0), a.nnz); };
    const int e0 = r1 > r ? rp(r) : 0;
    int e1 = r1 > r ? rp(r1) : 0;
    // ---- pieces of giant rows ----
    const int kGiant = 2 * a.T;
    if (r > 0) {
        const int s = rp(r - 1), e = r1 > r ? e0 : rp(r);
        if (e > lo && e - s > kGiant) {
            const float t = piece_sum(a, lo, min(e, hi), last_col, lane);
            words.ready();
            if (lane == 0) words.put(kNaSlots * k, t);
        }
    }
    int giant = -1;
    if (r1 > r) {
        const int s = rp(r1 - 1);
        if (e1 - s > kGiant) {
            giant = --r1;
            const float t = piece_sum(a, s, min(e1, hi), last_col, lane);
            words.ready();
            if (lane == 0) words.put(kNaSlots * k + 1, t);
            e1 = s;
        }
    }
    words.mark(k, giant, lane);

    // ---- the other rows, tile by tile ----
    float open = 0.f;   // partial sum of row r, begun in an earlier tile
    for (int base = e0 & ~3; base < e1; base += kNaTile) {
        const int lim = base + kNaTile;
        // the row pointers of the next 32 rows travel with the tile's entries
        // (r1 - r, not r + 32: row numbers may go up to INT_MAX)
        int s = lane <= r1 - r ? rp(r + lane) : INT_MAX;
        int s_next = 32 <= r1 - r ? rp(r + 32) : INT_MAX;
        if (base >= e0 && lim <= e1) tile_products<kVec, false>(a, base, e0, e1, last_col, lane, p);
        else tile_products<kVec, true>(a, base, e0, e1, last_col, lane, p);
        __syncwarp();
        while (true) {
            int e = __shfl_down_sync(0xffffffffu, s, 1);
            if (lane == 31) e = s_next;
            const bool started = lane < r1 - r && s < lim;
            const bool done = started && e <= lim;
            const unsigned started_m = __ballot_sync(0xffffffffu, started);
            const int nd = __popc(__ballot_sync(0xffffffffu, done));
            // the next rows' pointers, before the sums of these
            int s2 = INT_MAX, s2_next = INT_MAX;
            if (nd == 32) {
                const int v = __shfl_sync(0xffffffffu, s, 0);
                if (s_next == v) {   // 32 empty rows: zeros, and on to the last row of the run
                    a.y[r + lane] = 0.f;
                    r = skip_empty(a, rp, v, r + 32, r1, lane);
                    s = lane <= r1 - r ? rp(r + lane) : INT_MAX;
                    s_next = 32 <= r1 - r ? rp(r + 32) : INT_MAX;
                    continue;
                }
                s2 = 32 + lane <= r1 - r ? rp(r + 32 + lane) : INT_MAX;
                s2_next = 64 <= r1 - r ? rp(r + 64) : INT_MAX;
            }
            const int from = started ? max(s, base) - base : 0;
            const int to = started ? min(e, lim) - base : 0;
            const int rows = __popc(started_m);
            float sum = rows > 16 ? row_sums<0>(p, from, to, lane)
                        : rows > 8 ? row_sums<1>(p, from, to, lane)
                        : rows > 4 ? row_sums<2>(p, from, to, lane) : row_sums<3>(p, from, to, lane);
            if (lane == 0) sum += open;
            if (done) a.y[r + lane] = sum;
            open = 0.f;
            r += nd;
            if (nd < 32) {
                if ((started_m >> nd) & 1u) open = __shfl_sync(0xffffffffu, sum, nd);
                break;
            }
            s = s2;
            s_next = s2_next;
        }
        __syncwarp();   // p is free for the next tile
    }
    // empty rows after the last entry
    for (unsigned i = unsigned(r) + unsigned(lane); i < unsigned(r1); i += 32) a.y[i] = 0.f;
}

// The giant rows that begin in ranges [first, first + 32), a lane each (one
// after the other by the whole warp, 1,000 rows of 600 entries took 19.7 us, 10.5
// now); rows of more than kNaLanePieces pieces by the whole warp, lane-strided,
// then a tree.  A range's row number counts only if that
// row begins there and is a giant one in this call's row_ptr.
template <class Words>
__device__ __forceinline__ void finish_giants(const NaArgs& a, const Words& words, int first, int lane) {
    const int k = first + lane;
    const int row = k < a.ranges ? __float_as_int(words.get(kNaSlots * k + 2)) : -1;
    int to = k;   // last range with a piece
    if (row >= 0 && row < a.m) {
        const int s = __ldg(a.row_ptr + row), end = min(__ldg(a.row_ptr + row + 1), a.nnz);
        if (s >= k * a.T && s < min((k + 1) * a.T, a.nnz) && end - s > 2 * a.T) to = min((end - 1) / a.T, a.ranges - 1);
    }
    if (to > k && to - k <= kNaLanePieces) {
        float t[kNaLanePieces];   // added in the tree a warp with a piece per lane would use
#pragma unroll
        for (int j = 0; j < kNaLanePieces; ++j) t[j] = k + 1 + j <= to ? words.get(kNaSlots * (k + 1 + j)) : 0.f;
#pragma unroll
        for (int o = kNaLanePieces / 2; o > 0; o >>= 1)
#pragma unroll
            for (int j = 0; j < o; ++j) t[j] += t[j + o];
        a.y[row] = words.get(kNaSlots * k + 1) + t[0];
    }
    unsigned todo = __ballot_sync(0xffffffffu, to - k > kNaLanePieces);
    while (todo) {
        const int src = __ffs(int(todo)) - 1;
        todo &= todo - 1;
        const int r = __shfl_sync(0xffffffffu, row, src), last = __shfl_sync(0xffffffffu, to, src);
        const int from = first + src;
        float t = 0.f;
        for (int j = from + 1 + lane; j <= last; j += 32) t += words.get(kNaSlots * j);
        t = warp_total(t);
        if (lane == 0) a.y[r] = words.get(kNaSlots * from + 1) + t;
    }
}

template <bool kVec>
__global__ void __launch_bounds__(kNaWarps * 32, 6) noalloc_spmv_kernel(const NaArgs a) {
    __shared__ __align__(16) float products[kNaWarps][kNaTile];
    grid_dep_launch();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = blockIdx.x * kNaWarps + warp;
    if (k < a.ranges) range_product<kVec>(a, GlobalWords{a.carry}, k, lane, products[warp]);
}

__global__ void __launch_bounds__(256) noalloc_giants_kernel(const NaArgs a) {
    grid_dep_wait();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (32 * warp < a.ranges) finish_giants(a, GlobalWords{a.carry}, 32 * warp, threadIdx.x & 31);
}

// The whole product by one cluster.
template <bool kVec>
__global__ void __launch_bounds__(kNaWarps * 32, 6) noalloc_cluster_kernel(const NaArgs a) {
    __shared__ __align__(16) float products[kNaWarps][kNaTile];
    __shared__ float pieces[kNaSlots * kNaWarps * kNaClusterBlocks];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = blockIdx.x * kNaWarps + warp;
    const ClusterWords words(pieces);
    if (k < a.ranges) range_product<kVec>(a, words, k, lane, products[warp]);
    words.ready();
    // the pieces are visible after the barrier, to the first block's first two warps
    cluster_arrive();
    cluster_wait();
    if (32 * k < a.ranges) finish_giants(a, words, 32 * k, lane);
}
static_assert(kNaClusterBlocks * kNaWarps <= 32 * kNaWarps, "the first block finishes the cluster's giant rows");

template <bool kVec>
void launch(const NaArgs& a, cudaStream_t stream) {
    const int blocks = (a.ranges + kNaWarps - 1) / kNaWarps;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(blocks));
    cfg.blockDim = dim3(kNaWarps * 32);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (blocks <= kNaClusterBlocks) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = unsigned(blocks);
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        PB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, noalloc_cluster_kernel<kVec>, a));
        return;
    }
    noalloc_spmv_kernel<kVec><<<blocks, kNaWarps * 32, 0, stream>>>(a);
    PB_CUDA_CHECK(cudaGetLastError());
    // launched while the product drains; it waits for it before it reads the pieces
    cfg.gridDim = dim3(unsigned((a.ranges + 255) / 256));
    cfg.blockDim = dim3(256);
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    PB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, noalloc_giants_kernel, a));
}

// Device address of the scratch array for `dev`, looked up
// once per device with that device current and cached.  With lazy module
// loading this first lookup is also where the module, and with it the array,
// may be loaded onto the device.
float* carry_address(int dev) {
    if (dev < 0 || dev >= 64) throw InvalidArgument("device ordinal out of range");
    float* p = g_carry_addr[dev].load(std::memory_order_acquire);
    if (p) return p;
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    p = g_carry_addr[dev].load(std::memory_order_relaxed);
    if (!p) {
        void* addr = nullptr;
        PB_CUDA_CHECK(cudaGetSymbolAddress(&addr, g_noalloc_carry));
        p = static_cast<float*>(addr);
        g_carry_addr[dev].store(p, std::memory_order_release);
    }
    return p;
}

}  // namespace

// Host side of pramaan_spmv_noalloc; errors become exceptions handled by the
// extern "C" wrapper in abi.cu.
void spmv_noalloc(const int32_t* d_row_ptr, const int32_t* d_col_idx, const float* d_values,
                  int32_t m, int32_t n, int32_t nnz, const float* d_x, float* d_y,
                  cudaStream_t stream) {
    if (m < 0 || n < 0 || nnz < 0) throw InvalidArgument("negative dimension");
    if (nnz > kNoAllocMaxNnz)
        throw InvalidArgument("pramaan_spmv_noalloc: nnz " + std::to_string(nnz) +
                              " exceeds the scratch limit of " + std::to_string(kNoAllocMaxNnz) + " entries");
    if (m == 0) return;
    if (!d_row_ptr || !d_y) throw InvalidArgument("row_ptr and y must not be NULL");
    if (nnz > 0 && (!d_col_idx || !d_values || !d_x || n == 0))
        throw InvalidArgument("col_idx, values and x must not be NULL (and n > 0) when nnz > 0");
    int dev = 0;
    PB_CUDA_CHECK(cudaGetDevice(&dev));
    float* carry = carry_address(dev);
    if (nnz == 0) {
        PB_CUDA_CHECK(cudaMemsetAsync(d_y, 0, size_t(m) * sizeof(float), stream));
        return;
    }
    // Tiles per range: one per Mi entries, between one, so that a small product
    // spreads over the chip, and four, where the ranges fill it anyway and fewer
    // searches pay; more only where the scratch would not hold the ranges.  us with
    // 1 | 2 | 3 | 4 tiles: 1 M entries uniform 12.1 | 11.2 | 13.5 | 12.0, power law 13.1 |
    // 14.3 | 17.4 | 19.3; 2.2 M uniform 19.2 | 15.9 | 16.9 | 16.0, banded 12.7 | 9.8 | 9.6 |
    // 9.7; 4 M uniform 27.9 | 26.6 | 24.7 | 25.6, banded 18.7 | 15.0 | 12.9 | 13.3; 8 M uniform
    // 48.9 | 42.7 | 41.0 | 44.6.
    const int by_size = std::min(std::max(nnz >> 20, 1), 4);
    const int by_scratch = int((nnz + (long long)kNaTile * kNaMaxRanges - 1) / ((long long)kNaTile * kNaMaxRanges));
    // Products of up to 64 ranges (a cluster's warps) of a quarter or half a tile
    // take such short ranges: their warps' work is mostly rows, 32 a step, and long
    // rows are cut finer.  us with ranges of 256 | 64 entries (before: one block per
    // 2,048 entries): 1,000 rows of one entry 6.4 | 4.2 (5.6), 50 rows of 40 4.5 | 3.8
    // (4.7), 2 rows of 1,000 5.1 | 4.3 (4.3); of 128: 2,000 rows of 4 4.6 | 4.3 (10.6).
    const int cluster_ranges = kNaWarps * kNaClusterBlocks;
    const int T = nnz <= cluster_ranges * (kNaTile / 4)   ? kNaTile / 4
                  : nnz <= cluster_ranges * (kNaTile / 2) ? kNaTile / 2
                                                          : kNaTile * std::max(by_size, by_scratch);
    const NaArgs a{d_row_ptr, d_col_idx, d_values, d_x, d_y, carry, m, n, nnz, T, (nnz + T - 1) / T};
    const bool vec = ((reinterpret_cast<uintptr_t>(d_col_idx) | reinterpret_cast<uintptr_t>(d_values)) & 15) == 0;
    if (vec) launch<true>(a, stream);
    else launch<false>(a, stream);
}

}  // namespace pb
