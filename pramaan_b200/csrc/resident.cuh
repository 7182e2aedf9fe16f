// resident.cuh — iterations of one LP on one thread-block cluster, with the
// LP's matrix and vectors resident in the cluster's shared memory.
//
// Why.  An iteration of a small LP is a latency chain, not a stream: two
// products whose operands would fit on chip, yet every one of them reads its
// row pointers, entries and gathered vector from L2 again, and the halves are
// separated by kernel launches or by cluster barriers around L2 round trips.
// Here every block of a cluster of up to 16 keeps, for the whole launch, its
// rows of A and of A^T, its share of every vector, and the parts of y and of x̄
// that its rows refer to.  Measured, us per iteration: reference iteration on
// the 1,000 x 3,000 LP (12 K entries) 1.9 against 11.7 with the tiled products;
// Halpern iteration on a rolling-horizon LP of 180 periods and 28 products
// (30 K entries) 2.4 against 6.4 with halpern_cluster_kernel.
//
// What bounds it.  A half iteration is one warp's chain (entries, gather, sum,
// update, store to the others; about 900 cycles of mostly dependent
// instructions) plus the exchange (100 to 300 cycles).  Hence the layout: a lane
// per row with entry k of 32 rows in one line, constants in registers, no branch
// that can be a select, 16-byte remote stores.
//
// Exchange.  The rows and the columns of an LP are cut into contiguous shares,
// one of each per block, at multiples of kResSub elements.  A warp computes one
// sub-chunk (32 elements) of the new vector at a time and stores it straight
// into the shared memory of the blocks whose rows refer to that sub-chunk, and
// of those alone: 16-byte remote stores (st.async) that complete on the
// receiver's mbarrier.  A receiver waits for the bytes it expects; there is no
// cluster barrier per iteration.  Per
// iteration of a 12 K-entry LP: 2.9 us with bulk copies from a staging buffer,
// 2.6 with 4-byte stores, 1.9 now.  A receiver's gather
// vector holds the sub-chunks it needs back to back, and the entries' columns
// are rewritten to positions in it (16 bits) when the plan is built.
//   Overwriting an element of a gather vector is safe without further waiting:
//   the block that sends x̄_j owns column j.  If a row i of the receiver refers
//   to j, column j refers to y_i, so the sender has waited for the sub-chunk of
//   y with row i, whose elements are sent after their rows' sums have read x̄;
//   if no row refers to j, nothing reads the element.  The same holds the other
//   way round.  A barrier's next phase cannot complete early: thread 0 arrives
//   for it only after a block barrier that every thread reaches past its waits
//   of the iteration.
//
// Order of the sums.  A row of at most kResLongRow entries is one thread's, a
// longer one four lanes'.  Two orders, so that the iterates of a Halpern solve are
// the same bits whichever path runs them (the reference iteration uses kResFlat,
// whose bits are not those of its row-aligned tiles; kResTiled costs it 2.4 times
// the time on the 12 K-entry LP):
//   kResFlat   entries in CSR order; a long row lane-strided with an xor tree
//              (the order of halpern_cluster_kernel);
//   kResTiled  the order of the tiled products: pieces cut where the packed
//              position is a multiple of 16 (a lane's entries) or 512 (a tile),
//              FMAs in order within a piece, a tile's pieces by the segmented
//              scan's tree plus the last piece, tiles in order.
//
// Waits are bounded (kWaitLimitNs): a block that gives up sets the status word
// and leaves the loop, the blocks that wait for it follow, and all meet at the
// last cluster barrier.  A block that finished every iteration has waited for
// every store sent to it.  One that gave up has not, and neither the barrier
// nor its release covers them (st.async completes on the receiver's mbarrier
// alone): past the barrier, when nobody sends any more, it stays for
// kResDrainNs, far longer than a store is under way, before it retires.
#pragma once

#include <vector>

#include "adaptive.cuh"
#include "cluster.cuh"
#include "csr_device.cuh"

namespace pb {

constexpr int kResThreads = 512;
constexpr int kResSub = 32;            // vector elements per sub-chunk
constexpr int kResMaxCluster = 16;
constexpr int kResLean = -1;           // (a cluster size) kResMaxCluster blocks, constants in global memory
constexpr int kResWeights = 128;       // iterations whose weights are computed ahead
constexpr int kResLongRow = 16;
constexpr int kResFlat = 0, kResTiled = 1;
constexpr uint16_t kResNoSlot = 0xffff;
// How long a block that gave up outlives the last barrier (a remote store takes
// about a microsecond).
constexpr unsigned long long kResDrainNs = 10000000ull;   // 10 ms
// Entries a long row takes: 2 modulo 16, so that the 8 rows a warp sums at a
// time begin in different banks (rows of 48 back to back all began in the same
// one: a block with 130 of them took 4,300 cycles for its half, 3,200 now).
__host__ __device__ constexpr int res_long_stride(int len) { return len + ((2 - len) & 15); }
constexpr size_t kResMaxSmem = 232448;

// One block's share (rows of A, columns of A) and what it receives.
struct ResCta {
    int r0, r1, c0, c1;        // own rows and columns
    int lr0, lr1, lc0, lc1;    // its LP's
    int ell_a, ell_t;          // 32-entry lines of the short rows / columns
    int long_a, long_t;        // long rows / columns
    int lent_a, lent_t;        // their entries
    int need_x, need_y;        // sub-chunks of x̄ / y the own rows / columns refer to
};

struct ResView {
    const int* which = nullptr;         // plan LP of every launched cluster (null: all, in order)
    const ResCta* cta = nullptr;
    const uint16_t* slot_x = nullptr;   // [block][sub_x]: the block's slot of a sub-chunk of x̄
    const uint16_t* slot_y = nullptr;
    int sub_x = 0, sub_y = 0;
    const uint32_t* lines_a = nullptr;  // [block][sub_y]: first line of an own sub-chunk << 5 | lines
    const uint32_t* lines_t = nullptr;
    FlatCsr A{}, AT{};
    const uint16_t* idx_a = nullptr;    // positions of the entries' columns in the own gather vector
    const uint16_t* idx_t = nullptr;
    int* status = nullptr;
};

// Shared memory of one block.  The gather vectors come first, where senders
// find them: x̄'s at kGather, y's behind the sub-chunks of x̄ the block needs.
struct ResLayout {
    static constexpr int kBarX = 0, kBarY = 8, kCounts = 16, kWeights = 128, kGather = kWeights + 4 * kResWeights;
    int gx, gy, sx, sy, cols, rows, x, long_sum, ell_a, ell_t, lent_a, lent_t, range_a, range_t, lines_a, lines_t, long_a,
        long_t, to_x, to_y, n_to_x, n_to_y;
    int total;
    int R, C;
    // lean: the elements' constants stay in global memory
    __host__ __device__ ResLayout(const ResCta& c, int cluster, bool lean) {
        R = c.r1 - c.r0;
        C = c.c1 - c.c0;
        int at = kGather;
        auto take = [&](int bytes) {
            const int p = at;
            at += (bytes + 15) / 16 * 16;
            return p;
        };
        const int subs_x = (C + kResSub - 1) / kResSub, subs_y = (R + kResSub - 1) / kResSub;
        gx = take(c.need_x * kResSub * 4);
        gy = take(c.need_y * kResSub * 4);
        sx = take(subs_x * kResSub * 4);           // own x̄ (before: sums of long columns)
        sy = take(subs_y * kResSub * 4);           // own y
        cols = take(lean ? 0 : C * 16);            // {tau, c, lower, upper}
        rows = take(lean ? 0 : R * 16);            // {sigma, lower, upper, master y}
        x = take(C * 4);
        long_sum = take(R * 4);                    // sums of long rows
        ell_a = take(c.ell_a * 32 * 8);            // short rows: {value, address of the gathered element},
        ell_t = take(c.ell_t * 32 * 8);            // entry k of a sub-chunk's 32 rows in one line
        lent_a = take(c.lent_a * 8);               // long rows: row after row
        lent_t = take(c.lent_t * 8);
        range_a = take(R * 4);                     // packed position of the row's first entry % 16, length << 4
        range_t = take(C * 4);
        lines_a = take(subs_y * 4);
        lines_t = take(subs_x * 4);
        long_a = take(c.long_a * 16);              // {row, first entry, length, packed position}
        long_t = take(c.long_t * 16);
        to_x = take(subs_x * cluster * 8);         // receivers of every own sub-chunk: its slot's
        to_y = take(subs_y * cluster * 8);         // address in the cluster, the barrier's
        n_to_x = take(subs_x);
        n_to_y = take(subs_y);
        total = at;
    }
};

// ---- PTX ---------------------------------------------------------------------
__device__ __forceinline__ uint32_t map_to_cta(uint32_t shared_addr, uint32_t cta) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(shared_addr), "r"(cta));
    return r;
}
// Shared memory by 32-bit address: pointers kept in structs compile to generic
// loads, whose latency the half iterations would pay several times in a row.
__device__ __forceinline__ float lds_f32(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds_u8(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 lds_u64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ float4 lds_f128(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ int4 lds_i128(uint32_t a) {
    int4 v;
    asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts_f32(uint32_t a, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
// A 16-byte store into a block of the cluster, completing on that block's barrier.
__device__ __forceinline__ void store_async(uint32_t dst, float4 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
                 "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)),
                 "r"(__float_as_uint(v.w)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_cluster_bounded(uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    const unsigned long long t0 = global_timer_ns();
    while (true) {
        if (mbar_try_wait_cluster(bar, parity)) return true;
        if (global_timer_ns() - t0 > kWaitLimitNs) return false;
    }
}

// ---- row sums ------------------------------------------------------------------
// An entry is {value, shared address of the element it is multiplied with}.
__device__ __forceinline__ float res_fma(uint2 ent, float s) { return fmaf(__uint_as_float(ent.x), lds_f32(ent.y), s); }

// The short rows (at most kResLongRow entries) of a sub-chunk, a lane each:
// `line` is the address of entry 0 of the lane's row, entry k lies k lines on
// (a warp reads 256 consecutive bytes; rows in CSR order cost a bank conflict
// per load).  Shorter rows' lines end in padding, loaded and not added.
template <int kOrder>
__device__ __forceinline__ float res_short_sum(uint32_t line, int lines, int len, int cut) {
    constexpr uint32_t kLine = 32 * 8;
    float s = 0.0f, t = 0.0f;
    auto add = [&](uint2 r, float x, int k) {
        const float v = __uint_as_float(r.x);
        const float s2 = fmaf(v, x, s);
        s = k < cut ? s2 : s;
        if constexpr (kOrder == kResTiled) {
            const float t2 = fmaf(v, x, t);
            t = k >= cut && k < len ? t2 : t;
        }
    };
    int k = 0;
    for (; k + 4 <= lines; k += 4, line += 4 * kLine) {
        const uint2 r0 = lds_u64(line), r1 = lds_u64(line + kLine), r2 = lds_u64(line + 2 * kLine),
                    r3 = lds_u64(line + 3 * kLine);
        const float x0 = lds_f32(r0.y), x1 = lds_f32(r1.y), x2 = lds_f32(r2.y), x3 = lds_f32(r3.y);
        add(r0, x0, k); add(r1, x1, k + 1); add(r2, x2, k + 2); add(r3, x3, k + 3);
    }
    if (lines & 2) {
        const uint2 r0 = lds_u64(line), r1 = lds_u64(line + kLine);
        const float x0 = lds_f32(r0.y), x1 = lds_f32(r1.y);
        add(r0, x0, k); add(r1, x1, k + 1);
        k += 2;
        line += 2 * kLine;
    }
    if (lines & 1) {
        const uint2 r = lds_u64(line);
        add(r, lds_f32(r.y), k);
    }
    return kOrder == kResTiled && cut < len ? t + s : s;
}

// A longer row in the tiled order, by the whole warp; every lane returns the
// sum.  pos: the packed position of its first entry.
__device__ __forceinline__ float res_warp_tiled_sum(uint32_t ent, int len, int pos, int lane) {
    float sum = 0.0f;
    for (int base = pos / kSpmvTile * kSpmvTile; base < pos + len; base += kSpmvTile) {
        const int pb = pos - base, pe = pos + len - base;                    // the row in this tile's terms
        const int from = max(pb, lane * kSpmvIpt), to = min(pe, (lane + 1) * kSpmvIpt);
        float v = 0.0f;
        for (int k = from; k < to; ++k) v = res_fma(lds_u64(ent + (k - pb) * 8), v);
        const int first = max(pb, 0) / kSpmvIpt;                             // lanes of the row in this tile
        const int last = (min(pe, kSpmvTile) - 1) / kSpmvIpt;
        const float end = __shfl_sync(0xffffffffu, v, last);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float o = __shfl_up_sync(0xffffffffu, v, d);
            if (lane - d >= first) v += o;
        }
        const float before = __shfl_sync(0xffffffffu, v, last > 0 ? last - 1 : 0);
        const float total = last > first ? end + before : end;
        sum = pb >= 0 ? total : sum + total;
    }
    return sum;
}

// The sums of a block's long rows into out[row], 4 lanes per row so that a
// block's 128 rows overlap.
template <int kOrder>
__device__ __forceinline__ void res_long_sums(uint32_t longs, int n, uint32_t ents, uint32_t out, int warp, int lane) {
    constexpr int kWarps = kResThreads / 32;
    const int j = lane & 3;
    for (int base = warp * 8; base < n; base += kWarps * 8) {
        const int k = base + (lane >> 2);
        const int4 row = lds_i128(longs + min(k, n - 1) * 16);   // {row, first entry, length, packed position}
        const uint32_t ent = ents + row.y * 8;
        const int len = k < n ? row.z : 0;
        if constexpr (kOrder == kResFlat) {
            // lane j stands for lanes j, j + 4, ... j + 28 of a warp
            float s[8] = {};
            for (int q = j; q < len; q += 32) {
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const bool in = q + 4 * u < len;
                    const uint2 r = lds_u64(ent + (in ? q + 4 * u : q) * 8);
                    const float t = fmaf(__uint_as_float(r.x), lds_f32(r.y), s[u]);
                    s[u] = in ? t : s[u];
                }
            }
            float t = ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
            t += __shfl_xor_sync(0xffffffffu, t, 2);
            t += __shfl_xor_sync(0xffffffffu, t, 1);
            if (j == 0 && k < n) sts_f32(out + row.x * 4, t);
        } else {
            // a row inside one tile, over at most 8 of its 16-entry pieces: lane j has pieces 2 j and 2 j + 1
            const int at = row.w % kSpmvTile;
            const int first = at / kSpmvIpt;
            const int pieces = (at + row.z - 1) / kSpmvIpt - first + 1;
            const bool here = k < n && at + row.z <= kSpmvTile && pieces <= 8;
            float v[2] = {0.0f, 0.0f};
            if (here) {
                const int p0 = (first + 2 * j) * kSpmvIpt - at;
                const int from = max(0, p0), mid = min(len, p0 + kSpmvIpt), to = min(len, p0 + 2 * kSpmvIpt);
#pragma unroll 4
                for (int q = from; q < mid; ++q) v[0] = res_fma(lds_u64(ent + q * 8), v[0]);
#pragma unroll 4
                for (int q = max(0, p0 + kSpmvIpt); q < to; ++q) v[1] = res_fma(lds_u64(ent + q * 8), v[1]);
            }
            const int last = here ? pieces - 1 : 0, prev = here && pieces > 1 ? pieces - 2 : 0;
            auto piece = [&](int i) {
                const float a = __shfl_sync(0xffffffffu, v[0], i >> 1, 4), b = __shfl_sync(0xffffffffu, v[1], i >> 1, 4);
                return i & 1 ? b : a;
            };
            const float end = piece(last);
            const float up = __shfl_up_sync(0xffffffffu, v[1], 1, 4);   // distance 1 of the scan
            v[1] += v[0];
            if (j >= 1) v[0] += up;
#pragma unroll
            for (int d = 1; d < 4; d <<= 1) {                           // distances 2 and 4
                const float a = __shfl_up_sync(0xffffffffu, v[0], d, 4), b = __shfl_up_sync(0xffffffffu, v[1], d, 4);
                if (j >= d) {
                    v[0] += a;
                    v[1] += b;
                }
            }
            const float before = piece(prev);
            if (here && j == 0) sts_f32(out + row.x * 4, pieces > 1 ? end + before : end);
            unsigned other = __ballot_sync(0xffffffffu, k < n && !here && j == 0);
            while (other) {   // rows over two tiles, or very long ones
                const int src = __ffs(int(other)) - 1;
                other &= other - 1;
                const int wx = __shfl_sync(0xffffffffu, row.x, src), wy = __shfl_sync(0xffffffffu, row.y, src);
                const int wz = __shfl_sync(0xffffffffu, row.z, src), ww = __shfl_sync(0xffffffffu, row.w, src);
                const float t = res_warp_tiled_sum(ents + wy * 8, wz, ww, lane);
                if (lane == 0) sts_f32(out + wx * 4, t);
            }
        }
    }
}

// ---- the kernel ------------------------------------------------------------------
// Algo:
//   kColsFirst   the column half (A^T y -> x, x̄) comes first, else the row half
//   kOrder       order of the sums
//   kMaster      rows have a master y
//   kWeights     the weight depends on the iteration
//   begin(me), weight(it)   the LP's state, and iteration it's Halpern weight
//   col({tau, c, lower, upper}, x, sum, w, fpr), row({sigma, lower, upper,
//                master y}, y, sum, w, fpr)   one element's update from its
//                product sum; col returns x̄, row the new y; fpr: where the
//                element's residual term goes (null: nowhere)
//   fpr_col(it, iters), fpr_row(it, iters)   the iteration's residual terms, or null

// One side (the columns or the rows) of a block's share: shared addresses.
struct ResSide {
    uint32_t ell, lent, to, longs, range, lines;
    uint32_t k;           // the elements' constants
    uint32_t state, out;  // x and x̄, or y twice
    uint32_t long_sum, n_to;
    int n, subs, begin, nlong, cluster;
};

// The first kResCached sub-chunks of a warp on one side live in registers:
// nothing of them is read from shared memory but the entries and what those
// gather.  A half iteration is bound by the latency of one warp's chain, so every
// load and every instruction on it counts.
constexpr int kResCached = 2;
struct ResCached {
    uint32_t line;
    int lines, len, cut;
    float4 k;
    float state, out;
    uint2 to;             // the receiver of this lane's group of 8 (x = 0: none)
    int more;             // receivers beyond the first four
};

__device__ __forceinline__ int res_cut(int order, uint32_t range) {
    const int len = int(range >> 4);
    return order == kResTiled ? min(len, 16 - int(range & 15u)) : len;
}

// The constants of element j of a side: from shared memory, or (lean, for LPs
// that would not fit otherwise) from the global arrays.
template <class Algo, bool kCols, bool kLean>
__device__ __forceinline__ float4 res_constants(const ResSide& S, const Algo& a, int j) {
    if constexpr (!kLean) return lds_f128(S.k + j * 16);
    const int g = S.begin + j;
    if constexpr (kCols) return make_float4(__ldg(a.tau + g), __ldg(a.c + g), __ldg(a.l_x + g), __ldg(a.u_x + g));
    else return make_float4(__ldg(a.sigma + g), __ldg(a.r_lo + g), __ldg(a.r_hi + g),
                            Algo::kMaster ? __ldg(a.y_m + g) : 0.0f);
}

template <class Algo, bool kCols, bool kLean>
__device__ __forceinline__ void res_load_cached(const ResSide& S, ResCached (&c)[kResCached], const Algo& algo, int warp,
                                                int lane) {
#pragma unroll
    for (int u = 0; u < kResCached; ++u) {
        const int s = warp + u * (kResThreads / 32), j = s * kResSub + lane;
        c[u] = ResCached{S.ell, 0, 0, 0, make_float4(0.f, 0.f, 0.f, 0.f), 0.f, 0.f, make_uint2(0u, 0u), 0};
        if (s >= S.subs) continue;
        const uint32_t ln = lds_u32(S.lines + s * 4);
        c[u].line = S.ell + ((ln >> 5) * 32 + lane) * 8;
        c[u].lines = int(ln & 31u);
        const int n = int(lds_u8(S.n_to + s)), g = lane >> 3;
        if (g < n) {
            c[u].to = lds_u64(S.to + (s * S.cluster + g) * 8);
            c[u].to.x += (lane & 7) * 16;
        }
        c[u].more = n > 4 ? n : 0;
        if (j >= S.n) continue;
        const uint32_t range = lds_u32(S.range + j * 4);
        c[u].len = int(range >> 4);
        c[u].cut = res_cut(Algo::kOrder, range);
        c[u].k = res_constants<Algo, kCols, kLean>(S, algo, j);
        c[u].state = lds_f32(S.state + j * 4);
        c[u].out = lds_f32(S.out + j * 4);
    }
}

// One half iteration of one side: sums, updates, and with `send` the new
// values to their receivers.
template <class Algo, bool kCols, bool kLean>
__device__ __forceinline__ void res_half(const ResSide& S, ResCached (&c)[kResCached], const Algo& algo, float w,
                                         double* fpr, bool send, int warp, int lane) {
    constexpr int kWarps = kResThreads / 32;
    if (S.nlong > 0) {
        res_long_sums<Algo::kOrder>(S.longs, S.nlong, S.lent, S.long_sum, warp, lane);
        __syncthreads();
    }
    auto update = [&](float4 k, float& state, float sum, int j) {
        double* f = fpr ? fpr + S.begin + j : nullptr;
        if constexpr (kCols) return algo.col(k, state, sum, w, f);
        else return state = algo.row(k, state, sum, w, f);
    };
    // the 8 lanes of a group hold the sub-chunk's 32 values between them
    auto quad = [&](float v) {
        const int q = (lane & 7) * 4;
        return make_float4(__shfl_sync(0xffffffffu, v, q), __shfl_sync(0xffffffffu, v, q + 1),
                           __shfl_sync(0xffffffffu, v, q + 2), __shfl_sync(0xffffffffu, v, q + 3));
    };
#pragma unroll
    for (int u = 0; u < kResCached; ++u) {
        const int s = warp + u * kWarps, j = s * kResSub + lane;
        if (s >= S.subs) break;
        float v = 0.0f;
        const float sum = res_short_sum<Algo::kOrder>(c[u].line, c[u].lines, c[u].len, c[u].cut);
        if (j < S.n) {
            v = update(c[u].k, c[u].state, c[u].len > kResLongRow ? lds_f32(S.long_sum + j * 4) : sum, j);
            c[u].out = v;
        }
        if (send) {
            const float4 q = quad(v);
            if (c[u].to.x) store_async(c[u].to.x, q, c[u].to.y);
            for (int k = 4 + (lane >> 3); k < c[u].more; k += 4) {
                const uint2 d = lds_u64(S.to + (s * S.cluster + k) * 8);
                store_async(d.x + (lane & 7) * 16, q, d.y);
            }
        }
    }
    for (int s = warp + kResCached * kWarps; s < S.subs; s += kWarps) {
        const int j = s * kResSub + lane;
        const uint32_t ln = lds_u32(S.lines + s * 4), range = j < S.n ? lds_u32(S.range + j * 4) : 0u;
        const int len = int(range >> 4);
        const float4 k = j < S.n ? res_constants<Algo, kCols, kLean>(S, algo, j) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float sum = res_short_sum<Algo::kOrder>(S.ell + ((ln >> 5) * 32 + lane) * 8, int(ln & 31u), len,
                                                      res_cut(Algo::kOrder, range));
        float v = 0.0f;
        if (j < S.n) {
            float state = lds_f32(S.state + j * 4);
            v = update(k, state, len > kResLongRow ? lds_f32(S.long_sum + j * 4) : sum, j);
            sts_f32(S.state + j * 4, state);
            sts_f32(S.out + j * 4, v);
        }
        if (send) {
            const float4 q = quad(v);
            const int n = int(lds_u8(S.n_to + s));
            for (int k = lane >> 3; k < n; k += 4) {
                const uint2 d = lds_u64(S.to + (s * S.cluster + k) * 8);
                store_async(d.x + (lane & 7) * 16, q, d.y);
            }
        }
    }
}

template <class Algo, bool kLean>
__global__ void __launch_bounds__(kResThreads, 1) resident_kernel(const ResView v, Algo algo, const int iters) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kWarps = kResThreads / 32;
    const int cluster = int(cluster_blocks());
    const int first_cta = (v.which ? v.which[cluster_index_x()] : int(cluster_index_x())) * cluster;
    const int my_cta = first_cta + int(cluster_rank_in());
    const ResCta me = v.cta[my_cta];
    const ResLayout L(me, cluster, kLean);
    const int R = L.R, C = L.C;
    uint64_t* bar_x = reinterpret_cast<uint64_t*>(smem + ResLayout::kBarX);
    uint64_t* bar_y = reinterpret_cast<uint64_t*>(smem + ResLayout::kBarY);
    int* counts = reinterpret_cast<int*>(smem + ResLayout::kCounts);   // long rows and columns listed, their entries
    auto f32 = [&](int off) { return reinterpret_cast<float*>(smem + off); };
    auto u32 = [&](int off) { return reinterpret_cast<uint32_t*>(smem + off); };
    float *gx = f32(L.gx), *gy = f32(L.gy), *sx = f32(L.sx), *sy = f32(L.sy), *xs = f32(L.x);
    float *long_sum = f32(L.long_sum), *weights = f32(ResLayout::kWeights);
    float4 *cols = reinterpret_cast<float4*>(smem + L.cols), *rows = reinterpret_cast<float4*>(smem + L.rows);
    uint2 *ell_a = reinterpret_cast<uint2*>(smem + L.ell_a), *ell_t = reinterpret_cast<uint2*>(smem + L.ell_t);
    uint2 *lent_a = reinterpret_cast<uint2*>(smem + L.lent_a), *lent_t = reinterpret_cast<uint2*>(smem + L.lent_t);
    int4 *long_a = reinterpret_cast<int4*>(smem + L.long_a), *long_t = reinterpret_cast<int4*>(smem + L.long_t);
    uint32_t *range_a = u32(L.range_a), *range_t = u32(L.range_t), *lines_a = u32(L.lines_a), *lines_t = u32(L.lines_t);
    uint2 *to_x = reinterpret_cast<uint2*>(smem + L.to_x), *to_y = reinterpret_cast<uint2*>(smem + L.to_y);
    uint8_t *n_to_x = smem + L.n_to_x, *n_to_y = smem + L.n_to_y;
    const int subs_x = (C + kResSub - 1) / kResSub, subs_y = (R + kResSub - 1) / kResSub;

    if (tid == 0) {
        mbar_init(bar_x, 1);
        mbar_init(bar_y, 1);
        fence_mbar_init();
    }
    if (tid < 4) counts[tid] = 0;
    __syncthreads();

    // ---- the block's share of everything ----
    // Short rows line by line (a warp per sub-chunk), long rows listed in any
    // order (each is summed by itself).
    auto load_rows = [&](const FlatCsr& M, const uint16_t* idx, int begin, int n, int subs, const uint32_t* lines,
                         uint32_t* my_lines, uint2* ell, uint2* lent, int4* longs, uint32_t* range, uint32_t gather,
                         int* listed, int* entries) {
        for (int s = warp; s < subs; s += kWarps) {
            const int r = s * kResSub + lane;
            const int b = r < n ? M.row_ptr[begin + r] : 0, len = r < n ? M.row_ptr[begin + r + 1] - b : 0;
            const uint32_t ln = lines[s];
            if (lane == 0) my_lines[s] = ln;
            if (r < n) range[r] = uint32_t(b & 15) | uint32_t(len) << 4;
            uint2* line = ell + size_t(ln >> 5) * 32 + lane;
            for (int k = 0; k < int(ln & 31u); ++k)
                line[k * 32] = k < len && len <= kResLongRow
                                   ? make_uint2(__float_as_uint(M.val[b + k]), gather + 4u * idx[b + k])
                                   : make_uint2(0u, gather);
            const bool far = len > kResLongRow;
            int at = 0;
            if (far) {
                at = atomicAdd(entries, res_long_stride(len));
                longs[atomicAdd(listed, 1)] = make_int4(r, at, len, b);
            }
            unsigned todo = __ballot_sync(0xffffffffu, far);
            while (todo) {
                const int src = __ffs(int(todo)) - 1;
                todo &= todo - 1;
                const int fb = __shfl_sync(0xffffffffu, b, src), fl = __shfl_sync(0xffffffffu, len, src);
                const int fa = __shfl_sync(0xffffffffu, at, src);
                for (int k = lane; k < fl; k += 32)
                    lent[fa + k] = make_uint2(__float_as_uint(M.val[fb + k]), gather + 4u * idx[fb + k]);
            }
        }
    };
    load_rows(v.A, v.idx_a, me.r0, R, subs_y, v.lines_a + size_t(my_cta) * v.sub_y, lines_a, ell_a, lent_a, long_a, range_a,
              smem_u32(gx), &counts[0], &counts[2]);
    load_rows(v.AT, v.idx_t, me.c0, C, subs_x, v.lines_t + size_t(my_cta) * v.sub_x, lines_t, ell_t, lent_t, long_t, range_t,
              smem_u32(gy), &counts[1], &counts[3]);
    for (int j = tid; j < C; j += kResThreads) {
        const int g = me.c0 + j;
        xs[j] = algo.x[g];
        if constexpr (!kLean) cols[j] = make_float4(algo.tau[g], algo.c[g], algo.l_x[g], algo.u_x[g]);
        sx[j] = algo.x_bar[g];
    }
    for (int i = tid; i < R; i += kResThreads) {
        const int g = me.r0 + i;
        sy[i] = algo.y[g];
        if constexpr (!kLean) rows[i] = make_float4(algo.sigma[g], algo.r_lo[g], algo.r_hi[g], Algo::kMaster ? algo.y_m[g] : 0.0f);
    }
    // past the end of the last sub-chunks: sent, never read
    for (int j = C + tid; j < subs_x * kResSub; j += kResThreads) sx[j] = 0.0f;
    for (int i = R + tid; i < subs_y * kResSub; i += kResThreads) sy[i] = 0.0f;
    // the vector the first half reads, from global memory
    {
        const uint16_t* slot = Algo::kColsFirst ? v.slot_y + size_t(my_cta) * v.sub_y : v.slot_x + size_t(my_cta) * v.sub_x;
        const float* src = Algo::kColsFirst ? algo.y : algo.x_bar;
        float* dst = Algo::kColsFirst ? gy : gx;
        const int begin = Algo::kColsFirst ? me.lr0 : me.lc0, end = Algo::kColsFirst ? me.lr1 : me.lc1;
        for (int s = warp; begin + s * kResSub < end; s += kWarps) {
            const int at = slot[s];
            const int e = begin + s * kResSub + lane;
            if (at != kResNoSlot) dst[at * kResSub + lane] = e < end ? src[e] : 0.0f;
        }
    }
    // the receivers of every own sub-chunk
    const uint32_t gather_x = smem_u32(smem) + ResLayout::kGather;   // of block `lane` of the cluster
    const uint32_t gather_y =
        gather_x + (lane < cluster ? unsigned(v.cta[first_cta + lane].need_x) * (kResSub * 4) : 0u);
    auto find_receivers = [&](const uint16_t* slots, int stride, int first, int n, uint32_t gather, uint64_t* bar,
                              uint2* to, uint8_t* count) {
        for (int s = warp; s < n; s += kWarps) {
            const int at = lane < cluster ? slots[size_t(first_cta + lane) * stride + first + s] : kResNoSlot;
            const unsigned m = __ballot_sync(0xffffffffu, at != kResNoSlot);
            if (at != kResNoSlot)
                to[s * cluster + __popc(m & ((1u << lane) - 1u))] =
                    make_uint2(map_to_cta(gather + at * (kResSub * 4), lane), map_to_cta(smem_u32(bar), lane));
            if (lane == 0) count[s] = uint8_t(__popc(m));
        }
    };
    find_receivers(v.slot_x, v.sub_x, (me.c0 - me.lc0) / kResSub, subs_x, gather_x, bar_x, to_x, n_to_x);
    find_receivers(v.slot_y, v.sub_y, (me.r0 - me.lr0) / kResSub, subs_y, gather_y, bar_y, to_y, n_to_y);
    algo.begin(me);
    __syncthreads();
    const int nlong_a = counts[0], nlong_t = counts[1];
    // The first half reads what the last iteration's second half sent, the
    // second half what the first has sent; the last iteration's second half
    // sends nothing.  bar_first: the barrier of the vector the first half reads.
    uint64_t* bar_first = Algo::kColsFirst ? bar_y : bar_x;
    uint64_t* bar_second = Algo::kColsFirst ? bar_x : bar_y;
    const unsigned bytes_first = unsigned(Algo::kColsFirst ? me.need_y : me.need_x) * (kResSub * 4);
    const unsigned bytes_second = unsigned(Algo::kColsFirst ? me.need_x : me.need_y) * (kResSub * 4);
    if (tid == 0) mbar_arrive_expect_tx(bar_second, bytes_second);
    cluster_barrier();   // every block's mbarriers are ready

    auto side = [&](int ell, int lent, int to, int longs, int range, int lines, int k, int state, int out, int sums,
                    int n_to, int n, int subs, int begin, int nlong) {
        const uint32_t at = smem_u32(smem);
        return ResSide{at + ell, at + lent, at + to, at + longs, at + range, at + lines, at + k, at + state, at + out,
                       at + sums, at + n_to, n, subs, begin, nlong, cluster};
    };
    const ResSide SC = side(L.ell_t, L.lent_t, L.to_x, L.long_t, L.range_t, L.lines_t, L.cols, L.x, L.sx, L.sx, L.n_to_x, C,
                            subs_x, me.c0, nlong_t);
    const ResSide SR = side(L.ell_a, L.lent_a, L.to_y, L.long_a, L.range_a, L.lines_a, L.rows, L.sy, L.sy, L.long_sum,
                            L.n_to_y, R, subs_y, me.r0, nlong_a);
    ResCached cc[kResCached], cr[kResCached];
    res_load_cached<Algo, true, kLean>(SC, cc, algo, warp, lane);
    res_load_cached<Algo, false, kLean>(SR, cr, algo, warp, lane);

    bool ok = true;
    for (int it = 0; it < iters; ++it) {
        float w = 0.0f;
        if constexpr (Algo::kWeights) {
            if (it % kResWeights == 0) {   // an FP64 division each: computed once per block, not per thread
                if (tid < kResWeights) weights[tid] = algo.weight(it + tid);
                __syncthreads();
            }
            w = weights[it % kResWeights];
        }
        const uint32_t parity = uint32_t(it) & 1u;
        const bool more = it + 1 < iters;
        if (it > 0) ok = mbar_wait_cluster_bounded(bar_first, parity ^ 1u);
        // A block that gave up still runs its barriers; what it sends is discarded with the iterate.
        if constexpr (Algo::kColsFirst) res_half<Algo, true, kLean>(SC, cc, algo, w, algo.fpr_col(it, iters), true, warp, lane);
        else res_half<Algo, false, kLean>(SR, cr, algo, w, algo.fpr_row(it, iters), true, warp, lane);
        ok = mbar_wait_cluster_bounded(bar_second, parity) && ok;
        if constexpr (Algo::kColsFirst) res_half<Algo, false, kLean>(SR, cr, algo, w, algo.fpr_row(it, iters), more, warp, lane);
        else res_half<Algo, true, kLean>(SC, cc, algo, w, algo.fpr_col(it, iters), more, warp, lane);
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        // Every thread is past its waits of this iteration: bar_first takes the
        // phase its second half filled (perhaps already, before the bytes are
        // announced), bar_second the next iteration's.
        if (tid == 0 && more) {
            mbar_arrive_expect_tx(bar_first, bytes_first);
            mbar_arrive_expect_tx(bar_second, bytes_second);
        }
    }
    if (!ok) {
        if (tid == 0) atomicOr(v.status, kDevErrTimeout);
    } else {
#pragma unroll
        for (int u = 0; u < kResCached; ++u) {
            const int j = (warp + u * kWarps) * kResSub + lane;
            if (j < C) {
                algo.x[me.c0 + j] = cc[u].state;
                algo.x_bar[me.c0 + j] = cc[u].out;
            }
            if (j < R) algo.y[me.r0 + j] = cr[u].state;
        }
        for (int j = kResCached * kResThreads + tid; j < C; j += kResThreads) {
            algo.x[me.c0 + j] = xs[j];
            algo.x_bar[me.c0 + j] = sx[j];
        }
        for (int i = kResCached * kResThreads + tid; i < R; i += kResThreads) algo.y[me.r0 + i] = sy[i];
    }
    cluster_barrier();   // past it nobody stores into another block
    if (!ok) {           // what was sent to a block that gave up may not have landed
        const unsigned long long t0 = global_timer_ns();
        while (global_timer_ns() - t0 < kResDrainNs) __nanosleep(1000);
    }
}

// The reference iteration: rows first (y from A x̄), then columns (x, x̄ from A^T y).
struct ResReference {
    static constexpr bool kColsFirst = false;
    static constexpr int kOrder = kResFlat;
    static constexpr bool kMaster = false, kWeights = false;
    float *x, *x_bar, *y;
    const float *tau, *c, *l_x, *u_x, *sigma, *r_lo, *r_hi, *y_m;
    __device__ void begin(const ResCta&) {}
    __device__ double* fpr_col(int, int) const { return nullptr; }
    __device__ double* fpr_row(int, int) const { return nullptr; }
    __device__ float col(float4 s, float& xj, float aty, float, double*) const {
        float xb;
        xj = EpiPrimalRef::update(xj, s.x, s.y, s.z, s.w, aty, xb);
        return xb;
    }
    __device__ float row(float4 s, float y_old, float ax, float, double*) const {
        return EpiDualRef::update(y_old, s.x, s.y, s.z, ax);
    }
};

// The restarted Halpern iteration: columns first, then rows (EpiPrimalHalpern, EpiDualHalpern).
template <int kSumOrder>
struct ResHalpern {
    static constexpr bool kColsFirst = true;
    static constexpr int kOrder = kSumOrder;
    static constexpr bool kMaster = true, kWeights = true;
    float *x, *x_bar, *y;
    const float *tau, *c, *l_x, *u_x, *sigma, *r_lo, *r_hi, *y_m;
    const int *lp_row, *lp_col;        // null: one LP
    const int *restart_iter, *iter_base;
    double *fpr_c0, *fpr_c1, *fpr_r0, *fpr_r1;
    long long since;                   // iterations since the LP's restart, at the interval's start
    __device__ void begin(const ResCta& me) {
        const int q = lp_col && me.lc0 < me.lc1 ? lp_col[me.lc0] : (lp_row && me.lr0 < me.lr1 ? lp_row[me.lr0] : 0);
        since = (long long)(*iter_base) - restart_iter[q];
    }
    __device__ float weight(int it) const { return halpern_weight_of(since + it); }
    __device__ double* fpr_col(int it, int iters) const { return it == 0 ? fpr_c0 : (it == iters - 1 ? fpr_c1 : nullptr); }
    __device__ double* fpr_row(int it, int iters) const { return it == 0 ? fpr_r0 : (it == iters - 1 ? fpr_r1 : nullptr); }
    __device__ float col(float4 s, float& xj, float aty, float w, double* fpr) const {
        const EpiPrimalHalpern::In in{xj, s.x, s.y, s.z, s.w, 0.0f, w};
        float xb;
        xj = EpiPrimalHalpern::update(in, aty, xb, fpr);
        return xb;
    }
    __device__ float row(float4 s, float e_old, float ax, float w, double* fpr) const {
        const EpiDualHalpern::In in{s.x, e_old, s.w, s.z, s.y, 0.0f, w};
        return EpiDualHalpern::update(in, ax, fpr);
    }
};

// ---- host ------------------------------------------------------------------------
// How the LPs of an operand are cut over clusters.  Built once per layout, on
// the device, from the flat operands (kept by keep_flat).
class ResidentPlan {
public:
    // Blocks per cluster for LPs of these sizes ({rows, columns, non-zeros}):
    // the smallest size whose shared memory should hold each LP, and larger while
    // a warp would have more than one sub-chunk of a side (a half iteration lasts
    // as long as its longest warp) and all clusters together leave SMs idle.
    // kResLean: the largest clusters with the constants in global memory;
    // 0: too large for any cluster.
    static std::vector<int> sizes_for(const std::vector<int4>& shapes, int sms);
    // How often over clusters of these sizes fill the SMs (1 or less: they run
    // at the same time; infinite with a size 0).
    static constexpr double kMaxRounds = 8.0;
    static double rounds(const std::vector<int>& sizes, int sms);

    // Cuts the LPs {r0, r1, c0, c1} over clusters of `size` blocks, or of the
    // next size that holds them all.  Leaves ok() false when none does.
    // Synchronises `st`.
    void build(const CsrDevice& A, const CsrDevice& AT, const std::vector<int4>& lps, int size, cudaStream_t st);
    void reset() { clusters_ = 0; }
    bool ok() const { return clusters_ > 0; }
    int clusters() const { return clusters_; }
    int cluster_size() const { return size_; }

    template <class Algo>
    void launch(const CsrDevice& A, const CsrDevice& AT, const Algo& algo, int iters, int* status, cudaStream_t st) const {
        if (running_ == 0) return;
        const FlatCsr fa{A.row_ptr.get(), A.col.get(), A.val.get()}, ft{AT.row_ptr.get(), AT.col.get(), AT.val.get()};
        ResView v;
        v.which = which_.get();
        v.cta = cta_.get();
        v.slot_x = slot_x_.get();
        v.slot_y = slot_y_.get();
        v.lines_a = lines_a_.get();
        v.lines_t = lines_t_.get();
        v.sub_x = sub_x_;
        v.sub_y = sub_y_;
        v.A = fa;
        v.AT = ft;
        v.idx_a = idx_a_.get();
        v.idx_t = idx_t_.get();
        v.status = status;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        config(cfg, attr, st);
        if (lean_) PB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, resident_kernel<Algo, true>, v, algo, iters));
        else PB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, resident_kernel<Algo, false>, v, algo, iters));
    }
    // Launches only the LPs whose flag is set (plan order) from now on.
    void run_only(const std::vector<char>& flags, cudaStream_t st);

    // Sets the kernel's attributes and asks whether the device can run the
    // plan's clusters; clears the plan when it cannot.
    template <class Algo>
    void prepare() {
        if (!ok()) return;
        auto k = lean_ ? resident_kernel<Algo, true> : resident_kernel<Algo, false>;
        PB_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kResMaxSmem)));
        PB_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        config(cfg, attr, nullptr);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess || n < 1) {
            (void)cudaGetLastError();
            clusters_ = 0;
        }
    }

private:
    void config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, cudaStream_t st) const {
        cfg.gridDim = dim3(unsigned(running_ * size_));
        cfg.blockDim = dim3(kResThreads);
        cfg.dynamicSmemBytes = smem_;
        cfg.stream = st;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = unsigned(size_);
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    bool cut(const CsrDevice& A, const CsrDevice& AT, const std::vector<int4>& lps, int size, cudaStream_t st);

    bool lean_ = false;
    int clusters_ = 0, running_ = 0, size_ = 1, sub_x_ = 0, sub_y_ = 0;
    size_t smem_ = 0;
    DevBuf<int4> lps_;
    DevBuf<int> which_;
    DevBuf<ResCta> cta_;
    DevBuf<uint16_t> slot_x_, slot_y_, idx_a_, idx_t_;
    DevBuf<uint32_t> lines_a_, lines_t_;
};

}  // namespace pb
