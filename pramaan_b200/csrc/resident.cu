// resident.cu — builds the cluster plan of resident.cuh on the device.
#include "resident.cuh"

#include <algorithm>

namespace pb {

namespace {

// First row r of [r0, r1] whose rows before it weigh at least `part` of `parts`
// of the LP, an entry 2 and a row 1.  (By shared-memory bytes, 8 and 28, the
// blocks with a planning LP's coupling rows, 48 entries each at the end of A,
// had 190 of them, the largest share of memory and twice the others' time.)
__device__ int share_begin(const int* __restrict__ rp, int r0, int r1, int part, int parts) {
    if (part == 0) return r0;
    if (part == parts) return r1;
    const long long base = rp[r0];
    auto weight = [&](int r) { return 2 * ((long long)rp[r] - base) + (r - r0); };
    const long long want = weight(r1) * part / parts;
    int lo = r0, hi = r1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (weight(mid) >= want) hi = mid; else lo = mid + 1;
    }
    // shares begin at whole sub-chunks of their LP
    return min(r0 + (lo - r0 + kResSub / 2) / kResSub * kResSub, r1);
}

__global__ void share_kernel(const int4* __restrict__ lps, int blocks, int size, const int* __restrict__ rp_a,
                             const int* __restrict__ rp_t, ResCta* __restrict__ cta) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= blocks) return;
    const int4 lp = lps[b / size];
    const int part = b % size;
    ResCta c;
    c.lr0 = lp.x; c.lr1 = lp.y; c.lc0 = lp.z; c.lc1 = lp.w;
    c.r0 = share_begin(rp_a, lp.x, lp.y, part, size);
    c.r1 = share_begin(rp_a, lp.x, lp.y, part + 1, size);
    c.c0 = share_begin(rp_t, lp.z, lp.w, part, size);
    c.c1 = share_begin(rp_t, lp.z, lp.w, part + 1, size);
    c.need_x = c.need_y = c.ell_a = c.ell_t = c.long_a = c.long_t = c.lent_a = c.lent_t = 0;
    cta[b] = c;
}

// One block per share and side: which sub-chunks its entries refer to, their
// slots (in order), the entries' positions in the gather vector, and the lines
// its own sub-chunks' short rows take.
// Dynamic shared memory per sub-chunk of the LP: a word, a slot and a flag byte.
__global__ void __launch_bounds__(256) slot_kernel(ResCta* __restrict__ cta, int blocks, const int* __restrict__ rp_a,
                                                   const int* __restrict__ col_a, const int* __restrict__ rp_t,
                                                   const int* __restrict__ col_t, int sub_x, int sub_y,
                                                   uint16_t* __restrict__ slot_x, uint16_t* __restrict__ slot_y,
                                                   uint16_t* __restrict__ idx_a, uint16_t* __restrict__ idx_t,
                                                   uint32_t* __restrict__ lines_a, uint32_t* __restrict__ lines_t) {
    extern __shared__ uint32_t own_lines[];
    __shared__ int s_long, s_entries;
    const int b = blockIdx.x >> 1;
    const bool rows = (blockIdx.x & 1) == 0;   // rows of A refer to x̄, columns to y
    const ResCta c = cta[b];
    const int subs = rows ? sub_x : sub_y;
    const int most = sub_x > sub_y ? sub_x : sub_y;
    uint16_t* slots = reinterpret_cast<uint16_t*>(own_lines + most);
    unsigned char* flag = reinterpret_cast<unsigned char*>(slots + most);
    const int e0 = rows ? rp_a[c.r0] : rp_t[c.c0], e1 = rows ? rp_a[c.r1] : rp_t[c.c1];
    const int* col = rows ? col_a : col_t;
    const int base = rows ? c.lc0 : c.lr0;
    for (int s = threadIdx.x; s < subs; s += blockDim.x) flag[s] = 0;
    __syncthreads();
    for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) flag[(col[e] - base) / kResSub] = 1;
    __syncthreads();
    uint16_t* out = (rows ? slot_x : slot_y) + size_t(b) * subs;
    if (threadIdx.x < 32) {
        int count = 0;
        for (int s0 = 0; s0 < subs; s0 += 32) {
            const int s = s0 + int(threadIdx.x);
            const bool on = s < subs && flag[s];
            const unsigned m = __ballot_sync(0xffffffffu, on);
            const uint16_t at = on ? uint16_t(count + __popc(m & ((1u << threadIdx.x) - 1u))) : kResNoSlot;
            if (s < subs) out[s] = slots[s] = at;
            count += __popc(m);
        }
        if (threadIdx.x == 0) (rows ? cta[b].need_x : cta[b].need_y) = count;
    }
    __syncthreads();
    uint16_t* idx = rows ? idx_a : idx_t;
    for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
        const int o = col[e] - base;
        idx[e] = uint16_t(slots[o / kResSub] * kResSub + o % kResSub);
    }
    // ---- the own rows ----
    const int* rp = rows ? rp_a : rp_t;
    const int begin = rows ? c.r0 : c.c0, n = rows ? c.r1 - c.r0 : c.c1 - c.c0;
    const int own = (n + kResSub - 1) / kResSub, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) s_long = s_entries = 0;
    __syncthreads();
    for (int s = threadIdx.x >> 5; s < own; s += blockDim.x >> 5) {
        const int r = s * kResSub + lane;
        const int len = r < n ? rp[begin + r + 1] - rp[begin + r] : 0;
        const int lines = __reduce_max_sync(0xffffffffu, len <= kResLongRow ? len : 0);
        const int count = __popc(__ballot_sync(0xffffffffu, len > kResLongRow));
        const int entries = __reduce_add_sync(0xffffffffu, len > kResLongRow ? res_long_stride(len) : 0);
        if (lane == 0) {
            own_lines[s] = uint32_t(lines);
            if (count) {
                atomicAdd(&s_long, count);
                atomicAdd(&s_entries, entries);
            }
        }
    }
    __syncthreads();
    uint32_t* lines_out = (rows ? lines_a : lines_t) + size_t(b) * (rows ? sub_y : sub_x);
    if (threadIdx.x == 0) {
        uint32_t at = 0;
        for (int s = 0; s < own; ++s) {
            lines_out[s] = at << 5 | own_lines[s];
            at += own_lines[s];
        }
        (rows ? cta[b].ell_a : cta[b].ell_t) = int(at);
        (rows ? cta[b].long_a : cta[b].long_t) = s_long;
        (rows ? cta[b].lent_a : cta[b].lent_t) = s_entries;
    }
}

}  // namespace

bool ResidentPlan::cut(const CsrDevice& A, const CsrDevice& AT, const std::vector<int4>& lps, int size, cudaStream_t st) {
    const int blocks = int(lps.size()) * size;
    cta_.alloc(size_t(blocks));
    slot_x_.alloc(size_t(blocks) * sub_x_);
    slot_y_.alloc(size_t(blocks) * sub_y_);
    lines_a_.alloc(size_t(blocks) * sub_y_);
    lines_t_.alloc(size_t(blocks) * sub_x_);
    share_kernel<<<(blocks + 127) / 128, 128, 0, st>>>(lps_.get(), blocks, size, A.row_ptr.get(), AT.row_ptr.get(),
                                                       cta_.get());
    PB_CUDA_CHECK(cudaGetLastError());
    slot_kernel<<<2 * blocks, 256, size_t(std::max(sub_x_, sub_y_)) * 7, st>>>(
        cta_.get(), blocks, A.row_ptr.get(), A.col.get(), AT.row_ptr.get(), AT.col.get(), sub_x_, sub_y_, slot_x_.get(),
        slot_y_.get(), idx_a_.get(), idx_t_.get(), lines_a_.get(), lines_t_.get());
    PB_CUDA_CHECK(cudaGetLastError());
    std::vector<ResCta> h(static_cast<size_t>(blocks));
    PB_CUDA_CHECK(cudaMemcpyAsync(h.data(), cta_.get(), h.size() * sizeof(ResCta), cudaMemcpyDeviceToHost, st));
    PB_CUDA_CHECK(cudaStreamSynchronize(st));
    smem_ = 0;
    for (const ResCta& c : h) {
        if (std::max(c.need_x, c.need_y) * kResSub > 65536) return false;   // positions are 16 bits
        // before the layout's byte counts, which are ints
        const long long entries = 32LL * c.ell_a + 32LL * c.ell_t + c.lent_a + c.lent_t;
        if (8 * entries > (long long)kResMaxSmem) return false;
        smem_ = std::max(smem_, size_t(ResLayout(c, size, lean_).total));
    }
    return smem_ <= kResMaxSmem;
}

namespace {
// Cluster sizes: what tiles a GPC of 18 to 20 SMs well.
constexpr int kSizes[] = {1, 2, 3, 4, 6, 8, 16};
constexpr int kNumSizes = int(sizeof(kSizes) / sizeof(kSizes[0]));
static_assert(kSizes[kNumSizes - 1] == kResMaxCluster, "cluster sizes");
int next_size(int size) {
    for (int s : kSizes)
        if (s > size) return s;
    return 0;
}
}  // namespace

std::vector<int> ResidentPlan::sizes_for(const std::vector<int4>& shapes, int sms) {
    std::vector<int> size;
    for (const int4& q : shapes) {
        // both operands' entries, the vectors, and gather vectors of a few sub-chunks per row
        const long long elements = (long long)q.x + q.y, block = kResMaxSmem - 8192;
        int s = 1;
        while (s && 16LL * q.z + 36 * elements > s * block) s = next_size(s);
        if (s == 0 && 16LL * q.z + 20 * elements <= kResMaxCluster * block) s = kResLean;
        size.push_back(s);
    }
    while (true) {
        std::vector<int> larger = size;
        for (size_t k = 0; k < size.size(); ++k) {
            const int subs = (std::max(shapes[k].x, shapes[k].y) + kResSub - 1) / kResSub;
            if (size[k] > 0 && size[k] < kResMaxCluster && 4 * subs > 3 * size[k] * 16)
                larger[k] = next_size(size[k]);
        }
        if (larger == size || rounds(larger, sms) > 1.0) return size;
        size = std::move(larger);
    }
}

// A cluster lies in one GPC, of 18 to 20 SMs: the largest take a GPC each (7 at
// a time on 148 SMs).
double ResidentPlan::rounds(const std::vector<int>& sizes, int sms) {
    long long taken = 0;
    for (int s : sizes) {
        if (s == 0) return 1e30;
        taken += s == kResLean || s == kResMaxCluster ? 20 : s == 8 ? 9 : s;
    }
    return double(taken) / sms;
}

void ResidentPlan::build(const CsrDevice& A, const CsrDevice& AT, const std::vector<int4>& lps, int size,
                         cudaStream_t st) {
    clusters_ = running_ = 0;
    lean_ = size == kResLean;
    if (lean_) size = kResMaxCluster;
    if (lps.empty() || size <= 0 || A.nnz == 0 || !A.col.get() || !A.val.get() || !AT.col.get() || !AT.val.get()) return;
    sub_x_ = sub_y_ = 1;
    for (const int4& lp : lps) {
        sub_x_ = std::max(sub_x_, (lp.w - lp.z + kResSub - 1) / kResSub);
        sub_y_ = std::max(sub_y_, (lp.y - lp.x + kResSub - 1) / kResSub);
    }
    if (size_t(std::max(sub_x_, sub_y_)) * 7 > 48 * 1024) return;
    lps_.alloc(lps.size());
    idx_a_.alloc(size_t(A.nnz));
    idx_t_.alloc(size_t(AT.nnz));
    PB_CUDA_CHECK(cudaMemcpyAsync(lps_.get(), lps.data(), lps.size() * sizeof(int4), cudaMemcpyHostToDevice, st));
    for (; size > 0; size = next_size(size)) {
        if (!cut(A, AT, lps, size, st)) {
            if (size == kResMaxCluster && !lean_) {   // once more without the constants
                lean_ = true;
                if (!cut(A, AT, lps, size, st)) return;
            } else {
                continue;
            }
        }
        size_ = size;
        clusters_ = running_ = int(lps.size());
        which_.reset();
        return;
    }
}

void ResidentPlan::run_only(const std::vector<char>& flags, cudaStream_t st) {
    std::vector<int> list;
    for (size_t k = 0; k < flags.size(); ++k)
        if (flags[k]) list.push_back(int(k));
    running_ = int(list.size());
    if (list.empty()) return;
    if (which_.size() == 0) which_.alloc(size_t(clusters_));
    PB_CUDA_CHECK(cudaMemcpyAsync(which_.get(), list.data(), list.size() * sizeof(int), cudaMemcpyHostToDevice, st));
    PB_CUDA_CHECK(cudaStreamSynchronize(st));   // the list is freed on return
}

}  // namespace pb
