// gnn.cu — the warm-start network: graph packing, tensor-core dense layers,
// gather aggregations, deterministic reductions, loss, backward and Adam.
// The network itself is documented in gnn.cuh.
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <mutex>

#include "gnn.cuh"
#include "umma.cuh"

namespace pb {

using bf16 = __nv_bfloat16;

// ---------------------------------------------------------------------------
// Tensor maps
// ---------------------------------------------------------------------------
namespace {
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    if (!fn) throw CudaError("CUDA error in gnn.cu - cuTensorMapEncodeTiled is unavailable");
    return fn;
}
}  // namespace

CUtensorMap make_bf16_tile_map(const void* base, long long rows, int cols, int pitch_elems, int box_rows) {
    CUtensorMap m;
    std::memset(&m, 0, sizeof(m));
    const cuuint64_t dims[2] = {cuuint64_t(cols), cuuint64_t(rows > 0 ? rows : 1)};
    const cuuint64_t strides[1] = {cuuint64_t(pitch_elems) * 2};
    const cuuint32_t box[2] = {64u, cuuint32_t(box_rows)};
    const cuuint32_t estr[2] = {1u, 1u};
    const CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box,
                                   estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        throw CudaError("CUDA error in gnn.cu - cuTensorMapEncodeTiled failed (" + std::to_string(int(r)) + ")");
    return m;
}

namespace {

constexpr int kT = 256;
int grid_for(long long work) {
    long long g = (work + kT - 1) / kT;
    return int(std::max<long long>(1, std::min<long long>(g, 148LL * 32)));
}
// Grid of the kernels with 8 lanes per row (they stride by the grid).
int row_grid(long long rows) { return grid_for(rows * 8); }
#define GNN_STRIDE(i, n) \
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (n); i += (long long)gridDim.x * blockDim.x)

__device__ __forceinline__ float bf(bf16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float bfr(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// ---------------------------------------------------------------------------
// Dense layers on the tensor cores
// ---------------------------------------------------------------------------
constexpr int kRowsPerTile = 128;
constexpr uint32_t kBoxBytes = 128u * 128u;   // 128 rows x 64 BF16
constexpr int kDenseThreads = 128;

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
    return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}

// Each lane holds its own row of 32 FP32 values; row-wise stores would touch
// 32 half-used sectors an instruction, so a warp's rows go through 4 KB of
// shared memory (the tile's consumed TMA stage) and leave as whole 128-byte
// lines.  Chunk c of 16 bytes of row r lies at chunk c ^ (r & 7): neither side
// has bank conflicts.
__device__ __forceinline__ uint4* staged_chunk(uint8_t* buf, int r, int c) {
    return reinterpret_cast<uint4*>(buf + r * 128 + ((c ^ (r & 7)) << 4));
}
__device__ __forceinline__ void stage_bf16x32(uint8_t* buf, int lane, int half, const float (&v)[32]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            __nv_bfloat162 p = __floats2bfloat162_rn(v[8 * q + 2 * e], v[8 * q + 2 * e + 1]);
            w[e] = *reinterpret_cast<uint32_t*>(&p);
        }
        *staged_chunk(buf, lane, half * 4 + q) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}
__device__ __forceinline__ void stage_f32x32(uint8_t* buf, int lane, const float (&v)[32]) {
#pragma unroll
    for (int q = 0; q < 8; ++q)
        *reinterpret_cast<float4*>(staged_chunk(buf, lane, q)) =
            make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
}
// The staged rows (row0 .. row0 + 31, those below `rows`) to dst + row * pitch bytes, 128 bytes each.
__device__ __forceinline__ void unstage_rows(uint8_t* buf, int lane, uint8_t* dst, size_t pitch, int row0, int rows) {
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = 4 * i + (lane >> 3), c = lane & 7;
        const uint4 v = *staged_chunk(buf, r, c);
        if (row0 + r < rows) *reinterpret_cast<uint4*>(dst + size_t(row0 + r) * pitch + 16 * c) = v;
    }
    __syncwarp();
}
__device__ __forceinline__ void store_f32x32(float* dst, const float (&v)[32]) {
    float4* d = reinterpret_cast<float4*>(dst);
#pragma unroll
    for (int q = 0; q < 8; ++q) d[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
}

// Waits, with a limit, for the TMA copies still in flight on a stage before
// the block exits after an error.
__device__ __forceinline__ void drain(uint64_t* bar, bool pending, uint32_t parity) {
    if (pending) mbar_wait_bounded(bar, parity);
}

// A node head read off the last layer's rows: hat[r] = base[r] + (w . h[r] + b)
// (wb: 64 rounded weights, then the bias); wb null: none.
struct Head {
    const float* wb = nullptr;
    const float* base = nullptr;
    float* hat = nullptr;
};

// Forward: out[r][0:64] = bf16(relu(X[r] . W^T + b)), X = [rows][128] BF16.
// Shared memory: X stages 2 x 32 KB, W 16 KB, bias, head weights, barriers.
struct FwdSmem {
    static constexpr uint32_t kA = 0;
    static constexpr uint32_t kB = 2 * 2 * kBoxBytes;             // 65536
    static constexpr uint32_t kBias = kB + 2 * 64 * 128;          // 81920
    static constexpr uint32_t kHead = kBias + 64 * 4;             // 65 floats
    static constexpr uint32_t kBars = kHead + 68 * 4;
    static constexpr uint32_t kBytes = kBars + 64 + 1024;         // + alignment slack
};
constexpr uint32_t kIdescFwd = umma::idesc_bf16<128, 64, false, false>();
constexpr uint32_t kIdescDx = umma::idesc_bf16<128, 128, false, false>();
constexpr uint32_t kIdescDw = umma::idesc_bf16<128, 64, true, true>();

__global__ void __launch_bounds__(kDenseThreads) dense_fwd_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                  const __grid_constant__ CUtensorMap map_w,
                                                                  const float* __restrict__ bias, bf16* __restrict__ out,
                                                                  int ld_out, const Head head, int rows, int* status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = align1024(smem_raw);
    uint8_t* sA = sm + FwdSmem::kA;
    uint8_t* sB = sm + FwdSmem::kB;
    float* sbias = reinterpret_cast<float*>(sm + FwdSmem::kBias);
    uint64_t* full = reinterpret_cast<uint64_t*>(sm + FwdSmem::kBars);   // [2]
    uint64_t* wbar = full + 2;
    uint64_t* mbar = full + 3;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(full + 4);
    const int tid = threadIdx.x, warp = tid >> 5;
    const int ntiles = (rows + kRowsPerTile - 1) / kRowsPerTile;

    if (tid == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        mbar_init(wbar, 1);
        mbar_init(mbar, 1);
        fence_mbar_init();
        umma::tma_prefetch_map(&map_x);
        umma::tma_prefetch_map(&map_w);
    }
    if (warp == 0) umma::tmem_alloc(tslot, 64);
    float* shead = reinterpret_cast<float*>(sm + FwdSmem::kHead);
    if (tid < 64) sbias[tid] = bias[tid];
    if (head.wb && tid < 65) shead[tid] = head.wb[tid];
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tslot;

    bool pend[2] = {false, false};
    uint32_t uses[2] = {0, 0};
    if (tid == 0) {
        mbar_arrive_expect_tx(wbar, 2 * 64 * 128);
        umma::tma_load_2d(sB, &map_w, 0, 0, wbar);
        umma::tma_load_2d(sB + 64 * 128, &map_w, 64, 0, wbar);
        if (int(blockIdx.x) < ntiles) {
            mbar_arrive_expect_tx(&full[0], 2 * kBoxBytes);
            umma::tma_load_2d(sA, &map_x, 0, blockIdx.x * kRowsPerTile, &full[0]);
            umma::tma_load_2d(sA + kBoxBytes, &map_x, 64, blockIdx.x * kRowsPerTile, &full[0]);
            pend[0] = true;
        }
    }
    bool ok = true;
    bool w_pending = tid == 0;
    int it = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
        const int s = it & 1;
        if (tid == 0) {
            const int next = tile + gridDim.x;
            if (next < ntiles) {
                uint8_t* dst = sA + (s ^ 1) * 2 * kBoxBytes;
                mbar_arrive_expect_tx(&full[s ^ 1], 2 * kBoxBytes);
                umma::tma_load_2d(dst, &map_x, 0, next * kRowsPerTile, &full[s ^ 1]);
                umma::tma_load_2d(dst + kBoxBytes, &map_x, 64, next * kRowsPerTile, &full[s ^ 1]);
                pend[s ^ 1] = true;
            }
            bool w_ok = true;
            if (w_pending) { w_ok = mbar_wait_bounded(wbar, 0); w_pending = !w_ok; }
            const bool f_ok = w_ok && mbar_wait_bounded(&full[s], uses[s] & 1);
            if (f_ok) {
                pend[s] = false;
                ++uses[s];
                umma::fence_after_sync();
                const uint32_t a0 = smem_u32(sA + s * 2 * kBoxBytes), b0 = smem_u32(sB);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint64_t ad = umma::smem_desc(a0 + (k >> 2) * kBoxBytes + (k & 3) * 32, 16, 1024);
                    const uint64_t bd = umma::smem_desc(b0 + (k >> 2) * (64 * 128) + (k & 3) * 32, 16, 1024);
                    umma::mma_bf16(tmem, ad, bd, kIdescFwd, k > 0 ? 1u : 0u);
                }
                umma::mma_commit(mbar);
            } else {
                ok = false;
            }
        }
        ok = mbar_wait_bounded(mbar, it & 1) && ok;
        if (!__syncthreads_and(ok)) { ok = false; break; }
        umma::fence_after_sync();
        __syncwarp();
        const int row = tile * kRowsPerTile + tid;
        const uint32_t taddr = tmem + (uint32_t(warp * 32) << 16);
        uint8_t* buf = sA + s * 2 * kBoxBytes + warp * 4096;   // the MMAs have read this stage
        float dot[16];   // the head's dot product, feature pairs folded as a 32-lane xor tree folds them
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float v[32];
            umma::tmem_ld32(taddr + h * 32, v);
#pragma unroll
            for (int c = 0; c < 32; ++c) v[c] = fmaxf(v[c] + sbias[h * 32 + c], 0.0f);
            stage_bf16x32(buf, tid & 31, h, v);
            if (head.wb) {
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    const float2 w = *reinterpret_cast<const float2*>(shead + h * 32 + 2 * q);
                    const float d = fmaf(w.y, bfr(v[2 * q + 1]), __fmul_rn(w.x, bfr(v[2 * q])));
                    dot[q] = h == 0 ? d : dot[q] + d;
                }
            }
        }
        if (head.wb && row < rows) {
#pragma unroll
            for (int o = 8; o > 0; o >>= 1)
#pragma unroll
                for (int q = 0; q < o; ++q) dot[q] += dot[q + o];
            head.hat[row] = head.base[row] + (dot[0] + shead[64]);
        }
        unstage_rows(buf, tid & 31, reinterpret_cast<uint8_t*>(out), size_t(ld_out) * 2, tile * kRowsPerTile + warp * 32,
                     rows);
        fence_proxy_async_smem();   // before the next TMA load into the stage
        umma::fence_before_sync();
        __syncthreads();
    }
    if (tid == 0) {
        if (w_pending) mbar_wait_bounded(wbar, 0);   // a block without tiles still loaded W
        if (!ok) {
            atomicOr(status, kDevErrTimeout);
            drain(&full[0], pend[0], uses[0] & 1);
            drain(&full[1], pend[1], uses[1] & 1);
        }
    }
    __syncthreads();
    if (warp == 0) {
        umma::fence_after_sync();
        umma::tmem_dealloc(tmem, 64);
    }
}

// Input gradient: [dh_prev | dagg][r] = dZ[r] . W  (dZ [rows][64] BF16,
// W^T given as [128][64] BF16), FP32 outputs of 64 columns each.
struct DxSmem {
    static constexpr uint32_t kA = 0;                      // 2 stages x 16 KB
    static constexpr uint32_t kB = 2 * kBoxBytes;          // W^T 16 KB
    static constexpr uint32_t kBars = kB + kBoxBytes;
    // padded so that at most four blocks (4 x 128 tensor-memory columns) share an SM
    static constexpr uint32_t kBytes = 57 * 1024;
};

__global__ void __launch_bounds__(kDenseThreads) dense_dx_kernel(const __grid_constant__ CUtensorMap map_dz,
                                                                 const __grid_constant__ CUtensorMap map_wt,
                                                                 float* __restrict__ dh_prev, float* __restrict__ dagg,
                                                                 int rows, int* status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = align1024(smem_raw);
    uint8_t* sA = sm + DxSmem::kA;
    uint8_t* sB = sm + DxSmem::kB;
    uint64_t* full = reinterpret_cast<uint64_t*>(sm + DxSmem::kBars);
    uint64_t* wbar = full + 2;
    uint64_t* mbar = full + 3;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(full + 4);
    const int tid = threadIdx.x, warp = tid >> 5;
    const int ntiles = (rows + kRowsPerTile - 1) / kRowsPerTile;

    if (tid == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        mbar_init(wbar, 1);
        mbar_init(mbar, 1);
        fence_mbar_init();
        umma::tma_prefetch_map(&map_dz);
        umma::tma_prefetch_map(&map_wt);
    }
    if (warp == 0) umma::tmem_alloc(tslot, 128);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tslot;

    bool pend[2] = {false, false};
    uint32_t uses[2] = {0, 0};
    if (tid == 0) {
        mbar_arrive_expect_tx(wbar, kBoxBytes);
        umma::tma_load_2d(sB, &map_wt, 0, 0, wbar);
        if (int(blockIdx.x) < ntiles) {
            mbar_arrive_expect_tx(&full[0], kBoxBytes);
            umma::tma_load_2d(sA, &map_dz, 0, blockIdx.x * kRowsPerTile, &full[0]);
            pend[0] = true;
        }
    }
    bool ok = true;
    bool w_pending = tid == 0;
    int it = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
        const int s = it & 1;
        if (tid == 0) {
            const int next = tile + gridDim.x;
            if (next < ntiles) {
                mbar_arrive_expect_tx(&full[s ^ 1], kBoxBytes);
                umma::tma_load_2d(sA + (s ^ 1) * kBoxBytes, &map_dz, 0, next * kRowsPerTile, &full[s ^ 1]);
                pend[s ^ 1] = true;
            }
            bool w_ok = true;
            if (w_pending) { w_ok = mbar_wait_bounded(wbar, 0); w_pending = !w_ok; }
            const bool f_ok = w_ok && mbar_wait_bounded(&full[s], uses[s] & 1);
            if (f_ok) {
                pend[s] = false;
                ++uses[s];
                umma::fence_after_sync();
                const uint32_t a0 = smem_u32(sA + s * kBoxBytes), b0 = smem_u32(sB);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint64_t ad = umma::smem_desc(a0 + k * 32, 16, 1024);
                    const uint64_t bd = umma::smem_desc(b0 + k * 32, 16, 1024);
                    umma::mma_bf16(tmem, ad, bd, kIdescDx, k > 0 ? 1u : 0u);
                }
                umma::mma_commit(mbar);
            } else {
                ok = false;
            }
        }
        ok = mbar_wait_bounded(mbar, it & 1) && ok;
        if (!__syncthreads_and(ok)) { ok = false; break; }
        umma::fence_after_sync();
        __syncwarp();
        const uint32_t taddr = tmem + (uint32_t(warp * 32) << 16);
        uint8_t* buf = sA + s * kBoxBytes + warp * 4096;   // the MMAs have read this stage
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            float v[32];
            umma::tmem_ld32(taddr + h * 32, v);
            stage_f32x32(buf, tid & 31, v);
            float* dst = h < 2 ? dh_prev + h * 32 : dagg + (h - 2) * 32;
            unstage_rows(buf, tid & 31, reinterpret_cast<uint8_t*>(dst), 64 * 4, tile * kRowsPerTile + warp * 32, rows);
        }
        fence_proxy_async_smem();   // before the next TMA load into the stage
        umma::fence_before_sync();
        __syncthreads();
    }
    if (tid == 0) {
        if (w_pending) mbar_wait_bounded(wbar, 0);   // a block without tiles still loaded W
        if (!ok) {
            atomicOr(status, kDevErrTimeout);
            drain(&full[0], pend[0], uses[0] & 1);
            drain(&full[1], pend[1], uses[1] & 1);
        }
    }
    __syncthreads();
    if (warp == 0) {
        umma::fence_after_sync();
        umma::tmem_dealloc(tmem, 128);
    }
}

// Weight gradient: partial[block][f][g] = sum over this block's row tiles of
// X[r][f] dZ[r][g]  (D = X^T dZ, both operands MN-major, K = rows).
struct DwSmem {
    static constexpr uint32_t kStage = 3 * kBoxBytes;      // X (2 boxes) + dZ (1 box)
    static constexpr uint32_t kBars = 2 * kStage;          // 98304
    static constexpr uint32_t kBytes = kBars + 64 + 1024;
};

__global__ void __launch_bounds__(kDenseThreads) dense_dw_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                 const __grid_constant__ CUtensorMap map_dz,
                                                                 float* __restrict__ partial, int rows, int* status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = align1024(smem_raw);
    uint64_t* full = reinterpret_cast<uint64_t*>(sm + DwSmem::kBars);   // [2]
    uint64_t* empty = full + 2;                                          // [2]
    uint64_t* done = full + 4;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(full + 5);
    const int tid = threadIdx.x, warp = tid >> 5;
    const int ntiles = (rows + kRowsPerTile - 1) / kRowsPerTile;
    const int mine = ntiles > int(blockIdx.x) ? (ntiles - 1 - int(blockIdx.x)) / int(gridDim.x) + 1 : 0;

    if (tid == 0) {
        for (int i = 0; i < 5; ++i) mbar_init(&full[i], 1);
        fence_mbar_init();
        umma::tma_prefetch_map(&map_x);
        umma::tma_prefetch_map(&map_dz);
    }
    if (warp == 0) umma::tmem_alloc(tslot, 64);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tslot;

    bool ok = true;
    if (tid == 0) {
        bool pend[2] = {false, false};
        uint32_t fuses[2] = {0, 0}, euses[2] = {0, 0};
        auto load = [&](int i) {
            const int s = i & 1;
            const int r0 = (int(blockIdx.x) + i * int(gridDim.x)) * kRowsPerTile;
            uint8_t* st = sm + s * DwSmem::kStage;
            mbar_arrive_expect_tx(&full[s], 3 * kBoxBytes);
            umma::tma_load_2d(st, &map_x, 0, r0, &full[s]);
            umma::tma_load_2d(st + kBoxBytes, &map_x, 64, r0, &full[s]);
            umma::tma_load_2d(st + 2 * kBoxBytes, &map_dz, 0, r0, &full[s]);
            pend[s] = true;
        };
        if (mine > 0) load(0);
        if (mine > 1) load(1);
        for (int i = 0; i < mine; ++i) {
            const int s = i & 1;
            if (!mbar_wait_bounded(&full[s], fuses[s] & 1)) { ok = false; break; }
            pend[s] = false;
            ++fuses[s];
            umma::fence_after_sync();
            const uint32_t a0 = smem_u32(sm + s * DwSmem::kStage);
            const uint32_t b0 = a0 + 2 * kBoxBytes;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                // A: two 64-feature chunks 16 KB apart (LBO); B: one 64-wide chunk, so its
                // LBO is unused and kept small (every address stays inside this stage)
                const uint64_t ad = umma::smem_desc(a0 + k * 2048, kBoxBytes, 1024);
                const uint64_t bd = umma::smem_desc(b0 + k * 2048, 1024, 1024);
                umma::mma_bf16(tmem, ad, bd, kIdescDw, (i > 0 || k > 0) ? 1u : 0u);
            }
            umma::mma_commit(&empty[s]);
            if (i + 2 < mine) {
                if (!mbar_wait_bounded(&empty[s], euses[s] & 1)) { ok = false; break; }
                ++euses[s];
                load(i + 2);
            }
        }
        umma::mma_commit(done);
        if (!ok) {
            atomicOr(status, kDevErrTimeout);
            drain(&full[0], pend[0], fuses[0] & 1);
            drain(&full[1], pend[1], fuses[1] & 1);
        }
    }
    ok = mbar_wait_bounded(done, 0) && ok;
    ok = __syncthreads_and(ok);
    umma::fence_after_sync();
    __syncwarp();
    if (ok && mine > 0) {
        const uint32_t taddr = tmem + (uint32_t(warp * 32) << 16);
        float* dst = partial + (size_t(blockIdx.x) * 128 + tid) * 64;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float v[32];
            umma::tmem_ld32(taddr + h * 32, v);
            store_f32x32(dst + h * 32, v);
        }
    } else if (mine == 0) {
        float* dst = partial + (size_t(blockIdx.x) * 128 + tid) * 64;
        for (int c = 0; c < 64; ++c) dst[c] = 0.0f;
    }
    if (!ok && tid == 0) atomicOr(status, kDevErrTimeout);
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        umma::fence_after_sync();
        umma::tmem_dealloc(tmem, 64);
    }
}

// dW[g][f] = sum_b partial[b][f][g].  A block sums 32 consecutive elements,
// its 8 warps an eighth of the partials each (in order), then the eighths in
// order: bound by reading the partials (9.7 MB for 296 blocks) out of L2
// (one thread per element over all partials took 43 us on 16 windows).
__global__ void __launch_bounds__(256) dw_reduce_kernel(const float* __restrict__ partial, int blocks,
                                                        float* __restrict__ dw) {
    __shared__ float sums[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.x * 32 + lane;   // f * 64 + g
    float acc = 0.0f;
#pragma unroll 8
    for (int b = warp; b < blocks; b += 8) acc += __ldcg(partial + size_t(b) * (128 * 64) + t);
    sums[warp][lane] = acc;
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int w = 1; w < 8; ++w) acc += sums[w][lane];
        dw[(t & 63) * 128 + (t >> 6)] = acc;
    }
}

// ---------------------------------------------------------------------------
// CUDA-core kernels
// ---------------------------------------------------------------------------
constexpr int kF = kGnnFeat;

// One warp-wide load of 8 BF16 features per lane: 8 lanes hold a row of 64.
__device__ __forceinline__ uint4 ld_row8(const bf16* h, size_t row, int ld, int sub) {
    return *reinterpret_cast<const uint4*>(h + row * ld + 8 * sub);
}
__device__ __forceinline__ void unpack8(uint4 v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        f[2 * q] = __uint_as_float(w[q] << 16);
        f[2 * q + 1] = __uint_as_float(w[q] & 0xffff0000u);
    }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const __nv_bfloat162 p = __floats2bfloat162_rn(f[2 * q], f[2 * q + 1]);
        w[q] = *reinterpret_cast<const uint32_t*>(&p);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// h0[r][o] = bf16(relu(sum_f W[o][f] feat[r][f] + b[o])).  A lane keeps the
// weights of two outputs in registers and walks 32 nodes whose features its
// warp staged in shared memory: bound by instruction issue (28 per node and
// warp; a thread per output with the weights in shared memory took 70).
__global__ void __launch_bounds__(256) input_layer_kernel(const float* __restrict__ feat, int nodes,
                                                          const float* __restrict__ w, bf16* __restrict__ out, int ld) {
    constexpr int kPad = 12;   // floats per staged node: three 16-byte reads
    __shared__ __align__(16) float stage[8][32 * kPad];
    const int lane = threadIdx.x & 31;
    float* s = stage[threadIdx.x >> 5];
    float w0[kF], w1[kF];
#pragma unroll
    for (int q = 0; q < kF; ++q) {
        w0[q] = w[2 * lane * kF + q];
        w1[q] = w[(2 * lane + 1) * kF + q];
    }
    const float b0 = w[64 * kF + 2 * lane], b1 = w[64 * kF + 2 * lane + 1];
    const int warps = gridDim.x * 8;
    for (int base = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 32; base < nodes; base += warps * 32) {
        const int cnt = min(32, nodes - base);
        for (int t = lane; t < cnt * kF; t += 32) s[t / kF * kPad + t % kF] = feat[size_t(base) * kF + t];
        __syncwarp();
#pragma unroll 4
        for (int i = 0; i < cnt; ++i) {
            const float4* f4 = reinterpret_cast<const float4*>(s + i * kPad);
            const float4 fa = f4[0], fb = f4[1];
            const float f[kF] = {fa.x, fa.y, fa.z, fa.w, fb.x, fb.y, fb.z, fb.w, s[i * kPad + 8]};
            float a0 = 0.0f, a1 = 0.0f;
#pragma unroll
            for (int q = 0; q < kF; ++q) {
                a0 = fmaf(w0[q], f[q], a0);
                a1 = fmaf(w1[q], f[q], a1);
            }
            *reinterpret_cast<__nv_bfloat162*>(out + size_t(base + i) * ld + 2 * lane) =
                __floats2bfloat162_rn(fmaxf(a0 + b0, 0.0f), fmaxf(a1 + b1, 0.0f));
        }
        __syncwarp();
    }
}

// out[r][64:128] = bf16(sum_{e in row r} coef[e] h[col[e]][0:64]), entries in
// order.  8 lanes per row, 8 features each, so a warp works on four rows and
// an entry is one 16-byte load per lane; kEdges entries are in flight before
// the first is added.  Bound by those gathers' round trips: rows hold two to
// six entries.
template <int kEdges>
__global__ void __launch_bounds__(256) aggregate_kernel(const int* __restrict__ rp, const int* __restrict__ col,
                                                        const float* __restrict__ coef, const bf16* __restrict__ h,
                                                        int ldh, bf16* __restrict__ out, int ldo, int rows) {
    const int sub = threadIdx.x & 7;
    for (int r = (blockIdx.x * 256 + threadIdx.x) >> 3; r < rows; r += gridDim.x * 32) {
        const int beg = rp[r], end = rp[r + 1];
        float a[8] = {};
        for (int e = beg; e < end; e += kEdges) {
            int c[kEdges];
            float w[kEdges];
            uint4 v[kEdges];
#pragma unroll
            for (int u = 0; u < kEdges; ++u) {
                c[u] = e + u < end ? col[e + u] : 0;
                w[u] = e + u < end ? coef[e + u] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < kEdges; ++u) v[u] = e + u < end ? ld_row8(h, size_t(c[u]), ldh, sub) : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int u = 0; u < kEdges; ++u) {
                if (e + u < end) {
                    float f[8];
                    unpack8(v[u], f);
#pragma unroll
                    for (int q = 0; q < 8; ++q) a[q] = fmaf(w[u], f[q], a[q]);
                }
            }
        }
        *reinterpret_cast<uint4*>(out + size_t(r) * ldo + 64 + 8 * sub) = pack8(a);
    }
}

// One side's nodes cut into chunks of one LP each.
struct Chunks {
    const int* begin;      // [chunks + 1]
    const int* lp_first;   // [K + 1]
    int chunks;
};

// part[c][t] = sum of feature t of h over the nodes of chunk c, in node order:
// the variable side's chunks, then the constraint side's.  A warp per chunk, a
// lane two features, kPoolAhead rows in flight (one dependent add per row is
// the definition's order, so only the loads overlap).
constexpr int kPoolAhead = 32;
__global__ void __launch_bounds__(128) pool_kernel(const bf16* __restrict__ hv, Chunks cv, const bf16* __restrict__ hc,
                                                   Chunks cc, float* __restrict__ part) {
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < cv.chunks + cc.chunks; c += warps) {
        const bool v = c < cv.chunks;
        const int* begin = v ? cv.begin + c : cc.begin + (c - cv.chunks);
        const bf16* h = v ? hv : hc;
        const int b = begin[0], e = begin[1];
        float a0 = 0.0f, a1 = 0.0f;
        auto row = [&](int r) { return __ldg(reinterpret_cast<const uint32_t*>(h + size_t(r) * 64 + 2 * lane)); };
        auto add = [&](uint32_t x) {
            a0 += __uint_as_float(x << 16);
            a1 += __uint_as_float(x & 0xffff0000u);
        };
        int r = b;
        for (; r + kPoolAhead <= e; r += kPoolAhead) {
            uint32_t x[kPoolAhead];
#pragma unroll
            for (int u = 0; u < kPoolAhead; ++u) x[u] = row(r + u);
#pragma unroll
            for (int u = 0; u < kPoolAhead; ++u) add(x[u]);
        }
#pragma unroll 4
        for (; r < e; ++r) add(row(r));
        *reinterpret_cast<float2*>(part + size_t(c) * 64 + 2 * lane) = make_float2(a0, a1);
    }
}

// Sum of src[c * stride] for c in [b, e), in order, 32 loads in flight.
__device__ __forceinline__ float ordered_sum(const float* __restrict__ src, int b, int e, int stride) {
    float acc = 0.0f;
    int c = b;
    for (; c + 32 <= e; c += 32) {
        float v[32];
#pragma unroll
        for (int u = 0; u < 32; ++u) v[u] = src[size_t(c + u) * stride];
#pragma unroll
        for (int u = 0; u < 32; ++u) acc += v[u];
    }
#pragma unroll 8
    for (; c < e; ++c) acc += src[size_t(c) * stride];
    return acc;
}

// Per LP (a block): pooled means of both sides from the chunk sums, chunks in
// order, and rho_k = w_w . pooled_k + b_w (128 weights, then the bias).
__global__ void __launch_bounds__(128) pooled_rho_kernel(const float* __restrict__ part, Chunks cv, Chunks cc,
                                                         const float* __restrict__ inv_n,
                                                         const float* __restrict__ inv_m,
                                                         const float* __restrict__ wb, int K,
                                                         float* __restrict__ pooled, float* __restrict__ rho) {
    __shared__ float mean[128];
    const int t = threadIdx.x, lane = t & 31;
    for (int k = blockIdx.x; k < K; k += gridDim.x) {
        const bool v = t < 64;
        const int* first = v ? cv.lp_first + k : cc.lp_first + k;
        const float* src = part + (v ? size_t(t) : size_t(cv.chunks) * 64 + size_t(t - 64));
        const float p = ordered_sum(src, first[0], first[1], 64) * (v ? inv_n[k] : inv_m[k]);
        mean[t] = p;
        pooled[size_t(k) * 128 + t] = p;
        __syncthreads();
        if (t < 32) {
            float d = 0.0f;
#pragma unroll
            for (int q = 0; q < 4; ++q) d = fmaf(wb[4 * lane + q], mean[4 * lane + q], d);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
            if (lane == 0) rho[k] = d + wb[128];
        }
        __syncthreads();
    }
}

// One side of a loss or head gradient: predictions, targets, the LP of every
// node and the LP's loss weight.
struct HeadSide {
    const float* hat;
    const float* tgt;
    const int* lp;
    const float* lw;
};

// part[c] = sum over the nodes of chunk c of (hat - target)^2 lw, in node
// order (variable side, then constraint side): a warp loads 32 terms at a
// time and every lane adds them in order.
__global__ void __launch_bounds__(128) square_error_kernel(HeadSide sv, Chunks cv, HeadSide sc, Chunks cc,
                                                           float* __restrict__ part) {
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < cv.chunks + cc.chunks; c += warps) {
        const bool v = c < cv.chunks;
        const int* begin = v ? cv.begin + c : cc.begin + (c - cv.chunks);
        const HeadSide s = v ? sv : sc;
        const int b = begin[0], e = begin[1];
        static_assert(kGnnChunk % 32 == 0, "chunks are whole warps but for an LP's last");
        float sq[kGnnChunk / 32], lw[kGnnChunk / 32];
#pragma unroll
        for (int u = 0; u < kGnnChunk / 32; ++u) {
            const int r = b + u * 32 + lane;
            const float d = r < e ? s.hat[r] - s.tgt[r] : 0.0f;
            sq[u] = __fmul_rn(d, d);
            lw[u] = r < e ? s.lw[s.lp[r]] : 0.0f;
        }
        float acc = 0.0f;
#pragma unroll
        for (int u = 0; u < kGnnChunk / 32; ++u) {
            const int cnt = min(32, e - b - u * 32);
            for (int t = 0; t < cnt; ++t)
                acc = fmaf(__shfl_sync(0xffffffffu, sq[u], t), __shfl_sync(0xffffffffu, lw[u], t), acc);
        }
        if (lane == 0) part[c] = acc;
    }
}

// One block: each LP's x and y terms from the chunk sums (chunks in order),
// the loss (LPs in order, FP64) and drho_k = 2 (rho_k - tw_k) / K; with
// `grad` the gradient of the primal-weight head, sum_k drho_k [pooled_k ; 1].
__global__ void __launch_bounds__(256) loss_kernel(const float* __restrict__ part, Chunks cv, Chunks cc,
                                                   const float* __restrict__ rho, const float* __restrict__ tw, int K,
                                                   float inv_k, const float* __restrict__ pooled,
                                                   float* __restrict__ sums, float* __restrict__ drho,
                                                   float* __restrict__ grad, double* __restrict__ loss) {
    for (int t = threadIdx.x; t < 2 * K; t += blockDim.x) {
        const bool v = t < K;
        const int* first = v ? cv.lp_first + t : cc.lp_first + (t - K);
        sums[t] = ordered_sum(part + (v ? 0 : cv.chunks), first[0], first[1], 1);
    }
    for (int k = threadIdx.x; k < K; k += blockDim.x)
        drho[k] = __fmul_rn(float(2.0 * (double(rho[k]) - double(tw[k]))), inv_k);
    __syncthreads();
    if (threadIdx.x == 0) {
        double total = 0.0;
        for (int k = 0; k < K; ++k) {
            const double dw = double(rho[k]) - double(tw[k]);
            total = __dadd_rn(total, __dadd_rn(__dadd_rn(double(sums[k]), double(sums[K + k])), __dmul_rn(dw, dw)));
        }
        *loss = total / K;
    }
    if (!grad) return;
    for (int t = threadIdx.x; t < 129; t += blockDim.x) {
        float acc = 0.0f;
        for (int k = 0; k < K; ++k) acc += t < 128 ? drho[k] * pooled[size_t(k) * 128 + t] : drho[k];
        grad[t] = acc;
    }
}

// ---- gradient partials ------------------------------------------------------
// Every block of the node kernels below writes one row of gpart_; the columns:
constexpr int kColBias = 0;                              // dense layers' biases, (2 l + side) * 64
constexpr int kColHead = kColBias + 2 * kGnnLayers * 64; // w_x, b_x, then w_y, b_y
constexpr int kColIn = kColHead + 2 * 65;                // W_vin, b_vin, then W_cin, b_cin
constexpr int kInWide = 64 * kF + 64;
constexpr int kGradCols = kColIn + 2 * kInWide;

// Adds each thread's N partial vectors of 8 features (features 8 (tid & 7) ...)
// over the block into row[n * stride + feature], groups in a fixed order.
template <int N>
__device__ __forceinline__ void block_feature_sums(float (&acc)[N][8], float* __restrict__ row, const int (&at)[N]) {
    __shared__ float sums[8][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int n = 0; n < N; ++n) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            acc[n][q] += __shfl_xor_sync(0xffffffffu, acc[n][q], 8);
            acc[n][q] += __shfl_xor_sync(0xffffffffu, acc[n][q], 16);
        }
        __syncthreads();
        if (lane < 8) {
#pragma unroll
            for (int q = 0; q < 8; ++q) sums[warp][8 * lane + q] = acc[n][q];
        }
        __syncthreads();
        if (threadIdx.x < 64) {
            float t = 0.0f;
#pragma unroll
            for (int w = 0; w < 8; ++w) t += sums[w][threadIdx.x];
            row[at[n] + threadIdx.x] = t;
        }
    }
}

struct NodeBackward {
    int rows;
    // dh_r += sum_{e in row r} coef[e] dagg[col[e]]; rp null: no such terms
    const int* rp;
    const int* col;
    const float* coef;
    const float* dagg;
    float* dh;               // kHead: not read; kFinal: written
    const bf16* h;           // the layer's output rows
    int ldh;
    bf16* dz;                // !kFinal: bf16(h > 0 ? dh : 0)
    float* part;             // gpart_
    int col_bias, col_head;  // columns of the bias and head gradients
    // kHead: dh from the node head and the pooled primal-weight head
    HeadSide side;
    float inv_k;
    const float* w;          // head weights [64]
    const float* ww;         // this side's half of the primal-weight head [64]
    const float* drho;
    const float* inv;        // 1 / nodes of the LP
};

// One pass over a side's nodes on the way back: the gradient dh of every
// hidden row (the dense layer's own part, or the heads' with kHead, plus the
// other side's aggregation terms, entries in order), masked by the ReLU into
// the BF16 dz the dense gradients read, with the bias and head gradients
// summed on the way.  dh never returns to memory except for the input layer
// (kFinal).  8 lanes per row, 8 features each; bound by the FP32 rows it reads
// (256 bytes per node and per entry).
constexpr int kBackEdges = 4;
template <bool kHead, bool kFinal>
__global__ void __launch_bounds__(256) node_backward_kernel(const NodeBackward a) {
    const int sub = threadIdx.x & 7;
    float sums[kHead ? 2 : 1][8] = {};   // bias; head weights
    float dsum = 0.0f;
    float w[8], ww[8];
    if constexpr (kHead) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            w[q] = a.w[8 * sub + q];
            ww[q] = a.ww[8 * sub + q];
        }
    }
    for (int r = (blockIdx.x * 256 + threadIdx.x) >> 3; r < a.rows; r += gridDim.x * 32) {
        const int beg = a.rp ? a.rp[r] : 0, end = a.rp ? a.rp[r + 1] : 0;
        float dh[8], h[8];
        uint4 hv = make_uint4(0, 0, 0, 0);
        if constexpr (!kFinal) hv = ld_row8(a.h, size_t(r), a.ldh, sub);
        float d = 0.0f;
        if constexpr (kHead) {
            const int k = a.side.lp[r];
            d = 2.0f * (a.side.hat[r] - a.side.tgt[r]) * a.side.lw[k] * a.inv_k;
            const float dr = a.drho[k], iv = a.inv[k];
#pragma unroll
            for (int q = 0; q < 8; ++q) dh[q] = fmaf(d, w[q], dr * ww[q] * iv);
        } else {
            const float4* p = reinterpret_cast<const float4*>(a.dh + size_t(r) * 64 + 8 * sub);
            const float4 x = p[0], y = p[1];
            dh[0] = x.x; dh[1] = x.y; dh[2] = x.z; dh[3] = x.w;
            dh[4] = y.x; dh[5] = y.y; dh[6] = y.z; dh[7] = y.w;
        }
        float g[8] = {};
        for (int e = beg; e < end; e += kBackEdges) {
            int c[kBackEdges];
            float f[kBackEdges];
            float4 x[kBackEdges], y[kBackEdges];
#pragma unroll
            for (int u = 0; u < kBackEdges; ++u) {
                c[u] = e + u < end ? a.col[e + u] : 0;
                f[u] = e + u < end ? a.coef[e + u] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < kBackEdges; ++u) {
                const float4* p = reinterpret_cast<const float4*>(a.dagg + size_t(c[u]) * 64 + 8 * sub);
                x[u] = e + u < end ? p[0] : make_float4(0.f, 0.f, 0.f, 0.f);
                y[u] = e + u < end ? p[1] : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < kBackEdges; ++u) {
                if (e + u < end) {
                    g[0] = fmaf(f[u], x[u].x, g[0]); g[1] = fmaf(f[u], x[u].y, g[1]);
                    g[2] = fmaf(f[u], x[u].z, g[2]); g[3] = fmaf(f[u], x[u].w, g[3]);
                    g[4] = fmaf(f[u], y[u].x, g[4]); g[5] = fmaf(f[u], y[u].y, g[5]);
                    g[6] = fmaf(f[u], y[u].z, g[6]); g[7] = fmaf(f[u], y[u].w, g[7]);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) dh[q] += g[q];
        if constexpr (kFinal) {
            float4* p = reinterpret_cast<float4*>(a.dh + size_t(r) * 64 + 8 * sub);
            p[0] = make_float4(dh[0], dh[1], dh[2], dh[3]);
            p[1] = make_float4(dh[4], dh[5], dh[6], dh[7]);
        } else {
            unpack8(hv, h);
            float z[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) z[q] = h[q] > 0.0f ? dh[q] : 0.0f;
            const uint4 packed = pack8(z);
            *reinterpret_cast<uint4*>(a.dz + size_t(r) * 64 + 8 * sub) = packed;
            unpack8(packed, z);
#pragma unroll
            for (int q = 0; q < 8; ++q) sums[0][q] += z[q];
            if constexpr (kHead) {
#pragma unroll
                for (int q = 0; q < 8; ++q) sums[1][q] = fmaf(d, h[q], sums[1][q]);
                dsum += d;   // the same value in the 8 lanes of a row
            }
        }
    }
    if constexpr (!kFinal) {
        float* row = a.part + size_t(blockIdx.x) * kGradCols;
        if constexpr (kHead) {
            const int at[2] = {a.col_bias, a.col_head};
            block_feature_sums<2>(sums, row, at);
            __shared__ float ds[8];
            dsum += __shfl_xor_sync(0xffffffffu, dsum, 8);
            dsum += __shfl_xor_sync(0xffffffffu, dsum, 16);
            if ((threadIdx.x & 31) == 0) ds[threadIdx.x >> 5] = dsum;
            __syncthreads();
            if (threadIdx.x == 0) {
                float t = 0.0f;
#pragma unroll
                for (int q = 0; q < 8; ++q) t += ds[q];
                row[a.col_head + 64] = t;
            }
        } else {
            const int at[1] = {a.col_bias};
            block_feature_sums<1>(sums, row, at);
        }
    }
}

// Input-layer gradient: row[o*9 + q] = sum_r dz0[r][o] f[r][q], row[576 + o] =
// sum_r dz0[r][o] over the block's nodes, dz0 = dh masked by h0 > 0 (FP32).
// Four threads share an output feature o and take every fourth node; bound by
// the rows read (420 bytes per node).
constexpr int kInTile = 64;   // nodes whose features are staged at a time
__global__ void __launch_bounds__(256) inlayer_grad_kernel(const float* __restrict__ dh, const bf16* __restrict__ h0,
                                                           int ldh0, const float* __restrict__ feat, int nodes,
                                                           float* __restrict__ part, int col) {
    __shared__ float f[kInTile * kF];
    __shared__ float sums[4][64];
    const int o = threadIdx.x & 63, g = threadIdx.x >> 6;
    float acc[kF + 1] = {};
    for (int base = blockIdx.x * kInTile; base < nodes; base += gridDim.x * kInTile) {
        const int cnt = min(kInTile, nodes - base);
        __syncthreads();
        for (int t = threadIdx.x; t < cnt * kF; t += 256) f[t] = feat[size_t(base) * kF + t];
        float z[kInTile / 4];
#pragma unroll
        for (int u = 0; u < kInTile / 4; ++u) {
            const int i = min(4 * u + g, cnt - 1);   // past the end: the last node, not added
            const size_t r = size_t(base + i);
            const float hv = bf(h0[r * ldh0 + o]), d = dh[r * 64 + o];
            z[u] = hv > 0.0f ? d : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kInTile / 4; ++u) {
            const int i = 4 * u + g;
            if (i < cnt) {
#pragma unroll
                for (int q = 0; q < kF; ++q) acc[q] = fmaf(z[u], f[i * kF + q], acc[q]);
                acc[kF] += z[u];
            }
        }
    }
    float* row = part + size_t(blockIdx.x) * kGradCols + col;
#pragma unroll
    for (int q = 0; q <= kF; ++q) {
        __syncthreads();
        sums[g][o] = acc[q];
        __syncthreads();
        if (g == 0) row[q < kF ? o * kF + q : 64 * kF + o] = ((sums[0][o] + sums[1][o]) + sums[2][o]) + sums[3][o];
    }
}

// Place of gradient column c in the parameter vector; -1: a constraint-side
// column of a graph without constraints.
__device__ __forceinline__ int grad_place(int c, bool has_c) {
    if (c < kColHead) {
        const int d = c / 64;
        return (d & 1) == 0 && !has_c ? -1 : GnnParams::layer_b(d >> 1, d & 1) + c % 64;
    }
    if (c < kColIn) {
        const int t = c - kColHead;
        return t < 65 ? GnnParams::kHeadX + t : has_c ? GnnParams::kHeadY + (t - 65) : -1;
    }
    const int t = c - kColIn;
    return t < kInWide ? GnnParams::kVinW + t : has_c ? GnnParams::kCinW + (t - kInWide) : -1;
}
static_assert(GnnParams::kVinB == GnnParams::kVinW + 64 * kF && GnnParams::kCinB == GnnParams::kCinW + 64 * kF,
              "an input layer's bias follows its weights");

// The blocks' rows of gpart_ added per column: 8 warps an eighth of the rows
// each, then the eighths, in order.
__global__ void __launch_bounds__(256) grad_total_kernel(const float* __restrict__ part, int rows, bool has_c,
                                                         float* __restrict__ grad) {
    __shared__ float sums[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + lane;
    const int place = c < kGradCols ? grad_place(c, has_c) : -1;
    float acc = 0.0f;
    if (place >= 0) {
#pragma unroll 8
        for (int b = warp; b < rows; b += 8) acc += __ldcg(part + size_t(b) * kGradCols + c);
    }
    sums[warp][lane] = acc;
    __syncthreads();
    if (warp == 0 && place >= 0) {
#pragma unroll
        for (int w = 1; w < 8; ++w) acc += sums[w][lane];
        grad[place] = acc;
    }
}

__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, int n, float lr, float c1, float c2) {
    constexpr float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    GNN_STRIDE(i, n) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
    }
}

// pr = bf16-rounded parameters; w / wt = the dense layers' W and W^T in BF16.
__global__ void refresh_kernel(const float* __restrict__ p, int n, float* __restrict__ pr, bf16* __restrict__ w,
                               bf16* __restrict__ wt) {
    GNN_STRIDE(i, n) pr[i] = bfr(p[i]);
    GNN_STRIDE(t, 2LL * kGnnLayers * 64 * 128) {
        const int d = int(t / (64 * 128)), e = int(t % (64 * 128));
        const int l = d >> 1, side = d & 1;
        const int g = e / 128, f = e % 128;
        const bf16 v = __float2bfloat16_rn(p[GnnParams::layer_w(l, side) + e]);
        w[t] = v;
        wt[size_t(d) * 64 * 128 + size_t(f) * 64 + g] = v;
    }
}

// splitmix64 uniform in [-a, a)
uint64_t splitmix(uint64_t& s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
float uniform(uint64_t& s, float a) {
    const double u = double(splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
    return float((2.0 * u - 1.0) * a);
}

// Blocks of the node kernels that leave one row of gradient partials each.
int grad_blocks(int dev) { return 4 * device_sm_count(dev); }

int dense_blocks(int dev, int rows, int per_sm) {
    const int tiles = (rows + kRowsPerTile - 1) / kRowsPerTile;
    return std::max(1, std::min(tiles, per_sm * device_sm_count(dev)));
}

void set_smem_attrs_once() {
    static std::once_flag once;
    std::call_once(once, [] {
        PB_CUDA_CHECK(cudaFuncSetAttribute(dense_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           int(FwdSmem::kBytes)));
        PB_CUDA_CHECK(cudaFuncSetAttribute(dense_dx_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           int(DxSmem::kBytes)));
        PB_CUDA_CHECK(cudaFuncSetAttribute(dense_dw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           int(DwSmem::kBytes)));
    });
}

}  // namespace

// ---------------------------------------------------------------------------
// GnnGraph
// ---------------------------------------------------------------------------
GnnGraph::GnnGraph(const pramaan_lp* lps, int count_, const pramaan_warm_start* hints,
                   const pramaan_warm_start* targets, int dev) {
    device = dev;
    count = count_;
    has_targets = targets != nullptr;
    long long M = 0, N = 0, NZ = 0;
    for (int k = 0; k < count; ++k) {
        const pramaan_lp& lp = lps[k];
        if (lp.num_rows < 0 || lp.num_cols < 0 || lp.nnz < 0) throw InvalidArgument("gnn graph: negative size");
        if (lp.num_cols == 0) continue;
        index.push_back(k);
        r0.push_back(int(M));
        c0.push_back(int(N));
        M += lp.num_rows;
        N += lp.num_cols;
        NZ += lp.nnz;
        if (M > INT_MAX / 2 || N > INT_MAX / 2 || NZ > INT_MAX / 2)
            throw InvalidArgument("gnn graph: the packed batch exceeds 2^30 rows, columns or non-zeros");
    }
    K = int(index.size());
    m = int(M);
    n = int(N);
    nnz = int(NZ);
    r0.push_back(m);
    c0.push_back(n);
    PB_CUDA_CHECK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    if (K == 0) return;

    const size_t Mz = static_cast<size_t>(m), Nz = static_cast<size_t>(n), Ez = static_cast<size_t>(nnz);
    std::vector<int> hrp(Mz + 1, 0), hci(Ez), hlpr(Mz), hlpc(Nz);
    std::vector<double> hval(Ez), hvlo(Nz), hvhi(Nz), hcost(Nz), hrlo(Mz), hrhi(Mz);
    s_a.assign(size_t(K), 1.0);
    s_b.assign(size_t(K), 1.0);
    s_c.assign(size_t(K), 1.0);
    omega_ref.assign(size_t(K), 1.0);
    long long e0 = 0;
    for (int q = 0; q < K; ++q) {
        const pramaan_lp& lp = lps[index[size_t(q)]];
        if (lp.num_rows > 0 && !lp.row_ptr) throw InvalidArgument("gnn graph: row_ptr is NULL");
        if (lp.nnz > 0 && (!lp.col_idx || !lp.values)) throw InvalidArgument("gnn graph: col_idx/values is NULL");
        if (!lp.obj_coeffs || !lp.var_lower || !lp.var_upper) throw InvalidArgument("gnn graph: column data is NULL");
        if (lp.num_rows > 0 && (!lp.row_lower || !lp.row_upper)) throw InvalidArgument("gnn graph: row bounds are NULL");
        if (lp.num_rows > 0 && (lp.row_ptr[0] != 0 || lp.row_ptr[lp.num_rows] != lp.nnz))
            throw InvalidArgument("pramaan_lp: row_ptr must start at 0, be non-decreasing and end at nnz");
        const double sign = lp.obj_sense == PRAMAAN_MAXIMIZE ? -1.0 : 1.0;
        const int R = r0[size_t(q)], C = c0[size_t(q)];
        double a2 = 0.0, b2 = 0.0, c2 = 0.0;
        long long bc = 0;
        for (int i = 0; i < lp.num_rows; ++i) {
            if (lp.row_ptr[i + 1] < lp.row_ptr[i]) throw InvalidArgument("pramaan_lp: row_ptr must be non-decreasing");
            hrp[size_t(R + i)] = int(e0 + lp.row_ptr[i]);
            hlpr[size_t(R + i)] = q;
            const double lo = lp.row_lower[i], hi = lp.row_upper[i];
            hrlo[size_t(R + i)] = lo;
            hrhi[size_t(R + i)] = hi;
            if (lo > -1e29) { b2 += lo * lo; ++bc; }
            if (hi < 1e29 && !(lo > -1e29 && lo == hi)) { b2 += hi * hi; ++bc; }
        }
        for (int e = 0; e < lp.nnz; ++e) {
            const int j = lp.col_idx[e];
            if (j < 0 || j >= lp.num_cols) throw InvalidArgument("pramaan_lp: col_idx entry out of bounds");
            hci[size_t(e0 + e)] = C + j;
            hval[size_t(e0 + e)] = lp.values[e];
            a2 += lp.values[e] * lp.values[e];
        }
        for (int j = 0; j < lp.num_cols; ++j) {
            const double cj = sign * lp.obj_coeffs[j];
            hcost[size_t(C + j)] = cj;
            c2 += cj * cj;
            hvlo[size_t(C + j)] = lp.var_lower[j];
            hvhi[size_t(C + j)] = lp.var_upper[j];
            hlpc[size_t(C + j)] = q;
        }
        e0 += lp.nnz;
        const double sa = lp.nnz > 0 ? std::sqrt(a2 / lp.nnz) : 0.0;
        const double sb = bc > 0 ? std::sqrt(b2 / double(bc)) : 0.0;
        const double sc = std::sqrt(c2 / lp.num_cols);
        s_a[size_t(q)] = sa > 0.0 && std::isfinite(sa) ? sa : 1.0;
        s_b[size_t(q)] = sb > 0.0 && std::isfinite(sb) ? sb : 1.0;
        s_c[size_t(q)] = sc > 0.0 && std::isfinite(sc) ? sc : 1.0;
        const double cn = std::sqrt(c2), bn = std::sqrt(b2);
        omega_ref[size_t(q)] = cn > 1e-10 && bn > 1e-10 && std::isfinite(cn / bn) ? cn / bn : 1.0;
    }
    hrp[size_t(m)] = int(e0);

    // transpose (counting sort by column; rows of A^T list A's rows in order)
    std::vector<int> deg_c(Nz, 0), htp(Nz + 1, 0), hti(Ez), perm(Ez);
    for (int e = 0; e < nnz; ++e) ++deg_c[size_t(hci[size_t(e)])];
    for (int j = 0; j < n; ++j) htp[size_t(j) + 1] = htp[size_t(j)] + deg_c[size_t(j)];
    {
        std::vector<int> pos(htp.begin(), htp.end() - 1);
        for (int i = 0; i < m; ++i)
            for (int e = hrp[size_t(i)]; e < hrp[size_t(i) + 1]; ++e) {
                const int p = pos[size_t(hci[size_t(e)])]++;
                hti[size_t(p)] = i;
                perm[size_t(p)] = e;
            }
    }
    std::vector<float> hcr(Ez), hcc(Ez), htr(Ez), htc(Ez);
    for (int i = 0; i < m; ++i) {
        const int q = hlpr[size_t(i)];
        const int deg = hrp[size_t(i) + 1] - hrp[size_t(i)];
        for (int e = hrp[size_t(i)]; e < hrp[size_t(i) + 1]; ++e) {
            const int j = hci[size_t(e)];
            hcr[size_t(e)] = float(hval[size_t(e)] / (s_a[size_t(q)] * std::max(1, deg)));
            hcc[size_t(e)] = float(hval[size_t(e)] / (s_a[size_t(q)] * std::max(1, deg_c[size_t(j)])));
        }
    }
    for (int p = 0; p < nnz; ++p) {
        htr[size_t(p)] = hcr[size_t(perm[size_t(p)])];
        htc[size_t(p)] = hcc[size_t(perm[size_t(p)])];
    }

    // features (FP64 arithmetic, stored as FP32)
    auto clip = [](double v) { return std::min(10.0, std::max(-10.0, v)); };
    std::vector<float> hfv(Nz * kF), hfc(Mz * kF), hbx(Nz, 0.0f), hby(Mz, 0.0f);
    std::vector<char> hint_x(Nz, 0), hint_y(Mz, 0);
    if (hints) {
        for (int q = 0; q < K; ++q) {
            const pramaan_warm_start& h = hints[index[size_t(q)]];
            const int C = c0[size_t(q)], R = r0[size_t(q)];
            const int nk = c0[size_t(q) + 1] - C, mk = r0[size_t(q) + 1] - R;
            const double sa = s_a[size_t(q)], sb = s_b[size_t(q)], sc = s_c[size_t(q)];
            if (h.x)
                for (int j = 0; j < nk; ++j) {
                    if (!std::isfinite(h.x[j])) throw InvalidArgument("gnn graph: hint x must be finite");
                    hbx[size_t(C + j)] = float(h.x[j] * sa / sb);
                    hint_x[size_t(C + j)] = 1;
                }
            if (h.y)
                for (int i = 0; i < mk; ++i) {
                    if (!std::isfinite(h.y[i])) throw InvalidArgument("gnn graph: hint y must be finite");
                    hby[size_t(R + i)] = float(h.y[i] * sa / sc);
                    hint_y[size_t(R + i)] = 1;
                }
        }
    }
    for (int j = 0; j < n; ++j) {
        const int q = hlpc[size_t(j)];
        const double sa = s_a[size_t(q)], sb = s_b[size_t(q)], sc = s_c[size_t(q)];
        const double lo = hvlo[size_t(j)], hi = hvhi[size_t(j)];
        const bool fl = lo > -1e29, fu = hi < 1e29;
        double absum = 0.0;
        for (int p = htp[size_t(j)]; p < htp[size_t(j) + 1]; ++p) absum += std::fabs(hval[size_t(perm[size_t(p)])]);
        const int deg = deg_c[size_t(j)];
        float* f = &hfv[size_t(j) * kF];
        f[0] = float(hcost[size_t(j)] / sc);
        f[1] = fl ? 1.0f : 0.0f;
        f[2] = fu ? 1.0f : 0.0f;
        f[3] = fl ? float(clip(lo * sa / sb)) : 0.0f;
        f[4] = fu ? float(clip(hi * sa / sb)) : 0.0f;
        f[5] = float(std::log1p(double(deg)) / 4.0);
        f[6] = deg > 0 ? float(absum / (sa * deg)) : 0.0f;
        f[7] = hint_x[size_t(j)] ? 1.0f : 0.0f;
        f[8] = float(clip(double(hbx[size_t(j)])));
    }
    for (int i = 0; i < m; ++i) {
        const int q = hlpr[size_t(i)];
        const double sa = s_a[size_t(q)], sb = s_b[size_t(q)];
        const double lo = hrlo[size_t(i)], hi = hrhi[size_t(i)];
        const bool fl = lo > -1e29, fu = hi < 1e29;
        double absum = 0.0;
        for (int e = hrp[size_t(i)]; e < hrp[size_t(i) + 1]; ++e) absum += std::fabs(hval[size_t(e)]);
        const int deg = hrp[size_t(i) + 1] - hrp[size_t(i)];
        float* f = &hfc[size_t(i) * kF];
        f[0] = fl && fu && lo == hi ? 1.0f : 0.0f;
        f[1] = fl ? 1.0f : 0.0f;
        f[2] = fu ? 1.0f : 0.0f;
        f[3] = fl ? float(clip(lo / sb)) : 0.0f;
        f[4] = fu ? float(clip(hi / sb)) : 0.0f;
        f[5] = float(std::log1p(double(deg)) / 4.0);
        f[6] = deg > 0 ? float(absum / (sa * deg)) : 0.0f;
        f[7] = hint_y[size_t(i)] ? 1.0f : 0.0f;
        f[8] = float(clip(double(hby[size_t(i)])));
    }

    // chunk tables
    const size_t Kz = static_cast<size_t>(K);
    std::vector<int> cb, rb, clp, rlp, cfirst(Kz + 1), rfirst(Kz + 1);
    std::vector<float> hinv_n(Kz), hinv_m(Kz), hscale(Kz * 4);
    for (int q = 0; q < K; ++q) {
        cfirst[size_t(q)] = int(cb.size());
        for (int b = c0[size_t(q)]; b < c0[size_t(q) + 1]; b += kGnnChunk) { cb.push_back(b); clp.push_back(q); }
        rfirst[size_t(q)] = int(rb.size());
        for (int b = r0[size_t(q)]; b < r0[size_t(q) + 1]; b += kGnnChunk) { rb.push_back(b); rlp.push_back(q); }
        const int nk = c0[size_t(q) + 1] - c0[size_t(q)], mk = r0[size_t(q) + 1] - r0[size_t(q)];
        hinv_n[size_t(q)] = 1.0f / float(nk);
        hinv_m[size_t(q)] = mk > 0 ? 1.0f / float(mk) : 0.0f;
        hscale[size_t(q) * 4 + 0] = float(s_a[size_t(q)]);
        hscale[size_t(q) * 4 + 1] = float(s_b[size_t(q)]);
        hscale[size_t(q) * 4 + 2] = float(s_c[size_t(q)]);
        hscale[size_t(q) * 4 + 3] = 1.0f / float(K);
    }
    cfirst[size_t(K)] = int(cb.size());
    rfirst[size_t(K)] = int(rb.size());
    cchunks = int(cb.size());
    rchunks = int(rb.size());
    cb.push_back(n);
    rb.push_back(m);

    auto up = [&](auto& d, const auto& h) {
        d.alloc(h.size());
        if (!h.empty())
            PB_CUDA_CHECK(cudaMemcpyAsync(d.get(), h.data(), h.size() * sizeof(h[0]), cudaMemcpyHostToDevice, st));
    };
    up(rp, hrp); up(ci, hci); up(tp, htp); up(ti, hti);
    up(coef_r, hcr); up(coef_c, hcc); up(tcoef_r, htr); up(tcoef_c, htc);
    up(fv, hfv); up(fc, hfc); up(base_x, hbx); up(base_y, hby); up(lp_col, hlpc); up(lp_row, hlpr); up(lp_scale, hscale);
    up(vlo, hvlo); up(vhi, hvhi);
    up(cchunk_begin, cb); up(rchunk_begin, rb); up(cchunk_lp, clp); up(rchunk_lp, rlp);
    up(clp_first, cfirst); up(rlp_first, rfirst); up(inv_n, hinv_n); up(inv_m, hinv_m);
    h_vlo = std::move(hvlo);
    h_vhi = std::move(hvhi);

    if (has_targets) {
        std::vector<float> htx(Nz), hty(Mz), htw(Kz), hlx(Kz), hly(Kz);
        for (int q = 0; q < K; ++q) {
            const pramaan_warm_start& t = targets[index[size_t(q)]];
            const int nk = c0[size_t(q) + 1] - c0[size_t(q)], mk = r0[size_t(q) + 1] - r0[size_t(q)];
            if (!t.x || (mk > 0 && !t.y)) throw InvalidArgument("gnn graph: every target needs x (and y when m > 0)");
            if (!(t.primal_weight > 0.0) || !std::isfinite(t.primal_weight))
                throw InvalidArgument("gnn graph: target primal weights must be positive and finite");
            const double sa = s_a[size_t(q)], sb = s_b[size_t(q)], sc = s_c[size_t(q)];
            for (int j = 0; j < nk; ++j) htx[size_t(c0[size_t(q)] + j)] = float(t.x[j] * sa / sb);
            for (int i = 0; i < mk; ++i) hty[size_t(r0[size_t(q)] + i)] = float(t.y[i] * sa / sc);
            htw[size_t(q)] = float(std::log(t.primal_weight / omega_ref[size_t(q)]));
            // per-LP loss weights: squared errors relative to the mean square of the targets
            double sx = 0.0, sy = 0.0;
            for (int j = 0; j < nk; ++j) sx += double(htx[size_t(c0[size_t(q)] + j)]) * htx[size_t(c0[size_t(q)] + j)];
            for (int i = 0; i < mk; ++i) sy += double(hty[size_t(r0[size_t(q)] + i)]) * hty[size_t(r0[size_t(q)] + i)];
            hlx[size_t(q)] = float(1.0 / (nk * (sx / nk + kLossFloor)));
            hly[size_t(q)] = mk > 0 ? float(1.0 / (mk * (sy / mk + kLossFloor))) : 0.0f;
        }
        up(tx, htx); up(ty, hty); up(tw, htw); up(lw_x, hlx); up(lw_y, hly);
    }
    PB_CUDA_CHECK(cudaStreamSynchronize(st));
}

GnnGraph::~GnnGraph() {
    if (st) {
        cudaStreamSynchronize(st);
        cudaStreamDestroy(st);
    }
}

// ---------------------------------------------------------------------------
// GnnModel
// ---------------------------------------------------------------------------
GnnModel::GnnModel(int device, uint64_t seed) : dev_(device) {
    PB_CUDA_CHECK(cudaStreamCreateWithFlags(&st_, cudaStreamNonBlocking));
    set_smem_attrs_once();
    const int np = GnnParams::kCount;
    p_.alloc(np); g_.alloc(np); am_.alloc(np); av_.alloc(np); pr_.alloc(np);
    w_.alloc(size_t(2 * kGnnLayers) * 64 * 128);
    wt_.alloc(size_t(2 * kGnnLayers) * 64 * 128);
    status_.alloc(1);
    // He-uniform weights (fan-in), zero biases and heads
    std::vector<float> h(size_t(np), 0.0f);
    uint64_t s = seed;
    auto fill = [&](int off, int count_, int fan_in) {
        const float a = std::sqrt(6.0f / float(fan_in));
        for (int i = 0; i < count_; ++i) h[size_t(off + i)] = uniform(s, a);
    };
    fill(GnnParams::kVinW, 64 * kGnnFeat, kGnnFeat);
    fill(GnnParams::kCinW, 64 * kGnnFeat, kGnnFeat);
    for (int l = 0; l < kGnnLayers; ++l)
        for (int side = 0; side < 2; ++side) fill(GnnParams::layer_w(l, side), 64 * 128, 128);
    // the heads start at zero: an untrained network returns the hint (or 0)
    // and omega_ref, and learns a correction from there
    set_params(h.data());
}

GnnModel::~GnnModel() {
    if (st_) {
        cudaStreamSynchronize(st_);
        cudaStreamDestroy(st_);
    }
}

void GnnModel::get_params(float* host) const {
    PB_CUDA_CHECK(cudaMemcpyAsync(host, p_.get(), p_.bytes(), cudaMemcpyDeviceToHost, st_));
    PB_CUDA_CHECK(cudaStreamSynchronize(st_));
}

void GnnModel::set_params(const float* host) {
    PB_CUDA_CHECK(cudaMemcpyAsync(p_.get(), host, p_.bytes(), cudaMemcpyHostToDevice, st_));
    PB_CUDA_CHECK(cudaMemsetAsync(am_.get(), 0, am_.bytes(), st_));
    PB_CUDA_CHECK(cudaMemsetAsync(av_.get(), 0, av_.bytes(), st_));
    adam_t_ = 0;
    refresh_weights();
    PB_CUDA_CHECK(cudaStreamSynchronize(st_));
}

void GnnModel::refresh_weights() {
    refresh_kernel<<<grid_for(2LL * kGnnLayers * 64 * 128), kT, 0, st_>>>(p_.get(), GnnParams::kCount, pr_.get(),
                                                                         w_.get(), wt_.get());
    PB_CUDA_CHECK(cudaGetLastError());
}

void GnnModel::copy_grad(float* host) const {
    PB_CUDA_CHECK(cudaMemcpyAsync(host, g_.get(), g_.bytes(), cudaMemcpyDeviceToHost, st_));
    PB_CUDA_CHECK(cudaStreamSynchronize(st_));
}

void GnnModel::ensure_workspace(const GnnGraph& g) {
    const size_t m = size_t(std::max(g.m, 1)), n = size_t(std::max(g.n, 1)), k = size_t(std::max(g.K, 1));
    const size_t chunks = size_t(std::max(g.cchunks + g.rchunks, 1));
    if (m > cap_m_) {
        for (auto& b : xc_) b.alloc(m * 128);
        hc3_.alloc(m * 64);
        dhc_.alloc(m * 64);
        yhat_.alloc(m);
        cap_m_ = m;
    }
    if (n > cap_n_) {
        for (auto& b : xv_) b.alloc(n * 128);
        hv3_.alloc(n * 64);
        dhv_.alloc(n * 64);
        xhat_.alloc(n);
        cap_n_ = n;
    }
    const size_t mx = std::max(cap_m_, cap_n_);
    if (dz_.size() < mx * 64) {
        dz_.alloc(mx * 64);
        dagg_.alloc(mx * 64);
    }
    if (k > cap_k_) {
        pooled_.alloc(k * 128);
        rho_.alloc(k * 2);         // rho, drho
        lp_sums_.alloc(k * 2);
        cap_k_ = k;
    }
    if (chunks > cap_chunks_) {
        part_.alloc(chunks * 64);
        cap_chunks_ = chunks;
    }
    if (wpart_.size() == 0) {
        wpart_.alloc(size_t(2 * device_sm_count(dev_)) * 128 * 64);
        gpart_.alloc(size_t(grad_blocks(dev_)) * kGradCols);
        loss_.alloc(1);
    }
}

void GnnModel::forward(const GnnGraph& g) {
    last_ = &g;
    if (g.K == 0) return;
    ensure_workspace(g);
    PB_CUDA_CHECK(cudaMemsetAsync(status_.get(), 0, 4, st_));
    const float* pr = pr_.get();
    // input layers
    input_layer_kernel<<<grid_for(g.n), kT, 0, st_>>>(g.fv.get(), g.n, pr + GnnParams::kVinW, xv_[0].get(), 128);
    if (g.m > 0)
        input_layer_kernel<<<grid_for(g.m), kT, 0, st_>>>(g.fc.get(), g.m, pr + GnnParams::kCinW, xc_[0].get(), 128);
    PB_CUDA_CHECK(cudaGetLastError());
    for (int l = 0; l < kGnnLayers; ++l) {
        bf16* out_c = l + 1 < kGnnLayers ? xc_[l + 1].get() : hc3_.get();
        bf16* out_v = l + 1 < kGnnLayers ? xv_[l + 1].get() : hv3_.get();
        const int ldo = l + 1 < kGnnLayers ? 128 : 64;
        Head head_c, head_v;
        if (l + 1 == kGnnLayers) {
            head_c = {pr + GnnParams::kHeadY, g.base_y.get(), yhat_.get()};
            head_v = {pr + GnnParams::kHeadX, g.base_x.get(), xhat_.get()};
        }
        if (g.m > 0) {
            // constraint rows hold five entries or more, columns two or three
            aggregate_kernel<8><<<row_grid(g.m), kT, 0, st_>>>(g.rp.get(), g.ci.get(), g.coef_r.get(), xv_[l].get(),
                                                               128, xc_[l].get(), 128, g.m);
            PB_CUDA_CHECK(cudaGetLastError());
            const CUtensorMap mx = make_bf16_tile_map(xc_[l].get(), g.m, 128, 128, 128);
            const CUtensorMap mw = make_bf16_tile_map(w_.get() + size_t(2 * l) * 64 * 128, 64, 128, 128, 64);
            dense_fwd_kernel<<<dense_blocks(dev_, g.m, 2), kDenseThreads, FwdSmem::kBytes, st_>>>(
                mx, mw, pr + GnnParams::layer_b(l, 0), out_c, ldo, head_c, g.m, status_.get());
            PB_CUDA_CHECK(cudaGetLastError());
            aggregate_kernel<4><<<row_grid(g.n), kT, 0, st_>>>(g.tp.get(), g.ti.get(), g.tcoef_c.get(), out_c, ldo,
                                                               xv_[l].get(), 128, g.n);
        } else {
            // no constraints: the aggregated half of the variable input is zero
            PB_CUDA_CHECK(cudaMemset2DAsync(xv_[l].get() + 64, 256, 0, 128, size_t(g.n), st_));
        }
        PB_CUDA_CHECK(cudaGetLastError());
        const CUtensorMap mx = make_bf16_tile_map(xv_[l].get(), g.n, 128, 128, 128);
        const CUtensorMap mw = make_bf16_tile_map(w_.get() + size_t(2 * l + 1) * 64 * 128, 64, 128, 128, 64);
        dense_fwd_kernel<<<dense_blocks(dev_, g.n, 2), kDenseThreads, FwdSmem::kBytes, st_>>>(
            mx, mw, pr + GnnParams::layer_b(l, 1), out_v, ldo, head_v, g.n, status_.get());
        PB_CUDA_CHECK(cudaGetLastError());
    }
    // pooled means per LP, then rho
    const Chunks cv{g.cchunk_begin.get(), g.clp_first.get(), g.cchunks};
    const Chunks cc{g.rchunk_begin.get(), g.rlp_first.get(), g.rchunks};
    pool_kernel<<<std::min((cv.chunks + cc.chunks + 3) / 4, 148 * 16), 128, 0, st_>>>(hv3_.get(), cv, hc3_.get(), cc,
                                                                                  part_.get());
    pooled_rho_kernel<<<std::min(g.K, 148 * 8), 128, 0, st_>>>(part_.get(), cv, cc, g.inv_n.get(), g.inv_m.get(),
                                                             pr + GnnParams::kHeadW, g.K, pooled_.get(), rho_.get());
    PB_CUDA_CHECK(cudaGetLastError());
}

double GnnModel::backward(const GnnGraph& g, bool grad) {
    if (last_ != &g) throw std::logic_error("GnnModel::backward: forward() was run on another graph");
    if (!g.has_targets) throw InvalidArgument("gnn: the graph has no targets");
    if (g.K == 0) return 0.0;
    const float* pr = pr_.get();
    float* G = g_.get();
    const float inv_k = 1.0f / float(g.K);
    float* drho = rho_.get() + cap_k_;
    const Chunks cv{g.cchunk_begin.get(), g.clp_first.get(), g.cchunks};
    const Chunks cc{g.rchunk_begin.get(), g.rlp_first.get(), g.rchunks};
    const HeadSide sv{xhat_.get(), g.tx.get(), g.lp_col.get(), g.lw_x.get()};
    const HeadSide sc{yhat_.get(), g.ty.get(), g.lp_row.get(), g.lw_y.get()};
    // ---- loss per LP: x and y terms from chunk sums, omega term from rho ----
    if (grad) PB_CUDA_CHECK(cudaMemsetAsync(G, 0, g_.bytes(), st_));
    square_error_kernel<<<std::min((cv.chunks + cc.chunks + 3) / 4, 148 * 16), 128, 0, st_>>>(sv, cv, sc, cc,
                                                                                          part_.get());
    loss_kernel<<<1, 256, 0, st_>>>(part_.get(), cv, cc, rho_.get(), g.tw.get(), g.K, inv_k, pooled_.get(),
                                    lp_sums_.get(), drho, grad ? G + GnnParams::kHeadW : nullptr, loss_.get());
    PB_CUDA_CHECK(cudaGetLastError());
    if (grad) {
        const int blocks = grad_blocks(dev_);
        // Variable-side rows of the layer that `dh` belongs to; `head`: the last layer, from the heads.
        auto base = [&](bool head, bool v, int layer) {
            NodeBackward a{};
            a.rows = v ? g.n : g.m;
            a.dh = v ? dhv_.get() : dhc_.get();
            a.dagg = dagg_.get();
            a.ldh = layer + 1 < kGnnLayers ? 128 : 64;
            a.h = layer + 1 < kGnnLayers ? (v ? xv_[layer + 1].get() : xc_[layer + 1].get())
                                         : (v ? hv3_.get() : hc3_.get());
            a.dz = dz_.get();
            a.part = gpart_.get();
            a.col_bias = kColBias + (2 * layer + (v ? 1 : 0)) * 64;
            if (head) {
                a.col_head = kColHead + (v ? 0 : 65);
                a.side = v ? sv : sc;
                a.inv_k = inv_k;
                a.w = pr + (v ? GnnParams::kHeadX : GnnParams::kHeadY);
                a.ww = pr + GnnParams::kHeadW + (v ? 0 : 64);
                a.drho = drho;
                a.inv = v ? g.inv_n.get() : g.inv_m.get();
            }
            return a;
        };
        auto dense_back = [&](int layer, bool v, const bf16* x, float* dh) {
            const int rows = v ? g.n : g.m, side = v ? 1 : 0;
            const int wblocks = dense_blocks(dev_, rows, 2);
            const CUtensorMap mx = make_bf16_tile_map(x, rows, 128, 128, 128);
            const CUtensorMap mz = make_bf16_tile_map(dz_.get(), rows, 64, 64, 128);
            const CUtensorMap mwt = make_bf16_tile_map(wt_.get() + size_t(2 * layer + side) * 64 * 128, 128, 64, 64, 128);
            dense_dw_kernel<<<wblocks, kDenseThreads, DwSmem::kBytes, st_>>>(mx, mz, wpart_.get(), rows, status_.get());
            PB_CUDA_CHECK(cudaGetLastError());
            dw_reduce_kernel<<<64 * 128 / 32, 256, 0, st_>>>(wpart_.get(), wblocks, G + GnnParams::layer_w(layer, side));
            dense_dx_kernel<<<dense_blocks(dev_, rows, 4), kDenseThreads, DxSmem::kBytes, st_>>>(
                mz, mwt, dh, dagg_.get(), rows, status_.get());
            PB_CUDA_CHECK(cudaGetLastError());
        };
        // ---- message-passing layers, last to first ----
        node_backward_kernel<true, false><<<blocks, 256, 0, st_>>>(base(true, true, kGnnLayers - 1));
        PB_CUDA_CHECK(cudaGetLastError());
        for (int l = kGnnLayers - 1; l >= 0; --l) {
            dense_back(l, true, xv_[l].get(), dhv_.get());
            NodeBackward v = base(false, true, l - 1);
            if (g.m > 0) {
                // agg_v backward: dh_c[i] += sum_j A_ij/(s_a deg_j) dagg_v[j]
                const bool head = l + 1 == kGnnLayers;
                NodeBackward c = base(head, false, l);
                c.rp = g.rp.get(); c.col = g.ci.get(); c.coef = g.coef_c.get();
                if (head) node_backward_kernel<true, false><<<blocks, 256, 0, st_>>>(c);
                else node_backward_kernel<false, false><<<blocks, 256, 0, st_>>>(c);
                PB_CUDA_CHECK(cudaGetLastError());
                dense_back(l, false, xc_[l].get(), dhc_.get());
                // agg_c backward: dh_v[j] += sum_i A_ij/(s_a deg_i) dagg_c[i]
                v.rp = g.tp.get(); v.col = g.ti.get(); v.coef = g.tcoef_r.get();
            }
            if (l > 0) node_backward_kernel<false, false><<<blocks, 256, 0, st_>>>(v);
            else if (g.m > 0) node_backward_kernel<false, true><<<blocks, 256, 0, st_>>>(v);
            PB_CUDA_CHECK(cudaGetLastError());
        }
        // ---- input layers ----
        inlayer_grad_kernel<<<blocks, 256, 0, st_>>>(dhv_.get(), xv_[0].get(), 128, g.fv.get(), g.n, gpart_.get(), kColIn);
        if (g.m > 0)
            inlayer_grad_kernel<<<blocks, 256, 0, st_>>>(dhc_.get(), xc_[0].get(), 128, g.fc.get(), g.m, gpart_.get(),
                                                         kColIn + kInWide);
        grad_total_kernel<<<(kGradCols + 31) / 32, 256, 0, st_>>>(gpart_.get(), blocks, g.m > 0, G);
        PB_CUDA_CHECK(cudaGetLastError());
    }
    double loss = 0.0;
    int hstatus = 0;
    PB_CUDA_CHECK(cudaMemcpyAsync(&loss, loss_.get(), sizeof(double), cudaMemcpyDeviceToHost, st_));
    PB_CUDA_CHECK(cudaMemcpyAsync(&hstatus, status_.get(), 4, cudaMemcpyDeviceToHost, st_));
    PB_CUDA_CHECK(cudaStreamSynchronize(st_));
    if (hstatus & kDevErrTimeout) throw DeviceTimeout("gnn: a tensor-core tile wait exceeded its time limit");
    return loss;
}

void GnnModel::adam_step(float lr) {
    ++adam_t_;
    const float c1 = float(1.0 / (1.0 - std::pow(0.9, double(adam_t_))));
    const float c2 = float(1.0 / (1.0 - std::pow(0.999, double(adam_t_))));
    adam_kernel<<<grid_for(GnnParams::kCount), kT, 0, st_>>>(p_.get(), g_.get(), am_.get(), av_.get(),
                                                            GnnParams::kCount, lr, c1, c2);
    PB_CUDA_CHECK(cudaGetLastError());
    refresh_weights();
}

void GnnModel::predict(const GnnGraph& g, double* const* x, double* const* y, double* omega) {
    if (last_ != &g) throw std::logic_error("GnnModel::predict: forward() was run on another graph");
    if (g.K == 0) return;
    std::vector<float> hx(size_t(g.n)), hy(size_t(g.m)), hr(size_t(g.K));
    PB_CUDA_CHECK(cudaMemcpyAsync(hx.data(), xhat_.get(), size_t(g.n) * 4, cudaMemcpyDeviceToHost, st_));
    if (g.m) PB_CUDA_CHECK(cudaMemcpyAsync(hy.data(), yhat_.get(), size_t(g.m) * 4, cudaMemcpyDeviceToHost, st_));
    PB_CUDA_CHECK(cudaMemcpyAsync(hr.data(), rho_.get(), size_t(g.K) * 4, cudaMemcpyDeviceToHost, st_));
    int hstatus = 0;
    PB_CUDA_CHECK(cudaMemcpyAsync(&hstatus, status_.get(), 4, cudaMemcpyDeviceToHost, st_));
    PB_CUDA_CHECK(cudaStreamSynchronize(st_));
    if (hstatus & kDevErrTimeout) throw DeviceTimeout("gnn: a tensor-core tile wait exceeded its time limit");
    for (int q = 0; q < g.K; ++q) {
        const int k = g.index[size_t(q)];
        const double sa = g.s_a[size_t(q)], sb = g.s_b[size_t(q)], sc = g.s_c[size_t(q)];
        if (x && x[k]) {
            for (int j = g.c0[size_t(q)]; j < g.c0[size_t(q) + 1]; ++j) {
                double v = double(hx[size_t(j)]) * sb / sa;
                if (g.h_vhi[size_t(j)] < 1e29 && v > g.h_vhi[size_t(j)]) v = g.h_vhi[size_t(j)];
                if (g.h_vlo[size_t(j)] > -1e29 && v < g.h_vlo[size_t(j)]) v = g.h_vlo[size_t(j)];
                x[k][j - g.c0[size_t(q)]] = v;
            }
        }
        if (y && y[k])
            for (int i = g.r0[size_t(q)]; i < g.r0[size_t(q) + 1]; ++i)
                y[k][i - g.r0[size_t(q)]] = double(hy[size_t(i)]) * sc / sa;
        if (omega) {
            const double rho = std::min(10.0, std::max(-10.0, double(hr[size_t(q)])));
            omega[k] = g.omega_ref[size_t(q)] * std::exp(rho);
        }
    }
}

size_t GnnModel::trace_size(const GnnGraph& g) const {
    return size_t(kGnnLayers) * (size_t(g.m) + size_t(g.n)) * 128 + (size_t(g.m) + size_t(g.n)) * 64 + size_t(g.n) +
           size_t(g.m) + size_t(g.K) * 129;
}

namespace {
__global__ void bf16_to_f32_kernel(const bf16* __restrict__ src, long long count, float* __restrict__ dst) {
    GNN_STRIDE(i, count) dst[i] = bf(src[i]);
}
}  // namespace

void GnnModel::trace(const GnnGraph& g, float* host) const {
    if (last_ != &g) throw std::logic_error("GnnModel::trace: forward() was run on another graph");
    const size_t total = trace_size(g);
    if (total == 0) return;
    DevBuf<float> t(total);
    size_t off = 0;
    auto conv = [&](const bf16* src, size_t count) {
        if (count) bf16_to_f32_kernel<<<grid_for((long long)count), kT, 0, st_>>>(src, (long long)count, t.get() + off);
        off += count;
    };
    auto copy = [&](const float* src, size_t count) {
        if (count)
            PB_CUDA_CHECK(cudaMemcpyAsync(t.get() + off, src, count * 4, cudaMemcpyDeviceToDevice, st_));
        off += count;
    };
    for (int l = 0; l < kGnnLayers; ++l) conv(xc_[l].get(), size_t(g.m) * 128);
    for (int l = 0; l < kGnnLayers; ++l) conv(xv_[l].get(), size_t(g.n) * 128);
    conv(hc3_.get(), size_t(g.m) * 64);
    conv(hv3_.get(), size_t(g.n) * 64);
    copy(xhat_.get(), size_t(g.n));
    copy(yhat_.get(), size_t(g.m));
    copy(pooled_.get(), size_t(g.K) * 128);
    copy(rho_.get(), size_t(g.K));
    PB_CUDA_CHECK(cudaGetLastError());
    PB_CUDA_CHECK(cudaMemcpyAsync(host, t.get(), total * 4, cudaMemcpyDeviceToHost, st_));
    PB_CUDA_CHECK(cudaStreamSynchronize(st_));
}

}  // namespace pb
