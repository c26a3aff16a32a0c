// BF16 GEMM on the 5th-generation tensor cores of sm_103a: C = A * B^T with
// A [M x K] and B [N x K] both row-major (K contiguous), FP32 accumulation in
// tensor memory, operands staged into shared memory by TMA tensor copies
// (cp.async.bulk.tensor, 128-byte swizzle) through a STAGES-deep mbarrier ring.
//
// One CTA = 128 threads computes one 128 x BN tile of C over one K chunk
// (split-K: blockIdx.z selects the chunk; its partial goes to C + z*M*N):
//   warp 0, one lane : TMA producer
//   warp 1, one lane : tcgen05.mma issuer (kind::f16, BF16 x BF16 -> F32)
//   all 4 warps      : epilogue, tcgen05.ld of the accumulator (warp w owns
//                      TMEM lanes 32w..32w+31 = rows of the tile) -> global.
// Every wait is bounded by the global timer; a timeout sets *err and the CTA
// still drains what it issued and frees its tensor memory before returning.
//
// MN = true takes both operands stored [K x M] and [K x N] row-major (the K index is the row:
// C = A^T B), as MN-major tiles: TMA boxes of 64 columns x 64 rows, the transposition
// left to the tensor core's operand fetch. The weight gradients of a network (C = da^T h over
// the points) then need no transposed copies of da and h.
// HEAD = true writes the first three columns of a row as one 16-byte vector.
#pragma once
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

namespace nsfv1 {
namespace tc {

constexpr int BM = 128;          // rows per tile = TMEM lanes
constexpr int BK = 64;           // K per stage: 64 BF16 = 128 bytes = one swizzle span
constexpr int UK = 16;           // K per tcgen05.mma (kind::f16)
constexpr unsigned long long kWaitNs = 1000000000ull;   // 1 s per wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait for the phase of the given parity; false on timeout
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    while (!mbar_try_wait(bar, parity))
        if (global_ns() - t0 > kWaitNs) return false;
    return true;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// shared-memory matrix descriptor of a K-major tile written by TMA with the
// 128-byte swizzle: rows of 128 bytes, 8-row atoms 1024 bytes apart (SBO),
// descriptor version 1, swizzle mode 2 (128B); LBO is unused for this layout.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}

// the same for an MN-major tile of 64 K-rows per TMA box of 64 columns: 8-row atoms 1024 bytes
// apart along K (SBO), boxes of 64 columns 8192 bytes apart (LBO)
__device__ __forceinline__ uint64_t sw128_desc_mn(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(8192 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}
constexpr uint32_t kIdescMN = (1u << 15) | (1u << 16);   // A and B MN-major

// instruction descriptor of kind::f16: D F32, A and B BF16, both K-major, M x N
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

template <int BN, int STAGES>
struct GemmSmem {
    static constexpr int kA = BM * BK * 2;        // 16 KB
    static constexpr int kB = BN * BK * 2;        // BN * 128 bytes
    static constexpr int kStage = kA + kB;
    static constexpr int kBytes = STAGES * kStage + 1024 /* align */ + 256 /* barriers */;
};

// C[z][M][N] = A[M][kz..] * B[N][kz..]^T over K chunk z of kChunk columns.
// M % 128 == 0, N % BN == 0, K % 64 == 0, kChunk % 64 == 0 (host-checked).
template <int BN, int STAGES, bool MN = false, bool HEAD = false>
__global__ void __launch_bounds__(128, 1)
    k_gemm_bf16_tn(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, float* __restrict__ C,
                   int M, int N, int K, int kChunk, int* err) {
    static_assert(BN % 32 == 0 && BN >= 32 && BN <= 256, "tile N");
    extern __shared__ uint8_t smem_raw[];
    using S = GemmSmem<BN, STAGES>;
    uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(base + STAGES * S::kStage);
    uint32_t* tmemSlot = (uint32_t*)(bars + 2 * STAGES + 1);
    const uint32_t fullBar = smem_u32(bars), emptyBar = fullBar + 8 * STAGES, doneBar = fullBar + 16 * STAGES;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int k0 = blockIdx.z * kChunk;
    const int kEnd = min(K, k0 + kChunk);
    const int nk = (kEnd - k0) / BK;
    constexpr uint32_t kCols = BN < 32 ? 32 : BN;   // power of two >= 32

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(fullBar + 8 * s, 1); mbar_init(emptyBar + 8 * s, 1); }
        mbar_init(doneBar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmemSlot)), "r"(kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmemSlot;
    bool ok = true;

    if (warp == 0 && lane == 0) {
        // producer
        int issued = 0;
        for (int kt = 0; kt < nk; ++kt) {
            const int s = kt % STAGES;
            if (kt >= STAGES && !mbar_wait(emptyBar + 8 * s, ((kt / STAGES) & 1) ^ 1)) { ok = false; break; }
            const uint32_t sa = smem_u32(base + s * S::kStage), sb = sa + S::kA;
            mbar_expect_tx(fullBar + 8 * s, S::kStage);
            if constexpr (MN) {
#pragma unroll
                for (int i = 0; i < BM / 64; ++i) tma_load_2d(sa + i * 8192, &mapA, m0 + 64 * i, k0 + kt * BK, fullBar + 8 * s);
#pragma unroll
                for (int i = 0; i < BN / 64; ++i) tma_load_2d(sb + i * 8192, &mapB, n0 + 64 * i, k0 + kt * BK, fullBar + 8 * s);
            } else {
                tma_load_2d(sa, &mapA, k0 + kt * BK, m0, fullBar + 8 * s);
                tma_load_2d(sb, &mapB, k0 + kt * BK, n0, fullBar + 8 * s);
            }
            ++issued;
        }
        // drain: every issued copy has landed before the CTA may exit
        for (int kt = (issued > STAGES ? issued - STAGES : 0); kt < issued; ++kt)
            if (!mbar_wait(fullBar + 8 * (kt % STAGES), (kt / STAGES) & 1)) ok = false;
    } else if (warp == 1 && lane == 0) {
        // MMA issuer
        constexpr uint32_t idesc = idesc_bf16(BM, BN) | (MN ? kIdescMN : 0u);
        for (int kt = 0; kt < nk; ++kt) {
            const int s = kt % STAGES;
            if (!mbar_wait(fullBar + 8 * s, (kt / STAGES) & 1)) { ok = false; break; }
            fence_after();
            const uint32_t sa = smem_u32(base + s * S::kStage), sb = sa + S::kA;
#pragma unroll
            for (int k = 0; k < BK / UK; ++k)
                if constexpr (MN) mma_bf16(tmem, sw128_desc_mn(sa + k * UK * 128), sw128_desc_mn(sb + k * UK * 128), idesc, (kt | k) != 0);
                else mma_bf16(tmem, sw128_desc(sa + k * UK * 2), sw128_desc(sb + k * UK * 2), idesc, (kt | k) != 0);
            mma_commit(emptyBar + 8 * s);
        }
        mma_commit(doneBar);   // arrives once every MMA issued above has completed
    }
    __syncwarp();
    // epilogue
    // warp-uniform: tcgen05.ld below is a .sync.aligned instruction
    const bool done = __all_sync(0xffffffffu, mbar_wait(doneBar, 0));
    fence_after();
    if (!done) ok = false;
    if (HEAD && done) {
        float v[32];
        tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16), v);
        reinterpret_cast<float4*>(C)[m0 + warp * 32 + lane] = make_float4(v[0], v[1], v[2], 0.f);
    } else if (done && nk > 0) {
        const int row = m0 + warp * 32 + lane;
        float* crow = C + ((size_t)blockIdx.z * M + row) * N + n0;
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
            float v[32];
            tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + c, v);
#pragma unroll
            for (int i = 0; i < 32; i += 4) *(float4*)(crow + c + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
    } else if (done) {
        const int row = m0 + warp * 32 + lane;
        float* crow = C + ((size_t)blockIdx.z * M + row) * N + n0;
        for (int c = 0; c < BN; c += 4) *(float4*)(crow + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (!ok) atomicOr(err, 4);
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
    }
}

// ---------------------------------------------------------------------------
// One layer: a = h W^T on the tensor cores (W [256 x K]), with ACT its activation in the epilogue,
//   z = gamma (a + bias) + beta,  h_out = z sigmoid(z)  (BF16; 0 for rows >= P),
// and the FP32 a itself with STORE_A (the backward pass reads it; without ACT the plain product).
// W stays in shared memory for the whole launch, tiles of 128 rows of h stream
// through a ring, and the FP32 accumulators alternate between two TMEM halves, so the
// tensor core works on the next tile while this one's epilogue runs. A warp's results
// pass through shared memory so that a store covers 8 rows of 64 bytes instead of 32 of 16.
//   warps 0..EW-1 : epilogue (warp w: TMEM lanes 32 (w % 4).., columns of its quarter)
//   warp EW       : TMA producer (one lane)
//   warp EW + 1   : MMA issuer (one lane); the warp allocates and frees the tensor memory
// The activation's instructions bound it: a tile's MMAs take 1.2 us. Measured at K = 256:
// 81 us for 249,728 rows; with 16-byte stores straight from the lanes 121 us. 532,512 points
// through all layers and the head: 0.95 ms, 3.13 ms when the FP32 product went through memory to
// an activation kernel that also wrote a transposed copy. 96 registers a thread (576 threads); the
// training variant (ACT and STORE_A) spills 40 bytes, the others nothing.
// ---------------------------------------------------------------------------
template <int K>
struct LayerSmem {
    static constexpr int KB = K / BK, STAGES = 3, EW = 16;
    static constexpr int kA = BM * BK * 2, kW = 256 * BK * 2;
    static constexpr int kRow = 64 + 16, kOut = 32 * kRow;   // a warp's 32 rows of 64 bytes, padded
    static constexpr int kBytes = KB * kW + STAGES * kA + EW * kOut + 1024 /* align */ + 256 /* barriers */;
    static constexpr int THREADS = 32 * (EW + 2);
};

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

struct LayerArgs {
    int64_t P;               // rows that hold points (the others get 0)
    int nTiles;              // 128-row tiles
    const float* bias;       // [256]
    const float* film;       // [slot][...]: 256 gammas, 256 betas of this layer
    int64_t filmStride;      // floats between slots
    const int32_t* slot;     // [P] slot of a point
    uint16_t* h;             // [rows][256] BF16 bits
    float* a;                // [rows][256] (STORE_A)
    int* err;
};

// rows of 64 bytes (4 vectors of this lane's row) through the warp's buffer to row-major memory:
// dst = the 64-byte segment of row 0, rows 'pitch' vectors apart
__device__ __forceinline__ void store_rows(uint8_t* buf, int lane, const uint4 (&v)[4], uint4* __restrict__ dst, int64_t pitch) {
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(buf + lane * 80 + q * 16) = v[q];
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = q * 8 + (lane >> 2), part = lane & 3;
        dst[(int64_t)r * pitch + part] = *reinterpret_cast<const uint4*>(buf + r * 80 + part * 16);
    }
}

template <int K, bool ACT, bool STORE_A, class Act>
__global__ void __launch_bounds__(LayerSmem<K>::THREADS, 1)
    k_layer(const __grid_constant__ CUtensorMap mapH, const __grid_constant__ CUtensorMap mapW, const LayerArgs A, const Act act) {
    using S = LayerSmem<K>;
    constexpr int KB = S::KB, STAGES = S::STAGES, EW = S::EW;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sW = smem_u32(base), sA = sW + KB * S::kW;
    uint8_t* sOut = base + KB * S::kW + STAGES * S::kA;
    uint64_t* bars = (uint64_t*)(sOut + EW * S::kOut);
    uint32_t* tmemSlot = (uint32_t*)(bars + 2 * STAGES + 6);
    const uint32_t wBar = smem_u32(bars), fullBar = wBar + 8, emptyBar = fullBar + 8 * STAGES, accFull = emptyBar + 8 * STAGES,
                   accEmpty = accFull + 16, endBar = accEmpty + 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(wBar, 1);
        mbar_init(endBar, 1);
        for (int s = 0; s < STAGES; ++s) { mbar_init(fullBar + 8 * s, 1); mbar_init(emptyBar + 8 * s, 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(accFull + 8 * s, 1); mbar_init(accEmpty + 8 * s, EW); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == EW + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmemSlot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmemSlot;
    bool ok = true;

    if (warp == EW && lane == 0) {
        // producer: the weights once, then the tiles' K blocks
        mbar_expect_tx(wBar, KB * S::kW);
        for (int kb = 0; kb < KB; ++kb) tma_load_2d(sW + kb * S::kW, &mapW, kb * BK, 0, wBar);
        int n = 0;
        for (int tile = blockIdx.x; ok && tile < A.nTiles; tile += gridDim.x)
            for (int kb = 0; kb < KB; ++kb, ++n) {
                const int s = n % STAGES;
                if (n >= STAGES && !mbar_wait(emptyBar + 8 * s, ((n / STAGES) & 1) ^ 1)) { ok = false; break; }
                mbar_expect_tx(fullBar + 8 * s, S::kA);
                tma_load_2d(sA + s * S::kA, &mapH, kb * BK, tile * BM, fullBar + 8 * s);
            }
        // drain: every issued copy has landed before the CTA may exit
        if (!mbar_wait(wBar, 0)) ok = false;
        for (int q = n > STAGES ? n - STAGES : 0; q < n; ++q)
            if (!mbar_wait(fullBar + 8 * (q % STAGES), (q / STAGES) & 1)) ok = false;
    } else if (warp == EW + 1 && lane == 0) {
        // MMA issuer
        constexpr uint32_t idesc = idesc_bf16(BM, 256);
        if (!mbar_wait(wBar, 0)) ok = false;
        int n = 0, it = 0;
        for (int tile = blockIdx.x; ok && tile < A.nTiles; tile += gridDim.x, ++it) {
            const int buf = it & 1;
            if (it >= 2 && !mbar_wait(accEmpty + 8 * buf, ((it >> 1) & 1) ^ 1)) { ok = false; break; }
            fence_after();
            for (int kb = 0; kb < KB; ++kb, ++n) {
                const int s = n % STAGES;
                if (!mbar_wait(fullBar + 8 * s, (n / STAGES) & 1)) { ok = false; break; }
                fence_after();
                const uint32_t sa = sA + s * S::kA, sb = sW + kb * S::kW;
#pragma unroll
                for (int k = 0; k < BK / UK; ++k)
                    mma_bf16(tmem + buf * 256, sw128_desc(sa + k * UK * 2), sw128_desc(sb + k * UK * 2), idesc, (kb | k) != 0);
                mma_commit(emptyBar + 8 * s);
            }
            mma_commit(accFull + 8 * buf);
        }
        // every MMA issued above has completed before the tensor memory is freed
        mma_commit(endBar);
        if (!mbar_wait(endBar, 0)) ok = false;
    } else if (warp < EW) {
        constexpr int CW = 256 / (EW / 4);   // columns of a warp
        const int quarter = warp & 3, c0 = (warp >> 2) * CW;
        int it = 0;
        for (int tile = blockIdx.x; tile < A.nTiles; tile += gridDim.x, ++it) {
            const int buf = it & 1;
            const bool got = __all_sync(0xffffffffu, mbar_wait(accFull + 8 * buf, (it >> 1) & 1));
            if (!got) { ok = false; break; }
            fence_after();
            const int64_t row0 = (int64_t)tile * BM + quarter * 32, row = row0 + lane;
            const bool live = row < A.P;
            const float* __restrict__ film = ACT ? A.film + (live ? (int64_t)__ldg(A.slot + row) : 0) * A.filmStride : nullptr;
            uint8_t* buf_ = sOut + warp * S::kOut;
#pragma unroll 1
            for (int c = c0; c < c0 + CW; c += 32) {
                float v[32];
                tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + buf * 256 + c, v);
                if (c + 32 == c0 + CW) {
                    // this warp has read its part of the accumulator
                    fence_before();
                    if (lane == 0) mbar_arrive(accEmpty + 8 * buf);
                }
                if constexpr (STORE_A) {
                    uint4* dst = reinterpret_cast<uint4*>(A.a + row0 * 256 + c);
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        uint4 o[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            o[q] = make_uint4(__float_as_uint(v[16 * half + 4 * q]), __float_as_uint(v[16 * half + 4 * q + 1]),
                                              __float_as_uint(v[16 * half + 4 * q + 2]), __float_as_uint(v[16 * half + 4 * q + 3]));
                        store_rows(buf_, lane, o, dst + 4 * half, 64);
                    }
                }
                if constexpr (ACT) {
                    uint4 o[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint32_t w[4];
#pragma unroll
                        for (int p = 0; p < 2; ++p) {
                            const int k = 2 * q + p;
                            const float4 g = __ldg(reinterpret_cast<const float4*>(film + c) + k),
                                         be = __ldg(reinterpret_cast<const float4*>(film + 256 + c) + k),
                                         b = __ldg(reinterpret_cast<const float4*>(A.bias + c) + k);
                            const float h0 = act(v[4 * k], b.x, g.x, be.x), h1 = act(v[4 * k + 1], b.y, g.y, be.y);
                            const float h2 = act(v[4 * k + 2], b.z, g.z, be.z), h3 = act(v[4 * k + 3], b.w, g.w, be.w);
                            w[2 * p] = live ? act.pack(h0, h1) : 0u;
                            w[2 * p + 1] = live ? act.pack(h2, h3) : 0u;
                        }
                        o[q] = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                    store_rows(buf_, lane, o, reinterpret_cast<uint4*>(A.h + row0 * 256 + c), 32);
                }
            }
        }
    }
    __syncwarp();
    if (!ok) atomicOr(A.err, 4);
    fence_before();
    __syncthreads();
    if (warp == EW + 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

}  // namespace tc
}  // namespace nsfv1
