// Prefill dequantise + GEMM, warp-specialised and pipelined (tcgen05 + TMEM + TMA), sm_100a.
//
// Same arithmetic as gemm_tcgen05.cu (bit-exact fp16 weight tiles, fp32
// accumulation in tensor memory), organised so that the tensor cores are not
// left waiting for the reconstruction:
//
//   tile      TM*128 tokens x 128 outputs per block (TM = 1, 2 or 4 accumulators of
//             128 TMEM columns each).  Reconstructing a weight tile is repeated for
//             every token tile, so the token tile is made as tall as tensor memory
//             allows (512 tokens).
//   warp 0    TMA producer: per 64-wide K chunk, TM bulk-tensor loads of a
//             128-token x 64-column activation box (128-byte swizzle) into the
//             stage's A tiles, completion counted on the stage's `full` barrier; and,
//             some chunks ahead, the chunk's indices (16 Q rows x 64 columns) and
//             column scales into a ring of their own.
//   warp 1    MMA issuer: waits for `full`, issues TM x 4 tcgen05.mma
//             (M=128, N=128, K=16) and commits them to the stage's `empty`
//             barrier; the last commit also signals `acc_ready`.
//   warps 2-17 reconstruct the stage's 128-output x 64-column weight tile into the
//             no-swizzle core-matrix layout (2 indices per thread), make it visible
//             to the async proxy and arrive on `full`; afterwards they are the
//             epilogue: tcgen05.ld, bias, fp16, 256 contiguous bytes per token.
//
// No cluster, no multicast; every wait is bounded and ends in a status word.
//
// Reference counterpart: e8d4_wmma_v2_kernel (csrc/eptq_kernels.cu:309-461).

#include <cuda.h>
#include <atomic>
#include <cudaTypedefs.h>

#include "common.cuh"

namespace eptq {

struct GemmWsArgs {
    EptqLayer L;
    __half* y;             // (T, 8M)
    int* status;
    int T;
    int splits;            // K ranges (gridDim.z); above 1 their sums meet in `partial`
    float* partial;        // [tile][split][TM*128 tokens][NT outputs]
    unsigned* counters;    // one per tile, zero on entry and again on exit
};

namespace {

constexpr int kMaxStages = 3;
constexpr int kChunkK = 64;
constexpr int kATileBytes = 128 * kChunkK * 2;          // 16 KB: 128 tokens x 64 columns, 128-byte rows
// B tile: core matrices (8 rows x 16 B = 128 contiguous bytes) adjacent in K are placed 144 bytes apart instead of
// 128, so that the threads of a warp, which write the same row of neighbouring core matrices, hit different banks.
constexpr unsigned kB_LBO = 144;                        // bytes between core matrices adjacent in K
constexpr unsigned kB_SBO = (kChunkK / 8) * kB_LBO;     // bytes between 8-row groups (1152)
constexpr int kOutTile = 128;                           // measured: 256 outputs double the reconstruction per stage and run ~20 % slower
constexpr int kProducerWarps = 16;                      // reconstruction is latency-bound: many warps
constexpr int kWsThreads = (2 + kProducerWarps) * 32;   // 576
constexpr unsigned long long kWaitNs = 2000000000ull;     // limit of one mbarrier wait

// Blocks per SM: reconstruction waits more than it issues (48 % of issue slots with one block), so short E8-D4 tiles, the
// only ones whose registers and stages allow it, run two.
__host__ __device__ constexpr int ws_blocks(int kind, int tm) { return kind == EPTQ_E8D4 && tm == 1 ? 2 : 1; }
// Stages: 2 for 512x128 tiles (82 KB each) and where two blocks share the SM, otherwise 3 (50 or 34 KB).
__host__ __device__ constexpr int ws_stage_bytes(int tm, int nt) { return tm * kATileBytes + (nt / 8) * static_cast<int>(kB_SBO); }
__host__ __device__ constexpr int ws_stages(int kind, int tm, int nt) {
    return ws_stage_bytes(tm, nt) > 65536 || ws_blocks(kind, tm) == 2 ? 2 : 3;
}
// Index ring.  The reconstruction threads used to read their indices from global memory themselves: the fence that makes a
// weight tile visible to the tensor cores then waited for the next chunks' loads as well, a DRAM round trip in every chunk.
constexpr int kQStages = 6;
constexpr int kQBytes = 16 * kChunkK * 2;               // 16 Q rows x 64 columns
constexpr int kQStride = kQBytes + 2 * kChunkK * 2;     // + column scales h + group scales
__host__ __device__ constexpr int ws_smem_bytes(int kind, int tm, int nt) {
    return ws_stages(kind, tm, nt) * ws_stage_bytes(tm, nt) + kQStages * kQStride + 1024;
}

__device__ __forceinline__ unsigned smem_u32(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
    // Bounded by wall time (two seconds of the global timer, looked at every 1024 polls), not by a poll count
    // whose length would depend on the clock.
    unsigned long long t0 = 0;
    for (unsigned it = 0;; ++it) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
        if ((it & 1023u) == 1023u) {
            unsigned long long now;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (t0 == 0) t0 = now;
            else if (now - t0 > kWaitNs) return false;
        }
    }
}

// A tile: K-major, 128-byte swizzle (what the bulk-tensor load writes): 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t desc_a_sw128(unsigned addr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((addr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(1) << 16;                  // leading byte offset: unused with swizzled K-major
    d |= static_cast<uint64_t>(1024 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;                  // SWIZZLE_128B
    return d;
}
// B tile: K-major, no swizzle, core matrices of 8 rows x 16 bytes.
__device__ __forceinline__ uint64_t desc_b_plain(unsigned addr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((addr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(kB_LBO >> 4) << 16;
    d |= static_cast<uint64_t>(kB_SBO >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    return d;
}
__host__ __device__ constexpr uint32_t instr_desc(int nt) { return (1u << 4) | (static_cast<uint32_t>(nt >> 3) << 17) | ((128u >> 4) << 24); }

// First critical block of row m (CSR, sorted by column) at or behind column n.
__device__ __forceinline__ int first_marker(const EptqLayer& L, int m, int n) {
    int lo = __ldg(L.O_row_ptr + m), hi = __ldg(L.O_row_ptr + m + 1);
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(L.O_col + mid) < n) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Two fp32 multiplies, each rounded to nearest.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
        "mul.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

template <int KIND, int TM, int NT>
__global__ void __launch_bounds__(kWsThreads, ws_blocks(KIND, TM))
gemm_tcgen05_ws_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_q,
                       const GemmWsArgs p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(16) float4 tab_s[KIND == EPTQ_E8D4 ? 512 : 1];
    __shared__ __align__(8) unsigned long long bar_full[kMaxStages], bar_empty[kMaxStages], bar_qfull[kQStages], bar_qempty[kQStages], bar_acc;
    __shared__ unsigned tmem_base_slot, last_slot, read_sink[kProducerWarps];

    constexpr int kStages = ws_stages(KIND, TM, NT);
    constexpr int kStageBytes = ws_stage_bytes(TM, NT);
    constexpr unsigned kTmemCols = TM * NT;               // 128, 256 or 512: a power of two >= 32
    constexpr int kTileOuts = NT;
    constexpr uint32_t kInstrDesc = instr_desc(NT);
    const EptqLayer& L = p.L;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int N = L.N, out_dim = 8 * L.M;
    const int t0 = blockIdx.y * (TM * 128);
    const int m0 = blockIdx.x * (kTileOuts / 8);
    const int all_chunks = (N + kChunkK - 1) / kChunkK;
    const int c_begin = static_cast<int>(blockIdx.z) * all_chunks / p.splits;             // this block's K range
    const int n_chunks = (static_cast<int>(blockIdx.z) + 1) * all_chunks / p.splits - c_begin;
    // dynamic shared memory may start at an address that is not 1024-aligned: align by hand
    unsigned char* tiles = smem + ((1024u - (smem_u32(smem) & 1023u)) & 1023u);

    unsigned char* const qring = tiles + kStages * kStageBytes;
    // Group scales of one row serve the whole tile when no group ends inside it; otherwise the threads read their own.
    const bool s_shared = L.S_group != nullptr && (L.qb_size % kTileOuts) == 0;

    if (KIND == EPTQ_E8D4)
        for (int i = tid; i < 512; i += kWsThreads) tab_s[i] = __ldg(reinterpret_cast<const float4*>(L.table32) + i);
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&bar_full[s]), 1 + kProducerWarps);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        for (int s = 0; s < kQStages; ++s) {
            mbar_init(smem_u32(&bar_qfull[s]), 1);
            mbar_init(smem_u32(&bar_qempty[s]), kProducerWarps);
        }
        mbar_init(smem_u32(&bar_acc), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(reinterpret_cast<uint64_t>(&tmap_x)) : "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(&tmem_base_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem_acc = tmem_base_slot;
    bool ok = true;

    if (warp == 0) {
        // ---------------- TMA producer
        if (lane == 0) {
            auto load_indices = [&](int c) {
                const int s = c % kQStages, n0 = (c_begin + c) * kChunkK;
                if (!mbar_wait(smem_u32(&bar_qempty[s]), ((c / kQStages) & 1u) ^ 1u)) return false;
                const unsigned full = smem_u32(&bar_qfull[s]), dst = smem_u32(qring + s * kQStride);
                const unsigned cols = min(kChunkK, N - n0) * 2;           // bytes; N % 8 == 0: a multiple of 16
                mbar_arrive_expect_tx(full, kQBytes + cols + (s_shared ? cols : 0u));
                asm volatile(
                    "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                    :: "r"(dst), "l"(reinterpret_cast<uint64_t>(&tmap_q)), "r"(n0), "r"(m0), "r"(full) : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             :: "r"(dst + kQBytes), "l"(L.h + n0), "r"(cols), "r"(full) : "memory");
                if (s_shared)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                 :: "r"(dst + kQBytes + kChunkK * 2), "l"(L.S_group + static_cast<size_t>((8 * m0) / L.qb_size) * N + n0),
                                    "r"(cols), "r"(full) : "memory");
                return true;
            };
            constexpr int kAhead = kQStages - 1;             // chunk c + kAhead goes where chunk c - 1 was
            for (int c = 0; c < kAhead && c < n_chunks && ok; ++c) ok = load_indices(c);
            for (int c = 0; c < n_chunks && ok; ++c) {
                const int s = c % kStages;
                const unsigned phase = (c / kStages) & 1u;
                ok = mbar_wait(smem_u32(&bar_empty[s]), phase ^ 1u);
                if (!ok) break;
                const unsigned full = smem_u32(&bar_full[s]);
                mbar_arrive_expect_tx(full, TM * kATileBytes);
#pragma unroll
                for (int j = 0; j < TM; ++j) {
                    const unsigned dst = smem_u32(tiles + s * kStageBytes + j * kATileBytes);
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                        :: "r"(dst), "l"(reinterpret_cast<uint64_t>(&tmap_x)), "r"((c_begin + c) * kChunkK), "r"(t0 + j * 128), "r"(full)
                        : "memory");
                }
                if (c + kAhead < n_chunks) ok = load_indices(c + kAhead);
            }
            if (!ok) atomicExch(p.status, EPTQ_ERR_TIMEOUT);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer
        if (lane == 0) {
            for (int c = 0; c < n_chunks && ok; ++c) {
                const int s = c % kStages;
                const unsigned phase = (c / kStages) & 1u;
                ok = mbar_wait(smem_u32(&bar_full[s]), phase);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t db = desc_b_plain(smem_u32(tiles + s * kStageBytes + TM * kATileBytes));
#pragma unroll
                for (int j = 0; j < TM; ++j) {
                    const uint64_t da = desc_a_sw128(smem_u32(tiles + s * kStageBytes + j * kATileBytes));
#pragma unroll
                    for (int k = 0; k < kChunkK / 16; ++k) {
                        const unsigned accumulate = (c > 0 || k > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                            :: "r"(tmem_acc + j * NT), "l"(da + static_cast<uint64_t>((k * 32) >> 4)),
                               "l"(db + static_cast<uint64_t>((k * 2 * kB_LBO) >> 4)), "r"(kInstrDesc), "r"(accumulate)
                            : "memory");
                    }
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                             :: "r"(smem_u32(&bar_empty[s])) : "memory");
            }
            if (ok)
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                             :: "r"(smem_u32(&bar_acc)) : "memory");
            else
                atomicExch(p.status, EPTQ_ERR_TIMEOUT);
        }
    } else {
        // ---------------- weight-tile producers (512 threads), then epilogue
        // 16 Q rows x 64 columns per chunk: one warp per Q row, two neighbouring columns of the chunk per lane.
        static_assert(NT / 8 == kProducerWarps && kChunkK == 64, "one warp per Q row");
        const int qrow = warp - 2;
        const int bm = m0 + qrow;
        const bool b_valid = bm < L.M;
        float2 gk[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            gk[k] = b_valid ? make_float2(__half2float(__ldg(reinterpret_cast<const __half*>(L.g) + 8 * bm + 2 * k)),
                                          __half2float(__ldg(reinterpret_cast<const __half*>(L.g) + 8 * bm + 2 * k + 1)))
                            : make_float2(0.f, 0.f);
        const __half* srow = (L.S_group != nullptr && b_valid && !s_shared)
            ? reinterpret_cast<const __half*>(L.S_group) + static_cast<size_t>((8 * bm) / L.qb_size) * N : nullptr;
        const unsigned b_off = qrow * kB_SBO + (lane >> 2) * kB_LBO + (lane & 3) * 4;

        // What depends on a chunk's indices (E8 codewords in L2, critical blocks) is read one chunk ahead.  A critical
        // block's position is the row's running count plus the markers of lower columns (two ballots).
        struct Inputs { unsigned q, h, s; };
        struct Words { float4 lo[2], hi[2]; };               // E8: the codeword; a critical block: lo holds its 8 fp16
        auto fetch = [&](int c, Inputs& in) {
            const int n0 = (c_begin + c) * kChunkK + lane * 2;
            in.q = 0u; in.h = 0u; in.s = 0x3c003c00u;
            if (c >= n_chunks) return true;
            const int s = c % kQStages;
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_qfull[s]), (c / kQStages) & 1u))) return false;
            if (b_valid && n0 < N) {                          // N % 8 == 0: both columns are in or out
                const unsigned char* src = qring + s * kQStride + lane * 4;
                in.q = *reinterpret_cast<const unsigned*>(src + qrow * (kChunkK * 2));
                in.h = *reinterpret_cast<const unsigned*>(src + kQBytes);
                if (s_shared) in.s = *reinterpret_cast<const unsigned*>(src + kQBytes + kChunkK * 2);
                else if (srow != nullptr) in.s = __ldg(reinterpret_cast<const unsigned*>(srow + n0));
            }
            // The slot is free for the next TMA write once every lane's values are in registers.  An arrive alone does not
            // wait for that: shared-memory reads still under way saw the slot's next chunk.  So the arrive follows a store
            // that needs all of them.
            const unsigned read = __reduce_xor_sync(0xffffffffu, in.q ^ in.h ^ in.s);
            if (lane == 0) {
                *static_cast<volatile unsigned*>(&read_sink[qrow]) = read;
                mbar_arrive(smem_u32(&bar_qempty[s]));
            }
            return true;
        };
        int next_marker = b_valid ? first_marker(L, bm, c_begin * kChunkK) : 0;
        const unsigned below = (1u << lane) - 1u;
        auto index_of = [](unsigned q, int e) { return ((e ? q >> 16 : q) & 0xffffu) ^ 0x8000u; };
        // Returns whether the warp has a critical block in the chunk.
        auto lookup = [&](int c, const Inputs& in, Words& w) {
            const bool live = b_valid && (c_begin + c) * kChunkK + lane * 2 < N && c < n_chunks;
            const unsigned i0 = index_of(in.q, 0), i1 = index_of(in.q, 1);
            const bool k0 = live && i0 == kMarkerIndex, k1 = live && i1 == kMarkerIndex;
            if (KIND == EPTQ_E8 && live) {
                const float4* t0 = reinterpret_cast<const float4*>(L.table32 + static_cast<size_t>(k0 ? 0u : i0) * 8);
                const float4* t1 = reinterpret_cast<const float4*>(L.table32 + static_cast<size_t>(k1 ? 0u : i1) * 8);
                w.lo[0] = __ldg(t0); w.hi[0] = __ldg(t0 + 1);
                w.lo[1] = __ldg(t1); w.hi[1] = __ldg(t1 + 1);
            }
            if (__ballot_sync(0xffffffffu, k0 || k1) == 0u) return false;
            const unsigned m0b = __ballot_sync(0xffffffffu, k0), m1b = __ballot_sync(0xffffffffu, k1);
            const int r0 = next_marker + __popc(m0b & below) + __popc(m1b & below);
            next_marker += __popc(m0b) + __popc(m1b);
            if (k0) w.lo[0] = __ldg(reinterpret_cast<const float4*>(L.O_vals) + r0);
            if (k1) w.lo[1] = __ldg(reinterpret_cast<const float4*>(L.O_vals) + r0 + (k0 ? 1 : 0));
            return true;
        };
        // W16[8m .. 8m+7, n], bit-for-bit the reference's reconstruction (see gemm_tcgen05.cu): separate fp32 multiplies,
        // two dimensions per instruction.
        auto reconstruct8 = [&](unsigned idx, const float4& lo, const float4& hi, float hn, float sg, bool marked, float2 (&v)[4]) {
            float4 a = lo, b = hi;
            if (KIND == EPTQ_E8D4) {
                const unsigned ct = (idx >> 14) & 3u;
                a = tab_s[ct * 128 + ((idx >> 7) & 127u)];
                b = tab_s[ct * 128 + (idx & 127u)];
            }
            v[0] = make_float2(a.x, a.y); v[1] = make_float2(a.z, a.w); v[2] = make_float2(b.x, b.y); v[3] = make_float2(b.z, b.w);
            if (L.S_group != nullptr) {
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = mul2(v[k], make_float2(sg, sg));
            }
            if (marked && idx == kMarkerIndex) {
                float o8[8];
                unpack8(*reinterpret_cast<const uint4*>(&lo), o8);
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = make_float2(o8[2 * k], o8[2 * k + 1]);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = mul2(mul2(v[k], gk[k]), make_float2(hn, hn));
        };
        // E8 reads its codewords one chunk ahead; E8-D4 finds them in shared memory and looks ahead for critical blocks
        // only, behind the chunk's own work (registers for a second set would keep a second block off the SM).
        constexpr bool kTwoSets = KIND == EPTQ_E8;
        Inputs in0, in1;
        Words w0, w1;
        bool marked = false, marked1 = false;
#pragma unroll
        for (int e = 0; e < 2; ++e) w0.lo[e] = w0.hi[e] = w1.lo[e] = w1.hi[e] = make_float4(0.f, 0.f, 0.f, 0.f);
        ok = fetch(0, in0);
        if (ok) marked = lookup(0, in0, w0);
        for (int c = 0; c < n_chunks && ok; ++c) {
            const int s = c % kStages;
            const unsigned phase = (c / kStages) & 1u;
            const bool live = b_valid && (c_begin + c) * kChunkK + lane * 2 < N;
            if (kTwoSets) {
                ok = fetch(c + 1, in1);
                if (!ok) break;
                marked1 = lookup(c + 1, in1, w1);
            }
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_empty[s]), phase ^ 1u));     // the warp goes on together
            if (!ok) break;
            float2 v0[4], v1[4];
            const float2 h2f = __half22float2(*reinterpret_cast<const __half2*>(&in0.h));
            const float2 s2f = __half22float2(*reinterpret_cast<const __half2*>(&in0.s));
            reconstruct8(index_of(in0.q, 0), w0.lo[0], w0.hi[0], h2f.x, s2f.x, marked, v0);
            reconstruct8(index_of(in0.q, 1), w0.lo[1], w0.hi[1], h2f.y, s2f.y, marked, v1);
            unsigned char* dst = tiles + s * kStageBytes + TM * kATileBytes + b_off;
#pragma unroll
            for (int k = 0; k < 4; ++k) {                     // rows 2k, 2k+1 of the core matrix: two neighbouring columns
                const __half2 p0 = __floats2half2_rn(v0[k].x, v1[k].x), p1 = __floats2half2_rn(v0[k].y, v1[k].y);
                *reinterpret_cast<unsigned*>(dst + 2 * k * 16) = live ? *reinterpret_cast<const unsigned*>(&p0) : 0u;
                *reinterpret_cast<unsigned*>(dst + (2 * k + 1) * 16) = live ? *reinterpret_cast<const unsigned*>(&p1) : 0u;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_full[s]));
            if (kTwoSets) {
                in0 = in1; w0 = w1; marked = marked1;
            } else {
                ok = fetch(c + 1, in0);
                if (ok) marked = lookup(c + 1, in0, w0);
            }
        }
        if (!ok && lane == 0) atomicExch(p.status, EPTQ_ERR_TIMEOUT);

        // ---------------- epilogue
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_acc), 0u));
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // The accumulators occupy TMEM columns [0, TM*NT): sub-tile j (128 tokens) at columns [j*NT, (j+1)*NT).
        // Four groups of four warps (one warp per lane quarter) each take a quarter of those columns.
        const int quarter = warp & 3;                        // TMEM lanes this warp may read
        const int group = (warp - 2) >> 2;
        constexpr int kColsPerGroup = TM * NT / 4;           // 32 .. 128, a multiple of 32
        const int acc_col0 = group * kColsPerGroup;
        const int tok_in_tile = (acc_col0 / NT) * 128 + quarter * 32 + lane;
        const int col0 = acc_col0 % NT;                      // first output column (inside the tile) of this group
        const int token = t0 + tok_in_tile;
        const unsigned lane_addr = tmem_acc + (static_cast<unsigned>(quarter * 32) << 16) + acc_col0;
        constexpr size_t kTileFloats = static_cast<size_t>(TM) * 128 * NT;
        const unsigned tile = blockIdx.y * gridDim.x + blockIdx.x;
        // bias, fp16, 8 outputs of one token
        auto store8 = [&](const float (&f)[8], int tok, int o) {
            if (o >= out_dim) return;
            __half2 h2[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float f0 = f[2 * e], f1 = f[2 * e + 1];
                if (L.bias != nullptr) {
                    f0 += __half2float(__ldg(reinterpret_cast<const __half*>(L.bias) + o + 2 * e));
                    f1 += __half2float(__ldg(reinterpret_cast<const __half*>(L.bias) + o + 2 * e + 1));
                }
                h2[e] = __floats2half2_rn(f0, f1);
            }
            *reinterpret_cast<uint4*>(p.y + static_cast<size_t>(tok) * out_dim + o) = *reinterpret_cast<const uint4*>(h2);
        };
        if (ok) {
#pragma unroll
            for (int part = 0; part < kColsPerGroup / 32; ++part) {
                unsigned r[32];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                    "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                    "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                      "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                      "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                    : "r"(lane_addr + part * 32) : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (token < p.T) {
                    if (p.splits > 1) {
                        float* dst = p.partial + (static_cast<size_t>(tile) * p.splits + blockIdx.z) * kTileFloats +
                                     static_cast<size_t>(tok_in_tile) * NT + col0 + part * 32;
#pragma unroll
                        for (int v = 0; v < 8; ++v)
                            __stcg(reinterpret_cast<uint4*>(dst) + v, make_uint4(r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]));
                    } else {
#pragma unroll
                        for (int v8 = 0; v8 < 4; ++v8) {
                            float f[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[v8 * 8 + e]);
                            store8(f, token, blockIdx.x * kTileOuts + col0 + part * 32 + v8 * 8);
                        }
                    }
                }
            }
        } else if (lane == 0) {
            atomicExch(p.status, EPTQ_ERR_TIMEOUT);
        }
        if (p.splits > 1) {
            // Every block takes its ticket, a timed-out one too: the counter has to come back to zero.  The last one
            // adds the partial sums in split order.
            asm volatile("bar.sync 1, %0;" :: "n"(kProducerWarps * 32) : "memory");
            if (tid == 64) {
                unsigned ticket;
                asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(ticket) : "l"(p.counters + tile) : "memory");
                last_slot = ticket == static_cast<unsigned>(p.splits) - 1u ? 1u : 0u;
                if (last_slot != 0u) p.counters[tile] = 0u;
            }
            asm volatile("bar.sync 1, %0;" :: "n"(kProducerWarps * 32) : "memory");
            if (last_slot != 0u) {
                const float* src = p.partial + static_cast<size_t>(tile) * p.splits * kTileFloats;
                constexpr int kVec = NT / 8;                 // threads of neighbouring outputs, then tokens
                const int rows = min(TM * 128, p.T - t0);
                for (int i = tid - 64; i < rows * kVec; i += kProducerWarps * 32) {
                    const int tk = i / kVec, o8 = (i % kVec) * 8;
                    const float* s = src + static_cast<size_t>(tk) * NT + o8;
                    float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
                    for (int k = 0; k < p.splits; ++k) {
                        const float4 a = __ldcg(reinterpret_cast<const float4*>(s + k * kTileFloats));
                        const float4 b = __ldcg(reinterpret_cast<const float4*>(s + k * kTileFloats) + 1);
                        f[0] += a.x; f[1] += a.y; f[2] += a.z; f[3] += a.w;
                        f[4] += b.x; f[5] += b.y; f[6] += b.z; f[7] += b.w;
                    }
                    store8(f, t0 + tk, blockIdx.x * kTileOuts + o8);
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_acc), "r"(kTmemCols) : "memory");
    }
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
    }
    return fn;
}

template <int KIND, int TM, int NT>
int launch_ws(const CUtensorMap& tmap, const CUtensorMap& tmap_q, const GemmWsArgs& a, dim3 grid, cudaStream_t stream) {
    static std::atomic<bool> attr_done[64];       // setting the attribute twice is harmless; the flag itself must not race
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return EPTQ_ERR_LAUNCH;
    if (!attr_done[dev]) {
        if (cudaFuncSetAttribute(gemm_tcgen05_ws_kernel<KIND, TM, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 ws_smem_bytes(KIND, TM, NT)) != cudaSuccess)
            return EPTQ_ERR_LAUNCH;
        attr_done[dev] = true;
    }
    gemm_tcgen05_ws_kernel<KIND, TM, NT><<<grid, kWsThreads, ws_smem_bytes(KIND, TM, NT), stream>>>(tmap, tmap_q, a);
    count_launch(EPTQ_KERNEL_GEMM);
    return cudaPeekAtLastError() == cudaSuccess ? EPTQ_OK : EPTQ_ERR_LAUNCH;
}

template <int KIND>
int launch_ws_shape(int tm, const CUtensorMap& tmap, const CUtensorMap& tmap_q, const GemmWsArgs& a, dim3 grid, cudaStream_t stream) {
    switch (tm) {
        case 1: return launch_ws<KIND, 1, kOutTile>(tmap, tmap_q, a, grid, stream);
        case 2: return launch_ws<KIND, 2, kOutTile>(tmap, tmap_q, a, grid, stream);
        default: return launch_ws<KIND, 4, kOutTile>(tmap, tmap_q, a, grid, stream);
    }
}

int tile_tokens(int T) { return T <= 128 ? 128 : T <= 256 ? 256 : 512; }
int tile_count(int M, int T) { return ((8 * M + kOutTile - 1) / kOutTile) * ((T + tile_tokens(T) - 1) / tile_tokens(T)); }
size_t split_bytes(int M, int T, int splits) {
    return splits > 1 ? static_cast<size_t>(tile_count(M, T)) * splits * tile_tokens(T) * kOutTile * sizeof(float) : 0;
}

// K ranges per output tile: a 4096-output layer has 32 tiles for 148 SMs.  The times below are in hundredths of what a
// chunk takes an E8-D4 block (about 1 us; an E8 chunk 1.3), fitted to 1 to 16 ranges of eleven layers from 768 x 768 to
// 14336 x 4096 at 17 to 512 tokens: a block's chunks and its prologue and epilogue, for each round of blocks over the SMs
// (two blocks on one SM take 1.6 times as long as one); then once the last block's sum, which reads every token's partial
// sums of every range (5.7 ns a token and range).  Over that set the choice is within 2 % of the fastest in the mean
// and never more than 1 % behind one range.  Without that last term short rows at many tokens lost: 768 x 768 E8-D4 at 512
// tokens 34.5 us in three ranges, 25.7 in one; 1024 x 4096 71.3 us in sixteen, 49.0 in four.
// Bounded by the counters, by a K range of four chunks, and by 64 MiB of partial sums.
int plan_splits(int kind, int M, int N, int T) {
    const int tiles = tile_count(M, T), chunks = (N + kChunkK - 1) / kChunkK, tokens = T < tile_tokens(T) ? T : tile_tokens(T);
    const bool shared_sm = ws_blocks(kind, tile_tokens(T) / 128) == 2;
    if (tiles >= kMaxCounters - 1) return 1;
    int best = 1;
    long long best_cost = 0;
    for (int s = 1; s <= 16 && (s == 1 || chunks / s >= 4); ++s) {
        if (split_bytes(M, T, s) > (static_cast<size_t>(64) << 20)) break;
        const long long rounds = (static_cast<long long>(tiles) * s + kSms - 1) / kSms;
        const long long block = static_cast<long long>((chunks + s - 1) / s) * (kind == EPTQ_E8 ? 130 : 100) + 400 + 2 * tokens;
        const long long cost = rounds * block * (shared_sm && rounds > 1 ? 8 : 10) + (s > 1 ? 3000 + 10 * tokens + tokens * s * 57 / 10 : 0);
        if (s == 1 || cost < best_cost) { best = s; best_cost = cost; }
    }
    return best;
}

}  // namespace

// Bytes of partial sums a call's K ranges want behind the first MiB of scratch; with less it runs as one range.
size_t gemm_ws_partial_bytes(int kind, int M, int N, int T) { return split_bytes(M, T, plan_splits(kind, M, N, T)); }

// The pipelined kernel needs a tensor map over x: base 16-byte aligned, row pitch a multiple of 16 bytes.
bool gemm_ws_supported(const EptqLayer& L, const void* x, int T) {
    return T >= 1 && L.table32 != nullptr && (L.N % 8) == 0 && aligned16(x) && aligned16(L.Q) && aligned16(L.h) &&
           aligned16(L.table32) && (L.n_masked == 0 || aligned16(L.O_vals)) &&
           (L.S_group == nullptr || (L.qb_size > 0 && L.qb_size % 8 == 0 && aligned16(L.S_group))) &&
           tensor_map_encoder() != nullptr;
}

int launch_gemm_tcgen05_ws(const EptqLayer& L, const uint16_t* x, uint16_t* y, int T, void* workspace, size_t workspace_bytes,
                           cudaStream_t stream) {
    const int out_dim = 8 * L.M;
    const int tm = tile_tokens(T) / 128;
    int splits = plan_splits(L.quantizer, L.M, L.N, T);
    if (workspace_bytes < kPartialOffset + split_bytes(L.M, T, splits)) splits = 1;
    CUtensorMap tmap, tmap_q;
    auto encode = [&](CUtensorMap* m, CUtensorMapDataType type, const void* base, int rows, unsigned box_rows, CUtensorMapSwizzle swizzle) {
        const cuuint64_t dims[2] = {static_cast<cuuint64_t>(L.N), static_cast<cuuint64_t>(rows)};
        const cuuint64_t strides[1] = {static_cast<cuuint64_t>(L.N) * 2};
        const cuuint32_t box[2] = {kChunkK, box_rows};
        const cuuint32_t estr[2] = {1, 1};
        return tensor_map_encoder()(m, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                    swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    if (!encode(&tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x, T, 128, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode(&tmap_q, CU_TENSOR_MAP_DATA_TYPE_UINT16, L.Q, L.M, kOutTile / 8, CU_TENSOR_MAP_SWIZZLE_NONE))
        return EPTQ_ERR_LAUNCH;
    GemmWsArgs a;
    a.L = L;
    a.y = reinterpret_cast<__half*>(y);
    a.status = reinterpret_cast<int*>(workspace) + (kMaxCounters - 1);     // last counter word: never a tile
    a.T = T;
    a.splits = splits;
    a.partial = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + kPartialOffset);
    a.counters = reinterpret_cast<unsigned*>(workspace);
    const dim3 grid((out_dim + kOutTile - 1) / kOutTile, (T + tm * 128 - 1) / (tm * 128), splits);
    if (grid.y > 65535u) return EPTQ_ERR_SHAPE;
    return L.quantizer == EPTQ_E8 ? launch_ws_shape<EPTQ_E8>(tm, tmap, tmap_q, a, grid, stream)
                                  : launch_ws_shape<EPTQ_E8D4>(tm, tmap, tmap_q, a, grid, stream);
}

}  // namespace eptq
