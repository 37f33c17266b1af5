// Reconstruction of the fp16 weight from the quantized layer, bit-for-bit the
// arithmetic of the reference's `dequantize_layer` (algorithms/eptq.py:406-471):
//   v = table32[index]            (fp32; E8-D4: two 4-vectors of one class)
//   v = v * S_group[row/qb, col]  (only when group scales exist, and never on a
//                                  critical block)                 eptq.py:440-449
//   v = O_vals[rank]              (critical block)                  eptq.py:461-466
//   v = (v * g[row]) * h[col]     (two fp32 multiplies, left to right) eptq.py:469
//   W = fp16(v)                   (round to nearest even)           eptq.py:471
//
// 2 B of Q in, 16 B of W out per index.  One thread owns 8 consecutive columns of
// one Q row, so its output rows are each written as one 128-bit store.  Two kernels:
// dequant_vec_kernel for N % 8 == 0, dequant_kernel for the rest.

#include <atomic>

#include "common.cuh"

namespace eptq {

namespace {

// Rank of column `n` among the markers of row m (markers are sorted by column).
__device__ __forceinline__ int marker_rank(const int* __restrict__ O_col, int lo, int hi, int n) {
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (__ldg(O_col + mid) < n) lo = mid + 1; else hi = mid;
    }
    return lo;
}

template <int KIND>
__global__ void __launch_bounds__(256) dequant_kernel(EptqLayer L, __half* __restrict__ W, int chunks_per_row) {
    const long long gid = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int m = static_cast<int>(gid / chunks_per_row);
    if (m >= L.M) return;
    const int n0 = static_cast<int>(gid % chunks_per_row) * 8;
    const int N = L.N;
    const int16_t* qrow = L.Q + static_cast<size_t>(m) * N;
    const __half* g = reinterpret_cast<const __half*>(L.g);
    const __half* h = reinterpret_cast<const __half*>(L.h);
    const __half* O = reinterpret_cast<const __half*>(L.O_vals);
    const __half* S = reinterpret_cast<const __half*>(L.S_group);

    float gk[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) gk[k] = __half2float(__ldg(g + 8 * m + k));

    __half out[8][8];   // [k][e]
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int n = n0 + e;
        float v[8];
        if (n < N) {
            const unsigned idx = static_cast<unsigned>(static_cast<int>(qrow[n]) + 32768);
            if (idx == kMarkerIndex) {
                const int lo = __ldg(L.O_row_ptr + m), hi = __ldg(L.O_row_ptr + m + 1);
                const int r = marker_rank(L.O_col, lo, hi, n);
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = __half2float(__ldg(O + static_cast<size_t>(r) * 8 + k));
            } else {
                if (KIND == EPTQ_E8) {
                    const float4* t = reinterpret_cast<const float4*>(L.table32 + static_cast<size_t>(idx) * 8);
                    const float4 a = __ldg(t), b = __ldg(t + 1);
                    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
                    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
                } else {
                    const unsigned ct = (idx >> 14) & 3u, ii = (idx >> 7) & 127u, jj = idx & 127u;
                    const float4 a = __ldg(reinterpret_cast<const float4*>(L.table32) + ct * 128 + ii);
                    const float4 b = __ldg(reinterpret_cast<const float4*>(L.table32) + ct * 128 + jj);
                    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
                    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
                }
                if (S != nullptr) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int grp = (8 * m + k) / L.qb_size;
                        v[k] = __fmul_rn(v[k], __half2float(__ldg(S + static_cast<size_t>(grp) * N + n)));
                    }
                }
            }
            const float hn = __half2float(__ldg(h + n));
#pragma unroll
            for (int k = 0; k < 8; ++k) out[k][e] = __float2half_rn(__fmul_rn(__fmul_rn(v[k], gk[k]), hn));
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) out[k][e] = __float2half_rn(0.f);
        }
    }

    const bool full = (n0 + 8 <= N) && ((N & 7) == 0);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        __half* dst = W + static_cast<size_t>(8 * m + k) * N + n0;
        if (full) {
            *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(&out[k][0]);
        } else {
            for (int e = 0; e < 8 && n0 + e < N; ++e) dst[e] = out[k][e];
        }
    }
}

// Two fp32 multiplies, each rounded to nearest.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
        "mul.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// N % 8 == 0: 128-bit reads of Q, h and S, and no branch between the table reads of a thread's eight columns, so that they
// are all in flight together; critical blocks are put in afterwards, with one search per thread (its markers are
// neighbours in the row's list).  The general kernel above searches inside each index's branch and reads Q and h two
// bytes at a time.  E8-D4 keeps eight copies of the fp32 table in shared memory (64 KB): the eight lanes of a 128-bit read
// phase hit different banks.  E8 gathers its 32-byte codewords from L2; what bounds it is the L1's one line per cycle, so
// two neighbouring lanes share a codeword (dimensions 0-3 and 4-7) and a read of the warp touches 16 lines, not 32.
// 11008 x 4096, 101 MB of traffic: E8 60.3 us (general kernel), 61.9 (this one, a codeword per lane), 43.0 (shared); E8-D4
// 24.9 us, 15 us less than before in a call of 1024 tokens (144.1 -> 128.7 us).
constexpr int kCopies = 8;
constexpr int kVecThreadsD4 = 512, kVecThreadsE8 = 256;

template <int KIND, bool SCALED>
__global__ void __launch_bounds__(KIND == EPTQ_E8 ? kVecThreadsE8 : kVecThreadsD4, KIND == EPTQ_E8 ? 4 : 2)
dequant_vec_kernel(const EptqLayer L, __half* __restrict__ W, unsigned chunks_per_row, unsigned total) {
    constexpr int ROWS = KIND == EPTQ_E8 ? 4 : 8;              // output rows (dimensions) of a thread
    constexpr int PAIRS = ROWS / 2;
    extern __shared__ __align__(16) float4 tab[];
    const int N = L.N;
    const float4* mine = tab + (threadIdx.x & (kCopies - 1));
    if (KIND == EPTQ_E8D4) {
        for (int i = threadIdx.x; i < 512 * kCopies; i += blockDim.x) tab[i] = __ldg(reinterpret_cast<const float4*>(L.table32) + i / kCopies);
        __syncthreads();
    }
    for (unsigned id = blockIdx.x * blockDim.x + threadIdx.x; id < total; id += gridDim.x * blockDim.x) {
        const unsigned chunk = KIND == EPTQ_E8 ? id >> 1 : id;
        const unsigned half = KIND == EPTQ_E8 ? id & 1u : 0u;
        const unsigned m = chunk / chunks_per_row, n0 = (chunk - m * chunks_per_row) * 8;
        const unsigned row0 = 8 * m + ROWS * half;
        const uint4 qv = ldg128(L.Q + static_cast<size_t>(m) * N + n0);
        const uint4 hv = ldg128(L.h + n0);
        uint4 sv = make_uint4(0, 0, 0, 0);
        if (SCALED) sv = ldg128(L.S_group + static_cast<size_t>(8 * m / L.qb_size) * N + n0);
        float2 gk[PAIRS];
        {
            const uint2* gp = reinterpret_cast<const uint2*>(L.g + row0);
#pragma unroll
            for (int k = 0; k < PAIRS; k += 2) {
                const uint2 gv = __ldg(gp + k / 2);
                gk[k] = __half22float2(*reinterpret_cast<const __half2*>(&gv.x));
                gk[k + 1] = __half22float2(*reinterpret_cast<const __half2*>(&gv.y));
            }
        }
        const unsigned* qw = reinterpret_cast<const unsigned*>(&qv);
        unsigned marks = 0;                                    // markers are stored as 0x7fff
#pragma unroll
        for (int e = 0; e < 8; ++e) marks |= (((qw[e >> 1] >> (16 * (e & 1))) & 0xffffu) == 0x7fffu ? 1u : 0u) << e;
        unsigned out[ROWS][4];                                 // [row][column pair]
        constexpr int STEP = KIND == EPTQ_E8 ? 8 : 2;          // columns whose table reads are in flight
#pragma unroll
        for (int e0 = 0; e0 < 8; e0 += STEP) {
            float4 w[STEP][PAIRS / 2];
#pragma unroll
            for (int e = 0; e < STEP; ++e) {
                const unsigned idx = ((qw[(e0 + e) >> 1] >> (16 * (e & 1))) & 0xffffu) ^ 0x8000u;
                if (KIND == EPTQ_E8) {
                    w[e][0] = __ldg(reinterpret_cast<const float4*>(L.table32) + 2 * static_cast<size_t>(idx == kMarkerIndex ? 0u : idx) + half);
                } else {
                    w[e][0] = mine[(idx >> 7) * kCopies];                           // class and first half: 9 bits
                    w[e][PAIRS / 2 - 1] = mine[(((idx >> 7) & 0x180u) | (idx & 127u)) * kCopies];
                }
            }
#pragma unroll
            for (int pr = 0; pr < STEP; pr += 2) {
                const int j = (e0 + pr) >> 1;
                const float2 h2 = __half22float2(reinterpret_cast<const __half2*>(&hv)[j]);
                const float2 s2 = __half22float2(reinterpret_cast<const __half2*>(&sv)[j]);
                float2 v[2][PAIRS];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const float hs = c ? h2.y : h2.x, ss = c ? s2.y : s2.x;
#pragma unroll
                    for (int k = 0; k < PAIRS; ++k) {
                        const float4 q4 = w[pr + c][k >> 1];
                        v[c][k] = k & 1 ? make_float2(q4.z, q4.w) : make_float2(q4.x, q4.y);
                        if (SCALED) v[c][k] = mul2(v[c][k], make_float2(ss, ss));
                        v[c][k] = mul2(mul2(v[c][k], gk[k]), make_float2(hs, hs));
                    }
                }
#pragma unroll
                for (int k = 0; k < PAIRS; ++k) {
                    const __half2 r0 = __floats2half2_rn(v[0][k].x, v[1][k].x), r1 = __floats2half2_rn(v[0][k].y, v[1][k].y);
                    out[2 * k][j] = *reinterpret_cast<const unsigned*>(&r0);
                    out[2 * k + 1][j] = *reinterpret_cast<const unsigned*>(&r1);
                }
            }
        }
        __half* dst = W + static_cast<size_t>(row0) * N + n0;
#pragma unroll
        for (int k = 0; k < ROWS; ++k)
            *reinterpret_cast<uint4*>(dst + static_cast<size_t>(k) * N) = make_uint4(out[k][0], out[k][1], out[k][2], out[k][3]);
        if (marks != 0u) {                                     // overwrite the marked columns
            int r = marker_rank(L.O_col, __ldg(L.O_row_ptr + m), __ldg(L.O_row_ptr + m + 1), static_cast<int>(n0) + __ffs(marks) - 1);
            for (; marks != 0u; marks &= marks - 1u, ++r) {
                const int e = __ffs(marks) - 1;
                const float hn = __half2float(__ldg(reinterpret_cast<const __half*>(L.h) + n0 + e));
                const __half* O = reinterpret_cast<const __half*>(L.O_vals) + static_cast<size_t>(r) * 8 + ROWS * half;
#pragma unroll
                for (int k = 0; k < ROWS; ++k)
                    dst[static_cast<size_t>(k) * N + e] = __float2half_rn(
                        __fmul_rn(__fmul_rn(__half2float(__ldg(O + k)), __half2float(__ldg(reinterpret_cast<const __half*>(L.g) + row0 + k))), hn));
            }
        }
    }
}

template <int KIND, bool SCALED>
int launch_vec(const EptqLayer& L, __half* W, cudaStream_t stream) {
    constexpr int threads = KIND == EPTQ_E8 ? kVecThreadsE8 : kVecThreadsD4;
    constexpr int smem = KIND == EPTQ_E8 ? 0 : 512 * kCopies * 16;
    if (smem > 0) {
        static std::atomic<bool> attr_done[64];       // setting the attribute twice is harmless; the flag itself must not race
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return EPTQ_ERR_LAUNCH;
        if (!attr_done[dev]) {
            if (cudaFuncSetAttribute(dequant_vec_kernel<KIND, SCALED>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
                return EPTQ_ERR_LAUNCH;
            attr_done[dev] = true;
        }
    }
    const unsigned chunks = static_cast<unsigned>(L.N / 8);
    const unsigned total = static_cast<unsigned>(L.M) * chunks * (KIND == EPTQ_E8 ? 2 : 1);
    unsigned grid = (total + threads - 1) / threads;
    if (KIND == EPTQ_E8D4 && grid > 2 * 148) grid = 2 * 148;   // the table copies are made once per block
    dequant_vec_kernel<KIND, SCALED><<<grid, threads, smem, stream>>>(L, W, chunks, total);
    count_launch(EPTQ_KERNEL_OTHER);
    return cudaPeekAtLastError() == cudaSuccess ? EPTQ_OK : EPTQ_ERR_LAUNCH;
}

}  // namespace

int launch_dequant(const EptqLayer& L, uint16_t* W, cudaStream_t stream) {
    const int chunks = (L.N + 7) / 8;
    const long long total = static_cast<long long>(L.M) * chunks;
    const int block = 256;
    const long long grid = (total + block - 1) / block;
    if (grid > 0x7fffffffLL) return EPTQ_ERR_SHAPE;
    __half* Wh = reinterpret_cast<__half*>(W);
    // 32-bit thread numbers with room for a grid stride; g in 128-bit reads (its alignment is not part of the contract).
    if ((L.N & 7) == 0 && total <= 0x38000000LL && aligned16(L.g)) {
        if (L.quantizer == EPTQ_E8) return L.S_group != nullptr ? launch_vec<EPTQ_E8, true>(L, Wh, stream) : launch_vec<EPTQ_E8, false>(L, Wh, stream);
        return L.S_group != nullptr ? launch_vec<EPTQ_E8D4, true>(L, Wh, stream) : launch_vec<EPTQ_E8D4, false>(L, Wh, stream);
    }
    if (L.quantizer == EPTQ_E8) {
        dequant_kernel<EPTQ_E8><<<static_cast<unsigned>(grid), block, 0, stream>>>(L, Wh, chunks);
    } else {
        dequant_kernel<EPTQ_E8D4><<<static_cast<unsigned>(grid), block, 0, stream>>>(L, Wh, chunks);
    }
    count_launch(EPTQ_KERNEL_OTHER);
    return cudaPeekAtLastError() == cudaSuccess ? EPTQ_OK : EPTQ_ERR_LAUNCH;
}

}  // namespace eptq
