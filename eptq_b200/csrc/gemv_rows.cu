// Decode GEMV of 3 to 16 batch rows over a group of independent layers of one codebook (E8-D4 or E8), one pass
// over the weights.
//
// What bounds it: decoding an index (two conflict-free table reads of 2 wavefronts each for E8-D4, one conflicting
// read for E8, about eight integer instructions) costs more than streaming its two bytes, so every decoded
// codeword has to serve all batch rows.  The two-row kernel of gemv_group.cu, run once per pair of rows, decoded
// every index ceil(B / 2) times and left seven eighths of each MMA's columns to a diagonal.  Here a pair of
// codewords of neighbouring columns is transposed with PRMT (4 instructions per index) into ordinary A fragments
// (16 outputs x 16 columns), and the MMA columns are batch rows.
//
// Arithmetic as in gemv_group.cu: codewords unmodified in fp16, x*h*2^-e split into an fp16 part and an fp16
// remainder, fp32 accumulation.  NB = 4: the remainders take columns 4..7 of the one column tile; NB = 8, 16: they
// run as a second MMA into the same accumulators.
//
// Work split: a step is 32 Q rows x 32 columns; all steps (layer, row tile, column step) form one sequence, block b
// takes the contiguous share [W*b/G, W*(b+1)/G).  16 main warps: warp = (column group kq = warp / 4, row group
// rg = warp % 4); the four warps of a column group take every fourth step of the share, convert the step's
// activations once into a shared fragment buffer (double-buffered, one 128-thread barrier per step) and each decode 8
// Q rows.  At the end of a row tile (or of the share) the four column groups are added through shared memory and
// the block's partial sums go to scratch with plain stores; the block that takes the last
// ticket of a row tile, for its share or for a unit of corrections, adds the partials in block order, so results do not
// depend on arrival order.
//
// Group scales (SCALED; one layer, passes of 4 rows): the scale of a row group's 64 outputs multiplies x*h before the split,
// so the four warps of a column group need different fragments and each converts its own (4 values a lane and step).
// The SIMT kernel holds x*h*S and its products in 32 bits, and the split here loses none of that: each batch row is scaled
// by a power of two from its own max|x| (a pass over the rows while the table arrives), so that its values use the upper
// binades of fp16; the remainder is kept times 2^11; and codewords are lattice coordinates, small whole or half numbers,
// whose products with 11-bit parts the tensor core adds without loss.  Error of the sums against 64 bits, x of 1e-4 to 10,
// four shapes up to 4096 x 14336: log-normal S and h of sigma 0.1 and 0.25 1.2e-7 (SIMT kernel 1.4e-7), 0.5 and 0.3 1.3e-7
// (1.4e-7), 1.2 and 0.1 2.4e-7 (1.5e-7: the tensor core cuts where the other rounds); without the three up to 4e-2.
// Time with them, 14336 x 4096 at 1 row: E8-D4 19.6 -> 21.3 us, E8 25.4 -> 26.3 us.
// Taken for qb_size % 64 == 0 where it is the faster one (rows_scaled_supported); the SIMT kernel, which multiplies in its
// inner loop, stays for the rest.
//
// Critical blocks: while the table arrives, the warps of the launch walk the CSR tables in units of 4 Q rows (at most a
// unit or two per warp for the fractions in use) and store sum (O - code[65535])*h*x to a slot of their own that the
// last arrival adds; what does not need x is read before the dependency wait, and the ticket is looked at behind the main
// loop (4096 x 4096 E8-D4: 14.1 -> 13.3 us at 4 rows, 16.1 -> 15.2 at 8).  Dedicated warps for it would leave 96 registers a thread, and the main loop then spills: to L2,
// since nearly all of L1 is shared memory (4096 x 4096 E8-D4, 16 rows: 60.3 against 23.7 us a call).

#include <atomic>
#include <cmath>
#include <mutex>

#include "common.cuh"

namespace eptq {

namespace {

constexpr int kRowsMaxLayers = 32;
constexpr int kRowsFewLayers = 8;          // launches of few layers copy a smaller parameter block
constexpr int kTileRows = 32;              // Q rows of a row tile (256 outputs)
constexpr int kTileOut = kTileRows * 8;
constexpr int kColGroups = 4;
constexpr int kRowsWarps = 16;
constexpr int kRowsThreads = kRowsWarps * 32;
// Steps of Q, x and h in flight per warp.  Two cover the memory latency where a step is long (16 rows), and the
// registers of a third would spill there.
__host__ __device__ constexpr int ring_steps(int nb) { return nb == 16 ? 2 : 3; }
constexpr int kCorrPerTile = kTileRows / 4;
constexpr unsigned kRowsTableAddr = 0x10000u;                   // shared-window address of the replicated E8-D4 table
constexpr int kRowsSmemD4 = 2 * 65536 - 1024;                   // window [0x400, 0x20000)
constexpr int kRowsSmemE8 = 232448;                             // the most a block may ask for
// Control words: 0 last-arrival flag, 1 finished tiles, 4..7 row maxima, 16..31 a word per warp, 32.. the finished tiles.  Of
// those a block has at most 16 from units of corrections and 9 from its share, which touches at most tiles / G + 2 (148
// blocks, or shares of up to seven steps: plan_rows).
constexpr unsigned kCtrlBytes = 256;

// Fragment buffers ([column group][2][hi, lo][NB rows][32 columns] fp16), reused for the sum over column groups.
// With group scales every warp has its own buffers.
__host__ __device__ constexpr unsigned area_bytes(int nb, bool scaled) { return nb == 16 || scaled ? 16384u : 8192u; }
__host__ __device__ constexpr unsigned e8_table_offset(int nb, bool scaled) { return area_bytes(nb, scaled) + kCtrlBytes; }
__host__ __device__ constexpr unsigned e8_resident(int nb, bool scaled) { return (kRowsSmemE8 - e8_table_offset(nb, scaled)) / 4; }

struct RowsLayer {
    const int16_t* Q;
    const __half* g;
    const __half* h;
    const __half* x;
    const __half* O_vals;
    const int* O_col;
    const int* O_row_ptr;
    const __half* bias;
    __half* y;
    int step0;              // index of this layer's first step
    int tile0;              // index of its first row tile
    int corr0;              // index of its first correction unit
    int M, N;
    int ns;                 // steps per row tile = N / 32
    int row_tiles;          // ceil(M / 32)
    int corr_tile;          // correction units per row tile: 8, or 0 for a layer without critical blocks
    int qb_rows;            // Q rows per scale group, 0 without group scales
    const __half* S;
    float x_scale;          // power of two, <= 1 / max|h| (/ max|S|; then times the batch row's own power of two)
    float x_inv_scale;
};

template <int MAXL>
struct RowsArgs {
    RowsLayer L[MAXL];
    const uint2* table16;
    const unsigned* packed;
    unsigned* counters;     // zero on entry, zero again on exit
    float* partial;         // [block + tile][NB][256] main partials, then [tile][NB][256] corrections
    float code_unit;        // group scales, E8-D4: table16 = lattice coordinate * code_unit
    unsigned W;             // steps
    int G;                  // blocks with a share
    int tiles;
    int corr_units;
    int n_layers;
    int B;
};

__device__ __forceinline__ uint2 lds64(unsigned addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ unsigned lo_halves(unsigned a, unsigned b) { return __byte_perm(a, b, 0x5410); }
__device__ __forceinline__ unsigned hi_halves(unsigned a, unsigned b) { return __byte_perm(a, b, 0x7632); }
__device__ __forceinline__ void mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ldg_once(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void split_half(float v, __half& hi, __half& lo) {
    hi = __float2half_rn(v);
    lo = __float2half_rn(v - __half2float(hi));
}
// x * s = hi + lo * 2^-11 with one rounding of the remainder (a fused multiply-add forms it): 22 bits and the sign while hi
// is normal, and for |x * s| <= 2^15 a remainder times 2^11 is at most 2^15 too.
constexpr float kLoScale = 2048.f;
__device__ __forceinline__ void split_product(float x, float s, __half& hi, __half& lo) {
    hi = __float2half_rn(x * s);
    lo = __float2half_rn(fmaf(x, s, -__half2float(hi)) * kLoScale);
}
// 2^n, -126 <= n <= 127
__device__ __forceinline__ float exp2i(int n) { return __int_as_float((127 + n) << 23); }
// Biased fp16 exponent e of a row's largest |x| (bits): |x| < 2^(e-14).  Infinities and NaN count as the largest finite.
__device__ __forceinline__ int row_exponent(unsigned bits) { return min(max(static_cast<int>(bits >> 10), 1), 30); }
constexpr int kRowTop = 29;                 // a row's values times 2^(kRowTop - e) stay below 2^15

// A coordinate of the E8-D4 lattice from its fp16 table entry: the rounding of the entry is far less than half a step.
__device__ __forceinline__ float lattice(__half code, float inv_unit) { return rintf(__half2float(code) * inv_unit); }
__device__ __forceinline__ unsigned lattice2(unsigned codes, float inv_unit) {
    const __half2 c = *reinterpret_cast<const __half2*>(&codes);
    const __half2 v = __floats2half2_rn(lattice(__low2half(c), inv_unit), lattice(__high2half(c), inv_unit));
    return *reinterpret_cast<const unsigned*>(&v);
}

// Packed E8 entry -> fp16 pairs of dims (0,1), (2,3), (4,5), (6,7): the layout and the arithmetic are stated at
// e8_decode in gemv_group.cu.
__device__ __forceinline__ void e8_entry(unsigned e, unsigned (&r)[4]) {
    const unsigned rot = __funnelshift_r(e, e, 8);
    const unsigned magic = 0x64006400u;
    unsigned a[4] = {(e & 0x003C003Cu) | magic, (e & 0x03C003C0u) | magic, (rot & 0x003C003Cu) | magic, (rot & 0x03C003C0u) | magic};
    const __half2 kA = __floats2half2_rn(0.125f, 0.125f), cA = __floats2half2_rn(-131.f, -131.f);
    const __half2 kB = __floats2half2_rn(0.0078125f, 0.0078125f), cB = __floats2half2_rn(-11.f, -11.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __half2 v = __hfma2(*reinterpret_cast<__half2*>(&a[i]), i & 1 ? kB : kA, i & 1 ? cB : cA);
        r[i] = *reinterpret_cast<const unsigned*>(&v);
    }
}
template <int NB, bool SCALED>
__device__ __forceinline__ unsigned e8_fetch(unsigned u, unsigned tbase, const unsigned* packed) {
    unsigned v;
    asm volatile("{\n\t.reg .pred p;\n\t.reg .u64 ga;\n\t.reg .u32 sa;\n\t"
                 "setp.ge.u32 p, %1, %2;\n\t"
                 "mad.wide.u32 ga, %1, 4, %3;\n\t"
                 "mad.lo.u32 sa, %1, 4, %4;\n\t"
                 "@p ld.global.nc.u32 %0, [ga];\n\t"
                 "@!p ld.shared.u32 %0, [sa];\n\t}"
                 : "=r"(v) : "r"(u), "n"(e8_resident(NB, SCALED)), "l"(packed), "r"(tbase));
    return v;
}

// Block that owns step s when block b owns [b*W/G, (b+1)*W/G); the host keeps W * G below 2^32.
__device__ __forceinline__ int owner_block(unsigned s, unsigned W, unsigned G) {
    unsigned b = (s * G) / W;
    while (b + 1 < G && ((b + 1) * W) / G <= s) ++b;
    while (b > 0 && (b * W) / G > s) --b;
    return static_cast<int>(b);
}

// Adds the partial sums of a row tile in block order, then the corrections; writes y.  Run by `n` threads.
template <int NB, int MAXL>
__device__ __forceinline__ void finish_tile(const RowsArgs<MAXL>& p, const RowsLayer& L, int rt, int tid, int n) {
    const int tile = L.tile0 + rt;
    if (tid == 0) p.counters[tile] = 0u;
    const unsigned s0 = static_cast<unsigned>(L.step0 + rt * L.ns);
    const int first = owner_block(s0, p.W, p.G), last = owner_block(s0 + L.ns - 1, p.W, p.G);
    const size_t slot = static_cast<size_t>(NB) * kTileOut;
    const float* parts = p.partial + (first + tile) * slot;
    const float* corr = L.corr_tile != 0 ? p.partial + (p.G + p.tiles + tile) * slot : nullptr;
    for (int i = tid; i < p.B * (kTileOut / 4); i += n) {
        const int b = i / (kTileOut / 4), q = i % (kTileOut / 4);
        if (rt * kTileRows + (q >> 1) >= L.M) continue;
        const size_t off = static_cast<size_t>(b) * kTileOut + q * 4;
        const int o = rt * kTileOut + q * 4;
        const uint2 graw = __ldg(reinterpret_cast<const uint2*>(L.g + o));
        uint2 braw = make_uint2(0, 0);
        if (L.bias != nullptr) braw = __ldg(reinterpret_cast<const uint2*>(L.bias + o));
        float4 cv = make_float4(0.f, 0.f, 0.f, 0.f);
        if (corr != nullptr) cv = __ldcg(reinterpret_cast<const float4*>(corr + off));
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k = 0; k <= last - first; k += 8) {                     // eight loads in flight
            float4 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
                v[j] = k + j <= last - first ? __ldcg(reinterpret_cast<const float4*>(parts + (k + j) * slot + off)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 8; ++j) { s.x += v[j].x; s.y += v[j].y; s.z += v[j].z; s.w += v[j].w; }
        }
        s.x += cv.x; s.y += cv.y; s.z += cv.z; s.w += cv.w;
        const float2 g01 = __half22float2(*reinterpret_cast<const __half2*>(&graw.x));
        const float2 g23 = __half22float2(*reinterpret_cast<const __half2*>(&graw.y));
        const float2 b01 = __half22float2(*reinterpret_cast<const __half2*>(&braw.x));
        const float2 b23 = __half22float2(*reinterpret_cast<const __half2*>(&braw.y));
        const __half2 o01 = __floats2half2_rn(fmaf(s.x, g01.x, b01.x), fmaf(s.y, g01.y, b01.y));
        const __half2 o23 = __floats2half2_rn(fmaf(s.z, g23.x, b23.x), fmaf(s.w, g23.y, b23.y));
        uint2 ov;
        ov.x = *reinterpret_cast<const unsigned*>(&o01);
        ov.y = *reinterpret_cast<const unsigned*>(&o23);
        *reinterpret_cast<uint2*>(L.y + static_cast<size_t>(b) * 8 * L.M + o) = ov;
    }
}

// `row_max`: bits of max|x| of the four batch rows.
__device__ __forceinline__ bool any_nonfinite(const unsigned* row_max) {
    return max(max(row_max[0], row_max[1]), max(row_max[2], row_max[3])) >= 0x7c00u;
}
// The outputs, in the tiles a block finished, of batch rows with an infinity or a NaN in a layer with group scales.  The
// tensor core multiplies every column by every codeword, a critical block's stand-in and zero coordinates among them, and
// the split would subtract infinities; this is the SIMT kernel's arithmetic, which does neither.  Slow, and rare.
template <int KIND, int MAXL>
__device__ __noinline__ void finish_nonfinite(const RowsArgs<MAXL>& p, const unsigned* tiles, unsigned n_tiles, int tid, const unsigned* row_max) {
    const RowsLayer& L = p.L[0];
    for (int i = tid; i < static_cast<int>(n_tiles) * p.B * kTileOut; i += kRowsThreads) {
        const int b = i / kTileOut % p.B, rt = static_cast<int>(tiles[i / kTileOut / p.B]);
        const int dim = i % 8, row = rt * kTileRows + i % kTileOut / 8;
        if (row >= L.M || row_max[b] < 0x7c00u) continue;
        const __half* x = L.x + static_cast<size_t>(b) * L.N;
        const __half* S = L.S + static_cast<size_t>(row / L.qb_rows) * L.N;
        const __half* table = reinterpret_cast<const __half*>(p.table16);
        int block = __ldg(L.O_row_ptr + row);
        float sum = 0.f;
        for (int k = 0; k < L.N; ++k) {
            const unsigned idx = (static_cast<unsigned>(L.Q[static_cast<size_t>(row) * L.N + k]) & 0xffffu) ^ 0x8000u;
            float v = __half2float(L.h[k]), code;
            if (idx == kMarkerIndex) {
                code = __half2float(L.O_vals[static_cast<size_t>(block++) * 8 + dim]);
            } else {
                v *= __half2float(S[k]);
                code = __half2float(KIND == EPTQ_E8 ? table[static_cast<size_t>(idx) * 8 + dim]
                                                    : table[(((idx >> 7) & 0x180u) | ((dim >= 4 ? idx : idx >> 7) & 127u)) * 4 + dim % 4]);
            }
            sum = fmaf(code, v * __half2float(x[k]), sum);
        }
        const int o = row * 8 + dim;
        L.y[static_cast<size_t>(b) * 8 * L.M + o] =
            __float2half_rn(fmaf(sum, __half2float(L.g[o]), L.bias != nullptr ? __half2float(L.bias[o]) : 0.f));
    }
}

template <int MAXL>
__device__ __forceinline__ bool last_arrival(const RowsArgs<MAXL>& p, const RowsLayer& L, int rt) {
    unsigned ticket;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(ticket) : "l"(p.counters + L.tile0 + rt) : "memory");
    const unsigned s0 = static_cast<unsigned>(L.step0 + rt * L.ns);
    const int n = owner_block(s0 + L.ns - 1, p.W, p.G) - owner_block(s0, p.W, p.G) + 1;
    return ticket == static_cast<unsigned>(n + L.corr_tile) - 1u;
}

// A unit of corrections: 4 Q rows, 8 lanes per row.  `lo`, `hi`: this lane's row in the CSR tables; col, h, O: its first
// critical block, read ahead.
struct CorrUnit {
    int l, qt, lo, hi, col;
    float h;
    uint4 O;
};
template <int MAXL>
__device__ __forceinline__ CorrUnit corr_begin(const RowsArgs<MAXL>& p, int u, int lane) {
    CorrUnit c;
    c.l = 0;
    while (c.l + 1 < p.n_layers && p.L[c.l + 1].corr0 <= u) ++c.l;     // layers without units share their successor's corr0
    const RowsLayer& L = p.L[c.l];
    c.qt = u - L.corr0;
    const int row = c.qt * 4 + (lane >> 3);
    c.lo = c.hi = 0;
    if (row < L.M) { c.lo = __ldg(L.O_row_ptr + row); c.hi = __ldg(L.O_row_ptr + row + 1); }
    c.col = 0; c.h = 0.f; c.O = make_uint4(0, 0, 0, 0);
    const int i = c.lo + (lane & 7);
    if (i < c.hi) {
        c.col = __ldg(L.O_col + i);
        c.O = ldg128(L.O_vals + static_cast<size_t>(i) * 8);
        c.h = __half2float(__ldg(L.h + c.col));
    }
    return c;
}
// Four batch rows at a time; stores the sums and takes the tile's ticket.  Returns whether it was the last.
template <int KIND, int NB, bool SCALED, int MAXL>
__device__ __forceinline__ bool corr_finish(const RowsArgs<MAXL>& p, const CorrUnit& c, int lane) {
    float cstar[4] = {0.f, 0.f, 0.f, 0.f};                     // what the main loop adds for a marker (E8: zero)
    if (KIND == EPTQ_E8D4) {
        const uint2 raw = __ldg(p.table16 + 511);
        const float2 c01 = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
        const float2 c23 = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
        cstar[0] = c01.x; cstar[1] = c01.y; cstar[2] = c23.x; cstar[3] = c23.y;
        if constexpr (SCALED) {
#pragma unroll
            for (int k = 0; k < 4; ++k) cstar[k] = rintf(cstar[k] * (1.f / p.code_unit)) * p.code_unit;
        }
    }
    const RowsLayer& L = p.L[c.l];
    const int rt = c.qt / kCorrPerTile, sub = lane & 7;
    float* dst = p.partial + (static_cast<size_t>(p.G + p.tiles + L.tile0 + rt) * NB) * kTileOut + ((c.qt % kCorrPerTile) * 4 + (lane >> 3)) * 8;
    for (int b0 = 0; b0 < p.B; b0 += 4) {
        float acc[4][8];
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[b][k] = 0.f;
        int col = c.col;
        float hv = c.h;
        uint4 ov = c.O;
        for (int i = c.lo + sub; i < c.hi;) {
            float o8[8], xv[4], sg = 1.f;
            unpack8(ov, o8);
            if (SCALED && KIND == EPTQ_E8D4) sg = __half2float(__ldg(L.S + static_cast<size_t>((c.qt * 4 + (lane >> 3)) / L.qb_rows) * L.N + col));
#pragma unroll
            for (int b = 0; b < 4; ++b)
                xv[b] = b0 + b < p.B ? hv * __half2float(__ldg(L.x + static_cast<size_t>(b0 + b) * L.N + col)) : 0.f;
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int k = 0; k < 8; ++k) acc[b][k] = fmaf(SCALED ? fmaf(-sg, cstar[k & 3], o8[k]) : o8[k] - cstar[k & 3], xv[b], acc[b][k]);
            i += 8;
            if (i < c.hi) {
                col = __ldg(L.O_col + i);
                ov = ldg128(L.O_vals + static_cast<size_t>(i) * 8);
                hv = __half2float(__ldg(L.h + col));
            }
        }
        __syncwarp();
#pragma unroll
        for (int b = 0; b < 4; ++b) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                acc[b][k] += __shfl_xor_sync(0xffffffffu, acc[b][k], 1);
                acc[b][k] += __shfl_xor_sync(0xffffffffu, acc[b][k], 2);
                acc[b][k] += __shfl_xor_sync(0xffffffffu, acc[b][k], 4);
            }
            if (sub == 0 && b0 + b < p.B) {
                float4* d4 = reinterpret_cast<float4*>(dst + static_cast<size_t>(b0 + b) * kTileOut);
                __stcg(d4, make_float4(acc[b][0], acc[b][1], acc[b][2], acc[b][3]));
                __stcg(d4 + 1, make_float4(acc[b][4], acc[b][5], acc[b][6], acc[b][7]));
            }
        }
    }
    __syncwarp();
    return lane == 0 && last_arrival(p, L, rt);
}

// Row tiles whose last ticket went to a unit of corrections of this block, by warp.  With short shares a unit's chain of
// dependent reads ends last, and the one warp that had it took 32 rounds of reads to finish the tile; the block takes two
// (1024 x 4096 E8-D4, shares of four steps: 40.7 -> 16.5 us at 8 rows, 75.0 -> 24.7 at 16).  Not inlined: rare.
template <int NB, int MAXL>
__device__ __noinline__ void finish_for_units(const RowsArgs<MAXL>& p, const unsigned* done, int tid) {
    for (int w = 0; w < kRowsWarps; ++w) {
        const unsigned d = done[w];
        if (d != 0u) finish_tile<NB>(p, p.L[d >> 16 & 0x7fff], d & 0xffff, tid, kRowsThreads);
    }
}

template <int KIND, int NB, int MAXL, bool SCALED>
__global__ void __launch_bounds__(kRowsThreads, 1) gemv_rows_kernel(const __grid_constant__ RowsArgs<MAXL> p) {
    constexpr int RING = ring_steps(NB);
    constexpr int BT = NB == 16 ? 2 : 1;                       // accumulator column tiles
    // Fragment buffer: [16-column half ks][fp16 part, remainder][row][columns 8t + 4ks .. +3 for t = 0..3] fp16, so
    // that a warp's 64-bit reads of one half are contiguous.
    constexpr unsigned kLoPlane = NB * 32;                     // bytes from a row's fp16 parts to its remainders
    constexpr unsigned kHalf = NB * 64;                        // bytes between the halves
    constexpr unsigned kBuf = NB * 128;                        // one fragment buffer of a column group
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned base = static_cast<unsigned>(__cvta_generic_to_shared(smem_raw));     // 0x400: the first KB is reserved
    if (base != 0x400u) {                                      // the table address is part of the lookup arithmetic
        if (tid == 0) atomicExch(reinterpret_cast<int*>(p.counters) + (kMaxCounters - 1), static_cast<int>(EPTQ_ERR_LAUNCH));
        return;
    }
    unsigned* const flag = reinterpret_cast<unsigned*>(smem_raw + area_bytes(NB, SCALED));
    unsigned* const row_max = flag + 4;                        // group scales: bits of max|x| of the four batch rows
    unsigned* const finished = flag + 32;                      // group scales: flag[1] row tiles that this block finished
    auto fill_table = [&]() {
        if constexpr (KIND == EPTQ_E8) {
            const unsigned dst0 = base + e8_table_offset(NB, SCALED);
            const char* src0 = reinterpret_cast<const char*>(p.packed);
            for (unsigned off = tid * 16u; off < e8_resident(NB, SCALED) * 4u; off += kRowsThreads * 16u)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst0 + off), "l"(src0 + off) : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
        } else {
            // entry order follows the raw stored bits (true index ^ 0x100 on 9 bits), 16 copies of 8 bytes per entry
            unsigned char* tab = smem_raw + (kRowsTableAddr - base);
            static_assert(kRowsThreads == 512, "one table entry per thread");
            uint2 v = __ldg(p.table16 + (tid ^ 0x100));
            if constexpr (SCALED) { const float inv = 1.f / p.code_unit; v.x = lattice2(v.x, inv); v.y = lattice2(v.y, inv); }
            const uint4 vv = make_uint4(v.x, v.y, v.x, v.y);
    #pragma unroll
            for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(tab + tid * 128 + ((c + tid) & 7) * 16) = vv;
        }
    };
    // Layers with group scales ran in plain stream order on the SIMT kernel, so nothing of theirs is read before the wait:
    // weights that the previous kernel writes are seen.  (The other decode kernels read weights ahead of it and state so.)
    // The next kernel is let in behind it for the same reason.  The codebook, made once for all layers, comes ahead.
    if constexpr (SCALED) {
        if (tid < 4) row_max[tid] = 0u;
        if (tid == 0) flag[1] = 0u;
        fill_table();
        __syncthreads();
        asm volatile("griddepcontrol.wait;" ::: "memory");
    }
    asm volatile("griddepcontrol.launch_dependents;");

    const int g = lane >> 2, t = lane & 3;
    const int kq = warp >> 2, rg = warp & 3, ctid = tid & 127;
    const unsigned s_begin = (static_cast<unsigned>(blockIdx.x) * p.W) / p.G;
    const unsigned s_end = ((static_cast<unsigned>(blockIdx.x) + 1u) * p.W) / p.G;

    // A column group's position: row tile `rt` of layer `l`, its next step k, the end of the block's share of the
    // tile.  Past the last step l = n_layers.
    struct Pos { int l, rt; unsigned tile_s0; int k, kend; };
    auto settle = [&](Pos& c) {                                // move on to the tile that has the group's next step
        while (c.l < p.n_layers && c.k >= c.kend) {
            c.tile_s0 += p.L[c.l].ns;
            if (++c.rt == p.L[c.l].row_tiles) { c.rt = 0; ++c.l; }
            if (c.tile_s0 >= s_end) { c.l = p.n_layers; return; }
            c.kend = min(p.L[c.l].ns, static_cast<int>(s_end - c.tile_s0));
            c.k = kq;
        }
    };
    Pos cur;
    {
        int l = 0;
        while (l + 1 < p.n_layers && static_cast<unsigned>(p.L[l + 1].step0) <= s_begin) ++l;
        const unsigned local = s_begin - p.L[l].step0, ns = p.L[l].ns;
        cur.l = l;
        cur.rt = static_cast<int>(local / ns);
        cur.tile_s0 = p.L[l].step0 + cur.rt * ns;
        cur.k = static_cast<int>(s_begin - cur.tile_s0) + kq;
        cur.kend = min(static_cast<int>(ns), static_cast<int>(s_end - cur.tile_s0));
    }
    Pos pf = cur;
    settle(pf);
    // prefetch pointers of the position: Q row of this lane, x and h columns this thread converts
    static_assert(!SCALED || NB == 4, "group scales run in passes of four rows");
    constexpr int XC = NB == 16 || SCALED ? 4 : NB == 8 ? 2 : 1;         // columns converted per thread
    const int xtid = SCALED ? lane : ctid;
    const int xrow = xtid / (32 / XC), xcol = (xtid % (32 / XC)) * XC;
    const bool xlive = xrow < p.B;
    struct Raw { uint4 q; unsigned x[(XC + 1) / 2], h[(XC + 1) / 2], s[SCALED ? 2 : 1]; };
    const int16_t* qp = nullptr;
    const __half *xp = nullptr, *hp = nullptr, *sp = nullptr;
    auto place = [&]() {
        if (pf.l >= p.n_layers) return;
        const RowsLayer& L = p.L[pf.l];
        const int row = min(pf.rt * kTileRows + rg * 8 + g, L.M - 1);
        qp = L.Q + static_cast<size_t>(row) * L.N + pf.k * 32 + 8 * t;
        xp = L.x + static_cast<size_t>(xlive ? xrow : 0) * L.N + pf.k * 32 + xcol;
        hp = L.h + pf.k * 32 + xcol;
        if (SCALED) sp = L.S + static_cast<size_t>(min(pf.rt * kTileRows + rg * 8, L.M - 1) / L.qb_rows) * L.N + pf.k * 32 + xcol;
    };
    auto next = [&]() {
        pf.k += kColGroups;
        if (pf.k < pf.kend) { qp += 32 * kColGroups; xp += 32 * kColGroups; hp += 32 * kColGroups; if (SCALED) sp += 32 * kColGroups; }
        else { settle(pf); place(); }
    };
    auto load_cols = [&](const __half* src, unsigned (&v)[(XC + 1) / 2]) {
        if constexpr (XC == 4) { const uint2 w = __ldg(reinterpret_cast<const uint2*>(src)); v[0] = w.x; v[1] = w.y; }
        else if constexpr (XC == 2) v[0] = __ldg(reinterpret_cast<const unsigned*>(src));
        else v[0] = __half_as_ushort(__ldg(src));
    };
    Raw ring[RING];
    place();
    Pos pf0 = pf;
#pragma unroll
    for (int i = 0; i < RING; ++i) {                      // weights do not depend on the previous kernel
        ring[i].q = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int e = 0; e < (XC + 1) / 2; ++e) { ring[i].x[e] = 0u; ring[i].h[e] = 0u; }
#pragma unroll
        for (int e = 0; e < (SCALED ? 2 : 1); ++e) ring[i].s[e] = 0u;
        if (pf.l < p.n_layers) { ring[i].q = ldg_once(qp); load_cols(hp, ring[i].h); if constexpr (SCALED) load_cols(sp, ring[i].s); next(); }
    }

    if constexpr (!SCALED) fill_table();
    // group scales: the batch rows' values whose largest is sought, this thread's first 8 columns of each
    uint4 part[SCALED ? 4 : 1];
    const bool has_part = SCALED && tid * 8 < p.L[0].N;
    auto row_cols = [&](int b, int col) { return ldg128(p.L[0].x + static_cast<size_t>(b) * p.L[0].N + col); };
    if constexpr (SCALED) {
#pragma unroll
        for (int b = 0; b < 4; ++b) part[b] = has_part && b < p.B ? row_cols(b, tid * 8) : make_uint4(0, 0, 0, 0);
    }
    const int unit0 = warp * gridDim.x + blockIdx.x, unit_step = gridDim.x * kRowsWarps;
    CorrUnit corr = {};
    if (unit0 < p.corr_units) corr = corr_begin(p, unit0, lane);
    if constexpr (!SCALED) asm volatile("griddepcontrol.wait;" ::: "memory");
    {
        const Pos keep = pf;
        const int16_t* kq_ = qp; const __half *kx = xp, *kh = hp, *ks = sp;
        pf = pf0;
        place();
#pragma unroll
        for (int i = 0; i < RING; ++i)
            if (pf.l < p.n_layers) { if (xlive) load_cols(xp, ring[i].x); next(); }
        pf = keep; qp = kq_; xp = kx; hp = kh; sp = ks;
    }

    if constexpr (SCALED) {
        auto largest = [](const uint4& v) {
            return __vmaxu2(__vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu), __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu));
        };
        unsigned top[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) top[b] = largest(part[b]);
        for (int i = (tid + kRowsThreads) * 8; i < p.L[0].N; i += kRowsThreads * 8)
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if (b < p.B) top[b] = __vmaxu2(top[b], largest(row_cols(b, i)));
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const unsigned m = __reduce_max_sync(0xffffffffu, max(top[b] & 0xffffu, top[b] >> 16));
            if (lane == 0) atomicMax(row_max + b, m);
        }
        __syncthreads();                                       // a unit of corrections may finish a tile from here on
    }

    // The first unit's ticket is looked at behind the main loop (its round trip costs nothing there).
    bool corr_last = false;
    if (unit0 < p.corr_units) corr_last = corr_finish<KIND, NB, SCALED>(p, corr, lane);
    const unsigned corr_tile = 1u << 31 | static_cast<unsigned>(corr.l) << 16 | static_cast<unsigned>(corr.qt / kCorrPerTile);
    for (int u = unit0 + unit_step; !SCALED && u < p.corr_units; u += unit_step) {
        const CorrUnit c = corr_begin(p, u, lane);
        const bool last = corr_finish<KIND, NB, SCALED>(p, c, lane);
        if (__any_sync(0xffffffffu, last)) finish_tile<NB>(p, p.L[c.l], c.qt / kCorrPerTile, lane, 32);
        __syncwarp();
    }
    if constexpr (KIND == EPTQ_E8) asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                           // table complete

    const unsigned area = base;                                // fragment buffers / sums over column groups
    unsigned char* const area_p = smem_raw;
    const unsigned my_buf = (SCALED ? warp : kq) * 2 * kBuf;
    const unsigned wr_off = my_buf + ((xcol >> 2) & 1) * kHalf + xrow * 32 + (xcol >> 3) * 8 + (xcol & 3) * 2;
    const unsigned rd_addr = area + my_buf + g * 32 + t * 8;
    // this thread's rows: the one it converts, and the two it stores (behind `lo` of the same row pair where t >= 2)
    float row_up = 1.f, row_down[2] = {1.f, 1.f};
    if constexpr (SCALED) {
        row_up = exp2i(kRowTop - row_exponent(row_max[xrow]));
#pragma unroll
        for (int e = 0; e < 2; ++e)
            row_down[e] = exp2i(row_exponent(row_max[2 * (t & 1) + e]) - kRowTop) * (t >= 2 ? 1.f / kLoScale : 1.f);
    }
    const unsigned lane_tab = 8u * (lane & 15) | kRowsTableAddr;
    const unsigned tbase = base + e8_table_offset(NB, SCALED);

    float acc[BT][4][4];
#pragma unroll
    for (int i = 0; i < BT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.f;
    unsigned par = 0;

    // End of the block's share of a row tile: sum over the column groups, partial sums to scratch, ticket.
    auto flush = [&]() {
        const RowsLayer& L = p.L[cur.l];
        float* red = reinterpret_cast<float*>(area_p) + ctid;
        __syncthreads();             // fragment buffers are free
#pragma unroll
        for (int r = kColGroups - 1; r >= 0; --r) {
            if (kq == r) {
#pragma unroll
                for (int i = 0; i < BT; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            float v = acc[i][j][c];
                            if (r < kColGroups - 1) v += red[((i * 4 + j) * 4 + c) * 128];
                            if (r > 0) red[((i * 4 + j) * 4 + c) * 128] = v; else acc[i][j][c] = v;
                        }
            }
            if (r > 0) __syncthreads();
        }
        if (kq == 0) {
            float* dst = p.partial + (static_cast<size_t>(blockIdx.x + L.tile0 + cur.rt) * NB) * kTileOut + (rg * 8 + g) * 8;
#pragma unroll
            for (int i = 0; i < BT; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {                  // batch rows 2t and 2t+1 of the column tile
                    const float inv = SCALED ? L.x_inv_scale * row_down[e] : L.x_inv_scale;
                    float v[8];
#pragma unroll
                    for (int j = 0; j < 4; ++j) { v[2 * j] = acc[i][j][e] * inv; v[2 * j + 1] = acc[i][j][2 + e] * inv; }
                    if constexpr (NB == 4) {                   // columns 4..7 hold the remainders
#pragma unroll
                        for (int k = 0; k < 8; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], 2);
                    }
                    const int b = i * 8 + 2 * t + e;
                    if ((NB > 4 || t < 2) && b < p.B) {
                        float4* d4 = reinterpret_cast<float4*>(dst + static_cast<size_t>(b) * kTileOut);
                        __stcg(d4, make_float4(v[0], v[1], v[2], v[3]));
                        __stcg(d4 + 1, make_float4(v[4], v[5], v[6], v[7]));
                    }
                }
        }
#pragma unroll
        for (int i = 0; i < BT; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.f;
        __syncthreads();
        if (tid == 0) *flag = last_arrival(p, L, cur.rt) ? 1u : 0u;
        __syncthreads();
        if (*flag != 0u) {
            finish_tile<NB>(p, L, cur.rt, tid, kRowsThreads);
            if constexpr (SCALED)
                if (tid == 0) finished[flag[1]++] = cur.rt;
        }
    };
    // Segment after the current one; false when the block's share is done.
    auto next_segment = [&]() {
        cur.tile_s0 += p.L[cur.l].ns;
        if (cur.tile_s0 >= s_end) return false;
        if (++cur.rt == p.L[cur.l].row_tiles) { cur.rt = 0; ++cur.l; }
        cur.kend = min(p.L[cur.l].ns, static_cast<int>(s_end - cur.tile_s0));
        cur.k = kq;
        return true;
    };

    // E8 lookups run one step ahead: a seventh of them goes to L2, and waiting for those was half of a step (gate/up of a
    // 7B model: 48.9 -> 36.1 us at 4 rows, 57.4 -> 37.9 at 8, 64.5 -> 48.9 at 16).
    unsigned ent[8];
    auto lookup = [&](const uint4& q, unsigned (&e)[8]) {
        const unsigned w[4] = {q.x ^ 0x80008000u, q.y ^ 0x80008000u, q.z ^ 0x80008000u, q.w ^ 0x80008000u};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            e[2 * k] = e8_fetch<NB, SCALED>(w[k] & 0xFFFFu, tbase, p.packed);
            e[2 * k + 1] = e8_fetch<NB, SCALED>(w[k] >> 16, tbase, p.packed);
        }
    };
    if constexpr (KIND == EPTQ_E8) lookup(ring[0].q, ent);

    auto step = [&](Raw& in, const Raw& following) {
        const uint4 q = in.q;
        const unsigned qw[4] = {q.x, q.y, q.z, q.w};
        {
            const float sc = SCALED ? p.L[cur.l].x_scale * row_up : p.L[cur.l].x_scale;
            __half hi[XC], lo[XC];
#pragma unroll
            for (int e = 0; e < XC; ++e) {
                const unsigned short xb = static_cast<unsigned short>(in.x[e >> 1] >> (16 * (e & 1)));
                const unsigned short hb = static_cast<unsigned short>(in.h[e >> 1] >> (16 * (e & 1)));
                float hx = __half2float(__ushort_as_half(hb)) * sc;
                const float xv = __half2float(__ushort_as_half(xb));
                if constexpr (SCALED) {                        // h * S is exact: 22 bits
                    hx *= __half2float(__ushort_as_half(static_cast<unsigned short>(in.s[e >> 1] >> (16 * (e & 1)))));
                    split_product(xv, hx, hi[e], lo[e]);
                } else {
                    split_half(xv * hx, hi[e], lo[e]);
                }
            }
            unsigned char* w = area_p + wr_off + par * kBuf;
            if constexpr (XC == 4) {
                *reinterpret_cast<uint2*>(w) = *reinterpret_cast<const uint2*>(hi);
                *reinterpret_cast<uint2*>(w + kLoPlane) = *reinterpret_cast<const uint2*>(lo);
            } else if constexpr (XC == 2) {
                *reinterpret_cast<unsigned*>(w) = *reinterpret_cast<const unsigned*>(hi);
                *reinterpret_cast<unsigned*>(w + kLoPlane) = *reinterpret_cast<const unsigned*>(lo);
            } else {
                *reinterpret_cast<__half*>(w) = hi[0];
                *reinterpret_cast<__half*>(w + kLoPlane) = lo[0];
            }
        }
        if (pf.l < p.n_layers) {
            in.q = ldg_once(qp);
            load_cols(hp, in.h);
            if constexpr (SCALED) load_cols(sp, in.s);
            if (xlive) load_cols(xp, in.x);
            next();
        }
        if constexpr (SCALED) __syncwarp();
        else asm volatile("bar.sync %0, 128;" :: "r"(2 + kq) : "memory");     // the step's fragments are complete
        const unsigned rd = rd_addr + par * kBuf;
        par ^= 1;
        unsigned ahead[8];
        if constexpr (KIND == EPTQ_E8) lookup(following.q, ahead);       // behind the last step: an earlier step's indices
        constexpr int PLANES = NB == 4 ? 1 : 2 * BT;           // column tiles: fp16 parts, then remainders
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {                       // 16 columns: four of this lane's eight
            uint2 bf[PLANES];
#pragma unroll
            for (int i = 0; i < PLANES; ++i) bf[i] = lds64(rd + ks * kHalf + (i % BT) * 256 + (i / BT) * kLoPlane);
            unsigned c[4][4];                                  // [column][dim pair]
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if constexpr (KIND == EPTQ_E8) {
                    e8_entry(ent[4 * ks + e], c[e]);
                } else {
                    const unsigned v = (e & 1) ? qw[2 * ks + (e >> 1)] >> 16 : qw[2 * ks + (e >> 1)];
                    const uint2 a = lds64((v & 0xFF80u) | lane_tab);
                    const uint2 b = lds64(((v << 7) & 0x3F80u) | ((v & 0xC000u) | lane_tab));
                    c[e][0] = a.x; c[e][1] = a.y; c[e][2] = b.x; c[e][3] = b.y;
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const unsigned a[4] = {lo_halves(c[0][j], c[1][j]), hi_halves(c[0][j], c[1][j]),
                                       lo_halves(c[2][j], c[3][j]), hi_halves(c[2][j], c[3][j])};
#pragma unroll
                for (int i = 0; i < PLANES; ++i) mma(acc[i % BT][j], a, bf[i].x, bf[i].y);
            }
        }
        if constexpr (KIND == EPTQ_E8) {
#pragma unroll
            for (int e = 0; e < 8; ++e) ent[e] = ahead[e];
        }
    };

    for (bool more = true; more;) {
#pragma unroll
        for (int i = 0; i < RING; ++i) {
            while (more && cur.k >= cur.kend) { flush(); more = next_segment(); }
            if (!more) break;
            step(ring[i], ring[(i + 1) % RING]);
            cur.k += kColGroups;
        }
    }
    if (__syncthreads_or(corr_last)) {
        if (lane == 0) flag[16 + warp] = corr_last ? corr_tile : 0u;
        __syncthreads();
        finish_for_units<NB>(p, flag + 16, tid);
        if constexpr (SCALED) {
            if (lane == 0 && corr_last) finished[atomicAdd(flag + 1, 1u)] = corr_tile & 0xffffu;
            __syncthreads();
        }
    }
    if constexpr (SCALED)                                      // behind a barrier: the list and the outputs are written
        if (any_nonfinite(row_max)) finish_nonfinite<KIND>(p, finished, flag[1], tid, row_max);
}

struct RowsPlan {
    unsigned W = 0;
    int G = 0, tiles = 0, corr_units = 0;
    size_t bytes = 0;
};

int rows_of(int B) { return B <= 4 ? 4 : B <= 8 ? 8 : 16; }

bool plan_rows(const EptqLayer* layers, int n, int B, int n_sms, RowsPlan& plan) {
    if (n < 1 || n > kRowsMaxLayers || n_sms < 1) return false;
    long long W = 0, tiles = 0;
    for (int i = 0; i < n; ++i) {
        const long long rt = (layers[i].M + kTileRows - 1) / kTileRows;
        tiles += rt;
        W += rt * (layers[i].N / 32);
    }
    if (W < 1 || tiles > kMaxCounters - 1) return false;
    // A block has at least one step per column group, or the sums over blocks cost more than they spread.
    const long long G = W / kColGroups < n_sms ? (W / kColGroups > 0 ? W / kColGroups : 1) : n_sms;
    if (W * G >= (1LL << 32)) return false;
    plan.W = static_cast<unsigned>(W);
    plan.G = static_cast<int>(G);
    plan.tiles = static_cast<int>(tiles);
    plan.bytes = kPartialOffset + static_cast<size_t>(G + 2 * tiles) * rows_of(B) * kTileOut * sizeof(float);
    return true;
}

template <int KIND, int NB, bool SCALED = false, int MAXL>
int launch_kernel(const RowsArgs<MAXL>& a, int n_sms, cudaStream_t stream) {
    constexpr int smem = KIND == EPTQ_E8 ? kRowsSmemE8 : kRowsSmemD4;
    static std::atomic<bool> attr_done[64];       // setting the attribute twice is harmless; the flag itself must not race
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return EPTQ_ERR_LAUNCH;
    if (!attr_done[dev]) {
        if (cudaFuncSetAttribute(gemv_rows_kernel<KIND, NB, MAXL, SCALED>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return EPTQ_ERR_LAUNCH;
        attr_done[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_sms);
    cfg.blockDim = dim3(kRowsThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, gemv_rows_kernel<KIND, NB, MAXL, SCALED>, a);
    count_launch(EPTQ_KERNEL_GEMV_GROUP);
    return err == cudaSuccess ? EPTQ_OK : EPTQ_ERR_LAUNCH;
}

template <int MAXL>
int launch_sized(const RowsPlan& plan, const EptqLayer* layers, int n, const uint16_t* const* xs, uint16_t* const* ys, int B,
                 void* workspace, cudaStream_t stream) {
    const bool e8 = layers[0].quantizer == EPTQ_E8;
    RowsArgs<MAXL> a;
    a.table16 = reinterpret_cast<const uint2*>(layers[0].table16);
    a.packed = e8 ? layers[0].table_packed : nullptr;
    a.counters = reinterpret_cast<unsigned*>(workspace);
    a.partial = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + kPartialOffset);
    a.code_unit = layers[0].table8_scale;
    a.W = plan.W; a.G = plan.G; a.tiles = plan.tiles;
    a.n_layers = n;
    a.B = B;
    int step0 = 0, tile0 = 0, corr0 = 0;
    for (int i = 0; i < n; ++i) {
        const EptqLayer& L = layers[i];
        RowsLayer& R = a.L[i];
        if (xs[i] == nullptr || ys[i] == nullptr) return EPTQ_ERR_NULL;
        if (!aligned16(xs[i]) || !aligned16(ys[i])) return EPTQ_ERR_ALIGN;
        R.Q = L.Q;
        R.g = reinterpret_cast<const __half*>(L.g);
        R.h = reinterpret_cast<const __half*>(L.h);
        R.x = reinterpret_cast<const __half*>(xs[i]);
        R.O_vals = reinterpret_cast<const __half*>(L.O_vals);
        R.O_col = L.O_col;
        R.O_row_ptr = L.O_row_ptr;
        R.bias = reinterpret_cast<const __half*>(L.bias);
        R.y = reinterpret_cast<__half*>(ys[i]);
        R.M = L.M; R.N = L.N;
        R.ns = L.N / 32;
        R.row_tiles = (L.M + kTileRows - 1) / kTileRows;
        R.step0 = step0; R.tile0 = tile0; R.corr0 = corr0;
        R.S = reinterpret_cast<const __half*>(L.S_group);
        R.qb_rows = L.S_group != nullptr ? L.qb_size / 8 : 0;
        R.corr_tile = L.n_masked != 0 ? kCorrPerTile : 0;      // -1 (count unknown): the row pointers carry it
        int e = 0;
        std::frexp(std::fabs(L.h_absmax), &e);            // h_absmax = m * 2^e, m in [0.5, 1)  =>  2^-e <= 1/h_absmax
        R.x_scale = std::ldexp(1.0f, -e);
        R.x_inv_scale = std::ldexp(1.0f, e) * (e8 ? L.table_packed_scale : L.S_group != nullptr ? L.table8_scale : 1.0f);
        step0 += R.row_tiles * R.ns;
        tile0 += R.row_tiles;
        corr0 += R.row_tiles * R.corr_tile;
    }
    a.corr_units = corr0;
    if constexpr (MAXL == kRowsFewLayers)
        if (layers[0].S_group != nullptr) return e8 ? launch_kernel<EPTQ_E8, 4, true>(a, plan.G, stream) : launch_kernel<EPTQ_E8D4, 4, true>(a, plan.G, stream);
    switch (rows_of(B)) {
        case 4: return e8 ? launch_kernel<EPTQ_E8, 4>(a, plan.G, stream) : launch_kernel<EPTQ_E8D4, 4>(a, plan.G, stream);
        case 8: return e8 ? launch_kernel<EPTQ_E8, 8>(a, plan.G, stream) : launch_kernel<EPTQ_E8D4, 8>(a, plan.G, stream);
        default: return e8 ? launch_kernel<EPTQ_E8, 16>(a, plan.G, stream) : launch_kernel<EPTQ_E8D4, 16>(a, plan.G, stream);
    }
}

}  // namespace

// Scratch of the one-pass launch, 0 if the shapes do not fit its plan.  The layers are ones group_gemv_supported takes.
size_t rows_workspace_bytes(const EptqLayer* layers, int n, int B, int n_sms) {
    RowsPlan plan;
    return plan_rows(layers, n, B, n_sms, plan) ? (plan.bytes + 255) & ~static_cast<size_t>(255) : 0;
}

int launch_gemv_rows(const EptqLayer* layers, int n, const uint16_t* const* xs, uint16_t* const* ys, int B, int n_sms,
                     void* workspace, cudaStream_t stream) {
    RowsPlan plan;
    if (!plan_rows(layers, n, B, n_sms, plan)) return EPTQ_ERR_UNSUPPORTED;
    return n <= kRowsFewLayers ? launch_sized<kRowsFewLayers>(plan, layers, n, xs, ys, B, workspace, stream)
                               : launch_sized<kRowsMaxLayers>(plan, layers, n, xs, ys, B, workspace, stream);
}

// Where passes of four rows beat the SIMT kernel.  They cost a fixed part (table, row maxima, partial sums) once per four
// rows, that one its arithmetic per row, and few row tiles leave blocks with short shares.  E8-D4 / E8, scales per 128 rows,
// SIMT against this, us: 4096 x 4096 (2.1 M indices) 1 row 12.0, 15.5 / 14.3, 17.6; 4 rows 19.7, 15.8 / 22.9, 18.1; 8 rows
// 39.7, 31.1 / 51.8, 35.6; 16 rows 51.5, 62.0 / 69.3, 70.7.  5120 x 5120 (3.3 M) 1 row 21.1, 17.6 / 23.6, 20.2; 16 rows 74.1,
// 70.2 / 107, 81.  Few tiles: 2048 x 8192 (2.1 M) 4 rows 19.7, 17.6 / 23.0, 19.2; 12 rows 50.2, 52.1; 2048 x 14336 (3.7 M) 1
// row 17.3, 20.6 / 21.3, 23.1; 2432 x 14336 (4.4 M) 1 row 23.3, 21.3 / 24.5, 24.1; 1024 x 16384 (2.1 M) 4 rows 16.3, 23.4.
static bool rows_scaled_faster(long long M, long long N, int B) {
    if (M >= 288 && M * N >= 3LL << 20) return true;
    return B >= 3 && B <= 8 && M >= 256 && M * N >= 2LL << 20;
}

// One layer with group scales that are constant over 64 outputs; -h_absmax = max|h| * max|S_group| bounds x*h*S.
bool rows_scaled_supported(const EptqLayer& L, int B) {
    RowsPlan plan;                               // one unit of corrections per warp at most
    return rows_scaled_faster(L.M, L.N, B) && plan_rows(&L, 1, 4, kSms, plan) && plan.tiles * kCorrPerTile <= plan.G * kRowsWarps && L.S_group != nullptr && L.qb_size > 0 && (L.qb_size % 64) == 0 && L.h_absmax < 0.f && std::isfinite(L.h_absmax) && B >= 1 && B <= kGemmMinBatch &&
           (L.N % 32) == 0 && aligned16(L.Q) && aligned16(L.h) && aligned16(L.g) && aligned16(L.S_group) &&
           (L.bias == nullptr || aligned16(L.bias)) && (L.n_masked == 0 || aligned16(L.O_vals)) &&
           (L.quantizer == EPTQ_E8 ? L.table_packed != nullptr && aligned16(L.table_packed) && L.table_packed_scale > 0.f
                                   : L.table16 != nullptr && aligned16(L.table16) && L.table8 != nullptr && L.table8_scale > 0.f);
}

// Passes of four rows, the scratch of rows_workspace_bytes(&L, 1, 4, n_sms).
int launch_gemv_rows_scaled(const EptqLayer& L, const uint16_t* x, uint16_t* y, int B, int n_sms, void* workspace, cudaStream_t stream) {
    RowsPlan plan;
    if (!plan_rows(&L, 1, 4, n_sms, plan)) return EPTQ_ERR_UNSUPPORTED;
    for (int b = 0; b < B; b += 4) {
        const uint16_t* xs[1] = {x + static_cast<size_t>(b) * L.N};
        uint16_t* ys[1] = {y + static_cast<size_t>(b) * 8 * L.M};
        const int st = launch_sized<kRowsFewLayers>(plan, &L, 1, xs, ys, B - b < 4 ? B - b : 4, workspace, stream);
        if (st != EPTQ_OK) return st;
    }
    return EPTQ_OK;
}

}  // namespace eptq
