// int8 x int8 -> int32 contractions on the 5th-generation tensor cores (sm_100a):
// GEMM, implicit-GEMM convolution forward / error-backward, and convolution weight gradient.
//
// Common structure (one CTA per SM):
//   warp 0      TMA producer: cp.async.bulk.tensor into 128-byte-swizzled shared-memory stages
//   warp 1      allocates tensor memory, issues tcgen05.mma.kind::i8 (one lane), frees TMEM
//   warps 2..   epilogue (4, 8 or 16 warps): tcgen05.ld the int32 accumulators, reduce max|acc|, store
// Stages hand over through mbarriers (TMA complete_tx -> MMA, tcgen05.commit -> producer);
// accumulators are double-buffered in TMEM so the epilogue of one tile overlaps the main loop
// of the next.  All waits are bounded (ptx.cuh).
//
// Operand layouts in shared memory.  Every operand tile is rows of 128 bytes, 8-row groups of
// 1024 bytes, 128-byte swizzle -- exactly what a TMA box with a 128-byte inner extent writes.
//   K-major  (reduction index contiguous in memory): row = M/N index, 128 bytes = 128 reduction
//            elements; one MMA (K = 32) advances the descriptor by 32 bytes.
//   MN-major (M/N index contiguous, e.g. [pixels][channels] read as channels x pixels): row =
//            reduction index, 128 bytes = 128 M/N elements; one MMA advances by 32 rows = 4096 B;
//            a second 128-wide panel sits `rows * 128` bytes further (leading byte offset).
#include <cuda.h>
#include <cuda_runtime.h>
#include <atomic>
#include <cstdint>
#include <cstdio>

#include "../../include/niti_b200.h"
#include "internal.h"
#include "ptx.cuh"
#include "requant.cuh"
#include "grid_barrier.cuh"

namespace niti {
#ifdef NITI_PARKED_TIMING
__device__ unsigned long long g_dbg_stamps[32];
#define PARK_STAMP(i) do { if (blockIdx.x == 0) g_dbg_stamps[i] = global_timer_ns(); } while (0)
#define DBG_CLK(v) const long long v = clock64()
#define DBG_DECL long long dbg_acc[4] = {0, 0, 0, 0}
#define DBG_ACC(i, d) dbg_acc[(i) & 3] += (d)
#define DBG_OUT(base) do { if (blockIdx.x == 0 && (threadIdx.x & 31) == 0) for (int q_ = 0; q_ < 4; ++q_) g_dbg_stamps[(base) + q_] = dbg_acc[q_]; } while (0)
#else
#define DBG_CLK(v) do { } while (0)
#define DBG_DECL do { } while (0)
#define DBG_ACC(i, d) do { } while (0)
#define DBG_OUT(base) do { } while (0)
#define PARK_STAMP(i) do { } while (0)
#endif

// Pin a value in a register: kernel parameters live in the constant bank, and under register pressure the compiler
// re-reads them at every use; in the producer / MMA loops each such load sits on one warp's serial critical path.
__device__ __forceinline__ int keep_reg(int v) { asm volatile("" : "+r"(v)); return v; }

constexpr int BLOCK_M = 128;
constexpr int ROW_BYTES = 128;               // bytes per shared-memory row of an operand tile
constexpr int PANEL_BYTES = 128 * ROW_BYTES; // one 128-row operand panel
constexpr int UMMA_THREADS = 192;
constexpr uint32_t SWIZZLE_128B_CODE = 2;
constexpr uint32_t SWIZZLE_64B_CODE = 4;
constexpr uint32_t SWIZZLE_32B_CODE = 6;
constexpr int EPI_CHUNK_BYTES = 128 * 32 * 4;  // 128 rows x 32 int32 columns, one TMA store box
constexpr int EPI_BARRIER = 1;                 // named barrier of the 128 epilogue threads

// Epilogue staging: each thread owns one accumulator row of 32 int32 (128 bytes) and writes it as
// eight 16-byte chunks at the 128-byte-swizzled position the TMA store expects (chunk ^ row%8);
// that placement is also free of shared-memory bank conflicts.
__device__ __forceinline__ void stage_row(uint32_t buf, int row, const uint32_t (&v)[32]) {
    const uint32_t base = buf + static_cast<uint32_t>(row) * 128u;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        st_shared_v4(base + (static_cast<uint32_t>(j ^ (row & 7)) << 4), v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
}

// ------------------------------------------------------------------------------------------------
// GEMM / convolution forward / error-backward
// ------------------------------------------------------------------------------------------------
// Division of a non-negative int by a divisor fixed at launch: q = (umulhi(mul, n) + n) >> shift with
// shift = ceil(log2 d) and mul = floor(2^32 (2^shift - d) / d) + 1, exact for 0 <= n < 2^31.  The tile loops turn a
// tile number into coordinates once per tile; eight hardware-less 32-bit divisions there were a quarter of an epilogue.
struct FastDiv { unsigned mul, shift; int d; };
static FastDiv make_fastdiv(int d) {
    FastDiv f{1u, 0u, d < 1 ? 1 : d};
    while ((1ull << f.shift) < static_cast<unsigned long long>(f.d)) ++f.shift;
    f.mul = static_cast<unsigned>(((1ull << 32) * ((1ull << f.shift) - static_cast<unsigned long long>(f.d))) / static_cast<unsigned long long>(f.d) + 1ull);
    return f;
}
__device__ __forceinline__ int fdiv(int n, const FastDiv& f) {
    return static_cast<int>((__umulhi(f.mul, static_cast<unsigned>(n)) + static_cast<unsigned>(n)) >> f.shift);
}

struct GemmParams {
    int conv;              // 0: plain GEMM, 1: implicit-GEMM convolution (A tile = 4-D box of pixels)
    int M, N;              // output rows (GEMM rows or pixels) and columns
    int num_kb;            // reduction blocks of the whole problem
    int splits;            // split-K: each output tile is produced `splits` times over disjoint reduction ranges
    int m_tiles, n_tiles;
    int a_mn, b_mn;        // operand majors (0 = K-major, 1 = MN-major)
    int a_bytes;           // bytes one A stage receives from TMA
    int mma_n;             // columns of one MMA: the tile's, or of the only column tile those that exist (in sixteens)
    int b_bytes;           // bytes of one tap's B tile (of this CTA's half of it): fewer than the tile where the box is lower
    // Operands of 32-byte rows that lie in memory as the MMA reads them (32-byte swizzle: see patch_half), loaded with
    // one untiled bulk copy instead of a box of 128 rows.  1: A [M][32] and B [N][32], one reduction block;
    // 2: B [reduction][32] as 32 MN-major columns.
    int rows32;
    const int8_t* a32; const int8_t* b32;
    int K;                 // rows32 == 2: reduction length
    // convolution geometry
    int H, W, S, pad, Nimg;
    int flip;              // 1: error-backward, taps are read mirrored (offset pad - r instead of r - pad)
    int tapstride;         // elements between consecutive taps in a filter row
    int BW, BH, BI;        // pixels of one tile along w, h and images; BW*BH*BI <= 128
    int tiles_w, tiles_h;
    FastDiv fd_mn, fd_n, fd_tw, fd_th;  // by m_tiles * n_tiles, n_tiles, tiles_w, tiles_h (set by finish_params)
    int cblocks;           // 128-byte blocks per tap: ceil(reduction channels / 128)
    int red;               // reduction channels per tap (conv) -- the last block of a tap may be partial
    unsigned* maxabs;      // max|acc| is reduced into this word; may be null (split-K partials)
    int32_t* status;
    int group_m;           // GEMM tile order: row tiles per group (0 / 1: plain row-major)
    int nstages;           // stages of the ring actually used (<= the compiled maximum; tuning / experiments)
    int split_cols;        // 1: both epilogue warpgroups share every tile (alternate 128-column groups); 0: they alternate tiles
    // fused requantisation (FUSED kernels): int8 output narrowed by the shift in state[0].
    // state = {shift, max|acc|, redo flag, redo count, finished-CTA ticket}; the last CTA of a first
    // launch derives the true shift from max|acc|, publishes it with the exponent / shift outputs and
    // raises the redo flag when the applied shift was wrong.
    int32_t* state;
    int only_if_redo;      // 1: this launch does nothing unless state[2] != 0, and verifies nothing
    int kind, target_bits;
    const int32_t* exp_a; const int32_t* exp_b; int32_t* exp_out; int32_t* shift_out;
    int mode, relu;
    int8_t* out8;          // fused kernels: the int8 output as a plain pointer (rows = row_lin, pitch N bytes)
    const int8_t* mask;    // fused kernels: optional ReLU-backward mask, same shape as the output (zero where mask <= 0)
    int8_t* pool_out;      // parked kernel, forward convolutions: optional 2x2 / stride-2 max-pooled copy of the output [N][H/2][W/2][K]
    uint32_t* side;        // streaming fused kernel, round-to-nearest without ReLU: two more bits per output (16 per word, rows of
                           // N / 4 bytes) from which the output for the next LOWER shift follows exactly (requant_step_down)
    const unsigned long long* seed;
    unsigned rng_stream;
    unsigned long long rng_offset;
};

constexpr int GEMM_THREADS = 320;  // producer warp, MMA warp, two epilogue warpgroups of 4 warps
constexpr unsigned STEP_DOWN_RUN = 12;  // step-downs in a row after which the predicted shift is lowered (< 16)

template <int BN, bool TWO = false>
struct GemmCfg {
    static constexpr int B_STAGE_BYTES = (TWO ? BN / 2 : BN) * ROW_BYTES;  // a CTA of a pair holds half of the B columns
    static constexpr int STAGE_BYTES = PANEL_BYTES + B_STAGE_BYTES;
    static constexpr int EPI_GROUP_BYTES = 2 * EPI_CHUNK_BYTES;  // staging per epilogue warpgroup: two 128 x 32 int32 tiles
    static constexpr int EPI_BYTES = 2 * EPI_GROUP_BYTES;
    static constexpr int STAGES = (224 * 1024 - EPI_BYTES) / STAGE_BYTES;
    static constexpr int TMEM_COLS = 2 * BN;  // two accumulators; 256 or 512 columns
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
};

// a call of its own: its dozen instructions at every wait lay between the ones that a launch fetches and runs once
__device__ __noinline__ void report_abort(int32_t* status, int code, int role) {
    if (status != nullptr && atomicCAS(status, 0, code) == 0) {
        status[1] = static_cast<int32_t>(blockIdx.x + blockIdx.y * gridDim.x);
        status[2] = role;
    }
}

// Four accumulators of one row -> four int8 packed in a word, any rounding (the short forms are in requant.cuh).
__device__ __forceinline__ uint32_t narrow4(const uint32_t* v, int shift, int mode, int relu, const uint32_t* rnd) {
    uint32_t w = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        int y = narrow(static_cast<int>(v[j]), shift, mode, rnd[j]);
        if (relu && y < 0) y = 0;
        w |= static_cast<uint32_t>(static_cast<uint8_t>(y)) << (8 * j);
    }
    return w;
}

// Round-to-nearest narrowing of 16 values (one 16-byte piece of an output row) with shift S >= 2 that also keeps bits
// S-1 and S-2 of the rounded-up sum: with u = x + 2^(S-1) - (x < 0), T = u >> (S-2) = 4 * (u >> S) + code, and the value
// for shift S - 1, sign(x) * ((|x| + 2^(S-2)) >> (S-1)), is 2 * (u >> S) + (code == 3) - (code == 0) for either sign.
// The code of byte j of word q sits at bit 8 j + 2 q of the piece's code word.
__device__ __forceinline__ uint32_t narrow16_nearest_codes(const uint32_t* v, int shift2, int half, uint32_t* packed) {
    uint32_t codes = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        int y[4], t[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int x = static_cast<int>(v[4 * q + j]);
            t[j] = (x + half + (x >> 31)) >> shift2;
            y[j] = t[j] >> 2;
        }
        packed[q] = __vmaxs4(pack2_sat_s8(y[1], y[0], pack2_sat_s8(y[3], y[2], 0u)), 0x81818181u);
        // the low bytes of the four t side by side, their two low bits moved to this word's place in every byte
        const uint32_t low = __byte_perm(__byte_perm(t[0], t[1], 0x0040), __byte_perm(t[2], t[3], 0x0040), 0x5410);
        codes |= (low & 0x03030303u) << (2 * q);
    }
    return codes;
}
// Four outputs narrowed with shift S (one word) and their codes (bits 0-1 of each byte of e) -> the four outputs for
// shift S - 1, clamped to +-127.  Two 16-bit lanes per register, biased by 128 so that plain 32-bit arithmetic cannot
// borrow between lanes; the lane-wise add + min / max are single instructions.
__device__ __forceinline__ uint32_t step_down4(uint32_t y4, uint32_t e) {
    const uint32_t e1 = e >> 1;
    const uint32_t eq3 = e & e1;                       // bit 0 of a byte: code == 3
    const uint32_t eq0 = ~(e | e1) & 0x01010101u;      // code == 0
    const uint32_t dd = eq3 + 0x01010101u - eq0;       // d + 1 in {0, 1, 2} per byte
    const uint32_t yb = y4 ^ 0x80808080u;              // y + 128 per byte
    uint32_t la = (yb & 0x00FF00FFu) * 2u + (dd & 0x00FF00FFu);                // bytes 0, 2: 2 y + d + 257
    uint32_t lb = ((yb >> 8) & 0x00FF00FFu) * 2u + ((dd >> 8) & 0x00FF00FFu);  // bytes 1, 3
    la = __viaddmax_s16x2(__viaddmin_s16x2(la, 0xFFFFFFFFu, 0x017F017Fu), 0u, 0x00810081u);  // clamp(2 y + d, +-127) + 256
    lb = __viaddmax_s16x2(__viaddmin_s16x2(lb, 0xFFFFFFFFu, 0x017F017Fu), 0u, 0x00810081u);
    return __byte_perm(la, lb, 0x6240);                // the low byte of a lane is the value modulo 256
}
// The whole int8 output, narrowed with shift S by the launch before, rewritten for shift S - 1 from the side codes
// (every thread of the grid takes 16-byte pieces; the ReLU-backward mask is applied again, the codes ignore it).
__device__ void requant_step_down(int8_t* out8, const uint32_t* side, const int8_t* mask, long long pieces) {
    constexpr int U = 8;
    uint4* o = reinterpret_cast<uint4*>(out8);
    const uint4* m = reinterpret_cast<const uint4*>(mask);
    const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long i0 = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i0 < pieces; i0 += U * step) {
        uint4 y[U], k[U];
        uint32_t c[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = i0 + u * step;
            if (i < pieces) {
                y[u] = __ldcg(o + i);
                c[u] = __ldcg(side + i);
                if (mask != nullptr) k[u] = __ldg(m + i);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = i0 + u * step;
            if (i < pieces) {
                uint4 r;
                r.x = step_down4(y[u].x, c[u] & 0x03030303u); r.y = step_down4(y[u].y, (c[u] >> 2) & 0x03030303u);
                r.z = step_down4(y[u].z, (c[u] >> 4) & 0x03030303u); r.w = step_down4(y[u].w, (c[u] >> 6) & 0x03030303u);
                if (mask != nullptr) {
                    r.x &= __vcmpgts4(k[u].x, 0); r.y &= __vcmpgts4(k[u].y, 0);
                    r.z &= __vcmpgts4(k[u].z, 0); r.w &= __vcmpgts4(k[u].w, 0);
                }
                o[i] = r;
            }
        }
    }
}

// Output tile (row tile, column tile) of the mn-th tile in launch order.  Convolutions: row-major (the few column
// tiles of a row tile run together and share its activation tile).  GEMMs: row tiles in groups of 8, column-major
// inside a group, so the ~148 tiles in flight at any time cover a compact block of the output (8 x ~18 tiles) instead
// of 2-3 whole rows: a wave then re-reads ~36 MB of operands instead of all of B.  Only when the operands do not fit
// in L2 anyway (group_m is set on the host): 8192^3 406 -> 376 us, 16384^3 3679 -> 2977 us, 4096^3 unchanged.
__device__ __forceinline__ void tile_coords(const GemmParams& p, int mn, int* m_pair, int* n_t) {
    if (p.group_m <= 1) { *m_pair = fdiv(mn, p.fd_n); *n_t = mn - *m_pair * p.n_tiles; return; }
    const int GM = p.group_m;
    const int per_group = GM * p.n_tiles;
    const int group = mn / per_group, in_group = mn % per_group;
    const int first = group * GM;
    const int rows = min(GM, p.m_tiles - first);
    *m_pair = first + in_group % rows;
    *n_t = in_group / rows;
}

// ---- warp roles shared by the streaming kernel and the accumulator-parking kernel -------------
// stages of the ring in use (NITI_OPT_STAGE_CAP)
__device__ __forceinline__ int ring_stages(const GemmParams& p, int compiled) { return (p.nstages > 0 && p.nstages < compiled) ? p.nstages : compiled; }

// TMA producer: fills the stage ring for every tile of this CTA, in tile order.  The WHOLE warp runs the loop and
// an elected lane issues.  TMA and MMA instructions take their operands from uniform registers, and the compiler keeps
// addresses, coordinates and descriptors there only while every branch around them is provably warp-uniform: waits
// therefore spin INSIDE one asm statement and hand back a voted verdict (mbar_wait_uniform), values read from shared
// memory or special registers pass through a shuffle, and the issuing lane comes from elect.sync.  Measured on B200
// (clock64 around the instructions): 50 cycles per tcgen05.mma and ~20 per TMA instruction this way; 85-90 and ~50 when
// a loop-carried value depends on a per-lane asm result or the issuer is chosen by `lane == 0`; a loop entered by a
// single lane sits in between.  Per-tile integer divisions are skipped when the reduction is not split.
// TWO: this CTA is half of a CTA pair (cluster ranks 0/1).  Tiles are 256 rows high: rank r owns rows
// [128 r, 128 r + 128) of the pair's tile (m tile 2*pair_m + r) and columns [r BN/2, (r+1) BN/2) of the B
// operand; all byte counts are reported to rank 0's "full" barrier, which its MMA thread waits on.
// ROWS32: operands of 32-byte rows (p.rows32).  A variant of its own: as a branch of the one loop its byte counts and
// sources made every other product's issue slower (2048 x 128 x 4096: 20.5 us with the branch, 18.5 without; 8x8x8, 512 -> 256: 20.5, 18.5).
template <int BN, int STAGES, int STAGE_BYTES, bool TWO, bool ROWS32>
__device__ __forceinline__ void producer_role(uint8_t* smem, uint64_t* full_bar, uint64_t* empty_bar, const CUtensorMap* tmA,
                                              const CUtensorMap* tmB, const GemmParams& p, const int first, const int step,
                                              volatile int* abort_flag) {
    const int mn_tiles = p.m_tiles * p.n_tiles;
    const int total_tiles = mn_tiles * p.splits;
    const uint32_t rank = TWO ? __shfl_sync(0xFFFFFFFFu, cluster_ctarank(), 0) : 0u;  // a special register: make it provably uniform
    constexpr int BNH = TWO ? BN / 2 : BN;  // B columns this CTA loads
    const int nst = ring_stages(p, STAGES);
    const uint32_t abort_addr = smem_u32(const_cast<int*>(abort_flag));
    const uint32_t smem0 = smem_u32(smem), full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);
    const int conv = keep_reg(p.conv), flip = keep_reg(p.flip), pad = keep_reg(p.pad), S = keep_reg(p.S), cblocks = keep_reg(p.cblocks);
    const int tapstride = keep_reg(p.tapstride), b_mn = keep_reg(p.b_mn), a_mn = keep_reg(p.a_mn);
    const int rows32 = ROWS32 ? keep_reg(p.rows32) : 0;
    const uint32_t tx_full = static_cast<uint32_t>(keep_reg((TWO ? 2 : 1) * (p.a_bytes + p.b_bytes)));
    int s = 0; uint32_t ph = 0;
    uint32_t sa = smem0, fb_cur = full0, eb_cur = empty0;  // running stage pointers, wrapping with the ring
    DBG_DECL;
    DBG_CLK(c_begin);
    for (int tile = first; tile < total_tiles; tile += step) {
        int mn = tile, kb_lo = 0, kb_hi = p.num_kb;
        if (p.splits > 1) {
            const int split = fdiv(tile, p.fd_mn);
            mn = tile - split * mn_tiles;
            kb_lo = static_cast<int>(static_cast<long long>(split) * p.num_kb / p.splits);
            kb_hi = static_cast<int>(static_cast<long long>(split + 1) * p.num_kb / p.splits);
        }
        int m_pair, n_t;
        tile_coords(p, mn, &m_pair, &n_t);
        const int m_t = TWO ? 2 * m_pair + static_cast<int>(rank) : m_pair;
        int tw = 0, th = 0, tn = 0;
        if (conv) { const int q1 = fdiv(m_t, p.fd_tw); tw = m_t - q1 * p.tiles_w; tn = fdiv(q1, p.fd_th); th = q1 - tn * p.tiles_h; }
        const int ncol = n_t * BN + static_cast<int>(rank) * BNH;  // first B column of this CTA
        const int px = tw * p.BW, py = th * p.BH, pn = tn * p.BI;
        // This loop is one warp's serial instruction stream and sets the pace of the whole pipeline: the tap
        // (r, sx) and channel block cb of a reduction block are kept as running counters (four integer divisions per
        // block cost more than the block's MMAs), waits return nothing to branch on, pointers advance by addition.
        int cb = 0, sx = 0, r = 0;
        if (conv && kb_lo != 0) { const int tap0 = kb_lo / cblocks; cb = kb_lo % cblocks; r = tap0 / S; sx = tap0 % S; }
        for (int kb = kb_lo; kb < kb_hi; ++kb) {
            mbar_wait_quiet(eb_cur, ph ^ 1u, abort_addr);
            DBG_ACC(22, 1);
            const uint32_t sb = sa + PANEL_BYTES;
            uint32_t fb = fb_cur;
            uint32_t tx_bytes = tx_full, tx_b = 0;
            if (ROWS32) {  // the last rows of an operand may be fewer than a tile's; what they leave in the stage meets zeros or rows nobody stores
                const int b_rows = rows32 == 1 ? min(BN, p.N - ncol) : min(128, p.K - kb * 128);
                tx_b = static_cast<uint32_t>(b_rows) * 32u;
                tx_bytes = tx_b + (rows32 == 1 ? static_cast<uint32_t>(min(BLOCK_M, p.M - m_t * BLOCK_M)) * 32u : static_cast<uint32_t>(PANEL_BYTES));
            }
            if (elect_one()) {
                if (TWO) {
                    if (rank == 0) mbar_arrive_expect_tx(fb, tx_bytes);
                    fb = mapa_u32(fb, 0);
                } else {
                    mbar_arrive_expect_tx(fb, tx_bytes);
                }
                if (conv) {
                    const int tap = r * S + sx;
                    const int dx = flip ? pad - sx : sx - pad, dy = flip ? pad - r : r - pad;
                    if (TWO) tma_load_4d_pair(sa, tmA, fb, cb * ROW_BYTES, px + dx, py + dy, pn);
                    else     tma_load_4d(sa, tmA, fb, cb * ROW_BYTES, px + dx, py + dy, pn);
                    if (b_mn) {
#pragma unroll
                        for (int q = 0; q < (BNH + 127) / 128; ++q) {
                            if (TWO) tma_load_2d_pair(sb + q * PANEL_BYTES, tmB, fb, tap * tapstride + ncol + q * 128, cb * 128);
                            else     tma_load_2d(sb + q * PANEL_BYTES, tmB, fb, tap * tapstride + ncol + q * 128, cb * 128);
                        }
                    } else {
                        if (TWO) tma_load_2d_pair(sb, tmB, fb, tap * tapstride + cb * ROW_BYTES, ncol);
                        else     tma_load_2d(sb, tmB, fb, tap * tapstride + cb * ROW_BYTES, ncol);
                    }
                } else if (ROWS32 && rows32 == 1) {
                    bulk_load(sa, p.a32 + static_cast<long long>(m_t) * (BLOCK_M * 32), tx_bytes - tx_b, fb);
                    bulk_load(sb, p.b32 + static_cast<long long>(ncol) * 32, tx_b, fb);
                } else if (ROWS32) {
                    tma_load_2d(sa, tmA, fb, m_t * BLOCK_M, kb * 128);
                    bulk_load(sb, p.b32 + static_cast<long long>(kb) * (128 * 32), tx_b, fb);
                } else {
                    if (TWO) {
                        if (a_mn) tma_load_2d_pair(sa, tmA, fb, m_t * BLOCK_M, kb * 128);
                        else      tma_load_2d_pair(sa, tmA, fb, kb * ROW_BYTES, m_t * BLOCK_M);
                    } else {
                        if (a_mn) tma_load_2d(sa, tmA, fb, m_t * BLOCK_M, kb * 128);
                        else      tma_load_2d(sa, tmA, fb, kb * ROW_BYTES, m_t * BLOCK_M);
                    }
                    if (b_mn) {
#pragma unroll
                        for (int q = 0; q < BNH / 128; ++q) {
                            if (TWO) tma_load_2d_pair(sb + q * PANEL_BYTES, tmB, fb, ncol + q * 128, kb * 128);
                            else     tma_load_2d(sb + q * PANEL_BYTES, tmB, fb, ncol + q * 128, kb * 128);
                        }
                    } else {
                        if (TWO) tma_load_2d_pair(sb, tmB, fb, kb * ROW_BYTES, ncol);
                        else     tma_load_2d(sb, tmB, fb, kb * ROW_BYTES, ncol);
                    }
                }
            }
            if (conv && ++cb == cblocks) { cb = 0; if (++sx == S) { sx = 0; ++r; } }
            sa += STAGE_BYTES; fb_cur += 8u; eb_cur += 8u;
            if (++s == nst) { s = 0; ph ^= 1u; sa = smem0; fb_cur = full0; eb_cur = empty0; }
        }
    }
    if (*abort_flag) report_abort(p.status, 1, 0);  // a quiet wait of this role (or another role) gave up
    DBG_CLK(c_end); DBG_ACC(20, c_end - c_begin);
    DBG_OUT(20);
}

// MMA issuer: the whole warp runs the loop with warp-uniform control flow (see the producer), one elected lane issues
// the MMAs and the commits.  Streaming: NACC accumulators used in turn, each handed back by the
// epilogue (tempty).  Parked (NACC = 0): tile i of this CTA accumulates into TMEM columns [i*BN, (i+1)*BN) and
// stays there until the kernel ends, so no accumulator is ever waited for.
// TWO: run by rank 0 of a CTA pair only; M = 256 MMAs over both CTAs' shared and tensor memory, and every
// completion (stage free, accumulator full) is signalled to both CTAs.
template <bool TWO>
__device__ __forceinline__ void umma_issue(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    if (TWO) umma_i8_pair(d_tmem, a, b, idesc, accumulate); else umma_i8(d_tmem, a, b, idesc, accumulate);
}
template <int BN, int STAGES, int STAGE_BYTES, int NACC, bool TWO, bool ROWS32>
__device__ __forceinline__ void mma_role(uint8_t* smem, uint64_t* full_bar, uint64_t* empty_bar, uint64_t* tfull_bar,
                                         uint64_t* tempty_bar, uint32_t tmem_base_in, const GemmParams& p, const int first, const int step,
                                         volatile int* abort_flag) {
    constexpr bool PARKED = NACC == 0;
    const int rows32 = ROWS32 ? keep_reg(p.rows32) : 0;
    const int mn_tiles = p.m_tiles * p.n_tiles;
    const int total_tiles = mn_tiles * p.splits;
    const uint32_t idesc = make_idesc_i8(TWO ? 2 * BLOCK_M : BLOCK_M, p.mma_n, p.a_mn, p.b_mn);
    const int nst = ring_stages(p, STAGES);
    const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, tmem_base_in, 0);  // read from shared memory: make it provably uniform
    const uint32_t abort_addr = smem_u32(const_cast<int*>(abort_flag));
    const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);
    // operand descriptors of stage 0 (a stage's are these advanced by the stage offset) and the K = 32 steps
    const uint32_t s0 = smem_u32(smem);
    const uint64_t a_base = rows32 == 1 ? make_smem_desc(s0, 16, 256, SWIZZLE_32B_CODE) : p.a_mn ? make_smem_desc(s0, PANEL_BYTES, 1024, SWIZZLE_128B_CODE) : make_smem_desc(s0, 16, 1024, SWIZZLE_128B_CODE);
    // a 64-column MN-major operand has rows of 64 bytes: 64-byte swizzle, 8-row groups of 512 bytes
    const uint64_t b_base = ROWS32 ? make_smem_desc(s0 + PANEL_BYTES, 1024, 256, SWIZZLE_32B_CODE) : p.b_mn ? (BN == 64 ? make_smem_desc(s0 + PANEL_BYTES, 64 * ROW_BYTES, 512, SWIZZLE_64B_CODE)
                                               : make_smem_desc(s0 + PANEL_BYTES, PANEL_BYTES, 1024, SWIZZLE_128B_CODE))
                                   : make_smem_desc(s0 + PANEL_BYTES, 16, 1024, SWIZZLE_128B_CODE);
    const uint32_t a_step = static_cast<uint32_t>(keep_reg((p.a_mn ? 32 * ROW_BYTES : 32) >> 4));  // in descriptor units of 16 bytes
    const uint32_t b_step = static_cast<uint32_t>(keep_reg((rows32 == 2 ? 32 * 32 : p.b_mn ? 32 * (BN == 64 ? 64 : ROW_BYTES) : 32) >> 4));
    const int conv = keep_reg(p.conv), red = keep_reg(p.red), cblocks = keep_reg(p.cblocks), num_kb = keep_reg(p.num_kb), splits = keep_reg(p.splits);
    int s = 0; uint32_t ph = 0; bool ok = true; int it = 0;
    // every reduction block has four MMAs unless a conv tap's channel count ends in a partial 128-byte block
    const bool all4 = conv ? (red & 127) == 0 : rows32 != 1;
    // running stage pointers: descriptors and barrier addresses advance by one stage per block and wrap with the ring
    const uint64_t stage_step = STAGE_BYTES >> 4;
    uint64_t a_cur = a_base, b_cur = b_base;
    uint32_t full_cur = full0, empty_cur = empty0;
    DBG_DECL;
#ifdef NITI_PARKED_TIMING
    long long c_first = 0;
#endif
    for (int tile = first; ok && tile < total_tiles; tile += step, ++it) {
        const int acc = PARKED ? it : it % (PARKED ? 1 : NACC);
        if (!PARKED) {
            const uint32_t aph = (it / (PARKED ? 1 : NACC)) & 1u;
            ok = mbar_wait_uniform(smem_u32(&tempty_bar[acc]), aph ^ 1u, abort_addr);
            if (!ok) { *abort_flag = 1; report_abort(p.status, 2, 1); break; }
            tc_fence_after();
        }
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
        int kb_lo = 0, kb_hi = num_kb;
        if (splits > 1) {
            const int split = tile / mn_tiles;
            kb_lo = static_cast<int>(static_cast<long long>(split) * num_kb / splits);
            kb_hi = static_cast<int>(static_cast<long long>(split + 1) * num_kb / splits);
        }
        int cb = (conv && kb_lo != 0) ? kb_lo % cblocks : 0;  // channel block within the tap: a running counter, no division per block
        for (int kb = kb_lo; kb < kb_hi; ++kb) {
            DBG_ACC(19, 1);
#ifdef NITI_PARKED_TIMING
            if (it == 0 && kb == kb_lo) { c_first = clock64(); if (PARKED) PARK_STAMP(2); }
#endif
            if (all4) {
                // wait for the stage, four MMAs, commit: one asm statement, nothing for the loop to branch on
                umma_block4_wait<TWO>(d_tmem, a_cur, b_cur, a_step, b_step, idesc, static_cast<uint32_t>(kb != kb_lo), empty_cur,
                                      full_cur, ph, abort_addr);
            } else {
                // a partial block: issue only the MMAs (K = 32 each) that cover real channels (the rest is TMA zero fill)
                const int left = red - cb * 128;
                const int nmma = !conv ? 1 : left >= 128 ? 4 : (left + 31) >> 5;  // rows32 == 1: the one block is 32 deep
                if (++cb == cblocks) cb = 0;
                mbar_wait_quiet(full_cur, ph, abort_addr);
                if (elect_one()) {
                    for (int k = 0; k < nmma; ++k)
                        umma_issue<TWO>(d_tmem, a_cur + k * a_step, b_cur + k * b_step, idesc, static_cast<uint32_t>(kb != kb_lo || k != 0));
                    if (TWO) umma_commit_pair(empty_cur); else umma_commit(empty_cur);
                }
            }
            a_cur += stage_step; b_cur += stage_step; full_cur += 8u; empty_cur += 8u;
            if (++s == nst) { s = 0; ph ^= 1u; a_cur = a_base; b_cur = b_base; full_cur = full0; empty_cur = empty0; }
        }
        if (ok && elect_one()) { if (TWO) umma_commit_pair(smem_u32(&tfull_bar[acc])); else umma_commit(smem_u32(&tfull_bar[acc])); }
    }
    if (*abort_flag) report_abort(p.status, 3, 1);  // a quiet wait of this role (or another role) gave up
    if (PARKED) PARK_STAMP(3);
#ifdef NITI_PARKED_TIMING
    DBG_ACC(16, clock64() - c_first);
#endif
    DBG_OUT(16);
}

// ---- 3x3 convolutions whose tiles are 8 pixels wide: activations fetched once per filter COLUMN instead of once per tap
// A stage holds, for one 128-byte channel block and one filter column, the activations of a tile and of the pixel rows
// above and below it (a box of 8 x (BH + 2) pixels, 18 KB) and the weights of the column's three taps.  An image row of
// the box is 8 shared-memory rows of 128 bytes, one swizzle atom, so the operand of tap (r, column) is the same panel
// read from r atoms further on: a change of the descriptor's start address.  Against a box per tap (16 KB of activations
// and 16 KB of weights for four 128-column MMAs, 550 cycles against 256 on the tensor pipe) a tile moves 199 instead of
// 288 KB (64 columns: 127 instead of 216), and twelve MMAs instead of four ride on one hand-over between the roles.
constexpr int HALO_ATOM = 8 * ROW_BYTES;          // one image row of the box
constexpr int HALO_A_BYTES = 18 * HALO_ATOM;      // at most 16 + 2 image rows
// What a stage holds.  HALO_RESIDENT: layers of one channel block and one column tile keep their whole weights (nine taps,
// 72 or 144 KB) in shared memory behind the ring; they arrive with the first tile, column by column (one barrier each),
// and a stage is activations only.  The loads are paced by rows of 128 bytes (about 3 cycles each): 432 a tile instead
// of 1008 (64 columns) or 1584 (128).
// LOAD_ROWS32: operands of 32-byte rows (the thin layer; streaming only).
enum LoadMode : int { LOAD_TAPS = 0, LOAD_HALO = 1, LOAD_HALO_RESIDENT = 2, LOAD_ROWS32 = 3 };
constexpr bool shares_rows(int mode) { return mode == LOAD_HALO || mode == LOAD_HALO_RESIDENT; }
template <int BN, int STAGES, int STAGE_BYTES, bool RESIDENT>
__device__ __forceinline__ void producer_halo_role(uint8_t* smem, uint64_t* full_bar, uint64_t* empty_bar, uint32_t weights0, const CUtensorMap* tmA,
                                                   const CUtensorMap* tmB, const GemmParams& p, volatile int* abort_flag) {
    const int total_tiles = p.m_tiles * p.n_tiles;
    const uint32_t abort_addr = smem_u32(const_cast<int*>(abort_flag));
    const uint32_t smem0 = smem_u32(smem), full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);
    const int flip = keep_reg(p.flip), cblocks = keep_reg(p.cblocks), tapstride = keep_reg(p.tapstride), b_mn = keep_reg(p.b_mn);
    const uint32_t tx_bytes = static_cast<uint32_t>(keep_reg(p.a_bytes + (RESIDENT ? 0 : 3 * p.b_bytes)));
    const uint32_t res0 = smem0 + STAGES * STAGE_BYTES;  // resident weights: [column][filter row]
    bool weights_due = RESIDENT;
    const int nst = ring_stages(p, STAGES);
    int s = 0; uint32_t ph = 0;
    uint32_t sa = smem0, fb = full0, eb = empty0;
    for (int tile = static_cast<int>(blockIdx.x); tile < total_tiles; tile += static_cast<int>(gridDim.x)) {
        const int m_t = fdiv(tile, p.fd_n), n_t = tile - m_t * p.n_tiles;
        const int q1 = fdiv(m_t, p.fd_tw), tw = m_t - q1 * p.tiles_w, pn = fdiv(q1, p.fd_th), th = q1 - pn * p.tiles_h;
        const int ncol = n_t * BN, px = tw * 8, py = th * p.BH - 1;
        for (int cb = 0; cb < cblocks; ++cb)
            for (int sx = 0; sx < 3; ++sx) {
                mbar_wait_quiet(eb, ph ^ 1u, abort_addr);
                if (elect_one()) {
                    mbar_arrive_expect_tx(fb, tx_bytes);
                    tma_load_4d(sa, tmA, fb, cb * ROW_BYTES, px + (flip ? 1 - sx : sx - 1), py, pn);
                    if (!RESIDENT || weights_due) {
                        const uint32_t dst = RESIDENT ? res0 + sx * 3 * BN * ROW_BYTES : sa + HALO_A_BYTES;
                        const uint32_t bar = RESIDENT ? weights0 + 8u * sx : fb;
                        if (RESIDENT) mbar_arrive_expect_tx(bar, static_cast<uint32_t>(3 * p.b_bytes));
#pragma unroll
                        for (int r = 0; r < 3; ++r) {
                            const int x = (r * 3 + sx) * tapstride;
                            if (b_mn) tma_load_2d(dst + r * BN * ROW_BYTES, tmB, bar, x + ncol, cb * 128);
                            else      tma_load_2d(dst + r * BN * ROW_BYTES, tmB, bar, x + cb * ROW_BYTES, ncol);
                        }
                    }
                }
                sa += STAGE_BYTES; fb += 8u; eb += 8u;
                if (++s == nst) { s = 0; ph ^= 1u; sa = smem0; fb = full0; eb = empty0; }
            }
        weights_due = false;
    }
    if (*abort_flag) report_abort(p.status, 1, 0);
}
template <int BN, int STAGES, int STAGE_BYTES, int NACC, bool RESIDENT>
__device__ __forceinline__ void mma_halo_role(uint8_t* smem, uint64_t* full_bar, uint64_t* empty_bar, uint32_t weights0, uint64_t* tfull_bar,
                                              uint64_t* tempty_bar, uint32_t tmem_base_in, const GemmParams& p, volatile int* abort_flag) {
    constexpr bool PARKED = NACC == 0;
    constexpr int MOD = PARKED ? 1 : NACC;
    const int total_tiles = p.m_tiles * p.n_tiles;
    const uint32_t idesc = make_idesc_i8(BLOCK_M, p.mma_n, 0, p.b_mn);
    const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, tmem_base_in, 0);
    const uint32_t abort_addr = smem_u32(const_cast<int*>(abort_flag));
    const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar), s0 = smem_u32(smem);
    const uint64_t a_base = make_smem_desc(s0, 16, 1024, SWIZZLE_128B_CODE);
    const uint32_t b0 = RESIDENT ? s0 + STAGES * STAGE_BYTES : s0 + HALO_A_BYTES;
    const uint64_t b_base = !p.b_mn ? make_smem_desc(b0, 16, 1024, SWIZZLE_128B_CODE)
                            : BN == 64 ? make_smem_desc(b0, 64 * ROW_BYTES, 512, SWIZZLE_64B_CODE)
                                       : make_smem_desc(b0, PANEL_BYTES, 1024, SWIZZLE_128B_CODE);
    const uint32_t b_step = static_cast<uint32_t>(keep_reg((p.b_mn ? 32 * (BN == 64 ? 64 : ROW_BYTES) : 32) >> 4));
    const int flip = keep_reg(p.flip), red = keep_reg(p.red), cblocks = keep_reg(p.cblocks);
    // the panel of filter row r starts r image rows into the box (error-backward reads the taps mirrored)
    const uint64_t a_first = flip ? (2 * HALO_ATOM) >> 4 : 0;
    const uint64_t a_next = flip ? ~static_cast<uint64_t>(HALO_ATOM >> 4) + 1 : HALO_ATOM >> 4;
    const int nst = ring_stages(p, STAGES);
    int s = 0, it = 0; uint32_t ph = 0;
    uint64_t a_cur = a_base + a_first, b_cur = b_base;
    uint32_t full_cur = full0, empty_cur = empty0;
    for (int tile = static_cast<int>(blockIdx.x); tile < total_tiles; tile += static_cast<int>(gridDim.x), ++it) {
        const int acc = PARKED ? it : it % MOD;
        if (!PARKED) {
            if (!mbar_wait_uniform(smem_u32(&tempty_bar[acc]), ((it / MOD) & 1u) ^ 1u, abort_addr)) { *abort_flag = 1; report_abort(p.status, 2, 1); break; }
            tc_fence_after();
        }
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
        uint32_t accumulate = 0;
        for (int cb = 0; cb < cblocks; ++cb) {
            const int left = red - cb * 128;
            for (int sx = 0; sx < 3; ++sx) {
                mbar_wait_quiet(full_cur, ph, abort_addr);
                if (RESIDENT) {
                    if (accumulate == 0) b_cur = b_base;
                    if (it == 0) mbar_wait_quiet(weights0 + 8u * sx, 0, abort_addr);
                }
                if (left > 96) {
#pragma unroll
                    for (int r = 0; r < 3; ++r) {
                        umma_seq4(d_tmem, a_cur + r * a_next, b_cur + static_cast<uint64_t>(r * BN * ROW_BYTES >> 4), 2, b_step, idesc, accumulate);
                        accumulate = 1;
                    }
                    if (elect_one()) umma_commit(empty_cur);
                } else {  // only the MMAs (K = 32 each) that cover real channels; the rest of the rows is TMA zero fill
                    const int nmma = (left + 31) >> 5;
#pragma unroll
                    for (int r = 0; r < 3; ++r) {
                        umma_seq_upto3(d_tmem, a_cur + r * a_next, b_cur + static_cast<uint64_t>(r * BN * ROW_BYTES >> 4), 2, b_step, idesc, accumulate, nmma);
                        accumulate = 1;
                    }
                    if (elect_one()) umma_commit(empty_cur);
                }
                a_cur += STAGE_BYTES >> 4; b_cur += (RESIDENT ? 3 * BN * ROW_BYTES : STAGE_BYTES) >> 4; full_cur += 8u; empty_cur += 8u;
                if (++s == nst) {
                    s = 0; ph ^= 1u; a_cur = a_base + a_first; full_cur = full0; empty_cur = empty0;
                    if (!RESIDENT) b_cur = b_base;
                }
            }
        }
        if (elect_one()) umma_commit(smem_u32(&tfull_bar[acc]));
    }
    if (*abort_flag) report_abort(p.status, 3, 1);
}

__device__ __forceinline__ unsigned fold_minmax(const int (&vmax)[4], const int (&vmin)[4]) {
    const int hi = max(max(vmax[0], vmax[1]), max(vmax[2], vmax[3]));
    const int lo = min(min(vmin[0], vmin[1]), min(vmin[2], vmin[3]));
    return max(static_cast<unsigned>(hi), static_cast<unsigned>(-static_cast<long long>(lo)));
}
// The same two steps on 32 accumulators at a time, for epilogues that run once or twice per launch: there
// every instruction is fetched cold, so a rolled loop over four 32-column chunks (a quarter of the code, the
// last three trips from the instruction cache) beats the straight-line 128-column form.
__device__ __forceinline__ void minmax32(const uint32_t (&v)[32], int lim, int (&vmax)[4], int (&vmin)[4]) {
    if (lim >= 32) {
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            vmax[0] = __vimax3_s32(vmax[0], static_cast<int>(v[i]), static_cast<int>(v[i + 1]));
            vmin[0] = __vimin3_s32(vmin[0], static_cast<int>(v[i]), static_cast<int>(v[i + 1]));
            vmax[1] = __vimax3_s32(vmax[1], static_cast<int>(v[i + 2]), static_cast<int>(v[i + 3]));
            vmin[1] = __vimin3_s32(vmin[1], static_cast<int>(v[i + 2]), static_cast<int>(v[i + 3]));
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (i < lim) {
                vmax[0] = max(vmax[0], static_cast<int>(v[i]));
                vmin[0] = min(vmin[0], static_cast<int>(v[i]));
            }
    }
}
// Every other case (pseudo-stochastic rounding, shifts of 24 and more, ...): a call of its own on arrays in local memory, so that its
// registers are not the epilogue's.
__device__ __noinline__ void narrow32_general(const uint32_t* v, uint32_t* packed, int shift, int mode, int relu,
                                              unsigned long long seed, unsigned rng_stream, unsigned long long e0) {
    const bool stochastic = mode == ROUND_STOCHASTIC && shift > 0;
#pragma unroll 1
    for (int i = 0; i < 32; i += 4) {
        uint32_t rnd[4] = {0, 0, 0, 0};
        if (stochastic) {
            const unsigned long long e = e0 + i;
            if ((e & 3ull) == 0) random_block(seed, rng_stream, e >> 2, rnd);
            else {
#pragma unroll
                for (int t = 0; t < 4; ++t) rnd[t] = random_word(seed, rng_stream, e + t);
            }
        }
        packed[i >> 2] = narrow4(v + i, shift, mode, relu, rnd);
    }
}
__device__ __forceinline__ void narrow32(const uint32_t (&v)[32], uint32_t (&packed)[8], int shift, int mode, int relu,
                                         unsigned long long seed, unsigned rng_stream, unsigned long long e0) {
    if (mode == ROUND_NEAREST && shift > 0) {
        const int half = 1 << (shift - 1);
        if (relu) {
#pragma unroll
            for (int i = 0; i < 32; i += 4) packed[i >> 2] = narrow4_nearest<true>(&v[i], shift, half);
        } else {
#pragma unroll
            for (int i = 0; i < 32; i += 4) packed[i >> 2] = narrow4_nearest<false>(&v[i], shift, half);
        }
    } else if (mode == ROUND_STOCHASTIC && shift > 0 && shift < 24 && (e0 & 3ull) == 0 && static_cast<uint32_t>(e0 >> 2) <= 0xFFFFFFF8u) {
        // The random words of four neighbouring outputs come from one Philox block: ten rounds of two wide multiplications,
        // which with the short narrowing is what a stochastic epilogue costs; the general form works value by value.
        const uint32_t mask = (1u << shift) - 1u;
        // The eight blocks' counters differ in their low words: with the high word a value of its own, what the first rounds make
        // of it, of the stream and of the keys is worked out once (128->128 at 32x32, 128 images: 31.3 -> 30.6 us; 256->256, 256
        // 16x16 maps, error-backward: 45.3 -> 42.7).
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            uint32_t rnd[4];
            philox4x32_10(static_cast<uint32_t>(e0 >> 2) + (i >> 2), static_cast<uint32_t>(e0 >> 34), rng_stream, 0u, static_cast<uint32_t>(seed),
                          static_cast<uint32_t>(seed >> 32), rnd);
            packed[i >> 2] = relu ? narrow4_stochastic<true>(&v[i], shift, mask, rnd) : narrow4_stochastic<false>(&v[i], shift, mask, rnd);
        }
    } else if (shift == 0) {
        // The low bytes as they are: what a layer's first pass, whose guess is 0, narrows with before it contracts again.
        // Through the general form that pass cost more than the contraction (both passes of 94 x 32 x 32, 48 -> 272: 316 us,
        // 273 like this; 256 -> 256 on 500 16 x 16 maps: 166, 119).
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            const uint32_t w = __byte_perm(__byte_perm(v[i], v[i + 1], 0x0040), __byte_perm(v[i + 2], v[i + 3], 0x0040), 0x5410);
            packed[i >> 2] = relu ? __vmaxs4(w, 0u) : w;
        }
    } else {
        uint32_t in[32], out[8];
#pragma unroll
        for (int i = 0; i < 32; ++i) in[i] = v[i];
        narrow32_general(in, out, shift, mode, relu, seed, rng_stream, e0);
#pragma unroll
        for (int i = 0; i < 8; ++i) packed[i] = out[i];
    }
}
// ReLU backward folded into an error-backward epilogue: zero the packed int8 outputs where the layer's forward input
// (the ReLU's output) was not positive.  `m` points at this row's mask bytes for the same columns; `cols` of them exist.
template <int WORDS>
__device__ __forceinline__ void apply_relu_mask(uint32_t (&packed)[WORDS], const int8_t* m, int cols) {
#pragma unroll
    for (int q = 0; q < WORDS / 4; ++q)
        if (16 * q + 16 <= cols) {
            const uint4 x = __ldg(reinterpret_cast<const uint4*>(m) + q);
            packed[4 * q + 0] &= __vcmpgts4(x.x, 0); packed[4 * q + 1] &= __vcmpgts4(x.y, 0);
            packed[4 * q + 2] &= __vcmpgts4(x.z, 0); packed[4 * q + 3] &= __vcmpgts4(x.w, 0);
        }
}
// The same in two steps, so that the loads can be issued long before the bytes they gate exist: PIECES 16-byte pieces
// of the mask row into registers, then the AND.  m null: nothing to do.
template <int PIECES>
__device__ __forceinline__ void mask_load(const int8_t* m, int cols, uint4 (&mk)[PIECES]) {
#pragma unroll
    for (int q = 0; q < PIECES; ++q)
        if (m != nullptr && 16 * q + 16 <= cols) mk[q] = __ldg(reinterpret_cast<const uint4*>(m) + q);
}
template <int PIECES>
__device__ __forceinline__ void mask_apply(uint32_t* packed, const int8_t* m, int cols, const uint4 (&mk)[PIECES]) {
#pragma unroll
    for (int q = 0; q < PIECES; ++q)
        if (m != nullptr && 16 * q + 16 <= cols) {
            packed[4 * q + 0] &= __vcmpgts4(mk[q].x, 0); packed[4 * q + 1] &= __vcmpgts4(mk[q].y, 0);
            packed[4 * q + 2] &= __vcmpgts4(mk[q].z, 0); packed[4 * q + 3] &= __vcmpgts4(mk[q].w, 0);
        }
}
// Byte-wise maximum over a 2x2 pixel window whose four pixels are the rows of lanes l, l^1, l^bw, l^bw^1 of this warp
// (all 32 lanes call it): afterwards every lane of a window holds the window's maxima.
__device__ __forceinline__ void pool_window(uint32_t (&w)[8], int bw) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        uint32_t m = __vmaxs4(w[i], __shfl_xor_sync(0xFFFFFFFFu, w[i], 1));
        w[i] = __vmaxs4(m, __shfl_xor_sync(0xFFFFFFFFu, m, bw));
    }
}
// whether every 32-byte piece of a tensor of `n`-byte rows starts on a 32-byte boundary
__device__ __forceinline__ bool rows_of_32(const int8_t* base, int n) { return ((reinterpret_cast<uintptr_t>(base) | static_cast<uintptr_t>(n)) & 31) == 0; }
// 32 packed int8 of one output row to global memory: one 32-byte store (a whole L2 sector) or, where the rows are only
// 16-byte aligned, two.  `at` is null for rows outside the tensor; `cols` (a multiple of 16) exist from there on.
__device__ __forceinline__ void store_piece(int8_t* at, int cols, const uint32_t (&w)[8], bool wide) {
    if (at == nullptr) return;
    if (wide) {
        st_global_v8(at, w);  // rows of a multiple of 32 bytes: a piece that starts inside the row ends inside it
        return;
    }
    if (cols >= 16) *reinterpret_cast<uint4*>(at) = make_uint4(w[0], w[1], w[2], w[3]);
    if (cols >= 32) *reinterpret_cast<uint4*>(at + 16) = make_uint4(w[4], w[5], w[6], w[7]);
}

// Plain products: int32 out (+ max|acc|).
template <int BN, bool TWO, bool ROWS32>
__global__ void __launch_bounds__(GEMM_THREADS, 1)  // 10 warps: 3 on one scheduler -> at most 168 registers per thread
umma_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmC, const GemmParams p) {
    using Cfg = GemmCfg<BN, TWO>;
    constexpr int STAGES = Cfg::STAGES;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* epi_smem = smem + STAGES * Cfg::STAGE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(epi_smem + Cfg::EPI_BYTES);
    uint64_t* full_bar = bars;
    uint64_t* empty_bar = bars + STAGES;
    uint64_t* tfull_bar = bars + 2 * STAGES;
    uint64_t* tempty_bar = bars + 2 * STAGES + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile unsigned* warp_max = reinterpret_cast<volatile unsigned*>(tmem_slot + 4);  // one word per epilogue warp

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = TWO ? cluster_ctarank() : 0u;  // rank 0 of a pair issues the MMAs and owns the barriers the MMA thread waits on

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) { mbar_init(smem_u32(&full_bar[i]), 1); mbar_init(smem_u32(&empty_bar[i]), 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&tfull_bar[i]), 1); mbar_init(smem_u32(&tempty_bar[i]), (p.split_cols ? 8 : 4) * (TWO ? 2 : 1)); }
        *abort_flag = 0;
        fence_barrier_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        tma_prefetch_desc(&tmC);
    }
    if (warp == 1) {
        if (TWO) { tmem_alloc_pair(smem_u32(tmem_slot), Cfg::TMEM_COLS); tmem_relinquish_pair(); }
        else     { tmem_alloc(smem_u32(tmem_slot), Cfg::TMEM_COLS); tmem_relinquish(); }
    }
    tc_fence_before();
    __syncthreads();
    if (TWO) cluster_sync_all();  // the partner's barriers exist before anything is signalled across the pair
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const int mn_tiles = p.m_tiles * p.n_tiles;  // TWO: m_tiles counts 256-row tiles of the pair
    const int total_tiles = mn_tiles * p.splits;
    const int cta_first = TWO ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
    const int cta_step = TWO ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);

    // Only one lane of warps 0 and 1 works; the others wait at __syncwarp so that each warp reaches the
    // block-wide barrier of the teardown converged (an aligned barrier executed by a diverged warp is undefined).
    if (warp == 0) {
        producer_role<BN, STAGES, Cfg::STAGE_BYTES, TWO, ROWS32>(smem, full_bar, empty_bar, &tmA, &tmB, p, cta_first, cta_step, abort_flag);
        __syncwarp();
    } else if (warp == 1) {
        if (rank == 0)
            mma_role<BN, STAGES, Cfg::STAGE_BYTES, 2, TWO, ROWS32>(smem, full_bar, empty_bar, tfull_bar, tempty_bar, tmem_base, p, cta_first, cta_step, abort_flag);
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue (2 x 4 warps)
        // Two warpgroups.  With several tiles per CTA they alternate tiles (warpgroup g owns
        // accumulator g), so the epilogues of consecutive tiles overlap each other and the main
        // loop; with one or two wide tiles per CTA (split_cols) they share every tile, each taking
        // alternate 128-column groups, which halves the serial tail.  Per group of 128 columns:
        // four tcgen05.ld and ONE wait, the accumulator is handed back as soon as the warpgroup's
        // last columns sit in registers, max|acc| is tracked in registers, rows go to swizzled
        // staging tiles and leave through TMA stores (which clip rows/columns outside the tensor).
        // Two rounds of two 128 x 32 staging tiles per column group.
        const int grp = (warp - 2) >> 2;  // epilogue warpgroup 0 / 1
        const int q = warp & 3;           // TMEM lanes [32q, 32q+32) are the ones this warp may read
        const int row_in_tile = q * 32 + lane;
        const int bar_id = EPI_BARRIER + grp;
        const bool leader = (threadIdx.x == 64 + grp * 128);
        const uint32_t buf = smem_u32(epi_smem) + grp * Cfg::EPI_GROUP_BYTES;
        int vmax[4] = {0, 0, 0, 0}, vmin[4] = {0, 0, 0, 0};
        const int tile_step = p.split_cols ? cta_step : 2 * cta_step;
        int it = p.split_cols ? 0 : grp;
        // this thread's row inside a tile never changes: pixel offsets within the tile's box
        int row_w = 0, row_h = 0, row_n = 0;
        bool row_in_box = true;
        if (p.conv) {
            const int t_ = row_in_tile / p.BW;
            row_w = row_in_tile - t_ * p.BW; row_n = t_ / p.BH; row_h = t_ - row_n * p.BH;
            row_in_box = row_in_tile < p.BW * p.BH * p.BI;
        }
        for (int tile = cta_first + (p.split_cols ? 0 : grp * cta_step); tile < total_tiles; tile += tile_step, it += (p.split_cols ? 1 : 2)) {
            const int acc = it & 1; const uint32_t aph = (it >> 1) & 1u;
            // where the tile lies, before waiting for its accumulator: the arithmetic and the first touch of the mask hide in the wait
            int split = 0, mn = tile;
            if (p.splits > 1) { split = fdiv(tile, p.fd_mn); mn = tile - split * mn_tiles; }
            int m_pair, n_t;
            tile_coords(p, mn, &m_pair, &n_t);
            const int m_t = TWO ? 2 * m_pair + static_cast<int>(rank) : m_pair;
            bool valid; int cy, cz, cw;
            if (p.conv) {
                const int q1 = fdiv(m_t, p.fd_tw), tw = m_t - q1 * p.tiles_w, tn = fdiv(q1, p.fd_th), th = q1 - tn * p.tiles_h;
                cy = tw * p.BW; cz = th * p.BH; cw = tn * p.BI;
                const int w = cy + row_w, h = cz + row_h, n = cw + row_n;
                valid = row_in_box && w < p.W && h < p.H && n < p.Nimg;
            } else {
                valid = m_t * BLOCK_M + row_in_tile < p.M;
                cy = m_t * BLOCK_M; cz = split; cw = 0;
            }
            const uint32_t failed = mbar_wait(smem_u32(&tfull_bar[acc]), aph, abort_flag) ? 0u : 1u;
            if (barrier_or(bar_id, 128, failed)) {  // same verdict in all 128 threads of the warpgroup
                if (failed) report_abort(p.status, 4, 2);
                break;
            }
            tc_fence_after();
            const int col0 = n_t * BN;
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * BN);
            // column groups of this warpgroup: all of them, or every other one when the tile is shared
            const int g_first = p.split_cols ? grp * 128 : 0, g_step = p.split_cols ? 256 : 128;
            bool released = false;
#pragma unroll 1
            for (int g0 = g_first; g0 < BN && col0 + g0 < p.N; g0 += g_step) {
                uint32_t v[4][32];
#pragma unroll
                for (int j = 0; j < 4; ++j) tmem_ld_32x32(taddr + g0 + j * 32, v[j]);
                tmem_ld_wait();
                if (g0 + g_step >= BN || col0 + g0 + g_step >= p.N) {  // this warpgroup's last group of the tile
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (TWO) mbar_arrive_cluster(mapa_u32(smem_u32(&tempty_bar[acc]), 0));
                        else     mbar_arrive(smem_u32(&tempty_bar[acc]));
                    }
                    released = true;
                }
                const int lim = p.N - (col0 + g0);
                if (valid) {
                    // max|x| = max(max x, -min x): short chains of 3-input min/max
                    if (lim >= 128) {
#pragma unroll
                        for (int j = 0; j < 4; ++j)
#pragma unroll
                            for (int i = 0; i < 32; i += 2) {
                                vmax[j] = __vimax3_s32(vmax[j], static_cast<int>(v[j][i]), static_cast<int>(v[j][i + 1]));
                                vmin[j] = __vimin3_s32(vmin[j], static_cast<int>(v[j][i]), static_cast<int>(v[j][i + 1]));
                            }
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; ++j)
#pragma unroll
                            for (int i = 0; i < 32; ++i)
                                if (j * 32 + i < lim) {
                                    vmax[0] = max(vmax[0], static_cast<int>(v[j][i]));
                                    vmin[0] = min(vmin[0], static_cast<int>(v[j][i]));
                                }
                    }
                }
#pragma unroll
                for (int half_i = 0; half_i < 2; ++half_i) {
                    if (col0 + g0 + half_i * 64 >= p.N) break;
                    if (leader) bulk_wait_read<0>();  // the stores of the pass before have read the staging tiles
                    named_barrier(bar_id, 128);
                    stage_row(buf, row_in_tile, v[2 * half_i]);
                    stage_row(buf + EPI_CHUNK_BYTES, row_in_tile, v[2 * half_i + 1]);
                    fence_proxy_async();
                    named_barrier(bar_id, 128);
                    if (leader) {
                        tma_store_4d(&tmC, buf, col0 + g0 + half_i * 64, cy, cz, cw);
                        if (col0 + g0 + half_i * 64 + 32 < p.N) tma_store_4d(&tmC, buf + EPI_CHUNK_BYTES, col0 + g0 + half_i * 64 + 32, cy, cz, cw);
                        bulk_commit();
                    }
                }
            }
            if (!released) {  // a shared tile none of whose column groups fell to this warpgroup
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                        if (TWO) mbar_arrive_cluster(mapa_u32(smem_u32(&tempty_bar[acc]), 0));
                        else     mbar_arrive(smem_u32(&tempty_bar[acc]));
                    }
            }
        }
        if (leader) bulk_wait_read<0>();  // shared memory may go once the stores have read it; the writes land by the end of the grid
        const int hi = max(max(vmax[0], vmax[1]), max(vmax[2], vmax[3]));
        const int lo = min(min(vmin[0], vmin[1]), min(vmin[2], vmin[3]));
        unsigned local_max = max(static_cast<unsigned>(hi), static_cast<unsigned>(-static_cast<long long>(lo)));
        local_max = __reduce_max_sync(0xFFFFFFFFu, local_max);
        // one atomic per CTA: atomics on one address serialise at the L2, and there are 8 warps x 148 CTAs
        if (lane == 0) warp_max[warp - 2] = local_max;
        named_barrier(EPI_BARRIER + 2, 256);
        if (threadIdx.x == 64) {
            unsigned m = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) m = max(m, warp_max[i]);
            if (m != 0 && p.maxabs != nullptr) atomicMax(p.maxabs, m);
        }
    }

    // ---------------------------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if (TWO) cluster_sync_all();  // the partner may still signal this CTA's barriers / have MMAs reading its memory
    if (warp == 1) {
        if (*abort_flag) __nanosleep(200000);  // let copies and MMAs already in flight land
        tc_fence_after();
        __syncwarp();
        if (TWO) tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS); else tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
    }
}

// ------------------------------------------------------------------------------------------------
// The epilogue of the kernels that narrow to int8: sixteen warps (four per scheduler) in four groups of four.  Group g
// takes its own columns of EVERY tile, 32 at a time, so that the load of an accumulator chunk, the 32 dependent
// integer sequences of its narrowing and its store overlap between the four warps of a scheduler.  Eight warps that
// held whole 128-column rows had two warps per scheduler and ran at 2.4 times the bound of the integer pipe: a launch
// was paced by its epilogue and not by the tensor pipe (first layer at batch 1024, one MMA step per tile: 120 us).
//   BN = 128: one 32-column chunk per group and tile;   BN = 256: two;
//   BN = 64:  two groups share a tile, the other two the next one.
// 18 warps (five on one scheduler) leave 96 registers per thread, which 32 accumulators at a time fit into.
// ------------------------------------------------------------------------------------------------
constexpr int EPI_WARPS = 16;
constexpr unsigned long long GRID_BARRIER_LIMIT_NS = 500000000ull;  // 0.5 s
constexpr int REQUANT_THREADS = 64 + 32 * EPI_WARPS;  // producer warp, MMA warp, epilogue warps
template <int BN>
struct EpiSplit {
    static constexpr int GROUPS = BN >= 128 ? 4 : BN / 32;  // warp groups that share a tile
    static constexpr int TILES = 4 / GROUPS;                // tiles worked on side by side
    static constexpr int COLS = BN / GROUPS;                // columns of a group
    static constexpr int CHUNKS = COLS / 32;
};
// Operand ring and accumulators of the kernels that narrow.  BN = 64 serves layers of up to 64 output channels: with
// 128-column tiles half of the tensor work, of the accumulator reads and of the weight traffic was padding.
template <int BN, bool TWO, int MODE>
struct RequantCfg {
    static constexpr int B_STAGE_BYTES = (TWO ? BN / 2 : BN) * ROW_BYTES;
    static constexpr int STAGE_BYTES = MODE == LOAD_HALO_RESIDENT ? HALO_A_BYTES
                                       : MODE == LOAD_HALO ? HALO_A_BYTES + 3 * B_STAGE_BYTES : PANEL_BYTES + B_STAGE_BYTES;
    static constexpr int RESIDENT_BYTES = MODE == LOAD_HALO_RESIDENT ? 9 * B_STAGE_BYTES : 0;
    static constexpr int STAGES = (216 * 1024 - RESIDENT_BYTES) / STAGE_BYTES;
    static constexpr int NACC = BN == 256 ? 2 : 4;  // streaming: accumulators in flight
    static constexpr int TABLE_BYTES = 2 * 4 * 128 * 4;  // parked: output row and pooled row of every row of the CTA's tiles
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + RESIDENT_BYTES + TABLE_BYTES + 1024 /*alignment slack*/ + 512 /*barriers*/;
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of a CTA");
};

// Streaming kernel: narrows with the shift in state[0]; the last CTA derives the true one from max|acc|.
// CODES: with the side codes, where the call has room for them.  Without them the registers suffice (128 -> 128 at 32x32, 128 images,
// stochastic: 33.3 -> 32.1 us, at 80 images 28.2 -> 26.5); 64-column tiles are 3 % slower like that and keep them.
template <int BN, bool TWO, int MODE, bool CODES>
__global__ void __launch_bounds__(REQUANT_THREADS, 1)
umma_requant_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
    using Cfg = RequantCfg<BN, TWO, MODE>;
    using Split = EpiSplit<BN>;
    constexpr int STAGES = Cfg::STAGES, NACC = Cfg::NACC;
    if (p.only_if_redo) {
        const int verdict = p.state[2] & 3;
        if (verdict == 0) return;  // the prediction was right: nothing to redo
        if (CODES && verdict == 2) {  // one bit too many was shifted out and the side codes hold what is missing
            requant_step_down(p.out8, p.side, p.mask, static_cast<long long>(p.M) * p.N / 16);
            return;
        }
    }

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES + Cfg::RESIDENT_BYTES);
    uint64_t* full_bar = bars;
    uint64_t* empty_bar = bars + STAGES;
    uint64_t* tfull_bar = bars + 2 * STAGES;
    uint64_t* tempty_bar = bars + 2 * STAGES + NACC;
    uint64_t* weights_bar = bars + 2 * STAGES + 2 * NACC;  // one per filter column (resident weights)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 2 * NACC + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile unsigned* warp_max = reinterpret_cast<volatile unsigned*>(tmem_slot + 4);  // one word per epilogue warp

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = TWO ? cluster_ctarank() : 0u;  // rank 0 of a pair issues the MMAs and owns the barriers the MMA thread waits on

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) { mbar_init(smem_u32(&full_bar[i]), 1); mbar_init(smem_u32(&empty_bar[i]), 1); }
        for (int i = 0; i < NACC; ++i) { mbar_init(smem_u32(&tfull_bar[i]), 1); mbar_init(smem_u32(&tempty_bar[i]), 4 * Split::GROUPS * (TWO ? 2 : 1)); }
        for (int i = 0; i < 3; ++i) mbar_init(smem_u32(&weights_bar[i]), 1);
        *abort_flag = 0;
        fence_barrier_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
    }
    if (warp == 1) {
        if (TWO) { tmem_alloc_pair(smem_u32(tmem_slot), NACC * BN); tmem_relinquish_pair(); }
        else     { tmem_alloc(smem_u32(tmem_slot), NACC * BN); tmem_relinquish(); }
    }
    tc_fence_before();
    __syncthreads();
    if (TWO) cluster_sync_all();  // the partner's barriers exist before anything is signalled across the pair
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const int total_tiles = p.m_tiles * p.n_tiles;  // TWO: m_tiles counts 256-row tiles of the pair; the reduction is never split here
    const int cta_first = TWO ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
    const int cta_step = TWO ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);

    if (warp == 0) {
        if constexpr (shares_rows(MODE)) producer_halo_role<BN, STAGES, Cfg::STAGE_BYTES, MODE == LOAD_HALO_RESIDENT>(smem, full_bar, empty_bar, smem_u32(weights_bar), &tmA, &tmB, p, abort_flag);
        else producer_role<BN, STAGES, Cfg::STAGE_BYTES, TWO, MODE == LOAD_ROWS32>(smem, full_bar, empty_bar, &tmA, &tmB, p, cta_first, cta_step, abort_flag);
        __syncwarp();  // reach the teardown's block-wide barrier as a converged warp
    } else if (warp == 1) {
        if (rank == 0) {
            if constexpr (shares_rows(MODE)) mma_halo_role<BN, STAGES, Cfg::STAGE_BYTES, NACC, MODE == LOAD_HALO_RESIDENT>(smem, full_bar, empty_bar, smem_u32(weights_bar), tfull_bar, tempty_bar, tmem_base, p, abort_flag);
            else mma_role<BN, STAGES, Cfg::STAGE_BYTES, NACC, TWO, MODE == LOAD_ROWS32>(smem, full_bar, empty_bar, tfull_bar, tempty_bar, tmem_base, p, cta_first, cta_step, abort_flag);
        }
        __syncwarp();
    } else {
        const int grp = (warp - 2) >> 2;
        const int q = warp & 3;  // TMEM lanes [32q, 32q+32) are the ones this warp may read
        const int row_in_tile = q * 32 + lane;
        const int cg = (grp % Split::GROUPS) * Split::COLS;
        const int shift = p.state[0];
        const unsigned long long seed = (p.mode == ROUND_STOCHASTIC && shift > 0) ? *p.seed : 0ull;
        // a first launch also keeps what the next lower shift would need (see narrow16_nearest_codes)
        const bool with_codes = CODES && p.mode == ROUND_NEAREST && shift >= 2 && !p.relu && p.side != nullptr && !p.only_if_redo;
        const int half = CODES && shift > 0 ? 1 << (shift - 1) : 0;
        const bool wide = rows_of_32(p.out8, p.N);
        int vmax[4] = {0, 0, 0, 0}, vmin[4] = {0, 0, 0, 0};
        // this thread's row inside a tile never changes: pixel offsets within the tile's box
        int row_w = 0, row_h = 0, row_n = 0;
        bool row_in_box = true;
        if (p.conv) {
            const int t_ = row_in_tile / p.BW;
            row_w = row_in_tile - t_ * p.BW; row_n = t_ / p.BH; row_h = t_ - row_n * p.BH;
            row_in_box = row_in_tile < p.BW * p.BH * p.BI;
        }
        int it = grp / Split::GROUPS;
        for (int tile = cta_first + it * cta_step; tile < total_tiles; tile += Split::TILES * cta_step, it += Split::TILES) {
            const int acc = it & (NACC - 1); const uint32_t aph = (it / NACC) & 1u;
            // where the tile lies, and the mask of the first chunk, before waiting for its accumulator
            int m_pair, n_t;
            tile_coords(p, tile, &m_pair, &n_t);
            const int m_t = TWO ? 2 * m_pair + static_cast<int>(rank) : m_pair;
            bool valid; long long row;  // row of the output tensor (there may be more than 2^31)
            if (p.conv) {
                const int q1 = fdiv(m_t, p.fd_tw), tw = m_t - q1 * p.tiles_w, tn = fdiv(q1, p.fd_th), th = q1 - tn * p.tiles_h;
                const int w = tw * p.BW + row_w, h = th * p.BH + row_h, n = tn * p.BI + row_n;
                valid = row_in_box && w < p.W && h < p.H && n < p.Nimg;
                row = (static_cast<long long>(n) * p.H + h) * p.W + w;
            } else {
                row = static_cast<long long>(m_t) * BLOCK_M + row_in_tile;
                valid = row < p.M;
            }
            const int col0 = n_t * BN + cg;
            const long long off = row * p.N + col0;  // of this thread's first output
            const int8_t* mrow = (p.mask != nullptr && valid && col0 < p.N) ? p.mask + off : nullptr;
            uint4 mk[2];
            mask_load<2>(mrow, p.N - col0, mk);
            const bool up = mbar_wait(smem_u32(&tfull_bar[acc]), aph, abort_flag);
            if (!__all_sync(0xFFFFFFFFu, up)) { if (!up) report_abort(p.status, 4, 2); break; }
            tc_fence_after();
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * BN + cg);
#pragma unroll 1
            for (int c = 0; c < Split::CHUNKS; ++c) {
                const int cols = p.N - col0 - 32 * c;  // columns of the tensor from here on
                uint32_t v[32], packed[8];
                tmem_ld_32x32(taddr + 32 * c, v);
                if (c > 0) mask_load<2>(mrow == nullptr ? nullptr : mrow + 32 * c, cols, mk);
                tmem_ld_wait();
                if (c == Split::CHUNKS - 1) {  // this warp's last columns sit in registers: hand the accumulator back
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (TWO) mbar_arrive_cluster(mapa_u32(smem_u32(&tempty_bar[acc]), 0));
                        else     mbar_arrive(smem_u32(&tempty_bar[acc]));
                    }
                }
                if (cols <= 0) continue;
                if (valid) minmax32(v, cols, vmax, vmin);
                if (with_codes) {
                    uint32_t codes[2];
#pragma unroll
                    for (int i = 0; i < 32; i += 16) codes[i >> 4] = narrow16_nearest_codes(&v[i], shift - 2, half, &packed[i >> 2]);
                    if (valid) {  // 16 outputs per word, rows of N / 4 bytes
                        uint32_t* srow = p.side + ((off + 32 * c) >> 4);
                        srow[0] = codes[0];
                        if (cols >= 32) srow[1] = codes[1];
                    }
                } else {
                    narrow32(v, packed, shift, p.mode, p.relu, seed, p.rng_stream, p.rng_offset + static_cast<unsigned long long>(off) + 32 * c);
                }
                mask_apply<2>(packed, mrow, cols, mk);
                store_piece(valid ? p.out8 + off + 32 * c : nullptr, cols, packed, wide);
            }
        }
        const unsigned local_max = __reduce_max_sync(0xFFFFFFFFu, fold_minmax(vmax, vmin));
        // one atomic per CTA: atomics on one address serialise at the L2, and there are 16 warps x 148 CTAs
        if (lane == 0) warp_max[warp - 2] = local_max;
        named_barrier(EPI_BARRIER, 32 * EPI_WARPS);
        if (threadIdx.x == 64) {
            unsigned m = 0;
#pragma unroll
            for (int i = 0; i < EPI_WARPS; ++i) m = max(m, warp_max[i]);
            if (m != 0 && p.maxabs != nullptr) atomicMax(p.maxabs, m);
        }
        // the CTA that finishes last turns max|acc| into the true shift and checks the prediction
        if (!p.only_if_redo && threadIdx.x == 64) {
            __threadfence();
            int32_t* st = p.state;
            if (atomicAdd(&st[4], 1) == static_cast<int>(gridDim.x) - 1) {
                __threadfence();
                bool zero_out;
                const unsigned m = static_cast<unsigned>(atomicMax(reinterpret_cast<unsigned*>(&st[1]), 0u));
                const int true_shift = shift_for(m, p.kind, p.target_bits, &zero_out);
                // st[2] = verdict (0 right, 1 launch again, 2 step the output down one shift from the side codes)
                //         | run of step-downs << 4 | step-downs so far << 8
                const int pred = st[0];
                const unsigned old = static_cast<unsigned>(st[2]);
                unsigned run = (old >> 4) & 15u, downs = old >> 8;
                int verdict = 0;
                if (true_shift == pred) {
                    run = 0;
                } else if (CODES && p.side != nullptr && p.mode == ROUND_NEAREST && !p.relu && pred >= 2 && true_shift == pred - 1) {
                    // the prediction stays: a layer whose maximum hovers around a power of two keeps the upper
                    // shift as its guess and pays the cheap pass when the lower one applies; after
                    // STEP_DOWN_RUN lower ones in a row the guess follows
                    verdict = 2;
                    ++downs;
                    if (++run >= STEP_DOWN_RUN) { run = 0; st[0] = true_shift; }
                } else {
                    verdict = 1;
                    run = 0;
                    st[3] += 1;
                    st[0] = true_shift;
                }
                st[2] = static_cast<int>(static_cast<unsigned>(verdict) | (run << 4) | (downs << 8));
                st[1] = 0;  // ready for the next call
                st[4] = 0;
                if (p.exp_out) *p.exp_out = true_shift + (p.exp_a ? *p.exp_a : 0) + (p.exp_b ? *p.exp_b : 0);
                if (p.shift_out) *p.shift_out = true_shift;
            }
        }
    }

    // ---------------------------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if (TWO) cluster_sync_all();  // the partner may still signal this CTA's barriers / have MMAs reading its memory
    if (warp == 1) {
        if (*abort_flag) __nanosleep(200000);  // let copies and MMAs already in flight land
        tc_fence_after();
        __syncwarp();
        if (TWO) tmem_dealloc_pair(tmem_base, NACC * BN); else tmem_dealloc(tmem_base, NACC * BN);
    }
}

// The grid barrier of the narrowing kernels below (streaming in one launch, parked, shared tiles), run by a CTA's epilogue
// warps (which have left their maxima in warp_max): every CTA has contributed its maximum when it returns the shift that
// narrows the tensor, the same to all of them; -1 where the others did not arrive or a role of this CTA gave up.
// One atomic per CTA: atomics on one address serialise at the L2; the waiters poll with plain acquire loads for the same reason.
// The exit ticket (thread 64's) is drawn as soon as this CTA has read the barrier's words, so that its round trip runs under
// the narrowing; drawn at the end, behind a barrier of the epilogue warps, it was 0.45 us of every launch.
__device__ __forceinline__ int parked_grid_shift(const GemmParams& p, const volatile unsigned* warp_max, volatile int* shift_slot,
                                                 volatile int* abort_flag, int* ticket) {
    int32_t* st = p.state;
    named_barrier(EPI_BARRIER, 32 * EPI_WARPS);
    if (threadIdx.x == 64) {
        unsigned cta_max = 0;
#pragma unroll
        for (int i = 0; i < EPI_WARPS; ++i) cta_max = max(cta_max, warp_max[i]);
        // The maximum and the arrival count sit side by side (st[6], st[7]): two fire-and-forget reductions on the
        // way in (the count's release orders the maximum before it), ONE 64-bit acquire load per poll that returns
        // both -- a fence + atomicAdd + atomicMax read-back would add three round trips to the L2.
        if (cta_max != 0) red_relaxed_max(reinterpret_cast<unsigned*>(&st[6]), cta_max);
        red_release_add(&st[7], 1);
        const unsigned long long t0 = global_timer_ns();
        bool arrived = false;
        unsigned m = 0;
        for (unsigned spin = 0;; ++spin) {
            const unsigned long long both = ld_acquire_gpu_u64(&st[6]);
            if (static_cast<int>(both >> 32) >= static_cast<int>(gridDim.x)) { arrived = true; m = static_cast<unsigned>(both); break; }
            if ((spin & 63) == 63) {
                if (*abort_flag || global_timer_ns() - t0 > GRID_BARRIER_LIMIT_NS) break;
            }
        }
        bool zero_out;
        *shift_slot = arrived && !*abort_flag ? shift_for(m, p.kind, p.target_bits, &zero_out) : -1;
        if (!arrived) { *abort_flag = 1; report_abort(p.status, 5, 2); }
    }
    named_barrier(EPI_BARRIER, 32 * EPI_WARPS);
    if (threadIdx.x == 64) *ticket = atomicAdd(&st[4], 1);
    return *shift_slot;
}
// the CTA that drew the last ticket publishes the shift and clears the words for the next call
__device__ __forceinline__ void parked_leave(const GemmParams& p, int shift, int ticket) {
    int32_t* st = p.state;
    if (threadIdx.x == 64) {
        if (ticket == static_cast<int>(gridDim.x) - 1) {
            const int s_out = shift < 0 ? 0 : shift;
            st[0] = s_out; st[2] = 0; st[1] = 0; st[5] = 0; st[4] = 0; st[6] = 0; st[7] = 0;
            if (p.exp_out) *p.exp_out = s_out + (p.exp_a ? *p.exp_a : 0) + (p.exp_b ? *p.exp_b : 0);
            if (p.shift_out) *p.shift_out = s_out;
        }
    }
}

// Forward layers: a cooperative launch, whose CTAs meet at a grid barrier behind their last tile, know the true shift and where the
// guess was wrong contract and narrow again.  The conditional second launch of the kernel above cost a layer whose guess was right
// 1 us in a graph and 2 to 4 in a stream, and without masks and side codes the epilogue needs no spills (us, before / after: 64 ->
// 128 on 400 16x16 maps 17.9 / 15.6, 128 -> 128 at 32x32, 128 images 20.8 / 19.3 and stochastic 30.2 / 27.0, 500 8x8 maps of 512
// channels 54.8 / 51.9; the first layer's product the same way: evaluation of 500 images 397 / 392).  The error's way back keeps the kernel above: with the ReLU mask in the epilogue a second pass in the same
// kernel costs large layers up to 16 %, and a guess one shift too high is repaired from the side codes there.
// One pass of a CTA over its tiles, all warps; AGAIN: the second one, whose shift is known.  (A pass number in a loop around the
// body cost it 170 bytes of spills and up to 20 % of the time.)
template <int BN, int MODE, bool AGAIN>
__device__ __forceinline__ void requant_pass(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p, uint8_t* smem, uint64_t* bars,
                                             uint32_t* tmem_slot) {
    using Cfg = RequantCfg<BN, false, MODE>;
    using Split = EpiSplit<BN>;
    constexpr int STAGES = Cfg::STAGES, NACC = Cfg::NACC;
    const uint32_t tmem_base = *tmem_slot;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* again_slot = reinterpret_cast<volatile int*>(tmem_slot + 2);
    volatile int* shift_slot = reinterpret_cast<volatile int*>(tmem_slot + 3);
    volatile unsigned* warp_max = reinterpret_cast<volatile unsigned*>(tmem_slot + 4);  // one word per epilogue warp
    uint64_t* full_bar = bars;
    uint64_t* empty_bar = bars + STAGES;
    uint64_t* tfull_bar = bars + 2 * STAGES;
    uint64_t* tempty_bar = bars + 2 * STAGES + NACC;
    uint64_t* weights_bar = bars + 2 * STAGES + 2 * NACC;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int total_tiles = p.m_tiles * p.n_tiles;
    const int cta_first = static_cast<int>(blockIdx.x), cta_step = static_cast<int>(gridDim.x);

    if (warp == 0) {
        if constexpr (shares_rows(MODE)) producer_halo_role<BN, STAGES, Cfg::STAGE_BYTES, MODE == LOAD_HALO_RESIDENT>(smem, full_bar, empty_bar, smem_u32(weights_bar), &tmA, &tmB, p, abort_flag);
        else producer_role<BN, STAGES, Cfg::STAGE_BYTES, false, MODE == LOAD_ROWS32>(smem, full_bar, empty_bar, &tmA, &tmB, p, cta_first, cta_step, abort_flag);
        __syncwarp();  // reach the teardown's block-wide barrier as a converged warp
    } else if (warp == 1) {
        if constexpr (shares_rows(MODE)) mma_halo_role<BN, STAGES, Cfg::STAGE_BYTES, NACC, MODE == LOAD_HALO_RESIDENT>(smem, full_bar, empty_bar, smem_u32(weights_bar), tfull_bar, tempty_bar, tmem_base, p, abort_flag);
        else mma_role<BN, STAGES, Cfg::STAGE_BYTES, NACC, false, MODE == LOAD_ROWS32>(smem, full_bar, empty_bar, tfull_bar, tempty_bar, tmem_base, p, cta_first, cta_step, abort_flag);
        __syncwarp();
    } else {
        const int grp = (warp - 2) >> 2;
        const int q = warp & 3;  // TMEM lanes [32q, 32q+32) are the ones this warp may read
        const int row_in_tile = q * 32 + lane;
        const int cg = (grp % Split::GROUPS) * Split::COLS;
        const int shift = AGAIN ? *shift_slot : p.state[0];
        const unsigned long long seed = (p.mode == ROUND_STOCHASTIC && shift > 0) ? *p.seed : 0ull;
        const bool wide = rows_of_32(p.out8, p.N);
        int vmax[4] = {0, 0, 0, 0}, vmin[4] = {0, 0, 0, 0};
        // this thread's row inside a tile never changes: pixel offsets within the tile's box
        int row_w = 0, row_h = 0, row_n = 0;
        bool row_in_box = true;
        if (p.conv) {
            const int t_ = row_in_tile / p.BW;
            row_w = row_in_tile - t_ * p.BW; row_n = t_ / p.BH; row_h = t_ - row_n * p.BH;
            row_in_box = row_in_tile < p.BW * p.BH * p.BI;
        }
        int it = grp / Split::GROUPS;
        for (int tile = cta_first + it * cta_step; tile < total_tiles; tile += Split::TILES * cta_step, it += Split::TILES) {
            const int acc = it & (NACC - 1); const uint32_t aph = (it / NACC) & 1u;
            // where the tile lies, before waiting for its accumulator
            int m_t, n_t;
            tile_coords(p, tile, &m_t, &n_t);
            bool valid; long long row;  // row of the output tensor (there may be more than 2^31)
            if (p.conv) {
                const int q1 = fdiv(m_t, p.fd_tw), tw = m_t - q1 * p.tiles_w, tn = fdiv(q1, p.fd_th), th = q1 - tn * p.tiles_h;
                const int w = tw * p.BW + row_w, h = th * p.BH + row_h, n = tn * p.BI + row_n;
                valid = row_in_box && w < p.W && h < p.H && n < p.Nimg;
                row = (static_cast<long long>(n) * p.H + h) * p.W + w;
            } else {
                row = static_cast<long long>(m_t) * BLOCK_M + row_in_tile;
                valid = row < p.M;
            }
            const int col0 = n_t * BN + cg;
            const long long off = row * p.N + col0;  // of this thread's first output
            const bool up = mbar_wait(smem_u32(&tfull_bar[acc]), aph, abort_flag);
            if (!__all_sync(0xFFFFFFFFu, up)) { if (!up) report_abort(p.status, 4, 2); break; }
            tc_fence_after();
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * BN + cg);
#pragma unroll 1
            for (int c = 0; c < Split::CHUNKS; ++c) {
                const int cols = p.N - col0 - 32 * c;  // columns of the tensor from here on
                uint32_t v[32], packed[8];
                tmem_ld_32x32(taddr + 32 * c, v);
                tmem_ld_wait();
                if (c == Split::CHUNKS - 1) {  // this warp's last columns sit in registers: hand the accumulator back
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&tempty_bar[acc]));
                }
                if (cols <= 0) continue;
                if (!AGAIN && valid) minmax32(v, cols, vmax, vmin);
                narrow32(v, packed, shift, p.mode, p.relu, seed, p.rng_stream, p.rng_offset + static_cast<unsigned long long>(off) + 32 * c);
                store_piece(valid ? p.out8 + off + 32 * c : nullptr, cols, packed, wide);
            }
        }
        if (AGAIN) return;
        const unsigned local_max = __reduce_max_sync(0xFFFFFFFFu, fold_minmax(vmax, vmin));
        if (lane == 0) warp_max[warp - 2] = local_max;
        int ticket = -1;
        const int true_shift = parked_grid_shift(p, warp_max, shift_slot, abort_flag, &ticket);  // (releases the CTA's outputs too)
        if (threadIdx.x == 64) {
            *again_slot = true_shift >= 0 && true_shift != shift ? 1 : 0;
            if (ticket == static_cast<int>(gridDim.x) - 1) {  // every CTA has read its guess and the barrier's words
                int32_t* st = p.state;
                const int s_out = true_shift < 0 ? 0 : true_shift;
                const bool again = true_shift >= 0 && true_shift != shift;
                if (again) { st[3] += 1; st[0] = true_shift; }
                st[2] = again ? 1 : 0; st[1] = 0; st[4] = 0; st[5] = 0; st[6] = 0; st[7] = 0;  // ready for the next call
                if (p.exp_out) *p.exp_out = s_out + (p.exp_a ? *p.exp_a : 0) + (p.exp_b ? *p.exp_b : 0);
                if (p.shift_out) *p.shift_out = s_out;
            }
        }
    }
}

// What a CTA keeps in shared memory behind the operand ring: the barriers of one pass, of a second, and a few words.
template <int BN, int MODE>
struct RequantShared {
    static constexpr int BARS = 2 * RequantCfg<BN, false, MODE>::STAGES + 2 * RequantCfg<BN, false, MODE>::NACC + 3;  // stages full and free, accumulators, weights
    uint8_t* smem; uint64_t* bars; uint32_t* tmem_slot;
    __device__ __forceinline__ explicit RequantShared(uint8_t* raw) {
        using Cfg = RequantCfg<BN, false, MODE>;
        smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
        bars = reinterpret_cast<uint64_t*>(smem + Cfg::STAGES * Cfg::STAGE_BYTES + Cfg::RESIDENT_BYTES);
        tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * BARS);
    }
    // The same addresses worked out anew behind a pass instead of kept through it: its epilogue has no register to spare.
    static __device__ __forceinline__ RequantShared again(uint8_t* raw) {
        int zero;
        asm volatile("mov.u32 %0, 0;" : "=r"(zero));
        return RequantShared(raw + zero);
    }
};

template <int BN, int MODE>
__global__ void __launch_bounds__(REQUANT_THREADS, 1)
umma_requant_once_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
    using Cfg = RequantCfg<BN, false, MODE>;
    constexpr int NACC = Cfg::NACC, BARS = RequantShared<BN, MODE>::BARS;
    extern __shared__ uint8_t smem_raw[];
    {
        const RequantShared<BN, MODE> sh(smem_raw);
        if (threadIdx.x == 0) {
            for (int b = 0; b < 2; ++b)
                for (int i = 0; i < BARS; ++i)  // the accumulators come back from the warps that share a tile
                    mbar_init(smem_u32(&sh.bars[b * BARS + i]), i >= BARS - 3 - NACC && i < BARS - 3 ? 4 * EpiSplit<BN>::GROUPS : 1);
            sh.tmem_slot[1] = 0;  // abort flag
            sh.tmem_slot[2] = 0;  // a second pass
            fence_barrier_init();
            tma_prefetch_desc(&tmA);
            tma_prefetch_desc(&tmB);
        }
        if (threadIdx.x >> 5 == 1) { tmem_alloc(smem_u32(sh.tmem_slot), NACC * BN); tmem_relinquish(); }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        requant_pass<BN, MODE, false>(tmA, tmB, p, sh.smem, sh.bars, sh.tmem_slot);
    }
    const auto sh = RequantShared<BN, MODE>::again(smem_raw);
    tc_fence_before();
    __syncthreads();
    if (static_cast<volatile uint32_t*>(sh.tmem_slot)[2] != 0) {  // with barriers of its own: commits of the first pass may still be on their way to theirs
        tc_fence_after();
        requant_pass<BN, MODE, true>(tmA, tmB, p, sh.smem, sh.bars + BARS, sh.tmem_slot);
        tc_fence_before();
        __syncthreads();
    }
    if (threadIdx.x >> 5 == 1) {
        const uint32_t tmem_base = *sh.tmem_slot;
        if (static_cast<volatile uint32_t*>(sh.tmem_slot)[1]) __nanosleep(200000);  // let copies and MMAs already in flight land
        tc_fence_after();
        __syncwarp();
        tmem_dealloc(tmem_base, NACC * BN);
    }
}

// ------------------------------------------------------------------------------------------------
// Exact single-pass requantisation for problems whose accumulators all fit in tensor memory:
// every CTA owns at most 512 / BN output tiles and PARKS their int32 accumulators in TMEM.  After
// its main loops a CTA reduces max|acc| of its tiles into the global word, all CTAs meet at a grid
// barrier (cooperative launch: all resident; bounded spin), read the now final max, derive the true
// shift and only then narrow their parked accumulators to int8.  No prediction, no second launch,
// no int32 in memory.  state = {shift out, max|acc|, redo flag (cleared), redo count, exit ticket,
// -, max|acc| and barrier arrivals (adjacent: read with one 64-bit load)}; words 1, 4, 5, 6 and 7 are zero between calls.
// ------------------------------------------------------------------------------------------------
template <int BN, bool TWO, int MODE>
__global__ void __launch_bounds__(REQUANT_THREADS, 1)
umma_parked_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
    using Cfg = RequantCfg<BN, TWO, MODE>;
    using Split = EpiSplit<BN>;
    constexpr int STAGES = Cfg::STAGES;
    static_assert(BN >= 128 && 512 / BN <= 4, "all four warp groups share every tile; tables of four tiles");
    if (threadIdx.x == 0) PARK_STAMP(0);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    int32_t* out_row = reinterpret_cast<int32_t*>(smem + STAGES * Cfg::STAGE_BYTES + Cfg::RESIDENT_BYTES);  // [tile][row of the tile]; -1: outside the tensor
    int32_t* pool_row = out_row + 4 * 128;
    uint64_t* bars = reinterpret_cast<uint64_t*>(pool_row + 4 * 128);
    uint64_t* full_bar = bars;
    uint64_t* empty_bar = bars + STAGES;
    uint64_t* tfull_bar = bars + 2 * STAGES;  // one per parked tile (up to 4)
    uint64_t* weights_bar = bars + 2 * STAGES + 4;  // one per filter column (resident weights)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* shift_slot = reinterpret_cast<volatile int*>(tmem_slot + 2);
    volatile unsigned* warp_max = reinterpret_cast<volatile unsigned*>(tmem_slot + 4);  // one word per epilogue warp

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = TWO ? cluster_ctarank() : 0u;

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) { mbar_init(smem_u32(&full_bar[i]), 1); mbar_init(smem_u32(&empty_bar[i]), 1); }
        for (int i = 0; i < 4; ++i) mbar_init(smem_u32(&tfull_bar[i]), 1);
        for (int i = 0; i < 3; ++i) mbar_init(smem_u32(&weights_bar[i]), 1);
        *abort_flag = 0;
        fence_barrier_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
    }
    if (warp == 1) {
        if (TWO) { tmem_alloc_pair(smem_u32(tmem_slot), 512); tmem_relinquish_pair(); }
        else     { tmem_alloc(smem_u32(tmem_slot), 512); tmem_relinquish(); }
    }
    tc_fence_before();
    __syncthreads();
    if (TWO) cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (threadIdx.x == 0) PARK_STAMP(1);

    const int total_tiles = p.m_tiles * p.n_tiles;  // TWO: m_tiles counts 256-row tiles of the pair
    const int cta_first = TWO ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
    const int cta_step = TWO ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);

    if (warp == 0) {
        if constexpr (shares_rows(MODE)) producer_halo_role<BN, STAGES, Cfg::STAGE_BYTES, MODE == LOAD_HALO_RESIDENT>(smem, full_bar, empty_bar, smem_u32(weights_bar), &tmA, &tmB, p, abort_flag);
        else producer_role<BN, STAGES, Cfg::STAGE_BYTES, TWO, MODE == LOAD_ROWS32>(smem, full_bar, empty_bar, &tmA, &tmB, p, cta_first, cta_step, abort_flag);
        __syncwarp();  // reach the teardown's block-wide barrier as a converged warp
    } else if (warp == 1) {
        if (rank == 0) {
            if constexpr (shares_rows(MODE)) mma_halo_role<BN, STAGES, Cfg::STAGE_BYTES, 0, MODE == LOAD_HALO_RESIDENT>(smem, full_bar, empty_bar, smem_u32(weights_bar), tfull_bar, nullptr, tmem_base, p, abort_flag);
            else mma_role<BN, STAGES, Cfg::STAGE_BYTES, 0, TWO, false>(smem, full_bar, empty_bar, tfull_bar, nullptr, tmem_base, p, cta_first, cta_step, abort_flag);
        }
        __syncwarp();
    } else {
        const int grp = (warp - 2) >> 2;
        const int q = warp & 3;
        const int row_in_tile = q * 32 + lane;
        const int cg = grp * Split::COLS;
        int my_tiles = 0;
        for (int tile = cta_first; tile < total_tiles; tile += cta_step) ++my_tiles;

        // Where the rows of the CTA's tiles go is worked out while the main loop runs: group g fills the table of tile g.
        if (grp < my_tiles) {
            int m_pair, n_t;
            tile_coords(p, cta_first + grp * cta_step, &m_pair, &n_t);
            const int m_t = TWO ? 2 * m_pair + static_cast<int>(rank) : m_pair;
            const int q1 = fdiv(m_t, p.fd_tw), tw = m_t - q1 * p.tiles_w, tn = fdiv(q1, p.fd_th), th = q1 - tn * p.tiles_h;
            const int w = tw * p.BW + row_in_tile % p.BW;
            const int h = th * p.BH + (row_in_tile / p.BW) % p.BH;
            const int n = tn * p.BI + row_in_tile / (p.BW * p.BH);
            const bool valid = row_in_tile < p.BW * p.BH * p.BI && w < p.W && h < p.H && n < p.Nimg;
            const int row = valid ? (n * p.H + h) * p.W + w : -1;
            out_row[grp * 128 + row_in_tile] = row;
            // row of the 2x2-pooled tensor this pixel's window goes to; only the window's top-left pixel writes it
            pool_row[grp * 128 + row_in_tile] = (valid && ((w | h) & 1) == 0) ? (n * (p.H >> 1) + (h >> 1)) * (p.W >> 1) + (w >> 1) : -1;
            // the ReLU mask this row will be gated with after the main loop: start moving it towards the L2 now
            if (p.mask != nullptr && valid)
                for (int c = n_t * BN; c < p.N && c < n_t * BN + BN; c += 128) prefetch_l2(p.mask + static_cast<long long>(row) * p.N + c);
        }
        named_barrier(EPI_BARRIER, 32 * EPI_WARPS);

        // ---- pass 1: max|acc| of this CTA's tiles.  Rolled loops in both passes: code that runs a few times per launch is
        //      bound by instruction fetch, and the four warps of a scheduler hide each other's latencies
        int vmax[4] = {0, 0, 0, 0}, vmin[4] = {0, 0, 0, 0};
        bool ok = true;
#pragma unroll 1
        for (int it = 0; it < my_tiles; ++it) {
            const bool up = mbar_wait(smem_u32(&tfull_bar[it]), 0, abort_flag);
            if (!__all_sync(0xFFFFFFFFu, up)) { if (!up) report_abort(p.status, 4, 2); ok = false; break; }
            if (threadIdx.x == 64 && it == 0) PARK_STAMP(4);
            tc_fence_after();
            const int tile = cta_first + it * cta_step, col0 = (tile - fdiv(tile, p.fd_n) * p.n_tiles) * BN + cg;
            const bool valid = out_row[it * 128 + row_in_tile] >= 0;
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(it * BN + cg);
#pragma unroll 1
            for (int c = 0; c < Split::CHUNKS; ++c) {
                const int cols = p.N - col0 - 32 * c;
                if (cols <= 0) break;
                uint32_t v[32];
                tmem_ld_32x32(taddr + 32 * c, v);
                tmem_ld_wait();
                if (valid) minmax32(v, cols, vmax, vmin);
            }
        }
        const unsigned local_max = __reduce_max_sync(0xFFFFFFFFu, fold_minmax(vmax, vmin));
        if (lane == 0) warp_max[warp - 2] = local_max;
        if (threadIdx.x == 64) PARK_STAMP(5);
        int ticket = -1;
        const int shift = parked_grid_shift(p, warp_max, shift_slot, abort_flag, &ticket);
        if (threadIdx.x == 64) PARK_STAMP(6);

        // ---- pass 2: narrow the parked accumulators with the true shift
        if (ok && shift >= 0) {
            const unsigned long long seed = (p.mode == ROUND_STOCHASTIC && shift > 0) ? *p.seed : 0ull;
            const bool wide = rows_of_32(p.out8, p.N);
            // Max pooling in the same pass (TiMaxpool2d.forward): a warp's 32 rows are whole image rows of the tile
            // (BW is a power of two <= 16, BH even), so the 2x2 window of lane l is lanes l, l^1, l^BW, l^BW^1:
            // two shuffles and two byte-wise maxima per word, and the window's top-left lane stores the pooled piece.
            const bool pooling = p.pool_out != nullptr;  // the same for the whole grid
            const bool wide_pool = pooling && rows_of_32(p.pool_out, p.N);
#pragma unroll 1
            for (int it = 0; it < my_tiles; ++it) {
                const int tile = cta_first + it * cta_step, col0 = (tile - fdiv(tile, p.fd_n) * p.n_tiles) * BN + cg;
                const int row = out_row[it * 128 + row_in_tile], prow = pool_row[it * 128 + row_in_tile];
                const long long off = static_cast<long long>(max(row, 0)) * p.N + col0;  // rows outside the tensor go through the same form as the others
                const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(it * BN + cg);
#pragma unroll 1
                for (int c = 0; c < Split::CHUNKS; ++c) {
                    const int cols = p.N - col0 - 32 * c;  // columns of the tensor from here on; the same for the whole warp
                    if (cols <= 0) break;
                    const int8_t* mrow = (p.mask != nullptr && row >= 0) ? p.mask + off + 32 * c : nullptr;
                    uint32_t v[32], packed[8];
                    uint4 mk[2];
                    tmem_ld_32x32(taddr + 32 * c, v);
                    mask_load<2>(mrow, cols, mk);
                    tmem_ld_wait();
                    narrow32(v, packed, shift, p.mode, p.relu, seed, p.rng_stream, p.rng_offset + static_cast<unsigned long long>(off) + 32 * c);
                    mask_apply<2>(packed, mrow, cols, mk);
                    // every thread writes its own row straight from registers (32-byte pieces = whole L2 sectors)
                    store_piece(row >= 0 ? p.out8 + off + 32 * c : nullptr, cols, packed, wide);
                    if (pooling) {
                        pool_window(packed, p.BW);
                        store_piece(prow >= 0 ? p.pool_out + static_cast<long long>(prow) * p.N + col0 + 32 * c : nullptr, cols, packed, wide_pool);
                    }
                }
            }
        }
        if (threadIdx.x == 64) PARK_STAMP(7);
        parked_leave(p, shift, ticket);
    }

    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0) PARK_STAMP(8);
    if (TWO) cluster_sync_all();
    if (warp == 1) {
        if (*abort_flag) __nanosleep(200000);
        tc_fence_after();
        __syncwarp();
        if (TWO) tmem_dealloc_pair(tmem_base, 512); else tmem_dealloc(tmem_base, 512);
    }
}

// ------------------------------------------------------------------------------------------------
// Few output tiles: a cluster of CS thread blocks shares one tile's REDUCTION.
// A convolution of 16 tiles (512 -> 512 at 4x4, 32 images) kept 16 of the 148 SMs busy with 36 reduction blocks each, a
// single image one to four of them.  Here CTA r of a cluster contracts its share of the reduction blocks into its own tensor
// memory, the partial sums meet in distributed shared memory, and CTA r owns rows [r 128/CS, (r + 1) 128/CS) of the tile from
// there on: it adds the CS partial sums (int32, exact in any order), takes the tensor-wide maximum over the same grid barrier
// as the parked kernel and narrows its rows, so the epilogue is shared out as well.
//   exchange  every warp writes its 32 x 32 partial sums into the CTA's (by then idle) operand ring, 128-byte rows with their
//             16-byte chunks exchanged by the row number (both passes free of bank conflicts), and sends them to the rows'
//             owners as bulk copies of 2 or 4 KB into their receive slots, counted on their mbarriers, without waiting for the
//             other warps: (CS - 1) / CS x 64 KB per CTA and direction.
//   cluster   both cluster-wide barriers (peers exist; peers are done) are arrived at early and waited for late.
//   rows      a warp works on whole rows from here (lane = four columns): row coordinates are uniform, stores are 128
//             contiguous bytes, a lane's four outputs are one Philox block.
// state and grid barrier: as umma_parked_kernel.
// ------------------------------------------------------------------------------------------------
template <int CS>
struct SplitCfg {
    static constexpr int BN = 128;
    static constexpr int RPC = 128 / CS;                       // rows of the tile a CTA owns
    static constexpr int SLOT_BYTES = RPC * BN * 4;            // an owner's rows: four panels of 32 columns
    static constexpr int RECV_BYTES = (CS - 1) * SLOT_BYTES;
    static constexpr int STAGE_BYTES = PANEL_BYTES + BN * ROW_BYTES;
    static constexpr int STAGES = 5;
    static constexpr int POOL_BYTES = RPC * BN;                // the CTA's int8 rows, for the pooling windows
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + RECV_BYTES + POOL_BYTES + 1024 /*alignment slack*/ + 512 /*barriers*/;
    static_assert(CS * SLOT_BYTES <= STAGES * STAGE_BYTES, "the partial sums are staged in the ring");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of a CTA");
};

// Four accumulators, any rounding and shift, random words from any element on: a call of its own, so that the rare forms are
// not fetched on the way to the common ones.
__device__ __noinline__ uint32_t narrow4_general(uint32_t a, uint32_t b, uint32_t c, uint32_t d, int shift, int mode,
                                                 unsigned long long seed, unsigned rng_stream, unsigned long long e) {
    const uint32_t v[4] = {a, b, c, d};
    uint32_t w = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t rnd = mode == ROUND_STOCHASTIC && shift > 0 ? random_word(seed, rng_stream, e + j) : 0u;
        w |= static_cast<uint32_t>(static_cast<uint8_t>(narrow(static_cast<int>(v[j]), shift, mode, rnd))) << (8 * j);
    }
    return w;
}

template <int CS>
__global__ void __launch_bounds__(REQUANT_THREADS, 1)
umma_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
    using Cfg = SplitCfg<CS>;
    constexpr int STAGES = Cfg::STAGES, RPC = Cfg::RPC, BN = Cfg::BN;
    constexpr int ROWS = RPC / EPI_WARPS;  // rows of a warp: 4, 2 or 1
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* recv = smem + STAGES * Cfg::STAGE_BYTES;
    uint32_t* pool_rows = reinterpret_cast<uint32_t*>(recv + Cfg::RECV_BYTES);
    uint64_t* bars = reinterpret_cast<uint64_t*>(recv + Cfg::RECV_BYTES + Cfg::POOL_BYTES);
    uint64_t* full_bar = bars;
    uint64_t* empty_bar = bars + STAGES;
    uint64_t* tfull_bar = bars + 2 * STAGES;
    uint64_t* recv_bar = bars + 2 * STAGES + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* shift_slot = reinterpret_cast<volatile int*>(tmem_slot + 2);
    volatile unsigned* warp_max = reinterpret_cast<volatile unsigned*>(tmem_slot + 4);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int rank = static_cast<int>(__shfl_sync(0xFFFFFFFFu, cluster_ctarank(), 0));

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) { mbar_init(smem_u32(&full_bar[i]), 1); mbar_init(smem_u32(&empty_bar[i]), 1); }
        mbar_init(smem_u32(tfull_bar), 1);
        mbar_init(smem_u32(recv_bar), 1);
        *abort_flag = 0;
        fence_barrier_init();
        mbar_arrive_expect_tx(smem_u32(recv_bar), Cfg::RECV_BYTES);  // its one arrival; the peers' copies bring the bytes
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
    }
    if (warp == 1) { tmem_alloc(smem_u32(tmem_slot), BN); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    cluster_arrive();  // this CTA's barriers exist: peers may send (each warp waits for the others' before it sends)
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // the roles see a split reduction: one work item per CTA, numbered split-major
    const int mn_tiles = p.m_tiles * p.n_tiles;
    const int tile = static_cast<int>(blockIdx.x) / CS;
    const int cta_first = rank * mn_tiles + tile, cta_step = CS * mn_tiles;

    if (warp == 0) {
        producer_role<BN, STAGES, Cfg::STAGE_BYTES, false, false>(smem, full_bar, empty_bar, &tmA, &tmB, p, cta_first, cta_step, abort_flag);
        __syncwarp();
        cluster_wait();
        cluster_arrive();
    } else if (warp == 1) {
        mma_role<BN, STAGES, Cfg::STAGE_BYTES, 0, false, false>(smem, full_bar, empty_bar, tfull_bar, nullptr, tmem_base, p, cta_first, cta_step, abort_flag);
        __syncwarp();
        cluster_wait();
        cluster_arrive();
    } else {
        const int ew = warp - 2, grp = ew >> 2, q = warp & 3;
        int m_t, n_t;
        tile_coords(p, tile, &m_t, &n_t);
        const int col0 = n_t * BN + 4 * lane;  // this lane's four columns (N is a multiple of 16)
        const bool in_cols = col0 < p.N;
        // where this warp's rows lie in the output (and in the pooled output), and their ReLU masks, while the main loop runs
        int row[ROWS], prow[ROWS];
        uint32_t mk[ROWS];
        {
            const int q1 = fdiv(m_t, p.fd_tw), tw = m_t - q1 * p.tiles_w, tn = fdiv(q1, p.fd_th), th = q1 - tn * p.tiles_h;
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                const int t = rank * RPC + ew * ROWS + i;  // row of the tile
                const int w = tw * p.BW + t % p.BW, h = th * p.BH + (t / p.BW) % p.BH, n = tn * p.BI + t / (p.BW * p.BH);
                const bool valid = t < p.BW * p.BH * p.BI && w < p.W && h < p.H && n < p.Nimg;
                row[i] = valid ? (n * p.H + h) * p.W + w : -1;
                prow[i] = (valid && ((w | h) & 1) == 0) ? (n * (p.H >> 1) + (h >> 1)) * (p.W >> 1) + (w >> 1) : -1;
                mk[i] = 0;
                if (p.mask != nullptr && valid && in_cols) mk[i] = __ldg(reinterpret_cast<const uint32_t*>(p.mask + static_cast<long long>(row[i]) * p.N + col0));
            }
        }
        // ---- the partial sums: tensor memory -> staging -> the rows' owners
        cluster_wait();  // every CTA of the cluster has set up its barriers
        bool up = mbar_wait(smem_u32(tfull_bar), 0, abort_flag);
        if (!up) report_abort(p.status, 4, 2);
        if (__all_sync(0xFFFFFFFFu, up)) {
            tc_fence_after();
            const int t = q * 32 + lane, lr = t % RPC;  // row of the tile, row of its owner
            uint32_t v[32];
            tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(grp * 32), v);
            tmem_ld_wait();
            const uint32_t base = smem_u32(smem) + static_cast<uint32_t>(t / RPC) * Cfg::SLOT_BYTES + static_cast<uint32_t>(grp * RPC + lr) * 128u;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                st_shared_v4(base + ((static_cast<uint32_t>(j) ^ (static_cast<uint32_t>(lr) & 7u)) << 4), v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            fence_proxy_async();
            __syncwarp();
            // this warp's rows belong to two owners (16 rows each) or to one
            constexpr int PIECE = RPC < 32 ? RPC : 32, OWNERS = 32 / PIECE;
            if (lane < OWNERS) {
                const int t0 = q * 32 + lane * PIECE, owner = t0 / RPC;
                if (owner != rank) {
                    const uint32_t slot = static_cast<uint32_t>(rank - owner - 1) & static_cast<uint32_t>(CS - 1);
                    const uint32_t at = static_cast<uint32_t>(grp * RPC + t0 % RPC) * 128u;
                    bulk_copy_cluster(mapa_u32(smem_u32(recv) + slot * Cfg::SLOT_BYTES + at, owner), smem_u32(smem) + owner * Cfg::SLOT_BYTES + at,
                                      PIECE * 128, mapa_u32(smem_u32(recv_bar), owner));
                }
            }
            __syncwarp();
        }
        named_barrier(EPI_BARRIER, 32 * EPI_WARPS);  // this CTA's own rows lie in the staging area
        up = mbar_wait(smem_u32(recv_bar), 0, abort_flag);
        if (!up) report_abort(p.status, 4, 2);
        __syncwarp();
        cluster_arrive();  // nothing this warp waits for is still on its way
        // ---- this CTA's rows: the sum of CS partial sums, and their maximum
        uint32_t acc[ROWS][4];
        unsigned local_max = 0;
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const int lr = ew * ROWS + i;
            const uint32_t at = static_cast<uint32_t>((lane >> 3) * RPC + lr) * 128u + (static_cast<uint32_t>((lane ^ lr) & 7) << 4);
            int4 s = *reinterpret_cast<const int4*>(smem + rank * Cfg::SLOT_BYTES + at);
#pragma unroll
            for (int k = 0; k < CS - 1; ++k) {
                const int4 o = *reinterpret_cast<const int4*>(recv + k * Cfg::SLOT_BYTES + at);
                s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
            }
            acc[i][0] = static_cast<uint32_t>(s.x); acc[i][1] = static_cast<uint32_t>(s.y); acc[i][2] = static_cast<uint32_t>(s.z); acc[i][3] = static_cast<uint32_t>(s.w);
            if (row[i] >= 0 && in_cols)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    local_max = max(local_max, min(acc[i][j], 0u - acc[i][j]));  // |x|
        }
        local_max = __reduce_max_sync(0xFFFFFFFFu, local_max);
        if (lane == 0) warp_max[ew] = local_max;
        int ticket = -1;
        const int shift = parked_grid_shift(p, warp_max, shift_slot, abort_flag, &ticket);
        // ---- narrow, store, pool
        if (shift >= 0) {
            const unsigned long long seed = (p.mode == ROUND_STOCHASTIC && shift > 0) ? *p.seed : 0ull;
            const bool pooling = p.pool_out != nullptr;  // the same for the whole grid
            const unsigned long long e0 = p.rng_offset + static_cast<unsigned long long>(col0);
            uint32_t y[ROWS];
            if (p.mode == ROUND_NEAREST && shift > 0) {
#pragma unroll
                for (int i = 0; i < ROWS; ++i) y[i] = narrow4_nearest<false>(acc[i], shift, 1 << (shift - 1));
            } else if (p.mode == ROUND_STOCHASTIC && shift > 0 && shift < 24 && (e0 & 3ull) == 0) {
#pragma unroll
                for (int i = 0; i < ROWS; ++i) {
                    uint32_t rnd[4];
                    random_block(seed, p.rng_stream, (e0 + static_cast<unsigned long long>(static_cast<long long>(row[i]) * p.N)) >> 2, rnd);
                    y[i] = narrow4_stochastic<false>(acc[i], shift, (1u << shift) - 1u, rnd);
                }
            } else {
#pragma unroll
                for (int i = 0; i < ROWS; ++i)
                    y[i] = narrow4_general(acc[i][0], acc[i][1], acc[i][2], acc[i][3], shift, p.mode, seed, p.rng_stream,
                                           e0 + static_cast<unsigned long long>(static_cast<long long>(row[i]) * p.N));
            }
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                if (p.relu) y[i] = __vmaxs4(y[i], 0u);
                if (p.mask != nullptr) y[i] &= __vcmpgts4(mk[i], 0);
                if (row[i] >= 0 && in_cols) *reinterpret_cast<uint32_t*>(p.out8 + static_cast<long long>(row[i]) * p.N + col0) = y[i];
                if (pooling) pool_rows[(ew * ROWS + i) * 32 + lane] = y[i];
            }
            if (pooling) {
                // the 2x2 window of local row r is rows r, r + 1, r + BW, r + BW + 1: all in this CTA (split_cluster)
                named_barrier(EPI_BARRIER, 32 * EPI_WARPS);
#pragma unroll
                for (int i = 0; i < ROWS; ++i)
                    if (prow[i] >= 0 && in_cols) {
                        const uint32_t* at = pool_rows + (ew * ROWS + i) * 32 + lane;
                        const uint32_t m = __vmaxs4(__vmaxs4(at[0], at[32]), __vmaxs4(at[p.BW * 32], at[(p.BW + 1) * 32]));
                        *reinterpret_cast<uint32_t*>(p.pool_out + static_cast<long long>(prow[i]) * p.N + col0) = m;
                    }
            }
        }
        parked_leave(p, shift, ticket);
    }

    // ---------------------------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) __nanosleep(200000);  // a block that gave up: let copies in flight, its own and its peers', land
    cluster_wait();  // no CTA leaves while a peer may still send to it
    if (warp == 1) {
        tc_fence_after();
        __syncwarp();
        tmem_dealloc(tmem_base, BN);
    }
}

#ifdef NITI_PARKED_TIMING
}  // namespace niti
extern "C" __attribute__((visibility("default"))) int niti_debug_stamps(unsigned long long* out) {
    return cudaMemcpyFromSymbol(out, niti::g_dbg_stamps, sizeof(niti::g_dbg_stamps)) == cudaSuccess ? 0 : -3;
}
namespace niti {
#endif

// ------------------------------------------------------------------------------------------------
// Convolution weight gradient: g[k][r][s][c] = sum_pixels err[pixel][k] * x[pixel + (r,s) - pad][c]
// A = err tile (MN-major: 128 k-channels x <=128 pixels), B = shifted x tile (MN-major:
// 128 c-channels x the same pixels).  One CTA owns (128 k) x (128 c) x (one filter row r, all S
// taps) and a contiguous range of pixel chunks; its S accumulators live in TMEM side by side.
// Partial sums are written to scratch[split] and folded by wgrad_reduce_kernel.
//
// KMAJ: the same contraction of operands that hold the batch innermost, [channels][H][W][N] (the arrangement in which the
// reference writes a weight gradient as a convolution with image-sized filters): both operands are then K-major as they
// lie, a chunk is one pixel x 128 images, and nothing has to be transposed.  Turning the two 8.4 MB tensors of a
// 128 x 16 x 16 x 256 layer round first cost 72 us, more than three times the contraction itself.
// ------------------------------------------------------------------------------------------------
struct WgradParams {
    int H, W, C, K, R, S, pad, Nimg;
    int BW, BH, BI;
    int tiles_w, tiles_h, tiles_n;
    int chunks, splits;
    int k_tiles, c_tiles;
    int box_bytes;         // bytes of one TMA box (BW*BH*BI rows of 128 bytes)
    int mma_per_chunk;     // ceil(rows / 32)
    int32_t* partial;      // [splits][K*R*S*C]
    int32_t* status;
    int reduce_direct;     // 1: every CTA adds its tiles straight into the (zeroed) gradient with TMA reductions
    int flip;              // KMAJ: 1 = the column operand is read at pixel - (tap - pad) instead of pixel + (tap - pad)
};

constexpr int WG_MAX_S = 3;
constexpr int WG_STAGE_BYTES = (1 + WG_MAX_S) * PANEL_BYTES;  // 64 KB
constexpr int WG_STAGES = 3;
constexpr int WG_SMEM_BYTES = WG_STAGES * WG_STAGE_BYTES + 1024 + 256;
constexpr int WG_TMEM_COLS = 512;

// What surrounds the contraction in umma_wgrad_update_kernel.
struct WgradUpdate {
    int32_t* g32;
    int8_t* w;             // null: the update is a launch of its own, which counts in `words`
    unsigned* maxabs;
    uint32_t* words; int num_words;  // cleared
    long long n;           // gradient elements, a multiple of 4
    int mu, mode;
    const unsigned long long* seed;
    unsigned rng_stream;
    int32_t* state;        // {zeroed, barrier arrivals, max |g|, exit ticket}: zero between calls
};

// One CTA's share of one layer's weight gradient: work item `item` (filter row, k tile, c tile) over the pixel chunks of
// split `split`.  The tensor maps live in kernel parameter space (grid constants of the calling kernel).
template <bool KMAJ, bool UPDATE = false>
__device__ __forceinline__ void wgrad_body(const CUtensorMap& tmErr, const CUtensorMap& tmX, const CUtensorMap& tmP,
                                           const WgradParams& p, const int split, const int item, const bool probe_cta,
                                           const WgradUpdate* u = nullptr) {
    if (threadIdx.x == 0 && probe_cta) PARK_STAMP(10);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + WG_STAGES * WG_STAGE_BYTES);
    uint64_t* full_bar = bars;
    uint64_t* empty_bar = bars + WG_STAGES;
    uint64_t* tfull_bar = bars + 2 * WG_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * WG_STAGES + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    // Rows past the box (when a tile holds fewer than 128 pixels) are read by the MMA as part of
    // the reduction: they must be zero.  TMA only ever writes the first box_bytes of a panel.
    if ((p.box_bytes / ROW_BYTES) % 32 != 0) {  // full 32-row slabs leave nothing unwritten for the MMAs to read
        int4* z = reinterpret_cast<int4*>(smem);
        for (int i = threadIdx.x; i < WG_STAGES * WG_STAGE_BYTES / 16; i += UMMA_THREADS) z[i] = make_int4(0, 0, 0, 0);
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < WG_STAGES; ++i) { mbar_init(smem_u32(&full_bar[i]), 1); mbar_init(smem_u32(&empty_bar[i]), 1); }
        mbar_init(smem_u32(&tfull_bar[0]), 1);
        *abort_flag = 0;
        fence_barrier_init();
        tma_prefetch_desc(&tmErr);
        tma_prefetch_desc(&tmX);
        tma_prefetch_desc(&tmP);
    }
    if (warp == 1) { tmem_alloc(smem_u32(tmem_slot), WG_TMEM_COLS); tmem_relinquish(); }
    fence_proxy_async();  // zero fill (generic proxy) before TMA writes (async proxy)
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (threadIdx.x == 0 && probe_cta) PARK_STAMP(11);

    const int r = item % p.R;
    const int kt = (item / p.R) % p.k_tiles;
    const int ct = item / (p.R * p.k_tiles);
    const int chunk_lo = static_cast<int>(static_cast<long long>(split) * p.chunks / p.splits);
    const int chunk_hi = static_cast<int>(static_cast<long long>(split + 1) * p.chunks / p.splits);

    // Warps 0 and 1 run their loops whole, with warp-uniform control flow (see producer_role); an elected lane issues.
    const uint32_t abort_addr = smem_u32(const_cast<int*>(abort_flag));
    const uint32_t smem0 = smem_u32(smem), full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);
    const int S = keep_reg(p.S);
    if (warp == 0) {
        {
            const int flip = KMAJ ? keep_reg(p.flip) : 0;
            const int pad = keep_reg(p.pad), BW = keep_reg(p.BW), BH = keep_reg(p.BH), BI = keep_reg(p.BI);
            const int tiles_w = keep_reg(p.tiles_w), tiles_h = keep_reg(p.tiles_h);
            const uint32_t tx_bytes = static_cast<uint32_t>(keep_reg((1 + p.S) * p.box_bytes));
            int s = 0; uint32_t ph = 0;
            // tile coordinates as running counters: this instruction stream paces the pipeline
            int tw = chunk_lo % p.tiles_w, th = (chunk_lo / p.tiles_w) % p.tiles_h, tn = chunk_lo / (p.tiles_w * p.tiles_h);
            for (int ch = chunk_lo; ch < chunk_hi; ++ch) {
                if (!mbar_wait_uniform(empty0 + 8u * s, ph ^ 1u, abort_addr)) { *abort_flag = 1; report_abort(p.status, 11, 0); break; }
                const uint32_t fb = full0 + 8u * s;
                const uint32_t sa = smem0 + static_cast<uint32_t>(s) * WG_STAGE_BYTES;
                if (elect_one()) {
                    mbar_arrive_expect_tx(fb, tx_bytes);
                    if (KMAJ) {
                        tma_load_4d(sa, &tmErr, fb, tn * 128, tw, th, kt * 128);
                        const int y = flip ? th + pad - r : th + r - pad;
                        for (int sx = 0; sx < S; ++sx)
                            tma_load_4d(sa + (1 + sx) * PANEL_BYTES, &tmX, fb, tn * 128, flip ? tw + pad - sx : tw + sx - pad, y, ct * 128);
                    } else {
                        tma_load_4d(sa, &tmErr, fb, kt * 128, tw * BW, th * BH, tn * BI);
                        for (int sx = 0; sx < S; ++sx)
                            tma_load_4d(sa + (1 + sx) * PANEL_BYTES, &tmX, fb, ct * 128, tw * BW + sx - pad, th * BH + r - pad, tn * BI);
                    }
                }
                if (++s == WG_STAGES) { s = 0; ph ^= 1u; }
                if (++tw == tiles_w) { tw = 0; if (++th == tiles_h) { th = 0; ++tn; } }
            }
        }
        __syncwarp();  // reach the teardown's block-wide barrier as a converged warp
    } else if (warp == 1) {
        {
            constexpr int MN = KMAJ ? 0 : 1;
            const uint32_t idesc = make_idesc_i8(BLOCK_M, 128, MN, MN);
            const uint32_t idesc2 = make_idesc_i8(BLOCK_M, 256, MN, MN);
            const uint32_t tm = __shfl_sync(0xFFFFFFFFu, tmem_base, 0);
            const int nmma = keep_reg(p.mma_per_chunk);
            // 32 reduction rows (KMAJ: 32 bytes) per MMA, in descriptor units.  Adjacent panels are one operand of 256
            // columns in either major: 128-column panels one leading offset apart, or simply 256 rows.
            const uint64_t kstep = (KMAJ ? 32u : 32u * ROW_BYTES) >> 4;
            const uint64_t d0 = make_smem_desc(smem0, KMAJ ? 16 : PANEL_BYTES, 1024, SWIZZLE_128B_CODE);
            int s = 0; uint32_t ph = 0; bool ok = true;
            bool ready = false;  // the stage's "full" phase was seen complete by the previous chunk's probe
            for (int ch = chunk_lo; ch < chunk_hi; ++ch) {
                if (!ready && !mbar_wait_uniform(full0 + 8u * s, ph, abort_addr)) { ok = false; *abort_flag = 1; report_abort(p.status, 13, 1); break; }
                if (ch == chunk_lo && probe_cta) PARK_STAMP(12);
                const uint64_t a0 = d0 + ((static_cast<uint32_t>(s) * WG_STAGE_BYTES) >> 4);
                const uint32_t first = static_cast<uint32_t>(ch != chunk_lo);
                const int sn = (s + 1 == WG_STAGES) ? 0 : s + 1;
                const uint32_t phn = (sn == 0) ? ph ^ 1u : ph;
                const uint32_t eb = empty0 + 8u * s;
                // The taps' x tiles lie one panel apart, which is exactly the layout of an MN-major B operand of
                // two 128-column panels: two taps go through ONE 256-column MMA (half as many instructions to issue),
                // accumulating into the adjacent TMEM column blocks of the two taps.
                uint32_t probe;
                if (nmma == 4 && S == 3) {
                    umma_seq4(tm, a0, a0 + (PANEL_BYTES >> 4), kstep, kstep, idesc2, first);
                    probe = umma_block4<false>(tm + 256, a0, a0 + ((3 * PANEL_BYTES) >> 4), kstep, kstep, idesc, first, eb, full0 + 8u * sn, phn);
                } else {
                    if (elect_one()) {
                        int sx = 0;
                        for (; sx + 1 < S; sx += 2)
                            for (int k = 0; k < nmma; ++k)
                                umma_i8(tm + sx * 128, a0 + k * kstep, a0 + (((1 + sx) * PANEL_BYTES) >> 4) + k * kstep, idesc2,
                                        static_cast<uint32_t>(ch != chunk_lo || k != 0));
                        for (; sx < S; ++sx)
                            for (int k = 0; k < nmma; ++k)
                                umma_i8(tm + sx * 128, a0 + k * kstep, a0 + (((1 + sx) * PANEL_BYTES) >> 4) + k * kstep, idesc,
                                        static_cast<uint32_t>(ch != chunk_lo || k != 0));
                        umma_commit(eb);
                    }
                    probe = mbar_test_wait(full0 + 8u * sn, phn);
                }
                ready = __all_sync(0xFFFFFFFFu, probe != 0);
                s = sn; ph = phn;
            }
            if (ok && elect_one()) umma_commit(smem_u32(&tfull_bar[0]));
            if (probe_cta) PARK_STAMP(13);
        }
        __syncwarp();
    } else {
        // partial[split][k][r][s][c] viewed as a rank-4 tensor (c, r*S+s, k, split): per tap, four TMA
        // stores of 128 k-rows x 32 channels.  Once the last MMA has completed the operand stages
        // are dead, so stage `sx` serves as the staging area of tap `sx` (64 KB = 4 tiles each) and
        // no store ever waits for another.
        const int q = warp & 3;
        const int row_in_tile = q * 32 + lane;
        const bool leader = threadIdx.x == 64;
        const int ctas = static_cast<int>(gridDim.x * gridDim.y);
        if (UPDATE && p.splits > 1) {
            // the gradient is cleared here, under the contraction; nobody adds to it before every CTA has cleared its part
            int4* g = reinterpret_cast<int4*>(u->g32);
            const long long groups = u->n >> 2;
            for (long long i = static_cast<long long>(blockIdx.y * gridDim.x + blockIdx.x) * 128 + row_in_tile; i < groups; i += 128ll * ctas)
                g[i] = make_int4(0, 0, 0, 0);
            fence_proxy_async_global();
            __threadfence();
            named_barrier(EPI_BARRIER, 128);
            if (leader) red_release_add(&u->state[0], 1);
        }
        const uint32_t failed = mbar_wait(smem_u32(&tfull_bar[0]), 0, abort_flag) ? 0u : 1u;
        if (barrier_or(EPI_BARRIER, 128, failed)) {
            if (failed) report_abort(p.status, 14, 2);
        } else {
            tc_fence_after();
            if (leader && probe_cta) PARK_STAMP(14);
            bool cleared = true;
            if (UPDATE && p.splits > 1 && leader) {
                const unsigned long long t0 = global_timer_ns();
                for (unsigned spin = 0; ld_acquire_gpu(&u->state[0]) < ctas; ++spin)
                    if ((spin & 63) == 63 && global_timer_ns() - t0 > GRID_BARRIER_LIMIT_NS) { cleared = false; break; }
                if (!cleared) { *abort_flag = 1; report_abort(p.status, 15, 2); }
                fence_proxy_async_global();
            }
            for (int sx = 0; sx < p.S; ++sx) {
                const uint32_t buf = smem_u32(smem + sx * WG_STAGE_BYTES);
                uint32_t v[4][32];
#pragma unroll
                for (int j = 0; j < 4; ++j) tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + sx * 128 + j * 32, v[j]);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 4; ++j) stage_row(buf + j * EPI_CHUNK_BYTES, row_in_tile, v[j]);
                fence_proxy_async();
                named_barrier(EPI_BARRIER, 128);
                if (leader && cleared) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (ct * 128 + j * 32 < p.C) {
                            if (p.reduce_direct) tma_reduce_add_4d(&tmP, buf + j * EPI_CHUNK_BYTES, ct * 128 + j * 32, r * p.S + sx, kt * 128, 0);
                            else tma_store_4d(&tmP, buf + j * EPI_CHUNK_BYTES, ct * 128 + j * 32, r * p.S + sx, kt * 128, split);
                        }
                    bulk_commit();
                }
            }
            if (leader && probe_cta) PARK_STAMP(15);
            if (leader) { if (UPDATE) bulk_wait<0>(); else bulk_wait_read<0>(); }  // UPDATE: the sums are in memory
            if (UPDATE && leader) fence_proxy_async_global();
            if (leader && probe_cta) PARK_STAMP(16);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        if (*abort_flag) __nanosleep(200000);
        tc_fence_after();
        __syncwarp();
        tmem_dealloc(tmem_base, WG_TMEM_COLS);
    }
}

__global__ void __launch_bounds__(UMMA_THREADS, 1)
umma_wgrad_kernel(const __grid_constant__ CUtensorMap tmErr, const __grid_constant__ CUtensorMap tmX,
                  const __grid_constant__ CUtensorMap tmP, const __grid_constant__ WgradParams p) {
    wgrad_body<false>(tmErr, tmX, tmP, p, blockIdx.x, blockIdx.y, blockIdx.y == 0);
}
// The same with the gradient cleared under the contraction, and for small layers followed by the update (UpdateWeight.weight_update)
// in the same launch: a grid barrier when every CTA's sums are in memory, max |g|, a second one, the update.  A single layer's
// backward is launches: 48 -> 80 on 37 15x13 maps took 14.5 us with a memset, the contraction and the update in a row (and a gap of 1
// to 2 us behind each) and takes 11 as one.  Cooperative; one wave of CTAs, whose six warps are too few for the update of a large
// layer (589 thousand weights: even; 2.4 million: 44 us against 27).
constexpr long long WG_UPDATE_MAX = 200000;
__global__ void __launch_bounds__(UMMA_THREADS, 1)
umma_wgrad_update_kernel(const __grid_constant__ CUtensorMap tmErr, const __grid_constant__ CUtensorMap tmX,
                         const __grid_constant__ CUtensorMap tmP, const __grid_constant__ WgradParams p, const __grid_constant__ WgradUpdate u) {
    __shared__ int flag;
    __shared__ unsigned part[UMMA_THREADS / 32];
    if (blockIdx.x + blockIdx.y == 0)
        for (int i = threadIdx.x; i < u.num_words; i += UMMA_THREADS) u.words[i] = 0;
    wgrad_body<false, true>(tmErr, tmX, tmP, p, blockIdx.x, blockIdx.y, blockIdx.y == 0, &u);
    const int ctas = static_cast<int>(gridDim.x * gridDim.y);
    if (u.w == nullptr) {
        if (p.splits > 1 && threadIdx.x == 0 && atomicAdd(&u.state[3], 1) == ctas - 1) { u.state[0] = 0; u.state[3] = 0; }
        return;
    }
    const long long groups = u.n >> 2, step = static_cast<long long>(ctas) * UMMA_THREADS;
    const long long tid = static_cast<long long>(blockIdx.y * gridDim.x + blockIdx.x) * UMMA_THREADS + threadIdx.x;
    const int4* g4 = reinterpret_cast<const int4*>(u.g32);
    uint32_t* w4 = reinterpret_cast<uint32_t*>(u.w);
    // gradients and weights of a thread's first word groups stay in registers from the maximum to the update
    constexpr int KEEP = 2;
    int4 gv[KEEP];
    uint32_t wv[KEEP];
#pragma unroll
    for (int k = 0; k < KEEP; ++k)
        if (tid + k * step < groups) wv[k] = w4[tid + k * step];  // does not depend on the sums
    bool ok = bounded_grid_barrier(&u.state[1], ctas, p.status, 7, &flag);
    if (ok) {
        unsigned m = 0;
#pragma unroll
        for (int k = 0; k < KEEP; ++k)
            if (tid + k * step < groups) gv[k] = __ldcg(g4 + tid + k * step);
#pragma unroll
        for (int k = 0; k < KEEP; ++k)
            if (tid + k * step < groups) m = max(m, absmax4(gv[k]));
        for (long long g = tid + KEEP * step; g < groups; g += step) m = max(m, absmax4(__ldcg(g4 + g)));
        m = __reduce_max_sync(0xFFFFFFFFu, m);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
        __syncthreads();
        if (threadIdx.x == 0) {
#pragma unroll
            for (int i = 0; i < UMMA_THREADS / 32; ++i) m = max(m, part[i]);
            if (m != 0) red_relaxed_max(reinterpret_cast<unsigned*>(&u.state[2]), m);
        }
        ok = bounded_grid_barrier(&u.state[1], 2 * ctas, p.status, 7, &flag);
    }
    const unsigned mx = static_cast<unsigned>(ld_acquire_gpu(&u.state[2]));
    int ticket = -1;
    if (ok) {
        bool zero_out;
        const int shift = shift_for(mx, CALC_GRAD, u.mu, &zero_out);
        const bool stochastic = u.mode == ROUND_STOCHASTIC && shift > 0;
        const unsigned long long seed = stochastic ? *u.seed : 0ull;
        const auto one = [&](long long g, const int4 gvv, const uint32_t wvv) {
            uint32_t rnd[4] = {0, 0, 0, 0};
            if (stochastic) random_block(seed, u.rng_stream, static_cast<unsigned long long>(g), rnd);
            w4[g] = update_word(gvv, wvv, rnd, shift, u.mode, zero_out);
        };
#pragma unroll
        for (int k = 0; k < KEEP; ++k)
            if (tid + k * step < groups) one(tid + k * step, gv[k], wv[k]);
        for (long long g = tid + KEEP * step; g < groups; g += step) one(g, __ldcg(g4 + g), w4[g]);
    }
    __syncthreads();  // every thread has read the maximum
    if (threadIdx.x == 0) {
        ticket = atomicAdd(&u.state[3], 1);
        if (ticket == ctas - 1) {
            *u.maxabs = mx;
            u.state[0] = 0; u.state[1] = 0; u.state[2] = 0; u.state[3] = 0;
        }
    }
}
__global__ void __launch_bounds__(UMMA_THREADS, 1)
umma_wgrad_kmajor_kernel(const __grid_constant__ CUtensorMap tmErr, const __grid_constant__ CUtensorMap tmX,
                         const __grid_constant__ CUtensorMap tmP, const __grid_constant__ WgradParams p) {
    wgrad_body<true>(tmErr, tmX, tmP, p, blockIdx.x, blockIdx.y, blockIdx.y == 0);
}

// Several layers' weight gradients in ONE launch: CTAs [first_cta[l], first_cta[l + 1]) belong to layer l, split-major
// inside.  The host picks the splits so that every CTA of the launch walks about the same number of pixel chunks: a
// step's layers come in pairs of equal work (256->512 and 512->512 at 8x8, ...), which then fill one wave exactly and
// pay the launch, the prologue and the accumulator flush once instead of twice.
constexpr int WG_MULTI_MAX = 4;
struct WgradMultiMaps { CUtensorMap err[WG_MULTI_MAX], x[WG_MULTI_MAX], g[WG_MULTI_MAX]; };
struct WgradMultiParams { WgradParams layer[WG_MULTI_MAX]; int first_cta[WG_MULTI_MAX + 1]; int count; };
__global__ void __launch_bounds__(UMMA_THREADS, 1)
umma_wgrad_multi_kernel(const __grid_constant__ WgradMultiMaps maps, const __grid_constant__ WgradMultiParams mp) {
    int l = 0;
    while (l + 1 < mp.count && static_cast<int>(blockIdx.x) >= mp.first_cta[l + 1]) ++l;
    const int local = static_cast<int>(blockIdx.x) - mp.first_cta[l];
    const WgradParams& p = mp.layer[l];
    wgrad_body<false>(maps.err[l], maps.x[l], maps.g[l], p, local % p.splits, local / p.splits, blockIdx.x == 0);
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static void* driver_entry(const char* name) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    return cudaGetDriverEntryPoint(name, &sym, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess ? sym : nullptr;
}
static EncodeTiledFn get_encode() {
    static const EncodeTiledFn fn = reinterpret_cast<EncodeTiledFn>(driver_entry("cuTensorMapEncodeTiled"));
    return fn;
}
// A number for the current context that no other one has had or will have; 0: not known.
static unsigned long long context_number() {
    static const auto get_id = reinterpret_cast<CUresult (*)(CUcontext, unsigned long long*)>(driver_entry("cuCtxGetId"));
    unsigned long long id = 0;
    return get_id != nullptr && get_id(nullptr, &id) == CUDA_SUCCESS ? id + 1 : 0;
}

// Tensor map with 128-byte swizzle over uint8 (operands) or int32 (outputs) elements; dims/box
// innermost first, in elements; strides of dims 1.. in bytes.
static int encode_map(CUtensorMap* map, const void* ptr, bool int32_elems, int rank, const uint64_t* dims,
                      const uint64_t* strides, const uint32_t* box, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B,
                      CUtensorMapL2promotion promotion = CU_TENSOR_MAP_L2_PROMOTION_L2_256B) {
    EncodeTiledFn enc = get_encode();
    if (!enc) return set_cuda_error_text("cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t gdim[4]; cuuint64_t gstr[3]; cuuint32_t bx[4]; cuuint32_t es[4];
    for (int i = 0; i < rank; ++i) { gdim[i] = dims[i]; bx[i] = box[i]; es[i] = 1; }
    for (int i = 0; i + 1 < rank; ++i) gstr[i] = strides[i];
    CUresult r = enc(map, int32_elems ? CU_TENSOR_MAP_DATA_TYPE_INT32 : CU_TENSOR_MAP_DATA_TYPE_UINT8, rank,
                     const_cast<void*>(ptr), gdim, gstr, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     swizzle, promotion, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        char buf[160];
        snprintf(buf, sizeof buf, "cuTensorMapEncodeTiled failed with CUresult %d (rank %d)", static_cast<int>(r), rank);
        return set_cuda_error_text(buf);
    }
    return 0;
}

// The dynamic shared memory of a kernel, granted once per context: asked for at every launch it was about a microsecond of the host's
// time, and a single image's layers are bound by that.  Not once per device: a second context of a device, or its first one after a
// reset, starts without the grant, and a launch there would be refused.
template <auto KERNEL>
static cudaError_t allow_shared(int bytes) {
    static std::atomic<unsigned long long> granted[16];  // context numbers; two that share a place ask in turn
    const unsigned long long now = context_number();
    std::atomic<unsigned long long>& place = granted[now % 16];
    if (now != 0 && place.load(std::memory_order_acquire) == now) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess && now != 0) place.store(now, std::memory_order_release);
    return e;
}

// The result of a launch whose thread blocks have to be resident together: see LAUNCH_REFUSED.
static int launched_together(cudaError_t e) {
    if (e != cudaErrorCooperativeLaunchTooLarge && e != cudaErrorInvalidClusterSize && e != cudaErrorLaunchOutOfResources) return launched(e);
    cudaGetLastError();
    return LAUNCH_REFUSED;
}

static int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
    }
    return n;
}

// CTA pairs (TWO): clusters of two CTAs, p.m_tiles counts 256-row tiles
template <int BN, bool TWO, bool ROWS32 = false>
static int launch_gemm_inst(const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& c, const GemmParams& p, cudaStream_t st) {
    using Cfg = GemmCfg<BN, TWO>;
    cudaError_t e = allow_shared<umma_gemm_kernel<BN, TWO, ROWS32>>(Cfg::SMEM_BYTES);
    if (e != cudaSuccess) return set_cuda_error(e);
    int tiles = p.m_tiles * p.n_tiles * p.splits;
    if (tiles > sm_count() / (TWO ? 2 : 1)) tiles = sm_count() / (TWO ? 2 : 1);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(TWO ? 2 * tiles : tiles); cfg.blockDim = dim3(GEMM_THREADS); cfg.dynamicSmemBytes = Cfg::SMEM_BYTES; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = TWO ? 1 : 0;
    return launched(cudaLaunchKernelEx(&cfg, umma_gemm_kernel<BN, TWO, ROWS32>, a, b, c, p));
}
static int launch_gemm(int bn, bool pair, const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& c, const GemmParams& p,
                       cudaStream_t st) {
    if (pair) return bn == 256 ? launch_gemm_inst<256, true>(a, b, c, p, st) : launch_gemm_inst<128, true>(a, b, c, p, st);
    if (p.rows32) return bn == 256 ? launch_gemm_inst<256, false, true>(a, b, c, p, st) : launch_gemm_inst<128, false, true>(a, b, c, p, st);
    return bn == 256 ? launch_gemm_inst<256, false>(a, b, c, p, st) : launch_gemm_inst<128, false>(a, b, c, p, st);
}
// CTA pairs (M = 256 MMAs, B operand split between the two CTAs): bit 0 enables them for GEMMs, bit 1 for
// convolutions.  Measured on B200: +20 % on large GEMMs (2.2 -> 2.7 POP/s at 8192^3), nothing on the
// convolutions (their A tiles are re-read per filter tap and dominate), hence the default.
int g_two_cta = 1;
// a pair needs two 128-row tiles to share a B tile; an MN-major B splits only at 128-column panels
static bool pair_ok(int m_tiles, int bn, int b_mn, int conv) {
    return (g_two_cta & (conv ? 2 : 1)) && m_tiles >= 2 && (!b_mn || bn == 256);
}
// Kernels with a grid barrier are cooperative launches: every CTA must be resident at the same time
template <int BN, bool TWO, int MODE, bool PARKED, bool ONE = false, bool CODES = false>
static int launch_requant_inst(const CUtensorMap& a, const CUtensorMap& b, const GemmParams& p, cudaStream_t st) {
    using Cfg = RequantCfg<BN, TWO, MODE>;
    void (*kernel)(CUtensorMap, CUtensorMap, GemmParams);
    cudaError_t e;
    if constexpr (PARKED) { kernel = umma_parked_kernel<BN, TWO, MODE>; e = allow_shared<umma_parked_kernel<BN, TWO, MODE>>(Cfg::SMEM_BYTES); }
    else if constexpr (ONE) { kernel = umma_requant_once_kernel<BN, MODE>; e = allow_shared<umma_requant_once_kernel<BN, MODE>>(Cfg::SMEM_BYTES); }
    else { kernel = umma_requant_kernel<BN, TWO, MODE, CODES>; e = allow_shared<umma_requant_kernel<BN, TWO, MODE, CODES>>(Cfg::SMEM_BYTES); }
    if (e != cudaSuccess) return set_cuda_error(e);
    int tiles = p.m_tiles * p.n_tiles;
    if (tiles > sm_count() / (TWO ? 2 : 1)) tiles = sm_count() / (TWO ? 2 : 1);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(TWO ? 2 * tiles : tiles); cfg.blockDim = dim3(REQUANT_THREADS); cfg.dynamicSmemBytes = Cfg::SMEM_BYTES; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (PARKED || ONE) { attr[n].id = cudaLaunchAttributeCooperative; attr[n].val.cooperative = g_cooperative; ++n; }
    if (TWO) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 2; attr[n].val.clusterDim.y = 1; attr[n].val.clusterDim.z = 1; ++n;
    }
    cfg.attrs = attr; cfg.numAttrs = n;
    const cudaError_t r = cudaLaunchKernelEx(&cfg, kernel, a, b, p);
    return ONE ? launched_together(r) : launched(r);
}
template <bool ONE, bool CODES>
static int launch_streaming(int bn, int mode, const CUtensorMap& a, const CUtensorMap& b, const GemmParams& p, cudaStream_t st) {
    if constexpr (!CODES)
        if (mode == LOAD_ROWS32)
            return bn == 64    ? launch_requant_inst<64, false, LOAD_ROWS32, false, ONE>(a, b, p, st)
                   : bn == 256 ? launch_requant_inst<256, false, LOAD_ROWS32, false, ONE>(a, b, p, st)
                               : launch_requant_inst<128, false, LOAD_ROWS32, false, ONE>(a, b, p, st);
    if (mode == LOAD_HALO_RESIDENT)
        return bn == 64 ? launch_requant_inst<64, false, LOAD_HALO_RESIDENT, false, ONE, CODES>(a, b, p, st) : launch_requant_inst<128, false, LOAD_HALO_RESIDENT, false, ONE, CODES>(a, b, p, st);
    if (mode == LOAD_HALO) return bn == 64 ? launch_requant_inst<64, false, LOAD_HALO, false, ONE, CODES>(a, b, p, st) : launch_requant_inst<128, false, LOAD_HALO, false, ONE, CODES>(a, b, p, st);
    if (bn == 64) return launch_requant_inst<64, false, LOAD_TAPS, false, ONE, CODES>(a, b, p, st);
    return bn == 256 ? launch_requant_inst<256, false, LOAD_TAPS, false, ONE, CODES>(a, b, p, st) : launch_requant_inst<128, false, LOAD_TAPS, false, ONE, CODES>(a, b, p, st);
}
static int launch_requant(int bn, bool pair, int mode, bool parked, bool one, const CUtensorMap& a, const CUtensorMap& b, const GemmParams& p,
                          cudaStream_t st) {
    if (parked) {
        if (pair) return bn == 256 ? launch_requant_inst<256, true, LOAD_TAPS, true>(a, b, p, st) : launch_requant_inst<128, true, LOAD_TAPS, true>(a, b, p, st);
        if (mode == LOAD_HALO_RESIDENT) return launch_requant_inst<128, false, LOAD_HALO_RESIDENT, true>(a, b, p, st);
        if (mode == LOAD_HALO) return launch_requant_inst<128, false, LOAD_HALO, true>(a, b, p, st);
        return bn == 256 ? launch_requant_inst<256, false, LOAD_TAPS, true>(a, b, p, st) : launch_requant_inst<128, false, LOAD_TAPS, true>(a, b, p, st);
    }
    if (one) return launch_streaming<true, false>(bn, mode, a, b, p, st);
    if (pair) return bn == 256 ? launch_requant_inst<256, true, LOAD_TAPS, false, false, true>(a, b, p, st) : launch_requant_inst<128, true, LOAD_TAPS, false, false, true>(a, b, p, st);
    if (mode == LOAD_ROWS32) return launch_streaming<false, false>(bn, mode, a, b, p, st);
    return bn == 64 || (p.side != nullptr && p.mode == NITI_ROUND_NEAREST && !p.relu) ? launch_streaming<false, true>(bn, mode, a, b, p, st)
                                                                         : launch_streaming<false, false>(bn, mode, a, b, p, st);
}
template <int CS>
static cudaLaunchConfig_t split_config(int tiles, cudaLaunchAttribute* attr, cudaStream_t st) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative; attr[1].val.cooperative = g_cooperative;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(tiles * CS); cfg.blockDim = dim3(REQUANT_THREADS); cfg.dynamicSmemBytes = SplitCfg<CS>::SMEM_BYTES; cfg.stream = st;
    cfg.attrs = attr; cfg.numAttrs = 2;
    return cfg;
}
template <int CS>
static int launch_split(const CUtensorMap& a, const CUtensorMap& b, const GemmParams& p, cudaStream_t st) {
    cudaError_t e = allow_shared<umma_split_kernel<CS>>(SplitCfg<CS>::SMEM_BYTES);
    if (e != cudaSuccess) return set_cuda_error(e);
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = split_config<CS>(p.m_tiles * p.n_tiles, attr, st);
    return launched_together(cudaLaunchKernelEx(&cfg, umma_split_kernel<CS>, a, b, p));
}
// Clusters of CS CTAs (one CTA per SM) that the context holds at a time when idle; 0 where it cannot be asked (now: the next call
// asks again).  They lie within a GPC each, so that it is less than the number of SMs over CS.
template <int CS>
static int split_clusters() {
    static std::atomic<unsigned long long> known{0};  // the context's number, and the clusters in the low 16 bits
    const unsigned long long now = context_number(), was = known.load(std::memory_order_relaxed);
    if (now != 0 && was >> 16 == now) return static_cast<int>(was & 0xFFFF);
    int n = 0;
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = split_config<CS>(1, attr, nullptr);
    cfg.numAttrs = 1;
    if (allow_shared<umma_split_kernel<CS>>(SplitCfg<CS>::SMEM_BYTES) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, umma_split_kernel<CS>, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
    known.store(now << 16 | static_cast<unsigned>(n), std::memory_order_relaxed);
    return n;
}
// all accumulators of the problem fit in the tensor memory of one wave of CTAs (units: 128-row tiles,
// or 256-row pair tiles on sm/2 pairs)
static bool fits_parked(int bn, int tiles, bool pair) { return tiles <= (pair ? sm_count() / 2 : sm_count()) * (512 / bn); }

// Output tile width: 256 columns halve the A-operand traffic, but when that leaves fewer tiles than
// half the SMs, 128-column tiles put twice as many SMs to work.
static int pick_bn(int m_tiles, int n_cols) {
    if (n_cols <= 128) return 128;
    const int tiles256 = m_tiles * ((n_cols + 255) / 256);
    return tiles256 * 2 <= sm_count() ? 128 : 256;
}

// the streaming kernel that narrows also has 64-column tiles
static int requant_bn(int n_cols, int m_tiles) { return n_cols <= 64 ? 64 : pick_bn(m_tiles, n_cols); }

int g_stage_cap = 0;  // 0: use every compiled stage
// 1: kernels with a grid barrier are launched cooperatively (the driver guarantees that all their blocks are
// resident together).  0: plain launches of grids that fit the device in one wave; co-residency then rests on
// nothing else occupying the SMs, and a barrier that is not met ends in the bounded wait's error status.
int g_cooperative = 1;

static int mma_columns(int n, int bn, int n_tiles, bool pair) { return n_tiles == 1 && !pair ? (n + 15) / 16 * 16 : bn; }

static void finish_params(GemmParams* p) {
    p->fd_mn = make_fastdiv(p->m_tiles * p->n_tiles); p->fd_n = make_fastdiv(p->n_tiles);
    p->fd_tw = make_fastdiv(p->tiles_w); p->fd_th = make_fastdiv(p->tiles_h);
}

static void set_fused(GemmParams* p, const FusedArgs* f) {
    p->nstages = g_stage_cap;
    if (!f) return;
    p->state = f->state; p->only_if_redo = f->only_if_redo; p->mode = f->mode; p->relu = f->relu;
    p->seed = f->seed; p->rng_stream = f->rng_stream; p->rng_offset = f->rng_offset;
    p->kind = f->kind; p->target_bits = f->target_bits;
    p->exp_a = f->exp_a; p->exp_b = f->exp_b; p->exp_out = f->exp_out; p->shift_out = f->shift_out;
    p->mask = f->relu_mask;
    p->pool_out = nullptr;
    p->out8 = nullptr;
    p->side = static_cast<uint32_t*>(f->side);
    // max|acc| lives in state[1]; a redo launch must leave it alone (the last CTA of the first launch zeroed it)
    p->maxabs = f->only_if_redo ? nullptr : reinterpret_cast<unsigned*>(f->state + 1);
}

// Pixels of one 128-row tile: as much of a row as fits, then rows, then images.
static void pick_pixel_box(int Nimg, int H, int W, int* BW, int* BH, int* BI) {
    *BW = W < 128 ? W : 128;
    int bh = 128 / *BW; if (bh > H) bh = H; if (bh < 1) bh = 1;
    *BH = bh;
    int bi = 128 / (*BW * *BH); if (bi > Nimg) bi = Nimg; if (bi < 1) bi = 1;
    *BI = bi;
}

static bool pool_box_ok(int H, int W, int bw, int bh);

// Tiles of a convolution.  kernel: 0 = int32 out, 1 = streaming, 2 = parked.
struct ConvPlan { int BW, BH, BI, tiles_w, tiles_h, m_tiles, bn; bool pair, halo; };
// red: reduction channels per tap.  (`stochastic` turns down plans of more tiles only, so what fits in tensor memory does not
// depend on it.)
static ConvPlan conv_plan(int Nimg, int H, int W, int red, int outc, bool k3, int flip, int kernel, bool stochastic = false) {
    ConvPlan c{};
    pick_pixel_box(Nimg, H, W, &c.BW, &c.BH, &c.BI);
    c.tiles_w = (W + c.BW - 1) / c.BW; c.tiles_h = (H + c.BH - 1) / c.BH;
    c.m_tiles = c.tiles_w * c.tiles_h * ((Nimg + c.BI - 1) / c.BI);
    c.bn = kernel == 1 ? requant_bn(outc, c.m_tiles) : pick_bn(c.m_tiles, outc);
    c.pair = c.bn != 64 && pair_ok(c.m_tiles, c.bn, flip, 1);
    // 8-pixel-wide tiles of one image with the activations of three taps in one load (producer_halo_role): up to 128
    // columns, where the loads and not the MMAs set the pace (128 -> 128 at 32x32, batch 128: 28.0 -> 19.5 us; 64 -> 64,
    // batch 1024: 157 -> 119).
    // Maps that 8 x 16 pixels cover badly have more of these tiles; a tile takes about two thirds of the time, so up to half as
    // many more rounds of thread blocks are a gain (190 random layers, both ways timed; us, box per tap / shared rows, batch x map,
    // channels, rounds: 501x8x25 16->64, 7 / 14: 67 / 29; 437x28x10 32->96, 9 / 12: 42 / 24; 192x25x12 112->128, 4 / 6: 28.4 / 28.5;
    // 280x10x11 224->112, 2 / 4: 17.2 / 19.7; 154x10x5 48->128, 1 / 2: 10.6 / 11.9); where random words are drawn, for every row of
    // a tile, only up to a quarter unless the channels are few (300x20x20, 9 / 13: 96->96 37 / 42, 48->48 49 / 32).  Within one round they always are, but for
    // layers of 16 and 32 channels, whose time is the loading of the weights by every one of the thread blocks (60x28x4 16->128,
    // 60 / 120 blocks: 11.0 / 12.6; 36x8x26 80->128, 72 / 144: 10.9 / 10.2; 18x24x10 336->16, 36 / 72: 12.9 / 10.2).
    if (k3 && kernel != 0 && !c.pair && c.bn <= 128) {
        const int th = (H + 15) / 16, bh = (H + th - 1) / th, tw = (W + 7) / 8;
        const long long tiles = static_cast<long long>(tw) * th * Nimg;
        const long long n_tiles = (outc + c.bn - 1) / c.bn, sms = sm_count();
        const long long before = (c.m_tiles * n_tiles + sms - 1) / sms, after = (tiles * n_tiles + sms - 1) / sms;
        const bool gain = after == 1 ? red >= 48 || tiles * n_tiles <= 64 || 4 * tiles <= 5ll * c.m_tiles
                                     : (stochastic && red > 64 ? 4 * after <= 5 * before : 2 * after <= 3 * before) || (red == 16 && before > 1 && after <= 2 * before);
        if (gain && (kernel != 2 || fits_parked(c.bn, static_cast<int>(tiles) * ((outc + c.bn - 1) / c.bn), false))) {
            c.halo = true;
            c.BW = 8; c.BH = bh; c.BI = 1; c.tiles_w = tw; c.tiles_h = th; c.m_tiles = static_cast<int>(tiles);
        }
    }
    return c;
}

// The tiles of a call that pools too: with the shared activation rows unless that makes tiles of an odd number of rows
// (18, 22, 26, 30, 38 image rows), which would tear pooling windows apart; those keep the box per tap.
static ConvPlan pool_plan(int Nimg, int H, int W, int red, int outc, bool k3) {
    const ConvPlan c = conv_plan(Nimg, H, W, red, outc, k3, 0, 2);
    return pool_box_ok(H, W, c.BW, c.BH) ? c : conv_plan(Nimg, H, W, red, outc, false, 0, 2);
}

// CTAs that share the reduction of one output tile (umma_split_kernel); 1: none do.  bw: 0, or the width of the tile's pixel
// box in a call that pools (a CTA's rows are then whole pairs of image rows).
// Where the line lies: sharing costs about 1.6 us (exchange, cluster) and saves the (1 - 1 / cs) of the main loop that the
// others take over, 0.21 us per 128-byte reduction block with a box per tap and 0.14 where the rows of three taps come in one
// (us, before / after, batch x map, channels):
//   box per tap   32x4x4 512->512 15.3 / 10.6, 12x8x8 256->256 11.8 / 10.1, 32x8x8 256->512 11.7 / 11.0; 64x8x8 128->128 9.9 / 9.9
//   shared rows   1x8x8 512->512 12.7 / 10.1, 1x16x16 256->256 10.3 / 9.5; 16x16x16 256->256 10.6 / 11.4, 4x32x32 128->128 9.3 / 9.9,
//                 37x15x13 48->80 10.9 / 12.8
// and with random words, whose drawing is shared out too, it pays from half of that on: 64x8x8 128->128 11.9 / 10.6, 4x32x32
// 128->128 11.2 / 10.5; 8x32x32 64->64 10.4 / 12.1.
static int split_cluster(int tiles, int taps, int red, bool halo, bool stochastic, int bw) {
    if (tiles > sm_count() / 2 || (g_two_cta & 2) || !g_cooperative) return 1;  // without the guarantee a cluster more is a barrier that may not be met
    const int num_kb = taps * ((red + 127) / 128);
    const auto fits = [&](int cs, int clusters) { return tiles <= clusters && num_kb >= 2 * cs && (bw == 0 || 128 / cs % (2 * bw) == 0); };
    const int cs = fits(8, split_clusters<8>()) ? 8 : fits(4, split_clusters<4>()) ? 4 : fits(2, split_clusters<2>()) ? 2 : 1;
    // reduction steps of 32 channels that the other CTAs take over, in quarters of a block
    const int saved = taps * ((red + 31) / 32) * (cs - 1) / cs;
    return saved >= (stochastic ? 24 : halo ? 46 : 30) ? cs : 1;
}

int umma_gemm_splits(int M, int N, int K) {
    const int bn = (N > 128) ? 256 : 128;
    const int tiles = ((M + 127) / 128) * ((N + bn - 1) / bn);
    const int kb = (K + 127) / 128;
    if (tiles * 2 > sm_count() || kb < 8) return 1;
    int splits = sm_count() / tiles;
    if (splits > kb / 2) splits = kb / 2;
    return splits < 1 ? 1 : splits;
}

// out[splits][M][N] (splits == 1: the result itself) = op(A) * op(B) over disjoint reduction ranges.
// `fused` == null: int32 out; otherwise int8 out narrowed by the shift in fused->state[0] (splits must be 1).
// rows32: operands of 32-byte rows as im2col32 writes them (1: A and B, K = 32; 2: B only, N = 32).  As boxes of a
// tensor map such rows cost the TMA unit about 18 cycles each, inner extent beyond the row and all: one 128 x 128 tile of
// a first layer (256 rows) took 4600 cycles, whatever its epilogue did.  3 -> 128 channels, 500 images: 109 -> 68 us
// with the gather, 3 -> 64, 1024 images: the product alone 110 -> 44 us.
int umma_gemm(const int8_t* A, const int8_t* B, void* out, unsigned* maxabs, int M, int N, int K, int trans_a,
              int trans_b, int splits, const FusedArgs* fused, int32_t* status, cudaStream_t st, int rows32, int lda, int ldc) {
    CUtensorMap ma, mb, mc;
    const int a_mn = trans_a ? 1 : 0, b_mn = trans_b ? 0 : 1;
    const int bn = fused ? requant_bn(N, 1 << 20) : (N > 128) ? 256 : 128;
    const bool pair = rows32 == 0 && !fused && pair_ok((M + 127) / 128, bn, b_mn, 0);
    {
        uint64_t dims[2], str[1]; uint32_t box[2] = {128, 128};
        if (a_mn) { dims[0] = M; dims[1] = K; str[0] = lda > 0 ? lda : M; } else { dims[0] = K; dims[1] = M; str[0] = lda > 0 ? lda : K; }
        if (int e = encode_map(&ma, A, false, 2, dims, str, box)) return e;
        if (b_mn) { dims[0] = N; dims[1] = K; str[0] = N; box[1] = 128; } else { dims[0] = K; dims[1] = N; str[0] = K; box[1] = pair ? bn / 2 : bn; }
        if (int e = encode_map(&mb, B, false, 2, dims, str, box)) return e;
        uint64_t dc[4] = {(uint64_t)N, (uint64_t)M, (uint64_t)splits, 1};
        const uint64_t pitch = ldc > 0 ? ldc : N;
        uint64_t sc[3] = {pitch * 4, M * pitch * 4, splits * M * pitch * 4};
        uint32_t bc[4] = {32, 128, 1, 1};
        if (!fused) if (int e = encode_map(&mc, out, true, 4, dc, sc, bc)) return e;
    }
    GemmParams p{};
    p.conv = 0; p.M = M; p.N = N; p.num_kb = (K + 127) / 128; p.splits = splits;
    p.m_tiles = (M + 127) / 128; p.n_tiles = (N + bn - 1) / bn;
    if (pair) p.m_tiles = (p.m_tiles + 1) / 2;
    p.a_mn = a_mn; p.b_mn = b_mn; p.a_bytes = PANEL_BYTES; p.b_bytes = (pair ? bn / 2 : bn) * ROW_BYTES;
    p.mma_n = rows32 == 2 ? 32 : mma_columns(N, bn, p.n_tiles, pair);
    p.rows32 = rows32; p.a32 = A; p.b32 = B; p.K = K;
    p.maxabs = splits > 1 ? nullptr : maxabs; p.status = status;
    p.split_cols = (bn == 256 && p.m_tiles * p.n_tiles * splits <= 2 * (pair ? sm_count() / 2 : sm_count())) ? 1 : 0;
    // operands beyond ~half of the 126 MB L2: order the tiles in compact groups
    p.group_m = (static_cast<long long>(M) + N) * K > (48ll << 20) ? 8 : 0;
    set_fused(&p, fused);
    finish_params(&p);
    if (fused) { p.out8 = static_cast<int8_t*>(out); return launch_requant(bn, false, rows32 ? LOAD_ROWS32 : LOAD_TAPS, false, fused->one, ma, mb, p, st); }
    return launch_gemm(bn, pair, ma, mb, mc, p, st);
}

// Forward convolution (flip == 0: x [N,H,W,C] with w [K,R,S,C] -> [N,H,W,K]) or error-backward
// (flip == 1: err [N,H,W,K] with the same w -> [N,H,W,C]); "same" padding, stride 1.
// Forward reads w rows as the N operand (K-major); backward reads the very same tensor as the
// reduction operand (MN-major: 128 k rows of 128 c bytes per tap), so no transposed copy exists.
int umma_conv(const int8_t* x, const int8_t* w, void* out, unsigned* maxabs, int Nimg, int H, int W, int C, int K,
              int R, int S, int pad, int flip, const FusedArgs* fused, int32_t* status, cudaStream_t st) {
    CUtensorMap ma, mb, mc;
    const int red = flip ? K : C;   // reduction channels per tap
    const int outc = flip ? C : K;  // output channels
    GemmParams p{};
    const bool parked = fused && fused->parked;
    const bool k3 = R == 3 && S == 3 && pad == 1;
    ConvPlan plan = fused && fused->pool_out != nullptr ? pool_plan(Nimg, H, W, red, outc, k3)
                                                        : conv_plan(Nimg, H, W, red, outc, k3, flip, !fused ? 0 : parked ? 2 : 1,
                                                                    fused && fused->mode == NITI_ROUND_STOCHASTIC);
    int split = 1;
    if (parked && !fused->whole) {
        const ConvPlan taps = conv_plan(Nimg, H, W, red, outc, false, flip, 2);
        split = split_cluster(taps.m_tiles * ((outc + 127) / 128), R * S, red, plan.halo, fused->mode == NITI_ROUND_STOCHASTIC,
                              fused->pool_out != nullptr ? taps.BW : 0);
        if (split > 1) { plan = taps; plan.bn = 128; }
    }
    const int bn = plan.bn;
    const bool pair = plan.pair;
    p.BW = plan.BW; p.BH = plan.BH; p.BI = plan.BI;
    {
        uint64_t dims[4] = {(uint64_t)red, (uint64_t)W, (uint64_t)H, (uint64_t)Nimg};
        uint64_t str[3] = {(uint64_t)red, (uint64_t)W * red, (uint64_t)H * W * red};
        uint32_t box[4] = {128, (uint32_t)p.BW, (uint32_t)(plan.halo ? p.BH + 2 : p.BH), (uint32_t)p.BI};
        // Rows that end inside the box: without promotion (a TMA unit's cycles per row, 128-byte boxes of 16 / 48 / 64 / 80 / 96 / 128
        // channels: 4.2 / 4.9 / 2.0 / 5.0 / 2.5 / 1.85, with promotion 5.8 / 6.5 / 2.35 / 6.75 / 2.8 / 1.85)
        if (int e = encode_map(&ma, x, false, 4, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B,
                               red % 128 == 0 ? CU_TENSOR_MAP_L2_PROMOTION_L2_256B : CU_TENSOR_MAP_L2_PROMOTION_NONE)) return e;
        uint64_t d2[2] = {(uint64_t)R * S * C, (uint64_t)K};
        uint64_t s2[1] = {(uint64_t)R * S * C};
        const bool narrow_b = flip && bn == 64;  // MN-major rows of 64 bytes
        // Rows of a weight box: no more than there are output channels (the columns beyond are neither stored nor counted) or, where
        // they are the reduction, than its MMAs read.
        uint32_t b2[2] = {narrow_b ? 64u : 128u, flip ? 128u : (uint32_t)(pair ? bn / 2 : bn)};
        if (!pair && !flip && outc < bn) b2[1] = (uint32_t)outc;
        if (!pair && flip && red < 128) b2[1] = (uint32_t)((red + 31) / 32 * 32);
        p.b_bytes = flip ? (int)b2[1] * (pair ? bn / 2 : bn) : (int)b2[1] * ROW_BYTES;
        if (int e = encode_map(&mb, w, false, 2, d2, s2, b2, narrow_b ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B)) return e;
        uint64_t dc[4] = {(uint64_t)outc, (uint64_t)W, (uint64_t)H, (uint64_t)Nimg};
        uint64_t sc[3] = {(uint64_t)outc * 4, (uint64_t)W * outc * 4, (uint64_t)H * W * outc * 4};
        uint32_t bc[4] = {32, (uint32_t)p.BW, (uint32_t)p.BH, (uint32_t)p.BI};
        if (!fused) if (int e = encode_map(&mc, out, true, 4, dc, sc, bc)) return e;
    }
    p.conv = 1; p.flip = flip; p.splits = split;
    p.H = H; p.W = W; p.S = S; p.pad = pad; p.Nimg = Nimg; p.tapstride = C;
    p.tiles_w = plan.tiles_w; p.tiles_h = plan.tiles_h;
    p.cblocks = (red + 127) / 128; p.red = red;
    p.M = Nimg * H * W; p.N = outc; p.num_kb = R * S * p.cblocks;
    p.m_tiles = plan.m_tiles; p.n_tiles = (outc + bn - 1) / bn;
    if (pair) p.m_tiles = (p.m_tiles + 1) / 2;
    p.mma_n = mma_columns(outc, bn, p.n_tiles, pair);
    p.a_mn = 0; p.b_mn = flip ? 1 : 0; p.a_bytes = p.BW * (plan.halo ? p.BH + 2 : p.BH) * p.BI * ROW_BYTES;
    p.maxabs = maxabs; p.status = status;
    p.split_cols = (bn == 256 && p.m_tiles * p.n_tiles <= 2 * (pair ? sm_count() / 2 : sm_count())) ? 1 : 0;
    set_fused(&p, fused);
    finish_params(&p);
    if (fused) p.out8 = static_cast<int8_t*>(out);
    if (fused && fused->pool_out != nullptr) {
        if (!parked || flip || !pool_box_ok(H, W, p.BW, p.BH)) return NITI_ERR_UNSUPPORTED;
        p.pool_out = fused->pool_out;
    }
    if (parked && !fits_parked(bn, p.m_tiles * p.n_tiles, pair)) return NITI_ERR_UNSUPPORTED;
    if (split > 1) {
        const int rc = split == 8 ? launch_split<8>(ma, mb, p, st) : split == 4 ? launch_split<4>(ma, mb, p, st) : launch_split<2>(ma, mb, p, st);
        if (rc != LAUNCH_REFUSED) return rc;
        FusedArgs whole = *fused;  // fewer SMs than the device has: a CS-th of them may do
        whole.whole = 1;
        return umma_conv(x, w, out, maxabs, Nimg, H, W, C, K, R, S, pad, flip, &whole, status, st);
    }
    const int mode = !plan.halo ? LOAD_TAPS : p.cblocks == 1 && p.n_tiles == 1 ? LOAD_HALO_RESIDENT : LOAD_HALO;
    if (fused) return launch_requant(bn, pair, mode, parked, fused->one && !pair, ma, mb, p, st);
    return launch_gemm(bn, pair, ma, mb, mc, p, st);
}

// the parked kernel can pool 2x2 / stride 2 in its epilogue when every window lies inside one warp's 32 rows of a tile
static bool pool_box_ok(int H, int W, int bw, int bh) {
    return H % 2 == 0 && W % 2 == 0 && bh % 2 == 0 && (bw == 2 || bw == 4 || bw == 8 || bw == 16);
}
bool umma_conv_pool_fusable(int Nimg, int H, int W, int outc) {
    const ConvPlan c = conv_plan(Nimg, H, W, 0, outc, false, 0, 2);
    return pool_box_ok(H, W, c.BW, c.BH) && umma_conv_fits_parked(Nimg, H, W, 0, outc, false, 0);
}

bool umma_conv_fits_parked(int Nimg, int H, int W, int red, int outc, bool k3, int flip) {
    const ConvPlan c = conv_plan(Nimg, H, W, red, outc, k3, flip, 2);
    return fits_parked(c.bn, (c.pair ? (c.m_tiles + 1) / 2 : c.m_tiles) * ((outc + c.bn - 1) / c.bn), c.pair);
}

static void wgrad_plan(int Nimg, int H, int W, int C, int K, int R, int max_splits, WgradParams* p) {
    pick_pixel_box(Nimg, H, W, &p->BW, &p->BH, &p->BI);
    p->tiles_w = (W + p->BW - 1) / p->BW; p->tiles_h = (H + p->BH - 1) / p->BH; p->tiles_n = (Nimg + p->BI - 1) / p->BI;
    p->chunks = p->tiles_w * p->tiles_h * p->tiles_n;
    p->k_tiles = (K + 127) / 128; p->c_tiles = (C + 127) / 128;
    const int items = R * p->k_tiles * p->c_tiles;
    int splits = sm_count() / items;  // never more CTAs than SMs: a second wave of a few CTAs would double the time
    if (splits < 1) splits = 1;
    if (splits > p->chunks) splits = p->chunks;
    if (max_splits > 0 && splits > max_splits) splits = max_splits;
    p->splits = splits;
}

size_t umma_wgrad_scratch_bytes(int Nimg, int H, int W, int C, int K, int R, int S) {
    WgradParams p{};
    wgrad_plan(Nimg, H, W, C, K, R, 0, &p);
    return static_cast<size_t>(p.splits) * K * R * S * C * sizeof(int32_t);
}

// Tensor maps and kernel parameters of one layer; p->splits (and the rest of the plan) must already be set.
static int wgrad_setup(const int8_t* x, const int8_t* err, int32_t* out, int direct, int Nimg, int H, int W, int C, int K, int R,
                       int S, int pad, int32_t* status, WgradParams* p, CUtensorMap* me, CUtensorMap* mx, CUtensorMap* mp) {
    p->reduce_direct = direct;
    uint32_t box[4] = {128, (uint32_t)p->BW, (uint32_t)p->BH, (uint32_t)p->BI};
    uint64_t de[4] = {(uint64_t)K, (uint64_t)W, (uint64_t)H, (uint64_t)Nimg};
    uint64_t se[3] = {(uint64_t)K, (uint64_t)W * K, (uint64_t)H * W * K};
    if (int e = encode_map(me, err, false, 4, de, se, box)) return e;
    uint64_t dx[4] = {(uint64_t)C, (uint64_t)W, (uint64_t)H, (uint64_t)Nimg};
    uint64_t sx[3] = {(uint64_t)C, (uint64_t)W * C, (uint64_t)H * W * C};
    if (int e = encode_map(mx, x, false, 4, dx, sx, box)) return e;
    uint64_t dp[4] = {(uint64_t)C, (uint64_t)R * S, (uint64_t)K, (uint64_t)(direct ? 1 : p->splits)};
    uint64_t sp[3] = {(uint64_t)C * 4, (uint64_t)R * S * C * 4, (uint64_t)K * R * S * C * 4};
    uint32_t bp[4] = {32, 1, 128, 1};
    if (int e = encode_map(mp, out, true, 4, dp, sp, bp)) return e;
    p->H = H; p->W = W; p->C = C; p->K = K; p->R = R; p->S = S; p->pad = pad; p->Nimg = Nimg;
    const int rows = p->BW * p->BH * p->BI;
    p->box_bytes = rows * ROW_BYTES;
    p->mma_per_chunk = (rows + 31) / 32;
    p->partial = out; p->status = status;
    return NITI_OK;
}

// partial != null, direct == 0: CTA (split, tile) stores its sums to partial[split] (the caller folds them);
// direct == 1: `partial` is the gradient itself, zeroed by the caller, and every CTA adds into it.
int umma_conv_wgrad_partials(const int8_t* x, const int8_t* err, int32_t* partial, int* splits_out, int max_splits,
                             int Nimg, int H, int W, int C, int K, int R, int S, int pad, int32_t* status, cudaStream_t st,
                             int direct) {
    WgradParams p{};
    wgrad_plan(Nimg, H, W, C, K, R, max_splits, &p);
    CUtensorMap me, mx, mp;
    if (int e = wgrad_setup(x, err, partial, direct, Nimg, H, W, C, K, R, S, pad, status, &p, &me, &mx, &mp)) return e;
    *splits_out = p.splits;
    cudaError_t e = allow_shared<umma_wgrad_kernel>(WG_SMEM_BYTES);
    if (e != cudaSuccess) return set_cuda_error(e);
    dim3 grid(p.splits, R * p.k_tiles * p.c_tiles);
    umma_wgrad_kernel<<<grid, UMMA_THREADS, WG_SMEM_BYTES, st>>>(me, mx, mp, p);
    return launched(cudaGetLastError());
}

// The gradient into `out`, cleared by the launch, and where *updated says so the update of `w`; state: int32[4], zero between calls.
// words: cleared too, and the first becomes max |g| of an update.
bool umma_conv_wgrad_update_fits(int Nimg, int H, int W, int C, int K, int R) {
    WgradParams p{};
    wgrad_plan(Nimg, H, W, C, K, R, 0, &p);
    return p.splits * R * p.k_tiles * p.c_tiles <= sm_count();
}
int umma_conv_wgrad_update(const int8_t* x, const int8_t* err, int32_t* out, int8_t* w, uint32_t* words, int num_words, int32_t* state,
                           int Nimg, int H, int W, int C, int K, int R, int S, int pad, int mu, int mode, const unsigned long long* seed,
                           unsigned rng_stream, bool* updated, int32_t* status, cudaStream_t st) {
    WgradParams p{};
    wgrad_plan(Nimg, H, W, C, K, R, 0, &p);
    CUtensorMap me, mx, mp;
    if (int e = wgrad_setup(x, err, out, p.splits > 1 ? 1 : 0, Nimg, H, W, C, K, R, S, pad, status, &p, &me, &mx, &mp)) return e;
    const long long n = static_cast<long long>(K) * R * S * C;
    *updated = n <= WG_UPDATE_MAX;
    const WgradUpdate u{out, *updated ? w : nullptr, words, words, num_words, n, mu, mode, seed, rng_stream, state};
    cudaError_t e = allow_shared<umma_wgrad_update_kernel>(WG_SMEM_BYTES);
    if (e != cudaSuccess) return set_cuda_error(e);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(p.splits, R * p.k_tiles * p.c_tiles); cfg.blockDim = dim3(UMMA_THREADS); cfg.dynamicSmemBytes = WG_SMEM_BYTES; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative; attr[0].val.cooperative = g_cooperative;
    cfg.attrs = attr; cfg.numAttrs = 1;
    return launched_together(cudaLaunchKernelEx(&cfg, umma_wgrad_update_kernel, me, mx, mp, p, u));
}

// x_t [C][H][W][N], err_t [K][H][W][N] (batch innermost, N a multiple of 16) -> out [C][R][S][K], zeroed by the caller:
// out[c][r][s][k] = sum err_t[k][pixel] * x_t[c][pixel + (r, s) - pad].  x's channels are the rows of the product, so that
// the result needs no transposition either; the taps move the error instead, the other way.
int umma_conv_wgrad_batch_inner(const int8_t* x_t, const int8_t* err_t, int32_t* out, int Nimg, int H, int W, int C, int K, int R,
                                int S, int pad, int32_t* status, cudaStream_t st) {
    WgradParams p{};
    p.BW = p.BH = 1; p.BI = 128;
    p.tiles_w = W; p.tiles_h = H; p.tiles_n = (Nimg + 127) / 128;
    p.chunks = p.tiles_w * p.tiles_h * p.tiles_n;
    p.k_tiles = (C + 127) / 128; p.c_tiles = (K + 127) / 128;
    p.splits = sm_count() / (R * p.k_tiles * p.c_tiles);
    if (p.splits < 1) p.splits = 1;
    if (p.splits > p.chunks) p.splits = p.chunks;
    p.reduce_direct = 1; p.flip = 1;
    p.H = H; p.W = W; p.C = K; p.K = C; p.R = R; p.S = S; p.pad = pad; p.Nimg = Nimg;
    p.box_bytes = PANEL_BYTES;  // a box is always written whole; images beyond the batch are zero fill
    p.mma_per_chunk = Nimg < 128 ? (Nimg + 31) / 32 : 4;
    p.partial = out; p.status = status;
    CUtensorMap ma, mb, mc;
    const uint32_t box[4] = {128, 1, 1, 128};
    const uint64_t str[3] = {(uint64_t)Nimg, (uint64_t)W * Nimg, (uint64_t)H * W * Nimg};
    const uint64_t da[4] = {(uint64_t)Nimg, (uint64_t)W, (uint64_t)H, (uint64_t)C}, db[4] = {(uint64_t)Nimg, (uint64_t)W, (uint64_t)H, (uint64_t)K};
    if (int e = encode_map(&ma, x_t, false, 4, da, str, box)) return e;
    if (int e = encode_map(&mb, err_t, false, 4, db, str, box)) return e;
    const uint64_t dc[4] = {(uint64_t)K, (uint64_t)R * S, (uint64_t)C, 1};
    const uint64_t sc[3] = {(uint64_t)K * 4, (uint64_t)R * S * K * 4, (uint64_t)C * R * S * K * 4};
    const uint32_t bc[4] = {32, 1, 128, 1};
    if (int e = encode_map(&mc, out, true, 4, dc, sc, bc)) return e;
    cudaError_t e = allow_shared<umma_wgrad_kmajor_kernel>(WG_SMEM_BYTES);
    if (e != cudaSuccess) return set_cuda_error(e);
    umma_wgrad_kmajor_kernel<<<dim3(p.splits, R * p.k_tiles * p.c_tiles), UMMA_THREADS, WG_SMEM_BYTES, st>>>(ma, mb, mc, p);
    return launched(cudaGetLastError());
}

int umma_wgrad_multi_max() { return WG_MULTI_MAX; }

// Splits for layers whose items alone are more than the SMs: of several ways to cut them, the one whose thread blocks, longest
// first, are done earliest on `sms` SMs.  A thread block costs its chunks and about twelve chunks' time for its start and its
// flush.  Left uncut, the four last layers of VGG-13 at batch 1024 (48 + 48 items of 32 chunks, 48 + 24 of 128) were 168 blocks:
// 20 of 128 chunks started when the first ones were through.
static void wgrad_deal(WgradMultiParams* mp, const int* items, int count, int sms) {
    constexpr int OVERHEAD = 12, MAX_BLOCKS = 512;
    constexpr int CUTS[] = {1, 2, 3, 4, 6, 8};
    long long best = -1;
    int splits[WG_MULTI_MAX], chosen[WG_MULTI_MAX];
    for (int ref = 0; ref < count; ++ref)
        for (const int cut : CUTS) {
            const int len = (mp->layer[ref].chunks + cut - 1) / cut;  // chunks of a thread block
            int order[WG_MULTI_MAX], total = 0;
            for (int l = 0; l < count; ++l) {
                splits[l] = (mp->layer[l].chunks + len - 1) / len;
                total += splits[l] * items[l];
            }
            if (total > MAX_BLOCKS && best >= 0) continue;
            const auto cost = [&](int l) { return (mp->layer[l].chunks + splits[l] - 1) / splits[l] + OVERHEAD; };
            for (int l = 0; l < count; ++l) {
                int at = l;
                for (; at > 0 && cost(order[at - 1]) < cost(l); --at) order[at] = order[at - 1];
                order[at] = l;
            }
            // When SMs are free, earliest first, and how many then.  All that are free at a time take a layer's next blocks together,
            // so there are no more such times than layers and one, and a schedule is a few dozen steps (a heap of SMs dealt to block
            // by block took 20 to 44 us of the host's time in every call, these steps 1 to 4).
            struct Free { long long at; int sms; } free[WG_MULTI_MAX + 1] = {{0, sms}};
            int times = 1;
            long long end = 0;
            for (int o = 0; o < count; ++o)
                for (int left = splits[order[o]] * items[order[o]]; left > 0;) {
                    const int taken = left < free[0].sms ? left : free[0].sms;
                    const long long done = free[0].at + cost(order[o]);
                    left -= taken;
                    if ((free[0].sms -= taken) == 0) {
                        --times;
                        for (int i = 0; i < times; ++i) free[i] = free[i + 1];
                    }
                    int at = times;
                    while (at > 0 && free[at - 1].at > done) --at;
                    if (at > 0 && free[at - 1].at == done) {
                        free[at - 1].sms += taken;
                    } else {
                        for (int i = times++; i > at; --i) free[i] = free[i - 1];
                        free[at] = {done, taken};
                    }
                    if (done > end) end = done;
                }
            if (best < 0 || end < best) { best = end; for (int l = 0; l < count; ++l) chosen[l] = splits[l]; }
        }
    for (int l = 0; l < count; ++l) mp->layer[l].splits = chosen[l];
}

// Up to WG_MULTI_MAX layers' gradients added into their (zeroed or accumulating) int32 buffers by one launch.
int umma_conv_wgrad_multi(const WgradJob* jobs, int count, int32_t* status, cudaStream_t st) {
    if (count < 1 || count > WG_MULTI_MAX) return NITI_ERR_BAD_ARG;
    WgradMultiParams mp{};
    WgradMultiMaps maps;
    int items[WG_MULTI_MAX];
    long long work = 0;  // item-chunks of the whole launch
    for (int l = 0; l < count; ++l) {
        const WgradJob& j = jobs[l];
        wgrad_plan(j.N, j.H, j.W, j.C, j.K, j.R, 0, &mp.layer[l]);
        items[l] = j.R * mp.layer[l].k_tiles * mp.layer[l].c_tiles;
        work += static_cast<long long>(items[l]) * mp.layer[l].chunks;
    }
    // chunks per CTA: the smallest number for which the launch still fits in one wave
    const int sms = sm_count();
    long long per_cta = (work + sms - 1) / sms;
    if (per_cta < 1) per_cta = 1;
    for (;; ++per_cta) {
        int ctas = 0;
        for (int l = 0; l < count; ++l) {
            int sp = static_cast<int>((mp.layer[l].chunks + per_cta - 1) / per_cta);
            if (sp < 1) sp = 1;
            mp.layer[l].splits = sp;
            ctas += sp * items[l];
        }
        if (ctas <= sms) break;
        bool whole = true;  // nothing left to merge: every layer is down to one split
        for (int l = 0; l < count; ++l) whole = whole && mp.layer[l].splits == 1;
        if (whole) { wgrad_deal(&mp, items, count, sms); break; }
    }
    // the longest thread blocks first: where there are more than SMs, the short ones fill up behind them
    int order[WG_MULTI_MAX];
    for (int l = 0; l < count; ++l) {
        int at = l;
        const auto len = [&](int i) { return (mp.layer[i].chunks + mp.layer[i].splits - 1) / mp.layer[i].splits; };
        for (; at > 0 && len(order[at - 1]) < len(l); --at) order[at] = order[at - 1];
        order[at] = l;
    }
    const WgradMultiParams planned = mp;
    int grid = 0;
    for (int l = 0; l < count; ++l) {
        const WgradJob& j = jobs[order[l]];
        mp.layer[l] = planned.layer[order[l]];
        if (int e = wgrad_setup(j.x, j.err, j.g32, 1, j.N, j.H, j.W, j.C, j.K, j.R, j.S, j.pad, status, &mp.layer[l], &maps.err[l],
                                &maps.x[l], &maps.g[l])) return e;
        mp.first_cta[l] = grid;
        grid += mp.layer[l].splits * items[order[l]];
    }
    mp.first_cta[count] = grid;
    mp.count = count;
    cudaError_t e = allow_shared<umma_wgrad_multi_kernel>(WG_SMEM_BYTES);
    if (e != cudaSuccess) return set_cuda_error(e);
    umma_wgrad_multi_kernel<<<grid, UMMA_THREADS, WG_SMEM_BYTES, st>>>(maps, mp);
    return launched(cudaGetLastError());
}

}  // namespace niti
