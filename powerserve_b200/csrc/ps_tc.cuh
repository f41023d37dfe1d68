// ps_tc.cuh — tcgen05 (5th-gen tensor core) GEMM for token batches: dst{N, bs} = W{K, N} . x{K, bs}, Q4_K weights x Q8_K
// activations, BIT-IDENTICAL to ggml_vec_dot_q4_K_q8_K per column (ggml-quants.c:7809-7872).
//
// The reference's result is not a plain dot product: per super-block i and AVX lane l it forms the INTEGER
//   S_l = sum_{j<8} sc_j * sum_{t<4} q4[j][4l+t] * q8[j][4l+t]            (and P_k = m_2k*bs_2k + m_2k+1*bs_2k+1 for the mins)
// and then advances 8 + 4 fp32 FMA chains, acc_l = fma(d_x*d_y, (float)S_l, acc_l).  The integer part is a dense
// contraction, and it is EXACT on the tensor cores in fp16/fp32: the operands sc_j*q4 (<= 945) and q8 (|.| <= 127) are
// integers that fp16 represents exactly, every product is exact in fp32 and a 32-term sum stays below 2^24.
//
// What bounds it.  The 12 FMAs per (row, column, super-block) are CUDA-core work that nothing replaces, and 12 accumulators per output
// limit a tile that holds them all to 128 x 32; such a tile re-reads (and would have to de-quantise) its weights for every 32 columns.
// So a tile is 128 rows x NT columns (up to 64) and its chains are taken in six PASSES over K of two chains each - the lane pairs
// (0,4) (2,6) (1,5) (3,7), which hsum_float_8 adds first, and the mins pairs (0,2) (1,3) - with 2 x NT / 2 accumulators a thread.  A
// pass needs only its own quarter of the quants.  A pass ends with ONE number per output; the six are added in the reference's order
//   ((r04 + r26) + (r15 + r37)) + (m02 + m13).
//   * weights stay packed (20 480 B per 128 rows x 256, 1.11x the GGUF bytes; a tile reads 29 696, since every lane pass takes all scales and every
//     pass its factors): de-quantising warps (thread = row) turn the 16 bytes of a
//     (row, lane) into 32 halves - (1024 + nibble) by bit insertion, one HFMA2 per two values for the subtraction and the scale - and
//     write them with tcgen05.st straight into TENSOR MEMORY, from where tcgen05.mma takes its A operand: neither the expanded weights
//     nor their re-reads cross shared memory, whose bandwidth would otherwise be the first limit.
//   * activations (B): q8 as fp16 in canonical K-major tiles, written once per GEMM input by ps_k_tc_prep_b; TMA bulk copies.
//   * accumulators: a ring of tensor-memory entries; packed fma.rn.f32x2 advances two columns' chains per instruction.
// Pipeline: TMA producer -> de-quantising warps -> single-thread MMA issuer -> epilogue warps, linked by four kinds of mbarrier: a stage is
// full / empty, an entry may be computed (go: its A written, its accumulators drained) / is computed (done).
// Work: all passes of all tiles in a row, cut into one contiguous share per CTA, so that the shares differ by one pass at most and a CTA hands numbers
// over for two tiles at most, whatever the matrix.  The CTA that finishes a shared tile last adds the numbers and stores.
//
// Measured (time that each further super-block of a pass adds, at 1.92 GHz; 128 rows x 16 / 32 / 48 / 64 columns): 390 / 450 / 510 / 590 cycles, where a kernel with
// two units of work to a tile, epilogue warps of half the columns and a barrier per hand-over needed 720 to 820 at any width.  Where it goes (64 columns): the
// epilogue's own work 270 (16 FMUL2 and 32 FFMA2 a warp, 192 of pipe time), de-quantising 140 in a lane pass, and what the roles need for their waits and rings:
// 630 of 1 800 instructions.  28 672 x 4096 on 16 / 32 / 64 / 128 columns: 86 / 108 / 104 / 168 -> 45 / 53 / 71 / 126 us; 4096 x 14 336 on 128: 104 -> 76.
// An epilogue that reads more than eight columns at a time spills or moves registers (64 columns: 590 cycles with 8, 655 with 16, 676 with 32, 700 with two
// buffers of 8); the end of a pass is met once per pass with cold instructions, so its loops hold no branches (64 columns: 12 us a tile with, 3.5 without).
#pragma once
#include "ps_rw.cuh"

#define PS_TC_M 128
// K is taken in steps of TWO super-blocks (one stage, one bulk copy per operand; an odd count is padded by a super-block of zeros, which
// leaves every chain as it is: fma(0, 0, acc)).  nbp = super-blocks rounded up to even.
// packed weights of a 128-row tile: [4 lane passes][nbp][2 lanes][128 rows][16 B quants], [nbp][128 rows][8 fp16 scales], [nbp][128 d],
// [nbp][128 rows][8 mins], [nbp][128 -dmin]
#define PS_TC_A_Q 4096
#define PS_TC_A_SC 2048
#define PS_TC_A_MN 1024
#define PS_TC_A_D 512
#define PS_TC_A_BLOCK (4 * PS_TC_A_Q + PS_TC_A_SC + PS_TC_A_MN + 2 * PS_TC_A_D) // 20480 per (row tile, super-block)
#define PS_TC_A_OFF_SC(nbp) ((size_t)(nbp) * (4 * PS_TC_A_Q))
#define PS_TC_A_OFF_D(nbp) ((size_t)(nbp) * (4 * PS_TC_A_Q + PS_TC_A_SC))
#define PS_TC_A_OFF_MN(nbp) ((size_t)(nbp) * (4 * PS_TC_A_Q + PS_TC_A_SC + PS_TC_A_D))
#define PS_TC_A_OFF_DM(nbp) ((size_t)(nbp) * (4 * PS_TC_A_Q + PS_TC_A_SC + PS_TC_A_D + PS_TC_A_MN))
// activations of an NT-column tile: [4 lane passes][nbp][NT * 128 B], [2 mins passes][nbp][NT * 64 B], [nbp][NT d]
#define PS_TC_B_BLOCK(NT) ((NT) * 644)
#define PS_TC_PASSES 6
// lane pass p takes the AVX lanes l and l + 4 with l = 0, 2, 1, 3; this is the pass of lane l
PS_HD int ps_tc_pass(int l) { return ((l & 1) << 1) | ((l >> 1) & 1); }

// configuration by column-tile width
template <int NT> struct PsTc {
    static constexpr int EW = 8;                                // epilogue warps
    static constexpr int EC = NT * 4 / EW;                      // columns a thread owns (its warp's lane quadrant gives the row)
    // super-blocks of an entry: with two, every role waits half as often (48 columns: 510 cycles a super-block).  At 64 columns tensor memory holds three
    // entries of one super-block, or one of two
    static constexpr int XE = NT <= 48 ? 2 : 1;
    static constexpr int NE = XE == 1 ? 3 : NT == 16 ? 4 : 2;   // ring of accumulator entries with their A
    // de-quantising warpgroups, one per super-block of a step.  Where the epilogue is short they set the pace: four then take every second step
    // (16 columns: 450 -> 390 cycles, 32: 464 -> 450; 48 columns 510 -> 530, so two)
    static constexpr int ND = NT <= 32 ? 4 : 2;
    static constexpr int NS = NT <= 48 ? 6 : 5;                 // stages of two super-blocks (even where ND is 4: a group then sees every use of its slots)
    static constexpr int THREADS = (EW + 4 * ND + 4) * 32;
    // registers a thread of the epilogue and of the de-quantising warps (setmaxnreg; the rest has 24): they add up to what the block is launched with
    static constexpr int R_EPI = ND == 4 ? 128 : 160, R_DEQ = ND == 4 ? 56 : 64;
    static constexpr int TM_E = XE * 2 * NT;                    // tensor-memory columns of an entry's accumulators
    static constexpr int TM_A = NE * TM_E;                      // first column of the A buffers
    static constexpr int TM_USED = TM_A + NE * XE * 32;
    static constexpr int TM_COLS = TM_USED <= 256 ? 256 : 512;
    static constexpr int STAGE_SC = 2 * PS_TC_A_Q;              // quants, scales, B of the two super-blocks (a mins pass: mins at the front, B)
    static constexpr int STAGE_B = STAGE_SC + 2 * PS_TC_A_SC;
    static constexpr int STAGE = STAGE_B + 2 * NT * 128;
    static constexpr int NY = NS + (XE == 1 ? 2 : NE); // the factors' ring: the epilogue still reads them when the stage has been refilled
    static constexpr int FACT = 2 * (PS_TC_A_D + NT * 4);       // d or -dmin of the rows, d of the columns
    static constexpr int STASH = EW * 32 * EC * 4;              // numbers of a tile: the pass before, the sum of the pairs before
    static constexpr int SMEM = NS * STAGE + NY * FACT + 2 * STASH;
    static_assert(TM_USED <= 512 && SMEM <= 230000 && (ND == 2 || NS % 2 == 0), "");
};

// ---------------------------------------------------------------------------------------------------- operand builders
// packed blocks of a matrix, row tile by row tile.  One CTA per (super-block, row tile); rows >= n_rows and super-blocks >= nb are zero.
__global__ void __launch_bounds__(256) ps_k_tc_pack_a(uint8_t *__restrict__ dst, const uint8_t *__restrict__ w, int64_t n_rows, int64_t nb, int64_t tile0) {
    const int64_t i = blockIdx.x, rt = blockIdx.y, nbp = gridDim.x;
    uint8_t *out = dst + (tile0 + rt) * nbp * PS_TC_A_BLOCK;
    for (int idx = threadIdx.x; idx < PS_TC_M * 8; idx += blockDim.x) { // (row, AVX lane l); also sub-block j = l
        const int row = idx >> 3, l = idx & 7, j = l;
        const int64_t n = rt * PS_TC_M + row;
        const bool live = n < n_rows && i < nb;
        const uint8_t *blk = w + (n * nb + i) * PS_Q4_K_BYTES;
        int sc = 0, mn = 0;
        uint4 q = make_uint4(0, 0, 0, 0);
        if (live) { // get_scale_min_k4 (ggml-quants.c:1912-1919)
            const uint8_t *s = blk + 4;
            if (j < 4) { sc = s[j] & 63; mn = s[j + 4] & 63; }
            else { sc = (s[j + 4] & 0xF) | ((s[j - 4] >> 6) << 4); mn = (s[j + 4] >> 4) | ((s[j] >> 6) << 4); }
            const uint32_t *qs = reinterpret_cast<const uint32_t *>(blk + 16) + l; // word g: sub-block 2g (low nibbles), 2g + 1 (high)
            q = make_uint4(qs[0], qs[8], qs[16], qs[24]);
        }
        *reinterpret_cast<uint4 *>(out + (ps_tc_pass(l) * nbp + i) * PS_TC_A_Q + (l >> 2) * 2048 + row * 16) = q;
        // even sub-blocks are read from low nibbles, odd ones from high nibbles (16 x the value): the odd scales are stored / 16
        reinterpret_cast<__half *>(out + PS_TC_A_OFF_SC(nbp) + i * PS_TC_A_SC)[row * 8 + j] = __float2half_rn((j & 1) ? (float)sc * 0.0625f : (float)sc);
        out[PS_TC_A_OFF_MN(nbp) + i * PS_TC_A_MN + row * 8 + j] = (uint8_t)mn;
        if (j == 0) {
            reinterpret_cast<float *>(out + PS_TC_A_OFF_D(nbp) + i * PS_TC_A_D)[row] = live ? ps_half_bits_to_float(*reinterpret_cast<const unsigned short *>(blk)) : 0.f;
            reinterpret_cast<float *>(out + PS_TC_A_OFF_DM(nbp) + i * PS_TC_A_D)[row] = live ? -ps_half_bits_to_float(*reinterpret_cast<const unsigned short *>(blk + 2)) : 0.f;
        }
    }
}

// activation operand of a batch, column tile by column tile; one warp per (super-block, column): quantize_row_q8_K
// (the shared warp quantiser), the q8 of AVX lane l as 32 halves in the order the weights come out of their words - word g = k / 8:
// (2g: t 0, 2) (2g + 1: t 0, 2) (2g: t 1, 3) (2g + 1: t 1, 3) - then half-block sums for the mins and d.  Columns >= bs are zero.
// Tiles are canonical K-major without swizzle: [k / 8][column][8 halves].
__device__ __forceinline__ void ps_tc_store_b(uint8_t *__restrict__ out, int NT, int64_t nbp, int64_t i, int c, int lane, const uint32_t words[2], float yd) {
    // thread (g, l) of the warp builds the 16-byte piece g of lane l: it needs the words (sub-block 2g, l) and (2g + 1, l); natural word
    // (j, l) is words[j / 4] of thread (j % 4) * 8 + l
    const int g = lane >> 3, l = lane & 7, src = ((2 * g) & 3) * 8 + l;
    const uint32_t a0 = __shfl_sync(PS_FULL, words[0], src), a1 = __shfl_sync(PS_FULL, words[1], src);
    const uint32_t b0 = __shfl_sync(PS_FULL, words[0], src + 8), b1 = __shfl_sync(PS_FULL, words[1], src + 8);
    const uint32_t a = g < 2 ? a0 : a1, b = g < 2 ? b0 : b1;
    auto h2 = [](uint32_t w, int t0, int t1) {
        const __half2 h = __halves2half2(__int2half_rn((int)(signed char)(w >> (8 * t0))), __int2half_rn((int)(signed char)(w >> (8 * t1))));
        return *reinterpret_cast<const uint32_t *>(&h);
    };
    *reinterpret_cast<uint4 *>(out + (ps_tc_pass(l) * nbp + i) * NT * 128 + (size_t)(l >> 2) * NT * 64 + ((size_t)g * NT + c) * 16) =
        make_uint4(h2(a, 0, 2), h2(b, 0, 2), h2(a, 1, 3), h2(b, 1, 3));
    // half-block sums: threads of one sub-block, lanes l = 0..3 -> elements 0..15, l = 4..7 -> elements 16..31
    uint32_t hs[2]; // this thread's sub-blocks lane / 8 and 4 + lane / 8: (first half, second half) as half2
#pragma unroll
    for (int h = 0; h < 2; h++) {
        int s = __dp4a((int)words[h], 0x01010101, 0);
        s += __shfl_xor_sync(PS_FULL, s, 1);
        s += __shfl_xor_sync(PS_FULL, s, 2);
        const int s0 = __shfl_sync(PS_FULL, s, lane & 24), s1 = __shfl_sync(PS_FULL, s, (lane & 24) + 4);
        const __half2 v = __halves2half2(__int2half_rn(s0), __int2half_rn(s1)); // |.| <= 2032: exact
        hs[h] = *reinterpret_cast<const uint32_t *>(&v);
    }
    // mins chain k (sub-blocks 2k, 2k + 1): K positions 4k .. 4k + 3 hold its four half sums, the others are zero
    const uint32_t m0 = __shfl_sync(PS_FULL, hs[0], (lane & 1) * 16), m1 = __shfl_sync(PS_FULL, hs[0], (lane & 1) * 16 + 8);
    const uint32_t m2 = __shfl_sync(PS_FULL, hs[1], (lane & 1) * 16), m3 = __shfl_sync(PS_FULL, hs[1], (lane & 1) * 16 + 8);
    if (lane < 4) { // thread k: chain k; pass 4 + (k & 1), chain k / 2 of the pass
        const int k = lane;
        const uint32_t v0 = k < 2 ? m0 : m2, v1 = k < 2 ? m1 : m3;
        uint8_t *t = out + nbp * NT * 512 + ((k & 1) * nbp + i) * NT * 64 + (size_t)(k >> 1) * NT * 32;
        const uint4 mine = (k & 1) ? make_uint4(0, 0, v0, v1) : make_uint4(v0, v1, 0, 0), none = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4 *>(t + (size_t)c * 16) = k < 2 ? mine : none;
        *reinterpret_cast<uint4 *>(t + ((size_t)NT + c) * 16) = k < 2 ? none : mine;
    }
    if (lane == 0) reinterpret_cast<float *>(out + nbp * NT * 640)[i * NT + c] = yd;
}
__global__ void __launch_bounds__(128) ps_k_tc_prep_b(uint8_t *__restrict__ dst, const float *__restrict__ x, const float *__restrict__ u, int64_t K, int bs, int NT) {
    ps_grid_dep();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t nb = K / 256, nbp = (nb + 1) & ~(int64_t)1, i = (int64_t)blockIdx.x * 4 + warp;
    const int col = blockIdx.y, ct = col / NT, c = col % NT;
    if (i >= nbp) return;
    uint32_t words[2] = {0, 0}, bsp = 0;
    float yd = 0.f;
    if (col < bs && i < nb) {
        const int64_t at = (int64_t)col * K + i * 256;
        float e[8];
        ps_act8(x + at, u ? u + at : nullptr, lane, e);
        ps_quant_block_q8k_regs(e, lane, words, yd, bsp);
    }
    ps_tc_store_b(dst + ct * nbp * PS_TC_B_BLOCK(NT), NT, nbp, i, c, lane, words, yd);
}
// the same behind a norm, one CTA a column (128 columns of 4096: 7.0 + 4.2 us as two launches, together 6.2)
__global__ void __launch_bounds__(512) ps_k_tc_norm_b(uint8_t *__restrict__ dst, const float *__restrict__ x, const float *__restrict__ w, int64_t dim, float eps, int bs, int NT) {
    ps_grid_dep();
    __shared__ double sh[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t nb = dim / 256, nbp = (nb + 1) & ~(int64_t)1;
    const int col = blockIdx.x, ct = col / NT, c = col % NT;
    const float *xr = x + (int64_t)col * dim;
    const float scale = col < bs ? ps_rms_scale(xr, dim, eps, sh) : 0.f;
    for (int64_t i = warp; i < nbp; i += 16) {
        uint32_t words[2] = {0, 0}, bsp = 0;
        float yd = 0.f;
        if (col < bs && i < nb) {
            const int64_t at = i * 256 + 4 * lane;
            const float4 p = ps_norm4(xr + at, w + at, scale), q = ps_norm4(xr + at + 128, w + at + 128, scale);
            const float e[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
            ps_quant_block_q8k_regs(e, lane, words, yd, bsp);
        }
        ps_tc_store_b(dst + ct * nbp * PS_TC_B_BLOCK(NT), NT, nbp, i, c, lane, words, yd);
    }
}

// ---------------------------------------------------------------------------------------------------- GEMM
#define PS_TC_SEGS 3
struct PsTcArgs {
    const uint8_t *a;   // [row tiles][nbp * PS_TC_A_BLOCK]
    const uint8_t *b;   // [column tiles][nbp * PS_TC_B_BLOCK(NT)]
    int nbp, n_ct, n_tiles; // super-blocks (even); column tiles; row tiles x column tiles
    PsRwSeg seg[PS_TC_SEGS]; // rows row_begin .. row_end of the padded row space; dst of a segment is [bs][rows of the segment]
    int n_seg, bs;
    const float *residual;
    float *part;        // [CTA][pass][EC][epilogue threads]: numbers of the shared tile that begins in a CTA's share (there is one at most)
    int *cnt;           // [CTA]: how many of its passes have been handed over (left at zero)
    int *err;           // set if a pipeline wait gave up (results invalid)
    int give_up;        // warp whose first wait counts as run out (-1: none): how a test reaches the way out
    uint32_t limit;     // cycles a wait lasts at most
};

// eight columns of one row of an accumulator; they are there after ps_tc_ld_wait, and ps_tc_keep keeps whatever reads them behind it
PS_D void ps_tc_ld(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}
PS_D void ps_tc_keep(uint32_t (&v)[8]) {
    asm volatile("" : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])::"memory");
}
PS_D ps_f2 ps_f2_bits(uint32_t a, uint32_t b) { ps_f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b)); return r; }
PS_D void ps_tc_st8(uint32_t taddr, const uint32_t v[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]),
                 "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
PS_D void ps_tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
PS_D uint32_t ps_h2_fma(uint32_t a, uint32_t b, uint32_t c) { uint32_t r; asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r; }
PS_D uint32_t ps_h2_mul(uint32_t a, uint32_t b) { uint32_t r; asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }

// two words of nibbles of one (row, lane) -> 16 halves sc_j * q4 (two per register); s[j]: the scale of sub-block j twice (odd ones / 16),
// o[j] = -1024 s[j].  (1024 + n) s - 1024 s is exact: both terms are below 65504 and the fused result is an integer <= 945.
PS_D void ps_tc_dequant8(uint32_t w0, uint32_t w1, const uint32_t s[4], const uint32_t o[4], uint32_t v[8]) {
    const uint32_t w[2] = {w0, w1};
#pragma unroll
    for (int g = 0; g < 2; g++) {
        const uint32_t a = w[g], b = w[g] >> 8;
        v[4 * g + 0] = ps_h2_fma((a & 0x000F000Fu) | 0x64006400u, s[2 * g], o[2 * g]);
        v[4 * g + 1] = ps_h2_fma((a & 0x00F000F0u) | 0x64006400u, s[2 * g + 1], o[2 * g + 1]);
        v[4 * g + 2] = ps_h2_fma((b & 0x000F000Fu) | 0x64006400u, s[2 * g], o[2 * g]);
        v[4 * g + 3] = ps_h2_fma((b & 0x00F000F0u) | 0x64006400u, s[2 * g + 1], o[2 * g + 1]);
    }
}

template <int N> PS_D void ps_reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> PS_D void ps_reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// every lane waits for a barrier of its own; bounded like ps_tc_wait.  One such poll costs what a wait for one barrier does (about 80 cycles
// even when the phase is complete).  The vote orders no memory: what a lane acquired with its barrier reaches the other lanes at the __syncwarp
PS_D bool ps_tc_wait_all(uint32_t bar, uint32_t parity, uint32_t cycles) {
    bool ok = __all_sync(PS_FULL, ps_tc_poll(bar, parity));
    if (!ok) {
        const uint32_t t0 = __shfl_sync(PS_FULL, ps_clock32(), 0);
        do ok = __all_sync(PS_FULL, ps_tc_poll(bar, parity));
        while (!ok && __shfl_sync(PS_FULL, ps_clock32(), 0) - t0 < cycles);
    }
    __syncwarp();
    return ok;
}

PS_D int ps_add_acq_rel(int *p, int v) {
    int r;
    asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], %2;" : "=r"(r) : "l"(p), "r"(v) : "memory");
    return r;
}
// the CTA's passes: q = tile * 6 + pass, a contiguous share of all of them
PS_D int ps_tc_share(int c, int n_cta, int n_tiles) { return (int)((int64_t)n_tiles * PS_TC_PASSES * c / n_cta); }
// does a share begin at pass q?
PS_D bool ps_tc_cut(int q, int n_cta, int n_tiles) {
    const int64_t n = (int64_t)n_tiles * PS_TC_PASSES;
    return ps_tc_share((int)(((int64_t)q * n_cta + n - 1) / n), n_cta, n_tiles) == q;
}

// the CTA whose share holds pass q
PS_D int ps_tc_owner(int q, int n_cta, int n_tiles) {
    const int64_t n = (int64_t)n_tiles * PS_TC_PASSES;
    return (int)(((int64_t)(q + 1) * n_cta + n - 1) / n) - 1;
}

// where the operands of pass q lie, and the copies of its step i into a stage
template <int NT> struct PsTcSrc {
    const uint8_t *aq, *as, *ad, *bq, *by;
    bool lanes;
    PS_D PsTcSrc(const PsTcArgs &a, int q) {
        const int tile = q / PS_TC_PASSES, p = q % PS_TC_PASSES;
        const uint8_t *pa = a.a + (size_t)(tile / a.n_ct) * a.nbp * PS_TC_A_BLOCK, *pb = a.b + (size_t)(tile % a.n_ct) * a.nbp * PS_TC_B_BLOCK(NT);
        lanes = p < 4;
        aq = pa + (lanes ? (size_t)p * a.nbp * PS_TC_A_Q : PS_TC_A_OFF_MN(a.nbp));
        as = pa + PS_TC_A_OFF_SC(a.nbp);
        ad = pa + (lanes ? PS_TC_A_OFF_D(a.nbp) : PS_TC_A_OFF_DM(a.nbp));
        bq = pb + (lanes ? (size_t)p * a.nbp * (NT * 128) : (size_t)a.nbp * (NT * 512) + (size_t)(p - 4) * a.nbp * (NT * 64));
        by = pb + (size_t)a.nbp * (NT * 640);
    }
    PS_D void weights(int i, uint8_t *sm, uint8_t *sf, uint64_t *bar) const {
        const uint32_t na = lanes ? 2 * PS_TC_A_Q : 2 * PS_TC_A_MN;
        ps_mbar_expect_tx(bar, na + (lanes ? 2 * PS_TC_A_SC : 0) + 2 * PS_TC_A_D + (lanes ? 2 * NT * 128 : 2 * NT * 64) + 2 * NT * 4);
        ps_bulk_g2s(sm, aq + (size_t)i * na, na, bar);
        if (lanes) ps_bulk_g2s(sm + PsTc<NT>::STAGE_SC, as + (size_t)i * (2 * PS_TC_A_SC), 2 * PS_TC_A_SC, bar);
        ps_bulk_g2s(sf, ad + (size_t)i * (2 * PS_TC_A_D), 2 * PS_TC_A_D, bar);
    }
    PS_D void columns(int i, uint8_t *sm, uint8_t *sf, uint64_t *bar) const {
        const uint32_t nb = lanes ? 2 * NT * 128 : 2 * NT * 64;
        ps_bulk_g2s(sm + PsTc<NT>::STAGE_B, bq + (size_t)i * nb, nb, bar);
        ps_bulk_g2s(sf + 2 * PS_TC_A_D, by + (size_t)i * (2 * NT * 4), 2 * NT * 4, bar);
    }
};

template <int NT>
__global__ void __launch_bounds__(PsTc<NT>::THREADS, 1) ps_k_tc_gemm(const PsTcArgs a) {
    using T = PsTc<NT>;
    extern __shared__ __align__(1024) uint8_t ps_tc_smem[];
    // full: a stage has been copied; empty: its MMAs are complete; go: an entry's A is in tensor memory and its accumulators have been read;
    // done: its MMAs are complete (accumulators readable, A writable)
    __shared__ __align__(8) uint64_t bar_full[T::NS], bar_empty[T::NS], bar_go[T::NE], bar_done[T::NE], bar_end;
    __shared__ uint32_t tmem_base_smem;
    __shared__ int sh_last;
    const int tid = threadIdx.x, warp = __shfl_sync(PS_FULL, tid >> 5, 0), lane = tid & 31;
    const int ns = a.nbp >> 1; // steps of a pass
    const int q0 = ps_tc_share(blockIdx.x, gridDim.x, a.n_tiles), q1 = ps_tc_share(blockIdx.x + 1, gridDim.x, a.n_tiles);
    constexpr int W_TMA = T::EW + 4 * T::ND, W_MMA = W_TMA + 1;
    uint8_t *const ps_tc_fact = ps_tc_smem + (size_t)T::NS * T::STAGE;

    if (tid == 0) {
        for (int s = 0; s < T::NS; s++) {
            ps_mbar_init(&bar_full[s], 1);
            ps_mbar_init(&bar_empty[s], 1);
        }
        for (int s = 0; s < T::NE; s++) {
            ps_mbar_init(&bar_go[s], 4 * T::XE + T::EW);
            ps_mbar_init(&bar_done[s], 1);
        }
        ps_mbar_init(&bar_end, 1);
        ps_fence_barrier_init();
        for (int s = 0; s < T::NE; s++) // the entries are free at first
            for (int w = 0; w < T::EW; w++) ps_mbar_arrive(&bar_go[s]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == W_MMA) { // the MMA warp owns the tensor memory
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ps_smem_u32(&tmem_base_smem)), "n"(T::TM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    ps_tc_fence_before();
    __syncthreads();
    ps_tc_fence_after();
    const uint32_t tmem_base = tmem_base_smem;

    if (warp >= W_TMA) {
        ps_reg_dec<24>();
        if (warp == W_TMA) {
            // ===== TMA producer
            PsRing<T::NS> st;
            PsRing<T::NY> sy;
            int g = 0, ahead = 0;
            bool ok = warp != a.give_up;
            if (!ok) *a.err = 1;
            // the weights of the first steps do not depend on the kernel before: they are asked for while it still runs
            if (ok && q0 < q1) {
                const PsTcSrc<NT> src(a, q0);
                ahead = min(ns, T::NS);
                if (ps_elect_one())
                    for (int i = 0; i < ahead; i++) src.weights(i, ps_tc_smem + (size_t)i * T::STAGE, ps_tc_fact + i * T::FACT, &bar_full[i]);
                __syncwarp();
            }
            ps_grid_dep();
            for (int q = q0; q < q1 && ok; q++) {
                const PsTcSrc<NT> src(a, q);
                for (int i = 0; i < ns; i++, g++, st.step(), sy.step()) {
                    // the MMAs of stage g - NS are complete: its operands have been read; entries three super-blocks before have been drained, and
                    // with them the factors of stage g - NS - 2
                    if (g >= T::NS && !ps_tc_wait_warp(&bar_empty[st.i], st.round ^ 1, a.limit)) { *a.err = 1; ok = false; break; }
                    uint8_t *sm = ps_tc_smem + (size_t)st.i * T::STAGE, *sf = ps_tc_fact + sy.i * T::FACT;
                    if (ps_elect_one()) {
                        if (g >= ahead) src.weights(i, sm, sf, &bar_full[st.i]);
                        src.columns(i, sm, sf, &bar_full[st.i]);
                    }
                    __syncwarp();
                }
            }
            // copies in flight end before the CTA does (they have, unless a wait gave up)
            for (int k = g > T::NS ? g - T::NS : 0; k < g; k++)
                if (!ps_tc_wait(&bar_full[k % T::NS], (k / T::NS) & 1)) { *a.err = 5; break; }
        } else if (warp == W_MMA) {
            ps_grid_dep_wait();
            // ===== MMA issuer.  The warp stays converged and one thread, chosen by elect.sync, issues, so that descriptors and barrier addresses
            // live in uniform registers
            // kind::f16, D = F32 (bit 4), A = B = F16, K-major both, N >> 3 @ bit 17, M >> 4 @ bit 24
            constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(PS_TC_M >> 4) << 24);
            const uint64_t desc0 = ps_tc_smem_desc(ps_smem_u32(ps_tc_smem + T::STAGE_B), NT * 16, 128);
            PsRing<T::NS> st;
            PsRing<T::NE> re;
            bool ok = warp != a.give_up;
            if (!ok) *a.err = 2;
            for (int q = q0; q < q1 && ok; q++) {
                const bool lanes = q % PS_TC_PASSES < 4;
                for (int i = 0; i < ns && ok; i++, st.step()) {
                    const uint64_t ds = desc0 + (uint64_t)(st.i * (T::STAGE >> 4));
#pragma unroll
                    for (int e = 0; e < 2 / T::XE; e++, re.step()) {
                        const uint32_t ta = tmem_base + T::TM_A + re.i * (T::XE * 32), td = tmem_base + re.i * T::TM_E;
                        // (the de-quantising warps have waited for the stage, B with it)
                        if (!ps_tc_wait_warp(&bar_go[re.i], re.round, a.limit)) { *a.err = 2; ok = false; break; }
                        ps_tc_fence_after();
                        if (ps_elect_one()) {
                            if (lanes) {
#pragma unroll
                                for (int k = 0; k < 2 * T::XE; k++) { // super-block k / 2 of the entry, chain k % 2
                                    const uint64_t dk = ds + (2 * T::XE * e + k) * (NT * 4);
                                    ps_tc_mma_f16_ta(td + k * NT, ta + k * 16, dk, idesc, 0);
                                    ps_tc_mma_f16_ta(td + k * NT, ta + k * 16 + 8, dk + NT * 2, idesc, 1);
                                }
                            } else {
#pragma unroll
                                for (int k = 0; k < 2 * T::XE; k++) ps_tc_mma_f16_ta(td + k * NT, ta + (k >> 1) * 32, ds + (2 * T::XE * e + k) * (NT * 2), idesc, 0);
                            }
                            ps_tc_commit(&bar_done[re.i]);
                            if (e == 2 / T::XE - 1) ps_tc_commit(&bar_empty[st.i]);
                        }
                        __syncwarp();
                    }
                }
            }
            if (ps_elect_one()) ps_tc_commit(&bar_end); // MMAs in flight end before the tensor memory is given back
            __syncwarp();
            if (!ps_tc_wait(&bar_end, 0)) *a.err = 6;
        }
    } else if (warp >= T::EW) {
        // ===== de-quantising warps: a warpgroup takes super-block d of a step, of every second step where there are four; thread = row (warp % 4 is its
        // tensor-memory lane quadrant)
        ps_reg_dec<T::R_DEQ>();
        ps_grid_dep_wait(); // (nothing here reads global memory: the limits of the waits below count from here)
        const int group = (warp - T::EW) >> 2, d = group & 1, quad = warp & 3, row = quad * 32 + lane;
        const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16) + T::TM_A + (T::XE == 2 ? d * 32 : 0);
        PsRing<T::NS> st;
        PsRing<T::NE> re;
        constexpr int EN = 2 / T::XE; // entries of a step
        if (T::XE == 1 && d) re.step();
        bool ok = warp != a.give_up;
        if (!ok) *a.err = 7;
        int g = 0, fresh = T::NE - (T::XE == 1 ? d : 0); // entries ahead whose A buffer has not been used
        for (int q = q0; q < q1 && ok; q++) {
            const bool lanes = q % PS_TC_PASSES < 4;
            for (int i = 0; i < ns; i++, g++) {
                const bool used = fresh <= 0;
                fresh -= used ? 0 : EN;
                if (T::ND == 4 && ((g ^ (group >> 1)) & 1)) { // the other two groups' step
                    st.step();
                    re.step();
                    continue;
                }
                // one wait for two things: even lanes wait for the stage, odd ones for the A buffer
                const bool fa = (lane & 1) && used;
                if (!ps_tc_wait_all(ps_smem_u32(fa ? &bar_done[re.i] : &bar_full[st.i]), fa ? re.round ^ 1 : st.round, a.limit)) { *a.err = 7; ok = false; break; }
                ps_tc_fence_after();
                const uint8_t *sm = ps_tc_smem + (size_t)st.i * T::STAGE;
                const uint32_t td = t_lane + re.i * (T::XE * 32);
                uint32_t v[4][8];
                if (lanes) {
                    sm += d * PS_TC_A_Q;
                    const uint4 w0 = *reinterpret_cast<const uint4 *>(sm + row * 16), w1 = *reinterpret_cast<const uint4 *>(sm + 2048 + row * 16);
                    const uint4 sc = *reinterpret_cast<const uint4 *>(sm + T::STAGE_SC - d * (PS_TC_A_Q - PS_TC_A_SC) + row * 16);
#pragma unroll
                    for (int k = 0; k < 2; k++) { // words 2k, 2k + 1 of both lanes
                        uint32_t s2[4], o2[4];
                        const uint32_t s0 = k ? sc.z : sc.x, s1 = k ? sc.w : sc.y;
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            s2[j] = __byte_perm(j < 2 ? s0 : s1, 0, (j & 1) ? 0x3232 : 0x1010);
                            o2[j] = ps_h2_mul(s2[j], 0xE400E400u); // x -1024
                        }
                        ps_tc_dequant8(k ? w0.z : w0.x, k ? w0.w : w0.y, s2, o2, v[k]);
                        ps_tc_dequant8(k ? w1.z : w1.x, k ? w1.w : w1.y, s2, o2, v[2 + k]);
                    }
                } else { // K positions 4k + u hold m_(2k + u / 2): column 2k + u / 2 is that minimum twice
                    const uint2 mn = *reinterpret_cast<const uint2 *>(sm + d * PS_TC_A_MN + row * 8);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const uint32_t w = __byte_perm(j < 4 ? mn.x : mn.y, 0x64646464u, 0x4040 + 0x0101 * (j & 3)); // 1024 + m, twice
                        v[0][j] = ps_h2_fma(w, 0x3C003C00u, 0xE400E400u);
                    }
                }
                ps_tc_st8(td, v[0]);
                if (lanes) {
                    ps_tc_st8(td + 8, v[1]);
                    ps_tc_st8(td + 16, v[2]);
                    ps_tc_st8(td + 24, v[3]);
                }
                ps_tc_st_wait();
                ps_tc_fence_before();
                __syncwarp();
                if (lane == 0) ps_mbar_arrive(&bar_go[re.i]);
                st.step();
                for (int k = 0; k < EN; k++) re.step();
            }
        }
    } else {
        // ===== epilogue: warp w owns tensor-memory lanes 32 * (w % 4) .. +31 (rows) and EC columns
        ps_reg_inc<T::R_EPI>();
        ps_grid_dep_wait();
        const int quad = warp & 3, row = quad * 32 + lane, c0 = (warp >> 2) * T::EC;
        const uint32_t t_lane = tmem_base + ((uint32_t)(quad * 32) << 16) + c0;
        constexpr int ET = T::EW * 32, US = T::EC * ET;
        float *stash = reinterpret_cast<float *>(ps_tc_fact + T::NY * T::FACT) + tid, *whole = stash + US; // [EC][epilogue threads]
        PsRing<T::NY> sy;
        PsRing<T::NE> re;
        bool ok = warp != a.give_up;
        if (!ok) *a.err = 4;
        int pend = -1, pend_slot = 0, old = 0; // the shared tile handed over last, its slot, and (thread 0) how many of its passes were there by then
        ps_f2 acc[2][T::EC / 2];
        for (int q = q0; q < q1; q++) {
            const int tile = q / PS_TC_PASSES, p = q % PS_TC_PASSES;
#pragma unroll
            for (int c = 0; c < T::EC / 2; c++) acc[0][c] = acc[1][c] = 0ull;
            for (int i = 0; i < ns && ok; i++, sy.step()) {
                const uint8_t *sf = ps_tc_fact + sy.i * T::FACT;
                // one wait a step: entries are complete in order
                const int e0 = re.i;
                if (T::XE == 1) re.step();
                const int e1 = re.i;
                if (!ps_tc_wait_warp(&bar_done[e1], re.round, a.limit)) { *a.err = 4; ok = false; break; }
                re.step();
                ps_tc_fence_after();
                const uint32_t td[2] = {t_lane + e0 * T::TM_E, t_lane + e1 * T::TM_E + (T::XE == 2 ? 2 * NT : 0)};
#pragma unroll
                for (int x = 0; x < 2; x++) {
                    // (the factors came with the stage, and stay until this warp has drained the entry)
                    const float xd = *reinterpret_cast<const float *>(sf + x * PS_TC_A_D + row * 4);
                    const ps_f2 x2 = ps_f2_pack(xd, xd);
#pragma unroll
                    for (int c = 0; c < T::EC; c += 8) {
                        uint32_t v0[8], v1[8];
                        ps_tc_ld(td[x] + c, v0);
                        ps_tc_ld(td[x] + NT + c, v1);
                        const ulonglong2 *yd = reinterpret_cast<const ulonglong2 *>(sf + 2 * PS_TC_A_D + (x * NT + c0 + c) * 4);
                        const ulonglong2 y0 = yd[0], y1 = yd[1];
                        const ps_f2 dd[4] = {ps_f2_mul(y0.x, x2), ps_f2_mul(y0.y, x2), ps_f2_mul(y1.x, x2), ps_f2_mul(y1.y, x2)};
                        ps_tc_ld_wait();
                        ps_tc_keep(v0);
                        ps_tc_keep(v1);
                        if ((x == 1 || T::XE == 1) && c + 8 == T::EC) { // the entry is in registers
                            ps_tc_fence_before();
                            __syncwarp();
                            if (lane == 0) ps_mbar_arrive(&bar_go[x ? e1 : e0]);
                        }
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            acc[0][c / 2 + k] = ps_f2_fma(dd[k], ps_f2_bits(v0[2 * k], v0[2 * k + 1]), acc[0][c / 2 + k]);
                            acc[1][c / 2 + k] = ps_f2_fma(dd[k], ps_f2_bits(v1[2 * k], v1[2 * k + 1]), acc[1][c / 2 + k]);
                        }
                    }
                }
            }
            // ---- the pass's number: first step of hsum_float_8 (lane l + 4 and lane l), or of the mins sum (m_k and m_k+2); then
            // ((r04 + r26) + (r15 + r37)) + (m02 + m13)
            const bool alone = q - p >= q0 && q - p + PS_TC_PASSES <= q1; // a tile of this CTA alone; of any other, pairs or single numbers are written down
            const bool end = p == PS_TC_PASSES - 1 || q + 1 == q1;       // the CTA's part of the tile ends
            const int slot = alone ? 0 : ps_tc_owner(q - p, gridDim.x, a.n_tiles);
            float *part = a.part + ((size_t)slot * PS_TC_PASSES + p) * US + tid;
            // (loops without branches inside: the code is met once a pass, and every line of it is fetched anew)
            auto each = [&](auto f) {
#pragma unroll
                for (int c = 0; c < T::EC / 2; c++) {
                    float r0, r1;
                    ps_f2_unpack(acc[0][c], r0, r1);
                    f(2 * c * ET, r0);
                    f((2 * c + 1) * ET, r1);
                    acc[0][c] = ps_f2_pack(r0, r1);
                }
            };
#pragma unroll
            for (int c = 0; c < T::EC / 2; c++) acc[0][c] = ps_f2_add(acc[1][c], acc[0][c]);
            if (!(p & 1)) each([&](int o, float &r) { stash[o] = r; });
            else if (q > q0) each([&](int o, float &r) { r = __fadd_rn(stash[o], r); });
            if (!alone) {
                if ((p & 1) || end) each([&](int o, float &r) { __stcg(part + o, r); });
            } else if (p & 1) {
                if (p > 1) each([&](int o, float &r) { r = __fadd_rn(whole[o], r); });
                if (!end) each([&](int o, float &r) { whole[o] = r; });
            }
            if (!end) continue;
            // ---- the CTA's part of the tile ends: a tile of its own is stored.  Of a shared one, thread 0 tells for all (its release is cumulative
            // over the barrier) and learns at the CTA's next part, or at its end, when the answer has long come, whether its part was the tile's
            // last; if so the CTA adds the tile's numbers
            bool met = true;
#pragma unroll 1
            for (int r = alone ? 0 : 1; r < 3; r++) {
                int t = tile;
                if (r == 0) {
                    r = 1; // nothing to tell
                    if (!ok) continue;
                } else {
                    if (r == 2 && (q + 1 < q1 || pend < 0)) break;
                    // a warp that gave up comes here too, and all of them leave: no warp waits at a barrier that another has passed by
                    met = false;
                    if (!ps_bar_all(1, ET, ok)) break;
                    met = true;
                    if (tid == 0) {
                        const int last = pend >= 0 && old == PS_TC_PASSES;
                        if (last) a.cnt[pend_slot] = 0;
                        sh_last = last;
                    }
                    ps_bar_sync(1, ET);
                    const bool last = sh_last;
                    t = pend;
                    const float *w = a.part + (size_t)pend_slot * PS_TC_PASSES * US + tid;
                    pend = r == 2 ? -1 : tile;
                    pend_slot = slot;
                    if (r == 1 && tid == 0) {
                        const int n = q + 1 - max(q0, q - p);
                        old = ps_add_acq_rel(a.cnt + slot, n) + n;
                    }
                    if (!last) continue;
                    const int b = t * PS_TC_PASSES;
                    const bool cut[3] = {ps_tc_cut(b + 1, gridDim.x, a.n_tiles), ps_tc_cut(b + 3, gridDim.x, a.n_tiles), ps_tc_cut(b + 5, gridDim.x, a.n_tiles)};
#pragma unroll
                    for (int cb = 0; cb < T::EC; cb += 8) { // the loads of eight columns together
                        float y[3][8], z[3][8];
#pragma unroll
                        for (int j = 0; j < 3; j++)
#pragma unroll
                            for (int k = 0; k < 8; k++) y[j][k] = __ldcg(w + (2 * j + 1) * US + (cb + k) * ET);
#pragma unroll
                        for (int j = 0; j < 3; j++)
                            if (cut[j])
#pragma unroll
                                for (int k = 0; k < 8; k++) z[j][k] = __ldcg(w + 2 * j * US + (cb + k) * ET);
#pragma unroll
                        for (int j = 0; j < 3; j++)
                            if (cut[j])
#pragma unroll
                                for (int k = 0; k < 8; k++) y[j][k] = __fadd_rn(z[j][k], y[j][k]);
#pragma unroll
                        for (int k = 0; k < 8; k += 2)
                            acc[0][(cb + k) / 2] = ps_f2_pack(__fadd_rn(__fadd_rn(y[0][k], y[1][k]), y[2][k]), __fadd_rn(__fadd_rn(y[0][k + 1], y[1][k + 1]), y[2][k + 1]));
                    }
                }
                // bias / residual, dst[col][row]
                const int rt = t / a.n_ct, ct = t % a.n_ct, grow = rt * PS_TC_M + row;
                int sg = 0;
                if (a.n_seg > 1 && grow >= a.seg[1].row_begin) sg = 1;
                if (a.n_seg > 2 && grow >= a.seg[2].row_begin) sg = 2;
                const int n_col = grow < a.seg[sg].row_end ? a.bs - (ct * NT + c0) : 0; // columns of this thread that exist
                const int n = grow - a.seg[sg].row_begin, ld = a.seg[sg].row_end - a.seg[sg].row_begin;
                const size_t o0 = (size_t)(ct * NT + c0) * ld + n;
                auto columns = [&](auto f) {
                    size_t o = o0;
#pragma unroll
                    for (int c = 0; c < T::EC / 2; c++) {
                        float r0, r1;
                        ps_f2_unpack(acc[0][c], r0, r1);
                        if (2 * c < n_col) f(o, r0);
                        if (2 * c + 1 < n_col) f(o + ld, r1);
                        acc[0][c] = ps_f2_pack(r0, r1);
                        o += 2 * (size_t)ld;
                    }
                };
                if (a.seg[sg].bias) {
                    const float bias = n_col > 0 ? a.seg[sg].bias[n] : 0.f;
                    columns([&](size_t, float &v) { v = __fadd_rn(v, bias); });
                }
                if (a.residual) columns([&](size_t o, float &v) { v = __fadd_rn(a.residual[o], v); });
                float *dst = a.seg[sg].dst;
                columns([&](size_t o, float &v) { dst[o] = v; });
            }
            if (!met) break;
        }
        ps_tc_ld_wait();
    }
    ps_tc_fence_before();
    __syncthreads();
    if (warp == W_MMA) {
        ps_tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(T::TM_COLS) : "memory");
    }
}
