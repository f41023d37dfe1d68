// ps_mk.cuh - batch products of the 256-element block formats (Q4_K, Q5_K, Q6_K weights x Q8_K activations) on GGUF rows as they lie in memory, with the
// integer sums on the tensor cores: what the operator table's matrix product, files of mixed formats and models without packed copies use from two or a
// few columns up (one column and narrower ones: ps_k_matmul_q, ps_k_matmul_qb).  Replaces powerserve_compute_forward_mul_mat ->
// ggml_vec_dot_q4_K_q8_K / q5_K / q6_K (libs/ggml/src/ggml.c:13344-13432, ggml-quants.c:7809-7872, 8382-8460, 9039-9116), bit for bit.
//
// Per super-block and AVX lane l the reference forms the INTEGER S_l = sum_j sc_j sum_t q[j][4l + t] q8[j][4l + t] and advances acc_l = fma(d, (float)S_l, acc_l).  The
// 32 products of a lane are the k of two mma.sync m16n8k16: the weights enter as halves sc_j q (at most 63 x 31, exact), Q6_K's (up to 128 x 32) as two, 16 (sc_j >> 4) q and
// (sc_j & 15) q, each exact, so four MMAs.  Every partial sum is an integer below 2^24, so fp32 holds it exactly in any order.  An MMA makes 128 sums in 8 cycles;
// dp4a with its scale took 32 cycles a warp for 32 of them.  The mins are one more MMA: their k is (chain, half of a sub-block), masked to one chain (Q4_K) or whole
// (Q5_K, whose reference adds all four first).
// A CTA of four warps takes 16 rows x 8 NT columns; warp w the lanes w and w + 4 (and mins chain w).  Thread (g, t) of a warp unpacks sub-blocks 2t and 2t + 1 of rows g
// and g + 8, for all columns at once; that, not the MMAs, is the larger part with few columns.  Super-blocks pass through a ring of stages: the
// rows' bytes by cp.async in 16-byte lines around them (rows of Q6_K begin at any even address), the columns' records by bulk copies.
// Measured (K x rows on columns, us a product, cold caches; dp4a before): Q6_K 4096 x 4096 on 32 44 -> 24, on 128 120 -> 62; Q4_K 4096 x 4096 on 32 36.5 -> 21, 8192 x 8192 on 128
// 403 -> 169; Q5_K 2048 x 8192 on 64 70 -> 31.  The operator's call on Q6_K 4096 x 4096, 32 columns: 24.9 -> 18.7 us, quantiser included.
#pragma once
#include "ps_tc.cuh"

// activation record of (8 columns, super-block): [8 lanes][8 columns][4 t] 16-byte pieces - (2t: elements 0, 2) (2t + 1: 0, 2) (2t: 1, 3) (2t + 1: 1, 3) as halves -
// then the columns' d, then [8 columns][4 t] the sums of the halves of sub-blocks 2t and 2t + 1
#define PS_MK_D 4096
#define PS_MK_HS 4128
#define PS_MK_REC 4384
PS_HD size_t ps_mk_x_bytes(int64_t K, int64_t cols) { return (size_t)((cols + 7) / 8) * (size_t)(K / 256) * PS_MK_REC; }
PS_D void ps_mk_store(uint8_t *__restrict__ dst, const float e[8], int lane, int64_t i, int64_t col, int64_t nb) {
    uint32_t words[2], bsp;
    float yd;
    ps_quant_block_q8k_regs(e, lane, words, yd, bsp);
    uint8_t *rec = dst + ((col >> 3) * nb + i) * PS_MK_REC;
    const int n = (int)(col & 7), g = lane >> 3, l = lane & 7, src = ((2 * g) & 3) * 8 + l;
    const uint32_t a0 = __shfl_sync(PS_FULL, words[0], src), a1 = __shfl_sync(PS_FULL, words[1], src);
    const uint32_t b0 = __shfl_sync(PS_FULL, words[0], src + 8), b1 = __shfl_sync(PS_FULL, words[1], src + 8);
    const uint32_t a = g < 2 ? a0 : a1, b = g < 2 ? b0 : b1; // words (2g, l) and (2g + 1, l)
    auto h2 = [](uint32_t w, int t0, int t1) {
        const __half2 h = __halves2half2(__int2half_rn((int)(signed char)(w >> (8 * t0))), __int2half_rn((int)(signed char)(w >> (8 * t1))));
        return *reinterpret_cast<const uint32_t *>(&h);
    };
    *reinterpret_cast<uint4 *>(rec + ((l * 8 + n) * 4 + g) * 16) = make_uint4(h2(a, 0, 2), h2(b, 0, 2), h2(a, 1, 3), h2(b, 1, 3));
    uint32_t hs[2]; // sub-blocks lane / 8 and 4 + lane / 8: (first half, second half)
#pragma unroll
    for (int h = 0; h < 2; h++) {
        int s = __dp4a((int)words[h], 0x01010101, 0);
        s += __shfl_xor_sync(PS_FULL, s, 1);
        s += __shfl_xor_sync(PS_FULL, s, 2);
        const int s0 = __shfl_sync(PS_FULL, s, lane & 24), s1 = __shfl_sync(PS_FULL, s, (lane & 24) + 4);
        const __half2 v = __halves2half2(__int2half_rn(s0), __int2half_rn(s1)); // |.| <= 2032: exact
        hs[h] = *reinterpret_cast<const uint32_t *>(&v);
    }
    const int at = (lane & 1) * 16;
    const uint32_t m0 = __shfl_sync(PS_FULL, hs[0], at), m1 = __shfl_sync(PS_FULL, hs[0], at + 8), m2 = __shfl_sync(PS_FULL, hs[1], at), m3 = __shfl_sync(PS_FULL, hs[1], at + 8);
    if (lane < 4) *reinterpret_cast<uint2 *>(rec + PS_MK_HS + (n * 4 + lane) * 8) = lane < 2 ? make_uint2(m0, m1) : make_uint2(m2, m3);
    if (lane == 0) reinterpret_cast<float *>(rec + PS_MK_D)[n] = yd;
}
__global__ void __launch_bounds__(128) ps_k_mk_quantize(const float *__restrict__ x, const float *__restrict__ u, int64_t K, uint8_t *__restrict__ dst) {
    ps_grid_dep();
    const int lane = threadIdx.x & 31;
    const int64_t nb = K / 256, i = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5), col = blockIdx.y, at = col * K + i * 256;
    if (i >= nb) return;
    float e[8];
    ps_act8(x + at, u ? u + at : nullptr, lane, e);
    ps_mk_store(dst, e, lane, i, col, nb);
}
__global__ void __launch_bounds__(512) ps_k_mk_norm_quantize(const float *__restrict__ x, const float *__restrict__ w, int64_t dim, float eps, uint8_t *__restrict__ dst) {
    ps_grid_dep();
    __shared__ double sh[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t col = blockIdx.x, nb = dim / 256;
    const float *xr = x + col * dim;
    const float scale = ps_rms_scale(xr, dim, eps, sh);
    for (int64_t i = warp; i < nb; i += 16) {
        const int64_t at = i * 256 + 4 * lane;
        const float4 a = ps_norm4(xr + at, w + at, scale), b = ps_norm4(xr + at + 128, w + at + 128, scale);
        const float e[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        ps_mk_store(dst, e, lane, i, col, nb);
    }
}

struct PsMkArgs {
    PsMbSeg seg[3];     // w: GGUF rows; cta0: row tiles before the segment
    int n_seg, bs, nb, ns; // super-blocks of a row; stages of the ring
    const uint8_t *x;   // activation records
    const float *residual;
    int *err;
};
#define PS_MK_MAX_NS 8
// a row's bytes of one super-block and the 16-byte lines around them; rows lie PITCH apart (an odd number of lines, which spreads them over the banks)
template <int TYPE> PS_HD constexpr int ps_mk_lines() { return TYPE == 14 ? 15 : PsBlk<TYPE>::BYTES / 16; }
template <int TYPE> PS_HD constexpr int ps_mk_pitch() { return (ps_mk_lines<TYPE>() | 1) * 16; }
template <int TYPE, int NT> PS_HD constexpr int ps_mk_stage() { return 16 * ps_mk_pitch<TYPE>() + NT * PS_MK_REC; }
PS_D void ps_mk_mma(float (&s)[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(s[0]), "+f"(s[1]), "+f"(s[2]), "+f"(s[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
PS_D uint32_t ps_h2_add(uint32_t a, uint32_t b) { uint32_t r; asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
// (byte 2i + 0 of `bytes`, twice) as a half2 of the number
PS_D uint32_t ps_mk_byte2(uint32_t bytes, int i) { return ps_h2_add(__byte_perm(bytes, 0x64646464u, 0x4040 | i << 8 | i), 0xE400E400u); }
PS_D uint32_t ps_mk_word(const uint8_t *p, int odd) { // four bytes at an even address; odd: 0, or 16 where it is no multiple of four
    const uint32_t *q = reinterpret_cast<const uint32_t *>(p - (odd >> 3));
    return odd ? __funnelshift_r(q[0], q[1], 16) : q[0];
}

template <int TYPE, int NT>
__global__ void __launch_bounds__(128) ps_k_matmul_mk(const PsMkArgs a) {
    using B = PsBlk<TYPE>;
    constexpr int LINES = ps_mk_lines<TYPE>(), PITCH = ps_mk_pitch<TYPE>(), STAGE = ps_mk_stage<TYPE, NT>(), X0 = 16 * PITCH;
    extern __shared__ __align__(128) uint8_t ps_mk_smem[];
    __shared__ __align__(8) uint64_t bar[PS_MK_MAX_NS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gr = lane >> 2, t = lane & 3;
    const int nb = a.nb, ns = a.ns, n_ct = (a.bs + 7) / 8, ct0 = blockIdx.y * NT;
    const int sg = a.n_seg > 2 && (int)blockIdx.x >= a.seg[2].cta0 ? 2 : a.n_seg > 1 && (int)blockIdx.x >= a.seg[1].cta0 ? 1 : 0;
    const PsMbSeg &seg = a.seg[sg];
    const int row0 = ((int)blockIdx.x - seg.cta0) * 16;
    const int64_t row_bytes = (int64_t)nb * B::BYTES;
    if (tid == 0) {
        for (int s = 0; s < ns; s++) ps_mbar_init(&bar[s], 1);
        ps_fence_barrier_init();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    // a thread's lines of a stage (rows past the end: the last row again; a line past the row's last byte is not read)
    auto rows = [&](int i, int slot) {
        uint8_t *st = ps_mk_smem + (size_t)slot * STAGE;
        for (int c = tid; c < 16 * LINES; c += 128) {
            const int r = c / LINES, k = c - r * LINES;
            const uint8_t *src = seg.w + (int64_t)min(row0 + r, seg.n - 1) * row_bytes + (int64_t)i * B::BYTES;
            const uint8_t *line = reinterpret_cast<const uint8_t *>((uintptr_t)src & ~(uintptr_t)15) + 16 * k;
            if (TYPE != 14 || line < src + B::BYTES) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ps_smem_u32(st + r * PITCH + 16 * k)), "l"(line) : "memory");
        }
    };
    auto columns = [&](int i, int slot) { // one thread
        ps_mbar_expect_tx(&bar[slot], NT * PS_MK_REC);
#pragma unroll
        for (int j = 0; j < NT; j++) // (past the last tile: that one again)
            ps_bulk_g2s(ps_mk_smem + (size_t)slot * STAGE + X0 + j * PS_MK_REC, a.x + ((size_t)min(ct0 + j, n_ct - 1) * nb + i) * PS_MK_REC, PS_MK_REC, &bar[slot]);
    };
    for (int i = 0; i < ns - 1; i++) { // weights do not depend on the kernel before
        if (i < nb) rows(i, i);
        ps_cp_async_commit();
    }
    ps_grid_dep();
    __syncthreads(); // the barriers are there
    if (tid == 0)
        for (int i = 0; i < min(ns - 1, nb); i++) columns(i, i);
    ps_f2 acc[2][2][NT]; // [lane w, w + 4][row g, g + 8][column tile]: columns 2t, 2t + 1
    float accm[B::HAS_MIN ? NT : 1][4];
#pragma unroll
    for (int j = 0; j < NT; j++) {
        acc[0][0][j] = acc[0][1][j] = acc[1][0][j] = acc[1][1][j] = 0ull;
        if (B::HAS_MIN) accm[j][0] = accm[j][1] = accm[j][2] = accm[j][3] = 0.f;
    }
    int slot = 0;
    uint32_t phase = 0;
    const uint32_t mine = B::MIN_SCALAR || t == warp ? 0xFFFFFFFFu : 0u; // the mins chain's part of k
    for (int i = 0; i < nb; i++) {
        switch (ns) { // (groups still in flight: a constant of the instruction)
        case 2: ps_cp_async_wait<0>(); break;
        case 3: ps_cp_async_wait<1>(); break;
        case 4: ps_cp_async_wait<2>(); break;
        default: ps_cp_async_wait<3>(); break; // (ns 5 and more: some wait longer than they must)
        }
        // after a wait that gave up the results are invalid; the loop goes on and waits for the other copies, each within its limit
        if (!ps_tc_wait(&bar[slot], phase, PS_COPY_POLLS)) *a.err = PS_ERR_COPY;
        __syncthreads(); // everyone's lines have arrived, and everyone has read the slot before
        {
            const int nx = i + ns - 1, sl = slot == 0 ? ns - 1 : slot - 1;
            if (nx < nb) {
                rows(nx, sl);
                if (tid == 0) columns(nx, sl);
            }
            ps_cp_async_commit();
        }
        const uint8_t *st = ps_mk_smem + (size_t)slot * STAGE, *sx = st + X0;
        // ---- the weights of rows g and g + 8: halves av[lane][MMA][register], d, dmin, mins
        constexpr int NM = TYPE == 14 ? 4 : 2;
        uint32_t av[2][NM][4], mv[2][2];
        float xd[2], xm[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            if constexpr (TYPE == 14) {
                const int off = (int)((uintptr_t)(seg.w + (int64_t)min(row0 + gr + 8 * r, seg.n - 1) * row_bytes + (int64_t)i * B::BYTES) & 15);
                const uint8_t *blk = st + (gr + 8 * r) * PITCH + off;
                const int odd = (off & 2) << 3;
                const uint32_t sc = ps_mk_word(blk + 192 + 4 * t, odd); // of sub-blocks 2t, 2t + 1, first and second half
                xd[r] = ps_half_bits_to_float(*reinterpret_cast<const unsigned short *>(blk + 208));
#pragma unroll
                for (int h = 0; h < 2; h++) { // AVX lanes w, w + 4
                    const int l = warp + 4 * h;
                    const uint32_t l0 = ps_mk_word(blk + 64 * (t >> 1) + 4 * l, odd) >> (4 * (t & 1)), l1 = ps_mk_word(blk + 64 * (t >> 1) + 32 + 4 * l, odd) >> (4 * (t & 1));
                    const uint32_t qh = ps_mk_word(blk + 128 + 32 * (t >> 1) + 4 * l, odd) >> (4 * (t & 1));
#pragma unroll
                    for (int z = 0; z < 2; z++) { // sub-block 2t + z
                        const uint32_t lw = z ? l1 : l0, hw = z ? qh >> 2 : qh;
                        const int s = (int)(signed char)(sc >> (16 * z + 8 * h));
                        // 16 (s >> 4) and s & 15 as halves, twice: 1024 + 128 + 16 (s >> 4) - 1152
                        const uint32_t s_hi = ps_h2_add((uint32_t)(((s >> 4) * 16 + 128) * 0x00010001) | 0x64006400u, 0xE480E480u);
                        const uint32_t s_lo = ps_h2_add((uint32_t)((s & 15) * 0x00010001) | 0x64006400u, 0xE400E400u);
#pragma unroll
                        for (int p = 0; p < 2; p++) { // elements (0, 2), (1, 3)
                            const uint32_t q = ps_h2_add(((lw >> (8 * p)) & 0x000F000Fu) | (((hw >> (8 * p)) & 0x00030003u) << 4) | 0x64006400u, 0xE420E420u); // - 1056
                            av[h][p][2 * z + r] = ps_h2_mul(q, s_hi);
                            av[h][2 + p][2 * z + r] = ps_h2_mul(q, s_lo);
                        }
                    }
                }
            } else {
                const uint8_t *blk = st + (gr + 8 * r) * PITCH;
                const uint4 hd = *reinterpret_cast<const uint4 *>(blk);
                xd[r] = ps_half_bits_to_float(hd.x & 0xffffu);
                xm[r] = ps_half_bits_to_float(hd.x >> 16);
                // get_scale_min_k4 of sub-blocks 2t, 2t + 1 (ggml-quants.c:7816-7826)
                const uint32_t scw = t < 2 ? hd.y & 0x3f3f3f3fu : (hd.w & 0x0f0f0f0fu) | (((hd.y >> 6) & 0x03030303u) << 4);
                const uint32_t mnw = t < 2 ? hd.z & 0x3f3f3f3fu : ((hd.w >> 4) & 0x0f0f0f0fu) | (((hd.z >> 6) & 0x03030303u) << 4);
                const uint32_t sc = scw >> (16 * (t & 1)), mn = mnw >> (16 * (t & 1));
                const uint32_t s[2] = {ps_mk_byte2(sc, 0), ps_mk_byte2(sc, 1)};
                mv[r][0] = ps_mk_byte2(mn, 0);
                mv[r][1] = ps_mk_byte2(mn, 1);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int l = warp + 4 * h;
                    const uint32_t w = *reinterpret_cast<const uint32_t *>(blk + (TYPE == 13 ? 48 : 16) + 32 * t + 4 * l);
                    const uint32_t hi = TYPE == 13 ? *reinterpret_cast<const uint32_t *>(blk + 16 + 4 * l) >> (2 * t) : 0u; // bit 0 of a byte: sub-block 2t, bit 1: 2t + 1
#pragma unroll
                    for (int z = 0; z < 2; z++) {
                        const uint32_t o = ps_h2_mul(s[z], 0xE400E400u); // - 1024 sc
#pragma unroll
                        for (int p = 0; p < 2; p++) {
                            uint32_t q = ((w >> (8 * p + 4 * z)) & 0x000F000Fu) | 0x64006400u;
                            if (TYPE == 13) q |= ((hi >> (8 * p + z)) & 0x00010001u) << 4;
                            av[h][p][2 * z + r] = ps_h2_fma(q, s[z], o); // (1024 + q) sc - 1024 sc: exact
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < NT; j++) {
            const uint8_t *rec = sx + j * PS_MK_REC;
            const float2 yd = *reinterpret_cast<const float2 *>(rec + PS_MK_D + 8 * t);
            const ps_f2 y2 = ps_f2_pack(yd.x, yd.y);
            const ps_f2 d[2] = {ps_f2_mul(y2, ps_f2_pack(xd[0], xd[0])), ps_f2_mul(y2, ps_f2_pack(xd[1], xd[1]))};
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint4 b = *reinterpret_cast<const uint4 *>(rec + ((warp + 4 * h) * 32 + lane) * 16);
                float s[4] = {0.f, 0.f, 0.f, 0.f};
                ps_mk_mma(s, av[h][0], b.x, b.y);
                ps_mk_mma(s, av[h][1], b.z, b.w);
                if (TYPE == 14) {
                    ps_mk_mma(s, av[h][NM - 2], b.x, b.y);
                    ps_mk_mma(s, av[h][NM - 1], b.z, b.w);
                }
                acc[h][0][j] = ps_f2_fma(d[0], ps_f2_pack(s[0], s[1]), acc[h][0][j]);
                acc[h][1][j] = ps_f2_fma(d[1], ps_f2_pack(s[2], s[3]), acc[h][1][j]);
            }
            if (B::HAS_MIN && (!B::MIN_SCALAR || warp == 0)) {
                const uint2 hs = *reinterpret_cast<const uint2 *>(rec + PS_MK_HS + lane * 8);
                const uint32_t am[4] = {mv[0][0], mv[1][0], mv[0][1], mv[1][1]};
                float p[4] = {0.f, 0.f, 0.f, 0.f};
                ps_mk_mma(p, am, hs.x & mine, hs.y & mine);
                const float ym[2] = {-yd.x, -yd.y};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float dm = __fmul_rn(ym[e & 1], xm[e >> 1]);
                    accm[j][e] = B::MIN_SCALAR ? __fadd_rn(accm[j][e], __fmul_rn(dm, p[e])) : __fmaf_rn(dm, p[e], accm[j][e]);
                }
            }
        }
        if (++slot == ns) { slot = 0; phase ^= 1; }
    }
    // hsum_float_8: (x4 + x0, x5 + x1, x6 + x2, x7 + x3) -> (r0 + r2) + (r1 + r3), then the mins: (m0 + m2) + (m1 + m3), or the one sum
    __syncthreads();
    float *red = reinterpret_cast<float *>(ps_mk_smem), *redm = red + 4 * 8 * NT * 16; // [4 w][8 NT columns][16 rows]
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
        for (int r = 0; r < 2; r++) {
            float u, v;
            ps_f2_unpack(ps_f2_add(acc[1][r][j], acc[0][r][j]), u, v);
            const int at = (warp * 8 * NT + 8 * j + 2 * t) * 16 + 8 * r + gr;
            red[at] = u;
            red[at + 16] = v;
            if (B::HAS_MIN) {
                redm[at] = accm[j][2 * r];
                redm[at + 16] = accm[j][2 * r + 1];
            }
        }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NT; k++) {
        const int e = k * 128 + tid, c = 8 * ct0 + (e >> 4), n = row0 + (e & 15);
        float r = __fadd_rn(__fadd_rn(red[e], red[256 * NT + e]), __fadd_rn(red[128 * NT + e], red[384 * NT + e]));
        if (B::MIN_SCALAR) r = __fadd_rn(r, redm[e]);
        else if (B::HAS_MIN) r = __fadd_rn(r, __fadd_rn(__fadd_rn(redm[e], redm[256 * NT + e]), __fadd_rn(redm[128 * NT + e], redm[384 * NT + e])));
        if (c < a.bs && n < seg.n) {
            const int64_t o = (int64_t)c * seg.n + n;
            if (seg.bias) r = __fadd_rn(r, seg.bias[n]);
            if (a.residual) r = __fadd_rn(a.residual[o], r);
            seg.dst[o] = r;
        }
    }
}
