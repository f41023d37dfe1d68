// ps_arch_tc.cuh - tcgen05 GEMM for the layer-list executor's bfloat16 products: C[token][n] = sum_k X[token][k] W[n][k].
//
// The WEIGHT rows are the MMA's M side (128 output features per unit), the tokens its N side (128 per unit), so one
// accumulator column is one token (a grid with few units cuts the token tiles into parts of 64, 32 or 16) and an epilogue warp's 32 tensor-memory lanes are 32 consecutive output features: the
// stores of a column are coalesced.  Both operands reach shared memory as ready-made canonical K-major no-swizzle blocks
// ([k-chunk of 8][row][8 elements], 16 KB per 128 rows x 64 k) through ONE 1-D bulk copy each:
//   * weights are re-tiled once at bind time (pa_k_tc_tile_w), per expert for the routed feed-forward;
//   * activations are rounded to bfloat16 and tiled per call (pa_k_tc_prep_x), gathered and scaled per routed row.
// Roles per CTA (persistent over units): 4 epilogue warps, one producer lane, one MMA-issuing lane; 6 (4 for the fused
// gate|up pair) stages of 64 k; two accumulator buffers in tensor memory so the epilogue of unit i overlaps the MMAs of
// unit i + 1.  Every wait is bounded: a pipeline that loses step reports through the context's error flag.
#pragma once
#include "ps_ptx.cuh"

#define PT_M 128
#define PT_N 128
#define PT_KB 64
#define PT_BLOCK (128 * PT_KB * 2) // bytes of one operand block (either side)
#define PT_THREADS 192
#define PT_MAX_SEG 6 // operand sets of one product
#define PT_SMEM (192 * 1024 + 1024 + 2 * 16 * PT_M * 4) // stages, alignment, sixteen columns' sums and table entries

// ---------------------------------------------------------------------------------------------------- operand builders
// weights [groups][N][K] bf16 row-major -> blocks [group][row tile][k block][k-chunk 8][row 128][8]; zero outside N x K
// odd (or null): set if a weight is an infinity or no number
__global__ void __launch_bounds__(256) pa_k_tc_tile_w(uint8_t *__restrict__ dst, const bf16 *__restrict__ w, int N, int K, int n_rt, int nkb, int *__restrict__ odd) {
    const int kb = blockIdx.y, rt = blockIdx.x, grp = blockIdx.z; // (y ends at 65 535)
    const bf16 *src = w + (int64_t)grp * N * K;
    uint8_t *out = dst + (((int64_t)grp * n_rt + rt) * nkb + kb) * PT_BLOCK;
    for (int c = threadIdx.x; c < 128 * 8; c += 256) {
        const int kc = c & 7, row = c >> 3, n = rt * 128 + row, k0 = kb * PT_KB + kc * 8;
        uint16_t v[8];
#pragma unroll
        for (int t = 0; t < 8; t++) v[t] = (n < N && k0 + t < K) ? reinterpret_cast<const uint16_t *>(src)[(int64_t)n * K + k0 + t] : (uint16_t)0;
        if (odd) {
            bool any = false;
#pragma unroll
            for (int t = 0; t < 8; t++) any |= (v[t] & 0x7F80) == 0x7F80;
            if (any) *odd = 1;
        }
        uint4 pk;
        pk.x = v[0] | ((uint32_t)v[1] << 16); pk.y = v[2] | ((uint32_t)v[3] << 16); pk.z = v[4] | ((uint32_t)v[5] << 16); pk.w = v[6] | ((uint32_t)v[7] << 16);
        *reinterpret_cast<uint4 *>(out + kc * 2048 + row * 16) = pk;
    }
}

// activations fp32 -> bf16 blocks [column tile][k block][k-chunk][token 128][8].  Dense: tile t holds rows t * 128 ..;
// routed: tile t holds rows tile_row0[t] .. tile_end[t] of the row list (token gathered through row_token, scaled by row_w).
__global__ void __launch_bounds__(256) pa_k_tc_prep_x(uint8_t *__restrict__ dst, const float *__restrict__ x, int ldx, int M, int K, int nkb, const int *__restrict__ n_tiles,
                                                      const int *__restrict__ tile_row0, const int *__restrict__ tile_end, const int *__restrict__ row_token,
                                                      const float *__restrict__ row_w) {
    ps_grid_dep();
    const int kb = blockIdx.x, t = blockIdx.y;
    if (n_tiles && t >= *n_tiles) return;
    const int r0 = tile_row0 ? tile_row0[t] : t * 128, rend = tile_end ? tile_end[t] : M;
    uint8_t *out = dst + ((int64_t)t * nkb + kb) * PT_BLOCK;
    for (int c = threadIdx.x; c < 128 * 8; c += 256) {
        const int kc = c & 7, row = c >> 3, r = r0 + row, k0 = kb * PT_KB + kc * 8;
        uint16_t v[8];
        if (r < rend) {
            const float *src = x + (int64_t)(row_token ? row_token[r] : r) * ldx;
            const float sc = row_w ? row_w[r] : 1.0f;
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = (k0 + e < K) ? __bfloat16_as_ushort(__float2bfloat16_rn(src[k0 + e] * sc)) : (uint16_t)0;
        } else {
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = 0;
        }
        uint4 pk;
        pk.x = v[0] | ((uint32_t)v[1] << 16); pk.y = v[2] | ((uint32_t)v[3] << 16); pk.z = v[4] | ((uint32_t)v[5] << 16); pk.w = v[6] | ((uint32_t)v[7] << 16);
        *reinterpret_cast<uint4 *>(out + kc * 2048 + row * 16) = pk;
    }
}

// the operand sets of a segmented product: set 0 = x, set s = x + (x' - x) mu[s - 1] with x' the row of the token before (the batch's first
// token: row (pos - 1) & 1 of `ring`, zeros at position 0).  Grid (k blocks, column tiles, 4): a CTA takes 32 rows, a thread eight entries of all sets; set s starts s * set_bytes further on.
__global__ void __launch_bounds__(256) pa_k_tc_prep_shift(uint8_t *__restrict__ dst, const float *__restrict__ x, int M, int K, int nkb, const float *__restrict__ mu,
                                                          const float *__restrict__ ring, const int32_t *__restrict__ pos, int64_t set_bytes) {
    ps_grid_dep();
    const int kb = blockIdx.x, t = blockIdx.y, p0 = pos[0];
    const int kc = threadIdx.x & 7, row = blockIdx.z * 32 + (threadIdx.x >> 3), r = t * 128 + row, k0 = kb * PT_KB + kc * 8;
    uint8_t *out = dst + ((int64_t)t * nkb + kb) * PT_BLOCK + kc * 2048 + row * 16;
    const float *src = x + (int64_t)r * K, *prev = r > 0 ? src - K : ring + (int64_t)((p0 - 1) & 1) * K;
    const bool first = r == 0 && p0 == 0;
    float h[8], d[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const bool in = r < M && k0 + e < K;
        h[e] = in ? src[k0 + e] : 0.f;
        d[e] = in ? (first ? 0.f : prev[k0 + e]) - h[e] : 0.f;
    }
#pragma unroll
    for (int set = 0; set < PT_MAX_SEG; set++) {
        uint16_t v[8];
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = __bfloat16_as_ushort(__float2bfloat16_rn(set && k0 + e < K ? fmaf(d[e], mu[(int64_t)(set - 1) * K + k0 + e], h[e]) : h[e]));
        uint4 pk;
        pk.x = v[0] | ((uint32_t)v[1] << 16); pk.y = v[2] | ((uint32_t)v[3] << 16); pk.z = v[4] | ((uint32_t)v[5] << 16); pk.w = v[6] | ((uint32_t)v[7] << 16);
        *reinterpret_cast<uint4 *>(out + set * set_bytes) = pk;
    }
}

// ---------------------------------------------------------------------------------------------------- the GEMM
// A product whose output rows read different operand sets (activations that are mixtures of the same input): row tiles rt[s] .. rt[s + 1] - 1
// hold the rows row[s] .. row[s + 1] - 1 of the output and read set s.  n = 0: one set, all rows.
struct PtSegs {
    int n;
    int rt[PT_MAX_SEG + 1], row[PT_MAX_SEG + 1];
    int64_t set_bytes;
};
enum { PT_MODE_DENSE = 0, PT_MODE_EXPERT_UP = 1, PT_MODE_EXPERT_DOWN = 2 };

struct PtArgs {
    const uint8_t *a0, *a1; // weight blocks [group][row tiles][k blocks]; a1 = the second matrix of a fused pair (gate | up)
    const uint8_t *b;       // activation blocks [column tiles][k blocks]
    int nkb, n_rt, n_ct;    // n_ct: column tiles (an upper bound when n_ct_dev is given)
    int n_sub;              // dense: a column tile is cut into n_sub equal parts (0: one), n_ct counts the parts - more, narrower units for a grid that would not fill the GPU
    const int *n_ct_dev;
    const int *tile_e, *tile_row0, *tile_end; // routed: group, first row and end row of every column tile
    int M, N;               // dense: token rows; N: output features
    int mode;
    float *C;
    int ldc;
    const float *bias;
    const int *row_token, *row_slot;
    const float *row_w;
    int top, on_input;
    PaAct act;
    int act1;               // dense / expert up: the one-argument activation on the outputs n >= act_from (a feed-forward without a gate),
    int act_from, gap;      // which are stored `gap` columns further on
    PaRowMul mul;           // dense: the outputs times a table row per token
    PtSegs seg;
    int *err;
};

template <int NA>
__global__ void __launch_bounds__(PT_THREADS, 1) pa_k_tc_gemm(const __grid_constant__ PtArgs a) {
    constexpr int STAGES = NA == 1 ? 6 : 4;
    constexpr int STAGE_BYTES = (NA + 1) * PT_BLOCK;
    extern __shared__ __align__(1024) uint8_t pt_smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[STAGES], bar_empty[STAGES], bar_tmem_full[2], bar_tmem_empty[2], bar_done;
    __shared__ uint32_t tmem_base_smem;
    uint8_t *smem = reinterpret_cast<uint8_t *>(((uintptr_t)pt_smem_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int nkb = a.nkb;
    const int n_sub = max(a.n_sub, 1), tn = PT_N / n_sub; // tokens of a unit

    if (tid == 0) {
        for (int s = 0; s < STAGES; s++) { ps_mbar_init(&bar_full[s], 1); ps_mbar_init(&bar_empty[s], 1); }
        for (int b = 0; b < 2; b++) { ps_mbar_init(&bar_tmem_full[b], 1); ps_mbar_init(&bar_tmem_empty[b], 4); }
        ps_mbar_init(&bar_done, 1);
        ps_fence_barrier_init();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(ps_smem_u32(&tmem_base_smem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    ps_tc_fence_before();
    __syncthreads();
    ps_tc_fence_after();
    const uint32_t tmem_base = tmem_base_smem;
    // a dense product's first weights do not depend on the kernel before: they are asked for while it still runs
    int ahead = 0;
    if (warp == 4 && !a.n_ct_dev && !a.tile_e && (int)blockIdx.x < a.n_ct * a.n_rt) {
        ahead = min(STAGES, nkb);
        if (ps_elect_one()) {
            const int64_t b0 = (int64_t)((int)blockIdx.x % a.n_rt) * nkb * PT_BLOCK;
            for (int kb = 0; kb < ahead; kb++) {
                ps_mbar_expect_tx(&bar_full[kb], NA * PT_BLOCK + PT_BLOCK / n_sub);
                ps_bulk_g2s(smem + (size_t)kb * STAGE_BYTES, a.a0 + b0 + (int64_t)kb * PT_BLOCK, PT_BLOCK, &bar_full[kb]);
                if (NA == 2) ps_bulk_g2s(smem + (size_t)kb * STAGE_BYTES + PT_BLOCK, a.a1 + b0 + (int64_t)kb * PT_BLOCK, PT_BLOCK, &bar_full[kb]);
            }
        }
        __syncwarp();
    }
    ps_grid_dep();
    const int n_ct = a.n_ct_dev ? min(*a.n_ct_dev, a.n_ct) : a.n_ct;
    const int n_units = n_ct * a.n_rt;
    const int my_units = (n_units > (int)blockIdx.x) ? (n_units - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

    if (warp == 4) {
        // ===== producer: one bulk copy per operand block.  Producer and issuer stay converged warps and act through one elected thread: under
        // `lane == 0` descriptors and addresses go through vector registers and an MMA took 280 cycles to issue (128 x 128 x 16 itself: 64)
        PsRing<STAGES> st;
        int g = 0;
        bool ok = true;
        for (int mu = 0; mu < my_units && ok; mu++) {
            const int u = (int)blockIdx.x + mu * (int)gridDim.x, ct = u / a.n_rt, rt = u % a.n_rt;
            const int64_t grp = a.tile_e ? a.tile_e[ct] : 0;
            const uint8_t *pa0 = a.a0 + ((grp * a.n_rt + rt) * nkb) * (int64_t)PT_BLOCK;
            const uint8_t *pa1 = NA == 2 ? a.a1 + ((grp * a.n_rt + rt) * nkb) * (int64_t)PT_BLOCK : nullptr;
            const uint8_t *pb = a.b + ((int64_t)(ct / n_sub) * nkb) * PT_BLOCK + (ct % n_sub) * tn * 16;
            for (int sg = 1; sg < a.seg.n; sg++)
                if (rt >= a.seg.rt[sg]) pb += a.seg.set_bytes;
            for (int kb = 0; kb < nkb; kb++, g++, st.step()) {
                if (g >= STAGES && !ps_tc_wait_warp(&bar_empty[st.i], st.round ^ 1)) { *a.err = 1; ok = false; break; }
                uint8_t *sm = smem + (size_t)st.i * STAGE_BYTES;
                uint64_t *bar = &bar_full[st.i];
                if (ps_elect_one()) {
                    if (g >= ahead) {
                        ps_mbar_expect_tx(bar, NA * PT_BLOCK + PT_BLOCK / n_sub);
                        ps_bulk_g2s(sm, pa0, PT_BLOCK, bar);
                        if (NA == 2) ps_bulk_g2s(sm + PT_BLOCK, pa1, PT_BLOCK, bar);
                    }
                    if (n_sub == 1) ps_bulk_g2s(sm + NA * PT_BLOCK, pb, PT_BLOCK, bar);
                    else // the part's tokens of every k-chunk, at the places they have in the whole tile
#pragma unroll
                        for (int c = 0; c < 8; c++) ps_bulk_g2s(sm + NA * PT_BLOCK + c * 2048, pb + c * 2048, (uint32_t)(tn * 16), bar);
                }
                __syncwarp();
                pa0 += PT_BLOCK;
                pa1 += PT_BLOCK;
                pb += PT_BLOCK;
            }
        }
        for (int k = g > STAGES ? g - STAGES : 0; k < g; k++) // copies in flight end before the CTA does (they have, unless a wait gave up)
            if (!ps_tc_wait(&bar_full[k % STAGES], (k / STAGES) & 1)) { *a.err = 5; break; }
    } else if (warp == 5) {
        // ===== MMA issuer: kind::f16 with bfloat16 operands (a_format = b_format = 1), fp32 accumulators, K-major both
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(tn >> 3) << 17) | ((uint32_t)(PT_M >> 4) << 24);
        const uint64_t desc0 = ps_tc_smem_desc(ps_smem_u32(smem), 2048, 128);
        PsRing<STAGES> st;
        bool ok = true;
        for (int mu = 0; mu < my_units && ok; mu++) {
            const int tb = mu & 1;
            if (mu >= 2 && !ps_tc_wait_warp(&bar_tmem_empty[tb], ((mu >> 1) - 1) & 1)) { *a.err = 3; break; }
            const uint32_t td = tmem_base + tb * (NA * PT_N);
            for (int kb = 0; kb < nkb; kb++, st.step()) {
                if (!ps_tc_wait_warp(&bar_full[st.i], st.round)) { *a.err = 2; ok = false; break; }
                ps_tc_fence_after();
                const uint64_t da = desc0 + (uint64_t)(st.i * (STAGE_BYTES >> 4));
                if (ps_elect_one()) {
#pragma unroll
                    for (int j = 0; j < PT_KB / 16; j++) {
                        ps_tc_mma_f16(td, da + j * 256, da + NA * (PT_BLOCK >> 4) + j * 256, idesc, (kb | j) != 0);
                        if (NA == 2) ps_tc_mma_f16(td + PT_N, da + (PT_BLOCK >> 4) + j * 256, da + NA * (PT_BLOCK >> 4) + j * 256, idesc, (kb | j) != 0);
                    }
                    ps_tc_commit(&bar_empty[st.i]);
                    if (kb == nkb - 1) ps_tc_commit(&bar_tmem_full[tb]);
                }
                __syncwarp();
            }
        }
        if (ps_elect_one()) ps_tc_commit(&bar_done); // MMAs in flight end before the tensor memory is given back
        __syncwarp();
        if (!ps_tc_wait(&bar_done, 0)) *a.err = 6;
    } else {
        // ===== epilogue: warp w reads tensor-memory lanes 32 w .. 32 w + 31 = 32 consecutive output features
        for (int mu = 0; mu < my_units; mu++) {
            const int u = (int)blockIdx.x + mu * (int)gridDim.x, ct = u / a.n_rt, rt = u % a.n_rt, tb = mu & 1;
            if (!ps_tc_wait_warp(&bar_tmem_full[tb], (mu >> 1) & 1)) { *a.err = 4; break; }
            ps_tc_fence_after();
            int n = rt * PT_M + 32 * warp + lane, n_end = a.N;
            for (int sg = 0; sg < a.seg.n; sg++) // the segment's own rows
                if (rt >= a.seg.rt[sg] && rt < a.seg.rt[sg + 1]) { n += a.seg.row[sg] - a.seg.rt[sg] * PT_M; n_end = a.seg.row[sg + 1]; break; }
            const int r0 = a.tile_row0 ? a.tile_row0[ct] : ct * tn, rend = a.tile_end ? a.tile_end[ct] : a.M;
            const uint32_t t_lane = tmem_base + ((uint32_t)(32 * warp) << 16) + tb * (NA * PT_N);
            const float bias = (a.bias && n < n_end) ? a.bias[n] : 0.f;
            const int n_cols = min(tn, rend - r0); // warp-uniform
            for (int c0 = 0; c0 < n_cols; c0 += 16) {
                uint32_t v[16], w2[16];
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                               "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                             : "r"(t_lane + c0)
                             : "memory");
                if (NA == 2)
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                                 : "=r"(w2[0]), "=r"(w2[1]), "=r"(w2[2]), "=r"(w2[3]), "=r"(w2[4]), "=r"(w2[5]), "=r"(w2[6]), "=r"(w2[7]), "=r"(w2[8]), "=r"(w2[9]),
                                   "=r"(w2[10]), "=r"(w2[11]), "=r"(w2[12]), "=r"(w2[13]), "=r"(w2[14]), "=r"(w2[15])
                                 : "r"(t_lane + PT_N + c0)
                                 : "memory");
                float mulv[16]; // the table rows' entries: sixteen independent loads beside the tensor-memory loads
                if (NA == 1 && a.mul.table) {
#pragma unroll
                    for (int c = 0; c < 16; c++) mulv[c] = pa_ld(a.mul.table + (int64_t)a.mul.tok[min(r0 + c0 + c, rend - 1)] * a.mul.ld + min(n, n_end - 1));
                }
                ps_tc_ld_wait();
                // the branches of mode and activation lie outside the sixteen copies: a unit's stores are met once, instructions that have to be fetched (with them
                // inside, a product of 32 units took 22 us, 15 so; 256 tokens of Nufusun at 768 350 and 320)
                const int left = n_cols - c0;
                float *to = a.C + (int64_t)(r0 + c0) * a.ldc + n;
                auto each = [&](auto f) {
#pragma unroll
                    for (int c = 0; c < 16; c++)
                        if (c < left && n < n_end) to[(int64_t)c * a.ldc] = f(c);
                };
                auto sum = [&](int c) { return __uint_as_float(v[c]); };
                if (a.mode == PT_MODE_EXPERT_DOWN) {
                    const int r = min(r0 + c0 + (lane & 15), rend - 1);
                    const int64_t mine = ((int64_t)a.row_token[r] * a.top + a.row_slot[r]) * a.ldc;
                    const float rw = a.on_input ? 1.f : a.row_w[r];
#pragma unroll
                    for (int c = 0; c < 16; c++) {
                        const int64_t o = __shfl_sync(0xffffffffu, mine, c);
                        const float f = __shfl_sync(0xffffffffu, rw, c);
                        if (c < left && n < n_end) a.C[o + n] = sum(c) * f;
                    }
                } else if (NA == 2) {
                    PaAct act = a.act;
                    auto gated = [&](int kind) {
                        act.kind = kind;
                        each([&](int c) { return pa_expert_act(sum(c), __uint_as_float(w2[c]), act); });
                    };
                    if (act.kind == PS_ACT_RELU) gated(PS_ACT_RELU);
                    else if (act.kind == PS_ACT_GELU_TANH) gated(PS_ACT_GELU_TANH);
                    else gated(PS_ACT_SWISH);
                } else if (a.mode == PT_MODE_DENSE && !a.mul.table && !(a.act1 && n - lane + 31 >= a.act_from)) {
                    each([&](int c) { return sum(c) + bias; });
                } else { // one-argument activations, table rows: one copy, the sums by way of shared memory
                    float *red = reinterpret_cast<float *>(smem + STAGES * STAGE_BYTES) + 32 * warp + lane;
#pragma unroll
                    for (int c = 0; c < 16; c++) {
                        red[c * PT_M] = sum(c);
                        if (NA == 1 && a.mul.table) red[(16 + c) * PT_M] = mulv[c];
                    }
                    const bool act1 = a.mode == PT_MODE_EXPERT_UP || (a.act1 && n >= a.act_from);
                    if (a.mode == PT_MODE_DENSE && act1) to += a.gap;
                    if (n < n_end)
#pragma unroll 2
                        for (int c = 0; c < min(left, 16); c++) {
                            float val = a.mode == PT_MODE_DENSE ? red[c * PT_M] + bias : red[c * PT_M];
                            if (act1) val = pa_act1(val, a.act);
                            if (NA == 1 && a.mul.table) val *= red[(16 + c) * PT_M];
                            to[(int64_t)c * a.ldc] = val;
                        }
                }
            }
            ps_tc_fence_before();
            __syncwarp();
            if (lane == 0) ps_mbar_arrive(&bar_tmem_empty[tb]);
        }
    }
    ps_tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        ps_tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    }
}

// ---------------------------------------------------------------------------------------------------- float32 mode
// The same products without rounding.  The weights are bfloat16 as they are; an activation is cut into three bfloat16 parts, its upper, middle and lower
// eight significant bits (no part overflows; exact from 2^-103 up, below which a part may be subnormal and at worst 2^-126 is lost), so that three MMAs whose products are exact
// replace the FMAs.  What an MMA loses is the low end of the fp32 accumulator (it truncates where an FMA rounds), and that grows with the number of MMAs an accumulator sees and
// with its size.  So an accumulator takes ONE k block of 64 - lowest parts first, while it is small, the four MMAs of the upper parts last - and the epilogue adds the blocks' sums
// in fp32 with rounding.  The order of k is the same for every number of tokens and every portion.
// Error against 64 bits, root mean square over the result's: logits of two 1024-wide Vanapel layers 8e-7 with FMA tiles, 5.8e-7 so (150 tokens at 300); one product of K 512 / 2048 / 8192 with
// weights of both signs, activations of one sign or two, over a binade or ten: 2.1 / 3.0 / 5.8e-7 and 1.2 / 1.6 / 2.4e-7.  Truncation has a direction: where all products of a sum share a sign it
// does not average out.  Over one binade that is not seen (K 2048 1.1e-7 and 1.0e-7), over ten the sums are 1.1e-7 short: 1.0 / 1.0 / 1.8e-7 with FMAs, 1.2 / 1.4 / 2.0e-7 so.  Bound: the four upper MMAs
// of a block lose less than an ulp of 1/4 to 4/4 of its sum, together 2.5 * 2^-23.
// Bound by the epilogue, which drains an accumulator of TN tokens every 12 MMAs (24 with a gate), and by the copies: a stage of 64 k is 16 KB of weights a
// matrix and 384 B a token.  A unit is 128 output rows x TN tokens, TN as small as fills the GPU: its epilogue is shorter and the weights come from L2.
// 150 tokens, us with the cutting of the activations: K 1024 x 1024 outputs 12 + 4, K 2048 x 1024 20 + 4, gate | up of 2048 from K 1024 21 + 4, head of 4096 from K 1024 15 + 5 (a pass of two
// layers 606 -> 370)
#define PT_SPLIT 3
template <int TN> PS_HD constexpr int pt_xb() { return PT_SPLIT * TN * PT_KB * 2; } // bytes of a tile's k block: [part][k-chunk of 8][token TN][8]
// activations -> [column tile][k block][part][k-chunk][token][8]; tiles as in pa_k_tc_prep_x
__global__ void __launch_bounds__(256) pa_k_tc_prep_split(uint8_t *__restrict__ dst, const float *__restrict__ x, int ldx, int M, int K, int nkb, int TN, const int *__restrict__ n_tiles,
                                                          const int *__restrict__ tile_row0, const int *__restrict__ tile_end, const int *__restrict__ row_token, const float *__restrict__ row_w) {
    ps_grid_dep();
    const int kb = blockIdx.x, t = blockIdx.y;
    if (n_tiles && t >= *n_tiles) return;
    const int r0 = tile_row0 ? tile_row0[t] : t * TN, rend = tile_end ? tile_end[t] : M;
    uint8_t *out = dst + ((int64_t)t * nkb + kb) * (PT_SPLIT * TN * PT_KB * 2);
    for (int c = threadIdx.x; c < TN * 8; c += 256) {
        const int kc = c & 7, row = c >> 3, r = r0 + row, k0 = kb * PT_KB + kc * 8;
        const bool in = r < rend;
        const float *src = x + (int64_t)(in && row_token ? row_token[r] : in ? r : 0) * ldx;
        const float sc = in && row_w ? row_w[r] : 1.0f;
        uint32_t part[PT_SPLIT][4] = {};
#pragma unroll
        for (int e = 0; e < 8; e++) {
            float v = in && k0 + e < K ? src[k0 + e] * sc : 0.f;
            const bool odd = !(fabsf(v) < INFINITY);
            if (v != v) v = __uint_as_float(0x7FC00000u); // (a NaN's low bits alone would read as an infinity)
#pragma unroll
            for (int q = 0; q < PT_SPLIT; q++) {
                const uint32_t hi = __float_as_uint(v) & 0xFFFF0000u;
                part[q][e >> 1] |= (e & 1) ? hi : hi >> 16;
                v = odd ? 0.f : v - __uint_as_float(hi);
            }
        }
#pragma unroll
        for (int q = 0; q < PT_SPLIT; q++) *reinterpret_cast<uint4 *>(out + (q * 8 + kc) * (TN * 16) + row * 16) = make_uint4(part[q][0], part[q][1], part[q][2], part[q][3]);
    }
}

// a tile's sums wait in shared memory for a store loop of one copy: unrolled over its registers, with the modes' and activations' branches in every copy, a tile of 64
// tokens took longer to store than to multiply (instructions that are fetched once)
template <int NA, int TN> struct Pt3 {
    static constexpr int STAGE = NA * PT_BLOCK + pt_xb<TN>(), RED = NA * TN * PT_M * 4, FIT = (224 * 1024 - RED) / STAGE, STAGES = FIT < 8 ? FIT : 8, SMEM = STAGES * STAGE + RED + 1024;
};
template <int NA, int TN>
__global__ void __launch_bounds__(PT_THREADS, 1) pa_k_tc_gemm3(const __grid_constant__ PtArgs a) {
    constexpr int XB = pt_xb<TN>(), STAGE = Pt3<NA, TN>::STAGE, STAGES = Pt3<NA, TN>::STAGES;
    constexpr int TM = 2 * NA * TN < 32 ? 32 : 2 * NA * TN; // tensor-memory columns: two accumulator buffers
    extern __shared__ __align__(1024) uint8_t pt_smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[STAGES], bar_empty[STAGES], bar_tmem_full[2], bar_tmem_empty[2], bar_done;
    __shared__ uint32_t tmem_base_smem;
    uint8_t *smem = reinterpret_cast<uint8_t *>(((uintptr_t)pt_smem_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int nkb = a.nkb;
    if (tid == 0) {
        for (int s = 0; s < STAGES; s++) { ps_mbar_init(&bar_full[s], 1); ps_mbar_init(&bar_empty[s], 1); }
        for (int b = 0; b < 2; b++) { ps_mbar_init(&bar_tmem_full[b], 1); ps_mbar_init(&bar_tmem_empty[b], 4); }
        ps_mbar_init(&bar_done, 1);
        ps_fence_barrier_init();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ps_smem_u32(&tmem_base_smem)), "n"(TM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    ps_tc_fence_before();
    __syncthreads();
    ps_tc_fence_after();
    const uint32_t tmem_base = tmem_base_smem;
    int ahead = 0; // (as in pa_k_tc_gemm)
    if (warp == 4 && !a.n_ct_dev && !a.tile_e && (int)blockIdx.x < a.n_ct * a.n_rt) {
        ahead = min(STAGES, nkb);
        if (ps_elect_one()) {
            const int64_t b0 = (int64_t)((int)blockIdx.x % a.n_rt) * nkb * PT_BLOCK;
            for (int kb = 0; kb < ahead; kb++) {
                ps_mbar_expect_tx(&bar_full[kb], STAGE);
                ps_bulk_g2s(smem + (size_t)kb * STAGE, a.a0 + b0 + (int64_t)kb * PT_BLOCK, PT_BLOCK, &bar_full[kb]);
                if (NA == 2) ps_bulk_g2s(smem + (size_t)kb * STAGE + PT_BLOCK, a.a1 + b0 + (int64_t)kb * PT_BLOCK, PT_BLOCK, &bar_full[kb]);
            }
        }
        __syncwarp();
    }
    ps_grid_dep();
    const int n_ct = a.n_ct_dev ? min(*a.n_ct_dev, a.n_ct) : a.n_ct, n_units = n_ct * a.n_rt;

    if (warp == 4) {
        PsRing<STAGES> st;
        int g = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < n_units && ok; u += gridDim.x) {
            const int ct = u / a.n_rt, rt = u % a.n_rt;
            const int64_t grp = a.tile_e ? a.tile_e[ct] : 0;
            const uint8_t *pa0 = a.a0 + ((grp * a.n_rt + rt) * nkb) * (int64_t)PT_BLOCK, *pa1 = NA == 2 ? a.a1 + ((grp * a.n_rt + rt) * nkb) * (int64_t)PT_BLOCK : nullptr;
            const uint8_t *pb = a.b + (int64_t)ct * nkb * XB;
            for (int kb = 0; kb < nkb; kb++, g++, st.step()) {
                if (g >= STAGES && !ps_tc_wait_warp(&bar_empty[st.i], st.round ^ 1)) { *a.err = 1; ok = false; break; }
                uint8_t *sm = smem + (size_t)st.i * STAGE;
                uint64_t *bar = &bar_full[st.i];
                if (ps_elect_one()) {
                    if (g >= ahead) {
                        ps_mbar_expect_tx(bar, STAGE);
                        ps_bulk_g2s(sm, pa0 + (int64_t)kb * PT_BLOCK, PT_BLOCK, bar);
                        if (NA == 2) ps_bulk_g2s(sm + PT_BLOCK, pa1 + (int64_t)kb * PT_BLOCK, PT_BLOCK, bar);
                    }
                    ps_bulk_g2s(sm + NA * PT_BLOCK, pb + (int64_t)kb * XB, XB, bar);
                }
                __syncwarp();
            }
        }
        for (int k = g > STAGES ? g - STAGES : 0; k < g; k++) // copies in flight end before the CTA does (they have, unless a wait gave up)
            if (!ps_tc_wait(&bar_full[k % STAGES], (k / STAGES) & 1)) { *a.err = 5; break; }
    } else if (warp == 5) {
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(PT_M >> 4) << 24);
        const uint64_t desc_a = ps_tc_smem_desc(ps_smem_u32(smem), 2048, 128), desc_b = ps_tc_smem_desc(ps_smem_u32(smem + NA * PT_BLOCK), TN * 16, 128);
        PsRing<STAGES> st;
        bool ok = true;
        int m = 0;
        for (int u = blockIdx.x; u < n_units && ok; u += gridDim.x)
            for (int kb = 0; kb < nkb; kb++, m++, st.step()) {
                const int tb = m & 1;
                if (!ps_tc_wait_warp(&bar_full[st.i], st.round)) { *a.err = 2; ok = false; break; }
                if (m >= 2 && !ps_tc_wait_warp(&bar_tmem_empty[tb], ((m >> 1) - 1) & 1)) { *a.err = 3; ok = false; break; }
                ps_tc_fence_after();
                const uint64_t da = desc_a + (uint64_t)(st.i * (STAGE >> 4)), db = desc_b + (uint64_t)(st.i * (STAGE >> 4));
                const uint32_t td = tmem_base + tb * (NA * TN);
                if (ps_elect_one()) {
#pragma unroll
                    for (int q = PT_SPLIT - 1; q >= 0; q--) // lowest parts first
#pragma unroll
                        for (int j = 0; j < PT_KB / 16; j++) {
                            const uint64_t dq = db + (q * 8 + 2 * j) * TN;
                            ps_tc_mma_f16(td, da + j * 256, dq, idesc, q != PT_SPLIT - 1 || j != 0);
                            if (NA == 2) ps_tc_mma_f16(td + TN, da + (PT_BLOCK >> 4) + j * 256, dq, idesc, q != PT_SPLIT - 1 || j != 0);
                        }
                    ps_tc_commit(&bar_empty[st.i]);
                    ps_tc_commit(&bar_tmem_full[tb]);
                }
                __syncwarp();
            }
        if (ps_elect_one()) ps_tc_commit(&bar_done); // MMAs in flight end before the tensor memory is given back
        __syncwarp();
        if (!ps_tc_wait(&bar_done, 0)) *a.err = 6;
    } else {
        bool ok = true;
        int m = 0;
        for (int u = blockIdx.x; u < n_units && ok; u += gridDim.x) {
            const int ct = u / a.n_rt, rt = u % a.n_rt;
            float acc[NA][TN];
#pragma unroll
            for (int c = 0; c < TN; c++) acc[0][c] = acc[NA - 1][c] = 0.f;
            for (int kb = 0; kb < nkb; kb++, m++) {
                const int tb = m & 1;
                if (!ps_tc_wait_warp(&bar_tmem_full[tb], (m >> 1) & 1)) { *a.err = 4; ok = false; break; }
                ps_tc_fence_after();
                const uint32_t t_lane = tmem_base + ((uint32_t)(32 * warp) << 16) + tb * (NA * TN);
#pragma unroll
                for (int z = 0; z < NA; z++)
#pragma unroll
                    for (int c0 = 0; c0 < TN; c0 += 16) {
                        uint32_t v[16];
                        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                                       "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                                     : "r"(t_lane + z * TN + c0)
                                     : "memory");
                        ps_tc_ld_wait();
#pragma unroll
                        for (int c = 0; c < 16; c++) {
                            asm volatile("" : "+r"(v[c])); // (nothing reads it before the wait)
                            acc[z][c0 + c] += __uint_as_float(v[c]);
                        }
                    }
                ps_tc_fence_before();
                __syncwarp();
                if (lane == 0) ps_mbar_arrive(&bar_tmem_empty[tb]);
            }
            if (!ok) break;
            const int n = rt * PT_M + 32 * warp + lane, r0 = a.tile_row0 ? a.tile_row0[ct] : ct * TN, rend = a.tile_end ? a.tile_end[ct] : a.M;
            const float bias = a.bias && n < a.N ? a.bias[n] : 0.f;
            float *red = reinterpret_cast<float *>(smem + STAGES * STAGE) + 32 * warp + lane; // (a thread's own)
#pragma unroll
            for (int c = 0; c < TN; c++) {
                red[c * PT_M] = acc[0][c];
                if (NA == 2) red[(TN + c) * PT_M] = acc[1][c];
            }
            const int n_cols = min(TN, rend - r0); // warp-uniform
            if (a.mode == PT_MODE_EXPERT_DOWN) {
                int64_t to[(TN + 31) / 32]; // lane: rows lane and lane + 32 of the tile
                float rw[(TN + 31) / 32];
#pragma unroll
                for (int h = 0; h < (TN + 31) / 32; h++) {
                    const int r = min(r0 + 32 * h + lane, rend - 1);
                    to[h] = ((int64_t)a.row_token[r] * a.top + a.row_slot[r]) * a.ldc;
                    rw[h] = a.on_input ? 1.f : a.row_w[r];
                }
                for (int c = 0; c < n_cols; c++) {
                    const int64_t o = __shfl_sync(0xffffffffu, TN > 32 && c >= 32 ? to[(TN - 1) / 32] : to[0], c & 31);
                    const float rwc = __shfl_sync(0xffffffffu, TN > 32 && c >= 32 ? rw[(TN - 1) / 32] : rw[0], c & 31);
                    if (n < a.N) a.C[o + n] = red[c * PT_M] * rwc;
                }
            } else if (n < a.N) {
                const bool act1 = a.mode == PT_MODE_EXPERT_UP || (a.act1 && n >= a.act_from);
                float *to = a.C + (int64_t)r0 * a.ldc + (a.mode == PT_MODE_DENSE && act1 ? n + a.gap : n);
                if (NA == 2) {
                    for (int c = 0; c < n_cols; c++) to[(int64_t)c * a.ldc] = pa_expert_act(red[c * PT_M], red[(TN + c) * PT_M], a.act);
                } else if (act1) {
                    for (int c = 0; c < n_cols; c++) {
                        float v = pa_act1(red[c * PT_M] + bias, a.act);
                        if (a.mul.table) v *= pa_ld(a.mul.table + (int64_t)a.mul.tok[r0 + c] * a.mul.ld + n);
                        to[(int64_t)c * a.ldc] = v;
                    }
                } else {
                    for (int c = 0; c < n_cols; c++) {
                        float v = red[c * PT_M] + bias;
                        if (a.mul.table) v *= pa_ld(a.mul.table + (int64_t)a.mul.tok[r0 + c] * a.mul.ld + n);
                        to[(int64_t)c * a.ldc] = v;
                    }
                }
            }
            __syncwarp();
        }
    }
    ps_tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        ps_tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TM) : "memory");
    }
}
