// ps_mv32.cuh — fused decode mat-vec for the 32-element block formats (Q4_0, Q8_0 weights x Q8_0 activations):
// the counterpart of the Q4_K row-walker (ps_rw.cuh) for the models BASELINE configs[0] names (Qwen2-0.5B Q4_0) and for
// Q8_0 files.  Replaces powerserve_compute_forward_mul_mat -> ggml_vec_dot_q4_0_q8_0 / ggml_vec_dot_q8_0_q8_0
// (libs/ggml/src/ggml.c:13344-13432, ggml-quants.c:4205-4228, 5761-5782) with quantize_row_q8_0 (ggml-quants.c:957-1017),
// RMSNorm (ggml.c:12667-12721) or SiLU.up (src/backend/ggml/ggml.cpp:115-129) fused into the prologue and bias /
// residual / greedy-pick partials into the epilogue.
//
// Arithmetic (bit-exact, the same chains as PsBlk<2> / PsBlk<8> in ps_kernels.cuh): per row the reference keeps one
// __m256 accumulator; lane l of block b adds fl(d_x * d_y) * float(sum of the four int8 products 4l..4l+3) with ONE FMA,
// blocks in row order; hsum_float_8 at the end.  Four threads own a row (thread t = AVX lanes t and t + 4: for Q4_0 both
// come out of the same 32-bit word of nibbles, low nibbles = lane t, high nibbles = lane t + 4), a warp owns an octet of
// rows and walks the row's blocks in order.
//
// Weights are repacked once at bind time into an OCTET layout: [octet][block][8 rows x QB quant bytes | 8 x fp16 d]
// (144 B for Q4_0, 272 B for Q8_0 - a permutation of the GGUF bytes), so that a warp's stream is contiguous, every
// pipeline stage is one TMA bulk copy into the warp's private shared-memory ring and every warp-wide shared-memory load
// is conflict free.  Rings are filled BEFORE the dependency wait (weights never depend on the previous kernel).
#pragma once
#include "ps_decode.cuh"

#define PS_MV_WARPS 8
#define PS_MV_THREADS 256
#define PS_MV_MAX_NS 4
#define PS_MV_STAGE_CAP 6144

template <int TYPE> struct PsMv32;
template <> struct PsMv32<2> { static constexpr int QB = 16, BLK = 144, SRC = 18; };
template <> struct PsMv32<8> { static constexpr int QB = 32, BLK = 272, SRC = 34; };

// GGUF rows of 18- / 34-byte blocks -> octet layout (rows of a partial last octet stay zero: the buffer is cleared first)
template <int TYPE>
__global__ void ps_k_mv32_repack(uint8_t *__restrict__ dst, const uint8_t *__restrict__ w, int64_t n_rows, int64_t nb, int64_t oct0) {
    using G = PsMv32<TYPE>;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_rows * nb; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = t / nb, b = t % nb;
        const uint8_t *src = w + (row * nb + b) * G::SRC;
        uint8_t *o = dst + ((oct0 + row / 8) * nb + b) * G::BLK;
        const int r = (int)(row % 8);
        for (int k = 0; k < G::QB; k++) o[r * G::QB + k] = src[2 + k];
        o[8 * G::QB + 2 * r] = src[0];
        o[8 * G::QB + 2 * r + 1] = src[1];
    }
}

struct PsMvSeg {
    float *dst;            // [rows of the segment]
    const float *bias;     // optional
    int row_begin, row_end;
};
enum { PS_MV_PRO_PLAIN = 0, PS_MV_PRO_RMSNORM = 1, PS_MV_PRO_SILU = 2 };
struct PsMvArgs {
    const uint8_t *w;      // [n_oct][nb][BLK]
    int n_oct, K, sb, ns;  // sb = blocks per ring stage (divides nb), ns = ring stages per warp
    int kpar;              // block-parallel mode (one octet per CTA, long rows): slice capacity in bytes per warp, 0 = off
    const float *x;        // activation vector (PRO_SILU: the gate vector)
    const float *x2;       // PRO_SILU: the up vector
    const float *norm_w;   // PRO_RMSNORM
    float eps;
    double inv_k;
    int pro;
    PsMvSeg seg[3];        // q | k | v, gate | up, or a single matrix
    int n_seg;
    const float *residual; // optional, indexed like seg[0].dst (single-segment launches)
    float *part_val;       // optional greedy-pick partials, one per CTA
    int *part_idx;
};

// quantize_row_q8_0, AVX2 branch, for the four 32-blocks a warp holds (lane = 8 b + l owns elements 4l..4l+3 of block b):
// returns the packed word and d = fp16(max|x| / 127) widened back
PS_D void ps_mv_quant4(const float4 v, uint32_t &word, float &d_out) {
    float amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(PS_FULL, amax, o));
    const float d = __fdiv_rn(amax, 127.f);
    const float id = (amax != 0.0f) ? __fdiv_rn(127.f, amax) : 0.0f;
    const int q0 = __float2int_rn(__fmul_rn(v.x, id)), q1 = __float2int_rn(__fmul_rn(v.y, id));
    const int q2 = __float2int_rn(__fmul_rn(v.z, id)), q3 = __float2int_rn(__fmul_rn(v.w, id));
    word = (uint32_t)(q0 & 0xff) | ((uint32_t)(q1 & 0xff) << 8) | ((uint32_t)(q2 & 0xff) << 16) | ((uint32_t)(q3 & 0xff) << 24);
    d_out = __half2float(__float2half_rn(d));
}

// prologue of every launch: (RMSNorm | SiLU.up) + quantize_row_q8_0 of the activation vector into shared memory (all eight warps;
// ends with a CTA barrier)
PS_D void ps_mv_prologue(const PsMvArgs &a, uint32_t *s_qs, float *s_d, double *sh_red, int K, int nb, int tid, int warp, int lane) {
    float nscale = 1.f;
    if (a.pro == PS_MV_PRO_RMSNORM) {
        double ss = 0.0;
        for (int e = tid * 4; e < K; e += PS_MV_THREADS * 4) {
            const float4 v = *reinterpret_cast<const float4 *>(a.x + e);
            ss += (double)__fmul_rn(v.x, v.x);
            ss += (double)__fmul_rn(v.y, v.y);
            ss += (double)__fmul_rn(v.z, v.z);
            ss += (double)__fmul_rn(v.w, v.w);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(PS_FULL, ss, o);
        if (lane == 0) sh_red[warp] = ss;
        __syncthreads();
        double tot = 0.0;
#pragma unroll
        for (int w = 0; w < PS_MV_WARPS; w++) tot += sh_red[w];
        const float mean = (float)(a.inv_k != 0.0 ? tot * a.inv_k : tot / (double)K);
        nscale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, a.eps)));
    }
    for (int i0 = warp * 4; i0 < nb; i0 += PS_MV_WARPS * 4) { // four blocks per warp pass
        const int i = i0 + (lane >> 3), l = lane & 7;
        const bool valid = i < nb;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (valid) {
            v = *reinterpret_cast<const float4 *>(a.x + i * 32 + 4 * l);
            if (a.pro == PS_MV_PRO_RMSNORM) {
                const float4 wv = *reinterpret_cast<const float4 *>(a.norm_w + i * 32 + 4 * l);
                v.x = __fmul_rn(v.x, __fmul_rn(wv.x, nscale)); // y = x * (w * scale)
                v.y = __fmul_rn(v.y, __fmul_rn(wv.y, nscale));
                v.z = __fmul_rn(v.z, __fmul_rn(wv.z, nscale));
                v.w = __fmul_rn(v.w, __fmul_rn(wv.w, nscale));
            } else if (a.pro == PS_MV_PRO_SILU) {
                const float4 u = *reinterpret_cast<const float4 *>(a.x2 + i * 32 + 4 * l);
                v.x = ps_silu_mul(v.x, u.x);
                v.y = ps_silu_mul(v.y, u.y);
                v.z = ps_silu_mul(v.z, u.z);
                v.w = ps_silu_mul(v.w, u.w);
            }
        }
        uint32_t word;
        float d;
        ps_mv_quant4(v, word, d);
        if (valid) {
            s_qs[i * 8 + l] = word;
            if (l == 0) s_d[i] = d;
        }
    }
    __syncthreads();

}

// epilogue of one octet: hsum_float_8 across the row's four threads, bias / residual, store, running arg-max
PS_D void ps_mv_epilogue(const PsMvArgs &a, int oct, int r, int t, float a_lo, float a_hi, float &best_v, int &best_i) {
    // hsum_float_8 (ggml-quants.c:62-68): (x4 + x0, x5 + x1, x6 + x2, x7 + x3) -> (r0 + r2) + (r1 + r3)
    float res = __fadd_rn(a_hi, a_lo);
    res = __fadd_rn(res, __shfl_xor_sync(PS_FULL, res, 2));
    res = __fadd_rn(res, __shfl_xor_sync(PS_FULL, res, 1));
    const int row = oct * 8 + r;
    int sg = 0;
    if (a.n_seg > 1 && row >= a.seg[1].row_begin) sg = 1;
    if (a.n_seg > 2 && row >= a.seg[2].row_begin) sg = 2;
    if (t == 0 && row < a.seg[sg].row_end) {
        const int n = row - a.seg[sg].row_begin;
        if (a.seg[sg].bias) res = __fadd_rn(res, a.seg[sg].bias[n]);
        if (a.residual) res = __fadd_rn(a.residual[n], res);
        a.seg[sg].dst[n] = res;
        if (res > best_v || (res == best_v && n < best_i)) { best_v = res; best_i = n; } // first maximum wins
    }
}

// Dynamic shared memory: [s_qs: K bytes][s_d: nb floats, padded to 128][rings: 8 warps x ns x stage_bytes][bars: 8 x ns x 8]
//
// Block-parallel mode (a.kpar > 0; matrices with at most one octet per CTA and long rows, e.g. Qwen2's down projection:
// 112 octets of 152 blocks): a lone warp would walk the whole row serially, so the row's blocks are dealt to the CTA's eight
// warps instead.  Each warp streams its slice with one bulk copy, does the INTEGER work of its blocks and leaves, per block and
// lane, the three numbers the chains need - fl(d_x d_y), float(S_lo), float(S_hi), all exact - in shared memory; after one CTA
// barrier warp 0 advances the two FMA chains over all blocks IN ROW ORDER (the arithmetic of the one-warp walk) and runs
// the epilogue.  Shared memory: [s_qs][s_d][slices: 8 x kpar bytes][factors: nb x 3 x 32 floats][bars: 8 x 8].
template <int TYPE>
__global__ void __launch_bounds__(PS_MV_THREADS) ps_k_mv32(const PsMvArgs a) {
    using G = PsMv32<TYPE>;
    extern __shared__ __align__(128) uint8_t ps_mv_smem[];
    __shared__ double sh_red[PS_MV_WARPS];
    __shared__ float sv[PS_MV_WARPS];
    __shared__ int si[PS_MV_WARPS];
    const int K = a.K, nb = K / 32, sb = a.sb, ns = a.ns;
    const uint32_t stage_bytes = (uint32_t)sb * G::BLK;
    uint32_t *s_qs = reinterpret_cast<uint32_t *>(ps_mv_smem);
    float *s_d = reinterpret_cast<float *>(ps_mv_smem + K);
    uint8_t *s_ring = ps_mv_smem + (((size_t)K + (size_t)nb * 4 + 127) & ~(size_t)127);
    uint64_t *s_bar = reinterpret_cast<uint64_t *>(s_ring + (size_t)PS_MV_WARPS * ns * stage_bytes);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, t = lane & 3;
    const int o0 = (int)(((long long)blockIdx.x * a.n_oct) / gridDim.x), o1 = (int)(((long long)(blockIdx.x + 1) * a.n_oct) / gridDim.x);
    const int spo = nb / sb; // stages per octet
    const int n_mine = (o0 + warp < o1) ? (o1 - o0 - warp - 1) / PS_MV_WARPS + 1 : 0;
    const int n_stages = n_mine * spo;
    if (a.kpar) { // ---- block-parallel mode (see above)
        uint8_t *slice = s_ring + (size_t)warp * a.kpar;
        float *s_fac = reinterpret_cast<float *>(s_ring + (size_t)PS_MV_WARPS * a.kpar);
        uint64_t *bar = reinterpret_cast<uint64_t *>(s_fac + (size_t)nb * 96) + warp;
        const bool own = o0 < o1;                                       // CTAs beyond the octet count only take part in the dependency chain
        const int b_lo = nb * warp / PS_MV_WARPS, b_hi = nb * (warp + 1) / PS_MV_WARPS;
        if (lane == 0) {
            ps_mbar_init(bar, 1);
            ps_fence_barrier_init();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            if (own && b_hi > b_lo) {
                const uint32_t bytes = (uint32_t)(b_hi - b_lo) * G::BLK;
                ps_mbar_expect_tx(bar, bytes);
                ps_bulk_g2s(slice, a.w + ((size_t)o0 * nb + b_lo) * G::BLK, bytes, bar);
            }
        }
        __syncwarp();
        ps_grid_dep_wait();
        ps_grid_dep_launch();
        ps_mv_prologue(a, s_qs, s_d, sh_red, K, nb, tid, warp, lane);
        if (!own) return;
        if (b_hi > b_lo) ps_mbar_wait(bar, 0);
        for (int i = b_lo; i < b_hi; i++) {
            const uint8_t *blk = slice + (size_t)(i - b_lo) * G::BLK;
            int S_lo, S_hi;
            if (TYPE == 2) {
                const uint32_t w = *reinterpret_cast<const uint32_t *>(blk + r * 16 + 4 * t);
                const uint32_t lo = __vsub4(w & 0x0f0f0f0fu, 0x08080808u), hi = __vsub4((w >> 4) & 0x0f0f0f0fu, 0x08080808u);
                S_lo = __dp4a((int)lo, (int)s_qs[i * 8 + t], 0);
                S_hi = __dp4a((int)hi, (int)s_qs[i * 8 + 4 + t], 0);
            } else {
                const uint32_t w0 = *reinterpret_cast<const uint32_t *>(blk + r * 32 + 4 * t);
                const uint32_t w1 = *reinterpret_cast<const uint32_t *>(blk + r * 32 + 16 + 4 * t);
                S_lo = __dp4a((int)w0, (int)s_qs[i * 8 + t], 0);
                S_hi = __dp4a((int)w1, (int)s_qs[i * 8 + 4 + t], 0);
            }
            const float xd = ps_half_bits_to_float(*reinterpret_cast<const unsigned short *>(blk + 8 * G::QB + 2 * r));
            float *f = s_fac + (size_t)i * 96 + lane;
            f[0] = __fmul_rn(xd, s_d[i]);
            f[32] = __int2float_rn(S_lo);
            f[64] = __int2float_rn(S_hi);
        }
        __syncthreads();
        if (warp != 0) return;
        float a_lo = 0.f, a_hi = 0.f;
#pragma unroll 4
        for (int i = 0; i < nb; i++) { // the two chains of this thread's AVX lanes, block by block in row order
            const float *f = s_fac + (size_t)i * 96 + lane;
            const float d = f[0];
            a_lo = __fmaf_rn(d, f[32], a_lo);
            a_hi = __fmaf_rn(d, f[64], a_hi);
        }
        float best_v = -INFINITY;
        int best_i = 0x7fffffff;
        ps_mv_epilogue(a, o0, r, t, a_lo, a_hi, best_v, best_i);
        if (a.part_val) {
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                const float ov = __shfl_xor_sync(PS_FULL, best_v, o);
                const int oi = __shfl_xor_sync(PS_FULL, best_i, o);
                if (ov > best_v || (ov == best_v && oi < best_i)) { best_v = ov; best_i = oi; }
            }
            if (lane == 0) { a.part_val[blockIdx.x] = best_v; a.part_idx[blockIdx.x] = best_i; }
        }
        return;
    }
    uint8_t *my_ring = s_ring + (size_t)warp * ns * stage_bytes;
    uint64_t *my_bar = s_bar + warp * ns;
    auto issue = [&](int s) { // lane 0: request stage #s of this warp's stream into slot s % ns
        const int oct = o0 + warp + (s / spo) * PS_MV_WARPS;
        const uint8_t *src = a.w + ((size_t)oct * nb + (size_t)(s % spo) * sb) * G::BLK;
        uint64_t *bar = my_bar + (s % ns);
        ps_mbar_expect_tx(bar, stage_bytes);
        ps_bulk_g2s(my_ring + (size_t)(s % ns) * stage_bytes, src, stage_bytes, bar);
    };
    // every warp runs its own ring: barriers are warp-private, so no CTA-wide synchronisation guards them
    if (lane == 0) {
        for (int s = 0; s < ns; s++) ps_mbar_init(my_bar + s, 1);
        ps_fence_barrier_init();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        for (int s = 0; s < ns && s < n_stages; s++) issue(s);
    }
    __syncwarp();
    ps_grid_dep_wait();
    ps_grid_dep_launch();

    ps_mv_prologue(a, s_qs, s_d, sh_red, K, nb, tid, warp, lane);

    // ---- the stream
    float best_v = -INFINITY;
    int best_i = 0x7fffffff;
    int s = 0, slot = 0;
    uint32_t phase = 0;
#pragma unroll 1
    for (int m = 0; m < n_mine; m++) {
        const int oct = o0 + warp + m * PS_MV_WARPS;
        float a_lo = 0.f, a_hi = 0.f; // AVX lanes t and t + 4 of this row's accumulator
#pragma unroll 1
        for (int ss = 0; ss < spo; ss++, s++) {
            ps_mbar_wait(&my_bar[slot], phase);
            const uint8_t *st = my_ring + (size_t)slot * stage_bytes;
            const int ib = ss * sb;
#pragma unroll 4
            for (int b = 0; b < sb; b++) {
                const uint8_t *blk = st + (size_t)b * G::BLK;
                const int i = ib + b;
                int S_lo, S_hi;
                if (TYPE == 2) {
                    const uint32_t w = *reinterpret_cast<const uint32_t *>(blk + r * 16 + 4 * t);
                    const uint32_t lo = __vsub4(w & 0x0f0f0f0fu, 0x08080808u), hi = __vsub4((w >> 4) & 0x0f0f0f0fu, 0x08080808u);
                    S_lo = __dp4a((int)lo, (int)s_qs[i * 8 + t], 0);
                    S_hi = __dp4a((int)hi, (int)s_qs[i * 8 + 4 + t], 0);
                } else {
                    const uint32_t w0 = *reinterpret_cast<const uint32_t *>(blk + r * 32 + 4 * t);
                    const uint32_t w1 = *reinterpret_cast<const uint32_t *>(blk + r * 32 + 16 + 4 * t);
                    S_lo = __dp4a((int)w0, (int)s_qs[i * 8 + t], 0);
                    S_hi = __dp4a((int)w1, (int)s_qs[i * 8 + 4 + t], 0);
                }
                const float xd = ps_half_bits_to_float(*reinterpret_cast<const unsigned short *>(blk + 8 * G::QB + 2 * r));
                const float d = __fmul_rn(xd, s_d[i]);
                a_lo = __fmaf_rn(d, __int2float_rn(S_lo), a_lo);
                a_hi = __fmaf_rn(d, __int2float_rn(S_hi), a_hi);
            }
            __syncwarp(); // the slot is drained by every lane: re-arm it
            if (lane == 0 && s + ns < n_stages) issue(s + ns);
            if (++slot == ns) { slot = 0; phase ^= 1; }
        }
        ps_mv_epilogue(a, oct, r, t, a_lo, a_hi, best_v, best_i);
    }
    if (a.part_val) { // greedy pick, stage 1: the CTA's best (value, lowest index)
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const float ov = __shfl_xor_sync(PS_FULL, best_v, o);
            const int oi = __shfl_xor_sync(PS_FULL, best_i, o);
            if (ov > best_v || (ov == best_v && oi < best_i)) { best_v = ov; best_i = oi; }
        }
        if (lane == 0) { sv[warp] = best_v; si[warp] = best_i; }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < PS_MV_WARPS; w++)
                if (sv[w] > best_v || (sv[w] == best_v && si[w] < best_i)) { best_v = sv[w]; best_i = si[w]; }
            a.part_val[blockIdx.x] = best_v;
            a.part_idx[blockIdx.x] = best_i;
        }
    }
}

// ROPE(q), ROPE(k) and the two KV-cache COPY ops of NormAttention::build (norm_attention.cpp:76-105) in one launch for the
// token at pos_dev[0]: blocks [0, n_heads) rotate a query head into `qr`; the next n_kv_heads rotate a key head straight
// into row `pos` of the K cache; the last n_kv_heads write a value head into column `pos` of the transposed V cache.
// Rotation arithmetic = ps_k_rope (ggml_compute_forward_rope_f32, ggml.c:15368-15497; NORM pairs (2p, 2p+1), NEOX pairs
// (p, p + n_dims/2); products rounded separately).
__global__ void __launch_bounds__(64) ps_k_rope_kv(float *__restrict__ qr, const float *__restrict__ q, const float *__restrict__ k, const float *__restrict__ v,
                                                   float *__restrict__ kc, float *__restrict__ vct, int head_size, int n_heads, int n_kv_heads, int n_dims,
                                                   int neox, const int32_t *__restrict__ pos_dev, const float *__restrict__ table, int64_t n_ctx) {
    ps_grid_dep_wait();
    ps_grid_dep_launch();
    const int pos = pos_dev[0];
    const int b = blockIdx.x;
    if (b >= n_heads + n_kv_heads) { // value head
        const int h = b - n_heads - n_kv_heads;
        for (int e = threadIdx.x; e < head_size; e += blockDim.x) vct[((int64_t)h * head_size + e) * n_ctx + pos] = v[h * head_size + e];
        return;
    }
    const bool is_q = b < n_heads;
    const int h = is_q ? b : b - n_heads;
    const float *s = (is_q ? q : k) + (int64_t)h * head_size;
    float *d = is_q ? qr + (int64_t)h * head_size : kc + (int64_t)pos * head_size * n_kv_heads + (int64_t)h * head_size;
    const float *cache = table + (int64_t)pos * head_size;
    for (int p = threadIdx.x; p < head_size / 2; p += blockDim.x) {
        const int i0 = 2 * p;
        if (i0 < n_dims) {
            const float c = cache[i0], sn = cache[i0 + 1];
            const int ia = neox ? p : i0, ib = neox ? p + n_dims / 2 : i0 + 1;
            const float x0 = s[ia], x1 = s[ib];
            d[ia] = __fadd_rn(__fmul_rn(x0, c), -__fmul_rn(x1, sn));
            d[ib] = __fadd_rn(__fmul_rn(x0, sn), __fmul_rn(x1, c));
        } else {
            d[i0] = s[i0];
            d[i0 + 1] = s[i0 + 1];
        }
    }
}

// ---------------------------------------------------------------------------------------------------- token batches
// ps_k_matmul_qb's product (a thread = one AVX lane of two rows, C columns in registers) on the octet copies: a warp's eight rows are
// ONE contiguous stream, which it requests whole at the start - bulk copies in PS_MO_CHUNKS pieces with a barrier each - while the CTA stages
// the activations; rows of a 0.5B model are 4 to 22 KB.  On the GGUF bytes the kernel waited a memory round trip for every four
// blocks of a row, with one warp per scheduler to hide it: 896 x 4864 on 32 columns 84 us.  Pieces, us a layer on 4 / 32 / 128 columns: eight 108 /
// 150 / 312, sixteen 109 / 153 / 316, two 105 / 145 / 297 (0.5B, Q4_0); 138 / 541 / 1892, 145 / 563 / 1978, 135 / 525 / 1836 (2048 x 8192, Q8_0).
#define PS_MO_CHUNKS 8
#define PS_ERR_COPY 9 // error code: a bulk copy of ps_k_matmul_ob did not arrive
template <int TYPE> PS_HD size_t ps_mo_smem(int64_t K, int C, int warps) { return ps_mb_smem<TYPE>(K, C) + (size_t)warps * (size_t)(K / 32) * PsMv32<TYPE>::BLK; }
template <int TYPE, int C, bool REST>
__global__ void __launch_bounds__(PS_MB_WARPS * 32) ps_k_matmul_ob(const PsMbArgs a) {
    using G = PsMv32<TYPE>;
    constexpr int R = 2;
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ __align__(8) uint64_t bar[PS_MB_WARPS][PS_MO_CHUNKS];
    const int nb = (int)(a.K / 32), nbg = (nb + 3) / 4, col0 = blockIdx.y * C, ncol = min(C, a.bs - col0), warps = blockDim.x >> 5;
    int sg = 0;
    if (a.n_seg > 1 && (int)blockIdx.x >= a.seg[1].cta0) sg = 1;
    if (a.n_seg > 2 && (int)blockIdx.x >= a.seg[2].cta0) sg = 2;
    const PsMbSeg &seg = a.seg[sg];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l = lane & 7, r0 = lane >> 3;
    const int oct = ((int)blockIdx.x - seg.cta0) * warps + warp, n_oct = (seg.n + 7) / 8;
    const int cg = (nbg + PS_MO_CHUNKS - 1) / PS_MO_CHUNKS; // groups of four blocks per piece
    uint32_t *s_qs = reinterpret_cast<uint32_t *>(smem);                        // [C][group][8 lanes][4 blocks]
    float *s_d = reinterpret_cast<float *>(s_qs + (size_t)C * nbg * 32);        // [C][group][4 blocks]
    uint8_t *sw = smem + ps_mb_smem<TYPE>(a.K, C) + (size_t)warp * nb * G::BLK; // the warp's octet
    if (lane == 0) {
        for (int p = 0; p < PS_MO_CHUNKS; p++) ps_mbar_init(&bar[warp][p], 1);
        ps_fence_barrier_init();
        if (oct < n_oct)
            for (int p = 0, b0 = 0; b0 < nb; p++, b0 += 4 * cg) {
                const uint32_t bytes = (uint32_t)(min(4 * cg, nb - b0) * G::BLK);
                ps_mbar_expect_tx(&bar[warp][p], bytes);
                ps_bulk_g2s(sw + (size_t)b0 * G::BLK, seg.w + ((size_t)oct * nb + b0) * G::BLK, bytes, &bar[warp][p]);
            }
    }
    ps_grid_dep(); // (the weights are on their way)
    ps_mb_stage32<C>(s_qs, s_d, a.aqs + (int64_t)col0 * nb * 8, a.ad + (int64_t)col0 * nb, nb, nbg, ncol);
    __syncthreads();
    if (oct >= n_oct) return;
    float acc[R][C];
#pragma unroll
    for (int t = 0; t < R; t++)
#pragma unroll
        for (int c = 0; c < C; c++) acc[t][c] = 0.f;
    if (warp == a.give_up) *a.err = PS_ERR_COPY;
    for (int g = 0; g < nbg; g++) {
        // after a wait that gave up the results are invalid; the loop goes on and waits for the other pieces, each within its limit, so that none is in
        // flight when this shared memory becomes another CTA's
        if (g % cg == 0 && !ps_tc_wait(&bar[warp][g / cg], 0)) *a.err = PS_ERR_COPY;
        int q[R][4];
        float xd[R][4];
#pragma unroll
        for (int b = 0; b < 4; b++) {
            const uint8_t *blk = sw + (size_t)min(4 * g + b, nb - 1) * G::BLK; // past the end: the last block again, against zeros
#pragma unroll
            for (int t = 0; t < R; t++) {
                const int row = r0 + 4 * t;
                const uint32_t w = *reinterpret_cast<const uint32_t *>(blk + row * G::QB + (TYPE == 2 ? (l & 3) : l) * 4);
                q[t][b] = TYPE == 2 ? (int)__vsub4((l < 4) ? (w & 0x0f0f0f0fu) : ((w >> 4) & 0x0f0f0f0fu), 0x08080808u) : (int)w;
                xd[t][b] = !REST || 4 * g + b < nb ? ps_half_bits_to_float(*reinterpret_cast<const unsigned short *>(blk + 8 * G::QB + 2 * row)) : 0.f;
            }
        }
#pragma unroll
        for (int c = 0; c < C; c++) {
            const uint4 y = *reinterpret_cast<const uint4 *>(s_qs + ((size_t)(c * nbg + g) * 8 + l) * 4);
            const float4 yd = *reinterpret_cast<const float4 *>(s_d + (size_t)(c * nbg + g) * 4);
            const int yw[4] = {(int)y.x, (int)y.y, (int)y.z, (int)y.w};
            const float ydv[4] = {yd.x, yd.y, yd.z, yd.w};
#pragma unroll
            for (int b = 0; b < 4; b++)
#pragma unroll
                for (int t = 0; t < R; t++) {
                    const float S = __fsub_rn(__int_as_float(__dp4a(q[t][b], yw[b], 0x4B400000)), 12582912.f); // |sum| < 2^17: exact
                    acc[t][c] = __fmaf_rn(__fmul_rn(xd[t][b], ydv[b]), S, acc[t][c]);
                }
        }
    }
#pragma unroll
    for (int t = 0; t < R; t++) {
        const int n = oct * 8 + r0 + 4 * t;
#pragma unroll
        for (int c = 0; c < C; c++) {
            float r = acc[t][c]; // hsum_float_8 over the row's eight lanes
            r = __fadd_rn(r, __shfl_xor_sync(PS_FULL, r, 4));
            r = __fadd_rn(r, __shfl_xor_sync(PS_FULL, r, 2));
            r = __fadd_rn(r, __shfl_xor_sync(PS_FULL, r, 1));
            if (l == c % 8 && c < ncol && n < seg.n) {
                const int64_t o = (int64_t)(col0 + c) * seg.n + n;
                if (seg.bias) r = __fadd_rn(r, seg.bias[n]);
                if (a.residual) r = __fadd_rn(a.residual[o], r);
                seg.dst[o] = r;
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------- token batches on the tensor cores
// The same product on the tensor cores.  A block adds fl(d_x d_y) * S to each of eight chains, S the INTEGER sum of four products, and dp4a (2 cycles of the
// FMA pipe a warp), the integer-to-float step, the factor (every lane's own) and the FMA are five cycles of that pipe for 32 chain steps.
// mma.sync m16n8k8 makes 128 such sums, already float and exact (halves of 11 bits, products and sums of at most 17 bits in fp32), in 8 cycles of a
// pipe that runs beside the FMAs, and leaves a factor to eight chain steps.  Its k holds two AVX lanes, l and l + 4 (k = 2t: element t of lane l, k = 2t + 1: of
// lane l + 4), so the activation word is masked to one half for each of the two sums.  Any shape of mma.sync takes 8 cycles: 64 for 1024 chain steps.
// Warp w of a CTA takes lanes w and w + 4 of 16 rows x 8 NT columns; the chains of a row meet in shared memory at the end.  Weights and activations
// pass through a ring of stages that a fifth warp fills by bulk copies, over all of the CTA's tiles in a row, the first weights before the kernel
// before has ended.  The weights have an order of their own, in which a lane reads what it needs of four blocks at once: on the octet copies half of the
// instructions were byte loads and conversions of scales.
// Measured (Q4_0, 896 wide, 32 / 128 columns, us a product, cold caches; dp4a before): q|k|v 5.7 / 8.9 (9.4 / 17.6), o 6.5 / 9.1 (12 / 21), gate|up 16.4 / 47 (32 / 104), down 13.3 / 31
// (25 / 106); 32 tokens of six layers 632 -> 405 us.  HMMA pipe 30 % busy, issue 50 %: packed pairs need moves (14 instructions an MMA; with plain
// floats 13, and Q8_0 with two column tiles 162 -> 205 us).
//
// weight record of (16 rows, four blocks), g = lane / 4, t = lane % 4, rows g and g + 8: [4 w][32 lanes][2 rows][4 blocks] bytes (low nibble: element t of lane w,
// high nibble: of lane w + 4) or byte pairs (+ 128; of lanes w, w + 4), then [8 g][2 rows][4 blocks] scales.  Blocks past the row's end and rows past the matrix have scale zero
template <int TYPE> PS_HD constexpr int ps_mt_wq() { return TYPE == 2 ? 1024 : 2048; }
template <int TYPE> PS_HD constexpr int ps_mt_wrec() { return ps_mt_wq<TYPE>() + 256; }
PS_HD size_t ps_mt_w_bytes(int type, int64_t rows, int64_t K) { return (size_t)((rows + 15) / 16) * (size_t)((K / 32 + 3) / 4) * (type == 2 ? ps_mt_wrec<2>() : ps_mt_wrec<8>()); }
template <int TYPE> __global__ void __launch_bounds__(128) ps_k_mt_pack(uint8_t *__restrict__ dst, const uint8_t *__restrict__ w, int64_t n_rows, int64_t nb) { // grid (tiles, groups): y ends at 65 535
    constexpr int SRC = PsMv32<TYPE>::SRC;
    const int64_t g4 = blockIdx.y, tile = blockIdx.x;
    uint8_t *out = dst + (tile * gridDim.y + g4) * ps_mt_wrec<TYPE>();
    const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = lane & 3;
    for (int r = 0; r < 2; r++) {
        const int64_t row = tile * 16 + r * 8 + (lane >> 2);
        for (int b = 0; b < 4; b++) {
            const int64_t i = g4 * 4 + b;
            const bool live = row < n_rows && i < nb;
            const uint8_t *blk = w + (row * nb + i) * SRC;
            if (TYPE == 2) out[(threadIdx.x * 2 + r) * 4 + b] = live ? blk[2 + 4 * wp + t] : 0x88;
            else
                for (int h = 0; h < 2; h++) out[((threadIdx.x * 2 + r) * 4 + b) * 2 + h] = live ? blk[2 + 16 * h + 4 * wp + t] ^ 0x80 : 0x80;
            if (wp == 0 && t == 0)
                reinterpret_cast<float *>(out + ps_mt_wq<TYPE>())[(lane >> 2) * 8 + r * 4 + b] = live ? ps_half_bits_to_float((uint32_t)blk[0] | (uint32_t)blk[1] << 8) : 0.f;
        }
    }
}
// activation record of (8 columns, four blocks): [4 w][8 columns][4 t][4 blocks] pairs of halves (lane w, lane w + 4), then [4 t][4 blocks][columns 2t, 2t + 1] scales
#define PS_MT_REC 2176
PS_HD size_t ps_mt_x_bytes(int64_t K, int64_t cols) { return (size_t)((cols + 7) / 8) * (size_t)((K / 32 + 3) / 4) * PS_MT_REC; }
// one warp, four blocks of a column (lane = 8 b + l: word l of block b); blocks past the row's end are zeros
PS_D void ps_mt_store(uint8_t *__restrict__ dst, float4 v, int lane, int64_t g, int64_t col, int64_t nbg) {
    uint32_t word;
    float d;
    ps_mv_quant4(v, word, d);
    const int b = lane >> 3, l = lane & 7, n = (int)(col & 7);
    uint8_t *rec = dst + ((col >> 3) * nbg + g) * PS_MT_REC;
    const uint32_t other = __shfl_xor_sync(PS_FULL, word, 4), lo = l < 4 ? word : other, hi = l < 4 ? other : word; // lanes l % 4 and l % 4 + 4
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int t = (l >> 2) * 2 + k;
        const __half2 h = __halves2half2(__int2half_rn((int)(signed char)(lo >> (8 * t))), __int2half_rn((int)(signed char)(hi >> (8 * t))));
        reinterpret_cast<__half2 *>(rec)[(((l & 3) * 8 + n) * 4 + t) * 4 + b] = h;
    }
    if (l == 0) reinterpret_cast<float *>(rec + 2048)[((n >> 1) * 4 + b) * 2 + (n & 1)] = d;
}
__global__ void __launch_bounds__(128) ps_k_mt_quantize(const float *__restrict__ x, const float *__restrict__ u, int64_t K, uint8_t *__restrict__ dst) {
    ps_grid_dep();
    const int lane = threadIdx.x & 31;
    const int64_t nb = K / 32, nbg = (nb + 3) / 4, g = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5), i = g * 4 + (lane >> 3), col = blockIdx.y, at = col * K + i * 32 + 4 * (lane & 7);
    if (g >= nbg) return;
    ps_mt_store(dst, i < nb ? ps_act4(x + at, u ? u + at : nullptr) : make_float4(0.f, 0.f, 0.f, 0.f), lane, g, col, nbg);
}
__global__ void __launch_bounds__(512) ps_k_mt_norm_quantize(const float *__restrict__ x, const float *__restrict__ w, int64_t dim, float eps, uint8_t *__restrict__ dst) {
    ps_grid_dep();
    __shared__ double sh[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t col = blockIdx.x, nb = dim / 32, nbg = (nb + 3) / 4;
    const float *xr = x + col * dim;
    const float scale = ps_rms_scale(xr, dim, eps, sh);
    for (int64_t g = warp; g < nbg; g += 16) {
        const int64_t i = g * 4 + (lane >> 3), at = i * 32 + 4 * (lane & 7);
        ps_mt_store(dst, i < nb ? ps_norm4(xr + at, w + at, scale) : make_float4(0.f, 0.f, 0.f, 0.f), lane, g, col, nbg);
    }
}

struct PsMtSeg { const uint8_t *w; float *dst; const float *bias; int n, tile0; }; // w: weight records
struct PsMtArgs {
    PsMtSeg seg[3];
    int n_seg, bs, nbg, n_tiles, n_units, ns; // groups of four blocks; row tiles, x column groups: units of work; stages of the ring
    const uint8_t *x;   // activation records
    const float *residual;
    int *err, give_up;
};
#define PS_MT_MAX_NS 8
// groups of a stage: a wait and the issue of its copies cost some hundred cycles, a group's MMAs 64 NT (one group a stage, refilled by a thread of the first
// warp behind a CTA barrier: 1000 cycles a group whatever NT)
template <int NT> PS_HD constexpr int ps_mt_groups() { return NT == 1 ? 4 : 2; }
template <int TYPE, int NT> PS_HD constexpr int ps_mt_stage() { return ps_mt_groups<NT>() * (ps_mt_wrec<TYPE>() + NT * PS_MT_REC); }
template <int NT> PS_HD constexpr int ps_mt_red() { return 4 * 8 * NT * 16 * 4; } // [4 w][8 NT columns][16 rows] floats
// the sums of one AVX lane: (row g, columns 2t, 2t + 1), (row g + 8, the same)
PS_D void ps_mt_mma(float (&s)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=f"(s[0]), "=f"(s[1]), "=f"(s[2]), "=f"(s[3])
        : "r"(a0), "r"(a1), "r"(b), "f"(0.f));
}
template <int TYPE, int NT>
__global__ void __launch_bounds__(160) ps_k_matmul_mt(const PsMtArgs a) {
    constexpr int GS = ps_mt_groups<NT>(), WREC = ps_mt_wrec<TYPE>(), STAGE = ps_mt_stage<TYPE, NT>(), X0 = GS * WREC;
    extern __shared__ __align__(128) uint8_t ps_mt_smem[];
    __shared__ __align__(8) uint64_t bar_full[PS_MT_MAX_NS], bar_empty[PS_MT_MAX_NS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, t = lane & 3;
    const int nbg = a.nbg, ns = a.ns, n_st = (nbg + GS - 1) / GS, n_ct = (a.bs + 7) / 8;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ns; s++) {
            ps_mbar_init(&bar_full[s], 1);
            ps_mbar_init(&bar_empty[s], 4);
        }
        ps_fence_barrier_init();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    auto seg_of = [&](int tile) { return a.n_seg > 2 && tile >= a.seg[2].tile0 ? 2 : a.n_seg > 1 && tile >= a.seg[1].tile0 ? 1 : 0; };
    if (warp == 4) { // ===== copies
        auto weights = [&](int u, int k, int slot) { // stage k of unit u
            const int tile = u % a.n_tiles, n = min(GS, nbg - GS * k);
            const PsMtSeg &seg = a.seg[seg_of(tile)];
            ps_mbar_expect_tx(&bar_full[slot], (uint32_t)(n * (WREC + NT * PS_MT_REC)));
            ps_bulk_g2s(ps_mt_smem + (size_t)slot * STAGE, seg.w + ((size_t)(tile - seg.tile0) * nbg + GS * k) * WREC, (uint32_t)(n * WREC), &bar_full[slot]);
        };
        auto columns = [&](int u, int k, int slot) {
            const int ct0 = u / a.n_tiles * NT, n = min(GS, nbg - GS * k);
#pragma unroll
            for (int j = 0; j < NT; j++) // (past the last tile: that one again)
                ps_bulk_g2s(ps_mt_smem + (size_t)slot * STAGE + X0 + j * (GS * PS_MT_REC), a.x + ((size_t)min(ct0 + j, n_ct - 1) * nbg + GS * k) * PS_MT_REC, (uint32_t)(n * PS_MT_REC),
                            &bar_full[slot]);
        };
        const int ahead = min(ns, n_st);
        if (ps_elect_one())
            for (int k = 0; k < ahead; k++) weights(blockIdx.x, k, k);
        __syncwarp();
        ps_grid_dep();
        int slot = 0, n = 0;
        uint32_t phase = 0;
        for (int u = blockIdx.x; u < a.n_units; u += gridDim.x)
            for (int k = 0; k < n_st; k++, n++) {
                if (n >= ns && !ps_tc_wait_warp(&bar_empty[slot], phase ^ 1, PS_COPY_CYCLES)) *a.err = PS_ERR_COPY;
                if (ps_elect_one()) {
                    if (n >= ahead) weights(u, k, slot);
                    columns(u, k, slot);
                }
                __syncwarp();
                if (++slot == ns) { slot = 0; phase ^= 1; }
            }
        return; // (the other warps wait for every copy)
    }
    ps_grid_dep();
    if (warp == a.give_up) *a.err = PS_ERR_COPY;
    float *red = reinterpret_cast<float *>(ps_mt_smem + (size_t)ns * STAGE);
    int slot = 0;
    uint32_t phase = 0;
    for (int u = blockIdx.x; u < a.n_units; u += gridDim.x) {
        ps_f2 acc[2][2][NT]; // [lane w, w + 4][row g, g + 8][column tile]: columns 2t, 2t + 1
#pragma unroll
        for (int j = 0; j < NT; j++) acc[0][0][j] = acc[0][1][j] = acc[1][0][j] = acc[1][1][j] = 0ull;
        for (int k = 0; k < n_st; k++) {
            // after a wait that gave up the results are invalid; the loop goes on and waits for the other copies, each within its limit, so that none is in
            // flight when this shared memory becomes another CTA's
            if (!ps_tc_wait(&bar_full[slot], phase, PS_COPY_POLLS)) *a.err = PS_ERR_COPY;
            const uint8_t *st = ps_mt_smem + (size_t)slot * STAGE;
            auto group = [&](int g) {
                const uint8_t *sw = st + g * WREC;
                uint32_t av[2][4];  // [row g, g + 8][block]: the halves of lanes w and w + 4
                if (TYPE == 2) { // low nibble n, high nibble m of a byte: halves 1024 + n and 1024 + 16 m, made n - 8 and m - 8
                    const uint2 q = *reinterpret_cast<const uint2 *>(sw + (warp * 32 + lane) * 8);
#pragma unroll
                    for (int r = 0; r < 2; r++)
#pragma unroll
                        for (int b = 0; b < 4; b++) {
                            const uint32_t h = __byte_perm(r ? q.y : q.x, 0, b | 0x4040 | b << 8) & 0x00F0000Fu | 0x64006400u;
                            asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(av[r][b]) : "r"(h), "r"(0x2C003C00u), "r"(0xD480E408u)); // x (1, 1 / 16) + (-1032, -72)
                        }
                } else { // 1024 + 128 + q - 1152
                    const uint4 q = *reinterpret_cast<const uint4 *>(sw + (warp * 32 + lane) * 16);
                    const uint32_t w[2][2] = {{q.x, q.y}, {q.z, q.w}};
#pragma unroll
                    for (int r = 0; r < 2; r++)
#pragma unroll
                        for (int b = 0; b < 4; b++)
                            asm("add.rn.f16x2 %0, %1, %2;" : "=r"(av[r][b]) : "r"(__byte_perm(w[r][b >> 1], 0x64646464u, (b & 1) ? 0x4342 : 0x4140)), "r"(0xE480E480u));
                }
                const float4 d0 = *reinterpret_cast<const float4 *>(sw + ps_mt_wq<TYPE>() + gr * 32), d1 = *reinterpret_cast<const float4 *>(sw + ps_mt_wq<TYPE>() + gr * 32 + 16);
                const float xd[2][4] = {{d0.x, d0.y, d0.z, d0.w}, {d1.x, d1.y, d1.z, d1.w}};
#pragma unroll
                for (int j = 0; j < NT; j++) {
                    const uint8_t *sx = st + X0 + (j * GS + g) * PS_MT_REC;
                    const uint4 bq = *reinterpret_cast<const uint4 *>(sx + (warp * 32 + lane) * 16);
                    const ulonglong2 y01 = *reinterpret_cast<const ulonglong2 *>(sx + 2048 + t * 32), y23 = *reinterpret_cast<const ulonglong2 *>(sx + 2048 + t * 32 + 16);
                    const uint32_t bw[4] = {bq.x, bq.y, bq.z, bq.w};
                    const ps_f2 yd[4] = {y01.x, y01.y, y23.x, y23.y};
#pragma unroll
                    for (int b = 0; b < 4; b++) {
                        float s[2][4];
                        ps_mt_mma(s[0], av[0][b], av[1][b], bw[b] & 0xFFFFu);
                        ps_mt_mma(s[1], av[0][b], av[1][b], bw[b] & 0xFFFF0000u);
                        const ps_f2 d[2] = {ps_f2_mul(ps_f2_pack(xd[0][b], xd[0][b]), yd[b]), ps_f2_mul(ps_f2_pack(xd[1][b], xd[1][b]), yd[b])};
#pragma unroll
                        for (int l = 0; l < 2; l++)
#pragma unroll
                            for (int r = 0; r < 2; r++) acc[l][r][j] = ps_f2_fma(d[r], ps_f2_pack(s[l][2 * r], s[l][2 * r + 1]), acc[l][r][j]);
                    }
                }
            };
            if (GS * (k + 1) <= nbg) {
#pragma unroll(NT == 4 ? 1 : GS) // a warp is often alone on its scheduler: the loads of one group then fly beside the MMAs and FMAs of the other
                for (int g = 0; g < GS; g++) group(g);
            } else {
#pragma unroll 1
                for (int g = 0; g < nbg - GS * k; g++) group(g);
            }
            __syncwarp();
            if (lane == 0) ps_mbar_arrive(&bar_empty[slot]);
            if (++slot == ns) { slot = 0; phase ^= 1; }
        }
        // hsum_float_8: (x4 + x0, x5 + x1, x6 + x2, x7 + x3) -> (r0 + r2) + (r1 + r3)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                float p, q;
                ps_f2_unpack(ps_f2_add(acc[1][r][j], acc[0][r][j]), p, q);
                red[(warp * 8 * NT + 8 * j + 2 * t) * 16 + 8 * r + gr] = p;
                red[(warp * 8 * NT + 8 * j + 2 * t + 1) * 16 + 8 * r + gr] = q;
            }
        ps_bar_sync(1, 128);
        const int tile = u % a.n_tiles, ct0 = u / a.n_tiles * NT;
        const PsMtSeg &seg = a.seg[seg_of(tile)];
#pragma unroll
        for (int k = 0; k < NT; k++) {
            const int e = k * 128 + threadIdx.x, c = 8 * ct0 + (e >> 4), n = (tile - seg.tile0) * 16 + (e & 15);
            float r = __fadd_rn(__fadd_rn(red[e], red[256 * NT + e]), __fadd_rn(red[128 * NT + e], red[384 * NT + e]));
            if (c < a.bs && n < seg.n) {
                const int64_t o = (int64_t)c * seg.n + n;
                if (seg.bias) r = __fadd_rn(r, seg.bias[n]);
                if (a.residual) r = __fadd_rn(a.residual[o], r);
                seg.dst[o] = r;
            }
        }
        if (u + (int)gridDim.x < a.n_units) ps_bar_sync(1, 128); // (the next tile's numbers go to the same place)
    }
}
