// DSA / MLA sparse decode, fp32, any shape: ONE launch does what the reference spreads
// over eight launches and three materialised buffers (kernels/dsa/naive_dsa.cu:435-474):
// the three row gathers (:13-59), the 576-wide fused dot (:208-273), the scale (:321-324),
// the softmax (:278-294, here online) and the output projection (:300-316).
//
// Vector-aligned shapes take dsa_cluster_f32_kernel, everything else the general dsa_fused_f32_kernel:
// block = 8 warps = 8 heads of one query.  A tile of up to 32 selected rows (K = [Kc|Kp]
// and V) is staged in shared memory once and reused by the 8 heads; within a warp the
// lane is the row while scoring and the output column while accumulating P*V.
// Offsets are 64-bit; every listed index contributes (duplicates twice), any order.
#include <cfloat>

#include "common.cuh"

#include "cluster_f32.cuh"

void b200_count_launch(int n);

#define DSA_HB 8

template <int NJ>   // output columns per lane: Dc <= 32 * NJ
__global__ void __launch_bounds__(DSA_HB * 32)
dsa_fused_f32_kernel(const float* __restrict__ q_nope, const float* __restrict__ q_pe,
                     const float* __restrict__ kc, const float* __restrict__ kp, const float* __restrict__ v,
                     const int* __restrict__ idx, float* __restrict__ out,
                     int H, int Dc, int Dp, int S, int TS, float scale, int N) {
    extern __shared__ float sm[];
    const int Dk = Dc + Dp;
    const int ldk = Dk | 1;                       // odd row stride: lanes hit distinct banks
    float* qs = sm;                               // [DSA_HB][Dk]
    float* ks = qs + DSA_HB * Dk;                 // [TS][ldk]
    float* vs = ks + (size_t)TS * ldk;            // [TS][Dc]
    float* ps = vs + (size_t)TS * Dc;             // [DSA_HB][32]
    __shared__ long long row_id[32];

    const int q = blockIdx.x;
    const int h0 = blockIdx.y * DSA_HB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = h0 + warp;
    const bool head_ok = h < H;

    for (int i = threadIdx.x; i < DSA_HB * Dk; i += blockDim.x) {
        int hh = i / Dk, d = i % Dk;
        float val = 0.0f;
        if (h0 + hh < H)
            val = (d < Dc) ? q_nope[((size_t)q * H + h0 + hh) * Dc + d]
                           : q_pe[((size_t)q * H + h0 + hh) * Dp + (d - Dc)];
        qs[i] = val;
    }

    float m = -FLT_MAX, l = 0.0f;
    float acc[NJ];
#pragma unroll
    for (int j = 0; j < NJ; j++) acc[j] = 0.0f;

    for (int s0 = 0; s0 < S; s0 += TS) {
        const int rows = min(TS, S - s0);
        __syncthreads();                          // previous tile fully consumed (and qs visible)
        // an index that is negative or, when the cache size N is given, not below N is an empty entry: it
        // is not read and contributes nothing (the reference reads it unchecked, kernels/dsa/naive_dsa.cu:19-24)
        if (threadIdx.x < rows) {
            const int id = idx[(size_t)q * S + s0 + threadIdx.x];
            row_id[threadIdx.x] = (id < 0 || (N > 0 && id >= N)) ? -1ll : (long long)id;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < rows * Dk; i += blockDim.x) {
            int r = i / Dk, d = i % Dk;
            long long id = row_id[r];
            ks[(size_t)r * ldk + d] = id < 0 ? 0.0f : ((d < Dc) ? kc[id * Dc + d] : kp[id * Dp + (d - Dc)]);
        }
        for (int i = threadIdx.x; i < rows * Dc; i += blockDim.x) {
            int r = i / Dc, d = i % Dc;
            vs[(size_t)r * Dc + d] = row_id[r] < 0 ? 0.0f : v[row_id[r] * Dc + d];
        }
        __syncthreads();

        // scores: lane = row
        float sc = -FLT_MAX;
        const bool row_live = lane < rows && row_id[lane] >= 0;
        if (row_live) {
            const float* kr = ks + (size_t)lane * ldk;
            const float* qr = qs + warp * Dk;
            float sum = 0.0f;
            for (int d = 0; d < Dk; d++) sum = fmaf(qr[d], kr[d], sum);
            sc = sum * scale;
        }
        float tile_max = sc;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, o));
        const float m_new = fmaxf(m, tile_max);
        const float corr = expf(m - m_new);       // first tile: exp(-huge) = 0, acc and l are 0 anyway
        const float p = row_live ? expf(sc - m_new) : 0.0f;
        float psum = p;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) psum += __shfl_xor_sync(0xffffffffu, psum, o);
        l = l * corr + psum;
        m = m_new;
        ps[warp * 32 + lane] = p;
        __syncwarp();
        // P*V: lane = output column (d = lane + 32 j)
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            int d = lane + 32 * j;
            if (d < Dc) {
                float a = acc[j] * corr;
                for (int r = 0; r < rows; r++) a = fmaf(ps[warp * 32 + r], vs[(size_t)r * Dc + d], a);
                acc[j] = a;
            }
        }
    }
    if (head_ok) {
        const float inv = l > 0.0f ? 1.0f / l : 0.0f;      // every entry empty: zero row
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            int d = lane + 32 * j;
            if (d < Dc) out[((size_t)q * H + h) * Dc + d] = acc[j] * inv;
        }
    }
}

// ---------------------------------------------------------------------------
// Cluster version of the fused decode for vector-aligned shapes (Dc % 4 == 0, Dp % 4 == 0, Dc <= 512,
// Dc + Dp <= 640, 16-byte aligned tensors).  A decode call is small (a few MB) and what bounds it is latency:
// how many rows are fetched at once, and how long the chain of fetch, dot, softmax and P*V steps is.  So the
// selected rows of (query, 4 heads) are divided among the CTAs of a cluster (up to 8), each CTA takes its share in tiles
// of 32 rows, four per warp, with every load of the tile in flight at once, and the partial results (maximum, sum,
// accumulator) meet in distributed shared memory: still one launch, no workspace, a fixed order of additions.
// Q = 4, H = 16, Dc = 512, Dp = 64, S = 256: 389 us (one block per query and 8 heads, 8 blocks in all) -> 14.4 us; the
// error against 64-bit arithmetic falls from 8.6e-7 to 2.3e-7 (shorter chains).
//   scores  lane = 16-byte groups of the row (coalesced, K goes to registers only); one read of the query from
//           shared memory serves the warp's four rows; 16 sums per warp are folded by a 16-shuffle butterfly.
//   P*V     thread = two output columns (narrow heads: 256 / (Dc / 2) row groups side by side), V straight from
//           global memory, fetched before the scores are complete.
constexpr int FC_HB = 4, FC_THREADS = 256, FC_TR = 32;

template <int NG>      // 16-byte groups of [K | position] per lane: (Dc + Dp) / 4 <= 32 * NG
__global__ void __launch_bounds__(FC_THREADS)
dsa_cluster_f32_kernel(const float* __restrict__ q_nope, const float* __restrict__ q_pe,
                       const float* __restrict__ kc, const float* __restrict__ kp, const float* __restrict__ v,
                       const int* __restrict__ idx, float* __restrict__ out,
                       int H, int Dc, int Dp, int S, float scale, int N) {
    __shared__ __align__(16) float qs[FC_HB][NG * 128];
    __shared__ __align__(16) float acc_s[FC_HB * 512];      // [row group][head][Dc]: at most 256 column pairs x 4 heads
    __shared__ __align__(16) float sc_s[FC_TR][FC_HB];      // scores, then probabilities
    __shared__ float corr_s[FC_HB];
    __shared__ float ml_s[2][FC_HB];
    __shared__ long long row_s[2][FC_TR];

    uint32_t crank, csize;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
    const int q = blockIdx.z, h0 = blockIdx.y * FC_HB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ngr = (Dc + Dp) >> 2, ngc = Dc >> 2, vlines = (Dc + 31) >> 5;
    // whole tiles per CTA, so that every CTA but the last of a cluster works on full tiles
    const int tiles = (S + FC_TR - 1) / FC_TR;
    const int per = (tiles + (int)csize - 1) / (int)csize;
    const int s_begin = min(S, (int)crank * per * FC_TR), s_end = min(S, s_begin + per * FC_TR);

    // an index that is negative or, when the cache size N is given, not below N is an empty entry
    auto fetch_row = [&](int s) -> long long {
        if (s >= s_end) return -1ll;
        const int id = idx[(size_t)q * S + s];
        return (id < 0 || (N > 0 && id >= N)) ? -1ll : (long long)id;
    };
    if (threadIdx.x < FC_TR) row_s[0][threadIdx.x] = fetch_row(s_begin + threadIdx.x);
    for (int i = threadIdx.x; i < FC_HB * NG * 32; i += FC_THREADS) {
        const int hh = i / (NG * 32), g = i - hh * (NG * 32);
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (h0 + hh < H && g < ngr)
            x = (g < ngc) ? *reinterpret_cast<const float4*>(q_nope + ((size_t)q * H + h0 + hh) * Dc + g * 4)
                          : *reinterpret_cast<const float4*>(q_pe + ((size_t)q * H + h0 + hh) * Dp + (g - ngc) * 4);
        *reinterpret_cast<float4*>(&qs[hh][g * 4]) = x;
    }
    // P*V: column pair and row group of this thread
    const int cp = Dc >> 1, rgs = FC_THREADS / cp;
    const int rg = threadIdx.x / cp, col = (threadIdx.x - rg * cp) * 2;
    const bool pv = rg < rgs;
    float acc[FC_HB][2];
#pragma unroll
    for (int h = 0; h < FC_HB; h++) acc[h][0] = acc[h][1] = 0.0f;
    float m = -FLT_MAX, l = 0.0f;              // warps 0..3: running maximum and sum of head `warp`
    __syncthreads();

    int buf = 0;
    for (int s0 = s_begin; s0 < s_end; s0 += FC_TR, buf ^= 1) {
        const int rows = min(FC_TR, s_end - s0);
        // ---- scores: rows 4 warp .. 4 warp + 3 ----
        {
            float4 k[4][NG];
            bool live[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const long long id = row_s[buf][4 * warp + i];
                live[i] = id >= 0;
#pragma unroll
                for (int g = 0; g < NG; g++) {
                    const int gg = lane + 32 * g;
                    k[i][g] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (live[i] && gg < ngr)
                        k[i][g] = (gg < ngc) ? *reinterpret_cast<const float4*>(kc + id * Dc + gg * 4)
                                             : *reinterpret_cast<const float4*>(kp + id * Dp + (gg - ngc) * 4);
                }
            }
            // the V rows of the tile travel to L2 while the scores are formed
            for (int i = threadIdx.x; i < rows * vlines; i += FC_THREADS) {
                const long long id = row_s[buf][i / vlines];
                if (id >= 0)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(v + id * Dc + (i % vlines) * 32));
            }
            if (threadIdx.x < FC_TR) row_s[buf ^ 1][threadIdx.x] = fetch_row(s0 + FC_TR + threadIdx.x);
            float s16[16];
#pragma unroll
            for (int i = 0; i < 16; i++) s16[i] = 0.0f;
#pragma unroll
            for (int g = 0; g < NG; g++) {
#pragma unroll
                for (int h = 0; h < FC_HB; h++) {
                    const float4 x = *reinterpret_cast<const float4*>(&qs[h][(lane + 32 * g) * 4]);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        float a = s16[i * 4 + h];
                        a = fmaf(x.x, k[i][g].x, a); a = fmaf(x.y, k[i][g].y, a);
                        a = fmaf(x.z, k[i][g].z, a); a = fmaf(x.w, k[i][g].w, a);
                        s16[i * 4 + h] = a;
                    }
                }
            }
            // fold 16 sums over 32 lanes: after the step over `o` a lane keeps the half whose index bit matches its own
#pragma unroll
            for (int st = 0, n = 8; st < 4; st++, n >>= 1) {
                const int o = 16 >> st;
                const bool up = (lane & o) != 0;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    if (i < n) {
                        const float keep = up ? s16[i + n] : s16[i], give = up ? s16[i] : s16[i + n];
                        s16[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                    }
                }
            }
            const float tot = s16[0] + __shfl_xor_sync(0xffffffffu, s16[0], 1);
            const int which = lane >> 1;                     // sum `which`: row which / 4, head which % 4
            if ((lane & 1) == 0) sc_s[4 * warp + (which >> 2)][which & 3] = tot * scale;
        }
        __syncthreads();
        // ---- softmax step: warp h handles head h, lane = row ----
        if (warp < FC_HB) {
            const bool live = lane < rows && row_s[buf][lane] >= 0;
            const float sc = live ? sc_s[lane][warp] : -FLT_MAX;
            float tile_max = sc;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, o));
            const float m_new = fmaxf(m, tile_max);
            const float corr = expf(m - m_new);
            const float p = live ? expf(sc - m_new) : 0.0f;
            float psum = p;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) psum += __shfl_xor_sync(0xffffffffu, psum, o);
            l = l * corr + psum;
            m = m_new;
            sc_s[lane][warp] = p;
            if (lane == 0) corr_s[warp] = corr;
        }
        __syncthreads();
        // ---- P*V ----
        if (pv) {
            float c[FC_HB];
#pragma unroll
            for (int h = 0; h < FC_HB; h++) { c[h] = corr_s[h]; acc[h][0] *= c[h]; acc[h][1] *= c[h]; }
#pragma unroll 8
            for (int r = rg; r < rows; r += rgs) {
                const long long id = row_s[buf][r];
                const float2 vv = (id >= 0) ? *reinterpret_cast<const float2*>(v + id * Dc + col) : make_float2(0.f, 0.f);
                const float4 p4 = *reinterpret_cast<const float4*>(sc_s[r]);
                acc[0][0] = fmaf(p4.x, vv.x, acc[0][0]); acc[0][1] = fmaf(p4.x, vv.y, acc[0][1]);
                acc[1][0] = fmaf(p4.y, vv.x, acc[1][0]); acc[1][1] = fmaf(p4.y, vv.y, acc[1][1]);
                acc[2][0] = fmaf(p4.z, vv.x, acc[2][0]); acc[2][1] = fmaf(p4.z, vv.y, acc[2][1]);
                acc[3][0] = fmaf(p4.w, vv.x, acc[3][0]); acc[3][1] = fmaf(p4.w, vv.y, acc[3][1]);
            }
        }
        __syncthreads();                       // row_s[buf], sc_s and corr_s have been read
    }
    if (pv) {
#pragma unroll
        for (int h = 0; h < FC_HB; h++)
            *reinterpret_cast<float2*>(&acc_s[((size_t)rg * FC_HB + h) * Dc + col]) = make_float2(acc[h][0], acc[h][1]);
    }
    if (warp < FC_HB && lane == 0) { ml_s[0][warp] = m; ml_s[1][warp] = l; }
    cluster_sync();
    // ---- merge: CTA r of the cluster writes every csize-th run of outputs ----
    for (int i = (int)crank * FC_THREADS + threadIdx.x; i < FC_HB * Dc; i += (int)csize * FC_THREADS) {
        const int hh = i / Dc;
        float M = -FLT_MAX, mr[8], L = 0.0f, o = 0.0f;
        for (int r = 0; r < (int)csize; r++) {
            mr[r] = cluster_ld_f32(cluster_map(&ml_s[0][hh], r));
            M = fmaxf(M, mr[r]);
        }
        for (int r = 0; r < (int)csize; r++) {
            const float f = expf(mr[r] - M);
            L = fmaf(cluster_ld_f32(cluster_map(&ml_s[1][hh], r)), f, L);
            float part = 0.0f;
            for (int g = 0; g < rgs; g++) part += cluster_ld_f32(cluster_map(&acc_s[(size_t)g * FC_HB * Dc + i], r));
            o = fmaf(part, f, o);
        }
        // every entry empty: o = 0 and the factor 0; a NaN score or an overflow makes o and L NaN, and the product stays NaN
        if (h0 + hh < H) out[((size_t)q * H + h0) * Dc + i] = o * (L > 0.0f ? 1.0f / L : 0.0f);
    }
    cluster_sync();                        // nobody leaves while a neighbour still reads its shared memory
}

// ---------------------------------------------------------------------------
// stage kernels (the reference's per-stage launchers)
// ---------------------------------------------------------------------------
__global__ void gather_rows_f32_kernel(const float* __restrict__ src, const int* __restrict__ idx,
                                       float* __restrict__ dst, long long total, int Dm) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long stride = (long long)gridDim.x * blockDim.x;
    for (; i < total; i += stride) {
        long long pair = i / Dm;
        int d = (int)(i % Dm);
        dst[i] = src[(long long)idx[pair] * Dm + d];
    }
}

// scores[q,h,s] += q_nope . g_kc + q_pe . g_kp  (either part optional)
__global__ void dot_rows_f32_kernel(const float* __restrict__ qn, const float* __restrict__ qp,
                                    const float* __restrict__ gkc, const float* __restrict__ gkp,
                                    float* scores, int Q, int H, int S, int Dc, int Dp) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long total = (long long)Q * H * S;
    if (i >= total) return;
    int s = (int)(i % S);
    int h = (int)((i / S) % H);
    int q = (int)(i / ((long long)S * H));
    float sum = 0.0f;
    if (qn && gkc) {
        const float* a = qn + ((size_t)q * H + h) * Dc;
        const float* b = gkc + ((size_t)q * S + s) * Dc;
        for (int d = 0; d < Dc; d++) sum = fmaf(a[d], b[d], sum);
    }
    if (qp && gkp) {
        const float* a = qp + ((size_t)q * H + h) * Dp;
        const float* b = gkp + ((size_t)q * S + s) * Dp;
        for (int d = 0; d < Dp; d++) sum = fmaf(a[d], b[d], sum);
    }
    scores[i] += sum;
}

// one warp per (q,h) row
__global__ void softmax_rows_f32_kernel(float* scores, long long rows, int S) {
    long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (row >= rows) return;
    float* r = scores + row * S;
    float mx = -FLT_MAX;
    for (int s = lane; s < S; s += 32) mx = fmaxf(mx, r[s]);
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = 0.0f;
    for (int s = lane; s < S; s += 32) { float e = expf(r[s] - mx); r[s] = e; sum += e; }
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    float inv = 1.0f / sum;
    for (int s = lane; s < S; s += 32) r[s] *= inv;
}

__global__ void output_proj_f32_kernel(const float* __restrict__ attn, const float* __restrict__ gv,
                                       float* __restrict__ out, int Q, int H, int S, int Dc) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long total = (long long)Q * H * Dc;
    if (i >= total) return;
    int d = (int)(i % Dc);
    int h = (int)((i / Dc) % H);
    int q = (int)(i / ((long long)Dc * H));
    const float* a = attn + ((size_t)q * H + h) * S;
    const float* vv = gv + (size_t)q * S * Dc + d;
    float sum = 0.0f;
    for (int s = 0; s < S; s++) sum = fmaf(a[s], vv[(size_t)s * Dc], sum);
    out[i] = sum;
}

static int check_dsa(const b200_dsa_config* c) {
    if (!c) return B200_BAD_ARG;
    if (c->num_queries <= 0 || c->num_heads <= 0 || c->head_dim_compressed <= 0 || c->head_dim_positional < 0 ||
        c->num_selected_kv <= 0)
        return B200_BAD_SHAPE;
    return B200_OK;
}

template <int NJ>
static int launch_dsa_f32(const float* qn, const float* qp, const float* kc, const float* kp, const float* v,
                          const int* idx, float* out, const b200_dsa_config* c, size_t smem_limit,
                          cudaStream_t stream) {
    const int Dc = c->head_dim_compressed, Dp = c->head_dim_positional, Dk = Dc + Dp;
    int TS = 32;
    auto need = [&](int ts) {
        return sizeof(float) * ((size_t)DSA_HB * Dk + (size_t)ts * (Dk | 1) + (size_t)ts * Dc + DSA_HB * 32);
    };
    while (TS > 1 && need(TS) > smem_limit) TS >>= 1;
    if (need(TS) > smem_limit) return B200_UNSUPPORTED;
    size_t smem = need(TS);
    static B200PerDeviceOnce once;
    const int st = b200_allow_smem(once, dsa_fused_f32_kernel<NJ>, smem_limit);
    if (st) return st;
    dim3 grid(c->num_queries, ceil_div(c->num_heads, DSA_HB));
    float scale = 1.0f / sqrtf((float)Dk);        // naive_dsa.cu:464
    dsa_fused_f32_kernel<NJ><<<grid, DSA_HB * 32, smem, stream>>>(qn, qp, kc, kp, v, idx, out, c->num_heads, Dc, Dp,
                                                                   c->num_selected_kv, TS, scale, c->total_kv_tokens);
    b200_count_launch(1);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

template <int NG>
static int launch_dsa_f32_cluster(const float* qn, const float* qp, const float* kc, const float* kp, const float* v,
                                  const int* idx, float* out, const b200_dsa_config* c, int sm_count, cudaStream_t stream) {
    const int head_blocks = ceil_div(c->num_heads, FC_HB), tiles = ceil_div(c->num_selected_kv, FC_TR);
    // One tile of 32 rows per CTA, up to the portable cluster size, until the grid has two CTAs per SM (latency); beyond
    // that a CTA keeps eight tiles or more, and grids of six times that are cut once at most (less merging).
    // 256 queries x 8 heads, Dc = 512: S = 128 99 us split in four, 66 us not at all; S = 2048 736 us in four, 690 us in
    // two, 752 us not at all; 512 queries, Dc = 128, S = 2048: 638 us in two, 706 us not at all.
    const long long ctas = (long long)c->num_queries * head_blocks;
    auto room = [&](int cs) {
        return ctas * cs < 2ll * sm_count || (ctas * cs < 6ll * sm_count && tiles >= 16 * cs) ||
               (ctas < 8ll * sm_count && cs == 1 && tiles >= 32);
    };
    int cs = 1;
    while (cs < 8 && cs < tiles && room(cs)) cs *= 2;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(cs, head_blocks, c->num_queries);
    lc.blockDim = dim3(FC_THREADS);
    lc.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cs; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    lc.attrs = attr; lc.numAttrs = 1;
    const float scale = 1.0f / sqrtf((float)(c->head_dim_compressed + c->head_dim_positional));        // naive_dsa.cu:464
    B200_CUDA_TRY(cudaLaunchKernelEx(&lc, dsa_cluster_f32_kernel<NG>, qn, qp, kc, kp, v, idx, out, c->num_heads,
                                     c->head_dim_compressed, c->head_dim_positional, c->num_selected_kv, scale, c->total_kv_tokens));
    b200_count_launch(1);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

// Where the general kernel stays: batches that fill the machine with little work per (query, head).  Its eight heads share
// one staged tile, the cluster kernel's four fetch their rows themselves and pay for the cluster and the merge.  Measured
// with H a multiple of 8 (time of the general kernel / time of the cluster kernel; N = 8192; ctas = queries x groups
// of four heads):
//   ctas = 512    Dc = 16 0.90 .. 1.0, Dc = 32 from S = 64 on 1.1 and more, Dc = 128 S = 8 0.84, S = 32 1.1 and more
//   ctas = 1024   Dc = 16 0.66 .. 0.83, Dc = 32 0.69 (S = 8) 0.97 (128) 1.08 (512), Dc = 64 0.71 (8) 0.94 (32) 1.08 (64)
//   ctas = 4096   Dc = 32 0.42 (8) .. 0.91 (2048), Dc = 64 0.55 (8) 0.95 (64) 1.10 (128), Dc = 128 0.48 (8) 0.82 (32) 1.08
//                 (64), Dc = 256 0.86 (8) 1.7 (32), Dc = 512 2.4 (8)
// Heads that leave the general kernel's blocks partly empty shift the line: H = 2, ctas = 2048, Dc = 16 0.56 (8) 0.88 (64)
// 1.06 (128), Dc = 64 0.86 (8) 1.27 (32), Dc = 128 0.87 (8), Dc = 256 1.2 (1); H = 12, ctas = 1536 Dc = 16 0.50 .. 0.90,
// Dc = 32 0.94 (64), Dc = 64 0.70 (8), Dc = 128 0.66 (8), above 1 (32).
static bool dsa_f32_general_pays(const b200_dsa_config* c) {
    const int H = c->num_heads, Dc = c->head_dim_compressed;
    const long long ctas = (long long)c->num_queries * ceil_div(H, FC_HB), work = (long long)c->num_selected_kv * Dc;
    if (Dc > 256 || ctas < 512) return false;
    if (H <= 4) return ctas >= 2048 && Dc <= 128 && work <= 1024;
    if (Dc <= 16) return true;
    if (H >= 9 && H <= 12) return work <= (Dc <= 128 ? 2048 : 1024);
    if (Dc <= 32) return ctas >= 2048 || work <= 4096;
    return work <= (Dc <= 128 && ctas >= 2048 ? 4096 : 2048);
}

extern "C" {

int b200_dsa_forward_f32(b200_ws* ws, const float* q_nope, const float* q_pe, const float* kc, const float* kp,
                         const float* v, const int* idx, float* out, const b200_dsa_config* cfg,
                         b200_stream_t stream) {
    int st = check_dsa(cfg);
    if (st) return st;
    if (!q_nope || !kc || !v || !idx || !out) return B200_BAD_ARG;
    if (cfg->head_dim_positional > 0 && (!q_pe || !kp)) return B200_BAD_ARG;
    if (cfg->num_queries > 0x7fffffff / 1 || ceil_div(cfg->num_heads, DSA_HB) > 65535) return B200_UNSUPPORTED;
    if (!ws) ws = b200_default_ws();
    if (!ws) return B200_CUDA_ERROR;
    const size_t lim = ws->max_smem_optin - 1024;
    const int Dc = cfg->head_dim_compressed, Dp = cfg->head_dim_positional;
    // 16-byte groups of a row per lane, at most two output columns per thread; the query is the grid's z dimension
    const uintptr_t all = reinterpret_cast<uintptr_t>(q_nope) | reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(v) |
                          (Dp > 0 ? reinterpret_cast<uintptr_t>(q_pe) | reinterpret_cast<uintptr_t>(kp) : 0);
    if (Dc % 4 == 0 && Dp % 4 == 0 && Dc <= 512 && Dc + Dp <= 640 && (all & 15) == 0 && cfg->num_queries <= 65535 &&
        cfg->num_heads <= 65535 * FC_HB && !dsa_f32_general_pays(cfg)) {
        const int ng = ceil_div(Dc + Dp, 128);
        if (ng <= 1) return launch_dsa_f32_cluster<1>(q_nope, q_pe, kc, kp, v, idx, out, cfg, ws->sm_count, stream);
        if (ng <= 2) return launch_dsa_f32_cluster<2>(q_nope, q_pe, kc, kp, v, idx, out, cfg, ws->sm_count, stream);
        if (ng <= 3) return launch_dsa_f32_cluster<3>(q_nope, q_pe, kc, kp, v, idx, out, cfg, ws->sm_count, stream);
        return launch_dsa_f32_cluster<5>(q_nope, q_pe, kc, kp, v, idx, out, cfg, ws->sm_count, stream);
    }
    if (Dc <= 32) return launch_dsa_f32<1>(q_nope, q_pe, kc, kp, v, idx, out, cfg, lim, stream);
    if (Dc <= 64) return launch_dsa_f32<2>(q_nope, q_pe, kc, kp, v, idx, out, cfg, lim, stream);
    if (Dc <= 128) return launch_dsa_f32<4>(q_nope, q_pe, kc, kp, v, idx, out, cfg, lim, stream);
    if (Dc <= 256) return launch_dsa_f32<8>(q_nope, q_pe, kc, kp, v, idx, out, cfg, lim, stream);
    if (Dc <= 512) return launch_dsa_f32<16>(q_nope, q_pe, kc, kp, v, idx, out, cfg, lim, stream);
    if (Dc <= 1024) return launch_dsa_f32<32>(q_nope, q_pe, kc, kp, v, idx, out, cfg, lim, stream);
    return B200_UNSUPPORTED;
}

int b200_dsa_kv_gather_f32(const float* kc, const float* kp, const float* v, const int* idx, float* g_kc, float* g_kp,
                           float* g_v, const b200_dsa_config* cfg, b200_stream_t stream) {
    int st = check_dsa(cfg);
    if (st) return st;
    if (!idx) return B200_BAD_ARG;
    const long long pairs = (long long)cfg->num_queries * cfg->num_selected_kv;
    const int Dc = cfg->head_dim_compressed, Dp = cfg->head_dim_positional;
    auto run = [&](const float* src, float* dst, int Dm) {
        if (!src || !dst || Dm <= 0) return;
        long long total = pairs * Dm;
        long long blocks = (total + 255) / 256;
        if (blocks > 148 * 32) blocks = 148 * 32;
        gather_rows_f32_kernel<<<(unsigned)blocks, 256, 0, stream>>>(src, idx, dst, total, Dm);
        b200_count_launch(1);
    };
    run(kc, g_kc, Dc);
    run(kp, g_kp, Dp);
    run(v, g_v, Dc);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

int b200_dsa_dot_f32(const float* q_nope, const float* q_pe, const float* g_kc, const float* g_kp, float* scores,
                     const b200_dsa_config* cfg, b200_stream_t stream) {
    int st = check_dsa(cfg);
    if (st) return st;
    if (!scores) return B200_BAD_ARG;
    long long total = (long long)cfg->num_queries * cfg->num_heads * cfg->num_selected_kv;
    long long blocks = (total + 255) / 256;
    if (blocks > 0x7fffffffLL) return B200_UNSUPPORTED;
    dot_rows_f32_kernel<<<(unsigned)blocks, 256, 0, stream>>>(q_nope, q_pe, g_kc, g_kp, scores, cfg->num_queries,
                                                             cfg->num_heads, cfg->num_selected_kv,
                                                             cfg->head_dim_compressed, cfg->head_dim_positional);
    b200_count_launch(1);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

int b200_dsa_softmax_f32(float* scores, const b200_dsa_config* cfg, b200_stream_t stream) {
    int st = check_dsa(cfg);
    if (st) return st;
    if (!scores) return B200_BAD_ARG;
    long long rows = (long long)cfg->num_queries * cfg->num_heads;
    long long blocks = (rows + 7) / 8;
    if (blocks > 0x7fffffffLL) return B200_UNSUPPORTED;
    softmax_rows_f32_kernel<<<(unsigned)blocks, 256, 0, stream>>>(scores, rows, cfg->num_selected_kv);
    b200_count_launch(1);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

int b200_dsa_output_proj_f32(const float* attn, const float* g_v, float* out, const b200_dsa_config* cfg,
                             b200_stream_t stream) {
    int st = check_dsa(cfg);
    if (st) return st;
    if (!attn || !g_v || !out) return B200_BAD_ARG;
    long long total = (long long)cfg->num_queries * cfg->num_heads * cfg->head_dim_compressed;
    long long blocks = (total + 255) / 256;
    if (blocks > 0x7fffffffLL) return B200_UNSUPPORTED;
    output_proj_f32_kernel<<<(unsigned)blocks, 256, 0, stream>>>(attn, g_v, out, cfg->num_queries, cfg->num_heads,
                                                                cfg->num_selected_kv, cfg->head_dim_compressed);
    b200_count_launch(1);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

}  // extern "C"
