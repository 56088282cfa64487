// fp32 MoE layer (the reference's own data types): routing + permutation from
// moe_route.cu, then two grouped GEMM launches that cover every expert at once.
//
//   grouped_gemm1_f32  act[r, j] = silu(x_r . W1e[j]) * (x_r . W1e[I+j])   (SwiGLU fused;
//                      replaces tiled_gemm_bt_kernel + swiglu_strided_kernel,
//                      kernels/moe/naive_moe.cu:246-280, :297-310, called per expert at :437-455)
//   grouped_gemm2_f32  out[t, n] += w(t,e) * (act_r . W2e[n])             (router weight and
//                      scatter-add fused; replaces tiled_gemm_bt_kernel + scatter_kernel,
//                      naive_moe.cu:458-468, :315-335)
// Rows are addressed through the row -> (token, slot) map, so no gathered copy of the
// activations is made and the host never learns the per-expert counts.  Aligned shapes take the kernels of the
// vector path below; these two serve the rest.
#include <cfloat>
#include <type_traits>

#include "cluster_f32.cuh"
#include "common.cuh"
#include "moe_internal.cuh"

#define G_TM 32   // rows per tile
#define G_TN 32   // output columns per tile
#define G_TK 32

// grid: (ceil(N/G_TN), ceil(T/G_TM), E); tiles beyond an expert's row count exit at once.
template <int MODE>   // 1: GEMM1 + SwiGLU, 2: GEMM2 + weighted scatter-add
__global__ void __launch_bounds__(256)
grouped_gemm_f32_kernel(const float* __restrict__ a_src,     // MODE 1: x [T,D];  MODE 2: act [rows,I]
                        const float* __restrict__ w,         // MODE 1: W1 [E,2I,D]; MODE 2: W2 [E,D,I]
                        const int* __restrict__ offsets, const int* __restrict__ row_pair,
                        const float* __restrict__ wts, float* __restrict__ dst,
                        int K, int D, int I) {
    const int e = blockIdx.z;
    const int row0 = offsets[e], cnt = offsets[e + 1] - row0;
    const int m0 = blockIdx.y * G_TM;
    if (m0 >= cnt) return;
    const int n0 = blockIdx.x * G_TN;
    const int Kdim = (MODE == 1) ? D : I;      // reduction length
    const int Ncols = (MODE == 1) ? I : D;     // output columns

    __shared__ float As[G_TK][G_TM + 1];
    __shared__ float Bs[(MODE == 1) ? 2 : 1][G_TK][G_TN + 1];
    __shared__ long long a_row_off[G_TM];
    __shared__ int s_tok[G_TM];
    __shared__ float s_w[G_TM];

    if (threadIdx.x < G_TM) {
        int m = m0 + threadIdx.x;
        long long off = -1;
        int tok = 0; float wv = 0.0f;
        if (m < cnt) {
            int pair = row_pair[row0 + m];
            tok = pair / K;
            wv = wts ? wts[pair] : 0.0f;
            off = (MODE == 1) ? (long long)tok * D : (long long)(row0 + m) * I;
        }
        a_row_off[threadIdx.x] = off;
        s_tok[threadIdx.x] = tok;
        s_w[threadIdx.x] = wv;
    }
    __syncthreads();

    const float* we = w + (size_t)e * ((MODE == 1) ? (size_t)2 * I * D : (size_t)D * I);
    const int tx = threadIdx.x & 31;   // output column
    const int ty = threadIdx.x >> 5;   // 0..7 -> rows ty, ty+8, ty+16, ty+24
    float acc[2][4];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[h][i] = 0.0f;

    for (int k0 = 0; k0 < Kdim; k0 += G_TK) {
        // 256 threads load 32x32 tiles: thread -> (row = tid/8, 4 consecutive k)
        {
            int r = threadIdx.x >> 3, kk = (threadIdx.x & 7) * 4;
            long long off = a_row_off[r];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                int k = k0 + kk + i;
                As[kk + i][r] = (off >= 0 && k < Kdim) ? a_src[off + k] : 0.0f;
            }
            int n = n0 + r;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                int k = k0 + kk + i;
                bool ok = (n < Ncols) && (k < Kdim);
                Bs[0][kk + i][r] = ok ? we[(size_t)n * Kdim + k] : 0.0f;
                if (MODE == 1) Bs[1][kk + i][r] = ok ? we[(size_t)(I + n) * Kdim + k] : 0.0f;
            }
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < G_TK; k++) {
            float b0 = Bs[0][k][tx];
            float b1 = (MODE == 1) ? Bs[1][k][tx] : 0.0f;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float a = As[k][ty + 8 * i];
                acc[0][i] = fmaf(a, b0, acc[0][i]);
                if (MODE == 1) acc[1][i] = fmaf(a, b1, acc[1][i]);
            }
        }
        __syncthreads();
    }

    const int n = n0 + tx;
    if (n >= Ncols) return;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        int ml = ty + 8 * i;
        if (m0 + ml >= cnt) continue;
        if (MODE == 1) {
            float g = acc[0][i], u = acc[1][i];
            float sg = __fdiv_rn(g, 1.0f + expf(-g));      // silu as naive_moe.cu:308
            dst[(size_t)(row0 + m0 + ml) * I + n] = sg * u;
        } else {
            atomicAdd(&dst[(size_t)s_tok[ml] * D + n], s_w[ml] * acc[0][i]);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Vector path (D % 4 == 0, I % 4 == 0, 16-byte aligned tensors).  At these sizes (tens of tokens, weights of a few
// MB to 100 MB) the layer is bound by launches, by latency and by how much of the weights is in flight, so:
//   * three launches instead of eight: gate + selection + zero-fill of the output | GEMM1 | GEMM2, the later two
//     launched with programmatic stream serialisation (their first weight tiles are on the way before the kernel
//     in front of them has finished);
//   * no permutation kernel when the id list is short (T * K <= GV_PAIRS): every GEMM block reads the ids and
//     lists its expert's rows itself (a kilobyte against its 100 KB of weights);
//   * weights stream through a four-stage cp.async ring; a warp takes an eighth of every k-tile for the whole MT x 64
//     tile, thread = (MT / 4) x 8 outputs, operands read as 16-byte vectors along k from rows of 68 floats (odd
//     multiple of 16 bytes: no bank conflicts), the eight warps' sums are added at the end.  The multiply-adds of a
//     shared-memory read are what bounds the large case: with (MT / 4) x 4 outputs of a quarter of a 32-deep k-tile
//     per thread the T = 128 case below took 68 us;
//   * where the tiles do not fill the machine the reduction is split over a cluster of up to four CTAs and added in
//     rank order through distributed shared memory, so an output still receives one addition per (token, expert).
// T = 32, E = 8, K = 2, D = 128, I = 256: 67 -> 15 us a call; T = 128, E = 16, K = 2, D = 512, I = 1024: 350 -> 65 us
// (100 MB of weights); error against 64-bit arithmetic 9.2e-7 -> 5.0e-7.
// ---------------------------------------------------------------------------------------------
constexpr int GV_KT = 64, GV_LD = GV_KT + 4, GV_ST = 4, GV_N = 64, GV_THREADS = 256, GV_PAIRS = 2048, GV_IDS = GV_PAIRS / GV_THREADS;
constexpr int GV_MAXE = 4096;                                 // experts
constexpr int GV_W = GV_THREADS / 32, GV_RLD = GV_N + 8;      // warps; row stride of the warps' sums

__device__ __forceinline__ void gv_cp16(float* dst, const float* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ptx::smem_u32(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

struct GvParams {
    const float* a;          // MODE 1: x [T,D];  MODE 2: act [rows,I]
    const float* w;          // MODE 1: W1 [E,2I,D]; MODE 2: W2 [E,D,I]
    const int* ids;          // [T*K]
    const int* offsets;      // with row_pair: permutation made beforehand (long id lists)
    const int* row_pair;
    const float* wts;        // MODE 2
    float* dst;              // MODE 1: act [rows,I]; MODE 2: out [T,D]
    int TK, K, D, I, E;
};

template <int MT>
constexpr size_t gv_smem_bytes() { return sizeof(float) * (size_t)GV_ST * (GV_N + MT) * GV_LD; }

// MT rows x 64 weight rows per tile.  Which rows a block works on:
//   WALK  grid (ceil(N / tile columns), ny, E * cluster size): block (y, expert) takes the expert's row tiles y, y + ny, ...
//         and asks for the first one's weights before the routing is known where that tile is likely to exist.
//   DEAL  the same grid, for batches whose routing can leave an expert many tiles: those beyond its first ny are dealt out,
//         one each, to the E * ny blocks of the column, first to the ones without a tile (ny * MT is at least the mean row
//         count, so there are never more of them than blocks).  2048 rows on one of 128 experts (K = 1, D = 256, I = 512):
//         walked in series 1382 us, dealt out 256 us (347 us in the 32 x 32-tile kernels above, which have a block per
//         tile that may exist).
//   LIST  grid (ceil(N / tile columns), walkers, cluster size), long id lists with 32 rows and more per expert: the row
//         tiles of all experts in one list, taken in turn.  T = 8192, E = 16, K = 2, D = 128, I = 256: 360 us with a block
//         per tile that may exist, 225 us.
enum GvRows { WALK, DEAL, LIST };
template <int MODE, int MT, GvRows ROWS>
__global__ void __launch_bounds__(GV_THREADS, 2)
grouped_gemm_f32_vec_kernel(const GvParams p) {
    extern __shared__ __align__(16) float gv_smem[];
    __shared__ int s_pair[GV_PAIRS];
    __shared__ int s_scan[2][GV_W], s_rank, s_job[2];
    constexpr int RT = MT / 4;                               // rows per thread
    constexpr int STG = (GV_N + MT) * GV_LD;                 // floats per stage: weights, then activations
    static_assert(GV_W * MT * GV_RLD <= GV_ST * STG, "the warps' sums reuse the ring");
    uint32_t crank, csize;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
    const int E = p.E, own = blockIdx.z / csize, y = blockIdx.y, ny = ROWS == LIST ? 0 : gridDim.y;
    const int Kd = (MODE == 1) ? p.D : p.I, N = (MODE == 1) ? p.I : p.D;
    const int n0 = blockIdx.x * ((MODE == 1) ? GV_N / 2 : GV_N);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nkt = (Kd + GV_KT - 1) / GV_KT, per = (nkt + (int)csize - 1) / (int)csize;
    const int kt_b = min(nkt, (int)crank * per), nk = min(nkt, kt_b + per) - kt_b;

    // this thread's 16-byte pieces of a weight tile: tile rows tid / 16 + 16 i
    const int lr = tid >> 4, lk = (tid & 15) * 4;
    const float* wsrc[4];
    bool wok[4];
    auto weights_of = [&](int e) {
        const float* we = p.w + (size_t)e * ((MODE == 1) ? (size_t)2 * p.I * p.D : (size_t)p.D * p.I);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int c = lr + 16 * i;
            const int n = (MODE == 1) ? n0 + (c & 31) : n0 + c;
            wok[i] = n < N;
            wsrc[i] = we + (size_t)((MODE == 1 && c >= 32) ? p.I + (wok[i] ? n : 0) : (wok[i] ? n : 0)) * Kd;
        }
    };
    auto load_w = [&](int j) {                               // k-tile kt_b + j into ring slot j % GV_ST
        const int k = (kt_b + j) * GV_KT + lk;
        float* d = gv_smem + (j % GV_ST) * STG + lr * GV_LD + lk;
#pragma unroll
        for (int i = 0; i < 4; i++) gv_cp16(d + 16 * i * GV_LD, wsrc[i] + (k < Kd ? k : 0), wok[i] && k < Kd);
    };
    // The weights do not depend on the kernel in front: the first tiles are requested before waiting for it, where the block
    // is likely to have rows (T = 1, E = 256, K = 8, D = 512, I = 1024: 315 us with all experts' first tiles, 277 us without).
    bool requested = ROWS != LIST && (y == 0 ? 2 * p.TK > E : y * MT < p.TK / E);
    weights_of(own);
    if (requested)
        for (int j = 0; j < GV_ST - 1; j++)
            if (j < nk) load_w(j);
    // counts of all experts (short id list) in the ring's last slot, which nothing is on its way to before the main loop
    int* const hist = reinterpret_cast<int*>(gv_smem + (GV_ST - 1) * STG);
    static_assert(STG >= GV_MAXE, "a count per expert");
    if (ROWS == DEAL && !p.row_pair)
        for (int i = tid; i < E; i += GV_THREADS) hist[i] = 0;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // A short id list: thread = one pair, or GV_IDS consecutive ones.
    static_assert(GV_IDS * GV_THREADS == GV_PAIRS, "the whole list");
    const bool many = p.TK > GV_THREADS;
    const int pair0 = many ? tid * GV_IDS : tid;
    int id[GV_IDS];
    auto load_ids = [&]() {
#pragma unroll
        for (int i = 0; i < GV_IDS; i++) {
            if (i > 0 && !many) break;
            id[i] = (pair0 + i < p.TK) ? p.ids[pair0 + i] : -1;
        }
    };
    // Rows of an expert (ascending pairs) and, for the sorted position, the rows of lower experts
    int cnt = 0, base = 0;
    const int* rows = s_pair;
    auto list_rows = [&](int e) {
        if (ROWS == LIST || p.row_pair) {
            base = p.offsets[e];
            cnt = p.offsets[e + 1] - base;
            rows = p.row_pair + base;
            return;
        }
        int c = 0, lower = 0;
#pragma unroll
        for (int i = 0; i < GV_IDS; i++) {
            if (i > 0 && !many) break;
            c += id[i] == e ? 1 : 0;
            lower += id[i] >= 0 && id[i] < e ? 1 : 0;
        }
        int at = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int n = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= o) at += n;
        }
        lower = __reduce_add_sync(0xffffffffu, lower);
        if (lane == 31) { s_scan[0][warp] = at; s_scan[1][warp] = lower; }
        __syncthreads();
        at -= c;
        cnt = base = 0;
#pragma unroll
        for (int w = 0; w < GV_W; w++) {
            at += w < warp ? s_scan[0][w] : 0;
            cnt += s_scan[0][w];
            base += s_scan[1][w];
        }
#pragma unroll
        for (int i = 0; i < GV_IDS; i++) {
            if (i > 0 && !many) break;
            if (id[i] == e) s_pair[at++] = pair0 + i;
        }
        // (a barrier of the caller's makes the list visible)
    };
    auto tiles_of = [&](int e) { return ((ROWS == LIST || p.row_pair ? p.offsets[e + 1] - p.offsets[e] : hist[e]) + MT - 1) / MT; };
    // DEAL, LIST: the row tiles beyond each expert's first ny (LIST: all), numbered in order of (expert, tile); thread = a run of
    // experts.  idle: blocks without a tile of their own.
    const int run = (E + GV_THREADS - 1) / GV_THREADS, e_lo = min(E, tid * run), e_hi = min(E, e_lo + run);
    int mine = 0, before = 0, idle_before = 0, all = 0, idle_all = 0;
    auto number_tiles = [&]() {
        int idle = 0;
        for (int e = e_lo; e < e_hi; e++) {
            const int t = tiles_of(e);
            mine += max(0, t - ny);
            idle += max(0, ny - t);
        }
        before = mine; idle_before = idle;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, before, o), b = __shfl_up_sync(0xffffffffu, idle_before, o);
            if (lane >= o) { before += a; idle_before += b; }
        }
        if (lane == 31) { s_scan[0][warp] = before; s_scan[1][warp] = idle_before; }
        __syncthreads();
        before -= mine; idle_before -= idle;
#pragma unroll
        for (int w = 0; w < GV_W; w++) {
            const int a = s_scan[0][w], b = s_scan[1][w];
            if (w < warp) { before += a; idle_before += b; }
            all += a; idle_all += b;
        }
    };
    auto find_tile = [&](int n) {                            // s_job = expert and tile of number n
        if (n >= before && n < before + mine) {
            int left = n - before;
            for (int e = e_lo; e < e_hi; e++) {
                const int x = max(0, tiles_of(e) - ny);
                if (left < x) { s_job[0] = e; s_job[1] = ny + left; break; }
                left -= x;
            }
        }
        __syncthreads();
    };

    int m0 = y * MT, next = y;                               // the block's tile: rows m0 .. m0 + MT - 1 of the list
    bool more = false;
    if (ROWS == LIST) {
        number_tiles();
        if (next >= all) return;
        find_tile(next);
        weights_of(s_job[0]);
        list_rows(s_job[0]);
        m0 = s_job[1] * MT;
        __syncthreads();
    } else {
        if (!p.row_pair) load_ids();
        list_rows(own);
        bool over = false;                                   // any expert with more than ny tiles
        if (ROWS == DEAL) {
            if (!p.row_pair) {                               // (list_rows' barrier lies between clearing and counting)
#pragma unroll
                for (int i = 0; i < GV_IDS; i++) {
                    if (i > 0 && !many) break;
                    if (id[i] >= 0) atomicAdd(&hist[id[i]], 1);
                }
                __syncthreads();
            }
            for (int i = tid; i < E; i += GV_THREADS) over |= tiles_of(i) > ny;
        }
        if (ROWS == WALK) {
            __syncthreads();
        } else if (__syncthreads_or(over)) {
            number_tiles();
            if (own >= e_lo && own < e_hi) {                 // this block's turn: idle ones first, in order of (expert, y)
                int b = idle_before;
                for (int e = e_lo; e < own; e++) b += max(0, ny - tiles_of(e));
                const int t = min(ny, tiles_of(own));
                s_rank = y >= t ? b + y - t : idle_all + own * ny - b + y;
            }
            __syncthreads();
            more = s_rank < all;
            if (more) find_tile(s_rank);
        }
    }

    const int tx = lane & 7, ty = lane >> 3;
    constexpr int AR = (MT + 15) / 16;                       // activation rows per loader thread
    for (;;) {
        const bool live = m0 < cnt;
        const float* asrc[AR];
#pragma unroll
        for (int i = 0; i < AR; i++) {
            const int r = m0 + lr + 16 * i;
            asrc[i] = nullptr;
            if (lr + 16 * i < MT && r < cnt)
                asrc[i] = p.a + ((MODE == 1) ? (size_t)(rows[r] / p.K) * Kd : (size_t)(base + r) * Kd);
        }
        auto load_a = [&](int j) {
            const int k = (kt_b + j) * GV_KT + lk;
#pragma unroll
            for (int i = 0; i < AR; i++)
                if (lr + 16 * i < MT) {
                    const bool ok = asrc[i] != nullptr && k < Kd;
                    gv_cp16(gv_smem + (j % GV_ST) * STG + (GV_N + lr + 16 * i) * GV_LD + lk, ok ? asrc[i] + k : p.a, ok);
                }
        };
#pragma unroll
        for (int j = 0; j < GV_ST - 1; j++) {
            if (live && j < nk) {
                if (!requested) load_w(j);
                load_a(j);
            }
            ptx::cp_async_commit();                          // (early weights of an expert without rows are in a group too)
        }
        requested = false;
        if (live) {
            float acc[RT][8];
#pragma unroll
            for (int i = 0; i < RT; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = 0.0f;
            for (int j = 0; j < nk; j++) {
                ptx::cp_async_wait<GV_ST - 2>();
                __syncthreads();
                const float* sb = gv_smem + (j % GV_ST) * STG;
                const float* sa = sb + GV_N * GV_LD;
#pragma unroll
                for (int h = 0; h < GV_KT / 4 / GV_W; h++) {
                    const int k = (warp + GV_W * h) * 4;
                    float4 b[8];
#pragma unroll
                    for (int c = 0; c < 8; c++) b[c] = *reinterpret_cast<const float4*>(sb + (tx + 8 * c) * GV_LD + k);
#pragma unroll
                    for (int i = 0; i < RT; i++) {
                        const float4 a = *reinterpret_cast<const float4*>(sa + (ty + 4 * i) * GV_LD + k);
#pragma unroll
                        for (int c = 0; c < 8; c++) {
                            acc[i][c] = fmaf(a.x, b[c].x, acc[i][c]); acc[i][c] = fmaf(a.y, b[c].y, acc[i][c]);
                            acc[i][c] = fmaf(a.z, b[c].z, acc[i][c]); acc[i][c] = fmaf(a.w, b[c].w, acc[i][c]);
                        }
                    }
                }
                if (j + GV_ST - 1 < nk) { load_w(j + GV_ST - 1); load_a(j + GV_ST - 1); }
                ptx::cp_async_commit();
            }
            ptx::cp_async_wait<0>();
            __syncthreads();                                     // the ring is free: sums [warp][row][column]
#pragma unroll
            for (int i = 0; i < RT; i++)
#pragma unroll
                for (int c = 0; c < 8; c++) gv_smem[(warp * MT + ty + 4 * i) * GV_RLD + tx + 8 * c] = acc[i][c];
            __syncthreads();
            // add the warps' sums in place; thread = 4 consecutive columns
            for (int o = tid; o < MT * GV_N / 4; o += GV_THREADS) {
                float* q = gv_smem + (o >> 4) * GV_RLD + 4 * (o & 15);
                float4 s = *reinterpret_cast<const float4*>(q);
#pragma unroll
                for (int g = 1; g < GV_W; g++) {
                    const float4 v = *reinterpret_cast<const float4*>(q + g * MT * GV_RLD);
                    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
                }
                *reinterpret_cast<float4*>(q) = s;
            }
            if (csize > 1) cluster_sync(); else __syncthreads();
            auto total4 = [&](int m, int c4) -> float4 {         // the CTAs of the cluster in rank order
                const float* q = gv_smem + m * GV_RLD + 4 * c4;
                if (csize == 1) return *reinterpret_cast<const float4*>(q);
                float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
                for (uint32_t r = 0; r < csize; r++) {
                    const float4 v = cluster_ld_f32x4(cluster_map(q, r));
                    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
                }
                return s;
            };
            if (MODE == 1) {
                for (int o = (int)crank * GV_THREADS + tid; o < MT * GV_N / 8; o += (int)csize * GV_THREADS) {
                    const int m = o >> 3, c4 = o & 7;            // row, 4 activation columns: gate at 4 c4, up 32 further
                    if (m0 + m >= cnt || n0 + 4 * c4 >= N) continue;
                    const float4 g = total4(m, c4), u = total4(m, 8 + c4);
                    float4 r;
                    r.x = __fdiv_rn(g.x, 1.0f + expf(-g.x)) * u.x;   // silu as naive_moe.cu:308
                    r.y = __fdiv_rn(g.y, 1.0f + expf(-g.y)) * u.y;
                    r.z = __fdiv_rn(g.z, 1.0f + expf(-g.z)) * u.z;
                    r.w = __fdiv_rn(g.w, 1.0f + expf(-g.w)) * u.w;
                    *reinterpret_cast<float4*>(p.dst + (size_t)(base + m0 + m) * p.I + n0 + 4 * c4) = r;
                }
            } else {
                for (int o = (int)crank * GV_THREADS + tid; o < MT * GV_N / 4; o += (int)csize * GV_THREADS) {
                    const int m = o >> 4, c4 = o & 15;
                    if (m0 + m >= cnt || n0 + 4 * c4 >= N) continue;
                    const float4 s = total4(m, c4);
                    const int pair = rows[m0 + m];
                    const float wv = p.wts[pair];
                    float* d = p.dst + (size_t)(pair / p.K) * p.D + n0 + 4 * c4;
                    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(d), "f"(wv * s.x), "f"(wv * s.y), "f"(wv * s.z), "f"(wv * s.w)
                                 : "memory");
                }
            }
            // the ring is refilled (and the CTA may leave) only when nobody reads the sums any more
            if (csize > 1) cluster_sync(); else __syncthreads();
        }
        // nothing may be on its way into this block's shared memory when the ring is used again or the block leaves
        ptx::cp_async_wait<0>();
        if (ROWS == WALK) {
            m0 += ny * MT;
            if (m0 >= cnt) return;
            continue;
        }
        if (ROWS == LIST) {
            next += gridDim.y;
            more = next < all;
        }
        if (!more) return;
        more = false;
        __syncthreads();                                     // all threads' copies are over, s_job and the row list have been read
        if (ROWS == LIST) find_tile(next);
        weights_of(s_job[0]);
        if (ROWS == DEAL && !p.row_pair) load_ids();
        list_rows(s_job[0]);
        m0 = s_job[1] * MT;
        __syncthreads();                                     // the list is there, s_job has been read
    }
}

// Router of the vector path: block = 8 tokens x all (at most 32) experts, thread = one (token, expert) chain in the
// reference's order (multiply, then add, ascending d; naive_moe.cu:102-106), then one warp per token selects; the
// exponentials and divisions are spread over the lanes, sums and the K-slot scan stay in the reference's order.
// Also clears the block's output rows (GEMM2 adds into them).
constexpr int GR_T = 8, GR_KT = 128, GR_LD = GR_KT + 4, GR_ST = 4, GR_MAXE = 32;
constexpr size_t gr_smem_bytes(int E) { return sizeof(float) * (size_t)GR_ST * (E + GR_T) * GR_LD; }

__global__ void __launch_bounds__(GR_T * GR_MAXE)
gate_select_f32_kernel(const float* __restrict__ x, const float* __restrict__ wg, int* __restrict__ ids,
                       float* __restrict__ wts, float* __restrict__ out, int T, int E, int K, int D) {
    extern __shared__ __align__(16) float gr_smem[];
    __shared__ float s_p[GR_T][GR_MAXE];
    __shared__ float s_c[GR_T][GR_MAXE];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, t0 = blockIdx.x * GR_T;
    const int rowsz = E + GR_T, nkt = (D + GR_KT - 1) / GR_KT;
    auto load = [&](int j) {
        float* st = gr_smem + (size_t)(j % GR_ST) * rowsz * GR_LD;
        for (int i = tid; i < rowsz * (GR_KT / 4); i += blockDim.x) {
            const int r = i / (GR_KT / 4), k = j * GR_KT + (i % (GR_KT / 4)) * 4;
            const bool ok = k < D && (r < E || t0 + r - E < T);
            const float* src = r < E ? wg + (size_t)r * D + k : x + (size_t)(t0 + r - E) * D + k;
            gv_cp16(st + r * GR_LD + (i % (GR_KT / 4)) * 4, ok ? src : wg, ok);
        }
    };
#pragma unroll
    for (int j = 0; j < GR_ST - 1; j++) {
        if (j < nkt) load(j);
        ptx::cp_async_commit();
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int nrow = min(GR_T, T - t0);
    for (int i = tid; i < nrow * (D / 4); i += blockDim.x)
        reinterpret_cast<float4*>(out + (size_t)t0 * D)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    const int tok = tid / E, ex = tid - tok * E;
    const bool on = tok < GR_T;
    float acc = 0.0f;
    for (int j = 0; j < nkt; j++) {
        ptx::cp_async_wait<GR_ST - 2>();
        __syncthreads();
        if (on) {
            const float* st = gr_smem + (size_t)(j % GR_ST) * rowsz * GR_LD;
            const float *wr = st + ex * GR_LD, *xr = st + (E + tok) * GR_LD;
            const int kn = min(GR_KT, D - j * GR_KT);
#pragma unroll 8
            for (int k = 0; k < kn; k += 4) {
                const float4 a = *reinterpret_cast<const float4*>(xr + k), b = *reinterpret_cast<const float4*>(wr + k);
                acc = __fadd_rn(acc, __fmul_rn(a.x, b.x)); acc = __fadd_rn(acc, __fmul_rn(a.y, b.y));
                acc = __fadd_rn(acc, __fmul_rn(a.z, b.z)); acc = __fadd_rn(acc, __fmul_rn(a.w, b.w));
            }
        }
        if (j + GR_ST - 1 < nkt) load(j + GR_ST - 1);
        ptx::cp_async_commit();
    }
    ptx::cp_async_wait<0>();
    if (on) s_p[tok][ex] = acc;
    __syncthreads();
    for (int tt = warp; tt < nrow; tt += blockDim.x / 32) {
        // naive_moe.cu:109-141
        const float lg = lane < E ? s_p[tt][lane] : -FLT_MAX;
        float mx = -FLT_MAX;
        for (int i = 0; i < E; i++) mx = fmaxf(mx, s_p[tt][i]);
        __syncwarp();
        const float pe = (float)exp((double)__fsub_rn(lg, mx));      // correctly rounded expf
        if (lane < E) s_p[tt][lane] = pe;
        __syncwarp();
        float sum = 0.0f;
        for (int i = 0; i < E; i++) sum = __fadd_rn(sum, s_p[tt][i]);
        __syncwarp();
        if (lane < E) s_p[tt][lane] = __fdiv_rn(pe, sum);
        __syncwarp();
        if (lane == 0) {
            int* oi = ids + (size_t)(t0 + tt) * K;
            float* ow = wts + (size_t)(t0 + tt) * K;
            float* c = s_c[tt];
            for (int k = 0; k < K; k++) { c[k] = -FLT_MAX; oi[k] = -1; }
            for (int i = 0; i < E; i++) {
                const float pv = s_p[tt][i];
                int min_k = 0;
                for (int k = 1; k < K; k++)
                    if (c[k] < c[min_k]) min_k = k;
                if (pv > c[min_k]) { c[min_k] = pv; oi[min_k] = i; }
            }
            float tot = 0.0f;
            for (int k = 0; k < K; k++) tot = __fadd_rn(tot, c[k]);
            for (int k = 0; k < K; k++) ow[k] = (tot > 0.0f) ? __fdiv_rn(c[k], tot) : c[k];
        }
    }
}

// ---------------------------------------------------------------------------
// stage kernels (the reference's per-stage launchers; not on the fused path)
// ---------------------------------------------------------------------------
// naive_moe.cu:147-166 semantics, block-parallel: ascending token order kept by a
// ballot scan; rows copied by the whole block.
__global__ void __launch_bounds__(256)
gather_one_expert_kernel(const float* __restrict__ x, const int* __restrict__ ids, int expert, float* gathered,
                         int* token_map, int* count, int T, int K, int D) {
    __shared__ int warp_sums[8];
    __shared__ int s_running;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_running = 0;
    __syncthreads();
    for (int t0 = 0; t0 < T; t0 += 256) {
        int t = t0 + threadIdx.x;
        bool f = false;
        if (t < T)
            for (int k = 0; k < K; k++)
                if (ids[(size_t)t * K + k] == expert) { f = true; break; }
        unsigned bal = __ballot_sync(0xffffffffu, f);
        if (lane == 0) warp_sums[warp] = __popc(bal);
        __syncthreads();
        int before = s_running, total = 0;
        for (int w = 0; w < 8; w++) {
            if (w < warp) before += warp_sums[w];
            total += warp_sums[w];
        }
        if (f) token_map[before + __popc(bal & ((1u << lane) - 1))] = t;
        __syncthreads();
        if (threadIdx.x == 0) s_running += total;
        __syncthreads();
    }
    const int cnt = s_running;
    if (threadIdx.x == 0) *count = cnt;
    __threadfence_block();
    __syncthreads();
    for (long long i = threadIdx.x; i < (long long)cnt * D; i += 256) {
        int r = (int)(i / D), d = (int)(i % D);
        gathered[i] = x[(size_t)token_map[r] * D + d];
    }
}

// naive_moe.cu:205-238 (C = A * B, row-major)
__global__ void __launch_bounds__(256) gemm_nn_f32_kernel(const float* __restrict__ A, const float* __restrict__ B,
                                                          float* __restrict__ C, int M, int N, int Kd) {
    __shared__ float As[16][17], Bs[16][17];
    int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    int row = blockIdx.y * 16 + ty, col = blockIdx.x * 16 + tx;
    float sum = 0.0f;
    for (int k0 = 0; k0 < Kd; k0 += 16) {
        As[ty][tx] = (row < M && k0 + tx < Kd) ? A[(size_t)row * Kd + k0 + tx] : 0.0f;
        Bs[ty][tx] = (k0 + ty < Kd && col < N) ? B[(size_t)(k0 + ty) * N + col] : 0.0f;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 16; i++) sum = fmaf(As[ty][i], Bs[i][tx], sum);
        __syncthreads();
    }
    if (row < M && col < N) C[(size_t)row * N + col] = sum;
}

// naive_moe.cu:285-292
__global__ void swiglu_f32_kernel(const float* gate, const float* up, float* out, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float g = gate[i];
    out[i] = __fdiv_rn(g, 1.0f + expf(-g)) * up[i];
}

// naive_moe.cu:315-335, any D (grid.y tiles the columns)
__global__ void scatter_f32_kernel(const float* __restrict__ expert_out, const int* __restrict__ token_map,
                                   const float* __restrict__ wts, const int* __restrict__ ids, int expert,
                                   float* out, int count, int K, int D) {
    int i = blockIdx.x;
    int d = blockIdx.y * blockDim.x + threadIdx.x;
    if (i >= count || d >= D) return;
    int t = token_map[i];
    float w = 0.0f;
    for (int k = 0; k < K; k++)
        if (ids[(size_t)t * K + k] == expert) { w = wts[(size_t)t * K + k]; break; }
    atomicAdd(&out[(size_t)t * D + d], w * expert_out[(size_t)i * D + d]);
}

// one grouped GEMM launch of the vector path
template <int MODE, int MT, GvRows ROWS>
static int launch_gemm_vec(const GvParams& p, int ny, int sm_count, cudaStream_t stream) {
    static B200PerDeviceOnce once;
    const int st = b200_allow_smem(once, grouped_gemm_f32_vec_kernel<MODE, MT, ROWS>, gv_smem_bytes<MT>());
    if (st) return st;
    const int Kd = (MODE == 1) ? p.D : p.I, N = (MODE == 1) ? p.I : p.D;
    const int nx = ceil_div(N, (MODE == 1) ? GV_N / 2 : GV_N);
    // the list's TK / 32 + E tiles at most are walked by eight rounds of resident blocks (two per SM) or fewer
    if (ROWS == LIST) ny = (int)min((long long)p.TK / MT + p.E, (long long)max(1, 16 * sm_count / nx));
    const int nz = ROWS == LIST ? 1 : p.E;
    // cluster over k: until there are about two blocks per SM (what fits at a time)
    const int nkt = ceil_div(Kd, GV_KT);
    int cs = 1;
    while (cs < 4 && (long long)nx * (ROWS == LIST ? ny : p.E) * cs * 2 <= 2ll * sm_count && nkt >= 2 * cs) cs *= 2;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(nx, ny, nz * cs);
    lc.blockDim = dim3(GV_THREADS);
    lc.dynamicSmemBytes = gv_smem_bytes<MT>();
    lc.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = cs;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr; lc.numAttrs = 2;
    B200_CUDA_TRY(cudaLaunchKernelEx(&lc, grouped_gemm_f32_vec_kernel<MODE, MT, ROWS>, p));
    b200_count_launch(1);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

extern "C" {

int b200_moe_forward_f32(b200_ws* ws, const float* x, const float* gate_w, const float* w1, const float* w2,
                         float* out, const b200_moe_config* cfg, b200_stream_t stream) {
    if (!x || !gate_w || !w1 || !w2 || !out || !cfg) return B200_BAD_ARG;
    const int T = cfg->num_tokens, E = cfg->num_experts, K = cfg->top_k, D = cfg->hidden_dim,
              I = cfg->intermediate_dim;
    int st = check_route_cfg(T, E, K, D, B200_SCORE_SOFTMAX, 1, 1);
    if (st) return st;
    if (I <= 0) return B200_BAD_SHAPE;
    if (E > 65535 || ceil_div(T, G_TM) > 65535) return B200_UNSUPPORTED;
    if (!ws) ws = b200_default_ws();
    if (!ws) return B200_CUDA_ERROR;

    auto carve = [&](WsCarver& c, float*& partials, int*& ids, float*& wts, int*& counts, int*& offsets,
                     int*& row_pair, float*& act) {
        partials = c.take<float>((size_t)T * E);
        ids = c.take<int>((size_t)T * K);
        wts = c.take<float>((size_t)T * K);
        counts = c.take<int>(E);
        offsets = c.take<int>(E + 1);
        row_pair = c.take<int>((size_t)T * K);
        act = c.take<float>((size_t)T * K * I);
    };
    float *partials, *wts, *act; int *ids, *counts, *offsets, *row_pair;
    WsCarver sz(nullptr);
    carve(sz, partials, ids, wts, counts, offsets, row_pair, act);
    st = b200_ws_ensure(ws, sz.total());
    if (st) return st;
    WsCarver cv(ws->base);
    carve(cv, partials, ids, wts, counts, offsets, row_pair, act);

    const uintptr_t all = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gate_w) | reinterpret_cast<uintptr_t>(w1) |
                          reinterpret_cast<uintptr_t>(w2) | reinterpret_cast<uintptr_t>(out);
    const bool vec = D % 4 == 0 && I % 4 == 0 && (all & 15) == 0 && (long long)E * 4 <= 65535;
    const bool short_ids = vec && (long long)T * K <= GV_PAIRS;      // the GEMM blocks list their rows themselves
    // (the fused router clears the output while it reads its weights)
    const uintptr_t o0 = reinterpret_cast<uintptr_t>(out), g0 = reinterpret_cast<uintptr_t>(gate_w);
    const bool shared = o0 < g0 + sizeof(float) * (size_t)E * D && g0 < o0 + sizeof(float) * (size_t)T * D;
    if (vec && E <= GR_MAXE && short_ids && !shared) {
        static B200PerDeviceOnce once;
        st = b200_allow_smem(once, gate_select_f32_kernel, gr_smem_bytes(GR_MAXE));
        if (st) return st;
        gate_select_f32_kernel<<<ceil_div(T, GR_T), GR_T * GR_MAXE, gr_smem_bytes(E), stream>>>(x, gate_w, ids, wts, out, T, E, K, D);
        b200_count_launch(1);
        B200_CUDA_TRY(cudaGetLastError());
    } else {
        st = launch_gate_logits(x, nullptr, gate_w, partials, T, E, D, false, stream);
        if (st) return st;
        st = launch_route_select(partials, 1, nullptr, ids, wts, nullptr, nullptr, T, E, K, B200_SCORE_SOFTMAX, 1, 1,
                                 1.0f, stream);
        if (st) return st;
        if (!short_ids) {
            st = launch_permute(ids, T, K, E, true, counts, offsets, row_pair, stream);
            if (st) return st;
        }
        B200_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(float) * (size_t)T * D, stream));   // naive_moe.cu:413
    }
    if (vec) {
        GvParams p{};
        p.ids = ids; p.wts = wts; p.TK = T * K; p.K = K; p.D = D; p.I = I; p.E = E;
        if (!short_ids) { p.offsets = offsets; p.row_pair = row_pair; }
        // Row tiles of 8 .. 32: the smallest that holds the mean row count and twice its spread (binomial: at most
        // sqrt(mean)), because a second tile streams the weights again and an empty row costs as much as a full one.
        const float mean = (float)T * K / E;
        const int fit = min(T, (int)(mean + 2.0f * sqrtf(mean) + 0.999f));
        auto gemm = [&](auto mode) -> int {
            constexpr int M = decltype(mode)::value;
            auto own_blocks = [&](auto rows) -> int {
                constexpr int MT = decltype(rows)::value;
                // blocks per expert: one where the tile was chosen to hold the expert, else for the mean and a half
                const int ny = MT < 32 ? 1 : max(1, min(ceil_div(T, MT), ceil_div(3 * (p.TK / E + 1), 2 * MT)));
                // Knowing the other experts' counts costs a block 0.4 us (T = 32, E = 8, D = 128: 12.4 -> 13.2 us a call), so
                // tiles are dealt out where an expert could otherwise have more than four in series (T = 128, E = 16,
                // K = 2, D = 512, I = 1024: 69.6 -> 64.9 us), with 32 rows more than eight (at six, T = 300, E = 16,
                // D = 256, I = 512 took 55 us instead of 50).
                if (T > (MT < 32 ? 4 : 8) * ny * MT) return launch_gemm_vec<M, MT, DEAL>(p, ny, ws->sm_count, stream);
                return launch_gemm_vec<M, MT, WALK>(p, ny, ws->sm_count, stream);
            };
            if (fit <= 8) return own_blocks(std::integral_constant<int, 8>{});
            if (fit <= 16) return own_blocks(std::integral_constant<int, 16>{});
            if (fit <= 24) return own_blocks(std::integral_constant<int, 24>{});
            if (short_ids) return own_blocks(std::integral_constant<int, 32>{});
            return launch_gemm_vec<M, 32, LIST>(p, 0, ws->sm_count, stream);
        };
        p.a = x; p.w = w1; p.dst = act;
        st = gemm(std::integral_constant<int, 1>{});
        if (st) return st;
        p.a = act; p.w = w2; p.dst = out;
        return gemm(std::integral_constant<int, 2>{});
    }
    dim3 g1(ceil_div(I, G_TN), ceil_div(T, G_TM), E);
    grouped_gemm_f32_kernel<1><<<g1, 256, 0, stream>>>(x, w1, offsets, row_pair, nullptr, act, K, D, I);
    dim3 g2(ceil_div(D, G_TN), ceil_div(T, G_TM), E);
    grouped_gemm_f32_kernel<2><<<g2, 256, 0, stream>>>(act, w2, offsets, row_pair, wts, out, K, D, I);
    b200_count_launch(2);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

int b200_moe_gather_f32(const float* x, const int* expert_ids, int expert_id, float* gathered, int* token_map,
                        int* count, const b200_moe_config* cfg, b200_stream_t stream) {
    if (!x || !expert_ids || !gathered || !token_map || !count || !cfg) return B200_BAD_ARG;
    gather_one_expert_kernel<<<1, 256, 0, stream>>>(x, expert_ids, expert_id, gathered, token_map, count,
                                                    cfg->num_tokens, cfg->top_k, cfg->hidden_dim);
    b200_count_launch(1);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

int b200_gemm_f32(const float* A, const float* B, float* C, int M, int N, int K, b200_stream_t stream) {
    if (!A || !B || !C) return B200_BAD_ARG;
    if (M <= 0 || N <= 0 || K <= 0) return B200_BAD_SHAPE;
    dim3 grid(ceil_div(N, 16), ceil_div(M, 16));
    gemm_nn_f32_kernel<<<grid, 256, 0, stream>>>(A, B, C, M, N, K);
    b200_count_launch(1);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

int b200_swiglu_f32(const float* gate, const float* up, float* out, int n, b200_stream_t stream) {
    if (!gate || !up || !out) return B200_BAD_ARG;
    if (n <= 0) return n == 0 ? B200_OK : B200_BAD_SHAPE;
    swiglu_f32_kernel<<<ceil_div(n, 256), 256, 0, stream>>>(gate, up, out, n);
    b200_count_launch(1);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

int b200_moe_scatter_f32(const float* expert_out, const int* token_map, const float* expert_w, const int* expert_ids,
                         int expert_id, float* out, int count, const b200_moe_config* cfg, b200_stream_t stream) {
    if (!cfg) return B200_BAD_ARG;
    if (count == 0) return B200_OK;                  // naive_moe.cu:388
    if (!expert_out || !token_map || !expert_w || !expert_ids || !out) return B200_BAD_ARG;
    dim3 grid(count, ceil_div(cfg->hidden_dim, 256));
    scatter_f32_kernel<<<grid, 256, 0, stream>>>(expert_out, token_map, expert_w, expert_ids, expert_id, out, count,
                                                 cfg->top_k, cfg->hidden_dim);
    b200_count_launch(1);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

}  // extern "C"
