// FP8 (e4m3) block-scale MoE expert path for sm_100a.
//
// Replaces the reference's per-expert host loop (kernels/moe/naive_moe.cu:424-469: gather,
// D2H count + stream sync, GEMM1, SwiGLU, GEMM2, scatter; 5 launches and one host sync per
// expert) with one row-sort pass and two persistent grouped GEMM launches:
//
//   sort_rows_fp8_kernel   expert-sorted copy of the FP8 rows + 1x128 scales, and the
//                          row -> token / router-weight maps.
//   grouped_gemm_fp8<1>    act = requant_1x128( silu(x W1g^T) * (x W1u^T) )   (SwiGLU and
//                          requantisation fused in the epilogue: no fp32 GEMM1 output in HBM)
//   grouped_gemm_fp8<2>    out[token] += w * (act W2^T)                      (router weight and
//                          scatter-add fused in the epilogue)
//   grouped_gemm_fp8<3>    rows[r] = w * (act W2^T), then reduce_rows_kernel sums a token's rows
//                          in ascending expert order (the reference's order, naive_moe.cu:424):
//                          the bit-reproducible alternative to the scatter-add.
//
// GEMM structure (one CTA per SM, 384 threads, tiles 128 x 256 x 128 handed out round-robin,
// expert-major; E = 256, K = 8, D = 7168, I = 2048, a GPU that has just begun: T = 16 813 -> 733 us a call, T = 333 2070 -> 1876,
// T = 4096 3235 -> 2985; 32 experts x 1024 rows 2095 -> 1915, before and after what the comments below measure):
//   warp 8       TMA producer: A tile (128 rows x 128 B) and B tile (256 rows x 128 B) per
//                K block into a 4-stage shared-memory ring (128-byte swizzle, K-major).
//   warps 9,10   MMA issuers, one per 256-column TMEM accumulator stage (K blocks alternate between
//                them): 4 x tcgen05.mma kind::f8f6f4 (K = 32 each) per K block, started fresh for
//                every K block.  The issuers wait in mbarrier.try_wait: with 64 ns of sleep between polls they
//                noticed a free stage ~300 cycles late, and with 200 ns the producer an empty slot.
//   warps 0-7    promotion + epilogue: tcgen05.ld the K block's partial sums and fold them
//                into fp32 registers with a_scale[row,kb] * w_scale[nblk,kb] (the scales are
//                arbitrary fp32 values, so the scaling cannot be left to the tensor core).
//                Warp w owns TMEM lanes 32 (w % 4) .. +31 (the tile rows) and accumulator columns
//                128 (w / 4) .. +127: 128 running sums per thread.
//   warp 11      scales: a_scale[row,kb] * w_scale[nblk,kb] of the coming K blocks, and where the tile lies, into shared memory.
// Every mbarrier wait is bounded; on give-up the CTA flags B200_TIMEOUT and winds down.
#include "common.cuh"
#include "moe_internal.cuh"
#include "tma_host.cuh"

void b200_set_last_error_text(const char* text);

namespace {

constexpr int BM = 128, BN = 256, BK = 128;
constexpr int STAGES = 4;
constexpr int A_BYTES = BM * BK;            // 16384
constexpr int B_BYTES = BN * BK;            // 32768
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int NUM_PROMO_WARPS = 8;           // one barrier arrival per warp
constexpr int NQ = NUM_PROMO_WARPS / 4;      // column groups of the accumulator (TMEM lanes fix the row split at 4)
constexpr int QCOLS = BN / NQ;               // accumulator columns per promotion thread
constexpr int GEMM_THREADS = 32 * (NUM_PROMO_WARPS + 4);   // promotion/epilogue warpgroups, then the TMA + MMA warpgroup
constexpr int W_TMA = NUM_PROMO_WARPS, W_MMA0 = NUM_PROMO_WARPS + 1;
constexpr int MAX_E = 1024;
constexpr unsigned PRODUCER_SLEEP_NS = 40;
constexpr int DIRECT_ROWS = 16;              // GEMM2: rows of a warp up to which each lane adds its own row
// Register budgets after setmaxnreg.  The registers a warpgroup gives up are the only ones the others can
// take (the pool is what the CTA was launched with: GEMM_THREADS x LAUNCH_REGS), and setmaxnreg.inc waits
// without bound until its request is met, so the two sides must balance:
// promotion threads x (PROMO_REGS - LAUNCH_REGS) <= 128 x (LAUNCH_REGS - AUX_REGS).  The launcher checks
// the compiled register count against this before the first launch.
constexpr int LAUNCH_REGS = 168;
constexpr int PROMO_REGS = 232;
constexpr int AUX_REGS = 40;
constexpr int CH = 32;                       // columns per promotion load (two loads in flight)
constexpr int SW = 16;                       // columns per pass of the output transpose
constexpr int SC_RING = 4;                   // scales of four K blocks and the places of four tiles are in shared memory
static_assert(QCOLS % (2 * CH) == 0, "promotion chunks");
static_assert(NUM_PROMO_WARPS * (PROMO_REGS - LAUNCH_REGS) <= 4 * (LAUNCH_REGS - AUX_REGS), "setmaxnreg balance");
static_assert(GEMM_THREADS * LAUNCH_REGS <= 65536, "register file");

struct GemmSmem {
    uint64_t full[STAGES];
    uint64_t empty[STAGES];
    uint64_t tmem_full[2];
    uint64_t tmem_empty[2];
    uint64_t amax_bar[2];
    uint64_t sf_full[STAGES];      // block-scaled kernel only: the stage's scale factors are in shared memory
    uint64_t sc_free[SC_RING];     // CTA pairs: the promotion warps of this CTA have read the slot of the scale ring
    uint64_t pair_go;              // single-CTA tiles launched as clusters of two: the neighbour starts its tile
    uint32_t tmem_base;
    int abort_flag;
    int total_tiles;
    int tile_prefix[MAX_E + 1];
    float amax[2][NQ][BM];   // [tile parity][column group][row]
    alignas(16) float stage[NUM_PROMO_WARPS][32][SW + 4];   // per promotion warp: 32 rows x SW columns (+4 pad), output transpose
};

constexpr size_t GEMM_BASE_BYTES = 1024 /*alignment slack*/ + (size_t)STAGES * STAGE_BYTES + sizeof(GemmSmem);
// scales [K block % SC_RING][gate / up or column half][row], and where a tile lies [tile % SC_RING]
constexpr size_t GEMM_SMEM_BYTES = GEMM_BASE_BYTES + sizeof(float) * SC_RING * 2 * BM + sizeof(int4) * SC_RING;
static_assert(GEMM_SMEM_BYTES <= 232448, "shared memory budget of one CTA");
// block-scaled kernel: per stage one 512-byte scale atom for the 128 rows of A and two for the 256 rows of B
constexpr int SF_BYTES = 1536;
// block-scaled kernel: the accumulator is moved into fp32 registers every MX_FLUSH K blocks.  The tensor core's own
// accumulation over a long chain is less exact than fp32 additions (one chain over K = 7168 put ~1e-4 relative
// error on GEMM1, enough to flip one e4m3 code in a thousand at the requantisation and to push a few outputs of
// the full-size layer past the 1e-2 absolute bound); 32 MMAs per chain keep it near fp32.
constexpr int MX_FLUSH = 8;
constexpr size_t GEMM_MX_SMEM_BYTES = GEMM_BASE_BYTES + (size_t)STAGES * SF_BYTES;
static_assert(GEMM_MX_SMEM_BYTES <= 232448, "shared memory budget of one CTA (block-scaled kernel)");

struct GemmParams {
    const float* a_scale;      // scale of sorted row r, K block kb: a_scale[kb * a_ks + r]
    long long a_ks;
    const float* w_scale;      // MODE 1: [E, 2I/128, D/128]   MODE 2/3: [E, D/128, I/128]
    const int* offsets;        // [E+1]
    const int* row_tok;        // MODE 2
    const float* row_w;        // MODE 2/3
    uint8_t* act_q;            // MODE 1 out [rows, I]
    float* act_s;              // MODE 1 out: scale of row r, block b at act_s[r * s_rs + b * s_ks]
    long long s_rs, s_ks;
    float* out;                // MODE 2 out [T, D]; MODE 3 out [rows, D]
    int* status;
    int E, D, I;
    int packed;                // weights pre-tiled: one contiguous 256 x 128-byte block per (expert, n tile, K block)
#ifdef B200_GEMM_TRACE
    long long* trace;          // [8][TRACE_CAP] clock64 stamps of CTA 0's pipeline events (timeline builds only)
    int trace_warp;
#endif
};

#ifdef B200_GEMM_TRACE
constexpr int TRACE_CAP = 512;
long long* g_gemm_trace = nullptr;
int g_gemm_trace_warp = 0;
#define TRACE_STAMP(slot, idx) do { if (p.trace && blockIdx.x == 0 && (idx) < TRACE_CAP) p.trace[(slot) * TRACE_CAP + (idx)] = clock64(); } while (0)
#else
#define TRACE_STAMP(slot, idx) do { } while (0)
#endif

__device__ __forceinline__ void red_add_v4(float* addr, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}

// ---- CTA-pair (cta_group::2) helpers ------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_nctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// Tiles 2i and 2i+1 run on the two CTAs of a cluster at the same time; when an expert has 129..256 rows they are
// the two row tiles of one weight slab.  The slab comes from DRAM once only if both CTAs stream it within the
// time a line stays in L2 (~20 us at full DRAM rate), and without a rendezvous the CTA with the nearly empty row
// tile gains a few microseconds per tile and is a whole tile ahead after some rounds (measured: every second
// row tile re-read from DRAM, 11.7 GB instead of 7.8 GB per GEMM1 launch).  So the two producers meet before
// every tile: each arrives on the neighbour's barrier and waits on its own (bounded).
__device__ __forceinline__ bool pair_rendezvous(uint64_t* own_bar, uint32_t peer_bar_cluster_addr, uint32_t parity,
                                                volatile int* abort_flag) {
    if (ptx::elect_one())
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(peer_bar_cluster_addr) : "memory");
    return ptx::mbar_wait_relaxed(own_bar, parity, abort_flag, 100);
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of the same shared-memory location in CTA `rank` of the cluster (shared::cluster window)
__device__ __forceinline__ uint32_t map_to_cta(const void* p, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(ptx::smem_u32(p)), "r"(rank));
    return r;
}
// Arrival on a barrier of the pair's other CTA.  What it hands over is a TMEM stage whose reads have completed
// (tcgen05.wait::ld + tcgen05.fence::before_thread_sync) and no memory: the scales that were read with the stage go back inside the
// CTA (sc_free).  With .release.cluster, which would let the leader hand the scales back too, the arrival waits until all that the warp did
// in memory is visible to the other CTA: a K block of a pair then takes 1950 - 2280 cycles instead of 950 - 980 (32 experts x 1024
// rows 3.75 ms against 2.40, T = 4096 6.8 against 4.4).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_cluster(uint32_t cluster_addr, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(cluster_addr),
                 "r"(bytes)
                 : "memory");
}
// TMA tile load of one CTA of a pair: data lands in this CTA, completion bytes go to a barrier that may
// live in the pair's other CTA (no multicast: every CTA fetches its own tile)
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar_cluster_addr,
                                                 int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(ptx::smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t* smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ptx::smem_u32(smem_dst)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// one arrival on the mbarrier at this offset in both CTAs of the pair once all MMAs issued so far have
// retired (two commits, each addressed through the cluster window to one CTA; no multicast qualifier)
__device__ __forceinline__ void commit_both(uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .b32 r0, r1;\n\t"
        "mapa.shared::cluster.u32 r0, %0, 0;\n\t"
        "mapa.shared::cluster.u32 r1, %0, 1;\n\t"
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [r0];\n\t"
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [r1];\n\t}"
        ::"r"(ptx::smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void mma2_f8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Four e4m3 bytes, two per conversion instruction.  The epilogue runs once per tile, from a cold instruction cache (7700 of
// a decode tile's 72000 cycles, 9500 of a full one's 84000): what counts is how many instructions it has.
__device__ __forceinline__ uint32_t pack_e4m3x4(float a, float b, float c, float d) {
    return (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3) |
           ((uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3) << 16);
}

// tile_prefix[e] = tiles of experts < e.  Every CTA starts with this, so the offsets are fetched by all threads at once
// and scanned from shared memory (a warp that walked the global array 32 experts at a time spent 3 us on 256 of them).
__device__ __forceinline__ void count_tiles(GemmSmem* sm, const GemmParams& p, int rows_per_tile, int n_tiles) {
    for (int e = threadIdx.x; e < p.E; e += GEMM_THREADS)
        sm->tile_prefix[e] = ((p.offsets[e + 1] - p.offsets[e] + rows_per_tile - 1) / rows_per_tile) * n_tiles;
}
__device__ __forceinline__ void scan_tiles(GemmSmem* sm, int E) {
    __syncthreads();                                          // the counts are there
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x, per = (E + 31) / 32, b = min(E, lane * per), n = min(E, b + per);
        int sum = 0;
        for (int e = b; e < n; e++) sum += sm->tile_prefix[e];
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        int before = incl - sum;
        for (int e = b; e < n; e++) {
            const int t = sm->tile_prefix[e];
            sm->tile_prefix[e] = before;
            before += t;
        }
        if (lane == 31) { sm->tile_prefix[E] = incl; sm->total_tiles = incl; }
    }
}

// The GEMMs are launched programmatically, GEMM1 behind the sort, GEMM2 behind GEMM1.  The offsets are the sort's: GEMM1 waits for it
// before it reads them.  GEMM2 starts only when every CTA of GEMM1 has passed that wait, so it may read the offsets, and fetch
// weights, while GEMM1 drains; whoever touches GEMM1's results or the output waits with wait_for_gemm1 first.
template <int MODE>
__device__ __forceinline__ void wait_for_sort() {
    if (MODE == 1) {
        ptx::grid_wait();
        ptx::grid_release();
    }
}
template <int MODE>
__device__ __forceinline__ void wait_for_gemm1() {
    if (MODE != 1) ptx::grid_wait();
}

// The rows of an A tile that exist, in whole groups of eight: a decode batch has a few rows per expert, and a full box of 128
// would bring the next experts' rows along, a third of the stage's bytes.  The rows of the stage that are not loaded hold
// zeros until a fuller tile has been there (clear_a_tiles), then older bytes; their products go to accumulator rows that
// nobody reads, but multiplying zeros takes less power, and under sustained load power is what sets the clock.  Groups
// of 32 and no zeros: T = 16 748 us, T = 333 1950 us, T = 1024 2024 us; with zeros 733, 1905, 2015.
__device__ __forceinline__ uint32_t a_tile_bytes(int rows) { return rows > BM - 8 ? (uint32_t)A_BYTES : (uint32_t)((rows + 7) >> 3) * 8u * BK; }
__device__ __forceinline__ void load_a_rows(uint8_t* dst, const CUtensorMap* map128, const CUtensorMap* map32, const CUtensorMap* map8, uint64_t* bar,
                                            int x, int row0, uint32_t bytes) {
    if (bytes == A_BYTES) {
        ptx::tma_load_2d(dst, map128, bar, x, row0);
    } else {
        uint32_t o = 0;
        for (; o + 32 * BK <= bytes; o += 32 * BK) ptx::tma_load_2d(dst + o, map32, bar, x, row0 + (int)(o / BK));
        for (; o < bytes; o += 8 * BK) ptx::tma_load_2d(dst + o, map8, bar, x, row0 + (int)(o / BK));
    }
}
__device__ __forceinline__ void clear_a_tiles(uint8_t* tiles) {
    for (int i = threadIdx.x; i < STAGES * A_BYTES / 16; i += GEMM_THREADS)
        *reinterpret_cast<uint4*>(tiles + (size_t)(i / (A_BYTES / 16)) * STAGE_BYTES + (i % (A_BYTES / 16)) * 16) = make_uint4(0, 0, 0, 0);
    ptx::fence_proxy_async_smem();
}
// acc[0..N-1] += v[0..N-1] * s, two columns per instruction (the same bits as N fmaf in half the issue slots: with the scales out
// of the loop T = 4096 3576 -> 3449 us, 32 experts x 1024 rows 2245 -> 2180 us)
template <int N>
__device__ __forceinline__ void promote(float* acc, const uint32_t (&v)[N], float s) {
    const unsigned long long s2 = ptx::pack_f32x2(s, s);
#pragma unroll
    for (int i = 0; i < N / 2; i++) {
        const unsigned long long r = ptx::fma_f32x2(ptx::pack_f32x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), s2,
                                                    ptx::pack_f32x2(acc[2 * i], acc[2 * i + 1]));
        ptx::unpack_f32x2(r, acc[2 * i], acc[2 * i + 1]);
    }
}

// MODE 1: the tile's 256 accumulator columns are NQ groups [gate j0+g*QCOLS/2 .. | up j0+g*QCOLS/2 ..]
// (j0 = 128 n_tile, QCOLS/2 columns each), so that the gate and the up value of an activation column
// meet in one thread.
// MODE 2/3: plain output columns 256 n_tile .. +255.
//
// PAIR: two CTAs of a cluster (two SMs) work on one tile of 256 rows with tcgen05.mma.cta_group::2: CTA r holds
// rows 128 r .. +127 (its own A tile and accumulator) and HALF of the tile's weight rows (accumulator columns
// 128 r .. +127), so per K block each SM writes and reads 32 KB of shared memory instead of 48 KB, and a
// weight tile crosses L2 -> shared memory once per 256 rows.  The leader CTA (rank 0) issues the MMAs; both CTAs'
// loads complete on the leader's `full` barrier, both CTAs' promotion warps release the accumulator stage on
// the leader's `tmem_empty` barrier, and tcgen05.commit signals `empty` / `tmem_full` in both CTAs.
//
// What bounds a K block (GEMM1, 32 experts x 1024 rows, single-CTA tiles, clock stamps): 880 cycles as built, 880 without any TMA
// load, 560 with the loads but promotion warps that only hand the stage back, 520 with neither, 840 without the multiplications.
// So it is the round trip of an accumulator stage -- MMAs, commit, tcgen05.ld, release -- with two stages to hide it in, not shared
// memory (96 KB per K block pass in the 560), the weight stream or the multiplications.
template <int MODE, bool PAIR>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
grouped_gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_a32,
                        const __grid_constant__ CUtensorMap tmap_a8, const __grid_constant__ CUtensorMap tmap_b, const GemmParams p) {
    constexpr int TM = PAIR ? 2 * BM : BM;        // rows of a tile
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    GemmSmem* sm = reinterpret_cast<GemmSmem*>(tiles + (size_t)STAGES * STAGE_BYTES);
    float (*const scales)[2][BM] = reinterpret_cast<float (*)[2][BM]>(sm + 1);
    int4* const tile_at = reinterpret_cast<int4*>(scales + SC_RING);
    volatile int* abort_flag = &sm->abort_flag;

    const int warp = ptx::uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int Kdim = (MODE == 1) ? p.D : p.I;
    const int nkb = Kdim / BK;
    const int NT = (MODE == 1) ? p.I / 128 : p.D / 256;     // N tiles per expert
    const int w_rows = (MODE == 1) ? 2 * p.I : p.D;         // weight rows per expert

    // ---- prologue ---------------------------------------------------------
    const uint32_t crank = PAIR ? cluster_ctarank() : 0u;     // 0 = leader
    const bool duo = !PAIR && cluster_nctarank() == 2;        // single-CTA tiles, launched two CTAs to a cluster
    const int pair_count = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;     // tile walkers
    const int walker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    if (threadIdx.x == 0) {
        // PAIR: the leader's `full` takes one arrive.expect_tx from each CTA's producer, its `tmem_empty` one
        // arrival from every promotion warp of both CTAs
        for (int s = 0; s < STAGES; s++) { ptx::mbar_init(&sm->full[s], PAIR ? 2 : 1); ptx::mbar_init(&sm->empty[s], 1); }
        for (int a = 0; a < 2; a++) {
            ptx::mbar_init(&sm->tmem_full[a], 2);             // the commit and the scale warp
            ptx::mbar_init(&sm->tmem_empty[a], PAIR ? 2 * NUM_PROMO_WARPS : NUM_PROMO_WARPS);
            ptx::mbar_init(&sm->amax_bar[a], NUM_PROMO_WARPS);
        }
        for (int i = 0; i < SC_RING; i++) ptx::mbar_init(&sm->sc_free[i], NUM_PROMO_WARPS);
        ptx::mbar_init(&sm->pair_go, 1);
        sm->abort_flag = 0;
        ptx::fence_mbar_init();
    }
    if (warp == W_MMA0) {
        if (PAIR) { tmem_alloc2(&sm->tmem_base, 512); tmem_relinquish2(); }
        else      { ptx::tmem_alloc(&sm->tmem_base, 512); ptx::tmem_relinquish(); }
    }
    if (warp == W_TMA && lane == 0) {
        ptx::prefetch_tensormap(&tmap_a);
        ptx::prefetch_tensormap(&tmap_a32);
        ptx::prefetch_tensormap(&tmap_a8);
        ptx::prefetch_tensormap(&tmap_b);
    }
    clear_a_tiles(tiles);
    wait_for_sort<MODE>();
    count_tiles(sm, p, TM, NT);
    ptx::tc_fence_before();
    scan_tiles(sm, p.E);
    __syncthreads();
    if (PAIR || duo) cluster_sync_all();      // the peer's barriers are initialised before anyone signals them
    ptx::tc_fence_after();
    const uint32_t tmem_base = sm->tmem_base;
    const int total_tiles = ptx::uniform(sm->total_tiles);

    // tile -> (expert, m_tile, n_tile): expert-major, then n, then m, so the CTAs that run
    // together walk through one expert's weights once.
    auto locate = [&](int tile, int& e, int& m_tile, int& n_tile, int& cnt) {
        int lo = 0, hi = p.E;
        while (hi - lo > 1) {
            int mid = (lo + hi) >> 1;
            if (sm->tile_prefix[mid] <= tile) lo = mid; else hi = mid;
        }
        // experts with zero tiles repeat the prefix value; the search lands on the last
        // expert whose prefix is <= tile, which is the one that owns tiles.
        e = ptx::uniform(lo);
        cnt = ptx::uniform(p.offsets[e + 1] - p.offsets[e]);
        int mt = (cnt + TM - 1) / TM;
        int local = tile - ptx::uniform(sm->tile_prefix[e]);
        n_tile = local / mt;
        m_tile = local - n_tile * mt;
    };

    if (warp >= NUM_PROMO_WARPS) {
        ptx::setmaxnreg_dec<AUX_REGS>();
      if (warp == W_TMA) {
        // ===================== TMA producer =====================
        {
            int s = 0; uint32_t ph = 0; int gk = 0; (void)gk;
            uint32_t go_ph = 0;
            const uint32_t peer_go = duo ? map_to_cta(&sm->pair_go, cluster_ctarank() ^ 1u) : 0u;
            for (int tile = walker; tile < total_tiles; tile += pair_count) {
                int e, m_tile, n_tile, cnt;
                locate(tile, e, m_tile, n_tile, cnt);
                if (duo && (tile | 1) < total_tiles) {        // the neighbour has a tile in this pass over the grid too
                    if (!ptx::whole_warp(pair_rendezvous(&sm->pair_go, peer_go, go_ph, abort_flag))) goto done;
                    go_ph ^= 1;
                }
                const int row0 = ptx::uniform(p.offsets[e]) + m_tile * TM + (int)crank * BM;
                const uint32_t a_bytes = a_tile_bytes(cnt - m_tile * TM);
                const long long wrow0 = (long long)e * w_rows;
                auto load_b = [&](int kb, int st) {              // expects the whole stage
                    uint8_t* b_dst = tiles + (size_t)st * STAGE_BYTES + A_BYTES;
                    if (!ptx::elect_one()) return;
                    if (PAIR) {
                        // this CTA's half of the weight tile (accumulator columns 128 crank .. +127); the bytes are counted on the
                        // leader's barrier
                        const uint32_t fbar = map_to_cta(&sm->full[st], 0);
                        mbar_expect_tx_cluster(fbar, A_BYTES + B_BYTES / 2);
                        if (p.packed) {
                            tma_load_2d_pair(b_dst, &tmap_b, fbar, 0, (((e * NT + n_tile) * nkb) + kb) * BN + (int)crank * 128);
                        } else if (MODE == 1) {
                            const int j0 = n_tile * 128 + 64 * (int)crank;
                            tma_load_2d_pair(b_dst, &tmap_b, fbar, kb * BK, (int)(wrow0 + j0));
                            tma_load_2d_pair(b_dst + 8192, &tmap_b, fbar, kb * BK, (int)(wrow0 + p.I + j0));
                        } else {
                            tma_load_2d_pair(b_dst, &tmap_b, fbar, kb * BK, (int)(wrow0 + n_tile * 256 + 128 * (int)crank));
                        }
                        return;
                    }
                    ptx::mbar_expect_tx(&sm->full[st], a_bytes + B_BYTES);
                    if (p.packed) {
                        // the tile's K block is one contiguous 32 KB piece of the packed weights
                        ptx::tma_load_2d(b_dst, &tmap_b, &sm->full[st], 0, (((e * NT + n_tile) * nkb) + kb) * BN);
                    } else if (MODE == 1) {
                        // 2 NQ boxes of QCOLS/2 weight rows: group g = [gate j0 + g QCOLS/2 .. | up j0 + g QCOLS/2 ..]
                        const int j0 = n_tile * 128;
#pragma unroll
                        for (int bx = 0; bx < 2 * NQ; bx++)
                            ptx::tma_load_2d(b_dst + bx * (QCOLS / 2) * 128, &tmap_b, &sm->full[st], kb * BK,
                                             (int)(wrow0 + ((bx & 1) ? p.I : 0) + j0 + (QCOLS / 2) * (bx >> 1)));
                    } else {
                        ptx::tma_load_2d(b_dst, &tmap_b, &sm->full[st], kb * BK, (int)(wrow0 + n_tile * 256));
                    }
                };
                int ready = 0;                                   // K blocks whose weights have been requested
                if (MODE != 1 && tile == walker) {
                    for (; ready < min(nkb, STAGES); ready++) load_b(ready, ready);
                    wait_for_gemm1<MODE>();
                }
                for (int kb = 0; kb < nkb; kb++) {
                    if (kb >= ready) {
                        if (!ptx::whole_warp(ptx::mbar_wait_relaxed(&sm->empty[s], ph ^ 1, abort_flag, PRODUCER_SLEEP_NS))) goto done;
                        TRACE_STAMP(6, gk);
                        load_b(kb, s);
                    }
                    gk++;
                    if (ptx::elect_one()) {
                        uint8_t* a_dst = tiles + (size_t)s * STAGE_BYTES;
                        if (PAIR) tma_load_2d_pair(a_dst, &tmap_a, map_to_cta(&sm->full[s], 0), kb * BK, row0);
                        else      load_a_rows(a_dst, &tmap_a, &tmap_a32, &tmap_a8, &sm->full[s], kb * BK, row0, a_bytes);
                    }
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
        }
      } else if (warp == W_MMA0 || warp == W_MMA0 + 1) {
        // ===================== MMA issuers =====================
        // Two issuers, one per TMEM stage (K blocks alternate between them).  The thread that issues a
        // K block's MMAs stays tied up until they have run (in the issue of the later ones and in the
        // commits); with a single issuer it came back to look at the other stage's "free" barrier
        // hundreds of cycles after the promotion warps had released it.
        if (crank == 0) {
            constexpr uint32_t idesc = ptx::make_idesc(0, 0, 0, 0, TM, BN);
            const int role = warp - W_MMA0;                 // the TMEM stage this issuer owns
            int s = 0; uint32_t ph = 0;
            uint32_t acc_ph = 0; long long g = 0;           // g: K blocks since the kernel started
            for (int tile = walker; tile < total_tiles; tile += pair_count) {
                for (int kb = 0; kb < nkb; kb++, g++) {
                    if ((int)(g & 1) == role) {
                        // The operands first: they are there long before the stage is handed back, which starts the critical path.
                        // (waits on barriers that the peer CTA or tcgen05.commit signal need no cluster-scope
                        // acquire: what they hand over is a TMEM stage or TMA-written tiles, not memory data)
                        if (!ptx::whole_warp(ptx::mbar_wait(&sm->full[s], ph, abort_flag))) goto done;
                        TRACE_STAMP(0, g);
                        const uint32_t a_addr = ptx::smem_u32(tiles + (size_t)s * STAGE_BYTES);
                        const uint64_t ad = ptx::make_smem_desc(a_addr, 16, 1024, 2), bd = ptx::make_smem_desc(a_addr + A_BYTES, 16, 1024, 2);
                        const uint32_t d_tmem = tmem_base + role * BN;
                        if (!ptx::whole_warp(ptx::mbar_wait(&sm->tmem_empty[role], acc_ph ^ 1, abort_flag))) goto done;
                        TRACE_STAMP(1, g);
                        ptx::tc_fence_after();
                        if (ptx::elect_one()) {
#pragma unroll
                            for (int k4 = 0; k4 < 4; k4++) {        // 32 bytes further along K: 2 in the descriptor's 16-byte units
                                if (PAIR) mma2_f8(d_tmem, ad + 2 * k4, bd + 2 * k4, idesc, k4 > 0 ? 1u : 0u);
                                else      ptx::mma_f8(d_tmem, ad + 2 * k4, bd + 2 * k4, idesc, k4 > 0 ? 1u : 0u);
                            }
                            if (PAIR) {
                                commit_both(&sm->tmem_full[role]);
                                commit_both(&sm->empty[s]);
                            } else {
                                ptx::tc_commit(&sm->tmem_full[role]);   // partial sums ready for promotion
                                ptx::tc_commit(&sm->empty[s]);          // smem stage reusable once the MMAs have read it
                            }
                        }
                        TRACE_STAMP(2, g);
                        acc_ph ^= 1;
                    }
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
        }
      } else {
        // ===================== scales =====================
        // a_scale[row, kb] * w_scale[block, kb] of the tile's 128 rows into shared memory, K block by K block.  Loaded by the
        // promotion warps themselves one K block ahead, the scales' latency (32 rows of a row-major matrix are 32 cache lines) was
        // longer than a K block: it held the warps back by different amounts, and the last one sets the pace.
        const int nkb_w = Kdim / 128;
        uint32_t g = 0, tiles_done = 0;                     // K blocks, tiles since the kernel started
        wait_for_gemm1<MODE>();
        for (int tile = walker; tile < total_tiles; tile += pair_count, tiles_done++) {
            int e, m_tile, n_tile, cnt;
            locate(tile, e, m_tile, n_tile, cnt);
            const int trow0 = m_tile * TM + (int)crank * BM, left = cnt - trow0 - lane;      // rows lane + 32 i exist for 32 i < left
            const int off = p.offsets[e];
            const float* a_sc = p.a_scale + (long long)off + trow0 + lane;
            const float *w0, *w1;
            if (MODE == 1) {
                w0 = p.w_scale + ((size_t)e * (2 * p.I / 128) + n_tile) * nkb_w;             // gate rows' block
                w1 = w0 + (size_t)(p.I / 128) * nkb_w;                                       // up rows' block
            } else {
                w0 = p.w_scale + ((size_t)e * (p.D / 128) + n_tile * 2) * nkb_w;             // columns 0 .. 127 of the tile
                w1 = w0 + nkb_w;                                                             // columns 128 .. 255
            }
            // two K blocks ahead
            float a[2][4], w[2][2];
            auto fetch = [&](int kb, float (&av)[4], float (&wv)[2]) {
                if (kb < nkb) {
#pragma unroll
                    for (int i = 0; i < 4; i++) av[i] = 32 * i < left ? a_sc[kb * p.a_ks + 32 * i] : 0.0f;
                    wv[0] = w0[kb];
                    wv[1] = w1[kb];
                }
            };
            auto publish = [&](float (&av)[4], float (&wv)[2], bool first) -> bool {
                // Block g - 2 is through with this barrier, and with single-CTA tiles the slot's last K block, g - 4, has been read: the
                // MMAs of block g - 2 waited for that.  In a pair the leader's MMAs wait on an arrival that orders no memory of the peer,
                // so there each CTA's promotion warps hand the slot back themselves.
                if (g >= 2 && !ptx::whole_warp(ptx::mbar_wait(&sm->tmem_full[g & 1], ((g >> 1) & 1) ^ 1, abort_flag))) return false;
                if (PAIR && g >= SC_RING && !ptx::whole_warp(ptx::mbar_wait(&sm->sc_free[g % SC_RING], ((g / SC_RING) & 1) ^ 1, abort_flag))) return false;
                float (*const sc)[BM] = scales[g % SC_RING];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    sc[0][lane + 32 * i] = av[i] * wv[0];
                    sc[1][lane + 32 * i] = av[i] * wv[1];
                }
                // (a tile has a K block at least: the slot's last tile, four tiles ago, has been read as well)
                if (first && lane == 0) tile_at[tiles_done % SC_RING] = make_int4(off, cnt, trow0, n_tile);
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&sm->tmem_full[g & 1]);
                g++;
                return true;
            };
            fetch(0, a[0], w[0]);
            fetch(1, a[1], w[1]);
            for (int kb = 0; kb < nkb; kb += 2) {
                if (!publish(a[0], w[0], kb == 0)) goto done;
                fetch(kb + 2, a[0], w[0]);
                if (kb + 1 < nkb) {
                    if (!publish(a[1], w[1], false)) goto done;
                    fetch(kb + 3, a[1], w[1]);
                }
            }
        }
      }
    } else {
        // ===================== promotion + epilogue (warps 0-7) =====================
        ptx::setmaxnreg_inc<PROMO_REGS>();
        // The warp polls as one instruction (one lane that polls and tells the others costs a shuffle and a reconvergence per K
        // block: 32 experts x 1024 rows 2169 -> 2092 us, T = 4096 3130 -> 3036, T = 16 765 -> 748).
        auto warp_wait = [&](uint64_t* bar, uint32_t parity) -> bool { return ptx::whole_warp(ptx::mbar_wait(bar, parity, abort_flag)); };
        const int wq = warp >> 2;                         // column group of the accumulator
        const int row = (warp & 3) * 32 + lane;           // TMEM lane = tile row
        const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
        int acc = 0; uint32_t acc_ph = 0;
        int tile_par = 0; uint32_t amax_ph[2] = {0, 0};
        int gp = 0; (void)gp;
#ifdef B200_GEMM_TRACE
        const bool trw = (threadIdx.x == p.trace_warp * 32);
#endif
        // the stage's "free" barrier lives in the leader CTA
        const uint32_t tmem_empty_addr[2] = {PAIR ? map_to_cta(&sm->tmem_empty[0], 0) : 0u,
                                             PAIR ? map_to_cta(&sm->tmem_empty[1], 0) : 0u};
        auto release_stage = [&](int a, uint32_t g) {                // one lane; all of the warp's reads are behind a __syncwarp
            if (PAIR) ptx::mbar_arrive(&sm->sc_free[g % SC_RING]);
            if (PAIR && crank != 0) mbar_arrive_cluster(tmem_empty_addr[a]);
            else                    ptx::mbar_arrive(&sm->tmem_empty[a]);
        };
        uint32_t gsc = 0, tiles_done = 0;                     // K blocks, tiles since the kernel started
        wait_for_gemm1<MODE>();
        for (int tile = walker; tile < total_tiles; tile += pair_count, tiles_done++) {
            // Where the tile lies comes with the scales of its first K block: looked up here, it took 1200 - 2500 cycles of the gap
            // between two tiles.
            if (!warp_wait(&sm->tmem_full[acc], acc_ph)) goto done;
            const int4 at = tile_at[tiles_done % SC_RING];
            const int off = at.x, cnt = at.y, trow0 = at.z, n_tile = at.w;        // trow0: first row of this CTA inside the expert
            const long long grow = (long long)off + trow0 + row;                  // sorted row
            const bool row_ok = (trow0 + row) < cnt;
            const bool warp_valid = (trow0 + (warp & 3) * 32) < cnt;              // any valid row in this warp's 32
            const float row_weight = (MODE != 1 && row_ok) ? p.row_w[grow] : 0.0f;     // used by the epilogue
            const int row_token = (MODE == 2 && row_ok) ? p.row_tok[grow] : -1;
            float accv[QCOLS];
#pragma unroll
            for (int i = 0; i < QCOLS; i++) accv[i] = 0.0f;

            for (int kb = 0; kb < nkb; kb++, gsc++) {
                if (kb > 0 && !warp_wait(&sm->tmem_full[acc], acc_ph)) goto done;
#ifdef B200_GEMM_TRACE
                if (trw) TRACE_STAMP(3, gp);
#endif
                if (warp_valid) {
                    // warps whose 32 rows are all padding only hand the stage back
                    ptx::tc_fence_after();
                    const float (*const sc)[BM] = scales[gsc % SC_RING];
                    const float s0 = (MODE == 1) ? sc[0][row] : sc[(wq * QCOLS) / 128][row], s1 = (MODE == 1) ? sc[1][row] : s0;
                    const uint32_t t0 = tmem_base + lane_addr + acc * BN + wq * QCOLS;
                    // QCOLS columns in chunks of CH, two loads in flight; columns [0, QCOLS/2) take s0 (MODE 1:
                    // gate), the rest s1 (MODE 1: up)
                    constexpr int NPAIR = QCOLS / (2 * CH);
                    uint32_t ra[CH], rb[CH];
#pragma unroll
                    for (int c = 0; c < NPAIR; c++) {
                        ptx::tmem_ld_32x32(t0 + 2 * c * CH, ra);
                        ptx::tmem_ld_32x32(t0 + 2 * c * CH + CH, rb);
                        ptx::tc_wait_ld();
                        if (c == NPAIR - 1) {
                            ptx::tc_fence_before();
                            __syncwarp();
                            if (lane == 0) release_stage(acc, gsc);   // the stage is in registers now
#ifdef B200_GEMM_TRACE
                            if (trw) TRACE_STAMP(4, gp);
#endif
                        }
                        promote<CH>(accv + 2 * c * CH, ra, (2 * c * CH < QCOLS / 2) ? s0 : s1);
                        promote<CH>(accv + (2 * c + 1) * CH, rb, ((2 * c + 1) * CH < QCOLS / 2) ? s0 : s1);
                    }
                } else {
                    ptx::tc_fence_before();
                    __syncwarp();                            // (every lane has read tile_at)
                    if (lane == 0) release_stage(acc, gsc);
                }
#ifdef B200_GEMM_TRACE
                if (trw) TRACE_STAMP(5, gp);
                gp++;
#endif
                if (++acc == 2) { acc = 0; acc_ph ^= 1; }
            }
#ifdef B200_GEMM_TRACE
            if (trw) TRACE_STAMP(7, gp / nkb - 1);     // end of the main loop of each tile; epilogue follows
#endif

            if (MODE == 1) {
                // SwiGLU on 64 activation columns, 1x128 requantisation shared with the other half's warp.
                // Fast exp / reciprocal: the result is rounded to e4m3 next, an ulp of fp32 does not matter.
                constexpr int AC = QCOLS / 2;          // activation columns of this thread
                float amax = 0.0f;
                if (warp_valid) {
#pragma unroll
                    for (int i = 0; i < AC; i++) {
                        const float g = accv[i], u = accv[AC + i];
                        const float a = __fdividef(g, 1.0f + __expf(-g)) * u;
                        accv[i] = a;
                        amax = fmaxf(amax, fabsf(a));
                    }
                }
                sm->amax[tile_par][wq][row] = amax;
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&sm->amax_bar[tile_par]);
                if (!warp_wait(&sm->amax_bar[tile_par], amax_ph[tile_par])) goto done;
                amax_ph[tile_par] ^= 1;
#pragma unroll
                for (int g = 0; g < NQ; g++) amax = fmaxf(amax, sm->amax[tile_par][g][row]);
                if (row_ok) {
                    const float scale = amax > 0.0f ? __fdiv_rn(amax, 448.0f) : 1.0f;
                    const float inv = amax > 0.0f ? __fdiv_rn(448.0f, amax) : 1.0f;
                    uint32_t packed[AC / 4];
#pragma unroll
                    for (int i = 0; i < AC / 4; i++) {
                        packed[i] = pack_e4m3x4(accv[4 * i] * inv, accv[4 * i + 1] * inv, accv[4 * i + 2] * inv, accv[4 * i + 3] * inv);
                    }
                    uint4* dst = reinterpret_cast<uint4*>(p.act_q + grow * p.I + n_tile * 128 + wq * AC);
#pragma unroll
                    for (int i = 0; i < AC / 16; i++)
                        dst[i] = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
                    if (wq == 0) p.act_s[grow * p.s_rs + n_tile * p.s_ks] = scale;
                }
                tile_par ^= 1;
            } else if (warp_valid && cnt - (trow0 + (warp & 3) * 32) <= DIRECT_ROWS) {
                // Few rows: each lane adds its own row.  With 1 or 2 rows that takes 700 cycles instead of 3700; a row is a cache line
                // per instruction, so with all 32 it is no faster than the transpose below (up to 8 / 16 / 32 rows: T = 333
                // 1888 / 1876 / 1876 us, T = 4096 2992 / 2985 / 3012, 32 experts x 1024 rows 1919 / 1915 / 1917).
                if (row_ok) {
                    float* const dst = p.out + (size_t)(MODE == 2 ? row_token : grow) * p.D + n_tile * 256 + wq * QCOLS;
#pragma unroll
                    for (int i = 0; i < QCOLS; i += 4) {
                        const float4 x = make_float4(row_weight * accv[i], row_weight * accv[i + 1], row_weight * accv[i + 2], row_weight * accv[i + 3]);
                        if (MODE == 2) red_add_v4(dst + i, x.x, x.y, x.z, x.w);
                        else *reinterpret_cast<float4*>(dst + i) = x;
                    }
                }
            } else if (warp_valid) {
                // The accumulator row of a lane is transposed through shared memory SW columns at a time so that
                // one store / red instruction covers 32 / SEGS rows x 16 SEGS contiguous bytes instead of 32 rows
                // x 16 bytes (fewer, larger memory requests).
                const float w = row_weight;
                float (*st)[SW + 4] = sm->stage[warp];
                constexpr int SEGS = SW / 4;
                const int sub_row = lane / SEGS, seg = lane % SEGS;
                const int tok = row_token;
                // MODE 2: out[token] += w * acc.  MODE 3: rows[sorted row] = w * acc (plain stores).
                const long long grow0 = (long long)off + trow0 + (warp & 3) * 32;
                const int rows_ok = min(32, cnt - (trow0 + (warp & 3) * 32));
                float* const out_col = p.out + n_tile * 256 + wq * QCOLS;
#pragma unroll
                for (int pass = 0; pass < QCOLS / SW; pass++) {
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < SEGS; q++) {
                        const float* a4 = accv + pass * SW + q * 4;
                        *reinterpret_cast<float4*>(&st[lane][q * 4]) = make_float4(w * a4[0], w * a4[1], w * a4[2], w * a4[3]);
                    }
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < SEGS; k++) {
                        const int r = (32 / SEGS) * k + sub_row;
                        const float4 x4 = *reinterpret_cast<const float4*>(&st[r][seg * 4]);
                        if (MODE == 2) {
                            const int tok_r = __shfl_sync(0xffffffffu, tok, r);
                            if (tok_r >= 0)
                                red_add_v4(out_col + (size_t)tok_r * p.D + pass * SW + seg * 4, x4.x, x4.y, x4.z, x4.w);
                        } else if (r < rows_ok) {
                            *reinterpret_cast<float4*>(out_col + (size_t)(grow0 + r) * p.D + pass * SW + seg * 4) = x4;
                        }
                    }
                }
            }
        }
    }
done:
    ptx::tc_fence_before();
    __syncthreads();
    if (PAIR || duo) cluster_sync_all();     // the pair's MMAs, remote arrivals and TMEM reads are over in both CTAs
    if (warp == W_MMA0) {
        if (PAIR) tmem_dealloc2(tmem_base, 512);
        else      ptx::tmem_dealloc(tmem_base, 512);
    }
    if (threadIdx.x == 0 && sm->abort_flag) atomicExch(p.status, B200_TIMEOUT);
}

// -------------------------------------------------------------------------------------------------
// The same grouped GEMMs for power-of-two scales (B200_MOE_POW2_SCALES) on the hardware block-scaled MMA
// (tcgen05.mma kind::mxf8f6f4.block_scale, UE8M0 scale = the exponent byte of the fp32 scale): the tensor core
// multiplies every 32-deep slice of a row by its scale itself, so the accumulator of a tile stays in TMEM
// for the whole K loop, nothing is promoted in software and the K-block period is the MMA's own (or the
// weight stream's).  Differences from the kernel above:
//   * warp 10 builds the scale factors of every stage in shared memory: a 512-byte atom for the 128 rows of A
//     (row r -> byte (r % 32) * 16 + (r / 32) * 4 + step, four K = 32 steps of the 128-deep block share the
//     scale) and two atoms for the 256 rows of B (all rows of a 128-column weight block share its scale); it
//     also checks that every scale it sees is a power of two (B200_BAD_SCALE otherwise);
//   * the MMA warp copies the atoms into TMEM (tcgen05.cp 32x128b.warpx4: 4 + 8 columns per stage, at columns
//     256 + 16 stage) and issues the four MMAs of the K block with scale ids 0..3;
//   * ONE 256-column accumulator: the eight epilogue warps add it into registers (128 columns per thread) every
//     MX_FLUSH K blocks and free it at once, so the next segment's (or tile's) MMAs run under the additions and
//     the epilogue;
//   * GEMM1 requantises with a power-of-two scale as well.
// Single-CTA tiles only.
// -------------------------------------------------------------------------------------------------
template <int MODE>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
grouped_gemm_mx_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_a32,
                       const __grid_constant__ CUtensorMap tmap_a8, const __grid_constant__ CUtensorMap tmap_b, const GemmParams p) {
    constexpr int W_SF = W_MMA0 + 1;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sf_area = tiles + (size_t)STAGES * STAGE_BYTES;
    GemmSmem* sm = reinterpret_cast<GemmSmem*>(sf_area + (size_t)STAGES * SF_BYTES);
    volatile int* abort_flag = &sm->abort_flag;

    const int warp = ptx::uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int Kdim = (MODE == 1) ? p.D : p.I;
    const int nkb = Kdim / BK;
    const int NT = (MODE == 1) ? p.I / 128 : p.D / 256;     // N tiles per expert
    const int w_rows = (MODE == 1) ? 2 * p.I : p.D;         // weight rows per expert
    const int walkers = (int)gridDim.x, walker = (int)blockIdx.x;
    const bool duo = cluster_nctarank() == 2;               // launched two CTAs to a cluster

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            ptx::mbar_init(&sm->full[s], 1);
            ptx::mbar_init(&sm->empty[s], 1);
            ptx::mbar_init(&sm->sf_full[s], 1);
        }
        ptx::mbar_init(&sm->pair_go, 1);
        ptx::mbar_init(&sm->tmem_full[0], 1);
        ptx::mbar_init(&sm->tmem_empty[0], NUM_PROMO_WARPS);
        for (int a = 0; a < 2; a++) ptx::mbar_init(&sm->amax_bar[a], NUM_PROMO_WARPS);
        sm->abort_flag = 0;
        ptx::fence_mbar_init();
    }
    if (warp == W_MMA0) { ptx::tmem_alloc(&sm->tmem_base, 512); ptx::tmem_relinquish(); }
    if (warp == W_TMA && lane == 0) {
        ptx::prefetch_tensormap(&tmap_a);
        ptx::prefetch_tensormap(&tmap_a32);
        ptx::prefetch_tensormap(&tmap_a8);
        ptx::prefetch_tensormap(&tmap_b);
    }
    clear_a_tiles(tiles);
    wait_for_sort<MODE>();
    count_tiles(sm, p, BM, NT);
    ptx::tc_fence_before();
    scan_tiles(sm, p.E);
    __syncthreads();
    if (duo) cluster_sync_all();              // the neighbour's barrier is initialised before anyone signals it
    ptx::tc_fence_after();
    const uint32_t tmem_base = sm->tmem_base;
    const int total_tiles = ptx::uniform(sm->total_tiles);

    auto locate = [&](int tile, int& e, int& m_tile, int& n_tile, int& cnt) {
        int lo = 0, hi = p.E;
        while (hi - lo > 1) {
            int mid = (lo + hi) >> 1;
            if (sm->tile_prefix[mid] <= tile) lo = mid; else hi = mid;
        }
        e = ptx::uniform(lo);
        cnt = ptx::uniform(p.offsets[e + 1] - p.offsets[e]);
        int mt = (cnt + BM - 1) / BM;
        int local = tile - ptx::uniform(sm->tile_prefix[e]);
        n_tile = local / mt;
        m_tile = local - n_tile * mt;
    };
    auto warp_wait = [&](uint64_t* bar, uint32_t parity) -> bool { return ptx::whole_warp(ptx::mbar_wait(bar, parity, abort_flag)); };

    if (warp >= NUM_PROMO_WARPS) {
        ptx::setmaxnreg_dec<AUX_REGS>();
      if (warp == W_TMA) {
        // ===================== TMA producer (operand tiles) =====================
        {
            int s = 0; uint32_t ph = 0, go_ph = 0;
            const uint32_t peer_go = duo ? map_to_cta(&sm->pair_go, cluster_ctarank() ^ 1u) : 0u;
            for (int tile = walker; tile < total_tiles; tile += walkers) {
                int e, m_tile, n_tile, cnt;
                locate(tile, e, m_tile, n_tile, cnt);
                if (duo && (tile | 1) < total_tiles) {        // the neighbour has a tile in this pass over the grid too
                    if (!ptx::whole_warp(pair_rendezvous(&sm->pair_go, peer_go, go_ph, abort_flag))) goto done;
                    go_ph ^= 1;
                }
                const int row0 = ptx::uniform(p.offsets[e]) + m_tile * BM;
                const uint32_t a_bytes = a_tile_bytes(cnt - m_tile * BM);
                const long long wrow0 = (long long)e * w_rows;
                auto load_b = [&](int kb, int st) {              // expects the whole stage
                    uint8_t* b_dst = tiles + (size_t)st * STAGE_BYTES + A_BYTES;
                    if (!ptx::elect_one()) return;
                    ptx::mbar_expect_tx(&sm->full[st], a_bytes + B_BYTES);
                    if (p.packed) {
                        ptx::tma_load_2d(b_dst, &tmap_b, &sm->full[st], 0, (((e * NT + n_tile) * nkb) + kb) * BN);
                    } else if (MODE == 1) {
                        const int j0 = n_tile * 128;
#pragma unroll
                        for (int bx = 0; bx < 2 * NQ; bx++)
                            ptx::tma_load_2d(b_dst + bx * (QCOLS / 2) * 128, &tmap_b, &sm->full[st], kb * BK,
                                             (int)(wrow0 + ((bx & 1) ? p.I : 0) + j0 + (QCOLS / 2) * (bx >> 1)));
                    } else {
                        ptx::tma_load_2d(b_dst, &tmap_b, &sm->full[st], kb * BK, (int)(wrow0 + n_tile * 256));
                    }
                };
                int ready = 0;                                   // K blocks whose weights have been requested
                if (MODE != 1 && tile == walker) {
                    for (; ready < min(nkb, STAGES); ready++) load_b(ready, ready);
                    wait_for_gemm1<MODE>();
                }
                for (int kb = 0; kb < nkb; kb++) {
                    if (kb >= ready) {
                        if (!ptx::whole_warp(ptx::mbar_wait_relaxed(&sm->empty[s], ph ^ 1, abort_flag, PRODUCER_SLEEP_NS))) goto done;
                        load_b(kb, s);
                    }
                    if (ptx::elect_one())
                        load_a_rows(tiles + (size_t)s * STAGE_BYTES, &tmap_a, &tmap_a32, &tmap_a8, &sm->full[s], kb * BK, row0, a_bytes);
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
        }
      } else if (warp == W_MMA0) {
        // ===================== scale copies + MMAs =====================
        {
            int s = 0; uint32_t ph = 0, tph = 0;
            for (int tile = walker; tile < total_tiles; tile += walkers) {
              for (int kb0 = 0; kb0 < nkb; kb0 += MX_FLUSH) {
                // the epilogue warps have added the previous segment (or tile) into their registers
                if (!ptx::whole_warp(ptx::mbar_wait(&sm->tmem_empty[0], tph ^ 1, abort_flag))) goto done;
                ptx::tc_fence_after();
                const int kb1 = min(nkb, kb0 + MX_FLUSH);
                for (int kb = kb0; kb < kb1; kb++) {
                    if (!ptx::whole_warp(ptx::mbar_wait(&sm->full[s], ph, abort_flag))) goto done;
                    if (!ptx::whole_warp(ptx::mbar_wait(&sm->sf_full[s], ph, abort_flag))) goto done;
                    ptx::tc_fence_after();
                    const uint32_t a_addr = ptx::smem_u32(tiles + (size_t)s * STAGE_BYTES);
                    const uint64_t ad = ptx::make_smem_desc(a_addr, 16, 1024, 2), bd = ptx::make_smem_desc(a_addr + A_BYTES, 16, 1024, 2);
                    const uint64_t sd = ptx::make_smem_desc(ptx::smem_u32(sf_area + (size_t)s * SF_BYTES), 16, 128, 0);
                    const uint32_t tsfa = tmem_base + BN + 16 * s, tsfb = tsfa + 4;
                    if (ptx::elect_one()) {
                        ptx::tmem_cp_32x128b_warpx4(tsfa, sd);
                        ptx::tmem_cp_32x128b_warpx4(tsfb, sd + 512 / 16);
                        ptx::tmem_cp_32x128b_warpx4(tsfb + 4, sd + 1024 / 16);
#pragma unroll
                        for (int k4 = 0; k4 < 4; k4++)
                            ptx::mma_mxf8(tmem_base, ad + 2 * k4, bd + 2 * k4, ptx::make_idesc_mx(BM, BN, k4, k4), tsfa, tsfb,
                                          (kb > kb0 || k4 > 0) ? 1u : 0u);
                        ptx::tc_commit(&sm->empty[s]);          // operand tiles, scale atoms and their TMEM copies reusable
                    }
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
                if (ptx::elect_one()) ptx::tc_commit(&sm->tmem_full[0]);
                tph ^= 1;
              }
            }
        }
      } else if (warp == W_SF) {
        // ===================== scale factors of every stage =====================
        int s = 0; uint32_t ph = 0;
        uint32_t bad = 0;
        wait_for_gemm1<MODE>();
        auto expo = [&](float f) -> uint32_t {
            const uint32_t b = __float_as_uint(f);
            bad |= (b & 0x807FFFFFu) | (((b >> 23) == 0u) ? 1u : 0u);     // sign, mantissa bits, zero / denormal
            return ((b >> 23) & 0xFFu) * 0x01010101u;                    // the UE8M0 byte, once per K = 32 step
        };
        const int nkb_w = Kdim / 128;
        for (int tile = walker; tile < total_tiles; tile += walkers) {
            int e, m_tile, n_tile, cnt;
            locate(tile, e, m_tile, n_tile, cnt);
            const float* a_sc[4];
            bool ok[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int r = m_tile * BM + lane + 32 * q;
                ok[q] = r < cnt;
                a_sc[q] = p.a_scale + (ok[q] ? (long long)p.offsets[e] + r : 0);
            }
            const float* w_sc0;
            const float* w_sc1;
            if (MODE == 1) {
                const float* base = p.w_scale + (size_t)e * (2 * p.I / 128) * nkb_w;
                w_sc0 = base + (size_t)n_tile * nkb_w;                     // gate rows' block
                w_sc1 = base + (size_t)(p.I / 128 + n_tile) * nkb_w;       // up rows' block
            } else {
                const float* base = p.w_scale + (size_t)e * (p.D / 128) * nkb_w;
                w_sc0 = base + (size_t)(n_tile * 2) * nkb_w;               // columns 0..127 of the tile
                w_sc1 = w_sc0 + nkb_w;                                     // columns 128..255
            }
            float an[4], w0n = w_sc0[0], w1n = w_sc1[0];
#pragma unroll
            for (int q = 0; q < 4; q++) an[q] = ok[q] ? a_sc[q][0] : 1.0f;
            for (int kb = 0; kb < nkb; kb++) {
                const float a0 = an[0], a1 = an[1], a2 = an[2], a3 = an[3], w0 = w0n, w1 = w1n;
                if (kb + 1 < nkb) {
#pragma unroll
                    for (int q = 0; q < 4; q++) an[q] = ok[q] ? a_sc[q][(kb + 1) * p.a_ks] : 1.0f;
                    w0n = w_sc0[kb + 1];
                    w1n = w_sc1[kb + 1];
                }
                if (!warp_wait(&sm->empty[s], ph ^ 1)) goto done;
                const uint32_t sfp = ptx::smem_u32(sf_area + (size_t)s * SF_BYTES) + lane * 16;
                const uint32_t g = expo(w0), u = expo(w1);
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sfp), "r"(expo(a0)), "r"(expo(a1)), "r"(expo(a2)), "r"(expo(a3)) : "memory");
                if (MODE == 1) {
                    // accumulator columns [gate 64 | up 64 | gate 64 | up 64]
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sfp + 512), "r"(g), "r"(g), "r"(u), "r"(u) : "memory");
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sfp + 1024), "r"(g), "r"(g), "r"(u), "r"(u) : "memory");
                } else {
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sfp + 512), "r"(g), "r"(g), "r"(g), "r"(g) : "memory");
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sfp + 1024), "r"(u), "r"(u), "r"(u), "r"(u) : "memory");
                }
                ptx::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&sm->sf_full[s]);
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
        }
        if (__any_sync(0xffffffffu, bad != 0) && lane == 0) atomicExch(p.status, B200_BAD_SCALE);
      }
    } else {
        // ===================== epilogue (warps 0-7) =====================
        ptx::setmaxnreg_inc<PROMO_REGS>();
        const int wq = warp >> 2;                         // column half of the accumulator
        const int row = (warp & 3) * 32 + lane;           // TMEM lane = tile row
        const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
        uint32_t fph = 0;
        int tile_par = 0; uint32_t amax_ph[2] = {0, 0};
        wait_for_gemm1<MODE>();
        for (int tile = walker; tile < total_tiles; tile += walkers) {
            int e, m_tile, n_tile, cnt;
            locate(tile, e, m_tile, n_tile, cnt);
            const int trow0 = m_tile * BM;
            const long long grow = (long long)p.offsets[e] + trow0 + row;         // sorted row
            const bool row_ok = (trow0 + row) < cnt;
            const bool warp_valid = (trow0 + (warp & 3) * 32) < cnt;              // any valid row in this warp's 32
            float accv[QCOLS];
#pragma unroll
            for (int i = 0; i < QCOLS; i++) accv[i] = 0.0f;
            for (int kb0 = 0; kb0 < nkb; kb0 += MX_FLUSH) {
                if (!warp_wait(&sm->tmem_full[0], fph)) goto done;
                fph ^= 1;
                ptx::tc_fence_after();
                if (warp_valid) {
                    const uint32_t t0 = tmem_base + lane_addr + wq * QCOLS;
#pragma unroll
                    for (int c = 0; c < QCOLS / 32; c++) {
                        uint32_t r[32];
                        ptx::tmem_ld_32x32(t0 + 32 * c, r);
                        ptx::tc_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; i++) accv[32 * c + i] += __uint_as_float(r[i]);
                    }
                }
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&sm->tmem_empty[0]);  // the segment is in registers: the MMAs may go on
            }

            if (MODE == 1) {
                constexpr int AC = QCOLS / 2;          // activation columns of this thread
                float amax = 0.0f;
                if (warp_valid) {
#pragma unroll
                    for (int i = 0; i < AC; i++) {
                        const float g = accv[i], u = accv[AC + i];
                        const float a = __fdividef(g, 1.0f + __expf(-g)) * u;
                        accv[i] = a;
                        amax = fmaxf(amax, fabsf(a));
                    }
                }
                sm->amax[tile_par][wq][row] = amax;
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&sm->amax_bar[tile_par]);
                if (!warp_wait(&sm->amax_bar[tile_par], amax_ph[tile_par])) goto done;
                amax_ph[tile_par] ^= 1;
#pragma unroll
                for (int g = 0; g < NQ; g++) amax = fmaxf(amax, sm->amax[tile_par][g][row]);
                if (row_ok) {
                    // power-of-two scale: the reciprocal is exact
                    const float scale = amax > 0.0f ? ptx::pow2_scale_bits(__fdiv_rn(amax, 448.0f)) : 1.0f;
                    const float inv = __fdiv_rn(1.0f, scale);
                    uint32_t packed[AC / 4];
#pragma unroll
                    for (int i = 0; i < AC / 4; i++) {
                        packed[i] = pack_e4m3x4(accv[4 * i] * inv, accv[4 * i + 1] * inv, accv[4 * i + 2] * inv, accv[4 * i + 3] * inv);
                    }
                    uint4* dst = reinterpret_cast<uint4*>(p.act_q + grow * p.I + n_tile * 128 + wq * AC);
#pragma unroll
                    for (int i = 0; i < AC / 16; i++)
                        dst[i] = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
                    if (wq == 0) p.act_s[grow * p.s_rs + n_tile * p.s_ks] = scale;
                }
                tile_par ^= 1;
            } else if (warp_valid) {
                const float w = row_ok ? p.row_w[grow] : 0.0f;
                float (*st)[SW + 4] = sm->stage[warp];
                constexpr int SEGS = SW / 4;
                const int sub_row = lane / SEGS, seg = lane % SEGS;
                const int tok = (MODE == 2 && row_ok) ? p.row_tok[grow] : -1;
                const long long grow0 = (long long)p.offsets[e] + trow0 + (warp & 3) * 32;
                const int rows_ok = min(32, cnt - (trow0 + (warp & 3) * 32));
                float* const out_col = p.out + n_tile * 256 + wq * QCOLS;
#pragma unroll
                for (int pass = 0; pass < QCOLS / SW; pass++) {
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < SEGS; q++) {
                        const float* a4 = accv + pass * SW + q * 4;
                        *reinterpret_cast<float4*>(&st[lane][q * 4]) = make_float4(w * a4[0], w * a4[1], w * a4[2], w * a4[3]);
                    }
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < SEGS; k++) {
                        const int r = (32 / SEGS) * k + sub_row;
                        const float4 x4 = *reinterpret_cast<const float4*>(&st[r][seg * 4]);
                        if (MODE == 2) {
                            const int tok_r = __shfl_sync(0xffffffffu, tok, r);
                            if (tok_r >= 0)
                                red_add_v4(out_col + (size_t)tok_r * p.D + pass * SW + seg * 4, x4.x, x4.y, x4.z, x4.w);
                        } else if (r < rows_ok) {
                            *reinterpret_cast<float4*>(out_col + (size_t)(grow0 + r) * p.D + pass * SW + seg * 4) = x4;
                        }
                    }
                }
            }
        }
    }
done:
    ptx::tc_fence_before();
    __syncthreads();
    if (duo) cluster_sync_all();              // no remote arrival is in flight towards a CTA that has left
    if (warp == W_MMA0) ptx::tmem_dealloc(tmem_base, 512);
    if (threadIdx.x == 0 && sm->abort_flag) atomicExch(p.status, B200_TIMEOUT);
}

// Deterministic combine: out[t,:] = sum over the token's K slots, in ascending expert order (ties cannot
// occur: an expert appears at most once per token), of rows[row_of_pair[t*K+k],:].  One block per token.
__global__ void __launch_bounds__(256)
reduce_rows_kernel(const float* __restrict__ rows, const int* __restrict__ pair_row, const int* __restrict__ ids,
                   int K, int D, float* __restrict__ out) {
    const int t = blockIdx.x;
    __shared__ int order[64];
    if (threadIdx.x == 0) {
        // slots sorted by expert id (K <= 64), skipped slots (row < 0) dropped
        int n = 0;
        for (int k = 0; k < K; k++)
            if (pair_row[t * K + k] >= 0) order[n++] = k;
        for (int i = 1; i < n; i++) {
            const int kk = order[i];
            int j = i - 1;
            while (j >= 0 && ids[t * K + order[j]] > ids[t * K + kk]) { order[j + 1] = order[j]; j--; }
            order[j + 1] = kk;
        }
        for (int i = n; i < K; i++) order[i] = -1;
    }
    __syncthreads();
    for (int c = threadIdx.x * 4; c < D; c += blockDim.x * 4) {
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int i = 0; i < K; i++) {
            const int k = order[i];
            if (k < 0) break;
            const float4 v = *reinterpret_cast<const float4*>(rows + (size_t)pair_row[t * K + k] * D + c);
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        *reinterpret_cast<float4*>(out + (size_t)t * D + c) = acc;
    }
}

// 128 threads copy a row, four 16-byte loads in flight per thread
__device__ __forceinline__ void copy_row(uint4* __restrict__ dst, const uint4* __restrict__ src, int n) {
    for (int i0 = threadIdx.x; i0 < n; i0 += 512) {
        uint4 v[4];
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (i0 + 128 * j < n) v[j] = __ldg(src + i0 + 128 * j);
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (i0 + 128 * j < n) dst[i0 + 128 * j] = v[j];
    }
}

// Expert-sorted copy of the FP8 rows.  One block per sorted row, grid-stride (the number of valid
// rows is only known on the device: slots owned by other ranks are not rows).
__global__ void __launch_bounds__(128)
sort_rows_fp8_kernel(const uint8_t* __restrict__ xq, const float* __restrict__ xs, const int* __restrict__ row_pair,
                     const int* __restrict__ offsets, const float* __restrict__ wts, int E, int K, int D,
                     uint8_t* __restrict__ sq, float* __restrict__ ss, long long s_ks, int* __restrict__ row_tok,
                     float* __restrict__ row_w, int* __restrict__ pair_row) {
    ptx::grid_wait();
    ptx::grid_release();
    const int total = offsets[E];
    const int nb = D / 128;
    for (int r = blockIdx.x; r < total; r += gridDim.x) {
        const int pair = row_pair[r];
        const int tok = pair / K;
        const uint4* src = reinterpret_cast<const uint4*>(xq + (size_t)tok * D);
        uint4* dst = reinterpret_cast<uint4*>(sq + (size_t)r * D);
        copy_row(dst, src, D / 16);
        for (int i = threadIdx.x; i < nb; i += blockDim.x) ss[i * s_ks + r] = xs[(size_t)tok * nb + i];
        if (threadIdx.x == 0) {
            row_tok[r] = tok;
            row_w[r] = wts[pair];
            if (pair_row) pair_row[pair] = r;      // deterministic combine: sorted row of (token, slot)
        }
    }
}

// Permutation, expert-sorted copy and zero-fill of the output in one launch for short id lists of this library's own
// router (T * K <= SMALL_PAIRS; negative ids are not rows).  One block per (token, slot): its sorted row is the number
// of pairs that come before it (lower expert, or the same expert and a lower pair), counted from the list itself -- a
// few KB that every block reads -- instead of by a permutation kernel in front (decode batches are bound by the chain
// of launches, not by this work).  The block also clears its 1/K of the token's output row; one more block writes the
// experts' offsets.  With the router tiles and programmatic launches: E = 256, K = 8, D = 7168 layer at T = 1 175 -> 131 us,
// T = 16 963 -> 921 us.
constexpr int SMALL_PAIRS = 2048;
__global__ void __launch_bounds__(128)
sort_small_fp8_kernel(const uint8_t* __restrict__ xq, const float* __restrict__ xs, const int* __restrict__ ids,
                      const float* __restrict__ wts, int TK, int E, int K, int D, int* __restrict__ offsets,
                      uint8_t* __restrict__ sq, float* __restrict__ ss, long long s_ks, int* __restrict__ row_tok,
                      float* __restrict__ row_w, int* __restrict__ pair_row, float* __restrict__ out) {
    __shared__ int s_cnt[MAX_E];
    __shared__ int s_warp[4];
    ptx::grid_wait();
    ptx::grid_release();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if ((int)blockIdx.x == TK) {
        for (int e = tid; e < E; e += 128) s_cnt[e] = 0;
        __syncthreads();
        for (int i = tid; i < TK; i += 128) {
            const int id = ids[i];
            if (id >= 0 && id < E) atomicAdd(&s_cnt[id], 1);
        }
        __syncthreads();
        if (warp == 0) {
            int running = 0;
            for (int e0 = 0; e0 < E; e0 += 32) {
                const int c = (e0 + lane < E) ? s_cnt[e0 + lane] : 0;
                int incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                if (e0 + lane < E) offsets[e0 + lane] = running + incl - c;
                running += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) offsets[E] = running;
        }
        return;
    }
    const int pair = blockIdx.x, tok = pair / K, k = pair - tok * K;
    if (out) {
        const int d4 = D / 4, b = (int)((long long)d4 * k / K), e4 = (int)((long long)d4 * (k + 1) / K);
        float4* dst = reinterpret_cast<float4*>(out + (size_t)tok * D);
        for (int i = b + tid; i < e4; i += 128) dst[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const int mine = ids[pair];
    if (mine < 0 || mine >= E) {
        if (tid == 0 && pair_row) pair_row[pair] = -1;
        return;
    }
    int before = 0;
    for (int i = tid; i < TK; i += 128) {
        const int id = ids[i];
        before += (id >= 0 && (id < mine || (id == mine && i < pair))) ? 1 : 0;
    }
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) s_warp[warp] = before;
    __syncthreads();
    const int r = s_warp[0] + s_warp[1] + s_warp[2] + s_warp[3];
    const int nb = D / 128;
    const uint4* src = reinterpret_cast<const uint4*>(xq + (size_t)tok * D);
    uint4* dst = reinterpret_cast<uint4*>(sq + (size_t)r * D);
    copy_row(dst, src, D / 16);
    for (int i = tid; i < nb; i += 128) ss[i * s_ks + r] = xs[(size_t)tok * nb + i];
    if (tid == 0) {
        row_tok[r] = tok;
        row_w[r] = wts[pair];
        if (pair_row) pair_row[pair] = r;
    }
}

// Optional per-kernel timing: CUDA events recorded on the launch stream around the two grouped
// GEMMs (used by the benchmark for the roofline line; off by default).  The record belongs to the
// workspace, so host threads that drive different GPUs (or different workspaces) do not share it.
constexpr int PROF_SLOTS = 256;
}  // namespace
struct b200_gemm_profile {
    bool on = false;
    cudaEvent_t ev[PROF_SLOTS][4];
    long long calls = 0;      // layer calls recorded since profiling was enabled
};
namespace {

__global__ void pack_weights_kernel(int which, const uint8_t* __restrict__ src, uint8_t* __restrict__ packed, int E,
                                    int D, int I, long long chunks) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= chunks) return;
    const int Kdim = which == 1 ? D : I;
    const int nkb = Kdim / 128;
    const int NT = which == 1 ? I / 128 : D / 256;
    const int c16 = (int)(i & 7);
    const int r = (int)((i >> 3) & 255);
    long long t = i >> 11;
    const int kb = (int)(t % nkb); t /= nkb;
    const int nt = (int)(t % NT);
    const int e = (int)(t / NT);
    long long row;
    if (which == 1) {
        // group g of the tile's 256 rows = [gate j0 + g QCOLS/2 .. | up j0 + g QCOLS/2 ..], QCOLS/2 rows each
        const int j0 = nt * 128, g = r / QCOLS, up = (r / (QCOLS / 2)) & 1, rr = r % (QCOLS / 2);
        row = (long long)e * 2 * I + (up ? I : 0) + j0 + (QCOLS / 2) * g + rr;
    } else {
        row = (long long)e * D + nt * 256 + r;
    }
    const uint4 v = *reinterpret_cast<const uint4*>(src + row * Kdim + (long long)kb * 128 + c16 * 16);
    *reinterpret_cast<uint4*>(packed + i * 16) = v;
}

struct Fp8Scratch {
    RouteScratch route; int* ids; float* wts; int* range_hist; int* counts; int* offsets; int* row_pair;
    uint8_t* sq; float* ss; int* row_tok; float* row_w; uint8_t* act_q; float* act_s;
    int* pair_row; float* rows;     // deterministic combine only
};

void carve_fp8(WsCarver& c, const b200_moe_fp8_config* cfg, bool with_route, Fp8Scratch& s) {
    const size_t T = cfg->num_tokens, E = cfg->num_experts, K = cfg->top_k, D = cfg->hidden_dim,
                 I = cfg->intermediate_dim;
    const size_t TK = T * K;
    s.route = RouteScratch{};
    if (with_route) {
        const bool tc = moe_gate_tc_supported((int)T, (int)E, (int)D);
        s.route.partials = c.take<float>((size_t)max(moe_gate_chunks((int)D, true), moe_gate_tc_slots((int)D)) * T * E);
        s.route.whi = tc ? c.take<float>(E * D) : nullptr;
        s.route.wlo = tc ? c.take<float>(E * D) : nullptr;
        s.route.flag_list = tc ? c.take<int>(T) : nullptr;
        s.route.flag_n = tc ? c.take<int>(1) : nullptr;
    }
    s.ids = c.take<int>(TK);
    s.wts = c.take<float>(TK);
    s.range_hist = c.take<int>(permute_ranges_scratch_ints((int)T, (int)K, (int)E));
    s.counts = c.take<int>(E);
    s.offsets = c.take<int>(E + 1);
    s.row_pair = c.take<int>(TK);
    s.sq = c.take<uint8_t>(TK * D);
    s.ss = c.take<float>(TK * (D / 128));
    s.row_tok = c.take<int>(TK);
    s.row_w = c.take<float>(TK);
    s.act_q = c.take<uint8_t>(TK * I);
    s.act_s = c.take<float>(TK * (I / 128));
    const bool det = (cfg->flags & B200_MOE_DETERMINISTIC) != 0;
    s.pair_row = det ? c.take<int>(TK) : nullptr;
    s.rows = det ? c.take<float>(TK * D) : nullptr;
}

int check_fp8_cfg(const b200_moe_fp8_config* cfg) {
    if (!cfg) return B200_BAD_ARG;
    if (cfg->num_tokens <= 0 || cfg->num_experts <= 0 || cfg->top_k <= 0) return B200_BAD_SHAPE;
    if (cfg->hidden_dim <= 0 || cfg->intermediate_dim <= 0) return B200_BAD_SHAPE;
    if (cfg->hidden_dim % 256 || cfg->intermediate_dim % 128) return B200_BAD_SHAPE;
    if (cfg->num_experts > MAX_E) return B200_UNSUPPORTED;
    if ((cfg->flags & B200_MOE_DETERMINISTIC) && cfg->top_k > 64) return B200_UNSUPPORTED;
    if ((long long)cfg->num_experts * 2 * cfg->intermediate_dim > 0x7fffffffLL) return B200_UNSUPPORTED;
    if ((long long)cfg->num_experts * cfg->hidden_dim > 0x7fffffffLL) return B200_UNSUPPORTED;
    return B200_OK;
}

// permute + sort + GEMM1 (+ GEMM2) on given routing.  trusted: the ids are this library's router's (an expert
// appears at most once per token, nothing to check)
int run_experts(b200_ws* ws, const Fp8Scratch& s, const uint8_t* xq, const float* xs, const int* ids,
                const float* wts, const uint8_t* w1q, const float* w1s, const uint8_t* w2q, const float* w2s,
                float* out, const b200_moe_fp8_config* cfg, bool do_gemm2, bool packed, cudaStream_t stream,
                bool zero_out = true, bool trusted = false) {
    const int T = cfg->num_tokens, E = cfg->num_experts, K = cfg->top_k, D = cfg->hidden_dim,
              I = cfg->intermediate_dim;
    const long long TK = (long long)T * K;
    const bool det = (cfg->flags & B200_MOE_DETERMINISTIC) != 0 && do_gemm2;
    // The output is cleared early (the one-launch sort does it on the way), unless it shares memory with something that
    // the kernels in front of GEMM2 still read.
    const bool clear = do_gemm2 && !det && zero_out;
    const size_t out_bytes = sizeof(float) * (size_t)T * D, w1_blocks = (size_t)E * (2 * I / 128) * (D / 128);
    auto shares = [&](const void* p, size_t n) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(out), b = reinterpret_cast<uintptr_t>(p);
        return a < b + n && b < a + out_bytes;
    };
    const bool late = clear && (shares(xq, (size_t)T * D) || shares(xs, sizeof(float) * (size_t)T * (D / 128)) ||
                                shares(ids, sizeof(int) * (size_t)TK) || shares(wts, sizeof(float) * (size_t)TK) ||
                                shares(w1q, w1_blocks * 128 * 128) || shares(w1s, sizeof(float) * w1_blocks));
    int st = B200_OK;
    if (trusted && TK <= SMALL_PAIRS) {
        B200_CUDA_TRY(b200_launch_after(sort_small_fp8_kernel, dim3((unsigned)TK + 1), 128, 0, stream, xq, xs, ids, wts, (int)TK, E, K, D,
                                        s.offsets, s.sq, s.ss, TK, s.row_tok, s.row_w, det ? s.pair_row : nullptr,
                                        clear && !late ? out : nullptr));
    } else {
        if (clear && !late) B200_CUDA_TRY(cudaMemsetAsync(out, 0, out_bytes, stream));
        st = launch_permute_ranges(ids, T, K, E, trusted, s.range_hist, s.counts, s.offsets, s.row_pair, stream);
        if (st) return st;
        if (det) B200_CUDA_TRY(cudaMemsetAsync(s.pair_row, 0xFF, sizeof(int) * (size_t)TK, stream));
        const unsigned sort_blocks = (unsigned)(TK < (long long)ws->sm_count * 32 ? TK : (long long)ws->sm_count * 32);
        B200_CUDA_TRY(b200_launch_after(sort_rows_fp8_kernel, dim3(sort_blocks), 128, 0, stream, xq, xs, s.row_pair, s.offsets, wts, E, K, D,
                                        s.sq, s.ss, TK, s.row_tok, s.row_w, det ? s.pair_row : nullptr));
    }
    b200_count_launch(1);
    B200_CUDA_TRY(cudaGetLastError());

    static B200PerDeviceOnce once;
    st = b200_once_on_device(once, []() -> int {
        const void* kernels[9] = {(const void*)grouped_gemm_fp8_kernel<1, false>, (const void*)grouped_gemm_fp8_kernel<2, false>,
                                  (const void*)grouped_gemm_fp8_kernel<3, false>, (const void*)grouped_gemm_fp8_kernel<1, true>,
                                  (const void*)grouped_gemm_fp8_kernel<2, true>, (const void*)grouped_gemm_fp8_kernel<3, true>,
                                  (const void*)grouped_gemm_mx_kernel<1>, (const void*)grouped_gemm_mx_kernel<2>,
                                  (const void*)grouped_gemm_mx_kernel<3>};
        for (int i = 0; i < 9; i++)
            B200_CUDA_TRY(cudaFuncSetAttribute(kernels[i], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)(i < 6 ? GEMM_SMEM_BYTES : GEMM_MX_SMEM_BYTES)));
        // setmaxnreg.inc waits without bound for registers that only setmaxnreg.dec of the same CTA frees:
        // never launch a build whose compiled register count breaks the balance the budgets assume
        for (int i = 0; i < 9; i++) {
            cudaFuncAttributes a{};
            B200_CUDA_TRY(cudaFuncGetAttributes(&a, kernels[i]));
            const int n = a.numRegs;
            if (!(n * GEMM_THREADS <= 65536 && n <= PROMO_REGS && NUM_PROMO_WARPS * (PROMO_REGS - n) <= 4 * (n - AUX_REGS))) {
                b200_set_last_error_text("grouped GEMM: the compiled register count does not balance the setmaxnreg budgets");
                return B200_UNSUPPORTED;
            }
        }
        return B200_OK;
    });
    if (st) return st;
    b200_gemm_profile* prof = (ws->gemm_prof && ws->gemm_prof->on) ? ws->gemm_prof : nullptr;
    const int slot = prof ? (int)(prof->calls % PROF_SLOTS) : 0;
    // Single-CTA 128-row tiles unless the caller asks for CTA pairs.  Measured on B200 the pair tiles (256 rows,
    // half of the weight tile per SM, a third less shared-memory traffic) are slower at every shape tried
    // (E = 256, K = 8, D = 7168, I = 2048: T = 333 3.5 against 1.8 - 1.9 ms, T = 4096 4.3 - 4.5 against 3.2 - 3.4; 32 experts x 1024
    // rows 2.4 against 2.0): the K-block period is the round trip of an accumulator stage, which is longer across two
    // CTAs (950 - 980 against 880 cycles) and is not helped by less shared-memory traffic, and a pair idles half of its rows on
    // experts with fewer than 129 rows.
    const bool mx = (cfg->flags & B200_MOE_POW2_SCALES) != 0;      // power-of-two scales: hardware block-scaled MMA
    bool pair = (cfg->flags & B200_MOE_CTA_PAIR_TILES) != 0;
    if ((cfg->flags & B200_MOE_SINGLE_CTA_TILES) || mx) pair = false;
    if (ws->sm_count < 2) pair = false;
    const unsigned grid = pair ? (unsigned)(ws->sm_count / 2) * 2 : (unsigned)ws->sm_count;
    auto launch = [&](int mode, const CUtensorMap& ta, const CUtensorMap& ta32, const CUtensorMap& ta8, const CUtensorMap& tb, const GemmParams& p) -> int {
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3(grid); lc.blockDim = dim3(GEMM_THREADS); lc.stream = stream;
        lc.dynamicSmemBytes = mx ? GEMM_MX_SMEM_BYTES : GEMM_SMEM_BYTES;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = 2; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
#ifndef B200_GEMM_CLUSTER2
#define B200_GEMM_CLUSTER2 1
#endif
        // Single-CTA tiles are launched as clusters of two as well: tiles 2i and 2i+1 (the two 128-row tiles of
        // an expert's weight slab when it has 129..256 rows) then run on SMs of one GPC, behind the same L2
        // partition, and the slab comes from DRAM once instead of once per die.
        const bool cluster2 = pair || (B200_GEMM_CLUSTER2 && grid % 2 == 0);
        lc.attrs = attr; lc.numAttrs = cluster2 ? 2 : 1;
        cudaError_t err;
        if (mx) {
            if (mode == 1)      err = cudaLaunchKernelEx(&lc, grouped_gemm_mx_kernel<1>, ta, ta32, ta8, tb, p);
            else if (mode == 2) err = cudaLaunchKernelEx(&lc, grouped_gemm_mx_kernel<2>, ta, ta32, ta8, tb, p);
            else                err = cudaLaunchKernelEx(&lc, grouped_gemm_mx_kernel<3>, ta, ta32, ta8, tb, p);
        } else if (pair) {
            if (mode == 1)      err = cudaLaunchKernelEx(&lc, grouped_gemm_fp8_kernel<1, true>, ta, ta32, ta8, tb, p);
            else if (mode == 2) err = cudaLaunchKernelEx(&lc, grouped_gemm_fp8_kernel<2, true>, ta, ta32, ta8, tb, p);
            else                err = cudaLaunchKernelEx(&lc, grouped_gemm_fp8_kernel<3, true>, ta, ta32, ta8, tb, p);
        } else {
            if (mode == 1)      err = cudaLaunchKernelEx(&lc, grouped_gemm_fp8_kernel<1, false>, ta, ta32, ta8, tb, p);
            else if (mode == 2) err = cudaLaunchKernelEx(&lc, grouped_gemm_fp8_kernel<2, false>, ta, ta32, ta8, tb, p);
            else                err = cudaLaunchKernelEx(&lc, grouped_gemm_fp8_kernel<3, false>, ta, ta32, ta8, tb, p);
        }
        b200_count_launch(1);
        B200_CUDA_TRY(err);
        B200_CUDA_TRY(cudaGetLastError());
        return B200_OK;
    };
    CUtensorMap ta, ta32, ta8, tb;
    GemmParams p{};
    p.offsets = s.offsets; p.E = E; p.D = D; p.I = I; p.status = ws->d_status;
#ifdef B200_GEMM_TRACE
    p.trace = g_gemm_trace; p.trace_warp = g_gemm_trace_warp;
#endif

    // GEMM1 (a CTA of a pair fetches half of a weight tile: boxes of 128 rows instead of 256)
    st = b200_make_tmap_u8_sw128(&ta, s.sq, (unsigned long long)TK, D, 128);
    if (!st) st = b200_make_tmap_u8_sw128(&ta32, s.sq, (unsigned long long)TK, D, 32);
    if (!st) st = b200_make_tmap_u8_sw128(&ta8, s.sq, (unsigned long long)TK, D, 8);
    if (st) return st;
    p.packed = packed ? 1 : 0;
    if (packed) st = b200_make_tmap_u8_sw128(&tb, w1q, (unsigned long long)E * 2 * I * (D / 128), 128, pair ? 128 : 256);
    else        st = b200_make_tmap_u8_sw128(&tb, w1q, (unsigned long long)E * 2 * I, D, QCOLS / 2);
    if (st) return st;
    // Scales of the sorted rows lie K block by K block, as the GEMMs read them; alone, GEMM1 leaves its own row by row.
    p.a_scale = s.ss; p.a_ks = TK; p.w_scale = w1s; p.act_q = s.act_q; p.act_s = s.act_s;
    p.s_rs = do_gemm2 ? 1 : I / 128; p.s_ks = do_gemm2 ? TK : 1;
    if (prof) B200_CUDA_TRY(cudaEventRecord(prof->ev[slot][0], stream));
    st = launch(1, ta, ta32, ta8, tb, p);
    if (st) return st;
    if (prof) B200_CUDA_TRY(cudaEventRecord(prof->ev[slot][1], stream));
    if (!do_gemm2) return B200_OK;

    // GEMM2
    st = b200_make_tmap_u8_sw128(&ta, s.act_q, (unsigned long long)TK, I, 128);
    if (!st) st = b200_make_tmap_u8_sw128(&ta32, s.act_q, (unsigned long long)TK, I, 32);
    if (!st) st = b200_make_tmap_u8_sw128(&ta8, s.act_q, (unsigned long long)TK, I, 8);
    if (st) return st;
    if (packed) st = b200_make_tmap_u8_sw128(&tb, w2q, (unsigned long long)E * D * (I / 128), 128, pair ? 128 : 256);
    else        st = b200_make_tmap_u8_sw128(&tb, w2q, (unsigned long long)E * D, I, pair ? 128 : 256);
    if (st) return st;
    p.a_scale = s.act_s; p.w_scale = w2s; p.row_tok = s.row_tok; p.row_w = s.row_w;
#ifdef B200_GEMM_TRACE
    if (p.trace) p.trace += 8 * TRACE_CAP;      // second half of the buffer for GEMM2
#endif
    if (det) {
        p.out = s.rows;
        if (prof) B200_CUDA_TRY(cudaEventRecord(prof->ev[slot][2], stream));
        st = launch(3, ta, ta32, ta8, tb, p);
        if (st) return st;
        reduce_rows_kernel<<<T, 256, 0, stream>>>(s.rows, s.pair_row, ids, K, D, out);
        if (prof) { B200_CUDA_TRY(cudaEventRecord(prof->ev[slot][3], stream)); prof->calls++; }
        b200_count_launch(1);
        B200_CUDA_TRY(cudaGetLastError());
        return B200_OK;
    }
    p.out = out;
    if (late) B200_CUDA_TRY(cudaMemsetAsync(out, 0, out_bytes, stream));
    if (prof) B200_CUDA_TRY(cudaEventRecord(prof->ev[slot][2], stream));
    st = launch(2, ta, ta32, ta8, tb, p);
    if (st) return st;
    if (prof) { B200_CUDA_TRY(cudaEventRecord(prof->ev[slot][3], stream)); prof->calls++; }
    return B200_OK;
}

}  // namespace

extern "C" {

#ifdef B200_GEMM_TRACE
// Timeline builds only (-DB200_GEMM_TRACE; never part of the default library): CTA 0 of the next grouped
// GEMM launches fills dev_buf [2][8][512] with clock64 stamps of its pipeline events.
__attribute__((visibility("default"))) void b200_debug_gemm_trace(long long* dev_buf, int warp) {
    g_gemm_trace = dev_buf;
    g_gemm_trace_warp = warp;
}
#endif

int b200_moe_fp8_profile(b200_ws* ws, int enable) {
    if (!ws) ws = b200_default_ws();
    if (!ws) return B200_CUDA_ERROR;
    if (!ws->gemm_prof) {
        if (!enable) return B200_OK;
        b200_gemm_profile* pr = new b200_gemm_profile();
        for (int i = 0; i < PROF_SLOTS; i++)
            for (int j = 0; j < 4; j++) B200_CUDA_TRY(cudaEventCreate(&pr->ev[i][j]));
        ws->gemm_prof = pr;
    }
    ws->gemm_prof->on = enable != 0;
    ws->gemm_prof->calls = 0;
    return B200_OK;
}

int b200_moe_fp8_profile_read(b200_ws* ws, float* gemm1_ms, float* gemm2_ms, int* calls) {
    if (!gemm1_ms || !gemm2_ms || !calls) return B200_BAD_ARG;
    if (!ws) ws = b200_default_ws();
    if (!ws) return B200_CUDA_ERROR;
    const b200_gemm_profile* pr = ws->gemm_prof;
    const int n = pr ? (int)(pr->calls < PROF_SLOTS ? pr->calls : PROF_SLOTS) : 0;
    *calls = n;
    *gemm1_ms = *gemm2_ms = 0.0f;
    if (n == 0) return B200_OK;
    double s1 = 0.0, s2 = 0.0;
    for (int i = 0; i < n; i++) {
        float a = 0.f, b = 0.f;
        B200_CUDA_TRY(cudaEventSynchronize(pr->ev[i][3]));
        B200_CUDA_TRY(cudaEventElapsedTime(&a, pr->ev[i][0], pr->ev[i][1]));
        B200_CUDA_TRY(cudaEventElapsedTime(&b, pr->ev[i][2], pr->ev[i][3]));
        s1 += a; s2 += b;
    }
    *gemm1_ms = (float)(s1 / n);
    *gemm2_ms = (float)(s2 / n);
    return B200_OK;
}

static int experts_impl(b200_ws* ws, const uint8_t* xq, const float* xs, const int* expert_ids,
                        const float* expert_w, const uint8_t* w1q, const float* w1s, const uint8_t* w2q,
                        const float* w2s, float* out, const b200_moe_fp8_config* cfg, bool packed,
                        b200_stream_t stream, bool zero_out = true) {
    int st = check_fp8_cfg(cfg);
    if (st) return st;
    if (!xq || !xs || !expert_ids || !expert_w || !w1q || !w1s || !w2q || !w2s || !out) return B200_BAD_ARG;
    if (!ws) ws = b200_default_ws();
    if (!ws) return B200_CUDA_ERROR;
    Fp8Scratch s;
    WsCarver sz(nullptr);
    carve_fp8(sz, cfg, false, s);
    st = b200_ws_ensure(ws, sz.total());
    if (st) return st;
    WsCarver cv(ws->base);
    carve_fp8(cv, cfg, false, s);
    return run_experts(ws, s, xq, xs, expert_ids, expert_w, w1q, w1s, w2q, w2s, out, cfg, true, packed, stream,
                       zero_out);
}

}  // extern "C"

// Expert-parallel owner side (moe_ep.cu): `out` already holds zeros in every row that can receive a
// contribution (the push kernel of the previous step cleared what it read), so the scatter-add GEMM2
// runs without the zero-fill pass over the whole row capacity.
int b200_moe_fp8_experts_accumulate(b200_ws* ws, const uint8_t* xq, const float* xs, const int* expert_ids,
                                    const float* expert_w, const uint8_t* w1, const float* w1s, const uint8_t* w2,
                                    const float* w2s, float* out, const b200_moe_fp8_config* cfg, bool packed,
                                    cudaStream_t stream) {
    if (cfg && (cfg->flags & B200_MOE_DETERMINISTIC)) return B200_UNSUPPORTED;
    return experts_impl(ws, xq, xs, expert_ids, expert_w, w1, w1s, w2, w2s, out, cfg, packed, stream, false);
}

extern "C" {

int b200_moe_fp8_experts(b200_ws* ws, const uint8_t* xq, const float* xs, const int* expert_ids,
                         const float* expert_w, const uint8_t* w1q, const float* w1s, const uint8_t* w2q,
                         const float* w2s, float* out, const b200_moe_fp8_config* cfg, b200_stream_t stream) {
    return experts_impl(ws, xq, xs, expert_ids, expert_w, w1q, w1s, w2q, w2s, out, cfg, false, stream);
}

int b200_moe_fp8_experts_packed(b200_ws* ws, const uint8_t* xq, const float* xs, const int* expert_ids,
                                const float* expert_w, const uint8_t* w1p, const float* w1s, const uint8_t* w2p,
                                const float* w2s, float* out, const b200_moe_fp8_config* cfg, b200_stream_t stream) {
    return experts_impl(ws, xq, xs, expert_ids, expert_w, w1p, w1s, w2p, w2s, out, cfg, true, stream);
}

static int forward_impl(b200_ws* ws, const uint8_t* xq, const float* xs, const float* gate_w, const float* bias,
                        const uint8_t* w1q, const float* w1s, const uint8_t* w2q, const float* w2s, float* out,
                        const b200_moe_fp8_config* cfg, bool packed, b200_stream_t stream) {
    int st = check_fp8_cfg(cfg);
    if (st) return st;
    if (!xq || !xs || !gate_w || !w1q || !w1s || !w2q || !w2s || !out) return B200_BAD_ARG;
    const int T = cfg->num_tokens, E = cfg->num_experts, K = cfg->top_k, D = cfg->hidden_dim;
    st = check_route_cfg(T, E, K, D, cfg->scoring, cfg->n_group, cfg->topk_group);
    if (st) return st;
    if (!ws) ws = b200_default_ws();
    if (!ws) return B200_CUDA_ERROR;
    Fp8Scratch s;
    WsCarver sz(nullptr);
    carve_fp8(sz, cfg, true, s);
    st = b200_ws_ensure(ws, sz.total());
    if (st) return st;
    WsCarver cv(ws->base);
    carve_fp8(cv, cfg, true, s);
    st = moe_route_fp8_run(s.route, xq, xs, gate_w, bias, s.ids, s.wts, nullptr, nullptr, cfg, ws->d_status, stream);
    if (st) return st;
    ws->route_flag_n = (s.route.whi && cfg->scoring == B200_SCORE_SIGMOID_GROUPED && !(cfg->flags & B200_MOE_EXACT_ROUTER_LOGITS))
                           ? s.route.flag_n : nullptr;
    return run_experts(ws, s, xq, xs, s.ids, s.wts, w1q, w1s, w2q, w2s, out, cfg, true, packed, stream, true, true);
}

int b200_moe_fp8_forward(b200_ws* ws, const uint8_t* xq, const float* xs, const float* gate_w, const float* bias,
                         const uint8_t* w1q, const float* w1s, const uint8_t* w2q, const float* w2s, float* out,
                         const b200_moe_fp8_config* cfg, b200_stream_t stream) {
    return forward_impl(ws, xq, xs, gate_w, bias, w1q, w1s, w2q, w2s, out, cfg, false, stream);
}

int b200_moe_fp8_forward_packed(b200_ws* ws, const uint8_t* xq, const float* xs, const float* gate_w,
                                const float* bias, const uint8_t* w1p, const float* w1s, const uint8_t* w2p,
                                const float* w2s, float* out, const b200_moe_fp8_config* cfg, b200_stream_t stream) {
    return forward_impl(ws, xq, xs, gate_w, bias, w1p, w1s, w2p, w2s, out, cfg, true, stream);
}

// Weight pre-tiling.  which = 1: w1 [E,2I,D] -> tiles of 256 accumulator rows (gate j0..+63, up j0..+63,
// gate j0+64..+127, up j0+64..+127 for j0 = 128 * n_tile); which = 2: w2 [E,D,I] -> tiles of 256 rows.
// packed[(((e * NT + n_tile) * nkb + kb) * 256 + r) * 128 + b] = src[e][row(n_tile, r)][kb * 128 + b].
int b200_moe_fp8_pack_weights(int which, const uint8_t* src, uint8_t* packed, int E, int D, int I,
                              b200_stream_t stream) {
    if (!src || !packed) return B200_BAD_ARG;
    if (which != 1 && which != 2) return B200_BAD_ARG;
    if (E <= 0 || D <= 0 || I <= 0 || D % 256 || I % 128) return B200_BAD_SHAPE;
    const int Kdim = which == 1 ? D : I;
    const int NT = which == 1 ? I / 128 : D / 256;
    const long long chunks = (long long)E * NT * (Kdim / 128) * 256 * 8;     // 16-byte chunks
    long long blocks = (chunks + 255) / 256;
    if (blocks > 0x7fffffffLL) return B200_UNSUPPORTED;
    pack_weights_kernel<<<(unsigned)blocks, 256, 0, stream>>>(which, src, packed, E, D, I, chunks);
    b200_count_launch(1);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

int b200_moe_fp8_gemm1_stage(b200_ws* ws, const uint8_t* xq, const float* xs, const int* expert_ids,
                             const uint8_t* w1q, const float* w1s, uint8_t* act_q, float* act_s, int* offsets,
                             int* row_pair, const b200_moe_fp8_config* cfg, b200_stream_t stream) {
    int st = check_fp8_cfg(cfg);
    if (st) return st;
    if (!xq || !xs || !expert_ids || !w1q || !w1s || !act_q || !act_s || !offsets || !row_pair) return B200_BAD_ARG;
    if (!ws) ws = b200_default_ws();
    if (!ws) return B200_CUDA_ERROR;
    Fp8Scratch s;
    WsCarver sz(nullptr);
    carve_fp8(sz, cfg, false, s);
    float* dummy_w = sz.take<float>((size_t)cfg->num_tokens * cfg->top_k);
    st = b200_ws_ensure(ws, sz.total());
    if (st) return st;
    WsCarver cv(ws->base);
    carve_fp8(cv, cfg, false, s);
    dummy_w = cv.take<float>((size_t)cfg->num_tokens * cfg->top_k);
    const size_t TK = (size_t)cfg->num_tokens * cfg->top_k;
    B200_CUDA_TRY(cudaMemsetAsync(dummy_w, 0, sizeof(float) * TK, stream));
    B200_CUDA_TRY(cudaMemsetAsync(s.act_q, 0, TK * cfg->intermediate_dim, stream));
    B200_CUDA_TRY(cudaMemsetAsync(s.act_s, 0, sizeof(float) * TK * (cfg->intermediate_dim / 128), stream));
    st = run_experts(ws, s, xq, xs, expert_ids, dummy_w, w1q, w1s, nullptr, nullptr, nullptr, cfg, false, false, stream);
    if (st) return st;
    B200_CUDA_TRY(cudaMemcpyAsync(act_q, s.act_q, TK * cfg->intermediate_dim, cudaMemcpyDeviceToDevice, stream));
    B200_CUDA_TRY(cudaMemcpyAsync(act_s, s.act_s, sizeof(float) * TK * (cfg->intermediate_dim / 128),
                                  cudaMemcpyDeviceToDevice, stream));
    B200_CUDA_TRY(cudaMemcpyAsync(offsets, s.offsets, sizeof(int) * (cfg->num_experts + 1),
                                  cudaMemcpyDeviceToDevice, stream));
    B200_CUDA_TRY(cudaMemcpyAsync(row_pair, s.row_pair, sizeof(int) * TK, cudaMemcpyDeviceToDevice, stream));
    return B200_OK;
}

}  // extern "C"
