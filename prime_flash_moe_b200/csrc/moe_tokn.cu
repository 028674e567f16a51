// Fused MoE FFN with the routed rows on the N side of the MMA ("token-N" kernels), sm_100a, CTA pairs; bf16 and mxfp8.
//
// tcgen05 fixes M at 128 or 256 but takes any multiple of 16 as N. With the rows as M (moe_bf16.cu, moe_mxfp8.cu) an expert
// pays for whole 128-row blocks: 8 rows of a decode batch cost a 128-row MMA, 530 rows cost 640. Here the WEIGHT rows are
// M (256 per CTA pair, cta_group::2) and an expert's routed rows are N, cut into equal pieces of at most `cap` rows
// (a multiple of 32): 530 rows run as 3 x 192, and the operand feed per CTA and k-step (128 bytes of K) is 16 KB of weights
// + up to 16 KB of rows instead of 48 KB for the same MACs of a one-CTA 128 x 256 tile.
//
//   work item   (expert, first row of sorted_token_ids, rows of this piece): built on the device by CTA 0 of plan_kernel
//   gate/up     tile = item x 128 activation columns. Each CTA of the pair owns 64 of them: its A tile holds the 64
//               gate rows and the 64 up rows interleaved in groups of 16 (ONE five-dimensional TMA box per k-step), so
//               that lanes l and l + 16 of a TMEM lane quarter hold gate and up of the same activation and two
//               16-lane TMEM loads give a thread both. SwiGLU -> bf16 -> staging -> TMA store.
//   down        tile = item x 256 output columns, 128 per CTA; accumulator * routing weight -> bf16 -> transposed through the
//               warp's own staging buffer -> 16-byte vector reductions into out[token] by the epilogue warps themselves.
//               (A store warp's 256-byte bulk reductions, one a routed row, cost 31 ns each and SM and need 51 KB of staging:
//               8 experts, 128 rows each, K = 4096, N = 512 29.6 -> 25.0 us; mxfp8, T = 5003, K = 2048, N = 1536, top_k = 8
//               133 -> 101 us. Long rows take them all the same: tokn_bulk_down().)
//
//   backward    row-space GEMMs where an expert has few rows: tile = row block x 256 output columns, the rows by TMA from the
//               sorted copies, results rows of 16-byte stores through the warp's own tiles (D_ACT: SwiGLU derivative there).
//
// Warp roles: warp 0 TMA producer, warp 1 TMEM owner + MMA issuer (even CTA), warps 2-9 epilogue in two groups of four
// (a group takes every second 32-row chunk of the accumulator), gate/up and bulk reductions: warps 10-11 one store warp per
// group: it waits for a staged chunk, issues the bulk stores (mxfp8: quantises it) and hands the buffer back, so that the
// epilogue warps never wait for a store to be read; gate/up: four warps copy the routed rows of x straight into the ring (cp.async; no row-sorted copy of x
// in HBM, which cost 75 of 645 us at T = 8192, K = 2048, N = 1536, top_k = 8) and one publishes what has landed. Two
// accumulators in TMEM; every wait is bounded (ptx.cuh).
//
// mxfp8 (block-scaled MMAs, N <= 192: two accumulators of 192 columns leave 128 for the scales): the scale tiles of the rows
// come by TMA with their slot, those of w2 too; those of w have to be interleaved like the A tile and are put together by a
// warp of their own. The chunk staged by the gate/up epilogue is the fp32 SwiGLU value (an MX block runs over two warps'
// lanes); the store warps take a row a lane and quantise it as moe_mxfp8.cu does. Which calls take these kernels and which the
// row-M ones of moe_mxfp8.cu: take_token_n() there.
#include <algorithm>
#include <atomic>

#include "host_common.h"
#include "moe_tokn.h"
#include "mx_quant.cuh"
#include "ptx.cuh"
#include "tile_sched.cuh"

namespace pmoe {

__device__ int g_status_tokn = 0;

namespace {

constexpr int BM = kBlockM;
// What a launch contracts. The first three are the forward pass, the others the row-space GEMMs of the backward pass. D_ACT
// and D_XS read their weights with the output dimension contiguous (M-major operand: two 64 x 64 boxes a CTA and k-step).
enum : int {
    UP = 0,       // gate | up of the routed rows, SwiGLU
    DOWN = 1,     // act . W2[e]^T, weighted, added into out[token] by vector reductions ...
    DOWN_BULK = 2,   // ... by bulk reductions
    GATE_UP = 3,  // rows of x . W1[e]^T -> rows of the pre-activations
    D_ACT = 4,    // rows of d_out . W2[e], SwiGLU derivative -> d_gate | d_up, weight * act, d_weight
    D_XS = 5,     // d_gate | d_up . W1[e] -> rows of d_xs
};
constexpr uint32_t A_BYTES = 128 * 128;          // 16 KB: 128 weight rows x 128 bytes of K per CTA and k-step
template <bool kMx> constexpr int BK = kMx ? 128 : 64;            // K elements of a k-step (128 bytes)
template <bool kMx> constexpr uint32_t ACC_COLS = kMx ? 192 : 256; // TMEM columns of one of the two accumulators
constexpr int MAX_STAGES = 12;
constexpr uint32_t TMEM_COLS = 512;
constexpr int EPI_WARPS = 8;
constexpr int STORE_WARP = 2 + EPI_WARPS;        // gate/up: two store warps ...
constexpr int SCALE_WARP = STORE_WARP + 2;       // ... mxfp8: a scale warp and its publisher ...
template <bool kMx> constexpr int GATHER_WARP = SCALE_WARP + (kMx ? 2 : 0);   // ... four for the rows of x and their publisher
constexpr int GATHER_THREADS = 128;
template <int kMode, bool kMx>
constexpr int THREADS = (kMode == UP ? GATHER_WARP<kMx> + GATHER_THREADS / 32 + 1 : STORE_WARP + (kMode == DOWN_BULK ? 2 : 0)) * 32;
constexpr int CHUNK = 32;                        // rows per staged chunk
constexpr int UP_BUFS = 4;        // staging buffers per epilogue group
constexpr uint32_t UP_BUF_BYTES = CHUNK * 128;           // 32 rows x 64 activation columns, 128-byte swizzle
// down: a warp's own 32 routed rows x 32 output columns, a row padded so that neither stmatrix nor 16-byte loads conflict
constexpr uint32_t DOWN_ROW_BYTES = 64 + 16;
constexpr uint32_t DOWN_BUF_BYTES = CHUNK * DOWN_ROW_BYTES;
constexpr int BULK_BUFS = 3;                                      // ... bulk reductions: a group's 32 rows x 128 columns
constexpr uint32_t BULK_ROW_BYTES = 256 + 16;
constexpr uint32_t BULK_BUF_BYTES = CHUNK * BULK_ROW_BYTES;
constexpr int KEEP_BUFS = 2;                                      // gate/up with kept pre-activations: activation, gate
constexpr uint32_t KEEP_BUF_BYTES = 3 * UP_BUF_BYTES;             // and up chunks in one buffer
// mxfp8 gate/up: the staged chunk is the fp32 SwiGLU value, quantised by the store warps; 64 activations a row, padded so
// that neither the fragments' 4-byte stores nor the 16-byte loads of a row meet in a bank
constexpr int MX_UP_BUFS = 2;
constexpr uint32_t MX_UP_ROW_BYTES = 64 * 4 + 16;
constexpr uint32_t MX_UP_BUF_BYTES = CHUNK * MX_UP_ROW_BYTES;
constexpr uint32_t SF_TILE = 512;                // scales of 128 rows x 128 K elements: line l = rows l, l + 32, l + 64, l + 96
constexpr uint32_t D_ACT_TILE = CHUNK * 64;      // 32 routed rows x 32 activations, 64-byte swizzle
template <bool kUp> constexpr uint32_t SF_BYTES = kUp ? 1024 : 2048;   // of a slot: rows 2 x 512 (and, down, weights 512)
constexpr int SFA_BATCHES = 8;                   // gate/up: a ring of its own for the weights' scale tiles, two k-steps a batch
constexpr uint32_t SFA_BYTES = SFA_BATCHES * 2 * SF_TILE;
constexpr uint32_t SF_TMEM = 384;                // TMEM columns of the scales: eight regions of 4 (weights) + 8 (rows)
template <int kMode, bool kKeep, bool kMx>
constexpr int BUFS = kMode == DOWN_BULK ? BULK_BUFS : kMode != UP ? EPI_WARPS / 2 : kMx ? MX_UP_BUFS : kKeep ? KEEP_BUFS : UP_BUFS;
template <int kMode, bool kKeep, bool kMx>
constexpr uint32_t BUF_BYTES = kMode == D_ACT ? 5 * D_ACT_TILE : kMode == DOWN_BULK ? BULK_BUF_BYTES : kMode != UP ? DOWN_BUF_BYTES
                               : kMx ? MX_UP_BUF_BYTES : kKeep ? KEEP_BUF_BYTES : UP_BUF_BYTES;
constexpr uint32_t BAR_BYTES = 768;
constexpr uint32_t SMEM_LIMIT = 232448;
constexpr int ST_BAD_PAIR = 8;                   // bpc = 2 table whose 256-row pair holds two experts

struct Args {
    const uint8_t *x;         // in-kernel row gather: the caller's rows
    const int2 *row_info;     // per sorted row: token (-1 for padding) and routing weight (fp32 bits)
    __nv_bfloat16 *out;
    const int32_t *live_rows;
    const int4 *items;        // end of the item buffer: item i of n is items[i - n] (the planner fills it backwards)
    const int32_t *item_count;
    const uint32_t *w_scales;   // mxfp8 gate/up: scale tiles of w
    uint8_t *act_q, *act_sf;    // mxfp8 gate/up: e4m3 activations [sorted_num][H], their scale tiles [H / 128][blocks][512]
    int blocks;                 // 128-row blocks of the routing table
    // backward; M = routed pairs here
    ToknBlocks list;
    const int32_t *sorted_ids;
    const float *topk_weights;
    const __nv_bfloat16 *gu;    // gate | up pre-activations [sorted_num, 2 * H]
    __nv_bfloat16 *c, *actw;    // c: the rows that the launch writes, ldc columns
    float *dwt;
    int ldc, cols, k;           // cols: live output columns; k: contraction length
    int M, K, H;
    int stages;
    uint32_t stage_bytes, sf_off;
    int use_pdl, zero_out;
};

struct Smem {
    uint32_t ring, staging, sfa_ring, bars, stage_bytes, sf_off;
    __device__ __forceinline__ uint32_t a(int s) const { return ring + s * stage_bytes; }
    __device__ __forceinline__ uint32_t b(int s) const { return ring + s * stage_bytes + A_BYTES; }
    __device__ __forceinline__ uint32_t sf(int s) const { return ring + s * stage_bytes + sf_off; }
    __device__ __forceinline__ uint32_t full(int s) const { return bars + 8 * s; }
    __device__ __forceinline__ uint32_t empty(int s) const { return bars + 8 * (MAX_STAGES + s); }
    __device__ __forceinline__ uint32_t tmem_full(int b) const { return bars + 8 * (2 * MAX_STAGES + b); }
    __device__ __forceinline__ uint32_t tmem_empty(int b) const { return bars + 8 * (2 * MAX_STAGES + 2 + b); }
    __device__ __forceinline__ uint32_t staged(int i) const { return bars + 8 * (2 * MAX_STAGES + 4 + i); }
    __device__ __forceinline__ uint32_t freed(int i) const { return bars + 8 * (2 * MAX_STAGES + 4 + 2 * UP_BUFS + i); }
    __device__ __forceinline__ uint32_t sfa(int b) const { return sfa_ring + b * 2 * SF_TILE; }
    __device__ __forceinline__ uint32_t scaled(int b) const { return bars + 8 * (2 * MAX_STAGES + 6 + 4 * UP_BUFS + b); }
    __device__ __forceinline__ uint32_t gathered(int s) const { return scaled(3 * SFA_BATCHES + s); }
    __device__ __forceinline__ uint32_t sfa_full(int b) const { return scaled(SFA_BATCHES + b); }
    __device__ __forceinline__ uint32_t sfa_empty(int b) const { return scaled(2 * SFA_BATCHES + b); }
    __device__ __forceinline__ uint32_t tmem_slot() const { return bars + 8 * (2 * MAX_STAGES + 4 + 4 * UP_BUFS); }
};

__device__ __forceinline__ void tma_load_5d_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar_cluster_addr, int c0,
                                                 int c1, int c2, int c3, int c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar_cluster_addr), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
        : "memory");
}
// Shared-memory descriptor of an M-major operand made of 64 x 64 boxes (128-byte swizzle): one 128-byte line holds 64
// consecutive M indices of one k, eight lines (8 k) a 1024-byte atom; atoms follow each other along k every 1024 B (stride
// byte offset) and along M every box (leading byte offset). Stepping by one MMA (16 k) adds 2048 B.
__device__ __forceinline__ uint64_t smem_desc_m_sw128(uint32_t addr) {
    return static_cast<uint64_t>((addr & 0x3FFFFu) >> 4) | (static_cast<uint64_t>(8192 >> 4) << 16) |
           (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// 16 lanes x 32 columns of 32-bit in the fragment layout of an m16n8 accumulator: with i = lane id, d[4 j + {0, 1}] are
// columns 8 j + 2 (i % 4) + {0, 1} of TMEM lane i / 4, d[4 j + {2, 3}] the same columns of lane i / 4 + 8
__device__ __forceinline__ void tmem_ld_16x256b_x4(float (&d)[16], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]), "=f"(d[4]), "=f"(d[5]), "=f"(d[6]), "=f"(d[7]), "=f"(d[8]),
          "=f"(d[9]), "=f"(d[10]), "=f"(d[11]), "=f"(d[12]), "=f"(d[13]), "=f"(d[14]), "=f"(d[15])
        : "r"(addr)
        : "memory");
}
// four 8 x 8 matrices of bf16 fragments loaded / stored transposed; lane i gives the address of row i % 8 of matrix i / 8
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&v)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b),
                 "r"(c), "r"(d)
                 : "memory");
}

// four bytes of a 256-byte run that other lanes and the next k-step read too
__device__ __forceinline__ void cp_async_4_l2(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global.L2::256B [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void st_shared_f32(uint32_t addr, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ uint4 ld_shared_u4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float4 ld_shared_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// whole warp waits through lane 0
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, int *status, int code, int lane) {
    bool ok = true;
    if (lane == 0) ok = mbar_wait(bar, parity, status, code);
    return __shfl_sync(0xffffffffu, ok, 0);
}

// ---------------------------------------------------------------------------------------------
// work items (CTA 0 of plan_kernel). A run is a maximal sequence of consecutive row blocks of one expert whose
// blocks, except the last, are full; its n rows are cut into ceil(n / cap) pieces of equal size rounded up to `gran` rows (32,
// mxfp8: 64), the last one's to 32.
// Runs are found from the end of the table to its start, 512 blocks at a time, so that a run's first block already
// knows where the run ends; the items are written backwards from `items_end`, in table order.
// ---------------------------------------------------------------------------------------------
constexpr int PLAN_THREADS = 512;

// ext[i] = rows of block c0 + i up to and including the last routed one, for the chunk's 512 blocks; a warp reads a block
// with one load, eight blocks in flight
__device__ __forceinline__ void block_extents(const int32_t *sorted_ids, int c0, int blocks, int *ext) {
    constexpr int kWarps = PLAN_THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int u0 = 0; u0 < 32 && c0 + u0 * kWarps < blocks; u0 += 8) {
        int4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int b = c0 + (u0 + u) * kWarps + warp;
            v[u] = make_int4(-1, -1, -1, -1);
            if (b < blocks) v[u] = reinterpret_cast<const int4 *>(sorted_ids + static_cast<size_t>(b) * BM)[lane];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int last = v[u].w >= 0 ? 3 : v[u].z >= 0 ? 2 : v[u].y >= 0 ? 1 : v[u].x >= 0 ? 0 : -1;
            const int rows = __reduce_max_sync(0xffffffffu, last >= 0 ? 4 * lane + last + 1 : 0);
            if (lane == 0) ext[(u0 + u) * kWarps + warp] = rows;
        }
    }
}

__device__ void plan_items(const int32_t *sorted_ids, const int32_t *expert_ids, int blocks,
                           int cap, int gran, int bpc, int4 *items_end, int32_t *item_count) {
    constexpr int kWarps = PLAN_THREADS / 32;
    __shared__ int s_first[kWarps];    // first run start of every warp's 32 blocks (or INT_MAX)
    __shared__ int s_sum[kWarps];
    __shared__ int s_ext[PLAN_THREADS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int next_chunk = blocks;   // first run start after this chunk (or the end of the table) ...
    int next_ext = 0;          // ... and the extent of the block before it, taken in the chunk that holds that block
    int written = 0;           // items of the later chunks
    for (int c0 = (blocks + PLAN_THREADS - 1) / PLAN_THREADS * PLAN_THREADS - PLAN_THREADS; c0 >= 0; c0 -= PLAN_THREADS) {
        const int b = c0 + threadIdx.x;
        block_extents(sorted_ids, c0, blocks, s_ext);
        bool start = false;
        int e = 0;
        if (b < blocks) {
            e = expert_ids[b];
            start = b == 0 || expert_ids[b - 1] != e || sorted_ids[static_cast<size_t>(b) * BM - 1] < 0;
            if (bpc == 2 && (b & 1) && expert_ids[b - 1] != e) atomicCAS(&g_status_tokn, 0, ST_BAD_PAIR);
        }
        const uint32_t m = __ballot_sync(0xffffffffu, start);
        if (lane == 0) s_first[warp] = m ? c0 + warp * 32 + __ffs(m) - 1 : 0x7fffffff;
        __syncthreads();
        // that block is in this chunk: at the table's end, or where a run starts at the very next chunk's first block
        if (next_chunk <= c0 + PLAN_THREADS) next_ext = s_ext[next_chunk - 1 - c0];
        int next = next_chunk, first = next_chunk;
        for (int w = kWarps - 1; w >= 0; --w) {
            const int f = s_first[w];
            if (f != 0x7fffffff) {
                first = f;
                if (w > warp) next = f;
            }
        }
        const uint32_t later = lane < 31 ? m >> (lane + 1) : 0u;
        if (later) next = b + __ffs(later);
        int n = 0, pieces = 0;
        if (start) {
            const int last = next - 1;
            n = (last - b) * BM + (last < c0 + PLAN_THREADS ? s_ext[last - c0] : next_ext);
            pieces = (n + cap - 1) / cap;
        }
        int suffix = pieces;      // items of this and the later blocks of the chunk
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_down_sync(0xffffffffu, suffix, d);
            if (lane + d < 32) suffix += v;
        }
        if (lane == 0) s_sum[warp] = suffix;
        __syncthreads();
        int total = 0;
        for (int w = 0; w < kWarps; ++w) {
            const int v = s_sum[w];
            total += v;
            if (w > warp) suffix += v;
        }
        if (pieces) {
            const int width = ((n + pieces - 1) / pieces + gran - 1) & ~(gran - 1);
            int4 *dst = items_end - written - suffix;
            for (int i = 0; i < pieces; ++i) {
                const int r0 = i * width;
                const int rows = min(width, ((n - r0) + 31) & ~31);
                dst[i] = make_int4(e, b * BM + r0, max(rows, 0), 0);
            }
        }
        written += total;
        // a run of an earlier chunk that reaches into this one ends before this one's first run start
        if (first < next_chunk && first > c0) next_ext = s_ext[first - 1 - c0];
        next_chunk = first;
        __syncthreads();
    }
    if (threadIdx.x == 0) *item_count = written;
}

// mxfp8: the routed rows' scales (a word per row and 128 K elements) as 512-byte tiles [K / 128][max_blocks]; word w of a tile
// is row w / 4 + 32 (w % 4). A thread keeps its row, so that neighbouring threads write neighbouring words and the eight
// words of a sector of x_scales are read one after the other.
__device__ __forceinline__ void tile_row_scales(const int32_t *sorted_ids, const uint32_t *x_scales,
                                                uint32_t *__restrict__ tiles, int blocks, int max_blocks, int M, int top_k,
                                                int kt) {
    const int word = threadIdx.x & 127, part = threadIdx.x >> 7;      // four k ranges a CTA
    const int per = (kt + 3) / 4;
    for (int blk = blockIdx.x - 1; blk < blocks; blk += gridDim.x - 1) {
        const int pair = sorted_ids[blk * BM + (word >> 2) + 32 * (word & 3)];
        const int tok = pair >= 0 ? pair / top_k : -1;
        if (tok < 0 || tok >= M) continue;      // padding rows only feed accumulator columns that nothing reads
        const uint32_t *src = x_scales + static_cast<size_t>(tok) * kt;
        const int end = min(kt, (part + 1) * per);
        for (int k = part * per; k < end; k += 4) {      // four loads in flight
            uint32_t v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (k + u < end) v[u] = src[k + u];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (k + u < end) tiles[(static_cast<size_t>(k + u) * max_blocks + blk) * 128 + word] = v[u];
        }
    }
}

// CTA 0 builds the work items; the other CTAs write every row's token and routing weight where the GEMM kernels find both
// with one load instead of two dependent ones, and the scale tiles.
__global__ void __launch_bounds__(PLAN_THREADS)
plan_kernel(const int32_t *sorted_ids, const int32_t *expert_ids, const int32_t *npp, const float *topk_weights, int M,
            int top_k, int sorted_num, int cap, int gran, int bpc, int4 *items_end, int32_t *item_count,
            int2 *__restrict__ row_info, const uint32_t *x_scales, uint32_t *__restrict__ sf_tiles, int kt) {
    pdl_wait_primary();        // launched as a programmatic dependent of whatever the stream holds: the routing kernel
    pdl_launch_dependents();
    const int blocks = live_row_blocks(npp, sorted_num);
    if (blockIdx.x == 0) {
        plan_items(sorted_ids, expert_ids, blocks, cap, gran, bpc, items_end, item_count);
        return;
    }
    for (int row = (blockIdx.x - 1) * PLAN_THREADS + threadIdx.x; row < blocks * BM; row += (gridDim.x - 1) * PLAN_THREADS) {
        const int pair = sorted_ids[row];
        const int tok = pair >= 0 ? pair / top_k : -1;
        const bool live = tok >= 0 && tok < M;
        row_info[row] = make_int2(live ? tok : -1, live ? __float_as_int(topk_weights[pair]) : 0);
    }
    if (x_scales) tile_row_scales(sorted_ids, x_scales, sf_tiles, blocks, sorted_num / BM, M, top_k, kt);
}

// ---------------------------------------------------------------------------------------------
// the GEMM kernel
// ---------------------------------------------------------------------------------------------
struct Tile {
    int expert, row0, rows, n_tile;
};
// Every role fetches the tile after the one it works on: the item comes from L2 (0.4 us), a tenth of a short tile.
__device__ __forceinline__ Tile fetch_tile(const int4 *items, int t, int num_tiles, int n_items, int n_tiles) {
    Tile w{0, 0, 0, 0};
    if (t < num_tiles) {
        const Coord c = tile_coord(t, n_items, n_tiles);
        const int4 it = __ldcg(items + c.m_blk);
        w.expert = it.x, w.row0 = it.y, w.rows = it.z, w.n_tile = c.n_tile;
    }
    return w;
}
// Backward: a piece is a row block of the list, up to the expert's last routed row rounded up to a chunk.
__device__ __forceinline__ Tile fetch_block_tile(const ToknBlocks &l, int t, int num_tiles, int n_items, int n_tiles) {
    Tile w{0, 0, 0, 0};
    if (t < num_tiles) {
        const Coord c = tile_coord(t, n_items, n_tiles);
        const int it = __ldcg(l.blocks + c.m_blk);
        w.expert = it & 1023, w.row0 = (it >> 10) * BM, w.n_tile = c.n_tile;
        w.rows = min(BM, (__ldcg(l.row_end + w.expert) - w.row0 + CHUNK - 1) & ~(CHUNK - 1));
    }
    return w;
}
// pair (-1: padding) / weight of the rows `lane` of an epilogue group's chunks
__device__ __forceinline__ void fetch_pairs(const Args &a, const Tile &w, int grp, int lane, int2 (&r)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int ch = grp + 2 * j;
        r[j] = make_int2(-1, 0);
        if (ch * CHUNK < w.rows) {
            const int p = a.sorted_ids[w.row0 + ch * CHUNK + lane];
            if (p >= 0 && p < a.M) r[j] = make_int2(p, __float_as_int(a.topk_weights[p]));
        }
    }
}
// token / weight of the rows `lane` of an epilogue group's (at most four) chunks
__device__ __forceinline__ void fetch_rows(const int2 *row_info, const Tile &w, int grp, int lane, int2 (&r)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int ch = grp + 2 * j;
        r[j] = make_int2(-1, 0);
        if (ch * CHUNK < w.rows) r[j] = __ldcg(row_info + w.row0 + ch * CHUNK + lane);
    }
}

// 32 rows x 32 bf16 between a row-major matrix and a 64-byte-swizzled tile, four lanes a row, 16 bytes each
__device__ __forceinline__ uint32_t tile64(uint32_t r, uint32_t chunk) { return r * 64 + ((chunk ^ ((r >> 1) & 3)) << 4); }
__device__ __forceinline__ void load_tile64(uint32_t tile, const __nv_bfloat16 *src, size_t ld, int lane) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t r = 8 * i + (lane >> 2), c = lane & 3;
        cp_async_16(tile + tile64(r, c), src + r * ld + c * 8);
    }
}
__device__ __forceinline__ void store_tile64(uint32_t tile, __nv_bfloat16 *dst, size_t ld, int lane) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t r = 8 * i + (lane >> 2), c = lane & 3;
        *reinterpret_cast<uint4 *>(dst + r * ld + c * 8) = ld_shared_u4(tile + tile64(r, c));
    }
}
// SwiGLU derivative of one element, c = d_out . W2 before the routing weight
struct SwigluGrad {
    float act, gate, up;      // weight * act, d_gate, d_up
};
__device__ __forceinline__ SwigluGrad swiglu_grad(float c, float g, float u, float weight, bool valid, float &d_weight) {
    // a padding row of kept pre-activations is whatever the forward call found in its workspace; its products must be zeros
    // (the weight gradients contract over it), not 0 * NaN
    if (!valid) c = g = u = 0.f;
    const float s = 1.f / (1.f + __expf(-g));
    const float silu = g * s;
    const float act = silu * u;
    const float d = weight * c;
    d_weight += c * act;
    return {weight * act, d * u * s * (1.f + g * (1.f - s)), d * silu};
}

// kKeep: the gate/up kernel also stores the pre-activations (bf16, [sorted_num, N]) for a later backward pass
// kMx: OCP-MX operands (e4m3 + e8m0 scales per 32), block-scaled MMAs, MX activations between the two kernels
template <int kMode, bool kKeep = false, bool kMx = false>
__global__ void __launch_bounds__(THREADS<kMode, kMx>, 1)
moe_tokn_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_rows,
                const __grid_constant__ CUtensorMap map_rows16, const __grid_constant__ CUtensorMap map_act,
                const __grid_constant__ CUtensorMap map_gu, const Args a) {
    extern __shared__ uint8_t smem_raw[];
    constexpr bool kUp = kMode == UP, kBulk = kMode == DOWN_BULK, kDown = kMode == DOWN || kBulk, kBackward = kMode >= GATE_UP;
    constexpr bool kMMajor = kMode >= D_ACT;
    constexpr int kBufs = BUFS<kMode, kKeep, kMx>;
    constexpr uint32_t kBufBytes = BUF_BYTES<kMode, kKeep, kMx>;
    constexpr int kBK = BK<kMx>;
    constexpr int kBigBox = kMx ? 32 : 64;      // rows of a box of map_rows (mxfp8: half of 192 rows is three of them)
    // mxfp8 stores no tile by TMA: the two maps are those of the scale tiles (rows: two tiles a box; weights, down: one)
    const CUtensorMap &map_sfr = map_act, &map_sfw = map_gu;
    Smem sm;
    sm.stage_bytes = a.stage_bytes, sm.sf_off = a.sf_off;
    sm.ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    sm.staging = sm.ring + a.stages * a.stage_bytes;
    sm.sfa_ring = sm.staging + 2 * kBufs * kBufBytes;
    sm.bars = sm.sfa_ring + (kUp && kMx ? SFA_BYTES : 0);
    int *status = &g_status_tokn;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(sm.full(s), kUp ? 3 : 1);      // the even CTA's producer (and both CTAs' gather publishers)
            mbar_init(sm.empty(s), 1);
            if (kUp) mbar_init(sm.gathered(s), GATHER_THREADS);
        }
        for (int b = 0; kUp && kMx && b < SFA_BATCHES; ++b) {
            mbar_init(sm.scaled(b), 32);
            mbar_init(sm.sfa_full(b), 2);      // both CTAs' publishers
            mbar_init(sm.sfa_empty(b), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(sm.tmem_full(b), 1);
            mbar_init(sm.tmem_empty(b), 2 * EPI_WARPS);
        }
        for (int i = 0; i < 2 * kBufs; ++i) {
            mbar_init(sm.staged(i), 4);
            mbar_init(sm.freed(i), 1);
        }
        fence_mbar_init();
        tma_prefetch_desc(&map_w);
        if (!kUp) tma_prefetch_desc(&map_rows);
        if (!kUp) tma_prefetch_desc(&map_rows16);
        if (kUp || kMx) tma_prefetch_desc(&map_act);
        if (!kUp && kMx) tma_prefetch_desc(&map_gu);
    }
    if (warp == 1) tmem_alloc_pair(sm.tmem_slot(), TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();      // both CTAs' barriers are initialised and both halves of TMEM allocated
    tc_fence_after();
    uint32_t tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(sm.tmem_slot()));

    // Gate/up: everything comes from the preparation. Its dependents are let go only now: a down CTA that starts knows
    // that every gate/up CTA has passed this wait, hence that the items and row info are there, and that a CTA it shares
    // an SM with holds its TMEM already (it blocks in its own allocation until those columns are freed). The down
    // kernel's threads wait where they first touch what gate/up writes: activations and the zeroed `out`.
    if (kUp || kBackward) {
        if (a.use_pdl) pdl_wait_primary();
        pdl_launch_dependents();
    }

    const int n_items = __ldcg(kBackward ? a.list.count : a.item_count);
    const int4 *items = a.items - n_items;
    const int n_tiles = kUp ? a.H / 128 : ((kBackward ? a.cols : a.K) + 255) / 256;
    const int num_tiles = n_items * n_tiles;
    const int ksteps = (kBackward ? a.k : kUp ? a.K : a.H) / kBK;
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1;
    auto fetch = [&](int t) {
        return kBackward ? fetch_block_tile(a.list, t, num_tiles, n_items, n_tiles)
                         : fetch_tile(items, t, num_tiles, n_items, n_tiles);
    };

    if (warp == 0) {
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            long long issued = 0;
            bool ok = true;
            Tile w, next = fetch(first);
            for (int t = first; t < num_tiles && ok; t += step) {
                w = next;
                next = fetch(t + step);
                const int half = w.rows >> 1;
                const int row0 = w.row0 + static_cast<int>(rank) * half;
                const bool big = half > 32;
                const int box = big ? kBigBox : 16;
                const int boxes = (half + box - 1) / box;
                const uint32_t bytes = 2 * (A_BYTES + (kUp ? 0u : static_cast<uint32_t>(boxes * box) * 128u) +
                                            (!kMx ? 0 : kUp ? 2 * SF_TILE : 3 * SF_TILE));
                auto load_weights = [&](int slot, int ks) {
                    const uint32_t full_leader = mapa_shared(sm.full(slot), 0);
                    if (leader) mbar_arrive_expect_tx(sm.full(slot), bytes);
                    if (kMMajor) {
                        const int krow = w.expert * a.k + ks * kBK;
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            tma_load_2d_pair(sm.a(slot) + i * 8192, &map_w, full_leader,
                                             w.n_tile * 256 + static_cast<int>(rank) * 128 + i * 64, krow);
                    } else if (kUp)
                        tma_load_5d_pair(sm.a(slot), &map_w, full_leader, ks * kBK, 0, 0,
                                         w.n_tile * 8 + static_cast<int>(rank) * 4, w.expert);
                    else
                        tma_load_2d_pair(sm.a(slot), &map_w, full_leader, ks * kBK,
                                         w.expert * (kBackward ? a.cols : a.K) + w.n_tile * 256 + static_cast<int>(rank) * 128);
                    if (kMx && !kUp)
                        tma_load_2d_pair(sm.sf(slot) + 2 * SF_TILE, &map_sfw, full_leader, 0,
                                         ((w.expert * a.K + w.n_tile * 256) / 128 + static_cast<int>(rank)) * ksteps + ks);
                };
                // down: the weights of the first round of slots do not depend on gate/up, only their rows do
                const int early = kDown && t == first ? min(a.stages, ksteps) : 0;
                for (int ks = 0; ks < early; ++ks) load_weights(ks, ks);
                const long long before = issued;
                if (kDown && t == first && a.use_pdl) pdl_wait_primary();
                for (int ks = 0; ks < ksteps; ++ks) {
                    ok = mbar_wait(sm.empty(s), ph ^ 1, status, ST_TIMEOUT_EMPTY);
                    if (!ok) break;
                    const uint32_t full_leader = mapa_shared(sm.full(s), 0);
                    if (ks >= early) load_weights(s, ks);
                    if (kMx) tma_load_2d_pair(sm.sf(s), &map_sfr, full_leader, 0, ks * a.blocks + (w.row0 >> 7));
                    for (int j = 0; !kUp && j < boxes; ++j)
                        tma_load_2d_pair(sm.b(s) + j * box * 128, big ? &map_rows : &map_rows16, full_leader, ks * kBK,
                                         row0 + j * box);
                    ++issued;
                    if (++s == a.stages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (!ok) issued = max(issued, before + early);
            }
            if (!ok) drain_pair_fills(leader, [&](int slot) { return sm.full(slot); }, a.stages, issued);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (leader && elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            int it_n = 0;
            uint32_t fill = 0;
            bool ok = true;
            Tile w, next = fetch(first);
            for (int t = first; t < num_tiles && ok; t += step, ++it_n) {
                w = next;
                next = fetch(t + step);
                const uint32_t idesc = kMx ? idesc_mxf8_f32(256, static_cast<uint32_t>(w.rows))
                                           : idesc_bf16_f32(256, static_cast<uint32_t>(w.rows)) | (kMMajor ? 1u << 15 : 0u);
                // a piece starts at row 0 or 64 of a scale tile: 32 rows a TMEM column
                const uint32_t sf_col = (w.row0 & 64) >> 5;
                const bool two_tiles = (w.row0 & 64) + w.rows > 128;
                const int buf = it_n & 1;
                ok = mbar_wait(sm.tmem_empty(buf), ((it_n >> 1) & 1) ^ 1, status, ST_TIMEOUT_TMEM_EMPTY);
                if (!ok) break;
                tc_fence_after();
                const uint32_t d = tmem_base + buf * ACC_COLS<kMx>;
                for (int ks = 0; ks < ksteps; ++ks, ++fill) {
                    ok = mbar_wait(sm.full(s), ph, status, ST_TIMEOUT_FULL);
                    if (!ok) break;
                    tc_fence_after();
                    if (kMx) {
                        const uint32_t batch = (fill >> 1) % SFA_BATCHES, odd = fill & 1;
                        if (kUp && !odd) {
                            ok = mbar_wait(sm.sfa_full(batch), (fill / (2 * SFA_BATCHES)) & 1, status, ST_TIMEOUT_FULL);
                            if (!ok) break;
                            tc_fence_after();
                        }
                        const uint32_t sfa = tmem_base + SF_TMEM + 16u * (fill & 7), sfb = sfa + 4;
                        tmem_cp_sf_32x128b_warpx4_pair(sfa, smem_desc_sf(kUp ? sm.sfa(batch) + odd * SF_TILE
                                                                             : sm.sf(s) + 2 * SF_TILE));
                        tmem_cp_sf_32x128b_warpx4_pair(sfb, smem_desc_sf(sm.sf(s)));
                        if (two_tiles) tmem_cp_sf_32x128b_warpx4_pair(sfb + 4, smem_desc_sf(sm.sf(s) + SF_TILE));
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k)
                            umma_mxf8_pair(d, smem_desc_sw128(sm.a(s) + k * 32), smem_desc_sw128(sm.b(s) + k * 32),
                                           idesc_with_sf_ids(idesc, k, k), sfa, sfb + sf_col, (ks | k) != 0);
                        if (kUp && odd) umma_commit_pair(sm.sfa_empty(batch), 3);
                    } else {
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_f16_pair(d, kMMajor ? smem_desc_m_sw128(sm.a(s) + k * 2048) : smem_desc_sw128(sm.a(s) + k * 32),
                                          smem_desc_sw128(sm.b(s) + k * 32), idesc, (ks | k) != 0);
                    }
                    umma_commit_pair(sm.empty(s), 3);
                    if (++s == a.stages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (ok) umma_commit_pair(sm.tmem_full(buf), 3);
            }
        }
        __syncwarp();
    } else if (warp < 2 + EPI_WARPS) {
        // ---------------- epilogue ----------------
        const int grp = (warp - 2) >> 2;
        const uint32_t quarter = warp & 3;
        const uint32_t lane_base = quarter * 32;
        if (kUp && a.zero_out) {
            int4 *o4 = reinterpret_cast<int4 *>(a.out);
            const long long live = a.live_rows ? max(0, min(a.M, *a.live_rows)) : a.M;
            const long long n4 = live * a.K / 8;
            const int4 z = make_int4(0, 0, 0, 0);
            for (long long i = static_cast<long long>(blockIdx.x) * (EPI_WARPS * 32) + (threadIdx.x - 64); i < n4;
                 i += static_cast<long long>(gridDim.x) * (EPI_WARPS * 32))
                o4[i] = z;
        }
        // Lanes are weight rows, columns routed rows: the accumulator has to be transposed on its way to the staging
        // buffer. The 16-lane TMEM load gives matrix fragments that stmatrix stores transposed, eight elements a lane.
        // (One column a thread and 2-byte stores with a shuffle per element was bound by them: 4 us a tile.)
        const uint32_t mat = lane >> 3, mrow = lane & 7;
        const uint32_t off = kMode == D_ACT ? tile64(mrow, mat)
                             : kBulk ? mrow * BULK_ROW_BYTES + (quarter * 32 + 8 * mat) * 2
                             : !kUp ? mrow * DOWN_ROW_BYTES + 16 * mat
                             : kMx ? 2 * (lane & 3) * MX_UP_ROW_BYTES + (quarter * 16 + (lane >> 2)) * 4
                                   : (8 * (mat >> 1) + mrow) * 128 + (((2 * quarter + (mat & 1)) ^ mrow) << 4);
        int it_n = 0;
        uint32_t chunk_n = 0;       // chunks of this group so far
        bool ok = true;
        Tile w, next = fetch(first);
        int2 info[4], info_next[4];
        // D_ACT: pre-activations of a chunk, copied into one of the warp's two pairs of tiles while the chunk before is worked on
        uint32_t side = 0;
        bool loaded = false;
        auto load_gate_up = [&](const Tile &t, int ch, uint32_t to) {
            if (ch * CHUNK >= t.rows) return false;
            const int h0 = t.n_tile * 256 + static_cast<int>(rank * 128 + quarter * 32);
            const uint32_t tile = sm.staging + (warp - 2) * kBufBytes + 2 * to * D_ACT_TILE;
            const __nv_bfloat16 *src = a.gu + (static_cast<size_t>(t.row0) + ch * CHUNK) * 2 * a.H + h0;
            if (h0 < a.H) {
                load_tile64(tile, src, 2 * a.H, lane);
                load_tile64(tile + D_ACT_TILE, src + a.H, 2 * a.H, lane);
            }
            return true;
        };
        if (kDown) fetch_rows(a.row_info, next, grp, lane, info_next);
        if (kMode == D_ACT) fetch_pairs(a, next, grp, lane, info_next);
        if (kMode == DOWN && a.use_pdl) pdl_wait_primary();      // gate/up zeroes `out`
        for (int t = first; t < num_tiles && ok; t += step, ++it_n) {
            w = next;
            next = fetch(t + step);
            const int chunks = w.rows / CHUNK;
            const int buf = it_n & 1;
            if (kDown || kMode == D_ACT) {
#pragma unroll
                for (int j = 0; j < 4; ++j) info[j] = info_next[j];
            }
            if (kMode == D_ACT && !loaded) {
                loaded = load_gate_up(w, grp, side);
                cp_async_commit();
            }
            ok = warp_wait(sm.tmem_full(buf), (it_n >> 1) & 1, status, ST_TIMEOUT_TMEM_FULL, lane);
            if (!ok) break;
            tc_fence_after();
            const uint32_t acc = tmem_base + buf * ACC_COLS<kMx>;
            if (kDown) fetch_rows(a.row_info, next, grp, lane, info_next);
            if (kMode == D_ACT) fetch_pairs(a, next, grp, lane, info_next);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int ch = grp + 2 * j;
                if (ch >= chunks) break;
                float lo[16], hi[16];      // up: 16 gate rows, 16 up rows; down: output columns 0-15, 16-31 of the quarter
                tmem_ld_16x256b_x4(lo, tmem_addr(acc, lane_base, ch * CHUNK));
                tmem_ld_16x256b_x4(hi, tmem_addr(acc, lane_base + 16, ch * CHUNK));
                if (kMode == D_ACT) {
                    // SwiGLU derivative in the fragment layout; the pre-activations come, and d_gate / d_up go, through tiles
                    // in shared memory, so that a row's 64 bytes are four lanes' and the next chunk is on its way meanwhile
                    // (a lane a row, loading where it needs them: d_act 103 -> 106 us at 64 rows an expert, 205 -> 232 at 256)
                    const uint32_t mine = sm.staging + (warp - 2) * kBufBytes, actw = mine + 4 * D_ACT_TILE;
                    const uint32_t gate = mine + 2 * side * D_ACT_TILE, up = gate + D_ACT_TILE;
                    side ^= 1;
                    if (ch + 2 < chunks)
                        load_gate_up(w, ch + 2, side);
                    else
                        loaded = load_gate_up(next, grp, side);
                    cp_async_commit();
                    cp_async_wait_group<1>();
                    tmem_ld_wait();
                    __syncwarp();                   // this chunk's pre-activations have landed
                    const int h0 = w.n_tile * 256 + static_cast<int>(rank * 128 + quarter * 32);
                    float dwt = 0.f;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {   // 8 routed rows x 32 activations; two rows a lane, four activations of each
                        const int r = 8 * q + 2 * (lane & 3);
                        const bool v0 = __shfl_sync(0xffffffffu, info[j].x, r) >= 0;
                        const bool v1 = __shfl_sync(0xffffffffu, info[j].x, r + 1) >= 0;
                        const float w0 = __int_as_float(__shfl_sync(0xffffffffu, info[j].y, r));
                        const float w1 = __int_as_float(__shfl_sync(0xffffffffu, info[j].y, r + 1));
                        uint32_t g[4], u[4], av[4];
                        ldmatrix_x4_trans(gate + off + q * 512, g);
                        ldmatrix_x4_trans(up + off + q * 512, u);
                        float s0 = 0.f, s1 = 0.f;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float c0 = i < 2 ? lo[4 * q + 2 * i] : hi[4 * q + 2 * (i - 2)];
                            const float c1 = i < 2 ? lo[4 * q + 2 * i + 1] : hi[4 * q + 2 * (i - 2) + 1];
                            const SwigluGrad a0 = swiglu_grad(c0, __uint_as_float(g[i] << 16), __uint_as_float(u[i] << 16), w0, v0, s0);
                            const SwigluGrad a1 = swiglu_grad(c1, __uint_as_float(g[i] & 0xffff0000u),
                                                              __uint_as_float(u[i] & 0xffff0000u), w1, v1, s1);
                            av[i] = pack_bf16x2(a0.act, a1.act);
                            g[i] = pack_bf16x2(a0.gate, a1.gate);
                            u[i] = pack_bf16x2(a0.up, a1.up);
                        }
                        stmatrix_x4_trans(gate + off + q * 512, g[0], g[1], g[2], g[3]);
                        stmatrix_x4_trans(up + off + q * 512, u[0], u[1], u[2], u[3]);
                        stmatrix_x4_trans(actw + off + q * 512, av[0], av[1], av[2], av[3]);
#pragma unroll
                        for (int d = 4; d < 32; d <<= 1) {
                            s0 += __shfl_xor_sync(0xffffffffu, s0, d);
                            s1 += __shfl_xor_sync(0xffffffffu, s1, d);
                        }
                        const float t0 = __shfl_sync(0xffffffffu, s0, (lane & 7) >> 1);
                        const float t1 = __shfl_sync(0xffffffffu, s1, (lane & 7) >> 1);
                        if ((lane >> 3) == q) dwt = lane & 1 ? t1 : t0;
                    }
                    __syncwarp();
                    if (h0 < a.H) {
                        const size_t row = static_cast<size_t>(w.row0) + ch * CHUNK;
                        store_tile64(gate, a.c + row * 2 * a.H + h0, 2 * a.H, lane);
                        store_tile64(up, a.c + row * 2 * a.H + a.H + h0, 2 * a.H, lane);
                        store_tile64(actw, a.actw + row * a.H + h0, a.H, lane);
                        if (a.dwt && info[j].x >= 0) atomicAdd(a.dwt + info[j].x, dwt);
                    }
                    __syncwarp();
                    continue;
                }
                if (kBackward) {
                    const uint32_t mine = sm.staging + (warp - 2) * DOWN_BUF_BYTES;
                    tmem_ld_wait();
                    __syncwarp();                   // the previous chunk has been read
#pragma unroll
                    for (int q = 0; q < 4; ++q)     // 8 routed rows x 32 columns
                        stmatrix_x4_trans(mine + off + q * 8 * DOWN_ROW_BYTES, pack_bf16x2(lo[4 * q], lo[4 * q + 1]),
                                          pack_bf16x2(lo[4 * q + 2], lo[4 * q + 3]), pack_bf16x2(hi[4 * q], hi[4 * q + 1]),
                                          pack_bf16x2(hi[4 * q + 2], hi[4 * q + 3]));
                    __syncwarp();
                    const int col = w.n_tile * 256 + static_cast<int>(rank * 128 + quarter * 32) + (lane & 3) * 8;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {   // four lanes a row, 16 bytes each
                        const int r = 8 * i + (lane >> 2);
                        const uint4 v = ld_shared_u4(mine + r * DOWN_ROW_BYTES + (lane & 3) * 16);
                        if (col < a.cols)
                            *reinterpret_cast<uint4 *>(a.c + (static_cast<size_t>(w.row0) + ch * CHUNK + r) * a.ldc + col) = v;
                    }
                    continue;
                }
                if (kMode == DOWN) {
                    const uint32_t mine = sm.staging + (warp - 2) * DOWN_BUF_BYTES;
                    tmem_ld_wait();
                    __syncwarp();                   // the previous chunk has been read
#pragma unroll
                    for (int q = 0; q < 4; ++q) {   // 8 routed rows x 32 output columns
                        const int r = 8 * q + 2 * (lane & 3);
                        const float w0 = __int_as_float(__shfl_sync(0xffffffffu, info[j].y, r));
                        const float w1 = __int_as_float(__shfl_sync(0xffffffffu, info[j].y, r + 1));
                        stmatrix_x4_trans(mine + off + q * 8 * DOWN_ROW_BYTES, pack_bf16x2(w0 * lo[4 * q], w1 * lo[4 * q + 1]),
                                          pack_bf16x2(w0 * lo[4 * q + 2], w1 * lo[4 * q + 3]),
                                          pack_bf16x2(w0 * hi[4 * q], w1 * hi[4 * q + 1]),
                                          pack_bf16x2(w0 * hi[4 * q + 2], w1 * hi[4 * q + 3]));
                    }
                    __syncwarp();
                    const int col = w.n_tile * 256 + static_cast<int>(rank * 128 + quarter * 32) + (lane & 3) * 8;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {   // four lanes a row, 16 bytes each
                        const int r = 8 * i + (lane >> 2);
                        const uint4 v = ld_shared_u4(mine + r * DOWN_ROW_BYTES + (lane & 3) * 16);
                        const int tok = __shfl_sync(0xffffffffu, info[j].x, r);
                        if (tok >= 0 && col < a.K)
                            red_add_bf16x8(a.out + static_cast<size_t>(tok) * a.K + col, v.x, v.y, v.z, v.w);
                    }
                    continue;
                }
                const uint32_t slot = chunk_n % kBufs, round = chunk_n / kBufs;
                const uint32_t base = sm.staging + (grp * kBufs + slot) * kBufBytes + off;
                ok = warp_wait(sm.freed(grp * kBufs + slot), (round & 1) ^ 1, status, ST_TIMEOUT_ACT, lane);
                tmem_ld_wait();
                if (!ok) break;
                if (kUp) {
                    if (kKeep) {
#pragma unroll
                        for (int p = 0; p < 2; ++p) {
                            stmatrix_x4_trans(base + UP_BUF_BYTES + p * 16 * 128, pack_bf16x2(lo[8 * p], lo[8 * p + 1]),
                                              pack_bf16x2(lo[8 * p + 2], lo[8 * p + 3]),
                                              pack_bf16x2(lo[8 * p + 4], lo[8 * p + 5]),
                                              pack_bf16x2(lo[8 * p + 6], lo[8 * p + 7]));
                            stmatrix_x4_trans(base + 2 * UP_BUF_BYTES + p * 16 * 128, pack_bf16x2(hi[8 * p], hi[8 * p + 1]),
                                              pack_bf16x2(hi[8 * p + 2], hi[8 * p + 3]),
                                              pack_bf16x2(hi[8 * p + 4], hi[8 * p + 5]),
                                              pack_bf16x2(hi[8 * p + 6], hi[8 * p + 7]));
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 16; ++i) lo[i] = swiglu(lo[i], hi[i]);
                    if (kMx) {
#pragma unroll
                        for (int q = 0; q < 4; ++q)     // 8 routed rows x 16 activations
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                st_shared_f32(base + (8 * q + (i & 1)) * MX_UP_ROW_BYTES + (i >> 1) * 32, lo[4 * q + i]);
                    }
#pragma unroll
                    for (int p = 0; !kMx && p < 2; ++p)     // 16 routed rows x 16 activations
                        stmatrix_x4_trans(base + p * 16 * 128, pack_bf16x2(lo[8 * p], lo[8 * p + 1]),
                                          pack_bf16x2(lo[8 * p + 2], lo[8 * p + 3]), pack_bf16x2(lo[8 * p + 4], lo[8 * p + 5]),
                                          pack_bf16x2(lo[8 * p + 6], lo[8 * p + 7]));
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {   // 8 routed rows x 32 output columns
                        const int r = 8 * q + 2 * (lane & 3);
                        const float w0 = __int_as_float(__shfl_sync(0xffffffffu, info[j].y, r));
                        const float w1 = __int_as_float(__shfl_sync(0xffffffffu, info[j].y, r + 1));
                        stmatrix_x4_trans(base + q * 8 * BULK_ROW_BYTES, pack_bf16x2(w0 * lo[4 * q], w1 * lo[4 * q + 1]),
                                          pack_bf16x2(w0 * lo[4 * q + 2], w1 * lo[4 * q + 3]),
                                          pack_bf16x2(w0 * hi[4 * q], w1 * hi[4 * q + 1]),
                                          pack_bf16x2(w0 * hi[4 * q + 2], w1 * hi[4 * q + 3]));
                    }
                }
                if (!kMx) fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(sm.staged(grp * kBufs + slot));
                ++chunk_n;
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_peer_tcgen05(mapa_shared(sm.tmem_empty(buf), 0));
        }
        if (kMode == D_ACT) cp_async_wait_all();
    } else if (kUp && warp >= GATHER_WARP<kMx> && warp < GATHER_WARP<kMx> + GATHER_THREADS / 32) {
        // ---------------- gather warps ----------------
        // Rows of x straight into the B tile: 8 lanes copy a row's 128 bytes (thread g rows g / 8 + 16 i) to their place in
        // the 128-byte swizzle. Padding rows are not copied: whatever their lines of the tile hold feeds accumulator columns
        // that nothing reads (and 30 of the 32 rows of a decode piece would be reads of one line by every SM). A thread's copies of a slot arrive on gathered(s) by themselves when they have landed.
        const int g = threadIdx.x - GATHER_WARP<kMx> * 32;
        const int q = g >> 3, chunk = g & 7;
        const size_t row_bytes = static_cast<size_t>(ksteps) * 128;
        const uint32_t off = q * 128 + ((chunk ^ (q & 7)) << 4);
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        auto fetch_tokens = [&](const Tile &w, int (&tok)[8]) {
            const int half = w.rows >> 1;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                tok[i] = -1;
                if (16 * i < half) tok[i] = __ldcg(&a.row_info[w.row0 + static_cast<int>(rank) * half + 16 * i + q].x);
            }
        };
        Tile w, next = fetch(first);
        int tok[8];
        fetch_tokens(next, tok);
        for (int t = first; t < num_tiles && ok; t += step) {
            w = next;
            const uint8_t *src[8];
            uint32_t live = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                src[i] = a.x + max(0, tok[i]) * row_bytes + chunk * 16;
                live |= (tok[i] >= 0 ? 1u : 0u) << i;
            }
            next = fetch(t + step);
            fetch_tokens(next, tok);
            for (int ks = 0; ks < ksteps; ++ks) {
                ok = mbar_wait(sm.empty(s), ph ^ 1, status, ST_TIMEOUT_EMPTY);
                if (!ok) break;
                const uint32_t dst = sm.b(s) + off;
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (live >> i & 1) cp_async_16(dst + i * 16 * 128, src[i] + ks * 128);
                cp_async_mbar_arrive_noinc(sm.gathered(s));
                if (++s == a.stages) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
        cp_async_wait_all();
    } else if (kUp && warp == GATHER_WARP<kMx> + GATHER_THREADS / 32) {
        // ---------------- gather publisher ----------------
        // Landed rows (generic-proxy writes) -> visible to the MMA -> one arrival on the even CTA's barrier. Not done by the
        // gather warps, whose copies of the next slots are in flight: a proxy fence would wait for them.
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int t = first; t < num_tiles && ok; t += step)
                for (int ks = 0; ks < ksteps; ++ks) {
                    ok = mbar_wait(sm.gathered(s), ph, status, ST_TIMEOUT_FULL);
                    if (!ok) break;
                    fence_proxy_async_smem();
                    mbar_arrive_peer_tcgen05(mapa_shared(sm.full(s), 0));
                    if (++s == a.stages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
        }
        __syncwarp();
    } else if (kUp && kMx && warp == SCALE_WARP) {
        // ---------------- scale warp ----------------
        // The A tile interleaves 16 gate and 16 up rows in each group of 32; their scales lie in two 512-byte tiles of w_scales.
        // Lane l puts line l of the A tile's own scale tile together, a word from each group, with cp.async; a lane's
        // copies of a batch arrive on scaled(b) by themselves when they have landed. (The rows' scales gathered here as well,
        // six more words a lane and k-step, made the call 1.3 times as long at 300 rows per expert: plan_kernel tiles them.)
        int b = 0;
        uint32_t ph = 0;
        bool ok = true;
        Tile w, next = fetch(first);
        for (int t = first; t < num_tiles && ok; t += step) {
            w = next;
            next = fetch(t + step);
            const int tile_row = w.expert * 2 * a.H + (lane < 16 ? 0 : a.H) + w.n_tile * 128;
            const uint32_t *src = a.w_scales + static_cast<size_t>(tile_row >> 7) * ksteps * 128 + (lane & 15) * 4 + 2 * rank;
            for (int ks = 0; ks < ksteps; ks += 2) {       // K is a multiple of 256
                ok = warp_wait(sm.sfa_empty(b), ph ^ 1, status, ST_TIMEOUT_EMPTY, lane);
                if (!ok) break;
                const uint32_t dst = sm.sfa(b) + lane * 16;
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int g = 0; g < 4; ++g)   // group g: activations 16 g ... 16 g + 15 of this CTA's 64
                        cp_async_4_l2(dst + i * SF_TILE + 4 * g, src + i * 128 + (g & 1) * 64 + (g >> 1));
                src += 256;
                cp_async_mbar_arrive_noinc(sm.scaled(b));
                if (++b == SFA_BATCHES) {
                    b = 0;
                    ph ^= 1;
                }
            }
        }
        cp_async_wait_all();
    } else if (kUp && kMx && warp == SCALE_WARP + 1) {
        // ---------------- scale publisher ----------------
        // Landed scale tiles (generic-proxy writes) -> visible to tcgen05.cp -> one arrival on the even CTA's barrier. Not done
        // by the scale warp, whose copies of the next batches are in flight: a proxy fence would wait for them.
        if (elect_one()) {
            int b = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int t = first; t < num_tiles && ok; t += step)
                for (int ks = 0; ks < ksteps; ks += 2) {
                    ok = mbar_wait(sm.scaled(b), ph, status, ST_TIMEOUT_FULL);
                    if (!ok) break;
                    fence_proxy_async_smem();
                    mbar_arrive_peer_tcgen05(mapa_shared(sm.sfa_full(b), 0));
                    if (++b == SFA_BATCHES) {
                        b = 0;
                        ph ^= 1;
                    }
                }
        }
        __syncwarp();
    } else if (kUp || kBulk) {
        // ---------------- store warps ----------------
        const int grp = warp - STORE_WARP;
        uint32_t chunk_n = 0;
        bool ok = true;
        Tile w, next = fetch(first);
        int2 info[4], info_next[4];
        if (kBulk) fetch_rows(a.row_info, next, grp, lane, info_next);
        if (kBulk && a.use_pdl) pdl_wait_primary();      // gate/up zeroes `out`
        for (int t = first; t < num_tiles && ok; t += step) {
            w = next;
            next = fetch(t + step);
            const int chunks = w.rows / CHUNK;
            const int col0 = kBulk ? w.n_tile * 256 + static_cast<int>(rank) * 128 : w.n_tile * 128 + static_cast<int>(rank) * 64;
            if (kBulk) {
#pragma unroll
                for (int j = 0; j < 4; ++j) info[j] = info_next[j];
                fetch_rows(a.row_info, next, grp, lane, info_next);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int ch = grp + 2 * j;
                if (ch >= chunks) break;
                const uint32_t slot = chunk_n % kBufs, round = chunk_n / kBufs;
                const uint32_t base = sm.staging + (grp * kBufs + slot) * kBufBytes;
                ok = warp_wait(sm.staged(grp * kBufs + slot), round & 1, status, ST_TIMEOUT_ACT, lane);
                if (!ok) break;
                if (kMx) {
                    // a lane's row: two MX blocks of 32 activations, quantised as in moe_mxfp8.cu
                    const size_t row = static_cast<size_t>(w.row0) + ch * CHUNK + lane;
                    uint32_t e2 = 0;
#pragma unroll
                    for (int blk = 0; blk < 2; ++blk) {
                        float v[32];
                        float amax = 0.f;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float4 f = ld_shared_f4(base + lane * MX_UP_ROW_BYTES + blk * 128 + i * 16);
                            v[4 * i] = f.x, v[4 * i + 1] = f.y, v[4 * i + 2] = f.z, v[4 * i + 3] = f.w;
                        }
#pragma unroll
                        for (int i = 0; i < 32; ++i) amax = fmaxf(amax, fabsf(v[i]));
                        float inv;
                        e2 |= mx_block_scale(amax, &inv) << (8 * blk);
                        uint32_t q[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            q[i] = pack_e4m3x4(v[4 * i] * inv, v[4 * i + 1] * inv, v[4 * i + 2] * inv, v[4 * i + 3] * inv);
                        st_global_v8(a.act_q + row * a.H + col0 + blk * 32, q);
                    }
                    const uint32_t r = static_cast<uint32_t>(row) & 127;
                    *reinterpret_cast<uint16_t *>(a.act_sf + (static_cast<size_t>(w.n_tile) * a.blocks + (row >> 7)) * SF_TILE +
                                                  (r & 31) * 16 + (r >> 5) * 4 + rank * 2) = static_cast<uint16_t>(e2);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(sm.freed(grp * kBufs + slot));
                    ++chunk_n;
                    continue;
                }
                if (kBulk) {
                    if (info[j].x >= 0 && col0 < a.K)
                        bulk_reduce_add_bf16(a.out + static_cast<size_t>(info[j].x) * a.K + col0, base + lane * BULK_ROW_BYTES, 256);
                } else if (lane == 0) {
                    tma_store_2d(&map_act, base, col0, w.row0 + ch * CHUNK);
                    if (kKeep) {
                        tma_store_2d(&map_gu, base + UP_BUF_BYTES, col0, w.row0 + ch * CHUNK);
                        tma_store_2d(&map_gu, base + 2 * UP_BUF_BYTES, a.H + col0, w.row0 + ch * CHUNK);
                    }
                }
                tma_store_commit();
                tma_store_wait_read<1>();      // the previous chunk's buffer has been read
                __syncwarp();
                if (chunk_n > 0 && lane == 0) mbar_arrive(sm.freed(grp * kBufs + (chunk_n - 1) % kBufs));
                ++chunk_n;
            }
        }
        tma_store_wait<0>();
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync_all();      // nobody frees TMEM or exits while the peer may still use this CTA's memory
    if (warp == 1) tmem_dealloc_pair(tmem_base, TMEM_COLS);
}

// w1 [E, 2H, K] as (K, 16, gate | up, H / 16, E): one box = 128 bytes of k x (16 gate rows, 16 up rows) x 4 groups
int make_gate_up_map(CUtensorMap *map, const void *w, int E, int H, int K, bool mx) {
    const cuuint64_t k2 = static_cast<cuuint64_t>(K) * (mx ? 1 : 2);
    const cuuint64_t dims[5] = {static_cast<cuuint64_t>(K), 16, 2, static_cast<cuuint64_t>(H) / 16,
                                static_cast<cuuint64_t>(E)};
    const cuuint64_t strides[4] = {k2, static_cast<cuuint64_t>(H) * k2, 16 * k2, 2 * static_cast<cuuint64_t>(H) * k2};
    const cuuint32_t box[5] = {mx ? 128u : 64u, 16, 2, 4, 1};
    return make_tmap_nd(map, mx ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, w, dims, strides, box,
                        CU_TENSOR_MAP_SWIZZLE_128B, "w (gate | up interleaved)");
}

template <int kMode, bool kKeep = false, bool kMx = false>
int launch(const CUtensorMap &mw, const CUtensorMap &mrows, const CUtensorMap &m16, const CUtensorMap &mact,
           const CUtensorMap &mgu, Args a, int cap, long long max_tiles, cudaStream_t stream) {
    constexpr bool kUp = kMode == UP;
    // 1 KB-aligned slots: weights + the rows one CTA loads (a piece's half, in boxes) (+ scale tiles)
    a.sf_off = A_BYTES + (cap / 2) * 128;
    a.stage_bytes = a.sf_off + (kMx ? SF_BYTES<kUp> : 0);
    const uint32_t fixed = 1024 + 2 * BUFS<kMode, kKeep, kMx> * BUF_BYTES<kMode, kKeep, kMx> + (kUp && kMx ? SFA_BYTES : 0) + BAR_BYTES;
    a.stages = std::min<int>(MAX_STAGES, static_cast<int>((SMEM_LIMIT - fixed) / a.stage_bytes));
    const size_t smem = fixed + static_cast<size_t>(a.stages) * a.stage_bytes;
    auto kernel = moe_tokn_kernel<kMode, kKeep, kMx>;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(THREADS<kMode, kMx>);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = a.use_pdl ? 2 : 1;
    // CTA pairs that fit the device: one a SM pair whatever the ring depth, asked for once per device
    static std::atomic<int> pairs_of[64];
    int dev = 0;
    PMOE_CUDA_OK(cudaGetDevice(&dev));
    PMOE_REQUIRE(dev >= 0 && dev < 64, PMOE_ERR_UNSUPPORTED, "device ordinal %d out of range", dev);
    int max_clusters = pairs_of[dev].load(std::memory_order_acquire);
    if (max_clusters == 0) {
        PMOE_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SMEM_LIMIT)));
        cudaLaunchConfig_t probe = cfg;
        probe.gridDim = dim3(2);
        probe.numAttrs = 1;
        PMOE_CUDA_OK(cudaOccupancyMaxActiveClusters(&max_clusters, kernel, &probe));
        if (max_clusters < 1) return set_error(PMOE_ERR_CUDA, "no CTA pair of the token-N kernel fits on this device");
        pairs_of[dev].store(max_clusters, std::memory_order_release);
    }
    cfg.gridDim = dim3(2 * static_cast<unsigned>(std::min<long long>(max_tiles, max_clusters)));
    PMOE_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, mw, mrows, m16, mact, mgu, a));
    return PMOE_OK;
}

}  // namespace

// Rows of one work item at most, from the average rows per expert. Weight streaming wants many small ring slots (nine
// of 20 KB at cap 64), compute wants wide accumulators (256 leaves TMEM for a second one); a cap below an expert's rows
// reads its weights once per piece. Measured, us at cap 64 / 128 / 256: 28 rows 270 / 272 / 282; 41 rows 236 / 218 /
// 221; 65 rows 423 / 359 / 377; 122 rows 188 / 148 / 149; 140 rows 1118 / 862 / 777.
int tokn_cap(long long rows, int E, bool mx) {
    // mxfp8: 192 leaves a second accumulator; 128 is never the better one (us at 128 / 192: K = 6400, N = 1280, 87 rows 459 /
    // 416; K = 3584, N = 10240, 106 rows 301 / 270; below 32 rows 64 and 192 differ by 3 % either way)
    if (mx) return rows <= 32ll * E ? 64 : 192;
    return rows <= 32ll * E ? 64 : rows <= 112ll * E ? 128 : 256;
}

// How the down kernel adds its rows. Bulk reductions move 256 bytes an operation instead of 16, which counts at the power
// cap: with many rows and a contraction long enough to cover their 31 ns each (whole call, vector / bulk, us, runs of 1 s back
// to back: K = 4096, N = 3072, 524288 Zipf rows 18202 / 17875, 32 experts, 4096 rows each 4196 / 4163; K = 5120, N = 2048, 2200
// rows each 1018 / 1001; K = 6144, N = 5120, 2048 rows each 12118 / 11928). Shorter contractions do not cover them (N = 1536,
// 512 rows 677 / 682, 11000 rows 1.02; N = 1280, 3277 rows 1293 / 1352; N = 768, 4096 rows 1294 / 1441); at 512 rows per expert
// the two are within 1 % of each other, and below the staging's 51 KB, taken from the ring, cost more (1.00 - 1.09).
// mxfp8's MMAs take half the time: vector reductions everywhere (K = 2048, N = 1536, 5003 tokens 101 / 133).
static bool tokn_bulk_down(int M, int N, int E, int top_k) {
    return N >= 2048 && static_cast<long long>(M) * top_k >= 1024ll * E;
}

// the count, at most two pieces per 128-row block (cap 64) and the row info
size_t tokn_items_bytes(int sorted_num) {
    return (static_cast<size_t>(sorted_num / BM) * 2 + 1) * sizeof(int4) + static_cast<size_t>(sorted_num) * sizeof(int2);
}

int run_tokn(const ToknProblem &p, void *act, void *items, int phases, cudaStream_t stream) {
    const int H = p.N / 2;
    const int max_blocks = p.sorted_num / BM;
    const int cap = tokn_cap(static_cast<long long>(p.M) * p.top_k, p.E, p.w_scales != nullptr);
    int32_t *count = static_cast<int32_t *>(items);
    int4 *items_end = static_cast<int4 *>(items) + 1 + 2 * static_cast<size_t>(max_blocks);
    int2 *row_info = reinterpret_cast<int2 *>(items_end);
    Args a{};
    a.row_info = row_info;
    a.out = static_cast<__nv_bfloat16 *>(p.out);
    a.live_rows = p.live_rows;
    a.items = items_end, a.item_count = count;
    a.M = p.M, a.K = p.K, a.H = H;

    const bool mx = p.w_scales != nullptr;
    const int gran = mx ? 64 : 32;
    a.blocks = max_blocks;
    a.act_q = static_cast<uint8_t *>(act), a.act_sf = p.act_sf;

    CUtensorMap w1, w2, actb, act16, act_st;
    const auto type = mx ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const uint32_t elem = mx ? 1 : 2, bk = 128 / elem, big = mx ? 32 : 64;
    constexpr auto SW = CU_TENSOR_MAP_SWIZZLE_128B;
    if (int rc = make_gate_up_map(&w1, p.w, p.E, H, p.K, mx)) return rc;
    if (int rc = make_tmap_2d(&w2, type, elem, p.w2, static_cast<uint64_t>(p.E) * p.K, H, 128, bk, SW, "w2")) return rc;
    // (encoding a map takes the host 1 us: the larger box only where a CTA's half of a piece can have more than 32 rows)
    if (int rc = make_tmap_2d(&act16, type, elem, act, p.sorted_num, H, 16, bk, SW, "act (16 rows)")) return rc;
    actb = act16;
    if (cap > 64)
        if (int rc = make_tmap_2d(&actb, type, elem, act, p.sorted_num, H, big, bk, SW, "act")) return rc;
    if (!mx)
        if (int rc = make_tmap_2d(&act_st, type, elem, act, p.sorted_num, H, CHUNK, bk, SW, "act (store)")) return rc;

    a.x = static_cast<const uint8_t *>(p.x);
    const int sms = sm_count();
    const bool pdl = pdl_enabled();
    const long long max_items = std::min<long long>(2ll * max_blocks,
                                                    (static_cast<long long>(p.M) * p.top_k + cap - 1) / cap + max_blocks);
    // The work items and the row info are built in every call, whatever the phase mask: the kernels below index with them.
    {
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.blockDim = dim3(PLAN_THREADS);
        cfg.stream = stream;
        cfg.attrs = attr;
        cfg.numAttrs = pdl ? 1 : 0;
        const auto *x_scales = mx && (phases & 1) ? static_cast<const uint32_t *>(p.x_scales) : nullptr;
        // one CTA a scale tile column (128 rows), or a thread a row
        cfg.gridDim = dim3(1 + std::min(3 * sms, mx ? max_blocks : (p.sorted_num + PLAN_THREADS - 1) / PLAN_THREADS));
        PMOE_CUDA_OK(cudaLaunchKernelEx(&cfg, plan_kernel, p.sorted_ids, p.expert_ids, p.npp, p.topk_weights, p.M, p.top_k,
                                        p.sorted_num, cap, gran, p.bpc, items_end, count, row_info, x_scales,
                                        reinterpret_cast<uint32_t *>(p.x_sf), p.K / 128));
    }
    if (phases & 2) {
        Args up = a;
        up.use_pdl = pdl ? 1 : 0;
        up.zero_out = 1;
        up.w_scales = static_cast<const uint32_t *>(p.w_scales);
        const long long tiles = max_items * (H / 128);
        int rc = PMOE_OK;
        if (mx) {
            CUtensorMap sfx;
            if ((rc = make_tmap_2d(&sfx, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, p.x_sf, static_cast<uint64_t>(p.K / 128) * max_blocks,
                                   128, 2, 128, CU_TENSOR_MAP_SWIZZLE_NONE, "row scale tiles")))
                return rc;
            rc = launch<UP, false, true>(w1, w1, w1, sfx, sfx, up, cap, tiles, stream);
        } else if (p.gu_out) {
            CUtensorMap gu_st;
            if ((rc = make_tmap_2d(&gu_st, type, elem, p.gu_out, p.sorted_num, p.N, CHUNK, bk, SW, "gate | up (store)")))
                return rc;
            rc = launch<UP, true>(w1, w1, w1, act_st, gu_st, up, cap, tiles, stream);
        } else {
            rc = launch<UP>(w1, w1, w1, act_st, act_st, up, cap, tiles, stream);
        }
        if (rc) return rc;
    }
    if (phases & 4) {
        Args dn = a;
        dn.use_pdl = (pdl && (phases & 2)) ? 1 : 0;
        const long long tiles = max_items * ((p.K + 255) / 256);
        int rc = PMOE_OK;
        if (mx) {
            const uint64_t ht = H / 128;
            CUtensorMap sfa, sfw;
            if ((rc = make_tmap_2d(&sfa, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, p.act_sf, ht * max_blocks, 128, 2, 128,
                                   CU_TENSOR_MAP_SWIZZLE_NONE, "activation scale tiles")))
                return rc;
            if ((rc = make_tmap_2d(&sfw, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, p.w2_scales, static_cast<uint64_t>(p.E) * p.K / 128 * ht,
                                   128, 1, 128, CU_TENSOR_MAP_SWIZZLE_NONE, "w2 scale tiles")))
                return rc;
            rc = launch<DOWN, false, true>(w2, actb, act16, sfa, sfw, dn, cap, tiles, stream);
        } else {
            rc = tokn_bulk_down(p.M, p.N, p.E, p.top_k) ? launch<DOWN_BULK>(w2, actb, act16, act_st, act_st, dn, cap, tiles, stream)
                              : launch<DOWN>(w2, actb, act16, act_st, act_st, dn, cap, tiles, stream);
        }
        if (rc) return rc;
    }
    return PMOE_OK;
}

// Row-space GEMMs of the backward pass where an expert has few rows: every weight is read once and a row block costs what its
// rows need, where the 128-row tile of the kernels in moe_bwd_bf16.cu multiplies padding (K = 2048, N = 1536, 128 experts, 64
// rows each: recompute 154 -> 138 us, d_act 118 -> 103, d_xs 144 -> 140; where the line lies: there).
int tokn_block_gemm(const ToknBackward &p, ToknStep step, cudaStream_t stream) {
    constexpr auto BF16 = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    constexpr auto SW = CU_TENSOR_MAP_SWIZZLE_128B;
    const uint64_t E = p.E;
    const int H = p.N / 2;
    Args a{};
    a.list = p.list;
    a.use_pdl = pdl_enabled() ? 1 : 0;
    a.M = p.M * p.top_k, a.H = H;
    CUtensorMap w, rows, rows16;
    auto row_maps = [&](const void *src, int cols) {
        a.k = cols;
        if (int rc = make_tmap_2d(&rows, BF16, 2, src, p.sorted_num, cols, 64, 64, SW, "rows")) return rc;
        return make_tmap_2d(&rows16, BF16, 2, src, p.sorted_num, cols, 16, 64, SW, "rows (16)");
    };
    const long long tiles = static_cast<long long>(p.sorted_num / BM) *
                            (((step == ToknStep::gate_up ? p.N : step == ToknStep::d_act ? H : p.K) + 255) / 256);
    switch (step) {
        case ToknStep::gate_up:
            a.c = static_cast<__nv_bfloat16 *>(p.gu), a.ldc = a.cols = p.N;
            if (int rc = row_maps(p.xs, p.K)) return rc;
            if (int rc = make_tmap_2d(&w, BF16, 2, p.w1, E * p.N, p.K, 128, 64, SW, "w1 rows")) return rc;
            return launch<GATE_UP>(w, rows, rows16, rows, rows, a, BM, tiles, stream);
        case ToknStep::d_act:
            a.c = static_cast<__nv_bfloat16 *>(p.dgu), a.actw = static_cast<__nv_bfloat16 *>(p.actw);
            a.gu = static_cast<const __nv_bfloat16 *>(p.gu);
            a.sorted_ids = p.sorted_ids, a.topk_weights = p.topk_weights, a.dwt = p.dwt;
            a.cols = H;
            if (int rc = row_maps(p.dos, p.K)) return rc;
            if (int rc = make_tmap_2d(&w, BF16, 2, p.w2, E * p.K, H, 64, 64, SW, "w2 boxes")) return rc;
            return launch<D_ACT>(w, rows, rows16, rows, rows, a, BM, tiles, stream);
        default:
            a.c = static_cast<__nv_bfloat16 *>(p.dxs), a.ldc = a.cols = p.K;
            if (int rc = row_maps(p.dgu, p.N)) return rc;
            if (int rc = make_tmap_2d(&w, BF16, 2, p.w1, E * p.N, p.K, 64, 64, SW, "w1 boxes")) return rc;
            return launch<D_XS>(w, rows, rows16, rows, rows, a, BM, tiles, stream);
    }
}

int wait_ns_store_tokn(unsigned long long ns) {
    PMOE_CUDA_OK(cudaMemcpyToSymbol(g_wait_ns, &ns, sizeof(ns)));
    return PMOE_OK;
}

int status_fetch_tokn(int *value, bool reset) {
    if (value) PMOE_CUDA_OK(cudaMemcpyFromSymbol(value, g_status_tokn, sizeof(int)));
    if (reset) {
        const int zero = 0;
        PMOE_CUDA_OK(cudaMemcpyToSymbol(g_status_tokn, &zero, sizeof(int)));
    }
    return PMOE_OK;
}

}  // namespace pmoe

extern "C" int pmoe_debug_tokn_bulk_down(int M, int N, int num_experts, int top_k) {
    return pmoe::tokn_bulk_down(M, N, num_experts, top_k) ? 1 : 0;
}
