// Dense contraction on the sm_100a tensor cores (3xTF32, fp32 in and out) whose A operand is brought in by the copy engines:
// row-major and transposed matrices (GEMM, InnerProduct, the products of the Winograd algorithm) and "same" stride-1
// convolutions over channels in blocks of 32, with any K.  Same arithmetic, same packed weights and the same
// order of the sum over K as contraction_tf32x3_kernel.  What bounds that kernel is its A side: eight loader warps fetch every
// element of every k-block from global memory with a load of their own, and the loads an SM can have outstanding set a pace of
// about 1150 cycles per k-block (1900 for a row-major matrix, where a warp's load touches 32 rows) against the 768 cycles of
// the k-block's twelve MMAs.  Here
//
//   * A arrives in shared memory by tensor-map copies, one warp issuing them several slots ahead:
//       - K contiguous (row-major matrix): one box of 32 k x 128 rows per k-block, 128-byte swizzled, so that a thread reads its
//         row with eight conflict-free 16-byte loads;
//       - rows contiguous (NCHW pixels, a transposed matrix): the 128 rows of a tile are consecutive pixels that may run over
//         the end of an image, so a slot is put together from units of 32 pixels x 32 channels (4 KB), each one box of the
//         tensor [pixels, channels, images]; pixel q of a slot lies in unit q / 32 and bank q % 32.  No rows are spent on
//         clipped tiles (14x14 planes: 196 = 1.53 tiles);
//       - a convolution of T taps: the slot holds the tile's pixels and a halo to both sides, and serves the T k-blocks of its
//         channel block: tap (dy, dx) is the same pixels dy * W + dx further on.  Where a tap leaves the image (or wraps round
//         the end of a row) the thread reads from a unit of zeros instead.  Planes whose pitch is not a multiple of 16 bytes
//         (27x27) are put into the same slots by a copying warp, 4 bytes a lane;
//   * converter warps (two groups of four taking the k-blocks in turn) read their row's 32 values -- the next k-block's are
//     under way while the current one's are split --, split them into the TF32 part and the remainder and write both to the
//     tensor-memory ring that the MMAs read;
//   * two MMA issuer warps in turn, partial sums of eight k-blocks, as in the general kernel; weights through a ring of five
//     stages;
//   * two sets of four accumulate / epilogue warps, each with half of the tile's columns, hold the fp32 sums in registers
//     (setmaxnreg moves registers from the copying warps to them): the shared memory that the general kernel spends on sums
//     holds A slots here, and the epilogue has eight warps.
//   * Every wait is bounded (device status word + abort flag); each copy-issuing thread waits for its own copies before it
//     leaves, and tensor memory is freed on every path.
//
// What bounds it now is shared memory: per k-block of 128 columns the MMAs read 48 KB of weights (hi twice, lo once), the copies
// write 32 KB of weights and 16 KB (3 KB with nine taps) of A, and the converters read 16 KB: 112 KB at 128 bytes a cycle are 896
// cycles, and 1040 are measured (tensor pipe 75 % active on 4096 x 4096 x 4096; the SM clock then settles at 1.6 GHz).
// Measured against the general kernel, as whole calls (us): before this kernel and with it, 2048^3 A * B^T with the packing of B 134 -> 98.5,
// InnerProduct 2048 -> 1000 on 256 rows of raw weights 38.9 -> 25.1 and on one row of packed ones 24.6 -> 14.9 (launches that start early
// and a cheaper finishing pass are in both); calls captured one after the other, A as it is and four bytes off a 16-byte boundary,
// which is the general kernel's with single loads: 2048^3 A^T * B^T 90 against 107, InnerProduct 2048 -> 1000 on one row 14.7 against
// 17.5, 3x3 128 -> 128 on 28x28 at batch 256 271 against 277, 256 -> 256 on 14x14 283 against 285.
//
// Reference: the implicit GEMM and the plain GEMM of src/kernels/sgemm.cl:71-134.
#define DLP_INLINE_WAITS
#include "tc_device.cuh"
#include <cuda.h>
#include <algorithm>
#include <mutex>
#include <vector>
#include <cstring>

namespace dlp {
namespace st {

using namespace tc;

constexpr int BM = 128, BK = 32;
constexpr int T_STAGES = 4;                 // tensor-memory ring of A
constexpr int MAX_B_STAGES = 6;
constexpr int CHUNK_KB = 8;                 // k-blocks summed inside the tensor core before the sum moves to fp32 adds
constexpr int MAX_S_STAGES = 6;
constexpr int UNIT_BYTES = 32 * 32 * 4;     // 32 channels x 32 pixels
constexpr int MAX_UNITS = 10;               // of a slot
constexpr int MAX_TAPS = 64;
enum { SRC_K, SRC_UNITS, SRC_COPY };        // K contiguous; rows contiguous; rows contiguous at a pitch that a tensor map cannot have
constexpr int A_COL_BASE = 256, TMEM_COLS = 512;
constexpr int WARP_A = 0, WARP_MMA = 1 /* and 2 */, WARP_B = 3, WARP_ACC0 = 4, WARP_CONV0 = 8, WARP_ACC1 = 16;
constexpr int NUM_WARPS = 20, NUM_THREADS = NUM_WARPS * 32;
// Registers per thread of the warpgroups after the split (launched with 96): copies and issue 40, accumulate 128 (64 sums), convert 88:
// 40 + 2 * 128 + 2 * 88 = 472 of 5 * 96 = 480.
constexpr int REGS_LAUNCH = 96, REGS_ISSUE = 40, REGS_ACC = 128, REGS_CONV = 88;
// 96 at launch are what 640 threads leave each.  With units and copies the 128-column kernels spill 60 bytes a thread (88 loaded), the
// narrower ones 20 to 40; with K-major A the 128-column one 32 (64).
static_assert(REGS_ISSUE + 2 * REGS_ACC + 2 * REGS_CONV <= 5 * REGS_LAUNCH, "setmaxnreg draws on the launch's registers");
constexpr int SMEM_LIMIT = 227 * 1024;
constexpr int SMEM_FIXED = 1024 + 1024;     // alignment slack + the barrier block and tables (+ a unit of zeros when there are taps)

// codes left in the device status word
enum { ST_A_EMPTY = 401, ST_B_EMPTY = 402, ST_CONV_FULL = 404, ST_CONV_EMPTY = 405, ST_MMA_A = 406, ST_MMA_B = 407,
       ST_MMA_ACC = 408, ST_EPI_ACC = 409, ST_DRAIN = 411 };

struct Shared {
    unsigned long long sa_full[MAX_S_STAGES];  // a slot's copies landed
    unsigned long long sa_empty[MAX_S_STAGES]; // ... and the converter warps have read their last k-block from it
    unsigned long long full_a[T_STAGES];       // the k-block's hi/lo columns are written to tensor memory (4 converter warps)
    unsigned long long full_b[MAX_B_STAGES];   // a B stage landed
    unsigned long long empty_b[MAX_B_STAGES];  // ... and the MMAs that read it retired
    unsigned long long empty[T_STAGES / 2];    // the MMAs of a pair of k-blocks retired: their tensor-memory columns are free
    unsigned long long acc_full[2], acc_empty[2];
    unsigned long long drain;
    uint32_t tmem_base;
    int abort_flag;
    short2 tap[MAX_TAPS];                      // displacement (dy, dx) of each tap, padding included
};
static_assert(sizeof(Shared) <= 1024, "barrier block");

struct Params {
    long long rows;
    int cols;
    int P;                  // rows per image (the whole matrix when there are no images)
    int W, H;               // input plane of a convolution with taps
    int taps;               // k-blocks per slot (1: no halo, no masks)
    int kw, dil_h, dil_w, pad_h, pad_w;
    int dmin, dmax;         // smallest and largest displacement of a tap in pixels
    int kblocks;            // k-blocks per work item
    int kblocks_all;        // of the whole K (work items of a split K take equal parts)
    int n_tiles, splits;
    long long num_items;    // matrices * items_each
    long long items_each;   // row tiles * n_tiles * splits
    int slot_bytes, s_stages, b_stages;
    const float *a;         // SRC_COPY: the images, channels P floats apart
    long long a_image_stride;
    float *y;
    long long y_row_stride, y_col_stride, y_image_stride;    // y[b * image + pixel * row + col * col_stride]
    long long y_batch_stride, y_split_stride;
    int vec_store;          // columns contiguous and every row 16-byte aligned
    const float *bias;      // per column or null
    int act, post_act;
    const float *residual;  // addressed as y, or null
    float res_scale;
};

struct Item {
    long long m0;           // first row
    int n_tile, part, z;    // z: matrix of a batch
};
__device__ __forceinline__ Item decode(long long item, const Params &q)
{
    Item w;
    w.z = 0;
    if(q.items_each != q.num_items) {
        w.z = int(div32(item, q.items_each));
        item -= w.z * q.items_each;
    }
    long long t = item;
    w.part = 0;
    if(q.splits > 1) {
        t = unsigned(item) / unsigned(q.splits);           // few tiles whenever K is split
        w.part = int(unsigned(item) - unsigned(t) * unsigned(q.splits));
    }
    const long long mt = div32(t, q.n_tiles);
    w.n_tile = int(t - mt * q.n_tiles);
    w.m0 = mt * BM;
    return w;
}

// A copy-issuing thread waits (bounded) for the last `depth` copies it armed before it leaves: nothing may still be
// writing shared memory when the CTA ends.  count: copies issued; the n-th copy used barrier n % depth, phase n / depth.
__device__ __forceinline__ void drain_own(unsigned long long *bars, int depth, uint32_t count, int *status)
{
    for(uint32_t n = count > uint32_t(depth) ? count - depth : 0; n < count; n++) {
        const long long t0 = global_ns();
        while(!mbar_try_wait(&bars[n % depth], (n / depth) & 1)) {
            __nanosleep(256);
            if(global_ns() - t0 > WAIT_LIMIT_NS) { atomicCAS(status, 0, ST_DRAIN); break; }
        }
    }
}

template<int R> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template<int R> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }

// SRC: how A lies in memory and comes in (see the top of the file).
template<int BN, int SRC>
__global__ void __launch_bounds__(NUM_THREADS, 1)
stream_tf32x3_kernel(const __grid_constant__ CUtensorMap tm_a, const float *packed, const Params q, int *status)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    constexpr int B_TILE_BYTES = BN * BK * 4;
    constexpr int B_STAGE_BYTES = 2 * B_TILE_BYTES;              // hi tile, then lo tile
    constexpr bool KMAJOR = SRC == SRC_K;
    constexpr int SETS = BN >= 64 ? 2 : 1;                       // sets of accumulate warps
    constexpr int COLS = BN / SETS;                              // columns of a set
    const int S_STAGES = q.s_stages, B_STAGES = q.b_stages;
    Shared *sh = reinterpret_cast<Shared *>(smem);
    unsigned char *b_ring = smem + 1024;
    unsigned char *a_ring = b_ring + B_STAGES * B_STAGE_BYTES;   // 1024-byte aligned, as the swizzle asks for
    unsigned char *zeros = a_ring + S_STAGES * q.slot_bytes;
    int *abort_flag = &sh->abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kblocks = q.kblocks, T = q.taps;
    const long long my_items = blockIdx.x < q.num_items ? div32(q.num_items - blockIdx.x + gridDim.x - 1, gridDim.x) : 0;

    if(threadIdx.x == 0) {
        for(int s = 0; s < MAX_S_STAGES; s++) { mbar_init(&sh->sa_full[s], SRC == SRC_COPY ? 32 : 1); mbar_init(&sh->sa_empty[s], T == 1 ? 4 : 8); }
        for(int s = 0; s < T_STAGES; s++) mbar_init(&sh->full_a[s], 4);
        for(int s = 0; s < MAX_B_STAGES; s++) { mbar_init(&sh->full_b[s], 1); mbar_init(&sh->empty_b[s], 1); }
        for(int s = 0; s < T_STAGES / 2; s++) mbar_init(&sh->empty[s], 1);
        for(int a = 0; a < 2; a++) { mbar_init(&sh->acc_full[a], 1); mbar_init(&sh->acc_empty[a], 4 * SETS); }
        mbar_init(&sh->drain, 1);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if(!KMAJOR && T > 1) {
        for(int i = threadIdx.x; i < UNIT_BYTES / 4; i += NUM_THREADS) reinterpret_cast<float *>(zeros)[i] = 0.0f;
        if(int(threadIdx.x) < T) {
            const int ky = threadIdx.x / q.kw, kx = threadIdx.x - ky * q.kw;
            sh->tap[threadIdx.x] = make_short2(short(ky * q.dil_h - q.pad_h), short(kx * q.dil_w - q.pad_w));
        }
    }
    if(warp == WARP_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *(volatile uint32_t *)&sh->tmem_base;
    // (each role waits for the kernel before, pdl_wait(), where it first touches global memory or waits for another role: the
    // limit of a barrier wait counts from there, whatever the kernel before takes)

    if(warp < WARP_ACC0) {
        regs_dec<REGS_ISSUE>();
        if(warp == WARP_A) {
            // -------------------------------------------------------------- A copies
            // lane 0 waits for slots and arms them; with units, lane u asks for unit u of every slot of the work item (where it
            // lies is worked out once per item: on one thread that arithmetic was twice the MMAs' time)
            uint32_t pi = 0;
            bool live = true;
            const int slots = kblocks / T;
            for(long long item = blockIdx.x; item < q.num_items && live; item += gridDim.x) {
                const Item w = decode(item, q);
                const int c0 = w.part * slots;
                int units = 1, my_x = 0, my_b = w.z;
                if(!KMAJOR) {
                    int u = 0, b = int(div32(w.m0, q.P)), from = int(w.m0 - (long long)b * q.P), left = int(min((long long)BM, q.rows - w.m0));
                    while(left > 0) {
                        const int n = min(left, q.P - from);
                        const int lo = max(from + q.dmin, 0) & ~3, hi = min(from + n + q.dmax, q.P);
                        const int here = (hi - lo + 31) >> 5;
                        if(lane >= u && lane < u + here) { my_x = lo + (lane - u) * 32; my_b += b; }
                        u += here;
                        left -= n;
                        from = 0;
                        b++;
                    }
                    units = u;
                }
                if(pi == 0) pdl_wait();
                for(int c = 0; c < slots; c++, pi++) {
                    const int s = pi % S_STAGES;
                    if(!warp_wait(&sh->sa_empty[s], ((pi / S_STAGES) & 1) ^ 1, abort_flag, status, ST_A_EMPTY, lane)) { live = false; break; }
                    unsigned char *slot = a_ring + s * q.slot_bytes;
                    if(SRC == SRC_COPY) {
                        // planes whose rows of pixels start on any 4-byte boundary (7x7, 27x27): the warp copies 32 pixels of a channel at
                        // a time; the slot serves all taps, so this is an instruction per 32 * taps values that the MMAs read
                        const uint32_t dst0 = smem_u32(slot) + lane * 4;
                        #pragma unroll 1
                        for(int u = 0; u < units; u++) {
                            const int x = __shfl_sync(0xffffffffu, my_x, u) + lane, b = __shfl_sync(0xffffffffu, my_b, u);
                            const uint32_t bytes = x < q.P ? 4 : 0;                    // beyond the plane: zeros, nothing is read
                            const float *src = q.a + b * q.a_image_stride + (long long)(c0 + c) * BK * q.P + (x < q.P ? x : 0);
                            #pragma unroll 8
                            for(int ch = 0; ch < BK; ch++, src += q.P)
                                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst0 + u * UNIT_BYTES + ch * 128), "l"(src), "r"(bytes)
                                             : "memory");
                        }
                        asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(smem_u32(&sh->sa_full[s])) : "memory");
                        continue;
                    }
                    if(lane == 0) mbar_arrive_expect_tx(&sh->sa_full[s], KMAJOR ? BM * BK * 4 : units * UNIT_BYTES);
                    __syncwarp();
                    if(KMAJOR) { if(lane == 0) tma_load_3d(slot, &tm_a, (c0 + c) * BK, int(w.m0), my_b, &sh->sa_full[s]); }
                    else if(lane < units) tma_load_3d(slot + lane * UNIT_BYTES, &tm_a, my_x, (c0 + c) * BK, my_b, &sh->sa_full[s]);
                }
            }
            __syncwarp();
            if(SRC == SRC_COPY) asm volatile("cp.async.wait_all;" ::: "memory");
            else if(lane == 0) drain_own(sh->sa_full, S_STAGES, pi, status);
        }
        else if(warp == WARP_B) {
            // -------------------------------------------------------------- B copies
            if(lane == 0) {
                uint32_t it = 0;
                bool live = true;
                for(long long item = blockIdx.x; item < q.num_items && live; item += gridDim.x) {
                    const Item w = decode(item, q);
                    const float *src = packed + (((long long)w.z * q.n_tiles + w.n_tile) * q.kblocks_all + (long long)w.part * kblocks) *
                                                (B_STAGE_BYTES / 4);
                    if(it == 0) pdl_wait();
                    for(int kb = 0; kb < kblocks; kb++, it++) {
                        const int s = it % B_STAGES;
                        if(!mbar_wait(&sh->empty_b[s], ((it / B_STAGES) & 1) ^ 1, abort_flag, status, ST_B_EMPTY)) { live = false; break; }
                        mbar_arrive_expect_tx(&sh->full_b[s], B_STAGE_BYTES);
                        bulk_load(b_ring + s * B_STAGE_BYTES, src + (long long)kb * (B_STAGE_BYTES / 4), B_STAGE_BYTES, &sh->full_b[s]);
                    }
                }
                drain_own(sh->full_b, B_STAGES, it, status);
            }
        }
        else {
            // -------------------------------------------------------------- MMA issuers
            // As in contraction_tf32x3_kernel: two issuer warps take the iterations in turn (an iteration is a pair of k-blocks
            // when they start on an even stage inside one chunk), the whole warp runs the loop with warp-uniform control flow,
            // lanes 0..4 each watch one barrier, a named barrier carries the turn, and stages are released in pairs.
            constexpr uint32_t idesc = instr_desc_tf32(BN);
            constexpr uint32_t DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);   // SBO, version 1, SWIZZLE_128B
            const uint32_t ring_base = ((smem_u32(b_ring) & 0x3FFFF) >> 4) | (1u << 16);
            const uint32_t acc_empty0 = smem_u32(&sh->acc_empty[0]), empty0 = smem_u32(&sh->empty[0]), acc_full0 = smem_u32(&sh->acc_full[0]);
            const uint32_t full_a0 = smem_u32(&sh->full_a[0]), full_b0 = smem_u32(&sh->full_b[0]), empty_b0 = smem_u32(&sh->empty_b[0]);
            const uint32_t total = uint32_t(my_items * kblocks);
            uint32_t chunk = 0, s = 0, s_phase = 0, it = 0, step = 0;
            uint32_t sb = 0, sb_phase = 0;                       // B stage of the iteration's first k-block
            int kb = 0, in_chunk = 0;
            const int me = warp == WARP_MMA ? 0 : 1;
            bool dead = false;
            pdl_wait();
            #pragma unroll 1
            while(it < total) {
                const uint32_t buf = chunk & 1;
                const bool pair = (s & 1) == 0 && in_chunk + 2 <= CHUNK_KB && kb + 2 <= kblocks;
                const int n = pair ? 2 : 1;
                const bool closes_chunk = in_chunk + n == CHUNK_KB || kb + n == kblocks;
                const uint32_t ns = (s + n) & (T_STAGES - 1), nphase = ns < s ? s_phase ^ 1 : s_phase;
                const bool wrap1 = sb + 1 == uint32_t(B_STAGES);
                const uint32_t sb1 = wrap1 ? 0 : sb + 1, sb1_phase = wrap1 ? sb_phase ^ 1 : sb_phase;     // the second one's
                if(int(step & 1) == me) {
                    if(!dead) {
                        // lanes 0, 2: the A columns of the first / second stage; lanes 1, 3: their B stages; lane 4: the accumulator a chunk opens
                        const bool mine = lane < 2 || (lane < 4 && pair) || (lane == 4 && in_chunk == 0);
                        const uint32_t bar = lane == 4 ? acc_empty0 + 8 * buf
                                                       : (lane & 1 ? full_b0 + 8 * (lane >> 1 ? sb1 : sb) : full_a0 + 8 * (s + (lane >> 1)));
                        const uint32_t parity = lane == 4 ? ((chunk >> 1) & 1) ^ 1 : (lane & 1 ? (lane >> 1 ? sb1_phase : sb_phase) : s_phase);
                        const int code = lane == 4 ? ST_MMA_ACC : (lane & 1 ? ST_MMA_B : ST_MMA_A);
                        const bool ok = mine ? mbar_wait(bar, parity, abort_flag, status, code) : true;
                        if(!__all_sync(0xffffffffu, ok)) dead = true;
                    }
                    const uint32_t d = tmem_base + buf * BN, a = tmem_base + A_COL_BASE + s * 64;
                    uint32_t ah[2][4], al[2][4];
                    uint64_t bh[2][4], bl[2][4];
                    #pragma unroll
                    for(int h = 0; h < 2; h++) {
                        const uint32_t bhi = ring_base + (h ? sb1 : sb) * (B_STAGE_BYTES >> 4), blo = bhi + (B_TILE_BYTES >> 4);
                        #pragma unroll
                        for(int j = 0; j < 4; j++) {
                            ah[h][j] = a + h * 64 + 8 * j;
                            al[h][j] = a + h * 64 + 32 + 8 * j;
                            bh[h][j] = (uint64_t(DESC_HI) << 32) | (bhi + 2 * j);
                            bl[h][j] = (uint64_t(DESC_HI) << 32) | (blo + 2 * j);
                        }
                    }
                    const uint32_t accumulate = in_chunk != 0;
                    // my turn: the other warp has issued the iteration before this one
                    if(step > 0) asm volatile("bar.sync %0, 64;" ::"r"(3 + int((step - 1) & 1)) : "memory");
                    tc_fence_after();
                    if(!dead && elect_one()) {
                        mma_kblock(d, ah[0], al[0], bh[0], bl[0], idesc, accumulate);
                        if(pair) mma_kblock(d, ah[1], al[1], bh[1], bl[1], idesc, 1u);
                    }
                    __syncwarp();
                    tc_fence_before();
                    asm volatile("bar.arrive %0, 64;" ::"r"(3 + int(step & 1)) : "memory");      // the other warp's turn
                    if(!dead && elect_one()) {
                        mma_commit(empty_b0 + 8 * sb);
                        if(pair) mma_commit(empty_b0 + 8 * sb1);
                        if(pair || (s & 1)) mma_commit(empty0 + 8 * (s >> 1));   // frees the A columns of a pair of stages
                        if(closes_chunk) mma_commit(acc_full0 + 8 * buf);
                    }
                    __syncwarp();
                }
                step++;
                it += n;
                s = ns;
                s_phase = nphase;
                for(int h = 0; h < n; h++) { sb++; if(sb == uint32_t(B_STAGES)) { sb = 0; sb_phase ^= 1; } }
                in_chunk = closes_chunk ? 0 : in_chunk + n;
                kb = kb + n == kblocks ? 0 : kb + n;
                chunk = closes_chunk ? chunk + 1 : chunk;
            }
            // the last turn handed over is taken by nobody: meet it so that both barriers are left balanced
            if(step > 0 && int(step & 1) == me) asm volatile("bar.sync %0, 64;" ::"r"(3 + int((step - 1) & 1)) : "memory");
        }
    }
    else if(warp < WARP_CONV0 || warp >= WARP_ACC1) {
        // ------------------------------------------------------------------ accumulate + epilogue
        regs_inc<REGS_ACC>();
        const int quad = warp & 3;
        const int set = warp >= WARP_ACC1 ? 1 : 0;
        if(set < SETS) {
            const float2 clamp = act_clamp(q.act), post_clamp = act_clamp(q.post_act);
            const int chunks_per_tile = (kblocks + CHUNK_KB - 1) / CHUNK_KB;
            uint32_t chunk = 0;
            bool live = true;
            for(long long item = blockIdx.x; item < q.num_items && live; item += gridDim.x) {
                const Item w = decode(item, q);
                const long long row = w.m0 + quad * 32 + lane;
                const bool valid = row < q.rows;
                const int b = valid ? int(div32(row, q.P)) : 0;
                const int pix = valid ? int(row - (long long)b * q.P) : 0;
                const int col0 = w.n_tile * BN + set * COLS;
                const long long off = w.z * q.y_batch_stride + w.part * q.y_split_stride + b * q.y_image_stride +
                                      pix * q.y_row_stride + col0 * q.y_col_stride;
                if(item == blockIdx.x) pdl_wait();
                // asked for now, used when the last chunk is in: the bias of the set's columns (handed round by shuffles), and the
                // residual operand's lines into L2
                float bias_g[COLS / 32];
                #pragma unroll
                for(int g = 0; g < COLS / 32; g++)
                    bias_g[g] = q.bias && col0 + g * 32 + lane < q.cols ? ld_early(q.bias + col0 + g * 32 + lane) : 0.0f;
                if(q.residual) {
                    // each lane sees to two columns: the warp's first and last row (a column of the warp is one or two lines)
                    const long long first = __shfl_sync(0xffffffffu, off, 0), lastv = __shfl_sync(0xffffffffu, valid ? off : first, 31);
                    #pragma unroll
                    for(int g = 0; g < COLS / 32; g++)
                        if(w.m0 + quad * 32 < q.rows && col0 + g * 32 + lane < q.cols) {
                            const float *rp = q.residual + (g * 32 + lane) * q.y_col_stride;
                            asm volatile("prefetch.global.L2 [%0];" ::"l"(rp + first));
                            asm volatile("prefetch.global.L2 [%0];" ::"l"(rp + lastv));
                        }
                }
                float sum[COLS];
                #pragma unroll 1
                for(int c = 0; c < chunks_per_tile; c++, chunk++) {
                    const uint32_t buf = chunk & 1;
                    if(!warp_wait(&sh->acc_full[buf], (chunk >> 1) & 1, abort_flag, status, ST_EPI_ACC, lane)) { live = false; break; }
                    tc_fence_after();
                    const uint32_t taddr = tmem_base + (uint32_t(quad * 32) << 16) + buf * BN + set * COLS;
                    #pragma unroll
                    for(int g = 0; g < COLS / 16; g++) {
                        uint32_t v[16];
                        tmem_ld(taddr + g * 16, v);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        #pragma unroll
                        for(int j = 0; j < 16; j++) sum[g * 16 + j] = c == 0 ? __uint_as_float(v[j]) : sum[g * 16 + j] + __uint_as_float(v[j]);
                    }
                    tc_fence_before();
                    __syncwarp();
                    if(lane == 0) mbar_arrive(&sh->acc_empty[buf]);
                }
                if(!live) break;
                float *yp = q.y + off;
                const float *rp = q.residual + off;
                const bool with_res = q.residual != nullptr, res_ok = with_res && valid;
                const int cols_left = min(COLS, q.cols - col0);
                // residual values eight columns ahead of their use
                float res[2][8];
                auto load_res = [&](int h) {
                    #pragma unroll
                    for(int j = 0; j < 8; j++) {
                        res[h & 1][j] = res_ok && h * 8 + j < cols_left ? ld_plain(rp) : 0.0f;
                        rp += q.y_col_stride;
                    }
                };
                if(with_res) load_res(0);
                #pragma unroll
                for(int h = 0; h < COLS / 8; h++) {
                    if(h * 8 >= cols_left) break;
                    if(with_res && h + 1 < COLS / 8) load_res(h + 1);
                    #pragma unroll
                    for(int j = 0; j < 8; j++) {
                        float a = sum[h * 8 + j];
                        if(q.bias) a += __shfl_sync(0xffffffffu, bias_g[h / 4], (h & 3) * 8 + j);
                        a = fminf(fmaxf(a, clamp.x), clamp.y);
                        if(with_res) a = fminf(fmaxf(a + q.res_scale * res[h & 1][j], post_clamp.x), post_clamp.y);
                        sum[h * 8 + j] = a;
                    }
                    if(q.vec_store && h * 8 + 8 <= cols_left) {
                        if(valid) {
                            *reinterpret_cast<float4 *>(yp) = make_float4(sum[h * 8], sum[h * 8 + 1], sum[h * 8 + 2], sum[h * 8 + 3]);
                            *reinterpret_cast<float4 *>(yp + 4) = make_float4(sum[h * 8 + 4], sum[h * 8 + 5], sum[h * 8 + 6], sum[h * 8 + 7]);
                        }
                        yp += 8;
                    }
                    else {
                        #pragma unroll
                        for(int j = 0; j < 8; j++) {
                            if(valid && h * 8 + j < cols_left) *yp = sum[h * 8 + j];
                            yp += q.y_col_stride;
                        }
                    }
                }
            }
        }
    }
    else {
        // ------------------------------------------------------------------ converters
        if(REGS_CONV < REGS_LAUNCH) regs_dec<REGS_CONV>();
        const int quad = warp & 3, group = (warp - WARP_CONV0) >> 2;
        const int row_in_tile = quad * 32 + lane;
        const uint32_t total = uint32_t(my_items * kblocks);
        const uint32_t zero_base = smem_u32(zeros), ring = smem_u32(a_ring);
        const uint32_t full0 = smem_u32(&sh->sa_full[0]), sempty0 = smem_u32(&sh->sa_empty[0]);
        // position of the k-block whose values are fetched next: work item, k-block and tap in it, slot of the ring and its parity
        long long item = blockIdx.x;
        int kb = group, tap = T == 1 ? 0 : group, sa = T == 1 ? group : 0;
        uint32_t sa_phase = 0;
        bool new_item = true, new_slot = true;
        int rel = 0, oy = 0, ox = 0;       // the thread's pixel: its place in a slot, its output coordinates
        bool valid = false;
        while(kb >= kblocks) { kb -= kblocks; item += gridDim.x; }
        // values of the thread's row in the k-block at the position; false: a wait gave up
        auto fetch = [&](float (&v)[BK]) -> bool {
            if(!KMAJOR && new_item) {
                const Item w = decode(item, q);
                const long long row = w.m0 + row_in_tile;
                const int b0 = int(div32(w.m0, q.P)), pix0 = int(w.m0 - (long long)b0 * q.P);
                valid = row < q.rows;
                const int b = valid ? int(div32(row, q.P)) : b0;
                const int pix = valid ? int(row - (long long)b * q.P) : pix0;
                const int lo0 = max(pix0 + q.dmin, 0) & ~3;
                // units of the images before this one: the first from lo0 to its end, whole planes between
                rel = b == b0 ? pix - lo0 : (((q.P - lo0 + 31) >> 5) + (b - b0 - 1) * ((q.P + 31) >> 5)) * 32 + pix;
                if(T > 1) { oy = pix / q.W; ox = pix - oy * q.W; }
            }
            if(new_slot && !warp_wait(full0 + 8 * sa, sa_phase, abort_flag, status, ST_CONV_FULL, lane)) return false;
            const uint32_t base = ring + uint32_t(sa) * q.slot_bytes;
            if(KMAJOR) {
                const uint32_t r = base + row_in_tile * 128;
                #pragma unroll
                for(int c = 0; c < 8; c++)
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[4 * c]), "=f"(v[4 * c + 1]), "=f"(v[4 * c + 2]), "=f"(v[4 * c + 3])
                                 : "r"(r + ((c ^ (row_in_tile & 7)) << 4)));
            }
            else {
                uint32_t src = base + (uint32_t(rel) >> 5) * UNIT_BYTES + (uint32_t(rel) & 31) * 4;
                if(T > 1) {
                    const short2 d = sh->tap[tap];
                    const bool ok = valid && unsigned(oy + d.x) < unsigned(q.H) && unsigned(ox + d.y) < unsigned(q.W);
                    const int at = rel + d.x * q.W + d.y;
                    // (a row that reads zeros reads them from the bank its pixel would be in)
                    src = (ok ? base + (uint32_t(at) >> 5) * UNIT_BYTES : zero_base) + (uint32_t(at) & 31) * 4;
                }
                #pragma unroll
                for(int c = 0; c < BK; c++) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v[c]) : "r"(src + c * 128));
            }
            return true;
        };
        // split and publish as the A operand of stage it % T_STAGES
        auto publish = [&](uint32_t it, const float (&v)[BK]) -> bool {
            const int stg = it % T_STAGES;
            if(!warp_wait(&sh->empty[stg >> 1], ((it / T_STAGES) & 1) ^ 1, abort_flag, status, ST_CONV_EMPTY, lane)) return false;
            tc_fence_after();
            const uint32_t t_hi = tmem_base + (uint32_t(quad * 32) << 16) + A_COL_BASE + stg * 64;
            // The tensor core reads only the TF32 part of an fp32 word, so the value itself serves as "hi";
            // lo = v - tf32(v) goes to the 32 columns after it.
            #pragma unroll
            for(int h = 0; h < 2; h++) {
                uint32_t hi[16], lo[16];
                #pragma unroll
                for(int k = 0; k < 16; k++) {
                    const float x = v[h * 16 + k];
                    hi[k] = __float_as_uint(x);
                    lo[k] = __float_as_uint(x - __uint_as_float(__float_as_uint(x) & 0xffffe000u));
                }
                tmem_st16(t_hi + h * 16, hi);
                tmem_st16(t_hi + 32 + h * 16, lo);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if(lane == 0) mbar_arrive(&sh->full_a[stg]);
            return true;
        };
        float cur[BK], nxt[BK];
        bool have = false, release = false;
        uint32_t done = 0;
        pdl_wait();
        #pragma unroll 1
        for(uint32_t it = group;; it += 2) {
            const bool more = it < total;
            if(more) {
                if(!fetch(nxt)) break;
                // on to this group's next k-block; when it lies in another slot this warp is done with the current one
                done = sempty0 + 8 * sa;
                kb += 2;
                new_item = false;
                while(kb >= kblocks) { kb -= kblocks; item += gridDim.x; new_item = true; }
                int steps = 2;
                if(T > 1) { steps = 0; tap += 2; while(tap >= T) { tap -= T; steps++; } }
                new_slot = steps > 0;
                sa += steps;
                while(sa >= S_STAGES) { sa -= S_STAGES; sa_phase ^= 1; }
                release = new_slot || it + 2 >= total;
            }
            if(have && !publish(it - 2, cur)) break;
            if(!more) break;
            uint32_t all = 0;
            #pragma unroll
            for(int k = 0; k < BK; k++) { cur[k] = nxt[k]; all ^= __float_as_uint(nxt[k]); }
            // The slot is handed back once the loads from it have returned, not when they have been issued: the copy engine is
            // not ordered behind loads in flight.  The arrival's predicate hangs on all the loaded words (a square is never
            // 2 modulo 4), so it cannot be carried out before them.
            __syncwarp();
            if(release && lane == 0)
                asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tmul.lo.u32 t, %1, %1;\n\tand.b32 t, t, 3;\n\tsetp.ne.u32 p, t, 2;\n\t"
                             "@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(done), "r"(all) : "memory");
            have = true;
        }
    }

    // ---------------------------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if(*(volatile int *)abort_flag) {
        // a wait gave up: let the MMAs already issued retire (bounded) before tensor memory goes away
        if(warp == WARP_MMA && elect_one()) {
            mma_commit(smem_u32(&sh->drain));
            const long long t0 = global_ns();
            while(!mbar_try_wait(&sh->drain, 0)) {
                __nanosleep(256);
                if(global_ns() - t0 > WAIT_LIMIT_NS) { atomicCAS(status, 0, ST_DRAIN); break; }
            }
        }
        __syncthreads();
    }
    if(warp == WARP_MMA) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// ---------------------------------------------------------------------------------------------- host
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_fn()
{
    static std::mutex mutex;
    static EncodeTiledFn fn = nullptr;
    std::lock_guard<std::mutex> lock(mutex);
    if(!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult res;
        if(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &res) == cudaSuccess && res == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

struct Source {             // the A operand as a tensor [inner, outer, images] of floats
    int kind;               // SRC_...
    long long inner, outer, images, pitch, image_stride;
};

// The geometry of a launch, or false when the problem is not one for this kernel.
static bool plan(const Contraction &p, const TcPacked &L, int splits, const TcBatch &batch, Params &q, Source &src)
{
    memset(&q, 0, sizeof(q));
    if(!act_is_clamp(p.act) || !act_is_clamp(p.post_act) || p.beta != 0.0f || p.bias_mode == DLP_GEMM_BIAS_M) return false;
    if(p.rows >= (1ll << 31) - BM) return false;
    q.rows = p.rows;
    q.cols = p.cols;
    q.kblocks_all = L.k_pad / BK;
    q.splits = splits;
    q.kblocks = q.kblocks_all / splits;
    q.n_tiles = L.n_pad / L.bn;
    q.items_each = ceil_div<long long>(p.rows, BM) * q.n_tiles * splits;
    q.num_items = q.items_each * batch.count;
    if(splits > 1 && (batch.count > 1 || q.num_items >= (1ll << 31))) return false;
    q.taps = 1;
    q.kw = 1;
    q.P = int(p.rows);
    src.kind = SRC_UNITS;
    src.images = batch.count;
    src.image_stride = batch.a_stride;
    if(p.a_mode == A_STRIDED && p.plane == 0) {
        if(p.a_k_stride == 1) { src.kind = SRC_K; src.inner = p.k; src.outer = p.rows; src.pitch = p.a_row_stride; }
        else if(p.a_row_stride == 1) { src.inner = p.rows; src.outer = p.k; src.pitch = p.a_k_stride; }
        else return false;
    }
    else if(p.a_mode == A_TAPBLOCK) {
        // a convolution whose output pixel is its input pixel, displaced by the tap.  (1x1 convolutions do not come here: with one
        // tap a slot serves one k-block, and the general kernel, which does not pass A through shared memory, is the faster one:
        // 1024 -> 256 on 14x14 at batch 256 149 against 164 us, 512 -> 128 on 28x28 148 against 154 us.)
        if(batch.count != 1 || p.plane <= 0 || p.plane != p.in_h * p.in_w || p.out_w != p.in_w || p.rows % p.plane != 0) return false;
        if(p.stride_h != 1 || p.stride_w != 1 || p.a_k_stride != p.plane) return false;
        q.P = p.plane;
        q.W = p.in_w;
        q.H = p.in_h;
        q.taps = p.num_taps;
        q.kw = p.kw; q.dil_h = p.dil_h; q.dil_w = p.dil_w; q.pad_h = p.pad_h; q.pad_w = p.pad_w;
        if(q.taps < 2 || q.taps > MAX_TAPS || q.taps != p.kh * p.kw || p.k % (q.taps * BK) != 0) return false;
        if(2 * p.pad_h != p.dil_h * (p.kh - 1) || 2 * p.pad_w != p.dil_w * (p.kw - 1)) return false;
        if(q.kblocks % q.taps != 0) return false;                       // a part of a split K is whole channel blocks
        if((long long)p.pad_h * p.in_w + p.pad_w > MAX_UNITS * 32) return false;
        src.inner = p.plane;
        src.outer = p.k / q.taps;
        src.images = p.rows / p.plane;
        src.pitch = p.plane;
        src.image_stride = p.a_batch_stride;
        if(src.images > 1 && p.plane < 32) return false;                 // too many images per tile
        q.dmax = p.pad_h * p.in_w + p.pad_w;
        q.dmin = -q.dmax;
    }
    else return false;
    const bool mapped = reinterpret_cast<uintptr_t>(p.a) % 16 == 0 && src.pitch >= src.inner && src.pitch % 4 == 0 && src.pitch < (1ll << 37) &&
                        (src.images == 1 || (src.image_stride >= src.pitch * (src.outer - 1) + src.inner && src.image_stride % 4 == 0 &&
                                             src.image_stride < (1ll << 37))) && src.images < (1ll << 31);
    if(!mapped) {
        // One warp copies; with 25 taps to a slot it keeps up (5x5 64 -> 192 on 27x27 at batch 64 177 -> 167 us), with nine it does not
        // (3x3 512 -> 512 on 7x7 at batch 256 324 us in the general kernel, 515 here).
        if(q.taps < 16) return false;
        src.kind = SRC_COPY;
        q.a = p.a;
        q.a_image_stride = p.a_batch_stride;
    }
    if(src.kind == SRC_K) q.slot_bytes = BM * BK * 4;
    else {
        const int segs = p.plane > 0 && src.images > 1 ? (BM - 2) / q.P + 2 : 1;
        const int units = (BM + (q.taps > 1 ? 3 : 0) + q.dmax - q.dmin + 31 * segs) / 32;
        if(units > MAX_UNITS) return false;
        q.slot_bytes = units * UNIT_BYTES;
    }
    q.y = p.y;
    q.y_batch_stride = batch.y_stride;
    if(p.out_mode == OUT_NCHW) {
        if(p.plane <= 0) return false;
        q.y_row_stride = 1;
        q.y_col_stride = p.plane;
        q.y_image_stride = (long long)p.out_channels_total * p.plane;
    }
    else {
        q.y_row_stride = p.out_mode == OUT_COL_MAJOR ? 1 : p.ldc;
        q.y_col_stride = p.out_mode == OUT_COL_MAJOR ? p.ldc : 1;
        q.y_image_stride = q.y_row_stride * q.P;
    }
    q.vec_store = q.y_col_stride == 1 && p.ldc % 4 == 0 && batch.y_stride % 4 == 0 && reinterpret_cast<uintptr_t>(p.y) % 16 == 0;
    q.bias = p.bias_mode == DLP_GEMM_BIAS_N ? p.bias : nullptr;
    q.act = p.act;
    q.post_act = p.post_act;
    q.residual = p.residual;
    q.res_scale = p.residual_scale;
    return true;
}

template<int BN, int SRC>
static dlp_status launch_bn(const CUtensorMap &ta, const float *packed, const Params &q, cudaStream_t stream)
{
    {
        static std::mutex mutex;
        static std::vector<char> configured;          // by device ordinal: the attribute belongs to the function in that device's context
        int dev = 0;
        DLP_CUDA_OK(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lock(mutex);
        if(size_t(dev) >= configured.size()) configured.resize(size_t(dev) + 1, 0);
        if(!configured[dev]) {
            DLP_CUDA_OK(cudaFuncSetAttribute(stream_tf32x3_kernel<BN, SRC>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT));
            configured[dev] = 1;
        }
    }
    int *status = device_status_word();
    if(!status) return fail(DLP_CUDA_ERROR, "cannot resolve the device status word");
    Params r = q;
    constexpr int b_stage = 2 * BN * BK * 4;
    // Shared memory between the two rings.  A pair of B stages (64 KB for 128 columns, a trip to L2 and back) is refilled while
    // the others are read, so five serve better than four (4096 x 4096 x 4096: 739 -> 612 us), as long as two slots with taps, or
    // four of one k-block each, are left.  With one k-block to a slot the two converter groups take the slots in turn, and their
    // number has to be even: then a group meets a ring entry only in slots of its own, and an entry that its parity bit shows
    // as filled cannot be the one before, still on its way to the other group.
    const int room = SMEM_LIMIT - SMEM_FIXED - (r.taps > 1 ? UNIT_BYTES : 0), slots = r.taps > 1 ? 2 : 4;
    r.b_stages = std::max(4, std::min(MAX_B_STAGES, (room - slots * r.slot_bytes) / b_stage));
    r.s_stages = std::min(MAX_S_STAGES, (room - r.b_stages * b_stage) / r.slot_bytes);             // at least two of 40 KB
    if(r.taps == 1) r.s_stages &= ~1;
    const int smem_bytes = SMEM_LIMIT - room + r.b_stages * b_stage + r.s_stages * r.slot_bytes;
    const unsigned grid = unsigned(std::min<long long>(q.num_items, sm_count()));
    DLP_LAUNCH_PDL(launch_pdl(few_items(q.num_items), stream_tf32x3_kernel<BN, SRC>, grid, NUM_THREADS, smem_bytes, stream, ta,
                              packed, r, status), "stream_tf32x3_kernel");
    return DLP_OK;
}

} // namespace st

bool stream_tc_eligible(const Contraction &p, const TcPacked &L, int splits, const TcBatch &batch)
{
    st::Params q;
    st::Source src;
    return st::plan(p, L, splits, batch, q, src);
}

dlp_status launch_stream_tc(const Contraction &p, const TcPacked &L, const float *packed, cudaStream_t stream, int splits, long long split_stride,
                            const TcBatch &batch)
{
    st::Params q;
    st::Source src;
    if(!st::plan(p, L, splits, batch, q, src)) return fail(DLP_INVALID_ARGUMENT, "not a problem for the streaming kernel");
    q.y_split_stride = split_stride;
    note_route(src.kind == st::SRC_K ? "stream_k" : (src.kind == st::SRC_UNITS ? "stream_units" : "stream_copy"), L.bn, splits);
    CUtensorMap ta;
    memset(&ta, 0, sizeof(ta));
    if(src.kind != st::SRC_COPY) {
        st::EncodeTiledFn enc = st::encode_fn();
        if(!enc) return fail(DLP_CUDA_ERROR, "cuTensorMapEncodeTiled is not available from this driver");
        cuuint64_t dims[3] = { cuuint64_t(src.inner), cuuint64_t(src.outer), cuuint64_t(src.images) };
        cuuint64_t strides[2] = { cuuint64_t(src.pitch) * 4, cuuint64_t(src.images > 1 ? src.image_stride : src.pitch * src.outer) * 4 };
        cuuint32_t box[3] = { 32, cuuint32_t(src.kind == st::SRC_K ? st::BM : 32), 1 }, elem[3] = { 1, 1, 1 };
        const CUresult r = enc(&ta, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(p.a), dims, strides, box, elem,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, src.kind == st::SRC_K ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if(r != CUDA_SUCCESS) return fail(DLP_CUDA_ERROR, "cuTensorMapEncodeTiled failed with code " + std::to_string(int(r)));
    }
    switch(L.bn * 4 + src.kind) {
    case 32 * 4 + st::SRC_K: return st::launch_bn<32, st::SRC_K>(ta, packed, q, stream);
    case 32 * 4 + st::SRC_UNITS: return st::launch_bn<32, st::SRC_UNITS>(ta, packed, q, stream);
    case 32 * 4 + st::SRC_COPY: return st::launch_bn<32, st::SRC_COPY>(ta, packed, q, stream);
    case 64 * 4 + st::SRC_K: return st::launch_bn<64, st::SRC_K>(ta, packed, q, stream);
    case 64 * 4 + st::SRC_UNITS: return st::launch_bn<64, st::SRC_UNITS>(ta, packed, q, stream);
    case 64 * 4 + st::SRC_COPY: return st::launch_bn<64, st::SRC_COPY>(ta, packed, q, stream);
    case 128 * 4 + st::SRC_K: return st::launch_bn<128, st::SRC_K>(ta, packed, q, stream);
    case 128 * 4 + st::SRC_UNITS: return st::launch_bn<128, st::SRC_UNITS>(ta, packed, q, stream);
    case 128 * 4 + st::SRC_COPY: return st::launch_bn<128, st::SRC_COPY>(ta, packed, q, stream);
    default: return fail(DLP_INVALID_ARGUMENT, "unsupported column tile");
    }
}

} // namespace dlp
