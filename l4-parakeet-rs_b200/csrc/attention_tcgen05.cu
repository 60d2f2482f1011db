// Local relative-position multi-head attention (window +-128) on the 5th-generation tensor cores.
//
//   score[q,k] = ((Q_q + u_h) . K_k + (Q_q + v_h) . P_h[128 - q + k]) / sqrt(128)
//   keys k in [max(0, q-128), min(valid-1, q+128)] of the query's own utterance, fp32 softmax,
//   ctx = sum_k p . V_k  (definition: local_attention_simple_kernel; reference:
//   kernels/sm89/encoder.cu:1338-1461, tensor-core form :1500-2035).
//
// A tile = 128 consecutive queries of one head of one utterance; their keys lie in a window of three
// 128-key blocks, of which the ones outside the utterance are left out.  The kernel is persistent: a CTA
// takes a contiguous range of (head, tile) items.  The contractions run as tcgen05.mma kind::f16 (M = 128)
// with fp32 accumulators in tensor memory:
//     QP = Q . P_h^T   (N = 128 + 128 + 16: the 257 position rows)   TMEM columns [0, 272)
//     S  = Q . K^T     (key blocks of N = 128)                       [384, 512), [0, 128), [128, 256)
//     O  = Pr . V      (Pr = softmax probabilities, fp16, K = keys)  [384, 512), when S_0 has been read
// Operands arrive by TMA (cp.async.bulk.tensor, 128-byte swizzle, no multicast) into three 32 KB slots
// that hold blocks of P_h, then K, then V in turn, each load issued as soon as its slot is free.  Q, P
// and K are K-major operands; V is used as it lies in memory (rows = keys = the K dimension of
// Pr . V, features contiguous), i.e. as an MN-major B operand: instruction-descriptor bit 16, and a
// shared-memory descriptor whose leading-dimension offset is the distance between the two 64-feature
// atoms and whose stride is the 1024 bytes between 8-key groups.  The u / v biases are added in fp32
// outside the MMAs (u . K_k and v . P_j are per-column constants; v . P_j is formed once per head, u . K_k
// once per key block while the tiles of a CTA follow each other).  QP is drained to shared memory as fp16
// so that the relative shift is a plain gather (key kk of query ql reads column kk - ql).  The softmax is
// two passes by sixteen warps, four per TMEM lane quadrant: the first forms the scaled, masked scores,
// writes them back over the accumulators and takes the row maximum, the second reads them and writes the
// probabilities through swizzled shared memory (the space the position scores had) as the A operand of
// the last contraction.
//
// What bounds it: one tile is a chain of about ten dependent steps with one tile in flight per SM (tensor
// memory and shared memory are full), so what counts is the length of the chain and what the next tile can
// start meanwhile.  Q, P and the first key block of the next tile are loaded, and its QP product is issued,
// while the softmax warps finish this one.
// Measured back to back: 179 us at 45 056 rows, 33 us at 6144, 15 us at 768, 10.4 us at 128 (with the issuing roles
// behind a lane test 201, 36, 15.2, 10.7; one CTA per tile and two full passes over scores and position scores: 456
// and 66 us for the first two).  The softmax warps' issue slots, the tensor pipe and shared memory are each far from
// full; the first tile of a CTA takes about twice a later one, which is what the 48 tiles of 768 rows show.
// Every wait is a bounded mbarrier wait; when one expires the kernel raises the status word and all
// roles leave through the common teardown (tensor memory freed).
#include <cuda.h>
#include <cuda_fp16.h>
#include <float.h>
#include <stdint.h>

#include <type_traits>

#include "pk100_internal.h"
#include "ptx_sm100.cuh"

namespace pk100 {

namespace att5 {

constexpr int kHeads = 8;
constexpr int kDim = 128;                 // head width
constexpr int kTile = 128;                // queries per CTA
constexpr int kReach = 128;               // keys on each side
constexpr int kPosRows = 272;             // position rows per head (257 used)
constexpr float kSoftmaxScale = 0.08838834764831845f;
constexpr int kParts = 4;                 // softmax warps per TMEM lane quadrant: 32 columns of a block each
constexpr int kSoftmaxWarps = 4 * kParts;
constexpr int kSoftmaxThreads = 32 * kSoftmaxWarps;
constexpr int kThreads = kSoftmaxThreads + 64;       // + TMA producer warp + MMA warp

constexpr int kAtomBytes = 128 * 128;     // [128 rows x 64 halves], 128-byte swizzle
constexpr int kSlotBytes = 2 * kAtomBytes;           // one 128-row operand block: features 0-63 | 64-127
constexpr int kTailBytes = 2 * 16 * 128;  // position rows 256..271
constexpr int kQpPitch = 274;             // halves per QP row: 137 words, odd, so that the 32 rows of a
                                          // warp fall into 32 different banks

// barrier indices; each completes once per tile, the ones of a key block once per tile that has the block
enum : int {
    B_Q_IN = 0, B_P_IN, B_VP_DONE, B_QP_DONE, B_QP_DRAINED, B_PASS0_DONE, B_CTX_READ,
    B_K_IN,                    // 3
    B_UK_DONE = B_K_IN + 3,    // 3
    B_S_DONE = B_UK_DONE + 3,  // 3
    B_V_IN = B_S_DONE + 3,     // 3
    B_P_READY = B_V_IN + 3,    // 3
    B_PV_DONE = B_P_READY + 3, // 3
    B_SUM = B_PV_DONE + 3,     // 4 (one per lane quadrant)
    B_COUNT = B_SUM + 4
};

// Operand staging: three 32 KB slots take, in turn, the position rows (slots 0, 1 and the 4 KB tail), the
// key blocks (K0 -> slot 2 at once, K1 / K2 -> slots 0 / 1 when the position rows are done with) and the
// value blocks (V_b -> slot b, when the key block there and its bias term are done).  P_V frees slot 0
// first, so the next tile's position rows follow the value blocks in order.
struct Smem {
    alignas(1024) uint8_t q[kSlotBytes];
    alignas(1024) uint8_t slot[3][kSlotBytes];
    alignas(1024) uint8_t tail[kTailBytes];
    union {
        alignas(1024) __half qp[kTile * kQpPitch + 8];    // position scores, until the first pass is over
        alignas(1024) uint8_t pr[2][kSlotBytes];          // probabilities of two key blocks
    };
    float vp[288];                                        // 272 used, the rest read and dropped
    float uk[3][128];                                     // key block i of the utterance -> row i % 3
    alignas(16) float bias_u[4][36];                      // 32 features a row, rows in different banks
    float rowmax[kParts][kTile];
    float rowsum[kParts][kTile];
    uint64_t bar[B_COUNT];
    uint32_t tmem_base;
    int abort;
};

struct Params {
    const __half* bias_u;     // [8, 128]
    const __half* bias_v;
    __half* out; int ldo;
    int tiles;                // 128-row tiles of the batch
    pk100_rows rows;
    int early;                // position, bias_u, bias_v and rows were complete before the chain of launches began
    int* status;
};

// Place of a tile: first row of its utterance, first query inside it, the utterance's valid rows.
struct TilePlace {
    int base, q0, valid;
    __device__ __forceinline__ TilePlace(const pk100_rows& g, int tile) {
        if (g.tiles != nullptr) {
            const int2 t = __ldg(g.tiles + tile);
            base = t.x;
            valid = t.y;
        } else {
            const int seg = tile / (g.seg_stride / kTile);
            base = seg * g.seg_stride;
            valid = min(g.seg_valid != nullptr ? __ldg(g.seg_valid + seg) : g.valid_rows, g.seg_stride);
        }
        q0 = tile * kTile - base;
    }
    __device__ __forceinline__ bool padding() const { return q0 >= valid; }
    // key blocks that have keys: bit b = rows q0 - 128 + 128 b .. of the utterance
    __device__ __forceinline__ uint32_t blocks() const {
        return 2u | (q0 > 0 ? 1u : 0u) | (q0 + kTile < valid ? 4u : 0u);
    }
};

// byte offset of 16-byte chunk `chunk` (0..7) of row `row` inside a [rows x 64 halves] swizzled atom
__device__ __forceinline__ int swz(int row, int chunk) {
    return (row >> 3) * 1024 + (row & 7) * 128 + ((chunk ^ (row & 7)) << 4);
}

// a + b in fp32, a widened inside the instruction
__device__ __forceinline__ float add_half(__half a, float b) {
    float d;
    asm("add.rn.f32.f16 %0, %1, %2;" : "=f"(d) : "h"(__half_as_ushort(a)), "f"(b));
    return d;
}

// dot product of 32 fp32 bias values (in registers) with 32 consecutive halves (chunks first ..
// first + 3) of row `row` of a swizzled operand atom; two independent chains
__device__ __forceinline__ float bias_dot32(const uint8_t* atom, int row, int first, const float (&bias)[32]) {
    float acc0 = 0.0f, acc1 = 0.0f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const uint4 raw = *reinterpret_cast<const uint4*>(atom + swz(row, first + c));
        const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 x = __half22float2(h[i]);
            acc0 = fmaf(bias[8 * c + 2 * i], x.x, acc0);
            acc1 = fmaf(bias[8 * c + 2 * i + 1], x.y, acc1);
        }
    }
    return acc0 + acc1;
}

// The first poll is inlined (most waits of a tile find their phase complete; a call cost 250 cycles), the
// polling loop exists once.
__device__ __noinline__ bool att_poll(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    return mbar_wait_bounded(bar, parity, abort_flag);
}
__device__ __forceinline__ bool att_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    return mbar_try_wait(bar, parity) || att_poll(bar, parity, abort_flag);
}
#define ATT_WAIT(index, parity)                                                         \
    if (!(ok = att_wait(&sm.bar[index], (parity), abort_flag))) break
// a whole warp waits
#define ATT_WARP_WAIT(index, parity)                                                    \
    if (!(ok = __all_sync(0xffffffffu, att_wait(&sm.bar[index], (parity), abort_flag)) != 0)) break

__global__ void __launch_bounds__(kThreads, 1)
local_attention_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                               const __grid_constant__ CUtensorMap map_p, const __grid_constant__ CUtensorMap map_p16,
                               const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_out, const Params p) {
    extern __shared__ uint8_t att5_raw[];
    Smem& sm = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(att5_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid / 32, 0), lane = tid % 32;     // (warp: known to be the same in all lanes)
    // (head, tile) items of this CTA, heads outermost: a range meets two heads at most a few times
    const long long items = static_cast<long long>(kHeads) * p.tiles;
    const int first_item = static_cast<int>(items * blockIdx.x / gridDim.x);
    const int last_item = static_cast<int>(items * (blockIdx.x + 1) / gridDim.x);
    const int first_head = first_item / p.tiles, first_tile = first_item % p.tiles;

    grid_dependents_launch();
    volatile int* abort_flag = &sm.abort;
    if (tid == 0) {
        sm.abort = 0;
        for (int i = 0; i < B_COUNT; ++i) {
            int count = 1;                                             // TMA arrive / tcgen05.commit
            if (i == B_VP_DONE || i == B_QP_DRAINED || i == B_PASS0_DONE || i == B_CTX_READ ||
                (i >= B_UK_DONE && i < B_UK_DONE + 3) || (i >= B_P_READY && i < B_P_READY + 3))
                count = kSoftmaxWarps;
            if (i >= B_SUM) count = kParts;
            mbar_init(&sm.bar[i], count);
        }
        fence_barrier_init();
        prefetch_tensormap(&map_q);
        prefetch_tensormap(&map_k);
        prefetch_tensormap(&map_p);
        prefetch_tensormap(&map_p16);
        prefetch_tensormap(&map_v);
    }
    if (warp == kSoftmaxWarps + 1) {
        tmem_alloc(&sm.tmem_base, 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = sm.tmem_base;
    // Q, K and V come from the kernel before: the roles wait for it where they first need it (p.early: the
    // position rows and biases do not, so the first tile's are fetched and multiplied in its shadow)
    // slot of key block b (value block b: slot b)
    auto slot_of_key = [](int b) { return b == 0 ? 2 : b - 1; };
    // TMEM columns of the score block b and of the context
    auto score_col = [](int b) { return b == 0 ? 384u : (b == 1 ? 0u : 128u); };
    constexpr uint32_t kCtxCol = 384u;
    bool ok = true;
    // Parities of the current tile's phases.  Bit 1 is that of every barrier that completes once per tile
    // (the middle key block is in every tile), bits 0 and 2 those of the first and last key block.
    uint32_t ph = 0;

    // The two issuing roles run as whole warps and elect a lane for the TMA and MMA instructions alone: their operands
    // live in uniform registers, which the compiler has to fill one by one behind a lane test (about 130 cycles an
    // MMA, of which a tile has 72).
    if (warp == kSoftmaxWarps) {
        // ------------------------------------------------------------ TMA producer
        uint32_t before = 0, ph_before = 0;            // key blocks and parities of the tile before (0: none)
        if (!p.early) grid_dependency_wait();
        int head = first_head, tile = first_tile - 1;
        for (int item = first_item; ok && item < last_item; ++item) {
            if (++tile == p.tiles) { tile = 0; ++head; }
            const TilePlace at(p.rows, tile);
            if (at.padding()) continue;
            const uint32_t blocks = at.blocks(), par = (ph >> 1) & 1u;
            const int key_row = at.base + at.q0 - kReach;
            // one 128-row operand block: its two 64-feature atoms
            auto load_pair = [&](uint8_t* dst, int atom_bytes, const CUtensorMap* map, int bar, int x, int row, int arm_bytes) {
                if (elect_one()) {
                    if (arm_bytes > 0) mbar_arrive_expect_tx(&sm.bar[bar], arm_bytes);
                    tma_load_2d(dst, map, &sm.bar[bar], x, row);
                    tma_load_2d(dst + atom_bytes, map, &sm.bar[bar], x + 64, row);
                }
                __syncwarp();
            };
            auto load_block = [&](int slot, const CUtensorMap* map, int bar, int b) {
                load_pair(sm.slot[slot], kAtomBytes, map, bar, head * kDim, key_row + b * 128, kSlotBytes);
            };
            auto load_queries = [&] { load_pair(sm.q, kAtomBytes, &map_q, B_Q_IN, head * kDim, at.base + at.q0, kSlotBytes); };
            if (before != 0) load_queries();           // the score products of the tile before have retired
            // position rows: slot 0 held V0 (or K1), slot 1 held V1 of the tile before
            load_pair(sm.tail, kTailBytes / 2, &map_p16, B_P_IN, 0, head * kPosRows + 256, 2 * kSlotBytes + kTailBytes);
            if (before & 1u) ATT_WARP_WAIT(B_PV_DONE + 0, ph_before & 1u);
            if (before != 0 && !(before & 1u)) ATT_WARP_WAIT(B_PV_DONE + 1, (ph_before >> 1) & 1u);
            load_pair(sm.slot[0], kAtomBytes, &map_p, B_P_IN, 0, head * kPosRows, 0);
            if (before != 0) ATT_WARP_WAIT(B_PV_DONE + 1, (ph_before >> 1) & 1u);
            load_pair(sm.slot[1], kAtomBytes, &map_p, B_P_IN, 0, head * kPosRows + 128, 0);
            if (before & 4u) ATT_WARP_WAIT(B_PV_DONE + 2, (ph_before >> 2) & 1u);
            if (before == 0) {
                if (p.early) grid_dependency_wait();
                load_queries();
            }
            if (blocks & 1u) load_block(slot_of_key(0), &map_k, B_K_IN + 0, 0);
            // the other key blocks: once the position rows have been multiplied
            ATT_WARP_WAIT(B_QP_DONE, par);
            ATT_WARP_WAIT(B_VP_DONE, par);
            load_block(slot_of_key(1), &map_k, B_K_IN + 1, 1);
            if (blocks & 4u) load_block(slot_of_key(2), &map_k, B_K_IN + 2, 2);
            // values: V0 after K1, V1 after K2 (or the position rows), V2 after K0
            ATT_WARP_WAIT(B_S_DONE + 1, par);
            ATT_WARP_WAIT(B_UK_DONE + 1, par);
            if (blocks & 1u) load_block(0, &map_v, B_V_IN + 0, 0);
            if (blocks & 4u) {
                ATT_WARP_WAIT(B_S_DONE + 2, (ph >> 2) & 1u);
                ATT_WARP_WAIT(B_UK_DONE + 2, (ph >> 2) & 1u);
            }
            load_block(1, &map_v, B_V_IN + 1, 1);
            if (blocks & 4u) {
                if (blocks & 1u) {
                    ATT_WARP_WAIT(B_S_DONE + 0, ph & 1u);
                    ATT_WARP_WAIT(B_UK_DONE + 0, ph & 1u);
                }
                load_block(2, &map_v, B_V_IN + 2, 2);
            }
            before = blocks;
            ph_before = ph;
            ph ^= blocks;
        }
    } else if (warp == kSoftmaxWarps + 1) {
        // ------------------------------------------------------------- MMA issuer
        constexpr uint32_t idesc128 = make_instr_desc<KIND_F16>(128, 128);
        constexpr uint32_t idesc16 = make_instr_desc<KIND_F16>(128, 16);
        // B = V[keys, features] as it lies in memory: MN-major (features contiguous),
        // 8-key groups 1024 bytes apart, the second 64 features 16 KB on; 16 keys = 2048 bytes
        constexpr uint32_t idesc_v = idesc128 | (1u << 16);
        const uint64_t desc_q = make_smem_desc<128>(smem_u32(sm.q)), desc_tail = make_smem_desc<128>(smem_u32(sm.tail));
        const uint64_t desc_slot[2] = {make_smem_desc<128>(smem_u32(sm.slot[0])), make_smem_desc<128>(smem_u32(sm.slot[1]))};
        // K step of 16 halves inside a K-major operand block, in descriptor units of 16 bytes
        auto k_offset = [](int ks) { return static_cast<uint32_t>((ks / 4) * (kAtomBytes / 16) + 2 * (ks % 4)); };
        bool any = false;
        int tile = first_tile - 1;
        grid_dependency_wait();          // geometry, Q: the bounded waits begin behind the kernel in front
        for (int item = first_item; ok && item < last_item; ++item) {
            if (++tile == p.tiles) tile = 0;
            const TilePlace at(p.rows, tile);
            if (at.padding()) continue;
            const uint32_t blocks = at.blocks(), par = (ph >> 1) & 1u;
            ATT_WARP_WAIT(B_Q_IN, par);
            ATT_WARP_WAIT(B_P_IN, par);
            tc_fence_after_sync();
            // (columns [0, 272) are free: P_READY of the tile before came after their last read)
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) {           // 16 features per MMA
                    const uint32_t off = k_offset(ks);
                    tc_mma<KIND_F16>(tmem, desc_q + off, desc_slot[0] + off, idesc128, ks > 0);
                    tc_mma<KIND_F16>(tmem + 128u, desc_q + off, desc_slot[1] + off, idesc128, ks > 0);
                    tc_mma<KIND_F16>(tmem + 256u, desc_q + off, desc_tail + (ks / 4) * (kTailBytes / 32) + 2u * (ks % 4), idesc16, ks > 0);
                }
                tc_commit(&sm.bar[B_QP_DONE]);
            }
            __syncwarp();
            // S_0 and the context share their columns
            if (any) ATT_WARP_WAIT(B_CTX_READ, par ^ 1u);
            any = true;
#pragma unroll 1
            for (int b = 0; b < 3; ++b) {
                if (!((blocks >> b) & 1u)) continue;
                if (b == 1) ATT_WARP_WAIT(B_QP_DRAINED, par);   // columns [0, 272) are free
                ATT_WARP_WAIT(B_K_IN + b, (ph >> b) & 1u);
                tc_fence_after_sync();
                const uint64_t desc_k = desc_slot[0] + static_cast<uint32_t>(slot_of_key(b) * (kSlotBytes / 16));
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks)
                        tc_mma<KIND_F16>(tmem + score_col(b), desc_q + k_offset(ks), desc_k + k_offset(ks), idesc128, ks > 0);
                    tc_commit(&sm.bar[B_S_DONE + b]);
                }
                __syncwarp();
            }
            if (!ok) break;
            uint32_t accumulate = 0;
#pragma unroll 1
            for (int b = 0; b < 3; ++b) {
                if (!((blocks >> b) & 1u)) continue;
                ATT_WARP_WAIT(B_V_IN + b, (ph >> b) & 1u);
                ATT_WARP_WAIT(B_P_READY + b, (ph >> b) & 1u);
                tc_fence_after_sync();
                const uint64_t desc_v = static_cast<uint64_t>((smem_u32(sm.slot[b]) & 0x3FFFFu) >> 4) |
                                        (static_cast<uint64_t>(kAtomBytes >> 4) << 16) | (64ull << 32) |
                                        (1ull << 46) | (2ull << 61);
                const uint64_t desc_p = make_smem_desc<128>(smem_u32(sm.pr[b & 1]));
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks)         // 16 keys per MMA
                        tc_mma<KIND_F16>(tmem + kCtxCol, desc_p + k_offset(ks), desc_v + ks * 128u, idesc_v, ks > 0 ? 1u : accumulate);
                    tc_commit(&sm.bar[B_PV_DONE + b]);
                }
                __syncwarp();
                accumulate = 1;
            }
            ph ^= blocks;
        }
    } else {
        // ------------------------------------------ bias terms, QP drain, softmax, output
        const int quad = warp % 4, part = warp / 4;
        const int ql = quad * 32 + lane;                       // query row inside the tile = TMEM lane
        const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quad * 32) << 16);
        constexpr float kLog2e = 1.4426950408889634f;
        const float scale2 = kSoftmaxScale * kLog2e;
        const Pair scale22 = pair_of(scale2, scale2);
        // Bias terms: four lanes per operand row, 32 features each (32 * qt ..).  The eight lanes of a
        // 16-byte shared-memory access are four rows of one 64-feature atom: eight different chunks.
        const int qt = (lane & 1) | ((lane >> 2) & 2), bias_row = warp * 8 + (((lane >> 1) & 3) | ((lane >> 2) & 4));
        int head_now = -1, base_now = -1, q0_now = 0;          // what vp and uk in shared memory belong to
        int head = first_head, tile = first_tile - 1;
        if (!p.early) grid_dependency_wait();
        bool waited = !p.early;
        for (int item = first_item; ok && item < last_item; ++item) {
            if (++tile == p.tiles) { tile = 0; ++head; }
            const TilePlace at(p.rows, tile);
            const int q0 = at.q0, valid = at.valid;
            if (at.padding()) {                  // the whole tile is padding: zeros
                if (!waited) grid_dependency_wait();
                waited = true;
                for (int c = tid; c < kTile * 16; c += kSoftmaxThreads)
                    *reinterpret_cast<uint4*>(p.out + static_cast<size_t>(at.base + q0 + c / 16) * p.ldo + head * kDim + (c % 16) * 8) =
                        make_uint4(0, 0, 0, 0);
                continue;
            }
            const uint32_t blocks = at.blocks(), par = (ph >> 1) & 1u;
            const bool q_live = q0 + ql < valid;
            const int key_first = q0 - kReach;       // window index kk <-> key key_first + kk
            // u . K of the first two key blocks is there when the tile in front of this one was done last
            const bool follows = head == head_now && at.base == base_now && q0 == q0_now + kTile;
            if (head != head_now) {
                // v . P_j for the 272 position rows (per-column constant of QP): four threads per row,
                // 32 features each, from the staged operand tiles
                if (tid < kDim) sm.bias_u[tid / 32][tid % 32] = __half2float(p.bias_u[head * kDim + tid]);
                float bias[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) bias[i] = __half2float(p.bias_v[head * kDim + 32 * qt + i]);
                ATT_WAIT(B_P_IN, par);
#pragma unroll 1
                for (int row = bias_row; row < kPosRows; row += kSoftmaxThreads / 4) {   // (whole warps)
                    const uint8_t* atom = row < 256 ? sm.slot[row / 128] + (qt / 2) * kAtomBytes
                                                    : sm.tail + (qt / 2) * (kTailBytes / 2);
                    float acc = bias_dot32(atom, row < 256 ? row % 128 : row - 256, 4 * (qt % 2), bias);
                    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
                    acc += __shfl_xor_sync(0xffffffffu, acc, 8);
                    if (qt == 0) sm.vp[row] = acc;
                }
                __syncwarp();
            }
            head_now = head; base_now = at.base; q0_now = q0;
            if (!waited) grid_dependency_wait();
            waited = true;
            if (lane == 0) {
                bulk_wait_read_all();            // the staged context of the tile before has left
                mbar_arrive(&sm.bar[B_VP_DONE]);
            }
            ATT_WAIT(B_VP_DONE, par);
            // QP: tensor memory -> fp16 rows in shared memory, bias term added.  Row ql is stored shifted
            // right by (ql & 1) halves, so that the run of position columns a key piece needs (kk0 - ql ...)
            // starts on a 32-bit word for every thread.  Part p drains columns [64p, 64p + 64), the last
            // part the 16 columns beyond as well.
            ATT_WAIT(B_QP_DONE, par);
            tc_fence_after_sync();
            {
                uint32_t* row = reinterpret_cast<uint32_t*>(&sm.qp[ql * kQpPitch]) + 32 * part;
                const bool odd = (ql & 1) != 0;
                // An odd row's words hold (column 2m - 1, column 2m): one byte permute per word with a
                // selector per lane; the two words shared with the neighbouring parts are written as halves.
                const uint32_t sel = odd ? 0x5432u : 0x7654u;
                uint32_t carry = 0;
                // 32 columns per step (part 3: a last step of 16 columns)
                const int steps = part == kParts - 1 ? 3 : 2;
#pragma unroll 1
                for (int st = 0; st < steps; ++st) {
                    const int c0 = 64 * part + 32 * st;
                    uint32_t r[32], w[16];
                    tmem_ld_32x32(lane_addr + static_cast<uint32_t>(c0), r);    // (beyond column 272: never stored)
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float4 t = *reinterpret_cast<const float4*>(&sm.vp[c0 + 4 * i]);
                        const __half2 h0 = __floats2half2_rn(__uint_as_float(r[4 * i + 0]) + t.x, __uint_as_float(r[4 * i + 1]) + t.y);
                        const __half2 h1 = __floats2half2_rn(__uint_as_float(r[4 * i + 2]) + t.z, __uint_as_float(r[4 * i + 3]) + t.w);
                        w[2 * i + 0] = *reinterpret_cast<const uint32_t*>(&h0);
                        w[2 * i + 1] = *reinterpret_cast<const uint32_t*>(&h1);
                    }
                    uint32_t* dst = row + 16 * st;
                    if (st == 0 && odd)
                        reinterpret_cast<__half*>(dst)[1] = __ushort_as_half(static_cast<unsigned short>(w[0] & 0xFFFFu));
                    else
                        dst[0] = __byte_perm(carry, w[0], sel);
#pragma unroll
                    for (int i = 1; i < 8; ++i) dst[i] = __byte_perm(w[i - 1], w[i], sel);
                    if (st < 2) {
#pragma unroll
                        for (int i = 8; i < 16; ++i) dst[i] = __byte_perm(w[i - 1], w[i], sel);
                        carry = w[15];
                    } else {
                        carry = w[7];
                    }
                }
                if (odd)
                    reinterpret_cast<__half*>(row + (part == kParts - 1 ? 40 : 32))[0] =
                        __ushort_as_half(static_cast<unsigned short>(carry >> 16));
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.bar[B_QP_DRAINED]);
            ATT_WAIT(B_QP_DRAINED, par);

            // keys this query sees, in window coordinates: [lo, hi] (empty for a padding row)
            const int lo = max(ql, -key_first);
            const int hi = q_live ? min(ql + 2 * kReach, valid - 1 - key_first) : -1;
            const unsigned span = static_cast<unsigned>(hi - lo);          // hi < lo: nothing passes
            // the same for the whole warp: pieces outside [w_lo, w_hi] are skipped, pieces inside
            // [a_lo, a_hi] are seen whole by every row
            const int w_lo = max(quad * 32, -key_first), w_hi = min(quad * 32 + 31 + 2 * kReach, valid - 1 - key_first);
            const int a_lo = max(quad * 32 + 31, -key_first);
            const int a_hi = q0 + quad * 32 + 31 < valid ? min(quad * 32 + 2 * kReach, valid - 1 - key_first) : -1;
            const int ring = q0 / kTile + 2;                   // u . K of key block b of the tile: row (ring + b) % 3
            // A piece = 32 consecutive columns of this thread's scores, one per block.  Pass 0 writes the
            // scaled and masked scores back over the accumulators and finds the row maximum.
            float mx = -INFINITY, sum = 0.0f;
#pragma unroll 1
            for (int b = 0; b < 3; ++b) {
                if (!((blocks >> b) & 1u)) continue;
                if (b < 2 && follows) {
                    if (lane == 0) mbar_arrive(&sm.bar[B_UK_DONE + b]);
                } else {
                    // u . K_kk for the 128 keys of a new block: four threads per key, 32 features each
                    float bias[32];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float4 t = *reinterpret_cast<const float4*>(&sm.bias_u[qt][4 * i]);
                        bias[4 * i] = t.x; bias[4 * i + 1] = t.y; bias[4 * i + 2] = t.z; bias[4 * i + 3] = t.w;
                    }
                    ATT_WAIT(B_K_IN + b, (ph >> b) & 1u);
                    float acc = bias_dot32(sm.slot[slot_of_key(b)] + (qt / 2) * kAtomBytes, bias_row, 4 * (qt % 2), bias);
                    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
                    acc += __shfl_xor_sync(0xffffffffu, acc, 8);
                    if (qt == 0) sm.uk[(ring + b) % 3][bias_row] = acc;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sm.bar[B_UK_DONE + b]);
                    ATT_WAIT(B_UK_DONE + b, (ph >> b) & 1u);
                }
                ATT_WAIT(B_S_DONE + b, (ph >> b) & 1u);
                tc_fence_after_sync();
                const int kk0 = b * 128 + part * 32;
                if (kk0 + 31 < w_lo || kk0 > w_hi) continue;
                const bool whole = kk0 >= a_lo && kk0 + 31 <= a_hi;
                // two halves of 16 columns: 32 at a time spilled
#pragma unroll 1
                for (int c0 = 0; c0 < 32; c0 += 16) {
                    uint32_t r[16];
                    const uint32_t taddr = lane_addr + score_col(b) + static_cast<uint32_t>(part * 32 + c0);
                    tmem_ld_32x16(taddr, r);
                    // position scores of columns kk0 + c0 - ql ..: stored from half (ql & 1) on, so the
                    // run starts at a word of the row (kk0 is even)
                    const __half2* qp2 = reinterpret_cast<const __half2*>(&sm.qp[ql * kQpPitch + kk0 + c0 - ql + (ql & 1)]);
                    const float4* uk4 = reinterpret_cast<const float4*>(&sm.uk[(ring + b) % 3][part * 32 + c0]);
                    float s[16];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float4 u = uk4[c];
                        s[4 * c + 0] = add_half(__low2half(qp2[2 * c]), u.x);
                        s[4 * c + 1] = add_half(__high2half(qp2[2 * c]), u.y);
                        s[4 * c + 2] = add_half(__low2half(qp2[2 * c + 1]), u.z);
                        s[4 * c + 3] = add_half(__high2half(qp2[2 * c + 1]), u.w);
                    }
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const Pair sum2 = pair_add(pair_of(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), pair_of(s[2 * i], s[2 * i + 1]));
                        const float2 scaled = halves_of(pair_mul(sum2, scale22));
                        s[2 * i] = scaled.x;
                        s[2 * i + 1] = scaled.y;
                    }
                    if (!whole) {
                        const int off = kk0 + c0 - lo;
                        const bool some = hi >= lo;
#pragma unroll
                        for (int i = 0; i < 16; ++i) s[i] = some && static_cast<unsigned>(off + i) <= span ? s[i] : -INFINITY;
                    }
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        mx = fmaxf(mx, s[i]);
                        r[i] = __float_as_uint(s[i]);
                    }
                    tmem_st_32x16(taddr, r);
                }
            }
            if (!ok) break;
            tmem_st_wait();
            sm.rowmax[part][ql] = mx;
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.bar[B_PASS0_DONE]);
            // all warps are done with the position scores: their space takes the probabilities
            ATT_WAIT(B_PASS0_DONE, par);
            mx = fmaxf(fmaxf(sm.rowmax[0][ql], sm.rowmax[1][ql]), fmaxf(sm.rowmax[2][ql], sm.rowmax[3][ql]));
            if (mx == -INFINITY) mx = 0.0f;            // a query without keys: every probability is 0
            const Pair minus_mx2 = pair_of(-mx, -mx);
            // Pass 1: probabilities, block by block, into the A operand of the last contraction.
#pragma unroll 1
            for (int b = 0; b < 3; ++b) {
                if (!((blocks >> b) & 1u)) continue;
                uint32_t w[16];
                const int kk0 = b * 128 + part * 32;
                if (kk0 + 31 < w_lo || kk0 > w_hi) {
#pragma unroll
                    for (int e = 0; e < 16; ++e) w[e] = 0u;
                } else {
                    uint32_t r[32];
                    tmem_ld_32x32(lane_addr + score_col(b) + static_cast<uint32_t>(part * 32), r);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        float2 pr = halves_of(pair_add(pair_of(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])), minus_mx2));
                        asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(pr.x));     // ex2(-inf) = 0
                        asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(pr.y));
                        sum += pr.x + pr.y;
                        const __half2 h = __floats2half2_rn(pr.x, pr.y);
                        w[e] = *reinterpret_cast<const uint32_t*>(&h);
                    }
                }
                // the third block takes the first one's buffer
                if (b == 2 && (blocks & 1u)) ATT_WAIT(B_PV_DONE + 0, ph & 1u);
                uint8_t* atom = sm.pr[b & 1] + (part / 2) * kAtomBytes;   // keys 64 * (part / 2) .. + 63 of the block
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    *reinterpret_cast<uint4*>(atom + swz(ql, 4 * (part % 2) + e)) =
                        make_uint4(w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]);
                fence_proxy_async_smem();
                tc_fence_before_sync();                                   // the scores have been read
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.bar[B_P_READY + b]);
            }
            if (!ok) break;
            sm.rowsum[part][ql] = sum;
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.bar[B_SUM + quad]);
            ATT_WAIT(B_SUM + quad, par);
            sum = (sm.rowsum[0][ql] + sm.rowsum[1][ql]) + (sm.rowsum[2][ql] + sm.rowsum[3][ql]);
            const float inv = sum > 0.0f ? 1.0f / sum : 0.0f;
            const int last = (blocks & 4u) ? 2 : 1;
            ATT_WAIT(B_PV_DONE + last, (ph >> last) & 1u);
            tc_fence_after_sync();
            // context: this warp writes features [32 * part, +32) of its 32 queries
            {
                uint32_t r[32];
                tmem_ld_32x32(lane_addr + kCtxCol + static_cast<uint32_t>(part * 32), r);
                tmem_ld_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.bar[B_CTX_READ]);
                uint32_t w[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const __half2 h = __floats2half2_rn(__uint_as_float(r[2 * i]) * inv, __uint_as_float(r[2 * i + 1]) * inv);
                    w[i] = q_live ? *reinterpret_cast<const uint32_t*>(&h) : 0u;
                }
                // out through shared memory (64-byte rows, 64-byte swizzle; the probabilities there are done
                // with) and one TMA store per warp: 16-byte stores a row apart took 4.5k of a tile's 25k cycles
                uint8_t* stage = sm.pr[1] + warp * 2048;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    *reinterpret_cast<uint4*>(stage + lane * 64 + ((i ^ ((lane >> 1) & 3)) << 4)) =
                        make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    tma_store_2d(&map_out, stage, head * kDim + part * 32, at.base + q0 + quad * 32);
                    bulk_commit_group();
                }
            }
            ph ^= blocks;
        }
        if (lane == 0) bulk_wait_all();          // this warp's stores have landed
    }

    // ------------------------------------------------------------------- teardown
    if (*abort_flag != 0) {
        // give copies / MMAs still in flight time to land before shared and tensor memory are released
        const uint64_t start = global_timer_ns();
        while (global_timer_ns() - start < 200000ull) __nanosleep(1000);
        if (tid == 0 && p.status != nullptr) atomicExch(p.status, 1);
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == kSoftmaxWarps + 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, 512);
    }
}

}  // namespace att5
}  // namespace pk100

using namespace pk100;

int pk100_local_attention_rows(void* stream_v, const void* query, int ldq, const void* key, int ldk, const void* value, int ldv,
                               const void* position, const void* bias_u, const void* bias_v, void* output, int ldo,
                               int total_rows, const pk100_rows& geometry, bool constants_settled, int* status) {
    using namespace att5;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    const unsigned long long rows = static_cast<unsigned long long>(total_rows);
    CUtensorMap map_q, map_k, map_p, map_p16, map_v, map_out;
    int rc = pk100_tensor_map_2d(&map_q, query, 2, rows, 1024, ldq, kTile, 128);
    if (rc == PK100_OK) rc = pk100_tensor_map_2d(&map_k, key, 2, rows, 1024, ldk, 128, 128);
    if (rc == PK100_OK) rc = pk100_tensor_map_2d(&map_p, position, 2, kHeads * kPosRows, kDim, kDim, 128, 128);
    if (rc == PK100_OK) rc = pk100_tensor_map_2d(&map_p16, position, 2, kHeads * kPosRows, kDim, kDim, 16, 128);
    if (rc == PK100_OK) rc = pk100_tensor_map_2d(&map_v, value, 2, rows, 1024, ldv, 128, 128);
    if (rc == PK100_OK) rc = pk100_tensor_map_2d(&map_out, output, 2, rows, 1024, ldo, 32, 64);
    if (rc != PK100_OK) return rc;

    constexpr int smem_bytes = static_cast<int>(sizeof(Smem)) + 1024;
    const cudaError_t granted = pk100_grant_smem<local_attention_tcgen05_kernel>(smem_bytes);
    if (granted != cudaSuccess) return static_cast<int>(granted);
    const int tiles = total_rows / kTile;
    Params p{static_cast<const __half*>(bias_u), static_cast<const __half*>(bias_v), static_cast<__half*>(output), ldo,
             tiles, geometry, constants_settled ? 1 : 0, status};
    // one persistent CTA per SM; fewer while decoder clusters of earlier batches hold some of them
    const long long items = static_cast<long long>(kHeads) * tiles;
    const int ctas = static_cast<int>(items < pk100_cta_budget() ? items : pk100_cta_budget());
    pk100_launch_chained(local_attention_tcgen05_kernel, dim3(ctas), dim3(kThreads), smem_bytes, stream, map_q, map_k, map_p, map_p16, map_v, map_out, p);
    return pk100_launch_status();
}

extern "C" int pk100_local_relpos_attention_tcgen05(
    void* stream_v, const void* query, int ldq, const void* key, int ldk, const void* value, int ldv,
    const void* position, const void* bias_u, const void* bias_v, void* output, int ldo, int segments,
    int seg_stride, int valid_rows, const int* seg_valid, int* status) {
    using namespace att5;
    if (!query || !key || !value || !position || !bias_u || !bias_v || !output) return PK100_ERR_NULL;
    if (segments < 0 || seg_stride <= 0) return PK100_ERR_SHAPE;
    if (seg_stride % kTile != 0) return PK100_ERR_SHAPE;          // whole 128-query tiles
    if (ldq < 1024 || ldk < 1024 || ldv < 1024 || ldo < 1024 || (ldq | ldk | ldv | ldo) % 8 != 0) return PK100_ERR_SHAPE;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(query) | reinterpret_cast<uintptr_t>(key) |
                           reinterpret_cast<uintptr_t>(value) | reinterpret_cast<uintptr_t>(position) |
                           reinterpret_cast<uintptr_t>(output);
    if (bits & 15u) return PK100_ERR_ALIGN;
    if (segments == 0) return PK100_OK;
    return pk100_local_attention_rows(stream_v, query, ldq, key, ldk, value, ldv, position, bias_u, bias_v, output, ldo,
                                      segments * seg_stride, pk100_rows{nullptr, seg_stride, valid_rows, seg_valid}, false, status);
}
