// Cluster decoder (included by decoder_kernels.cu).
//
// One thread-block cluster of 16 CTAs decodes up to 8 utterances in lockstep rounds.  Every CTA owns
// 40 hidden units (160 gate rows per LSTM layer), 40 prediction rows and 65 joint rows; the phases of a
// round hand their vectors to the peers through distributed shared memory: a CTA pushes its slice into
// all 16 CTAs with st.async, which also credits the bytes to an mbarrier of the receiving CTA, and
// each CTA waits (bounded) on its own mbarriers only.  Every CTA runs the same control flow on
// replicated utterance state.
//
// A round is a latency chain (cell -> exchange -> prediction -> exchange -> joint -> exchange ->
// decision), so the CTA is split by role:
//   warps 0-19   matrix warps: mma.sync with the WEIGHTS as the 16-row A operand and the
//                activations of 4 utterances (hi, lo pairs) as the 8 columns of B, half the
//                instructions of the form that pads 8 utterances to 16 rows of A.  The product with the
//                recurrent weights only needs the new hidden state, not the next token, so it runs
//                right behind the prediction GEMM, under the prediction exchange, and is ready when the
//                next token is known.
//   control warps  one to four per utterance (their threads own its 40 units in registers): decision, LSTM
//                cell, reductions of the K-split partial sums, all sends.  The token's table row and the
//                new frame's encoder values go straight to the registers of the threads that use them.
//                The prediction slice is turned into the joint input relu(enc + pred) by its owner and
//                travels as such.
// Weights are resident where they fit: recurrent weights (two layers: the critical input weights of the
// second layer first) in tensor memory, joint rows in shared memory (one fp16 layer: half of them in
// tensor memory), prediction rows in
// registers; with two fp16 layers the rest streams from L2 in "fragment order" (16 contiguous bytes per
// lane and mma), off the critical path.  The input half of the first layer, W_ih . embedding[token],
// is a table [1025, 2560] computed once per call by one GEMM; a round gathers 4 x 40 floats of it.
//
// `Cache` = long-request numerics: recurrent weights and layer 1's input weights are INT8 codes, the
// hidden state that multiplies them is rne(h * 127): exact integer products (mma.sync m16n8k32 s8, one
// column per utterance).  Prediction projection and joint run in fp32 in the reference's
// summation order.
constexpr int kCl = 16;                          // CTAs per cluster
constexpr int kClUnits = kHidden / kCl;          // 40 hidden units / prediction rows per CTA
constexpr int kClJoint = 65;                     // joint rows per CTA (16 x 65 >= 1030)
constexpr int kMatrixWarps = 20;
constexpr int kMatrixThreads = kMatrixWarps * 32;
constexpr int cl_threads(int utts) { return kMatrixThreads + 32 * utts; }      // one control warp per utterance it is sized for
constexpr uint32_t kTmemColumns = 512;

// named barriers (0 is __syncthreads)
enum : int { BAR_CONTROL = 1, BAR_PRED = 2, BAR_GO = 3, BAR_LAYER1 = 4 };
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// How a [rows x K] slice is split over the matrix warps: KG k-groups x NG row groups; a warp walks KP
// k-pairs (64 bytes of K each: two mma k-steps) over NT tiles of 16 rows.
template <int KG_, int NG_, int KP_, int NT_, int TILES_>
struct Split {
    static constexpr int KG = KG_, NG = NG_, KP = KP_, NT = NT_, kTiles = TILES_;
    static constexpr int kPerCta = KG * KP * TILES_ * 64;       // uint4: [kg][kp][tile][k-step][lane]
    static_assert(KG * NG == kMatrixWarps && NG * NT >= TILES_ && (NG - 1) * NT < TILES_, "all warps, all tiles");
};
// The k-groups of the fp16 splits fix the order of the fp32 sums.
using LstmSplit = Split<4, 5, 5, 2, 10>;         // 160 gate rows x 640
using Lstm1Split = Split<2, 10, 10, 1, 10>;      // half of layer 1 (input or recurrent): 160 gate rows x 640
using CodeSplit = Split<2, 10, 5, 1, 10>;        // INT8 codes: 160 gate rows x 640
using PredSplit = Split<20, 1, 1, 3, 3>;         // 40 rows x 640 (third tile half empty)
using JointSplit = Split<10, 2, 2, 3, 5>;        // 65 rows x 640 (fifth tile: one row)
constexpr int kGatePitch = 168, kPredPitch = 40, kJointPitch = 72;   // = 8 (mod 32): conflict-free partial sums

struct ClLayout { size_t base, lstm, pred, joint, xtab, lstm1, cache, total; };
__host__ __device__ inline ClLayout cl_layout(int utts) {
    ClLayout l;
    const size_t a = dec_layout(utts).total, b = xch_layout(utts).total;
    l.base = ((a > b ? a : b) + 255) / 256 * 256;
    size_t off = l.base;
    l.lstm = off; off += static_cast<size_t>(kCl) * LstmSplit::kPerCta * 16;
    l.pred = off; off += static_cast<size_t>(kCl) * PredSplit::kPerCta * 16;
    l.joint = off; off += static_cast<size_t>(kCl) * JointSplit::kPerCta * 16;
    l.xtab = off; off += static_cast<size_t>(kTokenOutputs) * kGates * 4;
    l.lstm1 = off; off += static_cast<size_t>(kCl) * 2 * Lstm1Split::kPerCta * 16;   // input weights, then recurrent ones
    l.cache = off; off += 256;        // max |w| of the three tensors of the INT8 cache
    l.total = off;
    return l;
}

enum : int { CLPACK_GATES = 0, CLPACK_PRED = 1, CLPACK_JOINT = 2 };

// dst[cta][kg][kp][tile][k-step][lane] = the A fragment (a0..a3) of one mma: lane (g = lane / 4, t = lane % 4)
// holds rows g and g + 8 at bytes 4t and 4t + 16 of the k-step's 32 bytes.  Codes: the INT8 codes of the
// tensor (scale index `scale`), one byte per column.
template <typename S, int Mode, bool Codes>
__global__ void tdt_pack_kernel(uint4* dst, const __half* w, const float* absmax, int scale) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= kCl * S::kPerCta) return;
    int rest = idx;
    const int lane = rest % 32; rest /= 32;
    const int step = rest % 2; rest /= 2;
    const int tile = rest % S::kTiles; rest /= S::kTiles;
    const int kp = rest % S::KP; rest /= S::KP;
    const int kg = rest % S::KG; rest /= S::KG;
    const int r = rest;
    const int g = lane / 4, t = lane % 4;
    constexpr int kPerWord = Codes ? 4 : 2;
    const int k0 = ((kg * S::KP + kp) * 2 + step) * 8 * kPerWord;
    auto word = [&](int n, int k) -> unsigned {
        int row = -1;
        if (Mode == CLPACK_GATES) row = (n % 4) * kHidden + r * kClUnits + n / 4;   // gate-major rows
        else if (Mode == CLPACK_PRED) row = n < kClUnits ? r * kClUnits + n : -1;
        else if (n < kClJoint && r * kClJoint + n < kJointRows) row = r * kClJoint + n;
        if (row < 0) return 0u;
        const __half* src = w + static_cast<size_t>(row) * kHidden + k;
        if constexpr (Codes) {
            const float s = cache_scale(absmax, scale);
            unsigned out = 0;
            for (int i = 0; i < 4; ++i) out |= static_cast<unsigned>(cache_code(src[i], s) & 255) << (8 * i);
            return out;
        } else {
            return static_cast<unsigned>(__half_as_ushort(src[0])) | (static_cast<unsigned>(__half_as_ushort(src[1])) << 16);
        }
    };
    const int n = tile * 16 + g, ka = k0 + t * kPerWord, kb = ka + 4 * kPerWord;
    dst[idx] = make_uint4(word(n, ka), word(n + 8, ka), word(n, kb), word(n + 8, kb));
}

// Shared memory of one CTA; NU = utterances it is sized for (4 or 8).
template <int Layers, bool Cache, int NU>
struct CSmem {
    // activations that multiply weight matrices, one row per B column: fp16 rows 2u (hi) and 2u + 1 (lo),
    // Cache: one row of INT8 codes per utterance (8 rows always: the rows behind NU stay zero).  The
    // pitches keep ldmatrix free of bank conflicts.
    static constexpr int kActPitch = Cache ? 656 : 1296;               // bytes
    static constexpr int kActRows = Cache ? 8 : 2 * NU;
    using Act = uint8_t[kActRows * kActPitch];
    static constexpr bool kJointResident = Cache || Layers == 1 || NU == 4;
    // K pairs of the streamed matrix that fit beside the rest (see weight placement below)
    static constexpr int kSmemPairs = Layers == 1 ? 0 : Cache ? (NU == 4 ? 3 : 2) : (NU == 4 ? 1 : 2);
    static constexpr int kPairBytes = kMatrixWarps * (Cache ? 1 : 2) * 1024;
    static constexpr int kJointBytes = !kJointResident ? 0 : Cache ? kClJoint * 1280 : 10 * 2 * (4 * 1024 + 128);
    static constexpr int kGateParts = Cache ? 2 : 4;

    alignas(16) uint8_t joint[kJointBytes > 0 ? kJointBytes : 16];
    alignas(16) uint8_t pairs[kSmemPairs > 0 ? kSmemPairs * kPairBytes : 16];
    alignas(16) Act h0;                                   // hidden state of layer 0, written by all CTAs
    alignas(16) uint8_t h1[Layers == 2 ? sizeof(Act) : 16];            // of layer 1
    alignas(16) float hf[Cache ? NU : 1][Cache ? kHidden : 4];         // Cache: fp32 state of the top layer
    alignas(16) uint8_t ax[Cache ? NU * kHidden * 4 : kActRows * kActPitch];   // joint input: hi / lo rows or fp32
    alignas(16) float gates0[kGateParts * NU * kGatePitch];            // partial sums of the recurrent product
    alignas(16) float gates1[Layers == 2 ? 4 * NU * kGatePitch : 4];   // layer 1: parts 0, 1 input, 2, 3 recurrent
    alignas(16) float part[Cache ? NU * kJointPitch : (20 * NU * kPredPitch > 10 * NU * kJointPitch ? 20 * NU * kPredPitch : 10 * NU * kJointPitch)];
    alignas(16) uint8_t stage_act[NU][2][kClUnits * 2];   // outgoing slice: hi / lo halves, Cache: codes (first 40 bytes)
    alignas(16) float stage_f[NU][kClUnits];              // outgoing fp32 slice (Cache: hidden state / joint input)
    float pred[Cache ? NU : 1][kClUnits];                 // Cache: this CTA's prediction slice, finished by the matrix warps
    float bias0[kClUnits][4], bias1[Layers == 2 ? kClUnits : 1][4], pred_bias[kClUnits], joint_bias[kJointPitch];
    float cache_mul[3];                                   // scale / 127 of w_hh[0], w_hh[1], w_ih[1]
    unsigned long long keys[2][NU][3 * kCl];              // [round parity][utterance][source CTA, third of its rows]
    int dur[2][NU];                                       // [round parity][utterance] winning duration
    uint64_t hbar0, hbar1, abar, kbar[2];           // exchange mbarriers (count 1 + transaction bytes)
    uint32_t tmem_base;
    alignas(8) unsigned char done[8], need[8];            // read as 64-bit words; done = 1 behind the last utterance
    int abort;
#ifdef PK100_DEC_PROFILE
    long long prof[16], last_stamp;
#endif
};

constexpr size_t kCtaSmem = 227 * 1024;
static_assert(sizeof(CSmem<1, false, 4>) <= kCtaSmem && sizeof(CSmem<1, false, 8>) <= kCtaSmem && sizeof(CSmem<2, false, 4>) <= kCtaSmem &&
              sizeof(CSmem<2, false, 8>) <= kCtaSmem && sizeof(CSmem<1, true, 4>) <= kCtaSmem && sizeof(CSmem<1, true, 8>) <= kCtaSmem &&
              sizeof(CSmem<2, true, 4>) <= kCtaSmem && sizeof(CSmem<2, true, 8>) <= kCtaSmem, "fits one CTA's shared memory");

// Remote store that credits its bytes to an mbarrier of the destination CTA.  `addr` and `bar`
// are shared::cluster addresses of the same CTA.
__device__ __forceinline__ void st_async_v4(uint32_t addr, uint4 v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async_b64(uint32_t addr, unsigned long long v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];"
                 ::"r"(addr), "l"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async_b32(uint32_t addr, unsigned v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
                 ::"r"(addr), "r"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ float fast_sigmoid(float x) { return __fdividef(1.0f, 1.0f + __expf(-x)); }
__device__ __forceinline__ float fast_tanh(float x) { return 2.0f * fast_sigmoid(2.0f * x) - 1.0f; }

__device__ __forceinline__ void dec_mma_s8(int (&d)[4], const uint4& a, unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void dec_mma_f16(float (&d)[4], const uint4& a, unsigned b0, unsigned b1) {
    const unsigned av[4] = {a.x, a.y, a.z, a.w};
    dec_mma(d, av, b0, b1);
}
__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

// Index of a fragment in a packed slice.
template <typename S>
__device__ __forceinline__ int frag_index(int kg, int kp, int tile, int step, int lane) {
    return ((((kg * S::KP + kp) * S::kTiles + tile) * 2 + step) * 32) + lane;
}

// Accumulators of one warp: [tile][block of 8 B columns][4].
template <bool Codes> struct AccT { using type = float; };
template <> struct AccT<true> { using type = int; };

// One k-pair (64 bytes of K): `load(tile, step)` yields the A fragment, `act` is this lane's ldmatrix address
// of the pair (rows of block nb are 8 * pitch apart).
template <bool Codes, int NT, int NB, typename Load>
__device__ __forceinline__ void pair_mma(typename AccT<Codes>::type (&acc)[NT][NB][4], const uint8_t* act, int pitch,
                                         int tiles, Load&& load) {
    unsigned b[NB][4];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) dec_ldmatrix_x4(b[nb], act + nb * 8 * pitch);
#pragma unroll
    for (int step = 0; step < 2; ++step)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            if (NT > 1 && j >= tiles) continue;
            const uint4 a = load(j, step);
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
                if constexpr (Codes) dec_mma_s8(acc[j][nb], a, b[nb][2 * step], b[nb][2 * step + 1]);
                else dec_mma_f16(acc[j][nb], a, b[nb][2 * step], b[nb][2 * step + 1]);
            }
        }
}

// Partial sums of one tile: part[(kg * NU + u) * pitch + row].  fp16: column pair t of a block is (hi, lo) of
// utterance 4 * nb + t; codes: column = utterance.
template <bool Codes, int NB, int NU>
__device__ __forceinline__ void store_part(const typename AccT<Codes>::type (&acc)[NB][4], float* part, int kg, int row0,
                                           int rows, int pitch, int lane) {
    const int g = lane / 4, t = lane % 4;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int row = row0 + g + 8 * half;
            if (row >= rows) continue;
            if constexpr (Codes) {
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    if (2 * t + e < NU) part[(kg * NU + 2 * t + e) * pitch + row] = static_cast<float>(acc[nb][2 * half + e]);
            } else {
                part[(kg * NU + 4 * nb + t) * pitch + row] = acc[nb][2 * half] + acc[nb][2 * half + 1];
            }
        }
}

#ifdef PK100_DEC_PROFILE
#define CL_STAMP(i) do { if (tid == kMatrixThreads) { const long long now__ = clock64(); sm.prof[i] += now__ - sm.last_stamp; sm.last_stamp = now__; } } while (0)
#else
#define CL_STAMP(i) do { } while (0)
#endif

struct ClWeights {               // packed slices (see tdt_pack_kernel) and the input table
    const uint4 *lstm, *pred, *joint, *lstm1_in, *lstm1_rec;
    const float* xtab;
};

template <int Layers, bool Cache, int NU>
__global__ void __launch_bounds__(cl_threads(NU), 1)
tdt_cluster_kernel(const DecParams p, const ClWeights w) {
    using Smem = CSmem<Layers, Cache, NU>;
    constexpr int kClThreads = cl_threads(NU), kControlThreads = kClThreads - kMatrixThreads;
    constexpr int NB = Cache ? 1 : NU / 4;                 // blocks of 8 B columns
    constexpr int kPitch = Smem::kActPitch;
    using Gates0 = typename std::conditional<Cache, CodeSplit, LstmSplit>::type;
    using Gates1 = typename std::conditional<Cache, CodeSplit, Lstm1Split>::type;
    // tensor-memory columns of one warp: the matrix that is needed first, then what else fits
    constexpr int kCols0 = Layers == 2 && !Cache ? 16 : Gates0::KP * Gates0::NT * 8;      // w_hh[0] (two fp16 layers: one pair)
    constexpr int kCols1 = Layers == 2 ? Gates1::KP * 8 : 0;                              // w_ih[1]
    constexpr int kCols2 = Layers == 2 && Cache ? 16 : 0;                                 // w_hh[1]: two pairs
    constexpr int kColsJ = Layers == 1 && !Cache ? 16 : 0;                                // joint: the first pair of two tiles
    constexpr int kCols = kCols0 + kCols1 + kCols2 + kColsJ;
    static_assert(5 * kCols <= static_cast<int>(kTmemColumns), "fits tensor memory");

    extern __shared__ __align__(16) uint8_t cs_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(cs_raw);
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    const bool matrix = warp < kMatrixWarps;
    const int r = static_cast<int>(cluster_ctarank());
    const int U = p.utts;
    volatile int* abort_flag = &sm.abort;

    // ---- set-up: cleared state, biases, barriers
    for (int i = tid; i < static_cast<int>(sizeof(Smem) / 16); i += kClThreads) reinterpret_cast<uint4*>(cs_raw)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    if (tid < kClUnits * 4) {
        const int slot = tid / 4, gt = tid % 4, row = gt * kHidden + r * kClUnits + slot;
        sm.bias0[slot][gt] = p.b_ih[0][row] + p.b_hh[0][row];
        if constexpr (Layers == 2) sm.bias1[slot][gt] = p.b_ih[1][row] + p.b_hh[1][row];
    }
    if (tid < kClUnits) sm.pred_bias[tid] = p.b_pred[r * kClUnits + tid];
    if (tid < 3) sm.cache_mul[tid] = (Cache && (tid == 0 || Layers == 2)) ? cache_mul(cache_scale(p.cache_absmax, tid)) : 0.0f;
    if (tid < kClJoint && r * kClJoint + tid < kJointRows) sm.joint_bias[tid] = p.b_joint[r * kClJoint + tid];
    if (tid < 8) {
        const bool done = tid >= U || p.frames[tid] <= 0 || !in_window(p, tid);
        sm.done[tid] = done;
        sm.need[tid] = !done;
    }
    if (tid == 0) {
        mbar_init(&sm.hbar0, 1);
        mbar_init(&sm.hbar1, 1);
        mbar_init(&sm.abar, 1);
        mbar_init(&sm.kbar[0], 1);
        mbar_init(&sm.kbar[1], 1);
        fence_barrier_init();
    }
    if (warp == 1) {                 // one warp owns the tensor-memory allocation (all of it; one CTA per SM)
        tmem_alloc(&sm.tmem_base, kTmemColumns);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    // resident joint rows
    if constexpr (Cache) {
        // half-lane hl reads words hl + 16 s, s = 0..19: four of them per 16-byte group [row][s / 4][hl]
        for (int i = tid; i < kClJoint * 80; i += kClThreads) {
            const int n = i / 80, c = i % 80, row = r * kClJoint + n;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (row < kJointRows) {
                const uint32_t* src = reinterpret_cast<const uint32_t*>(p.w_joint + static_cast<size_t>(row) * kHidden) + (c / 16) * 64 + c % 16;
                v = make_uint4(__ldg(src), __ldg(src + 16), __ldg(src + 32), __ldg(src + 48));
            }
            *reinterpret_cast<uint4*>(sm.joint + n * 1280 + c * 16) = v;
        }
    } else if constexpr (Smem::kJointResident) {
        const uint4* src = w.joint + static_cast<size_t>(r) * JointSplit::kPerCta;
        for (int i = tid; i < JointSplit::kPerCta; i += kClThreads) {
            const int block = i / 320, rest = i % 320;           // block = (kg, kp): 5 tiles x 2 steps x 32 lanes
            uint4* dst = reinterpret_cast<uint4*>(sm.joint) + block * (256 + 8);
            if (rest < 256) dst[rest] = __ldg(src + i);
            else if (rest % 32 < 4) dst[256 + (rest - 256) / 32 * 4 + rest % 32] = __ldg(src + i);   // fifth tile: row 64 only
        }
    }
    __syncthreads();
    cluster_sync_all();      // every CTA's shared memory and mbarriers are ready before a peer writes

    // After the joint, all warps: warp (u, third) reduces a third of this CTA's joint rows of utterance u to
    // its best key, sent to every CTA by the same warp; the owner of the five duration rows sends the
    // first strict maximum among them.
    unsigned round = 0;
    auto publish_keys = [&](unsigned long long done8) {
        const int par = static_cast<int>(round & 1u);
        const int u = warp / 3, third = warp % 3;
        if (u >= U || ((done8 >> (8 * u)) & 1ull) != 0ull) return;
        const int n = third * 32 + lane, row = r * kClJoint + n;
        const bool owned = n < kClJoint && row < kJointRows;
        float total = 0.0f;
        if (owned) {
            if constexpr (Cache) {
                total = sm.part[u * kJointPitch + n];          // finished score of the fp32 joint
            } else {
                total = sm.joint_bias[n];
#pragma unroll
                for (int kg = 0; kg < JointSplit::KG; ++kg) total += sm.part[(kg * NU + u) * kJointPitch + n];
            }
        }
        const uint32_t bar = map_to_cta(smem_u32(&sm.kbar[par]), static_cast<uint32_t>(lane % kCl));
        constexpr int kDurCta = kTokenOutputs / kClJoint, kDurRow = kTokenOutputs % kClJoint;
        static_assert(kDurRow / 32 == (kDurRow + kDurations - 1) / 32 && kDurRow + kDurations <= kClJoint, "one warp holds the durations");
        if (r == kDurCta && third == kDurRow / 32) {
            int duration = 0;
            float best = __shfl_sync(0xffffffffu, total, kDurRow % 32);
#pragma unroll
            for (int i = 1; i < kDurations; ++i) {
                const float v = __shfl_sync(0xffffffffu, total, kDurRow % 32 + i);
                if (v > best) { best = v; duration = i; }
            }
            if (lane < kCl)
                st_async_b32(map_to_cta(smem_u32(&sm.dur[par][u]), static_cast<uint32_t>(lane)), static_cast<unsigned>(duration), bar);
        }
        unsigned ordered = 0;                                  // order-preserving bits; NaN and foreign rows never win
        if (owned && row < kTokenOutputs && total == total) {
            if (total == 0.0f) total = 0.0f;                   // canonicalise -0
            const unsigned bits = __float_as_uint(total);
            ordered = (bits & 0x80000000u) ? ~bits : (bits ^ 0x80000000u);
        }
        const unsigned top = __reduce_max_sync(0xffffffffu, ordered);
        // ties to the lower row; a third whose rows all produced NaN still publishes a (losing) key
        const unsigned first = __reduce_max_sync(0xffffffffu, ordered == top && top != 0u ? 2047u - static_cast<unsigned>(row) : 0u);
        const unsigned low = ((top != 0u ? first : 2047u - kTokenOutputs) << 21) | 1u;
        if (lane < kCl)
            st_async_b64(map_to_cta(smem_u32(&sm.keys[par][u][r * 3 + third]), static_cast<uint32_t>(lane)),
                         (static_cast<unsigned long long>(top) << 32) | low, bar);
    };

    if (matrix) {
        // ============================================================ matrix warps
        const uint32_t tm = sm.tmem_base + (static_cast<uint32_t>((warp % 4) * 32) << 16) + static_cast<uint32_t>((warp / 4) * kCols);
        const uint4* lstm = w.lstm + static_cast<size_t>(r) * Gates0::kPerCta;
        [[maybe_unused]] const uint4* in1 = w.lstm1_in + static_cast<size_t>(r) * Gates1::kPerCta;
        [[maybe_unused]] const uint4* rec1 = w.lstm1_rec + static_cast<size_t>(r) * Gates1::kPerCta;
        const int kg0 = warp / Gates0::NG, tile0 = (warp % Gates0::NG) * Gates0::NT;
        [[maybe_unused]] const int kg1 = warp / Gates1::NG, tile1 = warp % Gates1::NG;
        // ---- resident slices: tensor memory and the spare shared memory
        auto fill = [&](const uint4* src, uint32_t col) {          // two fragments of one (pair, tile)
            const uint4 a = __ldg(src), b = __ldg(src + 32);
            const uint32_t v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            tmem_st_32x8(tm + col, v);
        };
#pragma unroll
        for (int i = 0; i < kCols0 / 8; ++i)
            fill(lstm + frag_index<Gates0>(kg0, i / Gates0::NT, tile0 + i % Gates0::NT, 0, lane), i * 8);
        if constexpr (Layers == 2) {
#pragma unroll
            for (int i = 0; i < kCols1 / 8; ++i) fill(in1 + frag_index<Gates1>(kg1, i, tile1, 0, lane), kCols0 + i * 8);
#pragma unroll
            for (int i = 0; i < kCols2 / 8; ++i) fill(rec1 + frag_index<Gates1>(kg1, i, tile1, 0, lane), kCols0 + kCols1 + i * 8);
        }
        if constexpr (kColsJ > 0) {
            const uint4* src = w.joint + static_cast<size_t>(r) * JointSplit::kPerCta;
#pragma unroll
            for (int j = 0; j < 2; ++j)
                fill(src + frag_index<JointSplit>(warp / JointSplit::NG, 0, (warp % JointSplit::NG) * 2 + j, 0, lane), kCols0 + j * 8);
        }
        tmem_st_wait();
        uint4* pairs = reinterpret_cast<uint4*>(sm.pairs);         // [pair][warp][tile][step][lane]
        if constexpr (Smem::kSmemPairs > 0) {
#pragma unroll
            for (int i = 0; i < Smem::kSmemPairs; ++i)
#pragma unroll
                for (int j = 0; j < (Cache ? 1 : 2); ++j)
#pragma unroll
                    for (int step = 0; step < 2; ++step)
                        pairs[(((i * kMatrixWarps + warp) * (Cache ? 1 : 2) + j) * 2 + step) * 32 + lane] = __ldg(
                            Cache ? rec1 + frag_index<Gates1>(kg1, 2 + i, tile1, step, lane)
                                  : lstm + frag_index<Gates0>(kg0, 1 + i, tile0 + j, step, lane));
        }
        // prediction rows in registers: fp16 fragments of tiles 0 and 1 and the lower rows of tile 2;
        // Cache: rows `warp` and `warp + 20` of the caller's matrix, words lane + 32 i
        uint32_t predw[20];
        if constexpr (Cache) {
#pragma unroll
            for (int i = 0; i < 20; ++i)
                predw[i] = __ldg(reinterpret_cast<const uint32_t*>(
                    p.w_pred + static_cast<size_t>(r * kClUnits + warp + (i / 10) * kMatrixWarps) * kHidden) + lane + 32 * (i % 10));
        } else {
            const uint4* src = w.pred + static_cast<size_t>(r) * PredSplit::kPerCta;
#pragma unroll
            for (int tile = 0; tile < 3; ++tile)
#pragma unroll
                for (int step = 0; step < 2; ++step) {
                    const uint4 v = __ldg(src + frag_index<PredSplit>(warp, 0, tile, step, lane));
                    if (tile < 2) {
                        predw[tile * 8 + step * 4] = v.x; predw[tile * 8 + step * 4 + 1] = v.y;
                        predw[tile * 8 + step * 4 + 2] = v.z; predw[tile * 8 + step * 4 + 3] = v.w;
                    } else {
                        predw[16 + step * 2] = v.x; predw[17 + step * 2] = v.z;
                    }
                }
        }
        // this lane's ldmatrix address inside an activation block: row lane % 8, 16-byte column lane / 8
        const uint32_t lane_act = (lane % 8) * kPitch + (lane / 8) * 16;

        // part[kg] of one gate product.  Source of k-pair kp: tensor memory at column base + 8 * NT * kp for
        // kp < in_tmem, then `in_smem` pairs from shared memory, then the packed copy in L2; the next pair's
        // fragments are fetched under the mmas of the current one.
        auto gate_product = [&](auto split, const uint4* packed, const uint8_t* act, float* part, int kg, int tile,
                                int part_kg, auto tmem_pairs, auto smem_pairs, uint32_t col) {
            using S = decltype(split);
            constexpr int kTm = decltype(tmem_pairs)::value, kSm = decltype(smem_pairs)::value;
            typename AccT<Cache>::type acc[S::NT][NB][4] = {};
            uint32_t f[2][S::NT * 8];
            auto fetch = [&](int kp, uint32_t (&dst)[S::NT * 8]) {
                if (kp < kTm) {
                    if constexpr (S::NT == 2) tmem_ld_32x16(tm + col + kp * 16, dst);
                    else tmem_ld_32x8(tm + col + kp * 8, dst);
                } else {
#pragma unroll
                    for (int j = 0; j < S::NT; ++j)
#pragma unroll
                        for (int step = 0; step < 2; ++step) {
                            const uint4 v = kp < kTm + kSm
                                ? pairs[((((kp - kTm) * kMatrixWarps + warp) * S::NT + j) * 2 + step) * 32 + lane]
                                : __ldcg(packed + frag_index<S>(kg, kp, tile + j, step, lane));
                            dst[j * 8 + step * 4] = v.x; dst[j * 8 + step * 4 + 1] = v.y;
                            dst[j * 8 + step * 4 + 2] = v.z; dst[j * 8 + step * 4 + 3] = v.w;
                        }
                }
            };
            fetch(0, f[0]);
            if (kTm > 0) tmem_ld_wait();
            const uint8_t* a = act + kg * S::KP * 64 + lane_act;
#pragma unroll
            for (int kp = 0; kp < S::KP; ++kp) {
                if (kp + 1 < S::KP) fetch(kp + 1, f[(kp + 1) & 1]);
                pair_mma<Cache, S::NT, NB>(acc, a + kp * 64, kPitch, S::NT, [&](int j, int step) {
                    const uint32_t* v = &f[kp & 1][j * 8 + step * 4];
                    return make_uint4(v[0], v[1], v[2], v[3]);
                });
                if (kp + 1 < kTm) tmem_ld_wait();
            }
#pragma unroll
            for (int j = 0; j < S::NT; ++j)
                store_part<Cache, NB, NU>(acc[j], part, part_kg, (tile + j) * 16, 160, kGatePitch, lane);
        };
        using std::integral_constant;
        auto recurrent0 = [&]() {
            gate_product(Gates0{}, lstm, sm.h0, sm.gates0, kg0, tile0, kg0, integral_constant<int, kCols0 / (8 * Gates0::NT)>{},
                         integral_constant<int, Layers == 2 && !Cache ? Smem::kSmemPairs : 0>{}, 0);
        };

        uint32_t hphase = 0;
        while (true) {
            bar_sync(BAR_GO, kClThreads);
            const unsigned long long done8 = *reinterpret_cast<const unsigned long long*>(sm.done);
            const unsigned long long need8 = *reinterpret_cast<const unsigned long long*>(sm.need);
            if (done8 == 0x0101010101010101ull || sm.abort != 0) break;
            if (need8 != 0ull) {
                mbar_wait_bounded(&sm.hbar0, hphase, abort_flag);
                if constexpr (Layers == 2) {
                    gate_product(Gates1{}, in1, sm.h0, sm.gates1, kg1, tile1, kg1, integral_constant<int, kCols1 / 8>{},
                                 integral_constant<int, 0>{}, kCols0);
                    bar_arrive(BAR_LAYER1, kClThreads);
                    recurrent0();                          // under the second layer's cell and exchange
                    mbar_wait_bounded(&sm.hbar1, hphase, abort_flag);
                }
                const uint8_t* top = Layers == 2 ? sm.h1 : sm.h0;
                if constexpr (Cache) {
                    // fp32 in the reference's summation order (decoder.cu:672-684): lane l takes elements
                    // 2l + 64w as one fma chain that starts from the bias in lane 0, then a shuffle tree
                    for (int u = 0; u < U; ++u) {
                        if (((need8 >> (8 * u)) & 1ull) == 0ull) continue;
                        float s0 = lane == 0 ? sm.pred_bias[warp] : 0.0f, s1 = lane == 0 ? sm.pred_bias[warp + kMatrixWarps] : 0.0f;
#pragma unroll
                        for (int i = 0; i < 10; ++i) {
                            const float2 h = *reinterpret_cast<const float2*>(&sm.hf[u][2 * lane + 64 * i]);
                            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&predw[i]));
                            const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&predw[10 + i]));
                            s0 = fmaf(a.y, h.y, fmaf(a.x, h.x, s0));
                            s1 = fmaf(b.y, h.y, fmaf(b.x, h.x, s1));
                        }
#pragma unroll
                        for (int off = 16; off > 0; off /= 2) {
                            s0 += __shfl_down_sync(0xffffffffu, s0, off);
                            s1 += __shfl_down_sync(0xffffffffu, s1, off);
                        }
                        if (lane == 0) {
                            sm.pred[u][warp] = s0;
                            sm.pred[u][warp + kMatrixWarps] = s1;
                        }
                    }
                } else {
                    float acc[3][NB][4] = {};
                    pair_mma<false, 3, NB>(acc, top + warp * 64 + lane_act, kPitch, 3, [&](int j, int step) {
                        return j < 2 ? make_uint4(predw[j * 8 + step * 4], predw[j * 8 + step * 4 + 1], predw[j * 8 + step * 4 + 2], predw[j * 8 + step * 4 + 3])
                                     : make_uint4(predw[16 + step * 2], 0u, predw[17 + step * 2], 0u);
                    });
#pragma unroll
                    for (int j = 0; j < 3; ++j) store_part<false, NB, NU>(acc[j], sm.part, warp, j * 16, kClUnits, kPredPitch, lane);
                }
                bar_arrive(BAR_PRED, kClThreads);
                // the recurrent product of the NEXT step, under the prediction's reduction and exchange
                if constexpr (Layers == 2)
                    gate_product(Gates1{}, rec1, sm.h1, sm.gates1, kg1, tile1, 2 + kg1, integral_constant<int, kCols2 / 8>{},
                                 integral_constant<int, Cache ? Smem::kSmemPairs : 0>{}, kCols0 + kCols1);
                else
                    recurrent0();
            }
            // the joint rows' fragments do not depend on the activations: requested before the wait (all of them
            // where the registers allow it)
            constexpr int kAhead = Cache || (Layers == 2 && NU == 4) ? 0 : NU == 4 ? JointSplit::KP : 1;
            [[maybe_unused]] const int jkg = warp / JointSplit::NG, jng = warp % JointSplit::NG;
            [[maybe_unused]] uint4 jf[JointSplit::KP][3][2];
            [[maybe_unused]] uint32_t jt[16];                      // the pair that lives in tensor memory
            auto joint_fetch = [&](int kp) {
                const uint4* block = Smem::kJointResident
                    ? reinterpret_cast<const uint4*>(sm.joint) + (jkg * JointSplit::KP + kp) * (256 + 8)
                    : w.joint + static_cast<size_t>(r) * JointSplit::kPerCta + (jkg * JointSplit::KP + kp) * 320;
                if (kColsJ > 0 && kp == 0) tmem_ld_32x16(tm + kCols0, jt);
#pragma unroll
                for (int step = 0; step < 2; ++step) {
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        if (kColsJ == 0 || kp > 0) jf[kp][j][step] = block[((jng * 2 + j) * 2 + step) * 32 + lane];
                    jf[kp][2][step] = jng == 0 && lane < 4 ? block[256 + (Smem::kJointResident ? step * 4 : step * 32) + lane]
                                                           : make_uint4(0, 0, 0, 0);
                }
            };
            if constexpr (!Cache) {
#pragma unroll
                for (int kp = 0; kp < kAhead; ++kp) joint_fetch(kp);
            }
            mbar_wait_bounded(&sm.abar, round & 1u, abort_flag);
            if (need8 != 0ull) hphase ^= 1u;
            // ---- joint rows
            if constexpr (Cache) {
                // fp32 in the reference's summation order (decoder.cu:697-713): one row per half-warp, half-lane
                // l takes elements 2l + 32s as one fma chain that starts from the bias in half-lane 0,
                // then a shuffle tree.  Rows hw and hw + 40 share the loads of x.
                const int hw = tid / 16, hl = tid % 16;
                const bool second = hw + 40 < kClJoint;
                const uint4* w0 = reinterpret_cast<const uint4*>(sm.joint + hw * 1280) + hl;
                const uint4* w1 = reinterpret_cast<const uint4*>(sm.joint + (second ? hw + 40 : hw) * 1280) + hl;
                for (int u = 0; u < U; ++u) {
                    if (((done8 >> (8 * u)) & 1ull) != 0ull) continue;
                    const float* x = reinterpret_cast<const float*>(sm.ax) + u * kHidden + 2 * hl;
                    float s0 = hl == 0 ? sm.joint_bias[hw] : 0.0f, s1 = hl == 0 && second ? sm.joint_bias[hw + 40] : 0.0f;
#pragma unroll
                    for (int q = 0; q < 5; ++q) {
                        const uint4 a4 = w0[16 * q], b4 = w1[16 * q];
                        const uint32_t a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float2 xv = *reinterpret_cast<const float2*>(x + 32 * (4 * q + i));
                            const float2 av = __half22float2(*reinterpret_cast<const __half2*>(&a[i]));
                            const float2 bv = __half22float2(*reinterpret_cast<const __half2*>(&b[i]));
                            s0 = fmaf(av.y, xv.y, fmaf(av.x, xv.x, s0));
                            s1 = fmaf(bv.y, xv.y, fmaf(bv.x, xv.x, s1));
                        }
                    }
#pragma unroll
                    for (int off = 8; off > 0; off /= 2) {
                        s0 += __shfl_down_sync(0xffffffffu, s0, off, 16);
                        s1 += __shfl_down_sync(0xffffffffu, s1, off, 16);
                    }
                    if (hl == 0) {
                        sm.part[u * kJointPitch + hw] = s0;
                        if (second) sm.part[u * kJointPitch + hw + 40] = s1;
                    }
                }
            } else {
                float acc[3][NB][4] = {};
#pragma unroll
                for (int kp = 0; kp < JointSplit::KP; ++kp) {
                    if (kp >= kAhead) joint_fetch(kp);
                    if (kColsJ > 0 && kp == 0) tmem_ld_wait();
                    pair_mma<false, 3, NB>(acc, sm.ax + (jkg * JointSplit::KP + kp) * 64 + lane_act, kPitch, jng == 0 ? 3 : 2,
                                           [&](int j, int step) {
                        const int i = (j * 2 + step) * 4;
                        return kColsJ > 0 && kp == 0 && j < 2 ? make_uint4(jt[i], jt[i + 1], jt[i + 2], jt[i + 3]) : jf[kp][j][step];
                    });
                }
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    if (j < 2 || jng == 0)
                        store_part<false, NB, NU>(acc[j], sm.part, jkg, (j < 2 ? jng * 2 + j : 4) * 16, kClJoint, kJointPitch, lane);
            }
            __syncthreads();
            publish_keys(done8);
            round += 1;
        }
    } else {
        // ============================================================ control warps
        const int ct = tid - kMatrixThreads, cw = ct / 32;
        // sends: thread = (peer, item % kSubs); shared::cluster address of `x` in the peer = peer_base + offset of x
        constexpr int kSubs = kControlThreads / kCl;
        const uint32_t local_base = smem_u32(cs_raw), peer_base = map_to_cta(local_base, static_cast<uint32_t>(ct % kCl));
        const int sub = ct / kCl;
        auto in_peer = [&](const void* x) { return peer_base + (smem_u32(x) - local_base); };
        // 40 fp16 units as (hi, lo) rows 2u, 2u + 1 of `act`; `who` = utterances that send, one byte each
        auto send_halves = [&](uint8_t* act, uint64_t* bar_local, unsigned long long who) {
            const uint32_t bar = in_peer(bar_local);
            for (int u = 0; u < U; ++u) {
                if (((who >> (8 * u)) & 1ull) == 0ull) continue;
                for (int i = sub; i < 10; i += kSubs) {
                    const int lo = i / 5, chunk = i % 5;
                    st_async_v4(in_peer(act + (2 * u + lo) * kPitch + r * kClUnits * 2 + chunk * 16),
                                *reinterpret_cast<const uint4*>(&sm.stage_act[u][lo][chunk * 16]), bar);
                }
            }
        };
        auto send_floats = [&](float* dst, uint64_t* bar_local, unsigned long long who) {
            const uint32_t bar = in_peer(bar_local);
            for (int u = 0; u < U; ++u) {
                if (((who >> (8 * u)) & 1ull) == 0ull) continue;
                for (int i = sub; i < 10; i += kSubs)
                    st_async_v4(in_peer(dst + u * kHidden + r * kClUnits + i * 4), *reinterpret_cast<const uint4*>(&sm.stage_f[u][i * 4]), bar);
            }
        };
        auto send_codes = [&](uint8_t* act, uint64_t* bar_local, unsigned long long who) {
            const uint32_t bar = in_peer(bar_local);
            for (int u = 0; u < U; ++u) {
                if (((who >> (8 * u)) & 1ull) == 0ull || sub >= 5) continue;
                st_async_b64(in_peer(act + u * kPitch + r * kClUnits + sub * 8),
                             *reinterpret_cast<const unsigned long long*>(&sm.stage_act[u][0][sub * 8]), bar);
            }
        };
        auto gate_part = [&](const float* gates, int kg, int u, int slot) {
            return *reinterpret_cast<const float4*>(&gates[(kg * NU + u) * kGatePitch + slot * 4]);
        };
        // The warps of a team serve one utterance: its 40 slots (= this CTA's units) belong to fixed threads,
        // so cell state, gate inputs, encoder values and the utterance's counters live in registers (the
        // counters and the decision itself are replicated in the team's warps).
        const int team = NU == 8 || U > 2 ? 1 : (U == 2 ? 2 : 4);          // warps per utterance
        const int my = cw / team, first_slot = (cw % team) * 32 + lane, slot_step = team * 32;
        constexpr int kPasses = 2;                                         // slots per thread at most
        const bool serving = my < U;
        const bool leader = serving && cw % team == 0 && lane == 0;
        bool live = serving && !sm.done[serving ? my : 0];
        bool need = live;
        const int total_frames = live ? min(p.frames[my], p.seg_stride) : 0;   // never past the utterance's block
        const __half* enc_rows = p.enc_proj + static_cast<size_t>(serving ? my : 0) * p.seg_stride * kHidden + r * kClUnits;
        int frame = 0, symbols = 0, count = 0;
        float cell0[kPasses] = {}, cell1[kPasses] = {}, pred[kPasses] = {}, xg[kPasses][4] = {};
        __half enc[kPasses] = {};                                          // (converted where used: the load stays in flight)
        auto for_slots = [&](auto&& f) {                                   // f(pass, slot)
#pragma unroll
            for (int i = 0; i < kPasses; ++i) {
                const int slot = first_slot + i * slot_step;
                if (slot < kClUnits) f(i, slot);
            }
        };
        auto fetch_enc = [&]() {
            for_slots([&](int i, int slot) { enc[i] = __ldg(enc_rows + static_cast<size_t>(frame) * kHidden + slot); });
        };
        if (live) fetch_enc();
        // LSTM cell of one unit from its four gate sums; stages h for the exchange
        auto cell_update = [&](const float (&gsum)[4], float& cstate, int slot) {
            if constexpr (Cache) {
                // the reference's approximations: h is rounded to 8 bits next, and a code that flips moves a gate
                const float h = ref_lstm_cell(gsum, cstate);
                sm.stage_act[my][0][slot] = static_cast<uint8_t>(quantize_i8(h * 127.0f));
                sm.stage_f[my][slot] = h;
            } else {
                const float cell = fast_sigmoid(gsum[1]) * cstate + fast_sigmoid(gsum[0]) * fast_tanh(gsum[2]);
                cstate = cell;
                const float h = fast_sigmoid(gsum[3]) * fast_tanh(cell);
                const __half hi = __float2half_rn(h);
                reinterpret_cast<__half*>(sm.stage_act[my][0])[slot] = hi;
                reinterpret_cast<__half*>(sm.stage_act[my][1])[slot] = __float2half_rn(h - __half2float(hi));
            }
        };
        // bytes one utterance contributes to the exchanges
        constexpr uint32_t kTopTx = Cache ? kHidden + kHidden * 4 : kHidden * 4, kLowTx = Cache ? kHidden : kHidden * 4;
#ifdef PK100_DEC_PROFILE
        if (ct == 0) sm.last_stamp = clock64();
#endif
        while (true) {
            __syncwarp();
            bar_arrive(BAR_GO, kClThreads);                // this round's flags are published
            const int par = static_cast<int>(round & 1u);
            if (need) {
                // ---- cell of layer 0: table row + h . w_hh^T + bias
                for_slots([&](int i, int slot) {
                    float gsum[4];
                    if constexpr (Cache) {
                        // the scaled recurrent sum is rounded BEFORE the bias is added, as in the reference
                        // (decoder.cu:113, :626-640): a fused multiply-add here parts from the reference
                        // kernel's tokens after a few hundred steps
                        const float4 a = gate_part(sm.gates0, 0, my, slot), b = gate_part(sm.gates0, 1, my, slot);
                        const float rec[4] = {a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w};
#pragma unroll
                        for (int g = 0; g < 4; ++g)
                            gsum[g] = __fadd_rn(__fadd_rn(__fmul_rn(rec[g], sm.cache_mul[0]), sm.bias0[slot][g]), xg[i][g]);
                    } else {
#pragma unroll
                        for (int g = 0; g < 4; ++g) gsum[g] = sm.bias0[slot][g] + xg[i][g];
#pragma unroll
                        for (int kg = 0; kg < LstmSplit::KG; ++kg) {
                            const float4 v = gate_part(sm.gates0, kg, my, slot);
                            gsum[0] += v.x; gsum[1] += v.y; gsum[2] += v.z; gsum[3] += v.w;
                        }
                    }
                    cell_update(gsum, cell0[i], slot);
                });
            }
            CL_STAMP(0);
            bar_sync(BAR_CONTROL, kControlThreads);
            const unsigned long long done8 = *reinterpret_cast<const unsigned long long*>(sm.done);
            const unsigned long long need8 = *reinterpret_cast<const unsigned long long*>(sm.need);
            const unsigned long long live8 = ~done8 & 0x0101010101010101ull;
            // a wait that gave up raised sm.abort; it is read here, behind the barriers that end a round
            if (live8 == 0ull || sm.abort != 0) break;
            CL_STAMP(1);
            if (need8 != 0ull) {
                if constexpr (Cache) {
                    send_codes(sm.h0, &sm.hbar0, need8);
                    if constexpr (Layers == 1) send_floats(&sm.hf[0][0], &sm.hbar0, need8);
                } else {
                    send_halves(sm.h0, &sm.hbar0, need8);
                }
            }
            if (ct == kControlThreads - 1) {               // (transaction counts may trail the transactions)
                const uint32_t needs = static_cast<uint32_t>(__popcll(need8)), lives = static_cast<uint32_t>(__popcll(live8));
                if (need8 != 0ull) {
                    mbar_arrive_expect_tx(&sm.hbar0, needs * (Layers == 1 ? kTopTx : kLowTx));
                    if (Layers == 2) mbar_arrive_expect_tx(&sm.hbar1, needs * kTopTx);
                }
                mbar_arrive_expect_tx(&sm.abar, lives * kHidden * 4);
                mbar_arrive_expect_tx(&sm.kbar[par], lives * (3 * kCl * 8 + 4));
            }
            CL_STAMP(2);
            if (need8 != 0ull) {
                if constexpr (Layers == 2) {
                    bar_sync(BAR_LAYER1, kClThreads);
                    CL_STAMP(3);
                    // ---- cell of layer 1: [fresh h of layer 0 | own h] . [w_ih | w_hh]^T + bias
                    if (need) for_slots([&](int i, int slot) {
                        float gsum[4];
                        const float4 a = gate_part(sm.gates1, 0, my, slot), b = gate_part(sm.gates1, 1, my, slot);
                        const float4 c = gate_part(sm.gates1, 2, my, slot), d = gate_part(sm.gates1, 3, my, slot);
                        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
                        const float cv[4] = {c.x, c.y, c.z, c.w}, dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            // Cache: rounded recurrent product first, the input product fused onto it, bias last
                            // (decoder.cu:113, :655-663)
                            if constexpr (Cache)
                                gsum[g] = __fadd_rn(fmaf(av[g] + bv[g], sm.cache_mul[2], __fmul_rn(cv[g] + dv[g], sm.cache_mul[1])), sm.bias1[slot][g]);
                            else
                                gsum[g] = (((sm.bias1[slot][g] + av[g]) + bv[g]) + cv[g]) + dv[g];
                        }
                        cell_update(gsum, cell1[i], slot);
                    });
                    bar_sync(BAR_CONTROL, kControlThreads);
                    CL_STAMP(4);
                    if constexpr (Cache) {
                        send_codes(sm.h1, &sm.hbar1, need8);
                        send_floats(&sm.hf[0][0], &sm.hbar1, need8);
                    } else {
                        send_halves(sm.h1, &sm.hbar1, need8);
                    }
                }
                bar_sync(BAR_PRED, kClThreads);
            } else {
                bar_sync(BAR_CONTROL, kControlThreads);    // everyone has read the flags
            }
            CL_STAMP(5);
            // ---- prediction slice where the state moved; this CTA's 40 columns of the joint input relu(enc + pred)
            if (live) for_slots([&](int i, int slot) {
                if (need) {
                    if constexpr (Cache) {
                        pred[i] = sm.pred[my][slot];
                    } else {
                        float part[PredSplit::KG];
#pragma unroll
                        for (int kg = 0; kg < PredSplit::KG; ++kg) part[kg] = sm.part[(kg * NU + my) * kPredPitch + slot];
                        pred[i] = sm.pred_bias[slot];
#pragma unroll
                        for (int kg = 0; kg < PredSplit::KG; ++kg) pred[i] += part[kg];
                    }
                }
                const float x = fmaxf(__half2float(enc[i]) + pred[i], 0.0f);
                if constexpr (Cache) {
                    sm.stage_f[my][slot] = x;
                } else {
                    const __half hi = __float2half_rn(x);
                    reinterpret_cast<__half*>(sm.stage_act[my][0])[slot] = hi;
                    reinterpret_cast<__half*>(sm.stage_act[my][1])[slot] = __float2half_rn(x - __half2float(hi));
                }
            });
            bar_sync(BAR_CONTROL, kControlThreads);
            CL_STAMP(6);
            if constexpr (Cache) send_floats(reinterpret_cast<float*>(sm.ax), &sm.abar, live8);
            else send_halves(sm.ax, &sm.abar, live8);
            CL_STAMP(7);
            __syncthreads();                               // joint sums are complete
            CL_STAMP(8);
            publish_keys(done8);
            CL_STAMP(9);
            mbar_wait_bounded(&sm.kbar[par], (round >> 1) & 1u, abort_flag);
            CL_STAMP(10);

            // ---- decision (replicated in every CTA)
            if (live) {
                const unsigned long long k0 = sm.keys[par][my][lane], k1 = lane < kCl ? sm.keys[par][my][32 + lane] : 0ull;
                const unsigned long long best = k1 > k0 ? k1 : k0;
                const unsigned top = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(best >> 32));
                const unsigned low = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(best >> 32) == top ? static_cast<unsigned>(best) : 0u);
                int token = 2047 - static_cast<int>((low >> 21) & 0x7FFu);
                // keys not delivered (a wait gave up), or every token score of the round was NaN: a
                // blank; the second case is reported as status bit 4
                const bool no_score = token > kBlank;
                if (no_score) token = kBlank;
                need = token != kBlank;
                // requests for the next round: the token's table row, then the encoder values of the new frame
                if (need) {
                    const float* row = w.xtab + static_cast<size_t>(token) * kGates + r * kClUnits;
                    for_slots([&](int i, int slot) {
#pragma unroll
                        for (int g = 0; g < 4; ++g) xg[i][g] = __ldg(row + g * kHidden + slot);
                    });
                }
                const int duration = sm.dur[par][my];
                const int old_frame = frame;
                frame += duration;
                symbols += 1;
                if (duration != 0 || symbols == kMaxSymbols) {
                    if (duration == 0) frame += 1;
                    symbols = 0;
                }
                live = frame < total_frames;
                if (live && frame != old_frame) fetch_enc();
                if (leader) {
                    sm.done[my] = !live;
                    sm.need[my] = live && need;
                    if (r == 0) {
                        if (no_score && sm.abort == 0 && p.status != nullptr) atomicOr(p.status, 4);
                        if (need && count < p.max_tokens) {
                            p.tokens[static_cast<size_t>(my) * p.max_tokens + count] = token;
                            if (p.durations_out != nullptr) p.durations_out[static_cast<size_t>(my) * p.max_tokens + count] = duration;
                        }
                    }
                }
                count += need ? 1 : 0;
                need = need && live;
            }
            round += 1;
            CL_STAMP(11);
        }
        if (r == 0 && leader && in_window(p, my)) p.counts[my] = min(count, p.max_tokens);
    }
    // ---- teardown
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(sm.tmem_base, kTmemColumns);
    }
    cluster_sync_all();      // no CTA leaves while a peer may still address its shared memory
#ifdef PK100_DEC_PROFILE
    if (r == 0 && tid == 0)
        for (int i = 0; i < 16; ++i)
            reinterpret_cast<volatile long long*>(p.workspace + xch_layout(U).abort)[2 + i] = sm.prof[i];
#endif
    if (r == 0 && tid == kMatrixThreads) reinterpret_cast<volatile int*>(p.workspace + xch_layout(U).abort)[2] = static_cast<int>(round);
    if (sm.abort != 0 && tid == 0 && p.status != nullptr) atomicExch(p.status, 2);
}
