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
//                recurrent weights only needs the new hidden state, not the next token, so it runs off the
//                chain: behind the joint (one or two utterances: under the key exchange, the decision and
//                the next token's table row, so that nothing competes with the joint input's exchange) or
//                behind the prediction GEMM (more utterances: under the joint input's exchange, which is the
//                longest gap then).
//   control warps  LSTM cell, decision, reductions of the K-split partial sums, all sends.  One or two
//                utterances: five warps with 8 of the CTA's 40 units each, four lanes per unit (one per gate, so that
//                a gate sum is one chain of adds and the four activations run side by side), the decision replicated
//                in each of them (utterance state in lane u); more: one warp per utterance, a unit per lane.  The
//                token's table row and the new frame's encoder values go straight to the registers of the lanes
//                that use them.
//                The prediction slice is turned into the joint input relu(enc + pred) by its owner and
//                travels as such.
// Exchanges: a slice is staged in shared memory and consecutive lanes send consecutive 16-byte pieces to the
// same peer, whose buffer holds it in one piece ([source CTA][utterance][hi, lo][40 units]; 80-byte rows keep
// ldmatrix free of bank conflicts).  An instruction whose lanes address 16 different peers costs twice as
// much: all-to-all step with one utterance 835 cycles scattered, 560 so; eight utterances 3272, 1692.
// What bounds a round: three exchanges (about 400 cycles from the store to the wait's end each), the mma of
// the prediction and joint rows (240 and 420 cycles at 8 per instruction and scheduler), the table row's trip to L2
// (300) and the instructions in between.  us per round, scattered sends and one control warp per utterance against
// this form: one fp16 layer 3.24 -> 2.83 (1 utterance), 4.95 -> 3.97 (4), 7.00 -> 6.24 (8); two layers, long-request
// numerics 4.99 -> 4.37 (1), 18.3 -> 17.3 (8).
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
constexpr int control_warps(int utts) { return utts <= 2 ? 5 : utts; }
constexpr int cl_threads(int utts) { return kMatrixThreads + 32 * control_warps(utts); }
constexpr uint32_t kTmemColumns = 512;

// named barriers (0 is __syncthreads)
enum : int { BAR_CONTROL = 1, BAR_PRED = 2, BAR_GO = 3, BAR_LAYER1 = 4, BAR_JOINT = 5, BAR_GATES = 6 };
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

// Shared memory of one CTA; NU = utterances it is sized for (1, 2, 4 or 8).
template <int Layers, bool Cache, int NU>
struct CSmem {
    // activations that multiply weight matrices: fp16 [source CTA][utterance][hi, lo][40 units], Cache: one row
    // of INT8 codes per utterance.
    static constexpr int kSliceBytes = NU * 2 * kClUnits * 2;          // one source CTA's slice
    static constexpr int kCodePitch = 656;
    using Act = uint8_t[Cache ? NU * kCodePitch : kCl * kSliceBytes];
    // The recurrent product runs behind the joint: a peer may then be a round ahead, so the hidden state that
    // it reads is double-buffered.
    static constexpr bool kLate = NU <= 2;
    static constexpr bool kJointResident = Cache || Layers == 1 || NU <= 4;
    // K pairs of the streamed matrix that fit beside the rest (see weight placement below)
    static constexpr int kSmemPairs = Layers == 1 ? 0 : Cache ? (NU <= 4 ? 3 : 2) : (NU == 4 ? 1 : 2);
    static constexpr int kPairBytes = kMatrixWarps * (Cache ? 1 : 2) * 1024;
    static constexpr int kJointBytes = !kJointResident ? 0 : Cache ? kClJoint * 1280 : 10 * 2 * (4 * 1024 + 128);
    static constexpr int kGateParts = Cache ? 2 : 4;
    // Partial sums of the prediction and joint rows.  Up to two utterances: the parts of one row side by side
    // (16-byte loads); more: rows side by side (the stores of four utterances would collide).
    static constexpr bool kRowMajor = NU <= 2;
    static constexpr int kPredFloats = PredSplit::KG * NU * kPredPitch;
    static constexpr int kJointFloats = kRowMajor ? NU * kJointPitch * 12 : JointSplit::KG * NU * kJointPitch;
    static __device__ __forceinline__ int pred_index(int kg, int u, int row) {
        return kRowMajor ? (u * kPredPitch + row) * PredSplit::KG + kg : (kg * NU + u) * kPredPitch + row;
    }
    static __device__ __forceinline__ int joint_index(int kg, int u, int row) {
        return kRowMajor ? (u * kJointPitch + row) * 12 + kg : (kg * NU + u) * kJointPitch + row;
    }

    alignas(16) uint8_t joint[kJointBytes > 0 ? kJointBytes : 16];
    alignas(16) uint8_t pairs[kSmemPairs > 0 ? kSmemPairs * kPairBytes : 16];
    alignas(16) Act h0[kLate && Layers == 1 ? 2 : 1];     // hidden state of layer 0, written by all CTAs
    alignas(16) Act h1[Layers == 2 ? (kLate ? 2 : 1) : 1];             // of layer 1
    alignas(16) float hf[Cache ? NU : 1][Cache ? kHidden : 4];         // Cache: fp32 state of the top layer
    alignas(16) uint8_t ax[Cache ? NU * kHidden * 4 : kCl * kSliceBytes];      // joint input: hi / lo or fp32
    alignas(16) float gates0[kGateParts * NU * kGatePitch];            // partial sums of the recurrent product
    alignas(16) float gates1[Layers == 2 ? 4 * NU * kGatePitch : 4];   // layer 1: parts 0, 1 input, 2, 3 recurrent
    alignas(16) float part[Cache ? NU * kJointPitch : (kPredFloats > kJointFloats ? kPredFloats : kJointFloats)];
    alignas(16) uint8_t stage_act[NU][2][kClUnits * 2];   // outgoing slice: hi / lo halves, Cache: codes (first 40 bytes)
    alignas(16) float stage_f[NU][kClUnits];              // outgoing fp32 slice (Cache: hidden state / joint input)
    float pred[Cache ? NU : 1][kClUnits];                 // Cache: this CTA's prediction slice, finished by the matrix warps
    float bias0[4 * kClUnits], bias1[4 * kClUnits];       // [unit][gate]
    float pred_bias[kClUnits], joint_bias[kJointPitch];
    float cache_mul[3];                                   // scale / 127 of w_hh[0], w_hh[1], w_ih[1]
    unsigned long long keys[2][NU][3 * kCl];              // [round parity][utterance][source CTA, third of its rows]
    int dur[2][NU];                                       // [round parity][utterance] winning duration
    uint64_t hbar0, hbar1, abar, kbar[2];           // exchange mbarriers (count 1 + transaction bytes)
    uint32_t tmem_base;
    alignas(8) unsigned char need[8], live[8];            // of a round: 1 = steps, lives (read as 64-bit words)
    int stop;                                             // a wait gave up in an earlier round
    int abort;
#ifdef PK100_DEC_PROFILE
    long long prof[16], last_stamp;
#endif
};

constexpr size_t kCtaSmem = 227 * 1024;
template <int NU>
constexpr bool cl_smem_fits() {
    return sizeof(CSmem<1, false, NU>) <= kCtaSmem && sizeof(CSmem<2, false, NU>) <= kCtaSmem &&
           sizeof(CSmem<1, true, NU>) <= kCtaSmem && sizeof(CSmem<2, true, NU>) <= kCtaSmem;
}
static_assert(cl_smem_fits<1>() && cl_smem_fits<2>() && cl_smem_fits<4>() && cl_smem_fits<8>(), "fits one CTA's shared memory");

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
// of the pair (the rows of block nb are nb * kActBlock bytes on).
constexpr int kActBlock = 8 * 2 * kClUnits;
template <bool Codes, int NT, int NB, typename Load>
__device__ __forceinline__ void pair_mma(typename AccT<Codes>::type (&acc)[NT][NB][4], const uint8_t* act, int tiles, Load&& load) {
    unsigned b[NB][4];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) dec_ldmatrix_x4(b[nb], act + nb * kActBlock);
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

// Partial sums of one tile: put(utterance, row, value).  fp16: column pair t of a block is (hi, lo) of
// utterance 4 * nb + t; codes: column = utterance.  Columns behind NU are copies of others.
template <bool Codes, int NB, int NU, typename Put>
__device__ __forceinline__ void store_part(const typename AccT<Codes>::type (&acc)[NB][4], int row0, int rows, int lane, Put&& put) {
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
                    if (2 * t + e < NU) put(2 * t + e, row, static_cast<float>(acc[nb][2 * half + e]));
            } else {
                if (4 * nb + t < NU) put(4 * nb + t, row, acc[nb][2 * half] + acc[nb][2 * half + 1]);
            }
        }
}

#ifdef PK100_DEC_PROFILE
#define CL_STAMP(i) do { if (tid == kMatrixThreads) { const long long now__ = clock64(); sm.prof[i] += now__ - sm.last_stamp; sm.last_stamp = now__; } } while (0)
#else
#define CL_STAMP(i) do { } while (0)
#endif

// Bounded wait; the clock that bounds it is only read after some polls.
__device__ __forceinline__ void cl_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
        if (mbar_try_wait(bar, parity)) return;
    mbar_wait_bounded(bar, parity, abort_flag);
}
// Loads that stay in flight: the destination keeps its value where `take` is false, without a move that would
// wait for the load.
__device__ __forceinline__ void load_if(float& v, const float* p, bool take) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.global.nc.f32 %0, [%1];\n\t}" : "+f"(v) : "l"(p), "r"(static_cast<unsigned>(take)));
}
__device__ __forceinline__ void load_if(unsigned& v, const __half* p, bool take) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.global.nc.u16 %0, [%1];\n\t}" : "+r"(v) : "l"(p), "r"(static_cast<unsigned>(take)));
}
// eight flag bytes -> eight bits
__device__ __forceinline__ unsigned flag_bits(const unsigned char* bytes) {
    return static_cast<unsigned>((*reinterpret_cast<const volatile unsigned long long*>(bytes) * 0x0102040810204080ull) >> 56);
}

struct ClWeights {               // packed slices (see tdt_pack_kernel) and the input table
    const uint4 *lstm, *pred, *joint, *lstm1_in, *lstm1_rec;
    const float* xtab;
};

template <int Layers, bool Cache, int NU>
__global__ void __launch_bounds__(cl_threads(NU), 1)
tdt_cluster_kernel(const DecParams p, const ClWeights w) {
    using Smem = CSmem<Layers, Cache, NU>;
    constexpr int NB = Cache || NU < 4 ? 1 : NU / 4;       // blocks of 8 B columns
    constexpr int kControlWarps = control_warps(NU), kControlThreads = 32 * kControlWarps, kClThreads = cl_threads(NU);
    constexpr bool kLate = Smem::kLate;
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
    const int U = NU == 1 ? 1 : p.utts;
    volatile int* abort_flag = &sm.abort;
    volatile int* stop_flag = &sm.stop;

    // ---- set-up: cleared state, biases, barriers
    for (int i = tid; i < static_cast<int>(sizeof(Smem) / 16); i += kClThreads) reinterpret_cast<uint4*>(cs_raw)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    if (tid < 4 * kClUnits) {
        const int row = (tid % 4) * kHidden + r * kClUnits + tid / 4;
        sm.bias0[tid] = p.b_ih[0][row] + p.b_hh[0][row];
        if constexpr (Layers == 2) sm.bias1[tid] = p.b_ih[1][row] + p.b_hh[1][row];
    }
    if (tid < kClUnits) sm.pred_bias[tid] = p.b_pred[r * kClUnits + tid];
    if (tid < 3) sm.cache_mul[tid] = (Cache && (tid == 0 || Layers == 2)) ? cache_mul(cache_scale(p.cache_absmax, tid)) : 0.0f;
    if (tid < kClJoint && r * kClJoint + tid < kJointRows) sm.joint_bias[tid] = p.b_joint[r * kClJoint + tid];
    if (tid < U) sm.need[tid] = sm.live[tid] = p.frames[tid] > 0 && in_window(p, tid) ? 1 : 0;
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

    // Joint sums -> keys.  Publisher id = 3 * utterance + third: it reduces a third of this CTA's joint rows of
    // its utterance to their best key and sends that to every CTA; the owner of the five duration rows sends the
    // first strict maximum among them.  Ids go to the control warps first, then to matrix warps.
    unsigned round = 0;
    auto publish_keys = [&](int id, unsigned live) {
        const int par = static_cast<int>(round & 1u);
        const int u = id / 3, third = id % 3;
        if (((live >> u) & 1u) == 0u) return;
        const int n = third * 32 + lane, row = r * kClJoint + n;
        const bool owned = n < kClJoint && row < kJointRows;
        float total = 0.0f;
        if (owned) {
            if constexpr (Cache) {
                total = sm.part[u * kJointPitch + n];          // finished score of the fp32 joint
            } else {
                float part[JointSplit::KG];
                if constexpr (Smem::kRowMajor) {
                    const float* at = &sm.part[Smem::joint_index(0, u, n)];
                    const float4 a = *reinterpret_cast<const float4*>(at), b = *reinterpret_cast<const float4*>(at + 4);
                    const float2 c = *reinterpret_cast<const float2*>(at + 8);
                    part[0] = a.x; part[1] = a.y; part[2] = a.z; part[3] = a.w; part[4] = b.x;
                    part[5] = b.y; part[6] = b.z; part[7] = b.w; part[8] = c.x; part[9] = c.y;
                } else {
#pragma unroll
                    for (int kg = 0; kg < JointSplit::KG; ++kg) part[kg] = sm.part[Smem::joint_index(kg, u, n)];
                }
                total = sm.joint_bias[n];
#pragma unroll
                for (int kg = 0; kg < JointSplit::KG; ++kg) total += part[kg];
            }
        }
        const uint32_t peer = static_cast<uint32_t>(lane % kCl);
        const uint32_t bar = map_to_cta(smem_u32(&sm.kbar[par]), peer);
        unsigned ordered = 0;                                  // order-preserving bits; NaN and foreign rows never win
        if (owned && row < kTokenOutputs && total == total) {
            const unsigned bits = __float_as_uint(total == 0.0f ? 0.0f : total);          // (canonical -0)
            ordered = (bits & 0x80000000u) ? ~bits : (bits ^ 0x80000000u);
        }
        const unsigned top = __reduce_max_sync(0xffffffffu, ordered);
        // ties to the lower row; a third whose rows all produced NaN still publishes a (losing) key
        const unsigned first = __reduce_max_sync(0xffffffffu, ordered == top && top != 0u ? 2047u - static_cast<unsigned>(row) : 0u);
        const unsigned low = ((top != 0u ? first : 2047u - kTokenOutputs) << 21) | 1u;
        if (lane < kCl)
            st_async_b64(map_to_cta(smem_u32(&sm.keys[par][u][r * 3 + third]), peer), (static_cast<unsigned long long>(top) << 32) | low, bar);
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
            if (lane < kCl) st_async_b32(map_to_cta(smem_u32(&sm.dur[par][u]), peer), static_cast<unsigned>(duration), bar);
        }
    };

    uint32_t hphase = 0;                   // parity of the rounds with an LSTM step
    if (matrix) {
        // ============================================================ matrix warps
        const uint32_t tm = sm.tmem_base + (static_cast<uint32_t>((warp % 4) * 32) << 16) + static_cast<uint32_t>((warp / 4) * kCols);
        const uint4* lstm = w.lstm + static_cast<size_t>(r) * Gates0::kPerCta;
        [[maybe_unused]] const uint4* in1 = w.lstm1_in + static_cast<size_t>(r) * Gates1::kPerCta;
        [[maybe_unused]] const uint4* rec1 = w.lstm1_rec + static_cast<size_t>(r) * Gates1::kPerCta;
        const int kg0 = warp / Gates0::NG, tile0 = (warp % Gates0::NG) * Gates0::NT;
        [[maybe_unused]] const int kg1 = warp / Gates1::NG, tile1 = warp % Gates1::NG;
        // joint: the warps with three tiles and those with two alternate over the SM's four schedulers
        [[maybe_unused]] const int jkg = warp / JointSplit::NG, jng = (warp ^ (warp >> 2)) & 1;
        static_assert(JointSplit::NG == 2, "both row groups of a k-group in neighbouring warps");
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
            for (int j = 0; j < 2; ++j) fill(src + frag_index<JointSplit>(jkg, 0, jng * 2 + j, 0, lane), kCols0 + j * 8);
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
        // This lane's ldmatrix address of k-pair `pair`: row lane % 8 of the B columns, 16 bytes of K number
        // 4 * pair + lane / 8.  Rows behind the last utterance repeat the first ones.
        const int lane_row = (lane % 8) & ((Cache ? NU : NU < 4 ? 2 * NU : 8) - 1);
        auto act_at = [&](const uint8_t* act, int pair) {
            const int q = 4 * pair + lane / 8;
            if constexpr (Cache) return act + lane_row * Smem::kCodePitch + q * 16;
            const int src = (q * 205) >> 10;                       // q / 5 (five 16-byte pieces per source CTA), q < 80
            return act + src * (Smem::kSliceBytes - 2 * kClUnits) + q * 16 + lane_row * (2 * kClUnits);
        };

        // part[kg] of one gate product, for the utterances in `who` (double-buffered hidden states: the others' rows
        // are a step old and their sums stand).  Source of k-pair kp: tensor memory at column base + 8 * NT * kp for
        // kp < in_tmem, then `in_smem` pairs from shared memory, then the packed copy in L2; the next pair's
        // fragments are fetched under the mmas of the current one.
        auto gate_product = [&](auto split, const uint4* packed, const uint8_t* act, float* part, int kg, int tile,
                                int part_kg, auto tmem_pairs, auto smem_pairs, uint32_t col, unsigned who) {
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
#pragma unroll
            for (int kp = 0; kp < S::KP; ++kp) {
                if (kp + 1 < S::KP) fetch(kp + 1, f[(kp + 1) & 1]);
                pair_mma<Cache, S::NT, NB>(acc, act_at(act, kg * S::KP + kp), S::NT, [&](int j, int step) {
                    const uint32_t* v = &f[kp & 1][j * 8 + step * 4];
                    return make_uint4(v[0], v[1], v[2], v[3]);
                });
                if (kp + 1 < kTm) tmem_ld_wait();
            }
#pragma unroll
            for (int j = 0; j < S::NT; ++j)
                store_part<Cache, NB, NU>(acc[j], (tile + j) * 16, 160, lane,
                                          [&](int u, int row, float v) {
                                              if (!kLate || ((who >> u) & 1u) != 0u) part[(part_kg * NU + u) * kGatePitch + row] = v;
                                          });
        };
        using std::integral_constant;
        auto recurrent0 = [&](const uint8_t* h, unsigned who) {
            gate_product(Gates0{}, lstm, h, sm.gates0, kg0, tile0, kg0, integral_constant<int, kCols0 / (8 * Gates0::NT)>{},
                         integral_constant<int, Layers == 2 && !Cache ? Smem::kSmemPairs : 0>{}, 0, who);
        };
        // the recurrent product of the NEXT step of the top layer
        auto recurrent_top = [&](const uint8_t* h, unsigned who) {
            if constexpr (Layers == 2)
                gate_product(Gates1{}, rec1, h, sm.gates1, kg1, tile1, 2 + kg1, integral_constant<int, kCols2 / 8>{},
                             integral_constant<int, Cache ? Smem::kSmemPairs : 0>{}, kCols0 + kCols1, who);
            else
                recurrent0(h, who);
        };

        while (true) {
            bar_sync(BAR_GO, kClThreads);
            const unsigned need = flag_bits(sm.need), live = flag_bits(sm.live);
            if (live == 0u || *stop_flag != 0) break;
            const uint8_t* top = Layers == 2 ? sm.h1[kLate ? hphase : 0] : sm.h0[kLate ? hphase : 0];
            if (need != 0u) {
                cl_wait(&sm.hbar0, hphase, abort_flag);
                if constexpr (Layers == 2) {
                    gate_product(Gates1{}, in1, sm.h0[0], sm.gates1, kg1, tile1, kg1, integral_constant<int, kCols1 / 8>{},
                                 integral_constant<int, 0>{}, kCols0, 255u);
                    bar_arrive(BAR_LAYER1, kClThreads);
                    recurrent0(sm.h0[0], 255u);                  // under the second layer's cell and exchange
                    cl_wait(&sm.hbar1, hphase, abort_flag);
                }
                if constexpr (Cache) {
                    // fp32 in the reference's summation order (decoder.cu:672-684): lane l takes elements
                    // 2l + 64w as one fma chain that starts from the bias in lane 0, then a shuffle tree
                    for (int u = 0; u < U; ++u) {
                        if (((need >> u) & 1u) == 0u) continue;
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
                    pair_mma<false, 3, NB>(acc, act_at(top, warp), 3, [&](int j, int step) {
                        return j < 2 ? make_uint4(predw[j * 8 + step * 4], predw[j * 8 + step * 4 + 1], predw[j * 8 + step * 4 + 2], predw[j * 8 + step * 4 + 3])
                                     : make_uint4(predw[16 + step * 2], 0u, predw[17 + step * 2], 0u);
                    });
#pragma unroll
                    for (int j = 0; j < 3; ++j)
                        store_part<false, NB, NU>(acc[j], j * 16, kClUnits, lane,
                                                  [&](int u, int row, float v) { sm.part[Smem::pred_index(warp, u, row)] = v; });
                }
                bar_arrive(BAR_PRED, kClThreads);
                if constexpr (!kLate) recurrent_top(top, need);
            }
            // the joint rows' fragments do not depend on the activations: the first are requested before the wait
            // (where the registers allow it)
            constexpr int kAhead = Cache || (Layers == 2 && NU <= 4) ? 0 : 1;
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
            cl_wait(&sm.abar, round & 1u, abort_flag);
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
                    if (((live >> u) & 1u) == 0u) continue;
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
                    pair_mma<false, 3, NB>(acc, act_at(sm.ax, jkg * JointSplit::KP + kp), jng == 0 ? 3 : 2, [&](int j, int step) {
                        const int i = (j * 2 + step) * 4;
                        return kColsJ > 0 && kp == 0 && j < 2 ? make_uint4(jt[i], jt[i + 1], jt[i + 2], jt[i + 3]) : jf[kp][j][step];
                    });
                }
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    if (j < 2 || jng == 0)
                        store_part<false, NB, NU>(acc[j], (j < 2 ? jng * 2 + j : 4) * 16, kClJoint, lane,
                                                  [&](int u, int row, float v) { sm.part[Smem::joint_index(jkg, u, row)] = v; });
            }
            if (kControlWarps + warp < 3 * U) {
                bar_sync(BAR_JOINT, kClThreads);
                publish_keys(kControlWarps + warp, live);
            } else {
                bar_arrive(BAR_JOINT, kClThreads);
            }
            if (need != 0u) {
                if constexpr (kLate) {
                    recurrent_top(top, need);
                    if constexpr (Layers == 1) bar_arrive(BAR_GATES, kClThreads);
                }
                hphase ^= 1u;
            }
            round += 1;
        }
    } else {
        // ============================================================ control warps
        const int ct = tid - kMatrixThreads, cw = ct / 32;
        // sends: 16-byte piece i % kPieces of the outgoing slice (utterance piece / 10) to peer i / kPieces, counted
        // from another peer in every CTA
        constexpr int kPieces = 10 * NU;
        const uint32_t local_base = smem_u32(cs_raw);
        uint32_t peer_base[NU <= 2 ? NU : 1];              // the same peers in every send
        if constexpr (NU <= 2) {
#pragma unroll
            for (int j = 0; j < NU; ++j) peer_base[j] = map_to_cta(local_base, static_cast<uint32_t>((ct + j * kControlThreads) / kPieces + r) % kCl);
        }
        auto to_peers = [&](const uint64_t* bar_local, unsigned who, auto&& store) {    // store(piece, base, barrier)
            const uint32_t bar = smem_u32(bar_local) - local_base;
#pragma unroll
            for (int j = 0; j < kCl * kPieces / kControlThreads; ++j) {
                const int i = ct + j * kControlThreads, piece = i % kPieces;
                if (((who >> (piece / 10)) & 1u) == 0u) continue;
                const uint32_t base = NU <= 2 ? peer_base[j < NU ? j : 0] : map_to_cta(local_base, static_cast<uint32_t>(i / kPieces + r) % kCl);
                store(piece, base, base + bar);
            }
        };
        static_assert(kCl * kPieces % kControlThreads == 0, "whole passes of sends");
        // `who` = utterances that send
        auto send_halves = [&](const uint8_t* act, const uint64_t* bar, unsigned who) {
            const uint32_t dst = smem_u32(act) - local_base + r * Smem::kSliceBytes;
            to_peers(bar, who, [&](int piece, uint32_t base, uint32_t b) {
                st_async_v4(base + dst + piece * 16, reinterpret_cast<const uint4*>(sm.stage_act)[piece], b);
            });
        };
        auto send_floats = [&](const void* rows, const uint64_t* bar, unsigned who) {
            const uint32_t dst = smem_u32(rows) - local_base + r * kClUnits * 4;
            to_peers(bar, who, [&](int piece, uint32_t base, uint32_t b) {
                st_async_v4(base + dst + (piece / 10) * kHidden * 4 + (piece % 10) * 16, reinterpret_cast<const uint4*>(sm.stage_f)[piece], b);
            });
        };
        auto send_codes = [&](const uint8_t* act, const uint64_t* bar, unsigned who) {
            const uint32_t dst = smem_u32(act) - local_base + r * kClUnits;
            if constexpr (NU <= 2) {
                to_peers(bar, who, [&](int piece, uint32_t base, uint32_t b) {
                    const int u = piece / 10, c = piece % 10;
                    if (c < 5)
                        st_async_b64(base + dst + u * Smem::kCodePitch + c * 8, *reinterpret_cast<const unsigned long long*>(&sm.stage_act[u][0][c * 8]), b);
                });
            } else {                                       // 40-byte rows: scattered over the peers is the faster form
                const int c = ct / kCl;
                if (c >= 5) return;
                const uint32_t base = map_to_cta(local_base, static_cast<uint32_t>(ct % kCl)), b = base + smem_u32(bar) - local_base;
                for (int u = 0; u < U; ++u)
                    if (((who >> u) & 1u) != 0u)
                        st_async_b64(base + dst + u * Smem::kCodePitch + c * 8, *reinterpret_cast<const unsigned long long*>(&sm.stage_act[u][0][c * 8]), b);
            }
        };
        // Cell.  Up to two utterances: lane = (unit cw * 8 + lane / 4, gate lane % 4), gate row `ct` of the CTA's
        // slice, task i = utterance i.  More: task i = units lane and lane + 32 of utterance cw, all gates in the lane.
        constexpr int kCells = NU == 1 ? 1 : 2, kGatesHere = NU <= 2 ? 1 : 4;
        const int gate = lane % 4;
        const float* xrow = w.xtab + r * kClUnits + (NU <= 2 ? gate * kHidden + cw * 8 + lane / 4 : lane);
        float cell0[kCells] = {}, xg[kCells][kGatesHere] = {};
        [[maybe_unused]] float cell1[Layers == 2 ? kCells : 1] = {};
        auto for_cells = [&](auto&& f) {                   // f(task, utterance, first gate row)
#pragma unroll
            for (int i = 0; i < kCells; ++i) {
                if constexpr (NU <= 2) f(i, i, ct);
                else if (lane + 32 * i < kClUnits) f(i, cw, (lane + 32 * i) * 4);
            }
        };
        // joint input: pass i is (utterance x_u, unit x_unit(i))
        constexpr int kPasses = NU <= 2 ? 1 : 2;
        const int x_u = NU <= 2 ? (lane / 8) % NU : cw;
        auto x_unit = [&](int i) { return NU <= 2 ? cw * 8 + lane % 8 : lane + 32 * i; };
        auto x_lane = [&](int i) { return NU <= 2 ? lane < 8 * NU : i == 0 || lane < kClUnits - 32; };
        float pred[kPasses] = {};
        unsigned enc[kPasses] = {};                                        // fp16 bits
        // decision: this lane holds the state of utterance `my`
        const int my = NU <= 2 ? lane % NU : cw;
        const bool owner = NU <= 2 ? cw == 0 && lane < NU : lane == 0;
        unsigned need = flag_bits(sm.need), live = flag_bits(sm.live);      // bit masks, the same in all control threads
        const int total_frames = ((live >> my) & 1u) != 0u ? min(p.frames[my], p.seg_stride) : 0;   // never past the utterance's block
        int frame = 0, symbols = 0, count = 0;
        bool alive = total_frames > 0, steps = alive;
        int token = kBlank, duration = 0;
        bool emits = false, no_score = false;
        const __half* enc_base = p.enc_proj + static_cast<size_t>(x_u) * p.seg_stride * kHidden + r * kClUnits + x_unit(0);
        auto fetch_enc = [&](int f, bool take) {           // frame of x_u
#pragma unroll
            for (int i = 0; i < kPasses; ++i)
                load_if(enc[i], enc_base + static_cast<size_t>(f) * kHidden + 32 * i, take && x_lane(i));
        };
        fetch_enc(0, ((live >> x_u) & 1u) != 0u);
        // the emission of the round before (held back until this round's sends are out)
        auto flush_token = [&]() {
            if (r == 0 && owner) {
                if (no_score && sm.abort == 0 && p.status != nullptr) atomicOr(p.status, 4);
                if (emits && count <= p.max_tokens) {
                    p.tokens[static_cast<size_t>(my) * p.max_tokens + count - 1] = token;
                    if (p.durations_out != nullptr) p.durations_out[static_cast<size_t>(my) * p.max_tokens + count - 1] = duration;
                }
            }
            emits = no_score = false;
        };
        // One cell step of a unit of utterance u from its gate sums (one of them where four lanes share the unit);
        // stages h
        auto cell_update = [&](const float (&gsum)[kGatesHere], float& cstate, int u, int row, bool commit) {
            const int unit = row / 4;
            float ig, fg, gg, og;
            if constexpr (NU <= 2) {
                float a;
                if constexpr (Cache) {
                    a = gate == 2 ? ref_tanh(gsum[0]) : ref_sigmoid(gsum[0]);
                } else {
                    const float s = fast_sigmoid(gate == 2 ? 2.0f * gsum[0] : gsum[0]);
                    a = gate == 2 ? 2.0f * s - 1.0f : s;           // tanh(x) = 2 sigmoid(2x) - 1
                }
                const int unit0 = lane & ~3;
                ig = __shfl_sync(0xffffffffu, a, unit0); fg = __shfl_sync(0xffffffffu, a, unit0 + 1);
                gg = __shfl_sync(0xffffffffu, a, unit0 + 2); og = __shfl_sync(0xffffffffu, a, unit0 + 3);
            } else if constexpr (Cache) {
                ig = ref_sigmoid(gsum[0]); fg = ref_sigmoid(gsum[1]); gg = ref_tanh(gsum[2]); og = ref_sigmoid(gsum[3]);
            } else {
                ig = fast_sigmoid(gsum[0]); fg = fast_sigmoid(gsum[1]); gg = fast_tanh(gsum[2]); og = fast_sigmoid(gsum[3]);
            }
            if constexpr (Cache) {
                // the reference's approximations: h is rounded to 8 bits next, and a code that flips moves a gate
                const float cell = fmaf(ig, gg, __fmul_rn(fg, cstate));
                if (commit) cstate = cell;
                const float h = __fmul_rn(og, ref_tanh(cell));
                if (NU > 2 || gate == 0) sm.stage_act[u][0][unit] = static_cast<uint8_t>(quantize_i8(h * 127.0f));
                if (NU > 2 || gate == 1) sm.stage_f[u][unit] = h;
            } else {
                const float cell = fg * cstate + ig * gg;
                if (commit) cstate = cell;
                const float h = og * fast_tanh(cell);
                const __half hi = __float2half_rn(h), lo = __float2half_rn(h - __half2float(hi));
                if (NU > 2 || gate == 0) reinterpret_cast<__half*>(sm.stage_act[u][0])[unit] = hi;
                if (NU > 2 || gate == 1) reinterpret_cast<__half*>(sm.stage_act[u][1])[unit] = lo;
            }
        };
        // gate sums of a task from `Parts` partial sums
        auto gate_parts = [&](const float* gates, int k, int u, int row, float (&v)[kGatesHere]) {
            const float* at = gates + (k * NU + u) * kGatePitch + row;
            if constexpr (NU <= 2) {
                v[0] = *at;
            } else {
                const float4 f = *reinterpret_cast<const float4*>(at);
                v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
            }
        };
        // bytes one utterance contributes to the exchanges
        constexpr uint32_t kTopTx = Cache ? kHidden + kHidden * 4 : kHidden * 4, kLowTx = Cache ? kHidden : kHidden * 4;
        [[maybe_unused]] bool gates_pending = false;       // a recurrent product behind the joint is on its way
#ifdef PK100_DEC_PROFILE
        if (ct == 0) sm.last_stamp = clock64();
#endif
        while (true) {
            __syncwarp();
            bar_arrive(BAR_GO, kClThreads);                // this round's flags are published
            if (NU <= 2 && live == 0u) break;
            const int par = static_cast<int>(round & 1u);
            const int hbuf = kLate ? static_cast<int>(hphase) : 0;
            if (NU > 2 || need != 0u) {
                if constexpr (kLate && Layers == 1) {
                    if (gates_pending) bar_sync(BAR_GATES, kClThreads);
                    gates_pending = false;
                }
                CL_STAMP(0);
                // ---- cell of layer 0: table row + h . w_hh^T + bias
                if (NU <= 2 || steps) {
                    for_cells([&](int i, int u, int row) {
                        float gsum[kGatesHere], v[Smem::kGateParts][kGatesHere];
#pragma unroll
                        for (int k = 0; k < Smem::kGateParts; ++k) gate_parts(sm.gates0, k, u, row, v[k]);
#pragma unroll
                        for (int g = 0; g < kGatesHere; ++g) {
                            if constexpr (Cache) {
                                // the scaled recurrent sum is rounded BEFORE the bias is added, as in the reference
                                // (decoder.cu:113, :626-640): a fused multiply-add here parts from the reference
                                // kernel's tokens after a few hundred steps
                                gsum[g] = __fadd_rn(__fadd_rn(__fmul_rn(v[0][g] + v[1][g], sm.cache_mul[0]), sm.bias0[row + g]), xg[i][g]);
                            } else {
                                gsum[g] = sm.bias0[row + g] + xg[i][g];
#pragma unroll
                                for (int k = 0; k < Smem::kGateParts; ++k) gsum[g] += v[k][g];
                            }
                        }
                        cell_update(gsum, cell0[i], u, row, NU > 2 || ((need >> u) & 1u) != 0u);
                    });
                }
                __syncwarp();
                bar_sync(BAR_CONTROL, kControlThreads);
                CL_STAMP(1);
                if constexpr (NU > 2) {
                    need = flag_bits(sm.need);
                    live = flag_bits(sm.live);
                }
                if ((NU > 2 && live == 0u) || *stop_flag != 0) break;      // (as the matrix warps)
            }
            if (need != 0u) {
                gates_pending = true;
                if constexpr (Cache) {
                    send_codes(sm.h0[Layers == 1 ? hbuf : 0], &sm.hbar0, need);
                    if constexpr (Layers == 1) send_floats(&sm.hf[0][0], &sm.hbar0, need);
                } else {
                    send_halves(sm.h0[Layers == 1 ? hbuf : 0], &sm.hbar0, need);
                }
                if (ct == kControlThreads - 1) {           // (transaction counts may trail the transactions)
                    const uint32_t needs = static_cast<uint32_t>(__popc(need));
                    mbar_arrive_expect_tx(&sm.hbar0, needs * (Layers == 1 ? kTopTx : kLowTx));
                    if (Layers == 2) mbar_arrive_expect_tx(&sm.hbar1, needs * kTopTx);
                }
                __syncwarp();
                CL_STAMP(2);
                if constexpr (Layers == 2) {
                    bar_sync(BAR_LAYER1, kClThreads);
                    CL_STAMP(3);
                    // ---- cell of layer 1: [fresh h of layer 0 | own h] . [w_ih | w_hh]^T + bias
                    if (NU <= 2 || steps) {
                        for_cells([&](int i, int u, int row) {
                            float gsum[kGatesHere], v[4][kGatesHere];
#pragma unroll
                            for (int k = 0; k < 4; ++k) gate_parts(sm.gates1, k, u, row, v[k]);
#pragma unroll
                            for (int g = 0; g < kGatesHere; ++g) {
                                // Cache: rounded recurrent product first, the input product fused onto it, bias last
                                // (decoder.cu:113, :655-663)
                                if constexpr (Cache)
                                    gsum[g] = __fadd_rn(fmaf(v[0][g] + v[1][g], sm.cache_mul[2], __fmul_rn(v[2][g] + v[3][g], sm.cache_mul[1])), sm.bias1[row + g]);
                                else
                                    gsum[g] = (((sm.bias1[row + g] + v[0][g]) + v[1][g]) + v[2][g]) + v[3][g];
                            }
                            cell_update(gsum, cell1[i], u, row, NU > 2 || ((need >> u) & 1u) != 0u);
                        });
                    }
                    __syncwarp();
                    bar_sync(BAR_CONTROL, kControlThreads);
                    CL_STAMP(4);
                    if constexpr (Cache) {
                        send_codes(sm.h1[hbuf], &sm.hbar1, need);
                        send_floats(&sm.hf[0][0], &sm.hbar1, need);
                    } else {
                        send_halves(sm.h1[hbuf], &sm.hbar1, need);
                    }
                    __syncwarp();
                }
                hphase ^= 1u;
                bar_sync(BAR_PRED, kClThreads);
            }
            CL_STAMP(5);
            // ---- prediction slice where the state moved; this CTA's 40 columns of the joint input relu(enc + pred)
            const bool x_steps = ((need >> x_u) & 1u) != 0u;
#pragma unroll
            for (int i = 0; i < kPasses; ++i) {
                if (!x_lane(i) || x_u >= U) continue;
                const int unit = x_unit(i);
                if (x_steps) {
                    if constexpr (Cache) {
                        pred[i] = sm.pred[x_u][unit];
                    } else {
                        float part[PredSplit::KG];
                        if constexpr (Smem::kRowMajor) {
#pragma unroll
                            for (int kg = 0; kg < PredSplit::KG; kg += 4) {
                                const float4 v = *reinterpret_cast<const float4*>(&sm.part[Smem::pred_index(kg, x_u, unit)]);
                                part[kg] = v.x; part[kg + 1] = v.y; part[kg + 2] = v.z; part[kg + 3] = v.w;
                            }
                        } else {
#pragma unroll
                            for (int kg = 0; kg < PredSplit::KG; ++kg) part[kg] = sm.part[Smem::pred_index(kg, x_u, unit)];
                        }
                        pred[i] = sm.pred_bias[unit];
#pragma unroll
                        for (int kg = 0; kg < PredSplit::KG; ++kg) pred[i] += part[kg];
                    }
                }
                const float x = fmaxf(__half2float(__ushort_as_half(static_cast<unsigned short>(enc[i]))) + pred[i], 0.0f);
                if constexpr (Cache) {
                    sm.stage_f[x_u][unit] = x;
                } else {
                    const __half hi = __float2half_rn(x);
                    reinterpret_cast<__half*>(sm.stage_act[x_u][0])[unit] = hi;
                    reinterpret_cast<__half*>(sm.stage_act[x_u][1])[unit] = __float2half_rn(x - __half2float(hi));
                }
            }
            __syncwarp();
            bar_sync(BAR_CONTROL, kControlThreads);
            CL_STAMP(6);
            if (NU <= 2 && need == 0u && *stop_flag != 0) break;
            if constexpr (Cache) send_floats(sm.ax, &sm.abar, live);
            else send_halves(sm.ax, &sm.abar, live);
            if (ct == kControlThreads - 1) {
                const uint32_t lives = static_cast<uint32_t>(__popc(live));
                mbar_arrive_expect_tx(&sm.abar, lives * kHidden * 4);
                mbar_arrive_expect_tx(&sm.kbar[par], lives * (3 * kCl * 8 + 4));
            }
            flush_token();
            __syncwarp();
            CL_STAMP(7);
            bar_sync(BAR_JOINT, kClThreads);               // joint sums are complete
            CL_STAMP(8);
            if (cw < 3 * U) publish_keys(cw, live);
            CL_STAMP(9);
            cl_wait(&sm.kbar[par], (round >> 1) & 1u, abort_flag);
            CL_STAMP(10);

            // ---- decision (replicated in every CTA; up to two utterances: in every control warp)
            const bool was_live = ((live >> my) & 1u) != 0u;
            if (NU <= 2 || was_live) {
#pragma unroll
                for (int v = 0; v < (NU <= 2 ? NU : 1); ++v) {
                    const int u = NU <= 2 ? v : cw;
                    const unsigned long long k0 = sm.keys[par][u][lane], k1 = lane < kCl ? sm.keys[par][u][32 + lane] : 0ull;
                    const unsigned long long best = k1 > k0 ? k1 : k0;
                    const unsigned top = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(best >> 32));
                    const unsigned low = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(best >> 32) == top ? static_cast<unsigned>(best) : 0u);
                    const int id = 2047 - static_cast<int>((low >> 21) & 0x7FFu);
                    // the next step's table row
                    const bool row_too = ((live >> u) & 1u) != 0u && id < kBlank;
                    const float* row = xrow + static_cast<size_t>(row_too ? id : 0) * kGates;
                    if constexpr (NU <= 2) {
                        load_if(xg[v][0], row, row_too);
                    } else {
#pragma unroll
                        for (int i = 0; i < kCells; ++i)
#pragma unroll
                            for (int g = 0; g < 4; ++g) load_if(xg[i][g], row + g * kHidden + 32 * i, row_too && lane + 32 * i < kClUnits);
                    }
                    // keys not delivered (a wait gave up), or every token score of the round was NaN: a
                    // blank; the second case is reported as status bit 4
                    if (my == u) {
                        token = min(id, kBlank);
                        no_score = was_live && id > kBlank;
                    }
                }
                emits = was_live && token != kBlank;
                duration = sm.dur[par][my];
                const int old_frame = frame;
                if (was_live) {
                    frame += duration;
                    symbols += 1;
                    if (duration != 0 || symbols == kMaxSymbols) {
                        if (duration == 0) frame += 1;
                        symbols = 0;
                    }
                    count += emits ? 1 : 0;
                }
                alive = was_live && frame < total_frames;
                steps = alive && emits;
                if (owner) {
                    sm.need[my] = steps ? 1 : 0;
                    sm.live[my] = alive ? 1 : 0;
                }
                // the encoder values of the new frame
                if constexpr (NU <= 2) {
                    constexpr unsigned kLanes = (1u << NU) - 1u;
                    live = __ballot_sync(0xffffffffu, alive) & kLanes;
                    need = __ballot_sync(0xffffffffu, steps) & kLanes;
                    const unsigned moved = __ballot_sync(0xffffffffu, alive && frame != old_frame);
                    fetch_enc(NU == 1 ? frame : __shfl_sync(0xffffffffu, frame, x_u), ((moved >> x_u) & 1u) != 0u);
                } else {
                    fetch_enc(frame, alive && frame != old_frame);
                }
            }
            if (ct == 0) *stop_flag = *abort_flag;
            round += 1;
            CL_STAMP(11);
        }
        flush_token();
        if constexpr (kLate && Layers == 1) {
            __syncwarp();
            if (gates_pending) bar_sync(BAR_GATES, kClThreads);
        }
        if (r == 0 && owner && my < U && in_window(p, my)) p.counts[my] = min(count, p.max_tokens);
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
