// A whole network over large batches on the tensor cores (sm_100a, tcgen05 + TMEM), one kernel for all layers of a pass: 128 batch rows stay on the
// SM from the first layer to the last, and only what the pass owes its caller crosses HBM -- the inputs and the outputs of an evaluation, the
// pre-activations and outputs of a training forward pass. Serves
//   evaluate                 y = mlp(x)                                                        (nn_models/mlp/operations_generic.h:77-102)
//   forward                  the same, keeping pre-activations and outputs of every layer       (:103-120)
//   backward                 the chain d_pre = act'(pre) * (W^T d_pre of the layer above), every d_pre kept for the parameter gradients (mlp_grad.cu), and
//                            the input gradient (:152-173)
//
// Arithmetic: fp32 operands as two fp16 parts, x = lead + rest (11 + 11 significant bits), three passes rest * lead, lead * rest, lead * lead with
// fp32 accumulation -- the precision of three tf32 passes at twice their rate and half their shared memory. fp16's range is met by powers of two
// that divide out exactly: a layer's weights are scaled by their largest magnitude, every 64-column piece of an activation row by that piece's, so a
// remainder is subnormal only for values below 2^-17 of those maxima (and then off by at most 2^-39 of them). An output whose weights all lie more than
// 2^-12 below the layer's largest would lose bits by that (2.9e-5 of itself at 2^-24): it is scaled by its own largest, and a network that has such an
// output multiplies every sum by what it lacks when the layer ends. For other networks that is one test per layer: what stands between two layers counts
// (factors for all columns always: evaluate 1,447 -> 1,750 us at 1,048,576 rows; a test per piece: 1,551; two copies of the loop: the code to fetch costs 8 us
// per launch once the activations have pushed it out of L2). The tensor core truncates when it accumulates, so a chain of MMAs is kept to 64 summed columns
// (12 MMAs); the pieces are added, unscaled, to fp32 registers with fused multiply-adds.
//
// Roles: 16 warps (112 registers) move accumulators to registers and do everything element-wise; one thread each of two further warps issues MMAs, one
// of a third brings the weights in. A unit of work is one 64-column piece of the summed index into all outputs of a layer. An MMA of 128 rows takes about
// 128 cycles however narrow it is (the rows of A pass through the tensor core once per instruction), so that only N = 256 runs it at its rate:
//   - layers of more than 128 outputs: 12 MMAs M128 N256 K16 per unit (lead * rest, rest * lead, lead * lead);
//   - up to 128 outputs: the weights' two parts are stacked into one operand of twice the columns, 8 MMAs (rest * both, lead * both), and the two
//     column ranges are added when the accumulator is read.
// Two 256-column accumulators in turn. A thread that issues is held up until the tensor core has room, so two threads take the units in turn: one gets
// its barriers out of the way while the other's MMAs run.
// Element-wise work is a third of the MMAs' time per layer and cannot hide behind this tile's own MMAs as long as a layer needs all of its input; so
// every warp owns 16 columns of EVERY piece of its 32 rows, and the pieces are finished one after the other: the next layer's MMAs start on the first
// piece while the second is being split. A row's scale is the largest exponent among the four warps that share the row (a byte each, exchanged
// through shared memory at a barrier of those four warps).
// The activations of the 128 rows fill 128 KB of shared memory (both parts, up to 256 columns); the weights, split once per call into an image of
// exactly the shared-memory tiles, stream through three 32 KB slots by bulk copies (every CTA reads all weights from L2 for each of its row tiles: 592
// KB per tile of 64-256-256-256-16).
//
// Networks of at most 64 columns, input and outputs included (NARROW): a layer is one unit, 8 MMAs, and what a tile waits for is its own chain of MMAs, tensor-memory reads and splits,
// not any unit's rate. Two CTAs of eight element-wise warps share an SM (80 KB of shared memory, half the tensor memory, 104 registers), a tile each, so that one's chain
// fills the other's gaps; a warp owns columns 16 g ... + 15 of both halves of the piece, and two warps share a row. Wider networks need more than half an SM's shared memory.
// Measured, one CTA of 16 warps / this: evaluate 27-64-64-8 at 524,288 rows 214 / 118 us (11 us at the copy bandwidth); forward and backward chain 29-64-64-5 at 404,405
// rows 303 / 187 and 272 / 193 us (73 and 68), 31-32-32-32-1 at 251,600 rows 226 / 121 and 203 / 101 us.
//
// Bound by the tensor core and, between layers, by what the 16 warps do to a row tile before the next layer can start (about a third of the time), in
// the forward pass by the stores. Measured, 64-256-256-256-16 at 1,048,576 rows: evaluate 3,236 -> 1,450 us (0.58 ms at the rate of three fp16
// passes), forward 3,366 -> 2,850 us (6.8 GB, 1.0 ms at the copy bandwidth).
// Backward, 64-256-256-256-16 at 1,048,576 rows: 3.04 ms for the chain of d_pre (6.5 GB; the products per layer and the passes over d_pre took 4.1 ms).
#include "common.cuh"
#include "tcgen05.cuh"
#include "split_f16.cuh"
#include "dense.cuh"
#include <atomic>

namespace b200rl {

namespace {
constexpr int CH_ROWS = 128, CH_MAX_STEPS = 8, CH_STAGES = 3, CH_NARROW = 64;
constexpr uint32_t CH_TILE = 128 * 128;                           // one fp16 operand tile: 128 rows x 64 columns
constexpr uint32_t CH_PIECE = 2 * CH_TILE;                        // a piece of the activations: both parts
constexpr uint32_t CH_EXP = 4 * CH_ROWS + 2 * 4 * CH_ROWS;        // exponents of the pieces' scales; two buffers of the warps' exponents per row
// What a CTA consists of: an SM's worth, or half of it for networks of at most 64 columns (one piece, weights of one 64-row tile per part)
template <bool NARROW> struct Chain {
    static constexpr int WARPS = NARROW ? 8 : 16, THREADS = 32 * (WARPS + 4), PER_SM = NARROW ? 2 : 1;
    static constexpr int REGISTERS = NARROW ? 104 : 112;          // of the element-wise warps; 32 of the others: together what the CTA is launched with (80, 96 per thread)
    static constexpr int SLICES = NARROW ? 2 : 4, STEP = NARROW ? 32 : 64;   // slices of 16 columns of a warp; their distance
    static constexpr uint32_t A = NARROW ? CH_PIECE : 4 * CH_PIECE, STAGE = NARROW ? CH_TILE : 2 * CH_TILE;
    static constexpr uint32_t ACCUMULATOR = NARROW ? 128 : 256;   // columns of one of the two
    static constexpr uint32_t SMEM = A + CH_STAGES * STAGE + CH_EXP + 256 + 1024;
};
static_assert(Chain<false>::SMEM <= 227 * 1024 && Chain<true>::SMEM <= 113 * 1024, "shared memory");
constexpr size_t CH_TAIL = (3 * 256 + 4) * sizeof(float);        // behind an image: see ChainStep::tail
constexpr uint32_t CH_OWN_SCALE = 12;                             // powers of two below the layer's largest weight from which on an output has its own scale
constexpr long long CH_WAIT_LIMIT = 2000000000LL;
enum { CH_EVALUATE = 0, CH_FORWARD = 1, CH_BACKWARD = 2 };
}

struct ChainStep {
    int N, K, pieces, n, act;                         // n: N rounded up to 16
    const uint8_t* image; const float* tail;          // tail: 256 biases (zeros beyond N), the factors f that 256 outputs' sums lack, their biases x (1 - f), the inverse of the weights' scale, an
    // unused word, eight flags of a byte: whether any of 32 outputs lacks a factor
    float* pre; float* out; long long ld;             // forward: this layer's arenas [rows, N]; evaluate: the last layer's outputs with their row pitch
    // backward: pre_in = pre-activations [rows, N] of the layer below, act = its activation (identity where there is none), out = its d_pre with
    // row pitch ld, or the network's input gradient, or NULL
    const float* pre_in;
};
struct ChainArgs {
    int n_steps, rows, tiles;
    ChainStep step[CH_MAX_STEPS];
    const float* in; long long ld_in; int in_cols;
    // backward: in = gradient of the outputs; the last layer's pre-activations [rows, in_cols] and activation; its d_pre, NULL when that is `in` or not wanted
    const float* in_pre; int in_act;
    float* in_out; long long ld_in_out;
};

__device__ int g_chain_error = 0;

namespace {
// Where the 16 values (8 pairs of neighbouring columns) of a thread lie in its warp's 16 columns of a piece.
//   ROWS:  one row, 16 columns (tcgen05.ld 32x32b): no exchange within the warp, 16-byte shared-memory stores; pair i = columns 2 i, 2 i + 1 of row `lane`
//   !ROWS: four rows 8 apart, 4 columns each (16x256b): a global store instruction writes whole 32-byte sectors; pair 2 s + j = columns 8 j + 2 (lane & 3),
//          + 1 of row 8 s + (lane >> 2)
template <bool ROWS> struct Spread {
    static __device__ __forceinline__ int row(int lane, int i){ return ROWS ? lane : 8 * (i >> 1) + (lane >> 2); }
    static __device__ __forceinline__ int column(int lane, int i){ return ROWS ? 2 * i : 8 * (i & 1) + 2 * (lane & 3); }
};
typedef float2 Slice[8];
template <int ACT>
__device__ __forceinline__ void activate_slice(Slice& v){
#pragma unroll
    for(int i = 0; i < 8; i++){ v[i].x = activation<ACT>(v[i].x); v[i].y = activation<ACT>(v[i].y); }
}
__device__ __forceinline__ void activate_slice_rt(Slice& v, int act){
    switch(act){
        case B200RL_ACT_IDENTITY: break;
        case B200RL_ACT_RELU: activate_slice<B200RL_ACT_RELU>(v); break;
        case B200RL_ACT_TANH: activate_slice<B200RL_ACT_TANH>(v); break;
        case B200RL_ACT_FAST_TANH: activate_slice<B200RL_ACT_FAST_TANH>(v); break;
        default: activate_slice<B200RL_ACT_SIGMOID>(v); break;
    }
}
template <int ACT>
__device__ __forceinline__ void differentiate_slice(Slice& v, const Slice& pre){
#pragma unroll
    for(int i = 0; i < 8; i++){ v[i].x *= d_activation<ACT>(pre[i].x); v[i].y *= d_activation<ACT>(pre[i].y); }
}
__device__ __forceinline__ void differentiate_slice_rt(Slice& v, const Slice& pre, int act){
    switch(act){
        case B200RL_ACT_IDENTITY: break;
        case B200RL_ACT_RELU: differentiate_slice<B200RL_ACT_RELU>(v, pre); break;
        case B200RL_ACT_TANH: differentiate_slice<B200RL_ACT_TANH>(v, pre); break;
        case B200RL_ACT_FAST_TANH: differentiate_slice<B200RL_ACT_FAST_TANH>(v, pre); break;
        default: differentiate_slice<B200RL_ACT_SIGMOID>(v, pre); break;
    }
}
// a slice at (row0, col0) of a [rows, N] matrix with row pitch ld
struct Place { int row0, col0, rows, N; long long ld; };
__device__ __forceinline__ bool aligned_pairs(const float* p, long long ld){ return (ld & 1) == 0 && (reinterpret_cast<uintptr_t>(p) & 7u) == 0; }
__device__ __forceinline__ bool aligned_quads(const float* p, long long ld){ return (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
template <bool ROWS>
__device__ __forceinline__ void store_slice(const Place& p, float* dst, int lane, const Slice& v){
    const bool whole = p.col0 + 16 <= p.N && aligned_pairs(dst, p.ld), quads = ROWS && aligned_quads(dst, p.ld);
#pragma unroll
    for(int i = 0; i < 8; i++){
        const int row = p.row0 + Spread<ROWS>::row(lane, i), col = p.col0 + Spread<ROWS>::column(lane, i);
        if(row >= p.rows) continue;
        float* at = dst + (long long)row * p.ld + col;
        if(whole && quads){ if((i & 1) == 0) *reinterpret_cast<float4*>(at) = make_float4(v[i].x, v[i].y, v[i | 1].x, v[i | 1].y); }
        else if(whole) *reinterpret_cast<float2*>(at) = v[i];
        else{
            if(col < p.N) at[0] = v[i].x;
            if(col + 1 < p.N) at[1] = v[i].y;
        }
    }
}
template <bool ROWS>
__device__ __forceinline__ void load_slice(const Place& p, const float* src, int lane, Slice& v){
    const bool whole = p.col0 + 16 <= p.N && aligned_pairs(src, p.ld), quads = ROWS && aligned_quads(src, p.ld);
#pragma unroll
    for(int i = 0; i < 8; i++){
        const int row = p.row0 + Spread<ROWS>::row(lane, i), col = p.col0 + Spread<ROWS>::column(lane, i);
        const float* at = src + (long long)row * p.ld + col;
        if(whole && quads){
            if((i & 1) == 0){
                const float4 t = row < p.rows ? *reinterpret_cast<const float4*>(at) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                v[i] = make_float2(t.x, t.y); v[i | 1] = make_float2(t.z, t.w);
            }
        }
        else if(whole) v[i] = row < p.rows ? *reinterpret_cast<const float2*>(at) : make_float2(0.0f, 0.0f);
        else v[i] = make_float2(row < p.rows && col < p.N ? at[0] : 0.0f, row < p.rows && col + 1 < p.N ? at[1] : 0.0f);
    }
}
// columns of the slice beyond the layer (whatever lay in tensor memory, or an activation of zero that is not zero) become zeros
template <bool ROWS>
__device__ __forceinline__ void clear_beyond(int col0, int N, int lane, Slice& v){
    if(col0 + 16 <= N) return;
#pragma unroll
    for(int i = 0; i < 8; i++){
        const int col = col0 + Spread<ROWS>::column(lane, i);
        if(col >= N) v[i].x = 0.0f;
        if(col + 1 >= N) v[i].y = 0.0f;
    }
}
// a slice's sums, which started with the bias, times their outputs' factors, plus what the bias lacks then: at[0 ... 15] and at[256 ... 271]
template <bool ROWS>
__device__ __forceinline__ void finish_sums(const float* at, int lane, Slice& v){
    if constexpr(ROWS){
#pragma unroll
        for(int j = 0; j < 4; j++){
            const float4 f = __ldg(reinterpret_cast<const float4*>(at) + j), b = __ldg(reinterpret_cast<const float4*>(at + 256) + j);
            v[2 * j] = __ffma2_rn(v[2 * j], make_float2(f.x, f.y), make_float2(b.x, b.y));
            v[2 * j + 1] = __ffma2_rn(v[2 * j + 1], make_float2(f.z, f.w), make_float2(b.z, b.w));
        }
    }
    else{
#pragma unroll
        for(int j = 0; j < 2; j++){
            const float2 f = __ldg(reinterpret_cast<const float2*>(at + Spread<ROWS>::column(lane, j))), b = __ldg(reinterpret_cast<const float2*>(at + 256 + Spread<ROWS>::column(lane, j)));
#pragma unroll
            for(int s = 0; s < 4; s++) v[2 * s + j] = __ffma2_rn(v[2 * s + j], f, b);
        }
    }
}
__device__ __forceinline__ void ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]){
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
// 16 rows (lanes of the address on) x 16 columns: r[4 j + 2 s], r[4 j + 2 s + 1] = columns 8 j + 2 (lane & 3), + 1 of row 8 s + (lane >> 2)
__device__ __forceinline__ void ld_16x256b_x2(uint32_t taddr, uint32_t* r){
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
// a tile's rows of a matrix into L2
__device__ __forceinline__ void prefetch_rows(const float* p, long long ld, int row0, int rows){
    const uintptr_t from = (reinterpret_cast<uintptr_t>(p + row0 * ld) + 15) & ~(uintptr_t)15, to = reinterpret_cast<uintptr_t>(p + (long long)min(row0 + CH_ROWS, rows) * ld) & ~(uintptr_t)15;
    if(to > from) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(from), "r"((uint32_t)(to - from)) : "memory");
}
}  // namespace

template <int MODE, bool NARROW>
__global__ void __launch_bounds__(Chain<NARROW>::THREADS, Chain<NARROW>::PER_SM) mlp_chain_kernel(const __grid_constant__ ChainArgs a){
    typedef Chain<NARROW> H;
    constexpr bool ROWS = MODE == CH_EVALUATE;                          // only the last outputs go to memory
    constexpr int CH_WARPS = H::WARPS;
    constexpr uint32_t CH_STAGE = H::STAGE;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* stages = base + H::A;
    uint8_t* exps = stages + CH_STAGES * CH_STAGE;                      // [piece][row], then two exchange buffers [row][warp of the row]
    uint64_t* bars = reinterpret_cast<uint64_t*>(exps + CH_EXP);
    uint64_t* w_full = bars; uint64_t* w_empty = bars + CH_STAGES; uint64_t* acc_full = bars + 2 * CH_STAGES; uint64_t* acc_empty = acc_full + 2;
    uint64_t* turn = acc_empty + 2;                                     // whose unit's MMAs may be issued next
    uint64_t* a_full = turn + 2;                                        // [piece]: every warp has stored its columns of it
    uint32_t* slot = reinterpret_cast<uint32_t*>(a_full + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // asked for here, needed once tensor memory is there
    const uint2 own_flags = lane < a.n_steps ? __ldg(reinterpret_cast<const uint2*>(a.step[lane].tail + 770)) : make_uint2(0u, 0u);
    if(tid == 0){
        for(int i = 0; i < CH_STAGES; i++){ tc::mbar_init(w_full + i, 1); tc::mbar_init(w_empty + i, 1); }
        for(int i = 0; i < 2; i++){ tc::mbar_init(acc_full + i, 1); tc::mbar_init(acc_empty + i, CH_WARPS); tc::mbar_init(turn + i, 1); }
        for(int i = 0; i < 4; i++) tc::mbar_init(a_full + i, CH_WARPS);
        tc::fence_mbar_init(); *abort_flag = 0;
    }
    if(warp == CH_WARPS){ tc::tmem_alloc(slot, 2 * H::ACCUMULATOR); tc::tmem_relinquish(); }
    tc::fence_before_thread_sync();
    __syncthreads();
    tc::fence_after_thread_sync();
    const uint32_t tmem = *slot;
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
        if(tc::mbar_try_wait(bar, parity)) return true;
        const long long t0 = clock64();
        while(!tc::mbar_try_wait(bar, parity)){
            if(*abort_flag || clock64() - t0 > CH_WAIT_LIMIT){ *abort_flag = 1; g_chain_error = 1; return false; }
        }
        return true;
    };
    if(warp >= CH_WARPS){
        tc::setmaxnreg_dec<32>();
        if(lane == 0 && (warp == CH_WARPS || warp == CH_WARPS + 2)){
            // ---- the issuing threads: units 0, 2, ... and 1, 3, ...; both follow every fill of the activation pieces ----
            const uint32_t mine = warp == CH_WARPS ? 0u : 1u;
            uint32_t u = 0, w = 0, ready = 0;                           // running unit and slot; bit c: parity of piece c's next fill
            bool ok = true;
            for(int tile = blockIdx.x; tile < a.tiles && ok; tile += gridDim.x){
                for(int st = 0; st < a.n_steps && ok; st++){
                    const ChainStep& y = a.step[st];
                    const int pieces = y.pieces, K = y.K, n = y.n;
                    const bool stacked = NARROW || n <= 128;
                    const uint32_t idesc = tc::make_idesc_f16(CH_ROWS, stacked ? 2 * n : n);
                    for(int c = 0; c < pieces; c++, u++, w += stacked ? 1u : 2u){
                        if(!(ok = wait(a_full + c, (ready >> c) & 1u))) break;
                        ready ^= 1u << c;
                        if((u & 1u) != mine) continue;
                        const int ksteps = min(4, (K - 64 * c + 15) / 16);
                        const uint64_t lead = tc::make_desc_kmajor_sw128(tc::smem_u32(base + c * CH_PIECE)), rest = lead + (CH_TILE >> 4);
                        const uint32_t d = tmem + (u & 1u) * H::ACCUMULATOR, s0 = w % CH_STAGES;
                        if(!(ok = wait(acc_empty + (u & 1u), ((u >> 1) & 1u) ^ 1u))) break;
                        if(!(ok = wait(w_full + s0, (w / CH_STAGES) & 1u))) break;
                        const uint32_t s1 = (w + 1) % CH_STAGES;
                        if(!stacked && !(ok = wait(w_full + s1, ((w + 1) / CH_STAGES) & 1u))) break;
                        // units in order: interleaved, both would finish late and their accumulators be read late
                        if(u > 0 && !(ok = wait(turn + (u & 1u), ((u - 1) >> 1) & 1u))) break;
                        tc::fence_after_thread_sync();
                        const uint64_t w0 = tc::make_desc_kmajor_sw128(tc::smem_u32(stages + s0 * CH_STAGE));
                        // the small products first
                        const uint64_t first = stacked ? rest : lead;
                        for(int k = 0; k < ksteps; k++) tc::mma_f16_ss(d, first + (uint64_t)(2 * k), w0 + (uint64_t)(2 * k), idesc, k ? 1u : 0u);
                        if(stacked){
                            tc::mbar_arrive(turn + ((u + 1) & 1u));
                            for(int k = 0; k < ksteps; k++) tc::mma_f16_ss(d, lead + (uint64_t)(2 * k), w0 + (uint64_t)(2 * k), idesc, 1u);
                            tc::commit(acc_full + (u & 1u));
                            tc::commit(w_empty + s0);
                        }
                        else{
                            tc::commit(w_empty + s0);
                            const uint64_t w1 = tc::make_desc_kmajor_sw128(tc::smem_u32(stages + s1 * CH_STAGE));
                            for(int k = 0; k < ksteps; k++) tc::mma_f16_ss(d, rest + (uint64_t)(2 * k), w1 + (uint64_t)(2 * k), idesc, 1u);
                            tc::mbar_arrive(turn + ((u + 1) & 1u));      // a few MMAs early: the other thread needs about as long to get going
                            for(int k = 0; k < ksteps; k++) tc::mma_f16_ss(d, lead + (uint64_t)(2 * k), w1 + (uint64_t)(2 * k), idesc, 1u);
                            tc::commit(acc_full + (u & 1u));
                            tc::commit(w_empty + s1);
                        }
                    }
                }
            }
        }
        else if(lane == 0 && warp == CH_WARPS + 1){
            // ---- the weights: per unit a slot with the remainder tile and one with the leading tile, or one slot with both (up to 128 outputs) ----
            uint32_t w = 0;                                             // running slot
            bool ok = true;
            for(int tile = blockIdx.x; tile < a.tiles && ok; tile += gridDim.x){
                for(int st = 0; st < a.n_steps && ok; st++){
                    const ChainStep& y = a.step[st];
                    const uint32_t part = (uint32_t)y.n * 128;
                    const bool stacked = NARROW || y.n <= 128;
                    const uint8_t* unit = y.image;
                    if constexpr(MODE == CH_BACKWARD){                  // what the element-wise part will read, into L2 about a layer's MMAs ahead of it
                        if(y.act != B200RL_ACT_IDENTITY) prefetch_rows(y.pre_in, y.N, tile * CH_ROWS, a.rows);
                        if(st == 0 && tile + (int)gridDim.x < a.tiles){
                            prefetch_rows(a.in, a.ld_in, (tile + gridDim.x) * CH_ROWS, a.rows);
                            if(a.in_act != B200RL_ACT_IDENTITY) prefetch_rows(a.in_pre, a.in_cols, (tile + gridDim.x) * CH_ROWS, a.rows);
                        }
                    }
                    for(int c = 0; c < y.pieces && ok; c++, unit += 2 * part){
                        for(int k = stacked ? 0 : 1; k >= 0; k--, w++){
                            const uint32_t s = w % CH_STAGES, bytes = stacked ? 2 * part : part;
                            if(!(ok = wait(w_empty + s, ((w / CH_STAGES) & 1u) ^ 1u))) break;
                            tc::mbar_expect_tx(w_full + s, bytes);
                            tc::bulk_load(stages + s * CH_STAGE, unit + k * part, bytes, w_full + s);
                            tc::mbar_arrive(w_full + s);
                        }
                    }
                }
            }
            // every copy that was started must have landed before the CTA may leave
            for(uint32_t k = w < CH_STAGES ? 0 : w - CH_STAGES; k < w; k++) tc::mbar_wait_bounded(w_full + k % CH_STAGES, (k / CH_STAGES) & 1u, CH_WAIT_LIMIT);
        }
    }
    else{
        tc::setmaxnreg_inc<H::REGISTERS>();
        const int q = warp & 3, g = warp >> 2;                          // rows (TMEM lanes) 32 q ... + 31; columns 16 g ... + 15 of every piece, of every half of the only piece
        const uint32_t tmem_lane = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(16 * g);
        uint32_t u = 0, exchange = 0;                                   // running unit; running exchange of exponents
        bool ok = true;
        // this warp's slices of a piece of the next operand (one, or the first `n` of a narrow network's two): scaled by the largest magnitude of each row in the piece, split, stored
        auto store_operand = [&](int piece, const Slice* v, int n){
            constexpr int PER_ROW = NARROW ? 2 : 4;                      // warps that share a row
            uint8_t* buffer = exps + 4 * CH_ROWS + (exchange & 1u) * 4 * CH_ROWS + PER_ROW * q * 32;
            exchange++;
            constexpr int SLOTS = ROWS ? 1 : 4, PER = 8 / SLOTS;
#pragma unroll
            for(int s = 0; s < SLOTS; s++){
                float m0 = 0.0f, m1 = 0.0f;
#pragma unroll
                for(int p = 0; p < (NARROW ? 2 : 1); p++){
                    if(p >= n) break;
#pragma unroll
                    for(int j = 0; j < PER; j++){ m0 = fmaxf(m0, fabsf(v[p][s * PER + j].x)); m1 = fmaxf(m1, fabsf(v[p][s * PER + j].y)); }
                }
                float m = fmaxf(m0, m1);
                if constexpr(!ROWS){
                    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
                    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
                }
                if(ROWS || (lane & 3) == 0) buffer[PER_ROW * Spread<ROWS>::row(lane, s * PER) + g] = (uint8_t)scale_exponent(m);
            }
            tc::named_barrier_sync(1 + q, 32 * PER_ROW);                 // the warps of these rows; all of them have read the previous layer's sums
            uint8_t* tile_lead = base + piece * CH_PIECE;
            const float2 zero = make_float2(0.0f, 0.0f);
#pragma unroll
            for(int s = 0; s < SLOTS; s++){
                const int r = Spread<ROWS>::row(lane, s * PER);
                uint32_t e;
                if constexpr(NARROW){
                    const uint32_t two = *reinterpret_cast<const uint16_t*>(buffer + 2 * r);
                    e = max(two & 0xFFu, two >> 8);
                }
                else{
                    const uint32_t four = *reinterpret_cast<const uint32_t*>(buffer + 4 * r);
                    e = max(max(four & 0xFFu, (four >> 8) & 0xFFu), max((four >> 16) & 0xFFu, four >> 24));
                }
                if(g == 0 && (ROWS || (lane & 3) == 0)) exps[piece * CH_ROWS + q * 32 + r] = (uint8_t)e;
                const float2 f = make_float2(scale_of(e), scale_of(e));
                const uint32_t row = (uint32_t)(q * 32 + r), x = row & 7u;
#pragma unroll
                for(int p = 0; p < (NARROW ? 2 : 1); p++){
                    if(p >= n) break;
                    uint32_t lead[PER], rest[PER];
#pragma unroll
                    for(int j = 0; j < PER; j++) split_pair(__ffma2_rn(v[p][s * PER + j], f, zero), lead[j], rest[j]);
#pragma unroll
                    for(int j = 0; j < 2; j++){
                        const uint32_t off = row * 128 + (((uint32_t)(4 * p + 2 * g + j) ^ x) << 4) + (ROWS ? 0u : (uint32_t)(lane & 3) * 4);
                        if constexpr(ROWS){
                            *reinterpret_cast<uint4*>(tile_lead + off) = make_uint4(lead[4 * j], lead[4 * j + 1], lead[4 * j + 2], lead[4 * j + 3]);
                            *reinterpret_cast<uint4*>(tile_lead + CH_TILE + off) = make_uint4(rest[4 * j], rest[4 * j + 1], rest[4 * j + 2], rest[4 * j + 3]);
                        }
                        else{
                            *reinterpret_cast<uint32_t*>(tile_lead + off) = lead[j];
                            *reinterpret_cast<uint32_t*>(tile_lead + CH_TILE + off) = rest[j];
                        }
                    }
                }
            }
            tc::fence_proxy_async_smem();
            __syncwarp();
            if(lane == 0) tc::mbar_arrive(a_full + piece);
        };
        const int column = 16 * g;                                       // of slice p: column + STEP p
        // pieces of STEP columns in n of them
        auto slices = [](int n){ return (n + H::STEP - 1) / H::STEP; };
        // this warp's slice of a piece of a tile's inputs
        auto load_input = [&](int tile, int piece, Slice& v){
            load_slice<ROWS>(Place{tile * CH_ROWS + q * 32, H::STEP * piece + column, a.rows, a.in_cols, a.ld_in}, a.in, lane, v);
        };
        const bool some_own = __any_sync(0xffffffffu, (own_flags.x | own_flags.y) != 0u);        // some output of the network has a scale of its own
        Slice acc[4];                                                   // this layer's sums, a slice per piece
        bool loaded = false;                                            // acc[2], acc[3]: the tile's first two input pieces
        for(int tile = blockIdx.x; tile < a.tiles && ok; tile += gridDim.x){
            const int row0 = tile * CH_ROWS + q * 32;
            // ---- the first layer's input (every MMA of the previous tile has completed: its last unit was drained) ----
            const int ins = slices(a.in_cols);
#pragma unroll
            for(int p = 0; p < H::SLICES; p++){
                if(p >= ins) break;
                Slice& v = NARROW ? acc[MODE == CH_BACKWARD ? p : 2 + p] : acc[MODE == CH_BACKWARD ? 0 : p < 2 ? 2 + p : p - 2];
                if constexpr(MODE == CH_BACKWARD){
                    const Place at{row0, H::STEP * p + column, a.rows, a.in_cols, a.ld_in};
                    load_slice<ROWS>(at, a.in, lane, v);
                    if(a.in_act != B200RL_ACT_IDENTITY){
                        Slice& pre = acc[NARROW ? 2 : 1];
                        load_slice<ROWS>(Place{at.row0, at.col0, a.rows, a.in_cols, a.in_cols}, a.in_pre, lane, pre);
                        differentiate_slice_rt(v, pre, a.in_act);
                        clear_beyond<ROWS>(at.col0, a.in_cols, lane, v);
                    }
                }
                else if(p >= 2 || !loaded) load_input(tile, p, v);
                if(!NARROW) store_operand(p, &v, 1);
                if(!NARROW && MODE == CH_BACKWARD && a.in_out) store_slice<ROWS>(Place{row0, H::STEP * p + column, a.rows, a.in_cols, a.ld_in_out}, a.in_out, lane, v);
            }
            if constexpr(NARROW){
                store_operand(0, acc + (MODE == CH_BACKWARD ? 0 : 2), ins);
                if(MODE == CH_BACKWARD && a.in_out){
#pragma unroll
                    for(int p = 0; p < H::SLICES; p++) if(p < ins) store_slice<ROWS>(Place{row0, H::STEP * p + column, a.rows, a.in_cols, a.ld_in_out}, a.in_out, lane, acc[p]);
                }
            }
            loaded = false;
            for(int st = 0; st < a.n_steps && ok; st++){
                const ChainStep& y = a.step[st];
                const bool last = st + 1 == a.n_steps, stacked = NARROW || y.n <= 128;
                const int outs = slices(y.N);                           // of the output
#pragma unroll
                for(int p = 0; p < H::SLICES; p++){                      // the sums start with the bias
                    if(p >= outs) break;
                    const float* at = y.tail + H::STEP * p + column;
                    if constexpr(ROWS){
#pragma unroll
                        for(int j = 0; j < 4; j++){
                            const float4 b = __ldg(reinterpret_cast<const float4*>(at) + j);
                            acc[p][2 * j] = make_float2(b.x, b.y); acc[p][2 * j + 1] = make_float2(b.z, b.w);
                        }
                    }
                    else{
#pragma unroll
                        for(int j = 0; j < 2; j++){
                            const float2 b = __ldg(reinterpret_cast<const float2*>(at + Spread<ROWS>::column(lane, j)));
#pragma unroll
                            for(int s = 0; s < 4; s++) acc[p][2 * s + j] = b;
                        }
                    }
                }
                if(MODE != CH_BACKWARD && last && stacked && tile + (int)gridDim.x < a.tiles){  // a narrow last layer leaves room for the next tile's inputs
                    load_input(tile + gridDim.x, 0, acc[2]);
                    if(ins > 1) load_input(tile + gridDim.x, 1, acc[3]);
                    loaded = true;
                }
                const float weights = __ldg(y.tail + 768);              // inverse of the weights' scale
                Slice below;                                             // backward: pre-activations of the next piece
                for(int c = 0; c < y.pieces; c++, u++){
                    if constexpr(MODE == CH_BACKWARD){
                        if(c + 1 == y.pieces && y.act != B200RL_ACT_IDENTITY) load_slice<ROWS>(Place{row0, column, a.rows, y.N, y.N}, y.pre_in, lane, below);
                    }
                    if(!(ok = wait(acc_full + (u & 1u), (u >> 1) & 1u))) break;
                    tc::fence_after_thread_sync();
                    const uint8_t* e = exps + c * CH_ROWS + q * 32;
                    float inv[ROWS ? 1 : 4];
#pragma unroll
                    for(int s = 0; s < (ROWS ? 1 : 4); s++) inv[s] = weights * inverse_scale_of(e[Spread<ROWS>::row(lane, 2 * s)]);
                    const uint32_t from = tmem_lane + (u & 1u) * H::ACCUMULATOR;
#pragma unroll
                    for(int p = 0; p < H::SLICES; p++){
                        if(p >= outs) break;
                        uint32_t d[16], d2[16];
                        auto read = [&](uint32_t column, uint32_t (&r)[16]){
                            if constexpr(ROWS) ld_32x32b_x16(from + column, r);
                            else{ ld_16x256b_x2(from + column, r); ld_16x256b_x2(from + column + (16u << 16), r + 8); }
                        };
                        read((uint32_t)(H::STEP * p), d);
                        if(p < 2 && stacked) read((uint32_t)(H::STEP * p + y.n), d2);  // stacked parts: both column ranges
                        tc::tmem_wait_ld();
#pragma unroll
                        for(int i = 0; i < 8; i++){
                            // ROWS: register pair i = pair i; else register pair 4 x + 2 j + s = pair 2 (2 x + s) + j
                            const int at = ROWS ? i : 2 * (2 * (i >> 2) + (i & 1)) + ((i >> 1) & 1);
                            const float f = inv[ROWS ? 0 : at >> 1];
                            acc[p][at] = __ffma2_rn(make_float2(__uint_as_float(d[2 * i]), __uint_as_float(d[2 * i + 1])), make_float2(f, f), acc[p][at]);
                            if(p < 2 && stacked)
                                acc[p][at] = __ffma2_rn(make_float2(__uint_as_float(d2[2 * i]), __uint_as_float(d2[2 * i + 1])), make_float2(f, f), acc[p][at]);
                        }
                    }
                    tc::fence_before_thread_sync();
                    __syncwarp();
                    if(lane == 0) tc::mbar_arrive(acc_empty + (u & 1u));
                }
                if(!ok) break;
                if(some_own){                                           // one test per layer: it stands between this layer's MMAs and the next one's
#pragma unroll
                    for(int p = 0; p < H::SLICES; p++){
                        if(p >= outs) break;
                        finish_sums<ROWS>(y.tail + 256 + H::STEP * p + column, lane, acc[p]);
                    }
                }
                // every MMA of this layer has completed: its input may be overwritten
#pragma unroll
                for(int p = 0; p < H::SLICES; p++){
                    if(p >= outs) break;
                    const Place at{row0, H::STEP * p + column, a.rows, y.N, y.ld};
                    if constexpr(MODE == CH_FORWARD) store_slice<ROWS>(at, y.pre, lane, acc[p]);
                    if constexpr(MODE == CH_BACKWARD){
                        if(y.act != B200RL_ACT_IDENTITY){
                            differentiate_slice_rt(acc[p], below, y.act);
                            if(p + 1 < outs) load_slice<ROWS>(Place{row0, at.col0 + H::STEP, a.rows, y.N, y.N}, y.pre_in, lane, below);
                        }
                    }
                    else activate_slice_rt(acc[p], y.act);
                    clear_beyond<ROWS>(at.col0, y.N, lane, acc[p]);
                    if(!last){ if(!NARROW) store_operand(p, acc + p, 1); }
                    else if(MODE != CH_BACKWARD || y.out) store_slice<ROWS>(at, y.out, lane, acc[p]);
                }
                if(NARROW && !last) store_operand(0, acc, outs);
                if(MODE != CH_EVALUATE && !last && (MODE == CH_FORWARD || y.out)){
#pragma unroll
                    for(int p = 0; p < H::SLICES; p++){
                        if(p >= outs) break;
                        store_slice<ROWS>(Place{row0, H::STEP * p + column, a.rows, y.N, y.ld}, y.out, lane, acc[p]);
                    }
                }
            }
        }
    }
    tc::fence_before_thread_sync();
    __syncthreads();
    if(warp == CH_WARPS) tc::tmem_dealloc(tmem, 2 * H::ACCUMULATOR);
}

// ---- weight images: a CTA per 32 output rows of a product, a warp per row. Every CTA finds the
// largest magnitude of its layer's weights for itself (at most 256 KB from L2), which saves a launch in front ----------------------------------
// element (n, k) of the product's weights at W[n * stride_n + k * stride_k]
struct ChainImage { const float* W; const float* bias; uint8_t* image; float* tail; int N, K, block_begin, stride_n, stride_k; };
struct ChainImages { int n; ChainImage y[CH_MAX_STEPS]; int blocks; };
__global__ void __launch_bounds__(1024) chain_image_kernel(const __grid_constant__ ChainImages a){
    __shared__ uint32_t largest[32];
    int l = 0;
    while(l + 1 < a.n && (int)blockIdx.x >= a.y[l + 1].block_begin) l++;
    const ChainImage& y = a.y[l];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = (blockIdx.x - y.block_begin) * 32 + warp, rows = (y.N + 15) / 16 * 16, pieces = (y.K + 63) / 64;
    uint8_t* flags = reinterpret_cast<uint8_t*>(y.tail + 770);
    float v[4][2];
#pragma unroll
    for(int c = 0; c < 4; c++){
#pragma unroll
        for(int k = 0; k < 2; k++){
            const int i = 64 * c + 2 * lane + k;
            v[c][k] = n < y.N && i < y.K ? __ldg(y.W + (size_t)n * y.stride_n + (size_t)i * y.stride_k) : 0.0f;
        }
    }
    float m = 0.0f;
    const int count = y.N * y.K;
    if((reinterpret_cast<uintptr_t>(y.W) & 15u) == 0 && (count & 3) == 0){
#pragma unroll 8
        for(int i = threadIdx.x; i < count / 4; i += 1024){ const float4 t = __ldg(reinterpret_cast<const float4*>(y.W) + i); m = fmaxf(m, fmaxf(fmaxf(fabsf(t.x), fabsf(t.y)), fmaxf(fabsf(t.z), fabsf(t.w)))); }
    }
    else{
#pragma unroll 8
        for(int i = threadIdx.x; i < count; i += 1024) m = fmaxf(m, fabsf(__ldg(y.W + i)));
    }
    float m_row = 0.0f;
#pragma unroll
    for(int c = 0; c < 4; c++) m_row = fmaxf(m_row, fmaxf(fabsf(v[c][0]), fabsf(v[c][1])));
    // magnitudes compare like their bits (fmaxf has left NaNs out)
    if(const uint32_t t = __reduce_max_sync(0xffffffffu, __float_as_uint(m)); lane == 0) largest[warp] = t;
    m_row = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m_row)));
    __syncthreads();
    m = __uint_as_float(__reduce_max_sync(0xffffffffu, largest[lane]));
    const uint32_t e_layer = scale_exponent(m), e_row = scale_exponent(m_row);
    const bool apart = m_row > 0.0f && e_row + CH_OWN_SCALE < e_layer;   // a row of zeros fits any scale
    const uint32_t e = !apart ? e_layer : e_row + 126 < e_layer ? e_layer - 126 : e_row;      // the factor stays a normal number
    const float f = scale_of(e);
    const int some_apart = __syncthreads_or(apart);
    const int cta = blockIdx.x - y.block_begin;
    if(threadIdx.x == 0) flags[cta] = some_apart ? 1 : 0;
    if(cta == 0){
        for(int i = rows + threadIdx.x; i < 256; i += 1024){ y.tail[i] = 0.0f; y.tail[256 + i] = 0.0f; y.tail[512 + i] = 0.0f; }
        if((int)threadIdx.x >= (rows + 31) / 32 && threadIdx.x < 8) flags[threadIdx.x] = 0;
        if(threadIdx.x == 0) y.tail[768] = inverse_scale_of(e_layer);
    }
    if(lane == 0 && n < rows){
        const float bias = y.bias && n < y.N ? __ldg(y.bias + n) : 0.0f, lacks = scale_of(e_layer) * inverse_scale_of(e);       // 2^(e - e_layer)
        y.tail[n] = bias; y.tail[256 + n] = lacks; y.tail[512 + n] = bias - bias * lacks;
    }
    if(n >= rows) return;
    const uint32_t off = (uint32_t)n * 128 + ((((uint32_t)lane >> 2) ^ ((uint32_t)n & 7u)) << 4) + ((uint32_t)lane & 3u) * 4;
#pragma unroll
    for(int c = 0; c < 4; c++){
        if(c >= pieces) break;
        uint32_t lead, rest;
        split_pair(make_float2(v[c][0] * f, v[c][1] * f), lead, rest);
        uint8_t* unit = y.image + (size_t)c * rows * 256;
        *reinterpret_cast<uint32_t*>(unit + off) = lead;
        *reinterpret_cast<uint32_t*>(unit + (size_t)rows * 128 + off) = rest;
    }
}

// ---- host side ---------------------------------------------------------------------------------------------------------------------------
// Which passes run here: networks of two to eight layers, no wider than 256. A CTA takes 128 rows through all layers in the same time however few CTAs there
// are (34 us for 64-256-256-256-16, 54 us when everything is kept; 14 and 18 us for 27-64-64-8), while the kernels per layer gain from a smaller batch and
// start sooner; so the lines lie where the rows fill the SMs or the products are many. The lines for networks of at most 64 columns were drawn with one row tile per SM and still stand where they
// were: with two, 3-32-32-1 would gain from the chain in the forward pass at 65,536 rows and 10-16-2 in the gradients at 16,384. Measured, these kernels against the kernels per layer, us (graph of ten
// calls; rows x the network's weights in millions behind the rows):
//   evaluate            4-256-256-1 at 2,048: 23 and 29; 64-256-16 at 2,048 (42): 17 and 15, at 4,096 (84): 17 and 28; 8-256-4 at 8,192 (25): 15 and 13, at 16,384
//                       (50): 15 and 20; 64-128-4 at 8,192 (71): 14 and 13, at 16,384 (143): 15 and 17; 3-32-32-1 at 8,192 (9): 11 and 12, at 16,384 (19): 11 and 15
//   forward             33-200-200-7 at 2,048 (98): 37 and 23, at 4,096 (197): 37 and 34; 64-256-256-256-16 at 2,048 (310): 54 and 55; 27-64-64-8 at 8,192 (52): 17 and 17;
//                       3-64-64-1 at 16,384 (71): 17 and 24; 20-32-32-32-8 at 16,384 (48): 17 and 25; 3-50-50-1 at 16,384 (44): 17 and 24; 3-32-32-1 at 65,536
//                       (75): 28 and 42 (below the line of 2,048 weights; 50 and 41 with one tile per SM); 64-128-4 at 65,536 (570): 51 and 49
//   gradients           17-130-130-3 at 4,096 (80): 51 and 49, at 8,192 (160): 57 and 81; 33-200-200-7 at 2,048 (98): 58 and 53; 64-256-16 at 8,192 (168): 42 and 39, at
//                       16,384: 48 and 48; 256-256-256 at 2,048: 58 and 83; 64-128-4 at 8,192: 31 and 28, at 16,384: 34 and 40; 10-16-2 at 16,384 (3): 25 and 27
//   input gradient alone  17-130-130-3 at 2,048 (40): 27 and 18, at 4,096 (80): 27 and 35; 8-256-4 at 4,096 (13): 22 and 17, at 8,192: 22 and 99
bool mlp_chain_takes(const b200rl_mlp_shape* sh, int batch, int pass){
    if(sh->n_layers > CH_MAX_STEPS || sh->n_layers < 2) return false;
    int widest = sh->input_dim;
    long long weights = 0;
    for(int l = 0, I = sh->input_dim; l < sh->n_layers; I = sh->dims[l], l++){
        if(sh->dims[l] > widest) widest = sh->dims[l];
        weights += (long long)I * sh->dims[l];
    }
    const bool wide = widest > 128, two = sh->n_layers == 2;
    if(widest > 256 || batch < (wide ? 2048 : 8192)) return false;
    const long long million = 1000000, work = weights * batch;
    switch(pass){
        case CHAIN_EVALUATE: return two ? work >= (wide ? 50 : 72) * million : wide || work >= 16 * million;
        case CHAIN_FORWARD: return two ? wide && work >= 50 * million : wide ? batch >= 4096 || work >= 200 * million : weights >= 2048 && (batch >= 16384 || work >= 64 * million);
        case CHAIN_GRADIENTS: return two ? weights >= 32768 || (batch >= 16384 && (wide || weights >= 4096)) : !wide || work >= 90 * million;
        default: return batch >= 8192 || work >= 80 * million;
    }
}
static size_t chain_image_bytes(int N, int K){
    const size_t rows = (N + 15) / 16 * 16;
    return rows * ((K + 63) / 64) * 256 + CH_TAIL;
}
static size_t images_bytes(const b200rl_mlp_shape* sh){
    size_t n = 0; int I = sh->input_dim;
    for(int l = 0; l < sh->n_layers; l++){ n += chain_image_bytes(sh->dims[l], I); I = sh->dims[l]; }
    return n;
}
size_t mlp_chain_workspace_bytes(const b200rl_mlp_shape* sh, int batch){
    if(!mlp_chain_takes(sh, batch, CHAIN_EVALUATE) && !mlp_chain_takes(sh, batch, CHAIN_FORWARD)) return 0;
    return images_bytes(sh);
}
// the word that a kernel's expired wait sets, and its reset (b200rl_device_error_state, b200rl_device_error_clear)
int mlp_chain_error_get(int* word){ B200RL_CUDA_TRY(cudaMemcpyFromSymbol(word, g_chain_error, sizeof(int))); return B200RL_OK; }
int mlp_chain_error_clear(){ const int zero = 0; B200RL_CUDA_TRY(cudaMemcpyToSymbol(g_chain_error, &zero, sizeof(int))); return B200RL_OK; }

static void chain_step(ChainStep& y, ChainImages& images, const float* W, const float* bias, int N, int K, uint8_t*& ws, bool transposed = false){
    y.N = N; y.K = K; y.pieces = (K + 63) / 64; y.n = (N + 15) / 16 * 16;
    ChainImage& m = images.y[images.n++];
    m.W = W; m.N = N; m.K = K; m.stride_n = transposed ? 1 : K; m.stride_k = transposed ? N : 1; m.block_begin = images.blocks;
    m.bias = bias; m.image = ws; m.tail = reinterpret_cast<float*>(ws + chain_image_bytes(N, K) - CH_TAIL);
    images.blocks += (y.n + 31) / 32;
    y.image = m.image; y.tail = m.tail;
    ws += chain_image_bytes(N, K);
}
template <int MODE, bool NARROW>
static int launch_chain_kernel(ChainArgs& a, cudaStream_t s){
    typedef Chain<NARROW> H;
    static std::atomic<bool> configured[MAX_DEVICES];
    int dev = 0, sms = 0;
    int rc = current_device(&dev);
    if(rc) return rc;
    if((rc = sm_count(&sms))) return rc;
    if(!configured[dev].load(std::memory_order_acquire)){
        B200RL_CUDA_TRY(cudaFuncSetAttribute((mlp_chain_kernel<MODE, NARROW>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)H::SMEM));
        configured[dev].store(true, std::memory_order_release);
    }
    a.tiles = (a.rows + CH_ROWS - 1) / CH_ROWS;
    const int ctas = H::PER_SM * sms;
    mlp_chain_kernel<MODE, NARROW><<<a.tiles < ctas ? a.tiles : ctas, H::THREADS, H::SMEM, s>>>(a);
    B200RL_LAUNCH_CHECK("mlp_chain");
    return B200RL_OK;
}
template <int MODE>
static int launch_chain(ChainArgs& a, const ChainImages& images, cudaStream_t s, bool with_images = true){
    if(with_images){
        chain_image_kernel<<<images.blocks, 1024, 0, s>>>(images);
        B200RL_LAUNCH_CHECK("chain_image");
    }
    bool narrow = true;
    for(int l = 0; l < a.n_steps; l++) narrow = narrow && a.step[l].N <= CH_NARROW && a.step[l].K <= CH_NARROW;
    return narrow ? launch_chain_kernel<MODE, true>(a, s) : launch_chain_kernel<MODE, false>(a, s);
}

// pre == NULL: evaluate into y; otherwise forward into the arenas
int mlp_chain_forward(const b200rl_mlp_shape* sh, const float* params, const float* x, int ldx, float* pre, float* out, float* y, int ldy, int batch, void* workspace,
                      size_t workspace_bytes, cudaStream_t s){
    if(!workspace || workspace_bytes < images_bytes(sh) || (reinterpret_cast<uintptr_t>(workspace) & 15u)) return B200RL_ERR_UNSUPPORTED;
    // a CTA reads inputs while another one writes outputs: outputs over the inputs take the kernels per layer. Columns of one matrix do not overlap.
    if(y && y < x + (size_t)batch * ldx && x < y + (size_t)batch * ldy){
        const long long at = ldx == ldy ? ((y - x) % ldx + ldx) % ldx : 0;
        if(at < sh->input_dim || at + sh->dims[sh->n_layers - 1] > ldx) return B200RL_ERR_UNSUPPORTED;
    }
    ChainArgs a{};
    ChainImages images{};
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    a.rows = batch; a.in = x; a.ld_in = ldx; a.in_cols = sh->input_dim;
    int I = sh->input_dim;
    const float* p = params;
    for(int l = 0; l < sh->n_layers; l++){
        const int O = sh->dims[l];
        ChainStep& t = a.step[a.n_steps++];
        chain_step(t, images, p, p + (size_t)O * I, O, I, ws);
        t.act = sh->acts[l]; t.ld = O;
        if(pre){ t.pre = pre; t.out = out; pre += (size_t)batch * O; out += (size_t)batch * O; }
        else if(l + 1 == sh->n_layers){ t.out = y; t.ld = ldy; }
        p += (size_t)O * I + O; I = O;
    }
    return pre ? launch_chain<CH_FORWARD>(a, images, s) : launch_chain<CH_EVALUATE>(a, images, s);
}

// ---- backward: d_pre of every layer in one chain of transposed products, then all parameter gradients (mlp_grad.cu) ----
// Rows are taken in chunks of up to 2^18, so that the d_pre of all layers (784 columns of 64-256-256-256-16) take 0.8 GB, not a batch of them.
constexpr int CHAIN_BACKWARD_ROWS = 1 << 18;
int mlp_grad_splits(const b200rl_mlp_shape* sh);
int mlp_grad_launch(const b200rl_mlp_shape* sh, const float* const* input, const long long* ld_input, const float* const* d_pre, const long long* ld_pre, int rows,
                    float* partial, long long record, bool accumulate, cudaStream_t s);
int pad_rows(const float* from, long long ld, int rows, int cols, float* to, cudaStream_t s);
int reduce_partials_into(float* dst, const float* partial, int n, long long stride, int segments, cudaStream_t s);

static int chain_backward_rows(int batch){
    const int chunks = (batch + CHAIN_BACKWARD_ROWS - 1) / CHAIN_BACKWARD_ROWS;
    return ((batch + chunks - 1) / chunks + CH_ROWS - 1) / CH_ROWS * CH_ROWS;
}
static size_t aligned256(size_t n){ return (n + 255) / 256 * 256; }
static long long padded(int columns){ return (columns + 3) / 4 * 4; }           // row pitch for the gradient kernel: rows of whole 16 bytes
static size_t transposed_images_bytes(const b200rl_mlp_shape* sh){
    size_t n = 0; int I = sh->input_dim;
    for(int l = 0; l < sh->n_layers; l++){ n += chain_image_bytes(I, sh->dims[l]); I = sh->dims[l]; }
    return aligned256(n);
}
size_t mlp_chain_backward_scratch_bytes(const b200rl_mlp_shape* sh, int batch){
    if(!mlp_chain_takes(sh, batch, CHAIN_GRADIENTS) && !mlp_chain_takes(sh, batch, CHAIN_INPUT)) return 0;
    size_t columns = padded(sh->input_dim);                                  // padded copies of inputs; whether x needs one depends on where it lies
    bool copies = false;
    for(int l = 0; l < sh->n_layers; l++){
        copies = copies || sh->dims[l] % 4;                                  // a layer's outputs of such a width, or behind ones of such a width
        columns += padded(sh->dims[l]) * (copies && l + 1 < sh->n_layers ? 2 : 1);
    }
    return transposed_images_bytes(sh) + aligned256(sizeof(float) * mlp_grad_splits(sh) * b200rl_mlp_num_params(sh)) + sizeof(float) * columns * (size_t)chain_backward_rows(batch);
}
int mlp_chain_backward(const b200rl_mlp_shape* sh, const float* params, float* grads, const float* x, int ldx, const float* pre, const float* out, const float* d_out,
                       float* d_input, int batch, void* scratch, size_t scratch_bytes, cudaStream_t s){
    if(!scratch || scratch_bytes < mlp_chain_backward_scratch_bytes(sh, batch) || (reinterpret_cast<uintptr_t>(scratch) & 15u)) return B200RL_ERR_UNSUPPORTED;
    const int L = sh->n_layers, chunk = chain_backward_rows(batch);
    const size_t n_params = b200rl_mlp_num_params(sh);
    uint8_t* ws = static_cast<uint8_t*>(scratch);
    float* partial = reinterpret_cast<float*>(ws + transposed_images_bytes(sh));
    const float* input[CH_MAX_STEPS]; float* copy[CH_MAX_STEPS]; float* d_pre[CH_MAX_STEPS];
    long long ld_input[CH_MAX_STEPS], ld[CH_MAX_STEPS]; size_t poff[CH_MAX_STEPS], aoff[CH_MAX_STEPS]; int Is[CH_MAX_STEPS];
    {
        float* p = partial + aligned256(sizeof(float) * mlp_grad_splits(sh) * n_params) / sizeof(float);
        size_t po = 0, ao = 0; int I = sh->input_dim;
        for(int l = 0; l < L; l++){
            const int O = sh->dims[l];
            poff[l] = po; aoff[l] = ao; Is[l] = I; ld[l] = padded(O); d_pre[l] = p;
            p += (size_t)ld[l] * chunk;
            const bool aligned = l > 0 ? I % 4 == 0 : ldx % 4 == 0;
            const float* from = l > 0 ? out + aoff[l - 1] : x;
            copy[l] = aligned && (reinterpret_cast<uintptr_t>(from) & 15u) == 0 ? nullptr : p;
            ld_input[l] = copy[l] ? padded(I) : l > 0 ? I : ldx;
            if(copy[l]) p += (size_t)padded(I) * chunk;
            po += (size_t)O * I + O; ao += (size_t)batch * O; I = O;
        }
        if(reinterpret_cast<uint8_t*>(p) > ws + scratch_bytes) return B200RL_ERR_UNSUPPORTED;      // an output arena that is not aligned
    }
    const int O_last = sh->dims[L - 1], act_last = sh->acts[L - 1];
    const bool copy_last = act_last != B200RL_ACT_IDENTITY || (O_last & 3) != 0 || (reinterpret_cast<uintptr_t>(d_out) & 15u) != 0;
    if(!copy_last) ld[L - 1] = O_last;
    for(int row0 = 0; row0 < batch; row0 += chunk){
        ChainArgs a{};
        ChainImages images{};
        uint8_t* image = ws;
        a.rows = batch - row0 < chunk ? batch - row0 : chunk;
        a.in = d_out + (size_t)row0 * O_last; a.ld_in = O_last; a.in_cols = O_last;
        a.in_pre = pre + aoff[L - 1] + (size_t)row0 * O_last; a.in_act = act_last;
        a.in_out = grads && copy_last ? d_pre[L - 1] : nullptr; a.ld_in_out = ld[L - 1];
        if(!copy_last) d_pre[L - 1] = const_cast<float*>(a.in);
        for(int l = L - 1; l >= (d_input ? 0 : 1); l--){
            ChainStep& t = a.step[a.n_steps++];
            chain_step(t, images, params + poff[l], nullptr, Is[l], sh->dims[l], image, true);
            if(l > 0){
                t.act = sh->acts[l - 1]; t.pre_in = pre + aoff[l - 1] + (size_t)row0 * Is[l];
                t.out = grads ? d_pre[l - 1] : nullptr; t.ld = ld[l - 1];
            }
            else{ t.act = B200RL_ACT_IDENTITY; t.out = d_input + (size_t)row0 * Is[0]; t.ld = Is[0]; }
        }
        int rc = launch_chain<CH_BACKWARD>(a, images, s, row0 == 0);
        if(rc) return rc;
        if(!grads) continue;
        for(int l = 0; l < L; l++){
            const long long pitch = l > 0 ? Is[l] : ldx;
            input[l] = (l > 0 ? out + aoff[l - 1] : x) + row0 * pitch;
            if(copy[l]){
                if((rc = pad_rows(input[l], pitch, a.rows, Is[l], copy[l], s))) return rc;
                input[l] = copy[l];
            }
        }
        if((rc = mlp_grad_launch(sh, input, ld_input, d_pre, ld, a.rows, partial, (long long)n_params, row0 > 0, s))) return rc;
    }
    return grads ? reduce_partials_into(grads, partial, (int)n_params, (long long)n_params, mlp_grad_splits(sh), s) : B200RL_OK;
}

}  // namespace b200rl
