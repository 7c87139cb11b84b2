// A whole network walked by ONE team of CTAs per group of batch rows: forward, input gradients and parameter gradients without leaving the
// chip. The building block of the one-launch training steps (mlp_team.cu, ppo_team.cu).
//
// At the batch sizes of reinforcement learning (100 ... a few thousand rows) a layer is a microsecond of arithmetic, and what a step costs is the
// chain of dependent launches and of passes over memory between them. Here a team of C CTAs (a thread-block cluster, C = 1, 2, 4 or 8) takes R
// rows through every layer:
//   - the hidden units of every layer are dealt out over the team: CTA c holds the weight rows [c S, c S + S) of each layer in shared memory for
//     the whole launch, so that a network of a few hundred KB is spread over the team's shared memory;
//   - forward: a CTA computes its units' outputs for the R rows and stores them into the input buffer of the next layer in EVERY CTA of the team
//     (distributed shared memory), one cluster barrier per layer;
//   - backward: the input gradient is a sum over the units, i.e. over the team: each CTA forms the partial sums of its own units for all inputs
//     and stores each part into the CTA that owns that input, which adds the parts in a fixed order;
//   - parameter gradients: a patch of 4, 8 outputs x 4, 8 inputs per thread, or up to four of 4 x 4, in registers over all row tiles of the launch. The bias is column I of the
//     weight row (its input is the constant 1 in column I of the activation rows).
// A product of a layer is 4 x 4 register tiles with 16-byte shared-memory operands; the summed index of a tile is shared out over 1 ... 16 lanes of ONE warp, which
// add their parts by shuffles and go on with what follows the product (bias, activation, derivative; derivative of the layer below) on the sums in
// their registers: nothing but finished rows passes through shared memory, and a layer is one phase with one barrier behind it.
// Teams write their gradient sums to scratch memory; after a grid-wide barrier all CTAs share out the parameters, add the teams' sums in a fixed
// order and apply the optimizer step.
//
// A launch is bound by latency: counters of a PPO epoch of 27-64-64-8 (2,048 rows a minibatch) show 31 % of the issue slots used, the shared-memory pipe at 23 %, the multiply-adds at 16 %, and the
// warps at barriers for 47 % of their time (those of the CTA between phases and those of the grid). Within a product the reads come before the multiply-adds: a 16-byte read takes 4 cycles of an SM for a warp, 2 where all lanes of each half-phase read the same, so a 4 x 4 x 4 step costs 24 cycles of
// reads against 16 of multiply-adds; eight lanes in a row share the tile's rows (2 cycles) and read eight weight rows an odd number of 16 bytes apart
// (4 cycles, no conflicts). Patches of 8 x 8 read 12 cycles for 32 of multiply-adds.
//
// Loops over elements stay rolled: a minibatch walks the whole code once, and what does not fit the instruction caches is fetched anew for every one of them.
// The layers are unrolled: their sizes are then constants in the instructions, not loads at the head of every phase (64-64-64-4 at 64 rows 17.7 -> 16.4 us, 200-200-200-8 at 700 rows 57.6 -> 51.4,
// 32-32-13 at 32 rows 12.3 -> 11.2).
// Measured against products whose parts met in shared memory, element-wise passes behind them, 256 threads: 4-256-256-1 at 256 rows 28.7 -> 24.3 us a training step, 33-200-200-7 at 5,003 rows
// 121 -> 103, PPO epochs of 27-64-64-8 with 2,048 rows 20.8 -> 16.7 us per minibatch. Packed multiply-adds (two per instruction) were slower in the training step:
// 135 us for the second one, because the pairs take twice the registers; the PPO epoch, whose order of sums has the pairs, holds smaller gradient patches.
#pragma once
#include "common.cuh"
#include <algorithm>

namespace b200rl { namespace team {

// Four warps per scheduler: with the products' sums in registers until they are finished, more warps hide the shared-memory latencies.
// (Half as many for networks without work for more, by a number in the plan instead of a constant: no faster there, 3 to 8 % slower elsewhere.)
constexpr int THREADS = 512, WARPS = THREADS / 32, MAX_LAYERS = 4, MAX_PATCHES_PER_THREAD = 4;

// quotient by a divisor known on the host (n d < 2^32): one multiplication instead of a division's ~40 instructions, which on the path of a
// few microseconds per layer would be most of the time
struct Divisor { unsigned m; };
inline Divisor divisor(int d){ return Divisor{d <= 1 ? 0u : (unsigned)((0x100000000ull + (unsigned)d - 1) / (unsigned)d)}; }

struct Layer {
    int O, I, act;
    int S;                      // units per CTA (multiple of 4); unit u's weight row lies at row (u & 3) S / 4 + u / 4, so that the four units of a tile are S / 4 rows apart
    int P;                      // pitch of weight and activation rows in floats: I + 1 rounded up to four, an odd number of 16-byte pieces
    int K4;                     // 16-byte pieces of the summed index of a forward product (with the bias column, unless that starts a piece of its own)
    long long poff, aoff;       // offset in the parameter arena (weights, then bias), in the activation arenas (x batch)
    int w, a, p, g, d;          // shared-memory offsets (floats): weight rows [S][P], input rows [R][P]; [R][S]: pre-activations, activation derivatives, d_pre
    int fwd_tiles, fwd_shift, bwd_tiles, bwd_shift;            // 4 x 4 tiles of a product; 2^shift lanes share out its summed index
    int fwd_parts, bwd_parts;   // ORDERED: among so many of them
    int patch_begin, across;    // gradient patches: first index of this layer, patches along the inputs
    Divisor by_S4, by_I, by_row, by_I4, by_across, by_owner;
};
struct Net {
    int n_layers, C, R, n_params;            // C: CTAs per team
    int patch_o, patch_i, n_patches, quads;  // a patch is patch_o x patch_i pieces of four (1 x 1, 2 x 1, 2 x 2); patches per CTA; 16-byte pieces of gradient sums per CTA
    int a_alt;                               // the first layer's second buffer of input rows lies this much behind the first
    Divisor by_quads, by_patches, by_I0;
    int zero_begin, zero_end;                // weight and input rows of all layers (offsets, multiples of four floats)
    int rb[2];                               // exchange buffers of teams of several CTAs (offsets)
    int end;                                 // end of the network's shared memory (floats)
    Layer layer[MAX_LAYERS];
};

// lanes that share out the K4 pieces of a tile's summed index, as a power of two: by an estimate in cycles of an SM, reads or latencies of the steps, then the exchange
// and what follows the product (a lane keeps 4, 2, 1 of the tile's rows)
inline int lanes_of_a_tile(int tiles, int K4){
    int best = 0; double cost = 0.0;
    for(int s = 0; s <= 4; s++){
        const int warps = (tiles + (32 >> s) - 1) / (32 >> s), rounds = (warps + WARPS - 1) / WARPS, steps = (K4 + (1 << s) - 1) >> s, rows = s == 0 ? 4 : s == 1 ? 2 : 1;
        const double reads = 24.0 * warps * steps, latency = 70.0 * rounds * steps;
        const double c = (reads > latency ? reads : latency) + rounds * (80.0 * rows + 25.0 * s) + 8.0 * rows * warps;
        if(s == 0 || c < cost){ best = s; cost = c; }
    }
    return best;
}

// The same where the order of every sum is fixed (ORDERED, ppo_team.cu): the summed index of a tile is dealt out to a number of lanes that is part of the order, as many (a power of two) as
// give 256 threads a part each, of at least two pieces of a forward and one of a backward product. Up to three lanes without a part come on top where that leaves threads idle: they take some
// of the tile's rows to the end.
constexpr int ORDERED_LANES = 256;
inline int parts(int tiles, int pieces){
    int s = 0;
    while(s < 5 && (2 << s) * tiles <= ORDERED_LANES && (2 << s) <= pieces) s++;
    return s;
}
inline int lanes_of_parts(int tiles, int parts){
    while(parts < 2 && (2 << parts) * tiles <= ORDERED_LANES) parts++;
    return parts;
}
inline int parts_forward(const Net& n, int l){ return parts((n.R / 4) * (n.layer[l].S / 4), (n.layer[l].I / 4 + 1) / 2); }
inline int parts_backward(const Net& n, int l){ return parts((n.R / 4) * ((n.layer[l].I + 3) / 4), n.layer[l].S / 4); }
// Floats of shared memory that add_parts_in_order takes: 512 for each warp that has tiles of a product in four or more parts
inline int ordered_scratch(const Net& n){
    int warps = 0;
    for(int l = 0; l < n.n_layers; l++){
        const Layer& y = n.layer[l];
        const int forward = parts_forward(n, l), backward = l > 0 ? parts_backward(n, l) : 0;
        if(forward > 1) warps = std::max(warps, (((n.R / 4) * (y.S / 4) << forward) + 31) / 32);
        if(backward > 1) warps = std::max(warps, (((n.R / 4) * ((y.I + 3) / 4) << backward) + 31) / 32);
    }
    return 512 * warps;
}

// host: a plan is made in three parts, so that a search over team sizes and tiles pays for each of them once: what follows from the team size, what follows from the rows of a tile, and what
// only the chosen plan needs (32 candidates of 4-256-256-1: 0.5 us, 6.7 with everything made for each of them).
//
// Units, pitches and gradient patches for teams of C CTAs. False: a shape these kernels do not take. `least`: 0, or patches of at least 2 x 1 (1), 2 x 2 (2).
inline bool spread(const b200rl_mlp_shape* sh, int C, int least, Net* out){
    if(sh->n_layers > MAX_LAYERS) return false;
    Net n{};
    n.n_layers = sh->n_layers; n.C = C;
    int I = sh->input_dim;
    long long po = 0, ao = 0;
    for(int l = 0; l < sh->n_layers; l++){
        Layer& y = n.layer[l];
        y.O = sh->dims[l]; y.I = I; y.act = sh->acts[l];
        y.S = ((y.O + C - 1) / C + 3) / 4 * 4; y.P = 4 * (((I + 1 + 3) / 4) | 1); y.K4 = (I + 3) / 4;
        y.poff = po; y.aoff = ao;
        po += (long long)y.O * y.I + y.O; ao += y.O;
        I = y.O;
    }
    n.n_params = (int)po;
    // the smallest patch that gives every thread at most one; shapes that exceed the largest patch (layers of which its edges waste much) take up to four of the smallest: the same sums
    // in registers, twice the reads. 64-320-320-16 by teams of four (541 of the largest, 2,041 of the smallest): 70 us at 1,024 rows, 91 by teams of eight with one patch a
    // thread; 33-240-240-240-7: 87 and 107. Two of the largest do not fit the registers (32-512-512-4 at 256 rows: 102 us, 46 as a launch per pass)
    bool fits = false;
    for(int k = least; k < 4 && !fits; k++){
        const int more_o = k == 1 || k == 2, more_i = k == 2;
        n.patch_o = 1 + more_o; n.patch_i = 1 + more_i; n.n_patches = 0;
        for(int l = 0; l < n.n_layers; l++){
            Layer& y = n.layer[l];
            y.patch_begin = n.n_patches; y.across = (y.I / 4 + 1 + more_i) >> more_i;
            n.n_patches += ((y.S / 4 + more_o) >> more_o) * y.across;
        }
        fits = n.n_patches <= (k == 3 ? MAX_PATCHES_PER_THREAD : 1) * THREADS;
    }
    n.quads = n.n_patches * n.patch_o * 4 * n.patch_i;
    *out = n;
    return fits;
}
// Where everything lies for tiles of R rows (a multiple of four)
inline void place(Net& n, int R, bool keep_pre){
    n.R = R;
    int off = 0, rb = 0;
    for(int l = 0; l < n.n_layers; l++){                                 // what has to start at zero lies together
        Layer& y = n.layer[l];
        y.w = off; off += y.S * y.P;
        y.a = off; off += R * y.P;
        if(l == 0){ n.a_alt = R * y.P; off += R * y.P; }
    }
    n.zero_begin = 0; n.zero_end = off;
    for(int l = 0; l < n.n_layers; l++){
        Layer& y = n.layer[l];
        if(keep_pre){ y.p = off; off += R * y.S; }
        y.g = off; off += R * y.S;
        y.d = off; off += R * y.S;
        if(l > 0 && n.C > 1 && n.C * R * n.layer[l - 1].S > rb) rb = n.C * R * n.layer[l - 1].S;
    }
    off += 4;                                                            // a patch at the end of a row reads the piece behind it (into sums that nobody uses)
    n.rb[0] = off; off += rb;
    n.rb[1] = off; off += rb;
    n.end = off;
}
// What only the kernel reads: tiles, lanes and divisors. `ordered`: sums in the order of parts() and, with the bias column, in as many pieces as a weight row has
inline void complete(Net& n, bool ordered){
    for(int l = 0; l < n.n_layers; l++){
        Layer& y = n.layer[l];
        const int I4 = (y.I + 3) / 4;
        y.fwd_tiles = (n.R / 4) * (y.S / 4); y.bwd_tiles = (n.R / 4) * I4;
        if(ordered){
            y.K4 = y.I / 4 + 1;
            y.fwd_parts = 1 << parts_forward(n, l); y.fwd_shift = lanes_of_parts(y.fwd_tiles, parts_forward(n, l));
            y.bwd_parts = 1 << parts_backward(n, l); y.bwd_shift = lanes_of_parts(y.bwd_tiles, parts_backward(n, l));
        }
        else{ y.fwd_shift = lanes_of_a_tile(y.fwd_tiles, y.K4); y.bwd_shift = l > 0 ? lanes_of_a_tile(y.bwd_tiles, y.S / 4) : 0; }
        y.by_S4 = divisor(y.S / 4); y.by_I4 = divisor(I4); y.by_I = divisor(y.I); y.by_row = divisor(y.I / 4); y.by_owner = divisor(l > 0 ? n.layer[l - 1].S : 1); y.by_across = divisor(y.across);
    }
    n.by_quads = divisor(n.quads); n.by_patches = divisor(n.n_patches); n.by_I0 = divisor(n.layer[0].I);
}

#ifdef __CUDACC__
__device__ __forceinline__ int quotient(int n, Divisor d){ return d.m ? (int)__umulhi((unsigned)n, d.m) : n; }

// threadIdx.x, as a value that the compiler does not take out of the loop around: what a thread does in each of the layers, kept from one minibatch to the next, would
// cost the registers of the gradient sums
__device__ __forceinline__ int thread_here(){ int t = threadIdx.x; asm volatile("" : "+r"(t)); return t; }

// ---- cluster primitives -----------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank(){ uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
template <int C> __device__ __forceinline__ void sync_team(){
    if constexpr(C == 1) __syncthreads();
    else asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t remote(const void* p, int rank){
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void store_remote(float* p, int rank, float v){ asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(remote(p, rank)), "f"(v) : "memory"); }
__device__ __forceinline__ void store_remote(float* p, int rank, float4 v){
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" :: "r"(remote(p, rank)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
template <int C, typename V> __device__ __forceinline__ void store_to(float* p, int rank, V v){
    if constexpr(C == 1) *reinterpret_cast<V*>(p) = v;
    else store_remote(p, rank, v);
}
__device__ __forceinline__ void copy4_async(float* smem, const float* gmem){
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy16_async(float* smem, const float* gmem){
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copies_wait(){ asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory"); }

// activation and its derivative in one evaluation (the derivatives of nn/activation_functions.h:57-85 in terms of the value), on four units
template <typename F> __device__ __forceinline__ float4 each(float4 x, float4& derivative, F f){
    return make_float4(f(x.x, derivative.x), f(x.y, derivative.y), f(x.z, derivative.z), f(x.w, derivative.w));
}
__device__ __forceinline__ float4 activate(float4 x, int act, float4& derivative){
    switch(act){
        case B200RL_ACT_IDENTITY: derivative = make_float4(1.0f, 1.0f, 1.0f, 1.0f); return x;
        case B200RL_ACT_RELU: return each(x, derivative, [](float v, float& d){ d = v > 0.0f ? 1.0f : 0.0f; return v > 0.0f ? v : 0.0f; });
        case B200RL_ACT_TANH: return each(x, derivative, [](float v, float& d){ const float a = tanhf(v); d = 1.0f - a * a; return a; });
        case B200RL_ACT_FAST_TANH: return each(x, derivative, [](float v, float& d){ const float a = fast_tanh_dev(v); d = 1.0f - a * a; return a; });
        default: return each(x, derivative, [](float v, float& d){ const float a = 1.0f / (1.0f + expf(-v)); d = a * (1.0f - a); return a; });
    }
}

// Units beyond a layer's width carry the derivative -0, which no activation has, and their d_pre is 0 whatever stands in their place (targets that were never copied; in the layers below the sums
// of the bias column). A derivative of 0 is not that: it is a factor like any other, so that what is not finite stays so.
constexpr float BEYOND = -0.0f;
__device__ __forceinline__ float d_pre(float d_out, float derivative){ return __float_as_uint(derivative) == 0x80000000u ? 0.0f : d_out * derivative; }

// Once per launch: the weight and input rows start at zero (the padding behind a row and the rows beyond the layer's width stay so), with the
// constant 1 in the bias column of every input row. A CTA-wide barrier, then load_weights.
template <int L>
__device__ __forceinline__ void clear_rows(const Net& n, float* smem){
    for(int i = n.zero_begin + 4 * (int)threadIdx.x; i < n.zero_end; i += 4 * THREADS) *reinterpret_cast<float4*>(smem + i) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncthreads();
#pragma unroll
    for(int l = 0; l < L; l++) if((int)threadIdx.x < n.R) smem[n.layer[l].a + threadIdx.x * n.layer[l].P + n.layer[l].I] = 1.0f;
    if((int)threadIdx.x < n.R) smem[n.layer[0].a + n.a_alt + threadIdx.x * n.layer[0].P + n.layer[0].I] = 1.0f;
}
// this CTA's weight rows of every layer into shared memory by asynchronous copies; the caller waits for them
template <int L>
__device__ __forceinline__ void load_weights(const Net& n, float* smem, const float* params, int rank){
#pragma unroll 1
    for(int l = 0; l < L; l++){
        const Layer& y = n.layer[l];
        const float* W = params + y.poff + (size_t)rank * y.S * y.I;
        float* sw = smem + y.w;
        const int rows = min(y.S, y.O - rank * y.S), S4 = y.S >> 2;
        if((y.I & 3) == 0 && (reinterpret_cast<uintptr_t>(W) & 15u) == 0){
            const int q = y.I >> 2;
#pragma unroll 2
            for(int i = threadIdx.x; i < rows * q; i += THREADS){
                const int o = quotient(i, y.by_row), k = i - o * q;
                copy16_async(sw + ((o & 3) * S4 + (o >> 2)) * y.P + 4 * k, W + 4 * i);
            }
        }
        else{
#pragma unroll 2
            for(int i = threadIdx.x; i < rows * y.I; i += THREADS){
                const int o = quotient(i, y.by_I), k = i - o * y.I;
                copy4_async(sw + ((o & 3) * S4 + (o >> 2)) * y.P + k, W + i);
            }
        }
#pragma unroll 1
        for(int o = threadIdx.x; o < rows; o += THREADS) copy4_async(sw + ((o & 3) * S4 + (o >> 2)) * y.P + y.I, params + y.poff + (size_t)y.O * y.I + rank * y.S + o);
    }
}

// the lanes' parts of a 4 x 4 tile are added: v[0 ... rows - 1] of the tile's rows from `first` on stay with a lane (4, 2, 1 of them). Lanes beyond four per tile all
// get the sums.
struct Share { int tile, part, first, rows, copy, copies; };     // tile of the round, part of the summed index; kept rows; which of `copies` lanes with the same sums this is
__device__ __forceinline__ Share share(int shift, int lane){
    Share s;
    const int per_warp = 32 >> shift;
    s.tile = lane & (per_warp - 1); s.part = lane >> (5 - shift);
    s.first = (shift >= 1 ? (lane >> 3) & 2 : 0) + (shift >= 2 ? (lane >> 3) & 1 : 0);
    s.rows = shift == 0 ? 4 : shift == 1 ? 2 : 1;
    s.copies = shift > 2 ? 1 << (shift - 2) : 1; s.copy = s.part & (s.copies - 1);
    return s;
}
__device__ __forceinline__ void add_parts(float4 (&v)[4], int shift, int lane){
    auto add_to = [](float4& a, float4 b){ a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; };
    auto exchange = [](float4 a, int mask){
        return make_float4(__shfl_xor_sync(0xffffffffu, a.x, mask), __shfl_xor_sync(0xffffffffu, a.y, mask), __shfl_xor_sync(0xffffffffu, a.z, mask), __shfl_xor_sync(0xffffffffu, a.w, mask));
    };
    if(shift >= 1){
        const bool upper = lane & 16;
        const float4 s0 = upper ? v[0] : v[2], s1 = upper ? v[1] : v[3];
        v[0] = upper ? v[2] : v[0]; v[1] = upper ? v[3] : v[1];
        add_to(v[0], exchange(s0, 16)); add_to(v[1], exchange(s1, 16));
    }
    if(shift >= 2){
        const bool upper = lane & 8;
        const float4 s0 = upper ? v[0] : v[1];
        v[0] = upper ? v[1] : v[0];
        add_to(v[0], exchange(s0, 8));
    }
    if(shift >= 3) add_to(v[0], exchange(v[0], 4));
    if(shift >= 4) add_to(v[0], exchange(v[0], 2));
}

// The same with the parts added in their order: of up to two parts there is one (lanes without a part hold zeros); four or more meet in shared memory, 64 bytes for each lane,
// which all have a part of one tile then
__device__ __forceinline__ void add_parts_in_order(float4 (&v)[4], int n_parts, int shift, int lane, int warp, const Share& sh, float* scratch){
    if(n_parts < 4){ add_parts(v, shift, lane); return; }
    float4* rows = reinterpret_cast<float4*>(scratch) + 128 * warp;
#pragma unroll
    for(int i = 0; i < 4; i++) rows[32 * i + lane] = v[i];
    __syncwarp();
    const float4* from = rows + 32 * sh.first + sh.tile;
    v[0] = from[0];
#pragma unroll 4
    for(int p = 1; p < 1 << shift; p++){ const float4 t = from[p << (5 - shift)]; v[0].x += t.x; v[0].y += t.y; v[0].z += t.z; v[0].w += t.w; }
}

// A lane's part of a 4 x 4 tile of a forward product: the pieces first, first + G, ... of four activation and four weight rows. PAIRS: even and odd summed indices apart, their sums added at the
// end (packed multiply-adds; the pairs cost 16 more registers).
template <bool PAIRS>
__device__ __forceinline__ void tile_products(const float4* a, const float4* w, int P4, int S4, int first, int K4, int G, float4 (&v)[4]){
    float2 pair[4][PAIRS ? 4 : 1];
    float acc[4][PAIRS ? 1 : 4];
#pragma unroll
    for(int i = 0; i < 4; i++)
#pragma unroll
        for(int j = 0; j < 4; j++){ if constexpr(PAIRS) pair[i][j] = make_float2(0.0f, 0.0f); else acc[i][j] = 0.0f; }
#pragma unroll 1
    for(int k = first; k < K4; k += G){
        float4 xv[4], wv[4];
#pragma unroll
        for(int i = 0; i < 4; i++) xv[i] = a[i * P4 + k];
#pragma unroll
        for(int j = 0; j < 4; j++) wv[j] = w[j * S4 * P4 + k];
#pragma unroll
        for(int i = 0; i < 4; i++)
#pragma unroll
            for(int j = 0; j < 4; j++){
                if constexpr(PAIRS){
                    pair[i][j] = __ffma2_rn(make_float2(xv[i].x, xv[i].y), make_float2(wv[j].x, wv[j].y), pair[i][j]);
                    pair[i][j] = __ffma2_rn(make_float2(xv[i].z, xv[i].w), make_float2(wv[j].z, wv[j].w), pair[i][j]);
                }
                else{
                    acc[i][j] = fmaf(xv[i].x, wv[j].x, acc[i][j]); acc[i][j] = fmaf(xv[i].y, wv[j].y, acc[i][j]);
                    acc[i][j] = fmaf(xv[i].z, wv[j].z, acc[i][j]); acc[i][j] = fmaf(xv[i].w, wv[j].w, acc[i][j]);
                }
            }
    }
#pragma unroll
    for(int i = 0; i < 4; i++){
        if constexpr(PAIRS) v[i] = make_float4(pair[i][0].x + pair[i][0].y, pair[i][1].x + pair[i][1].y, pair[i][2].x + pair[i][2].y, pair[i][3].x + pair[i][3].y);
        else v[i] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
}

// One layer of the forward pass; `a`: where its input rows lie. The values go into the next layer's input rows of the whole team; after the last layer
// finish(row, first unit, values, derivatives) runs for every row and four units of this CTA. Ends without a barrier.
template <int C, int L, bool KEEP_PRE, bool ORDERED, typename FINISH>
__device__ __forceinline__ void forward_layer(const Net& n, int l, int a_rows, float* smem, int rank, float* scratch, FINISH finish){
    const Layer& y = n.layer[l];
    const int tid = thread_here(), lane = tid & 31, warp = tid >> 5, S4 = y.S >> 2, P4 = y.P >> 2, shift = y.fwd_shift, G = ORDERED ? y.fwd_parts : 1 << shift;
    const Share sh = share(shift, lane);
#pragma unroll 1
    for(int t0 = warp << (5 - shift); t0 < y.fwd_tiles; t0 += WARPS << (5 - shift)){
        const int t = min(t0 + sh.tile, y.fwd_tiles - 1), rg = quotient(t, y.by_S4), og = t - rg * S4;
        const bool mine = t0 + sh.tile < y.fwd_tiles;
        const float4* a = reinterpret_cast<const float4*>(smem + a_rows) + rg * 4 * P4;
        const float4* w = reinterpret_cast<const float4*>(smem + y.w) + og * P4;
        float4 v[4];
        tile_products<ORDERED>(a, w, P4, S4, ORDERED && sh.part >= G ? y.K4 : sh.part, y.K4, G, v);
        if constexpr(ORDERED) add_parts_in_order(v, y.fwd_parts, shift, lane, warp, sh, scratch);
        else add_parts(v, shift, lane);
        if(!mine) continue;                                              // no barrier or exchange below
        float4 bias = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if(!ORDERED && (y.I & 3) == 0){                                  // the bias column is not among the pieces summed
            const float* b = smem + y.w + og * y.P + y.I;
            bias = make_float4(b[0], b[S4 * y.P], b[2 * S4 * y.P], b[3 * S4 * y.P]);
        }
        const int unit = rank * y.S + 4 * og, beyond = unit + 4 - y.O;   // how many of the four units lie beyond the layer
        float* next = nullptr;
        if(l + 1 < L) next = smem + n.layer[l + 1].a + unit;
#pragma unroll 1
        for(int i = 0; i < sh.rows; i++){
            const int r = rg * 4 + sh.first + i;
            const float4 pre = make_float4(v[0].x + bias.x, v[0].y + bias.y, v[0].z + bias.z, v[0].w + bias.w);
            v[0] = v[1]; v[1] = v[2]; v[2] = v[3];
            float4 dv;
            const float4 value = activate(pre, y.act, dv);
            if(beyond > 0){ dv.w = BEYOND; if(beyond > 1) dv.z = BEYOND; if(beyond > 2) dv.y = BEYOND; if(beyond > 3) dv.x = BEYOND; }
            const int at = r * y.S + 4 * og;
            if(sh.copy == 0){
                *reinterpret_cast<float4*>(smem + y.g + at) = dv;
                if constexpr(KEEP_PRE) *reinterpret_cast<float4*>(smem + y.p + at) = pre;
                if(l + 1 == L) finish(r, 4 * og, value, dv);
            }
            if(l + 1 < L){
                float* dst = next + r * n.layer[l + 1].P;
#pragma unroll 1
                for(int c = sh.copy; c < C; c += sh.copies){
                    if(beyond <= 0) store_to<C>(dst, c, value);
                    else{
                        if(beyond < 4) store_to<C>(dst, c, value.x);
                        if(beyond < 3) store_to<C>(dst + 1, c, value.y);
                        if(beyond < 2) store_to<C>(dst + 2, c, value.z);
                    }
                }
            }
        }
    }
}
// pre-activations and outputs of the tile's rows that lie in [keep_from, rows) to the activation arenas (row - keep_from of `stride` rows per
// layer). Called once all layers are done: a global store in front of a cluster barrier would make the barrier wait for it.
template <int L>
__device__ __forceinline__ void store_activations(const Net& n, const float* smem, const float* last_out, int rank, int row0, int rows, int keep_from, int stride, float* pre, float* out){
    if(row0 + n.R <= keep_from) return;
#pragma unroll 1
    for(int l = 0; l < L; l++){
        const Layer& y = n.layer[l];
        const int S4 = y.S >> 2, count = n.R * S4;
        const size_t base = (size_t)y.aoff * stride;
        const bool quads = (y.O & 3) == 0 && (base & 3) == 0 && ((reinterpret_cast<uintptr_t>(pre) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
#pragma unroll 2
        for(int i = threadIdx.x; i < count; i += THREADS){
            const int r = quotient(i, y.by_S4), og = i - r * S4, unit = rank * y.S + 4 * og, row = row0 + r;
            if(unit >= y.O || row >= rows || row < keep_from) continue;
            const size_t at = base + (size_t)(row - keep_from) * y.O + unit;
            const float* p = smem + y.p + 4 * i;
            const float* o = l + 1 < L ? smem + n.layer[l + 1].a + r * n.layer[l + 1].P + unit : last_out + 4 * i;
            if(quads){ *reinterpret_cast<float4*>(pre + at) = *reinterpret_cast<const float4*>(p); *reinterpret_cast<float4*>(out + at) = *reinterpret_cast<const float4*>(o); }
            else for(int k = 0; k < min(4, y.O - unit); k++){ pre[at + k] = p[k]; out[at + k] = o[k]; }
        }
    }
}

// Input gradient of layer l > 0 from its d_pre (own units), then d_pre of layer l - 1 (own units): in teams of several CTAs by way of the owners of the inputs, through
// one of two exchange buffers (`turn` alternates).
template <int C, bool ORDERED>
__device__ __forceinline__ void backward_layer(const Net& n, int l, float* smem, int rank, int turn, float* scratch){
    const Layer& y = n.layer[l];
    const Layer& z = n.layer[l - 1];
    float* rb = smem + n.rb[turn];
    const int tid = thread_here(), lane = tid & 31, warp = tid >> 5, I4 = (y.I + 3) >> 2, S4 = y.S >> 2, P4 = y.P >> 2, shift = y.bwd_shift, G = ORDERED ? y.bwd_parts : 1 << shift;
    const Share sh = share(shift, lane);
    auto below = [&](int at, float4 v){
        const float4 dv = *reinterpret_cast<const float4*>(smem + z.g + at);
        *reinterpret_cast<float4*>(smem + z.d + at) = make_float4(d_pre(v.x, dv.x), d_pre(v.y, dv.y), d_pre(v.z, dv.z), d_pre(v.w, dv.w));
    };
#pragma unroll 1
    for(int t0 = warp << (5 - shift); t0 < y.bwd_tiles; t0 += WARPS << (5 - shift)){
        const int t = min(t0 + sh.tile, y.bwd_tiles - 1), rg = quotient(t, y.by_I4), i4 = t - rg * I4;
        const bool mine = t0 + sh.tile < y.bwd_tiles;
        const float4* d = reinterpret_cast<const float4*>(smem + y.d) + rg * 4 * S4;
        const float4* w = reinterpret_cast<const float4*>(smem + y.w) + i4;
        float4 v[4];
#pragma unroll
        for(int i = 0; i < 4; i++) v[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 1
        for(int o4 = ORDERED && sh.part >= G ? S4 : sh.part; o4 < S4; o4 += G){
            float4 dv[4], wv[4];
#pragma unroll
            for(int i = 0; i < 4; i++) dv[i] = d[i * S4 + o4];
#pragma unroll
            for(int q = 0; q < 4; q++) wv[q] = w[(q * S4 + o4) * P4];
#pragma unroll
            for(int i = 0; i < 4; i++){
                const float e[4] = {dv[i].x, dv[i].y, dv[i].z, dv[i].w};
#pragma unroll
                for(int q = 0; q < 4; q++) v[i] = make_float4(fmaf(e[q], wv[q].x, v[i].x), fmaf(e[q], wv[q].y, v[i].y), fmaf(e[q], wv[q].z, v[i].z), fmaf(e[q], wv[q].w, v[i].w));
            }
        }
        if constexpr(ORDERED) add_parts_in_order(v, y.bwd_parts, shift, lane, warp, sh, scratch);
        else add_parts(v, shift, lane);
        if(!mine || sh.copy != 0) continue;
        const int owner = C == 1 ? 0 : quotient(i4 * 4, y.by_owner), col = i4 * 4 - owner * z.S;
#pragma unroll 1
        for(int i = 0; i < sh.rows; i++){
            const int r = rg * 4 + sh.first + i;
            if constexpr(C == 1) below(r * z.S + col, v[0]);
            else store_remote(rb + (rank * n.R + r) * z.S + col, owner, v[0]);
            v[0] = v[1]; v[1] = v[2]; v[2] = v[3];
        }
    }
    if constexpr(C > 1){
        sync_team<C>();
        const int count = n.R * z.S;
#pragma unroll 1
        for(int at = 4 * threadIdx.x; at < count; at += 4 * THREADS){
            float4 v = *reinterpret_cast<const float4*>(rb + at);
#pragma unroll
            for(int p = 1; p < C; p++){ const float4 t = *reinterpret_cast<const float4*>(rb + p * count + at); v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w; }
            below(at, v);
        }
    }
    __syncthreads();
}

// ---- parameter gradients: thread t owns the patches t, t + THREADS, ... (up to four) of the CTA's weight rows ------------------------------
struct Patch { int d, a, pitch, alt; };                 // pitch: of the d_pre rows in the low half, of the input rows in the high half; alt: distance of the other input buffer
// layer, first output quad and first input quad of a patch; patches ascend over the layers
template <int L>
__device__ __forceinline__ void locate(const Net& n, int at, int& l, int& o4, int& i4){
    l = 0;
#pragma unroll
    for(int k = 1; k < L; k++) if(at >= n.layer[k].patch_begin) l = k;
    int begin = n.layer[0].patch_begin, across = n.layer[0].across; Divisor by = n.layer[0].by_across;
#pragma unroll
    for(int k = 1; k < L; k++) if(l == k){ begin = n.layer[k].patch_begin; across = n.layer[k].across; by = n.layer[k].by_across; }
    const int o = quotient(at - begin, by);
    o4 = o * n.patch_o; i4 = (at - begin - o * across) * n.patch_i;
}
template <int L>
__device__ __forceinline__ Patch patch(const Net& n, int at){
    Patch p{0, 0, 0, 0};
    if(at >= n.n_patches) return p;
    int l, o4, i4;
    locate<L>(n, at, l, o4, i4);
#pragma unroll
    for(int k = 0; k < L; k++) if(l == k){ const Layer& y = n.layer[k]; p.d = y.d + 4 * o4; p.a = y.a + 4 * i4; p.pitch = y.S | (y.P << 16); p.alt = k == 0 ? n.a_alt : 0; }
    return p;
}
// a thread's sums: N patches of PO x PI pieces
template <int N, int PO, int PI> struct Sums { float4 v[N][4 * PO][PI]; };
template <int N, int PO, int PI>
__device__ __forceinline__ void clear_sums(Sums<N, PO, PI>& acc){
#pragma unroll
    for(int k = 0; k < N; k++)
#pragma unroll
        for(int o = 0; o < 4 * PO; o++)
#pragma unroll
            for(int i = 0; i < PI; i++) acc.v[k][o][i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}
// `other`: the first layer's rows lie in its second buffer
template <int N, int PO, int PI>
__device__ __forceinline__ void accumulate_gradients(const Net& n, const float* smem, const Patch (&p)[N], Sums<N, PO, PI>& acc, bool other){
#pragma unroll
    for(int k = 0; k < N; k++){
        if(k * THREADS + (int)threadIdx.x >= n.n_patches) continue;
        const float* d = smem + p[k].d; const float* a = smem + p[k].a + (other ? p[k].alt : 0);
        const int ds = p[k].pitch & 0xFFFF, as = p[k].pitch >> 16;
#pragma unroll (PO * PI == 1 ? 4 : PO * PI == 2 ? 2 : 1)
        for(int r = 0; r < n.R; r++){
            float4 dv[PO], av[PI];
#pragma unroll
            for(int o = 0; o < PO; o++) dv[o] = *reinterpret_cast<const float4*>(d + r * ds + 4 * o);
#pragma unroll
            for(int i = 0; i < PI; i++) av[i] = *reinterpret_cast<const float4*>(a + r * as + 4 * i);
#pragma unroll
            for(int o = 0; o < PO; o++){
                const float e[4] = {dv[o].x, dv[o].y, dv[o].z, dv[o].w};
#pragma unroll
                for(int q = 0; q < 4; q++)
#pragma unroll
                    for(int i = 0; i < PI; i++){
                        float4& s = acc.v[k][4 * o + q][i];
                        s.x = fmaf(e[q], av[i].x, s.x); s.y = fmaf(e[q], av[i].y, s.y); s.z = fmaf(e[q], av[i].z, s.z); s.w = fmaf(e[q], av[i].w, s.w);
                    }
            }
        }
    }
}
// gradient sums of one CTA of a team: [output of the patch][piece of the inputs][patch] x 16 bytes, so that the lanes of a warp write neighbouring pieces
template <int N, int PO, int PI>
__device__ __forceinline__ void store_gradients(const Net& n, float4* partial, int rank, const Sums<N, PO, PI>& acc){
#pragma unroll
    for(int k = 0; k < N; k++){
        const int at = k * THREADS + (int)threadIdx.x;
        if(at >= n.n_patches) continue;
        float4* dst = partial + (size_t)rank * n.quads + at;
#pragma unroll
        for(int o = 0; o < 4 * PO; o++)
#pragma unroll
            for(int i = 0; i < PI; i++) __stcg(dst + (o * PI + i) * n.n_patches, acc.v[k][o][i]);
    }
}
// arena index of component `comp` of quad `u` (= (CTA of the team, output of the patch, piece of the inputs, patch)); -1 where the patch reaches beyond the layer
template <int L>
__device__ __forceinline__ int arena_index(const Net& n, int u, int comp){
    const int rank = quotient(u, n.by_quads), rest = u - rank * n.quads, j = quotient(rest, n.by_patches), at = rest - j * n.n_patches;
    int l, o4, i4, index = -1;
    locate<L>(n, at, l, o4, i4);
    const int out = n.patch_i == 2 ? j >> 1 : j, piece = n.patch_i == 2 ? j & 1 : 0;
#pragma unroll
    for(int k = 0; k < L; k++) if(l == k){
        const Layer& y = n.layer[k];
        const int unit = o4 * 4 + out, o = rank * y.S + unit, i = (i4 + piece) * 4 + comp;
        if(unit < y.S && o < y.O && i <= y.I) index = (int)y.poff + (i < y.I ? o * y.I + i : y.O * y.I + o);
    }
    return index;
}

// shared-memory offset of the four weights that quad `u` of a team of one CTA holds the gradients of; -1 where the patch reaches beyond the layer
template <int L>
__device__ __forceinline__ int weights_of_quad(const Net& n, int u){
    const int j = quotient(u, n.by_patches), at = u - j * n.n_patches, out = n.patch_i == 2 ? j >> 1 : j, piece = n.patch_i == 2 ? j & 1 : 0;
    int l, o4, i4, off = -1;
    locate<L>(n, at, l, o4, i4);
#pragma unroll
    for(int k = 0; k < L; k++) if(l == k){
        const Layer& y = n.layer[k];
        const int unit = o4 * 4 + out, i = (i4 + piece) * 4;
        if(unit < y.O && i <= y.I) off = y.w + ((unit & 3) * (y.S >> 2) + (unit >> 2)) * y.P + i;
    }
    return off;
}

static __device__ __noinline__ float adam_bias_correction(float beta, uint32_t age){
    const float pw = (float)pow((double)beta, (double)(float)age);      // rounded to float once, as the per-arena kernel does
    return 1.0f / (1.0f - pw);
}
// utils/polyak/operations_generic.h:72-88 and nn/optimizers/adam/instance/operations_generic.h:25-61, every intermediate rounded like the reference's
__device__ __forceinline__ float adam_update(float p, float g, float& m, float& v, const b200rl_adam_hyper& h, float c1, float c2){
    m = __fadd_rn(__fmul_rn(h.beta_1, m), __fmul_rn(1.0f - h.beta_1, g));
    v = __fadd_rn(__fmul_rn(h.beta_2, v), __fmul_rn(__fmul_rn(1.0f - h.beta_2, g), g));
    const float pre_sqrt = fmaxf(__fmul_rn(v, c2), h.epsilon_sqrt);
    return __fsub_rn(p, __fdiv_rn(__fmul_rn(__fmul_rn(h.alpha, c1), m), __fadd_rn(__fsqrt_rn(pre_sqrt), h.epsilon)));
}

// All CTAs of the grid share out the parameters: `lanes` threads per quad (a power of two from 4 on) add the teams' sums (thread y of a quad takes teams y, y + lanes, ... ascending,
// then they are added pairwise, neighbours first or, ORDERED, halves first: a fixed order), the first four each finish one parameter. Lanes of neighbouring quads lie side by side.
struct Owner { int quad, part, step; };
__device__ __forceinline__ Owner owner(int lanes, int cta, int ctas){
    const int bits = __popc(lanes - 1), per_warp = 32 >> bits, lane = threadIdx.x & 31;
    return Owner{(cta * WARPS + ((int)threadIdx.x >> 5)) * per_warp + (lane & (per_warp - 1)), lane >> (5 - bits), ctas * WARPS * per_warp};
}
template <bool ORDERED>
__device__ __forceinline__ float sum_of_teams(const float4* partial, int u, int quads, int teams, int part, int lanes){
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if(u < quads){
        const float4* src = partial + u;
        constexpr int AHEAD = ORDERED ? 10 : 8;                          // loads under way; ten are the 74 teams of half the SMs over eight lanes
        for(int t = part; t < teams; t += AHEAD * lanes){
            float4 v[AHEAD];
#pragma unroll
            for(int k = 0; k < AHEAD; k++) v[k] = t + k * lanes < teams ? __ldcg(src + (size_t)(t + k * lanes) * quads) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for(int k = 0; k < AHEAD; k++){ s.x += v[k].x; s.y += v[k].y; s.z += v[k].z; s.w += v[k].w; }
        }
    }
    auto add = [&](int o){
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o); s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        s.z += __shfl_xor_sync(0xffffffffu, s.z, o); s.w += __shfl_xor_sync(0xffffffffu, s.w, o);
    };
    const int least = 32 >> __popc(lanes - 1);
    if(ORDERED) for(int o = 16; o >= least; o >>= 1) add(o);
    else for(int o = least; o < 32; o <<= 1) add(o);
    return part == 0 ? s.x : part == 1 ? s.y : part == 2 ? s.z : s.w;
}
// sink(arena index, gradient, what prefetch(arena index) returned before the sums were loaded)
template <int C, int L, typename PREFETCH, typename SINK>
__device__ __forceinline__ void reduce_gradients(const Net& n, const float4* partial, int teams, int cta, int ctas, int lanes, PREFETCH prefetch, SINK sink){
    const int quads = C * n.quads;
    const Owner me = owner(lanes, cta, ctas);
    const int first = me.quad - (threadIdx.x & 31 & ((32 / lanes) - 1));                 // the same for all lanes of a warp
    for(int u0 = first; u0 < quads; u0 += me.step){
        const int u = u0 + me.quad - first, index = u < quads && me.part < 4 ? arena_index<L>(n, u, me.part) : -1;
        const auto early = prefetch(index);
        const float g = sum_of_teams<false>(partial, u, quads, teams, me.part, lanes);
        if(index >= 0) sink(index, g, early);
    }
}
#endif

}}  // namespace b200rl::team
