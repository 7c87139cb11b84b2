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
//   - parameter gradients: 4 x 4 patches per thread, in registers over all row tiles of the launch. The bias is column I of the weight row
//     (its input is the constant 1 in column I of the activation rows), so it needs no code of its own in either direction.
// Every product runs as 4 x 4 register tiles on packed multiply-adds with 16-byte shared-memory operands; where a product has fewer tiles than
// the CTA has threads, the summed index is split over thread groups and the parts are added in group order.
// Teams write their gradient sums to scratch memory; after a grid-wide barrier all CTAs share out the parameters, add the teams' sums in a fixed
// order and apply the optimizer step.
//
// Loops over elements and layers stay rolled: a minibatch walks the whole code once, and what does not fit the instruction caches is fetched anew for every one of
// them (PPO epoch kernel 220 -> 108 KB of code: 27-64-64-8, 2,048 rows 22.4 -> 20.3 us per minibatch).
#pragma once
#include "common.cuh"

namespace b200rl { namespace team {

// 256 threads: a tile of a few rows is bound by the latency of its phases and by instruction issue (address arithmetic around short products), which
// more warps only repeat. Measured with 512: 64-wide networks 12.8 -> 15.7 us per step at batch 512, 18.1 -> 19.8 us at batch 2,048.
constexpr int THREADS = 256, MAX_LAYERS = 4, MAX_TILES_PER_THREAD = 8;

// quotient by a divisor known on the host (both below 2^16): one multiplication instead of a division's ~40 instructions, which on the path of a
// few microseconds per layer would be most of the time
struct Divisor { unsigned m; };
inline Divisor divisor(int d){ return Divisor{d <= 1 ? 0u : (unsigned)((0x100000000ull + (unsigned)d - 1) / (unsigned)d)}; }

struct Layer {
    int O, I, act;
    int S;                      // units per CTA (multiple of 4)
    int P;                      // pitch of weight and activation rows in floats: I + 1 rounded up to four, an odd number of 16-byte pieces
    int K4;                     // 16-byte pieces of a row that hold data
    long long poff, aoff;       // offset in the parameter arena (weights, then bias), in the activation arenas (x batch)
    int w, a, p, g, d;          // shared-memory offsets (floats): weight rows [S][P], input rows [R][P]; [R][S]: pre-activations, activation derivatives, d_pre
    int fwd_threads, fwd_groups, bwd_threads, bwd_groups;      // threads of one pass over all tiles, groups that share out the summed index
    int tile_begin, tiles_i;    // gradient patches: first index of this layer, patches along the inputs
    Divisor by_S, by_S4, by_fwd, by_bwd, by_I, by_row, by_I4, by_tiles_i;
};
struct Net {
    int n_layers, R, n_tiles, n_params;      // n_tiles: gradient patches per CTA
    Divisor by_tiles, by_I0;
    int zero_begin, zero_end;                // weight and input rows of all layers (offsets, multiples of four floats)
    int rb[2];                               // exchange buffers (offsets); rb_floats each
    int end;                                 // end of the network's shared memory (floats)
    Layer layer[MAX_LAYERS];
};

// host: lays a network out for teams of C CTAs and R rows per tile, from shared-memory offset `base` on. False: a shape these kernels do not take.
inline bool plan(const b200rl_mlp_shape* sh, int C, int R, int base, Net* out){
    if(sh->n_layers > MAX_LAYERS) return false;
    Net n{};
    n.n_layers = sh->n_layers; n.R = R;
    int I = sh->input_dim, off = base, rb = 0;
    long long po = 0, ao = 0;
    for(int l = 0, i = sh->input_dim; l < sh->n_layers; i = sh->dims[l], l++){            // what has to start at zero lies together
        const int S = ((sh->dims[l] + C - 1) / C + 3) / 4 * 4, P = 4 * (((i + 1 + 3) / 4) | 1);
        n.layer[l].w = off; off += S * P;
        n.layer[l].a = off; off += R * P;
    }
    n.zero_begin = base; n.zero_end = off;
    for(int l = 0; l < sh->n_layers; l++){
        Layer& y = n.layer[l];
        y.O = sh->dims[l]; y.I = I; y.act = sh->acts[l];
        y.S = ((y.O + C - 1) / C + 3) / 4 * 4;
        y.K4 = (I + 1 + 3) / 4;
        y.P = 4 * (y.K4 | 1);
        y.poff = po; y.aoff = ao;
        po += (long long)y.O * I + y.O; ao += y.O;
        y.p = off; off += R * y.S;
        y.g = off; off += R * y.S;
        y.d = off; off += R * y.S;
        y.fwd_threads = (R / 4) * (y.S / 4);
        y.fwd_groups = 1;
        while(2 * y.fwd_groups * y.fwd_threads <= THREADS && 4 * y.fwd_groups <= y.K4) y.fwd_groups *= 2;
        if(y.fwd_groups * R * y.S > rb) rb = y.fwd_groups * R * y.S;
        if(l > 0){
            y.bwd_threads = (R / 4) * ((I + 3) / 4);
            y.bwd_groups = 1;
            while(2 * y.bwd_groups * y.bwd_threads <= THREADS && 2 * y.bwd_groups <= y.S / 4) y.bwd_groups *= 2;
            const int need = C * y.bwd_groups * R * n.layer[l - 1].S;
            if(need > rb) rb = need;
        }
        y.tile_begin = n.n_tiles; y.tiles_i = y.K4;
        n.n_tiles += (y.S / 4) * y.tiles_i;
        y.by_S = divisor(y.S); y.by_S4 = divisor(y.S / 4); y.by_fwd = divisor(y.fwd_threads); y.by_bwd = divisor(l > 0 ? y.bwd_threads : 1); y.by_I4 = divisor((I + 3) / 4);
        y.by_tiles_i = divisor(y.tiles_i); y.by_I = divisor(I); y.by_row = divisor(I / 4);
        I = y.O;
    }
    if(n.n_tiles > MAX_TILES_PER_THREAD * THREADS || off % 4 != 0) return false;
    n.n_params = (int)po;
    n.by_tiles = divisor(n.n_tiles); n.by_I0 = divisor(sh->input_dim);
    n.rb[0] = off; off += rb;
    n.rb[1] = off; off += rb;
    n.end = off;
    *out = n;
    return true;
}

#ifdef __CUDACC__
__device__ __forceinline__ int quotient(int n, Divisor d){ return d.m ? (int)__umulhi((unsigned)n, d.m) : n; }

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
template <int C, typename T> __device__ __forceinline__ void store_to(float* p, int rank, T v){
    if constexpr(C == 1) *reinterpret_cast<T*>(p) = v;
    else store_remote(p, rank, v);
}
__device__ __forceinline__ void copy4_async(float* smem, const float* gmem){
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy16_async(float* smem, const float* gmem){
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copies_wait(){ asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory"); }

// activation and its derivative in one evaluation (the derivatives of nn/activation_functions.h:57-85 in terms of the value)
__device__ __forceinline__ float activate(float x, int act, float& derivative){
    switch(act){
        case B200RL_ACT_IDENTITY: derivative = 1.0f; return x;
        case B200RL_ACT_RELU: derivative = x > 0.0f ? 1.0f : 0.0f; return x > 0.0f ? x : 0.0f;
        case B200RL_ACT_TANH: { const float a = tanhf(x); derivative = 1.0f - a * a; return a; }
        case B200RL_ACT_FAST_TANH: { const float a = fast_tanh_dev(x); derivative = 1.0f - a * a; return a; }
        default: { const float a = 1.0f / (1.0f + expf(-x)); derivative = a * (1.0f - a); return a; }
    }
}

// Once per launch: the weight and input rows start at zero (the padding behind a row and the rows beyond the layer's width stay so), with the
// constant 1 in the bias column of every input row. A CTA-wide barrier, then load_weights.
template <int L>
__device__ __forceinline__ void clear_rows(const Net& n, float* smem){
    for(int i = n.zero_begin + 4 * (int)threadIdx.x; i < n.zero_end; i += 4 * THREADS) *reinterpret_cast<float4*>(smem + i) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for(int i = threadIdx.x; i < n.R * n.layer[L - 1].S; i += THREADS) smem[n.layer[L - 1].d + i] = 0.0f;      // columns beyond the output stay zero
    __syncthreads();
#pragma unroll
    for(int l = 0; l < L; l++) if((int)threadIdx.x < n.R) smem[n.layer[l].a + threadIdx.x * n.layer[l].P + n.layer[l].I] = 1.0f;
}
// this CTA's weight rows of every layer into shared memory by asynchronous copies; the caller waits for them
template <int L>
__device__ __forceinline__ void load_weights(const Net& n, float* smem, const float* params, int rank){
#pragma unroll 1
    for(int l = 0; l < L; l++){
        const Layer& y = n.layer[l];
        const float* W = params + y.poff + (size_t)rank * y.S * y.I;
        float* sw = smem + y.w;
        const int rows = min(y.S, y.O - rank * y.S);
        if((y.I & 3) == 0 && (reinterpret_cast<uintptr_t>(W) & 15u) == 0){
            const int q = y.I >> 2;
#pragma unroll 2
            for(int i = threadIdx.x; i < rows * q; i += THREADS) copy16_async(sw + 4 * i + quotient(i, y.by_row) * (y.P - y.I), W + 4 * i);
        }
        else{
#pragma unroll 2
            for(int i = threadIdx.x; i < rows * y.I; i += THREADS) copy4_async(sw + i + quotient(i, y.by_I) * (y.P - y.I), W + i);
        }
#pragma unroll 1
        for(int o = threadIdx.x; o < rows; o += THREADS) copy4_async(sw + o * y.P + y.I, params + y.poff + (size_t)y.O * y.I + rank * y.S + o);
    }
}

// partial sums of one layer's pre-activations for the CTA's units: exchange buffer [group][R][S]
__device__ __forceinline__ void forward_products(const Net& n, const Layer& y, const float* smem, float* rb){
    const int g = quotient(threadIdx.x, y.by_fwd), S4 = y.S >> 2, P4 = y.P >> 2;
    if(g >= y.fwd_groups) return;
    for(int t = threadIdx.x - g * y.fwd_threads; t < y.fwd_threads; t += THREADS){           // more than one round only with a single group
        const int rg = quotient(t, y.by_S4), og = t - rg * S4;      // unit og + S4 j: the weight rows of consecutive lanes lie in different banks
        const float4* a = reinterpret_cast<const float4*>(smem + y.a) + rg * 4 * P4;
        const float4* w = reinterpret_cast<const float4*>(smem + y.w) + og * P4;
        float2 acc[4][4];
#pragma unroll
        for(int i = 0; i < 4; i++)
#pragma unroll
            for(int j = 0; j < 4; j++) acc[i][j] = make_float2(0.0f, 0.0f);
#pragma unroll 2
        for(int k = g; k < y.K4; k += y.fwd_groups){
            float4 xv[4], wv[4];
#pragma unroll
            for(int i = 0; i < 4; i++) xv[i] = a[i * P4 + k];
#pragma unroll
            for(int j = 0; j < 4; j++) wv[j] = w[j * S4 * P4 + k];
#pragma unroll
            for(int i = 0; i < 4; i++)
#pragma unroll
                for(int j = 0; j < 4; j++){
                    acc[i][j] = __ffma2_rn(make_float2(xv[i].x, xv[i].y), make_float2(wv[j].x, wv[j].y), acc[i][j]);
                    acc[i][j] = __ffma2_rn(make_float2(xv[i].z, xv[i].w), make_float2(wv[j].z, wv[j].w), acc[i][j]);
                }
        }
        float* dst = rb + (g * n.R + rg * 4) * y.S + og;
#pragma unroll
        for(int i = 0; i < 4; i++)
#pragma unroll
            for(int j = 0; j < 4; j++) dst[i * y.S + j * S4] = acc[i][j].x + acc[i][j].y;
    }
}

// One layer of the forward pass. epilogue(r, unit, index in [R][S], value, derivative) runs once per row and own unit; the value goes into the
// next layer's input rows of the whole team (unless this is the last layer). Ends without a barrier.
template <int C, int L, typename EPILOGUE>
__device__ __forceinline__ void forward_layer(const Net& n, int l, float* smem, int rank, EPILOGUE epilogue){
    const Layer& y = n.layer[l];
    float* rb = smem + n.rb[0];
    forward_products(n, y, smem, rb);
    __syncthreads();
    const int count = n.R * y.S, next_a = l + 1 < L ? n.layer[l + 1].a : 0, next_p = l + 1 < L ? n.layer[l + 1].P : 0;
#pragma unroll 1
    for(int idx = threadIdx.x; idx < count; idx += THREADS){
        const int r = quotient(idx, y.by_S), o = idx - r * y.S, unit = rank * y.S + o;
        float v = rb[idx], dv;
#pragma unroll 4
        for(int g = 1; g < y.fwd_groups; g++) v += rb[g * count + idx];
        const float value = activate(v, y.act, dv);
        if(unit >= y.O) dv = 0.0f;
        smem[y.g + idx] = dv;
        smem[y.p + idx] = v;
        if(unit < y.O){
            if(l + 1 < L){
                float* dst = smem + next_a + r * next_p + unit;
                if constexpr(C == 1) *dst = value;
                else{
#pragma unroll
                    for(int c = 0; c < C; c++) store_remote(dst, c, value);
                }
            }
            epilogue(r, unit, idx, value, dv);
        }
    }
}
// pre-activations and outputs of the tile's rows that lie in [keep_from, rows) to the activation arenas (row - keep_from of `stride` rows per
// layer). Called once all layers are done: a global store in front of a cluster barrier would make the barrier wait for it.
template <int L>
__device__ __forceinline__ void store_activations(const Net& n, const float* smem, const float* last_out, int rank, int row0, int rows, int keep_from, int stride, float* pre, float* out){
    if(row0 + n.R <= keep_from) return;
#pragma unroll
    for(int l = 0; l < L; l++){
        const Layer& y = n.layer[l];
        const int count = n.R * y.S;
        const size_t base = (size_t)y.aoff * stride;
        for(int idx = threadIdx.x; idx < count; idx += THREADS){
            const int r = quotient(idx, y.by_S), unit = rank * y.S + idx - r * y.S, row = row0 + r;
            if(unit >= y.O || row >= rows || row < keep_from) continue;
            const size_t at = base + (size_t)(row - keep_from) * y.O + unit;
            pre[at] = smem[y.p + idx];
            out[at] = l + 1 < L ? smem[n.layer[l + 1].a + r * n.layer[l + 1].P + unit] : last_out[idx];
        }
    }
}

// Input gradient of layer l > 0 from its d_pre (own units): partial sums to the owners of the inputs, then d_pre of layer l - 1 (own units).
// `turn` alternates between the two exchange buffers.
template <int C>
__device__ __forceinline__ void backward_layer(const Net& n, int l, float* smem, int rank, int turn){
    const Layer& y = n.layer[l];
    const Layer& z = n.layer[l - 1];
    float* rb = smem + n.rb[turn];
    const int g = quotient(threadIdx.x, y.by_bwd), I4 = (y.I + 3) >> 2, S4 = y.S >> 2, P4 = y.P >> 2;
    for(int t = g < y.bwd_groups ? threadIdx.x - g * y.bwd_threads : y.bwd_threads; t < y.bwd_threads; t += THREADS){
        const int rg = quotient(t, y.by_I4), i4 = t - rg * I4;
        const float4* d = reinterpret_cast<const float4*>(smem + y.d) + rg * 4 * S4;
        const float4* w = reinterpret_cast<const float4*>(smem + y.w) + i4;
        float2 acc[4][2];
#pragma unroll
        for(int i = 0; i < 4; i++){ acc[i][0] = make_float2(0.0f, 0.0f); acc[i][1] = make_float2(0.0f, 0.0f); }
#pragma unroll 2
        for(int o4 = g; o4 < S4; o4 += y.bwd_groups){
            float4 dv[4], wv[4];
#pragma unroll
            for(int i = 0; i < 4; i++) dv[i] = d[i * S4 + o4];
#pragma unroll
            for(int q = 0; q < 4; q++) wv[q] = w[(o4 * 4 + q) * P4];
#pragma unroll
            for(int i = 0; i < 4; i++){
                const float e[4] = {dv[i].x, dv[i].y, dv[i].z, dv[i].w};
#pragma unroll
                for(int q = 0; q < 4; q++){
                    acc[i][0] = __ffma2_rn(make_float2(e[q], e[q]), make_float2(wv[q].x, wv[q].y), acc[i][0]);
                    acc[i][1] = __ffma2_rn(make_float2(e[q], e[q]), make_float2(wv[q].z, wv[q].w), acc[i][1]);
                }
            }
        }
        const int owner = C == 1 ? 0 : quotient(i4 * 4, z.by_S), col = i4 * 4 - owner * z.S;
        float* dst = rb + ((rank * y.bwd_groups + g) * n.R + rg * 4) * z.S + col;
#pragma unroll
        for(int i = 0; i < 4; i++) store_to<C>(dst + i * z.S, owner, make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y));
    }
    sync_team<C>();
    const int count = n.R * z.S, parts = C * y.bwd_groups;
#pragma unroll 1
    for(int idx = threadIdx.x; idx < count; idx += THREADS){
        const float dv = smem[z.g + idx];
        float v = 0.0f;
#pragma unroll 4
        for(int p = 0; p < parts; p++) v += rb[p * count + idx];
        smem[z.d + idx] = dv != 0.0f ? v * dv : 0.0f;             // units beyond the layer's width have derivative 0
    }
    __syncthreads();
}

// ---- parameter gradients: thread t owns the patches t, t + THREADS, ... of the CTA's weight rows -------------------------------------------
struct Patch { int d, a, pitch; };                      // pitch: of the d_pre rows in the low half, of the input rows in the high half
// layer, output quad and input quad of a patch; tiles ascend over the layers
template <int L>
__device__ __forceinline__ void locate(const Net& n, int tile, int& l, int& o4, int& i4){
    l = 0;
#pragma unroll
    for(int k = 1; k < L; k++) if(tile >= n.layer[k].tile_begin) l = k;
    int begin = n.layer[0].tile_begin, tiles_i = n.layer[0].tiles_i; Divisor by = n.layer[0].by_tiles_i;
#pragma unroll
    for(int k = 1; k < L; k++) if(l == k){ begin = n.layer[k].tile_begin; tiles_i = n.layer[k].tiles_i; by = n.layer[k].by_tiles_i; }
    o4 = quotient(tile - begin, by); i4 = tile - begin - o4 * tiles_i;
}
template <int L>
__device__ __forceinline__ Patch patch(const Net& n, int tile){
    Patch p{0, 0, 0};
    if(tile >= n.n_tiles) return p;
    int l, o4, i4;
    locate<L>(n, tile, l, o4, i4);
#pragma unroll
    for(int k = 0; k < L; k++) if(l == k){ const Layer& y = n.layer[k]; p.d = y.d + 4 * o4; p.a = y.a + 4 * i4; p.pitch = y.S | (y.P << 16); }
    return p;
}
template <int TPT>
__device__ __forceinline__ void accumulate_gradients(const Net& n, const float* smem, const Patch (&p)[TPT], float2 (&acc)[TPT][4][2]){
#pragma unroll
    for(int k = 0; k < TPT; k++){
        if(k * THREADS + (int)threadIdx.x >= n.n_tiles) continue;
        const float* d = smem + p[k].d; const float* a = smem + p[k].a;
        const int ds = p[k].pitch & 0xFFFF, as = p[k].pitch >> 16;
#pragma unroll 4
        for(int r = 0; r < n.R; r++){
            const float4 dv = *reinterpret_cast<const float4*>(d + r * ds), av = *reinterpret_cast<const float4*>(a + r * as);
            const float e[4] = {dv.x, dv.y, dv.z, dv.w};
#pragma unroll
            for(int i = 0; i < 4; i++){
                acc[k][i][0] = __ffma2_rn(make_float2(e[i], e[i]), make_float2(av.x, av.y), acc[k][i][0]);
                acc[k][i][1] = __ffma2_rn(make_float2(e[i], e[i]), make_float2(av.z, av.w), acc[k][i][1]);
            }
        }
    }
}
// gradient sums of one team: [CTA of the team][patch][output of the patch] x 16 bytes
template <int C, int TPT>
__device__ __forceinline__ void store_gradients(const Net& n, float4* partial, int rank, const float2 (&acc)[TPT][4][2]){
#pragma unroll
    for(int k = 0; k < TPT; k++){
        const int tile = k * THREADS + (int)threadIdx.x;
        if(tile >= n.n_tiles) continue;
        float4* dst = partial + ((size_t)rank * n.n_tiles + tile) * 4;
#pragma unroll
        for(int i = 0; i < 4; i++) __stcg(dst + i, make_float4(acc[k][i][0].x, acc[k][i][0].y, acc[k][i][1].x, acc[k][i][1].y));
    }
}
// arena index of component `comp` of quad `u` (= (CTA of the team, patch, output)); -1 where the patch reaches beyond the layer
template <int L>
__device__ __forceinline__ int arena_index(const Net& n, int u, int comp){
    const int q = u & 3, rank = quotient(u >> 2, n.by_tiles), tile = (u >> 2) - rank * n.n_tiles;
    int l, o4, i4, index = -1;
    locate<L>(n, tile, l, o4, i4);
#pragma unroll
    for(int k = 0; k < L; k++) if(l == k){
        const Layer& y = n.layer[k];
        const int o = rank * y.S + o4 * 4 + q, i = i4 * 4 + comp;
        if(o < y.O && i <= y.I) index = (int)y.poff + (i < y.I ? o * y.I + i : y.O * y.I + o);
    }
    return index;
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

// All CTAs of the grid (cta of ctas) share out the parameters: `lanes` threads per quad (a power of two from 4 on) add the teams' sums (lane y
// takes teams y, y + lanes, ... ascending, then the lanes pairwise: a fixed order), the first four lanes each finish one parameter:
// sink(arena index, gradient, what prefetch(arena index) returned before the sums were loaded).
template <int C, int L, typename PREFETCH, typename SINK>
__device__ __forceinline__ void reduce_gradients(const Net& n, const float4* partial, int teams, int cta, int ctas, int lanes, PREFETCH prefetch, SINK sink){
    const int quads = C * n.n_tiles * 4, lane = threadIdx.x & (lanes - 1), lane_bits = __popc(lanes - 1), per_cta = THREADS >> lane_bits;
    for(int u0 = cta * per_cta; u0 < quads; u0 += ctas * per_cta){
        const int u = u0 + ((int)threadIdx.x >> lane_bits);
        const int index = u < quads && lane < 4 ? arena_index<L>(n, u, lane) : -1;
        const auto early = prefetch(index);
        float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if(u < quads){
            const float4* src = partial + u;
            for(int t = lane; t < teams; t += 8 * lanes){
                float4 v[8];
#pragma unroll
                for(int k = 0; k < 8; k++) v[k] = t + k * lanes < teams ? __ldcg(src + (size_t)(t + k * lanes) * quads) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                for(int k = 0; k < 8; k++){ s.x += v[k].x; s.y += v[k].y; s.z += v[k].z; s.w += v[k].w; }
            }
        }
        for(int o = lanes >> 1; o > 0; o >>= 1){
            s.x += __shfl_xor_sync(0xffffffffu, s.x, o); s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
            s.z += __shfl_xor_sync(0xffffffffu, s.z, o); s.w += __shfl_xor_sync(0xffffffffu, s.w, o);
        }
        if(index >= 0) sink(index, lane == 0 ? s.x : lane == 1 ? s.y : lane == 2 ? s.z : s.w, early);
    }
}
#endif

}}  // namespace b200rl::team
