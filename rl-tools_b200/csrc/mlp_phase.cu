// Whole-pass kernels for wide networks at small batches (e.g. 4 -> 256 -> 256 -> 1 at batch 256: the critic of the off-policy algorithms).
//
// At this size a layer's products are a few microseconds of work spread over 64 tiles each, and a backward pass through per-layer kernels is a chain of
// dependent launches (five per layer: d_pre and the bias sums, the weight gradient, its reduction, the input gradient). The weights (256 KB
// per 256 x 256 layer) do not fit one CTA, so the pass cannot be a kernel of independent CTAs like the one for small networks; here it is one launch per
// layer whose CTAs share out the tiles of everything that the layer's d_pre gives:
//   dW_l += d_pre_l^T in_l, db_l += column sums of d_pre_l, and d_pre_(l-1) = (d_pre_l W_l) * act'(pre_(l-1)), the
//   derivative folded into the epilogue of the input-gradient tiles (nn/layers/dense/operations_generic.h:151-243)
// A tile is 32 x 32 outputs; the CTA brings both operands of up to 256 summed indices into shared memory with all of its copies in flight
// at once (one L2 round trip per tile), its eight warps take every eighth group of four summed indices and each lane a 4 x 8 patch,
// and the eight partial tiles are added in warp order (deterministic).
//
// Bound by latency, so what the epilogues read (old gradients, pre-activations) and a column's rows for the bias sums are under way together with the operands (a launch of the critic's backward
// pass 6.0 -> 5.6 us on average). Measured, 4-256-256-1 at batch 256 in a captured graph: 16.7 us (one cooperative launch with grid barriers between the layers 24 us: a
// barrier costs more than a graph's next node, and two such launches take turns on the SMs).
#include "common.cuh"
#include <atomic>

namespace b200rl {

constexpr int PH_T = 32, PH_KC = 256, PH_THREADS = 256, PH_WARPS = 8;
constexpr size_t PH_SMEM = sizeof(float) * 2 * PH_KC * PH_T;          // both operand tiles; the eight partial tiles (32 KB) reuse the space

struct PhaseProduct {                    // C(m, n) = sum_k A(m, k) B(n, k)
    const float* A; const float* B; float* C; const float* aux;
    int lda, ldb, ldc, ldaux, M, N, K, act, tiles_n, tiles;
};
enum { PH_PHASE_PRODUCTS = 0, PH_PHASE_DPRE = 1 };
struct Phase {
    int type;
    PhaseProduct dx, dw;                 // input gradient; weight gradient, added to what is there
    const float* bias_src; float* bias_dst; int bias_ld, bias_rows, bias_cols, bias_items;      // db += column sums
    float* d_out; const float* pre; int ew_ldd, ew_ldpre, ew_rows, ew_cols, ew_act;                              // d_pre of the last layer, in place
};
constexpr int PH_MAX_LAYERS = 4, PH_MAX_PHASES = PH_MAX_LAYERS + 1;
struct PhaseArgs { int n_phases; Phase phase[PH_MAX_PHASES]; };

// Operand tiles, brought in by asynchronous copies in the order in which they lie in memory (zeros outside the operand):
//   summed index contiguous: [row][256], 16-byte pieces swizzled by the row, read four summed indices at a time
//   row index contiguous   : [k][32], read four rows of one k at a time
__device__ __forceinline__ void phase_copy(float* to, const float* from, const float* valid, int floats, bool vec){       // four floats, zeros behind the first `floats`
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(to);
    if(vec) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(at), "l"(floats > 0 ? from : valid), "r"(floats > 0 ? 16 : 0) : "memory");
    else{
#pragma unroll
        for(int k = 0; k < 4; k++) asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"(at + 4 * k), "l"(k < floats ? from + k : valid), "r"(k < floats ? 4 : 0) : "memory");
    }
}
__device__ __forceinline__ void phase_load(float* S, const float* P, int ld, bool kcontig, int r0, int R, int k0, int kc){
    const bool vec = ld % 4 == 0 && (reinterpret_cast<uintptr_t>(P) & 15u) == 0 && (kcontig ? kc : R) % 4 == 0;
    const int pieces = (kc + 3) / 4;
    if(kcontig){
        const int c = threadIdx.x & 63;
        if(c < pieces){
#pragma unroll
            for(int j = 0; j < PH_T / 4; j++){
                const int r = (threadIdx.x >> 6) + 4 * j;
                phase_copy(S + r * PH_KC + 4 * (c ^ (r & 7)), P + (size_t)(r0 + r) * ld + k0 + 4 * c, P, r0 + r < R ? kc - 4 * c : 0, vec);
            }
        }
    }
    else{
        const int r = 4 * (threadIdx.x & 7);
#pragma unroll
        for(int j = 0; j < PH_KC / 32; j++){
            const int k = (threadIdx.x >> 3) + 32 * j;
            if(k < 4 * pieces) phase_copy(S + k * PH_T + r, P + (size_t)(k0 + k) * ld + r0 + r, P, k < kc ? R - r0 - r : 0, vec);
        }
    }
}

// the first operand in either order, the second with its rows contiguous
template <bool A_KCONTIG>
__device__ __forceinline__ void phase_product_tile(const PhaseProduct& g, int tile, float* smem){
    const float* A = opaque(g.A); const float* B = opaque(g.B); const float* aux = opaque(g.aux); float* C = opaque(g.C);
    float* As = smem;
    float* Bs = smem + PH_T * PH_KC;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rg = lane >> 2, cg = lane & 3;
    const int m0 = (tile / g.tiles_n) * PH_T, n0 = (tile % g.tiles_n) * PH_T;
    float2 acc[4][4];                                      // rows rg + 8 i (4 rg + i), columns 8 cg + 2 j, + 1
#pragma unroll
    for(int i = 0; i < 4; i++)
#pragma unroll
        for(int j = 0; j < 4; j++) acc[i][j] = make_float2(0.0f, 0.0f);
    // what the epilogue reads, asked for while the operands are on their way: the old gradients, the pre-activations of the layer below
    const int r = tid >> 3, c4 = (tid & 7) * 4, m = m0 + r;
    float early[4];
#pragma unroll
    for(int j = 0; j < 4; j++){
        const int n = n0 + c4 + j;
        early[j] = 0.0f;
        if(m < g.M && n < g.N){
            if(!A_KCONTIG) early[j] = C[(size_t)m * g.ldc + n];
            else if(g.aux) early[j] = __ldg(aux + (size_t)m * g.ldaux + n);
        }
    }
    for(int k0 = 0; k0 < g.K; k0 += PH_KC){
        const int kc = min(PH_KC, g.K - k0);
        if(k0) __syncthreads();                            // whoever read the previous chunk is done
        phase_load(As, A, g.lda, A_KCONTIG, m0, g.M, k0, kc);
        phase_load(Bs, B, g.ldb, false, n0, g.N, k0, kc);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        for(int c = warp; c < (kc + 3) / 4; c += PH_WARPS){
            float a[4][4];                                 // [k][i]
#pragma unroll
            for(int i = 0; i < 4; i++){
                const float4 t = *reinterpret_cast<const float4*>(A_KCONTIG ? As + (rg + 8 * i) * PH_KC + 4 * (c ^ rg) : As + (4 * c + i) * PH_T + 4 * rg);
                if(A_KCONTIG){ a[0][i] = t.x; a[1][i] = t.y; a[2][i] = t.z; a[3][i] = t.w; }
                else{ a[i][0] = t.x; a[i][1] = t.y; a[i][2] = t.z; a[i][3] = t.w; }
            }
#pragma unroll
            for(int k = 0; k < 4; k++){
                const float4 b0 = *reinterpret_cast<const float4*>(Bs + (4 * c + k) * PH_T + 8 * cg), b1 = *reinterpret_cast<const float4*>(Bs + (4 * c + k) * PH_T + 8 * cg + 4);
                const float2 b[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w), make_float2(b1.x, b1.y), make_float2(b1.z, b1.w)};
#pragma unroll
                for(int i = 0; i < 4; i++)
#pragma unroll
                    for(int j = 0; j < 4; j++) acc[i][j] = __ffma2_rn(make_float2(a[k][i], a[k][i]), b[j], acc[i][j]);
            }
        }
    }
    __syncthreads();
    float* R = smem;                                       // [warp][32][32]
#pragma unroll
    for(int i = 0; i < 4; i++){
        float* row = R + (warp * PH_T + (A_KCONTIG ? rg + 8 * i : 4 * rg + i)) * PH_T + 8 * cg;
        *reinterpret_cast<float4*>(row) = make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y);
        *reinterpret_cast<float4*>(row + 4) = make_float4(acc[i][2].x, acc[i][2].y, acc[i][3].x, acc[i][3].y);
    }
    __syncthreads();
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for(int w = 0; w < PH_WARPS; w++){
        const float4 p = *reinterpret_cast<const float4*>(R + (w * PH_T + r) * PH_T + c4);
        v[0] += p.x; v[1] += p.y; v[2] += p.z; v[3] += p.w;
    }
    if(m >= g.M) return;
#pragma unroll
    for(int j = 0; j < 4; j++){
        const int n = n0 + c4 + j;
        if(n >= g.N) continue;
        float s = v[j];
        if(A_KCONTIG){                                     // input gradient, through the activation below
            if(g.aux) s *= d_activation_rt(early[j], g.act);
            C[(size_t)m * g.ldc + n] = s;
        }
        else C[(size_t)m * g.ldc + n] = early[j] + s;
    }
}

// 32 columns of the bias gradient: eight row lanes per column, added in lane order
__device__ void phase_bias_item(const Phase& p, int item, float* smem){
    const int tid = threadIdx.x, c = tid & 31, seg = tid >> 5, col = item * 32 + c;
    const float* src = opaque(p.bias_src);
    const float old = seg == 0 && col < p.bias_cols ? p.bias_dst[col] : 0.0f;
    float s = 0.0f;
    if(col < p.bias_cols)
        for(int b = seg; b < p.bias_rows; b += 32 * PH_WARPS){         // 32 loads under way, added in order
            float v[32];
#pragma unroll
            for(int k = 0; k < 32; k++) v[k] = b + k * PH_WARPS < p.bias_rows ? src[(size_t)(b + k * PH_WARPS) * p.bias_ld + col] : 0.0f;
#pragma unroll
            for(int k = 0; k < 32; k++) s += v[k];
        }
    __syncthreads();
    smem[seg * 32 + c] = s;
    __syncthreads();
    if(tid < 32 && col < p.bias_cols){
        float t = 0.0f;
#pragma unroll
        for(int w = 0; w < PH_WARPS; w++) t += smem[w * 32 + tid];
        p.bias_dst[col] = old + t;
    }
}

__global__ void __launch_bounds__(PH_THREADS, 2) mlp_phase_kernel(const __grid_constant__ Phase p){
    extern __shared__ __align__(16) float smem[];
    after_predecessor();
    if(p.type == PH_PHASE_DPRE){
        const int total = p.ew_rows * p.ew_cols, idx = blockIdx.x * PH_THREADS + threadIdx.x;
        if(idx >= total) return;
        const int r = idx / p.ew_cols, c = idx % p.ew_cols;
        float* d = opaque(p.d_out) + (size_t)r * p.ew_ldd + c;
        *d = *d * d_activation_rt(opaque(p.pre)[(size_t)r * p.ew_ldpre + c], p.ew_act);
    }
    else{
        const int item = blockIdx.x, t0 = p.dx.tiles, t1 = p.dw.tiles;
        if(item < t0) phase_product_tile<true>(p.dx, item, smem);
        else if(item < t0 + t1) phase_product_tile<false>(p.dw, item - t0, smem);
        else phase_bias_item(p, item - t0 - t1, smem);
    }
}

// ---------------------------------------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------------------------------------
bool mlp_fused_eligible(const b200rl_mlp_shape* sh, int batch);

// Which passes run here.
bool mlp_phase_eligible(const b200rl_mlp_shape* sh, int batch){
    if(batch < 1 || batch > 512 || sh->n_layers > PH_MAX_LAYERS || sh->input_dim > 512 || mlp_fused_eligible(sh, batch)) return false;
    for(int l = 0; l < sh->n_layers; l++) if(sh->dims[l] > 512) return false;
    return true;
}

static void set_tiles(PhaseProduct& g){ g.tiles_n = (g.N + PH_T - 1) / PH_T; g.tiles = ((g.M + PH_T - 1) / PH_T) * g.tiles_n; }

static int launch_phases(PhaseArgs& a, cudaStream_t s){
    static std::atomic<bool> configured[MAX_DEVICES];
    int dev = 0;
    const int rc = current_device(&dev);
    if(rc) return rc;
    if(!configured[dev].load(std::memory_order_acquire)){
        B200RL_CUDA_TRY(cudaFuncSetAttribute(mlp_phase_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PH_SMEM));
        configured[dev].store(true, std::memory_order_release);
    }
    for(int ph = 0; ph < a.n_phases; ph++){
        const Phase& p = a.phase[ph];
        const int items = p.type == PH_PHASE_DPRE ? (p.ew_rows * p.ew_cols + PH_THREADS - 1) / PH_THREADS
                                                  : p.dx.tiles + p.dw.tiles + p.bias_items;
        B200RL_CUDA_TRY(launch_after(mlp_phase_kernel, dim3(items), dim3(PH_THREADS), PH_SMEM, s, p));
    }
    return B200RL_OK;
}

int mlp_phase_backward(const b200rl_mlp_shape* sh, const float* params, float* grads, const float* x, int ldx, const float* pre, const float* out,
                      float* d_out, float* d_input, float* tick, float* tock, int batch, cudaStream_t s){
    const int L = sh->n_layers;
    size_t poff[PH_MAX_LAYERS], aoff[PH_MAX_LAYERS]; int Is[PH_MAX_LAYERS];
    { size_t po = 0, ao = 0; int I = sh->input_dim;
      for(int l = 0; l < L; l++){ poff[l] = po; aoff[l] = ao; Is[l] = I; po += (size_t)sh->dims[l] * I + sh->dims[l]; ao += (size_t)batch * sh->dims[l]; I = sh->dims[l]; } }
    PhaseArgs a{};
    if(sh->acts[L - 1] != B200RL_ACT_IDENTITY){                   // otherwise d_out is d_pre
        Phase& ph = a.phase[a.n_phases++];
        ph.type = PH_PHASE_DPRE; ph.d_out = d_out; ph.pre = pre + aoff[L - 1]; ph.ew_ldd = sh->dims[L - 1]; ph.ew_ldpre = sh->dims[L - 1];
        ph.ew_rows = batch; ph.ew_cols = sh->dims[L - 1]; ph.ew_act = sh->acts[L - 1];
    }
    const float* d_cur = d_out; int ldd = sh->dims[L - 1];
    for(int l = L - 1; l >= 0; l--){
        const int O = sh->dims[l], I = Is[l];
        const float* in = l == 0 ? x : out + aoff[l - 1];
        const int ldin = l == 0 ? ldx : I;
        float* d_in = l == 0 ? d_input : ((l % 2 == 0) ? tick : tock);
        if(!grads && !d_in) break;
        Phase& ph = a.phase[a.n_phases++];
        ph.type = PH_PHASE_PRODUCTS;
        if(grads){
            PhaseProduct& g = ph.dw;
            g.A = d_cur; g.lda = ldd; g.B = in; g.ldb = ldin; g.M = O; g.N = I; g.K = batch;
            g.C = grads + poff[l]; g.ldc = I;
            set_tiles(g);
            ph.bias_src = d_cur; ph.bias_ld = ldd; ph.bias_rows = batch; ph.bias_cols = O; ph.bias_dst = grads + poff[l] + (size_t)O * I;
            ph.bias_items = (O + 31) / 32;
        }
        if(d_in){
            PhaseProduct& g = ph.dx;
            g.A = d_cur; g.lda = ldd; g.B = params + poff[l]; g.ldb = I; g.M = batch; g.N = I; g.K = O;
            g.C = d_in; g.ldc = I;
            if(l > 0){ g.aux = pre + aoff[l - 1]; g.ldaux = I; g.act = sh->acts[l - 1]; }
            set_tiles(g);
        }
        d_cur = d_in; ldd = I;
    }
    return launch_phases(a, s);
}

}  // namespace b200rl
