// One training step of a network in ONE cooperative launch: gradients zeroed, forward, mean-squared-error gradient, backward, gradient sums over
// the whole batch, optimizer step -- for batches that leave the tensor-core kernels without enough row tiles (the replay batches of the off-policy
// algorithms, the minibatches of the on-policy ones). Built on the team walk of mlp_team.cuh: a team of C CTAs takes tiles of R rows through the
// network, the teams' gradient sums meet in scratch memory behind one grid-wide barrier.
// Same operations as zero_gradient, forward, mse::gradient, backward, step (nn_models/mlp/operations_generic.h:77-217,
// nn/loss_functions/mse/operations_generic.h:43-58, nn/optimizers/adam/operations_generic.h:49-64) run one after the other.
#include "common.cuh"
#include "grid_barrier.cuh"
#include "mlp_team.cuh"
#include <atomic>
#include <mutex>

namespace b200rl {
using namespace team;

struct TeamStepArgs {
    Net net;
    float* params; float* grads; float* m; float* v; uint32_t* adam_state;
    b200rl_adam_hyper hyper;
    const float* x; const float* target; int ldx, ldt;
    float* pre; float* out;
    float4* partial; GridBarrier barrier;
    int rows, chunk_rows, n_total, optimize, row_tiles, teams, lanes;
    Divisor by_S;
    float constant;                          // 2 / (rows of a chunk x columns) x loss weight, evaluated like the reference does
    int y_off, y_alt, out_off;               // shared-memory offsets: targets of a tile, distance of the next tile's, outputs
};

template <int C, int L, int N, int PO, int PI>
__global__ void __launch_bounds__(THREADS, 1) mlp_team_step_kernel(const __grid_constant__ TeamStepArgs a){
    extern __shared__ __align__(16) float smem[];
    __shared__ float s_scalars[2];
    __shared__ int s_ok;
    __shared__ uint32_t s_age;
    const Net& n = a.net;
    const int tid = threadIdx.x, rank = C == 1 ? 0 : (int)cluster_rank(), t = blockIdx.x / C;
    const Layer& last = n.layer[L - 1];
    const int I0 = n.layer[0].I, R = n.R;
    auto stage = [&](int tile, bool other){  // the tile's input rows and this CTA's target columns, zero beyond the batch
        const int row0 = tile * R, P = n.layer[0].P;
        float* rows = smem + n.layer[0].a + (other ? n.a_alt : 0);
        if(((I0 | a.ldx) & 3) == 0 && (reinterpret_cast<uintptr_t>(a.x) & 15u) == 0){
#pragma unroll 1
            for(int i = tid; i < R * (I0 >> 2); i += THREADS){
                const int r = quotient(i, n.layer[0].by_row), k = 4 * (i - r * (I0 >> 2));
                if(row0 + r < a.rows) copy16_async(rows + r * P + k, a.x + (size_t)(row0 + r) * a.ldx + k);
                else *reinterpret_cast<float4*>(rows + r * P + k) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        }
        else{
#pragma unroll 1
            for(int i = tid; i < R * I0; i += THREADS){
                const int r = quotient(i, n.by_I0), k = i - r * I0;
                if(row0 + r < a.rows) copy4_async(rows + r * P + k, a.x + (size_t)(row0 + r) * a.ldx + k);
                else rows[r * P + k] = 0.0f;
            }
        }
#pragma unroll 1
        for(int i = tid; i < R * last.S; i += THREADS){
            const int r = quotient(i, a.by_S), unit = rank * last.S + i - r * last.S;
            if(row0 + r < a.rows && unit < last.O) copy4_async(smem + a.y_off + (other ? a.y_alt : 0) + i, a.target + (size_t)(row0 + r) * a.ldt + unit);
        }
    };
    clear_rows<L>(n, smem);
    __syncthreads();
    stage(t, false);
    load_weights<L>(n, smem, a.params, rank);
    // the optimizer's age, too, is here before this CTA arrives at the grid barrier: once all have arrived, the first CTA may store the next one
    if(tid == 0 && a.optimize) copy4_async(reinterpret_cast<float*>(&s_age), reinterpret_cast<const float*>(a.adam_state));
    Patch patches[N];
    Sums<N, PO, PI> acc;
#pragma unroll
    for(int k = 0; k < N; k++) patches[k] = patch<L>(n, k * THREADS + tid);
    clear_sums(acc);
    const int keep_from = a.rows - a.chunk_rows;          // the activations of the last chunk stay behind in pre / out
    bool other = false;                                   // which of the two buffers this tile's rows are in
    for(int tile = t; tile < a.row_tiles; tile += a.teams, other = !other){
        copies_wait();
        sync_team<C>();                                   // the rows are there; every CTA of the team has left the previous tile (or set its buffers up)
        if(tile + a.teams < a.row_tiles) stage(tile + a.teams, !other);
        const int row0 = tile * R;
        const float* y = smem + a.y_off + (other ? a.y_alt : 0);
#pragma unroll
        for(int l = 0; l < L; l++){
            forward_layer<C, L, true, false>(n, l, n.layer[l].a + (l == 0 && other ? n.a_alt : 0), smem, rank, nullptr, [&](int r, int unit, float4 value, float4 derivative){
                const int at = r * last.S + unit;
                const float4 target = *reinterpret_cast<const float4*>(y + at);
                auto d = [&](float v, float wanted, float dv){ return row0 + r < a.rows ? d_pre(__fmul_rn(__fsub_rn(v, wanted), a.constant), dv) : 0.0f; };
                *reinterpret_cast<float4*>(smem + last.d + at) = make_float4(d(value.x, target.x, derivative.x), d(value.y, target.y, derivative.y), d(value.z, target.z, derivative.z), d(value.w, target.w, derivative.w));
                *reinterpret_cast<float4*>(smem + a.out_off + at) = value;
            });
            if(l == L - 1) __syncthreads();
            else sync_team<C>();
        }
#pragma unroll
        for(int l = L - 1; l > 0; l--) backward_layer<C, false>(n, l, smem, rank, (L - l) & 1, nullptr);
        store_activations<L>(n, smem, smem + a.out_off, rank, row0, a.rows, keep_from, a.chunk_rows, a.pre, a.out);
        accumulate_gradients<N, PO, PI>(n, smem, patches, acc, other);
    }
    store_gradients<N, PO, PI>(n, a.partial + (size_t)t * C * n.quads, rank, acc);
    __syncthreads();
    if(tid == 0){ grid_barrier_arrive(a.barrier); s_ok = grid_barrier_wait(a.barrier, gridDim.x); }
    else if(a.optimize && (tid == 32 || tid == 33)) s_scalars[tid - 32] = adam_bias_correction(tid == 32 ? a.hyper.beta_1 : a.hyper.beta_2, s_age);
    __syncthreads();
    if(!s_ok){ if(tid == 0) grid_barrier_leave(a.barrier, gridDim.x); return; }
    const float c1 = s_scalars[0], c2 = s_scalars[1];
    struct Moments { float p, m, v; };
    auto prefetch = [&](int i){ return a.optimize && i >= 0 ? Moments{a.params[i], a.m[i], a.v[i]} : Moments{0.0f, 0.0f, 0.0f}; };
    auto sink = [&](int i, float g, Moments s){
        a.grads[i] = g;
        if(a.optimize){
            a.params[i] = adam_update(s.p, g, s.m, s.v, a.hyper, c1, c2);
            a.m[i] = s.m; a.v[i] = s.v;
        }
    };
    reduce_gradients<C, L>(n, a.partial, a.teams, blockIdx.x, gridDim.x, a.lanes, prefetch, sink);
    if(blockIdx.x == 0){
        for(int i = n.n_params + tid; i < a.n_total; i += THREADS) sink(i, 0.0f, prefetch(i));      // parameters outside the layers: no gradient from this loss
        if(tid == 0 && a.optimize){ a.adam_state[0] = s_age + 1u; a.adam_state[1] = 0u; a.adam_state[2] = __float_as_uint(c1); a.adam_state[3] = __float_as_uint(c2); }
    }
    if(tid == 0) grid_barrier_leave(a.barrier, gridDim.x);
}

// ---- host side ---------------------------------------------------------------------------------------------------------------------------
struct TeamChoice { Net net; int teams, row_tiles, y_off, y_alt, out_off; size_t smem; };

constexpr size_t TEAM_SMEM = 220 * 1024;
constexpr int TEAM_MAX_ROWS = 8192;          // what was measured; up to there the caller asks for steps of little work only (dense.cu)

// teams of C CTAs that are resident at once on the current device (clusters do not tile every GPC completely); 0: unknown
static int team_capacity(int C);

// Team size and rows per tile by an estimate of the launch: a layer of a tile costs its latencies (more where the team exchanges through cluster barriers) and its products, loading the weights
// and storing and adding the teams' sums cost per float, the grid barrier and the sums per CTA. The constants, in no unit but their own, are fitted to all teams and tiles of 110 shapes (16 ... 256
// wide, 2 to 4 layers, 32 ... 6,000 rows): the choice is 1.3 % from the fastest on average, the worst 9 % off (18-200-200-3 at 563 rows: 24.3 and 22.5 us). Without the cost of a CTA small
// networks were spread too thin: 12-16-16-3 at 838 rows 12.7 us on 105 CTAs, 12.0 on 42; 5-100-100-2 at 50 rows 15.2 us on 13 CTAs, 13.6 in teams of four.
// Only plans whose sums fit into scratch_bytes: the scratch of a smaller batch serves a larger one, by its own plan or a better one that fits.
static bool choose_team(const b200rl_mlp_shape* sh, int rows, size_t scratch_bytes, TeamChoice* out){
    for(int l = 0, I = sh->input_dim; l < sh->n_layers; I = sh->dims[l], l++) if(sh->dims[l] > 512 || I > 512) return false;
    double best = 0.0;
    for(int C = 1; C <= 8; C *= 2){
        const int max_teams = team_capacity(C);
        TeamChoice c{};
        if(max_teams < 1 || !spread(sh, C, 0, &c.net)) continue;
        double weights = 0.0;
        for(int l = 0; l < c.net.n_layers; l++) weights += (double)c.net.layer[l].S * c.net.layer[l].P;
        const Layer& last = c.net.layer[c.net.n_layers - 1];
        for(int R = 4; R <= 32; R += 4){
            place(c.net, R, true);
            int off = (c.net.end + 3) / 4 * 4;
            c.y_off = off; c.y_alt = R * last.S; off += 2 * R * last.S;
            c.out_off = off; off += R * last.S;
            c.smem = sizeof(float) * (size_t)off;
            if(c.smem > TEAM_SMEM) break;                                // more rows take more
            c.row_tiles = (rows + R - 1) / R;
            c.teams = c.row_tiles < max_teams ? c.row_tiles : max_teams;
            if(sizeof(float4) * (size_t)c.teams * C * c.net.quads > scratch_bytes) continue;
            const double tile = (C == 1 ? 3800.0 : 4700.0) * c.net.n_layers + 0.13 * R * weights;
            const double cost = 0.15 * weights + tile * ((c.row_tiles + c.teams - 1) / c.teams) + 0.3 * c.net.quads + 0.0013 * C * c.net.quads * c.teams + 45.0 * C * c.teams;
            if(best == 0.0 || cost < best){ best = cost; *out = c; }
        }
    }
    if(best > 0.0) complete(out->net, false);
    return best > 0.0;
}

// what the plan of this batch needs for any number of rows (a training step may run over several chunks of the batch the scratch was asked for)
size_t mlp_team_scratch_bytes(const b200rl_mlp_shape* sh, int rows){
    TeamChoice c;
    if(rows < 1 || !choose_team(sh, rows, SIZE_MAX, &c)) return 0;
    return sizeof(float4) * (size_t)team_capacity(c.net.C) * c.net.C * c.net.quads;
}

static void team_attributes(cudaLaunchAttribute (&attr)[2], int C){
    attr[0].id = cudaLaunchAttributeClusterDimension; attr[0].val.clusterDim.x = C; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative; attr[1].val.cooperative = 1;
}
template <int C>
static int query_capacity(){
    int n = 0;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    team_attributes(attr, C);
    cfg.gridDim = dim3(NUM_SMS / C * C); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = TEAM_SMEM; cfg.attrs = attr; cfg.numAttrs = 1;
    if(cudaFuncSetAttribute(mlp_team_step_kernel<C, 3, 1, 1, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TEAM_SMEM) != cudaSuccess ||
       cudaOccupancyMaxActiveClusters(&n, mlp_team_step_kernel<C, 3, 1, 1, 1>, &cfg) != cudaSuccess){ cudaGetLastError(); return 0; }
    return n;
}
static int team_capacity(int C){
    static std::atomic<int> cached[MAX_DEVICES][4];                      // capacity + 1
    const int k = C == 1 ? 0 : C == 2 ? 1 : C == 4 ? 2 : 3;
    int dev = 0;
    if(cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES){ cudaGetLastError(); return 0; }
    int n = cached[dev][k].load(std::memory_order_relaxed);
    if(n == 0){
        n = 1 + (k == 0 ? query_capacity<1>() : k == 1 ? query_capacity<2>() : k == 2 ? query_capacity<4>() : query_capacity<8>());
        cached[dev][k].store(n, std::memory_order_relaxed);
    }
    return n - 1;
}

template <int C, int L, int N, int PO, int PI>
static int launch_team_step(const TeamStepArgs& a, size_t smem, cudaStream_t s){
    static std::atomic<bool> configured[MAX_DEVICES];
    int dev = 0;
    int rc = current_device(&dev);
    if(rc) return rc;
    if(!configured[dev].load(std::memory_order_acquire)){
        B200RL_CUDA_TRY(cudaFuncSetAttribute(mlp_team_step_kernel<C, L, N, PO, PI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TEAM_SMEM));
        configured[dev].store(true, std::memory_order_release);
    }
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    team_attributes(attr, C);
    cfg.gridDim = dim3(a.teams * C); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = s; cfg.attrs = attr; cfg.numAttrs = 2;
    B200RL_CUDA_TRY(cudaLaunchKernelEx(&cfg, mlp_team_step_kernel<C, L, N, PO, PI>, a));
    return B200RL_OK;
}
template <int C, int L>
static int launch_team_step_l(const TeamStepArgs& a, size_t smem, cudaStream_t s){
    if(a.net.n_patches > THREADS) return launch_team_step<C, L, MAX_PATCHES_PER_THREAD, 1, 1>(a, smem, s);
    if(a.net.patch_i == 2) return launch_team_step<C, L, 1, 2, 2>(a, smem, s);
    if(a.net.patch_o == 2) return launch_team_step<C, L, 1, 2, 1>(a, smem, s);
    return launch_team_step<C, L, 1, 1, 1>(a, smem, s);
}
template <int C>
static int launch_team_step_c(const TeamStepArgs& a, size_t smem, cudaStream_t s){
    switch(a.net.n_layers){
        case 1: return launch_team_step_l<C, 1>(a, smem, s);
        case 2: return launch_team_step_l<C, 2>(a, smem, s);
        case 3: return launch_team_step_l<C, 3>(a, smem, s);
        default: return launch_team_step_l<C, 4>(a, smem, s);
    }
}

int mlp_team_step(const b200rl_mlp_shape* sh, float* params, float* grads, float* m, float* v, size_t n_total, const b200rl_adam_hyper& hyper, uint32_t* adam_state,
                  const float* x, int ldx, const float* target, int ldt, int rows, int chunk_rows, float loss_weight, float* pre, float* out, void* scratch, size_t scratch_bytes,
                  int optimize, cudaStream_t s){
    TeamChoice c;
    if(rows > TEAM_MAX_ROWS || !scratch || (reinterpret_cast<uintptr_t>(scratch) & 15u) || !choose_team(sh, rows, scratch_bytes, &c)) return B200RL_ERR_UNSUPPORTED;
    TeamStepArgs a{};
    a.net = c.net;
    a.params = params; a.grads = grads; a.m = m; a.v = v; a.adam_state = adam_state; a.hyper = hyper;
    a.x = x; a.ldx = ldx; a.target = target; a.ldt = ldt; a.pre = pre; a.out = out;
    a.partial = static_cast<float4*>(scratch);
    a.rows = rows; a.chunk_rows = chunk_rows; a.n_total = (int)n_total; a.optimize = optimize; a.row_tiles = c.row_tiles; a.teams = c.teams;
    a.constant = 2.0f / ((float)chunk_rows * (float)sh->dims[sh->n_layers - 1]) * loss_weight;
    a.y_off = c.y_off; a.y_alt = c.y_alt; a.out_off = c.out_off; a.by_S = divisor(c.net.layer[c.net.n_layers - 1].S);
    // threads per quad of the reduction: as many as let the grid take all quads in one pass, no more than there are sums to add
    const int quads = c.net.C * c.net.quads, threads = c.teams * c.net.C * THREADS;
    a.lanes = 4;
    while(a.lanes < 32 && 2 * a.lanes <= c.teams && (long long)quads * 2 * a.lanes <= threads) a.lanes *= 2;
    int rc = grid_barriers(1, s, &a.barrier);
    if(rc) return rc;
    if(c.net.C == 1) return launch_team_step_c<1>(a, c.smem, s);
    if(c.net.C == 2) return launch_team_step_c<2>(a, c.smem, s);
    if(c.net.C == 4) return launch_team_step_c<4>(a, c.smem, s);
    return launch_team_step_c<8>(a, c.smem, s);
}

}  // namespace b200rl
