// One epoch of the PPO update -- all of its minibatches, actor and critic -- in ONE cooperative launch.
//
// A minibatch update is about 24 dependent launches of two to thirteen microseconds each (65 us per update even when they are replayed as a CUDA
// graph), for arithmetic of a microsecond. Here half of the CTAs keep the actor and half the critic; the two never wait for each other. A CTA
// takes its rows of a minibatch through the network (mlp_team.cuh, teams of one CTA), the row-wise loss gradient of the clipped surrogate or of
// the value regression in between, writes its gradient sums, and behind a barrier over the network's CTAs every thread adds the sums of the one
// parameter it owns and steps the optimizer for it, with the moments in registers for the whole epoch. A second barrier publishes the new
// parameters, in quads of four neighbours of a weight row whose places in shared memory every CTA has a table of; log_std is quads like the weights. Replaces the
// per-minibatch body of train (rl/algorithms/ppo/operations_generic.h:159-336), per sample :214-296; Gaussian head random/operations_generic.h:87-121.
//
// The order of every sum is fixed (ORDERED in mlp_team.cuh): it follows from the networks and the rows of a minibatch by the rules of parts(), `lanes` below and the two orders of adding, and a
// change for speed keeps it. The clipped surrogate jumps where a sample's ratio crosses the clipping bound, so a rounding of one sum becomes percents of the actor's first moments once a sample
// has crossed: with sums in another order an update of 320 minibatches of 27-64-64-8 ended 4e-2 (2-norm, first moments) from this one for some data, 7e-7 for others. Sums in the order that suits
// the lanes best take 15.9 us per minibatch of it (2,048 rows) and 14.4 of 3-64-64-1 (512 rows, with the loop around it), these 16.7 and 15.3.
#include "common.cuh"
#include "grid_barrier.cuh"
#include "mlp_team.cuh"
#include <atomic>
#include <math.h>

namespace b200rl {
using namespace team;

struct PpoNetArgs {
    Net net;
    float* params; float* grads; float* m; float* v; uint32_t* adam_state;
    b200rl_adam_hyper hyper;
    float4* partial; float* fresh; GridBarrier barrier;       // gradient sums [team][quad] x 16 bytes; parameters on their way to all CTAs [quad] x 16 bytes
    int ctas, teams, lanes, row_tiles;
    int quads;                               // those of the layers and, behind them, of log_std
    int aux, aux_alt, out;                   // shared memory: columns of a tile (actions [R][S], log-probabilities [R], advantages [R]; targets [R]), distance of the next tile's; outputs [R][S]
    int std_warp;                            // the first of the warps that add the sums of log_std's quads
    int scratch;                             // shared memory of add_parts_in_order
    int places, log_std;                     // where the weights of every quad go [quads]; log_std [action dimension rounded up to four]
    int lp, ps, dl;                          // the surrogate's log-probability terms [R][S], (action - mean) / std [R][S], dL / d log-probability [R]
    Divisor by_S;
};
struct PpoEpochArgs {
    PpoNetArgs actor, critic;
    const float* observations; const float* actions; const float* log_probs; const float* advantages; const float* targets;
    const float* stats;                      // [minibatch][2]: mean and standard deviation of its advantages
    int ld, batch, minibatches, action_dim;
    float epsilon_clip, entropy_coefficient, advantage_epsilon, neg_log_sqrt_pi;
    int normalize_advantage, learn_action_std;
};

constexpr int PPO_TEAM_MAX_ACTIONS = 64, PPO_TEAM_MAX_PARAMS = 18944;       // parameters of a network's layers: what was measured

// mean and standard deviation of every minibatch's advantages (:173-184), one CTA each
__global__ void __launch_bounds__(1024) ppo_epoch_stats_kernel(const float* __restrict__ advantages, int ld, int batch, float* __restrict__ stats){
    __shared__ float s_sum[32], s_sq[32];
    after_predecessor();
    const float* adv = opaque(advantages) + (size_t)blockIdx.x * batch * ld;
    float sum = 0.0f, sq = 0.0f;
    for(int b = threadIdx.x; b < batch; b += blockDim.x){ const float a = adv[(size_t)b * ld]; sum += a; sq = fmaf(a, a, sq); }
    for(int o = 16; o > 0; o >>= 1){ sum += __shfl_xor_sync(0xffffffffu, sum, o); sq += __shfl_xor_sync(0xffffffffu, sq, o); }
    if((threadIdx.x & 31) == 0){ s_sum[threadIdx.x >> 5] = sum; s_sq[threadIdx.x >> 5] = sq; }
    __syncthreads();
    if(threadIdx.x == 0){
        float ts = 0.0f, tq = 0.0f;
        for(int w = 0; w < 32; w++){ ts += s_sum[w]; tq += s_sq[w]; }
        const float mean = ts / batch, msq = tq / batch;
        stats[2 * blockIdx.x] = mean; stats[2 * blockIdx.x + 1] = sqrtf(fmaxf(0.0f, msq - mean * mean));
    }
}

template <bool ACTOR, int L, int N, int PO, int PI>
__device__ __forceinline__ void ppo_epoch(const PpoEpochArgs& a, const PpoNetArgs& w, int cta, float* smem){
    __shared__ float s_scalars[2][64];       // bias corrections of the next minibatches
    __shared__ float s_std[PPO_TEAM_MAX_ACTIONS];
    __shared__ int s_ok;
    const Net& n = w.net;
    const Layer& last = n.layer[L - 1];
    const int tid = threadIdx.x, R = n.R, I0 = n.layer[0].I, A = a.action_dim, S = last.S;
    const bool has_rows = cta < w.row_tiles;
    auto stage = [&](int minibatch, int tile, bool other){
        const int tid = thread_here();
        const int row0 = tile * R;
        const size_t base = (size_t)minibatch * a.batch + row0;
        const int rows = min(R, a.batch - row0);
        float* in = smem + n.layer[0].a + (other ? n.a_alt : 0);
        float* aux = smem + w.aux + (other ? w.aux_alt : 0);
#pragma unroll 1
        for(int i = tid; i < R * I0; i += THREADS){
            const int r = quotient(i, n.by_I0), k = i - r * I0;
            if(r < rows) copy4_async(in + r * n.layer[0].P + k, a.observations + (base + r) * a.ld + k);
            else in[r * n.layer[0].P + k] = 0.0f;
        }
        if constexpr(ACTOR){
#pragma unroll 1
            for(int i = tid; i < R * S; i += THREADS){
                const int r = quotient(i, w.by_S), k = i - r * S;
                if(r < rows && k < A) copy4_async(aux + i, a.actions + (base + r) * a.ld + k);
            }
            if(tid < rows){
                copy4_async(aux + R * S + tid, a.log_probs + (base + tid) * a.ld);
                copy4_async(aux + R * S + R + tid, a.advantages + (base + tid) * a.ld);
            }
        }
        else if(tid < rows) copy4_async(aux + tid, a.targets + (base + tid) * a.ld);
    };
    clear_rows<L>(n, smem);
    __syncthreads();
    if(has_rows) stage(0, cta, false);
    load_weights<L>(n, smem, w.params, 0);
    if(ACTOR && tid < A) smem[w.log_std + tid] = w.params[n.n_params + tid];
    // the parameter this thread owns: `lanes` threads per quad of the layers, a warp behind them per quad of log_std, one pass over all quads (guaranteed by the host's choice of lanes)
    Owner me = owner(w.lanes, cta, w.ctas);
    const int quads = w.quads, std_quad = cta * WARPS + (tid >> 5) - w.std_warp;
    int lanes = w.lanes;
    if(me.quad >= n.quads) me.quad = quads;
    if(ACTOR && std_quad >= 0 && std_quad < quads - n.quads){ me.quad = n.quads + std_quad; me.part = tid & 31; lanes = 32; }
    const int u = me.quad;
    auto place_of_quad = [&](int q){ return ACTOR && q >= n.quads ? w.log_std + 4 * (q - n.quads) : weights_of_quad<L>(n, q); };
    int* places = reinterpret_cast<int*>(smem + w.places);
    for(int i = tid; i < quads; i += THREADS) places[i] = place_of_quad(i);
    const bool adds = u < quads && place_of_quad(u) >= 0;
    int index = -1;
    if(adds && me.part < 4){
        if(!ACTOR || u < n.quads) index = arena_index<L>(n, u, me.part);
        else if(4 * (u - n.quads) + me.part < A) index = n.n_params + 4 * (u - n.quads) + me.part;
    }
    float my_p = 0.0f, my_m = 0.0f, my_v = 0.0f, my_g = 0.0f;
    if(index >= 0){ my_p = w.params[index]; my_m = w.m[index]; my_v = w.v[index]; }
    unsigned target = 0;
    const uint32_t age0 = *reinterpret_cast<volatile uint32_t*>(w.adam_state);
    Patch patches[N];
#pragma unroll
    for(int k = 0; k < N; k++) patches[k] = patch<L>(n, k * THREADS + tid);
    bool other = false;                      // which of the two buffers this tile's rows are in
    const float value_constant = 2.0f / ((float)a.batch * 1.0f) * 0.5f;
    for(int mb = 0; mb < a.minibatches; mb++){
        const int tid = thread_here();
        if((mb & 63) == 0){
            __syncthreads();                                              // the last of the old ones have been read
            if(tid < 128) s_scalars[tid & 1][tid >> 1] = adam_bias_correction(tid & 1 ? w.hyper.beta_2 : w.hyper.beta_1, age0 + (uint32_t)(mb + (tid >> 1)));
            __syncthreads();
        }
        Sums<N, PO, PI> acc;
        clear_sums(acc);
        float std_gradient = 0.0f;
        float mean = 0.0f, deviation = 1.0f;
        if(ACTOR && a.normalize_advantage){ mean = __ldg(a.stats + 2 * mb); deviation = __fadd_rn(__ldg(a.stats + 2 * mb + 1), a.advantage_epsilon); }
        for(int tile = cta; tile < w.row_tiles; tile += w.teams, other = !other){
            const int rows = min(R, a.batch - tile * R);
            const float* aux = smem + w.aux + (other ? w.aux_alt : 0);
            copies_wait();
            __syncthreads();
            if(ACTOR && tid < A) s_std[tid] = expf(smem[w.log_std + tid]);
            if(tile + w.teams < w.row_tiles) stage(mb, tile + w.teams, !other);
            else if(mb + 1 < a.minibatches) stage(mb + 1, cta, !other);
#pragma unroll
            for(int l = 0; l < L; l++){
                forward_layer<1, L, false, true>(n, l, n.layer[l].a + (l == 0 && other ? n.a_alt : 0), smem, 0, smem + w.scratch, [&](int r, int unit, float4 value, float4 derivative){
                    if constexpr(ACTOR) *reinterpret_cast<float4*>(smem + w.out + r * S + unit) = value;
                    else *reinterpret_cast<float4*>(smem + last.d + r * S + unit) =
                        make_float4(r < rows ? __fmul_rn(__fsub_rn(value.x, aux[r]), value_constant) * derivative.x : 0.0f, 0.0f, 0.0f, 0.0f);       // one output
                });
                __syncthreads();
            }
            if constexpr(ACTOR){
                // eight lanes a row; what one of them needs from the others of its row goes through shared memory
                float* lp = smem + w.lp; float* ps = smem + w.ps; float* dl = smem + w.dl;
                const int part = tid & 7;
#pragma unroll 1
                for(int r = tid >> 3; r < R; r += THREADS / 8){          // the same number of rounds for all lanes of a warp: R is a multiple of four
#pragma unroll 1
                    for(int k = part; k < A; k += 8){
                        const int i = r * S + k;
                        const float p = __fdiv_rn(__fsub_rn(aux[i], smem[w.out + i]), s_std[k]);
                        // (constant - log_std) - 0.5 p^2 rounded once: p^2 as an exact float pair (see ppo.cu)
                        const float h = __fmul_rn(p, p), lo = __fmaf_rn(p, p, -h);
                        const float c = __fsub_rn(a.neg_log_sqrt_pi, smem[w.log_std + k]), hh = __fmul_rn(0.5f, h);
                        const float d = __fsub_rn(c, hh), db = __fsub_rn(d, c);
                        const float de = __fsub_rn(__fsub_rn(c, __fsub_rn(d, db)), __fadd_rn(hh, db));
                        lp[i] = __fadd_rn(d, __fmaf_rn(-0.5f, lo, de));
                        ps[i] = p;
                    }
                    __syncwarp();
                    float d = 0.0f;
                    if(r < rows){
                        float log_prob = 0.0f;
#pragma unroll 4
                        for(int k = 0; k < A; k++) log_prob = __fadd_rn(log_prob, lp[r * S + k]);
                        float advantage = aux[R * S + R + r];
                        if(a.normalize_advantage) advantage = __fdiv_rn(__fsub_rn(advantage, mean), deviation);
                        const float ratio = expf(__fsub_rn(log_prob, aux[R * S + r]));
                        const float lo = 1.0f - a.epsilon_clip, hi = 1.0f + a.epsilon_clip;
                        const float clipped_ratio = ratio < lo ? lo : (ratio > hi ? hi : ratio);
                        const bool clipped = ratio != clipped_ratio;
                        const bool unclipped_is_smaller = __fsub_rn(__fmul_rn(ratio, advantage), __fmul_rn(clipped_ratio, advantage)) <= 0.0f;
                        const float d_ratio = unclipped_is_smaller ? advantage : (clipped ? 0.0f : advantage);
                        d = __fmul_rn(__fmul_rn(-1.0f / (float)a.batch, d_ratio), ratio);
                    }
                    if(part == 0) dl[r] = d;
#pragma unroll 1
                    for(int k = part; k < S; k += 8){
                        const int i = r * S + k;
                        smem[last.d + i] = r < rows && k < A ? __fmul_rn(__fdiv_rn(ps[i], s_std[k]), d) * smem[last.g + i] : 0.0f;
                    }
                }
                __syncthreads();
                if(tid >= THREADS - 64 && tid < THREADS - 64 + A){       // the log_std gradient of the CTA's rows, in row order
                    const int k = tid - (THREADS - 64);
#pragma unroll 4
                    for(int r = 0; r < rows; r++) std_gradient += __fmul_rn(dl[r], __fadd_rn(-1.0f, __fmul_rn(ps[r * S + k], ps[r * S + k])));
                }
            }
#pragma unroll
            for(int l = L - 1; l > 0; l--) backward_layer<1, true>(n, l, smem, 0, 0, smem + w.scratch);
            accumulate_gradients<N, PO, PI>(n, smem, patches, acc, other);
        }
        if(has_rows){
            store_gradients<N, PO, PI>(n, w.partial + (size_t)cta * quads, 0, acc);
            if(ACTOR && tid >= THREADS - 64 && tid - (THREADS - 64) < 4 * (quads - n.quads)) __stcg(reinterpret_cast<float*>(w.partial + (size_t)cta * quads + n.quads) + tid - (THREADS - 64), std_gradient);
        }
        __syncthreads();
        target += (unsigned)w.ctas;
        if(tid == 0){ grid_barrier_arrive(w.barrier); s_ok = grid_barrier_wait(w.barrier, target); }
        __syncthreads();
        if(!s_ok) break;
        const float c1 = s_scalars[0][mb & 63], c2 = s_scalars[1][mb & 63];
        const float g = sum_of_teams<true>(w.partial, adds ? u : quads, quads, w.teams, me.part, lanes);
        if(index >= 0){
            // log_std: the entropy bonus of every sample (:262-266); no gradient where it is not learnt
            my_g = !ACTOR || index < n.n_params ? g : a.learn_action_std ? __fadd_rn(g, __fmul_rn((float)a.batch, -1.0f / (float)a.batch * a.entropy_coefficient)) : 0.0f;
            my_p = adam_update(my_p, my_g, my_m, my_v, w.hyper, c1, c2);
        }
        if(adds && me.part < 4) __stcg(w.fresh + 4 * u + me.part, my_p);
        if(mb + 1 == a.minibatches) break;
        __syncthreads();
        target += (unsigned)w.ctas;
        if(tid == 0){ grid_barrier_arrive(w.barrier); s_ok = grid_barrier_wait(w.barrier, target); }
        __syncthreads();
        if(!s_ok) break;
        if(has_rows){
#pragma unroll 4
            for(int q = tid; q < quads; q += THREADS){ const int at = places[q]; if(at >= 0) copy16_async(smem + at, w.fresh + 4 * q); }
        }
    }
    copies_wait();
    if(!s_ok){ if(tid == 0) grid_barrier_leave(w.barrier, (unsigned)w.ctas); return; }
    if(index >= 0){ w.params[index] = my_p; w.m[index] = my_m; w.v[index] = my_v; w.grads[index] = my_g; }
    if(cta == 0 && tid == 0){
        const int last_mb = (a.minibatches - 1) & 63;
        w.adam_state[0] = age0 + (uint32_t)a.minibatches; w.adam_state[1] = 0u;
        w.adam_state[2] = __float_as_uint(s_scalars[0][last_mb]); w.adam_state[3] = __float_as_uint(s_scalars[1][last_mb]);
    }
    if(tid == 0) grid_barrier_leave(w.barrier, (unsigned)w.ctas);
}

template <int L, int PO, int PI>
__global__ void __launch_bounds__(THREADS, 1) ppo_epoch_kernel(const __grid_constant__ PpoEpochArgs a){
    extern __shared__ __align__(16) float smem[];
    if((int)blockIdx.x < a.actor.ctas) ppo_epoch<true, L, 1, PO, PI>(a, a.actor, blockIdx.x, smem);
    else ppo_epoch<false, L, 1, PO, PI>(a, a.critic, blockIdx.x - a.actor.ctas, smem);
}

// ---- host side ---------------------------------------------------------------------------------------------------------------------------
constexpr size_t PPO_TEAM_SMEM = 220 * 1024, PPO_TEAM_MOST_SMEM = 225 * 1024;      // the second: for the smallest tiles, which nothing smaller can stand in for (1.3 KB more are static)

// rows per tile: one tile per CTA where the batch allows it
static bool plan_ppo_net(const b200rl_mlp_shape* sh, int batch, int ctas, bool actor, int least, PpoNetArgs* w, size_t* smem){
    const int want = (batch + ctas - 1) / ctas, A = sh->dims[sh->n_layers - 1];
    Net n;
    if(!spread(sh, 1, least, &n) || n.n_patches > THREADS || n.n_params > PPO_TEAM_MAX_PARAMS || A > PPO_TEAM_MAX_ACTIONS) return false;
    for(int R = want >= 32 ? 32 : (want + 3) / 4 * 4; R >= 4; R -= 4){
        place(n, R, false);
        const int S = n.layer[n.n_layers - 1].S;
        int off = (n.end + 3) / 4 * 4;
        w->quads = n.quads + (actor ? (A + 3) / 4 : 0);
        w->aux = off; w->aux_alt = R * S + 2 * R; off += 2 * w->aux_alt;
        w->out = off; off += R * S;
        w->places = off; off += (w->quads + 3) / 4 * 4;
        if(actor){ w->log_std = off; off += (A + 3) / 4 * 4; w->lp = off; off += R * S; w->ps = off; off += R * S; w->dl = off; off += R; }
        w->by_S = divisor(S);
        w->scratch = off; off += ordered_scratch(n);
        if(sizeof(float) * (size_t)off > (R > 4 ? PPO_TEAM_SMEM : PPO_TEAM_MOST_SMEM)) continue;
        w->net = n; w->ctas = ctas; w->row_tiles = (batch + R - 1) / R; w->teams = w->row_tiles < ctas ? w->row_tiles : ctas;
        // How many threads add a quad's sums is part of their order: as many as give 256 threads of each CTA the pieces of four parameters that there are. One pass over the quads (of patches, whose
        // edges are quads as well) has to fit all threads
        int pieces = 0;
        for(int l = 0; l < n.n_layers; l++) pieces += n.layer[l].S * (n.layer[l].I / 4 + 1);
        w->lanes = 4;
        while(w->lanes < 32 && 2 * w->lanes <= w->teams && 2ll * w->lanes * pieces <= ctas * ORDERED_LANES) w->lanes *= 2;
        auto warps = [&](){ return (n.quads + 32 / w->lanes - 1) / (32 / w->lanes); };
        while(w->lanes > 4 && warps() + w->quads - n.quads > ctas * WARPS) w->lanes /= 2;
        w->std_warp = warps();
        if(w->std_warp + w->quads - n.quads > ctas * WARPS) return false;
        *smem = sizeof(float) * (size_t)off;
        return true;
    }
    return false;
}
// gradient sums of the teams and the parameters on their way
static size_t ppo_exchange_bytes(const PpoNetArgs& w){ return sizeof(float4) * (size_t)(w.teams + 1) * w.quads; }
struct PpoChoice { PpoNetArgs actor, critic; size_t smem, bytes; };
static bool choose_ppo(const b200rl_mlp_shape* actor, const b200rl_mlp_shape* critic, int batch, int minibatches, PpoChoice* out){
    int sms = 0;
    if(!actor || !critic || actor->n_layers != critic->n_layers || actor->n_layers < 1 || actor->n_layers > 3 || batch < 1 || sm_count(&sms) != B200RL_OK) return false;
    PpoChoice c{};
    size_t sa = 0, sc = 0;
    int least = 0;                           // both networks take patches of the same size
    for(int k = 0; k < 2; k++){
        if(!plan_ppo_net(actor, batch, sms / 2, true, least, &c.actor, &sa) || !plan_ppo_net(critic, batch, sms / 2, false, least, &c.critic, &sc)) return false;
        const int pa = c.actor.net.patch_o + c.actor.net.patch_i, pc = c.critic.net.patch_o + c.critic.net.patch_i;
        if(pa == pc) break;
        least = (pa > pc ? pa : pc) - 2;
    }
    complete(c.actor.net, true); complete(c.critic.net, true);
    c.smem = sa > sc ? sa : sc;
    c.bytes = ppo_exchange_bytes(c.actor) + ppo_exchange_bytes(c.critic) + sizeof(float) * 2 * (size_t)minibatches;
    *out = c;
    return true;
}

template <int L, int PO, int PI>
static int launch_ppo_epoch(const PpoEpochArgs& a, size_t smem, cudaStream_t s){
    static std::atomic<bool> configured[MAX_DEVICES];
    int dev = 0;
    int rc = current_device(&dev);
    if(rc) return rc;
    if(!configured[dev].load(std::memory_order_acquire)){
        B200RL_CUDA_TRY(cudaFuncSetAttribute(ppo_epoch_kernel<L, PO, PI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PPO_TEAM_MOST_SMEM));
        configured[dev].store(true, std::memory_order_release);
    }
    PpoEpochArgs copy = a;
    void* params[] = { &copy };
    B200RL_CUDA_TRY(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(ppo_epoch_kernel<L, PO, PI>), dim3(a.actor.ctas + a.critic.ctas), dim3(THREADS), params, smem, s));
    return B200RL_OK;
}
template <int L>
static int launch_ppo_epoch_l(const PpoEpochArgs& a, size_t smem, cudaStream_t s){
    if(a.actor.net.patch_i == 2) return launch_ppo_epoch<L, 2, 2>(a, smem, s);
    if(a.actor.net.patch_o == 2) return launch_ppo_epoch<L, 2, 1>(a, smem, s);
    return launch_ppo_epoch<L, 1, 1>(a, smem, s);
}

}  // namespace b200rl
using namespace b200rl;

extern "C" size_t b200rl_ppo_train_epoch_scratch_bytes(const b200rl_mlp_shape* actor, const b200rl_mlp_shape* critic, int batch, int n_minibatches){
    PpoChoice c;
    return choose_ppo(actor, critic, batch, n_minibatches, &c) ? c.bytes : 0;
}

extern "C" int b200rl_ppo_train_epoch(const b200rl_mlp_shape* actor, const b200rl_mlp_arenas* actor_arenas, const b200rl_mlp_shape* critic, const b200rl_mlp_arenas* critic_arenas,
                                      const float* observations, const float* actions, const float* log_probs, const float* advantages, const float* target_values, int ld,
                                      int batch, int n_minibatches, float epsilon_clip, float entropy_coefficient, float advantage_epsilon, int normalize_advantage,
                                      int learn_action_std, void* scratch, size_t scratch_bytes, b200rl_stream_t stream){
    if(!actor || !critic || !actor_arenas || !critic_arenas || !observations || !actions || !log_probs || !advantages || !target_values || batch < 1 || n_minibatches < 0 || ld < 1)
        return B200RL_ERR_INVALID_ARGUMENT;
    const size_t na = b200rl_mlp_num_params(actor), nc = b200rl_mlp_num_params(critic);
    if(na == 0 || nc == 0) return B200RL_ERR_INVALID_ARGUMENT;
    const int A = actor->dims[actor->n_layers - 1];
    for(const b200rl_mlp_arenas* r : {actor_arenas, critic_arenas}) if(!r->params || !r->grads || !r->m || !r->v || !r->adam_state) return B200RL_ERR_INVALID_ARGUMENT;
    if(actor_arenas->n != na + (size_t)A || critic_arenas->n != nc) return B200RL_ERR_UNSUPPORTED;
    PpoChoice c;
    if(critic->dims[critic->n_layers - 1] != 1 || actor->input_dim != critic->input_dim || !choose_ppo(actor, critic, batch, n_minibatches, &c)) return B200RL_ERR_UNSUPPORTED;
    if(n_minibatches == 0) return B200RL_OK;
    if(!scratch || scratch_bytes < c.bytes || (reinterpret_cast<uintptr_t>(scratch) & 15u)) return B200RL_ERR_INVALID_ARGUMENT;
    PpoEpochArgs a{};
    a.actor = c.actor; a.critic = c.critic;
    auto arenas = [](PpoNetArgs& w, const b200rl_mlp_arenas* r){ w.params = r->params; w.grads = r->grads; w.m = r->m; w.v = r->v; w.adam_state = r->adam_state; w.hyper = r->hyper; };
    arenas(a.actor, actor_arenas); arenas(a.critic, critic_arenas);
    uint8_t* p = static_cast<uint8_t*>(scratch);
    for(PpoNetArgs* w : {&a.actor, &a.critic}){
        w->partial = reinterpret_cast<float4*>(p); w->fresh = reinterpret_cast<float*>(w->partial + (size_t)w->teams * w->quads);
        p += ppo_exchange_bytes(*w);
    }
    float* stats = reinterpret_cast<float*>(p);
    a.observations = observations; a.actions = actions; a.log_probs = log_probs; a.advantages = advantages; a.targets = target_values; a.stats = stats;
    a.ld = ld; a.batch = batch; a.minibatches = n_minibatches; a.action_dim = A;
    a.epsilon_clip = epsilon_clip; a.entropy_coefficient = entropy_coefficient; a.advantage_epsilon = advantage_epsilon;
    a.neg_log_sqrt_pi = (float)(-0.5 * (double)logf(2.0f * 3.14159265358979323846f));
    a.normalize_advantage = normalize_advantage; a.learn_action_std = learn_action_std;
    cudaStream_t s = (cudaStream_t)stream;
    GridBarrier bars[2];
    int rc = grid_barriers(2, s, bars);
    if(rc) return rc;
    a.actor.barrier = bars[0]; a.critic.barrier = bars[1];
    if(normalize_advantage){
        B200RL_CUDA_TRY(launch_after(ppo_epoch_stats_kernel, dim3(n_minibatches), dim3(1024), 0, s, advantages, ld, batch, stats));
    }
    switch(actor->n_layers){
        case 1: return launch_ppo_epoch_l<1>(a, c.smem, s);
        case 2: return launch_ppo_epoch_l<2>(a, c.smem, s);
        default: return launch_ppo_epoch_l<3>(a, c.smem, s);
    }
}
