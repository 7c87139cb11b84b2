// PPO update pieces that the reference runs as host scalar loops (rl/algorithms/ppo/operations_generic.h): generalized
// advantage estimation (one backward scan per environment) and the minibatch loss gradient with respect to the actor
// output and log_std (advantage normalisation, clipped surrogate, entropy bonus). All are HBM/latency-bound
// element-wise or scan kernels over columns of the on-policy dataset, addressed with an element pitch so that they work
// directly on the reference's row-major dataset matrix (row = step * N_ENVIRONMENTS + env) as well as on SoA arrays.
#include "common.cuh"

namespace b200rl {

// rl/algorithms/ppo/operations_generic.h:59-95. A CTA per environment: all threads read the steps and form the temporal differences, one thread runs the
// recurrence through shared memory (the reference's operations in their order), all threads write. Only the recurrence is serial, three operations a step; with
// a thread per environment every step waits for its loads (64 environments x 1,024 steps: 185 to 288 us by the columns' pitch, 20 us this way).
constexpr int GAE_CHUNK = 1024, GAE_THREADS = 256;
__global__ void __launch_bounds__(GAE_THREADS) gae_kernel(const float* __restrict__ rewards, long long ld_r, const float* __restrict__ all_values, long long ld_v,
                           const float* __restrict__ terminated, long long ld_te, const float* __restrict__ truncated, long long ld_tr,
                           float* advantages, long long ld_a, float* target_values, long long ld_t, int n_envs, int steps, float gamma, float lambda, int ignore_termination){
    __shared__ float s_adv[GAE_CHUNK], s_value[GAE_CHUNK];                // temporal differences, then advantages
    __shared__ float s_keep[GAE_CHUNK];                                   // 0: the recurrence starts anew
    const int e = blockIdx.x;
    const float lambda_gamma = __fmul_rn(lambda, gamma);
    float previous_advantage = 0.0f;
    for(int end = steps; end > 0; end -= GAE_CHUNK){
        const int first = max(0, end - GAE_CHUNK), count = end - first;
        for(int i = threadIdx.x; i < count; i += GAE_THREADS){
            const long long pos = (long long)(first + i) * n_envs + e;
            const bool term = terminated[pos * ld_te] != 0.0f, trunc = truncated[pos * ld_tr] != 0.0f;
            const float current = all_values[pos * ld_v];
            const float next = (term && !ignore_termination) ? 0.0f : all_values[(pos + n_envs) * ld_v];
            float td = __fsub_rn(__fadd_rn(rewards[pos * ld_r], __fmul_rn(gamma, next)), current);
            if(trunc && !term) td = 0.0f;
            s_adv[i] = td; s_value[i] = current; s_keep[i] = trunc ? 0.0f : 1.0f;
        }
        __syncthreads();
        if(threadIdx.x == 0){
            int i = count - 1;
            for(; i >= 7; i -= 8){
                float td[8], keep[8];
#pragma unroll
                for(int k = 0; k < 8; k++){ td[k] = s_adv[i - k]; keep[k] = s_keep[i - k]; }
#pragma unroll
                for(int k = 0; k < 8; k++){
                    previous_advantage = __fadd_rn(__fmul_rn(lambda_gamma, keep[k] != 0.0f ? previous_advantage : 0.0f), td[k]);
                    s_adv[i - k] = previous_advantage;
                }
            }
            for(; i >= 0; i--){
                previous_advantage = __fadd_rn(__fmul_rn(lambda_gamma, s_keep[i] != 0.0f ? previous_advantage : 0.0f), s_adv[i]);
                s_adv[i] = previous_advantage;
            }
        }
        __syncthreads();
        for(int i = threadIdx.x; i < count; i += GAE_THREADS){
            const long long pos = (long long)(first + i) * n_envs + e;
            advantages[pos * ld_a] = s_adv[i];
            target_values[pos * ld_t] = __fadd_rn(s_adv[i], s_value[i]);
        }
        __syncthreads();
    }
}

// The same with a thread per environment, neighbouring threads on neighbouring rows: for so many environments that they hide each other's loads. Same bits.
constexpr int GAE_ENVS = 64;
__global__ void __launch_bounds__(GAE_ENVS) gae_many_kernel(const float* __restrict__ rewards, long long ld_r, const float* __restrict__ all_values, long long ld_v,
                           const float* __restrict__ terminated, long long ld_te, const float* __restrict__ truncated, long long ld_tr,
                           float* advantages, long long ld_a, float* target_values, long long ld_t, int n_envs, int steps, float gamma, float lambda, int ignore_termination){
    const int e = blockIdx.x * GAE_ENVS + threadIdx.x;
    if(e >= n_envs) return;
    const float lambda_gamma = __fmul_rn(lambda, gamma);
    float next_value = all_values[((long long)steps * n_envs + e) * ld_v], advantage = 0.0f;
    for(int step = steps - 1; step >= 0; step--){
        const long long pos = (long long)step * n_envs + e;
        const bool term = terminated[pos * ld_te] != 0.0f, trunc = truncated[pos * ld_tr] != 0.0f;
        const float current = all_values[pos * ld_v];
        float td = __fsub_rn(__fadd_rn(rewards[pos * ld_r], __fmul_rn(gamma, term && !ignore_termination ? 0.0f : next_value)), current);
        if(trunc && !term) td = 0.0f;
        advantage = __fadd_rn(__fmul_rn(lambda_gamma, trunc ? 0.0f : advantage), td);
        advantages[pos * ld_a] = advantage;
        target_values[pos * ld_t] = __fadd_rn(advantage, current);
        next_value = current;
    }
}
// Measured, a CTA per environment against a thread per environment, us (columns of their own; columns of a 13-wide matrix): 4,096 x 16 8.8 and 7.6; 8.7 and 8.6.
// 4,096 x 64 16.8 and 14.7; 16.8 and 25.0. 8,192 x 16 14.7 and 8.2; 14.8 and 8.7. 8,192 x 256 99 and 52; 92 and 92. 8,192 x 1,024 369 and 543; 453 and 561.
// 16,384 x 256 196 and 124; 182 and 153. 65,536 x 16 87 and 7.7; 89 and 14.8. 65,536 x 64 201 and 37; 201 and 72.
static bool gae_many(int n_envs, int steps){ return n_envs >= 8192 ? steps <= n_envs / 32 : n_envs >= 4096 && steps <= 16; }

// random/operations_generic.h:87-121 with the reference's float/double promotions
struct GaussianTerms { float log_prob, d_mean, d_log_std; };
__device__ __forceinline__ GaussianTerms gaussian_terms(float mean, float log_std, float value){
    const float neg_log_sqrt_pi = (float)(-0.5 * (double)logf(2.0f * 3.14159265358979323846f));
    const float diff = __fsub_rn(value, mean);
    const float std = expf(log_std);
    const float pre_square = __fdiv_rn(diff, std);
    GaussianTerms t;
    // (neg_log_sqrt_pi - log_std) - 0.5 * pre_square^2, which the reference takes in double and rounds to float: here the square is an exact
    // float pair and the difference is rounded to float once (no double-precision instruction: they issue at 1/64 rate on this part and were
    // most of this kernel's time), as in the rollout's Gaussian head
    {
        const float h = __fmul_rn(pre_square, pre_square), l = __fmaf_rn(pre_square, pre_square, -h);          // pre_square^2 = h + l exactly
        const float a = __fsub_rn(neg_log_sqrt_pi, log_std), hh = __fmul_rn(0.5f, h);
        const float d = __fsub_rn(a, hh), db = __fsub_rn(d, a);
        const float de = __fsub_rn(__fsub_rn(a, __fsub_rn(d, db)), __fadd_rn(hh, db));                         // a - hh = d + de exactly
        t.log_prob = __fadd_rn(d, __fmaf_rn(-0.5f, l, de));
    }
    t.d_mean = __fdiv_rn(pre_square, std);
    t.d_log_std = __fadd_rn(-1.0f, __fmul_rn(pre_square, pre_square));
    return t;
}

// the same d_mean and d_log_std without the log-probability (no double-precision instruction)
__device__ __forceinline__ GaussianTerms gaussian_derivatives(float mean, float log_std, float value){
    const float diff = __fsub_rn(value, mean);
    const float std = expf(log_std);
    const float pre_square = __fdiv_rn(diff, std);
    GaussianTerms t;
    t.log_prob = 0.0f;
    t.d_mean = __fdiv_rn(pre_square, std);
    t.d_log_std = __fadd_rn(-1.0f, __fmul_rn(pre_square, pre_square));
    return t;
}

// :173-184: mean and std of the minibatch advantages -> stats[0], stats[1]
__global__ void __launch_bounds__(1024) ppo_adv_stats_kernel(const float* __restrict__ adv, long long ld, int B, float* stats){
    __shared__ float s_sum[32], s_sq[32];
    float sum = 0.0f, sq = 0.0f;
    for(int b = threadIdx.x; b < B; b += blockDim.x){ const float a = adv[b * ld]; sum += a; sq = fmaf(a, a, sq); }
    for(int o = 16; o > 0; o >>= 1){ sum += __shfl_xor_sync(0xffffffffu, sum, o); sq += __shfl_xor_sync(0xffffffffu, sq, o); }
    if((threadIdx.x & 31) == 0){ s_sum[threadIdx.x >> 5] = sum; s_sq[threadIdx.x >> 5] = sq; }
    __syncthreads();
    if(threadIdx.x == 0){
        float ts = 0.0f, tq = 0.0f;
        for(int w = 0; w < (int)(blockDim.x >> 5); w++){ ts += s_sum[w]; tq += s_sq[w]; }
        const float mean = ts / B, msq = tq / B;
        stats[0] = mean; stats[1] = sqrtf(fmaxf(0.0f, msq - mean * mean));
    }
}

struct PpoArgs {
    const float* current_actions; long long ld_cur;
    const float* rollout_actions; long long ld_roll;
    const float* log_std;
    const float* rollout_log_probs; long long ld_lp;
    const float* advantages; long long ld_adv;
    float* d_actions; long long ld_d;
    const float* stats; float* partial;       // partial[block][A]
    int B, A;
    float epsilon_clip, advantage_epsilon; int normalize_advantage, learn_action_std;
};
constexpr int PPO_THREADS = 256, PPO_MAX_ACTION_DIM = 64;

// :214-296, one thread per sample; per-block partial sums of the log_std gradient (warp shuffle + shared memory)
__global__ void __launch_bounds__(PPO_THREADS) ppo_gradient_kernel(PpoArgs a){
    __shared__ float s_part[PPO_MAX_ACTION_DIM][PPO_THREADS / 32];
    const int b = blockIdx.x * PPO_THREADS + threadIdx.x;
    const bool valid = b < a.B;
    float d_loss_d_lp = 0.0f;
    if(valid){
        float action_log_prob = 0.0f;
        for(int i = 0; i < a.A; i++){
            const GaussianTerms t = gaussian_terms(a.current_actions[b * a.ld_cur + i], a.log_std[i], a.rollout_actions[b * a.ld_roll + i]);
            action_log_prob = __fadd_rn(action_log_prob, t.log_prob);
        }
        float advantage = a.advantages[b * a.ld_adv];
        if(a.normalize_advantage) advantage = __fdiv_rn(__fsub_rn(advantage, a.stats[0]), __fadd_rn(a.stats[1], a.advantage_epsilon));
        const float ratio = expf(__fsub_rn(action_log_prob, a.rollout_log_probs[b * a.ld_lp]));
        const float lo = 1.0f - a.epsilon_clip, hi = 1.0f + a.epsilon_clip;
        const float clipped_ratio = ratio < lo ? lo : (ratio > hi ? hi : ratio);
        const bool clipped = ratio != clipped_ratio;
        const bool ratio_min_switch = __fsub_rn(__fmul_rn(ratio, advantage), __fmul_rn(clipped_ratio, advantage)) <= 0.0f;
        const float d_surrogate_d_ratio = ratio_min_switch ? advantage : (clipped ? 0.0f : advantage);
        d_loss_d_lp = __fmul_rn(__fmul_rn(-1.0f / (float)a.B, d_surrogate_d_ratio), ratio);
    }
    // second pass over the actions: only the float terms of the Gaussian (the double-precision log-probability is not needed again); the
    // warps' sums of the log_std gradient meet in shared memory once, after the loop
    for(int i = 0; i < a.A; i++){
        float contrib = 0.0f;
        if(valid){
            const GaussianTerms t = gaussian_derivatives(a.current_actions[b * a.ld_cur + i], a.log_std[i], a.rollout_actions[b * a.ld_roll + i]);
            a.d_actions[b * a.ld_d + i] = __fmul_rn(t.d_mean, d_loss_d_lp);
            contrib = __fmul_rn(d_loss_d_lp, t.d_log_std);
        }
        if(a.learn_action_std){
            for(int o = 16; o > 0; o >>= 1) contrib += __shfl_xor_sync(0xffffffffu, contrib, o);
            if((threadIdx.x & 31) == 0) s_part[i][threadIdx.x >> 5] = contrib;
        }
    }
    if(a.learn_action_std){
        __syncthreads();
        for(int i = threadIdx.x; i < a.A; i += PPO_THREADS){
            float t = 0.0f;
            for(int w = 0; w < PPO_THREADS / 32; w++) t += s_part[i][w];
            a.partial[(long long)blockIdx.x * a.A + i] = t;
        }
    }
}
// d_log_std[i] += sum over blocks (fixed order) + B * (-coefficient / B) (the entropy bonus of every sample, :262-266)
__global__ void ppo_log_std_reduce_kernel(float* d_log_std, const float* __restrict__ partial, int blocks, int A, int B, float entropy_coefficient){
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= A) return;
    float t = 0.0f;
    for(int k = 0; k < blocks; k++) t += partial[(long long)k * A + i];
    const float d_entropy = -1.0f / (float)B * entropy_coefficient;
    d_log_std[i] += t + (float)B * d_entropy;
}

}  // namespace b200rl
using namespace b200rl;

extern "C" {

int b200rl_gae(const float* rewards, int ld_rewards, const float* all_values, int ld_values, const float* terminated, int ld_terminated,
               const float* truncated, int ld_truncated, float* advantages, int ld_advantages, float* target_values, int ld_targets,
               int n_envs, int steps, float gamma, float lambda, int ignore_termination, b200rl_stream_t stream){
    if(!rewards || !all_values || !terminated || !truncated || !advantages || !target_values || n_envs < 0 || steps < 0 ||
       ld_rewards < 1 || ld_values < 1 || ld_terminated < 1 || ld_truncated < 1 || ld_advantages < 1 || ld_targets < 1) return B200RL_ERR_INVALID_ARGUMENT;
    if(n_envs == 0 || steps == 0) return B200RL_OK;
    if(gae_many(n_envs, steps))
        gae_many_kernel<<<(n_envs + GAE_ENVS - 1) / GAE_ENVS, GAE_ENVS, 0, (cudaStream_t)stream>>>(rewards, ld_rewards, all_values, ld_values, terminated, ld_terminated, truncated,
                                                                  ld_truncated, advantages, ld_advantages, target_values, ld_targets, n_envs, steps, gamma, lambda, ignore_termination);
    else
        gae_kernel<<<n_envs, GAE_THREADS, 0, (cudaStream_t)stream>>>(rewards, ld_rewards, all_values, ld_values, terminated, ld_terminated, truncated, ld_truncated,
                                                                  advantages, ld_advantages, target_values, ld_targets, n_envs, steps, gamma, lambda, ignore_termination);
    B200RL_LAUNCH_CHECK("gae");
    return B200RL_OK;
}

size_t b200rl_ppo_scratch_bytes(int batch, int action_dim){
    if(batch < 1 || action_dim < 1) return 0;
    return sizeof(float) * (2 + (size_t)((batch + PPO_THREADS - 1) / PPO_THREADS) * action_dim);
}

int b200rl_ppo_policy_gradient(const float* current_actions, int ld_current, const float* rollout_actions, int ld_rollout, const float* log_std,
                               const float* rollout_log_probs, int ld_log_probs, const float* advantages, int ld_advantages, float* d_actions, int ld_d,
                               float* d_log_std, int batch, int action_dim, float epsilon_clip, float entropy_coefficient, float advantage_epsilon,
                               int normalize_advantage, int learn_action_std, void* scratch, size_t scratch_bytes, b200rl_stream_t stream){
    if(!current_actions || !rollout_actions || !log_std || !rollout_log_probs || !advantages || !d_actions || batch < 0 || action_dim < 1 ||
       ld_current < action_dim || ld_rollout < action_dim || ld_d < action_dim || ld_log_probs < 1 || ld_advantages < 1) return B200RL_ERR_INVALID_ARGUMENT;
    if(learn_action_std && !d_log_std) return B200RL_ERR_INVALID_ARGUMENT;
    if(action_dim > PPO_MAX_ACTION_DIM) return B200RL_ERR_UNSUPPORTED;
    if(batch == 0) return B200RL_OK;
    if(!scratch || scratch_bytes < b200rl_ppo_scratch_bytes(batch, action_dim)) return B200RL_ERR_INVALID_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    float* stats = reinterpret_cast<float*>(scratch);
    const int blocks = (batch + PPO_THREADS - 1) / PPO_THREADS;
    if(normalize_advantage){
        ppo_adv_stats_kernel<<<1, 1024, 0, s>>>(advantages, ld_advantages, batch, stats);
        B200RL_LAUNCH_CHECK("ppo_adv_stats");
    }
    PpoArgs a{current_actions, ld_current, rollout_actions, ld_rollout, log_std, rollout_log_probs, ld_log_probs, advantages, ld_advantages, d_actions, ld_d,
              stats, stats + 2, batch, action_dim, epsilon_clip, advantage_epsilon, normalize_advantage, learn_action_std};
    ppo_gradient_kernel<<<blocks, PPO_THREADS, 0, s>>>(a);
    B200RL_LAUNCH_CHECK("ppo_gradient");
    if(learn_action_std){
        ppo_log_std_reduce_kernel<<<1, PPO_MAX_ACTION_DIM, 0, s>>>(d_log_std, stats + 2, blocks, action_dim, batch, entropy_coefficient);
        B200RL_LAUNCH_CHECK("ppo_log_std_reduce");
    }
    return B200RL_OK;
}

}

// ---------------------------------------------------------------------------------------------------------------
// Epoch shuffle: apply a row permutation to selected columns of the dataset matrix (gather into scratch, write back).
// ---------------------------------------------------------------------------------------------------------------
namespace b200rl {
// A CTA takes PERMUTE_ROWS rows, a thread every 256th element of them; the columns are found in a table. Bound by latency, then by HBM (65,536 rows of 38
// columns: 36 us with a 64-bit division and a walk through the mask per element).
constexpr int PERMUTE_ROWS = 64;
template <bool GATHER>
__global__ void __launch_bounds__(256) permute_rows_kernel(float* __restrict__ data, int ld, int n_rows, const int32_t* __restrict__ perm, unsigned long long mask, int n_cols,
                                    float* __restrict__ scratch){
    __shared__ int s_col[64], s_row[PERMUTE_ROWS];
    after_predecessor();
    data = opaque(data); perm = opaque(perm); scratch = opaque(scratch);
    const int row0 = blockIdx.x * PERMUTE_ROWS, rows = min(PERMUTE_ROWS, n_rows - row0);
    if(threadIdx.x < 64 && (mask >> threadIdx.x & 1)) s_col[__popcll(mask & ((1ull << threadIdx.x) - 1))] = threadIdx.x;
    if(threadIdx.x < rows) s_row[threadIdx.x] = GATHER ? perm[row0 + threadIdx.x] : row0 + threadIdx.x;
    __syncthreads();
    float* part = scratch + (size_t)row0 * n_cols;
    const int n = rows * n_cols;
#pragma unroll 4
    for(int i = threadIdx.x; i < n; i += 256){
        const int r = (int)((unsigned)i / (unsigned)n_cols), c = i - r * n_cols;
        float* at = data + (size_t)s_row[r] * ld + s_col[c];
        if(GATHER) part[i] = *at;
        else *at = part[i];
    }
}
}  // namespace b200rl

extern "C" size_t b200rl_permute_rows_scratch_bytes(int n_rows, unsigned long long column_mask){
    return sizeof(float) * (size_t)(n_rows > 0 ? n_rows : 0) * (size_t)__builtin_popcountll(column_mask);
}

extern "C" int b200rl_permute_rows(float* data, int ld, int n_rows, const int32_t* perm, unsigned long long column_mask, void* scratch, size_t scratch_bytes,
                                   b200rl_stream_t stream){
    const int n_cols = __builtin_popcountll(column_mask);
    if(!data || !perm || n_rows < 0 || ld < 1 || (ld < 64 && (column_mask >> ld) != 0)) return B200RL_ERR_INVALID_ARGUMENT;
    if(n_rows == 0 || n_cols == 0) return B200RL_OK;
    if(!scratch || scratch_bytes < b200rl_permute_rows_scratch_bytes(n_rows, column_mask)) return B200RL_ERR_INVALID_ARGUMENT;
    const int threads = 256;
    const unsigned blocks = (unsigned)((n_rows + b200rl::PERMUTE_ROWS - 1) / b200rl::PERMUTE_ROWS);
    cudaStream_t s = (cudaStream_t)stream;
    for(auto kernel : {b200rl::permute_rows_kernel<true>, b200rl::permute_rows_kernel<false>})
        B200RL_CUDA_TRY(b200rl::launch_after(kernel, dim3(blocks), dim3(threads), 0, s, data, ld, n_rows, perm, column_mask, n_cols, static_cast<float*>(scratch)));
    return B200RL_OK;
}

// Native, because a loop of small networks calls it every 100 us: as a dozen calls from Python it took 92 us of the host, more than an epoch's kernels (64 x 64 networks, 4,096 rows).
extern "C" int b200rl_shuffle_rows(float* data, int ld, int n_rows, unsigned long long column_mask, uint32_t* rng, int32_t* perm_host, int32_t* perm, void* scratch,
                                   size_t scratch_bytes, void* sent, void* used, b200rl_stream_t copy_stream, b200rl_stream_t stream){
    if(!data || !rng || !perm_host || !perm || !sent || !used || n_rows < 0 || ld < 1 || (ld < 64 && (column_mask >> ld) != 0) ||
       (n_rows > 0 && column_mask != 0 && (!scratch || scratch_bytes < b200rl_permute_rows_scratch_bytes(n_rows, column_mask)))) return B200RL_ERR_INVALID_ARGUMENT;
    cudaStream_t copies = (cudaStream_t)copy_stream, s = (cudaStream_t)stream;
    B200RL_CUDA_TRY(cudaEventSynchronize((cudaEvent_t)sent));
    int rc = b200rl_shuffle_permutation_host(rng, n_rows, perm_host);
    if(rc) return rc;
    B200RL_CUDA_TRY(cudaStreamWaitEvent(copies, (cudaEvent_t)used, 0));
    B200RL_CUDA_TRY(cudaMemcpyAsync(perm, perm_host, sizeof(int32_t) * (size_t)n_rows, cudaMemcpyHostToDevice, copies));
    B200RL_CUDA_TRY(cudaEventRecord((cudaEvent_t)sent, copies));
    B200RL_CUDA_TRY(cudaStreamWaitEvent(s, (cudaEvent_t)sent, 0));
    if((rc = b200rl_permute_rows(data, ld, n_rows, perm, column_mask, scratch, scratch_bytes, stream))) return rc;
    B200RL_CUDA_TRY(cudaEventRecord((cudaEvent_t)used, s));
    return B200RL_OK;
}
