// Fused rollout for environments given as device-function policies: reset-if-truncated, observe, actor forward
// (OBS_DIM -> H -> H -> 1, H one of 16 / 32 / 64 / 128), environment step, reward and episode counters for T steps in ONE launch, LANES threads per
// environment, the runner state in registers between steps, the actor's weights in shared memory. Serves the hidden
// widths other than 64 and, at width 64, the Acrobot variants with few environments; the rest of width 64 runs on the tensor-core kernel (rollout_tc.cu).
//
// A step is a serial chain and there are few environments: bound by latency. So an environment's hidden units are dealt out over LANES threads of a
// warp, a layer's units advance side by side with the summed index outermost (packed multiply-adds; per unit the order of the sums is that of
// the reference: bias first, inputs ascending, so the results do not depend on LANES), and the double-precision sines and cosines of an Acrobot step
// are evaluated by different lanes at the same time (envs.cuh).
#include "common.cuh"
#include "envs.cuh"
#include "rollout.cuh"

namespace b200rl {

struct EnvRolloutArgs {
    const float* params;        // actor arena: W1[H,OBS] b1[H] W2[H,H] b2[H] W3[1,H] b3[1]
    float* states;              // [n_envs, STATE_DIM]
    int32_t* episode_step; uint8_t* truncated; float* episode_return;
    const float* reset_states;  // [n_reset_rounds, n_envs, RESET_DIM]
    uint8_t* terminated;        // [n_steps * n_envs] or NULL
    int n_reset_rounds, n_envs, n_steps, step_limit;
    float* obs; float* act; float* rew;         // [n_steps * n_envs, OBS_DIM | 1 | 1], row = step * n_envs + env
    int* error_flag;
    int acts[3];
};

// v[2 c], v[2 c + 1] of lane l: units 4 (c LANES + l) ... + 3
template <int ACT, int N> __device__ __forceinline__ void activate_units(float2 (&v)[N]){
#pragma unroll
    for(int i = 0; i < N; i++){ v[i].x = activation<ACT>(v[i].x); v[i].y = activation<ACT>(v[i].y); }
}
template <int N> __device__ __forceinline__ void activate_units_rt(float2 (&v)[N], int act){
    B200RL_DISPATCH_ACT(act, activate_units<ACT>(v));
}
template <int H, int LANES> __device__ __forceinline__ void load_units(const float* row, int lane, float2 (&v)[H / LANES / 2]){
#pragma unroll
    for(int c = 0; c < H / LANES / 4; c++){
        const float4 t = *reinterpret_cast<const float4*>(row + 4 * (c * LANES + lane));
        v[2 * c] = make_float2(t.x, t.y); v[2 * c + 1] = make_float2(t.z, t.w);
    }
}
template <int H, int LANES> __device__ __forceinline__ void store_units(float* row, int lane, const float2 (&v)[H / LANES / 2]){
#pragma unroll
    for(int c = 0; c < H / LANES / 4; c++) *reinterpret_cast<float4*>(row + 4 * (c * LANES + lane)) = make_float4(v[2 * c].x, v[2 * c].y, v[2 * c + 1].x, v[2 * c + 1].y);
}
template <int H, int LANES> __device__ __forceinline__ void add_products(const float* weights, float x, int lane, float2 (&acc)[H / LANES / 2]){
    float2 w[H / LANES / 2];
    load_units<H, LANES>(weights, lane, w);
#pragma unroll
    for(int i = 0; i < H / LANES / 2; i++) acc[i] = __ffma2_rn(w[i], make_float2(x, x), acc[i]);
}

constexpr int ENV_MAX_WARPS = 8;
__host__ __device__ constexpr int env_pitch(int h){ return h + 4; }        // rows of the weights and of an environment's activations: 16-byte aligned, neighbours four banks apart
__host__ __device__ constexpr int env_weight_floats(int h, int obs){ return h * env_pitch(h) + obs * h + 3 * h + 4; }

template <typename ENV, int H, int LANES>
__global__ void __launch_bounds__(32 * ENV_MAX_WARPS, H / LANES <= 32 ? 2 : 1) rollout_env_kernel(EnvRolloutArgs a){
    constexpr int S = ENV::STATE_DIM, O = ENV::OBS_DIM, PER_WARP = 32 / LANES, PITCH = env_pitch(H);
    extern __shared__ __align__(16) float smem[];
    float* W2 = smem;                 // [H inputs][H units], rows of PITCH
    float* W1 = W2 + H * PITCH;       // [O inputs][H units]
    float* b1 = W1 + O * H;
    float* b2 = b1 + H;
    float* W3 = b2 + H;
    float* b3 = W3 + H;
    {
        const float* p = a.params;
        for(int i = threadIdx.x; i < H * O; i += blockDim.x) W1[(i % O) * H + i / O] = __ldg(p + i);
        p += H * O;
        for(int i = threadIdx.x; i < H; i += blockDim.x){ b1[i] = __ldg(p + i); b2[i] = __ldg(p + H + H * H + i); W3[i] = __ldg(p + H + H * H + H + i); }
        if(threadIdx.x == 0) *b3 = __ldg(p + H + H * H + 2 * H);
        p += H;
        for(int i = threadIdx.x; i < H * H; i += blockDim.x) W2[(i % H) * PITCH + i / H] = __ldg(p + i);
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, in_warp = (threadIdx.x & 31) / LANES, lane = threadIdx.x % LANES;
    const int first = (blockIdx.x * (blockDim.x >> 5) + warp) * PER_WARP;
    if(first >= a.n_envs) return;
    const bool valid = first + in_warp < a.n_envs;
    const int e = valid ? first + in_warp : a.n_envs - 1;                    // lanes without an environment of their own follow the last one and store nothing
    float* row1 = smem + env_weight_floats(H, O) + (warp * PER_WARP + in_warp) * PITCH;      // this environment's activations: written by its lanes, read by all of them
    float state[S];
#pragma unroll
    for(int k = 0; k < S; k++) state[k] = a.states[(size_t)e * S + k];
    int es = a.episode_step[e];
    bool trunc = a.truncated[e] != 0;
    float er = a.episode_return[e];
    int resets = 0;
    __syncwarp();                                    // every lane has the state before any lane may write it
    for(int t = 0; t < a.n_steps; t++){
        if(trunc){                                   // prologue: rl/components/off_policy_runner/operations_generic_per_env.h:8-61
            if(a.reset_states != nullptr && resets < a.n_reset_rounds){
                const float* rsp = a.reset_states + ((size_t)resets * a.n_envs + e) * ENV::RESET_DIM;      // scalar loads: the table may be a view at any 4-byte offset
                float draws[ENV::RESET_DIM];
#pragma unroll
                for(int k = 0; k < ENV::RESET_DIM; k++) draws[k] = __ldg(rsp + k);
                ENV::reset(state, draws);
            }
            else if(a.error_flag) *a.error_flag = 1;
            resets++; es = 0; er = 0.0f;
        }
        __syncwarp();
        float o[O];
        ENV::template observe_lanes<LANES>(state, o);
        const size_t row = (size_t)t * a.n_envs + e;
        if(valid){
#pragma unroll
            for(int k0 = 0; k0 < O; k0 += LANES){
                float v = o[k0];
#pragma unroll
                for(int k = 1; k < LANES && k0 + k < O; k++) v = lane == k ? o[k0 + k] : v;
                if(k0 + lane < O) a.obs[row * O + k0 + lane] = v;
            }
        }
        float2 acc[H / LANES / 2];                   // exact fp32 FMA chains in the reference's summation order
        load_units<H, LANES>(b1, lane, acc);
#pragma unroll
        for(int k = 0; k < O; k++) add_products<H, LANES>(W1 + k * H, o[k], lane, acc);
        activate_units_rt(acc, a.acts[0]);
        store_units<H, LANES>(row1, lane, acc);
        __syncwarp();
        load_units<H, LANES>(b2, lane, acc);
#pragma unroll (H / LANES <= 8 ? 4 : 1)
        for(int k = 0; k < H; k += 4){
            const float4 h = *reinterpret_cast<const float4*>(row1 + k);
            add_products<H, LANES>(W2 + (k + 0) * PITCH, h.x, lane, acc);
            add_products<H, LANES>(W2 + (k + 1) * PITCH, h.y, lane, acc);
            add_products<H, LANES>(W2 + (k + 2) * PITCH, h.z, lane, acc);
            add_products<H, LANES>(W2 + (k + 3) * PITCH, h.w, lane, acc);
        }
        activate_units_rt(acc, a.acts[1]);
        __syncwarp();
        store_units<H, LANES>(row1, lane, acc);
        __syncwarp();
        float out = *b3;
#pragma unroll 8
        for(int k = 0; k < H; k += 4){
            const float4 w = *reinterpret_cast<const float4*>(W3 + k), h = *reinterpret_cast<const float4*>(row1 + k);
            out = fmaf(w.x, h.x, out); out = fmaf(w.y, h.y, out); out = fmaf(w.z, h.z, out); out = fmaf(w.w, h.w, out);
        }
        const float action = activation_rt(out, a.acts[2]);
        float next[S];
        const float r = ENV::template transition_lanes<LANES>(state, action, next);        // epilogue: operations_generic_per_env.h:62-108
        es += 1; er = __fadd_rn(er, r);
        const bool term = ENV::TERMINATES && ENV::template terminated_lanes<LANES>(next);
        trunc = term || (es == a.step_limit);                        // operations_generic_per_env.h:93-97
        if(valid && lane == 0){
            a.act[row] = action; a.rew[row] = r;
            if(a.terminated) a.terminated[row] = term ? 1 : 0;
        }
#pragma unroll
        for(int k = 0; k < S; k++) state[k] = next[k];
    }
    if(!valid || lane != 0) return;
#pragma unroll
    for(int k = 0; k < S; k++) a.states[(size_t)e * S + k] = state[k];
    a.episode_step[e] = es; a.truncated[e] = trunc ? 1 : 0; a.episode_return[e] = er;
}

template <typename ENV, int H, int LANES>
static int launch_env_lanes(const EnvRolloutArgs& a, int sms, cudaStream_t s){
    constexpr int PER_WARP = 32 / LANES;
    const int warps = (a.n_envs + PER_WARP - 1) / PER_WARP;
    int per_cta = (warps + sms - 1) / sms;                           // spread over all SMs before CTAs grow
    if(per_cta > ENV_MAX_WARPS) per_cta = ENV_MAX_WARPS;
    constexpr size_t per_warp = sizeof(float) * PER_WARP * env_pitch(H), weights = sizeof(float) * env_weight_floats(H, ENV::OBS_DIM), largest = weights + ENV_MAX_WARPS * per_warp;
    static_assert(largest <= 227 * 1024, "shared memory");
    const size_t smem = weights + per_cta * per_warp;
    // always the largest, never this launch's: the limit belongs to the kernel, and another thread may be about to launch it for more environments
    if constexpr(largest > 48 * 1024) B200RL_CUDA_TRY(cudaFuncSetAttribute(rollout_env_kernel<ENV, H, LANES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)largest));
    rollout_env_kernel<ENV, H, LANES><<<(warps + per_cta - 1) / per_cta, 32 * per_cta, smem, s>>>(a);
    B200RL_LAUNCH_CHECK("rollout_env");
    return B200RL_OK;
}

// The hidden width is a template parameter (a lane's units live in registers): the widths of the reference's example policies are
// instantiated, any other is refused. The more lanes an environment has, the shorter its step and the fewer environments fill the GPU:
// measured (us per step), the lines cross near 24 environments per SM (Acrobot, width 64, 4,000 environments: 6.0 with 16 lanes, 5.8 with 4; 1,003: 3.8 and
// 5.2) and 64 per SM (width 32, 16,384: 5.8 with 4 lanes, 5.9 with 1; width 128: 40 and 26; 8,000: 19 and 22). Before, with one thread per
// environment and a dot product at a time, a step took 12.0 us at width 32 and 74 us at width 128.
template <typename ENV, int H>
static int launch_env_width(const EnvRolloutArgs& a, cudaStream_t s){
    int sms = 0;
    const int rc = sm_count(&sms);
    if(rc) return rc;
    if constexpr(H >= 64){
        if(a.n_envs <= 24 * sms) return launch_env_lanes<ENV, H, 16>(a, sms, s);
    }
    if(H == 64 || a.n_envs <= 64 * sms) return launch_env_lanes<ENV, H, 4>(a, sms, s);
    if constexpr(H != 64) return launch_env_lanes<ENV, H, 1>(a, sms, s);
    return B200RL_ERR_UNSUPPORTED;
}
template <typename ENV>
static int launch_env(const EnvRolloutArgs& a, int hidden, cudaStream_t s){
    switch(hidden){
        case 16:  return launch_env_width<ENV, 16>(a, s);
        case 32:  return launch_env_width<ENV, 32>(a, s);
        case 64:
            if constexpr(ENV::STATE_DIM == 4) return launch_env_width<ENV, 64>(a, s);
            return B200RL_ERR_UNSUPPORTED;
        case 128: return launch_env_width<ENV, 128>(a, s);
        default:  return B200RL_ERR_UNSUPPORTED;
    }
}

}  // namespace b200rl
using namespace b200rl;

extern "C" int b200rl_env_observation_dim(int env){ return env == B200RL_ENV_PENDULUM ? 3 : (env == B200RL_ENV_ACROBOT_SWINGUP || env == B200RL_ENV_ACROBOT) ? 6 : 0; }
extern "C" int b200rl_env_state_dim(int env){ return env == B200RL_ENV_PENDULUM ? 2 : (env == B200RL_ENV_ACROBOT_SWINGUP || env == B200RL_ENV_ACROBOT) ? 4 : 0; }
extern "C" int b200rl_env_reset_dim(int env){ return env == B200RL_ENV_ACROBOT ? 4 : (env == B200RL_ENV_PENDULUM || env == B200RL_ENV_ACROBOT_SWINGUP) ? 2 : 0; }

extern "C" int b200rl_env_rollout(int env, const b200rl_mlp_shape* actor, const float* actor_params, float* states, int32_t* episode_step, uint8_t* truncated,
                                  float* episode_return, const float* reset_states, int n_reset_rounds, int n_envs, int n_steps, int step_limit, float* obs,
                                  float* act, float* rew, int* error_flag, b200rl_stream_t stream){
    return b200rl_env_rollout_flags(env, actor, actor_params, states, episode_step, truncated, episode_return, reset_states, n_reset_rounds, n_envs, n_steps, step_limit,
                                    obs, act, rew, nullptr, error_flag, stream);
}
extern "C" int b200rl_env_rollout_flags(int env, const b200rl_mlp_shape* actor, const float* actor_params, float* states, int32_t* episode_step, uint8_t* truncated,
                                        float* episode_return, const float* reset_states, int n_reset_rounds, int n_envs, int n_steps, int step_limit, float* obs,
                                        float* act, float* rew, uint8_t* terminated, int* error_flag, b200rl_stream_t stream){
    const int O = b200rl_env_observation_dim(env);
    if(O == 0 || !actor) return B200RL_ERR_INVALID_ARGUMENT;
    if(actor->n_layers != 3 || actor->input_dim != O || actor->dims[0] != actor->dims[1] || actor->dims[2] != 1) return B200RL_ERR_UNSUPPORTED;
    const int H = actor->dims[0];
    if(H != 16 && H != 32 && H != 64 && H != 128) return B200RL_ERR_UNSUPPORTED;
    for(int l = 0; l < 3; l++) if(!valid_activation(actor->acts[l])) return B200RL_ERR_INVALID_ARGUMENT;
    if(!actor_params || !states || !episode_step || !truncated || !episode_return || !obs || !act || !rew || n_envs < 0 || n_steps < 0 || n_reset_rounds < 0 || step_limit < 1)
        return B200RL_ERR_INVALID_ARGUMENT;
    if(reset_states == nullptr && n_reset_rounds != 0) return B200RL_ERR_INVALID_ARGUMENT;
    if(n_envs == 0 || n_steps == 0) return B200RL_OK;
    // Width 64: the tensor-core kernel (second layer as split-fp16 MMAs, the environment as its compile-time policy) for the Pendulum, whose results are the
    // same bits whatever the number of environments, and for the Acrobots beyond 60 environments per SM (9.4 us per step from 500 environments to
    // 65,536; the lanes' 7.5 us at 8,000 environments, 12.6 at 16,384).
    int sms = 0;
    const int rc = sm_count(&sms);
    if(rc) return rc;
    if(H == 64 && (env == B200RL_ENV_PENDULUM || n_envs > 60 * sms)){
        RolloutArgs t{};
        t.params = actor_params; t.states = states; t.episode_step = episode_step; t.truncated = truncated; t.episode_return = episode_return;
        t.reset_states = reset_states; t.n_reset_rounds = n_reset_rounds; t.n_envs = n_envs; t.env_begin = 0; t.env_count = n_envs;
        t.n_steps = n_steps; t.step_limit = step_limit; t.obs = obs; t.act = act; t.rew = rew; t.terminated = terminated; t.error_flag = error_flag;
        for(int l = 0; l < 3; l++) t.acts[l] = actor->acts[l];
        return launch_env_rollout_tc(env, t, (cudaStream_t)stream);
    }
    EnvRolloutArgs a{};
    a.params = actor_params; a.states = states; a.episode_step = episode_step; a.truncated = truncated; a.episode_return = episode_return;
    a.reset_states = reset_states; a.n_reset_rounds = n_reset_rounds; a.n_envs = n_envs; a.n_steps = n_steps; a.step_limit = step_limit;
    a.obs = obs; a.act = act; a.rew = rew; a.terminated = terminated; a.error_flag = error_flag;
    for(int l = 0; l < 3; l++) a.acts[l] = actor->acts[l];
    if(env == B200RL_ENV_PENDULUM) return launch_env<PendulumEnv>(a, H, (cudaStream_t)stream);
    if(env == B200RL_ENV_ACROBOT) return launch_env<AcrobotEnv>(a, H, (cudaStream_t)stream);
    return launch_env<AcrobotSwingupEnv>(a, H, (cudaStream_t)stream);
}
