// Weight and bias gradients of all layers over large batches in one launch (sm_100a, tcgen05 + TMEM): dW_l += d_pre_l^T input_l for the d_pre that the
// backward pass of mlp_chain.cu has left in memory (the gradient part of nn/layers/dense/operations_generic.h's backward).
//
// Arithmetic: fp32 operands as two fp16 parts and three passes, as in mlp_chain.cu. The summed index is the batch row here, so the powers of two that bring
// the values into fp16's range belong to columns: every column of a unit of 32 rows is scaled by its largest magnitude. A chain of MMAs is
// one unit (6 MMAs); the units are added, unscaled, in fp32 registers.
//
// A CTA works on one job (up to 128 columns of one operand by up to 256 of the other: two jobs for a 256 x 256 layer) over a contiguous range of rows; all
// jobs have the same number of ranges, as many as fill the SMs. Both operands lie in memory with the rows as the outer index and go into shared memory
// in that order: the tensor core takes them MN-major, nothing is transposed. TMA brings the fp32 rows of the next units into a ring of
// shared-memory slots, zeros outside the matrices. Twelve warps (40 registers) stage: a warp takes 32 columns of a unit, largest magnitude per column by
// shuffles, split, 8-byte stores into the 128-byte-swizzled tile, and the sums of the d_pre columns (the bias gradient) on the way; if a job has few
// such column groups, the warps form teams that take the units in turn. Eight warps (168 registers) hold the sums, 128 a thread, and move the units
// from tensor memory into them. One thread each of two further warps issues the copies and the MMAs. (All warps staging and summing in turn
// took twice as long: both are chains of latencies, and the one waited for the other; so did a staging warp that also issued the copies.)
//
// Bound by the staging warps (shared memory: a unit crosses it four times), about 3,300 cycles per unit of 128 + 256 columns. Measured, 64-256-256-256-16
// at 1,048,576 rows: 2.53 ms for the gradients of all layers (6.8 GB, 1.0 ms at the copy bandwidth; the products per layer with their reductions took 3.6 ms),
// 0.65 ms less than asynchronous copies of each thread's own values, 1.0 ms less than the copies in registers.
#include "common.cuh"
#include "tcgen05.cuh"
#include "split_f16.cuh"
#include <atomic>
#include <cuda.h>
#include <cudaTypedefs.h>

namespace b200rl {

namespace {
constexpr int GR_SUM_WARPS = 8, GR_STAGING_WARPS = 12, GR_THREADS = 32 * (GR_SUM_WARPS + GR_STAGING_WARPS + 4), GR_UNIT = 32, GR_MAX_STAGES = 6, GR_MAX_JOBS = 2 * 8;
constexpr uint32_t GR_BLOCK = GR_UNIT * 128;                     // one part of 64 columns of a unit: 32 rows x 128 bytes
constexpr uint32_t GR_TILES = 2 * 48 * 1024, GR_RAW = 2 * 48 * 1024;        // two stages of tiles and two slots of fp32 rows of 128 + 256 columns; up to six of narrower ones
                                                                              // (64 + 64 columns: a copy takes longer than a unit; 202,203 rows of 29-64-64-5 114 us with four, 102 with six)
// inverse scales of the columns, by unit: who stages unit u has waited for the MMAs of a unit at least u - GR_MAX_STAGES, which have waited for
// the accumulator of the unit two before it to be read
constexpr uint32_t GR_SCALES = 128 + 256, GR_SCALE_BUFFERS = GR_MAX_STAGES + 2;
constexpr uint32_t GR_SMEM = GR_TILES + GR_RAW + 4 * GR_SCALES * GR_SCALE_BUFFERS + 256 + 1024;
static_assert(GR_SMEM <= 227 * 1024, "shared memory");
constexpr long long GR_WAIT_LIMIT = 2000000000LL;
constexpr int GR_SEGMENT = 128;                                  // units that are added in registers before they go into the record: one sum over a range of
                                                                 // 390 units (2^18 rows) is off by 3.8e-7, four of a hundred by 2.6e-7, the products with their own splits before by 2.6e-7
}

struct GradJob {
    CUtensorMap a, b;                                 // boxes of a unit's rows by M (up to 128) and N (up to 256) columns, rounded up to 32
    int M, N, from;                                   // a's first column
    long long at, stride_m, stride_n;                 // where element (m, n) goes in a record
    long long bias; int bias_of;                      // 1: a's column sums are the bias gradient, 2: b's; 0: another job's business
};
struct GradArgs { GradJob job[GR_MAX_JOBS]; int n_jobs, splits, rows, accumulate; float* partial; long long record; };

__device__ int g_grad_error = 0;

namespace {
// operand with the row as the outer index, columns in blocks of 64 (128 bytes, swizzled): 8-row groups 1024 bytes apart, column blocks GR_BLOCK apart
__device__ __forceinline__ uint64_t make_desc_mnmajor_sw128(uint32_t smem_addr){
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
    d |= (uint64_t)(GR_BLOCK >> 4) << 16;                 // leading byte offset: next 64 columns
    d |= (uint64_t)(1024 >> 4) << 32;                     // stride byte offset: next 8 rows
    d |= (uint64_t)1 << 46;                               // descriptor version (Blackwell)
    d |= (uint64_t)2 << 61;                               // layout type: SWIZZLE_128B
    return d;
}
__device__ __forceinline__ void ld_16_columns(uint32_t taddr, uint32_t (&r)[16]){
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* smem, const CUtensorMap* map, int column, int row, uint64_t* bar){
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 :: "r"(tc::smem_u32(smem)), "l"(map), "r"(column), "r"(row), "r"(tc::smem_u32(bar)) : "memory");
}
// this thread's rows of a unit: t = lane >> 3 and load i -> row. Rows 4 apart land in different halves of the banks (the swizzle): the two rows of a
// half warp, so that an 8-byte store of a warp takes two wavefronts, not four
__device__ __forceinline__ int unit_row(int t, int i){ return (t >> 1) + 4 * (t & 1) + 2 * (i & 1) + 8 * (i >> 1); }
}  // namespace

__global__ void __launch_bounds__(GR_THREADS, 1) mlp_grad_kernel(const __grid_constant__ GradArgs a){
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* raw = base + GR_TILES;
    float* bias = reinterpret_cast<float*>(raw);                                    // at the end: [team][256]
    float* scales = reinterpret_cast<float*>(raw + GR_RAW);                          // [unit % GR_SCALE_BUFFERS][128 of a, 256 of b]
    uint64_t* full = reinterpret_cast<uint64_t*>(scales + GR_SCALE_BUFFERS * GR_SCALES);
    uint64_t* empty = full + GR_MAX_STAGES; uint64_t* raw_full = empty + GR_MAX_STAGES; uint64_t* raw_empty = raw_full + GR_MAX_STAGES;
    uint64_t* acc_full = raw_empty + GR_MAX_STAGES; uint64_t* acc_empty = acc_full + 2;
    uint32_t* slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    after_predecessor();
    const int split = blockIdx.x / a.n_jobs;
    const GradJob& y = a.job[blockIdx.x - split * a.n_jobs];
    const int M = y.M, N = y.N, n = (N + 15) / 16 * 16;
    const int groups_a = (M + 31) / 32, groups_b = (N + 31) / 32, groups = groups_a + groups_b;
    const uint32_t blocks_a = (M + 63) / 64, blocks_b = (N + 63) / 64, stage_bytes = 2 * GR_BLOCK * (blocks_a + blocks_b);
    const uint32_t row_a = 128 * groups_a, row_b = 128 * groups_b, raw_bytes = GR_UNIT * (row_a + row_b);       // bytes of a row
    // A team always comes back to the same slots and stages (their numbers are multiples of the number of teams): a warp that waits for a phase has
    // itself seen the one before it complete, which a wait by parity takes for granted.
    const int room = min(min(GR_MAX_STAGES, (int)(GR_TILES / stage_bytes)), (int)(GR_RAW / raw_bytes)), teams = min(room, GR_STAGING_WARPS / groups);
    const int stages = room / teams * teams, slots = stages;
    const int all = (a.rows + GR_UNIT - 1) / GR_UNIT, first = (int)((long long)all * split / a.splits), units = (int)((long long)all * (split + 1) / a.splits) - first;
    if(tid == 0){
        for(int i = 0; i < GR_MAX_STAGES; i++){ tc::mbar_init(full + i, groups); tc::mbar_init(empty + i, 1); tc::mbar_init(raw_full + i, 1); tc::mbar_init(raw_empty + i, groups); }
        for(int i = 0; i < 2; i++){ tc::mbar_init(acc_full + i, 1); tc::mbar_init(acc_empty + i, GR_SUM_WARPS); }
        tc::fence_mbar_init(); *abort_flag = 0;
    }
    if(warp == 0){ tc::tmem_alloc(slot, 512); tc::tmem_relinquish(); }
    tc::fence_before_thread_sync();
    __syncthreads();
    tc::fence_after_thread_sync();
    const uint32_t tmem = *slot;
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
        if(tc::mbar_try_wait(bar, parity)) return true;
        const long long t0 = clock64();
        while(!tc::mbar_try_wait(bar, parity)){
            if(*abort_flag || clock64() - t0 > GR_WAIT_LIMIT){ *abort_flag = 1; g_grad_error = 1; return false; }
        }
        return true;
    };
    if(warp < GR_SUM_WARPS){
        tc::setmaxnreg_inc<168>();
        const int q = warp & 3, g = warp >> 2, chunks = n / 16;
        const uint32_t tmem_lane = tmem + ((uint32_t)(q * 32) << 16);
        const float2 zero = make_float2(0.0f, 0.0f);
        float2 acc[8][8];                                               // row 32 q + lane; columns 16 (2 p + g) + 2 i, + 1
#pragma unroll
        for(int p = 0; p < 8; p++)
#pragma unroll
            for(int i = 0; i < 8; i++) acc[p][i] = zero;
        // A range may have no unit (2,048 rows of 128-256-16: 64 units for 74 ranges): one segment of none, whose record is zeros
        const int segments = max(1, (units + GR_SEGMENT - 1) / GR_SEGMENT), segment = (units + segments - 1) / segments;
        for(int begin = 0; ; begin += segment){
        const int end = min(units, begin + segment);
        for(int d = begin; d < end; d++){
            if(!wait(acc_full + (d & 1), (d >> 1) & 1u)) break;
            tc::fence_after_thread_sync();
            const float* inverse = scales + (d % GR_SCALE_BUFFERS) * GR_SCALES;
            const float mine = inverse[32 * q + lane];
            const float2 row = make_float2(mine, mine);
#pragma unroll
            for(int p = 0; p < 8; p++){
                const int c = 2 * p + g;
                if(c >= chunks) break;
                uint32_t x[16];
                ld_16_columns(tmem_lane + (uint32_t)(d & 1) * 256 + 16 * c, x);
                tc::tmem_wait_ld();
#pragma unroll
                for(int j = 0; j < 4; j++){
                    const float4 f = *reinterpret_cast<const float4*>(inverse + 128 + 16 * c + 4 * j);
                    acc[p][2 * j] = __ffma2_rn(make_float2(__uint_as_float(x[4 * j]), __uint_as_float(x[4 * j + 1])), __ffma2_rn(row, make_float2(f.x, f.y), zero), acc[p][2 * j]);
                    acc[p][2 * j + 1] = __ffma2_rn(make_float2(__uint_as_float(x[4 * j + 2]), __uint_as_float(x[4 * j + 3])), __ffma2_rn(row, make_float2(f.z, f.w), zero), acc[p][2 * j + 1]);
                }
            }
            tc::fence_before_thread_sync();
            __syncwarp();
            if(lane == 0) tc::mbar_arrive(acc_empty + (d & 1));
        }
        // ---- this range's record ----
        if(32 * q + lane < M){
            float* to = a.partial + split * a.record + y.at + (32 * q + lane) * y.stride_m;
            const bool add = begin > 0 || a.accumulate;
#pragma unroll
            for(int p = 0; p < 8; p++){
                if(16 * (2 * p + g) >= N) break;
                float old[16];                                           // all of them asked for before the first store
#pragma unroll
                for(int i = 0; i < 16; i++){ const int c = 16 * (2 * p + g) + i; old[i] = add && c < N ? to[c * y.stride_n] : 0.0f; }
#pragma unroll
                for(int i = 0; i < 16; i++){
                    const int c = 16 * (2 * p + g) + i;
                    const float v = i & 1 ? acc[p][i >> 1].y : acc[p][i >> 1].x;
                    if(c < N) to[c * y.stride_n] = add ? old[i] + v : v;
                }
            }
        }
        if(end >= units || *abort_flag) break;
#pragma unroll
        for(int p = 0; p < 8; p++)
#pragma unroll
            for(int i = 0; i < 8; i++) acc[p][i] = zero;
        }
    }
    else if(warp >= GR_SUM_WARPS + GR_STAGING_WARPS){
        tc::setmaxnreg_dec<24>();
        if(warp == GR_SUM_WARPS + GR_STAGING_WARPS && lane == 0){
            const uint32_t idesc = tc::make_idesc_f16(128, n) | (1u << 15) | (1u << 16);          // both operands MN-major
            for(int u = 0; u < units; u++){
                const uint32_t s = (uint32_t)(u % stages), d = tmem + (u & 1u) * 256;
                if(!wait(acc_empty + (u & 1), ((u >> 1) & 1u) ^ 1u) || !wait(full + s, (u / stages) & 1u)) break;
                tc::fence_after_thread_sync();
                // (a's descriptors span 128 columns: from a narrower operand's second block, whatever lies there, come rows of the accumulator that nobody reads)
                const uint32_t at = tc::smem_u32(base + s * stage_bytes), at_b = at + 2 * blocks_a * GR_BLOCK;
                const uint64_t a_lead = make_desc_mnmajor_sw128(at), a_rest = make_desc_mnmajor_sw128(at + blocks_a * GR_BLOCK);
                const uint64_t b_lead = make_desc_mnmajor_sw128(at_b), b_rest = make_desc_mnmajor_sw128(at_b + blocks_b * GR_BLOCK);
                // the small products first; 16 rows are 2048 bytes
                for(int k = 0; k < 2; k++) tc::mma_f16_ss(d, a_rest + (uint64_t)(128 * k), b_lead + (uint64_t)(128 * k), idesc, k ? 1u : 0u);
                for(int k = 0; k < 2; k++) tc::mma_f16_ss(d, a_lead + (uint64_t)(128 * k), b_rest + (uint64_t)(128 * k), idesc, 1u);
                for(int k = 0; k < 2; k++) tc::mma_f16_ss(d, a_lead + (uint64_t)(128 * k), b_lead + (uint64_t)(128 * k), idesc, 1u);
                tc::commit(acc_full + (u & 1));
                tc::commit(empty + s);
            }
        }
        else if(warp == GR_SUM_WARPS + GR_STAGING_WARPS + 1 && lane == 0){
            int u = 0;
            for(; u < units; u++){
                uint64_t* bar = raw_full + u % slots;
                uint8_t* to = raw + u % slots * raw_bytes;
                if(!wait(raw_empty + u % slots, ((u / slots) & 1u) ^ 1u)) break;
                tc::mbar_expect_tx(bar, raw_bytes);
                tma_load_2d(to, &y.a, y.from, (first + u) * GR_UNIT, bar);
                tma_load_2d(to + GR_UNIT * row_a, &y.b, 0, (first + u) * GR_UNIT, bar);
                tc::mbar_arrive(bar);
            }
            // every copy that was started must have landed before the CTA may leave
            for(int k = max(0, u - slots); k < u; k++) tc::mbar_wait_bounded(raw_full + k % slots, (k / slots) & 1u, GR_WAIT_LIMIT);
        }
    }
    else{
        tc::setmaxnreg_dec<40>();
        const int w = warp - GR_SUM_WARPS, team = w / groups, group = w - team * groups, t = lane >> 3;
        const bool of_a = group < groups_a, loads = team < teams;
        const int col = 32 * (of_a ? group : group - groups_a) + 4 * (lane & 7);          // of the operand
        const bool sums = loads && y.bias_of == (of_a ? 1 : 2);
        const uint32_t part = (of_a ? blocks_a : blocks_b) * GR_BLOCK, row_bytes = of_a ? row_a : row_b;
        const uint32_t chunk = (uint32_t)(col & 63) >> 3;
        const uint32_t tile = (of_a ? 0u : 2 * blocks_a * GR_BLOCK) + (uint32_t)(col >> 6) * GR_BLOCK + (uint32_t)(col & 4) * 2;
        const float2 zero = make_float2(0.0f, 0.0f);
        // column sums: of eight units' rows, of all. One sum over a range's thousands of rows loses three times what sums of this kind lose (2^18 rows:
        // 1.2e-6 of the bias gradient, 3.7e-7 this way; the pass before this kernel 3.6e-7)
        float2 sum0 = zero, sum1 = zero, some0 = zero, some1 = zero;
        int in_some = 0;
        for(int u = team; loads && u < units; u += teams){
            const int s = u % stages, k = u % slots;
            bool ok = wait(raw_full + k, (u / slots) & 1u);
            if(!__all_sync(0xffffffffu, ok)) break;
            const uint8_t* from = raw + k * raw_bytes + (of_a ? 0u : GR_UNIT * row_a) + 4 * col;
            float4 big = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for(int i = 0; i < 8; i++){
                const float4 v = *reinterpret_cast<const float4*>(from + unit_row(t, i) * row_bytes);
                big.x = fmaxf(big.x, fabsf(v.x)); big.y = fmaxf(big.y, fabsf(v.y)); big.z = fmaxf(big.z, fabsf(v.z)); big.w = fmaxf(big.w, fabsf(v.w));
                if(sums){ some0 = __fadd2_rn(some0, make_float2(v.x, v.y)); some1 = __fadd2_rn(some1, make_float2(v.z, v.w)); }
            }
            if((++in_some & 7) == 0){ sum0 = __fadd2_rn(sum0, some0); sum1 = __fadd2_rn(sum1, some1); some0 = zero; some1 = zero; }
#pragma unroll
            for(int o = 8; o <= 16; o += 8){
                big.x = fmaxf(big.x, __shfl_xor_sync(0xffffffffu, big.x, o)); big.y = fmaxf(big.y, __shfl_xor_sync(0xffffffffu, big.y, o));
                big.z = fmaxf(big.z, __shfl_xor_sync(0xffffffffu, big.z, o)); big.w = fmaxf(big.w, __shfl_xor_sync(0xffffffffu, big.w, o));
            }
            const uint32_t e0 = scale_exponent(big.x), e1 = scale_exponent(big.y), e2 = scale_exponent(big.z), e3 = scale_exponent(big.w);
            const float2 f0 = make_float2(scale_of(e0), scale_of(e1)), f1 = make_float2(scale_of(e2), scale_of(e3));
            ok = wait(empty + s, ((u / stages) & 1u) ^ 1u);
            if(!__all_sync(0xffffffffu, ok)) break;
            if(t == 0)
                *reinterpret_cast<float4*>(scales + (u % GR_SCALE_BUFFERS) * GR_SCALES + (of_a ? 0 : 128) + col) =
                    make_float4(inverse_scale_of(e0), inverse_scale_of(e1), inverse_scale_of(e2), inverse_scale_of(e3));
            uint8_t* to = base + s * stage_bytes + tile;
#pragma unroll
            for(int i = 0; i < 8; i++){
                const float4 v = *reinterpret_cast<const float4*>(from + unit_row(t, i) * row_bytes);
                const uint32_t r = unit_row(t, i), off = r * 128 + ((chunk ^ (r & 7u)) << 4);
                uint32_t l0, l1, r0, r1;
                split_pair(__ffma2_rn(make_float2(v.x, v.y), f0, zero), l0, r0);
                split_pair(__ffma2_rn(make_float2(v.z, v.w), f1, zero), l1, r1);
                *reinterpret_cast<uint2*>(to + off) = make_uint2(l0, l1);
                *reinterpret_cast<uint2*>(to + part + off) = make_uint2(r0, r1);
            }
            tc::fence_proxy_async_smem();
            __syncwarp();
            if(lane == 0){
                tc::mbar_arrive(full + s);
                tc::mbar_arrive(raw_empty + k);
            }
        }
        tc::named_barrier_sync(1, 32 * GR_STAGING_WARPS);               // every warp's last reads of `raw`
        if(sums){
            sum0 = __fadd2_rn(sum0, some0); sum1 = __fadd2_rn(sum1, some1);
#pragma unroll
            for(int o = 8; o <= 16; o += 8){
                sum0.x += __shfl_xor_sync(0xffffffffu, sum0.x, o); sum0.y += __shfl_xor_sync(0xffffffffu, sum0.y, o);
                sum1.x += __shfl_xor_sync(0xffffffffu, sum1.x, o); sum1.y += __shfl_xor_sync(0xffffffffu, sum1.y, o);
            }
            if(t == 0) *reinterpret_cast<float4*>(bias + 256 * team + col) = make_float4(sum0.x, sum0.y, sum1.x, sum1.y);
        }
    }
    tc::fence_before_thread_sync();
    __syncthreads();
    if(y.bias_of && tid < (y.bias_of == 1 ? M : N)){
        float s = 0.0f;
        for(int k = 0; k < teams; k++) s += bias[256 * k + tid];
        float* at = a.partial + split * a.record + y.bias + tid;
        *at = a.accumulate ? *at + s : s;
    }
    if(warp == 0) tc::tmem_dealloc(tmem, 512);
}

// Rows of `from` with row pitch ld into rows of a pitch that is a multiple of four, zeros behind the columns. A thread takes four 16-byte pieces of the result, with all of their
// loads under way; bound by HBM (202,203 rows of 29 columns, 49 MB: 21.9 us with an element and a 64-bit division at a time, 9.1 us this way).
constexpr int PAD_PIECES = 4;
__global__ void __launch_bounds__(256) pad_rows_kernel(const float* __restrict__ from, long long ld, unsigned pieces, unsigned per_row, int cols, float4* __restrict__ to){
    after_predecessor();
    from = opaque(from);
    const unsigned first = blockIdx.x * (256u * PAD_PIECES) + threadIdx.x;
    float v[PAD_PIECES][4];
#pragma unroll
    for(int k = 0; k < PAD_PIECES; k++){
        const unsigned i = first + 256u * k, r = i / per_row;
        const int c = 4 * (int)(i - r * per_row);
#pragma unroll
        for(int j = 0; j < 4; j++) v[k][j] = i < pieces && c + j < cols ? __ldg(from + (long long)r * ld + c + j) : 0.0f;
    }
#pragma unroll
    for(int k = 0; k < PAD_PIECES; k++) if(first + 256u * k < pieces) to[first + 256u * k] = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
}

// ---- host side ---------------------------------------------------------------------------------------------------------------------------
// the word that a kernel's expired wait sets, and its reset (b200rl_device_error_state, b200rl_device_error_clear)
int mlp_grad_error_get(int* word){ B200RL_CUDA_TRY(cudaMemcpyFromSymbol(word, g_grad_error, sizeof(int))); return B200RL_OK; }
int mlp_grad_error_clear(){ const int zero = 0; B200RL_CUDA_TRY(cudaMemcpyToSymbol(g_grad_error, &zero, sizeof(int))); return B200RL_OK; }

int pad_rows(const float* from, long long ld, int rows, int cols, float* to, cudaStream_t s){
    const unsigned per_row = (unsigned)(cols + 3) / 4, pieces = (unsigned)rows * per_row;            // at most 2^18 rows (a chunk of the backward pass) of 64 pieces
    B200RL_CUDA_TRY(launch_after(pad_rows_kernel, dim3((pieces + 256 * PAD_PIECES - 1) / (256 * PAD_PIECES)), dim3(256), 0, s, from, ld, pieces, per_row, cols, reinterpret_cast<float4*>(to)));
    return B200RL_OK;
}
// Which operand gives the 128 rows of an accumulator: the input, whose gradient elements then lie next to each other in memory, unless that takes more jobs
static bool grad_rows_are_inputs(int O, int I){ return (I + 127) / 128 <= (O + 127) / 128; }
static int grad_jobs(int O, int I){ return ((grad_rows_are_inputs(O, I) ? I : O) + 127) / 128; }
int mlp_grad_splits(const b200rl_mlp_shape* sh){
    int jobs = 0, I = sh->input_dim;
    for(int l = 0; l < sh->n_layers; l++){ jobs += grad_jobs(sh->dims[l], I); I = sh->dims[l]; }
    return NUM_SMS / jobs;
}
// cuTensorMapEncodeTiled, from the driver through the runtime (nothing links against libcuda)
static int tensor_map_encoder(PFN_cuTensorMapEncodeTiled_v12000* encode){
    static std::atomic<void*> entry{nullptr};
    void* p = entry.load(std::memory_order_acquire);
    if(!p){
        cudaDriverEntryPointQueryResult result;
        B200RL_CUDA_TRY(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &result));
        if(result != cudaDriverEntryPointSuccess || !p) return B200RL_ERR_UNSUPPORTED;
        entry.store(p, std::memory_order_release);
    }
    *encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    return B200RL_OK;
}
// For every layer: d_pre[l] [rows, dims[l]] and input[l] [rows, its inputs], bases and row pitches multiples of 16 bytes. partial: mlp_grad_splits
// records of a gradient arena each; accumulate: add to what is there.
int mlp_grad_launch(const b200rl_mlp_shape* sh, const float* const* input, const long long* ld_input, const float* const* d_pre, const long long* ld_pre, int rows,
                    float* partial, long long record, bool accumulate, cudaStream_t s){
    static std::atomic<bool> configured[MAX_DEVICES];
    int dev = 0;
    int rc = current_device(&dev);
    if(rc) return rc;
    PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if((rc = tensor_map_encoder(&encode))) return rc;
    if(!configured[dev].load(std::memory_order_acquire)){
        B200RL_CUDA_TRY(cudaFuncSetAttribute(mlp_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GR_SMEM));
        configured[dev].store(true, std::memory_order_release);
    }
    GradArgs a{};
    a.rows = rows; a.splits = mlp_grad_splits(sh); a.partial = partial; a.record = record; a.accumulate = accumulate;
    auto operand = [&](CUtensorMap* map, const float* p, long long ld, int cols, int box){
        const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * sizeof(float)};
        const cuuint32_t boxes[2] = {(cuuint32_t)((box + 31) / 32 * 32), (cuuint32_t)GR_UNIT}, steps[2] = {1, 1};
        return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(p), dims, strides, boxes, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    bool encoded = true;
    int I = sh->input_dim;
    long long at = 0;
    for(int l = 0; l < sh->n_layers; l++){
        const int O = sh->dims[l], jobs = grad_jobs(O, I);
        const bool rows_are_inputs = grad_rows_are_inputs(O, I);
        for(int j = 0; j < jobs; j++){
            GradJob& y = a.job[a.n_jobs++];
            const int from = 128 * j, all = rows_are_inputs ? I : O, cols = all - from < 128 ? all - from : 128;
            y.M = cols; y.from = from;
            if(rows_are_inputs){
                y.N = O;
                encoded = encoded && operand(&y.a, input[l], ld_input[l], I, cols) && operand(&y.b, d_pre[l], ld_pre[l], O, O);
                y.at = at + from; y.stride_m = 1; y.stride_n = I;
                y.bias_of = j == 0 ? 2 : 0; y.bias = at + (long long)O * I;
            }
            else{
                y.N = I;
                encoded = encoded && operand(&y.a, d_pre[l], ld_pre[l], O, cols) && operand(&y.b, input[l], ld_input[l], I, I);
                y.at = at + (long long)from * I; y.stride_m = I; y.stride_n = 1;
                y.bias_of = 1; y.bias = at + (long long)O * I + from;
            }
        }
        at += (long long)O * I + O;
        I = O;
    }
    if(!encoded) return B200RL_ERR_INVALID_ARGUMENT;
    B200RL_CUDA_TRY(launch_after(mlp_grad_kernel, dim3(a.n_jobs * a.splits), dim3(GR_THREADS), GR_SMEM, s, a));
    B200RL_LAUNCH_CHECK("mlp_grad");
    return B200RL_OK;
}

}  // namespace b200rl
