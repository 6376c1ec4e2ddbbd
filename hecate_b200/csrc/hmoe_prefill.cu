// Prefill path of the MoE expert layer (hundreds to tens of thousands of rows), sm_100a: token permutation on the device
// and two grouped GEMMs on the tcgen05 tensor cores with the int4 weights converted on the way into tensor memory.
//
// Replaces, behind the same operator surface (packed int4 experts in the reference's fragment order, (sel, rw) routing, fp32
// output added into `out`):
//   * the host-side permutation of runtime/tier/tier_split.py:404-412,433-455 (stable argsort by expert id, bincount with a
//     host sync, numpy row blocks from runtime/tier/rtx_split.py:236-255 copied to the device per group) by three small
//     kernels with no host synchronisation: histogram per 1024-pick chunk, scan + balanced row-block table, stable scatter;
//   * gather_kernel / p4t_gu_kernel / p4t_gemm_kernel of runtime/tier/moe4/moe4t.cu:113-433 by the kernels below.
//
// GEMM orientation: D[channel][pick] = W[channel][k] . X[pick][k]: the weights are the M = 128 operand, converted into tensor
// memory, the picks of one row block (<= 128, one expert) the N operand in shared memory, fp32 accumulators in tensor memory. An
// item is a row block x two 128-channel tiles (gate and up, or two tiles of down) over the same inputs, so that every input tile
// feeds two MMA sequences. Per 128-column stage (one scale group):
//   warp 16    brings the packed codes and scales into shared memory by 1-D bulk copies, four stages ahead;
//   warps 0-15 in two groups that take the stages in turn: 16 bytes of codes per lane and strip -> fp16 (times the bf16 group scale)
//              -> tcgen05.st. The stored fragment order of the codes is the row / word order of the 16x256b store, so the weights never
//              pass through shared memory as fp16: at N <= 128 reading a 128-row operand from shared memory for every MMA, and writing it
//              there, would ask for more than the 128 bytes per cycle that shared memory gives;
//   warp 17    brings the stage's inputs (picks x 128 columns) as 2-D TMA boxes of 64 and 16 rows (128-byte swizzle), four stages ahead;
//   warps 18, 19  issue tcgen05.mma (M 128, N = picks rounded up to 16, K 16), one warp per accumulator, and commit the stage back;
//   warps 20-27   read the finished sums out of tensor memory (one quarter of the lanes = 32 channels each): gate_up writes
//              act = SiLU(g) * u * routing weight in fp16; down adds scale * sum into out[token] with coalesced fp32 reductions.
// What bounds it: up to about 64 picks per expert HBM (every expert's codes once), next to it the conversion (a code costs two of
// the half-rate instructions, whatever the number of picks); from there on the tensor core at the clock the power cap leaves.
// Measured, 256 experts of 6144 x 2048, us per call on new inputs: 777 rows, Zipf(1.1) 1713; 2048 rows, fp32 row scales 1758; 8192 rows, Zipf(1.1) 6178 (the
// last two at 1.45 GHz under the power cap). With fp16 weights staged through shared memory and row blocks of up to 256 picks: 2874, 2825 and
// 6971. Experts of 150 to 256 picks were converted once there and twice here, which a layer of few experts pays for (1500 rows over 64
// experts of 8192 x 1536, scale groups: 1110 there, 1165 here).
// The converting warps' issue slots are what a stage of few picks waits for (measured alone, four warps on a scheduler: 280 cycles per 16 words
// of group-scaled codes, 210 of plain ones; beside them eight MMAs of 16 picks take 1240 cycles to issue instead of 470), so all that is not
// conversion is kept short: the stage's inputs count their bytes on the barrier that the MMA warps wait for, a group steps over the other
// group's stages, and slots and parities follow from running numbers.
// Blocks are persistent (one per SM) over (row block, channel tile) items, channel tile fastest, so the blocks working at
// the same time share one input tile and one expert's weights through L2.
// Every wait is bounded (see pf_wait); tensor memory is released by the warp that allocated it on every path.
#include <cuda.h>
#include <type_traits>
#include "hmoe_common.cuh"
#include "hmoe_internal.h"
#include "hmoe_prefill_order.h"

namespace hmoe {
namespace {

// Diagnostic build (-DHMOE_PROBE_WAITS): every role adds up the cycles it spends in each of its waits (in registers, one atomic
// per thread at the end of the kernel); hmoe_probe_read() returns the sums. 32 counters per kernel: 0 / 2 first MMA warp waiting
// for a converted stage (and its inputs) / free accumulators, 10 / 4 converting warp 0 waiting for codes / for its operand slot, 9 its
// store completion + arrive, 6 input warp waiting for a slot, 7 / 8 first read-out warp waiting for a tile / reading it out, 15
// the block's lifetime. Not part of the normal build.
#ifdef HMOE_PROBE_WAITS
__device__ unsigned long long g_probe[64];
#define PROBE_T0() const long long pt0_ = clock64()
#define PROBE_ADD(i) pacc_[i] += (unsigned long long) (clock64() - pt0_)
#define PROBE_ON(c) (c)
#else
#define PROBE_T0()
#define PROBE_ADD(i)
#define PROBE_ON(c) false
#endif
constexpr int TM = 128, TN = 128, TK = 64;
constexpr int NDQ = 16;                         // converting warps; then codes, inputs, MMA, MMA, read-out
constexpr int NEPI = 8;
constexpr int PF_THREADS = (NDQ + 4 + NEPI) * 32;
constexpr int CHUNK = 1024;                     // picks per permutation block (one warp)

// ---------------------------------------------------------------------------------------------------------------------
// permutation
struct Plan
{
    int total;          // routed local picks + shared rows
    int nrb;            // row blocks
    int pad[2];
};

// per 1024-pick chunk: how many picks of each local expert
__global__ void __launch_bounds__(32) permute_hist_kernel(const int64_t* __restrict__ sel, int P, int lo, int n_local, int* __restrict__ block_hist)
{
    __shared__ int hist[256];
    const int lane = threadIdx.x, base = blockIdx.x * CHUNK;
    for (int e = lane; e < n_local; e += 32) hist[e] = 0;
    __syncwarp();
    for (int i = base + lane; i < base + CHUNK && i < P; i += 32)
    {
        const int64_t e = sel[i] - lo;
        if (e >= 0 && e < n_local) atomicAdd(&hist[(int) e], 1);
    }
    __syncwarp();
    for (int e = lane; e < n_local; e += 32) block_hist[(size_t) blockIdx.x * n_local + e] = hist[e];
}

// one block: chunk offsets per expert, expert offsets, the shared expert's segment, balanced row blocks
// (runtime/tier/rtx_split.py:236-255 with one pick group: experts without picks emit nothing, an expert's blocks get
// near-equal sizes when `balance`, {expert, first pick, picks, 0})
__global__ void __launch_bounds__(256) permute_scan_kernel(int* __restrict__ block_hist, int nblocks, int n_local, int shared_rows, int bm,
                                                          int balance, int* __restrict__ counts, int* __restrict__ offs, int* __restrict__ rbt,
                                                          Plan* __restrict__ plan)
{
    __shared__ int cnt[257], off[258], rb0[258];
    const int t = threadIdx.x;
    const int ne = n_local + (shared_rows > 0 ? 1 : 0);
    for (int e = t; e < n_local; e += blockDim.x)
    {
        int run = 0;
        for (int b = 0; b < nblocks; ++b) { const int v = block_hist[(size_t) b * n_local + e]; block_hist[(size_t) b * n_local + e] = run; run += v; }
        cnt[e] = run;
    }
    if (t == 0 && shared_rows > 0) cnt[n_local] = shared_rows;
    __syncthreads();
    if (t == 0)
    {
        int o = 0, r = 0;
        for (int e = 0; e < ne; ++e) { off[e] = o; rb0[e] = r; o += cnt[e]; r += (cnt[e] + bm - 1) / bm; }
        off[ne] = o; rb0[ne] = r;
        plan->total = o; plan->nrb = r; plan->pad[0] = plan->pad[1] = 0;
    }
    __syncthreads();
    for (int e = t; e <= ne; e += blockDim.x) { offs[e] = off[e]; if (e < ne) counts[e] = cnt[e]; }
    for (int e = t; e < ne; e += blockDim.x)
    {
        const int c = cnt[e], nb = (c + bm - 1) / bm;
        for (int k = 0; k < nb; ++k)
        {
            int rows, start;
            if (balance) { const int base = c / nb, extra = c % nb; rows = base + (k < extra ? 1 : 0); start = k * base + (k < extra ? k : extra); }
            else { rows = c - bm * k < bm ? c - bm * k : bm; start = bm * k; }
            int* r = rbt + 4 * (rb0[e] + k);
            r[0] = e; r[1] = off[e] + start; r[2] = rows; r[3] = 0;
        }
    }
}

// stable scatter: pick i goes to offs[e] + (picks of e in earlier chunks) + (picks of e earlier in this chunk)
__global__ void __launch_bounds__(32) permute_scatter_kernel(const int64_t* __restrict__ sel, const __half* __restrict__ rw, int P, int topk,
    int lo, int n_local, int shared_rows, int shared_row0, const int* __restrict__ block_hist, const int* __restrict__ offs, int nblocks,
    int* __restrict__ order, int* __restrict__ tok, int* __restrict__ eid, float* __restrict__ wt)
{
    const int lane = threadIdx.x;
    if ((int) blockIdx.x >= nblocks)
    {
        // the shared expert's rows: every row once, in order, weight 1
        const int base = ((int) blockIdx.x - nblocks) * CHUNK, o = offs[n_local];
        for (int r = base + lane; r < base + CHUNK && r < shared_rows; r += 32) { tok[o + r] = shared_row0 + r; eid[o + r] = n_local; wt[o + r] = 1.f; if (order) order[o + r] = -1; }
        return;
    }
    __shared__ int seen[256];
    for (int e = lane; e < n_local; e += 32) seen[e] = 0;
    __syncwarp();
    const int base = blockIdx.x * CHUNK;
    for (int i0 = base; i0 < base + CHUNK && i0 < P; i0 += 32)
    {
        const int i = i0 + lane;
        int e = -1;
        if (i < P) { const int64_t v = sel[i] - lo; if (v >= 0 && v < n_local) e = (int) v; }
        const unsigned same = __match_any_sync(0xffffffffu, e);
        if (e >= 0)
        {
            const int rank = __popc(same & ((1u << lane) - 1u));
            const int pos = offs[e] + block_hist[(size_t) blockIdx.x * n_local + e] + seen[e] + rank;
            if (order) order[pos] = i;
            tok[pos] = i / topk; eid[pos] = e; wt[pos] = __half2float(rw[i]);
        }
        __syncwarp();
        if (e >= 0 && (same >> lane) == 1u) seen[e] += __popc(same);      // the highest lane of each group updates the count
        __syncwarp();
    }
}

// xg[pos][H] = fp16(x[tok[pos]]), optionally after the CPU engine's int8 round trip (runtime/tier/cpuband.cpp:106-111)
__global__ void __launch_bounds__(192) gather_kernel(const void* __restrict__ x, int x_bf16, const int* __restrict__ tok, const Plan* __restrict__ plan,
                                                     int H, int act_quant, __half* __restrict__ xg)
{
    const int pos = blockIdx.x;
    if (pos >= plan->total) return;
    const int r = tok[pos];
    for (int gi = threadIdx.x; gi < H / 32; gi += blockDim.x)
    {
        float v[32];
        if (x_bf16)
        {
            const uint4* p = (const uint4*) ((const uint16_t*) x + (size_t) r * H + gi * 32);
            #pragma unroll
            for (int j = 0; j < 4; ++j)
            {
                const uint4 u = p[j]; const uint32_t w[4] = {u.x, u.y, u.z, u.w};
                #pragma unroll
                for (int k = 0; k < 4; ++k) { v[j * 8 + 2 * k] = __uint_as_float(w[k] << 16); v[j * 8 + 2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u); }
            }
        }
        else
        {
            const uint4* p = (const uint4*) ((const __half*) x + (size_t) r * H + gi * 32);
            #pragma unroll
            for (int j = 0; j < 4; ++j)
            {
                const uint4 u = p[j]; const uint32_t w[4] = {u.x, u.y, u.z, u.w};
                #pragma unroll
                for (int k = 0; k < 4; ++k) { const float2 f = __half22float2(*(const __half2*) &w[k]); v[j * 8 + 2 * k] = f.x; v[j * 8 + 2 * k + 1] = f.y; }
            }
        }
        if (act_quant)
        {
            float m = 0.f;
            #pragma unroll
            for (int k = 0; k < 32; ++k) m = fmaxf(m, fabsf(v[k]));
            const float s = m > 0.f ? __fdiv_rn(m, 127.f) : 1.f, inv = __fdiv_rn(1.f, s);
            #pragma unroll
            for (int k = 0; k < 32; ++k) v[k] = __fmul_rn((float) __float2int_rn(__fmul_rn(v[k], inv)), s);
        }
        const size_t rowlen = act_quant ? 2 * (size_t) H : (size_t) H;       // int8 mode: [hi | lo] halves, code x scale kept to ~22 bits
        // The columns are stored in the order the converted weights use (operand_pos): the thread's two 16-column steps stay in place, and inside
        // a step the pairs of columns 2q (+ 8 h) become positions 4q + 2h: four consecutive 4-byte pairs = one 16-byte store.
        #pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            uint32_t w[4], wl[4];
            #pragma unroll
            for (int i = 0; i < 4; ++i)
            {
                const int c = (q >> 1) * 16 + (i & 1) * 8 + 2 * ((q & 1) * 2 + (i >> 1));      // step q / 2, half i % 2, pair 2 (q % 2) + i / 2
                const __half2 h = __floats2half2_rn(v[c], v[c + 1]);
                w[i] = *(const uint32_t*) &h;
                const float2 f = __half22float2(h);
                const __half2 l = __floats2half2_rn(v[c] - f.x, v[c + 1] - f.y);
                wl[i] = *(const uint32_t*) &l;
            }
            *(uint4*) (xg + (size_t) pos * rowlen + gi * 32 + q * 8) = make_uint4(w[0], w[1], w[2], w[3]);
            if (act_quant) *(uint4*) (xg + (size_t) pos * rowlen + H + gi * 32 + q * 8) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// tcgen05 helpers
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// shared-memory operand descriptor: K-major tile, 128-byte swizzle, rows of 128 bytes, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr)
{
    return (uint64_t) ((addr & 0x3FFFFu) >> 4) | ((uint64_t) 1 << 16) | ((uint64_t) (1024 >> 4) << 32) | ((uint64_t) 1 << 46) | ((uint64_t) 2 << 61);
}
// A from tensor memory: 128 lanes x 8 words (16 fp16 columns) per instruction
template <bool FIRST>
__device__ __forceinline__ void mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc)
{
    if (FIRST) asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, 0, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc) : "memory");
    else asm volatile("{\n .reg .pred p;\n setp.eq.b32 p, 0, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc) : "memory");
}
__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}
// 16 lanes x 32 words (see the 64-word form below)
__device__ __forceinline__ void tmem_st_16x256_half(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                   "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
// 16 lanes x 64 words: register 4 i + {0, 1} of lane (g, q) = row g, words 8 i + 2 q, + 1; register 4 i + {2, 3} = row g + 8
__device__ __forceinline__ void tmem_st_16x256(uint32_t taddr, const uint32_t (&r)[32])
{
    asm volatile("tcgen05.st.sync.aligned.16x256b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
                 "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                   "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
                   "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
                   "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"((uint64_t) map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ void red_add_sys(float* p, float v)
{
    asm volatile("red.relaxed.sys.global.add.f32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "f"(v) : "memory");
}
__device__ __forceinline__ uint2 lds64(uint32_t addr)
{
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}

// Bounded wait of a whole warp, like mbar_wait in fewer instructions (these kernels' converting warps leave few issue slots to spare). Every lane leaves it
// with the same answer: what follows are instructions of the whole warp (tensor-memory loads and stores, votes, shuffles), which lanes that gave up
// must not miss. The first try is a short one: parked for long from the first try on, the thread wakes up later (measured: 64 to 2048 rows 3 to 7 %
// slower).
__device__ __forceinline__ bool pf_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, unsigned* status)
{
    if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
    unsigned long long t0 = 0;
    while (!__all_sync(0xffffffffu, mbar_try_hint(bar, parity, 20000u)))
    {
        const unsigned long long now = globaltimer_ns();
        const bool late = t0 != 0 && now - t0 > 1000000000ull;
        if (t0 == 0) t0 = now;
        if (late) { *abort_flag = 1; if (status) atomicOr(status, ST_WAIT_TIMEOUT); }
        if (__any_sync(0xffffffffu, late || *abort_flag)) return false;
    }
    return true;
}

struct GemmArgs
{
    int K, N;                 // reduction length and output channels of the matrix (gate_up: K = H, N = I; down: K = I, N = H)
    int grouped;              // bf16 scale per 128 columns (else fp32 per row)
    int act_quant;
    int kfold;                // 1, or 2 in the int8 mode: the inputs are [hi | lo] halves over 2 K columns, the weights are walked twice
    int nsub;                 // sub-blocks of at most TN picks per row block of the table (1; 2 for a caller's table with up to 2 TN picks)
    const int64_t* w0; const int64_t* w1;     // pointer tables of the matrix (gate, up) or (down, -)
    const int64_t* s0; const int64_t* s1;     // scale tables
    const void* sh_w0; const void* sh_w1; const void* sh_s0; const void* sh_s1;   // shared expert (expert id n_local)
    int sh_i8;                // the shared expert is in the reference's int8 format (dense GEMV fragment order, fp32 scale per row)
    int n_local;
    const Plan* plan; const int* rbt; const int* tok; const float* wt;
    __half* act;              // gate_up: output [pos][I]
    float* out;               // down: output [R][H], added into
    float* out_peer[8];       // expert parallel, combine over peer memory: row t belongs to rank t / rows_per_rank and is added
    int rows_per_rank;        //   into out_peer[rank][(t % rows_per_rank)][H] (peer pointers over NVLink); 0 = off
    unsigned* status;
};

// Column order of the GEMM operands inside every block of 64 columns. The tensor core only needs both operands to agree on
// which stored position holds which column, so the order is chosen for the weights: in the 16 columns of one MMA step a lane (g, q)
// of a converting warp holds, of rows g and g + 8, the columns 8 h + 2 q + cc (h, cc = 0..1), and the tensor-memory store puts a
// lane's two words of a row at 32-bit columns 2 q and 2 q + 1, i.e. operand positions 4 q + 2 h + cc. The gathered inputs and the
// intermediate activations are written in the same order (gather_kernel, the gate_up read-out).
__host__ __device__ __forceinline__ int operand_pos(int k) { return (k & ~15) + ((k >> 1) & 3) * 4 + ((k >> 3) & 1) * 2 + (k & 1); }

// One 16-row x 64-column strip of packed codes (one 16-byte word per lane) -> the four registers of each of its four 16-column
// steps in the order the tensor-memory store takes them (row g: two words, row g + 8: two words), times the group scale.
// Logic / shift instructions and half2 arithmetic each run at one warp instruction per two cycles and scheduler, so what counts is
// the larger of the two counts. UNSCALED: frag_from_codes (5 + 4 per word). SCALED (any scale): a multiply behind it makes that 5 + 8. FUSED:
// the two codes of the upper byte are instead brought to mantissa bits 6..9 under the exponent of 16, where one fused multiply-add does
// both steps: (16 + c) s - 24 s, exact because 24 s has at most ten significant bits (s comes from bf16) and (c - 8) s at most eleven: 6 + 6.
// It needs 31 s inside fp16's range, so a stage with a scale of 2048 or more takes SCALED.
enum Conv { UNSCALED, SCALED, FUSED };
template <Conv MODE>
__device__ __forceinline__ void convert_strip(const uint4& w, uint32_t s_lo, uint32_t s_hi, uint32_t* r)
{
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
    uint32_t o_lo = 0, o_hi = 0;
    if (MODE == FUSED) { asm("mul.f16x2 %0, %1, %2;" : "=r"(o_lo) : "r"(s_lo), "r"(0xce00ce00u)); asm("mul.f16x2 %0, %1, %2;" : "=r"(o_hi) : "r"(s_hi), "r"(0xce00ce00u)); }     // -24 s
    #pragma unroll
    for (int t = 0; t < 4; ++t)
    {
        if (MODE != FUSED)
        {
            uint32_t a[4];
            frag_from_codes(ww[t], a);
            if (MODE == SCALED)
            {
                asm("mul.f16x2 %0, %0, %1;" : "+r"(a[0]) : "r"(s_lo)); asm("mul.f16x2 %0, %0, %1;" : "+r"(a[2]) : "r"(s_lo));
                asm("mul.f16x2 %0, %0, %1;" : "+r"(a[1]) : "r"(s_hi)); asm("mul.f16x2 %0, %0, %1;" : "+r"(a[3]) : "r"(s_hi));
            }
            r[4 * t] = a[0]; r[4 * t + 1] = a[2]; r[4 * t + 2] = a[1]; r[4 * t + 3] = a[3];
        }
        else
        {
            uint32_t lo, hi, lo1, hi1;
            asm("lop3.b32 %0, %1, 0x000f000f, 0x64006400, 0xea;" : "=r"(lo) : "r"(ww[t]));           // row g, columns 2q (+ 1): 1024 + c
            asm("lop3.b32 %0, %1, 0x00f000f0, 0x64006400, 0xea;" : "=r"(hi) : "r"(ww[t]));           // row g + 8: 1024 + 16 c
            asm("lop3.b32 %0, %1, 0x03c003c0, 0x4c004c00, 0xea;" : "=r"(lo1) : "r"(ww[t] >> 2));     // row g, columns 2q + 8 (+ 1): 16 + c
            asm("lop3.b32 %0, %1, 0x03c003c0, 0x4c004c00, 0xea;" : "=r"(hi1) : "r"(ww[t] >> 6));     // row g + 8
            asm("sub.f16x2 %0, %0, %1;" : "+r"(lo) : "r"(0x64086408u));
            asm("fma.rn.f16x2 %0, %0, %1, %2;" : "+r"(hi) : "r"(0x2c002c00u), "r"(0xd480d480u));
            asm("mul.f16x2 %0, %1, %2;" : "=r"(r[4 * t]) : "r"(lo), "r"(s_lo));
            asm("mul.f16x2 %0, %1, %2;" : "=r"(r[4 * t + 2]) : "r"(hi), "r"(s_hi));
            asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r[4 * t + 1]) : "r"(lo1), "r"(s_lo), "r"(o_lo));
            asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r[4 * t + 3]) : "r"(hi1), "r"(s_hi), "r"(o_hi));
        }
    }
}
// whether one of the four bf16 scales is 2048 or more in size (0x4500): adding 0x3b00 to such a half, its sign removed, sets its top bit
__device__ __forceinline__ bool large_scale(const uint2 s) { return ((((s.x & 0x7fff7fffu) + 0x3b003b00u) | ((s.y & 0x7fff7fffu) + 0x3b003b00u)) & 0x80008000u) != 0u; }
// the same for 32 columns of the int8 format (16 bytes per lane)
__device__ __forceinline__ void convert_strip_i8(const uint4& w, uint32_t* r)
{
    dec_i8(w.x, r[0], r[2]); dec_i8(w.y, r[1], r[3]); dec_i8(w.z, r[4], r[6]); dec_i8(w.w, r[5], r[7]);
}

// bf16 pair (rows g, g + 8 of a strip) -> two fp16x2 broadcast registers
__device__ __forceinline__ void scale_pair(uint32_t bf2, uint32_t& s_lo, uint32_t& s_hi)
{
    const __half2 lo = __float2half2_rn(__uint_as_float(bf2 << 16)), hi = __float2half2_rn(__uint_as_float(bf2 & 0xffff0000u));
    s_lo = *(const uint32_t*) &lo; s_hi = *(const uint32_t*) &hi;
}

// shared memory: the packed codes (four 64-row x 128-column blocks of 4 KB and their scales) and the inputs (two 64-column tiles) of
// the stages in flight. Codes are requested NCODE stages ahead (68 KB per SM: more than the 45 KB that cover a microsecond at the
// memory's full rate; seven slots, with three for the inputs, measured no faster), inputs NB stages ahead; the converted weights never come here.
struct PfSmem
{
    static constexpr int NCODE = PF_NCODE, NB = 4;           // powers of two: a running stage number gives slot and parity
    static constexpr int CODE_SLOT = 4 * 4096 + 4 * 128;
    static constexpr int B_TILE = TN * TK * 2, B_SLOT = 2 * B_TILE;
    static constexpr int b = 0;
    static constexpr int code = NB * B_SLOT;
    static constexpr int bars = code + NCODE * CODE_SLOT;   // code_full, code_empty [NCODE], b_empty, a_full [NB], a_empty, done, acc_free [2], i8_done
    static constexpr int misc = bars + (2 * NCODE + 2 * NB + 7) * 8 + 8;
    static constexpr int total = misc + 32 + 1024;          // + slack to align the base to 1024
};
// tensor memory: columns 0..255 accumulators (two slots of 128: a block of up to 64 picks takes one slot for its two accumulators, a larger
// one both), columns 256..511 two stages of converted weights (two matrices x 128 columns of fp16 = 64 words each)
constexpr int TMEM_COLS = 512, TMEM_A = 256;

// The accumulator slots of a block's successive tiles; every role steps through the same sequence.
struct AccSeq
{
    uint32_t small = 0, u0 = 0, u1 = 0, d0 = 0, d1 = 0;      // next slot of a small tile; tiles so far that took slot 0 / 1, that completed on slot 0 / 1
    uint32_t mask, slot, up;                 // this tile: slots taken (bits), first slot, column distance of the second accumulator
    uint32_t need0, need1, done_par;         // earlier uses of each slot; parity of the tile's completion barrier
    __device__ __forceinline__ void next(int n)
    {
        const bool big = n > 64;
        slot = big ? 0u : small; mask = big ? 3u : 1u << small; up = big ? 128u : 64u;
        if (!big) small ^= 1u;
        need0 = u0; need1 = u1;
        u0 += mask & 1u; u1 += mask >> 1;
        done_par = (slot ? d1 : d0) & 1u;
        d0 += slot ^ 1u; d1 += slot;
    }
};

// One item: a sub-block of a row block's picks (<= TN, one expert) x one 128-channel tile of gate and of up, or two 128-channel tiles of down.
struct ItemPos { int e, pos0, n, ct, nmat; };
template <bool DOWN>
__device__ __forceinline__ ItemPos item_pos(const GemmArgs& a, int item, int nct)
{
    ItemPos it;
    const int rs = item / nct;
    it.ct = item - rs * nct;
    const int rb = a.nsub == 1 ? rs : rs / a.nsub, sub = a.nsub == 1 ? 0 : rs - rb * a.nsub;
    const int* r = a.rbt + 4 * (size_t) rb;                 // word by word: a caller's table (hmoe_prefill_sorted) need not start on 16 bytes
    it.e = __ldg(r); it.pos0 = __ldg(r + 1) + sub * TN; it.n = min(__ldg(r + 2) - sub * TN, TN);
    it.nmat = DOWN ? (2 * it.ct + 1 < a.N / TM ? 2 : 1) : 2;
    return it;
}

// DOWN = false: gate and up over one input tile, SiLU read-out. DOWN = true: two channel tiles of down, scatter-add read-out.
template <bool DOWN>
__global__ void __launch_bounds__(PF_THREADS, 1) prefill_gemm_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap tmap16, const __grid_constant__ GemmArgs a)
{
    using L = PfSmem;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t sbase = (raw + 1023u) & ~1023u;
    unsigned char* smem = smem_raw + (sbase - raw);
    const uint32_t code_full = sbase + L::bars, code_empty = code_full + L::NCODE * 8, b_empty = code_empty + L::NCODE * 8, a_full = b_empty + L::NB * 8,
                   a_empty = a_full + L::NB * 8, done = a_empty + 16, acc_free = done + 16, i8_done = acc_free + 16;
    uint32_t* tmem_slot = (uint32_t*) (smem + L::misc);
    volatile int* abort_flag = (volatile int*) (smem + L::misc + 8);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0)
    {
        for (int i = 0; i < L::NCODE; ++i) { mbar_init(code_full + i * 8, 1); mbar_init(code_empty + i * 8, NDQ / 2); }
        for (int i = 0; i < L::NB; ++i) { mbar_init(a_full + i * 8, NDQ / 2 + 1); mbar_init(b_empty + i * 8, 2); }       // the converting warps and the inputs
        for (int i = 0; i < 2; ++i) { mbar_init(a_empty + i * 8, 2); mbar_init(done + i * 8, 2); mbar_init(acc_free + i * 8, NEPI); }
        mbar_init(i8_done, NDQ);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == NDQ + 2)
    {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    const int KS = a.K / 128, KST = KS * a.kfold;                    // 128-column stages of the weights / of a tile
    const int NCT = DOWN ? (a.N / TM + 1) / 2 : a.N / TM;
#ifdef HMOE_PROBE_WAITS
    unsigned long long pacc_[16] = {};
#endif
    PROBE_T0();
    const int nitems = a.plan->nrb * a.nsub * NCT;

    if (warp < NDQ)
    {
        // ---- convert: two groups of eight warps take the stages in turn, so that one group's waits (for codes, for its operand slot, for its
        // stores) lie under the other's arithmetic. Warp w of a group takes, of matrix w / 4, the 32 rows of tensor-memory lane
        // quarter w % 4 (a warp can only reach the quarter that matches its number) as two 16-row strips. In down's last item of an
        // odd number of channel tiles the second tile's warps convert whatever the slot holds; nothing reads it.
        const int g = lane >> 2, quarter = warp & 3, mat = (warp >> 2) & 1;
        const uint32_t group = warp >> 3;
        const uint32_t code0 = sbase + L::code + (mat * 2 + (quarter >> 1)) * 4096 + (quarter & 1) * 1024 + lane * 16;
        const uint32_t sc0 = sbase + L::code + 4 * 4096 + (mat * 2 + (quarter >> 1)) * 128 + (g * 8 + (quarter & 1) * 4) * 2;
        const uint32_t ta = tmem + TMEM_A + group * 128 + mat * 64 + ((uint32_t) (quarter * 32) << 16);      // the group's operand slot
        uint32_t t0 = 0, c0 = 0;                                               // stages and code slots before this item
        CodeOrder order;
        for (int item = blockIdx.x; item < nitems; item += gridDim.x)
        {
            const ItemPos it = item_pos<DOWN>(a, item, NCT);
            if (it.n <= 0) continue;
            if (__any_sync(0xffffffffu, *abort_flag)) break;
            const bool i8 = a.sh_i8 && it.e >= a.n_local;
            auto code_wait = [&](uint32_t c) -> bool { PROBE_T0(); const bool w_ = pf_wait(code_full + (c % L::NCODE) * 8, (c / L::NCODE) & 1, abort_flag, a.status); if (PROBE_ON(threadIdx.x == 0)) PROBE_ADD(10); return w_; };
            auto code_release = [&](uint32_t c) {
                __syncwarp();
                mbar_arrive_if(code_empty + (c % L::NCODE) * 8, lane == 0);
            };
            auto slot_wait = [&](uint32_t t) -> bool {
                PROBE_T0(); const bool w_ = pf_wait(a_empty + group * 8, ((t >> 1) & 1) ^ 1, abort_flag, a.status); if (PROBE_ON(threadIdx.x == 0)) PROBE_ADD(4);
                tc_fence_after();
                return w_;
            };
            // both strips are stored: hand the slot to the MMA warps
            auto put = [&](uint32_t t) {
                PROBE_T0();
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                mbar_arrive_if(a_full + (t % L::NB) * 8, lane == 0);
                if (PROBE_ON(threadIdx.x == 0)) PROBE_ADD(9);
            };
            auto run = [&](auto grouped_tag) -> bool {
                constexpr bool GROUPED = decltype(grouped_tag)::value;
                #pragma unroll 1
                for (uint32_t j = (t0 ^ group) & 1; j < (uint32_t) KST; j += 2)
                {
                    const uint32_t t = t0 + j, c = c0 + j;
                    if (!code_wait(c)) return false;
                    const uint32_t at = code0 + (c % L::NCODE) * L::CODE_SLOT;
                    uint2 sp = make_uint2(0, 0);
                    if (GROUPED) sp = lds64(sc0 + (c % L::NCODE) * L::CODE_SLOT);
                    auto strips = [&](auto mode_tag) -> bool {
                        constexpr Conv MODE = decltype(mode_tag)::value;
                        uint32_t r[32], s_lo = 0, s_hi = 0;
                        uint4 wa = lds128(at), wb = lds128(at + 2048);
                        if (GROUPED) scale_pair(sp.x, s_lo, s_hi);
                        convert_strip<MODE>(wa, s_lo, s_hi, r);
                        convert_strip<MODE>(wb, s_lo, s_hi, r + 16);
                        wa = lds128(at + 512); wb = lds128(at + 2048 + 512);
                        if (!slot_wait(t)) return false;
                        tmem_st_16x256(ta, r);
                        if (GROUPED) scale_pair(sp.y, s_lo, s_hi);
                        convert_strip<MODE>(wa, s_lo, s_hi, r);
                        convert_strip<MODE>(wb, s_lo, s_hi, r + 16);
                        code_release(c);
                        tmem_st_16x256(ta + (16u << 16), r);
                        return true;
                    };
                    bool ok;
                    if (!GROUPED) ok = strips(std::integral_constant<Conv, UNSCALED>());
                    else if (__any_sync(0xffffffffu, large_scale(sp))) ok = strips(std::integral_constant<Conv, SCALED>());
                    else ok = strips(std::integral_constant<Conv, FUSED>());
                    if (!ok) return false;
                    put(t);
                }
                return true;
            };
            // The shared expert in the reference's int8 format (runtime/tier/tier_split.py:495-514): 2 KB units of 64 rows x 32
            // columns, so a code slot holds 64 columns and a stage takes two. Its fp32 row scales are applied by the read-out.
            auto run_i8 = [&]() -> bool {
                #pragma unroll 1
                for (uint32_t j = (t0 ^ group) & 1; j < (uint32_t) KST; j += 2)
                {
                    const uint32_t t = t0 + j;
                    if (!slot_wait(t)) return false;
                    #pragma unroll 1
                    for (uint32_t h = 0; h < 2; ++h)
                    {
                        const uint32_t c = c0 + 2 * j + h;
                        if (!code_wait(c)) return false;
                        const uint32_t at = code0 + (c % L::NCODE) * L::CODE_SLOT;
                        uint32_t r[16];
                        convert_strip_i8(lds128(at), r);
                        convert_strip_i8(lds128(at + 2048), r + 8);
                        tmem_st_16x256_half(ta + h * 32, r);
                        convert_strip_i8(lds128(at + 512), r);
                        convert_strip_i8(lds128(at + 2048 + 512), r + 8);
                        tmem_st_16x256_half(ta + h * 32 + (16u << 16), r);
                        code_release(c);
                    }
                    put(t);
                }
                return true;
            };
            if (order.wait_first(i8))
            {
                __syncwarp();
                mbar_arrive_if(i8_done, lane == 0);
                if (!pf_wait(i8_done, (order.crossings - 1) & 1, abort_flag, a.status)) break;
            }
            if (!(i8 ? run_i8() : a.grouped ? run(std::true_type()) : run(std::false_type()))) break;
            t0 += KST; c0 += i8 ? 2 * KST : KST;
        }
    }
    else if (warp == NDQ)
    {
        // ---- codes: per stage (int8: half stage) one bulk copy of 4 KB per matrix and 64-row group, lanes 0..3, and its 128 bytes of scales, lanes 4..7
        uint32_t c = 0;
        bool ok = true;
        const int blk = lane & 3, mat = blk >> 1, unit = blk & 1;
        for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x)
        {
            const ItemPos it = item_pos<DOWN>(a, item, NCT);
            if (it.n <= 0) continue;
            const bool sh = it.e >= a.n_local, i8 = a.sh_i8 && sh, scaled = a.grouped && !i8;
            const bool second = !DOWN && mat;
            const char* wp = (const char*) (sh ? (second ? a.sh_w1 : a.sh_w0) : (const void*) (second ? a.w1 : a.w0)[it.e]);
            const char* sp = (const char*) (sh ? (second ? a.sh_s1 : a.sh_s0) : (const void*) (second ? a.s1 : a.s0)[it.e]);
            const int gr = DOWN ? (2 * it.ct + mat) * 2 + unit : 2 * it.ct + unit;          // 64-row group
            const char* src = lane < 4 ? wp + (size_t) gr * (a.K / 64) * (i8 ? 4096 : 2048) : sp + (size_t) gr * KS * 128;
            const bool on = mat < it.nmat && (lane < 4 || (lane < 8 && scaled));
            const uint32_t bytes = lane < 4 ? 4096 : 128, dst0 = sbase + L::code + (lane < 4 ? blk * 4096 : 4 * 4096 + blk * 128);
            const uint32_t total = (uint32_t) it.nmat * 2 * (4096 + (scaled ? 128 : 0));
            const int steps = i8 ? 2 * KS : KS;                      // copies of one pass over the weights
            for (int f = 0; f < a.kfold && ok; ++f)
                for (int j = 0; j < steps; ++j)
                {
                    const uint32_t s = c % L::NCODE;
                    if (!pf_wait(code_empty + s * 8, ((c / L::NCODE) & 1) ^ 1, abort_flag, a.status)) { ok = false; break; }
                    if (lane == 0) mbar_expect_tx(code_full + s * 8, total);
                    __syncwarp();
                    if (on) bulk_g2s(dst0 + s * L::CODE_SLOT, src + (size_t) j * bytes, bytes, code_full + s * 8);
                    ++c;
                }
        }
    }
    else if (warp == NDQ + 1)
    {
        // ---- inputs: the picks' 128 columns of a stage as two tiles of 64 columns, in boxes of 64 rows and, for the last rows, of 16, so that a
        // block with few picks brings in little more than the rows the MMAs read (n rounded up to 16)
        uint32_t t = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x)
        {
            const ItemPos it = item_pos<DOWN>(a, item, NCT);
            if (it.n <= 0) continue;
            const int n16 = (it.n + 15) & ~15, nbig = n16 >> 6, nbox = nbig + ((n16 & 63) >> 4);
            const int tile = lane / nbox, box = lane - tile * nbox, row = box < nbig ? box * 64 : nbig * 64 + (box - nbig) * 16;
            const bool on = lane < 2 * nbox;
            for (int j = 0; j < KST; ++j)
            {
                const uint32_t s = t % L::NB;
                { PROBE_T0(); const bool w_ = pf_wait(b_empty + s * 8, ((t / L::NB) & 1) ^ 1, abort_flag, a.status); if (PROBE_ON(lane == 0)) PROBE_ADD(6); if (!w_) { ok = false; break; } }
                if (lane == 0) mbar_expect_tx(a_full + s * 8, (uint32_t) n16 * (2 * TK * 2));
                __syncwarp();
                if (on) tma_load_2d(sbase + L::b + s * L::B_SLOT + tile * L::B_TILE + row * (TK * 2), box < nbig ? &tmap : &tmap16, j * 128 + tile * 64, it.pos0 + row, a_full + s * 8);
                ++t;
            }
        }
    }
    else if (warp < NDQ + 4)
    {
        // ---- MMA: one warp per accumulator (gate / up, or the two channel tiles); the whole warp steps through the stages, one elected lane
        // issues. Between two stages' MMAs lie a few hundred cycles of waiting, fencing and committing while the converting warps take most of
        // the issue slots (measured with one warp for both accumulators: 450 cycles per stage against 16 x 17 for the MMAs of a block of
        // few picks); with two warps one's stage is under way meanwhile. All 512 columns are allocated, so the allocation starts at
        // column 0 (checked here): the addresses of the operands are plain arithmetic on loop counters.
        const uint32_t acc = warp - (NDQ + 2);
        uint32_t t = 0;
        const uint64_t bdesc0 = smem_desc_sw128(sbase + L::b);
        AccSeq seq;
        bool ok = tmem == 0u;
        if (!ok && lane == 0) { *abort_flag = 1; atomicOr(a.status, ST_WAIT_TIMEOUT); }
        for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x)
        {
            const ItemPos it = item_pos<DOWN>(a, item, NCT);
            if (it.n <= 0) continue;
            const uint32_t n16 = (uint32_t) ((it.n + 15) & ~15);
            const uint32_t idesc = (1u << 4) | ((n16 >> 3) << 17) | ((uint32_t) (TM >> 4) << 24);
            seq.next(it.n);
            // the accumulators are free once the tiles that used their slots last have been read out
            PROBE_T0();
            if ((seq.mask & 1) && seq.need0 && !pf_wait(acc_free, (seq.need0 - 1) & 1, abort_flag, a.status)) ok = false;
            if ((seq.mask & 2) && seq.need1 && !pf_wait(acc_free + 8, (seq.need1 - 1) & 1, abort_flag, a.status)) ok = false;
            if (PROBE_ON(acc == 0)) PROBE_ADD(2);
            if (!ok) break;
            tc_fence_after();
            const uint32_t d = seq.slot * 128 + acc * seq.up;
            const bool live = !DOWN || (int) acc < it.nmat;
            for (int j = 0; j < KST; ++j, ++t)
            {
                const uint32_t sb = t % L::NB, sa = t & 1;
                bool w;
                { PROBE_T0(); w = pf_wait(a_full + sb * 8, (t / L::NB) & 1, abort_flag, a.status); if (PROBE_ON(acc == 0)) PROBE_ADD(0); }
                if (!w) { ok = false; break; }
                tc_fence_after();
                const uint32_t at = TMEM_A + sa * 128 + acc * 64;
                const uint64_t bd = bdesc0 + sb * (L::B_SLOT >> 4);
                if (elect_one())
                {
                    if (live)
                    {
                        if (j == 0) mma_f16_ts<true>(d, at, bd, idesc); else mma_f16_ts<false>(d, at, bd, idesc);
                        #pragma unroll
                        for (int k = 1; k < 8; ++k) mma_f16_ts<false>(d, at + k * 8, bd + (k >> 2) * (L::B_TILE >> 4) + (k & 3) * 2, idesc);
                    }
                    tc_commit(a_empty + sa * 8);
                    tc_commit(b_empty + sb * 8);
                    if (j + 1 == KST) tc_commit(done + seq.slot * 8);
                }
                __syncwarp();
            }
        }
    }
    else
    {
        // ---- read-out: warp i reads the tensor-memory lanes of quarter i % 4, i.e. 32 output channels per accumulator. gate_up: SiLU(gate)
        // * up * routing weight -> fp16 activations, the two warps of a quarter take half of the picks each; down: out[token] += scale *
        // sum, one fp32 reduction per element (32 lanes = 32 consecutive channels = 128 contiguous bytes), one of the two channel
        // tiles per warp. These warps do nothing else, so the read-out of a tile overlaps the conversion (and for blocks of up to 64 picks,
        // which leave the other accumulator slot free, the MMAs) of the next one.
        const int lq = warp & 3, half = (warp - (NDQ + 4)) >> 2;
        AccSeq seq;
        bool ok = true;
        for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x)
        {
            const ItemPos it = item_pos<DOWN>(a, item, NCT);
            if (it.n <= 0) continue;
            if (__any_sync(0xffffffffu, *abort_flag)) break;
            const int e = it.e, pos0 = it.pos0, n = it.n, n16 = (n + 15) & ~15;
            seq.next(n);
            const bool live = !DOWN || half < it.nmat;
            const int ch = (DOWN ? 2 * it.ct + (live ? half : 0) : it.ct) * TM + lq * 32 + lane;
            const uint32_t tacc = tmem + seq.slot * 128 + ((uint32_t) (lq * 32) << 16);
            // Everything the read-out needs besides the sums is fetched BEFORE the wait for the tile's last MMA, so that no global
            // load stands between that MMA and the release of the accumulators: the row scales, and in gate_up the
            // routing weights of the warp's columns (lane l holds picks cbeg + 32 i + l).
            float sc0 = 1.f, sc1 = 1.f;
            if (!a.grouped || (a.sh_i8 && e >= a.n_local))      // one fp32 scale per output row: applied here, not in the operand
            {
                const void* s0p = e < a.n_local ? (const void*) a.s0[e] : a.sh_s0;
                sc0 = __ldg((const float*) s0p + ch);
                if (!DOWN) { const void* s1p = e < a.n_local ? (const void*) a.s1[e] : a.sh_s1; sc1 = __ldg((const float*) s1p + ch); }
            }
            if constexpr (!DOWN)
            {
                const int csplit = ((n16 + 31) >> 5) << 4;          // the quarter's two warps take columns [0, csplit) and [csplit, n16)
                const int cbeg = half ? csplit : 0, cend = half ? n16 : csplit;
                float wv[2] = {0.f, 0.f};
                #pragma unroll
                for (int i = 0; i < 2; ++i) { const int pj = cbeg + 32 * i + lane; if (pj < n) wv[i] = __ldg(a.wt + pos0 + pj); }
                { PROBE_T0(); const bool w_ = pf_wait(done + seq.slot * 8, seq.done_par, abort_flag, a.status); if (PROBE_ON(threadIdx.x == (NDQ + 4) * 32)) PROBE_ADD(7); if (!w_) break; }
                PROBE_T0();
                tc_fence_after();
                const int chp = (ch & ~63) + operand_pos(ch & 63);       // where the down GEMM expects this channel of the activations
                // Eight columns at a time. The loops carry no branch per column: a conditional region per column costs
                // convergence-barrier instructions that run one after the other (measured: ~70 cycles per column); the arithmetic runs
                // for the padding columns too and only the store is predicated; the int8 mode is a compile-time variant of the whole loop.
                auto read_out = [&](auto aq_tag) {
                    constexpr bool AQ = decltype(aq_tag)::value;
                    uint32_t g0[8], u0[8];
                    for (int c0 = cbeg; c0 < cend; c0 += 8)
                    {
                        tmem_ld8(tacc + c0, g0); tmem_ld8(tacc + seq.up + c0, u0);
                        tmem_ld_wait();
                        const int rel = c0 - cbeg;
                        const float wsel = rel < 32 ? wv[0] : wv[1];
                        float ws[8];
                        #pragma unroll
                        for (int j = 0; j < 8; ++j) ws[j] = __shfl_sync(0xffffffffu, wsel, (rel & 31) + j);
                        #pragma unroll
                        for (int j = 0; j < 8; ++j)
                        {
                            const int p = c0 + j;
                            const float w = ws[j];
                            const float gg = __uint_as_float(g0[j]) * sc0, uu = __uint_as_float(u0[j]) * sc1;
                            if (AQ)
                            {
                                float v = gg / (1.f + expf(-gg)) * uu * w;
                                // second int8 round trip of the CPU engine: 32 consecutive channels = this warp
                                float m = fabsf(v);
                                #pragma unroll
                                for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                                const float sq8 = m > 0.f ? __fdiv_rn(m, 127.f) : 1.f;
                                v = __fmul_rn((float) __float2int_rn(__fmul_rn(v, __fdiv_rn(1.f, sq8))), sq8);
                                // code x scale does not fit fp16: keep it as hi + lo halves, the down GEMM walks both
                                const __half hi = __float2half_rn(v), lo = __float2half_rn(v - __half2float(hi));
                                __half* dst = a.act + (size_t) (pos0 + p) * (2 * a.N) + chp;
                                if (p < n) { dst[0] = hi; dst[a.N] = lo; }
                            }
                            else
                            {
                                // fp16 result: the fast exponential and division are far inside its rounding (the reference's
                                // kernels make the same choice, runtime/tier/moe4/moe4t.cu:404-425 built with fast-math)
                                const __half v = __float2half_rn(__fdividef(gg, 1.f + __expf(-gg)) * uu * w);
                                if (p < n) a.act[(size_t) (pos0 + p) * a.N + chp] = v;
                            }
                        }
                    }
                };
                if (a.act_quant) read_out(std::true_type()); else read_out(std::false_type());
                if (PROBE_ON(threadIdx.x == (NDQ + 4) * 32)) PROBE_ADD(8);
            }
            else
            {
                // lane l holds the tokens of picks l, l + 32, ... (of the last pick beyond them); fetched before the wait, and sixteen columns per
                // step instead of eight with a load in each: 10 % of this kernel's time at 8192 rows, whose blocks of more than 64 picks keep the
                // MMAs waiting for the read-out
                int tok[TN / 32];
                #pragma unroll
                for (int i = 0; i < TN / 32; ++i) tok[i] = __ldg(a.tok + pos0 + min(32 * i + lane, n - 1));
                { PROBE_T0(); const bool w_ = pf_wait(done + seq.slot * 8, seq.done_par, abort_flag, a.status); if (PROBE_ON(threadIdx.x == (NDQ + 4) * 32)) PROBE_ADD(7); if (!w_) break; }
                PROBE_T0();
                tc_fence_after();
                // Sixteen columns at a time; no branch per column here either: the padding columns add 0 to the row of the block's last pick.
                const uint32_t td = tacc + half * seq.up;
                auto read_out = [&](auto peer_tag) {
                    constexpr bool PEER = decltype(peer_tag)::value;
                    #pragma unroll
                    for (int i = 0; i < TN / 32; ++i)
                    {
                        #pragma unroll 1
                        for (int c0 = 32 * i; c0 < min(n16, 32 * i + 32); c0 += 16)
                        {
                            uint32_t r[16];
                            tmem_ld16(td + c0, r);
                            tmem_ld_wait();
                            auto add = [&](int j, float v) {
                                const int tk = __shfl_sync(0xffffffffu, tok[i], (c0 & 16) + j);
                                if (PEER)
                                {
                                    // the row's owner may be another GPU, and up to eight GPUs add into the same addresses: the
                                    // reduction has to be atomic at system scope (a gpu-scope one is only atomic among this GPU's threads)
                                    const int pr = tk / a.rows_per_rank;
                                    red_add_sys(a.out_peer[pr] + (size_t) (tk - pr * a.rows_per_rank) * a.N + ch, v);
                                }
                                else atomicAdd(a.out + (size_t) tk * a.N + ch, v);
                            };
                            if (c0 + 16 <= n)
                            {
                                #pragma unroll
                                for (int j = 0; j < 16; ++j) add(j, __uint_as_float(r[j]) * sc0);
                            }
                            else
                            {
                                #pragma unroll
                                for (int j = 0; j < 16; ++j) add(j, c0 + j < n ? __uint_as_float(r[j]) * sc0 : 0.f);
                            }
                        }
                    }
                };
                if (live) { if (a.rows_per_rank) read_out(std::true_type()); else read_out(std::false_type()); }
                if (PROBE_ON(threadIdx.x == (NDQ + 4) * 32)) PROBE_ADD(8);
            }
            tc_fence_before();
            __syncwarp();
            #pragma unroll
            for (int i = 0; i < 2; ++i) mbar_arrive_if(acc_free + i * 8, lane == 0 && (seq.mask >> i & 1));
        }
    }
#ifdef HMOE_PROBE_WAITS
    if (threadIdx.x == 0) PROBE_ADD(15);
    #pragma unroll
    for (int i = 0; i < 16; ++i) if (pacc_[i] && !(warp >= NDQ + 2 && warp < NDQ + 4 && lane)) atomicAdd(&g_probe[(DOWN ? 0 : 1) * 32 + i], pacc_[i]);
#endif
    tc_fence_before();
    __syncthreads();
    abort_drain(abort_flag);
    __syncthreads();
    if (warp == NDQ + 2)
    {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

typedef CUresult (*encode_fn_t)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

encode_fn_t encode_fn()
{
    static encode_fn_t f = nullptr;
    if (!f)
    {
        void* p = nullptr; cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess) f = (encode_fn_t) p;
    }
    return f;
}

// row-major fp16 [rows][K] in boxes of 64 columns x `box_rows` rows, 128-byte swizzle
bool make_map(CUtensorMap* m, const void* ptr, int K, size_t rows, int box_rows)
{
    encode_fn_t f = encode_fn();
    if (!f) return false;
    cuuint64_t dims[2] = {(cuuint64_t) K, (cuuint64_t) rows};
    cuuint64_t strides[1] = {(cuuint64_t) K * 2};
    cuuint32_t box[2] = {TK, (cuuint32_t) box_rows}, es[2] = {1, 1};
    return f(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*) ptr, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

size_t up256(size_t b) { return (b + 255) / 256 * 256; }

// the kernels' dynamic shared memory exceeds the default limit: raise it once per device
void set_gemm_attributes()
{
    static DeviceOnce once;
    if (!once.first()) return;
    cudaFuncSetAttribute(prefill_gemm_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, PfSmem::total);
    cudaFuncSetAttribute(prefill_gemm_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, PfSmem::total);
}

struct WsLayout
{
    size_t status, plan, counts, offs, hist, order, tok, eid, wt, rbt, xg, act, total;
    int nblocks, rows_cap, maxrb;
};

WsLayout ws_layout(int R, int topk, int n_local, int H, int I, int bm, int kfold = 1)
{
    WsLayout w;
    const size_t P = (size_t) R * topk;
    w.nblocks = (int) ((P + CHUNK - 1) / CHUNK);
    w.rows_cap = (int) (P + R);
    w.maxrb = (int) ((P + R) / bm + n_local + 2);
    size_t o = 0;
    w.status = o; o += 256;
    w.plan = o; o += 256;
    w.counts = o; o += up256((size_t) (n_local + 2) * 4);
    w.offs = o; o += up256((size_t) (n_local + 3) * 4);
    w.hist = o; o += up256((size_t) w.nblocks * (n_local > 0 ? n_local : 1) * 4);
    w.order = o; o += up256((size_t) w.rows_cap * 4);
    w.tok = o; o += up256((size_t) w.rows_cap * 4);
    w.eid = o; o += up256((size_t) w.rows_cap * 4);
    w.wt = o; o += up256((size_t) w.rows_cap * 4);
    w.rbt = o; o += up256((size_t) w.maxrb * 16);
    w.xg = o; o += up256((size_t) w.rows_cap * H * 2 * kfold);
    w.act = o; o += up256((size_t) w.rows_cap * I * 2 * kfold);
    w.total = o;
    return w;
}

int run_permute(const int64_t* sel, const void* rw, int R, int topk, int lo, int n_local, int shared_rows, int shared_row0, int bm, int balance,
                int* counts, int* offs, int* hist, int nblocks, int* order, int* tok, int* eid, float* wt, int* rbt, Plan* plan, cudaStream_t st)
{
    const int P = R * topk;
    permute_hist_kernel<<<nblocks, 32, 0, st>>>(sel, P, lo, n_local, hist);
    permute_scan_kernel<<<1, 256, 0, st>>>(hist, nblocks, n_local, shared_rows, bm, balance, counts, offs, rbt, plan);
    const int sb = shared_rows > 0 ? (shared_rows + CHUNK - 1) / CHUNK : 0;
    permute_scatter_kernel<<<nblocks + sb, 32, 0, st>>>(sel, (const __half*) rw, P, topk, lo, n_local, shared_rows, shared_row0, hist, offs, nblocks, order, tok, eid, wt);
    count_launches(3);
    return cudaGetLastError() == cudaSuccess ? HMOE_OK : fail(HMOE_E_CUDA, "hmoe_permute: launch failed");
}

}  // namespace

size_t prefill_ws_bytes(int R, int topk, int n_local, int H, int I, int act_quant) { return ws_layout(R, topk, n_local, H, I, TN, act_quant ? 2 : 1).total; }

namespace {
__global__ void set_plan_kernel(Plan* plan, int total, int nrb) { plan->total = total; plan->nrb = nrb; plan->pad[0] = plan->pad[1] = 0; }
}

// The reference's calling convention (moe4t.forward, runtime/tier/moe4/moe4t.cu:498-524): the caller has already sorted the
// picks by expert (tok, wt in that order) and built the row-block table; npos picks, nrb row blocks of <= 256 picks.
size_t prefill_sorted_ws_bytes(int npos, int H, int I, int act_quant)
{
    const int f = act_quant ? 2 : 1;
    return 512 + up256((size_t) npos * H * 2 * f) + up256((size_t) npos * I * 2 * f);
}

int prefill_sorted_launch(const hmoe_layer* L, const void* x, int x_dtype, const int32_t* tok, const float* wt, const int32_t* rbt, int nrb,
                          int npos, int n_local, int act_quant, float* out, void* ws, size_t ws_bytes, cudaStream_t st)
{
    const int H = L->H, I = L->I;
    if (npos < 0 || nrb < 0) return fail(HMOE_E_ARG, "hmoe_prefill_sorted: sizes");
    if (npos == 0 || nrb == 0) return HMOE_OK;
    if (H % 128 || I % 128 || H < 128 || I < 128) return fail(HMOE_E_ARG, "hmoe_prefill_sorted: H and I must be multiples of 128");
    if (!(L->group == 0 && L->scale_dtype == HMOE_F32) && !(L->group == 128 && L->scale_dtype == HMOE_BF16))
        return fail(HMOE_E_ARG, "hmoe_prefill_sorted: scales must be fp32 per row (group 0) or bf16 per 128 columns");
    if (x_dtype != HMOE_F16 && x_dtype != HMOE_BF16) return fail(HMOE_E_ARG, "hmoe_prefill_sorted: x must be fp16 or bf16");
    if (!x || !tok || !wt || !rbt || !out || !ws) return fail(HMOE_E_ARG, "hmoe_prefill_sorted: null pointer");
    const int kf = act_quant ? 2 : 1;
    if (ws_bytes < prefill_sorted_ws_bytes(npos, H, I, act_quant)) return fail(HMOE_E_WS, "hmoe_prefill_sorted: workspace too small");
    const int sms = device_sms();
    if (sms <= 0) return fail(HMOE_E_CUDA, "hmoe_prefill_sorted: no current CUDA device");
    set_gemm_attributes();
    char* b = (char*) ws;
    unsigned* status = (unsigned*) b;
    Plan* plan = (Plan*) (b + 256);
    __half* xg = (__half*) (b + 512);
    __half* act = (__half*) (b + 512 + up256((size_t) npos * H * 2 * kf));
    set_plan_kernel<<<1, 1, 0, st>>>(plan, npos, nrb);
    gather_kernel<<<npos, 192, 0, st>>>(x, x_dtype == HMOE_BF16, tok, plan, H, act_quant, xg);
    CUtensorMap mx, ma, mx16, ma16;
    if (!make_map(&mx, xg, H * kf, (size_t) npos, 64) || !make_map(&ma, act, I * kf, (size_t) npos, 64) || !make_map(&mx16, xg, H * kf, (size_t) npos, 16) ||
        !make_map(&ma16, act, I * kf, (size_t) npos, 16)) return fail(HMOE_E_CUDA, "hmoe_prefill_sorted: cuTensorMapEncodeTiled failed");
    GemmArgs g;
    g.grouped = L->group != 0; g.act_quant = act_quant; g.n_local = n_local; g.kfold = kf; g.nsub = 2;                // the caller's row blocks hold up to 256 picks
    g.sh_i8 = L->shared_format == 1 && L->sh_gate_w != nullptr;
    g.plan = plan; g.rbt = rbt; g.tok = tok; g.wt = wt; g.act = act; g.out = out; g.status = status;
    g.rows_per_rank = 0;
    for (int p = 0; p < 8; ++p) g.out_peer[p] = nullptr;
    g.K = H; g.N = I; g.w0 = L->gate_w; g.w1 = L->up_w; g.s0 = L->gate_s; g.s1 = L->up_s;
    g.sh_w0 = L->sh_gate_w; g.sh_w1 = L->sh_up_w; g.sh_s0 = L->sh_gate_s; g.sh_s1 = L->sh_up_s;
    prefill_gemm_kernel<false><<<sms, PF_THREADS, PfSmem::total, st>>>(mx, mx16, g);
    g.K = I; g.N = H; g.w0 = L->down_w; g.w1 = nullptr; g.s0 = L->down_s; g.s1 = nullptr;
    g.sh_w0 = L->sh_down_w; g.sh_w1 = nullptr; g.sh_s0 = L->sh_down_s; g.sh_s1 = nullptr;
    prefill_gemm_kernel<true><<<sms, PF_THREADS, PfSmem::total, st>>>(ma, ma16, g);
    count_launches(4);
    const cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? HMOE_OK : fail(HMOE_E_CUDA, cudaGetErrorString(err));
}

int permute_launch(const int64_t* sel, const void* rw, int R, int topk, int lo, int n_local, int shared_rows, int bm, int balance,
                   int32_t* order, int32_t* tok, int32_t* eid, float* wt, int32_t* counts, int32_t* rbt, int32_t* plan2, void* ws, size_t ws_bytes,
                   cudaStream_t st)
{
    if (R < 1 || topk < 1 || n_local < 1 || n_local > 256 || bm < 1) return fail(HMOE_E_ARG, "hmoe_permute: needs R >= 1, 1 <= n_local <= 256, bm >= 1");
    if (!sel || !rw || !tok || !eid || !wt || !counts || !rbt || !plan2 || !ws) return fail(HMOE_E_ARG, "hmoe_permute: null pointer");
    const size_t P = (size_t) R * topk;
    const int nblocks = (int) ((P + CHUNK - 1) / CHUNK);
    const size_t need = up256((size_t) nblocks * n_local * 4) + up256((size_t) (n_local + 3) * 4);
    if (ws_bytes < need) return fail(HMOE_E_WS, "hmoe_permute: workspace too small");
    int* hist = (int*) ws;
    int* offs = (int*) ((char*) ws + up256((size_t) nblocks * n_local * 4));
    return run_permute(sel, rw, R, topk, lo, n_local, shared_rows, 0, bm, balance, counts, offs, hist, nblocks, order, tok, eid, wt, rbt, (Plan*) plan2, st);
}

size_t permute_ws_bytes(int R, int topk, int n_local)
{
    const size_t P = (size_t) R * topk;
    const int nblocks = (int) ((P + CHUNK - 1) / CHUNK);
    return up256((size_t) nblocks * n_local * 4) + up256((size_t) (n_local + 3) * 4);
}

int prefill_launch(const hmoe_layer* L, const void* x, int x_dtype, const int64_t* sel, const void* rw, int R, int lo, int n_local,
                   int act_quant, float* out, void* ws, size_t ws_bytes, cudaStream_t st, int shared_row0, int shared_rows,
                   void* const* out_peer, int world, int rows_per_rank)
{
    if (shared_rows < 0) { shared_row0 = 0; shared_rows = R; }
    if (out_peer && (world < 1 || world > 8 || rows_per_rank < 1 || (long long) world * rows_per_rank < R))
        return fail(HMOE_E_ARG, "hmoe_prefill_ep_peer: world must be 1..8 and world * rows_per_rank must cover the rows");          // default: the shared expert takes every row
    if (shared_row0 < 0 || shared_row0 + shared_rows > R) return fail(HMOE_E_ARG, "hmoe_prefill: shared row range outside the rows");
    const int H = L->H, I = L->I;
    if (R < 1) return fail(HMOE_E_ARG, "hmoe_prefill: rows must be >= 1");
    if (L->topk < 1 || L->topk > TOPK_MAX) return fail(HMOE_E_ARG, "hmoe_prefill: topk must be 1..8");
    if (H % 128 || I % 128 || H < 128 || I < 128) return fail(HMOE_E_ARG, "hmoe_prefill: H and I must be multiples of 128");
    if (n_local < 1 || n_local > 256) return fail(HMOE_E_ARG, "hmoe_prefill: 1..256 local experts");
    if (!(L->group == 0 && L->scale_dtype == HMOE_F32) && !(L->group == 128 && L->scale_dtype == HMOE_BF16))
        return fail(HMOE_E_ARG, "hmoe_prefill: scales must be fp32 per row (group 0) or bf16 per 128 columns");
    if (x_dtype != HMOE_F16 && x_dtype != HMOE_BF16) return fail(HMOE_E_ARG, "hmoe_prefill: x must be fp16 or bf16");
    if (!x || !sel || !rw || (!out && !out_peer) || !ws) return fail(HMOE_E_ARG, "hmoe_prefill: null pointer");
    const int kf = act_quant ? 2 : 1;
    const WsLayout w = ws_layout(R, L->topk, n_local, H, I, TN, kf);
    if (ws_bytes < w.total) return fail(HMOE_E_WS, "hmoe_prefill: workspace too small (the int8 mode needs hmoe_prefill_ws_bytes(..., act_quant = 1))");
    const int sms = device_sms();
    if (sms <= 0) return fail(HMOE_E_CUDA, "hmoe_prefill: no current CUDA device");
    set_gemm_attributes();
    char* b = (char*) ws;
    unsigned* status = (unsigned*) (b + w.status);
    Plan* plan = (Plan*) (b + w.plan);
    int* counts = (int*) (b + w.counts); int* offs = (int*) (b + w.offs); int* hist = (int*) (b + w.hist);
    int* order = (int*) (b + w.order); int* tok = (int*) (b + w.tok); int* eid = (int*) (b + w.eid); float* wt = (float*) (b + w.wt);
    int* rbt = (int*) (b + w.rbt);
    __half* xg = (__half*) (b + w.xg); __half* act = (__half*) (b + w.act);
    const int has_shared = L->sh_gate_w != nullptr;
    int rc = run_permute(sel, rw, R, L->topk, lo, n_local, has_shared ? shared_rows : 0, shared_row0, TN, 1, counts, offs, hist, w.nblocks, order, tok, eid, wt,
                         rbt, plan, st);
    if (rc) return rc;
    gather_kernel<<<w.rows_cap, 192, 0, st>>>(x, x_dtype == HMOE_BF16, tok, plan, H, act_quant, xg);
    CUtensorMap mx, ma, mx16, ma16;
    if (!make_map(&mx, xg, H * kf, (size_t) w.rows_cap, 64) || !make_map(&ma, act, I * kf, (size_t) w.rows_cap, 64) ||
        !make_map(&mx16, xg, H * kf, (size_t) w.rows_cap, 16) || !make_map(&ma16, act, I * kf, (size_t) w.rows_cap, 16)) return fail(HMOE_E_CUDA, "hmoe_prefill: cuTensorMapEncodeTiled failed");
    GemmArgs g;
    g.grouped = L->group != 0; g.act_quant = act_quant; g.n_local = n_local; g.kfold = kf; g.nsub = 1;
    g.sh_i8 = L->shared_format == 1 && L->sh_gate_w != nullptr;
    g.plan = plan; g.rbt = rbt; g.tok = tok; g.wt = wt; g.act = act; g.out = out; g.status = status;
    g.rows_per_rank = out_peer ? rows_per_rank : 0;
    for (int p = 0; p < 8; ++p) g.out_peer[p] = (out_peer && p < world) ? (float*) out_peer[p] : nullptr;
    g.K = H; g.N = I; g.w0 = L->gate_w; g.w1 = L->up_w; g.s0 = L->gate_s; g.s1 = L->up_s;
    g.sh_w0 = L->sh_gate_w; g.sh_w1 = L->sh_up_w; g.sh_s0 = L->sh_gate_s; g.sh_s1 = L->sh_up_s;
    prefill_gemm_kernel<false><<<sms, PF_THREADS, PfSmem::total, st>>>(mx, mx16, g);
    g.K = I; g.N = H; g.w0 = L->down_w; g.w1 = nullptr; g.s0 = L->down_s; g.s1 = nullptr;
    g.sh_w0 = L->sh_down_w; g.sh_w1 = nullptr; g.sh_s0 = L->sh_down_s; g.sh_s1 = nullptr;
    prefill_gemm_kernel<true><<<sms, PF_THREADS, PfSmem::total, st>>>(ma, ma16, g);
    count_launches(3);
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return fail(HMOE_E_CUDA, cudaGetErrorString(err));
    return HMOE_OK;
}

}  // namespace hmoe

#ifdef HMOE_PROBE_WAITS
extern "C" int hmoe_probe_read(unsigned long long* out, int clear)
{
    cudaDeviceSynchronize();
    cudaMemcpyFromSymbol(out, hmoe::g_probe, sizeof(unsigned long long) * 64);
    if (clear) { unsigned long long z[64] = {}; cudaMemcpyToSymbol(hmoe::g_probe, z, sizeof(z)); }
    return 0;
}
#endif
