// The streaming kernel of the decode and short-prefill paths, what it is given, and its launch. Instantiated in hmoe_decode.cu and, for the widest
// layers, in hmoe_decode_wide.cu.
#pragma once
#include "hmoe_common.cuh"
#include "hmoe_internal.h"

namespace hmoe {

// The expert-parallel combine, done by the down launch itself when its blocks run out of weights to stream (instead of a kernel
// of its own after it). The block that finishes last raises this rank's generation in every peer's flag array (release, system
// scope); every block then waits, bounded, until all peers have raised theirs here, and sums its slice of the peers' partial slots
// into the layer output in rank order (all rows: identical bits on every rank; or only the rows this rank owns when the tokens
// are data-parallel), and clears its slice of the other slot for the step after next. Blocks that finish early wait on SMs that
// would otherwise idle: the tail costs one flag round trip and one round of peer loads after the slowest rank's last weight.
struct EpTail
{
    int rank, world, own_rows, n;     // n = rows * H
    float* slots[8];                  // slots[p] = rank p's two partial slots as seen from here
    unsigned* flags[8];               // flags[p] = rank p's flag array [world]
    float* f;                         // layer output, added into
    unsigned* done;                   // arrival counter of this launch's blocks (in the workspace, returns to zero)
    unsigned* status;                 // status word for a wait that gives up
};

struct DecodeArgs
{
    int H, I;
    const int64_t* gate_w; const int64_t* up_w; const int64_t* down_w;
    const int64_t* gate_s; const int64_t* up_s; const int64_t* down_s;
    const void* sh_gw; const void* sh_uw; const void* sh_dw; const void* sh_gs; const void* sh_us; const void* sh_ds;
    const Route* route;
    const __half* xf;      // [R][H] prepared rows
    const float* xscale;   // [R][H/32] (Q8)
    __half* act;           // [tiles][8][I] gate_up output = down input
    float* ascale;         // [tiles][8][I/32] (Q8)
    float* G;              // register-resident path: [pick rows][gate | up][I] fp32 sums (shares memory with act)
    float* y;              // [R][H] (expert-parallel: base of two slots, the step's slot is chosen by *gen_ptr & 1)
    const unsigned* gen_ptr; size_t slot_stride;
    unsigned* status;
    EpTail ep;             // expert parallel: the combine over peer memory as the tail of the down launch (world = 0: none)
};

namespace {

constexpr int CW = 16;                   // warps per block
constexpr int NTHREADS = CW * 32;
constexpr int NSTAGE = 3;

__device__ __forceinline__ void ep_st_release_sys(unsigned* p, unsigned v) { asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ unsigned ep_ld_acquire_sys(const unsigned* p)
{
    unsigned v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float4 ep_ld_peer(const float4* p)
{
    float4 v;
    asm volatile("ld.relaxed.sys.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

// called by all threads of every block of the down launch, after the block's last reduction has been issued
__device__ __forceinline__ void ep_tail_combine(const EpTail& e, unsigned gen, size_t slot_floats, int H)
{
    __shared__ int ok_sh;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        if (atomicAdd(e.done, 1u) == gridDim.x - 1)
        {
            *e.done = 0u;
            __threadfence_system();
            for (int p = 0; p < e.world; ++p) ep_st_release_sys(e.flags[p] + e.rank, gen);
        }
        int ok = 1;
        const unsigned long long t0 = globaltimer_ns();
        for (int p = 0; p < e.world && ok; ++p)
            while ((int) (ep_ld_acquire_sys(e.flags[e.rank] + p) - gen) < 0)
                if (globaltimer_ns() - t0 > 2000000000ull) { ok = 0; atomicOr(e.status, ST_WAIT_TIMEOUT); break; }
        ok_sh = ok;
    }
    __syncthreads();
    if (!ok_sh) return;
    const int parity = gen & 1;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) * 4; i < e.n; i += gridDim.x * blockDim.x * 4)
    {
        *(float4*) (e.slots[e.rank] + (size_t) (parity ^ 1) * slot_floats + i) = make_float4(0.f, 0.f, 0.f, 0.f);
        int o = i;
        if (e.own_rows)
        {
            const int r = i / H;
            if (r % e.world != e.rank) continue;
            o = (r / e.world) * H + (i - r * H);
        }
        // all peers' loads are issued before the first sum (a warp issues in order: a sum between two loads would serialise
        // the NVLink round trips); the sums then run in rank order
        float4 v[8];
        #pragma unroll
        for (int p = 0; p < 8; ++p)
            if (p < e.world) v[p] = ep_ld_peer((const float4*) (e.slots[p] + (size_t) parity * slot_floats + i));
        float4 acc = *(float4*) (e.f + o);
        #pragma unroll
        for (int p = 0; p < 8; ++p)
            if (p < e.world) { acc.x += v[p].x; acc.y += v[p].y; acc.z += v[p].z; acc.w += v[p].w; }
        *(float4*) (e.f + o) = acc;
    }
}

// Two 64-column blocks (one scale group) of a 64-row group: 4 strips x 8 steps of MMAs on the tile, added into acc with
// the scales applied. wsm = shared address of the first block's 2 KB unit; the second follows it.
template <bool GROUPED, bool Q8>
__device__ __forceinline__ void consume_group(uint32_t wsm, const uint32_t (&bx)[2][8], const uint4 sc, const float4 sx0, const float4 sx1,
                                              float (*acc)[4], int lane)
{
    const uint32_t scw[4] = {sc.x, sc.y, sc.z, sc.w};
    const float sxa[4] = {sx0.x, sx0.y, sx0.z, sx0.w}, sxb[4] = {sx1.x, sx1.y, sx1.z, sx1.w};
    // The four strips' sums are independent MMA chains; the steps are interleaved across strips so that consecutive MMAs
    // never wait on each other.
    float part[4][4];
    #pragma unroll
    for (int s = 0; s < 4; ++s) part[s][0] = part[s][1] = part[s][2] = part[s][3] = 0.f;
    #pragma unroll
    for (int blk = 0; blk < 2; ++blk)
    {
        uint4 w4[4];
        #pragma unroll
        for (int s = 0; s < 4; ++s) w4[s] = lds128(wsm + blk * 2048 + s * 512 + lane * 16);
        #pragma unroll
        for (int t = 0; t < 4; ++t)
        {
            #pragma unroll
            for (int s = 0; s < 4; ++s)
            {
                const uint32_t w = t == 0 ? w4[s].x : t == 1 ? w4[s].y : t == 2 ? w4[s].z : w4[s].w;
                uint32_t a[4];
                frag_from_codes(w, a);
                mma_f16((GROUPED || Q8) ? part[s] : acc[s], a, bx[blk][2 * t], bx[blk][2 * t + 1]);
            }
            if (Q8 && (t & 1))
            {
                // int8 activations: the sums of 32 columns are exact integers; one multiply by (activation scale x weight scale)
                const int qt = blk * 2 + (t >> 1);
                #pragma unroll
                for (int s = 0; s < 4; ++s)
                {
                    float s0 = 1.f, s1 = 1.f;
                    if (GROUPED) { s0 = __uint_as_float(scw[s] << 16); s1 = __uint_as_float(scw[s] & 0xffff0000u); }
                    acc[s][0] = fmaf(part[s][0], sxa[qt] * s0, acc[s][0]); acc[s][1] = fmaf(part[s][1], sxb[qt] * s0, acc[s][1]);
                    acc[s][2] = fmaf(part[s][2], sxa[qt] * s1, acc[s][2]); acc[s][3] = fmaf(part[s][3], sxb[qt] * s1, acc[s][3]);
                    part[s][0] = part[s][1] = part[s][2] = part[s][3] = 0.f;
                }
            }
        }
    }
    if (GROUPED && !Q8)
    {
        #pragma unroll
        for (int s = 0; s < 4; ++s)
        {
            const float s0 = __uint_as_float(scw[s] << 16), s1 = __uint_as_float(scw[s] & 0xffff0000u);
            acc[s][0] = fmaf(s0, part[s][0], acc[s][0]); acc[s][1] = fmaf(s0, part[s][1], acc[s][1]);
            acc[s][2] = fmaf(s1, part[s][2], acc[s][2]); acc[s][3] = fmaf(s1, part[s][3], acc[s][3]);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// The streaming kernel of the register-resident path, used twice per call: gate_up (DOWN = false) and down (DOWN = true).
//
// An item is (tile, matrix, 64-row group of the output): 64 rows x all K input columns of codes (gate_up: 192 KB for
// K = 6144, down: 64 KB). Items are dealt out to the blocks as contiguous ranges with the row group fastest, then the
// matrix (gate, up), then the tile, so a block walks the matrices in address order and stays with one tile - one set of
// activations - for a long time. The K columns are cut into KC chunks of 2048; warp w owns the 128 columns
// [2048 kc + 128 w, + 128) of every chunk: one scale group, 4 KB of codes, contiguous in memory. Its activation fragments
// for those columns (16 registers per chunk) stay in registers for the whole tile, so the inner loop reads nothing but
// shared memory. Every warp has a private ring of NSTAGE slots (4 KB of codes + the 128 bytes of bf16 scales of the same
// 64 rows x 128 columns), each with its own mbarrier; when the warp has read a slot its lane 0 at once issues the copies
// for the slot's next use, so the warps stream independently and no warp ever waits for another.
// A warp ends an item with a 64 x 8 partial tile over its KC x 128 columns; the real tile columns are added to the result
// with fp32 reductions in global memory (sixteen per output element, one per warp):
//   gate_up -> G[pick row][gate | up][I]  (zeroed by the prepare kernel; pick row = Route::rowbase[tile] + tile column)
//   down    -> y[row][H]
// Between the two launches nothing else runs: the down kernel turns G into its own MMA operand when it enters a tile
// (SiLU(gate) * up * routing weight, in the int8 mode followed by the CPU engine's second int8 round trip).
// Programmatic dependent launch: a kernel lets the next one in the stream start as its own blocks retire (the next kernel's
// blocks set up their barriers and request their first weights meanwhile), and the next kernel waits here for the full
// completion of its predecessor, memory included, before it reads anything the predecessor wrote. Both are no-ops for a
// kernel launched without the attribute.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ void red_add(float* p, float v)
{
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "f"(v) : "memory");
}

struct StreamSmem
{
    static constexpr int SLOT = 4096 + 128;
    static constexpr int bars = NSTAGE * CW * SLOT;
    static constexpr int flags = bars + NSTAGE * CW * 8;
    static constexpr int total = flags + 16;
};

// WIDE: layers wider than 6144 x 2048, whose SiLU has always been computed with expf, as in the int8 mode, and which the fused combine does not serve.
template <bool GROUPED, bool Q8, bool DOWN, int KC, typename RT = Route, bool WIDE = false>
__global__ void __launch_bounds__(NTHREADS, 1) decode_stream_kernel(const DecodeArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    constexpr int SLOT = StreamSmem::SLOT;
    const uint32_t sbase = smem_u32(smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const uint32_t ring = sbase + warp * SLOT, full0 = sbase + StreamSmem::bars + warp * 8;      // slot st: + st * CW * SLOT / + st * CW * 8
    volatile int* abort_flag = (volatile int*) (smem + StreamSmem::flags);
    if (threadIdx.x == 0)
    {
        for (int i = 0; i < NSTAGE * CW; ++i) mbar_init(sbase + StreamSmem::bars + i * 8, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    __syncthreads();
    // gate_up follows the prepare kernel, which wrote the route; down follows gate_up, but the route and the weights it
    // needs to fill its rings are older than that: it waits only before it reads the gate / up sums.
    // Ordering rule of the chain: a kernel lets its dependents start only after its own wait has returned, i.e. after the
    // kernel before it has completed with its memory visible. So whatever a dependent reads before ITS wait (down: the route,
    // the step counter) was written at least two kernels back and is complete, whatever the occupancy. Blocks without work
    // wait too, so that a grid with nothing to do cannot release its dependents early.
    TL_MIN(DOWN ? 8 : 0);
    if (!DOWN) { pdl_wait(); pdl_launch_dependents(); TL_MIN(2); }
    const RT* rt = reinterpret_cast<const RT*>(a.route);          // RT = RouteShort: the same fields with room for more tiles
    const int K = DOWN ? a.I : a.H, N = DOWN ? a.H : a.I;          // input columns and output rows of one matrix
    const int KB = K / 64, NG = N / 64, J = DOWN ? NG : 2 * NG;
    const int p0 = rt->split[DOWN][blockIdx.x], p1 = rt->split[DOWN][blockIdx.x + 1];      // cut at equal cost by the prepare kernel
    float* const out0 = DOWN ? a.y + (a.gen_ptr ? (size_t) (*a.gen_ptr & 1u) * a.slot_stride : 0) : a.G;
    if (p0 < p1 && 2 * warp < KB)
    {
        // ---- fill cursor (lane 0): the next slot to request is chunk f_kc of item (f_tile, f_j)
        int f_p = p0, f_tile = p0 / J, f_j = p0 % J, f_kc = 0;
        const char* f_w = nullptr; const char* f_s = nullptr;
        auto fill_next = [&](uint32_t slot) {
            if (f_p >= p1) return;
            const int mat = (!DOWN && f_j >= NG) ? 1 : 0, gr = f_j - mat * NG;
            if (f_w == nullptr || (gr == 0 && f_kc == 0))
            {
                const int e = rt->expert[f_tile];
                const void* w = DOWN ? (e >= 0 ? (const void*) a.down_w[e] : a.sh_dw)
                                     : (mat ? (e >= 0 ? (const void*) a.up_w[e] : a.sh_uw) : (e >= 0 ? (const void*) a.gate_w[e] : a.sh_gw));
                f_w = (const char*) w + (size_t) warp * 4096;
                if (GROUPED)
                {
                    const void* sc = DOWN ? (e >= 0 ? (const void*) a.down_s[e] : a.sh_ds)
                                          : (mat ? (e >= 0 ? (const void*) a.up_s[e] : a.sh_us) : (e >= 0 ? (const void*) a.gate_s[e] : a.sh_gs));
                    f_s = (const char*) sc + (size_t) warp * 128;
                }
            }
            const uint32_t bar = full0 + slot * CW * 8, dst = ring + slot * CW * SLOT;
            mbar_expect_tx(bar, GROUPED ? SLOT : 4096);
            bulk_g2s(dst, f_w + ((size_t) gr * KB + f_kc * 32) * 2048, 4096, bar);
            if (GROUPED) bulk_g2s(dst + 4096, f_s + ((size_t) gr * (K / 128) + f_kc * 16) * 128, 128, bar);
            if (++f_kc == KC || f_kc * 32 + 2 * warp >= KB)
            {
                f_kc = 0; ++f_p;
                if (++f_j == J) { f_j = 0; ++f_tile; f_w = nullptr; }
            }
        };
        if (lane == 0)
            for (uint32_t i = 0; i < NSTAGE; ++i) fill_next(i);

        // ---- consume (all lanes)
        uint32_t bx[KC][2][8];                  // the tile's activation fragments of this warp's columns
        float4 sx[KC][2];                       // Q8: their scales per 32 columns for tile columns 2q and 2q + 1
        #pragma unroll
        for (int kc = 0; kc < KC; ++kc) sx[kc][0] = sx[kc][1] = make_float4(1.f, 1.f, 1.f, 1.f);
        int nrows = 0;
        float* outA = nullptr; float* outB = nullptr;         // result rows of tile columns 2q and 2q + 1, at this lane's row g
        const float* sdp[2] = {nullptr, nullptr};             // !GROUPED: per-row scales, at this lane's row g
        auto enter_tile = [&](int tile) {
            const int e = rt->expert[tile];
            nrows = rt->nrows[tile];
            if (!DOWN)
            {
                const char* xb = (const char*) (a.xf + (size_t) rt->rows[tile][g] * a.H) + (size_t) warp * 256 + q * 32;
                #pragma unroll
                for (int kc = 0; kc < KC; ++kc)
                {
                    uint4 b0 = make_uint4(0, 0, 0, 0), b1 = b0, b2 = b0, b3 = b0;
                    if (kc * 32 + 2 * warp < KB)
                    {
                        const char* xk = xb + kc * 4096;
                        b0 = ldg128(xk); b1 = ldg128(xk + 16); b2 = ldg128(xk + 128); b3 = ldg128(xk + 144);
                        if (Q8)
                        {
                            sx[kc][0] = *(const float4*) (a.xscale + (size_t) rt->rows[tile][2 * q] * (a.H / 32) + 64 * kc + 4 * warp);
                            sx[kc][1] = *(const float4*) (a.xscale + (size_t) rt->rows[tile][2 * q + 1] * (a.H / 32) + 64 * kc + 4 * warp);
                        }
                    }
                    bx[kc][0][0] = b0.x; bx[kc][0][1] = b0.y; bx[kc][0][2] = b0.z; bx[kc][0][3] = b0.w;
                    bx[kc][0][4] = b1.x; bx[kc][0][5] = b1.y; bx[kc][0][6] = b1.z; bx[kc][0][7] = b1.w;
                    bx[kc][1][0] = b2.x; bx[kc][1][1] = b2.y; bx[kc][1][2] = b2.z; bx[kc][1][3] = b2.w;
                    bx[kc][1][4] = b3.x; bx[kc][1][5] = b3.y; bx[kc][1][6] = b3.z; bx[kc][1][7] = b3.w;
                }
                const size_t rb = (size_t) rt->rowbase[tile] + 2 * q;
                outA = a.G + rb * 2 * a.I + g; outB = outA + 2 * a.I;
                if (!GROUPED)
                {
                    sdp[0] = (const float*) (e >= 0 ? (const void*) a.gate_s[e] : a.sh_gs) + g;
                    sdp[1] = (const float*) (e >= 0 ? (const void*) a.up_s[e] : a.sh_us) + g;
                }
            }
            else
            {
                // The operand of tile column t is computed by the whole warp, lane L taking columns 2L, 2L + 1 of each of the
                // warp's two blocks (= word L of the block), and handed to the lanes g == t in the order the MMAs read:
                // word [blk][2t' + h] of lane (g, q) is word 8t' + 4h + q of the block.
                #pragma unroll
                for (int kc = 0; kc < KC; ++kc)
                {
                    #pragma unroll
                    for (int blk = 0; blk < 2; ++blk)
                        #pragma unroll
                        for (int wd = 0; wd < 8; ++wd) bx[kc][blk][wd] = 0u;
                    if (KC > 1 && kc * 32 + 2 * warp >= KB) continue;
                    float sa[4] = {1.f, 1.f, 1.f, 1.f}, sb[4] = {1.f, 1.f, 1.f, 1.f};
                    const float* gp = a.G + (size_t) rt->rowbase[tile] * 2 * a.I + (size_t) kc * 2048 + (size_t) warp * 128 + 2 * lane;
                    for (int t = 0; t < nrows; ++t, gp += 2 * a.I)
                    {
                        const float2 g0 = __ldcg((const float2*) gp), g1 = __ldcg((const float2*) (gp + 64));
                        const float2 u0 = __ldcg((const float2*) (gp + a.I)), u1 = __ldcg((const float2*) (gp + a.I + 64));
                        const float wt = rt->w[tile][t];
                        // fp16 operands: the fast exponential is far inside their rounding; the int8 mode follows the CPU engine
                        constexpr bool EXACT = Q8 || WIDE;
                        float v[2][2];
                        v[0][0] = g0.x / (1.f + (EXACT ? expf(-g0.x) : __expf(-g0.x))) * u0.x * wt;
                        v[0][1] = g0.y / (1.f + (EXACT ? expf(-g0.y) : __expf(-g0.y))) * u0.y * wt;
                        v[1][0] = g1.x / (1.f + (EXACT ? expf(-g1.x) : __expf(-g1.x))) * u1.x * wt;
                        v[1][1] = g1.y / (1.f + (EXACT ? expf(-g1.y) : __expf(-g1.y))) * u1.y * wt;
                        #pragma unroll
                        for (int blk = 0; blk < 2; ++blk)
                        {
                            if (Q8)
                            {
                                // second int8 round trip of the CPU engine (cpuband.cpp:200-207): 32 consecutive values = 16 lanes
                                float m = fmaxf(fabsf(v[blk][0]), fabsf(v[blk][1]));
                                #pragma unroll
                                for (int o = 8; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                                const float sc = m > 0.f ? __fdiv_rn(m, 127.f) : 1.f, inv = __fdiv_rn(1.f, sc);
                                v[blk][0] = (float) __float2int_rn(__fmul_rn(v[blk][0], inv));
                                v[blk][1] = (float) __float2int_rn(__fmul_rn(v[blk][1], inv));
                                // the MMA results of a lane are tile columns 2q and 2q + 1: those lanes keep this column's scales
                                const float s_lo = __shfl_sync(0xffffffffu, sc, 0), s_hi = __shfl_sync(0xffffffffu, sc, 16);
                                if (2 * q == t) { sa[2 * blk] = s_lo; sa[2 * blk + 1] = s_hi; }
                                if (2 * q + 1 == t) { sb[2 * blk] = s_lo; sb[2 * blk + 1] = s_hi; }
                            }
                            const __half2 h = __floats2half2_rn(v[blk][0], v[blk][1]);
                            const uint32_t word = *(const uint32_t*) &h;
                            #pragma unroll
                            for (int wd = 0; wd < 8; ++wd)
                            {
                                const uint32_t got = __shfl_sync(0xffffffffu, word, (wd >> 1) * 8 + (wd & 1) * 4 + q);
                                if (g == t) bx[kc][blk][wd] = got;
                            }
                        }
                    }
                    if (Q8) { sx[kc][0] = make_float4(sa[0], sa[1], sa[2], sa[3]); sx[kc][1] = make_float4(sb[0], sb[1], sb[2], sb[3]); }
                }
                outA = out0 + (size_t) rt->rows[tile][2 * q] * a.H + g; outB = out0 + (size_t) rt->rows[tile][2 * q + 1] * a.H + g;
                if (!GROUPED) sdp[0] = (const float*) (e >= 0 ? (const void*) a.down_s[e] : a.sh_ds) + g;
            }
        };
        // !GROUPED: the eight per-row scales of this lane's rows for item jj, applied to the finished sums
        auto load_row_scales = [&](int jj, float* sd) {
            const int mat = (!DOWN && jj >= NG) ? 1 : 0, gr = jj - mat * NG;
            #pragma unroll
            for (int i = 0; i < 8; ++i) sd[i] = __ldg(sdp[mat] + gr * 64 + i * 8);
        };
        float sd[8];
        #pragma unroll
        for (int i = 0; i < 8; ++i) sd[i] = 1.f;
        float acc[4][4];
        #pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
        uint32_t st = 0, par = 0;
        int tile = p0 / J, j = p0 % J;
        if (DOWN) { pdl_wait(); pdl_launch_dependents(); TL_MIN(10); }
        // With scale groups a tile is entered in one place of the code: a second copy made the kernel a fifth larger, and a one-row step depended on
        // where its code lay (65.2 or 67.5 us). With row scales the copy is the better one (11 rows, 256 experts: 331 against 335 us).
        bool alive = true, enter = GROUPED;
        if (!GROUPED) { enter_tile(tile); load_row_scales(j, sd); }
        for (int p = p0; p < p1 && alive; ++p)
        {
            if (GROUPED && enter) { enter_tile(tile); enter = false; }
            float sdn[8];
            #pragma unroll
            for (int k = 0; k < 8; ++k) sdn[k] = 1.f;
            const bool same_tile = j + 1 < J;
            if (!GROUPED && same_tile && p + 1 < p1) load_row_scales(j + 1, sdn);          // one item ahead
            #pragma unroll
            for (int kc = 0; kc < KC; ++kc)
            {
                if (kc * 32 + 2 * warp < KB)
                {
                    if (!mbar_wait(full0 + st * CW * 8, par, abort_flag, a.status)) { alive = false; break; }
                    TL_MIN(DOWN ? 12 : 4);
                    const uint32_t slot = ring + st * CW * SLOT;
                    uint4 sc = make_uint4(0, 0, 0, 0);
                    if (GROUPED) sc = lds128(slot + 4096 + g * 16);
                    consume_group<GROUPED, Q8>(slot, bx[kc], sc, sx[kc][0], sx[kc][1], acc, lane);
                    __syncwarp();
                    if (lane == 0) fill_next(st);
                    if (++st == NSTAGE) { st = 0; par ^= 1; }
                }
            }
            if (!alive) break;
            // this warp's partial sums of the real tile columns join the result
            #pragma unroll
            for (int c = 0; c < 2; ++c)
            {
                if (2 * q + c < nrows)
                {
                    float* yr = (c ? outB : outA) + j * 64;
                    #pragma unroll
                    for (int ss = 0; ss < 4; ++ss)
                    {
                        red_add(yr + ss * 16, acc[ss][c] * sd[2 * ss]);
                        red_add(yr + ss * 16 + 8, acc[ss][2 + c] * sd[2 * ss + 1]);
                    }
                }
            }
            #pragma unroll
            for (int ss = 0; ss < 4; ++ss) acc[ss][0] = acc[ss][1] = acc[ss][2] = acc[ss][3] = 0.f;
            if (same_tile)
            {
                ++j;
                #pragma unroll
                for (int k = 0; k < 8; ++k) sd[k] = sdn[k];
            }
            else if (p + 1 < p1)
            {
                j = 0; ++tile;
                if (GROUPED) enter = true;
                else { enter_tile(tile); load_row_scales(j, sd); }
            }
        }
    }
    else if (DOWN) { pdl_wait(); pdl_launch_dependents(); }
    __syncthreads();
    abort_drain(abort_flag);
    TL_MAX(DOWN ? 9 : 1);
    if (DOWN && !WIDE && a.ep.world > 0) ep_tail_combine(a.ep, *a.gen_ptr, a.slot_stride, a.H);
}

template <typename Kern>
static void launch_dependent(Kern kern, int grid, const DecodeArgs& a, cudaStream_t st, bool dependent)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(NTHREADS); cfg.dynamicSmemBytes = StreamSmem::total; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = dependent ? 1 : 0;
    cfg.attrs = at; cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, a);
}

template <bool G, bool Q, bool DOWN, int KC, bool WIDE = false>
static void launch_stream(int grid, const DecodeArgs& a, cudaStream_t st, bool dependent)
{
    static DeviceOnce once;
    if (once.first()) cudaFuncSetAttribute(decode_stream_kernel<G, Q, DOWN, KC, Route, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, StreamSmem::total);
    launch_dependent(decode_stream_kernel<G, Q, DOWN, KC, Route, WIDE>, grid, a, st, dependent);
}

}  // namespace
}  // namespace hmoe
