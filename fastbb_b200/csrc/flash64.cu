// O = softmax(scale . Q K^T) V for head dimension 64, no mask, any N: tcgen05 UMMA for both products, softmax in
// registers, K/V tiles streamed by TMA. Replaces flash64_r{1,2}_{hh,fh,ff} (fastbb/fastbb_kernels.cu:58-312) and the
// SDPA fallback for small inputs (fastbb/vit.py:146-150). Q, K, V are read in place from the strided [b, n, h, 64]
// views of the packed qkv GEMM output; O is written as [b, n, h*64].
//
// Work: a "tile group" is NQ (1 or 2) tiles of 128 queries of one (batch, head); it walks the keys in blocks of 128, so
// the whole problem is groups x key blocks "units". Without a workspace every CTA takes exactly one group. With a
// workspace, and when the groups do not fill the SMs evenly, the grid is persistent (one CTA per SM): every CTA first
// takes whole groups round-robin (group = round * G + cta, so CTAs running together share heads, i.e. K/V tiles in L2)
// for all but the last full wave, then an equal share of the units of what is left (between one and two waves' worth,
// so a share is at least one group long and a group is split over at most two CTAs):
//   - the CTA whose share starts in the middle of a group (always the first item of its share) leaves the unnormalised
//     O (fp32), the running maxima and sums in its workspace slot and raises the slot's per-warp flags;
//   - the CTA that began that group (always the last item of its share, so it needs the slot late) merges the slot into
//     its own accumulators, clears the flags and writes the rows.
// With 400 groups on 148 SMs (ViT-L/14 at 896x1344) this replaces 3 waves by 2.7; part of the gain is lost because the
// two tiles of a long-lived CTA drift into step (see below): 2.5 % on whole-model time.
//
//   warp 0          TMA producer: the Q tiles of each item, then K_j and V_j into a ring of stages (128-byte swizzle, zero fill)
//   warps 1, 2      UMMA issuers, one per tile: S_t = Q_t K_j^T (both K-major, 4 x K16) into tensor memory, issued as
//                   soon as the softmax group holds the previous S_t in registers - also across items, so the first
//                   product of the next group overlaps the last softmax and the write-out of this one; once the group
//                   has written P_t (fp16) back into tensor memory, O_t += P_t V_j (A from tensor memory, V as the
//                   MN-major B operand, 8 x K16); O_t stays in tensor memory (fp32) over the key blocks of an item
//   warps 4..11/12..19 softmax group t, 16 query rows per warp: tcgen05.ld 16x256b hands thread i the key pairs
//                   8k + 2(i%4), +1 of rows i/4 and i/4 + 8 (the m16n8 accumulator fragment), and P (fp16 pairs) goes back
//                   with the matching 16x128b store. The 128-key block is loaded at once; the maximum is taken with 3-input
//                   max, p = 2^(s*scale*log2e - m) with packed f32x2 FMAs. The running maximum m is only raised when a block
//                   exceeds it by more than 2^8 (then O_t and the running sum are rescaled in place, a rare event after the
//                   first blocks); otherwise P is taken relative to the older maximum, which keeps it <= 256 and exactly as
//                   accurate in fp16. The loop over an item's blocks holds only what every block needs: each thread compares
//                   its own share of a row with the row's limit and the warp votes. What other blocks need stands outside it:
//                   an item's first block (which takes the maximum, with two shuffles among the four threads that share a
//                   row) before the loop; a ragged last block in a masking copy of the loop's code; a block that has to raise
//                   the maximum in code that reads S again from tensor memory in halves. An item's rows are written by
//                   16-row TMA stores in the NEXT item's first block, behind that block's exponentials, a CTA's last rows by
//                   plain stores, and Q has two buffers, so that neither tile stops between items. One loop for all of this,
//                   the write-out between items, one Q buffer / this form, us a call, in turn in one process, from CUDA graphs:
//                   1496 / 1337 (1 x 16385 tokens x 16 heads), 217 / 198 (1 x 6145 x 16), 81.5 / 71.5 (1 x 4097 x 12),
//                   13.8 / 11.5 (1 x 1041 x 12), 81.8 / 74.8 (4 x 1370 x 24), 59.0 / 52.5 (32 x 257 x 16), 6.9 / 6.2 (1 x 257 x
//                   16).
//                   Four softmax warps share each SM sub-partition and cover one another's waits (measured against
//                   one-thread-per-row groups of four warps: 740 -> 849 TFLOP/s at N = 16385).
// With NQ = 2 the two groups alternate on the tensor core (S of one tile is computed while the other tile is in its
// softmax). Variants (fastbb/attention.py:5-7) name the accumulate types of the two products in the reference's
// mma.sync kernels, where fp16 accumulation doubles the GeForce tensor rate. On tcgen05 an f16 accumulator runs at the
// same rate as an fp32 one, and reading it back costs a conversion per element (measured: 215 vs 201 us per launch at
// N = 6145), so ff, fh and hh all run with fp32 S here; the softmax arithmetic is fp32 as in the reference. P.V
// accumulates in fp32 as well, because O lives in tensor memory across all key blocks: an fp16 accumulator there would
// add N terms in fp16, where the reference's fh / hh only ever add 64 (one key block) before going to fp32. Every
// variant is therefore at least as accurate as the reference's.
// The kernel is bound by the exponentials, not the tensor core: 128 x 128 of them per S tile against 16 results per
// clock per SM from the transcendental unit is twice the time of the tile's two matrix products (1024 vs 2 x 256 clocks).
// A launch of 6145 tokens x 16 heads keeps that unit 82 % busy over its active clocks, the tensor pipe 41 %. Measured dynamics
// worth knowing before changing the pipeline: a softmax warp alone cannot saturate the unit, so the two tiles run fastest half a
// period apart; in step, every phase collides with its twin. The half-period offset set at start-up is not stable: over some
// tens of units the later tile catches up. CTAs that live for one group (<= ~130 units) mostly keep it; the persistent form
// loses part of what it gains from the removed wave this way. On the older loop (clocks per unit 2800 half a period apart, 3800
// in step; 198 - 200 us at 6145 tokens with 25 groups a head) every way of forcing the offset that was built measured slower than
// letting the tiles run free: strict turns around a whole unit (3100 clocks per unit); turns around the exponential loop only,
// per SM sub-partition (218 us: the two warps a tile has on a sub-partition do not saturate its unit on their own, four
// contending warps use it better); a one-sided lock that only holds a tile back until the other is 4/16 .. 14/16 of the way
// through its exponentials (201 - 212 us). So did writing P back in two halves (a second wait, 212 us).
// Short launches (N <= 300, one tile per CTA) are chains of latencies: 1650 clocks from the dependency wait to the first Q and K in
// shared memory, 650 more to S, 1200 - 1600 for a block's softmax, 1650 from the last P.V to the end.
#include "common.cuh"
#include <cstdlib>
#include <type_traits>

#include "internal.h"

namespace fbb {

constexpr int FQ = 128;       // queries per tile
constexpr int FK = 128;       // keys per block
constexpr int kKVStages = 4;
constexpr int kTileBytes = 128 * 64 * 2;  // one [128 x 64] fp16 tile
constexpr float kLazyMax = 8.0f;          // raise the running maximum only beyond 2^8
// Key groups of eight whose exponentials a thread takes before the test of the running maximum is known: the test's vote then
// costs no wait, and S_t is released that much later. Measured on B200 (us at 1 x 16385 x 16 / 1 x 6145 x 16 / 1 x 1041 x 12 / 32 x
// 257 x 16): 0 -> 1396 / 198 / 11.9 / 52.7, 2 -> 1360 / 195 / 11.6 / 52.5, 4 -> 1337 / 198 / 11.5 / 52.5, 8 -> 1386 / 200 / 11.8 / 53.4.
constexpr int kEarly = 4;
// Register split of the 640-thread (NQ = 2) kernel. It is launched with 96 registers per thread (the most 20 warps can
// get); setmaxnreg.inc WAITS until the CTA's own pool has the registers, so the split must fit in that pool or the
// kernel never starts its softmax: 128 * kRegsCtl + 512 * kRegsSoftmax <= 640 * 96. A softmax thread holds 64 scores and up to
// 32 packed probabilities; 104 hold them (one predicate word spills), and the issuers keep their loop state in registers with 56 (us at
// 1 x 16385 x 16 / 1 x 6145 x 16 / 4 x 1370 x 24: 1337 / 198 / 74.8; with 32 / 112: 1368 / 202 / 80.1).
constexpr int kRegsCtl = 56, kRegsSoftmax = 104;
static_assert(128 * kRegsCtl + 512 * kRegsSoftmax <= 640 * 96, "setmaxnreg split exceeds the CTA's register pool");

// tensor-memory columns of tile t: S_t (128 columns) at t * kColTileS, O_t (fp32, 64 columns) at kColO + t * kColTileOP,
// P_t (fp16 pairs, 64 columns) kColP after O_t
constexpr uint32_t kColTileS = 128, kColO = 256, kColTileOP = 64, kColP = 128;

struct FlashSmem {
    static constexpr int kQOff = 0;                                  // two items x NQ (<= 2) tiles x 16 KB
    static constexpr int kKOff = 4 * kTileBytes;                     // stages x 16 KB
    static constexpr int kVOff = kKOff + kKVStages * kTileBytes;     // stages x 16 KB
    static constexpr int kOOff = kVOff + kKVStages * kTileBytes;     // output rows on their way out: 16 warps x 2 KB
    static constexpr int kBarOff = kOOff + 2 * kTileBytes;
    // barriers: q_full[2], q_empty[2], k_full[S], v_full[S], k_empty[S], v_empty[S], s_full[2], p_ready[2], pv_done[2], s_free[2], t1_go
    static constexpr int kNumBars = 4 + 4 * kKVStages + 8 + 1;
    static constexpr int kTailOff = kBarOff + kNumBars * 8 + 16;    // TailItems (40 bytes)
    static constexpr int kBytes = kTailOff + 48;
    // no slack for aligning by hand (the array is declared 1024-byte aligned)
    static constexpr int kDynamic = kBytes;
};
static_assert(FlashSmem::kDynamic <= 232448, "more shared memory than a CTA can have");

// Workspace of the split form: per CTA one slot for the group it starts in the middle. A slot holds, for each of the 16
// softmax warps, 36 values per lane stored [value][lane] (32 accumulator registers of the 16x256b fragment, then the two
// running maxima and the lane's shares of the two running sums), preceded by one flag word per warp.
constexpr int kSlotWarps = 16;
constexpr int kSlotValues = 36;
constexpr size_t kSlotFloats = (size_t)kSlotWarps * kSlotValues * 32;
constexpr size_t kFlagBytesPerCta = kSlotWarps * sizeof(unsigned);
// Leftover query rows: every ViT token count is a multiple of the 256-row tile group plus the cls token (and a few
// registers), and a 25th group per head for ONE row costs the N = 6145 launch 3.5 % (N = 6144: 189 us, 6145: 200 us).
// Up to kSideMaxRows rows beyond the last full group are therefore not tiled: a second, small launch
// (flash64_side_rows_kernel) computes them on the CUDA cores. It is the tiled launch's programmatic dependent, so its
// CTAs (128 threads, 32 registers, no shared memory: what the tiled kernel leaves free on an SM) run beside the tiled
// kernel's, and it waits for that kernel only at its very end, so that whatever depends on it depends on both.
constexpr int kSideMaxRows = 8;
constexpr int kSideMaxChunks = 64;
constexpr int kSideValues = 66;  // per (row, key chunk): 64 outputs, maximum, sum
constexpr int kSideMaxTasks = 1024;
// flag words of the split form, then one counter per leftover row
constexpr size_t flag_region_bytes(int ctas) { return ((size_t)ctas * (kFlagBytesPerCta + sizeof(unsigned)) + 255) & ~(size_t)255; }
constexpr size_t side_region_bytes() { return ((size_t)kSideMaxTasks * kSideValues * sizeof(float) + 255) & ~(size_t)255; }
int64_t flash64_workspace_bytes();
static bool split_pays(int64_t groups, int sms);

// Built-in workspace of fbb_flash64_f16_static: room for the split form on a device of up to kStaticMaxSms SMs
// (11.5 MiB; zero-initialised when the module is loaded, as the flag words must be).
constexpr int kStaticMaxSms = 160;
constexpr size_t kStaticWsBytes = flag_region_bytes(kStaticMaxSms) + (size_t)kStaticMaxSms * kSlotFloats * sizeof(float) + side_region_bytes();
static __device__ __align__(256) unsigned char g_flash_static_ws[kStaticWsBytes];

#ifdef FBB_FLASH_TRACE
// Development aid: per-iteration clock stamps of one softmax warp (CTA 0, lane 0 of warps 4 and 8) and of the UMMA
// issuer, written to a global buffer set through fbb_flash_trace_buffer(). Not compiled into the shipped library.
__device__ unsigned* g_flash_trace = nullptr;
#define FBB_TRACE(slot, j, k)                                                                                         \
    do {                                                                                                              \
        if (trace_to != nullptr && (j) < 160) {                                                                          \
            unsigned c_;                                                                                                \
            asm volatile("mov.u32 %0, %%clock;" : "=r"(c_)::"memory");                                                  \
            trace_to[((slot) * 160 + (j)) * 8 + (k)] = c_;                                                               \
        }                                                                                                             \
    } while (0)
#else
#define FBB_TRACE(slot, j, k) do { } while (0)
#endif

struct FlashArgs {
    __half* o;
    int N, H;
    int64_t o_sb, o_sn, o_sh;
    float scale_log2;
    int groups_per_head;     // ceil(N / (128 * NQ))
    int nkb;                 // key blocks per group
    int rounds;              // whole groups every CTA takes round-robin before the tail region
    long long tail_units;    // (groups - rounds * gridDim.x) * nkb, dealt out in equal contiguous shares
    unsigned* ws_flags;      // [gridDim.x][16], all zero between launches; null when no group is ever split
    float* ws_data;          // [gridDim.x][kSlotFloats]
    int Nq;                  // query rows covered by tiles; rows [Nq, N) are left to flash64_side_rows_kernel
};

struct SideArgs {
    const __half *q, *k, *v;
    __half* o;
    int64_t q_sb, q_sn, q_sh, k_sb, k_sn, k_sh, v_sb, v_sn, v_sh, o_sb, o_sn, o_sh;
    int N, H, row0, rows, chunks, tasks;  // rows [row0, row0 + rows) of every (batch, head); tasks = B * H * rows * chunks
    float scale_log2;
    unsigned* count;         // [B * H * rows], all zero between launches
    float* part;             // [tasks][kSideValues]
};

// A CTA's work is a list of items (group w, key blocks [kb0, kb1)): first `rounds` whole groups taken round-robin
// (group = round * G + cta, so that the CTAs running at the same time share heads, i.e. K/V tiles in L2), then its share
// of the tail region, whose (group, key block) units are dealt out in contiguous runs of at least one group's length:
// at most three items (the end of a group another CTA began, a whole group, the beginning of one the next CTA ends).
// Thread 0 writes the tail items to shared memory once; every role walks the list by item index.
struct TailItems {
    int n;
    int w[3], kb0[3], kb1[3];
};

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Lane 0 polls a workspace flag until it is raised (bounded like every other wait); the result is warp-uniform.
__device__ __forceinline__ bool wait_slot_flag(const unsigned* flag, int lane, volatile int* abort_flag, unsigned detail) {
    bool ok = true;
    if (lane == 0 && ld_acquire_gpu(flag) == 0u) {
        const uint64_t t0 = globaltimer_ns();
        for (;;) {
            __nanosleep(200);
            if (ld_acquire_gpu(flag) != 0u) break;
            if (*abort_flag) { ok = false; break; }
            if (globaltimer_ns() - t0 > kWaitLimitNs) {
                report_error(DEV_TIMEOUT_OTHER, detail);
                *abort_flag = 1;
                __threadfence_block();
                ok = false;
                break;
            }
        }
    }
    ok = __all_sync(0xffffffffu, ok) != 0;
    __syncwarp();
    if (ok) (void)ld_acquire_gpu(flag);  // every lane orders its own reads of the slot after the flag
    return ok;
}

// One warp per (leftover query row, chunk of the keys). Scores: lane j takes key j of each 32-key step (fp32 dot product
// over the 64 dimensions); then the lanes switch to two output dimensions each and add p_j * v_j for the step's keys, p_j
// broadcast by shuffle: an online softmax in the scaled log2 domain of the tiled path (x = s * scale_log2). The partial
// (64 outputs, maximum, sum) goes to the workspace; the warp whose counter update completes a row merges its chunks and
// stores the row. No warp waits for another. 32 registers (16 CTAs of 128 threads would fit an SM): the point is to fit
// beside a resident CTA of the tiled kernel, which leaves 4096 registers and no shared memory to spare.
__global__ void __launch_bounds__(128, 16) flash64_side_rows_kernel(const SideArgs a) {
    grid_launch_dependents();
    const int lane = threadIdx.x & 31;
    const int task = (int)blockIdx.x * 4 + (int)(threadIdx.x >> 5);
    if (task < a.tasks) {
        const int chunk = task % a.chunks, rid = task / a.chunks;
        const int bh = rid / a.rows;
        const int row = a.row0 + (rid - bh * a.rows);
        const int b = bh / a.H, h = bh - b * a.H;
        const int per = (a.N + a.chunks - 1) / a.chunks;
        const int k0 = chunk * per, k1 = min(a.N, k0 + per);
        const uint4* qv = reinterpret_cast<const uint4*>(a.q + b * a.q_sb + (int64_t)row * a.q_sn + h * a.q_sh);
        const __half* kb = a.k + b * a.k_sb + h * a.k_sh;
        const __half* vb = a.v + b * a.v_sb + h * a.v_sh + 2 * lane;
        float m = -INFINITY, l = 0.f, o0 = 0.f, o1 = 0.f;
#pragma unroll 1
        for (int j0 = k0; j0 < k1; j0 += 32) {
            const int j = j0 + lane;
            float sc = -INFINITY;
            if (j < k1) {
                const uint4* kv = reinterpret_cast<const uint4*>(kb + (int64_t)j * a.k_sn);
                float acc = 0.f;
#pragma unroll 2
                for (int d = 0; d < 8; ++d) {
                    const uint4 kk = __ldcg(kv + d), qq = __ldg(qv + d);  // K and V stream past L1: each byte is used once
                    const __half2* kh = reinterpret_cast<const __half2*>(&kk);
                    const __half2* qh = reinterpret_cast<const __half2*>(&qq);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 kf = __half22float2(kh[e]), qf = __half22float2(qh[e]);
                        acc = fmaf(kf.x, qf.x, acc);
                        acc = fmaf(kf.y, qf.y, acc);
                    }
                }
                sc = acc * a.scale_log2;
            }
            float mx = sc;
#pragma unroll
            for (int sft = 16; sft > 0; sft >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, sft));
            const float mn = fmaxf(m, mx);       // finite: the step holds at least one key
            const float c = ex2_approx(m - mn);   // 0 on the first step (m = -inf)
            const float p = ex2_approx(sc - mn);  // 0 for lanes beyond the chunk
            float ps = p;
#pragma unroll
            for (int sft = 16; sft > 0; sft >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, sft);
            l = l * c + ps;
            o0 *= c;
            o1 *= c;
            m = mn;
            const int cnt = min(32, k1 - j0);
#pragma unroll 4
            for (int jj = 0; jj < cnt; ++jj) {
                const float pj = __shfl_sync(0xffffffffu, p, jj);
                const unsigned vw = __ldcg(reinterpret_cast<const unsigned*>(vb + (int64_t)(j0 + jj) * a.v_sn));
                const float2 vf = __half22float2(*reinterpret_cast<const __half2*>(&vw));
                o0 = fmaf(pj, vf.x, o0);
                o1 = fmaf(pj, vf.y, o1);
            }
        }
        float* part = a.part + (size_t)task * kSideValues;
        *reinterpret_cast<float2*>(part + 2 * lane) = make_float2(o0, o1);
        if (lane == 0) {
            part[64] = m;
            part[65] = l;
        }
        __threadfence();
        __syncwarp();
        unsigned prev = 0u;
        if (lane == 0) prev = atomicAdd(a.count + rid, 1u);
        prev = __shfl_sync(0xffffffffu, prev, 0);
        if (prev + 1u == (unsigned)a.chunks) {
            // this warp completed the row: merge the chunks (an empty chunk has m = -inf and contributes nothing)
            __threadfence();
            const float* parts = a.part + (size_t)rid * a.chunks * kSideValues;
            float M = -INFINITY;
            for (int ci = 0; ci < a.chunks; ++ci) M = fmaxf(M, __ldcg(parts + ci * kSideValues + 64));
            float L = 0.f, O0 = 0.f, O1 = 0.f;
            for (int ci = 0; ci < a.chunks; ++ci) {
                const float* pc = parts + ci * kSideValues;
                const float w = ex2_approx(__ldcg(pc + 64) - M);
                const float2 oc = __ldcg(reinterpret_cast<const float2*>(pc + 2 * lane));
                L = fmaf(__ldcg(pc + 65), w, L);
                O0 = fmaf(oc.x, w, O0);
                O1 = fmaf(oc.y, w, O1);
            }
            const float inv = 1.f / L;
            __half* dst = a.o + b * a.o_sb + (int64_t)row * a.o_sn + h * a.o_sh + 2 * lane;
            *reinterpret_cast<__half2*>(dst) = __floats2half2_rn(O0 * inv, O1 * inv);
            if (lane == 0) a.count[rid] = 0u;  // free for the next launch
        }
    }
    // The tiled launch before this one in the stream is still running. Nothing above depends on it (q, k and v were complete
    // before it started, and the rows written here are not its rows), but whoever waits for THIS grid must find that one
    // complete as well.
    grid_dependency_wait();
}

// ---- softmax pieces. A warp's 16 rows of a key block in the 16x256b fragment: registers 4k, 4k+1 = keys 8k + 2(lane%4), +1 of
// row A = lane/4; 4k+2, 4k+3 = the same keys of row B = lane/4 + 8.
template <int K>  // K groups of 8 keys (even)
__device__ __forceinline__ void max_frag(const uint32_t* v, float& mxA, float& mxB) {
    // two chains per row: half the latency before the caller's test
    float a0 = fmaxf(__uint_as_float(v[0]), __uint_as_float(v[1])), a1 = fmaxf(__uint_as_float(v[4]), __uint_as_float(v[5]));
    float b0 = fmaxf(__uint_as_float(v[2]), __uint_as_float(v[3])), b1 = fmaxf(__uint_as_float(v[6]), __uint_as_float(v[7]));
#pragma unroll
    for (int k = 2; k < K; k += 2) {
        a0 = fmax3(a0, __uint_as_float(v[4 * k]), __uint_as_float(v[4 * k + 1]));
        b0 = fmax3(b0, __uint_as_float(v[4 * k + 2]), __uint_as_float(v[4 * k + 3]));
        a1 = fmax3(a1, __uint_as_float(v[4 * k + 4]), __uint_as_float(v[4 * k + 5]));
        b1 = fmax3(b1, __uint_as_float(v[4 * k + 6]), __uint_as_float(v[4 * k + 7]));
    }
    mxA = fmaxf(a0, a1);
    mxB = fmaxf(b0, b1);
}
__device__ __forceinline__ void mask_frag(uint32_t* v, int key0, int n) {  // 64 keys
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (key0 + 8 * k >= n) v[4 * k] = v[4 * k + 2] = 0xff800000u;
        if (key0 + 8 * k + 1 >= n) v[4 * k + 1] = v[4 * k + 3] = 0xff800000u;
    }
}
// p = 2^(s*sl - m) in fp32, this thread's shares of the row sums, and P as fp16 pairs (the 16x128b fragment)
template <int K>
__device__ __forceinline__ void exp_frag(const uint32_t* v, float sl, float mA, float mB, float2& accA, float2& accB, uint32_t* pk) {
    const float2 sl2 = make_float2(sl, sl), nmA = make_float2(-mA, -mA), nmB = make_float2(-mB, -mB);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const float2 xA = ffma2(make_float2(__uint_as_float(v[4 * k]), __uint_as_float(v[4 * k + 1])), sl2, nmA);
        const float2 xB = ffma2(make_float2(__uint_as_float(v[4 * k + 2]), __uint_as_float(v[4 * k + 3])), sl2, nmB);
        const float2 pA = make_float2(ex2_approx(xA.x), ex2_approx(xA.y)), pB = make_float2(ex2_approx(xB.x), ex2_approx(xB.y));
        accA = fadd2(accA, pA);
        accB = fadd2(accB, pB);
        pk[2 * k] = pack_h2(pA.x, pA.y);
        pk[2 * k + 1] = pack_h2(pB.x, pB.y);
    }
}

template <int NQ>
__global__ void __launch_bounds__(128 + 256 * NQ, 1)
flash64_umma_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                    const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_o, const FlashArgs a) {
    using S = FlashSmem;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t base = smem_u32(smem_raw);
    uint8_t* gen = smem_raw;
    const uint32_t bar0 = base + S::kBarOff;
    auto q_full = [&](int i) { return bar0 + 8u * i; };
    auto q_empty = [&](int i) { return bar0 + 8u * (2 + i); };
    auto k_full = [&](int s) { return bar0 + 8u * (4 + s); };
    auto v_full = [&](int s) { return bar0 + 8u * (4 + kKVStages + s); };
    auto k_empty = [&](int s) { return bar0 + 8u * (4 + 2 * kKVStages + s); };
    auto v_empty = [&](int s) { return bar0 + 8u * (4 + 3 * kKVStages + s); };
    auto s_full = [&](int t) { return bar0 + 8u * (4 + 4 * kKVStages + t); };
    auto p_ready = [&](int t) { return bar0 + 8u * (4 + 4 * kKVStages + 2 + t); };
    auto pv_done = [&](int t) { return bar0 + 8u * (4 + 4 * kKVStages + 4 + t); };
    auto s_free = [&](int t) { return bar0 + 8u * (4 + 4 * kKVStages + 6 + t); };
    const uint32_t t1_go = bar0 + 8u * (4 + 4 * kKVStages + 8);  // completes once: tile 0's issuer has seen its group take the first block
    volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(gen + S::kBarOff + S::kNumBars * 8);
    volatile int* s_abort = reinterpret_cast<volatile int*>(gen + S::kBarOff + S::kNumBars * 8 + 4);
    TailItems* s_tail = reinterpret_cast<TailItems*>(gen + S::kTailOff);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int nkb = a.nkb;
#ifdef FBB_FLASH_TRACE
    if (threadIdx.x == 0 && g_flash_trace != nullptr) { unsigned* q_ = g_flash_trace + 20 * 160 * 8 + blockIdx.x * 4; q_[0] = (unsigned)globaltimer_ns(); unsigned c_; asm volatile("mov.u32 %0, %%clock;" : "=r"(c_)); q_[2] = c_; }
    unsigned* trace_to = (blockIdx.x == 0 && lane == 0) ? g_flash_trace : nullptr;
#endif

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(q_full(i), 1);
            mbar_init(q_empty(i), NQ);  // one commit per tile issuer, after the item's last Q K^T
        }
        for (int s = 0; s < kKVStages; ++s) {
            mbar_init(k_full(s), 1);
            mbar_init(v_full(s), 1);
            mbar_init(k_empty(s), NQ);
            mbar_init(v_empty(s), NQ);
        }
        for (int t = 0; t < 2; ++t) {
            mbar_init(s_full(t), 1);
            mbar_init(p_ready(t), 8);
            mbar_init(pv_done(t), 1);
            mbar_init(s_free(t), 8);
        }
        mbar_init(t1_go, 1);
        *s_abort = 0;
        // this CTA's share [tb, te) of the tail region's units, cut into items at group boundaries
        long long tb = 0, te = 0;
        if (a.tail_units > 0) {
            tb = (long long)(((unsigned long long)a.tail_units * blockIdx.x) / gridDim.x);
            te = (long long)(((unsigned long long)a.tail_units * (blockIdx.x + 1u)) / gridDim.x);
        }
        int n = 0;
        for (long long uu = tb; uu < te && n < 3; ++n) {  // (no iterations without a tail region)
            const int wt = (int)(uu / nkb);
            const int kb0 = (int)(uu - (long long)wt * nkb);
            const int kb1 = (int)((te - uu < (long long)(nkb - kb0)) ? kb0 + (te - uu) : nkb);
            s_tail->w[n] = a.rounds * (int)gridDim.x + wt;
            s_tail->kb0[n] = kb0;
            s_tail->kb1[n] = kb1;
            uu += kb1 - kb0;
        }
        s_tail->n = n;
        fence_barrier_init();
        tma_prefetch_desc(&tmap_q);
        tma_prefetch_desc(&tmap_k);
        tma_prefetch_desc(&tmap_v);
        tma_prefetch_desc(&tmap_o);
    }
    if (warp == 1) {
        __syncwarp();
        tmem_alloc<512>(smem_u32(const_cast<uint32_t*>(s_tmem)));
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *s_tmem;
    grid_dependency_wait();  // the set-up above may overlap the previous kernel's tail; its outputs are visible from here
    grid_launch_dependents();

    // Item list of this CTA (see TailItems): items [0, rounds) are whole groups, the rest come from the table.
    const int n_items = a.rounds + s_tail->n;
    auto item_at = [&](int it, int& w, int& kb0, int& kb1) {
        if (it < a.rounds) {
            w = it * (int)gridDim.x + (int)blockIdx.x;
            kb0 = 0;
            kb1 = nkb;
        } else {
            w = s_tail->w[it - a.rounds];
            kb0 = s_tail->kb0[it - a.rounds];
            kb1 = s_tail->kb1[it - a.rounds];
        }
    };

    // Warpgroup 0 holds the two single-thread roles (and two idle warps) and gives registers away; the softmax
    // warpgroups take them: a softmax thread keeps a whole 128-key row of S in registers.
    if (warp < 4) {
    if constexpr (NQ == 2) setmaxnreg_dec<kRegsCtl>();
    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
#pragma unroll 1
            for (int it = 0; it < n_items && ok; ++it) {
                int w, kb0, kb1;
                item_at(it, w, kb0, kb1);
                const int bh = w / a.groups_per_head;
                const int q0 = (w - bh * a.groups_per_head) * (FQ * NQ);
                const int b = bh / a.H, h = bh - b * a.H;
                // Q goes to one of two buffers, free when both tiles have left the item before the previous one. The tiles run about
                // a unit and a half apart and up to four units behind this loop: the next Q is there when a tile gets to it.
                // (One code path for all items: a separate load of the first Q put 1100 clocks between it and the first K, the
                // coordinates worked out twice and instruction fetches in between, where 400 do.)
                const int i = it & 1;
                if (!mbar_wait(q_empty(i), (((uint32_t)it >> 1) & 1u) ^ 1u, s_abort, DEV_TIMEOUT_SMEM_EMPTY, 32)) { ok = false; break; }
                mbar_arrive_expect_tx(q_full(i), NQ * kTileBytes);
                for (int t = 0; t < NQ; ++t) tma_load_4d(base + S::kQOff + (2 * i + t) * kTileBytes, &tmap_q, q_full(i), 0, h, q0 + t * FQ, b);
#pragma unroll 1
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!mbar_wait(k_empty(s), ph ^ 1u, s_abort, DEV_TIMEOUT_SMEM_EMPTY, s)) { ok = false; break; }
                    mbar_arrive_expect_tx(k_full(s), kTileBytes);
                    tma_load_4d(base + S::kKOff + s * kTileBytes, &tmap_k, k_full(s), 0, h, kb * FK, b);
                    if (!mbar_wait(v_empty(s), ph ^ 1u, s_abort, DEV_TIMEOUT_SMEM_EMPTY, 16 + s)) { ok = false; break; }
                    mbar_arrive_expect_tx(v_full(s), kTileBytes);
                    tma_load_4d(base + S::kVOff + s * kTileBytes, &tmap_v, v_full(s), 0, h, kb * FK, b);
                    if (++s == kKVStages) { s = 0; ph ^= 1u; }
                }
            }
            if (!ok) __nanosleep(20000);
        }
    } else if (warp - 1 < NQ) {
        // ------------------------------------------------------------------ UMMA issuers: warp 1 for tile 0, warp 2 for tile 1
        // Each tile has its own issuer so that neither tile ever waits for the other one's turn. The whole warp runs the
        // code and one elected lane issues each instruction (descriptors and addresses stay warp-uniform).
        // Per unit g (one key block of the current item) the order follows the softmax group's events:
        //   S_t free (the group has unit g in registers)  ->  S_t(g+1) = Q_t K^T of the next unit, which may belong to
        //                                                      the next item (other Q buffer), issued while the group works on g
        //   P_t(g) written                                 ->  O_t (+)= P_t(g) V
        const int t = warp - 1;
        const uint32_t idesc_qk = make_idesc_f16(FQ, FK, true, false, false);
        const uint32_t idesc_pv = make_idesc_f16(FQ, 64, true, false, true);
        constexpr uint64_t desc_hi = make_smem_desc_hi(16, 1024);
        const uint64_t qd0 = smem_desc(base + S::kQOff + t * kTileBytes, desc_hi);
        const uint64_t kd0 = smem_desc(base + S::kKOff, desc_hi);
        const uint64_t vd0 = smem_desc(base + S::kVOff, desc_hi);
        const uint32_t dS = tmem_base + t * kColTileS, dO = tmem_base + kColO + t * kColTileOP, aP = dO + kColP;
        auto all_ok = [&](bool mine) { return __all_sync(0xffffffffu, mine) != 0; };
        // S_t = Q_t K^T for one unit: Q buffer of item `it`, K in stage s; `last` = the item's last unit
        auto issue_qk = [&](int it, int s, bool last) {
            const uint64_t qd = qd0 + (uint64_t)((it & 1) * (2 * kTileBytes >> 4));
            const uint64_t kd = kd0 + (uint64_t)(s * (kTileBytes >> 4));
            umma_kblock_commit2_warp(dS, qd, kd, idesc_qk, s_full(t), k_empty(s));
            if (last) umma_commit_warp(q_empty(it & 1));  // this buffer may be loaded again
        };
        int it = 0, kb = 0, kb1 = 0;
        bool ok = n_items > 0;
        if (ok) {
            int w;
            item_at(0, w, kb, kb1);
        }
        if (ok) ok = all_ok(mbar_wait(q_full(0), 0, s_abort, DEV_TIMEOUT_TMA_FULL, 100));
        if (ok) ok = all_ok(mbar_wait(k_full(0), 0, s_abort, DEV_TIMEOUT_TMA_FULL, 0));
        // Tile 1 starts once tile 0's group has its first block in registers: the two groups then run slightly out of
        // step, so that one group's load / maximum / store phases overlap the other group's exponentials (measured at
        // N = 6145: 668 -> 695 TFLOP/s for ff, 600 -> 667 for hh; longer offsets change nothing).
        // (a barrier of its own that completes exactly once: waiting on s_free(0) by parity could be overtaken by tile 0's
        // second block and then never return)
        if (ok && t == 1 && (n_items > 1 || kb1 - kb > 2)) ok = all_ok(mbar_wait(t1_go, 0, s_abort, DEV_TIMEOUT_TMEM_EMPTY, 50));
        if (ok) {
            tc_fence_after();
            issue_qk(0, 0, kb + 1 == kb1);
        }
        int s = 0;
        uint32_t ph = 0, g = 0;
        bool first = true;  // this unit starts an item: O_t is overwritten, not accumulated
#pragma unroll 1
        while (ok) {
            const int sn = (s + 1 == kKVStages) ? 0 : s + 1;
            const uint32_t phn = (s + 1 == kKVStages) ? ph ^ 1u : ph;
            // the unit after this one
            int nit = it, nkb_ = kb + 1, nkb1 = kb1;
            bool nfirst = false, have_next = true;
            if (nkb_ == kb1) {
                nit = it + 1;
                nfirst = true;
                have_next = nit < n_items;
                if (have_next) {
                    int w;
                    item_at(nit, w, nkb_, nkb1);
                }
            }
            if (have_next) {
                if (nfirst && !all_ok(mbar_wait(q_full(nit & 1), ((uint32_t)nit >> 1) & 1u, s_abort, DEV_TIMEOUT_TMA_FULL, 101))) { ok = false; break; }
                if (!all_ok(mbar_wait(k_full(sn), phn, s_abort, DEV_TIMEOUT_TMA_FULL, sn))) { ok = false; break; }
                if (!all_ok(mbar_wait(s_free(t), g & 1u, s_abort, DEV_TIMEOUT_TMEM_EMPTY, t))) { ok = false; break; }
                if (NQ == 2 && t == 0 && g == 0 && lane == 0) mbar_arrive(t1_go);  // tile 1 may start (see the gate above)
                tc_fence_after();
                issue_qk(nit, sn, nkb_ + 1 == nkb1);
                FBB_TRACE(2 + t, g + 1, 3);
            }
            if (!all_ok(mbar_wait(v_full(s), ph, s_abort, DEV_TIMEOUT_TMA_FULL, 16 + s))) { ok = false; break; }
            if (!all_ok(mbar_wait(p_ready(t), g & 1u, s_abort, DEV_TIMEOUT_OTHER, 200 + t))) { ok = false; break; }
            tc_fence_after();
            FBB_TRACE(2 + t, g, 1);
            const uint64_t vd = vd0 + (uint64_t)(s * (kTileBytes >> 4));
            umma_ts8_commit2_warp(dO, aP, vd, idesc_pv, first ? 0u : 1u, pv_done(t), v_empty(s));
            FBB_TRACE(2 + t, g, 2);
            if (!have_next) {
                // The CTA gives its tensor memory and barriers up when all warps are past their loops. A tile that ends in an item
                // of padding has no softmax warp that waits for this last product, so the issuer does.
                (void)all_ok(mbar_wait(pv_done(t), g & 1u, s_abort, DEV_TIMEOUT_TMEM_FULL, 10 + t));
                break;
            }
            it = nit;
            kb = nkb_;
            kb1 = nkb1;
            first = nfirst;
            s = sn;
            ph = phn;
            ++g;
        }
    }
    } else {
        // ------------------------------------------------------------------ softmax groups
        // Eight warps per tile, 16 query rows per warp (tensor-memory lanes 32*(u%4) + 16*(u/4) ..+15), read with the
        // 16x256b shape: thread i holds, for rows i/4 and i/4 + 8, the key pairs 8k + 2*(i%4), +1 (k = 0..15) - the
        // m16n8 accumulator fragment. Row maxima and sums are finished with two shuffles inside the four threads that
        // share a row; P goes back with the 16x128b shape, whose layout is exactly those key pairs as fp16x2.
        // Four softmax warps per SM sub-partition keep the transcendental unit busy across one another's waits.
        if constexpr (NQ == 2) setmaxnreg_inc<kRegsSoftmax>();
        const int u = (warp - 4) & 7;
        const int t = (warp - 4) >> 3;
        const int lane_base = (u & 3) * 32 + (u >> 2) * 16;      // first tensor-memory lane (= row in the tile) of this warp
        const int cq = lane & 3;
        const uint32_t tS = tmem_base + ((uint32_t)lane_base << 16) + t * kColTileS;  // this warp's lanes of S_t
        const uint32_t tO = tmem_base + ((uint32_t)lane_base << 16) + kColO + t * kColTileOP;  // ... of O_t; P_t is kColP further
        const float sl = a.scale_log2;
        const float lazy = kLazyMax / sl;
        float tA = 0.f, tB = 0.f;  // raw scores beyond which the running maxima are raised
        float mA = -INFINITY, mB = -INFINITY, lA = 0.f, lB = 0.f;  // running maximum and (this thread's share of the) sum
        bool ok = true;
        uint32_t g = 0;  // units done: the phase of the per-tile barriers

        // An item's rows are written (or handed over, or merged) when its last P.V has completed, which is only waited for in
        // the next item's first unit, after that unit's exponentials: `done` is the item, lA .. mB its sums and maxima.
        int done = -1;
        float dlA = 0.f, dlB = 0.f, dmA = 0.f, dmB = 0.f;
        auto finish = [&](bool last) -> bool {
            int w, kb0, kb1;
            item_at(done, w, kb0, kb1);
            done = -1;
            float lA = dlA, lB = dlB, mA = dmA, mB = dmB;
            uint32_t o[32];
            tmem_ld_16x256b_x8(tO, o);
            tmem_wait_ld();
            const int wslot = t * 8 + u;
            if (kb0 > 0) {
                // Another CTA began this group: leave the partial result for it.
                float* dst = a.ws_data + ((size_t)blockIdx.x * kSlotWarps + wslot) * (kSlotValues * 32) + lane;
#pragma unroll
                for (int i = 0; i < 32; ++i) dst[i * 32] = __uint_as_float(o[i]);
                dst[32 * 32] = mA;
                dst[33 * 32] = mB;
                dst[34 * 32] = lA;
                dst[35 * 32] = lB;
                __threadfence();
                __syncwarp();
                if (lane == 0) st_release_gpu(a.ws_flags + (size_t)blockIdx.x * kSlotWarps + wslot, 1u);
                return true;
            }
            if (kb1 != nkb) {
                // The next CTA holds the rest of this group's keys (the first thing it did in its tail share).
                unsigned* flag = a.ws_flags + (size_t)(blockIdx.x + 1u) * kSlotWarps + wslot;
                if (!wait_slot_flag(flag, lane, s_abort, 300 + wslot)) return false;
                const float* src = a.ws_data + ((size_t)(blockIdx.x + 1u) * kSlotWarps + wslot) * (kSlotValues * 32) + lane;
                const float pmA = __ldcg(src + 32 * 32), pmB = __ldcg(src + 33 * 32);
                const float nA = fmaxf(mA, pmA), nB = fmaxf(mB, pmB);
                const float cA = ex2_approx(mA - nA), cB = ex2_approx(mB - nB);
                const float dA = ex2_approx(pmA - nA), dB = ex2_approx(pmB - nB);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    o[4 * k] = __float_as_uint(__uint_as_float(o[4 * k]) * cA + __ldcg(src + (4 * k) * 32) * dA);
                    o[4 * k + 1] = __float_as_uint(__uint_as_float(o[4 * k + 1]) * cA + __ldcg(src + (4 * k + 1) * 32) * dA);
                    o[4 * k + 2] = __float_as_uint(__uint_as_float(o[4 * k + 2]) * cB + __ldcg(src + (4 * k + 2) * 32) * dB);
                    o[4 * k + 3] = __float_as_uint(__uint_as_float(o[4 * k + 3]) * cB + __ldcg(src + (4 * k + 3) * 32) * dB);
                }
                lA = lA * cA + __ldcg(src + 34 * 32) * dA;
                lB = lB * cB + __ldcg(src + 35 * 32) * dB;
                __syncwarp();
                if (lane == 0) *flag = 0u;  // the slot is free for the next launch
            }
            // a row's sum is spread over the four threads that share it
            lA += __shfl_xor_sync(0xffffffffu, lA, 1);
            lB += __shfl_xor_sync(0xffffffffu, lB, 1);
            lA += __shfl_xor_sync(0xffffffffu, lA, 2);
            lB += __shfl_xor_sync(0xffffffffu, lB, 2);
            const float invA = 1.f / lA, invB = 1.f / lB;
            const int bh = w / a.groups_per_head;
            const int b = bh / a.H, h = bh - b * a.H;
            // The warp's 16 rows of 128 bytes leave through its own 2 KB of shared memory and one TMA store, which clips rows
            // at Nq: the fragment is four stmatrix of 8x8 tiles (lane i supplies the address of row i%8 of tile i/8), 16-byte
            // units swizzled as the tensor map's 128-byte mode expects them.
            if (lane == 0) bulk_wait_read_all();  // the previous item's rows have left
            __syncwarp();
            const uint32_t st = base + S::kOOff + (uint32_t)(t * 8 + u) * 2048u;
            const uint32_t strow = (uint32_t)(lane & 15);              // tiles 0, 1 of a call: rows 0-7, 8-15 of one column group; 2, 3: the next one
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
                const uint32_t unit = (uint32_t)(k + (lane >> 4)) ^ (strow & 7u);
                stmatrix_x4(st + strow * 128u + unit * 16u,
                            pack_h2(__uint_as_float(o[4 * k]) * invA, __uint_as_float(o[4 * k + 1]) * invA),
                            pack_h2(__uint_as_float(o[4 * k + 2]) * invB, __uint_as_float(o[4 * k + 3]) * invB),
                            pack_h2(__uint_as_float(o[4 * k + 4]) * invA, __uint_as_float(o[4 * k + 5]) * invA),
                            pack_h2(__uint_as_float(o[4 * k + 6]) * invB, __uint_as_float(o[4 * k + 7]) * invB));
            }
            const int row0 = (w - bh * a.groups_per_head) * (FQ * NQ) + t * FQ + lane_base;
            if (last) {
                // A CTA's last rows (in short launches its only ones) have nothing running behind them: plain 16-byte stores, a row's
                // by eight lanes, wait for no proxy fence and need not be drained before the CTA leaves. us with the TMA store / now:
                // 1 x 64 tokens x 6 heads 4.05 / 3.97, 1 x 223 x 16 5.74 / 5.50, 1 x 257 x 16 6.33 / 6.08; straight from the
                // registers, four bytes a thread, they are slower than the TMA store (1 x 256 x 6 5.9 / 6.4).
                __syncwarp();
                __half* dst = a.o + (int64_t)b * a.o_sb + (int64_t)h * a.o_sh + 8 * (lane & 7);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int r = 4 * i + (lane >> 3);
                    if (row0 + r < a.Nq)
                        *reinterpret_cast<uint4*>(dst + (int64_t)(row0 + r) * a.o_sn) =
                            ld_shared_16(st + (uint32_t)r * 128u + (uint32_t)(((lane & 7) ^ (r & 7)) * 16));
                }
                return true;
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                tma_store_4d(&tmap_o, st, 0, h, row0, b);
                bulk_commit();
            }
            return true;
        };

#pragma unroll 1
        for (int it = 0; ok && it < n_items; ++it) {
            int n;               // key blocks of this item still to do
            bool to_end;         // the item runs to the group's last key block
            bool warp_has_rows;  // a warp whose 16 rows all lie beyond N (padding of the last tile) only keeps the barriers moving
            {
                int w, kb0, kb1;
                item_at(it, w, kb0, kb1);
                n = kb1 - kb0;
                to_end = kb1 == nkb;
                warp_has_rows = (w % a.groups_per_head) * (FQ * NQ) + t * FQ + lane_base < a.Nq;
            }
            if (!warp_has_rows) {
#pragma unroll 1
                for (; n > 0; --n, ++g) {
                    // This warp only keeps the barriers moving. Its arrival for unit g must wait until the issuer has taken
                    // p_ready of unit g-1 (it commits pv_done right after issuing that unit's P.V): a tile whose warps are
                    // all padding would otherwise complete p_ready for g-1 and for g back to back, and the issuer, which
                    // waits by phase parity, would see the barrier back at the parity it started from and never wake up.
                    // (Working warps are held the same way by their own wait for pv_done before they overwrite P.)
                    // S_t is released at once (the next Q K^T needs no more from this warp; its arrival for unit g + 1 can
                    // only follow S_t(g+1), which the issuer computes after it has seen this unit's release).
                    if (!mbar_wait(s_full(t), g & 1u, s_abort, DEV_TIMEOUT_TMEM_FULL, t)) { ok = false; break; }
                    tc_fence_after();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(s_free(t));
                    if (g > 0 && !mbar_wait(pv_done(t), (g - 1u) & 1u, s_abort, DEV_TIMEOUT_OTHER, 210 + t)) { ok = false; break; }
                    tc_fence_after();
                    if (done >= 0 && !finish(false)) { ok = false; break; }
                    tc_fence_before();  // finish() read O_t, which the P.V that this arrival lets go overwrites
                    __syncwarp();
                    if (lane == 0) mbar_arrive(p_ready(t));
                }
                continue;
            }
            const bool ragged = to_end && (a.N & (FK - 1)) != 0;  // the group's last key block has keys beyond N
            const int key0 = (nkb - 1) * FK + 2 * cq;
            // That block has no key in its upper half. A ragged block goes through S once like any other, with its own copy of the
            // code (masks, half of the work where half is empty). Through the two passes of the blocks that raise a maximum, us
            // with / now: 1 x 223 tokens x 16 heads 6.26 / 5.74, 32 x 257 x 16 56.5 / 53.2, 4 x 1370 x 12 39.8 / 38.0.
            const bool half = a.N - (nkb - 1) * FK <= 64;
            {
                // ---- the item's first unit takes the running maxima
                if (!mbar_wait(s_full(t), g & 1u, s_abort, DEV_TIMEOUT_TMEM_FULL, t)) { ok = false; break; }
                tc_fence_after();
                uint32_t sc[64], pk[32];
                float mxA, mxB;
                // In halves in the one-tile kernel, whose launches are the short ones: the upper half of a ragged block may hold no
                // key. (The two-tile kernel has no registers to spare for this.)
                const bool lower = NQ == 1 && half && ragged && n == 1;
                if constexpr (NQ == 1) {
                    tmem_ld_16x256b_x8(tS, sc);
                    if (!lower) tmem_ld_16x256b_x8(tS + 64u, sc + 32);
                } else {
                    tmem_ld_16x256b_x16(tS, sc);
                }
                tmem_wait_ld();
                tmem_tie32(sc);
                tmem_tie32(sc + 32);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(s_free(t));
                if (ragged && n == 1) {
                    if (half || NQ == 2) mask_frag(sc, key0, a.N);
                    if (!half || NQ == 2) mask_frag(sc + 32, key0 + 64, a.N);
                }
                if constexpr (NQ == 1) {
                    max_frag<8>(sc, mxA, mxB);
                    if (!lower) {
                        float xA, xB;
                        max_frag<8>(sc + 32, xA, xB);
                        mxA = fmaxf(mxA, xA);
                        mxB = fmaxf(mxB, xB);
                    }
                } else {
                    max_frag<16>(sc, mxA, mxB);
                }
                mxA = fmaxf(mxA, __shfl_xor_sync(0xffffffffu, mxA, 1));
                mxB = fmaxf(mxB, __shfl_xor_sync(0xffffffffu, mxB, 1));
                mxA = fmaxf(mxA, __shfl_xor_sync(0xffffffffu, mxA, 2));
                mxB = fmaxf(mxB, __shfl_xor_sync(0xffffffffu, mxB, 2));
                mA = mxA * sl;
                mB = mxB * sl;
                tA = mxA + lazy;
                tB = mxB + lazy;
                float2 accA = make_float2(0.f, 0.f), accB = make_float2(0.f, 0.f);
                if constexpr (NQ == 1) {
                    exp_frag<8>(sc, sl, mA, mB, accA, accB, pk);
                    if (!lower) {
                        exp_frag<8>(sc + 32, sl, mA, mB, accA, accB, pk + 16);
                    } else {
#pragma unroll
                        for (int i = 16; i < 32; ++i) pk[i] = 0u;
                    }
                } else {
                    exp_frag<16>(sc, sl, mA, mB, accA, accB, pk);
                }
                if (g > 0) {
                    if (!mbar_wait(pv_done(t), (g - 1u) & 1u, s_abort, DEV_TIMEOUT_TMEM_FULL, 8 + t)) { ok = false; break; }
                    tc_fence_after();
                }
                tmem_st_16x128b_x16(tO + kColP, pk);
                if (done >= 0 && !finish(false)) { ok = false; break; }  // before this item's first P.V overwrites O_t
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_ready(t));
                lA = accA.x + accA.y;
                lB = accB.x + accB.y;
                --n;
                ++g;
            }
            int plain = n - (ragged ? 1 : 0);
            // One unit in a single pass over S, in registers: kDone, kRaise (a row's maximum must be raised first; nothing has been
            // released or written) or kFail (a wait ran out).
            enum { kDone, kRaise, kFail };
            auto unit = [&](auto masked) -> int {
                FBB_TRACE(4 + u + 8 * t, g, 0);
                if (!mbar_wait(s_full(t), g & 1u, s_abort, DEV_TIMEOUT_TMEM_FULL, t)) return kFail;
                tc_fence_after();
                FBB_TRACE(4 + u + 8 * t, g, 1);
                uint32_t sc[64], pk[32];
                float mxA, mxB;
                float2 accA = make_float2(0.f, 0.f), accB = make_float2(0.f, 0.f);
                if constexpr (decltype(masked)::value) {
                    if (half) {  // no key in the block's upper half
                        tmem_ld_16x256b_x8(tS, sc);
                        tmem_wait_ld();
                        tmem_tie32(sc);
                        mask_frag(sc, key0, a.N);
                        max_frag<8>(sc, mxA, mxB);
                        if (__any_sync(0xffffffffu, mxA > tA || mxB > tB)) return kRaise;
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(s_free(t));
                        exp_frag<8>(sc, sl, mA, mB, accA, accB, pk);
#pragma unroll
                        for (int i = 16; i < 32; ++i) pk[i] = 0u;
                    }
                }
                if (!decltype(masked)::value || !half) {
                    tmem_ld_16x256b_x16(tS, sc);
                    tmem_wait_ld();
                    tmem_tie32(sc);
                    tmem_tie32(sc + 32);
                    if constexpr (decltype(masked)::value) mask_frag(sc + 32, key0 + 64, a.N);
                    max_frag<16>(sc, mxA, mxB);
                    exp_frag<kEarly>(sc, sl, mA, mB, accA, accB, pk);
                    if (__any_sync(0xffffffffu, mxA > tA || mxB > tB)) return kRaise;
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(s_free(t));  // S_t is in registers: the next Q K^T may overwrite it
                    FBB_TRACE(4 + u + 8 * t, g, 2);
                    exp_frag<16 - kEarly>(sc + 4 * kEarly, sl, mA, mB, accA, accB, pk + 2 * kEarly);
                }
                // P_t is read by the previous unit's P.V until that product has completed: waiting here, not before the
                // exponentials, keeps the issue and run time of that product off the softmax warps' path
                if (!mbar_wait(pv_done(t), (g - 1u) & 1u, s_abort, DEV_TIMEOUT_TMEM_FULL, 8 + t)) return kFail;
                tc_fence_after();
                tmem_st_16x128b_x16(tO + kColP, pk);
                FBB_TRACE(4 + u + 8 * t, g, 3);
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_ready(t));
                FBB_TRACE(4 + u + 8 * t, g, 4);
                lA += accA.x + accA.y;
                lB += accB.x + accB.y;
                return kDone;
            };
#pragma unroll 1
            while (n > 0) {
                // ---- the units that are all alike, then the ragged one
                int got = kDone;
#pragma unroll 1
                for (; plain > 0; --plain, --n, ++g) {
                    got = unit(std::false_type());
                    if (got != kDone) break;
                }
                if (got == kDone && n > 0) {
                    got = unit(std::true_type());
                    if (got == kDone) {
                        --n;
                        ++g;
                    }
                }
                ok = got != kFail;
                if (!ok || n == 0) break;
                // ---- a block that exceeds a row's running maximum by more than 2^kLazyMax (raises them and rescales O and the sums),
                // half of it at a time from tensor memory
                const bool mask = plain == 0;
                float2 accA = make_float2(0.f, 0.f), accB = make_float2(0.f, 0.f);
                if (!mbar_wait(s_full(t), g & 1u, s_abort, DEV_TIMEOUT_TMEM_FULL, t)) { ok = false; break; }
                tc_fence_after();
                float mxA = -INFINITY, mxB = -INFINITY;
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    uint32_t v[32];
                    tmem_ld_16x256b_x8(tS + 64u * h, v);
                    tmem_wait_ld();
                    tmem_tie32(v);
                    if (mask) mask_frag(v, key0 + 64 * h, a.N);
                    float xA, xB;
                    max_frag<8>(v, xA, xB);
                    mxA = fmaxf(mxA, xA);
                    mxB = fmaxf(mxB, xB);
                }
                mxA = fmaxf(mxA, __shfl_xor_sync(0xffffffffu, mxA, 1));
                mxB = fmaxf(mxB, __shfl_xor_sync(0xffffffffu, mxB, 1));
                mxA = fmaxf(mxA, __shfl_xor_sync(0xffffffffu, mxA, 2));
                mxB = fmaxf(mxB, __shfl_xor_sync(0xffffffffu, mxB, 2));
                // P_t and O_t are in use by the previous unit's P.V until that product has completed
                if (!mbar_wait(pv_done(t), (g - 1u) & 1u, s_abort, DEV_TIMEOUT_TMEM_FULL, 8 + t)) { ok = false; break; }
                tc_fence_after();
                if (__any_sync(0xffffffffu, mxA > tA || mxB > tB)) {
                    const float nA = fmaxf(mA, mxA * sl), nB = fmaxf(mB, mxB * sl);
                    const float cA = ex2_approx(mA - nA), cB = ex2_approx(mB - nB);
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        uint32_t o[8];
                        tmem_ld_16x256b_x2(tO + 16u * c, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            o[4 * k] = __float_as_uint(__uint_as_float(o[4 * k]) * cA);
                            o[4 * k + 1] = __float_as_uint(__uint_as_float(o[4 * k + 1]) * cA);
                            o[4 * k + 2] = __float_as_uint(__uint_as_float(o[4 * k + 2]) * cB);
                            o[4 * k + 3] = __float_as_uint(__uint_as_float(o[4 * k + 3]) * cB);
                        }
                        tmem_st_16x256b_x2(tO + 16u * c, o);
                    }
                    lA *= cA;
                    lB *= cB;
                    mA = nA;
                    mB = nB;
                    tA = fmaxf(tA, mxA + lazy);
                    tB = fmaxf(tB, mxB + lazy);
                }
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    uint32_t v[32], pk[16];
                    if (mask && (nkb - 1) * FK + 64 * h >= a.N) {  // no key in this half
#pragma unroll
                        for (int i = 0; i < 16; ++i) pk[i] = 0u;
                    } else {
                        tmem_ld_16x256b_x8(tS + 64u * h, v);
                        tmem_wait_ld();
                        tmem_tie32(v);
                        if (mask) mask_frag(v, key0 + 64 * h, a.N);
                        exp_frag<8>(v, sl, mA, mB, accA, accB, pk);
                    }
                    tmem_st_16x128b_x8(tO + kColP + 32u * h, pk);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(s_free(t));
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_ready(t));
                lA += accA.x + accA.y;
                lB += accB.x + accB.y;
                --n;
                --plain;
                ++g;
            }
            if (!ok) continue;
            done = it;
            dlA = lA;
            dlB = lB;
            dmA = mA;
            dmB = mB;
        }
        if (ok && done >= 0 && mbar_wait(pv_done(t), (g - 1u) & 1u, s_abort, DEV_TIMEOUT_TMEM_FULL, 8 + t)) {
            tc_fence_after();
            finish(true);
        }
        if (lane == 0) bulk_wait_all();
    }

    tc_fence_before();
    __syncthreads();
#ifdef FBB_FLASH_TRACE
    if (threadIdx.x == 0 && g_flash_trace != nullptr) { unsigned* q_ = g_flash_trace + 20 * 160 * 8 + blockIdx.x * 4; q_[1] = (unsigned)globaltimer_ns(); unsigned c_; asm volatile("mov.u32 %0, %%clock;" : "=r"(c_)); q_[3] = c_; }
#endif
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc<512>(tmem_base);
    }
}

template <int NQ>
static int launch_flash_variant(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to, FlashArgs a, int B, void* ws,
                                int64_t ws_bytes, cudaStream_t stream) {
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    auto kern = flash64_umma_kernel<NQ>;
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FlashSmem::kDynamic);
        if (e != cudaSuccess) return fail((int)e, "cudaFuncSetAttribute(flash64_umma_kernel): %s", cudaGetErrorString(e));
        configured[dev] = true;
    }
    a.groups_per_head = (a.Nq + FQ * NQ - 1) / (FQ * NQ);
    a.nkb = (a.N + FK - 1) / FK;
    const int64_t groups = (int64_t)a.groups_per_head * B * a.H;
    if (groups > 0x7FFFFFFFll) return fail(FBB_ERR_SHAPE, "flash64: too many query tiles (%lld)", (long long)groups);
    a.ws_flags = nullptr;
    a.ws_data = nullptr;
    // One CTA per tile group, unless the groups do not fill the SMs evenly and the caller lent a workspace: then one
    // persistent CTA per SM takes whole groups round-robin for all but the last full wave, and an equal share of the
    // (group, key block) units of what is left (between one and two waves' worth, so every share is at least one group
    // long and a group is split over at most two CTAs, which merge through the workspace).
    const int sms = num_sms();
    int64_t ctas = groups;
    a.rounds = 1;
    a.tail_units = 0;
    const bool plain_only = getenv("FBB_FLASH_NO_SPLIT") != nullptr;  // tuning aid: always one CTA per group
    if (groups > sms && groups % sms == 0 && !plain_only) {
        ctas = sms;
        a.rounds = (int)(groups / sms);
    } else if (ws != nullptr && !plain_only && split_pays(groups, sms)) {
        if (ws_bytes < flash64_workspace_bytes()) return fail(FBB_ERR_SHAPE, "flash64: workspace of %lld bytes, %lld needed", (long long)ws_bytes, (long long)flash64_workspace_bytes());
        ctas = sms;
        a.rounds = (int)(groups / sms) - 1;
        a.tail_units = (groups - (int64_t)a.rounds * sms) * a.nkb;
        a.ws_flags = reinterpret_cast<unsigned*>(ws);
        a.ws_data = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(ws) + flag_region_bytes(sms));
    }
    if ((int64_t)a.rounds * a.nkb + 2 * (int64_t)a.nkb * 2 > 0x7FFFFFFFll) return fail(FBB_ERR_SHAPE, "flash64: too many key blocks per CTA");
    cudaError_t e = launch_pdl(kern, dim3((unsigned)ctas), dim3(128 + 256 * NQ), FlashSmem::kDynamic, stream, tq, tk, tv, to, a);
    if (e != cudaSuccess) return fail((int)e, "flash64_umma_kernel launch: %s", cudaGetErrorString(e));
    return FBB_OK;
}

#ifdef FBB_FLASH_TRACE
extern "C" int fbb_flash_trace_buffer(void* buf) {
    unsigned* p = reinterpret_cast<unsigned*>(buf);
    return (int)cudaMemcpyToSymbol(g_flash_trace, &p, sizeof(p));
}
#endif

// Whether the persistent split form is worth it: the groups do not fill the SMs evenly and the partly filled last wave
// wastes at least 9 % of the whole-wave schedule. Measured, about a third of that waste is recovered (long-lived CTAs
// lose some speed to the two tiles drifting into step), so smaller savings do not pay: 8 % -> -0.6 %, 10 % -> +2.5 %,
// 31 % -> +11 % on whole-model time.
static bool split_pays(int64_t groups, int sms) {
    if (groups <= sms || groups % sms == 0) return false;
    const int64_t whole = (groups + sms - 1) / sms;
    const char* f = getenv("FBB_FLASH_SPLIT_WASTE");  // tuning aid: the least wasted share of the whole-wave schedule that splits
    const double least = f != nullptr ? atof(f) : 0.09;
    return (double)(whole * sms - groups) >= least * (double)(whole * sms);
}

// Two query tiles per CTA once that still gives every SM a CTA; small inputs take one tile per CTA (the small-token path).
static bool two_tiles_per_cta(int B, int N, int H) { return (int64_t)((N + 2 * FQ - 1) / (2 * FQ)) * B * H >= num_sms(); }

int64_t flash64_workspace_bytes() {
    return (int64_t)(flag_region_bytes(num_sms()) + (size_t)num_sms() * kSlotFloats * sizeof(float) + side_region_bytes());
}

// Query rows beyond the last full two-tile group that the side launch takes instead of a tile group of their own
// (0: none): a few rows (cls token, registers), few enough in all and a sequence long enough for the side launch to
// hide behind the tiled one, and the rest still worth two tiles per CTA. FBB_FLASH_NO_SIDE switches it off (tuning and test aid).
static int side_rows_for(int B, int N, int H) {
    const int r = N % (2 * FQ);
    if (r < 1 || r > kSideMaxRows || N <= 2 * FQ || getenv("FBB_FLASH_NO_SIDE") != nullptr || getenv("FBB_FLASH_NO_SPLIT") != nullptr) return 0;
    const int sms = num_sms();
    // The side launch gets four warps per SM (what fits beside the tiled kernel) and each of them is bound by the latency
    // of its loads, so it only hides behind the tiled launch when that is long and the rows are few. Measured on B200
    // (side / tiled only, us): N = 6145, 16 rows 194 / 200; 4097, 12 rows 76.1 / 77.5; 3073, 16 rows 61.5 / 62.6; 2561
    // 47.8 / 47.4; but 6149 (5 rows per head: 80 rows) 308 / 200 and 1281 with 64 rows 63.6 / 55.5.
    if ((int64_t)B * H * r > sms / 8 || N < 3072 || !two_tiles_per_cta(B, N - r, H)) return 0;
    // Only where the tiled launch stays in a persistent form (split, or whole groups in equal rounds). One CTA per group
    // measured 3 % slower per group than the persistent forms at N = 16385, where dropping the 65th group per head would
    // have moved the launch from the split form (1040 groups) to one CTA per group (1024): 1453 against 1430 us.
    const int64_t groups = (int64_t)((N - r) / (2 * FQ)) * B * H;
    if (!(split_pays(groups, sms) || (groups > sms && groups % sms == 0))) return 0;
    return r;
}

int64_t flash64_workspace_bytes_for(int B, int N, int H) {
    if (B <= 0 || N <= 0 || H <= 0 || getenv("FBB_FLASH_NO_SPLIT") != nullptr) return 0;
    const int r = side_rows_for(B, N, H);
    const int nq = two_tiles_per_cta(B, N - r, H) ? 2 : 1;
    const int64_t groups = (int64_t)((N - r + FQ * nq - 1) / (FQ * nq)) * B * H;
    const int sms = num_sms();
    return (r > 0 || split_pays(groups, sms)) ? flash64_workspace_bytes() : 0;
}

int flash64_launches(int B, int N, int H, bool has_workspace) { return (B > 0 && N > 0 && H > 0 && has_workspace && side_rows_for(B, N, H) > 0) ? 2 : 1; }

// The leftover rows [N - rows, N): enqueued right after the tiled launch (see kSideMaxRows).
static int launch_side_rows(const FlashArgs& f, const void* q, const void* k, const void* v, int B, const int64_t* qs, const int64_t* ks,
                            const int64_t* vs, int rows, void* ws, cudaStream_t stream) {
    SideArgs a = {};
    a.q = reinterpret_cast<const __half*>(q);
    a.k = reinterpret_cast<const __half*>(k);
    a.v = reinterpret_cast<const __half*>(v);
    a.o = f.o;
    a.q_sb = qs[0]; a.q_sn = qs[1]; a.q_sh = qs[2];
    a.k_sb = ks[0]; a.k_sn = ks[1]; a.k_sh = ks[2];
    a.v_sb = vs[0]; a.v_sn = vs[1]; a.v_sh = vs[2];
    a.o_sb = f.o_sb; a.o_sn = f.o_sn; a.o_sh = f.o_sh;
    a.N = f.N;
    a.H = f.H;
    a.row0 = f.N - rows;
    a.rows = rows;
    a.scale_log2 = f.scale_log2;
    const int sms = num_sms();
    const int64_t nrows = (int64_t)B * f.H * rows;  // <= sms
    int64_t chunks = (4 * (int64_t)sms) / nrows;     // about four warps per SM
    const int64_t most = (f.N + 63) / 64;            // at least two 32-key steps per chunk
    chunks = chunks > most ? most : chunks;
    chunks = chunks > kSideMaxChunks ? kSideMaxChunks : (chunks < 1 ? 1 : chunks);
    while (nrows * chunks > kSideMaxTasks) --chunks;
    a.chunks = (int)chunks;
    a.tasks = (int)(nrows * chunks);
    uint8_t* w8 = reinterpret_cast<uint8_t*>(ws);
    a.count = reinterpret_cast<unsigned*>(w8 + (size_t)sms * kFlagBytesPerCta);
    a.part = reinterpret_cast<float*>(w8 + flag_region_bytes(sms) + (size_t)sms * kSlotFloats * sizeof(float));
    cudaError_t e = launch_pdl(flash64_side_rows_kernel, dim3((unsigned)((a.tasks + 3) / 4)), dim3(128), 0, stream, a);
    if (e != cudaSuccess) return fail((int)e, "flash64_side_rows_kernel launch: %s", cudaGetErrorString(e));
    return FBB_OK;
}

// Address and size of the built-in workspace on the current device; the address is looked up once per device. Enqueues
// the clearing of its flag words on `stream` (calls share the array, and a launch that gave up a wait may have left some
// raised). No memory is allocated.
int flash64_static_workspace(void** ptr, int64_t* bytes, cudaStream_t stream) {
    static void* addr[64] = {};
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail((int)e, "cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= 64) return fail(FBB_ERR_SHAPE, "flash64 static workspace: device ordinal %d not supported", dev);
    if (addr[dev] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_flash_static_ws);
        if (e != cudaSuccess || p == nullptr) return fail(e != cudaSuccess ? (int)e : FBB_ERR_DRIVER, "cudaGetSymbolAddress(static workspace): %s", cudaGetErrorString(e));
        addr[dev] = p;
    }
    if (flash64_workspace_bytes() > (int64_t)kStaticWsBytes)
        return fail(FBB_ERR_SHAPE, "flash64 static workspace holds %lld bytes (%d SMs), this device needs %lld", (long long)kStaticWsBytes,
                    kStaticMaxSms, (long long)flash64_workspace_bytes());
    e = cudaMemsetAsync(addr[dev], 0, flag_region_bytes(num_sms()), stream);
    if (e != cudaSuccess) return fail((int)e, "cudaMemsetAsync(static workspace flags): %s", cudaGetErrorString(e));
    *ptr = addr[dev];
    *bytes = (int64_t)kStaticWsBytes;
    return FBB_OK;
}

int launch_flash64(const void* q, const void* k, const void* v, void* o, int B, int N, int H, const int64_t* qs,
                   const int64_t* ks, const int64_t* vs, const int64_t* os, float scale, int variant, void* ws, int64_t ws_bytes,
                   cudaStream_t stream) {
    CUtensorMap tq, tk, tv;
    const uint64_t dims[4] = {64, (uint64_t)H, (uint64_t)N, (uint64_t)B};
    const uint32_t box[4] = {64, 1, 128, 1};
    const void* ptrs[3] = {q, k, v};
    const int64_t* strides[3] = {qs, ks, vs};
    CUtensorMap* maps[3] = {&tq, &tk, &tv};
    for (int i = 0; i < 3; ++i) {
        // innermost first: d (contiguous), head, token, batch; a size-1 dimension may carry any stride, use a valid one
        int64_t st[4] = {1, strides[i][2], strides[i][1], strides[i][0]};
        if (H == 1 && st[1] == 0) st[1] = 64;
        if (B == 1 && st[3] == 0) st[3] = st[2] * (int64_t)N;
        int rc = make_tmap_f16(maps[i], ptrs[i], 4, dims, st, box);
        if (rc != FBB_OK) return rc;
    }
    FlashArgs a = {};
    a.o = reinterpret_cast<__half*>(o);
    a.N = N;
    a.H = H;
    a.o_sb = os[0];
    a.o_sn = os[1];
    a.o_sh = os[2];
    a.scale_log2 = scale * 1.4426950408889634f;
    (void)variant;  // ff, fh and hh run the same kernel on this part (see the note on variants at the top of the file)
    // leftover rows go to the side launch only when the caller lent a workspace (their partial results live there)
    const int side = ws != nullptr ? side_rows_for(B, N, H) : 0;
    if (side > 0 && ws_bytes < flash64_workspace_bytes())
        return fail(FBB_ERR_SHAPE, "flash64: workspace of %lld bytes, %lld needed", (long long)ws_bytes, (long long)flash64_workspace_bytes());
    a.Nq = N - side;
    CUtensorMap to;  // 16 rows of one head at a time; rows from Nq on are not this kernel's
    {
        const uint64_t odims[4] = {64, (uint64_t)H, (uint64_t)a.Nq, (uint64_t)B};
        const uint32_t obox[4] = {64, 1, 16, 1};
        int64_t st[4] = {1, os[2], os[1], os[0]};
        if (H == 1 && st[1] == 0) st[1] = 64;
        if (B == 1 && st[3] == 0) st[3] = st[2] * (int64_t)N;
        const int rc = make_tmap_f16(&to, o, 4, odims, st, obox);
        if (rc != FBB_OK) return rc;
    }
    int rc;
    if (two_tiles_per_cta(B, a.Nq, H)) rc = launch_flash_variant<2>(tq, tk, tv, to, a, B, ws, ws_bytes, stream);
    else rc = launch_flash_variant<1>(tq, tk, tv, to, a, B, ws, ws_bytes, stream);  // (never with side rows: see side_rows_for)
    if (rc != FBB_OK || side == 0) return rc;
    return launch_side_rows(a, q, k, v, B, qs, ks, vs, side, ws, stream);
}

}  // namespace fbb
