// The streamed shift-and-stack: the stacking pass of stack.cu for motions that
// pack into blocks of five sharing their column in every frame and at most one row
// apart (velocity lattices of about a quarter pixel a motion), for up to 255 frames.
//
// One CTA owns a 32 x 16 output tile and takes the motions in groups of sixteen
// blocks, one block a warp. A warp holds its block's 5 x 16 sums a lane (one
// column, sixteen rows) in registers while the frames stream past in ascending
// order: the group's windows of a run of frames are copied by TMA (zero fill
// outside the frame) into one of three buffers of shared memory, and run after run,
// group after group and tile after tile follow without a pause. A lane loads its
// column of a frame's window once, 17 rows, and adds it to all five motions.
//
// What bounds it: issue and the FMA pipe, with four warps a scheduler. A paired add
// (add.rn.f32x2) takes the pipe for two cycles, as two single adds do, so 128 adds a
// cycle and SM need every other cycle's issue slot and leave the rest to loads,
// descriptors and branches. A block and frame takes 105 instructions with its share of
// the maxima, 40 of them the adds (120 frames of 1024 x 512: issue active 57 % of the
// cycles, the FMA pipe 50 %; stalls on fixed latencies 2.0 an issue, on loads and the
// copies 1.5, on the pipe 0.7). Five motions a load and not four, which have 32 adds
// beside the same loads; more need more than the 128 registers that sixteen warps have;
// fewer warps leave the load latency open (blocks of eight on eight warps 9 T adds/s).
// Measured: 15.4 T adds/s at 120 frames of 2048 x 1024 (462 ms; 32 x 8 and 32 x 4 tiles
// with resident windows 1080), 14.3 T at 40 frames of 2048^2 (46.4 ms; resident windows
// 42.4).
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <cstddef>
#include <stdexcept>
#include <string>
#include <vector>

#include "ft_internal.h"
#include "stack_device.cuh"
#include "stack_stream.h"

namespace ftb {

namespace {

constexpr int kBuffers = 3;                             // runs of frames in shared memory
constexpr int kMostFrames = 32;                         // frames of a run at most (a lane copies one)
constexpr int kThreads = 32 * kStreamWarps;

struct StreamArgs {
    int w, h, n, min_count;
    int g0, g1;            // groups of this launch
    int splits;            // work items a tile (its groups cut into as many runs)
    int tiles_x;
    int rows, frames;      // a window's rows, a run's frames
    long long item0;       // its first work item in the batch
    const StreamGroup* groups;
    const StreamWin* wins;
    const uint32_t* desc;
    const int* slot_motion;
    const float* inv_sqrt;
    unsigned long long* keys;  // the maps' running maxima (null: one item a tile writes the maps itself)
    float* max_snr;
    int* best_v;
};

// A run of frames in a buffer (p < 0: the end).
struct Run {
    int p, x0, y0, g, gb, i0, frames, n;
    int window, inside;  // floats of a window; whether the tile lies inside the frame
    float inv_n;
};

struct alignas(128) Shared {
    uint32_t desc[kBuffers][(kMostFrames + 1) * kStreamWarps];  // a frame more than is read
    int motion[kBuffers][kStreamWarps * kStreamBlock];
    StreamGroup group[kBuffers];
    unsigned long long keys[32 * kStreamRows];
    uint64_t full[kBuffers];
    uint64_t tile_bar;       // every warp, at a tile's end
    int left[kBuffers];      // warps that are past a buffer's run
    Run run[kBuffers];
    Run next;                // the next run to copy
    int abort;               // a wait ran out: every warp gives up
};

static_assert(offsetof(Shared, motion) % 16 == 0 && offsetof(Shared, group) % 16 == 0 && sizeof(StreamGroup) == 16 &&
                  kStreamWarps * kStreamBlock * 4 % 16 == 0,
              "16-byte copies into shared memory");

// Bounded wait of a whole warp that also ends when another warp of the CTA gave
// up; the same answer in every lane.
__device__ __forceinline__ bool ring_wait(Shared& sh, uint64_t* bar, uint32_t parity, int* err, long long limit) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    const long long t0 = clock64();
    while (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) {
        const bool late = clock64() - t0 > limit;
        if (late) {
            *reinterpret_cast<volatile int*>(&sh.abort) = 1;
            atomicExch(err, 1);
        }
        if (__any_sync(0xffffffffu, late || *reinterpret_cast<volatile int*>(&sh.abort))) return false;
    }
    return true;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}

__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

__device__ __forceinline__ uint32_t order_bits(float s) {
    const uint32_t b = __float_as_uint(__fadd_rn(s, 0.0f));  // as snr_key
    return b ^ (static_cast<uint32_t>(static_cast<int>(b) >> 31) | 0x80000000u);
}

// ---- the adds of one frame for a block
//
// A pair of sums is one 64-bit register pair, rows (q, q + 8) of a motion; A[r]
// holds the window's rows (r, r + 8), so a motion on the upper row adds A[q + 1] to
// its pair q (add.rn.f32x2: two independent round-to-nearest adds). Two lines of
// code add the motions from the lower (L) and the upper row (U); a step changes
// lines before its motion. Written out because the compiler's switch over the
// patterns cost more: a tree of compares, and moves for the operands of adds that
// it shared between cases.
#define FTB_ADD(S, A) "add.rn.f32x2 %" #S ", %" #S ", %" #A ";\n\t"
// motion k's eight pairs from the lower row (FTB_Mk_0) or the upper (FTB_Mk_1): sums %8k .., A %40 ..
#define FTB_M0_0 FTB_ADD(0, 40) FTB_ADD(1, 41) FTB_ADD(2, 42) FTB_ADD(3, 43) FTB_ADD(4, 44) FTB_ADD(5, 45) \
    FTB_ADD(6, 46) FTB_ADD(7, 47)
#define FTB_M0_1 FTB_ADD(0, 41) FTB_ADD(1, 42) FTB_ADD(2, 43) FTB_ADD(3, 44) FTB_ADD(4, 45) FTB_ADD(5, 46) \
    FTB_ADD(6, 47) FTB_ADD(7, 48)
#define FTB_M1_0 FTB_ADD(8, 40) FTB_ADD(9, 41) FTB_ADD(10, 42) FTB_ADD(11, 43) FTB_ADD(12, 44) FTB_ADD(13, 45) \
    FTB_ADD(14, 46) FTB_ADD(15, 47)
#define FTB_M1_1 FTB_ADD(8, 41) FTB_ADD(9, 42) FTB_ADD(10, 43) FTB_ADD(11, 44) FTB_ADD(12, 45) FTB_ADD(13, 46) \
    FTB_ADD(14, 47) FTB_ADD(15, 48)
#define FTB_M2_0 FTB_ADD(16, 40) FTB_ADD(17, 41) FTB_ADD(18, 42) FTB_ADD(19, 43) FTB_ADD(20, 44) FTB_ADD(21, 45) \
    FTB_ADD(22, 46) FTB_ADD(23, 47)
#define FTB_M2_1 FTB_ADD(16, 41) FTB_ADD(17, 42) FTB_ADD(18, 43) FTB_ADD(19, 44) FTB_ADD(20, 45) FTB_ADD(21, 46) \
    FTB_ADD(22, 47) FTB_ADD(23, 48)
#define FTB_M3_0 FTB_ADD(24, 40) FTB_ADD(25, 41) FTB_ADD(26, 42) FTB_ADD(27, 43) FTB_ADD(28, 44) FTB_ADD(29, 45) \
    FTB_ADD(30, 46) FTB_ADD(31, 47)
#define FTB_M3_1 FTB_ADD(24, 41) FTB_ADD(25, 42) FTB_ADD(26, 43) FTB_ADD(27, 44) FTB_ADD(28, 45) FTB_ADD(29, 46) \
    FTB_ADD(30, 47) FTB_ADD(31, 48)
#define FTB_M4_0 FTB_ADD(32, 40) FTB_ADD(33, 41) FTB_ADD(34, 42) FTB_ADD(35, 43) FTB_ADD(36, 44) FTB_ADD(37, 45) \
    FTB_ADD(38, 46) FTB_ADD(39, 47)
#define FTB_M4_1 FTB_ADD(32, 41) FTB_ADD(33, 42) FTB_ADD(34, 43) FTB_ADD(35, 44) FTB_ADD(36, 45) FTB_ADD(37, 46) \
    FTB_ADD(38, 47) FTB_ADD(39, 48)

__device__ __forceinline__ void block_frame(unsigned long long (&s)[40], const unsigned long long (&A)[9], uint32_t d) {
    asm volatile(
        "{\n\t"
        ".reg .pred p1, p2, p3, p4, u;\n\t"
        ".reg .u32 t;\n\t"
        "and.b32 t, %49, 131072;\n\tsetp.ne.u32 p1, t, 0;\n\t"
        "and.b32 t, %49, 262144;\n\tsetp.ne.u32 p2, t, 0;\n\t"
        "and.b32 t, %49, 524288;\n\tsetp.ne.u32 p3, t, 0;\n\t"
        "and.b32 t, %49, 1048576;\n\tsetp.ne.u32 p4, t, 0;\n\t"
        "and.b32 t, %49, 16777216;\n\tsetp.ne.u32 u, t, 0;\n\t"
        "@u bra.uni U0;\n\t"
        "L0:\n\t" FTB_M0_0 "@p1 bra.uni U1;\n\t"
        "L1:\n\t" FTB_M1_0 "@p2 bra.uni U2;\n\t"
        "L2:\n\t" FTB_M2_0 "@p3 bra.uni U3;\n\t"
        "L3:\n\t" FTB_M3_0 "@p4 bra.uni U4;\n\t"
        "L4:\n\t" FTB_M4_0 "bra.uni E;\n\t"
        "U0:\n\t" FTB_M0_1 "@p1 bra.uni L1;\n\t"
        "U1:\n\t" FTB_M1_1 "@p2 bra.uni L2;\n\t"
        "U2:\n\t" FTB_M2_1 "@p3 bra.uni L3;\n\t"
        "U3:\n\t" FTB_M3_1 "@p4 bra.uni L4;\n\t"
        "U4:\n\t" FTB_M4_1
        "E:\n\t}"
        : "+l"(s[0]), "+l"(s[1]), "+l"(s[2]), "+l"(s[3]), "+l"(s[4]), "+l"(s[5]), "+l"(s[6]), "+l"(s[7]),
          "+l"(s[8]), "+l"(s[9]), "+l"(s[10]), "+l"(s[11]), "+l"(s[12]), "+l"(s[13]), "+l"(s[14]), "+l"(s[15]),
          "+l"(s[16]), "+l"(s[17]), "+l"(s[18]), "+l"(s[19]), "+l"(s[20]), "+l"(s[21]), "+l"(s[22]), "+l"(s[23]),
          "+l"(s[24]), "+l"(s[25]), "+l"(s[26]), "+l"(s[27]), "+l"(s[28]), "+l"(s[29]), "+l"(s[30]), "+l"(s[31]),
          "+l"(s[32]), "+l"(s[33]), "+l"(s[34]), "+l"(s[35]), "+l"(s[36]), "+l"(s[37]), "+l"(s[38]), "+l"(s[39])
        : "l"(A[0]), "l"(A[1]), "l"(A[2]), "l"(A[3]), "l"(A[4]), "l"(A[5]), "l"(A[6]), "l"(A[7]), "l"(A[8]),
          "r"(d));
}

// The next run into buffer b, which every warp is past: its windows and
// descriptors, or the end. By one warp at a time.
__device__ __forceinline__ void copy_run(Shared& sh, unsigned char* windows, const StreamArgs* passes,
                                         const CUtensorMap* maps, int npasses, long long items, unsigned long long* queue,
                                         int b, unsigned extra_tx, int lane) {
    Run r = sh.next;
    if (r.g >= r.gb && r.p >= -1) {  // a new item (p = -1 before the first, -2 after the last)
        unsigned long long q = 0;
        if (lane == 0) q = atomicAdd(queue, 1ull);
        const long long item = static_cast<long long>(__shfl_sync(0xffffffffu, q, 0));
        r.p = -2;
        if (item < items) {
            r.p = 0;
            while (r.p + 1 < npasses && passes[r.p + 1].item0 <= item) ++r.p;
            const StreamArgs& a = passes[r.p];
            const long long e = item - a.item0;
            const int split = static_cast<int>(e % a.splits), tile = static_cast<int>(e / a.splits);
            r.x0 = (tile % a.tiles_x) * 32;
            r.y0 = (tile / a.tiles_x) * kStreamRows;
            const long long ng = a.g1 - a.g0;
            r.g = a.g0 + static_cast<int>(ng * split / a.splits);
            r.gb = a.g0 + static_cast<int>(ng * (split + 1) / a.splits);
            r.n = a.n;
            r.i0 = 0;
            r.window = a.rows * kStreamPitch;
            r.inside = r.x0 + 31 < a.w && r.y0 + kStreamRows - 1 < a.h;
            r.inv_n = a.inv_sqrt[a.n];
        }
    }
    __syncwarp();
    if (r.p < 0) {
        if (lane == 0) {
            sh.next = r;
            sh.run[b].p = -1;
            mbar_arrive(&sh.full[b]);
        }
        return;
    }
    const StreamArgs& a = passes[r.p];
    r.frames = min(a.frames, r.n - r.i0);
    const int window = r.window * 4;
    StreamWin wv;
    if (lane < r.frames) wv = a.wins[static_cast<size_t>(r.g) * r.n + r.i0 + lane];
    if (lane == 0) {
        sh.run[b] = r;
        Run t = r;
        t.i0 += r.frames;
        if (t.i0 >= t.n) {
            t.i0 = 0;
            ++t.g;
        }
        sh.next = t;
        const uint32_t words = static_cast<uint32_t>(r.frames) * kStreamWarps * 4;
        const bool ends = r.i0 + r.frames >= r.n;  // the run after which the group's maxima are taken
        const uint32_t tail = ends ? sizeof(sh.motion[0]) + sizeof(StreamGroup) : 0;
        mbar_expect_tx(&sh.full[b], static_cast<uint32_t>(r.frames * window) + words + tail + extra_tx);
        if (ends) {
            bulk_load(sh.motion[b], a.slot_motion + static_cast<size_t>(r.g) * kStreamWarps * kStreamBlock,
                      sizeof(sh.motion[0]), &sh.full[b]);
            bulk_load(&sh.group[b], a.groups + r.g, sizeof(StreamGroup), &sh.full[b]);
        }
        bulk_load(sh.desc[b], a.desc + (static_cast<size_t>(r.g) * r.n + r.i0) * kStreamWarps, words, &sh.full[b]);
    }
    __syncwarp();
    if (lane < r.frames)
        tma_load_3d(windows + lane * window, maps + r.p, r.x0 + wv.dx0, r.y0 + wv.dy0, r.i0 + lane, &sh.full[b]);
    __syncwarp();
}

__global__ void __launch_bounds__(kThreads, 1)
    stack_stream_kernel(const StreamArgs* __restrict__ passes, const CUtensorMap* __restrict__ maps, int npasses,
                        long long items, unsigned long long* queue, int* err, int buffer, unsigned extra_tx,
                        long long limit) {
    constexpr int P = kStreamRows, H = P / 2, WP = kStreamPitch, M = kStreamBlock;
    extern __shared__ __align__(128) unsigned char smem[];  // the only shared memory, at a fixed 128-byte boundary
    Shared& sh = *reinterpret_cast<Shared*>(smem);
    unsigned char* ring = smem + sizeof(Shared);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int b = 0; b < kBuffers; ++b) {
            mbar_init(&sh.full[b], 1);
            sh.left[b] = 0;
        }
        mbar_init(&sh.tile_bar, kStreamWarps);
        sh.abort = 0;
        sh.next.p = -1;
        sh.next.g = sh.next.gb = 0;
    }
    for (int q = tid; q < 32 * P; q += kThreads) sh.keys[q] = 0ull;
    tensor_maps_acquire(maps, npasses);
    __syncthreads();
    if (warp == 0)
        for (int b = 0; b < kBuffers; ++b)
            copy_run(sh, ring + b * buffer, passes, maps, npasses, items, queue, b, extra_tx, lane);

    unsigned long long acc[M * H];  // [motion][row pair]
    int b = 0;
    uint32_t phase = 0, tile_phase = 0;
    for (;;) {
        if (!ring_wait(sh, &sh.full[b], phase, err, limit)) break;
        const Run& run = sh.run[b];
        if (run.p < 0) return;
        // the buffer before this one, once every warp is past it: the first warp that
        // finds it so copies the run after next (warps ahead of the others do it)
        const int before = b == 0 ? kBuffers - 1 : b - 1;
        int claimed = 0;
        if (lane == 0 && *reinterpret_cast<volatile int*>(&sh.left[before]) == kStreamWarps)
            claimed = atomicCAS(&sh.left[before], kStreamWarps, 0) == kStreamWarps;
        if (__shfl_sync(0xffffffffu, claimed, 0)) {
            __threadfence_block();
            fence_proxy_async();
            copy_run(sh, ring + before * buffer, passes, maps, npasses, items, queue, before, extra_tx, lane);
        }
        if (run.i0 == 0) {
#pragma unroll
            for (int e = 0; e < M * H; ++e) acc[e] = 0ull;
        }
        const int frames = run.frames, window = run.window;
        const uint32_t* dp = sh.desc[b] + warp;
        const float* src = reinterpret_cast<const float*>(ring + b * buffer) + lane;
        uint32_t d = *dp;
        const bool idle = d == kStreamIdle;
        if (!idle) {
#pragma unroll 1
            for (int i = 0; i < frames; ++i) {
                const float* col = src + (d & 0xffffu);
                unsigned long long A[H + 1];
#pragma unroll
                for (int r = 0; r <= H; ++r) A[r] = pack2(col[r * WP], col[(r + H) * WP]);
                dp += kStreamWarps;  // (one word beyond the run's: inside the buffers, not used)
                const uint32_t next = *dp;
                src += window;
                block_frame(acc, A, d);
                d = next;
            }
        }
        const bool ends = run.i0 + frames >= run.n;
        if (ends) {
            const int x0 = run.x0, y0 = run.y0, g = run.g, n = run.n;
            const bool tile_ends = g + 1 == run.gb;
            const StreamArgs& a = passes[run.p];
            if (!idle) {
                const StreamGroup G = sh.group[b];
                const int* motion = sh.motion[b] + warp * M;
                const bool interior = run.inside && x0 + G.gdxmin >= 0 && x0 + 31 + G.gdxmax < a.w &&
                                      y0 + G.gdymin >= 0 && y0 + P - 1 + G.gdymax < a.h;
                if (interior) {
                    // all n frames cover every pixel. The largest sum gives the largest
                    // S/N (one positive factor, a monotone rounding), and only where it
                    // reaches the tile's running maximum are the motions looked at; a
                    // block's motions ascend and a pad repeats the last one's sums
                    const float inv_n = run.inv_n;
#pragma unroll
                    for (int q = 0; q < P; ++q) {
                        float s[M];
#pragma unroll
                        for (int k = 0; k < M; ++k) {
                            const float2 v = unpack2(acc[H * k + q % H]);
                            s[k] = q < H ? v.x : v.y;
                        }
                        const float top = max3(max3(s[0], s[1], s[2]), s[3], s[4]);
                        unsigned long long* key = sh.keys + q * 32 + lane;
                        const uint32_t held = *(reinterpret_cast<volatile uint32_t*>(key) + 1);
                        if (order_bits(__fmul_rn(top, inv_n)) >= held) {
                            float best = -CUDART_INF_F;
                            int arg = -1;
#pragma unroll
                            for (int k = 0; k < M; ++k) {
                                const float v = __fmul_rn(s[k], inv_n);
                                const int j = motion[k];
                                if (j >= 0 && v > best) {
                                    best = v;
                                    arg = j;
                                }
                            }
                            if (arg >= 0) atomicMax(key, snr_key(best, arg));
                        }
                    }
                } else {
                    // each motion's frames that cover a pixel: `whole` those that cover the
                    // tile (a lane looks at a frame), cx those whose rows do and whose column
                    // covers this lane's, part the others, one byte a row (255 frames at most)
                    const uint32_t* desc = a.desc + static_cast<size_t>(g) * n * kStreamWarps + warp;
                    const StreamWin* wins = a.wins + static_cast<size_t>(g) * n;
#pragma unroll
                    for (int k = 0; k < M; ++k) {
                        const int j = motion[k];
                        if (j < 0) break;
                        int whole = 0, cx = 0;
                        uint32_t part[P / 4] = {};
                        for (int c = 0; c < n; c += 32) {
                            const bool in = c + lane < n;
                            int sx = 0, sy = 0;
                            if (in) {
                                const uint32_t e = desc[static_cast<size_t>(c + lane) * kStreamWarps];
                                const StreamWin wv = wins[c + lane];
                                const int off = static_cast<int>(e & 0xffffu), row = off / WP;
                                sx = wv.dx0 + off - row * WP;
                                sy = wv.dy0 + row + stream_row(e, k);
                            }
                            const bool rows = y0 + sy >= 0 && y0 + P - 1 + sy < a.h;
                            const bool cols = x0 + sx >= 0 && x0 + 31 + sx < a.w;
                            whole += __popc(__ballot_sync(0xffffffffu, in && rows && cols));
                            unsigned some = __ballot_sync(0xffffffffu, in && !(rows && cols));
                            while (some) {
                                const int f = __ffs(some) - 1;
                                some &= some - 1;
                                const int fx = __shfl_sync(0xffffffffu, sx, f), fy = __shfl_sync(0xffffffffu, sy, f);
                                const bool inx = static_cast<unsigned>(x0 + lane + fx) < static_cast<unsigned>(a.w);
                                const int lo = max(0, -(y0 + fy)), hi = min(P - 1, a.h - 1 - (y0 + fy));
                                if (lo == 0 && hi == P - 1) {
                                    cx += inx;
                                } else if (lo <= hi) {
                                    const uint32_t m = inx ? (0xffffffffu >> (31 - hi)) & (0xffffffffu << lo) : 0u;
#pragma unroll
                                    for (int w = 0; w < P / 4; ++w)
                                        part[w] += (((m >> (4 * w)) & 15u) * 0x00204081u) & 0x01010101u;
                                }
                            }
                        }
                        whole += cx;
#pragma unroll
                        for (int q = 0; q < P; ++q) {
                            const int c = whole + static_cast<int>((part[q >> 2] >> (8 * (q & 3))) & 0xffu);
                            if (c < a.min_count) continue;
                            const float2 s = unpack2(acc[H * k + q % H]);
                            const float v = __fmul_rn(q < H ? s.x : s.y, a.inv_sqrt[c]);
                            unsigned long long* key = sh.keys + q * 32 + lane;
                            const uint32_t held = *(reinterpret_cast<volatile uint32_t*>(key) + 1);
                            if (v > -CUDART_INF_F && order_bits(v) >= held) atomicMax(key, snr_key(v, j));
                        }
                    }
                }
            }
            if (tile_ends) {
                // every warp's maxima are in: the tile's keys go out and are cleared
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.tile_bar);
                if (!ring_wait(sh, &sh.tile_bar, tile_phase, err, limit)) break;
                const int q = tid, xx = x0 + (q & 31), yy = y0 + (q >> 5);
                const unsigned long long key = sh.keys[q];
                sh.keys[q] = 0ull;
                if (xx < a.w && yy < a.h) {
                    const size_t o = static_cast<size_t>(yy) * a.w + xx;
                    if (a.keys) {
                        if (key) atomicMax(a.keys + o, key);
                    } else {
                        float best = -CUDART_INF_F;
                        int arg = -1;
                        if (key) snr_unkey(key, best, arg);
                        a.max_snr[o] = isfinite(best) ? best : 0.0f;
                        a.best_v[o] = arg;
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.tile_bar);
                if (!ring_wait(sh, &sh.tile_bar, tile_phase ^ 1u, err, limit)) break;
            }
        }
        // this warp is past the buffer
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            atomicAdd(&sh.left[b], 1);
        }
        if (++b == kBuffers) {
            b = 0;
            phase ^= 1u;
        }
    }
    // a wait ran out: the copies in flight land before the shared memory is given up
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) {
    }
}

// The maps of a pass whose maxima were merged in global keys.
__global__ void __launch_bounds__(256) stream_maps_kernel(const unsigned long long* keys, size_t pixels, float* max_snr,
                                                          int* best_v) {
    const size_t o = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x;
    if (o >= pixels) return;
    float b = -CUDART_INF_F;
    int ar = -1;
    if (keys[o]) snr_unkey(keys[o], b, ar);
    max_snr[o] = isfinite(b) ? b : 0.0f;
    best_v[o] = ar;
}

}  // namespace

int stream_splits(const std::vector<const StackPlan*>& plans, int sms) {
    long long tiles = 0;
    size_t groups = 1;
    for (const StackPlan* p : plans) {
        tiles += static_cast<long long>((p->w + 31) / 32) * ((p->h + kStreamRows - 1) / kStreamRows);
        groups = std::max(groups, p->stream.groups.size());
    }
    const long long want = (4LL * sms + tiles - 1) / tiles;
    return static_cast<int>(std::max<long long>(1, std::min<long long>(want, static_cast<long long>(groups))));
}

size_t stream_desc_bytes(int npasses) { return 128 + (128 + sizeof(StreamArgs)) * static_cast<size_t>(npasses); }

int stream_launch(const std::vector<BatchPass>& batch, int splits, unsigned char* d_desc, size_t desc_bytes, int* d_err,
                  int sms, cudaStream_t s) {
    const size_t np = batch.size();
    if (np == 0) return 0;
    int launches = 0;
    std::vector<unsigned char> host(stream_desc_bytes(static_cast<int>(np)), 0);
    if (host.size() > desc_bytes) throw std::runtime_error("stack batch: descriptor buffer too small");
    CUtensorMap* maps = reinterpret_cast<CUtensorMap*>(host.data() + 128);
    StreamArgs* args = reinterpret_cast<StreamArgs*>(host.data() + 128 + 128 * np);
    long long items = 0;
    int buffer = 0;
    for (size_t k = 0; k < np; ++k) {
        const BatchPass& bp = batch[k];
        const StackPlan& plan = *bp.plan;
        const int rows = plan.stream.rows;
        const cuuint64_t dims[3] = {static_cast<cuuint64_t>(plan.w), static_cast<cuuint64_t>(plan.h),
                                    static_cast<cuuint64_t>(plan.n)};
        const cuuint64_t strides[2] = {static_cast<cuuint64_t>(plan.pitch) * 4,
                                       static_cast<cuuint64_t>(plan.pitch) * plan.h * 4};
        const cuuint32_t box[3] = {kStreamPitch, static_cast<cuuint32_t>(rows), 1};
        const cuuint32_t estr[3] = {1, 1, 1};
        const CUresult r = tensor_map_encoder()(
            &maps[k], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(bp.frames), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
            throw CudaError("cuTensorMapEncodeTiled failed (" + std::to_string(static_cast<int>(r)) + ")");
        const StackPlanDev& dev = *bp.dev;
        StreamArgs& a = args[k];
        a.w = plan.w;
        a.h = plan.h;
        a.n = plan.n;
        a.min_count = plan.min_count;
        a.g0 = bp.g0;
        a.g1 = bp.g1;
        a.splits = std::max(1, std::min(splits, bp.g1 - bp.g0));
        a.tiles_x = (plan.w + 31) / 32;
        a.rows = rows;
        a.frames = stream_frames(plan.n, rows);
        if (a.frames > kMostFrames) throw std::runtime_error("stack stream: too many frames in a run");
        buffer = std::max(buffer, a.frames * rows * kStreamPitch * 4);
        a.item0 = items;
        items += static_cast<long long>(a.tiles_x) * ((plan.h + kStreamRows - 1) / kStreamRows) * a.splits;
        a.groups = dev.stream_groups;
        a.wins = dev.stream_wins;
        a.desc = dev.stream_desc;
        a.slot_motion = dev.slot_motion;
        a.inv_sqrt = dev.inv_sqrt;
        a.keys = bp.keys;
        a.max_snr = bp.max_snr;
        a.best_v = bp.best_v;
        if (!bp.keys && (a.splits > 1 || !bp.first || !bp.last))
            throw std::runtime_error("stack stream: a pass in parts needs its keys");
        if (bp.keys && bp.first)
            FTB_CHECK(cudaMemsetAsync(bp.keys, 0, sizeof(unsigned long long) * static_cast<size_t>(plan.w) * plan.h, s));
    }
    FTB_CHECK(cudaMemcpyAsync(d_desc, host.data(), host.size(), cudaMemcpyHostToDevice, s));
    unsigned extra_tx;
    long long wait_limit;
    wait_test(extra_tx, wait_limit);
    const size_t smem = sizeof(Shared) + static_cast<size_t>(kBuffers) * buffer;
    allow_dynamic_smem(reinterpret_cast<const void*>(stack_stream_kernel), smem);
    const int ctas = static_cast<int>(std::min<long long>(items, sms));
    stack_stream_kernel<<<ctas, kThreads, smem, s>>>(
        reinterpret_cast<const StreamArgs*>(d_desc + 128 + 128 * np), reinterpret_cast<const CUtensorMap*>(d_desc + 128),
        static_cast<int>(np), items, reinterpret_cast<unsigned long long*>(d_desc), d_err, buffer, extra_tx, wait_limit);
    FTB_CHECK(cudaGetLastError());
    ++launches;
    for (const BatchPass& bp : batch) {
        if (!bp.keys || !bp.last) continue;
        const size_t px = static_cast<size_t>(bp.plan->w) * bp.plan->h;
        stream_maps_kernel<<<static_cast<unsigned>((px + 255) / 256), 256, 0, s>>>(bp.keys, px, bp.max_snr, bp.best_v);
        FTB_CHECK(cudaGetLastError());
        ++launches;
    }
    return launches;
}

}  // namespace ftb
