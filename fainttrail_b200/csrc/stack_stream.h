// The streamed stacking pass (stack_stream.cu): its plan and the constants its
// planner, kernel and host emulation share.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

namespace ftb {

constexpr int kStreamBlock = 5;      // motions a warp accumulates together
constexpr int kStreamWarps = 16;     // blocks of a group, one a warp
constexpr int kStreamRows = 16;      // output rows of a tile (32 columns)
constexpr int kStreamPitch = 40;     // window pitch in floats
constexpr int kStreamBox = 4;        // rows of one TMA box
constexpr int kStreamMaxRows = 36;   // window rows at most
constexpr int kStreamBuffer = 68 * 1024;  // bytes of one of the three window buffers

// A block's motions in one frame share their column and take at most one step of
// one row between them. Its descriptor: bits 0-15 the window offset of the lowest
// row, bit 16 + k (k = 1 .. 4) a step between motions k - 1 and k, bit 24 the first
// motion on the upper row. kStreamIdle: a block without motions.
constexpr uint32_t kStreamIdle = 0xffffffffu;
__host__ __device__ constexpr int stream_row(uint32_t desc, int k) {
    int row = static_cast<int>(desc >> 24 & 1u);
    for (int q = 1; q <= k; ++q) row ^= static_cast<int>(desc >> (16 + q) & 1u);
    return row;
}

// One frame's window of a group: its origin relative to the tile (dx0 a multiple
// of 4).
struct StreamWin {
    int dx0 = 0, dy0 = 0;
};

// A group: the blocks that stream through one set of windows, one block a warp.
struct StreamGroup {
    int gdxmin = 0, gdxmax = 0, gdymin = 0, gdymax = 0;  // shift extremes over its motions and frames
};

struct StreamPlan {
    std::vector<StreamGroup> groups;
    std::vector<StreamWin> wins;     // [group][frame]
    std::vector<uint32_t> desc;      // [group][frame][block]
    std::vector<int> slot_motion;    // [group][block][kStreamBlock] ascending, -1: a pad
    int rows = 0;                    // rows of every window (a multiple of kStreamBox)
    bool empty() const { return groups.empty(); }
};

// Frames of a stage: the frames in equal parts of at most what a buffer holds.
__host__ __device__ inline int stream_frames(int n, int rows) {
    const int fit = kStreamBuffer / (rows * kStreamPitch * 4), most = fit < 32 ? fit : 32;
    const int parts = (n + most - 1) / most;
    return (n + parts - 1) / parts;
}

// The plan of a pass, or an empty one where its motions do not pack for it: the
// other tile shapes then.
StreamPlan make_stream_plan(int w, int h, int n, const int* dx, const int* dy, int m);

}  // namespace ftb
