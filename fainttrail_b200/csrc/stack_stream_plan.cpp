// The host planner of the streamed stacking pass (stack_stream.cu).
#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <unordered_map>
#include <vector>

#include "stack_stream.h"

namespace ftb {

namespace {

struct Block {
    int motion[kStreamBlock];
    int count = 0;
    int ex = 0, ey = 0;  // its first motion's shift in the frame of widest spread
};

inline int floor4(int v) { return (v >> 2) * 4; }  // arithmetic shift: floor for negatives too

}  // namespace

StreamPlan make_stream_plan(int w, int h, int n, const int* dx, const int* dy, int m) {
    StreamPlan P;
    if (m < 1 || n < 1) return P;
    const size_t N = static_cast<size_t>(n);
    // clamped shifts: beyond +-w / +-h a frame never covers, as within
    auto X = [&](int j, size_t i) { return std::clamp(dx[static_cast<size_t>(j) * N + i], -w, w); };
    auto Y = [&](int j, size_t i) { return std::clamp(dy[static_cast<size_t>(j) * N + i], -h, h); };
    // A block lies at no more than two positions in a frame, and at most m / 4.5 blocks keep
    // to the pad limit below: more than 4 m / 9 positions in one frame, as coarse lattices
    // have in their widest, do not pack (looked at in the frame that moves the first motion
    // most; the whole way to a refusal took 3 of 25 ms of the plan for 100 frames and 9008
    // motions).
    {
        size_t i = 0;
        for (size_t q = 1; q < N; ++q)
            if (std::abs(X(0, q)) + std::abs(Y(0, q)) > std::abs(X(0, i)) + std::abs(Y(0, i))) i = q;
        int lx = X(0, i), hx = lx, ly = Y(0, i), hy = ly;
        for (int j = 1; j < m; ++j) {
            lx = std::min(lx, X(j, i));
            hx = std::max(hx, X(j, i));
            ly = std::min(ly, Y(j, i));
            hy = std::max(hy, Y(j, i));
        }
        const long long wide = static_cast<long long>(hx) - lx + 1, tall = static_cast<long long>(hy) - ly + 1;
        if (wide * tall <= 8LL * m) {
            std::vector<unsigned char> seen(static_cast<size_t>(wide * tall), 0);
            long long positions = 0;
            for (int j = 0; j < m; ++j) {
                unsigned char& at = seen[static_cast<size_t>((Y(j, i) - ly) * wide + (X(j, i) - lx))];
                positions += !at;
                at = 1;
            }
            if (positions * 9 > 4LL * m) return P;
        }
    }
    // classes of motions whose columns agree in every frame, each in index order
    std::vector<int> rep, chain;
    std::vector<std::vector<int>> members;
    std::unordered_map<uint64_t, int> by_hash;
    for (int j = 0; j < m; ++j) {
        const int* a = dx + static_cast<size_t>(j) * N;
        uint64_t hsh = 1469598103934665603ull;
        for (size_t i = 0; i < N; ++i) hsh = (hsh ^ static_cast<uint32_t>(a[i])) * 1099511628211ull;
        auto it = by_hash.find(hsh);
        int c = -1;
        if (it != by_hash.end())
            for (int k = it->second; k >= 0 && c < 0; k = chain[static_cast<size_t>(k)])
                if (std::memcmp(dx + static_cast<size_t>(rep[static_cast<size_t>(k)]) * N, a, sizeof(int) * N) == 0) c = k;
        if (c < 0) {
            c = static_cast<int>(rep.size());
            rep.push_back(j);
            chain.push_back(it != by_hash.end() ? it->second : -1);
            by_hash[hsh] = c;
            members.emplace_back();
        }
        members[static_cast<size_t>(c)].push_back(j);
    }
    // blocks: consecutive motions of a class whose rows, in every frame, take at
    // most one step, of one row
    std::vector<Block> blocks;
    std::vector<int> stepped(N);
    // pads cost what motions cost: up to a tenth of the slots, looked at before each class as
    // if the motions left filled their blocks (slots only become more)
    size_t left = static_cast<size_t>(m);
    auto padded = [&]() {
        const long long slots = static_cast<long long>(blocks.size()) * kStreamBlock + static_cast<long long>(left);
        return (slots - m) * 10 > slots;
    };
    for (const std::vector<int>& mem : members) {
        if (padded()) return P;
        left -= mem.size();
        Block b;
        auto close = [&]() {
            if (b.count == 0) return;
            blocks.push_back(b);
            b.count = 0;
        };
        for (int j : mem) {
            if (b.count == kStreamBlock) close();
            if (b.count > 0) {
                const int prev = b.motion[b.count - 1];
                int bad = 0;
                for (size_t i = 0; i < N; ++i) {
                    const int e = Y(j, i) - Y(prev, i);
                    bad |= (e > 1) | (e < -1) | ((e != 0) & stepped[i]);
                    stepped[i] |= e != 0;
                }
                if (bad) close();
            }
            if (b.count == 0) std::fill(stepped.begin(), stepped.end(), 0);
            b.motion[b.count++] = j;
        }
        close();
    }
    if (padded()) return P;
    // the frame whose shifts spread most orders the blocks
    std::vector<int> lo(N, INT_MAX), hi(N, INT_MIN);
    for (int j = 0; j < m; ++j) {
        const int* a = dx + static_cast<size_t>(j) * N;
        const int* b = dy + static_cast<size_t>(j) * N;
        for (size_t i = 0; i < N; ++i) {
            lo[i] = std::min(lo[i], std::min(a[i], b[i]));
            hi[i] = std::max(hi[i], std::max(a[i], b[i]));
        }
    }
    size_t ie = 0;
    for (size_t i = 1; i < N; ++i)
        if (static_cast<long long>(hi[i]) - lo[i] > static_cast<long long>(hi[ie]) - lo[ie]) ie = i;
    for (Block& b : blocks) {
        b.ex = X(b.motion[0], ie);
        b.ey = Y(b.motion[0], ie);
    }
    // groups of kStreamWarps blocks with close shifts: strips of columns about two
    // pixels wide at frame ie, each walked up or down in turn
    auto kx = [&](const Block& b) { return b.ex >> 1; };
    std::stable_sort(blocks.begin(), blocks.end(), [&](const Block& a, const Block& b) {
        if (kx(a) != kx(b)) return kx(a) < kx(b);
        const int s = (kx(a) & 1) ? -1 : 1;
        if (a.ey != b.ey) return s * a.ey < s * b.ey;
        return a.ex < b.ex;
    });
    std::vector<int> lx(N), hx(N), ly(N), hy(N), tx(N), ux(N), ty(N), uy(N);
    std::vector<const Block*> open;
    auto flush = [&]() {
        StreamGroup g;
        g.gdxmin = g.gdymin = INT_MAX;
        g.gdxmax = g.gdymax = INT_MIN;
        const size_t s0 = P.slot_motion.size(), d0 = P.desc.size(), w0 = P.wins.size();
        P.slot_motion.resize(s0 + static_cast<size_t>(kStreamWarps) * kStreamBlock, -1);
        P.desc.resize(d0 + N * kStreamWarps, kStreamIdle);
        for (size_t i = 0; i < N; ++i) {
            P.wins.push_back({floor4(lx[i]), ly[i]});
            P.rows = std::max(P.rows, (hy[i] - ly[i] + kStreamRows + 1 + kStreamBox - 1) / kStreamBox * kStreamBox);
            g.gdxmin = std::min(g.gdxmin, lx[i]);
            g.gdxmax = std::max(g.gdxmax, hx[i]);
        }
        for (size_t q = 0; q < open.size(); ++q) {
            const Block& b = *open[q];
            std::copy(b.motion, b.motion + b.count, P.slot_motion.begin() + static_cast<std::ptrdiff_t>(s0 + q * kStreamBlock));
            for (size_t i = 0; i < N; ++i) {
                int row[kStreamBlock];
                for (int k = 0; k < b.count; ++k) {
                    row[k] = Y(b.motion[k], i);
                    g.gdymin = std::min(g.gdymin, row[k]);
                    g.gdymax = std::max(g.gdymax, row[k]);
                }
                uint32_t d = 0;
                int base = row[0];
                for (int k = 1; k < b.count; ++k) {  // (a pad repeats the last motion)
                    base = std::min(base, row[k]);
                    if (row[k] != row[k - 1]) d |= 1u << (16 + k);
                }
                if (row[0] > base) d |= 1u << 24;
                const StreamWin& wv = P.wins[w0 + i];
                d |= static_cast<uint32_t>((base - wv.dy0) * kStreamPitch + (X(b.motion[0], i) - wv.dx0));
                P.desc[d0 + i * kStreamWarps + q] = d;
            }
        }
        P.groups.push_back(g);
        open.clear();
    };
    // the windows of the open group with block b in it; false: they do not fit
    auto extend = [&](const Block& b) {
        const bool first = open.empty();
        int bad = 0;
        for (size_t i = 0; i < N; ++i) {
            int l = Y(b.motion[0], i);
            for (int k = 1; k < b.count; ++k) l = std::min(l, Y(b.motion[k], i));
            const int x = X(b.motion[0], i);
            tx[i] = first ? x : std::min(lx[i], x);
            ux[i] = first ? x : std::max(hx[i], x);
            ty[i] = first ? l : std::min(ly[i], l);
            uy[i] = first ? l : std::max(hy[i], l);
            bad |= (ux[i] - floor4(tx[i]) + 32 > kStreamPitch) | (uy[i] - ty[i] + kStreamRows + 1 > kStreamMaxRows);
        }
        return !bad;
    };
    for (const Block& b : blocks) {
        if (open.size() == static_cast<size_t>(kStreamWarps)) flush();
        if (!extend(b)) {
            flush();
            extend(b);  // a block's own windows always fit
        }
        lx.swap(tx);
        hx.swap(ux);
        ly.swap(ty);
        hy.swap(uy);
        open.push_back(&b);
    }
    flush();
    // groups left a quarter empty leave warps idle
    if (P.groups.size() > 4 && blocks.size() * 4 < P.groups.size() * kStreamWarps * 3) return StreamPlan();
    return P;
}

}  // namespace ftb
