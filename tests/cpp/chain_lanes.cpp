// The chain kernel's device code on the host, for tests/test_chain_lanes.py: the 32 lanes of a warp are
// fibers, and each runs on its own up to its next warp-wide operation (shuffle, ballot, reduction,
// __syncwarp), in an order that the caller picks -- the freedom that independent thread scheduling
// gives the device.  A lane that reads or updates what another lane also updates, without a
// warp-wide operation in between, then gives another result than lanes in lockstep.  All lanes have
// to meet at the same operation; a lane that finishes or meets another one is reported.
//
// Compiled twice: CHAIN_PLAN, the host pass that sizes a chain's scratch (with the namespace renamed,
// as both builds hold the same inline functions), and without it, the kernel and main().
#include <climits>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#define __host__
#define __device__
#define __global__
#define __shared__
#define __forceinline__ inline
#define __launch_bounds__(...)

struct Dim { unsigned x; };
struct int2 { int x, y; };
struct alignas(16) int4 { int x, y, z, w; };
struct alignas(16) uint4 { unsigned x, y, z, w; };
inline uint4 make_uint4(unsigned x, unsigned y, unsigned z, unsigned w) { return uint4{x, y, z, w}; }
using cudaStream_t = void *;

struct Problem {
    int32_t m, n, seeds;
    int32_t anchor[4], gap[4];        // match, mismatch, extend, open
    int32_t free_ends, band_ext, affine, max_traces;
};
void plan_chain(const Problem &p, const int32_t *seeds, void *plan, int64_t *bytes);

#ifdef CHAIN_PLAN
#define chain chain_plan
#include "../../seqan_gb300/csrc/chain_kernels.cuh"

void plan_chain(const Problem &p, const int32_t *seeds, void *plan, int64_t *bytes)
{
    chain::Plan pl{};
    pl.gseg_cap = p.m + p.n + 8;
    chain::Engine e{};
    e.plan = true;
    e.anchor = chain::Scheme{p.anchor[0], p.anchor[1], p.anchor[2], p.anchor[3]};
    e.gap = chain::Scheme{p.gap[0], p.gap[1], p.gap[2], p.gap[3]};
    e.fe = p.free_ends;
    e.affine = p.affine;
    e.k = p.band_ext;
    e.max_traces = p.max_traces;
    e.m = p.m;
    e.n = p.n;
    e.pl = &pl;
    e.run(seeds, p.seeds);
    pl.status = e.err;
    if (pl.set_cap < pl.mp_cap) pl.set_cap = pl.mp_cap;
    if (pl.col_rows < 1) pl.col_rows = 1;
    *bytes = chain::layout(pl, p.max_traces, nullptr, nullptr) + 16;
    std::memcpy(plan, &pl, sizeof pl);
}

#else
#include <ucontext.h>

namespace lanes {

enum Kind { SYNC, SHFL, BALLOT, MINIMUM, MAXIMUM, ALL };
constexpr int kLanes = 32, kStack = 256 * 1024;
ucontext_t scheduler, lane_context[kLanes];
std::vector<char> stack[kLanes];
bool finished[kLanes];
int kind[kLanes];
int64_t given[kLanes], taken[kLanes];   // what the lanes bring to this operation; what they all brought
int current;
void (*body)();

void start() { body(); finished[current] = true; swapcontext(&lane_context[current], &scheduler); }

void meet(int k, int64_t value)
{
    kind[current] = k;
    given[current] = value;
    swapcontext(&lane_context[current], &scheduler);
}

// Runs `f` on all lanes; order: 0 first to last, 1 last to first, else a random one, new at every operation.
// False when the lanes do not meet.
bool run(void (*f)(), unsigned order, Dim &thread)
{
    body = f;
    for (int l = 0; l < kLanes; ++l) {
        stack[l].resize(kStack);
        finished[l] = false;
        getcontext(&lane_context[l]);
        lane_context[l].uc_stack.ss_sp = stack[l].data();
        lane_context[l].uc_stack.ss_size = kStack;
        lane_context[l].uc_link = nullptr;
        makecontext(&lane_context[l], start, 0);
    }
    uint32_t random = order * 2654435761u + 1;
    for (;;) {
        int turn[kLanes];
        for (int l = 0; l < kLanes; ++l) turn[l] = order == 1 ? kLanes - 1 - l : l;
        if (order > 1)
            for (int l = kLanes - 1; l > 0; --l) {
                random = random * 1664525u + 1013904223u;
                const int q = int((random >> 8) % unsigned(l + 1)), t = turn[l];
                turn[l] = turn[q];
                turn[q] = t;
            }
        int done = 0;
        for (int l : turn) {
            current = l;
            thread.x = unsigned(l);
            swapcontext(&scheduler, &lane_context[l]);
            done += finished[l];
        }
        if (done == kLanes) return true;
        if (done > 0) return false;
        for (int l = 1; l < kLanes; ++l)
            if (kind[l] != kind[0]) return false;
        std::memcpy(taken, given, sizeof taken);
    }
}

}  // namespace lanes

static Dim threadIdx, blockIdx, blockDim{32};

inline void __syncwarp() { lanes::meet(lanes::SYNC, 0); }
inline int __shfl_sync(unsigned, int v, int from) { lanes::meet(lanes::SHFL, v); return int(lanes::taken[from & 31]); }
inline unsigned __ballot_sync(unsigned, bool v)
{
    lanes::meet(lanes::BALLOT, v);
    unsigned b = 0;
    for (int l = 0; l < 32; ++l) b |= unsigned(lanes::taken[l] != 0) << l;
    return b;
}
inline bool __all_sync(unsigned, bool v)
{
    lanes::meet(lanes::ALL, v);
    for (int l = 0; l < 32; ++l)
        if (!lanes::taken[l]) return false;
    return true;
}
inline int __reduce_min_sync(unsigned, int v)
{
    lanes::meet(lanes::MINIMUM, v);
    int64_t r = lanes::taken[0];
    for (int64_t x : lanes::taken) r = x < r ? x : r;
    return int(r);
}
inline int __reduce_max_sync(unsigned, int v)
{
    lanes::meet(lanes::MAXIMUM, v);
    int64_t r = lanes::taken[0];
    for (int64_t x : lanes::taken) r = x > r ? x : r;
    return int(r);
}
inline int __popc(unsigned x) { return __builtin_popcount(x); }
inline int atomicAdd(int *p, int v) { const int old = *p; *p += v; return old; }

#define __CUDA_ARCH__ 1030
#define SEQAN_GB300_CHAIN_KERNELS
#include "../../seqan_gb300/csrc/chain_kernels.cuh"

uint4 chain_shared[chain::kSharedPerWarp / sizeof(uint4)];

static ChainArgs args;
static void kernel() { k_banded_chain(args); }

template <typename T>
static bool read(T *to, size_t count) { return count == 0 || std::fread(to, sizeof(T), count, stdin) == count; }

// stdin: problems (Problem, H, V, 4 integers per seed); stdout: per problem (met, status, score, traces,
// segments) and the segments.  Argument: the order of the lanes.
int main(int, char **argv)
{
    const unsigned order = unsigned(std::atoi(argv[1]));
    Problem p;
    while (read(&p, 1)) {
        std::vector<uint8_t> h(size_t(p.m) + 16), v(size_t(p.n) + 16);
        std::vector<int32_t> seeds(size_t(p.seeds) * 4);
        if (!read(h.data(), size_t(p.m)) || !read(v.data(), size_t(p.n)) || !read(seeds.data(), seeds.size())) return 1;
        chain::ChainDesc d{};
        int64_t bytes = 0;
        plan_chain(p, seeds.data(), &d.plan, &bytes);
        d.m = p.m;
        d.n = p.n;
        d.n_seeds = p.seeds;
        std::vector<uint4> arena(size_t(bytes) / sizeof(uint4) + 1);
        std::memset(arena.data(), 0xcd, arena.size() * sizeof(uint4));
        std::memset(chain_shared, 0xcd, sizeof chain_shared);
        int32_t out[4] = {0, 0, 0, 0}, next = 0;
        args = ChainArgs{};
        args.seq_h = h.data();
        args.seq_v = v.data();
        args.seeds = seeds.data();
        args.chains = &d;
        args.num_chains = 1;
        args.arena = reinterpret_cast<uint8_t *>(arena.data());
        args.anchor = chain::Scheme{p.anchor[0], p.anchor[1], p.anchor[2], p.anchor[3]};
        args.gap = chain::Scheme{p.gap[0], p.gap[1], p.gap[2], p.gap[3]};
        args.free_ends = p.free_ends;
        args.band_ext = p.band_ext;
        args.affine = p.affine;
        args.max_traces = p.max_traces;
        args.score = out;
        args.status = out + 1;
        args.n_traces = out + 2;
        args.seg_count = out + 3;
        args.next = &next;
        blockDim.x = 32;
        const bool met = lanes::run(kernel, order, threadIdx);
        std::vector<chain::Seg> segs(size_t(met && out[3] > 0 ? out[3] : 0));
        if (!segs.empty()) {
            const int64_t at = 0;
            threadIdx.x = 0;
            blockDim.x = 1;
            k_chain_pack(&d, 1, args.arena, p.max_traces, args.seg_count, &at, segs.data());
        }
        const int32_t head[5] = {met, out[1], out[0], out[2], int32_t(segs.size())};
        std::fwrite(head, sizeof head, 1, stdout);
        std::fwrite(segs.data(), sizeof(chain::Seg), segs.size(), stdout);
    }
    return 0;
}
#endif
