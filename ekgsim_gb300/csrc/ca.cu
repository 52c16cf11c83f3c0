// ca.cu -- activation times of the excitation-sequence cellular automaton on the device.
//
// The reference runs a Dijkstra search over the 26-neighbour cube (simlib/simulator.cpp:212-286):
// start voxels get time 1.0; a popped voxel u offers time(u) + lag to each unexcited non-empty
// neighbour v, lag = T[L(u)][L(v)] * sqrt(|u - v|^2), each step rounded in FP64.  With positive
// lags that search returns the unique fixed point of
//     at(v) = min(init(v), min_u fl(at(u) + fl(T[L(u)][L(v)] * sqrt(k))))
// (every offered time is >= the offering voxel's own time), so a chaotic min-relaxation from
// +inf converges to the same doubles bit for bit, in any order.  The products are formed on the host,
// the sums with __dadd_rn.
//
// Layout: the grid is cut into 8x8x8 tiles.  A round visits the tiles that hold pending times, one
// CTA each: the tile and a one-voxel halo are staged in shared memory (the FP64 times as their bit
// patterns, which order like the values for non-negative doubles, + uint8 layers), the tile settles up to
// the round's horizon, the settled times are written back, and the tiles that were offered a time or
// hold later ones form the next round's list (k_ca_round).  The host queues rounds in chunks and reads
// the lists' length once per chunk.
//
// GB300 (relaxation alone, CUDA events): 24^3 0.11 ms, 64^3 0.31, 128^3 0.71, 160^3 0.94
// (49 rounds), 192^3 1.23, 256^3 2.07.  One launch per time bucket over queues in global memory took
// 0.24, 0.57, 1.40, 1.96, 3.04 and 5.64 ms (9 us a bucket, every access of its chain a trip to L2); rounds
// of block-wide sweeps to local convergence, without a horizon, 3.4 ms at 160^3 in the calls that
// allocate nothing.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <mutex>
#include <vector>

#include "ekg_internal.h"

namespace ekg {

namespace {

constexpr int TS = 8;            // tile edge
constexpr int HS = TS + 2;       // tile + halo
constexpr int HCELLS = HS * HS * HS;
constexpr int CA_THREADS = TS * TS * TS;  // one thread per voxel of the tile
constexpr int CA_WARPS = CA_THREADS / 32;

__device__ __forceinline__ uint8_t layer_id(uint8_t v) { return v; }
__device__ __forceinline__ uint8_t layer_id(int32_t v) { return (uint8_t)(v < 0 ? -v : v); }

// While the relaxation runs, a cell's entry holds 2 * (bits of its time) + 1 while the time is pending (the
// cell has not offered it to its neighbours yet), 2 * bits once it has.  Entries order by time, and
// an offer of the same time does not replace a settled one.
typedef unsigned long long u64;
constexpr u64 INF_BITS = 0x7ff0000000000000ULL;

// The active tiles of consecutive rounds.  Round r walks list r & 1 (counts[r % 3] tiles), appends the
// tiles that hold pending times to list (r + 1) & 1 and clears the slot of round r + 2.
struct TileLists {
    int32_t *list;     // [2][cap]
    int cap;
    int32_t *counts;   // [3] tiles of a round, then the number of rounds that had a tile
    uint32_t *first;   // [3] high word of the earliest pending time of a round
    uint32_t *flags;   // one byte per tile, in words: bit (r & 1) set while the tile is in round r's list
};
constexpr int CA_CTRL_WORDS = 4 + 3;  // words of counts and first, one behind the other

__device__ __forceinline__ void tile_append(const TileLists &T, int tile, int round) {
    const uint32_t bit = 1u << (8 * (tile & 3) + (round & 1));
    if (!(atomicOr(&T.flags[tile >> 2], bit) & bit))
        T.list[(size_t)(round & 1) * T.cap + atomicAdd(&T.counts[round % 3], 1)] = tile;
}
// One round: a block per active tile, the grid walking the list, so that rounds can be queued back to
// back without the host reading the count.
//
// What bounds it: latency -- a chain of rounds, in a round the slowest tile's chain of settling steps,
// in a step its barriers and dependent shared-memory accesses.  Hence:
//  - a tile settles in steps: every voxel whose pending time lies within the round's horizon offers it to its
//    26 neighbours, a warp per voxel and a lane per neighbour, and offers again where a later step brings
//    it an earlier time (settling the earliest pending times first took as long, 1.11 and 1.12 ms at 160^3);
//  - a step has one barrier and no list: a warp expands the selected ones of its own 32 voxels, which
//    lie spread over the tile so that a front falls on all warps, and another step follows where
//    a voxel was selected, or an offer within the horizon may have come after its target's read;
//  - offers across the tile's surface go to the neighbour's cells in global memory (an atomicMin whose
//    result nothing waits for), so that a visit starts from the pending cells alone;
//  - a round settles only times up to its horizon, the earliest pending time of the heart + `window`
//    (a few of the largest lags), and later ones wait for their round: the front then moves at the
//    speed of the wave and not a tile per round, so that times which a faster path would replace are
//    not spread first.
template <typename LT>
__global__ void __launch_bounds__(CA_THREADS, 3)
    k_ca_round(int round, int nz, int ny, int nx, int ntz, int nty, int ntx, const LT *__restrict__ layers,
               const double *__restrict__ lag, int nl1, double window, u64 *__restrict__ at, TileLists T) {
    __shared__ u64 s_e[HCELLS];       // entries of the tile and its halo
    __shared__ uint8_t s_l[HCELLS];   // layers
    __shared__ uint8_t s_dir[HCELLS]; // which of the 27 tiles a cell lies in, 13 = this one ((dz+1)*9+(dy+1)*3+(dx+1))
    __shared__ uint32_t s_mark;       // tiles to queue, one bit each
    __shared__ uint32_t s_first;      // earliest time they wait for
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t NONE = 0xffffffffu;
    for (int i = tid; i < HCELLS; i += CA_THREADS) {
        const int hx = i % HS, hy = (i / HS) % HS, hz = i / (HS * HS);
        s_dir[i] = (uint8_t)((hz == 0 ? 0 : (hz > TS ? 18 : 9)) + (hy == 0 ? 0 : (hy > TS ? 6 : 3)) +
                             (hx == 0 ? 0 : (hx > TS ? 2 : 1)));
    }
    // the thread's voxel: a warp's 32 voxels share no plane of the tile with more than a few of one another
    const int q4 = (warp + 5 * (lane >> 2) + 3 * (lane & 3)) & 15;
    const int lx = (q4 & 7) + 1, ly = 2 * (lane & 3) + (q4 >> 3) + 1, lz = (lane >> 2) + 1;
    const int me = (lz * HS + ly) * HS + lx;
    // lane -> neighbour (26 of the 32 lanes)
    int off = 0, kind = 0;
    if (lane < 26) {
        const int c = lane < 13 ? lane : lane + 1;  // skip the centre of the 3x3x3 cube
        const int dz = c / 9 - 1, dy = (c / 3) % 3 - 1, dx = c % 3 - 1;
        off = (dz * HS + dy) * HS + dx;
        kind = (dz != 0) + (dy != 0) + (dx != 0) - 1;
    }
    // everything above runs beside the round before (programmatic launch)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int n = T.counts[round % 3];
    const u64 upto = (u64)__double_as_longlong(__dadd_rn(__hiloint2double((int)T.first[round % 3], -1), window));
    if (blockIdx.x == 0 && tid == 0) {
        T.counts[(round + 2) % 3] = 0;
        T.first[(round + 2) % 3] = NONE;
        if (n > 0) T.counts[3] = round + 1;
    }
    for (int it = blockIdx.x; it < n; it += gridDim.x) {
        const int tile = T.list[(size_t)(round & 1) * T.cap + it];
        const int tx0 = (tile % ntx) * TS, ty0 = ((tile / ntx) % nty) * TS, tz0 = (tile / (ntx * nty)) * TS;
        __syncthreads();  // the previous tile's reads of the shared arrays are done
        if (tid == 0) {
            atomicAnd(&T.flags[tile >> 2], ~(1u << (8 * (tile & 3) + (round & 1))));
            s_mark = 0;
            s_first = NONE;
        }
        // stage tile + halo
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int i = tid + q * CA_THREADS;
            if (i >= HCELLS) break;
            const int hx = i % HS, hy = (i / HS) % HS, hz = i / (HS * HS);
            const int gx = tx0 + hx - 1, gy = ty0 + hy - 1, gz = tz0 + hz - 1;
            u64 e = 2 * INF_BITS;
            uint8_t l = 0;
            if (gx >= 0 && gx < nx && gy >= 0 && gy < ny && gz >= 0 && gz < nz) {
                const size_t g = ((size_t)gz * ny + gy) * nx + gx;
                l = layer_id(layers[g]);
                const u64 v = at[g];
                if (l) e = v;
            }
            s_e[i] = e;
            s_l[i] = l;
        }
        __syncthreads();
        const u64 orig = s_e[me];
        const int myl = s_l[me];
        u64 offered = orig & 1 ? ~0ULL : orig >> 1;  // the time that the voxel has offered
        uint32_t mark = 0, first = NONE;
        bool sent = false;  // an offer of the last step within the tile and the horizon
        // settling steps: every voxel with a pending time up to the horizon offers it; they end, as times only fall
        for (;;) {
            const u64 mine = s_e[me] >> 1;
            const bool sel = mine != offered && mine <= upto;
            // an offer made in the last step may have come too late for its target's read
            if (!__syncthreads_or(sel || sent)) break;
            sent = false;
            if (sel) offered = mine;
            for (unsigned b = __ballot_sync(0xffffffffu, sel); b; b &= b - 1) {
                const int src = __ffs(b) - 1;
                const u64 t = __shfl_sync(0xffffffffu, mine, src);
                const int v = __shfl_sync(0xffffffffu, me, src) + off, lu = __shfl_sync(0xffffffffu, myl, src);
                const int lv = s_l[v];
                const u64 ev = s_e[v];
                if (lane < 26 && lv && 2 * t < ev) {
                    const u64 c = (u64)__double_as_longlong(__dadd_rn(
                        __longlong_as_double((long long)t), __ldg(lag + ((size_t)lu * nl1 + lv) * 3 + kind)));
                    const u64 ce = 2 * c + 1;
                    if (ce < ev && ce < atomicMin(&s_e[v], ce)) {
                        const int dir = s_dir[v];
                        if (dir == 13) {
                            sent = sent || c <= upto;
                        } else {
                            const int hx = v % HS, hy = (v / HS) % HS, hz = v / (HS * HS);
                            atomicMin(&at[((size_t)(tz0 + hz - 1) * ny + (ty0 + hy - 1)) * nx + (tx0 + hx - 1)], ce);
                            mark |= 1u << dir;
                            first = min(first, (uint32_t)(c >> 32));
                        }
                    }
                }
            }
        }
        // write back (a neighbour tile's block may have offered an earlier time meanwhile, and then has
        // queued this tile); a tile with waiting voxels stays queued
        const u64 mine = s_e[me] >> 1;
        if (myl) {
            const u64 e = 2 * mine + (mine != offered);
            if (e != orig) atomicMin(&at[((size_t)(tz0 + lz - 1) * ny + (ty0 + ly - 1)) * nx + (tx0 + lx - 1)], e);
            if (mine != offered) {
                mark |= 1u << 13;
                first = min(first, (uint32_t)(mine >> 32));
            }
        }
        mark = __reduce_or_sync(0xffffffffu, mark);
        first = __reduce_min_sync(0xffffffffu, first);
        if (lane == 0 && mark) {
            atomicOr(&s_mark, mark);
            atomicMin(&s_first, first);
        }
        __syncthreads();
        if (tid < 27 && (s_mark >> tid) & 1u) {
            const int tz = tz0 / TS + tid / 9 - 1, ty = ty0 / TS + (tid / 3) % 3 - 1, tx = tx0 / TS + tid % 3 - 1;
            tile_append(T, (tz * nty + ty) * ntx + tx, round + 1);  // inside the grid: it holds a voxel
        }
        if (tid == 32 && s_mark) atomicMin(&T.first[(round + 1) % 3], s_first);
    }
}

// The caller's grid: layers stripped of the stimulus sign, the header, and with `at` the entries before
// round 0 and the stimulus tiles in its list.
__global__ void __launch_bounds__(256) k_ca_grid(int nz, int ny, int nx, int nty, int ntx, const int32_t *__restrict__ grid,
                                                 uint8_t *__restrict__ lay, GridHeader *__restrict__ hdr,
                                                 u64 *__restrict__ at, TileLists T) {
    __shared__ uint32_t s_present[8];
    if (threadIdx.x < 8) s_present[threadIdx.x] = 0;
    __syncthreads();
    const size_t n = (size_t)nz * ny * nx;
    int bad = 0, starts = 0, vox = 0, last = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int32_t v = grid[i];
        // widened before the negation, so that INT32_MIN is rejected rather than overflowing
        const int64_t a = v < 0 ? -(int64_t)v : (int64_t)v;
        if (a > 254) {
            bad = 1;
            continue;
        }
        lay[i] = (uint8_t)a;
        vox += a != 0;
        if (a && (int)a != last) {
            last = (int)a;
            atomicOr(&s_present[last >> 5], 1u << (last & 31));
        }
        if (v < 0) ++starts;
        if (at) {
            at[i] = a ? (v < 0 ? 2 * 0x3ff0000000000000ULL + 1 : 2 * INF_BITS) : 0;
            if (v < 0) {
                const int x = (int)(i % nx), y = (int)((i / nx) % ny), z = (int)(i / ((size_t)nx * ny));
                tile_append(T, ((z / TS) * nty + (y / TS)) * ntx + (x / TS), 0);
            }
        }
    }
    starts = __reduce_add_sync(0xffffffffu, starts);
    vox = __reduce_add_sync(0xffffffffu, vox);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
        if (starts) atomicAdd(&hdr->nstart, starts);
        if (vox) atomicAdd(&hdr->nvox, vox);
        if (bad) atomicOr(&hdr->bad, 1);
    }
    __syncthreads();
    if (threadIdx.x < 8 && s_present[threadIdx.x]) atomicOr(&hdr->present[threadIdx.x], s_present[threadIdx.x]);
}

// entries -> times; unreachable voxels keep excitationDelay 0.  Queued behind every chunk of rounds, it
// leaves the entries alone while tiles are left: the host's look at the counters then is the call's last
// wait (launched after that look it cost 16 us more).
__global__ void k_ca_finish(size_t n, u64 *__restrict__ at, const int32_t *__restrict__ left) {
    if (*left) return;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const u64 t = at[i] >> 1;
        at[i] = t == INF_BITS ? 0 : t;
    }
}

}  // namespace

// The lists over `ctrl` (CA_CTRL_WORDS words), and its words before round 0, when the stimulus tiles are yet
// to be appended: the earliest pending time is the stimulus', 1.0.
static TileLists tile_lists(int32_t *ctrl, uint32_t *flags, int32_t *list, int cap) {
    TileLists T;
    T.counts = ctrl;
    T.first = reinterpret_cast<uint32_t *>(ctrl + 4);
    T.flags = flags;
    T.list = list;
    T.cap = cap;
    return T;
}
static const int32_t FIRST_ROUND[CA_CTRL_WORDS] = {0, 0, 0, 0, 0x3ff00000 /* high word of 1.0 */, -1, -1};

// The width of a round, 5 of the largest lag between present layers: in a narrower one the rounds' fixed
// cost shows (launch, staging, write-back), in a wider one the wave leaves the tile and its successors
// wait.  160^3 heart with lags 1, 2, 2 ms (a whole call): 1.06, 1.07, 1.07, 1.10, 1.11, 1.16 and 1.71 ms at 2.5, 4, 5,
// 6, 8, 16 and without an end, repeats within 2 %; 256^3, ten layers: 2.42, 2.45, 2.47, 2.51, 2.58, 2.91, 6.1 ms.
static double round_window(const double *lag, int nl1, const char *present) {
    double hi = 0.0;
    for (int a = 1; a < nl1; ++a)
        for (int b = 1; b < nl1; ++b)
            if (present[a] && present[b]) hi = std::max(hi, lag[((size_t)a * nl1 + b) * 3]);
    return 5.0 * hi;
}

// Queues rounds in chunks until a round has no tile; the host reads the counts once per chunk (rounds
// after convergence find an empty list).  `read` copies the four counters to the host, waiting.
// A chunk's end costs some 22 us (the copy, the wait, the next launch without its predecessor to overlap), a
// round too many 2.5: the first chunk is as long as hearts of 24 to 256 cells were seen to need, 2.2 to 3.5
// rounds per tile of the longest side (160^3, 49 rounds: five chunks of 12 1.02 ms, one of 50 0.95), but no
// more than 128, and later ones are a quarter of the rounds behind: how many a long strip takes depends on its
// stimuli (8 x 8 x 524,288 cells: 3 rounds with one in every tile, 364 ms behind a first chunk of 163,840,
// 5.3 now; 147,337 rounds with a single one, 2.05 s and 1.99).
template <typename LT, class Read>
static int run_rounds(cudaStream_t s, int nz, int ny, int nx, const LT *layers, const double *lag, int nl1, double w,
                      u64 *at, const TileLists &T, int cap, int sm_count, Read read) {
    const int ntz = (nz + TS - 1) / TS, nty = (ny + TS - 1) / TS, ntx = (nx + TS - 1) / TS;
    cudaLaunchAttribute pdl;
    pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)std::max(1, std::min(ntz * nty * ntx, 3 * std::max(1, sm_count))));
    cfg.blockDim = dim3(CA_THREADS);
    cfg.stream = s;
    cfg.attrs = &pdl;
    cfg.numAttrs = 1;
    constexpr int CHUNK = 12, FIRST_MAX = 128;
    int chunk = std::max(CHUNK, std::min(FIRST_MAX, 5 * std::min(FIRST_MAX, std::max({ntz, nty, ntx})) / 2));
    int32_t h[4];
    for (int r = 0;;) {
        const int end = (int)std::min<int64_t>(cap, (int64_t)r + chunk);
        for (; r < end; ++r) {
            EKG_CUDA(cudaLaunchKernelEx(&cfg, k_ca_round<LT>, r, nz, ny, nx, ntz, nty, ntx, layers, lag, nl1, w, at, T));
        }
        chunk = std::max(CHUNK, r / 4);
        k_ca_finish<<<1024, 256, 0, s>>>((size_t)nz * ny * nx, at, T.counts + r % 3);
        EKG_CUDA(cudaGetLastError());
        read(h);
        if (h[r % 3] == 0) return h[3];
        if (r >= cap) throw Error{EKG_ERR_CA_NOT_CONVERGED, "activation-time relaxation did not converge"};
    }
}

static int tile_count(int nz, int ny, int nx) {
    return ((nz + TS - 1) / TS) * ((ny + TS - 1) / TS) * ((nx + TS - 1) / TS);
}
// scratch: control words, flags, two lists
static TileLists scratch_lists(void *scratch, int ntiles) {
    int32_t *p = static_cast<int32_t *>(scratch);
    const size_t nflag = (size_t)(ntiles + 3) / 4;
    return tile_lists(p, reinterpret_cast<uint32_t *>(p + CA_CTRL_WORDS), p + CA_CTRL_WORDS + nflag, ntiles);
}
size_t ca_scratch_bytes(int nz, int ny, int nx) {
    const size_t nt = (size_t)tile_count(nz, ny, nx);
    return (CA_CTRL_WORDS + (nt + 3) / 4 + 2 * nt) * sizeof(int32_t);
}

void ca_grid(cudaStream_t s, int nz, int ny, int nx, const int32_t *d_grid, uint8_t *d_lay, GridHeader *d_hdr,
             double *d_at, void *scratch) {
    const int nt = tile_count(nz, ny, nx), nty = (ny + TS - 1) / TS, ntx = (nx + TS - 1) / TS;
    const TileLists T = scratch_lists(scratch, nt);
    EKG_CUDA(cudaMemsetAsync(T.flags, 0, (size_t)(nt + 3) / 4 * sizeof(int32_t), s));
    EKG_CUDA(cudaMemsetAsync(d_hdr, 0, sizeof(GridHeader), s));
    // the kernel appends the stimulus tiles
    EKG_CUDA(cudaMemcpyAsync(T.counts, FIRST_ROUND, sizeof(FIRST_ROUND), cudaMemcpyHostToDevice, s));
    k_ca_grid<<<1216, 256, 0, s>>>(nz, ny, nx, nty, ntx, d_grid, d_lay, d_hdr, reinterpret_cast<u64 *>(d_at), T);
    EKG_CUDA(cudaGetLastError());
}

CaResult ca_run(cudaStream_t s, int nz, int ny, int nx, const uint8_t *d_layers, const std::vector<double> &lag_h,
                const std::vector<char> &present, int nl1, const double *d_lag, double *d_at, void *scratch,
                int round_cap, int sm_count) {
    CaResult res;
    const size_t n = (size_t)nz * ny * nx;
    const TileLists T = scratch_lists(scratch, tile_count(nz, ny, nx));
    struct Events {
        cudaEvent_t a = nullptr, b = nullptr;
        ~Events() {
            if (a) cudaEventDestroy(a);
            if (b) cudaEventDestroy(b);
        }
    } ev;
    EKG_CUDA(cudaEventCreate(&ev.a));
    EKG_CUDA(cudaEventCreate(&ev.b));
    EKG_CUDA(cudaEventRecord(ev.a, s));
    u64 *entries = reinterpret_cast<u64 *>(d_at);
    // every round settles at least the voxels with the earliest pending time for good
    const int cap = round_cap > 0 ? round_cap : (int)std::min<size_t>(n, INT32_MAX / 2) + 64;
    res.rounds = run_rounds(s, nz, ny, nx, d_layers, d_lag, nl1, round_window(lag_h.data(), nl1, present.data()),
                            entries, T, cap, sm_count, [&](int32_t *h) {
                                EKG_CUDA(cudaMemcpyAsync(h, T.counts, 4 * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
                                EKG_CUDA(cudaStreamSynchronize(s));
                            });
    EKG_CUDA(cudaEventRecord(ev.b, s));
    EKG_CUDA(cudaEventSynchronize(ev.b));
    EKG_CUDA(cudaEventElapsedTime(&res.ms, ev.a, ev.b));
    return res;
}

// ------------------------------------------------------------------ no-allocation entry point
// ekg_activation_noalloc: the same relaxation for callers that cannot allocate device memory
// (for example code running under a memory pool or allocator that forbids new cudaMalloc calls
// after start-up, or inside a host loop that must not touch the allocator).  All scratch lives in
// one file-scope device array, g_noalloc, of fixed size; the caller supplies the layer grid and
// the output as device buffers it already owns.  Every call shares g_noalloc and leaves its last
// contents behind, so the counters and flags are cleared at the start of each call; a host mutex
// serialises callers in this process, and calls whose device work overlaps (for example from
// another thread that bypasses this entry point's lock) would race on the array.
namespace {
constexpr int NOALLOC_MAX_TILES = 65536;  // 8x8x8 tiles, e.g. a 320^3 grid
constexpr int NOALLOC_MAX_LAYER = 31;     // highest layer id (lag table 32 x 32 x 3)
struct NoAllocScratch {
    int32_t list[2][NOALLOC_MAX_TILES];
    uint32_t flag[NOALLOC_MAX_TILES / 4];  // one byte per tile (TileLists)
    int32_t ctrl[CA_CTRL_WORDS];
    int32_t nstart;
    uint32_t layer_mask;
    int32_t bad;
    double lag[(NOALLOC_MAX_LAYER + 1) * (NOALLOC_MAX_LAYER + 1) * 3];
};
static __device__ __align__(256) NoAllocScratch g_noalloc;

// per-device address of g_noalloc (host code may not use the symbol itself as an address)
std::mutex g_noalloc_mu;
NoAllocScratch *g_noalloc_ptr[64] = {nullptr};

// What the host hands over with a launch: a copy of a few words between two kernels takes 4 to 8 us.
struct CtrlWords {
    int32_t v[CA_CTRL_WORDS];
};
constexpr int LAG_WORDS = 432;  // 11 layers; longer tables are copied
struct LagTable {
    int n;
    double v[LAG_WORDS];
};

__global__ void k_na_validate(size_t n, const int32_t *__restrict__ layers, NoAllocScratch *sc, CtrlWords first) {
    if (blockIdx.x == 0 && threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < CA_CTRL_WORDS; ++k) sc->ctrl[k] = first.v[k];
    uint32_t mask = 0;
    int32_t starts = 0, bad = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int32_t v = layers[i];
        // widened before the negation: INT32_MIN is out of range, not a negative shift
        const int64_t a = v < 0 ? -(int64_t)v : (int64_t)v;
        if (a > NOALLOC_MAX_LAYER) bad = 1;
        else mask |= 1u << (uint32_t)a;
        starts += v < 0;
    }
    mask = __reduce_or_sync(0xffffffffu, mask);
    starts = __reduce_add_sync(0xffffffffu, starts);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
        if (mask) atomicOr(&sc->layer_mask, mask);
        if (starts) atomicAdd(&sc->nstart, starts);
        if (bad) atomicOr(&sc->bad, 1);
    }
}

__global__ void k_na_init(int nz, int ny, int nx, int nty, int ntx, const int32_t *__restrict__ layers,
                          u64 *__restrict__ at, TileLists T, const __grid_constant__ LagTable lag, double *__restrict__ d_lag) {
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < lag.n; i += blockDim.x) d_lag[i] = lag.v[i];
    const size_t n = (size_t)nz * ny * nx;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int32_t v = layers[i];
        u64 a = 0;
        if (v < 0) {
            a = 2 * 0x3ff0000000000000ULL + 1;
            const int x = (int)(i % nx), y = (int)((i / nx) % ny), z = (int)(i / ((size_t)nx * ny));
            tile_append(T, ((z / TS) * nty + (y / TS)) * ntx + (x / TS), 0);
        } else if (v > 0) {
            a = 2 * INF_BITS;
        }
        at[i] = a;
    }
}

NoAllocScratch *noalloc_scratch() {
    int dev = 0;
    EKG_CUDA(cudaGetDevice(&dev));
    EKG_CHECK(dev >= 0 && dev < 64, EKG_ERR_DEVICE, "device index out of range");
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        EKG_CUDA(cudaGetSymbolAddress(&p, g_noalloc));
        g_noalloc_ptr[dev] = reinterpret_cast<NoAllocScratch *>(p);
    }
    return g_noalloc_ptr[dev];
}
}  // namespace

}  // namespace ekg

extern "C" int ekg_activation_noalloc(int32_t nz, int32_t ny, int32_t nx, const int32_t *d_layers, int32_t n_transfer,
                                      const double *transfer, double *d_at, int32_t *rounds_out) {
    using namespace ekg;
    return guard([&] {
        EKG_CHECK(d_layers && transfer && d_at && n_transfer >= 1, EKG_ERR_BAD_INPUT, "null argument");
        EKG_CHECK(nz >= 1 && ny >= 1 && nx >= 1, EKG_ERR_BAD_INPUT, "grid extents must be positive");
        const int ntz = (nz + TS - 1) / TS, nty = (ny + TS - 1) / TS, ntx = (nx + TS - 1) / TS;
        const int64_t ntiles = (int64_t)ntz * nty * ntx;
        EKG_CHECK(ntiles <= NOALLOC_MAX_TILES, EKG_ERR_BAD_INPUT,
                  "grid too large for ekg_activation_noalloc: at most 65536 tiles of 8x8x8 cells");
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        NoAllocScratch *sc = noalloc_scratch();
        const size_t n = (size_t)nz * ny * nx;
        cudaStream_t s = 0;
        // clear what must start at zero: flags, counters, layer mask (they are contiguous)
        EKG_CUDA(cudaMemsetAsync(sc->flag, 0, offsetof(NoAllocScratch, lag) - offsetof(NoAllocScratch, flag), s));
        CtrlWords first;
        std::copy(std::begin(FIRST_ROUND), std::end(FIRST_ROUND), first.v);
        k_na_validate<<<1024, 256, 0, s>>>(n, d_layers, sc, first);
        EKG_CUDA(cudaGetLastError());
        struct {
            int32_t nstart;
            uint32_t mask;
            int32_t bad;
        } hdr;
        EKG_CUDA(cudaMemcpy(&hdr, &sc->nstart, sizeof(hdr), cudaMemcpyDeviceToHost));
        EKG_CHECK(!hdr.bad, EKG_ERR_BAD_INPUT, "layer ids must be at most 31 for ekg_activation_noalloc");
        EKG_CHECK(hdr.nstart > 0, EKG_ERR_NO_START, "Could not find starting point for excitation sequence");
        int nl = 0;
        for (int a = 1; a <= NOALLOC_MAX_LAYER; ++a)
            if (hdr.mask & (1u << a)) {
                nl = a;
                if (a >= n_transfer)
                    throw Error{EKG_ERR_TRANSFER, "transfer (conduction) matrix does not define layer " + std::to_string(a)};
            }
        const int nl1 = nl + 1;
        char present[NOALLOC_MAX_LAYER + 1];
        for (int a = 0; a <= NOALLOC_MAX_LAYER; ++a) present[a] = (hdr.mask >> a) & 1u;
        double lag[(NOALLOC_MAX_LAYER + 1) * (NOALLOC_MAX_LAYER + 1) * 3];
        for (int i = 0; i < nl1 * nl1 * 3; ++i) lag[i] = 0.0;
        for (int a = 1; a <= nl; ++a)
            for (int b = 1; b <= nl; ++b) {
                if (!((hdr.mask >> a) & 1u) || !((hdr.mask >> b) & 1u)) continue;
                const double t = transfer[(size_t)a * n_transfer + b];
                EKG_CHECK(t >= 0 && std::isfinite(t), EKG_ERR_BAD_INPUT,
                          "conduction delays between present layers must be finite and non-negative");
                for (int k = 1; k <= 3; ++k) {
                    double l = t;
                    l *= std::sqrt((double)k);
                    lag[((size_t)a * nl1 + b) * 3 + (k - 1)] = l;
                }
            }
        const TileLists T = tile_lists(sc->ctrl, sc->flag, sc->list[0], NOALLOC_MAX_TILES);
        LagTable table;
        table.n = nl1 * nl1 * 3 <= LAG_WORDS ? nl1 * nl1 * 3 : 0;
        std::copy(lag, lag + table.n, table.v);
        if (table.n == 0) EKG_CUDA(cudaMemcpy(sc->lag, lag, (size_t)nl1 * nl1 * 3 * sizeof(double), cudaMemcpyHostToDevice));
        // k_na_init appends the stimulus tiles (k_na_validate has set the words before the first round)
        u64 *entries = reinterpret_cast<u64 *>(d_at);
        k_na_init<<<1024, 256, 0, s>>>(nz, ny, nx, nty, ntx, d_layers, entries, T, table, sc->lag);
        EKG_CUDA(cudaGetLastError());
        int dev = 0, sm_count = 0;
        EKG_CUDA(cudaGetDevice(&dev));
        EKG_CUDA(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev));
        const int rounds = run_rounds(s, nz, ny, nx, d_layers, sc->lag, nl1, round_window(lag, nl1, present), entries, T,
                                      (int)std::min<size_t>(n, INT32_MAX / 2) + 64, sm_count, [&](int32_t *h) {
                                          EKG_CUDA(cudaMemcpy(h, T.counts, 4 * sizeof(int32_t), cudaMemcpyDeviceToHost));
                                      });
        EKG_CUDA(cudaStreamSynchronize(s));
        if (rounds_out) *rounds_out = rounds;
    });
}
