// setup.cu -- the de-duplication part of a heart's set-up on the device.
//
// Simulation::setApIndices (simlib/simulator.cpp:561-621) gives every distinct (layer, activation
// time) pair of the non-empty voxels an AP.  Here the voxels are listed in raster order
// (compaction by a two-level scan), sorted by (layer, activation time) with a stable LSD radix
// sort on 8-bit digits of the time's bit pattern (non-negative doubles order like their bit
// patterns) and then of the layer -- stability keeps raster (cell) order inside an AP -- and the
// runs of equal keys are the APs.  Then the per-AP arrays in the padded per-layer K layout and the
// per-voxel records of the dipole kernels are written by one thread per AP slot / voxel.  The
// results are the arrays a host sort by (layer, time bits, cell) gives, element for element.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "ekg_internal.h"

namespace ekg {

namespace {

constexpr int ST = 256;             // threads per block
constexpr int SITEMS = 8;           // items per thread in the scans
constexpr int STILE = ST * SITEMS;  // scan tile
constexpr unsigned FULL = 0xffffffffu;

// Exclusive scan of one value per thread across the block (fixed order); *total gets the sum.
__device__ __forceinline__ int block_exscan(int v, int *total, int *s_warp) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = lane < ST / 32 ? s_warp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, t, o);
            if (lane >= o) t += y;
        }
        if (lane < ST / 32) s_warp[lane] = t;
    }
    __syncthreads();
    const int r = (w > 0 ? s_warp[w - 1] : 0) + x - v;
    *total = s_warp[ST / 32 - 1];
    __syncthreads();
    return r;
}

// Flag functions: cell c is a voxel; sorted voxel i starts a new (layer, time) run.
struct IsVoxel {
    const uint8_t *lay;
    __device__ int operator()(int64_t c) const { return lay[c] != 0; }
};
struct StartsRun {
    const uint8_t *lay;
    const uint64_t *key;
    __device__ int operator()(int64_t i) const {
        return i == 0 || lay[i] != lay[i - 1] || key[i] != key[i - 1];
    }
};

// Flags per STILE tile: tile sums, then (one block) their exclusive scan, then each tile writes the
// indices of its flagged items to out[] at their ranks.
template <class F>
__global__ void __launch_bounds__(ST) k_tile_counts(F f, int64_t n, int *__restrict__ tsum) {
    __shared__ int s_warp[ST / 32];
    const int64_t base = (int64_t)blockIdx.x * STILE + (int64_t)threadIdx.x * SITEMS;
    int c = 0;
#pragma unroll
    for (int k = 0; k < SITEMS; ++k)
        if (base + k < n) c += f(base + k);
    int total;
    block_exscan(c, &total, s_warp);
    if (threadIdx.x == 0) tsum[blockIdx.x] = total;
}

// exclusive scan of tsum[0..nt) in place by one block; tsum[nt] = total
__global__ void __launch_bounds__(ST) k_scan_counts(int *__restrict__ tsum, int nt) {
    __shared__ int s_warp[ST / 32];
    int carry = 0;
    for (int b = 0; b < nt; b += ST) {
        const int i = b + (int)threadIdx.x;
        const int v = i < nt ? tsum[i] : 0;
        int total;
        const int ex = block_exscan(v, &total, s_warp);
        if (i < nt) tsum[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) tsum[nt] = carry;
}

template <class F>
__global__ void __launch_bounds__(ST) k_compact(F f, int64_t n, const int *__restrict__ tsum, int *__restrict__ out) {
    __shared__ int s_warp[ST / 32];
    const int64_t base = (int64_t)blockIdx.x * STILE + (int64_t)threadIdx.x * SITEMS;
    int flags = 0, c = 0;
#pragma unroll
    for (int k = 0; k < SITEMS; ++k)
        if (base + k < n && f(base + k)) {
            flags |= 1 << k;
            ++c;
        }
    int total;
    int pos = tsum[blockIdx.x] + block_exscan(c, &total, s_warp);
#pragma unroll
    for (int k = 0; k < SITEMS; ++k)
        if (flags & (1 << k)) out[pos++] = (int)(base + k);
}

// ---- stable LSD radix sort of (layer, time bits) with the cell as payload, 8-bit digits
// pass p < 8: byte p of the time bits; pass 8: the layer.  Tiles of RTILE elements.  A pass is bound by its
// three launches and their chains, not by the 26 bytes an element that it moves (160^3, 661,216 voxels:
// 30 us a pass with a tile per 256 elements and a launch for the digits' bases; 21.5, and 18.5 with a pass's
// kernels launched ahead).
constexpr int RITEMS = 4, RTILE = ST * RITEMS;
__device__ __forceinline__ int digit(int pass, uint64_t key, uint8_t lay) {
    return pass < 8 ? (int)((key >> (8 * pass)) & 0xffu) : (int)lay;
}

// The kernels of a pass are launched while their predecessor runs: each lets its successor's blocks take
// the places that it leaves and waits for its own predecessor's results before its first access (none of
// their pointers is __restrict__: a load of data that is declared constant may be moved before the wait).
__device__ __forceinline__ void pass_begin() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

__global__ void __launch_bounds__(ST) k_digit_hist(int pass, int n, const uint64_t *key,
                                                   const uint8_t *lay, int nblk, int *hist) {
    __shared__ int s_h[256];
    s_h[threadIdx.x] = 0;
    pass_begin();
    int d[RITEMS];
#pragma unroll
    for (int k = 0; k < RITEMS; ++k) {
        const int i = blockIdx.x * RTILE + k * ST + threadIdx.x;
        d[k] = i < n ? digit(pass, pass < 8 ? key[i] : 0, pass < 8 ? (uint8_t)0 : lay[i]) : -1;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RITEMS; ++k)
        if (d[k] >= 0) atomicAdd(&s_h[d[k]], 1);
    __syncthreads();
    hist[(size_t)threadIdx.x * nblk + blockIdx.x] = s_h[threadIdx.x];
}

// per digit (block): exclusive scan of its counts over the tiles; totals[d] = the digit's count
__global__ void __launch_bounds__(ST) k_digit_scan(int *hist, int nblk, int *totals) {
    __shared__ int s_warp[ST / 32];
    int *h = hist + (size_t)blockIdx.x * nblk;
    int carry = 0;
    pass_begin();
    for (int b = 0; b < nblk; b += ST) {
        const int i = b + (int)threadIdx.x;
        const int v = i < nblk ? h[i] : 0;
        int total;
        const int ex = block_exscan(v, &total, s_warp);
        if (i < nblk) h[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// rank = the digit's base (every block scans the 256 totals) + the tile's offset for the digit + equal
// digits before it in the tile: a warp takes 32 RITEMS consecutive elements, 32 at a time, with its
// running counts in shared memory and a match mask for the lanes before; then the earlier warps' counts.
__global__ void __launch_bounds__(ST) k_digit_scatter(int pass, int n, const uint64_t *key_in,
                                                      const uint8_t *lay_in, const int *val_in,
                                                      int nblk, const int *hist,
                                                      const int *totals, uint64_t *key_out,
                                                      uint8_t *lay_out, int *val_out) {
    __shared__ int s_cnt[ST / 32][256];
    __shared__ int s_warp[ST / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i0 = blockIdx.x * RTILE + w * (32 * RITEMS) + lane;
    pass_begin();
    uint64_t kv[RITEMS];
    uint8_t lv[RITEMS];
    int vv[RITEMS], rank[RITEMS], dg[RITEMS];
#pragma unroll
    for (int k = 0; k < RITEMS; ++k) {
        const int i = i0 + 32 * k;
        kv[k] = i < n ? key_in[i] : 0;
        lv[k] = i < n ? lay_in[i] : (uint8_t)0;
        vv[k] = i < n ? val_in[i] : 0;
    }
    const int off = hist[(size_t)threadIdx.x * nblk + blockIdx.x];
    int all;
    const int base = block_exscan(totals[threadIdx.x], &all, s_warp);
    for (int k = threadIdx.x; k < (ST / 32) * 256; k += ST) (&s_cnt[0][0])[k] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RITEMS; ++k) {
        const bool valid = i0 + 32 * k < n;
        dg[k] = valid ? digit(pass, kv[k], lv[k]) : 256 + lane;  // invalid lanes match nothing
        const unsigned m = __match_any_sync(FULL, dg[k]);
        const int before = valid ? s_cnt[w][dg[k]] : 0, in = __popc(m & ((1u << lane) - 1u));
        rank[k] = before + in;
        __syncwarp();
        if (valid && in == 0) s_cnt[w][dg[k]] = before + __popc(m);
        __syncwarp();
    }
    __syncthreads();
    int run = base + off;  // thread = digit
#pragma unroll
    for (int k = 0; k < ST / 32; ++k) {
        const int c = s_cnt[k][threadIdx.x];
        s_cnt[k][threadIdx.x] = run;
        run += c;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RITEMS; ++k)
        if (i0 + 32 * k < n) {
            const int pos = s_cnt[w][dg[k]] + rank[k];
            key_out[pos] = kv[k];
            lay_out[pos] = lv[k];
            val_out[pos] = vv[k];
        }
}

__global__ void k_gather_keys(int nv, const int *__restrict__ cell, const double *__restrict__ at,
                              const uint8_t *__restrict__ lay, uint64_t *__restrict__ key, uint8_t *__restrict__ vl) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nv) return;
    const int64_t c = cell[i];
    key[i] = (uint64_t)__double_as_longlong(at[c]);
    vl[i] = lay[c];
}

// out[0] = the number of APs (*na); out[L] = first AP of layer L (APs are ordered by layer; the others keep
// what they held)
__global__ void k_layer_first(const int *__restrict__ na, const int *__restrict__ gstart, const uint8_t *__restrict__ vl,
                              int *__restrict__ out) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x, n = *na;
    if (a == 0) out[0] = n;
    if (a >= n) return;
    const uint8_t L = vl[gstart[a]];
    if (a == 0 || vl[gstart[a - 1]] != L) out[L] = a;
}

// stage order: sort key (most voxels first) and payload of each 32-AP stage
__global__ void k_stage_keys(int nst, uint32_t top, const int64_t *__restrict__ a_vb, uint64_t *__restrict__ key,
                             int *__restrict__ val) {
    const int st = blockIdx.x * blockDim.x + threadIdx.x;
    if (st >= nst) return;
    key[st] = top - (uint32_t)(a_vb[(int64_t)st * 32 + 32] - a_vb[(int64_t)st * 32]);
    val[st] = st;
}

// per padded AP slot p: its layer (present layer k with pbase[k] <= p < pbase[k + 1]), the AP's
// time (FP64 and FP32 hi/lo), layer index and first voxel; padding slots get +inf and the first
// voxel of the layer's next AP
__global__ void k_ap_arrays(int64_t apad, int npl, const int *__restrict__ pl_layer, const int64_t *__restrict__ pbase,
                            const int *__restrict__ pfirst, const int *__restrict__ pcount, int na, int nv,
                            const int *__restrict__ gstart, const int *__restrict__ cell, const double *__restrict__ at_cells,
                            double *__restrict__ at, float2 *__restrict__ at_hilo, int32_t *__restrict__ a_layer,
                            int64_t *__restrict__ a_vb) {
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p == apad) a_vb[apad] = nv;
    if (p >= apad) return;
    int lo = 0, hi = npl - 1;  // last k with pbase[k] <= p
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (pbase[mid] <= p) lo = mid;
        else hi = mid - 1;
    }
    const int64_t j = p - pbase[lo];
    a_layer[p] = pl_layer[lo] - 1;
    if (j < pcount[lo]) {
        const int ap = pfirst[lo] + (int)j;
        const double t = at_cells[cell[gstart[ap]]];
        at[p] = t;
        const float h = __double2float_rn(t);
        at_hilo[p] = make_float2(h, __double2float_rn(t - (double)h));
        a_vb[p] = gstart[ap];
    } else {
        const int next = pfirst[lo] + pcount[lo];
        at[p] = __longlong_as_double(0x7ff0000000000000ll);
        at_hilo[p] = make_float2(__int_as_float(0x7f800000), 0.f);
        a_vb[p] = next < na ? gstart[next] : nv;
    }
}

// per voxel (sorted order): packed position, neighbour masks, bordered position relative to the
// centre with the mask and flags (interior, few absent neighbours, last voxel of its AP), out-offset sum
struct VoxelGeom {
    int nz, ny, nx, nnb;
    int8_t dif[26 * 3];
    uint32_t interior_mask;
    int few_max;
    double cz, cy, cx;  // heart centre; bordered coordinates relative to it, (float)((z + 1) - cz)
};
__global__ void k_voxel_records(int nv, VoxelGeom g, const int *__restrict__ cell, const uint8_t *__restrict__ lay,
                                const uint8_t *__restrict__ vl, const uint64_t *__restrict__ key,
                                int32_t *__restrict__ vzyx, uint32_t *__restrict__ vin, uint32_t *__restrict__ vout,
                                float4 *__restrict__ vpos, float4 *__restrict__ vosum,
                                unsigned long long *__restrict__ n_interior) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool interior = false;
    if (i < nv) {
        const int64_t c = cell[i];
        const int z = (int)(c / ((int64_t)g.ny * g.nx)), y = (int)((c / g.nx) % g.ny), x = (int)(c % g.nx);
        vzyx[i] = (z << 20) | (y << 10) | x;
        uint32_t mi = 0, mo = 0;
        int oz = 0, oy = 0, ox = 0;
        for (int q = 0; q < g.nnb; ++q) {
            const int dz = g.dif[3 * q], dy = g.dif[3 * q + 1], dx = g.dif[3 * q + 2];
            int z2 = z + dz, y2 = y + dy, x2 = x + dx;
            if (z2 >= 0 && z2 < g.nz && y2 >= 0 && y2 < g.ny && x2 >= 0 && x2 < g.nx &&
                lay[((int64_t)z2 * g.ny + y2) * g.nx + x2])
                mi |= 1u << q;
            z2 = z - dz;
            y2 = y - dy;
            x2 = x - dx;
            if (z2 >= 0 && z2 < g.nz && y2 >= 0 && y2 < g.ny && x2 >= 0 && x2 < g.nx &&
                lay[((int64_t)z2 * g.ny + y2) * g.nx + x2]) {
                mo |= 1u << q;
                oz += dz;
                oy += dy;
                ox += dx;
            }
        }
        vin[i] = mi;
        vout[i] = mo;
        uint32_t mbits = mi;
        if (g.interior_mask && mi == g.interior_mask && oz == 0 && oy == 0 && ox == 0) {
            mbits |= 1u << 31;
            interior = true;
        } else if (g.interior_mask && __popc(g.interior_mask & ~mi) <= g.few_max) {
            mbits |= 1u << 29;
        }
        const bool ends = i == nv - 1 || vl[i + 1] != vl[i] || key[i + 1] != key[i];
        if (ends) mbits |= 1u << 30;
        vpos[i] = make_float4((float)((double)(z + 1) - g.cz), (float)((double)(y + 1) - g.cy),
                              (float)((double)(x + 1) - g.cx), __uint_as_float(mbits));
        vosum[i] = make_float4((float)oz, (float)oy, (float)ox, mo ? 1.f : 0.f);
    }
    const unsigned b = __ballot_sync(FULL, interior);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(n_interior, (unsigned long long)__popc(b));
}

}  // namespace

// Sorts n (key, layer, payload) triples by the digit passes listed; the pointers are left at the sorted
// buffers (first) and the other ones.
static void sort_passes(cudaStream_t s, int n, int first, int passes, uint64_t *&key, uint64_t *&key2, uint8_t *&lay,
                        uint8_t *&lay2, int *&val, int *&val2, int *hist, int *totals) {
    const int nblk = (n + RTILE - 1) / RTILE;
    cudaLaunchAttribute pdl;
    pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(ST);
    cfg.stream = s;
    cfg.attrs = &pdl;
    cfg.numAttrs = 1;
    auto go = [&](auto kern, int blocks, auto... args) {
        cfg.gridDim = dim3((unsigned)blocks);
        EKG_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
    };
    for (int pass = first; pass < first + passes; ++pass) {
        go(k_digit_hist, nblk, pass, n, (const uint64_t *)key, (const uint8_t *)lay, nblk, hist);
        go(k_digit_scan, 256, hist, nblk, totals);
        go(k_digit_scatter, nblk, pass, n, (const uint64_t *)key, (const uint8_t *)lay, (const int *)val, nblk,
           (const int *)hist, (const int *)totals, key2, lay2, val2);
        std::swap(key, key2);
        std::swap(lay, lay2);
        std::swap(val, val2);
    }
}

// elements the sort's buffers hold: the voxels, or the stages of the padded APs
static size_t sort_capacity(int64_t nvox) { return (size_t)std::max<int64_t>(nvox, nvox / 32 + 2 * 256 + 2); }

size_t setup_scratch_bytes(int64_t n_cells, int64_t nvox) {
    const size_t m = sort_capacity(nvox), tiles = (size_t)(n_cells + STILE - 1) / STILE + 1;
    return 2 * (Arena::part(m * 8) + Arena::part(m) + Arena::part(m * 4)) + Arena::part((m + 1) * 4) +
           Arena::part((m + RTILE - 1) / RTILE * 256 * 4) + Arena::part(256 * 4) + Arena::part(tiles * 4) +
           Arena::part(257 * 4) + Arena::part(8);
}

void setup_voxels_device(cudaStream_t s, int nz, int ny, int nx, const uint8_t *d_lay, const double *d_at_cells,
                         int nl, int64_t nvox, Arena &scratch, DedupResult &r) {
    const int64_t n = (int64_t)nz * ny * nx;
    const int nv = (int)nvox;
    const size_t m = sort_capacity(nvox);
    r.key = scratch.take<uint64_t>(m);
    r.key2 = scratch.take<uint64_t>(m);
    r.vl = scratch.take<uint8_t>(m);
    r.vl2 = scratch.take<uint8_t>(m);
    r.cell = scratch.take<int>(m);
    r.cell2 = scratch.take<int>(m);
    r.gstart = scratch.take<int>(m + 1);
    r.hist = scratch.take<int>((m + RTILE - 1) / RTILE * 256);
    r.totals = scratch.take<int>(256);
    r.tsum = scratch.take<int>((size_t)(n + STILE - 1) / STILE + 1);
    int *info = scratch.take<int>(257);
    r.n_interior = scratch.take<unsigned long long>(1);
    r.nvox = nv;
    // 1. voxels in raster order
    const int nt = (int)((n + STILE - 1) / STILE);
    k_tile_counts<<<nt, ST, 0, s>>>(IsVoxel{d_lay}, n, r.tsum);
    k_scan_counts<<<1, ST, 0, s>>>(r.tsum, nt);
    k_compact<<<nt, ST, 0, s>>>(IsVoxel{d_lay}, n, r.tsum, r.cell);
    // 2. stable radix sort by (layer, time bits); payload = cell
    k_gather_keys<<<(nv + 255) / 256, 256, 0, s>>>(nv, r.cell, d_at_cells, d_lay, r.key, r.vl);
    EKG_CUDA(cudaGetLastError());
    sort_passes(s, nv, 0, 9, r.key, r.key2, r.vl, r.vl2, r.cell, r.cell2, r.hist, r.totals);
    // 3. runs of equal (layer, time): the APs
    const int nt2 = (nv + STILE - 1) / STILE;
    k_tile_counts<<<nt2, ST, 0, s>>>(StartsRun{r.vl, r.key}, nv, r.tsum);
    k_scan_counts<<<1, ST, 0, s>>>(r.tsum, nt2);
    k_compact<<<nt2, ST, 0, s>>>(StartsRun{r.vl, r.key}, nv, r.tsum, r.gstart);
    // 4. their number and the first one of each layer
    EKG_CUDA(cudaMemsetAsync(info, 0xff, 257 * sizeof(int), s));
    k_layer_first<<<(nv + 255) / 256, 256, 0, s>>>(r.tsum + nt2, r.gstart, r.vl, info);
    EKG_CUDA(cudaGetLastError());
    int lf[257];
    EKG_CUDA(cudaMemcpyAsync(lf, info, sizeof(lf), cudaMemcpyDeviceToHost, s));
    EKG_CUDA(cudaStreamSynchronize(s));
    const int na = lf[0];
    r.naps = na;
    // present layers in order with their AP ranges and padded (multiple of 64) bases
    r.pl_layer.clear();
    r.pfirst.clear();
    r.pcount.clear();
    r.pbase.clear();
    int64_t pad = 0;
    for (int L = 1; L <= nl; ++L)
        if (lf[L] >= 0) {
            int next = na;
            for (int L2 = L + 1; L2 <= nl; ++L2)
                if (lf[L2] >= 0) {
                    next = lf[L2];
                    break;
                }
            r.pl_layer.push_back(L);
            r.pfirst.push_back(lf[L]);
            r.pcount.push_back(next - lf[L]);
            r.pbase.push_back(pad);
            pad += (int64_t)(next - lf[L] + 63) / 64 * 64;
        }
    r.apad = pad;
}

// bases first (8 bytes), then layers, first APs, counts
size_t setup_ap_tables(const DedupResult &r, uint8_t *host) {
    const size_t npl = r.pl_layer.size();
    if (host) {
        std::memcpy(host, r.pbase.data(), npl * 8);
        std::memcpy(host + npl * 8, r.pl_layer.data(), npl * 4);
        std::memcpy(host + npl * 12, r.pfirst.data(), npl * 4);
        std::memcpy(host + npl * 16, r.pcount.data(), npl * 4);
    }
    return npl * 20;
}

void setup_ap_arrays_device(cudaStream_t s, const DedupResult &r, const uint8_t *d_tables, const double *d_at_cells,
                            double *at, float2 *at_hilo, int32_t *a_layer, int64_t *a_vb) {
    const size_t npl = r.pl_layer.size();
    const int64_t slots = r.apad + 1;
    k_ap_arrays<<<(unsigned)((slots + 255) / 256), 256, 0, s>>>(
        r.apad, (int)npl, reinterpret_cast<const int *>(d_tables + npl * 8), reinterpret_cast<const int64_t *>(d_tables),
        reinterpret_cast<const int *>(d_tables + npl * 12), reinterpret_cast<const int *>(d_tables + npl * 16), (int)r.naps,
        (int)r.nvox, r.gstart, r.cell, d_at_cells, at, at_hilo, a_layer, a_vb);
    EKG_CUDA(cudaGetLastError());
}

void setup_voxel_records_device(cudaStream_t s, const DedupResult &r, int nz, int ny, int nx, const uint8_t *d_lay,
                                const HeartDev &D, int few_max, int32_t *vzyx, uint32_t *vin, uint32_t *vout,
                                float4 *vpos, float4 *vosum) {
    VoxelGeom g;
    g.nz = nz;
    g.ny = ny;
    g.nx = nx;
    g.nnb = D.nnb;
    for (int i = 0; i < 26 * 3; ++i) g.dif[i] = D.nb_dif[i];
    g.interior_mask = D.interior_mask;
    g.few_max = few_max;
    g.cz = D.centre[0];
    g.cy = D.centre[1];
    g.cx = D.centre[2];
    EKG_CUDA(cudaMemsetAsync(r.n_interior, 0, sizeof(unsigned long long), s));
    const int nv = (int)r.nvox;
    k_voxel_records<<<(nv + 255) / 256, 256, 0, s>>>(nv, g, r.cell, d_lay, r.vl, r.key, vzyx, vin, vout, vpos, vosum,
                                                     r.n_interior);
    EKG_CUDA(cudaGetLastError());
}

// Keys top - voxels ascend as the voxel counts descend; the sort is stable, so ties keep their index
// order.  As many 8-bit digits as a count can have.
void setup_stage_order_device(cudaStream_t s, DedupResult &r, const int64_t *a_vox_begin, int32_t *stage_order) {
    const int nst = (int)(r.apad / 32);
    if (nst <= 0) return;
    int digits = 1;
    while (digits < 4 && (r.nvox >> (8 * digits))) ++digits;
    const uint32_t top = digits == 4 ? 0xffffffffu : (1u << (8 * digits)) - 1u;
    k_stage_keys<<<(nst + 255) / 256, 256, 0, s>>>(nst, top, a_vox_begin, r.key, r.cell);
    EKG_CUDA(cudaGetLastError());
    sort_passes(s, nst, 0, digits, r.key, r.key2, r.vl, r.vl2, r.cell, r.cell2, r.hist, r.totals);
    EKG_CUDA(cudaMemcpyAsync(stage_order, r.cell, (size_t)nst * 4, cudaMemcpyDeviceToDevice, s));
}

// ------------------------------------------------------------------ stage bounding boxes
// Block per 32-AP stage: the lowest and highest voxel position over the stage's voxels, so that the
// operand kernel can tell for a whole stage whether every voxel is far from a lead.
__global__ void k_stage_boxes(int64_t nst, const int64_t *__restrict__ a_vox_begin, const float4 *__restrict__ vox_pos,
                              float4 *__restrict__ box) {
    __shared__ float red[6][4];
    const int64_t st = blockIdx.x;
    const int64_t v0 = a_vox_begin[st * 32], v1 = a_vox_begin[st * 32 + 32];
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int64_t v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
        const float4 p = vox_pos[v];
        lo[0] = fminf(lo[0], p.x);
        lo[1] = fminf(lo[1], p.y);
        lo[2] = fminf(lo[2], p.z);
        hi[0] = fmaxf(hi[0], p.x);
        hi[1] = fmaxf(hi[1], p.y);
        hi[2] = fmaxf(hi[2], p.z);
    }
    for (int o = 16; o > 0; o >>= 1)
        for (int k = 0; k < 3; ++k) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 3; ++k) {
            red[k][w] = lo[k];
            red[3 + k][w] = hi[k];
        }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int j = 1; j < (int)(blockDim.x >> 5); ++j)
            for (int k = 0; k < 3; ++k) {
                red[k][0] = fminf(red[k][0], red[k][j]);
                red[3 + k][0] = fmaxf(red[3 + k][0], red[3 + k][j]);
            }
        box[2 * st] = make_float4(red[0][0], red[1][0], red[2][0], 0.f);
        box[2 * st + 1] = make_float4(red[3][0], red[4][0], red[5][0], 0.f);
    }
}

void setup_stage_boxes_device(cudaStream_t s, int64_t apad, const int64_t *a_vox_begin, const float4 *vox_pos,
                              float4 *stage_box) {
    const int64_t nst = apad / 32;
    if (nst <= 0) return;
    k_stage_boxes<<<(unsigned)nst, 128, 0, s>>>(nst, a_vox_begin, vox_pos, stage_box);
    EKG_CUDA(cudaGetLastError());
}

}  // namespace ekg
