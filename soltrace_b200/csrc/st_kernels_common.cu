// Precision-independent kernels: the grid probe's pre-test, scans, ordered compaction and
// counting sort of the probe's hits, the run-state update.
#define ST_COMMON_KERNELS
#include <algorithm>
#include "st_launch.h"
#include "st_trace_impl.cuh"

namespace stb {
void launch_sun_candidates(const SceneDev &S, uint64_t s0, uint32_t n, const ProbeOut &o, const RunState *rs,
                           cudaStream_t st) {
    const uint32_t nblocks = (n + kCandRays - 1) / kCandRays;
    cudaMemsetAsync(o.cand_count, 0, sizeof(uint32_t), st);
    k_sun_candidates<<<nblocks, kProbeBlock, 0, st>>>(S, s0, n, o, rs);
}
bool launch_sun_probe_flat(const SceneDev &S, uint64_t s0, uint32_t n, const ProbeOut &o, const RunState *rs,
                           cudaStream_t st) {
    // outputs a caller without room for the undecided rays (or with one word per ray) asks for
    // come from the general grid probe
    if (!S.sun.exact_flat || !S.stages[0].flat_only || !o.amb || !o.cand_el || !o.hit_mask || o.hit_elem) return false;
    constexpr int kWarps = kFlatBlock / 32 * kFlatWarpBytes, kMost = kWarps + kMaxOccWords * int(sizeof(uint32_t));
    if (S.sun.occ_words > kMaxOccWords) return false;
    // the limit belongs to the kernel on its device, for every thread: always the largest bitmap's, so
    // that a thread setting it never lowers it under another's launch
    if (cudaFuncSetAttribute(k_sun_probe_flat, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost) != cudaSuccess) {
        cudaGetLastError();  // not an error of the run, which takes the general grid probe
        return false;
    }
    const int smem = kWarps + S.sun.occ_words * int(sizeof(uint32_t));
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaMemsetAsync(o.cand_count, 0, sizeof(uint32_t), st);
    cudaMemsetAsync(o.amb_count, 0, sizeof(uint32_t), st);
    FlatKeys keys;
    for (uint32_t r = 0; r < 7; ++r) {
        keys.k0[r] = S.seed + (r + 3) * 0x9E3779B9u;
        keys.k1[r] = 0x50C7A5E1u + (r + 3) * 0xBB67AE85u;
    }
    // persistent grid; fewer blocks where each warp would get less than one unit of kProbeBlock rays
    const uint32_t blocks = std::max(1u, (n + kFlatBlock * 8 - 1) / (kFlatBlock * 8));
    k_sun_probe_flat<<<std::min<uint32_t>(blocks, uint32_t(2 * sms)), kFlatBlock, smem, st>>>(S, keys, s0, n, o, rs);
    return true;
}
void launch_offsets(const uint32_t *counts, uint32_t nb, uint32_t *offsets, uint32_t *total, cudaStream_t st) {
    k_offsets<<<1, 1024, 0, st>>>(counts, nb, offsets, total);
}
int launch_scan(const uint32_t *counts, uint32_t nb, uint32_t *offsets, uint32_t *total, uint32_t *parts,
                cudaStream_t st) {
    if (nb <= kScanOneBlock) {
        k_offsets<<<1, 1024, 0, st>>>(counts, nb, offsets, total);
        return 1;
    }
    const uint32_t chunks = std::max(1u, (nb + kScanChunk - 1) / kScanChunk);
    k_scan_parts<<<chunks, kScanBlock, 0, st>>>(counts, nb, parts);
    k_scan_chunks<<<chunks, kScanBlock, 0, st>>>(counts, nb, parts, offsets, total);
    return 2;
}
// chunk scans from the scanned chunk sums (k_scan_chunks with the sum of the chunks before
// each read instead of added up)
__global__ void __launch_bounds__(kScanBlock) k_scan_apply(const uint32_t *counts, uint32_t nb,
                                                           const uint32_t *part_off, uint32_t *offsets) {
    constexpr int kPer = kScanChunk / kScanBlock;
    __shared__ uint32_t wsum[kScanBlock / 32];
    const uint32_t i0 = blockIdx.x * kScanChunk + threadIdx.x * kPer;
    uint32_t v[kPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        v[k] = (i0 + k < nb) ? counts[i0 + k] : 0u;
        sum += v[k];
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    uint32_t run = part_off[blockIdx.x] + x - sum;
    for (int k = 0; k < w; ++k) run += wsum[k];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        if (i0 + k < nb) offsets[i0 + k] = run;
        run += v[k];
    }
}
void launch_scan_large(const uint32_t *counts, uint32_t nb, uint32_t *offsets, uint32_t *total, uint32_t *parts,
                       uint32_t *parts2, cudaStream_t st) {
    const uint32_t chunks = std::max(1u, (nb + kScanChunk - 1) / kScanChunk);
    k_scan_parts<<<chunks, kScanBlock, 0, st>>>(counts, nb, parts);
    // the chunk sums scanned in place (parts has one spare entry beyond the chunks)
    launch_scan(parts, chunks, parts, total, parts2, st);
    k_scan_apply<<<chunks, kScanBlock, 0, st>>>(counts, nb, parts, offsets);
}

__device__ __forceinline__ bool rec_key(const RecOrder &o, const RecordDev &r, int &s) {
    s = r.stage - 1;
    if (s < 0 || s >= o.nst) return false;
    if (o.drop_later && s >= 1) return false;  // raytrace.cpp:786-797
    if (s >= 1 && r.element == 0 && o.tt_drop[s] != 0 && r.raynum == o.tt_drop[s]) return false;  // 810-811
    return true;
}
__global__ void __launch_bounds__(256) k_rec_count(const RecOrder o) {
    __shared__ unsigned long long per[kMaxStages];
    if (threadIdx.x < kMaxStages) per[threadIdx.x] = 0;
    __syncthreads();
    for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < o.n; i += gridDim.x * 256ull) {
        const RecordDev &r = o.recs[i];
        int s;
        if (!rec_key(o, r, s)) continue;
        if (r.raynum > o.rb) {
            atomicOr(o.bad, 1u);
            continue;
        }
        atomicAdd(&o.key[size_t(s) * (o.rb + 1) + r.raynum], 1u);
        atomicAdd(&per[s], 1ull);
    }
    __syncthreads();
    if (threadIdx.x < o.nst && per[threadIdx.x]) atomicAdd(&o.stage_count[threadIdx.x], per[threadIdx.x]);
}
__global__ void __launch_bounds__(256) k_rec_scatter(const RecOrder o) {
    for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < o.n; i += gridDim.x * 256ull) {
        const RecordDev r = o.recs[i];
        int s;
        if (!rec_key(o, r, s) || r.raynum > o.rb) continue;
        const size_t k0 = size_t(s) * (o.rb + 1);
        // place in the stage's (ray number, hit index) order; the hit indices of a key are 0..m-1
        const uint32_t li = o.key[k0 + r.raynum] + r.seq - o.key[k0];
        int lo = o.run_seg[s], hi = o.run_seg[s + 1] - 1;  // last run starting at or before li
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (o.run_src[mid] <= li)
                lo = mid;
            else
                hi = mid - 1;
        }
        const unsigned long long d = o.run_dst[lo] + (li - o.run_src[lo]);
        if (d >= o.total) {
            atomicOr(o.bad, 2u);
            continue;
        }
        for (int q = 0; q < 3; ++q) {
            o.col_d[q * o.total + d] = r.pos[q];
            o.col_d[(3 + q) * o.total + d] = r.cos[q];
        }
        o.col_i[d] = r.element;
        o.col_i[o.total + d] = r.stage;
        o.col_i[2 * o.total + d] = int(r.raynum);
    }
}
static uint32_t rec_blocks(unsigned long long n) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return uint32_t(std::max<unsigned long long>(1, std::min<unsigned long long>((n + 255) / 256, 8ull * sms)));
}
void launch_rec_count(const RecOrder &o, cudaStream_t st) { k_rec_count<<<rec_blocks(o.n), 256, 0, st>>>(o); }
void launch_rec_scatter(const RecOrder &o, cudaStream_t st) { k_rec_scatter<<<rec_blocks(o.n), 256, 0, st>>>(o); }

__global__ void __launch_bounds__(256) k_set_rotations(ElemRec *el, uint32_t n, const double *rot) {
    const uint32_t i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
#pragma unroll
    for (int q = 0; q < 9; ++q) el[i].R[q] = rot[size_t(i) * 9 + q];
}
void launch_set_rotations(ElemRec *el, uint32_t n, const double *rot, cudaStream_t st) {
    if (n) k_set_rotations<<<(n + 255) / 256, 256, 0, st>>>(el, n, rot);
}

// ------------------------------------------------------------------------------------
// Sun-plane grids of batched positions (PosGrid): one thread per position and element projects
// the footprint, counts it into the cells it reaches and marks the bitmap; after the scan of the
// counts it lists itself there, and k_pos_entries puts a cell's entries in ascending element order and
// writes them out.  A host core took 5 to 7 ms for one position of 2,000
// heliostats, and its 3.4 MB of tables crossed PCIe; 24 positions take 0.3 ms here.  Every test is
// sun_setup's, with its margins (which also cover another rounding of the same expressions).
// ------------------------------------------------------------------------------------
// whether element f may be hit from cell (gx, gy); one function for the count and the fill, so
// that both list the same cells
__device__ __noinline__ bool pos_cell_reached(const PosGrid &g, const PosFoot &f, int gx, int gy) {
    const double ax = g.x0 + gx * g.cell, bx = ax + g.cell, ay = g.y0 + gy * g.cell, by = ay + g.cell;
    const double dx = fmax(fmax(ax - f.cx, 0.0), f.cx - bx), dy = fmax(fmax(ay - f.cy, 0.0), f.cy - by);
    if (dx * dx + dy * dy > f.pad * f.pad) return false;
    const double qx = 0.5 * (ax + bx) - f.disc.x, qy = 0.5 * (ay + by) - f.disc.y;
    const double h = 0.5 * g.cell + 2.0 * g.eps + 4e-7 * (fabs(qx) + fabs(qy) + g.box_ext);
    return fabs(f.par.x * qx + f.par.y * qy) <= 1.0 + 1e-5 + (fabs(f.par.x) + fabs(f.par.y)) * h &&
           fabs(f.par.z * qx + f.par.w * qy) <= 1.0 + 1e-5 + (fabs(f.par.z) + fabs(f.par.w)) * h;
}
__device__ __forceinline__ void rotate(const double *R, const double *v, double o[3]) {
    for (int q = 0; q < 3; ++q) o[q] = R[3 * q] * v[0] + R[3 * q + 1] * v[1] + R[3 * q + 2] * v[2];
}
__global__ void __launch_bounds__(128) k_pos_footprints(const PosGridBuild b) {
    const int j = blockIdx.x * 128 + threadIdx.x;
    if (j >= b.n_elem) return;
    const PosGrid &g = b.grids[blockIdx.y];
    const ElemRec &e = g.elems[b.first_elem + j];
    PosFoot f{};
    f.x0 = 0;
    f.x1 = -1;
    if (e.enabled && 0.0 <= e.zap && e.ap[0] >= 0.0 && e.ap[1] >= 0.0) {  // others accept no hit
        double c[3], a[3], bb[3], n[3], ax3[3], ay3[3], nz3[3];
        const double hx = e.ap[0] / 2.0, hy = e.ap[1] / 2.0, rad = e.bound_r;
        for (int q = 0; q < 3; ++q) {
            ax3[q] = e.R[q];
            ay3[q] = e.R[3 + q];
            nz3[q] = e.R[6 + q];
        }
        rotate(g.Rs, e.o, c);
        rotate(g.Rs, ax3, a);   // unit half-axes
        rotate(g.Rs, ay3, bb);
        rotate(g.Rs, nz3, n);
        f.cx = c[0];
        f.cy = c[1];
        const double cpad = rad * (1.0 + 1e-9) + 1e-6 * (1.0 + fabs(c[0]) + fabs(c[1]));
        f.pad = cpad + 2.0 * g.eps;
        const double fr = cpad + 4e-7 * (fabs(c[0]) + fabs(c[1]) + g.box_ext + cpad);
        f.disc = make_float4(float(c[0]), float(c[1]), float(fr), __int_as_float(j));
        // padded parallelogram (the pre-test's) and exact footprint
        const double wide = 1e-3 + 2e-6 * (1.0 + fabs(c[0]) + fabs(c[1]) + g.box_ext + rad);
        const double d1 = a[0] * bb[1] - a[1] * bb[0];
        const double la = sqrt(a[0] * a[0] + a[1] * a[1]), lb = sqrt(bb[0] * bb[0] + bb[1] * bb[1]);
        const bool flat_on = fabs(d1) > 1e-3 * la * lb;
        if (flat_on) {
            const double wx = hx + wide, wy = hy + wide;
            const double i00 = bb[1] / (d1 * wx), i01 = -bb[0] / (d1 * wx), i10 = -a[1] / (d1 * wy), i11 = a[0] / (d1 * wy);
            const double z0 = wide * n[0], z1 = wide * n[1];
            const double Q0 = 2.0 * (wx * la + wy * lb + sqrt(z0 * z0 + z1 * z1)) + 1.0;
            const double lu = (1.0 + fabs(i00 * z0 + i01 * z1)) * (1.0 + 1e-5) + 1e-6 * (fabs(i00) + fabs(i01)) * Q0;
            const double lv = (1.0 + fabs(i10 * z0 + i11 * z1)) * (1.0 + 1e-5) + 1e-6 * (fabs(i10) + fabs(i11)) * Q0;
            f.par = make_float4(float(i00 / lu), float(i01 / lu), float(i10 / lv), float(i11 / lv));
        }
        // bitmap squares within (ex, ey) of the centre
        auto mark = [&](double ex, double ey, const double i4[4]) {
            const double x = c[0] - g.x0, y = c[1] - g.y0, h = 0.5 * g.side + g.pad;
            const double lu = i4 ? 1.0 + 1e-5 + (fabs(i4[0]) + fabs(i4[1])) * h : 0.0;
            const double lv = i4 ? 1.0 + 1e-5 + (fabs(i4[2]) + fabs(i4[3])) * h : 0.0;
            const int x0 = max(0, int(floor((x - ex) / g.side))), x1 = min(g.onx - 1, int(floor((x + ex) / g.side)));
            const int y0 = max(0, int(floor((y - ey) / g.side))), y1 = min(g.ony - 1, int(floor((y + ey) / g.side)));
            for (int iy = y0; iy <= y1; ++iy)
                for (int ix = x0; ix <= x1; ++ix) {
                    const double qx = (ix + 0.5) * g.side - x, qy = (iy + 0.5) * g.side - y;
                    if (i4 && (fabs(i4[0] * qx + i4[1] * qy) > lu || fabs(i4[2] * qx + i4[3] * qy) > lv)) continue;
                    atomicOr(&b.occ[g.occ0 + uint32_t(iy) * uint32_t(g.ostride) + uint32_t(ix >> 5)], 1u << (ix & 31));
                }
        };
        const double gx = -n[0] / n[2], gy = -n[1] / n[2];
        const double Q = f.disc.z + 1.5 * g.cell, err = g.eps * (1.0 + fabs(gx) + fabs(gy));
        const double tol = 1e-6 * (fabs(c[2]) + (fabs(gx) + fabs(gy)) * Q) + err + 1e-5;
        if (!flat_on || !(fabs(n[2]) > 1e-3) || !before_start_plane(c[2] - hx * fabs(a[2]) - hy * fabs(bb[2]), tol)) {
            f.xc = make_float4(0.f, 0.f, 0.f, INFINITY);  // always decided in double
            const double r = f.disc.z + 2.0 * g.eps + g.pad;
            mark(r, r, nullptr);
        } else {
            const double i4[4] = {bb[1] / (d1 * hx), -bb[0] / (d1 * hx), -a[1] / (d1 * hy), a[0] / (d1 * hy)};
            const double row = fmax(fabs(i4[0]) + fabs(i4[1]), fabs(i4[2]) + fabs(i4[3]));
            f.xb = make_float4(float(i4[0]), float(i4[1]), float(i4[2]), float(i4[3]));
            f.xc = make_float4(float(gx), float(gy), float(c[2]), float((6e-7 * Q + err) * row + 1e-6));
            f.xtol = float(tol);
            mark((hx * fabs(a[0]) + hy * fabs(bb[0])) * (1.0 + 1e-5) + g.pad,
                 (hx * fabs(a[1]) + hy * fabs(bb[1])) * (1.0 + 1e-5) + g.pad, i4);
        }
        f.x0 = max(0, int(floor((f.cx - f.pad - g.x0) / g.cell)));
        f.x1 = min(g.nx - 1, int(floor((f.cx + f.pad - g.x0) / g.cell)));
        f.y0 = max(0, int(floor((f.cy - f.pad - g.y0) / g.cell)));
        f.y1 = min(g.ny - 1, int(floor((f.cy + f.pad - g.y0) / g.cell)));
        for (int gy = f.y0; gy <= f.y1; ++gy)
            for (int gx = f.x0; gx <= f.x1; ++gx)
                if (pos_cell_reached(g, f, gx, gy))
                    atomicAdd(&b.counts[g.cell0 + uint32_t(gy) * uint32_t(g.nx) + uint32_t(gx)], 1u);
    }
    b.feet[size_t(blockIdx.y) * size_t(b.n_elem) + size_t(j)] = f;
}
__global__ void __launch_bounds__(128) k_pos_fill(const PosGridBuild b) {
    const int j = blockIdx.x * 128 + threadIdx.x;
    if (j >= b.n_elem) return;
    const PosGrid &g = b.grids[blockIdx.y];
    const PosFoot f = b.feet[size_t(blockIdx.y) * size_t(b.n_elem) + size_t(j)];
    for (int gy = f.y0; gy <= f.y1; ++gy)
        for (int gx = f.x0; gx <= f.x1; ++gx)
            if (pos_cell_reached(g, f, gx, gy)) {
                const uint32_t c = g.cell0 + uint32_t(gy) * uint32_t(g.nx) + uint32_t(gx);
                const uint32_t k = atomicAdd(&b.cursor[c], 1u);
                if (k < b.counts[c]) b.list[b.offsets[c] + k] = uint32_t(j);
            }
}
// Entries of cells in ascending element order.  A cell of a few entries is one thread's insertion sort;
// where a distant element stretches the box, thousands of elements share a cell: such cells are left
// to the whole block, which marks a window of elements in a bitmap and writes the marked ones out
// in order.  Set-up of a position with 10,000 elements in one cell: 1,406 ms with the insertion sort
// alone, 3.3 so; 1,000 elements 17.5 and 1.0.
constexpr int kPosThreads = 128;
constexpr uint32_t kPosSortMost = 32;      // entries sorted by one thread (at most 500 steps)
constexpr int kPosWindowWords = 1024;      // 32,768 elements of a window
__global__ void __launch_bounds__(kPosThreads) k_pos_entries(const PosGridBuild b) {
    const PosGrid &g = b.grids[blockIdx.y];
    const PosFoot *feet = b.feet + size_t(blockIdx.y) * size_t(b.n_elem);
    const uint32_t n_cells = uint32_t(g.nx) * uint32_t(g.ny);
    __shared__ uint32_t window[kPosWindowWords], crowded[kPosThreads], n_crowded, part[kPosThreads / 32];
    auto put = [&](uint32_t at, uint32_t j, double x0, double y0) {
        const PosFoot &f = feet[j];
        b.disc[at] = f.disc;
        b.par[at] = f.par;
        b.xa[at] = make_float4(float(f.cx - x0), float(f.cy - y0), f.xtol, f.disc.w);
        b.xb[at] = f.xb;
        b.xc[at] = f.xc;
    };
    auto corner = [&](uint32_t k, double &x0, double &y0) {
        x0 = g.x0 + double(k % uint32_t(g.nx)) * g.cell;
        y0 = g.y0 + double(k / uint32_t(g.nx)) * g.cell;
    };
    for (uint32_t k0 = blockIdx.x * kPosThreads; k0 < n_cells; k0 += gridDim.x * kPosThreads) {
        const uint32_t k = k0 + threadIdx.x;
        if (threadIdx.x == 0) n_crowded = 0;
        __syncthreads();
        if (k < n_cells) {
            const uint32_t c = g.cell0 + k, a = b.offsets[c], n = b.counts[c];
            b.cells[c] = make_int2(int(a), int(a + n));
            if (n > kPosSortMost) {
                crowded[atomicAdd(&n_crowded, 1u)] = k;
            } else {
                uint32_t *l = b.list + a;
                for (uint32_t i = 1; i < n; ++i) {
                    const uint32_t v = l[i];
                    uint32_t m = i;
                    for (; m > 0 && l[m - 1] > v; --m) l[m] = l[m - 1];
                    l[m] = v;
                }
                double x0, y0;
                corner(k, x0, y0);
                for (uint32_t i = 0; i < n; ++i) put(a + i, l[i], x0, y0);
            }
        }
        __syncthreads();
        for (uint32_t h = 0; h < n_crowded; ++h) {
            const uint32_t c = g.cell0 + crowded[h], a = b.offsets[c], n = b.counts[c];
            const uint32_t *l = b.list + a;
            double x0, y0;
            corner(crowded[h], x0, y0);
            uint32_t at = a;  // the same in every thread
            for (uint32_t e0 = 0; e0 < uint32_t(b.n_elem) && at < a + n; e0 += kPosWindowWords * 32) {
                for (int w = threadIdx.x; w < kPosWindowWords; w += kPosThreads) window[w] = 0;
                __syncthreads();
                for (uint32_t i = threadIdx.x; i < n; i += kPosThreads) {
                    const uint32_t v = l[i] - e0;  // elements before the window wrap beyond it
                    if (v < kPosWindowWords * 32) atomicOr(&window[v >> 5], 1u << (v & 31));
                }
                __syncthreads();
                for (int w = threadIdx.x; w < kPosWindowWords; w += kPosThreads) {
                    uint32_t bits = window[w];
                    const uint32_t mine = __popc(bits);
                    uint32_t before = mine;  // inclusive over the warp, then over the block
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t v = __shfl_up_sync(0xffffffffu, before, o);
                        if (int(threadIdx.x & 31) >= o) before += v;
                    }
                    if ((threadIdx.x & 31) == 31) part[threadIdx.x >> 5] = before;
                    __syncthreads();
                    uint32_t all = 0;
                    for (int q = 0; q < kPosThreads / 32; ++q) {
                        if (q < int(threadIdx.x >> 5)) before += part[q];
                        all += part[q];
                    }
                    uint32_t to = at + before - mine;
                    for (; bits; bits &= bits - 1) put(to++, e0 + uint32_t(w) * 32u + uint32_t(__ffs(int(bits)) - 1), x0, y0);
                    at += all;
                    __syncthreads();
                }
            }
        }
        __syncthreads();
    }
}
void launch_pos_footprints(const PosGridBuild &b, cudaStream_t st) {
    k_pos_footprints<<<dim3((b.n_elem + 127) / 128, b.n_pos), 128, 0, st>>>(b);
}
void launch_pos_entries(const PosGridBuild &b, cudaStream_t st) {
    k_pos_fill<<<dim3((b.n_elem + 127) / 128, b.n_pos), 128, 0, st>>>(b);
    k_pos_entries<<<dim3(128, b.n_pos), kPosThreads, 0, st>>>(b);
}

void launch_compact(uint64_t s0, uint32_t n, const uint32_t *hit_elem, const uint32_t *counts,
                    const uint32_t *offsets, uint64_t *hit_sid, uint32_t *hit_el, cudaStream_t st) {
    const uint32_t nb = (n + kProbeBlock - 1) / kProbeBlock;
    k_compact<<<nb, kProbeBlock, 0, st>>>(s0, n, hit_elem, counts, offsets, hit_sid, hit_el);
}
void launch_advance(const uint32_t *total, const uint64_t *hit_sid, uint64_t s0, uint32_t n, RunState *rs,
                    cudaStream_t st) {
    k_advance<<<1, 1, 0, st>>>(total, hit_sid, s0, n, rs);
}
void launch_list_rank(uint64_t s0, const ProbeOut &o, const uint32_t *offsets, const uint32_t *total, RunState *rs,
                      HitRec *hits, uint32_t max_n, cudaStream_t st) {
    const uint32_t blocks = std::max(1u, std::min<uint32_t>((max_n + 255) / 256, 148u * 8u));
    k_list_rank<<<blocks, 256, 0, st>>>(s0, o, offsets, total, rs, hits);
}
void launch_list_sort(uint64_t s0, const ProbeOut &o, const uint32_t *offsets, const uint32_t *total, RunState *rs,
                      uint32_t n_elem0, uint32_t *elem_count, uint32_t *elem_cursor, uint32_t *scratch_total,
                      HitRec *hits, uint32_t max_n, cudaStream_t st) {
    cudaMemsetAsync(elem_count, 0, size_t(n_elem0) * 4, st);
    if (n_elem0 <= uint32_t(kSortBins)) {
        int dev = 0, sms = 148;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const uint32_t blocks = std::max(1u, std::min<uint32_t>((max_n + 4095) / 4096, uint32_t(2 * sms)));
        k_list_hist_sh<<<blocks, kSortBlock, 0, st>>>(o.cand_count, o.cand_el, n_elem0, elem_count);
        k_offsets<<<1, 1024, 0, st>>>(elem_count, n_elem0, elem_cursor, scratch_total);
        k_list_scatter_sh<<<blocks, kSortBlock, 0, st>>>(s0, o, offsets, total, rs, n_elem0, elem_cursor, hits);
        return;
    }
    const uint32_t blocks = std::max(1u, std::min<uint32_t>((max_n + 255) / 256, 148u * 8u));
    k_list_hist<<<blocks, 256, 0, st>>>(o.cand_count, o.cand_el, elem_count);
    k_offsets<<<1, 1024, 0, st>>>(elem_count, n_elem0, elem_cursor, scratch_total);
    k_list_scatter<<<blocks, 256, 0, st>>>(s0, o, offsets, total, rs, elem_cursor, hits);
}
}  // namespace stb
