// GPU voxelizer, bit-exact with src/geom/voxelize.cpp:14-243.
//
// The reference runs on one host thread: a separating-axis triangle/box test
// over each triangle's candidate cells, then a queue BFS that marks the
// exterior from the six domain faces.  Here:
//   * one warp per triangle, its lanes striding over the candidate cells;
//     every float operation is spelled with an explicit rounding intrinsic
//     (__fadd_rn, __fmul_rn, ...), so nvcc cannot contract it into an FMA and
//     each result equals the reference's uncontracted x86-64 float result;
//   * the grid is held as one bit per cell, 32 cells along x to a word;
//   * the exterior flood fill is a reachability fixed point: one block per (x, y)
//     plane floods its plane to the end in shared memory, then one per (x, z)
//     plane, until a round changes nothing; the reachable set is unique, so the
//     mask is identical to the BFS result whatever the visiting order;
//   * the optional refine^3 coverage downsample (voxelize.cpp:187-226) is one
//     thread per coarse cell.
#include "lbm_common.cuh"
#include "lbm_internal.h"

namespace lbm {
namespace {

__device__ __forceinline__ float fmin_ref(float a, float b) { return (b < a) ? b : a; }   // std::min
__device__ __forceinline__ float fmax_ref(float a, float b) { return (a < b) ? b : a; }   // std::max

// a*b - c*d with both products rounded, as GLM's cross evaluates each term
__device__ __forceinline__ float dif2(float a, float b, float c, float d) {
    return __fsub_rn(__fmul_rn(a, b), __fmul_rn(c, d));
}
// ((a0*b0 + a1*b1) + a2*b2) left to right
__device__ __forceinline__ float dot3(float a0, float a1, float a2, float b0, float b1, float b2) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a0, b0), __fmul_rn(a1, b1)), __fmul_rn(a2, b2));
}

// voxelize.cpp:23-81
__device__ bool tri_box(const float c[3], const float h[3], const float v0[3], const float v1[3], const float v2[3]) {
    float t0[3], t1[3], t2[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        t0[k] = __fsub_rn(v0[k], c[k]);
        t1[k] = __fsub_rn(v1[k], c[k]);
        t2[k] = __fsub_rn(v2[k], c[k]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float mn = fmin_ref(fmin_ref(t0[k], t1[k]), t2[k]);
        const float mx = fmax_ref(fmax_ref(t0[k], t1[k]), t2[k]);
        if (mx < -h[k] || mn > h[k]) return false;
    }
    float e[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        e[0][k] = __fsub_rn(t1[k], t0[k]);
        e[1][k] = __fsub_rn(t2[k], t1[k]);
        e[2][k] = __fsub_rn(t0[k], t2[k]);
    }
    // n = cross(e0, e1): (a.y*b.z - b.y*a.z, a.z*b.x - b.z*a.x, a.x*b.y - b.x*a.y)
    const float n0 = dif2(e[0][1], e[1][2], e[1][1], e[0][2]);
    const float n1 = dif2(e[0][2], e[1][0], e[1][2], e[0][0]);
    const float n2 = dif2(e[0][0], e[1][1], e[1][0], e[0][1]);
    const float r = dot3(h[0], h[1], h[2], fabsf(n0), fabsf(n1), fabsf(n2));
    const float s = fabsf(dot3(n0, n1, n2, t0[0], t0[1], t0[2]));
    if (s > r) return false;
#pragma unroll
    for (int ei = 0; ei < 3; ++ei) {
        const float* ed = e[ei];
        if (__fadd_rn(__fadd_rn(fabsf(ed[0]), fabsf(ed[1])), fabsf(ed[2])) < 1e-12f) continue;
#pragma unroll
        for (int ai = 0; ai < 3; ++ai) {
            const float ax[3] = {ai == 0 ? 1.f : 0.f, ai == 1 ? 1.f : 0.f, ai == 2 ? 1.f : 0.f};
            const float L0 = dif2(ed[1], ax[2], ax[1], ed[2]);
            const float L1 = dif2(ed[2], ax[0], ax[2], ed[0]);
            const float L2 = dif2(ed[0], ax[1], ax[0], ed[1]);
            const float l2 = dot3(L0, L1, L2, L0, L1, L2);
            if (l2 < 1e-20f) continue;
            const float p0 = dot3(L0, L1, L2, t0[0], t0[1], t0[2]);
            const float p1 = dot3(L0, L1, L2, t1[0], t1[1], t1[2]);
            const float p2 = dot3(L0, L1, L2, t2[0], t2[1], t2[2]);
            const float minp = fmin_ref(p0, fmin_ref(p1, p2));
            const float maxp = fmax_ref(p0, fmax_ref(p1, p2));
            const float rp = dot3(h[0], h[1], h[2], fabsf(L0), fabsf(L1), fabsf(L2));
            if (maxp < -rp || minp > rp) return false;
        }
    }
    return true;
}

// voxelize.cpp:83-113: vertex' = s*vertex + trans, per component
__global__ void fit_kernel(const float* __restrict__ in, float* __restrict__ out, int64_t n, float s, float t0,
                           float t1, float t2) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float tr = (i % 3 == 0) ? t0 : ((i % 3 == 1) ? t1 : t2);
        out[i] = __fadd_rn(__fmul_rn(s, in[i]), tr);
    }
}

// voxelize.cpp:115-149: one warp per triangle
__global__ void surface_kernel(const float* __restrict__ vt, int64_t ntri, int nx, int ny, int nz,
                               int wx, uint32_t* __restrict__ surf) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const float h[3] = {__fdiv_rn(0.5f, (float)nx), __fdiv_rn(0.5f, (float)ny), __fdiv_rn(0.5f, (float)nz)};
    const float eps = 1e-6f;
    for (int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < ntri; t += warps) {
        const float* p = vt + t * 9;
        const float v0[3] = {p[0], p[1], p[2]}, v1[3] = {p[3], p[4], p[5]}, v2[3] = {p[6], p[7], p[8]};
        int lo[3], hi[3];
        const int n[3] = {nx, ny, nz};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float mn = __fsub_rn(fmin_ref(v0[k], fmin_ref(v1[k], v2[k])), eps);
            const float mx = __fadd_rn(fmax_ref(v0[k], fmax_ref(v1[k], v2[k])), eps);
            lo[k] = max(0, (int)floorf(__fmul_rn(mn, (float)n[k])));
            hi[k] = min(n[k] - 1, (int)floorf(__fmul_rn(mx, (float)n[k])));
        }
        if (hi[0] < lo[0] || hi[1] < lo[1] || hi[2] < lo[2]) continue;
        const int64_t sx = hi[0] - lo[0] + 1, sy = hi[1] - lo[1] + 1, sz = hi[2] - lo[2] + 1;
        const int64_t cnt = sx * sy * sz;
        for (int64_t c = lane; c < cnt; c += 32) {
            const int x = lo[0] + (int)(c % sx);
            const int y = lo[1] + (int)((c / sx) % sy);
            const int z = lo[2] + (int)(c / (sx * sy));
            const float cc[3] = {__fdiv_rn(__fadd_rn((float)x, 0.5f), (float)nx),
                                 __fdiv_rn(__fadd_rn((float)y, 0.5f), (float)ny),
                                 __fdiv_rn(__fadd_rn((float)z, 0.5f), (float)nz)};
            if (tri_box(cc, h, v0, v1, v2)) atomicOr(surf + ((int64_t)z * ny + y) * wx + (x >> 5), 1u << (x & 31));
        }
    }
}

// One plane of the flood fill: `rows` rows of `wx` words, open cells O, reached
// cells R (a subset of O), `pitch` words from row to row.  Sweeps along x and across the rows
// alternate until nothing changes.
//   x: a carry ripples through a run of ones, so (O + R) ^ O marks the run from a
//      seed upward; one thread per row, the carry going from word to word, then
//      the same on reversed bits.
//   rows: 32 cells at a time; every word column is cut into segments, one thread
//      per segment finds what leaves it (from inside, and with everything entering),
//      the segments are chained, and each is swept once more with what enters it.
__device__ bool flood_plane(const uint32_t* __restrict__ O, uint32_t* R, int rows, int wx, int64_t pitch,
                            uint32_t* seg) {
    const int T = (int)blockDim.x, tid = (int)threadIdx.x;
    const int nseg = max(1, min(T / wx, rows)), len = (rows + nseg - 1) / nseg;
    uint32_t *sa = seg, *sb = seg + T;
    bool ever = false;
    for (;;) {
        bool any = false;
        for (int y = tid; y < rows; y += T) {
            const uint32_t* o = O + (int64_t)y * pitch;
            uint32_t* r = R + (int64_t)y * pitch;
            uint32_t in = 0;      // the last cell of the word before is reached
            for (int w = 0; w < wx; ++w) {
                const uint32_t ow = o[w], rw = r[w];
                const uint32_t sd = rw | (in & ow);
                const uint32_t n = sd | (ow & (ow ^ (ow + sd)));
                if (n != rw) { r[w] = n; any = true; }
                in = n >> 31;
            }
            in = 0;
            for (int w = wx - 1; w >= 0; --w) {
                const uint32_t rw = r[w], ow = __brev(o[w]), rv = __brev(rw);
                const uint32_t sd = rv | (in & ow);
                const uint32_t n = sd | (ow & (ow ^ (ow + sd)));
                if (n != rv) { r[w] = __brev(n); any = true; }
                in = n >> 31;
            }
        }
        __syncthreads();
        for (int c0 = 0; c0 < wx; c0 += T) {          // word columns in groups of at most T
            const int cols = min(wx - c0, T);
            for (int dir = 0; dir < 2; ++dir) {
                const int w = c0 + tid % cols, k = tid / cols;
                const int y0 = k * len, y1 = min(rows, y0 + len);
                const bool on = k < nseg && y0 < rows;
                auto row = [&](int i) { return (int64_t)(dir ? rows - 1 - i : i) * pitch + w; };
                if (on) {
                    uint32_t out = 0, through = 0xffffffffu;
                    for (int i = y0; i < y1; ++i) {
                        const uint32_t o = O[row(i)];
                        out = R[row(i)] | (out & o);
                        through &= o;
                    }
                    sa[tid] = out;
                    sb[tid] = through;
                }
                __syncthreads();
                if (on) {
                    uint32_t c = 0;
                    for (int j = 0; j < k; ++j) c = sa[j * cols + tid % cols] | (c & sb[j * cols + tid % cols]);
                    for (int i = y0; i < y1; ++i) {
                        const uint32_t o = O[row(i)], r = R[row(i)];
                        c = r | (c & o);
                        if (c != r) { R[row(i)] = c; any = true; }
                    }
                }
                __syncthreads();
            }
        }
        if (!__syncthreads_or(any)) return ever;
        ever = true;
    }
}

// Flood of one (x, y) plane per block (AXIS 2) or one (x, z) plane (AXIS 1).
// first: the exterior starts from the open cells on the six faces.  A round whose
// predecessor changed nothing (changed[round - 1] == 0) has nothing to do.  SHARED:
// the plane's words fit in shared memory; otherwise it is flooded where it lies.  Whole
// calls, copies included, against sweeps of one byte per cell along all lines of the grid,
// both with an icosphere: in shared memory 1024x800x64 18.4 -> 12.0 ms, in global memory
// 1024x1024x64 23.9 -> 15.7, 2048x2048x16 25.9 -> 17.1, 4096x4096x8 52 -> 38,
// 1024x1024x512 165 -> 125; with a serpentine of 24 walls 1024x1024x256 221 -> 97.
template <int AXIS, bool SHARED>
__global__ void __launch_bounds__(512) flood_kernel(const uint32_t* __restrict__ surf, uint32_t* vis, int nx, int ny,
                                                    int nz, int wx, int first, int round, int* changed) {
    extern __shared__ uint32_t buf[];
    __shared__ uint32_t seg[2 * 512];
    if (round > 0 && changed[round - 1] == 0) return;
    const int rows = AXIS == 2 ? ny : nz;
    const int64_t pitch = AXIS == 2 ? wx : (int64_t)ny * wx;
    const int64_t base = AXIS == 2 ? (int64_t)blockIdx.x * ny * wx : (int64_t)blockIdx.x * wx;
    const uint32_t last = nx % 32 ? (1u << (nx % 32)) - 1u : 0xffffffffu;
    uint32_t* O = buf;                          // (not SHARED: vis + the second half of the buffer)
    uint32_t* R = SHARED ? buf + rows * wx : vis + base;
    const bool face = AXIS == 2 && (blockIdx.x == 0 || blockIdx.x == (unsigned)nz - 1);
    bool seeded = false;
    for (int i = threadIdx.x; i < rows * wx; i += blockDim.x) {
        const int y = i / wx, w = i - y * wx;
        const int64_t g = base + (int64_t)y * pitch + w;
        const uint32_t o = ~surf[g] & (w == wx - 1 ? last : 0xffffffffu);
        uint32_t r;
        if (first) {
            uint32_t m = face || y == 0 || y == ny - 1 ? 0xffffffffu : 0u;
            if (w == 0) m |= 1u;
            if (w == wx - 1) m |= 1u << ((nx - 1) & 31);
            r = o & m;
            seeded = seeded || r != 0;
        } else {
            r = vis[g];
        }
        if (SHARED) { O[i] = o; R[i] = r; }
        else if (first) vis[g] = r;
    }
    bool ch;
    if constexpr (SHARED) {
        __syncthreads();
        ch = flood_plane(O, R, rows, wx, wx, seg);
        if (ch || first)
            for (int i = threadIdx.x; i < rows * wx; i += blockDim.x) {
                const int y = i / wx, w = i - y * wx;
                vis[base + (int64_t)y * pitch + w] = R[i];
            }
    } else {
        __syncthreads();
        ch = flood_plane(vis + (int64_t)nz * ny * wx + base, vis + base, rows, wx, pitch, seg);   // open cells: second half
    }
    if (__syncthreads_or(ch || seeded) && threadIdx.x == 0) changed[round] = 1;
}

// the open cells of a grid whose planes do not fit in shared memory
__global__ void open_kernel(const uint32_t* __restrict__ surf, uint32_t* __restrict__ open, int64_t words, int wx,
                            uint32_t last) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (int64_t)gridDim.x * blockDim.x)
        open[i] = ~surf[i] & (i % wx == wx - 1 ? last : 0xffffffffu);
}

// Solid = surface or not reached; with refinement r the coverage of r^3 fine cells
// against thr (voxelize.cpp:187-226).  One thread per coarse cell, whose r cells of
// a fine row lie in one or two words (r <= 32) or are counted word by word.
__global__ void mask_kernel(const uint32_t* __restrict__ surf, const uint32_t* __restrict__ vis, int r, int nx, int ny,
                            int nz, int wx, float thr, uint8_t* __restrict__ out) {
    const int64_t N = (int64_t)nx * ny * nz;
    const int64_t fy = (int64_t)ny * r;
    const int r3 = r * r * r;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
        const int x = (int)(i % nx);
        const int64_t row = i / nx;
        const int y = (int)(row % ny), z = (int)(row / ny);
        int cnt = 0;
        for (int dz = 0; dz < r; ++dz)
            for (int dy = 0; dy < r; ++dy) {
                const int64_t b = (((int64_t)z * r + dz) * fy + (int64_t)y * r + dy) * wx;
                int64_t x0 = (int64_t)x * r, left = r;
                while (left > 0) {
                    const int bit = (int)(x0 & 31), take = (int)min((int64_t)(32 - bit), left);
                    const uint32_t m = (take == 32 ? 0xffffffffu : ((1u << take) - 1u)) << bit;
                    cnt += __popc((surf[b + (x0 >> 5)] | ~vis[b + (x0 >> 5)]) & m);
                    x0 += take;
                    left -= take;
                }
            }
        if (r == 1) out[i] = (uint8_t)cnt;
        else {
            const float cov = __fdiv_rn((float)cnt, (float)r3);
            out[i] = (cov > 0.0f && cov >= thr) ? 1 : 0;
        }
    }
}

}  // namespace

cudaError_t launch_voxelize(const float* d_tris, int64_t ntri, const float* bb, int nx, int ny, int nz, float scale,
                            const float* translate, int refine, float thr, uint8_t* d_mask, cudaStream_t s) {
    if (refine < 1) refine = 1;
    // compute_fit_transform (voxelize.cpp:83-91), float, uncontracted
    const float bs[3] = {bb[3] - bb[0], bb[4] - bb[1], bb[5] - bb[2]};
    const float maxDim = (bs[0] < ((bs[1] < bs[2]) ? bs[2] : bs[1])) ? ((bs[1] < bs[2]) ? bs[2] : bs[1]) : bs[0];
    volatile float sv = (maxDim > 0.0f) ? (scale / maxDim) : 1.0f;
    const float sf = sv;
    float tr[3];
    for (int k = 0; k < 3; ++k) {
        volatile float center = 0.5f * (bb[k] + bb[3 + k]);
        volatile float prod = sf * center;
        tr[k] = translate[k] - prod;
    }
    const int fx = nx * refine, fy = ny * refine, fz = nz * refine;
    const int64_t NF = (int64_t)fx * fy * fz;
    const int wx = (fx + 31) / 32;
    const int64_t words = NF / fx * wx;
    const size_t sm2 = sizeof(uint32_t) * 2 * (size_t)fy * wx, sm1 = sizeof(uint32_t) * 2 * (size_t)fz * wx;
    constexpr size_t kShared = 200 * 1024;     // beyond it a plane is flooded in global memory
    const bool shared = sm2 <= kShared && sm1 <= kShared;
    constexpr int kRounds = 16;                // rounds queued between two looks at the result
    float* vt = nullptr;
    uint32_t *surf = nullptr, *vis = nullptr;
    int* changed = nullptr;
    cudaError_t e = cudaSuccess;
#define VX_CK(x) do { e = (x); if (e != cudaSuccess) goto done; } while (0)
    VX_CK(scratch_alloc((void**)&vt, sizeof(float) * 9 * (size_t)(ntri > 0 ? ntri : 1), s));
    VX_CK(scratch_alloc((void**)&surf, sizeof(uint32_t) * (size_t)words, s));
    VX_CK(scratch_alloc((void**)&vis, sizeof(uint32_t) * (size_t)words * (shared ? 1 : 2), s));
    VX_CK(scratch_alloc((void**)&changed, sizeof(int) * kRounds, s));
    VX_CK(cudaMemsetAsync(surf, 0, sizeof(uint32_t) * (size_t)words, s));
    if (ntri > 0) {
        fit_kernel<<<num_sms() * 4, 256, 0, s>>>(d_tris, vt, ntri * 9, sf, tr[0], tr[1], tr[2]);
        const int64_t blocks = (ntri + 7) / 8;   // 8 warps per block
        surface_kernel<<<(int)(blocks < 65535 ? blocks : 65535), 256, 0, s>>>(vt, ntri, fx, fy, fz, wx, surf);
        VX_CK(cudaGetLastError());
    }
    if (shared) {
        VX_CK(cudaFuncSetAttribute((const void*)flood_kernel<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kShared));
        VX_CK(cudaFuncSetAttribute((const void*)flood_kernel<1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kShared));
    } else {
        const uint32_t last = fx % 32 ? (1u << (fx % 32)) - 1u : 0xffffffffu;
        open_kernel<<<num_sms() * 8, 256, 0, s>>>(surf, vis + words, words, wx, last);
        VX_CK(cudaGetLastError());
    }
    for (int pass = 0;; ++pass) {
        // (the first batch: most obstacles are done after one round, which the second one confirms)
        // a grid of one plane is done when that is flooded (8192x8192x1: the call 37 -> 28 ms)
        const bool plane = fy == 1 || fz == 1;
        const int n = plane ? 1 : (pass == 0 ? 3 : kRounds);
        int h[kRounds];
        VX_CK(cudaMemsetAsync(changed, 0, sizeof(int) * kRounds, s));
        for (int k = 0; k < n; ++k) {
            const int first = pass == 0 && k == 0;
            if (shared) {
                flood_kernel<2, true><<<fz, 512, sm2, s>>>(surf, vis, fx, fy, fz, wx, first, k, changed);
                if (fz > 1) flood_kernel<1, true><<<fy, 512, sm1, s>>>(surf, vis, fx, fy, fz, wx, 0, k, changed);
            } else {
                flood_kernel<2, false><<<fz, 512, 0, s>>>(surf, vis, fx, fy, fz, wx, first, k, changed);
                if (fz > 1) flood_kernel<1, false><<<fy, 512, 0, s>>>(surf, vis, fx, fy, fz, wx, 0, k, changed);
            }
            VX_CK(cudaGetLastError());
        }
        if (plane) break;
        VX_CK(cudaMemcpyAsync(h, changed, sizeof(int) * kRounds, cudaMemcpyDeviceToHost, s));
        VX_CK(cudaStreamSynchronize(s));
        if (!h[n - 1]) break;
    }
    mask_kernel<<<num_sms() * 8, 256, 0, s>>>(surf, vis, refine, nx, ny, nz, wx,
                                              fmaxf(0.0f, fminf(1.0f, thr)), d_mask);
    VX_CK(cudaGetLastError());
done:
#undef VX_CK
    if (vt) cudaFreeAsync(vt, s);
    if (surf) cudaFreeAsync(surf, s);
    if (vis) cudaFreeAsync(vis, s);
    if (changed) cudaFreeAsync(changed, s);
    return e;
}

}  // namespace lbm
