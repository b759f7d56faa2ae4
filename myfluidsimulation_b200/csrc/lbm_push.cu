// Reference-compatible Legacy / Hybrid step (LBM_BOUNCE_REFERENCE).
//
// The reference's opposite table (src/lbm/lbm3d_legacy.cu:29-32,
// src/lbm/lbm3d_hybrid.cu:28-31) pairs every diagonal direction with its
// mirror image in x (xy and xz diagonals) or y (yz diagonals) instead of its
// opposite.  In the reference's push kernels (legacy.cu:92-108,
// hybrid.cu:140-169) that has two consequences next to solid cells:
//   * a slot (q, y) whose upstream cell y - c_q is solid is written only if the
//     cell's own reflection of direction opp_ref(q) happens to target a solid
//     cell too; otherwise it is never written and keeps what the second buffer
//     held (after the element-wise swap: the populations of the previous step);
//   * a slot written by a neighbour's streaming AND by the cell's own
//     reflection is written twice by two threads (a race in the reference).
// This kernel reproduces that step deterministically: two buffers swapped by
// pointer (the same contents as the reference's swap kernel leaves), unwritten
// slots keep the old buffer's value, and in a doubly written slot the
// reflection wins.  It is the compatibility path, not the fast one: the AA
// kernels (lbm_aa.cu) implement halfway bounce-back with true opposites in
// one buffer.
#include "lbm_common.cuh"
#include "lbm_internal.h"

namespace lbm {
namespace {

__host__ __device__ constexpr int opp_ref(int q) { return opp_tab(q); }

// Whether the target of direction q reflects into the slot that q streams into:
// a diagonal's target x + c_q, and from there c_opp_ref(q), is the cell two rows
// or planes on (c_q + c_opp_ref(q) = (0, +-2, 0) or (0, 0, +-2)).  The flags
// builder left those four answers in the link word.
__host__ __device__ constexpr uint32_t far_bit(int q) {
    if (opp_ref(q) == opp(q)) return 0u;
    const int dy = cy(q) + cy(opp_ref(q)), dz = cz(q) + cz(opp_ref(q));
    return dy > 0 ? LK_YP2 : (dy < 0 ? LK_YM2 : (dz > 0 ? LK_ZP2 : LK_ZM2));
}

// One cell per thread in cell order, so that no thread idles whatever nx is.
// Bound by HBM: 19 populations read, 19 written, a flag byte.  The link word is
// read for cells within two cells of a solid one; every other test is a bit of
// it.  (With the solid flags of the neighbours looked up per direction in 64-bit
// arithmetic, and rows of 256 threads, 128 x 128 x 96 cells took 279 us.)
template <int MODE, class IDX>
__global__ void __launch_bounds__(256, 4) ref_push(AAParams p, const float* fa, float* fb) {
    constexpr bool MACRO = MODE >= 1, STATS = MODE == 2;
    step_begin();
    const IDX N = (IDX)p.N;
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    const uint8_t* __restrict__ fl = p.flags;
    double acc[NSTAT];
#pragma unroll
    for (int k = 0; k < NSTAT; ++k) acc[k] = 0.0;

    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t id64 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; id64 < p.N; id64 += stride) {
        const IDX id = (IDX)id64;
        const uint32_t f8 = fl ? fl[id] : 0u;
        float c[19];
#pragma unroll
        for (int q = 0; q < 19; ++q) c[q] = fa[(IDX)q * N + id];
        if (f8 & F_SOLID) {   // legacy.cu:72-76
#pragma unroll
            for (int q = 0; q < 19; ++q) fb[(IDX)q * N + id] = c[q];
            if (MACRO) { p.rho[id] = 1.f; p.ux[id] = 0.f; p.uy[id] = 0.f; p.uz[id] = 0.f; }
            continue;
        }
        const uint32_t lk = (f8 & (F_SPECIAL | F_NEAR2)) ? p.links[id] : 0u;
        const IDX row = id / (IDX)nx;
        const int x = (int)(id - row * (IDX)nx);
        const int z = (int)(row / (IDX)ny);
        const int y = (int)(row - (IDX)z * (IDX)ny);
        IDX r0[3][3];    // first cells of the nine rows around [dy+1][dz+1], periodic
        {
            const int yy[3] = {y == 0 ? ny - 1 : y - 1, y, y == ny - 1 ? 0 : y + 1};
            const int zz[3] = {z == 0 ? nz - 1 : z - 1, z, z == nz - 1 ? 0 : z + 1};
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) r0[a][b] = ((IDX)zz[b] * (IDX)ny + (IDX)yy[a]) * (IDX)nx;
        }
        const int xs[3] = {x == 0 ? nx - 1 : x - 1, x, x == nx - 1 ? 0 : x + 1};
        float r = 0.f, jx = 0.f, jy = 0.f, jz = 0.f;
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            r += c[q];
            if (cx(q) > 0) jx += c[q]; else if (cx(q) < 0) jx -= c[q];
            if (cy(q) > 0) jy += c[q]; else if (cy(q) < 0) jy -= c[q];
            if (cz(q) > 0) jz += c[q]; else if (cz(q) < 0) jz -= c[q];
        }
        const float ux = ((r > 0.f) ? jx / r : 0.f) + p.fx;
        const float uy = ((r > 0.f) ? jy / r : 0.f) + p.fy;
        const float uz = ((r > 0.f) ? jz / r : 0.f) + p.fz;
        const bool bgk = !p.hybrid || (f8 & F_BAND);
        // legacy.cu:54-58,92-96 with the rounding of every operation spelled out, so that
        // the result does not hang on which of them the compiler fuses
        const float uu = __fmaf_rn(uz, uz, __fmaf_rn(ux, ux, __fmul_rn(uy, uy)));
        const float ws = __fsub_rn(p.omega_s, p.omega_h);
        float o[19];
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            const float eiu = (float)cx(q) * ux + (float)cy(q) * uy + (float)cz(q) * uz;
            const float poly = __fmaf_rn(-1.5f, uu, __fmaf_rn(__fmul_rn(4.5f, eiu), eiu, __fmaf_rn(3.0f, eiu, 1.0f)));
            const float d = __fsub_rn(__fmul_rn(__fmul_rn(wq(q), r), poly), c[q]);      // feq - f
            o[q] = __fmaf_rn(bgk ? p.omega : p.omega_h, d, c[q]);
            if (!bgk) o[q] = __fmaf_rn(ws, d, o[q]);
        }
        const bool at_in = p.duct && x == 0, at_out = p.duct && x == nx - 1;
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            const IDX t = r0[cy(q) + 1][cz(q) + 1] + (IDX)xs[cx(q) + 1];
            if ((lk >> q) & 1u) {
                if (cx(q) < 0 && at_in) {                 // inlet (true opposite, as in the AA kernels)
                    fb[(IDX)opp(q) * N + id] = feq_ref(opp(q), r, p.u_in, 0.f, 0.f);
                } else if (cx(q) > 0 && at_out) {         // outlet
                    fb[(IDX)opp(q) * N + id] = o[opp(q)];
                } else {                                  // reflection into slot opp_ref(q)
                    fb[(IDX)opp_ref(q) * N + id] = o[q];
                    if (STATS) {
                        if (fl[t] & F_OBST) {
                            acc[2] += (double)(cx(q) - cx(opp_ref(q))) * o[q];
                            acc[3] += (double)(cy(q) - cy(opp_ref(q))) * o[q];
                            acc[4] += (double)(cz(q) - cz(opp_ref(q))) * o[q];
                        }
                    }
                }
            } else if (!(lk & far_bit(q))) {   // else the target's own reflection lands in the slot
                fb[(IDX)q * N + t] = o[q];
            }
        }
        if (MACRO) { p.rho[id] = r; p.ux[id] = ux; p.uy[id] = uy; p.uz[id] = uz; }
        if (STATS) {
            acc[0] += (double)r;
            acc[1] += 0.5 * ((double)ux * ux + (double)uy * uy + (double)uz * uz);
            acc[5] += (double)r * ux;
            acc[6] += (double)r * uy;
            acc[7] += (double)r * uz;
        }
    }
    if constexpr (STATS) block_reduce_stats(acc, p.partials);
}

template <class IDX>
void push_idx(const AAParams& p, const float* fa, float* fb, LaunchCfg cfg, cudaStream_t s) {
    // one block per 256 cells; with statistics the cfg.blocks whose partial sums the caller has room for
    const int64_t all = (p.N + cfg.threads - 1) / cfg.threads;
    const unsigned blocks = (unsigned)(all < ((int64_t)1 << 30) ? all : ((int64_t)1 << 30));
    if (p.stats) launch_after(ref_push<2, IDX>, cfg.blocks, cfg.threads, 0, s, p, fa, fb);
    else if (p.macro) launch_after(ref_push<1, IDX>, blocks, cfg.threads, 0, s, p, fa, fb);
    else launch_after(ref_push<0, IDX>, blocks, cfg.threads, 0, s, p, fa, fb);
}

}  // namespace

cudaError_t launch_ref_push(const AAParams& p, const float* fa, float* fb, LaunchCfg cfg, cudaStream_t s) {
    // 32-bit element offsets while every slot index 19*N fits in them
    if ((uint64_t)p.N * 19u < (1ull << 32)) push_idx<uint32_t>(p, fa, fb, cfg, s);
    else push_idx<int64_t>(p, fa, fb, cfg, s);
    return cudaGetLastError();
}

}  // namespace lbm
