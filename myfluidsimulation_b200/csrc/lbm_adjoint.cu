// Hand-written discrete adjoint of the BGK duct step, with checkpointing.
//
// The differentiated model is the duct step of the AA kernels (lbm_aa.cu) in
// two-buffer push form, in FP32 or FP64 (template R):
//   f*_q(x) = f_q(x) + w (feq_q(rho, u) - f_q(x)),   rho = sum f, u = j/rho + F
//   f'_q(x + c_q) = f*_q(x)                             streaming link
//   f'_opp(q)(x)  = f*_q(x)                             x + c_q solid (halfway bounce-back)
//   f'_opp(q)(x)  = w_q rho(x) (1 + 3 u_in + 3 u_in^2)  x + c_q before the inlet plane,
//                                                        u_in = u_in(y, z) (the inlet control)
//   f'_opp(q)(x)  = f*_opp(q)(x)                        x + c_q past the outlet plane
// with the drag of a step D = sum over links into obstacle cells of 2 c_qx f*_q.
// The objective is J = mean of D over the steps [window_begin, window_end]
// (1-based, the drag of step n uses the collision of f^{n-1}); the controls are
// the inlet profile u_in(y, z) and the initial velocity field u0 (f^0 =
// feq(1, u0)).
//
// Reverse pass, one kernel per step, gather form (lambda = dJ/df):
//   lambda*_q(x) = lambda'_q(x + c_q)            streaming link
//               = lambda'_opp(q)(x) [+ 2 c_qx / nwin if x + c_q is an obstacle in the window]
//               = 0                                inlet / outlet links (f*_q leaves)
//   outlet copies: lambda*_opp(q)(x) += lambda'_opp(q)(x)
//   lambda_p(x) = (1 - w) lambda*_p + w (A + sum_a B_a (c_pa - (u_a - F_a)) / rho) + A_in
//   A = sum_q lambda*_q feq_q / rho,  B_a = sum_q lambda*_q w_q rho (3 c_qa + 9 (c_q.u) c_qa - 3 u_a)
//   A_in = sum over inlet links lambda'_opp(q)(x) w_q kin   (rho enters the inlet value)
//   dJ/du_in(y,z) += sum over inlet links lambda'_opp(q)(x) w_q rho (3 + 6 u_in)
// and at the end dJ/du0_a = sum_q lambda^0_q w_q (3 c_qa + 9 (c_q.u0) c_qa - 3 u0_a).
// The forward states the reverse pass needs are recomputed segment by segment
// from checkpoints taken every `checkpoint_every` steps.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <utility>
#include <vector>

#include "lbm_capi.h"
#include "lbm_common.cuh"
#include "lbm_internal.h"
#include "lbm_vec.cuh"

namespace lbm {
void set_error(const std::string& msg);

namespace {

template <class R>
__device__ __forceinline__ constexpr R wR(int q) {
    return q == 0 ? R(1) / R(3) : (q <= 6 ? R(1) / R(18) : R(1) / R(36));
}

template <class R>
struct AdjP {
    const uint8_t* flags;
    const uint32_t* links;
    int nx, ny, nz;
    int64_t N;
    R omega, fx, fy, fz;
};

// Every loop over the directions is unrolled, so that c_q is a literal, the 19
// populations stay in registers and a product with c_q = 0 is no instruction.
// With the loops rolled the arrays lived in local memory: 315 us (forward) and
// 320 us (reverse) per 128x64x64 step in FP32, against 12 us of traffic; the
// gradient of 100 such steps (checkpoints every 25) went from 105.6 to 17.4 ms,
// host copies and allocations included, and has come to 7.4 ms with sums over
// opposite pairs, one allocation and controls that stay on the GPU.
template <int C, class R>
__device__ __forceinline__ R plus_c(R s, R v) { return C > 0 ? s + v : (C < 0 ? s - v : s); }
// c_q . u
template <int q, class R>
__device__ __forceinline__ R cdot(R ux, R uy, R uz) {
    return plus_c<cz(q)>(plus_c<cy(q)>(plus_c<cx(q)>(R(0), ux), uy), uz);
}
template <int q> struct QC { static constexpr int value = q; };
template <int Q0, int Q1, class F>
__device__ __forceinline__ void for_q(F&& fn) {
    if constexpr (Q0 < Q1) {
        fn(QC<Q0>{});
        for_q<Q0 + 1, Q1>(fn);
    }
}

// One cell and its neighbours' indices, periodic in every axis (a link past the
// duct's ends never streams, so its index is not used).
template <class IDX>
struct AdjCell {
    int x, y, z;
    IDX row[3][3];   // [dy+1][dz+1]
    int xs[3];
    __device__ __forceinline__ void init(uint32_t id, int nx, int ny, int nz) {
        const uint32_t r = id / (uint32_t)nx;
        x = (int)(id - r * (uint32_t)nx);
        z = (int)(r / (uint32_t)ny);
        y = (int)(r - (uint32_t)z * (uint32_t)ny);
        const int yy[3] = {y == 0 ? ny - 1 : y - 1, y, y == ny - 1 ? 0 : y + 1};
        const int zz[3] = {z == 0 ? nz - 1 : z - 1, z, z == nz - 1 ? 0 : z + 1};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) row[a][b] = ((IDX)zz[b] * (IDX)ny + (IDX)yy[a]) * (IDX)nx;
        xs[0] = x == 0 ? nx - 1 : x - 1;
        xs[1] = x;
        xs[2] = x == nx - 1 ? 0 : x + 1;
    }
    template <int q>
    __device__ __forceinline__ IDX to() const { return row[cy(q) + 1][cz(q) + 1] + (IDX)xs[cx(q) + 1]; }
};

template <class R>
__global__ void adj_init(AdjP<R> p, const double* __restrict__ u0, R* __restrict__ f) {
    for (int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; id < p.N; id += (int64_t)gridDim.x * blockDim.x) {
        const R ux = (R)u0[id], uy = (R)u0[p.N + id], uz = (R)u0[2 * p.N + id];
        const R uu = ux * ux + uy * uy + uz * uz;
        for_q<0, 19>([&](auto qi) {
            constexpr int q = decltype(qi)::value;
            const R cu = cdot<q>(ux, uy, uz);
            f[q * p.N + id] = wR<R>(q) * (R(1) + R(3) * cu + R(4.5) * cu * cu - R(1.5) * uu);
        });
    }
}

// one push step f -> fn, one cell per thread; drag_part (or null: the step is
// outside the window, or recomputed) adds the block's drag sum (FP64).
// Bound by the latency of its loads at 24 warps per SM: 256x128x128 FP32 124 us
// where its traffic (the state read and written once) takes 98, DRAM 59 % and
// issue slots 57 % busy; 128x64x64 19 us, traffic 12.
template <class R, class IDX>
__global__ void __launch_bounds__(256) adj_fwd(AdjP<R> p, const R* f, R* fn,
                                               const double* __restrict__ uin, double* __restrict__ drag_part) {
    step_begin();
    double drag = 0.0;
    const IDX N = (IDX)p.N;
    const int64_t id64 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id64 < p.N) {
        const IDX id = (IDX)id64;
        const uint32_t fl = p.flags[id];
        R fq[19];
        for_q<0, 19>([&](auto qi) {
            constexpr int q = decltype(qi)::value;
            fq[q] = f[(IDX)q * N + id];
        });
        if (fl & F_SOLID) {
            for_q<0, 19>([&](auto qi) {
                constexpr int q = decltype(qi)::value;
                fn[(IDX)q * N + id] = fq[q];
            });
        } else {
            AdjCell<IDX> c;
            c.init((uint32_t)id64, p.nx, p.ny, p.nz);
            const CellV<R> m = moments<false>(fq, p.fx, p.fy, p.fz);   // u = j / rho + F whatever the sign of rho
            collide(fq, m, p.omega);
            const uint32_t lk = (fl & F_SPECIAL) ? p.links[id] : 0u;
            for_q<0, 19>([&](auto qi) {
                constexpr int q = decltype(qi)::value;
                constexpr int o = opp(q);
                const IDX t = c.template to<q>();
                if (!((lk >> q) & 1u)) {
                    fn[(IDX)q * N + t] = fq[q];
                } else {
                    R v = fq[q];
                    if (cx(q) < 0 && c.x == 0) {
                        const R u = (R)uin[(int64_t)c.z * p.ny + c.y];
                        v = wR<R>(q) * m.r * (R(1) + R(3) * u + R(3) * u * u);
                    } else if (cx(q) > 0 && c.x == p.nx - 1) {
                        v = fq[o];
                    } else if (cx(q) != 0 && drag_part && (p.flags[t] & F_OBST)) {
                        drag += 2.0 * cx(q) * (double)fq[q];
                    }
                    fn[(IDX)o * N + id] = v;
                }
            });
        }
    }
    if (!drag_part) return;
    __shared__ double red[8];
    for (int o = 16; o > 0; o >>= 1) drag += __shfl_down_sync(0xffffffffu, drag, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = drag;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
        drag_part[blockIdx.x] += s;
    }
}

// out = the sum of n values in a fixed order (one block)
__global__ void __launch_bounds__(1024) adj_sum(const double* __restrict__ v, int64_t n, double* __restrict__ out) {
    double s = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += v[i];
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = red[threadIdx.x];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) *out = s;
    }
}

// one reverse step, one cell per thread: lam0 = (d f'/d f)^T lam1 (+ the drag
// term when wdrag != 0).  Bound as adj_fwd: 256x128x128 FP32 182 us where its
// traffic (f and lam1 read, lam0 written) takes 146, DRAM 61 %, issue slots 50 %.
template <class R, class IDX>
__global__ void __launch_bounds__(256) adj_bwd(AdjP<R> p, const R* f, const R* lam1, R* lam0,
                                               const double* __restrict__ uin, double* g_uin, R wdrag) {
    step_begin();
    const IDX N = (IDX)p.N;
    const int64_t id64 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id64 >= p.N) return;
    const IDX id = (IDX)id64;
    const uint32_t fl = p.flags[id];
    if (fl & F_SOLID) {
        for_q<0, 19>([&](auto qi) {
            constexpr int q = decltype(qi)::value;
            lam0[(IDX)q * N + id] = R(0);
        });
        return;
    }
    AdjCell<IDX> c;
    c.init((uint32_t)id64, p.nx, p.ny, p.nz);
    CellV<R> m;
    {
        R fq[19];
        for_q<0, 19>([&](auto qi) {
            constexpr int q = decltype(qi)::value;
            fq[q] = f[(IDX)q * N + id];
        });
        m = moments<false>(fq, p.fx, p.fy, p.fz);
    }
    const uint32_t lk = (fl & F_SPECIAL) ? p.links[id] : 0u;
    R ls[19];
    R a_in = 0;
    // what arrives over each link: a streaming one from the neighbour, another
    // from the cell's own slot opp(q)
    for_q<0, 19>([&](auto qi) {
        constexpr int q = decltype(qi)::value;
        constexpr int o = opp(q);
        const bool nn = (lk >> q) & 1u;
        ls[q] = lam1[nn ? (IDX)o * N + id : (IDX)q * N + c.template to<q>()];
    });
    if (lk) {
        double g_in = 0.0;
        R keep[19];      // outlet copies, added once every direction is resolved
        for_q<0, 19>([&](auto qi) {
            constexpr int q = decltype(qi)::value;
            constexpr int o = opp(q);
            keep[o] = 0;
            if ((lk >> q) & 1u) {
                const R lo = ls[q];
                if (cx(q) < 0 && c.x == 0) {
                    const R u = (R)uin[(int64_t)c.z * p.ny + c.y];
                    a_in += lo * wR<R>(q) * (R(1) + R(3) * u + R(3) * u * u);
                    g_in += (double)(lo * wR<R>(q) * m.r * (R(3) + R(6) * u));
                    ls[q] = 0;
                } else if (cx(q) > 0 && c.x == p.nx - 1) {
                    keep[o] = lo;
                    ls[q] = 0;
                } else if (cx(q) != 0 && wdrag != R(0) && (p.flags[c.template to<q>()] & F_OBST)) {
                    ls[q] += wdrag * R(2 * cx(q));
                }
            }
        });
        for_q<0, 19>([&](auto qi) {
            constexpr int q = decltype(qi)::value;
            ls[q] += keep[q];
        });
        if (c.x == 0 && g_uin) g_uin[(int64_t)c.z * p.ny + c.y] += g_in;
    }
    // A and B from sums over the opposite pairs (q, o) of one weight w, with
    // S = ls_q + ls_o, D = ls_q - ls_o:
    //   A = sum w [(1 - 1.5 u^2) sum S + sum c.u (4.5 c.u S + 3 D)]
    //   B = rho sum w [sum c (9 c.u S + 3 D) - 3 u sum S]
    // The weights are multiplied in once per sum, their own rounding compensated (mulk), as
    // the forward step does: sum w_q of the rounded weights is 1.5e-8 too large, a bias of
    // omega times that per step, 2.7e-6 over 100 steps at tau 0.56.  dJ/du0 of 48x32x32 after
    // 100 steps is off by 4.4e-7 (2-norm, relative to FP64), by 2.5e-6 with rounded weights.
    // (B carries rho, and the derivative of u divides by it.)
    const R iso = R(1) - R(1.5) * (m.ux * m.ux + m.uy * m.uy + m.uz * m.uz);
    const R l0 = mulk(ls[0], K3_HI, K3_LO), n0 = R(-3) * l0;
    R A = iso * l0, gx = m.ux * n0, gy = m.uy * n0, gz = m.uz * n0;
    auto add_pairs = [&](auto q0, auto q1, float hi, float lo) {
        R s = 0, a = 0, bx = 0, by = 0, bz = 0;
        for_q<decltype(q0)::value, decltype(q1)::value>([&](auto qi) {
            constexpr int q = decltype(qi)::value, o = opp(q);
            if constexpr (q < o) {
                const R S = ls[q] + ls[o], D = ls[q] - ls[o];
                const R cu = cdot<q>(m.ux, m.uy, m.uz);
                const R e = R(4.5) * cu * S, k = e + R(3) * D;
                s += S;
                a += cu * k;
                bx = plus_c<cx(q)>(bx, e + k);
                by = plus_c<cy(q)>(by, e + k);
                bz = plus_c<cz(q)>(bz, e + k);
            }
        });
        const R s3 = R(3) * s;
        A += mulk(a + iso * s, hi, lo);
        gx += mulk(bx - m.ux * s3, hi, lo);
        gy += mulk(by - m.uy * s3, hi, lo);
        gz += mulk(bz - m.uz * s3, hi, lo);
    };
    add_pairs(QC<1>{}, QC<7>{}, K18_HI, K18_LO);
    add_pairs(QC<7>{}, QC<19>{}, K36_HI, K36_LO);
    const R om = p.omega;
    const R base = om * (A - (gx * (m.ux - p.fx) + gy * (m.uy - p.fy) + gz * (m.uz - p.fz))) + a_in;
    for_q<0, 19>([&](auto qi) {
        constexpr int q = decltype(qi)::value;
        lam0[(IDX)q * N + id] = (R(1) - om) * ls[q] + (om * cdot<q>(gx, gy, gz) + base);
    });
}

template <class R>
__global__ void adj_grad_u0(AdjP<R> p, const double* __restrict__ u0, const R* __restrict__ lam, double* __restrict__ g) {
    for (int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; id < p.N; id += (int64_t)gridDim.x * blockDim.x) {
        const R ux = (R)u0[id], uy = (R)u0[p.N + id], uz = (R)u0[2 * p.N + id];
        R gx = 0, gy = 0, gz = 0;
        for_q<0, 19>([&](auto qi) {
            constexpr int q = decltype(qi)::value;
            const R cu = cdot<q>(ux, uy, uz);
            const R t = lam[q * p.N + id] * wR<R>(q);
            const R k = R(3) + R(9) * cu;
            gx += t * plus_c<cx(q)>(-R(3) * ux, k);
            gy += t * plus_c<cy(q)>(-R(3) * uy, k);
            gz += t * plus_c<cz(q)>(-R(3) * uz, k);
        });
        g[id] = (double)gx;
        g[p.N + id] = (double)gy;
        g[2 * p.N + id] = (double)gz;
    }
}

int blocks_for(int64_t n) { return (int)((n + 255) / 256); }

#define ACK(call)                                                                          \
    do {                                                                                   \
        cudaError_t e_ = (call);                                                           \
        if (e_ != cudaSuccess) {                                                           \
            set_error(std::string("lbm_adjoint: ") + #call + ": " + cudaGetErrorString(e_)); \
            return LBM_ERR_CUDA;                                                           \
        }                                                                                  \
    } while (0)

// The device buffers of one run, one allocation: laid out by add(), taken by
// alloc(), released by the destructor.  (Thirteen allocations and their releases
// cost 4 ms of a call.)
struct AdjBuffers {
    char* base = nullptr;
    size_t bytes = 0;
    std::vector<std::pair<void**, size_t>> parts;
    template <class T>
    void add(T** p, size_t n) {
        parts.push_back({reinterpret_cast<void**>(p), bytes});
        bytes += (sizeof(T) * (n ? n : 1) + 255) / 256 * 256;
    }
    bool alloc() {
        if (cudaMalloc((void**)&base, bytes) != cudaSuccess) return false;
        for (auto& q : parts) *q.first = base + q.second;
        return true;
    }
    ~AdjBuffers() { cudaFree(base); }
};

template <class R>
void run_fwd(const AdjP<R>& p, const R* f, R* fn, const double* uin, double* drag, cudaStream_t s) {
    // 32-bit element offsets while every slot index 19*N fits in them
    if ((uint64_t)p.N * 19u < (1ull << 32)) launch_after(adj_fwd<R, uint32_t>, blocks_for(p.N), 256, 0, s, p, f, fn, uin, drag);
    else launch_after(adj_fwd<R, int64_t>, blocks_for(p.N), 256, 0, s, p, f, fn, uin, drag);
}
template <class R>
void run_bwd(const AdjP<R>& p, const R* f, const R* lam1, R* lam0, const double* uin, double* guin, R wd,
             cudaStream_t s) {
    if ((uint64_t)p.N * 19u < (1ull << 32))
        launch_after(adj_bwd<R, uint32_t>, blocks_for(p.N), 256, 0, s, p, f, lam1, lam0, uin, guin, wd);
    else launch_after(adj_bwd<R, int64_t>, blocks_for(p.N), 256, 0, s, p, f, lam1, lam0, uin, guin, wd);
}

template <class R>
int adjoint_run(const lbm_adj_problem* pr, const uint8_t* h_mask, const double* h_uin,
                const double* h_u0, double* J, double* h_g_uin, double* h_g_u0, cudaStream_t s) {
    const int64_t N = (int64_t)pr->nx * pr->ny * pr->nz;
    const int64_t NI = (int64_t)pr->ny * pr->nz;
    const int steps = pr->n_steps, K = pr->checkpoint_every;
    const int wb = pr->window_begin, we = pr->window_end;
    const int nwin = we - wb + 1;
    const bool want_grad = h_g_uin || h_g_u0;
    AdjP<R> p{nullptr, nullptr, pr->nx, pr->ny, pr->nz, N, R(1) / (R)pr->tau, (R)pr->force[0], (R)pr->force[1],
              (R)pr->force[2]};
    const int grid = blocks_for(N);
    const int small = grid < num_sms() * 8 ? grid : num_sms() * 8;   // the set-up kernels stride over the cells
    AdjBuffers B;
    double *d_uin = nullptr, *d_u0 = nullptr, *d_drag = nullptr, *d_J = nullptr, *d_guin = nullptr, *d_gu0 = nullptr;
    R *fa = nullptr, *fb = nullptr;
    const int nseg = (steps - 1) / K + 1;
    const int last0 = (nseg - 1) * K;                 // first state of the last segment
    const size_t state = 19 * (size_t)N;
    const int inner = std::min(K, steps) - 1;         // states of a segment behind its checkpoint
    R* ckpt = nullptr;     // f^{kK}, k = 0 .. nseg-1, written there by the step that produces them
    R* seg = nullptr;      // f^{n0+1} .. f^{n0+inner} of the segment being reversed
    uint8_t *mask = nullptr, *flags = nullptr;
    uint32_t* links = nullptr;
    B.add(&mask, N); B.add(&flags, N); B.add(&links, N);
    B.add(&d_uin, NI); B.add(&d_u0, 3 * N); B.add(&d_drag, grid); B.add(&d_J, 1);
    B.add(&fa, state); B.add(&fb, state);
    if (want_grad) {
        B.add(&ckpt, (size_t)nseg * state); B.add(&seg, (size_t)inner * state);
        B.add(&d_guin, NI); B.add(&d_gu0, 3 * N);
    }
    if (!B.alloc()) { set_error("lbm_adjoint: device allocation failed"); return LBM_ERR_ALLOC; }
    ACK(cudaMemcpyAsync(mask, h_mask, (size_t)N, cudaMemcpyDefault, s));
    ACK(launch_build_flags(mask, nullptr, flags, links, pr->nx, pr->ny, pr->nz, 1, s));
    p.flags = flags;
    p.links = links;
    auto seg_state = [&](int k, int j) { return j == 0 ? ckpt + (size_t)k * state : seg + (size_t)(j - 1) * state; };
    ACK(cudaMemcpyAsync(d_uin, h_uin, sizeof(double) * NI, cudaMemcpyDefault, s));
    ACK(cudaMemcpyAsync(d_u0, h_u0, sizeof(double) * 3 * N, cudaMemcpyDefault, s));
    ACK(cudaMemsetAsync(d_drag, 0, sizeof(double) * grid, s));
    R* cur = want_grad ? ckpt : fa;
    adj_init<R><<<small, 256, 0, s>>>(p, d_u0, cur);
    ACK(cudaGetLastError());
    // forward: f^{n-1} -> f^n.  Checkpoints and the last segment's states are
    // written where the reverse pass reads them, so nothing is copied and the
    // last segment is not recomputed; the drag of the window's steps adds up in d_drag.
    for (int n = 1; n <= steps; ++n) {
        R* dst = cur == fa ? fb : fa;
        if (want_grad && n < steps) {
            if (n % K == 0) dst = seg_state(n / K, 0);
            else if (n > last0) dst = seg_state(nseg - 1, n - last0);
        }
        run_fwd<R>(p, cur, dst, d_uin, n >= wb && n <= we ? d_drag : nullptr, s);
        ACK(cudaGetLastError());
        cur = dst;
    }
    adj_sum<<<1, 1024, 0, s>>>(d_drag, grid, d_J);
    ACK(cudaGetLastError());
    if (want_grad) {
        // reverse: lambda^steps = 0; lambda^{n-1} from lambda^n and f^{n-1}
        R* lam1 = fa;
        R* lam0 = fb;
        ACK(cudaMemsetAsync(lam1, 0, sizeof(R) * state, s));
        ACK(cudaMemsetAsync(d_guin, 0, sizeof(double) * NI, s));
        for (int k = nseg - 1; k >= 0; --k) {
            const int n0 = k * K;                            // f^{n0} is the checkpoint
            const int n1 = std::min(steps, n0 + K);          // states f^{n0} .. f^{n1-1} are needed
            if (k < nseg - 1)
                for (int j = 1; j < n1 - n0; ++j) {
                    run_fwd<R>(p, seg_state(k, j - 1), seg_state(k, j), d_uin, nullptr, s);
                    ACK(cudaGetLastError());
                }
            for (int n = n1; n > n0; --n) {
                const R wd = (n >= wb && n <= we) ? R(1) / (R)nwin : R(0);
                run_bwd<R>(p, seg_state(k, n - 1 - n0), lam1, lam0, d_uin, d_guin, wd, s);
                ACK(cudaGetLastError());
                std::swap(lam0, lam1);
            }
        }
        adj_grad_u0<R><<<small, 256, 0, s>>>(p, d_u0, lam1, d_gu0);
        ACK(cudaGetLastError());
        if (h_g_uin) ACK(cudaMemcpyAsync(h_g_uin, d_guin, sizeof(double) * NI, cudaMemcpyDefault, s));
        if (h_g_u0) ACK(cudaMemcpyAsync(h_g_u0, d_gu0, sizeof(double) * 3 * N, cudaMemcpyDefault, s));
    }
    double acc = 0.0;
    ACK(cudaMemcpyAsync(&acc, d_J, sizeof(double), cudaMemcpyDeviceToHost, s));
    ACK(cudaStreamSynchronize(s));
    *J = acc / nwin;
    return LBM_OK;
}

}  // namespace

}  // namespace lbm

extern "C" int lbm_adjoint_run(const lbm_adj_problem* p, const uint8_t* host_mask, const double* u_inlet,
                               const double* u0, double* objective, double* grad_inlet, double* grad_u0) {
    using lbm::set_error;
    if (!p || !host_mask || !u_inlet || !u0 || !objective) { set_error("lbm_adjoint_run: null argument"); return LBM_ERR_INVALID; }
    if (p->nx < 3 || p->ny < 1 || p->nz < 1 || !(p->tau > 0.5) || p->n_steps < 1 || p->checkpoint_every < 1 ||
        p->window_begin < 1 || p->window_end < p->window_begin || p->window_end > p->n_steps ||
        (p->precision != 0 && p->precision != 1)) {
        set_error("lbm_adjoint_run: bad problem (nx >= 3, tau > 0.5, 1 <= window_begin <= window_end <= n_steps, "
                  "checkpoint_every >= 1, precision 0|1)");
        return LBM_ERR_INVALID;
    }
    if ((int64_t)p->nx * p->ny * p->nz > ((int64_t)1 << 31)) { set_error("lbm_adjoint_run: grid too large"); return LBM_ERR_SIZE; }
    cudaStream_t s = nullptr;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) {
        set_error("lbm_adjoint_run: cannot create a stream");
        return LBM_ERR_CUDA;
    }
    const int rc = p->precision == 0
                       ? lbm::adjoint_run<float>(p, host_mask, u_inlet, u0, objective, grad_inlet, grad_u0, s)
                       : lbm::adjoint_run<double>(p, host_mask, u_inlet, u0, objective, grad_inlet, grad_u0, s);
    cudaStreamDestroy(s);
    return rc;
}
