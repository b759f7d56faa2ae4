// Two Legacy/Hybrid steps in one pass over memory (FP32, no solid cells, no duct).
//
// A BGK step is bound by the 152 B per cell that every step reads and writes
// (0.87-0.94 of the measured copy bandwidth one step at a time, lbm_aa.cu), so
// the way to a faster step is to touch memory once for two of them.  This kernel
// runs the odd AA step and the even step behind it: it gathers f_q from slot
// opp(q) of x - c_q, collides, streams into shared memory, collides again and
// stores f*_q into slot opp(q) of x -- the layout it started from, in a second
// buffer (a cell's sources are other blocks' cells, so it cannot run in place).
// Per two steps it reads each population once (plus the tile's halo) and writes
// it once.  The arithmetic is that of the single steps (lbm_vec.cuh), so states
// are the same bits.
//
// The block shape is the HOME kernel's (lbm_home.cu): a 32 x 8 tile of an (x, y)
// plane marching along z, two x-adjacent cells per lane on paired FP32
// instructions; four tile warps, one halo-row warp and one warp of halo-column
// positions, which run the first step for the cells around the tile.  The first
// step's populations go into a ring in shared memory, indexed by the cell that
// receives them and grouped by c_z: 3 plane slots for c_z = +1, 2 for c_z = 0 and 1
// for c_z = -1.  The next plane's populations are loaded into registers before the
// second step of the plane behind, so that they arrive during it.
//
// Measured (512^3, us per step): 3320 one step at a time, 2290 here (4.5 TB/s of
// populations).  What bounds it is the latency of its loads and barriers at 12
// warps per SM: without the collisions it takes 2200, without the loads 1500,
// without the stores 1820.  Slower: 3 blocks/SM (spills) 3180, a 32 x 12 tile at 16
// warps 2510, a ring that needs one barrier per plane (82 KB) 2430, aligned loads
// with shuffles for the shifted pairs 2310-2340, the loads staged in shared memory
// by 16-byte asynchronous copies 2890 (1.6 times the L2 sectors).
#include <algorithm>

#include "lbm_common.cuh"
#include "lbm_internal.h"
#include "lbm_vec.cuh"

namespace lbm {
namespace {

constexpr int TX = 32, TY = 8;              // tile (cells); 16 pairs of cells in a row
constexpr int NCW = TY / 2;                 // tile warps: two rows of 16 pairs
constexpr int NCOL = 2 * TY + 4;            // halo-column positions and corners
constexpr int NT = (NCW + 2) * 32;          // + the halo-row warp + the halo-column warp
constexpr int NB = 2;                       // blocks per SM: 168 registers hold the next plane's 19 pairs
// ring plane: the tile with a margin of one row and two columns, so that every position
// stores all its populations without a test; margins are never read.  Halo rows reach
// one row past them: a spare row lies before the ring and one behind it.
constexpr int RP = TX + 4, PL = RP * (TY + 2);
constexpr int UP_SZ = 5 * PL, MID_SZ = 9 * PL, DN_SZ = 5 * PL;
constexpr int UP_OFF = RP, MID_OFF = UP_OFF + 3 * UP_SZ, DN_OFF = MID_OFF + 2 * MID_SZ;
constexpr int SMEM_FLOATS = DN_OFF + DN_SZ + RP;       // 54.9 KB

// index of q inside its c_z group
__host__ __device__ constexpr int gidx(int q) {
    constexpr int t[19] = {0, 1, 2, 3, 4, 0, 0, 5, 6, 7, 8, 1, 2, 1, 2, 3, 4, 3, 4};
    return t[q];
}
template <int q> struct QI { static constexpr int value = q; };
template <int Q0, int Q1, class F>
__device__ __forceinline__ void static_for(F&& fn) {
    if constexpr (Q0 < Q1) {
        fn(QI<Q0>{});
        static_for<Q0 + 1, Q1>(fn);
    }
}

// base + 4 idx in one instruction
__device__ __forceinline__ const float* at(const float* base, uint32_t idx) {
    uint64_t a;
    asm("mad.wide.u32 %0, %1, 4, %2;" : "=l"(a) : "r"(idx), "l"(base));
    return reinterpret_cast<const float*>(a);
}

// VEC: nx is even, so a pair's two cells are one aligned 8-byte word of every plane
template <bool VEC>
__global__ void __launch_bounds__(NT, NB) aa_pair(AAParams p, const float* __restrict__ fa, float* __restrict__ fb,
                                                  int zchunk) {
    extern __shared__ __align__(16) float sm[];
    step_begin();
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    const int tiles_x = (nx + TX - 1) / TX, tiles_y = (ny + TY - 1) / TY;
    int b = blockIdx.x;
    const int x0 = (b % tiles_x) * TX; b /= tiles_x;
    const int y0 = (b % tiles_y) * TY; b /= tiles_y;
    const int z0 = b * zchunk, z1 = min(nz, z0 + zchunk);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto mod = [](int v, int n) { const int r = v % n; return r < 0 ? r + n : r; };
    const uint32_t plane = (uint32_t)nx * (uint32_t)ny;
    const uint32_t N = (uint32_t)p.N;

    // this thread's role and the tile position of its first cell
    enum { TILE, ROW, COL, IDLE };
    int role, px, py;
    if (warp < NCW) { role = TILE; px = 2 * (lane & 15); py = 2 * warp + (lane >> 4); }
    else if (warp == NCW) { role = ROW; px = 2 * (lane & 15); py = (lane >> 4) ? TY : -1; }
    else if (lane < 2 * TY) { role = COL; px = lane < TY ? -1 : TX; py = lane & (TY - 1); }
    else if (lane < NCOL) { role = COL; px = (lane & 1) ? TX : -1; py = (lane & 2) ? TY : -1; }
    else { role = IDLE; px = 0; py = 0; }
    const bool pair = role == TILE || role == ROW;
    const bool own0 = role == TILE && y0 + py < ny && x0 + px < nx;
    const bool own1 = role == TILE && y0 + py < ny && x0 + px + 1 < nx;
    // the cells it stands for, periodic
    const int gy = mod(y0 + py, ny), gx0 = mod(x0 + px, nx), gx1 = gx0 + 1 == nx ? 0 : gx0 + 1;
    const uint32_t cell0 = (uint32_t)gy * (uint32_t)nx + (uint32_t)gx0;
    const int pos = (py + 1) * RP + px + 2;      // in a ring plane
    const float omega = p.hybrid ? p.omega_s : p.omega;      // without a band every Hybrid cell takes omega_s
    // element offsets of rows y-1, y, y+1 (at its first cell) and of the cells x-1, x+1, x+2 from the first
    const uint32_t yo[3] = {(uint32_t)mod(gy - 1, ny) * (uint32_t)nx + (uint32_t)gx0, cell0,
                            (uint32_t)mod(gy + 1, ny) * (uint32_t)nx + (uint32_t)gx0};
    const int dm = gx0 == 0 ? nx - 1 : -1, d1 = gx1 - gx0, d2 = (gx1 + 1 == nx ? 0 : gx1 + 1) - gx0;

    float2 v[19];                  // the populations of the plane that arrives next (halo columns: .x)
    auto load = [&](int pz) {
        const int zc = pz < 0 ? pz + nz : (pz >= nz ? pz - nz : pz);
        const uint32_t zb[3] = {(uint32_t)(zc == 0 ? nz - 1 : zc - 1) * plane, (uint32_t)zc * plane,
                                (uint32_t)(zc == nz - 1 ? 0 : zc + 1) * plane};
        // a population arriving along q was left in slot opp(q) of x - c_q
        auto from = [&](auto qi) -> const float* {
            constexpr int q = decltype(qi)::value;
            return at(fa, (uint32_t)opp(q) * N + zb[1 - cz(q)] + yo[1 - cy(q)]);
        };
        if (pair) {
            static_for<0, 19>([&](auto qi) {
                constexpr int q = decltype(qi)::value;
                const float* const s = from(qi);
                if constexpr (cx(q) == 0) {
                    if constexpr (VEC) v[q] = __ldg(reinterpret_cast<const float2*>(s));
                    else v[q] = make_float2(__ldg(s), __ldg(s + d1));
                } else if constexpr (cx(q) > 0) {
                    v[q] = make_float2(__ldg(s + dm), __ldg(s));
                } else {
                    v[q] = make_float2(__ldg(s + (VEC ? 1 : d1)), __ldg(s + d2));
                }
            });
        } else {
            static_for<0, 19>([&](auto qi) {
                constexpr int q = decltype(qi)::value;
                v[q].x = __ldg(from(qi) + (cx(q) == 0 ? 0 : (cx(q) > 0 ? dm : d1)));
            });
        }
    };

    int t3 = mod(z0 - 1, 3);        // pz mod 3: the UP slot of plane pz
    load(z0 - 1);
    for (int pz = z0 - 1; pz <= z1; ++pz) {
        const int stage = min(pz - (z0 - 1), 2);      // 0: only upward populations are wanted, 1: + in-plane, 2: all
        float* const UPp = sm + UP_OFF + t3 * UP_SZ;               // leave pz upward
        float* const MIDp = sm + MID_OFF + (pz & 1) * MID_SZ;
        float* const DNg = sm + DN_OFF;                            // arrive at pz - 1 from above
        auto slot = [&](auto qi) -> float* {       // where q of this position streams to
            constexpr int q = decltype(qi)::value;
            return (cz(q) > 0 ? UPp : (cz(q) == 0 ? MIDp : DNg)) + gidx(q) * PL + pos + (cy(q) * RP + cx(q));
        };
        // 1. plane pz: first step, into the ring
        if (pair) {
            const CellV<float2> m = moments(v, p.fx, p.fy, p.fz);
            collide(v, m, make_float2(omega, omega));
            auto put = [&](auto qi) {
                constexpr int q = decltype(qi)::value;
                float* const d = slot(qi);
                if constexpr (cx(q) == 0) st_pair(d, v[q]);
                else { d[0] = v[q].x; d[1] = v[q].y; }
            };
            auto group = [&](auto zi) {
                constexpr int Z = decltype(zi)::value;
                static_for<0, 19>([&](auto qi) {
                    constexpr int q = decltype(qi)::value;
                    if constexpr (cz(q) == Z && cy(q) != 0) put(qi);
                });
                if (role == TILE)
                    static_for<0, 19>([&](auto qi) {
                        constexpr int q = decltype(qi)::value;
                        if constexpr (cz(q) == Z && cy(q) == 0) put(qi);
                    });
            };
            group(QI<1>{});
            if (stage >= 1) group(QI<0>{});
            if (stage >= 2) group(QI<-1>{});
        } else if (role == COL) {
            float c[19];
            static_for<0, 19>([&](auto qi) { c[decltype(qi)::value] = v[decltype(qi)::value].x; });
            const CellV<float> m = moments(c, p.fx, p.fy, p.fz);
            collide(c, m, omega);
            static_for<0, 19>([&](auto qi) {
                constexpr int q = decltype(qi)::value;
                if constexpr (cx(q) != 0) {
                    if (cz(q) > 0 || (cz(q) == 0 && stage >= 1) || stage >= 2) *slot(qi) = c[q];
                }
            });
        }
        if (pz < z1) load(pz + 1);
        if (stage >= 2) {
            __syncthreads();      // the ring of pz - 1 is complete
            // 2. plane pz - 1: second step, from the ring to memory
            if (own0) {
                const int z = pz - 1;
                const float* const g_up = sm + UP_OFF + (t3 == 2 ? 0 : t3 + 1) * UP_SZ + pos;     // left pz - 2
                const float* const g_mid = sm + MID_OFF + (z & 1) * MID_SZ + pos;
                const float* const g_dn = DNg + pos;
                float2 o[19];
                static_for<0, 19>([&](auto qi) {
                    constexpr int q = decltype(qi)::value;
                    o[q] = ld_pair((cz(q) > 0 ? g_up : (cz(q) == 0 ? g_mid : g_dn)) + gidx(q) * PL);
                });
                const CellV<float2> m = moments(o, p.fx, p.fy, p.fz);
                collide(o, m, make_float2(omega, omega));
                static_for<0, 19>([&](auto qi) {
                    constexpr int q = decltype(qi)::value;
                    float* const dst = const_cast<float*>(at(fb, (uint32_t)opp(q) * N + (uint32_t)z * plane + cell0));
                    if constexpr (VEC) {
                        __stcs(reinterpret_cast<float2*>(dst), o[q]);
                    } else {
                        __stcs(dst, o[q].x);
                        if (own1) __stcs(dst + 1, o[q].y);
                    }
                });
            }
            __syncthreads();      // the ring of pz - 2 is free
        }
        t3 = t3 == 2 ? 0 : t3 + 1;
    }
}

}  // namespace

// Planes per block.  A block runs zchunk + 2 planes (two of them only to fill the
// ring), so long chunks do less work and short ones leave more blocks: the chunk
// with the least a (waves + 1/4)(zchunk + 2) + b blocks (zchunk + 2), the measured
// time of one step in us to about 5 % from 32^3 to 384^3 (64^3: 4 planes 7.2 us, 2
// and 8 planes 8.3; 96^3: 12 planes 18.4, 8 and 16 planes 20.6 and 22.3; 256x128x128:
// 16 planes 78.6, 4 planes 88, 48 planes 94).  Against single steps (us per step
// before -> with it): 32^3 6.2 -> 4.1, 64^3 12.3 -> 7.2, 128^3 58.4 -> 41.0,
// 33x64x300 (half-empty tiles) 27.0 -> 22.5, 300x33x64 18.6 -> 17.2, 256x128x128
// 107.6 -> 78.6, 256^3 419 -> 285, 384^3 1467 -> 980.  It is taken wherever its
// 32-bit element offsets reach; 0 elsewhere.
int pair_zchunk(int nx, int ny, int nz, int storage) {
    if (storage != 0 || (uint64_t)nx * ny * nz * 19u >= (1ull << 32)) return 0;
    const int64_t tiles = (int64_t)((nx + TX - 1) / TX) * ((ny + TY - 1) / TY), slots = (int64_t)num_sms() * NB;
    int best = 1;
    double least = 1e300;
    for (int c : {1, 2, 4, 6, 8, 12, 16, 24, 32, 48}) {
        const int z = std::min(c, nz);
        const int64_t blocks = tiles * ((nz + z - 1) / z);
        const double cost = 0.73 * ((double)((blocks + slots - 1) / slots) + 0.25) * (z + 2) +
                            0.00124 * (double)(tiles * (nz + 2 * ((nz + z - 1) / z)));
        if (cost < least) { least = cost; best = z; }
    }
    return best;
}

cudaError_t launch_aa_pair(const AAParams& p, const float* fa, float* fb, int zchunk, cudaStream_t s) {
    const int grid = ((p.nx + TX - 1) / TX) * ((p.ny + TY - 1) / TY) * ((p.nz + zchunk - 1) / zchunk);
    const size_t smem = sizeof(float) * SMEM_FLOATS;
    return p.nx % 2 == 0 ? launch_after(aa_pair<true>, grid, NT, smem, s, p, fa, fb, zchunk)
                         : launch_after(aa_pair<false>, grid, NT, smem, s, p, fa, fb, zchunk);
}

cudaError_t pair_prepare() {
    const int smem = (int)(sizeof(float) * SMEM_FLOATS);
    cudaError_t e = cudaFuncSetAttribute((const void*)aa_pair<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute((const void*)aa_pair<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return e;
}

}  // namespace lbm
