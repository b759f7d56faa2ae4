// Two Legacy/Hybrid steps in one pass over memory (FP32).
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
// Links that do not stream (solid cells, a duct's ends): the first step lets every
// population go to the place in the ring that it would stream to, inlet and outlet
// values in place of what leaves the duct, and the second step of a cell takes back
// what it left over such a link, where otherwise it would take what came.  Solid
// cells are not touched; their populations are copied to the second buffer once a call.
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
// Ring plane: the tile with a margin of two columns on either side and of one row above
// and two below, so that every position stores all its populations without a test.
// What a tile cell left in the margin (or in a solid cell's place) is what comes back
// to it over a link that does not stream; nothing else is read there.  Halo rows reach
// two rows above: into the last row of the plane before, or the spare row before the ring.
// With a mask the down-going group has 2 slots: a cell of plane p that gets a downward
// population back needs it when p is gathered, one plane after it left.
constexpr int RP = TX + 4, PL = RP * (TY + 3);
constexpr int UP_SZ = 5 * PL, MID_SZ = 9 * PL, DN_SZ = 5 * PL;
constexpr int UP_OFF = RP, MID_OFF = UP_OFF + 3 * UP_SZ, DN_OFF = MID_OFF + 2 * MID_SZ;
__host__ __device__ constexpr int smem_floats(bool mask) { return DN_OFF + (mask ? 2 : 1) * DN_SZ; }   // 60.3, 68.3 KB

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

// base + 4 idx
__device__ __forceinline__ const float* at(const float* base, uint32_t idx) {
    uint64_t a;
    asm("mad.wide.u32 %0, %1, 4, %2;" : "=l"(a) : "r"(idx), "l"(base));
    return reinterpret_cast<const float*>(a);
}

// the same rule as the single steps' (lbm_aa.cu)
__device__ __forceinline__ float inlet_value(int q, float r, float kin) { return wq(q) * r * kin; }

// VEC: nx is even, so a pair's two cells are one aligned 8-byte word of every plane.
// MASK: the grid has solid cells, a band or a duct's ends (flags and links).
template <bool MASK, bool VEC>
__global__ void __launch_bounds__(NT, NB) aa_pair(AAParams p, const float* fa, float* fb, int zchunk) {
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
    const uint32_t cell0 = (uint32_t)gy * (uint32_t)nx + (uint32_t)gx0, cell1 = (uint32_t)gy * (uint32_t)nx + (uint32_t)gx1;
    const int pos = (py + 1) * RP + px + 2;      // in a ring plane
    const float omega = p.hybrid ? p.omega_s : p.omega;      // of the cells outside the band
    const float kin = 1.f + 3.f * p.u_in + 3.f * p.u_in * p.u_in;
    // element offsets of rows y-1, y, y+1 (at its first cell) and of the cells x-1, x+1, x+2 from the first
    const uint32_t yo[3] = {(uint32_t)mod(gy - 1, ny) * (uint32_t)nx + (uint32_t)gx0, cell0,
                            (uint32_t)mod(gy + 1, ny) * (uint32_t)nx + (uint32_t)gx0};
    const int dm = gx0 == 0 ? nx - 1 : -1, d1 = gx1 - gx0, d2 = (gx1 + 1 == nx ? 0 : gx1 + 1) - gx0;

    float2 v[19];                  // the populations of the plane that arrives next (halo columns: .x)
    // Flag bytes and link words of the two cells: of the plane in v, of the one behind it (they
    // decide its loads) and of the plane that is gathered.  Flags are requested one plane
    // before the links they tell to read, so that neither is waited for.
    uint32_t fl = 0, lk0 = 0, lk1 = 0, fn = 0, ln0 = 0, ln1 = 0, fg = 0, lg0 = 0, lg1 = 0, ff = 0;
    auto plane_of = [&](int pz) {
        return (uint32_t)(pz < 0 ? pz + nz : (pz >= nz ? pz - nz : pz)) * plane;
    };
    auto load_flags = [&](int pz) {
        if constexpr (MASK) {
            const uint32_t zb = plane_of(pz);
            if (VEC && pair) ff = __ldg(reinterpret_cast<const uint16_t*>(p.flags + (zb + cell0)));
            else ff = __ldg(p.flags + (zb + cell0)) | ((pair ? (uint32_t)__ldg(p.flags + (zb + cell1)) : 0u) << 8);
        }
    };
    auto load_links = [&](int pz) {       // of the plane whose flags are in ff
        if constexpr (MASK) {
            const uint32_t zb = plane_of(pz);
            fn = ff;
            ln0 = (fn & F_SPECIAL) ? __ldg(p.links + (zb + cell0)) & 0x7ffffu : 0u;
            ln1 = (fn & (F_SPECIAL << 8)) ? __ldg(p.links + (zb + cell1)) & 0x7ffffu : 0u;
        }
    };
    auto load = [&](int pz) {
        const int zc = pz < 0 ? pz + nz : (pz >= nz ? pz - nz : pz);
        const uint32_t zb[3] = {(uint32_t)(zc == 0 ? nz - 1 : zc - 1) * plane, (uint32_t)zc * plane,
                                (uint32_t)(zc == nz - 1 ? 0 : zc + 1) * plane};
        // a population arriving along q was left in slot opp(q) of x - c_q, or, where that
        // link does not stream, in the cell's own slot q
        auto place = [&](auto qi) -> uint32_t {
            constexpr int q = decltype(qi)::value;
            return (uint32_t)opp(q) * N + zb[1 - cz(q)] + yo[1 - cy(q)];
        };
        auto from = [&](auto qi) { return at(fa, place(qi)); };
        fl = fn; lk0 = ln0; lk1 = ln1;
        if (MASK && __any_sync(0xffffffffu, (lk0 | lk1) != 0u)) {
            static_for<0, 19>([&](auto qi) {
                constexpr int q = decltype(qi)::value;
                const uint32_t s = place(qi), own = (uint32_t)q * N + zb[1];
                const uint32_t s0 = s + (uint32_t)(cx(q) == 0 ? 0 : (cx(q) > 0 ? dm : d1));
                const uint32_t s1 = s + (uint32_t)(cx(q) == 0 ? d1 : (cx(q) > 0 ? 0 : d2));
                v[q].x = __ldca(at(fa, ((lk0 >> opp(q)) & 1u) ? own + cell0 : s0));
                if (pair) v[q].y = __ldca(at(fa, ((lk1 >> opp(q)) & 1u) ? own + cell1 : s1));
            });
        } else if (pair) {
            static_for<0, 19>([&](auto qi) {
                constexpr int q = decltype(qi)::value;
                const float* const s = from(qi);
                if constexpr (cx(q) == 0) {
                    if constexpr (VEC) v[q] = __ldca(reinterpret_cast<const float2*>(s));
                    else v[q] = make_float2(__ldca(s), __ldca(s + d1));
                } else if constexpr (cx(q) > 0) {
                    v[q] = make_float2(__ldca(s + dm), __ldca(s));
                } else {
                    v[q] = make_float2(__ldca(s + (VEC ? 1 : d1)), __ldca(s + d2));
                }
            });
        } else {
            static_for<0, 19>([&](auto qi) {
                constexpr int q = decltype(qi)::value;
                v[q].x = __ldca(from(qi) + (cx(q) == 0 ? 0 : (cx(q) > 0 ? dm : d1)));
            });
        }
    };

    int t3 = mod(z0 - 1, 3);        // pz mod 3: the UP slot of plane pz
    load_flags(z0 - 1);
    load_links(z0 - 1);
    load_flags(z0);
    load(z0 - 1);
    load_links(z0);
    load_flags(z0 + 1);
    for (int pz = z0 - 1; pz <= z1; ++pz) {
        const int stage = min(pz - (z0 - 1), 2);      // 0: only upward populations are wanted, 1: + in-plane, 2: all
        float* const UPp = sm + UP_OFF + t3 * UP_SZ;               // leave pz upward
        float* const MIDp = sm + MID_OFF + (pz & 1) * MID_SZ;
        float* const DNg = sm + DN_OFF + (MASK ? (pz - 1) & 1 : 0) * DN_SZ;       // arrive at pz - 1 from above
        auto slot = [&](auto qi) -> float* {       // where q of this position streams to
            constexpr int q = decltype(qi)::value;
            return (cz(q) > 0 ? UPp : (cz(q) == 0 ? MIDp : DNg)) + gidx(q) * PL + pos + (cy(q) * RP + cx(q));
        };
        // 1. plane pz: first step, into the ring
        if (pair) {
            const CellV<float2> m = moments(v, p.fx, p.fy, p.fz);
            float2 om = make_float2(omega, omega);
            if constexpr (MASK) {
                if (fl & F_BAND) om.x = p.omega;
                if (fl & (F_BAND << 8)) om.y = p.omega;
            }
            collide(v, m, om);
            if (MASK && p.duct) {
                // what leaves past the inlet is the inlet population that comes back, past the
                // outlet the population of the opposite direction
                if (gx0 == 0) static_for<0, 19>([&](auto qi) {
                    constexpr int q = decltype(qi)::value;
                    if constexpr (cx(q) < 0) v[q].x = inlet_value(q, m.r.x, kin);
                });
                if (gx0 == nx - 1) static_for<0, 19>([&](auto qi) {
                    constexpr int q = decltype(qi)::value;
                    if constexpr (cx(q) > 0) v[q].x = v[opp(q)].x;
                });
                if (gx1 == nx - 1) static_for<0, 19>([&](auto qi) {
                    constexpr int q = decltype(qi)::value;
                    if constexpr (cx(q) > 0) v[q].y = v[opp(q)].y;
                });
            }
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
            if (stage >= (MASK ? 1 : 2)) group(QI<-1>{});
        } else if (role == COL) {
            float c[19];
            static_for<0, 19>([&](auto qi) { c[decltype(qi)::value] = v[decltype(qi)::value].x; });
            const CellV<float> m = moments(c, p.fx, p.fy, p.fz);
            collide(c, m, (MASK && (fl & F_BAND)) ? p.omega : omega);
            static_for<0, 19>([&](auto qi) {
                constexpr int q = decltype(qi)::value;
                if constexpr (cx(q) != 0) {
                    if (cz(q) > 0 || (cz(q) == 0 && stage >= 1) || stage >= 2) *slot(qi) = c[q];
                }
            });
        }
        const uint32_t fp = fl, lp0 = lk0, lp1 = lk1;
        if (pz < z1) load(pz + 1);
        if (pz + 1 < z1) {
            load_links(pz + 2);
            if (pz + 2 < z1) load_flags(pz + 3);
        }
        if (stage >= 2) {
            __syncthreads();      // the ring of pz - 1 is complete
            // 2. plane pz - 1: second step, from the ring to memory; solid cells keep what they have
            const bool st0 = own0 && !(MASK && (fg & F_SOLID)), st1 = own1 && !(MASK && (fg & (F_SOLID << 8)));
            const bool special = MASK && __any_sync(0xffffffffu, (lg0 | lg1) != 0u);
            if (st0 || st1) {
                const int z = pz - 1;
                const float* const g_up = sm + UP_OFF + (t3 == 2 ? 0 : t3 + 1) * UP_SZ + pos;     // left pz - 2
                const float* const g_mid = sm + MID_OFF + (z & 1) * MID_SZ + pos;
                const float* const g_dn = DNg + pos;
                float2 o[19];
                static_for<0, 19>([&](auto qi) {
                    constexpr int q = decltype(qi)::value;
                    o[q] = ld_pair((cz(q) > 0 ? g_up : (cz(q) == 0 ? g_mid : g_dn)) + gidx(q) * PL);
                });
                if (special) {
                    // over a link that does not stream the cell's own population comes back: it
                    // left it in slot opp(q) of the cell at the link's end
                    const float* const h_up = sm + UP_OFF + (t3 == 0 ? 2 : t3 - 1) * UP_SZ + pos;     // left pz - 1
                    const float* const h_dn = sm + DN_OFF + (pz & 1) * DN_SZ + pos;
                    static_for<1, 19>([&](auto qi) {
                        constexpr int q = decltype(qi)::value, n = opp(q);
                        const float* const h = (cz(n) > 0 ? h_up : (cz(n) == 0 ? g_mid : h_dn)) + gidx(n) * PL + (cy(n) * RP + cx(n));
                        if ((lg0 >> n) & 1u) o[q].x = h[0];
                        if ((lg1 >> n) & 1u) o[q].y = h[1];
                    });
                }
                const CellV<float2> m = moments(o, p.fx, p.fy, p.fz);
                float2 om = make_float2(omega, omega);
                if constexpr (MASK) {
                    if (fg & F_BAND) om.x = p.omega;
                    if (fg & (F_BAND << 8)) om.y = p.omega;
                }
                collide(o, m, om);
                if (MASK && p.duct) {
                    const bool in = gx0 == 0, out0 = gx0 == nx - 1, out1 = gx1 == nx - 1;
                    if (in || out0 || out1) {
                        static_for<0, 19>([&](auto qi) {
                            constexpr int q = decltype(qi)::value;
                            if constexpr (cx(q) > 0) {
                                // outlet: slot opp(q) takes f*_opp(q); inlet: slot q takes the inlet population
                                constexpr int n = opp(q);
                                if (out0) o[q].x = o[n].x;
                                if (out1) o[q].y = o[n].y;
                                if (in) o[n].x = inlet_value(n, m.r.x, kin);
                            }
                        });
                    }
                }
                auto to = [&](auto qi) {
                    return const_cast<float*>(at(fb, (uint32_t)opp(decltype(qi)::value) * N + (uint32_t)z * plane + cell0));
                };
                if (VEC && (!MASK || (st0 && st1))) {
                    static_for<0, 19>([&](auto qi) { __stcs(reinterpret_cast<float2*>(to(qi)), o[decltype(qi)::value]); });
                } else {
                    static_for<0, 19>([&](auto qi) {
                        float* const dst = to(qi);
                        if (st0) __stcs(dst, o[decltype(qi)::value].x);
                        if (st1) __stcs(dst + 1, o[decltype(qi)::value].y);
                    });
                }
            }
            __syncthreads();      // the ring of pz - 2 is free
        }
        fg = fp; lg0 = lp0; lg1 = lp1;
        t3 = t3 == 2 ? 0 : t3 + 1;
    }
}

// the solid cells' populations into the second buffer (the two-step kernel does not touch them)
__global__ void __launch_bounds__(256) pair_solids(const uint8_t* __restrict__ flags, const float* fa, float* fb,
                                                   int64_t N) {
    step_begin();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N || !(flags[i] & F_SOLID)) return;
    for (int q = 0; q < 19; ++q) fb[q * N + i] = fa[q * N + i];
}

}  // namespace

// Planes per block, or 0 where single steps are faster.
//
// A block runs zchunk + 2 planes (two of them only to fill the ring), so long chunks do
// less work and short ones leave more blocks: the chunk with the least
// a (waves + t)(zchunk + 2) + b blocks (zchunk + 2), t = 1/4, the measured time of one
// step in us to about 5 % from 32^3 to 384^3 (64^3: 4 planes 7.2 us, 2 and 8 planes 8.3;
// 96^3: 12 planes 18.4, 8 and 16 planes 20.6 and 22.3; 256x128x128: 16 planes 78.6, 4
// planes 88, 48 planes 94); with a mask the blocks at walls take longer, and t = 1 keeps
// the last wave short (8 and 12 planes 100, 16 planes 104, 32 planes 115).
//
// Against single steps (us per step, before -> with it): 32^3 4.2 -> 2.5, 64^3 6.8 -> 6.4,
// 128x128x96 38.1 -> 32.4, 160^3 107 -> 81, 256x128x128 104 -> 81 (with walls and an
// obstacle 109 -> 100, as an inlet duct 116 -> 108), 256^3 414 -> 288 (442 -> 356,
// 468 -> 393).  Tiles that stick out of the grid do idle work: 33x64x300 (half of it)
// 20.0 -> 23.7, 300x33x64 (a quarter) 14.5 -> 17.0, 70x20x500 17.4 -> 20.5 -- but beyond
// L2 it pays even so (40x400x300, 62 % used: 138 -> 109).  With a mask it pays beyond
// L2 only (201x93x77 39.3 -> 44.8, 192x96x96 43.9 -> 45.7).
int pair_zchunk(int nx, int ny, int nz, int storage, bool mask) {
    if (storage != 0 || (uint64_t)nx * ny * nz * 19u >= (1ull << 32)) return 0;
    const int64_t tiles = (int64_t)((nx + TX - 1) / TX) * ((ny + TY - 1) / TY), slots = (int64_t)num_sms() * NB;
    const double used = (double)nx * ny / (double)(tiles * TX * TY);
    const bool big = (double)nx * ny * nz * 76.0 >= 200e6;      // the populations do not stay in L2
    if (mask ? !(big && used >= 0.75) : !(used >= 0.85 || (big && used >= 0.6))) return 0;
    int best = 1;
    double least = 1e300;
    for (int c : {1, 2, 4, 6, 8, 12, 16, 24, 32, 48}) {
        const int z = std::min(c, nz);
        const int64_t chunks = (nz + z - 1) / z, blocks = tiles * chunks;
        const double cost = 0.73 * ((double)((blocks + slots - 1) / slots) + (mask ? 1.0 : 0.25)) * (z + 2) +
                            0.00124 * (double)(tiles * (nz + 2 * chunks));
        if (cost < least) { least = cost; best = z; }
    }
    return best;
}

cudaError_t launch_aa_pair(const AAParams& p, const float* fa, float* fb, int zchunk, cudaStream_t s) {
    const int grid = ((p.nx + TX - 1) / TX) * ((p.ny + TY - 1) / TY) * ((p.nz + zchunk - 1) / zchunk);
    const bool mask = p.flags != nullptr;
    const size_t smem = sizeof(float) * smem_floats(mask);
    const bool vec = p.nx % 2 == 0;
    if (mask) return vec ? launch_after(aa_pair<true, true>, grid, NT, smem, s, p, fa, fb, zchunk)
                         : launch_after(aa_pair<true, false>, grid, NT, smem, s, p, fa, fb, zchunk);
    return vec ? launch_after(aa_pair<false, true>, grid, NT, smem, s, p, fa, fb, zchunk)
               : launch_after(aa_pair<false, false>, grid, NT, smem, s, p, fa, fb, zchunk);
}

cudaError_t launch_pair_solids(const AAParams& p, const float* fa, float* fb, cudaStream_t s) {
    if (!p.flags) return cudaSuccess;
    return launch_after(pair_solids, (unsigned)((p.N + 255) / 256), 256, 0, s, p.flags, fa, fb, p.N);
}

cudaError_t pair_prepare() {
    cudaError_t e = cudaSuccess;
    auto set = [&](const void* fn, bool mask) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(float) * smem_floats(mask)));
    };
    set((const void*)aa_pair<false, false>, false);
    set((const void*)aa_pair<false, true>, false);
    set((const void*)aa_pair<true, false>, true);
    set((const void*)aa_pair<true, true>, true);
    return e;
}

}  // namespace lbm
