// pipe_solve.cuh -- the 3D linear solve as a pipeline of specialised warps, one
// block per SM: the same iteration as krylov_solve (subsurface.cu) for handles
// with few tiles per SM, where that kernel is bound by latency.
//
// krylov_solve marches a thread down each column; every plane costs the chain of
// its stencil, sums and recurrence (1,300 cycles for a 128x128x30 domain, with
// everything it reads already in shared memory), plus a block barrier per chunk
// and two global round trips per batch of the back substitution.  Here the planes
// of a tile are computed by different warps at the same time, since only the two
// recurrences of the column solve have an order in k, and these run from shared
// memory.  All solves of a pass, krylov_solve / this in ms: 32x32x20 FP64 two steps
// 3.77 / 2.24, 53x37x21 FP64 2.16 / 1.22, 128x128x30 5.36 / 2.65, 384x384x40 48.8 /
// 33.2; more sizes at use_pipe.  What bounds it: in small handles the chain of a sweep
// (issue of the copies, recurrences, sums, grid barrier; 128x128x30 issues in 27 % of
// the cycles); in larger ones the chains of the plane warps' instructions, of which an
// SM has eight (384x384x40: issue 41 %, DRAM 39 % of peak).  krylov_solve spreads them
// over 28 warps per SM -- it keeps the largest handles (use_pipe).
#pragma once

#include "device_common.cuh"
#include "staging.cuh"

#define MAX_CYCLES 30
#define STEP_GROUPS 3  // tiles a block of k_step_pipe works on at the same time

namespace pipe {

// columns a 16-byte unit of an array holds: the x offset of a halo box
template <typename V>
__host__ __device__ constexpr int xoff() {
    return 16 / (int)sizeof(V);
}
// Bytes of one plane of a halo box of a tile of tx x ty columns.
template <typename V>
__host__ __device__ constexpr unsigned halo_bytes(int tx, int ty) {
    return (unsigned)((tx + 2 * xoff<V>()) * (ty + 2) * (int)sizeof(V));
}
// Box loads of the planes from k on of the tile at (x0, y0): of one array, or of
// a set of arrays (one behind the other).
template <typename V>
__device__ __forceinline__ void tma_halo(void *dst, const CUtensorMap *map, int x0, int y0, int k, uint64_t *bar) {
    tma_load_3d(dst, map, x0 - xoff<V>(), y0 - 1, k, bar);
}
template <typename V>
__device__ __forceinline__ void tma_halo4(void *dst, const CUtensorMap *map, int x0, int y0, int k, uint64_t *bar) {
    tma_load_4d(dst, map, x0 - xoff<V>(), y0 - 1, k, bar);
}
__device__ __forceinline__ void tma_own(void *dst, const CUtensorMap *map, int x0, int y0, int k, uint64_t *bar) {
    tma_load_3d(dst, map, x0, y0, k, bar);
}
__device__ __forceinline__ void tma_own4(void *dst, const CUtensorMap *map, int x0, int y0, int k, uint64_t *bar) {
    tma_load_4d(dst, map, x0, y0, k, bar);
}

// Two neighbouring columns' values.  FP32 pairs use sm_100's packed FP32
// instructions (two IEEE operations each), FP64 pairs two FP64 ones.
template <typename T>
struct Pair;
template <>
struct Pair<float> {
    using type = float2;
};
template <>
struct Pair<double> {
    using type = double2;
};
template <typename T>
using P2 = typename Pair<T>::type;
template <typename T>
__device__ __forceinline__ P2<T> mk2(T x, T y) {
    P2<T> r;
    r.x = x;
    r.y = y;
    return r;
}
template <typename T>
__device__ __forceinline__ P2<T> mk2(T x) { return mk2<T>(x, x); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
// a - b as one packed operation (b times -1 is exact)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ double2 fma2(double2 a, double2 b, double2 c) {
    return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
__device__ __forceinline__ double2 add2(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 mul2(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ double2 sub2(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// sum + a / b
__device__ __forceinline__ float2 add_quot2(float2 sum, float2 a, float2 b) {
    return add2(sum, make_float2(quot(a.x, b.x), quot(a.y, b.y)));
}
__device__ __forceinline__ double2 add_quot2(double2 sum, double2 a, double2 b) {
    return make_double2(add_quot(sum.x, a.x, b.x), add_quot(sum.y, a.y, b.y));
}
template <typename T, typename F>
__device__ __forceinline__ P2<T> get2(const F *p) {
    const P2<F> v = *reinterpret_cast<const P2<F> *>(p);
    return mk2<T>((T)v.x, (T)v.y);
}
template <typename T>
__device__ __forceinline__ void put2(T *p, P2<T> v) {
    *reinterpret_cast<P2<T> *>(p) = v;
}

// A ring stage of the inner sweep: a unit of UNIT planes of a tile -- z, t, p of
// the previous iteration (one box), K (halo), then the own planes of D, 1/den,
// c', d (FP32) or D, d and 1/den, c' in FP32 (FP64 mode); of each array the
// planes one behind the other.  Both tile shapes fit the same slots.
enum { UNIT = STAGE_PLANES };
template <typename T>
struct Stage {
    using F = typename Fac<T>::type;
    static constexpr bool same = sizeof(F) == sizeof(T);
    static constexpr unsigned up(unsigned b) { return (b + 127u) & ~127u; }
    static constexpr unsigned h32 = halo_bytes<T>(32, 4), h16 = halo_bytes<T>(16, 8), h = UNIT * (h32 > h16 ? h32 : h16);
    static constexpr unsigned ob = UNIT * TILE_THREADS * sizeof(T), of = UNIT * TILE_THREADS * sizeof(F);
    static constexpr unsigned K = up(3 * h), own = K + up(h);
    static constexpr unsigned D = own, inv = same ? own + ob : own + 2 * ob, c = inv + of,
                              d = same ? own + 3 * ob : own + ob;
    static constexpr unsigned bytes = own + 2 * ob + 2 * of;
};
// A ring stage of phase R: a unit in FP64 -- x, K64 (halo), D64, b (own) -- and
// the stored factors (own).
template <typename T>
struct StageR {
    using F = typename Fac<T>::type;
    static constexpr unsigned h32 = halo_bytes<double>(32, 4), h16 = halo_bytes<double>(16, 8),
                              hs = (UNIT * (h32 > h16 ? h32 : h16) + 127u) & ~127u, ob = UNIT * TILE_THREADS * 8,
                              of = UNIT * TILE_THREADS * sizeof(F);
    static constexpr unsigned x = 0, K = hs, D = 2 * hs, b = D + ob, inv = b + ob, c = inv + of, bytes = c + of;
};
// A column buffer: of every cell of a tile's columns, plane by plane, the right-
// hand side of the column solve in T and then the factors c' and 1/den (two arrays
// of F), or in a solve's first phase R the matrix they are formed from: in FP32 the
// vertical coupling and the diagonal, in FP64 the diagonal (the coupling is then
// left in the d array, which is free there).
template <typename T>
__host__ __device__ constexpr int col_bytes(int nz) {
    constexpr int factors = 2 * (int)sizeof(typename Fac<T>::type), matrix = (sizeof(T) == 4 ? 2 : 1) * (int)sizeof(T);
    return TILE_THREADS * ((int)sizeof(T) + (factors > matrix ? factors : matrix)) * nz;
}

// What the roles need to know of a tile.  A block's first TILE_TABLE tiles are
// kept in shared memory for the whole solve: each sweep starts with a grid
// barrier, after which the descriptors' lines are no longer in L1.
struct TileCtx {
    int dom, x0, y0, nx, ny, nz, nxp, tx;
    int begin, end;        // the domain's tiles
    unsigned off, sxy;     // the domain's first cell, cells of a plane
    double ix2, iy2, iz2;  // 1 / dx^2, ...
};
enum { TILE_TABLE = 64 };
__device__ __forceinline__ TileCtx tile_ctx(const DevPtrs &P, int t) {
    const TileDesc td = P.tiles[t];
    const DomainDesc &D = P.dom[td.dom];
    return TileCtx{td.dom, td.x0, td.y0, D.nx, D.ny, D.nz, D.nxp, D.tx, D.tile_begin, D.tile_end, (unsigned)D.off3,
                   (unsigned)D.nxp * (unsigned)D.ny, 1.0 / (D.dx * D.dx), 1.0 / (D.dy * D.dy), 1.0 / (D.dz * D.dz)};
}

// A plane warp's place in a unit (UNIT_WARPS share one): its plane e and its
// lane's pair of columns of the UNIT_WARPS / UNIT x 32 in a plane.
enum { UNIT_WARPS = 4 };
__device__ __forceinline__ int unit_sub() { return ((int)threadIdx.x / 32) % UNIT_WARPS; }
__device__ __forceinline__ int unit_plane() { return unit_sub() / 2; }

// That pair in a tile, and its face weights: the stencil weight times the 1/2 of
// the face average, zero on a domain face, so that a face coefficient is one
// add and one multiply, f = h (K_c + K_nb).  we: the outer faces of the pair (w
// of the first column, e of the second); in: the face between them.  Past an odd
// nx the second column is padding: everything staged there is zero, its inner
// face too, and so is all that is written there (to the arrays' padding).
template <typename T>
struct PairRef {
    int own, halo;   // place in an own plane and in a halo plane
    unsigned g;      // cell (i, j, e)
    P2<T> we, s, n;
    T in;
    bool valid;
};
template <typename T, int TX>
__device__ __forceinline__ PairRef<T> pair_of(const TileCtx &td, T hx, T hy) {
    constexpr int PAIRS = TX / 2, XO = xoff<T>();
    PairRef<T> r;
    const int pair = (unit_sub() & 1) * 32 + ((int)threadIdx.x & 31);
    const int px = pair & (PAIRS - 1), row = pair / PAIRS;
    const int i = td.x0 + 2 * px, j = td.y0 + row;
    r.own = row * TX + 2 * px;
    r.halo = (row + 1) * (TX + 2 * XO) + XO + 2 * px;
    r.g = td.off + (unsigned)j * (unsigned)td.nxp + (unsigned)i + (unsigned)unit_plane() * td.sxy;
    r.valid = i < td.nx && j < td.ny;
    r.we = mk2<T>(i > 0 ? hx : T(0), i + 2 < td.nx ? hx : T(0));
    r.in = i + 1 < td.nx ? hx : T(0);
    r.s = mk2<T>(j > 0 ? hy : T(0));
    r.n = mk2<T>(j < td.ny - 1 ? hy : T(0));
    return r;
}

// Step scalars of a domain in one sweep: of the inner solve, or of phase R, where
// active means the outer solve runs and first a solve's first cycle, which
// factors M.
struct SweepCtl {
    int dom, active, parity;
    bool first, keep_p;
    double alpha, beta;
};
template <bool RESIDUAL, typename Get>
__device__ __forceinline__ void load_ctl(SweepCtl &c, int dom, const KrylovCtrl *k, Get get) {
    if (c.dom == dom) return;
    c.dom = dom;
    c.active = get(RESIDUAL ? &k->active : &k->inner_active);
    c.parity = get(&k->parity);
    c.first = RESIDUAL ? get(&k->cycles) == 0 : get(&k->first_inner) != 0;
    c.keep_p = get(&k->keep_p) != 0;
    c.alpha = get(&k->alpha);
    c.beta = get(&k->beta);
}

// A solver block is a pipeline of four roles over the tiles it owns:
//   two producer warps stage units of planes into the ring (TMA),
//   the observer warp waits for them in order and counts those that have landed
//     (an mbarrier wait can tell a phase only from the one before it, and a plane
//     warp does not see every unit),
//   the PLANE_WARPS plane warps take the units as they land -- the stencil has no
//     order in k -- and leave what the column solve needs (q and the factors) in
//     a column buffer in shared memory,
//   the column warps (one thread per column) run the two recurrences down and
//     up the column from that buffer and write the result,
// so that with two column buffers a tile's recurrences run while the next
// tile's planes are computed and those after it are in flight.
enum { COL_THREADS = TILE_THREADS, PLANE_WARPS = 8 };
static_assert(SOLVE_THREADS == COL_THREADS + 32 * PLANE_WARPS + 96, "column, plane, producer and observer warps");
__host__ __device__ constexpr int units_of(int nz) { return (nz + UNIT - 1) / UNIT; }

struct PipeBars {
    uint64_t full[RING_MAX], empty[RING_MAX];  // ring stages: landed; done with by the unit and its two neighbours
    uint64_t cfull[2], cempty[2];              // column buffers: written by all plane warps; solved by the column warps
    uint64_t red[2];                           // plane warps' sums of a domain are in PipeShared::sums
};
struct PipeShared {
    PipeBars c, r;                             // of the inner sweeps and of phase R
    double sums[2][PLANE_WARPS][3];
    double csum[2][COL_THREADS / 32];
    unsigned landed_c, landed_r;               // units that have landed in each ring, counted by the observer
    unsigned issued[2];                        // stages each producer warp has issued (for an error exit)
    TileCtx tiles[TILE_TABLE];
    KrylovCtrl ctl;                            // of a handle's only domain
};

// One role's place in a pipeline.
struct Pipe {
    PipeBars *b;
    unsigned char *col, *ring;  // column buffers, stages
    int n, stage, nb, colb;     // stages and bytes of one; column buffers and bytes of one
    unsigned *landed;           // PipeShared::landed_c or _r
    int slot;                   // stage of the tile's first unit, and the parity its "full" completes with
    unsigned par;
    int buf;                    // column buffer of the tile and the parity its "cfull" completes with
    unsigned cpar;
    unsigned unit;              // units before the tile, over the whole launch
    unsigned flushes;           // domains finished

    __device__ __forceinline__ void step(int &s, unsigned &p, int m) const {
        s += m;
        while (s >= n) {
            s -= n;
            p ^= 1u;
        }
    }
    __device__ __forceinline__ unsigned char *at(int s) const { return ring + s * stage; }
    __device__ __forceinline__ unsigned char *cbuf() const { return col + buf * colb; }
    __device__ __forceinline__ void next_tile(int nz) {
        step(slot, par, units_of(nz));
        unit += (unsigned)units_of(nz);
        if (++buf == nb) {
            buf = 0;
            cpar ^= 1u;
        }
    }
    // producer, on an error exit: waits, DRAIN_TIMEOUT_NS at most, for the last
    // copies of every stage issued, so no TMA write into the block's shared
    // memory is in flight when the block exits
    __device__ __forceinline__ void drain(unsigned issued) const {
        const unsigned long long t0 = global_ns();
        int q = slot;
        unsigned p = par;
        for (unsigned left = issued < (unsigned)n ? issued : (unsigned)n; left > 0; --left) {
            if (--q < 0) {
                q = n - 1;
                p ^= 1u;
            }
            while (!mbar_try_wait(b->full + q, p) && global_ns() - t0 < DRAIN_TIMEOUT_NS) {
            }
        }
    }
};

struct SolveBlock {
    Pipe c, r;
    PipeShared *sh;
    unsigned int target;  // of the solve's grid barrier
    unsigned int phase;   // grid barriers passed: even and odd phases keep their partials apart
};
enum Role { ROLE_COLUMN, ROLE_PLANE, ROLE_PRODUCER, ROLE_OBSERVER };
__device__ __forceinline__ int role_of() {
    return threadIdx.x < COL_THREADS         ? ROLE_COLUMN
           : threadIdx.x < SOLVE_THREADS - 96 ? ROLE_PLANE
           : threadIdx.x < SOLVE_THREADS - 32 ? ROLE_PRODUCER
                                              : ROLE_OBSERVER;
}

// ---- the producer ----------------------------------------------------------
// Stages one tile's units: each of the two producer warps issues a part of the
// copies (`half` 0 or 1), since the issue of a few copies takes one warp longer
// than the unit's bytes take to arrive.  On a wait that gave up nothing more is
// issued.
template <typename Issue>
__device__ __forceinline__ void produce(const DevPtrs &P, Pipe &pp, unsigned *issued, int nz, unsigned bytes,
                                        Issue issue) {
    unsigned done = 0;
    for (int k = 0; k < nz; k += UNIT, ++done) {
        if (!mbar_sleep(pp.b->empty + pp.slot, pp.par ^ 1u, P.barrier)) break;
        uint64_t *bar = pp.b->full + pp.slot;
        mbar_expect_tx(bar, bytes);
        issue(pp.at(pp.slot), k, bar);
        pp.step(pp.slot, pp.par, 1);
    }
    *issued += done;
}

template <typename T>
__device__ __forceinline__ void produce_R(const DevPtrs &P, const TileCtx &td, const SweepCtl &c, int half, Pipe &pp,
                                          unsigned *issued) {
    using S = StageR<T>;
    const CUtensorMap *m = P.tmaps + (size_t)td.dom * NMAP;
    const int x0 = td.x0, y0 = td.y0;
    if (half == 0) {
        produce(P, pp, issued, td.nz, 2 * UNIT * halo_bytes<double>(td.tx, TILE_THREADS / td.tx),
                [&](unsigned char *B, int k, uint64_t *bar) {
                    tma_halo<double>(B + S::x, m + PMAP_X64_H, x0, y0, k, bar);
                    tma_halo<double>(B + S::K, m + PMAP_K64_H, x0, y0, k, bar);
                });
    } else {
        produce(P, pp, issued, td.nz, 2 * S::ob + (c.first ? 0 : 2 * S::of), [&](unsigned char *B, int k, uint64_t *bar) {
            tma_own(B + S::D, m + PMAP_D64_O, x0, y0, k, bar);
            tma_own(B + S::b, m + PMAP_B_O, x0, y0, k, bar);
            if (!c.first) tma_own4(B + S::inv, m + PMAP_FAC_O, x0, y0, k, bar);
        });
    }
}

// The first sweep of a cycle has no previous t or d (alpha = 0, d starts at
// zero), and no p either unless it continues the previous cycle's direction.
template <typename T>
__device__ __forceinline__ void produce_C(const DevPtrs &P, const TileCtx &td, const SweepCtl &c, int half, Pipe &pp,
                                          unsigned *issued) {
    using S = Stage<T>;
    const CUtensorMap *m = P.tmaps + (size_t)td.dom * NMAP;
    const unsigned hb = UNIT * halo_bytes<T>(td.tx, TILE_THREADS / td.tx);
    const int x0 = td.x0, y0 = td.y0;
    if (half == 0) {
        if (!c.first) {
            const CUtensorMap *mv = m + (c.parity ? PMAP_ZTP1_H : PMAP_ZTP0_H);
            produce(P, pp, issued, td.nz, 3 * hb,
                    [&](unsigned char *B, int k, uint64_t *bar) { tma_halo4<T>(B, mv, x0, y0, k, bar); });
        } else {
            const CUtensorMap *mz = m + (c.parity ? PMAP_Z1_H : PMAP_Z0_H), *mp = m + (c.parity ? PMAP_P1_H : PMAP_P0_H);
            const bool with_p = c.keep_p;
            produce(P, pp, issued, td.nz, (with_p ? 2 : 1) * hb, [&](unsigned char *B, int k, uint64_t *bar) {
                tma_halo<T>(B, mz, x0, y0, k, bar);
                if (with_p) tma_halo<T>(B + 2 * hb, mp, x0, y0, k, bar);
            });
        }
    } else {
        const bool all = !c.first && S::same, d_too = !c.first;
        produce(P, pp, issued, td.nz, hb + (d_too ? 2 : 1) * S::ob + 2 * S::of,
                [&](unsigned char *B, int k, uint64_t *bar) {
                    tma_halo<T>(B + S::K, m + PMAP_K_H, x0, y0, k, bar);
                    if (d_too) tma_own4(B + S::own, m + PMAP_OWN_O, x0, y0, k, bar);
                    else tma_own(B + S::D, m + PMAP_D_O, x0, y0, k, bar);
                    if (!all) tma_own4(B + S::inv, m + PMAP_FAC_O, x0, y0, k, bar);
                });
    }
}

// The L2 prefetch of a unit of the inner sweep: the DRAM reads of planes that the
// ring has no room for yet.
#ifndef PF_UNITS
#define PF_UNITS 4
#endif
template <typename T>
__device__ __forceinline__ void prefetch_C(const DevPtrs &P, const TileCtx &td, const SweepCtl &c, int k, int x0, int y0) {
    const CUtensorMap *m = P.tmaps + (size_t)td.dom * NMAP;
    if (!c.first) {
        tma_prefetch_4d(m + (c.parity ? PMAP_ZTP1_H : PMAP_ZTP0_H), x0 - xoff<T>(), y0 - 1, k);
        tma_prefetch_4d(m + PMAP_OWN_O, x0, y0, k);
        if (!Stage<T>::same) tma_prefetch_4d(m + PMAP_FAC_O, x0, y0, k);
    } else {
        tma_prefetch_3d(m + (c.parity ? PMAP_Z1_H : PMAP_Z0_H), x0 - xoff<T>(), y0 - 1, k);
        if (c.keep_p) tma_prefetch_3d(m + (c.parity ? PMAP_P1_H : PMAP_P0_H), x0 - xoff<T>(), y0 - 1, k);
        tma_prefetch_3d(m + PMAP_D_O, x0, y0, k);
        tma_prefetch_4d(m + PMAP_FAC_O, x0, y0, k);
    }
    tma_prefetch_3d(m + PMAP_K_H, x0 - xoff<T>(), y0 - 1, k);
}

// ---- the plane warps -------------------------------------------------------
// Waits until `units` units have landed (PipeShared::landed, in stage order).
__device__ __forceinline__ void wait_landed(const DevPtrs &P, const unsigned *landed, unsigned units) {
    auto enough = [&]() {
        unsigned v;
        asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(smem_addr(landed)) : "memory");
        return (int)(v - units) >= 0;
    };
    if (enough()) return;
    const unsigned long long t0 = global_ns();
    for (unsigned spins = 1;; ++spins) {
        if (enough() || ((spins & 63u) == 0 && *(volatile int *)&P.barrier->error)) return;
        if ((spins & 1023u) == 0 && global_ns() - t0 > MBAR_TIMEOUT_NS) {
            atomicExch(&P.barrier->error, 1);
            return;
        }
    }
}

// Walks this warp's units of a tile: fn(plane, own stage, and the halo planes --
// `hb` bytes each, of the first array of a stage -- above it, its own and below
// it) once they have landed (its own in the place of a plane that does not
// exist).  Four plane warps share a unit, each with half a plane and each lane
// with one pair of columns, so that few stages are held by planes being computed
// and most of the ring is in flight; the two groups of four take alternate
// units.  `turn` counts the block's tiles of the domain: with an odd number of
// units it alternates which group begins, and it depends on nothing else the
// block works on, so a domain's sums do not either.
enum { PLANE_GROUPS = PLANE_WARPS / UNIT_WARPS };
static_assert(UNIT == 2, "a unit's two planes are its warps' upper and lower halves");
template <typename Fn>
__device__ __forceinline__ void planes(const DevPtrs &P, Pipe &pp, int nz, int turn, int hb, Fn fn) {
    const int units = units_of(nz), e = unit_plane();
    const int first = (((int)threadIdx.x - COL_THREADS) / (32 * UNIT_WARPS) + turn * units) % PLANE_GROUPS;
    const bool lane0 = (threadIdx.x & 31) == 0;
    // the tile's column buffer is free once its last user's columns are solved
    mbar_sleep(pp.b->cempty + pp.buf, pp.cpar ^ 1u, P.barrier);
    int s = pp.slot;
    unsigned par = 0;  // not used here
    pp.step(s, par, first);
    for (int q = first; q < units; q += PLANE_GROUPS) {
        const int k = q * UNIT + e;
        // the upper half reads the unit above too, the lower half the one below
        int other = s;
        if (e == 0) {
            if (q > 0) other = s == 0 ? pp.n - 1 : s - 1;
        } else if (q + 1 < units) {
            other = s + 1 == pp.n ? 0 : s + 1;
        }
        wait_landed(P, pp.landed, pp.unit + (unsigned)(q + (e == 1 && q + 1 < units ? 2 : 1)));
        if (k < nz) {
            const unsigned char *B = pp.at(s), *O = pp.at(other), *C = B + e * hb;
            const unsigned char *U = e == 0 ? O + hb : B, *N = e == 0 ? B + hb : O;
            fn(k, B, k == 0 ? C : U, C, k + 1 == nz ? C : N);
        }
        __syncwarp();
        // a stage is free once its own unit's warps, the lower half of the unit
        // above and the upper half of the unit below are done with it; the
        // arrivals of units that do not exist are made here
        if (lane0) {
            mbar_arrive(pp.b->empty + s);
            mbar_arrive(pp.b->empty + other);
        }
        s += PLANE_GROUPS;
        if (s >= pp.n) s -= pp.n;
    }
    __syncwarp();
    if (lane0) mbar_arrive(pp.b->cfull + pp.buf);  // the warp's writes are done
    pp.next_tile(nz);
}

// Leaves the warp's three sums of a domain for the column warps.
__device__ __forceinline__ void plane_sums(Pipe &pp, PipeShared *sh, double (&v)[3]) {
    const int w = ((int)threadIdx.x - COL_THREADS) >> 5, f = pp.flushes & 1;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
    }
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int i = 0; i < 3; ++i) sh->sums[f][w][i] = v[i];
        mbar_arrive(pp.b->red + f);
    }
    pp.flushes += 1;
}

// Phase R, a tile's planes: r = b - A x with the FP64 coefficients; to the
// column buffer r_T = (T) r and, in a solve's first cycle, the column block of
// M from the inner operator's T coefficients (the same rounding as the stored
// K, D): the diagonal without its vertical couplings (-1 on a fixed cell) and
// the coupling to the plane below; in later cycles the stored factors.
template <typename T, int TX>
__device__ __forceinline__ void planes_R(const DevPtrs &P, const TileCtx &td, const SweepCtl &c, int turn, Pipe &pp,
                                         double (&v)[3]) {
    using S = StageR<T>;
    using F = typename Fac<T>::type;
    using D2 = double2;
    constexpr int BW = TX + 2 * xoff<double>(), HALO = BW * (TILE_THREADS / TX + 2);
    const T hx = T(0.5) * (T)td.ix2, hy = T(0.5) * (T)td.iy2, hz = T(0.5) * (T)td.iz2;
    const double cx = (double)(T)td.ix2, cy = (double)(T)td.iy2, cz = (double)(T)td.iz2;
    const int nz = td.nz, own = unit_plane() * TILE_THREADS;
    T *const cq = (T *)pp.cbuf();
    // face masks: 1/2 of the face average, zero on a domain face
    const PairRef<double> r = pair_of<double, TX>(td, 0.5, 0.5);
    planes(P, pp, nz, turn, HALO * 8, [&](int k, const unsigned char *B, const unsigned char *U, const unsigned char *C,
                                          const unsigned char *N) {
        if (!r.valid) return;
        const double *sx = (const double *)(C + S::x) + r.halo, *sK = (const double *)(C + S::K) + r.halo;
        const D2 xc = get2<double>(sx), Kc = get2<double>(sK);
        const D2 xu = get2<double>((const double *)(U + S::x) + r.halo), Ku = get2<double>((const double *)(U + S::K) + r.halo);
        const D2 xd = get2<double>((const double *)(N + S::x) + r.halo), Kd = get2<double>((const double *)(N + S::K) + r.halo);
        const double md = k + 1 < nz ? 0.5 : 0.0, mu = k > 0 ? 0.5 : 0.0;
        const D2 xs = get2<double>(sx - BW), Ks = get2<double>(sK - BW);
        const D2 xn = get2<double>(sx + BW), Kn = get2<double>(sK + BW);
        const D2 xo = mk2<double>(sx[-1], sx[2]), Ko = mk2<double>(sK[-1], sK[2]);
        const D2 Dk = get2<double>((const double *)(B + S::D) + own + r.own),
                 bk = get2<double>((const double *)(B + S::b) + own + r.own);
        const D2 kwe = mul2(r.we, add2(Kc, Ko));
        const double kin = r.in * (Kc.x + Kc.y);
        const D2 ks = mul2(r.s, add2(Kc, Ks)), kn = mul2(r.n, add2(Kc, Kn));
        const D2 ku = mul2(mk2<double>(mu), add2(Kc, Ku)), kd = mul2(mk2<double>(md), add2(Kc, Kd));
        const double din = xc.x - xc.y;
        const D2 qx = fma2(mk2<double>(kin), mk2<double>(din, -din), mul2(kwe, sub2(xc, xo)));
        const D2 qy = fma2(kn, sub2(xc, xn), mul2(ks, sub2(xc, xs)));
        const D2 qz = fma2(kd, sub2(xc, xd), mul2(ku, sub2(xc, xu)));
        const D2 Ax = fma2(mk2<double>(cz), qz, fma2(mk2<double>(cy), qy, fma2(mk2<double>(cx), qx, mul2(Dk, xc))));
        // D < 0 marks a Dirichlet (fixed) cell: identity row, x already holds its
        // value, so its residual is zero and the preconditioner leaves it alone
        D2 rk = sub2(bk, Ax);
        if (Dk.x < 0.0) rk.x = 0.0;
        if (Dk.y < 0.0) rk.y = 0.0;
        v[0] += rk.x * rk.x;
        v[0] += rk.y * rk.y;
        v[1] += bk.x * bk.x;
        v[1] += bk.y * bk.y;
        const int o = k * TILE_THREADS + r.own;
        put2<T>(cq + o, mk2<T>((T)rk.x, (T)rk.y));
        if (c.first) {
            const P2<T> Kt = mk2<T>((T)Kc.x, (T)Kc.y);
            const P2<T> fwe = mul2(mk2<T>(r.we.x != 0.0 ? hx : T(0), r.we.y != 0.0 ? hx : T(0)),
                                   add2(Kt, mk2<T>((T)Ko.x, (T)Ko.y)));
            const T fin = (r.in != 0.0 ? hx : T(0)) * (Kt.x + Kt.y);
            const P2<T> fs = mul2(mk2<T>(r.s.x != 0.0 ? hy : T(0)), add2(Kt, mk2<T>((T)Ks.x, (T)Ks.y)));
            const P2<T> fn = mul2(mk2<T>(r.n.x != 0.0 ? hy : T(0)), add2(Kt, mk2<T>((T)Kn.x, (T)Kn.y)));
            const P2<T> fu = mul2(mk2<T>(k + 1 < nz ? hz : T(0)), add2(Kt, mk2<T>((T)Kd.x, (T)Kd.y)));
            P2<T> bl = add2(add2(mk2<T>((T)Dk.x, (T)Dk.y), add2(fwe, mk2<T>(fin))), add2(fs, fn));
            if (Dk.x < 0.0) bl.x = T(-1);
            if (Dk.y < 0.0) bl.y = T(-1);
            T *const m = cq + nz * TILE_THREADS;
            put2<T>(m + o, bl);
            if constexpr (sizeof(T) == 4) put2<T>(m + nz * TILE_THREADS + o, fu);
            else put2<T>((T *)P.d + r.g + (unsigned)(k - unit_plane()) * td.sxy, fu);
        } else {
            F *const m = (F *)(cq + nz * TILE_THREADS);
            put2<F>(m + o, get2<F>((const F *)(B + S::c) + own + r.own));
            put2<F>(m + nz * TILE_THREADS + o, get2<F>((const F *)(B + S::inv) + own + r.own));
        }
    });
}

// ---- inner sweep C: one PCG iteration --------------------------------------
// With ap = alpha_{i-1} and bt = beta_i (ap zero in a cycle's first sweep, bt
// too unless the sweep continues the previous cycle's direction):
// z = z_prev - ap t_prev and p = z + bt p_prev at a pair of columns and its
// lateral and vertical neighbours (from the staged halo boxes), q = A p,
// d += ap p_prev.  Writes z, p into the buffers other than `prev`, q and the
// factors into the column buffer, and adds p.q, z.q and z.M z to v (the column
// warps add q.t and write t = M^-1 q).  The three forms of a sweep (a cycle's
// first without or with the previous direction, and the general one) are
// compiled separately: MODE 0 p = z, 1 p = z + bt p_prev, 2 z and p from t and
// p_prev.
template <typename T, int TX, int MODE>
__device__ __forceinline__ void planes_C(const DevPtrs &P, const TileCtx &td, const SweepCtl &c, int turn, Pipe &pp,
                                         P2<T> (&a)[3]) {
    using S = Stage<T>;
    using F = typename Fac<T>::type;
    using V = P2<T>;
    // BW: a row of a halo plane; HALO: the plane; SET: from one array of a box to the next
    constexpr int BW = TX + 2 * xoff<T>(), HALO = BW * (TILE_THREADS / TX + 2), SET = UNIT * HALO;
    constexpr int KT = S::K / sizeof(T);  // from z to K
    const T hz = T(0.5) * (T)td.iz2;
    const int nz = td.nz;
    const PairRef<T> r = pair_of<T, TX>(td, T(0.5) * (T)td.ix2, T(0.5) * (T)td.iy2);
    const int own = unit_plane() * TILE_THREADS + r.own;
    T *__restrict__ z_out = (T *)(c.parity ? P.z0 : P.z1);
    T *__restrict__ p_out = (T *)(c.parity ? P.p0 : P.p1);
    T *__restrict__ d_out = (T *)P.d;
    const V nap = mk2<T>(-(T)c.alpha), ap = mk2<T>((T)c.alpha), bt = mk2<T>((T)c.beta);
    T *const cq = (T *)pp.cbuf();
    F *const cc = (F *)(cq + nz * TILE_THREADS), *const ci = cc + nz * TILE_THREADS;
    // z and p from the staged previous z, t, p
    auto zv = [&](V z, V t) {
        if constexpr (MODE == 2) return fma2(nap, t, z);
        else return z;
    };
    auto pz = [&](V z, V p) {
        if constexpr (MODE == 0) return z;
        else return fma2(bt, p, z);
    };
    auto z_at = [&](const T *s) {
        const V z = get2<T>(s);
        if constexpr (MODE == 2) return zv(z, get2<T>(s + SET));
        else return z;
    };
    auto p_prev_at = [&](const T *s) {
        if constexpr (MODE > 0) return get2<T>(s + 2 * SET);
        else return V{};
    };
    auto p_at = [&](const T *s) { return pz(z_at(s), p_prev_at(s)); };
    // the columns left of the first and right of the second
    auto outer = [&](const T *s) { return mk2<T>(s[-1], s[2]); };
    planes(P, pp, nz, turn, HALO * (int)sizeof(T), [&](int k, const unsigned char *B, const unsigned char *U,
                                                       const unsigned char *C, const unsigned char *N) {
        if (!r.valid) return;
        const T *sc = (const T *)C + r.halo, *su = (const T *)U + r.halo, *sn = (const T *)N + r.halo;
        const V pu = p_at(su), Ku = get2<T>(su + KT);
        const V zc = z_at(sc), qc = p_prev_at(sc), pc = pz(zc, qc), Kc = get2<T>(sc + KT);
        const V zd = z_at(sn), pd = pz(zd, p_prev_at(sn)), Kd = get2<T>(sn + KT);
        V zo = outer(sc);
        if constexpr (MODE == 2) zo = zv(zo, outer(sc + SET));
        V po = zo;
        if constexpr (MODE > 0) po = pz(zo, outer(sc + 2 * SET));
        const V ps = p_at(sc - BW), pn = p_at(sc + BW);
        const V fwe = mul2(r.we, add2(Kc, outer(sc + KT)));
        const T fin = r.in * (Kc.x + Kc.y);
        const V fs = mul2(r.s, add2(Kc, get2<T>(sc + KT - BW)));
        const V fn = mul2(r.n, add2(Kc, get2<T>(sc + KT + BW)));
        const V fu = mul2(mk2<T>(k > 0 ? hz : T(0)), add2(Kc, Ku));
        const V fd = mul2(mk2<T>(k + 1 < nz ? hz : T(0)), add2(Kc, Kd));
        const T din = pc.x - pc.y;
        const V qx = fma2(mk2<T>(fin), mk2<T>(din, -din), mul2(fwe, sub2(pc, po)));
        const V qy = fma2(fn, sub2(pc, pn), mul2(fs, sub2(pc, ps)));
        const V qz = fma2(fd, sub2(pc, pd), mul2(fu, sub2(pc, pu)));
        // A Dirichlet cell (D < 0, identity row) has z = p = 0 and 1/den = c' = 0:
        // whatever q is there, it enters no sum and not the column solve
        const V q = add2(add2(fma2(get2<T>((const T *)(B + S::D) + own), pc, qx), qy), qz);
        // z.M z with M = L D L^T from the stored factors: the sum of
        // (z_k + c'_k z_{k+1})^2 / inv_k; where inv = 0 (a fixed cell, padding)
        // the numerator is 0; c' of the last plane is 0
        const P2<F> inv_s = get2<F>((const F *)(B + S::inv) + own), cp_s = get2<F>((const F *)(B + S::c) + own);
        const V inv = mk2<T>((T)inv_s.x, (T)inv_s.y), cp = mk2<T>((T)cp_s.x, (T)cp_s.y);
        V u = fma2(cp, zd, zc);
        u = mul2(u, u);
        constexpr T tiny = sizeof(T) == 4 ? T(1e-37) : T(1e-300);
        a[0] = fma2(pc, q, a[0]);
        a[1] = fma2(zc, q, a[1]);
        a[2] = add_quot2(a[2], u, mk2<T>(inv.x > tiny ? inv.x : tiny, inv.y > tiny ? inv.y : tiny));
        const unsigned g = r.g + (unsigned)(k - unit_plane()) * td.sxy;
        put2<T>(z_out + g, zc);
        put2<T>(p_out + g, pc);
        if constexpr (MODE == 2) put2<T>(d_out + g, fma2(ap, qc, get2<T>((const T *)(B + S::d) + own)));
        else put2<T>(d_out + g, V{});
        const int o = k * TILE_THREADS + r.own;
        put2<T>(cq + o, q);
        put2<F>(cc + o, cp_s);
        put2<F>(ci + o, inv_s);
    });
}

// ---- the column warps ------------------------------------------------------
// One thread per column: out = M^-1 q from the column buffer, returns
// q.M^-1 q.  FACTOR: the buffer holds the matrix instead of the factors, which
// are formed, used and stored.  The loads of COL_BATCH planes are issued
// together, ahead of the recurrence.
#ifndef COL_BATCH
#define COL_BATCH 8
#endif
template <typename T, bool FACTOR>
__device__ __forceinline__ T solve_column(const DevPtrs &P, unsigned char *buf, int nz, unsigned g0, unsigned sxy,
                                          T *__restrict__ out) {
    using F = typename Fac<T>::type;
    T *const q = (T *)buf + threadIdx.x;
    T *const m = q + nz * TILE_THREADS;  // FACTOR: the diagonal
    F *const cc = (F *)((T *)buf + nz * TILE_THREADS) + threadIdx.x, *const iv = cc + nz * TILE_THREADS;
    T cprev = T(0), yprev = T(0), fd = T(0), sum = T(0);
    for (int k0 = 0; k0 < nz; k0 += COL_BATCH) {
        T qk[COL_BATCH], ck[COL_BATCH], ik[COL_BATCH];
#pragma unroll
        for (int e = 0; e < COL_BATCH; ++e) {
            // past the end: the last plane again, not used
            const int k = k0 + e < nz ? k0 + e : nz - 1, o = k * TILE_THREADS;
            qk[e] = q[o];
            if constexpr (!FACTOR) {
                ck[e] = (T)cc[o];
                ik[e] = (T)iv[o];
            } else {
                ik[e] = m[o];
                if constexpr (sizeof(T) == 4) ck[e] = m[nz * TILE_THREADS + o];
                else ck[e] = ldcg((const T *)P.d + g0 + (unsigned)k * sxy);
            }
        }
#pragma unroll
        for (int e = 0; e < COL_BATCH; ++e) {
            const int k = k0 + e;
            if (k >= nz) break;
            T cp = ck[e], inv = ik[e];
            if constexpr (FACTOR) {
                // ck: the coupling fu to the next plane; ik: the diagonal without
                // the vertical couplings, negative on a fixed cell
                const T fu = ck[e];
                const T den = ((ik[e] + fd) + fu) + fd * cprev;  // b_k - a_k c'_{k-1}, a_k = -fd
                // the stored (rounded) factors are the ones applied, here as in the sweeps
                const F inv_s = (F)(ik[e] < T(0) ? T(0) : recip(den));
                inv = (T)inv_s;
                const F cp_s = (F)(-fu * inv);
                cp = (T)cp_s;
                ((F *)P.finv)[g0 + (unsigned)k * sxy] = inv_s;
                ((F *)P.fc)[g0 + (unsigned)k * sxy] = cp_s;
                m[k * TILE_THREADS] = cp;
                fd = fu;
            }
            const T y = qk[e] - cprev * yprev;
            const T dp = y * inv;
            sum += y * dp;
            q[k * TILE_THREADS] = dp;
            cprev = cp;
            yprev = y;
        }
    }
    T zn = T(0);
    for (int k0 = nz - 1; k0 >= 0; k0 -= COL_BATCH) {
        T dk[COL_BATCH], ck[COL_BATCH];
#pragma unroll
        for (int e = 0; e < COL_BATCH; ++e) {
            const int o = (k0 - e >= 0 ? k0 - e : 0) * TILE_THREADS;
            dk[e] = q[o];
            if constexpr (FACTOR) ck[e] = m[o];  // c' over the diagonal
            else ck[e] = (T)cc[o];
        }
#pragma unroll
        for (int e = 0; e < COL_BATCH; ++e) {
            const int k = k0 - e;
            if (k < 0) break;
            zn = dk[e] - ck[e] * zn;
            out[g0 + (unsigned)k * sxy] = zn;
        }
    }
    return sum;
}

// One tile's columns; returns the thread's q.M^-1 q.
template <typename T, bool FACTOR>
__device__ __forceinline__ double columns(const DevPtrs &P, const TileCtx &td, Pipe &pp, T *out) {
    const int i = td.x0 + ((int)threadIdx.x & (td.tx - 1)), j = td.y0 + (int)threadIdx.x / td.tx;
    mbar_sleep(pp.b->cfull + pp.buf, pp.cpar, P.barrier);
    T s = T(0);
    if (i < td.nx && j < td.ny)
        s = solve_column<T, FACTOR>(P, pp.cbuf(), td.nz, td.off + (unsigned)j * (unsigned)td.nxp + (unsigned)i, td.sxy, out);
    return (double)s;
}
__device__ __forceinline__ void columns_done(Pipe &pp, int nz) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(pp.b->cempty + pp.buf);
    pp.next_tile(nz);
}

// The decisions after a phase R and after an inner sweep, on a domain's control
// record from its sums.  `report`: also into the domain's diagnostics and the
// count of active domains.  live: the phase's count of live domains (null with
// one domain, whose record tells).
__device__ __forceinline__ void finalize_R(const DevPtrs &P, int dom, KrylovCtrl &c, bool report, int *live,
                                           const double (&v)[4]) {
    const DomainDesc &D = P.dom[dom];
    const double rr64 = v[0], bb = v[1];
    c.bb = bb;
    c.rr64 = rr64;
    c.cycles += 1;
    const double tol2 = D.krylov_tol * D.krylov_tol;
    const bool conv = rr64 <= tol2 * bb;
    const bool bad = !(rr64 == rr64) || !(bb == bb) || isinf(rr64);
    if (conv || bad || c.total_iter >= D.krylov_maxiter || c.cycles > MAX_CYCLES) {
        c.active = 0;
        if (report) {
            atomicSub(&P.gctrl->n_active, 1);
            DevDiag &dg = P.diag[dom];
            if (!conv) dg.krylov_nonconverged += 1;
            if (bad) dg.nonfinite = 1;
            dg.krylov_relres_last = bb > 0 ? sqrt(rr64 / bb) : sqrt(rr64);
        }
    } else {
        c.inner_active = 1;
        if (live) atomicAdd(live, 1);
        c.inner_iter = 0;
        c.first_inner = 1;
        c.rz = v[2];
        c.alpha = 0.0;
        // A later cycle continues the direction of the previous one: the true
        // residual replaces the recursive one (z = M^-1 r from phase R) and
        // p = z + beta p with beta = rho_true / rho_last ("reliable update"),
        // so refinement does not discard the Krylov space built so far.
        c.keep_p = (c.total_iter > 0 && c.rho_last > 0.0) ? 1 : 0;
        c.beta = c.keep_p ? v[2] / c.rho_last : 0.0;
        // the inner solve reduces r.M^-1 r by inner_tol^2 (mixed mode), or far
        // enough that ||r|| should meet the outer tolerance (half of it, with
        // the M^-1-norm standing in for the 2-norm); R checks the true residual
        c.inner_target2 = v[2] * fmax(D.inner_tol * D.inner_tol, 0.25 * tol2 * bb / rr64);
    }
}

__device__ __forceinline__ void finalize_C(const DevPtrs &P, int dom, KrylovCtrl &c, int *live, const double (&v)[4]) {
    const DomainDesc &D = P.dom[dom];
    const double sigma = v[0], mu = v[1], nu = v[2], rho = v[3];
    const double alpha = rho / sigma;
    const double rho_next = rho - 2.0 * alpha * mu + alpha * alpha * nu;
    const bool bad = !(sigma > 0.0) || isinf(sigma) || !(rho > 0.0) || !(rho_next == rho_next);
    c.alpha = bad ? 0.0 : alpha;  // a broken iteration leaves x alone
    c.beta = bad ? 0.0 : rho_next / rho;
    c.rz = rho_next;
    c.rho_last = bad ? 0.0 : rho;
    c.parity ^= 1;
    c.first_inner = 0;
    c.inner_iter += 1;
    c.total_iter += 1;
    if (bad || rho_next <= c.inner_target2 || c.inner_iter >= D.inner_maxiter || c.total_iter >= D.krylov_maxiter)
        c.inner_active = 0;
    else if (live)
        atomicAdd(live, 1);
}

// The sums of a domain's partials (a warp; lane 0 gets them).  A phase's are not
// overwritten in the next one, where a slow block may still be reading them; nor
// by the Picard check (row 0), which follows a solve's last phase R in k_step_pipe
// with no barrier between them.
enum { PART_ROW0 = 4 };
static_assert(PART_ROW0 + 8 <= NPART, "four rows each for even and odd phases");
__device__ __forceinline__ double *part_at(const DevPtrs &P, unsigned phase, int i, int t) {
    return P.partials + ((size_t)(PART_ROW0 + 4 * (phase & 1u)) + i) * P.ntiles + t;
}
__device__ __forceinline__ void sum_parts(const DevPtrs &P, unsigned phase, int begin, int parts, double (&v)[4]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = 0.0;
#pragma unroll 5
    for (int t = begin + lane; t < begin + parts; t += 32)
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] += __ldcg(part_at(P, phase, i, t));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
    }
}

// A domain's sums over this block's tiles (three from the plane warps, `mine`
// from the column threads, third of the four) into the domain's partials, at the
// block's first tile of the domain; min(tiles, blocks) blocks contribute.  With
// several domains the last block to arrive decides for the domain; one domain's
// blocks all decide for themselves after the grid barrier (decide), which leaves
// the chain between two sweeps shorter.  The partials are summed in the same
// order either way, whichever block is last, so the result is reproducible.
template <bool RESIDUAL>
__device__ __forceinline__ void block_reduce(const DevPtrs &P, Pipe &pp, PipeShared *sh, unsigned phase, int tile,
                                             const TileCtx &td, double mine) {
    const int f = pp.flushes & 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, o);
    if (lane == 0) sh->csum[f][warp] = mine;
    mbar_sleep(pp.b->red + f, (pp.flushes >> 1) & 1u, P.barrier);
    pp.flushes += 1;
    group_sync<STEP_GROUPS>();
    if (warp != 0) return;
    const int n = td.end - td.begin, grid = (int)gridDim.x, parts = n < grid ? n : grid;
    if (lane < 4) {
        const double *w = sh->csum[f];
        static_assert(COL_THREADS == 128 && PLANE_WARPS == 8, "sums in pairs: a chain of three additions");
        double a = (w[0] + w[1]) + (w[2] + w[3]);
        if (lane != 2) {
            const double(*q)[3] = sh->sums[f];
            const int i = lane == 3 ? 2 : lane;
            a = ((q[0][i] + q[1][i]) + (q[2][i] + q[3][i])) + ((q[4][i] + q[5][i]) + (q[6][i] + q[7][i]));
        }
        __stcg(part_at(P, phase, lane, td.begin + (tile - td.begin) % grid), a);
    }
    if (P.ndom == 1) return;
    __syncwarp();
    unsigned int prev = 0;
    if (lane == 0)
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(prev) : "l"(&P.arrive[td.dom * 4]) : "memory");
    prev = __shfl_sync(0xffffffffu, prev, 0);
    if (prev != (unsigned int)(parts - 1)) return;
    __threadfence();
    double v[4];
    sum_parts(P, phase, td.begin, parts, v);
    if (lane != 0) return;
    P.arrive[td.dom * 4] = 0u;
    if (RESIDUAL) finalize_R(P, td.dom, P.kctrl[td.dom], true, live_slot(P, phase), v);
    else finalize_C(P, td.dom, P.kctrl[td.dom], live_slot(P, phase), v);
}

// One domain: every block sums the partials after the grid barrier and keeps the
// control record in shared memory; block 0 also writes it back and reports.
template <bool RESIDUAL>
__device__ __forceinline__ void decide(const DevPtrs &P, SolveBlock &b) {
    if (threadIdx.x < 32) {
        const int grid = (int)gridDim.x;
        double v[4];
        sum_parts(P, b.phase - 1, 0, P.ntiles < grid ? P.ntiles : grid, v);
        if (threadIdx.x == 0) {
            const bool report = blockIdx.x == 0;
            if (RESIDUAL) finalize_R(P, 0, b.sh->ctl, report, nullptr, v);
            else finalize_C(P, 0, b.sh->ctl, nullptr, v);
            if (report) P.kctrl[0] = b.sh->ctl;
        }
    }
    __syncthreads();
}

// One sweep of phase R (RESIDUAL) or of the inner solve over this block's tiles
// (those at blockIdx.x + n gridDim.x), in this thread's role.  A domain's
// control record changes only when the last block's sums of it have arrived,
// after every role is past the domain's tiles, so within a sweep each role
// reads it once per domain.
template <typename T, int TXC, bool RESIDUAL>
__device__ __forceinline__ void run_sweep(const DevPtrs &P, SolveBlock &b, int role) {
    Pipe &pp = RESIDUAL ? b.r : b.c;
    SweepCtl c{-1, 0, 0, false, false, 0.0, 0.0};
    live_begin(P, b.phase);
    // fn(tile, its record, how many tiles of its domain the block had before,
    // whether it is the block's last one) for every tile of a live domain
    auto each_tile = [&](auto fn) {
        int n = 0;
        for (int t = blockIdx.x; t < P.ntiles; t += gridDim.x, ++n) {
            const TileCtx td = n < TILE_TABLE ? b.sh->tiles[n] : tile_ctx(P, t);
            if (P.ndom == 1) load_ctl<RESIDUAL>(c, td.dom, &b.sh->ctl, [](auto *q) { return *q; });
            else load_ctl<RESIDUAL>(c, td.dom, &P.kctrl[td.dom], [](auto *q) { return ldcg(q); });
            if (c.active) fn(t, td, (t - td.begin) / (int)gridDim.x, t + (int)gridDim.x >= td.end);
        }
    };
    if (role == ROLE_PRODUCER) {
        const int half = (threadIdx.x >> 5) & 1;
        if ((threadIdx.x & 31) == 0)
            each_tile([&](int, const TileCtx &td, int, bool) {
                if constexpr (RESIDUAL) produce_R<T>(P, td, c, half, pp, &b.sh->issued[half]);
                else produce_C<T>(P, td, c, half, pp, &b.sh->issued[half]);
            });
        __syncwarp();
    } else if (role == ROLE_OBSERVER) {
        if ((threadIdx.x & 31) == 0)
            each_tile([&](int t, const TileCtx &td, int, bool last) {
                const int units = units_of(td.nz);
                for (int q = 0; q < units; ++q) {
                    if (!mbar_sleep(pp.b->full + pp.slot, pp.par, P.barrier)) return;
                    pp.unit += 1;
                    asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_addr(pp.landed)), "r"(pp.unit)
                                 : "memory");
                    pp.step(pp.slot, pp.par, 1);
                    if constexpr (PF_UNITS > 0 && !RESIDUAL) {
                        // the L2 prefetch of the unit PF_UNITS beyond the ring, in this
                        // tile or the block's next one of the domain
                        const int ahead = q + pp.n + PF_UNITS;
                        if (ahead < units) prefetch_C<T>(P, td, c, ahead * UNIT, td.x0, td.y0);
                        else if (!last && ahead - units < units) {
                            const TileDesc nt = P.tiles[t + (int)gridDim.x];
                            prefetch_C<T>(P, td, c, (ahead - units) * UNIT, nt.x0, nt.y0);
                        }
                    }
                }
            });
        __syncwarp();
    } else if (role == ROLE_PLANE) {
        double s[3] = {0.0, 0.0, 0.0};  // the domain's sums over this warp's planes: a tile's in T, tiles in FP64
        each_tile([&](int, const TileCtx &td, int turn, bool last) {
            const bool wide = TXC == TILE_X || (TXC == 0 && td.tx == TILE_X);
            if constexpr (RESIDUAL) {
                if (wide) planes_R<T, TILE_X>(P, td, c, turn, pp, s);
                else planes_R<T, 16>(P, td, c, turn, pp, s);
            } else {
                P2<T> a[3] = {};
                if (wide) {
                    if (!c.first) planes_C<T, TILE_X, 2>(P, td, c, turn, pp, a);
                    else if (c.keep_p) planes_C<T, TILE_X, 1>(P, td, c, turn, pp, a);
                    else planes_C<T, TILE_X, 0>(P, td, c, turn, pp, a);
                } else {
                    if (!c.first) planes_C<T, 16, 2>(P, td, c, turn, pp, a);
                    else if (c.keep_p) planes_C<T, 16, 1>(P, td, c, turn, pp, a);
                    else planes_C<T, 16, 0>(P, td, c, turn, pp, a);
                }
#pragma unroll
                for (int i = 0; i < 3; ++i) s[i] += (double)a[i].x + (double)a[i].y;
            }
            if (last) {
                plane_sums(pp, b.sh, s);
                s[0] = s[1] = s[2] = 0.0;
            }
        });
    } else {
        double s = 0.0;
        each_tile([&](int t, const TileCtx &td, int, bool last) {
            // R: z goes into the buffer that holds the last iteration's p (the
            // next sweep reads both from there); C: t beside the new z and p
            T *out = RESIDUAL ? (T *)(c.parity ? P.z1 : P.z0) : (T *)(c.parity ? P.t0 : P.t1);
            if (RESIDUAL && c.first) s += columns<T, RESIDUAL>(P, td, pp, out);
            else s += columns<T, false>(P, td, pp, out);
            if (last) {
                // before the buffer is given back: the plane warps' next sums but one
                // of a domain go where these are
                if constexpr (RESIDUAL) {
                    block_reduce<true>(P, pp, b.sh, b.phase, t, td, s);  // ||r||^2, ||b||^2, r.z
                } else {
                    block_reduce<false>(P, pp, b.sh, b.phase, t, td, s);  // p.q, z.q, q.t, z.M z
                }
                s = 0.0;
            }
            columns_done(pp, td.nz);
        });
    }
}

// U: x += d + alpha p (the pending update of a cycle's last iteration), a plane
// of a tile per compute warp at a time.
template <typename T>
__device__ __forceinline__ void update_x(const DevPtrs &P, SolveBlock &b) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = SOLVE_THREADS / 32;
    int n = 0;
    for (int t = blockIdx.x; t < P.ntiles; t += gridDim.x, ++n) {
        const TileCtx td = n < TILE_TABLE ? b.sh->tiles[n] : tile_ctx(P, t);
        const KrylovCtrl *kc = P.ndom == 1 ? &b.sh->ctl : &P.kctrl[td.dom];
        auto get = [&](auto *q) { return P.ndom == 1 ? *q : ldcg(q); };
        if (!get(&kc->active) || get(&kc->first_inner)) continue;
        const T *__restrict__ d = (const T *)P.d;
        const T *__restrict__ p = (const T *)(get(&kc->parity) ? P.p1 : P.p0);
        const double a = get(&kc->alpha);
        double *__restrict__ x = P.x;
        const int px = lane & (td.tx / 2 - 1), row = lane / (td.tx / 2), rows = 64 / td.tx;
        const int i = td.x0 + 2 * px;
        // two rows of up to two planes at once: eight pairs of loads in flight
        for (int k = warp; k < td.nz; k += 2 * warps) {
            unsigned g[4];
            bool ok[4];
            P2<T> dd[4], pp[4];
            double2 xx[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int kk = k + (e >> 1) * warps, j = td.y0 + row + (e & 1) * rows;
                ok[e] = kk < td.nz && i < td.nx && j < td.ny;
                g[e] = td.off + (unsigned)j * (unsigned)td.nxp + (unsigned)i + (unsigned)kk * td.sxy;
                if (ok[e]) {
                    dd[e] = get2<T>(d + g[e]);
                    pp[e] = get2<T>(p + g[e]);
                    xx[e] = get2<double>(x + g[e]);
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (ok[e]) {
                    xx[e].x += (double)dd[e].x + a * (double)pp[e].x;
                    xx[e].y += (double)dd[e].y + a * (double)pp[e].y;
                    put2<double>(x + g[e], xx[e]);
                }
        }
    }
}

__device__ __forceinline__ SolveBlock solve_block(const DevPtrs &P, unsigned char *smem_raw, PipeShared *sh) {
    if (threadIdx.x == 0) {
        sh->issued[0] = sh->issued[1] = sh->landed_c = sh->landed_r = 0;
        for (PipeBars *q : {&sh->c, &sh->r}) {
            for (int i = 0; i < RING_MAX; ++i) {
                mbar_init(q->full + i, 2);
                mbar_init(q->empty + i, 2 * UNIT_WARPS);
            }
            for (int i = 0; i < 2; ++i) {
                mbar_init(q->cfull + i, PLANE_WARPS);
                mbar_init(q->cempty + i, COL_THREADS / 32);
                mbar_init(q->red + i, PLANE_WARPS);
            }
        }
        mbar_fence_init();
    }
    for (int n = threadIdx.x, t = blockIdx.x + n * gridDim.x; n < TILE_TABLE && t < P.ntiles;
         n += blockDim.x, t += blockDim.x * gridDim.x)
        sh->tiles[n] = tile_ctx(P, t);
    __syncthreads();
    unsigned char *mem = smem_raw + ((128u - (smem_addr(smem_raw) & 127u)) & 127u);
    auto pipe = [&](PipeBars *q, const PipeShape &s, unsigned *landed) {
        return Pipe{q, mem, mem + s.nb * s.colb, s.n, s.stage, s.nb, s.colb, landed, 0, 0u, 0, 0u, 0u, 0u};
    };
    return SolveBlock{pipe(&sh->c, P.pipe_c, &sh->landed_c), pipe(&sh->r, P.pipe_r, &sh->landed_r), sh, 0u, 0u};
}

// Grid barrier of the solve: a counter (zeroed by the assembly before it) that
// every block adds to once per phase.  What the phase wrote is read by the TMA
// in the next one, so both sides order it for the async proxy.  So is what it
// wrote to shared memory: the two kinds of sweep may have another number of
// column buffers (FP64 columns of 26 to 35 layers, mixed ones of 48 and 49), and
// one's second buffer is then where the other's TMA writes its first stages.
__device__ __forceinline__ bool solve_sync(const DevPtrs &P, SolveBlock &b) {
    asm volatile("fence.proxy.async;\n" ::: "memory");
    b.target += gridDim.x;
    b.phase += 1;
    const bool ok = counter_sync(&P.gctrl->kry_bar, b.target, P.barrier);
    asm volatile("fence.proxy.async.global;\n" ::: "memory");
    return ok;
}

// The whole linear solve of one Picard iteration for every active domain (the
// body of k_krylov, also run by k_step).  Returns false when a grid barrier
// gave up (the handle's error flag is set); the block must then return.
// TXC: the tile width when every domain of the handle has the same (the sweeps
// are then compiled for it), 0 when it differs by domain (each tile is
// dispatched to the sweep of its shape).
template <typename T, int TXC>
__device__ __forceinline__ bool solve(const DevPtrs &P, SolveBlock &b) {
    const int role = role_of();
    // every error exit first lets this block's in-flight stage copies land
    auto fail = [&]() {
        if (threadIdx.x == SOLVE_THREADS - 96 || threadIdx.x == SOLVE_THREADS - 64) {
            b.c.drain(b.sh->issued[(threadIdx.x >> 5) & 1]);
            b.r.drain(b.sh->issued[(threadIdx.x >> 5) & 1]);
        }
        return false;
    };
    b.target = 0;
    const bool one = P.ndom == 1;
    if (one) {
        if (threadIdx.x == 0) b.sh->ctl = P.kctrl[0];
        __syncthreads();
        // its Picard iteration has converged: no sweep would visit a tile, and there
        // are no sums to decide on
        if (b.sh->ctl.active == 0) return true;
    }
    for (;;) {
        // ---- R: outer residual
        run_sweep<T, TXC, true>(P, b, role);
        if (!solve_sync(P, b)) return fail();
        if (one) decide<true>(P, b);
        if (one ? b.sh->ctl.active == 0 : ldcg(&P.gctrl->n_active) == 0) break;
        // ---- inner PCG: one sweep and one grid barrier per iteration
        while (one ? b.sh->ctl.inner_active != 0 : ldcg(live_slot(P, b.phase - 1)) > 0) {
            run_sweep<T, TXC, false>(P, b, role);
            if (!solve_sync(P, b)) return fail();
            if (one) decide<false>(P, b);
        }
        // ---- U
        live_begin(P, b.phase);
        update_x<T>(P, b);
        if (!solve_sync(P, b)) return fail();
    }
    return true;
}

}  // namespace pipe
