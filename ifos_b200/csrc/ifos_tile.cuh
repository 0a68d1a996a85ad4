// Persistent, TMA-pipelined stencil kernels (fp32).
//
// Each block loops over 64 x TY tiles of the grid (all shot slots).  A
// producer warp streams every input plane of a tile into a ring of NST
// shared-memory stages with bulk tensor loads (cp.async.bulk.tensor, never
// with cluster multicast): the planes that need neighbours (the stresses in
// the velocity update, the velocities in the stress update) as tile + halo
// boxes, the per-cell planes (fields, memory variables, coefficients) as
// plain tile boxes.  The compute warps release a stage as soon as they have
// read it and write their results straight to HBM with vector stores (on
// snapshot steps also the stored wavefield components, into the snapshot
// buffer), so the ring only ever waits on loads.
//
// A thread owns four adjacent cells of one row and a warp two rows of the
// tile, or two cells and one row (Pipe's V).  Warps whose rows need nothing but the plain update (no CPML strip cell, no
// free surface, receiver, source or ragged edge) take a path without any of
// that code.  The per-cell arithmetic is the reference's, in the same order
// and with the same float/double promotions as the one-thread-per-cell
// kernels of ifos_kernels.cuh.
#pragma once
#include <limits.h>
#include <algorithm>
#include <type_traits>

#include "ifos_kernels.cuh"
#include "ifos_snap.cuh"
#include "ifos_tma.cuh"

// 1: the reference's double-promoted terms are evaluated in double (bit-exact);
// 0: in single precision
#ifndef IFOS_EXACT
#define IFOS_EXACT 1
#endif

namespace ifos {

// Resident blocks per SM that the launch bounds and the ring are sized for.
// More blocks cap the registers and spill: 64 shots of 400 x 160 at FDORDER 4
// with 4, 5 and 6 blocks: velocity 47, 51 and 54 us, stress 46, 52 and 51;
// 4000 x 1200 at FDORDER 8 with 3, 5 and 6: velocity 53, 56 and 57, stress 46,
// 49 and 53.  The viscoelastic stress fills the shared memory with two blocks
// of two 46 KB stages; three or four blocks of one stage were slower (2000 x
// 600: 42 us against 46 and 52).
constexpr int sblocks(int fdoh) { return fdoh <= 2 ? 4 : 3; }
constexpr int vblocks(int fdoh) { return fdoh <= 2 ? 4 : 3; }
constexpr int visc_blocks(int LL) { return LL <= 1 ? 3 : 2; }
// Half widths and memory variables for which the viscoelastic stress's DIRECT
// form is faster on large batches (Launcher::s_visc_pipe), 4 shots of 2000 x
// 600, forward + adjoint step without and with it (us), with one model, and
// with a model per shot:
//   L 3, FDORDER 2, 4, 6, 8 and 12: 144 + 161 and 140 + 158, 144 + 165 and 139 + 161,
//     145 + 161 and 140 + 160, 147 + 163 and 141 + 160, 140 + 145 and 133 + 138; models
//     160 + 178 and 157 + 176, 160 + 183 and 156 + 179, 160 + 179 and 156 + 176, 163 +
//     181 and 156 + 176, 157 + 162 and 149 + 155;
//   L 4, FDORDER 4, 8 and 12: 171 + 192 and 167 + 184, 174 + 192 and 162 + 185, 161 +
//     168 and 160 + 166; models 187 + 209 and 182 + 202, 190 + 210 and 178 + 201, 167 +
//     174 and 174 + 181 (24 shots of 1300 x 400: 436 + 451 and 544 + 558);
//   L 1, FDORDER 2, 4, 6, 8, 10 and 12: 98 + 116 and 129 + 115, 100 + 145 and 126 +
//     123 (24 of 1300 x 400: 243 + 334 and 327 + 325), 124 + 135 and 101 + 153, 130 +
//     143 and 107 + 142, 103 + 111 and 105 + 112, 103 + 111 and 91 + 102;
//   L 2, FDORDER 4, 8 and 12: 115 + 138 and 122 + 144, 118 + 134 and 124 + 142, 111 +
//     116 and 111 + 117; L 5: 183 + 204 and 195 + 214, 187 + 202 and 194 + 217, 176 + 183
//     and 188 + 195.
constexpr bool visc_direct(int fdoh, int LL) {
    return LL == 3 || (LL == 4 && fdoh <= 4) || (LL == 1 && (fdoh == 3 || fdoh == 4 || fdoh == 6));
}
constexpr int kTileX = 64;
// Cells per thread.  Four halve the loads, addresses and bookkeeping per cell;
// two leave room for twice the warps.  Four win where instructions bound the
// op (64 shots of 400 x 160, FDORDER 4: velocity 48 against 54 us, stress 48
// against 60; 4000 x 1200, FDORDER 8: elastic stress 47.2 against 48.7, SH
// 28.7 against 30.8), two in the viscoelastic stress, whose four cells need
// 168 registers (6 shots of 2000 x 600: 177 against 185 us; 3000 x 1000: 76
// against 82), and in the P-SV velocity of the wide stencils (4000 x 1200,
// FDORDER 8: 47.1 against 49.8).
constexpr int kCells = 4, kCellsVisc = 2;
// Tiles a block up to which a launch of the P-SV elastic FDORDER 2 and 4 ops
// is a programmatic dependent one (the others always are).  Their four blocks
// of 96 registers fill the register file, and while the blocks of the
// preceding launch leave one by one the next one's do not pack: 15 tiles a
// block (64 shots of 400 x 160) took 47 instead of 38 ms a forward loop, 21
// tiles 14.9 instead of 13.4, 5.4 tiles 56.6 instead of 53.6; below that the
// hidden start wins (2.2 tiles: 4.0 instead of 4.75 ms).
constexpr int kDepTiles = 5;
constexpr int cells_v(int fdoh) { return fdoh <= 2 ? 4 : 2; }

using D = std::conditional<IFOS_EXACT != 0, double, float>::type;

// Plane ids for the TMA z coordinate: state plane = slot * planes_per_slot + pid,
// model plane = model * model_planes + mid; snap_comp: the snapshot
// component of a state plane.
struct KTma {
    int planes_per_slot;
    int pid[NP_FIELD];
    int mem_pid[N_MEM];
    int model_planes;
    int mid[NM_PLANE];
    int snap_comp[NP_FIELD];  // component index of a state plane (-1: not stored)
};

// The tensor maps of a launch: the halo planes of a tile are one box of NH_
// consecutive state planes, the per-cell planes up to five boxes of
// consecutive state or model planes each (Op::GD, Op::GM).
constexpr int kMaxGroups = 5;
struct KMaps {
    CUtensorMap halo;             // state planes, box (64+2XH) x (TY+2H) x NH_
    CUtensorMap grp[kMaxGroups];  // state or model planes, box 64 x TY x GD[k]
};

// the snapshot a stencil launch stores (base NULL: none)
struct KSnapOut {
    char *base;            // this snapshot of slot 0
    long long slot_bytes;  // bytes between slots
    long long n;           // NX*NY
    int align;             // 4, 2 or 1: cells of a row that are aligned for vector stores (by NX)
    int f16;               // fp16 segments (IFOS_SNAP_F16S); else fp32
    long long ex_off;      // fp16: bytes from a snapshot to its segment scales [comp][NY][segs]
    int segs;              // fp16: segments per row
};

// The shared-memory ring of an op: NH halo planes and NP plain planes a stage,
// NST stages; V cells per thread: 4 (a compute warp takes two tile rows) or 2
// (one row); BCAP resident blocks per SM that the launch bounds aim for.
template <int FDOH, int TY, int NH, int NP, int NST, int BCAP = 3, int V = 4>
struct Pipe {
    static constexpr int ROWS = V / 2;                // tile rows of a compute warp
    static constexpr int NCW = TY / ROWS;             // compute warps; the block adds one producer warp
    static constexpr int THREADS = 32 * NCW + 32;
    static constexpr int TX = kTileX, H = FDOH;
    static constexpr int XH = ((FDOH + 3) / 4) * 4;  // staged x halo (16-byte TMA alignment)
    static constexpr int BW = TX + 2 * XH, BH = TY + 2 * H;
    static constexpr int BOXS = BW * BH;                        // a plane of the halo box
    static constexpr int HALO = (NH * BOXS + 31) / 32 * 32;     // the halo box, 128-byte aligned
    static constexpr int PLS = TX * TY;
    static constexpr int STAGES = NST;
    static constexpr int STAGE = HALO + NP * PLS;
    static constexpr int TILE_Y = TY;
    static constexpr uint32_t TXB = (uint32_t)((NH * BW * BH + NP * PLS) * 4);
    static constexpr size_t bytes() { return (size_t)NST * STAGE * 4; }
    static constexpr int BLOCK_CAP = BCAP;
    static_assert((V == 4 || V == 2) && TY % ROWS == 0 && NCW <= 8, "tile rows and compute warps");
};

// One tile as the producer hands it to the compute warps.
struct __align__(16) TileInfo {
    int slot, i0, j0;
    int bits;  // model index of the slot * 256, + bit w: the rows of compute warp w need more than the plain update
    __device__ __forceinline__ int model() const { return bits >> 8; }
    __device__ __forceinline__ bool edge(int w) const { return (bits >> w) & 1; }
};

// a / b and the remainder for 0 <= a < 2^24, rb = 1/b: the float quotient is
// off by at most one
__device__ __forceinline__ int div_small(int a, int b, float rb, int &rem) {
    int q = (int)((float)a * rb);
    rem = a - q * b;
    if (rem < 0) q--, rem += b;
    if (rem >= b) q++, rem -= b;
    return q;
}

// Tile t of a launch.  Slot-major order walks all tiles of slot 0, then of
// slot 1, ...; slot-minor order gives consecutive t the same tile of
// consecutive slots, so the CTAs resident at one time share the model tiles
// of shots over the same model (one HBM read, the rest from L2).
//
// CPML-first order (tile order bit 1): the spatial rank runs over the tiles
// that meet a CPML strip first -- the tile rows in a y strip (top without a
// free surface, bottom), then the x-strip columns (left, right) of the other
// rows -- and the interior last, each region row by row.  Strip tiles take
// the slower CPML path of every op; ranked first, the round-robin of tiles
// over the persistent CTAs hands each CTA the same number of them (within
// one), so the CTAs finish together instead of the ones that drew the strip
// columns finishing last.  A bijection on [0, ntx*nty).
//
// The launcher makes the struct (Launcher::pipelined) with everything the
// producer warp needs before its first loads, in a few adjacent words of the
// parameters.  Worked out on the device from the members of the op, the first
// tile's indices took 2600-3200 cycles in front of every launch's first loads,
// twice what the whole producer start had taken with one lane and no classes of
// warps; so they take 1100-1300 (400 x 160, FDORDER 4, no dependent launches:
// 9.8 to 7.5 us a forward step; with them acoustic 777 x 259 8.2 to 7.6, 1010 x
// 336 viscoelastic, two shots, 23.7 to 22.6).
struct TileWalk {
    int ntx, per, nshots, ntiles;  // tile columns, tiles of a slot, slots, all tiles
    float r_ntx, r_shots, r_per;
    // tile order (slot-minor, CPML first) and its CPML-first regions: rows in a
    // top y strip, first row of the bottom one, tiles in y-strip rows; left
    // x-strip columns, first right one, x-strip columns and their tiles in the
    // other rows, columns between
    int minor, cpml;
    int rt, yb0, ny_tiles, cl, xr0, ce, nx_tiles, mid;
    float r_ce, r_mid;
    // Compute warps whose rows need more than the plain update: all of a tile
    // outside the tile columns px0..px1-1 (an x strip, cells outside the grid)
    // or of the top tiles if `top` (rows imaged at the free surface, velocity);
    // else those with a row of the ranges lo..hi: top y strip or the surface
    // itself, bottom y strip and rows outside the grid, the probe's row,
    // receiver rows, source rows
    enum { R_TOP, R_BOTTOM, R_PROBE, R_REC, R_SRC, NR };
    int px0, px1, top;
    int lo[NR], hi[NR];
    // The receiver and source ranges span all slots.  Where one holds more than
    // one row, the slot's own rows are looked up (KRec::rows; NULL: the range says
    // it all), so that shots at several depths, or receivers in
    // a shallow and a deep row, do not put all rows between on the longer path.
    // A forward step with the ranges alone, with the lookup, and with one row
    // (us): six viscoelastic shots of 2000 x 600 at six depths 261, 217 and 215;
    // four acoustic shots of 1500 x 500 at four depths 47.2, 34.9 and 32.2; a
    // P-SV shot of 4000 x 1200 with two receiver rows 88.5, 73.9 and 71.9.
    // The lookup is out of line: a block works out its first tiles in code that
    // comes cold from the instruction cache, and this part is rarely needed.
    int lookup;
    const unsigned char *own[2];
    long long own_stride;
    // TMA z coordinates: planes of a slot and of a model, the halo box's first plane, the groups'
    int slot_planes, model_planes, zh, zg[kMaxGroups];

    template <typename Op>
    static TileWalk of(const Op &op, int shots) {
        using std::max;
        using std::min;
        const KGrid &g = op.g;
        constexpr int TY = Op::P::TILE_Y;
        TileWalk w{};
        const int nty = (g.ny + TY - 1) / TY;
        w.ntx = (g.nx + kTileX - 1) / kTileX;
        w.per = w.ntx * nty;
        w.nshots = shots;
        w.ntiles = w.per * shots;
        w.r_ntx = 1.0f / w.ntx, w.r_shots = 1.0f / shots, w.r_per = 1.0f / w.per;
        w.minor = g.tile_order & 1;
        w.cpml = (g.tile_order & 2) && g.fw > 0;
        w.cl = min(w.ntx, (g.fw - 1) / kTileX + 1);  // tile columns with i0 <= FW
        const int vx = g.nx - g.fw + 1 - kTileX;     // right strip: min(i0+63, NX) >= NX-FW+1
        w.xr0 = max(w.cl, vx <= 0 ? 0 : (vx + kTileX - 1) / kTileX);
        w.rt = g.free_surf ? 0 : min(nty, (g.fw - 1) / TY + 1);  // tile rows with j0 <= FW
        const int vy = g.ny - g.fw + 1 - TY;                     // bottom strip: j0+TY-1 >= NY-FW+1
        w.yb0 = min(nty, max(w.rt, vy <= 0 ? 0 : (vy + TY - 1) / TY));
        w.ny_tiles = (w.rt + nty - w.yb0) * w.ntx;
        w.ce = w.cl + (w.ntx - w.xr0);
        w.nx_tiles = (w.yb0 - w.rt) * w.ce;
        w.mid = w.ntx - w.ce;
        w.r_ce = 1.0f / w.ce, w.r_mid = w.mid > 0 ? 1.0f / w.mid : 0.0f;

        const bool ystrips = Op::CPML && g.fw > 0, xstrips = ystrips && !g.boundary;
        w.px0 = xstrips ? (g.fw - 1) / kTileX + 1 : 0;
        w.px1 = (g.nx - (xstrips ? g.fw : 0)) / kTileX;
        w.top = Op::MIRROR && g.free_surf;
        auto range = [&](int k, bool on, int a, int b) { w.lo[k] = on ? a : 1, w.hi[k] = on ? b : 0; };
        range(R_TOP, g.free_surf ? op.fsurf != 0 : ystrips, 1, g.free_surf ? 1 : g.fw);
        range(R_BOTTOM, true, ystrips ? g.ny - g.fw + 1 : g.ny + 1, INT_MAX);
        range(R_PROBE, op.probe, g.ny / 2, g.ny / 2);
        range(R_REC, op.rec_mode, op.rec_j0, op.rec_j1);
        range(R_SRC, op.fps || op.fvs, op.src_j0, op.src_j1);
        static_assert(TY == 8, "a tile's rows are one byte of the row tables");
        w.own[0] = w.hi[R_REC] > w.lo[R_REC] ? op.rec.rows : nullptr;
        w.own[1] = w.hi[R_SRC] > w.lo[R_SRC] ? op.rec.rows + op.rec.row_bytes : nullptr;
        w.own_stride = op.rec.map_stride * 4;
        w.lookup = w.own[0] || w.own[1];

        int z[Op::NG];
        op.planes(w.zh, z);
        for (int k = 0; k < Op::NG; k++) w.zg[k] = z[k];
        w.slot_planes = op.tm.planes_per_slot;
        w.model_planes = op.tm.model_planes;
        return w;
    }
    // tile row and column of a spatial rank in CPML-first order
    __device__ __forceinline__ int first(int rank, int &tx) const {
        if (rank < ny_tiles) {
            const int r = div_small(rank, ntx, r_ntx, tx);
            return r < rt ? r : yb0 + (r - rt);
        }
        rank -= ny_tiles;
        int c;
        if (rank < nx_tiles) {  // rows between the y strips: rt .. yb0-1
            const int r = div_small(rank, ce, r_ce, c);
            tx = c < cl ? c : xr0 + (c - cl);
            return rt + r;
        }
        rank -= nx_tiles;
        const int r = div_small(rank, mid, r_mid, c);  // mid > 0 here: the regions above hold every tile when it is not
        tx = cl + c;
        return rt + r;
    }
    // Tile t of the launch: slot, first cell, the slot's model (models NULL: 0),
    // and the bits of the compute warps of ROWS rows each that need more than the
    // plain update
    template <int TY, int ROWS>
    __device__ __forceinline__ TileInfo tile(int t, const int *models) const {
        TileInfo r;
        int rem, tx;
        if (nshots == 1) r.slot = 0, rem = t;
        else if (minor) rem = div_small(t, nshots, r_shots, r.slot);
        else r.slot = div_small(t, per, r_per, rem);
        const int model = models ? models[r.slot] : 0;  // requested before the rest is worked out
        const int ty = cpml ? first(rem, tx) : div_small(rem, ntx, r_ntx, tx);
        r.i0 = tx * kTileX + 1;
        r.j0 = ty * TY + 1;
        unsigned rows = tx < px0 || tx >= px1 || (top && ty == 0) ? (1u << TY) - 1 : 0u;
#pragma unroll
        for (int k = 0; k < R_REC; k++) rows |= range<TY>(k, r.j0);
        if (lookup) {
            rows |= own_rows<TY>(r.slot, ty, r.j0);
        } else {
            rows |= range<TY>(R_REC, r.j0) | range<TY>(R_SRC, r.j0);
        }
        r.bits = model * 256 + warps_of_rows<ROWS>(rows);
        return r;
    }
    // rows of range k in the tile that starts at row j0
    template <int TY>
    __device__ __forceinline__ unsigned range(int k, int j0) const {
        const int a = max(lo[k] - j0, 0), b = min(hi[k] - j0, TY - 1);
        return a <= b ? (2u << b) - (1u << a) : 0u;
    }
    // the slot's receiver and source rows in tile row ty
    template <int TY>
    __device__ __noinline__ unsigned own_rows(int slot, int ty, int j0) const {
        unsigned m = 0;
        for (int k = R_REC; k <= R_SRC; k++) {
            const unsigned r = range<TY>(k, j0);
            const unsigned char *p = own[k - R_REC];
            if (r) m |= p ? p[slot * own_stride + ty] : r;
        }
        return m;
    }
    // bit w: one of the rows of compute warp w
    template <int ROWS>
    static __device__ __forceinline__ int warps_of_rows(unsigned rows) {
        static_assert(ROWS == 1 || ROWS == 2, "rows of a compute warp");
        if (ROWS == 1) return (int)rows;
        unsigned m = (rows | rows >> 1) & 0x55u;
        m = (m | m >> 1) & 0x33u;
        return (int)((m | m >> 2) & 0x0fu);
    }
};

// The profiles a block reads: in shared memory (staged once per block) when
// the strips are no wider than kProfX columns and kProfY rows, else the global
// tables.  Read from global memory the four profiles of a strip cell were four
// L2 round trips one after another, 2000 of the 3000 cycles of a strip tile.
struct ProfTab {
    const float *x, *y;  // K a b at the full points, K a b at the half points
    int xs, ys;          // values between two of them
    bool local;          // x is indexed by the column of a strip row, else by the grid column
};
// Tiles whose indices the producer warp works out at a time, one per lane.
constexpr int kTileBatch = 32;

// Warp-specialised persistent driver.  Warps 0..NCW-1 compute; the
// last warp produces: it walks the same tile sequence, waits until a stage
// has been released by all compute warps ("empty" barrier, one arrival per
// warp), and issues the bulk tensor loads of the next tile into it ("full"
// barrier, completed by the transaction bytes).  The indices of 32 tiles at a
// time are worked out by the 32 lanes into shared memory (tq), ahead of their
// loads; a compute warp may read those of its next tile as soon as the
// batch's barrier has completed, and starts the loads that its CPML needs
// (Op::prefetch) before it waits for the stage.  One lane working out one tile
// after another took 1700-2300 cycles a tile, more than the update itself
// (4000 x 1200, FDORDER 8: 900-1900), and held back the first loads of every
// launch by 2 us.  The planes of a tile arrive as a few boxes of consecutive
// planes (about 100 cycles of issue per box).
//
// Every wait is bounded: a wait that gives up records its code in *err (16/17:
// a compute warp on a stage's loads, 18: the producer on a stage's release,
// 19: a compute warp on a batch of tile indices) and the block winds down
// after its copies in flight: when the producer gives up before tile k_stop it
// records k_stop (stop_at) and issues nothing more; the compute warps still
// wait for every tile it issued (so that no copy into the ring is in flight
// when the block exits), compute none of them, and leave at k_stop.
template <typename P, typename Op>
__device__ __forceinline__ void run_pipeline(const KGrid &g, const KMaps &mp, const TileWalk &walk, const Op &op, int *err) {
    constexpr int NST = P::STAGES, TY = P::TILE_Y;
    extern __shared__ __align__(1024) unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t full[NST], empty[NST], filled;
    __shared__ TileInfo tq[2 * kTileBatch];
    __shared__ __align__(16) float sprof[Op::CPML ? 6 * (kProfX + kProfY) : 4];
    __shared__ int stop_at;  // -1 while the producer runs, else the first tile it did not issue
    float *smem = reinterpret_cast<float *>(sm_raw);
    const int ntiles = walk.ntiles;
    const int warp = threadIdx.y, lane = threadIdx.x;
    if (warp == P::NCW && lane == 0) {
        for (int s = 0; s < NST; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], P::NCW);
        }
        mbar_init(&filled, 1);
        stop_at = -1;
        fence_mbar_init();
    }
    __syncthreads();
    volatile int *stop = &stop_at;
    if (warp == P::NCW) {
        // tiles k0 .. k0+31 of this block; the entries they replace belong to
        // tiles the compute warps have left (they are at most NST behind)
        auto fill = [&](int k0) {
            const int k = k0 + lane, t = blockIdx.x + k * gridDim.x;
            if (t < ntiles) {
                tq[k % (2 * kTileBatch)] = walk.tile<TY, P::ROWS>(t, op.M.one_model ? nullptr : op.M.slot_model);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&filled);
        };
        auto issue = [&](int k, int st, bool halo, bool plain) {
            const TileInfo ti = tq[k % (2 * kTileBatch)];
            float *stage = smem + st * P::STAGE;
            uint64_t *bar = &full[st];
            const int zs = ti.slot * walk.slot_planes, zm = ti.model() * walk.model_planes;
            if (plain) mbar_expect_tx(bar, P::TXB);
            if (halo)
                tma_load_3d(stage, &mp.halo, HX + ti.i0 - 1 - P::XH, HY + ti.j0 - 1 - P::H, zs + walk.zh, bar);
            if (plain) {
                const int px = HX + ti.i0 - 1, py = HY + ti.j0 - 1;
                int q = 0;
#pragma unroll
                for (int k = 0; k < Op::NG; k++) {
                    tma_load_3d(stage + P::HALO + q * P::PLS, &mp.grp[k], px, py, (Op::gm(k) ? zm : zs) + walk.zg[k], bar);
                    q += Op::gd(k);
                }
            }
        };
        fill(0);
        // The per-cell planes of the first NST tiles are not written by the
        // preceding kernel of the stream, so they are requested before
        // waiting for it; everything else after.
        int npre = 0;
        if (lane == 0) {
            for (; npre < NST && blockIdx.x + npre * gridDim.x < ntiles; npre++) issue(npre, npre, false, true);
            pdl_wait();
            for (int k = 0; k < npre; k++) issue(k, k, true, false);
        }
        npre = __shfl_sync(0xffffffffu, npre, 0);
        int st = 0;
        uint32_t parity = 0;
        for (int k = npre, t = blockIdx.x + k * gridDim.x; t < ntiles; k++, t += gridDim.x) {
            if (k % kTileBatch == 0) {
                __syncwarp();
                if (*stop >= 0) break;
                fill(k);
            }
            if (lane == 0 && *stop < 0) {
                if (mbar_wait_bounded(&empty[st], parity, err, 18, (long)g.prod_polls)) issue(k, st, true, true);
                else *stop = k;
            }
            if (++st == NST) {
                st = 0;
                parity ^= 1;
            }
        }
        // Only now may the next kernel's blocks start: they then find this
        // launch's blocks leaving and spread evenly over the SMs.  Released
        // after the first tiles they took the slots of the blocks that left
        // first and the SMs ended with two to four of them (4000 x 1200: 54
        // instead of 36 us a block).
        pdl_launch();
        return;
    }
    ProfTab pt{op.M.profx, op.M.prof + 6 * (2 * g.fw + 1), g.psy, 2 * g.fw + 1, false};
    if constexpr (Op::CPML) {
        if (op.M.proftab) {
            constexpr int n = 6 * (kProfX + kProfY) / 4;
            for (int k = warp * 32 + lane; k < n; k += 32 * P::NCW)
                reinterpret_cast<float4 *>(sprof)[k] = reinterpret_cast<const float4 *>(op.M.proftab)[k];
            asm volatile("bar.sync 1, %0;" ::"n"(32 * P::NCW) : "memory");
            pt = ProfTab{sprof, sprof + 6 * kProfX, kProfX, kProfY, true};
        }
    }
    int st = -1;
    uint32_t parity = 1;
    for (int k = 0, t = blockIdx.x; t < ntiles; k++, t += gridDim.x) {
        st = st + 1 == NST ? 0 : st + 1;
        if (st == 0) parity ^= 1;
        if (k % kTileBatch == 0) {
            bool ready = false;
            for (long it = 0; it < (1L << 16) && !ready; it++) {
                ready = mbar_try_wait(&filled, (uint32_t)(k / kTileBatch) & 1);
                if (!ready && *stop >= 0 && k >= *stop) return;  // never filled
            }
            if (!ready) {
                if (err) atomicExch(err, 19);
                mbar_wait_bounded(&full[st], parity, err, 17);
                return;
            }
        }
        const TileInfo ti = tq[k % (2 * kTileBatch)];
        const bool edge = ti.edge(warp);
        typename Op::Pre pre;
        if (edge) op.prefetch(ti, pre);
        if constexpr (Op::EARLY) {
            if (edge) op.template early<true>(ti, pre);
            else op.template early<false>(ti, pre);
        }
        bool landed = false;
        for (long it = 0; it < (1L << 16) && !landed; it++) {
            landed = mbar_try_wait(&full[st], parity);
            if (!landed && *stop >= 0 && k >= *stop) return;  // never issued: nothing in flight for it
        }
        if (!landed) {
            if (err) atomicExch(err, 16);
            mbar_wait_bounded(&full[st], parity, err, 17);
            return;
        }
        if (*stop >= 0) continue;  // the producer stopped: drain the tiles it issued, compute none
        const float *stage = smem + st * P::STAGE;
        if (edge) op.template rows<true>(ti, pre, pt, stage, stage + P::HALO, &empty[st]);
        else op.template rows<false>(ti, pre, pt, stage, stage + P::HALO, &empty[st]);
    }
}

// ---------------------------------------------------------------------------
// A thread owns V = 4 adjacent cells of one row (16-byte shared-memory reads
// and global stores): 16 lanes cover a tile row, a warp two rows; or 2, and a
// warp one row (kCells).  Against two cells, four halve the loads, the address
// arithmetic and the per-row bookkeeping of a cell; the stencils were bound by
// instruction issue, not by HBM (400 x 160, 64 shots, FDORDER 4: 263
// instructions a cell in the velocity update with DRAM at 25 % of its peak).

// FD weights of one launch
template <int FDOH>
struct Hc {
    float w[FDOH + 1];
    __device__ __forceinline__ explicit Hc(const KGrid &g) {
#pragma unroll
        for (int m = 0; m <= FDOH; m++) w[m] = g.hc[m];
    }
};

// V adjacent cells
template <int V>
struct FV {
    float v[V];
    __device__ __forceinline__ static FV of(float x) {
        FV r;
#pragma unroll
        for (int e = 0; e < V; e++) r.v[e] = x;
        return r;
    }
};
template <int V>
__device__ __forceinline__ FV<V> ldv(const float *p) {
    if constexpr (V == 4) {
        const float4 a = *reinterpret_cast<const float4 *>(p);
        return {{a.x, a.y, a.z, a.w}};
    } else {
        const float2 a = *reinterpret_cast<const float2 *>(p);
        return {{a.x, a.y}};
    }
}
// the same from L2, past this SM's L1
template <int V>
__device__ __forceinline__ FV<V> ldv_l2(const float *p) {
    if constexpr (V == 4) {
        const float4 a = __ldcg(reinterpret_cast<const float4 *>(p));
        return {{a.x, a.y, a.z, a.w}};
    } else {
        const float2 a = __ldcg(reinterpret_cast<const float2 *>(p));
        return {{a.x, a.y}};
    }
}
template <int V>
__device__ __forceinline__ void stv(float *p, const float (&v)[V]) {
    if constexpr (V == 4) *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
}

// Difference stencils of a thread's cells.  The m=1 term starts each sum
// and the others are added in order, as in the reference's written-out
// expressions (src/update_v_PML.c:164-175); Z0: the sum is accumulated from
// zero, as in its generic loops (the FDORDER 10/12 default branches, e.g.
// src/update_p_PML.c:275-287).  fwd: sum_m w_m (f[+m] - f[-m+1]);
// bwd: sum_m w_m (f[+m-1] - f[-m]).

// staged values of one row at columns c0-XB .. c0+V-1+XB (c0 a multiple of V)
template <int FDOH, int V>
struct XWin {
    static constexpr int XB = (FDOH + V - 1) / V * V, N = V + 2 * XB;
    float v[N];
    __device__ __forceinline__ void load(const float *row, int c0) {
#pragma unroll
        for (int q = 0; q < N / V; q++) {
            const FV<V> a = ldv<V>(row + c0 - XB + V * q);
#pragma unroll
            for (int e = 0; e < V; e++) v[V * q + e] = a.v[e];
        }
    }
};
template <bool Z0 = false, int FDOH, int V>
__device__ __forceinline__ float xfwd(const Hc<FDOH> &hc, const XWin<FDOH, V> &W, int e) {
    constexpr int XB = XWin<FDOH, V>::XB;
    float s = hc.w[1] * (W.v[XB + e + 1] - W.v[XB + e]);
    if (Z0) s = 0.0f + s;
#pragma unroll
    for (int m = 2; m <= FDOH; m++) s += hc.w[m] * (W.v[XB + e + m] - W.v[XB + e - m + 1]);
    return s;
}
template <bool Z0 = false, int FDOH, int V>
__device__ __forceinline__ float xbwd(const Hc<FDOH> &hc, const XWin<FDOH, V> &W, int e) {
    constexpr int XB = XWin<FDOH, V>::XB;
    float s = hc.w[1] * (W.v[XB + e] - W.v[XB + e - 1]);
    if (Z0) s = 0.0f + s;
#pragma unroll
    for (int m = 2; m <= FDOH; m++) s += hc.w[m] * (W.v[XB + e + m - 1] - W.v[XB + e - m]);
    return s;
}

// A thread's cells of a staged halo box at row offset dy from tile row jj.  MIR: the
// tile is the top one under a free surface, whose rows j<=0 read the imaged
// value the reference's ghost rows hold when the velocity is updated:
// -f(2-j) for syy, syz, sp (src/surface_elastic_PML.c:59) and -f(1-j) for sxy
// (:60).
template <bool MIR, bool ODD, typename P, int V>
__device__ __forceinline__ FV<V> ldy(const float *t, int jj, int c0, int dy) {
    const int rr = jj + P::H + dy;
    if (MIR && rr < P::H) {
        FV<V> a = ldv<V>(t + (ODD ? 2 * P::H - rr - 1 : 2 * P::H - rr) * P::BW + c0);
#pragma unroll
        for (int e = 0; e < V; e++) a.v[e] = -a.v[e];
        return a;
    }
    return ldv<V>(t + rr * P::BW + c0);
}
// FWD: rows +m and 1-m, else m-1 and -m
template <bool FWD, bool MIR, bool ODD, typename P, bool Z0 = false, int FDOH, int V>
__device__ __forceinline__ void ydiff(const Hc<FDOH> &hc, const float *t, int jj, int c0, float (&s)[V]) {
#pragma unroll
    for (int m = 1; m <= FDOH; m++) {
        const FV<V> a = ldy<MIR, ODD, P, V>(t, jj, c0, FWD ? m : m - 1);
        const FV<V> b = ldy<MIR, ODD, P, V>(t, jj, c0, FWD ? 1 - m : -m);
#pragma unroll
        for (int e = 0; e < V; e++) {
            const float d = hc.w[m] * (a.v[e] - b.v[e]);
            if (m == 1) s[e] = Z0 ? 0.0f + d : d;
            else s[e] += d;
        }
    }
}
// the same with the imaged rows where mir is set (the velocity ops)
template <bool FWD, bool EDGE, bool ODD, typename P, bool Z0 = false, int FDOH, int V>
__device__ __forceinline__ void ydiff_fs(const Hc<FDOH> &hc, const float *t, int jj, int c0, bool mir, float (&s)[V]) {
    if (EDGE && mir) ydiff<FWD, true, ODD, P, Z0>(hc, t, jj, c0, s);
    else ydiff<FWD, false, ODD, P, Z0>(hc, t, jj, c0, s);
}

// A thread's place in its tile: row jj, staged column c0, cell (j, i) of its
// first column, and the number of its cells inside the grid (nv; V on tiles
// that are not EDGE).
struct Lane {
    int jj, c, i, j, nv;
    template <bool EDGE, int V>
    static __device__ __forceinline__ Lane of(const KGrid &g, const TileInfo &ti) {
        Lane q;
        q.jj = V == 4 ? 2 * threadIdx.y + (threadIdx.x >> 4) : threadIdx.y;
        q.c = V == 4 ? 4 * (threadIdx.x & 15) : 2 * threadIdx.x;
        q.i = ti.i0 + q.c;
        q.j = ti.j0 + q.jj;
        q.nv = !EDGE ? V : (q.j > g.ny ? 0 : max(0, min(V, g.nx - q.i + 1)));
        return q;
    }
};

// CPML of the thread's cells (src/update_v_PML.c:177-226).  The strip rows are
// laid out so that a thread's group of cells is one aligned access
// (KGrid::psx, psy); cells of the group outside the strip have zero factors
// and keep their difference.  The memory values are loaded before the wait
// for the stage (Op::prefetch) and used after the differences.
//
// These loads may run before the preceding kernel has completed, in warps that
// never wait for it.  Their values were stored two launches back or earlier, and
// the launch between has waited for that one (griddepcontrol.wait, after which
// its stores are performed) before it let this one start, so they are in L2.
// They are read from there: a dependent launch may find lines of earlier
// launches in L1.  No line is read twice in a launch, so nothing is lost by it.
template <int V>
struct Psi {
    int at;  // index of the group in its strip (-1: in no strip)
    FV<V> v;
};
template <int V>
__device__ __forceinline__ void psi_x(const KGrid &g, const float *strip, const Lane &q, Psi<V> &s) {
    s.at = -1;
    if (g.boundary || g.fw == 0 || q.nv == 0) return;
    const bool right = q.i + V - 1 >= g.nx - g.fw + 1;
    if (q.i > g.fw && !right) return;
    s.at = (q.j - 1) * g.psx + (right ? q.i - 1 - g.psx_rs + g.psx_lw : q.i - 1);
    s.v = ldv_l2<V>(strip + s.at);
}
template <int V>
__device__ __forceinline__ void psi_y(const KGrid &g, const float *strip, const Lane &q, Psi<V> &s) {
    s.at = -1;
    const int hy = q.nv == 0 ? 0 : strip_y(g, q.j);
    if (!hy) return;
    s.at = (hy - 1) * g.psy + (q.i - 1);
    s.v = ldv_l2<V>(strip + s.at);
}
// cells lo..hi of the group lie in the strip
template <int V>
__device__ __forceinline__ void cpml_group(const KGrid &g, float *strip, Psi<V> &s, const FV<V> &b, const FV<V> &a,
                                           const FV<V> &K, int lo, int hi, float (&d)[V]) {
#pragma unroll
    for (int e = 0; e < V; e++) s.v.v[e] = b.v[e] * s.v.v[e] + a.v[e] * d[e];
    stv<V>(strip + s.at, s.v.v);
    if (g.k_one) {  // every K is 1: d/K is d
#pragma unroll
        for (int e = 0; e < V; e++) {
            const float t = d[e] + s.v.v[e];
            d[e] = e >= lo && e <= hi ? t : d[e];
        }
    } else {
#pragma unroll
        for (int e = 0; e < V; e++)
            if (e >= lo && e <= hi) d[e] = div_rn_pinned(d[e], K.v[e]) + s.v.v[e];
    }
}
// A group that meets both x strips (2 FW close to NX): its left cells one by
// one; its right cells are the group's own.
template <int V>
__device__ __noinline__ FV<V> cpml_left_cells(const KGrid &g, const KModel<float> &M, float *strip, Lane q, bool half,
                                              FV<V> d) {
#pragma unroll
    for (int e = 0; e < V; e++) {
        const int h = q.i + e;
        if (h <= g.fw && e < q.nv)
            d.v[e] = cpml(strip + (q.j - 1) * g.psx + (h - 1), prof(M, g, half ? B_XH : B_X, h),
                          prof(M, g, half ? A_XH : A_X, h), prof(M, g, half ? K_XH : K_X, h), d.v[e]);
    }
    return d;
}
// x strips; half: the profiles at half points
template <int V>
__device__ __forceinline__ void cpml_x(const KGrid &g, const KModel<float> &M, const ProfTab &pt, float *strip,
                                       Psi<V> &s, const Lane &q, bool half, float (&d)[V]) {
    if (s.at < 0) return;
    const bool left = q.i <= g.fw, right = q.i + V - 1 >= g.nx - g.fw + 1;
    const float *pr = pt.x + (half ? 3 * pt.xs : 0) + (pt.local ? s.at - (q.j - 1) * g.psx : q.i - 1);
    if (left && right) {
        FV<V> t;
#pragma unroll
        for (int e = 0; e < V; e++) t.v[e] = d[e];
        t = cpml_left_cells<V>(g, M, strip, q, half, t);
#pragma unroll
        for (int e = 0; e < V; e++) d[e] = t.v[e];
    }
    FV<V> K{};
    if (!g.k_one) K = ldv<V>(pr);
    cpml_group(g, strip, s, ldv<V>(pr + 2 * pt.xs), ldv<V>(pr + pt.xs), K, right ? g.nx - g.fw + 1 - q.i : 0,
               right ? q.nv - 1 : g.fw - q.i, d);
}
template <int V>
__device__ __forceinline__ void cpml_y(const KGrid &g, const ProfTab &pt, float *strip, Psi<V> &s, const Lane &q,
                                       bool half, float (&d)[V]) {
    if (s.at < 0) return;
    const int hy = strip_y(g, q.j);
    const float *pr = pt.y + (half ? 3 * pt.ys : 0) + hy;
    const float k = g.k_one ? 1.0f : pr[0], a = pr[pt.ys], b = pr[2 * pt.ys];
    cpml_group(g, strip, s, FV<V>::of(b), FV<V>::of(a), FV<V>::of(k), 0, V - 1, d);
}

// x / DH of a thread's values, rounded as the division: by the reciprocal when DH
// is a power of two, else by the reciprocal and two exact-remainder
// corrections (Markstein, IBM J. Res. Dev. 34, 1990: with the correctly
// rounded reciprocal, one correction of a quotient that is off by less than
// one ulp rounds correctly; the first correction makes it so).  Outside the
// range where the remainders are exact the division itself runs; a zero is
// its own quotient.
template <int V>
__device__ __forceinline__ void div_dh(const KGrid &g, float (&x)[V]) {
    if (g.dh_pow2) {
#pragma unroll
        for (int e = 0; e < V; e++) x[e] = x[e] * g.inv_dh;
        return;
    }
#pragma unroll
    for (int e = 0; e < V; e++) {
        const float a = x[e], m = fabsf(a);
        float q = a * g.inv_dh;
        q = __fmaf_rn(__fmaf_rn(-q, g.dh, a), g.inv_dh, q);
        q = __fmaf_rn(__fmaf_rn(-q, g.dh, a), g.inv_dh, q);
        if (!(m >= g.div_lo && m <= g.div_hi)) q = a == 0.0f ? a : div_rn_pinned(a, g.dh);
        x[e] = q;
    }
}

// Where a thread's cells go: the state of a slot and, on snapshot steps, the
// snapshot being stored.
template <bool EDGE, int V>
struct RowOut {
    float *st;  // state plane 0 at (j, i)
    int nv;
    __device__ __forceinline__ RowOut(const KGrid &g, const KState<float> &S, int slot, const Lane &q) {
        st = S.base + (long long)slot * S.slot_stride + ((q.j - 1 + HY) * g.pitch + (q.i - 1 + HX));
        nv = q.nv;
    }
    __device__ __forceinline__ void put(long long off, const float (&v)[V]) const {
        float *p = st + off;
        if (!EDGE || nv == V) {
            stv<V>(p, v);
        } else {
#pragma unroll
            for (int e = 0; e < V - 1; e++)
                if (e < nv) p[e] = v[e];
        }
    }
};

// Component comp of the snapshot being stored, at the thread's cells.  Every
// lane of the warp calls it: an fp16 segment is one tile row.
template <bool EDGE, int V>
__device__ __forceinline__ void snap(const KGrid &g, const KSnapOut &so, int slot, const Lane &q, int comp,
                                      const float (&v)[V]) {
    if (comp < 0) return;
    char *b = so.base + slot * so.slot_bytes;
    const long long at = comp * so.n + ((long long)(q.j - 1) * g.nx + (q.i - 1));
    if (!so.f16) {
        float *p = reinterpret_cast<float *>(b) + at;
        if (so.align >= V && q.nv == V) {
            stv<V>(p, v);
        } else if (V == 4 && so.align == 2 && q.nv == V) {
#pragma unroll
            for (int e = 0; e < V; e += 2) *reinterpret_cast<float2 *>(p + e) = make_float2(v[e], v[e + 1]);
        } else {
#pragma unroll
            for (int e = 0; e < V; e++)
                if (e < q.nv) p[e] = v[e];
        }
        return;
    }
    unsigned m = 0;
#pragma unroll
    for (int e = 0; e < V; e++)
        if (!EDGE || e < q.nv) m = max(m, __float_as_uint(v[e]) & 0x7fffffffu);
    if constexpr (V == 4) {
        const bool low = threadIdx.x < 16;
        const unsigned m0 = __reduce_max_sync(0xffffffffu, low ? m : 0u);
        const unsigned m1 = __reduce_max_sync(0xffffffffu, low ? 0u : m);
        m = low ? m0 : m1;
    } else {
        m = __reduce_max_sync(0xffffffffu, m);
    }
    float f, inv;
    seg_scales(__uint_as_float(m), f, inv);
    if (EDGE && q.nv == 0) return;
    __half *p = reinterpret_cast<__half *>(b) + at;
    if (so.align >= 2 && q.nv == V) {
        unsigned w[V / 2];
#pragma unroll
        for (int e = 0; e < V; e += 2) {
            const __half2 h2 = __floats2half2_rn(v[e] * f, v[e + 1] * f);
            w[e / 2] = *reinterpret_cast<const unsigned *>(&h2);
        }
        if (V == 4 && so.align == 4) {
            *reinterpret_cast<uint2 *>(p) = make_uint2(w[0], w[V / 2 - 1]);
        } else {
#pragma unroll
            for (int e = 0; e < V / 2; e++) reinterpret_cast<unsigned *>(p)[e] = w[e];
        }
    } else {
#pragma unroll
        for (int e = 0; e < V; e++)
            if (e < q.nv) p[e] = __float2half_rn(v[e] * f);
    }
    if (q.c == 0)
        reinterpret_cast<float *>(b + so.ex_off)[((long long)comp * g.ny + (q.j - 1)) * so.segs + (q.i - 1) / kSegCells] = inv;
}

// release a stage once every lane of the warp has read its part of it
__device__ __forceinline__ void release_stage(uint64_t *empty) {
    __syncwarp();
    if (threadIdx.x == 0) mbar_arrive(empty);
}

// The rarely taken rows (sources, free surface, receivers) are out of line
// and by value, so that they add nothing to the register budget of the main
// path.

// Explosive sources of step nt on row j, as src/psource.c:47-55 applies
// them after the stress update and before the free surface
// (src/IFOS2D.c:1758-1764): the lane holding a source cell adds half the
// source term to its sxx and syy, sources in list order (psource_apply).
struct SxxSyy {
    float xx[4], yy[4];
};
static __device__ __noinline__ SxxSyy psource_row(const KGrid &g, const KSrc &src, int slot, int nt, Lane q, SxxSyy v) {
    const float *pos = src.pos + (long long)slot * 8 * src.max_src;
    const int n = src.nsrc[slot];
    // the first source's place, type and term are requested with the count: one round trip for the usual single source
    const float x0 = pos[0], y0 = pos[src.max_src], type0 = pos[7 * src.max_src];
    const float amp0 = psource_amp(src, slot, 0, nt, g.dh);
    if (n <= 0 || (int)(n == 1 ? type0 : pos[7 * src.max_src + n - 1]) != 1) return v;  // psource_fires
    for (int l = 0; l < n; l++) {
        if ((int)(l ? pos[src.max_src + l] : y0) != q.j) continue;
        const int e = (int)(l ? pos[l] : x0) - q.i;
        if (e < 0 || e >= q.nv) continue;
        const float amp = l ? psource_amp(src, slot, l, nt, g.dh) : amp0;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (e == k) {
                v.xx[k] = (float)((double)v.xx[k] + 0.5 * (double)amp);
                v.yy[k] = (float)((double)v.yy[k] + 0.5 * (double)amp);
            }
    }
    return v;
}

// The free surface of row 1 on a stress op's results (surface_cell: the
// elastic src/surface_elastic_PML.c:53-104 and, with L memory variables, the
// viscoelastic src/surface_PML.c:60-157), from the zero-started differences
// of the staged velocities (vxx, vyy, formed before the stage was released):
// scaled by 1/DH, vxx with its own x CPML (psi_vxxs).  p and q are the p and q
// memory variables (LL each).
template <int LL, int V>
struct SurfVals {
    float xx[V], yy[V], vxx[V], vyy[V], p[LL > 0 ? LL : 1][V], q[LL > 0 ? LL : 1][V];
};
template <int LL, int V>
__device__ __noinline__ SurfVals<LL, V> surface_row(const KGrid &g, const KState<float> &S, const KModel<float> &M,
                                                 ProfTab pt, Lane c, int slot, int model, SurfVals<LL, V> r) {
    const float DT = g.dt, DH = g.dh;
    const float dh24 = (float)(1.0 / (double)DH), dthalbe = (float)((double)DT / 2.0);
    const float *srf = M.srf + (long long)model * M.srf_stride;
    float vx4[V];
#pragma unroll
    for (int e = 0; e < V; e++) vx4[e] = r.vxx[e] * dh24;
    // the surface has its x CPML also where the stress update has none (10/12)
    float *strip = S.psix[X_VXXS] + slot * S.psix_slot;
    Psi<V> ps;
    psi_x(g, strip, c, ps);
    cpml_x<V>(g, M, pt, strip, ps, c, false, vx4);
#pragma unroll
    for (int e = 0; e < V; e++) {
        if (e >= c.nv) continue;
        const int i = c.i + e;
        r.yy[e] = 0.0f;
#pragma unroll
        for (int l = 0; l < LL; l++) r.q[l][e] = 0.0f;
        const float vxx = vx4[e], vyy = r.vyy[e] * dh24;
        const float fjm = srf[i - 1], gg = srf[g.nx + i - 1];
        if (LL == 0) {
            r.xx[e] += -DT * ((gg * gg) / (gg + fjm) * vxx + gg * vyy);
            continue;
        }
        const float djm = srf[2 * g.nx + i - 1], ee = srf[3 * g.nx + i - 1];
        float sump = 0;
#pragma unroll
        for (int l = 0; l < LL; l++) sump += r.p[l][e];
        r.xx[e] += -(DT * (gg - fjm) * (gg - fjm) * vxx / gg) - (DT * (gg - fjm) * vyy) - (dthalbe * sump);
        sump = 0;
#pragma unroll
        for (int l = 0; l < LL; l++) {
            const float bjm = g.bjm_srf[l + 1];
            r.p[l][e] = (float)((double)r.p[l][e] + (double)bjm * (((double)(djm - ee) * ((double)(fjm / gg) - 1.0) *
                                                                    (double)vxx) - (double)((djm - ee) * vyy)));
            sump += r.p[l][e];
        }
        r.xx[e] += (dthalbe * sump);
    }
    return r;
}

// The receivers of the thread's cells in row j on the new vx, vy before they
// are stored: mode 1 copies them into the seismograms of step nt, as
// src/seismo_ssg.c:26-140 samples vx, vy after the step (SEISMO 1); mode 2
// adds the adjoint sources of step nt, as src/update_v_PML.c:567-578 does
// after the velocity update (ADJOINT_TYPE 1: both components, 2: vy, 3: vx).
// The slot's cell map gives each cell its receiver (-1: none).
struct RecIdx {
    int l[4];
};
__device__ __forceinline__ RecIdx rec_lookup(const KGrid &g, const KRec &rec, bool one_row, int slot, const Lane &q) {
    RecIdx r{{-1, -1, -1, -1}};
    const int *m = rec.map + (long long)slot * rec.map_stride;
    // with one receiver row its index is 0 and the row table need not be read
    const int rr = q.nv <= 0 ? -1 : (one_row ? 0 : m[q.j - 1]);
    if (rr < 0) return r;
    const int *cells = m + g.ny + (long long)rr * g.nx + (q.i - 1);
#pragma unroll
    for (int e = 0; e < 4; e++)
        if (e < q.nv) r.l[e] = cells[e];
    return r;
}
static __device__ __noinline__ SxxSyy rec_row(const KGrid &g, const KRec &rec, int mode, int slot, int nt, RecIdx r,
                                              SxxSyy v) {
    const long long cs = (long long)rec.max_rec * g.nt_total;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const int l = r.l[e];
        if (l < 0) continue;
        const long long o = (long long)l * g.nt_total + nt - 1;
        if (mode == 2) {
            const float *adj = rec.adj + (long long)slot * 3 * cs + o;
            const int at = g.adjoint_type;
            if (at == 1 || at == 3) v.xx[e] += adj[0];
            if (at == 1 || at == 2) v.yy[e] += adj[cs];
        } else {
            float *sec = rec.sec + (long long)slot * 6 * cs + o;
            sec[0] = v.xx[e];
            sec[cs] = v.yy[e];
        }
    }
    return v;
}

// One value per cell: the SH velocity (plane 2 of the seismograms) and the
// acoustic pressure (plane 3, -p); both take component 2 of the adjoint
// sources (src/seismo_ssg.c, src/update_v_PML_SH.c, src/psource.c:61-74).
struct Cells4 {
    float v[4];
};
template <bool PRESSURE>
__device__ __noinline__ Cells4 rec_row1(const KGrid &g, const KRec &rec, int mode, int slot, int nt, RecIdx r, Cells4 v) {
    const long long cs = (long long)rec.max_rec * g.nt_total;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        if (r.l[e] < 0) continue;
        const long long o = (long long)r.l[e] * g.nt_total + nt - 1;
        if (mode == 2) v.v[e] += rec.adj[(long long)slot * 3 * cs + 2 * cs + o];
        else rec.sec[(long long)slot * 6 * cs + (PRESSURE ? 3 : 2) * cs + o] = PRESSURE ? -v.v[e] : v.v[e];
    }
    return v;
}
__device__ __forceinline__ bool any_receiver(const RecIdx &r) {
    return max(max(r.l[0], r.l[1]), max(r.l[2], r.l[3])) >= 0;
}

// Explosive sources on the acoustic pressure (psource_apply), in list order.
static __device__ __noinline__ Cells4 psource_row_p(const KGrid &g, const KSrc &src, int slot, int nt, Lane q, Cells4 v) {
    const float *pos = src.pos + (long long)slot * 8 * src.max_src;
    const int n = src.nsrc[slot];
    const float x0 = pos[0], y0 = pos[src.max_src], type0 = pos[7 * src.max_src];  // requested with the count
    const float amp0 = psource_amp(src, slot, 0, nt, g.dh);
    if (n <= 0 || (int)(n == 1 ? type0 : pos[7 * src.max_src + n - 1]) != 1) return v;  // psource_fires
    for (int l = 0; l < n; l++) {
        const int e = (int)(l ? pos[l] : x0) - q.i;
        if ((int)(l ? pos[src.max_src + l] : y0) != q.j || e < 0 || e >= q.nv) continue;
        const float amp = l ? psource_amp(src, slot, l, nt, g.dh) : amp0;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (e == k) v.v[k] += amp;
    }
    return v;
}
// Force sources on the SH velocity, as src/update_v_PML_SH.c:327-333 adds
// them after the update, in list order; rjp: the cells' reciprocal densities.
static __device__ __noinline__ Cells4 force_row_sh(const KGrid &g, const KSrc &src, int slot, int nt, Lane q, Cells4 rjp,
                                                   Cells4 v) {
    const float *pos = src.pos + (long long)slot * 8 * src.max_src;
    const float *sig = src.sig + (long long)slot * src.max_src * src.nt_total + nt - 1;
    const int n = src.nsrc[slot];
    const float x0 = pos[0], y0 = pos[src.max_src], a0 = sig[0];  // requested with the count
    const float DT = g.dt, DH = g.dh;
    for (int l = 0; l < n; l++) {
        const int e = (int)(l ? pos[l] : x0) - q.i;
        if ((int)(l ? pos[src.max_src + l] : y0) != q.j || e < 0 || e >= q.nv) continue;
        const float a = l ? sig[(long long)l * src.nt_total] : a0;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (e == k)
                v.v[k] = (float)((double)v.v[k] + ((double)(rjp.v[k] * DT) * 1.0 * (double)a) / (double)(DH * DH));
    }
    return v;
}

// rows<true> runs on warps whose rows of the tile need anything beyond the
// plain update (TileInfo::edge), rows<false> on the others.  prefetch starts
// the loads of the CPML memories that rows<true> uses (Pre); they are written
// by the op's own previous launch only, which has completed before this one
// starts.
// the common members of an op
// nt: the time step.  What the ops do beside the update, so that a step needs
// no other kernel:
// fps: the stress and pressure ops apply the explosive sources of step nt,
// fsurf: and the free surface of row 1;
// fvs: the SH velocity op applies the force sources (rows src_j0..src_j1 hold
// every slot's sources);
// rec_mode 1: the op copies its new values at the receivers into the
// seismograms (P-SV and acoustic velocity: vx, vy; SH velocity: vz; pressure:
// -p), 2: it adds the adjoint sources there (rows rec_j0..rec_j1 hold every
// slot's receivers);
// probe: the velocity op checks the centre cell for NaN.
#define IFOS_OP_MEMBERS \
    KGrid g;            \
    KState<float> S;    \
    KModel<float> M;    \
    KTma tm;            \
    KSnapOut so;        \
    KSrc src;           \
    int nt;             \
    int fsurf;          \
    int fps;            \
    int fvs;            \
    int probe;          \
    int src_j0, src_j1; \
    KRec rec;           \
    int rec_mode;       \
    int rec_j0, rec_j1; \
    int *bad;

// ---------------------------------------------------------------------------
// stress, P-SV viscoelastic with LL SLS (src/update_s_visc_PML.c; the
// reference 10/12 default :615-660 has no CPML and zero-started sums: QUIRK)
// halo: vx vy; plain: sxx syy sxy, r[LL] p[LL] q[LL], fipjp f g mu pi muipjp;
// writes sxx syy sxy r p q.  Non-uniform tau planes are read from HBM.
// DIRECT: the model's coefficients are loaded into registers before the wait
// for the stage instead of through the ring, whose stages shrink (L 3: from 46
// to 34 KB, three instead of two).
template <int FDOH, int TY, int LL, int NST, bool QUIRK, bool DIRECT>
struct OpSVisc {
    static constexpr int V = kCellsVisc;
    static constexpr bool EARLY = DIRECT;
    static constexpr int DEP_TILES = INT_MAX;
    static constexpr int NH_ = 2, NP_ = 3 + 3 * LL + (DIRECT ? 0 : 6);
    static constexpr bool CPML = !QUIRK, MIRROR = false;
    using P = Pipe<FDOH, TY, NH_, NP_, NST, visc_blocks(LL), V>;
    IFOS_OP_MEMBERS
    // boxes of consecutive planes: their number, planes of box k, whether they are model planes
    static constexpr int NG = DIRECT ? 2 : 3;
    __host__ __device__ static constexpr int gd(int k) { return k == 0 ? 3 : (k == 1 ? 3 * LL : 6); }
    __host__ __device__ static constexpr bool gm(int k) { return k == 2; }
    void planes(int &hz, int (&gz)[NG]) const {  // first planes of the boxes, in slot 0 and model 0
        hz = tm.pid[P_VX];
        gz[0] = tm.pid[P_SXX];
        gz[1] = tm.mem_pid[MEM_R];
        if (!DIRECT) gz[2 % NG] = tm.mid[M_FIPJPV];
    }
    // DIRECT: fipjp f g mu pi muipjp of the thread's cells, loaded before the wait
    struct Pre {
        FV<V> c[DIRECT ? 6 : 1];
        Psi<V> x0, x1, y0, y1;
    };
    template <bool EDGE>
    __device__ __forceinline__ void early(const TileInfo &ti, Pre &pre) const {
        const Lane q = Lane::of<EDGE, V>(g, ti);
        const float *p = M.m[M_FIPJPV] + (long long)ti.model() * M.model_stride + (q.j - 1 + HY) * g.pitch + (q.i - 1 + HX);
#pragma unroll
        for (int k = 0; k < 6; k++) pre.c[k] = !EDGE || q.nv > 0 ? ldv<V>(p + k * g.plane) : FV<V>::of(0.0f);
    }
    __device__ __forceinline__ void prefetch(const TileInfo &ti, Pre &pre) const {
        if (!CPML) return;
        const Lane q = Lane::of<true, V>(g, ti);
        psi_x<V>(g, S.psix[X_VXX] + ti.slot * S.psix_slot, q, pre.x0);
        psi_x<V>(g, S.psix[X_VYX] + ti.slot * S.psix_slot, q, pre.x1);
        psi_y<V>(g, S.psiy[Y_VYY] + ti.slot * S.psiy_slot, q, pre.y0);
        psi_y<V>(g, S.psiy[Y_VXY] + ti.slot * S.psiy_slot, q, pre.y1);
    }
    template <bool EDGE>
    __device__ __forceinline__ void rows(const TileInfo &ti, Pre &pre, const ProfTab &pt, const float *h,
                                         const float *pl, uint64_t *empty) const {
        const Lane q = Lane::of<EDGE, V>(g, ti);
        const float *t_vx = h, *t_vy = h + P::BOXS;
        const int c0 = P::XH + q.c;
        const Hc<FDOH> hc(g);
        const float DT = g.dt, DH = g.dh;
        const float dhi = (float)(1.0 / (double)DH), dthalbe = (float)((double)DT / 2.0);
        const int slot = ti.slot;
        const bool surf = EDGE && fsurf && q.j == 1;
        float vxx[V], vyx[V], vxy[V], vyy[V], sx[V], sy[V];  // sx, sy: the surface's zero-started differences
        {
            XWin<FDOH, V> w;
            w.load(t_vx + (q.jj + P::H) * P::BW, c0);
#pragma unroll
            for (int e = 0; e < V; e++) vxx[e] = xbwd<QUIRK>(hc, w, e) * dhi;
            if (surf) {
#pragma unroll
                for (int e = 0; e < V; e++) sx[e] = xbwd<true>(hc, w, e);
            }
            w.load(t_vy + (q.jj + P::H) * P::BW, c0);
#pragma unroll
            for (int e = 0; e < V; e++) vyx[e] = xfwd<QUIRK>(hc, w, e) * dhi;
        }
        ydiff<true, false, false, P, QUIRK>(hc, t_vx, q.jj, c0, vxy);
        ydiff<false, false, false, P, QUIRK>(hc, t_vy, q.jj, c0, vyy);
        if (surf) ydiff<false, false, false, P, true>(hc, t_vy, q.jj, c0, sy);
#pragma unroll
        for (int e = 0; e < V; e++) vxy[e] *= dhi, vyy[e] *= dhi;
        if (EDGE && CPML) {
            cpml_x<V>(g, M, pt, S.psix[X_VXX] + slot * S.psix_slot, pre.x0, q, false, vxx);
            cpml_x<V>(g, M, pt, S.psix[X_VYX] + slot * S.psix_slot, pre.x1, q, true, vyx);
            cpml_y<V>(g, pt, S.psiy[Y_VYY] + slot * S.psiy_slot, pre.y0, q, false, vyy);
            cpml_y<V>(g, pt, S.psiy[Y_VXY] + slot * S.psiy_slot, pre.y1, q, true, vxy);
        }
        const float *in = pl + q.jj * kTileX + q.c;
        auto ld = [&](int k) { return ldv<V>(in + k * P::PLS); };
        const FV<V> s0 = ld(0), s1 = ld(1), s2 = ld(2);
        FV<V> co[6];
#pragma unroll
        for (int k = 0; k < 6; k++) co[k] = DIRECT ? pre.c[DIRECT ? k : 0] : ld(3 + 3 * LL + k);
        const FV<V> &fipjp = co[0], &f = co[1], &gg = co[2], &mu = co[3], &pi = co[4], &muij = co[5];
        FV<V> mr[LL], mp[LL], mq[LL];
#pragma unroll
        for (int l = 0; l < LL; l++) mr[l] = ld(3 + l), mp[l] = ld(3 + LL + l), mq[l] = ld(3 + 2 * LL + l);
        release_stage(empty);
        const RowOut<EDGE, V> out(g, S, slot, q);
        float div[V], shear[V], o[3][V], sumr[V], sump[V], sumq[V];
#pragma unroll
        for (int e = 0; e < V; e++) {
            div[e] = vxx[e] + vyy[e], shear[e] = vxy[e] + vyx[e];
            sumr[e] = sump[e] = sumq[e] = 0;
#pragma unroll
            for (int l = 0; l < LL; l++) {
                sumr[e] += mr[l].v[e];
                sump[e] += mp[l].v[e];
                sumq[e] += mq[l].v[e];
            }
            const D gd = (D)(gg.v[e] * div[e]), f2 = (D)2 * (D)f.v[e];
            o[2][e] = s2.v[e] + ((fipjp.v[e] * shear[e]) + (dthalbe * sumr[e]));
            o[0][e] = (float)((D)s0.v[e] + (gd - f2 * (D)vyy[e] + (D)(dthalbe * sump[e])));
            o[1][e] = (float)((D)s1.v[e] + (gd - f2 * (D)vxx[e] + (D)(dthalbe * sumq[e])));
            sumr[e] = sump[e] = sumq[e] = 0;
        }
        FV<V> ts = FV<V>::of(g.taus0), tp = FV<V>::of(g.taup0), tsij = FV<V>::of(g.tausipjp0);
        if (M.m[M_TAUS]) {  // the three tau planes are present together; pad cells read what is there
            const long long at = (long long)ti.model() * M.model_stride + (min(q.j, g.ny) - 1 + HY) * g.pitch +
                                 (q.nv ? q.i - 1 + HX : 0);
            ts = ldv<V>(M.m[M_TAUS] + at);
            tp = ldv<V>(M.m[M_TAUP] + at);
            tsij = ldv<V>(M.m[M_TAUSIPJP] + at);
        }
#pragma unroll
        for (int l = 0; l < LL; l++) {
            const float eta = g.eta[l + 1];
#pragma unroll
            for (int e = 0; e < V; e++) {
                // dip, d, e of src/prepare_update_s.c:57-59, formed in the same order
                const float dip = muij.v[e] * eta * tsij.v[e], dd = mu.v[e] * eta * ts.v[e], ee = pi.v[e] * eta * tp.v[e];
                const D d2 = (D)2 * (D)dd;
                mr[l].v[e] = g.bip[l + 1] * (mr[l].v[e] * g.cip[l + 1] - (dip * shear[e]));
                mp[l].v[e] = (float)((D)g.bjm[l + 1] * ((D)(mp[l].v[e] * g.cjm[l + 1] - (ee * div[e])) + (d2 * (D)vyy[e])));
                mq[l].v[e] = (float)((D)g.bjm[l + 1] * ((D)(mq[l].v[e] * g.cjm[l + 1] - (ee * div[e])) + (d2 * (D)vxx[e])));
                sumr[e] += mr[l].v[e];
                sump[e] += mp[l].v[e];
                sumq[e] += mq[l].v[e];
            }
            out.put(S.mem_off[MEM_R] + l * g.plane, mr[l].v);
            out.put(S.mem_off[MEM_P] + l * g.plane, mp[l].v);
            out.put(S.mem_off[MEM_Q] + l * g.plane, mq[l].v);
        }
#pragma unroll
        for (int e = 0; e < V; e++) {
            o[0][e] = o[0][e] + (dthalbe * sump[e]);
            o[1][e] = o[1][e] + (dthalbe * sumq[e]);
            o[2][e] = o[2][e] + (dthalbe * sumr[e]);
        }
        if (EDGE) {
            if (fps && q.j >= src_j0 && q.j <= src_j1) {
                SxxSyy v{};
#pragma unroll
                for (int e = 0; e < V; e++) v.xx[e] = o[0][e], v.yy[e] = o[1][e];
                v = psource_row(g, src, slot, nt, q, v);
#pragma unroll
                for (int e = 0; e < V; e++) o[0][e] = v.xx[e], o[1][e] = v.yy[e];
            }
            if (surf) {  // changes the thread's own p and q of row 1, stored above
                SurfVals<LL, V> r;
#pragma unroll
                for (int e = 0; e < V; e++) r.xx[e] = o[0][e], r.yy[e] = o[1][e], r.vxx[e] = sx[e], r.vyy[e] = sy[e];
#pragma unroll
                for (int l = 0; l < LL; l++)
#pragma unroll
                    for (int e = 0; e < V; e++) {
                        r.p[l][e] = e < q.nv ? out.st[S.mem_off[MEM_P] + l * g.plane + e] : 0.0f;
                        r.q[l][e] = 0.0f;
                    }
                r = surface_row<LL, V>(g, S, M, pt, q, slot, ti.model(), r);
#pragma unroll
                for (int e = 0; e < V; e++) o[0][e] = r.xx[e], o[1][e] = r.yy[e];
#pragma unroll
                for (int l = 0; l < LL; l++) {
                    out.put(S.mem_off[MEM_P] + l * g.plane, r.p[l]);
                    out.put(S.mem_off[MEM_Q] + l * g.plane, r.q[l]);
                }
            }
        }
        out.put(S.off[P_SXX], o[0]);
        out.put(S.off[P_SYY], o[1]);
        out.put(S.off[P_SXY], o[2]);
        if (so.base) {
            snap<EDGE, V>(g, so, slot, q, tm.snap_comp[P_SXX], o[0]);
            snap<EDGE, V>(g, so, slot, q, tm.snap_comp[P_SYY], o[1]);
            snap<EDGE, V>(g, so, slot, q, tm.snap_comp[P_SXY], o[2]);
        }
    }
};

// stress, P-SV elastic (src/update_s_elastic_PML.c:151-241; 10/12: :442-535)
// halo: vx vy; plain: sxx syy sxy uipjp f g (reference 10/12 branch: uipjp vs vp);
// writes sxx syy sxy
// SMALL: see Launcher::small
template <int FDOH, int TY, int NST, bool QUIRK, bool SMALL = false>
struct OpSEl {
    static constexpr int V = SMALL ? 2 : kCells;
    static constexpr bool EARLY = false;
    static constexpr int DEP_TILES = FDOH <= 2 ? kDepTiles : INT_MAX;
    static constexpr int NH_ = 2, NP_ = 6;
    static constexpr bool CPML = !QUIRK, MIRROR = false;
    using P = Pipe<FDOH, TY, NH_, NP_, NST, SMALL ? 2 : sblocks(FDOH), V>;
    IFOS_OP_MEMBERS
    // boxes of consecutive planes: their number, planes of box k, whether they are model planes
    static constexpr int NG = QUIRK ? 4 : 2;
    __host__ __device__ static constexpr int gd(int k) { return k == 0 || !QUIRK ? 3 : 1; }
    __host__ __device__ static constexpr bool gm(int k) { return k > 0; }
    void planes(int &hz, int (&gz)[NG]) const {  // first planes of the boxes, in slot 0 and model 0
        hz = tm.pid[P_VX];
        gz[0] = tm.pid[P_SXX];
        gz[1] = tm.mid[M_UIPJP];
        if (QUIRK) gz[2 % NG] = tm.mid[M_VS], gz[3 % NG] = tm.mid[M_VP];
    }
    struct Pre {
        Psi<V> x0, x1, y0, y1;
    };
    __device__ __forceinline__ void prefetch(const TileInfo &ti, Pre &pre) const {
        if (!CPML) return;
        const Lane q = Lane::of<true, V>(g, ti);
        psi_x<V>(g, S.psix[X_VXX] + ti.slot * S.psix_slot, q, pre.x0);
        psi_x<V>(g, S.psix[X_VYX] + ti.slot * S.psix_slot, q, pre.x1);
        psi_y<V>(g, S.psiy[Y_VYY] + ti.slot * S.psiy_slot, q, pre.y0);
        psi_y<V>(g, S.psiy[Y_VXY] + ti.slot * S.psiy_slot, q, pre.y1);
    }
    template <bool EDGE>
    __device__ __forceinline__ void rows(const TileInfo &ti, Pre &pre, const ProfTab &pt, const float *h,
                                         const float *pl, uint64_t *empty) const {
        const Lane q = Lane::of<EDGE, V>(g, ti);
        const float *t_vx = h, *t_vy = h + P::BOXS;
        const int c0 = P::XH + q.c;
        const Hc<FDOH> hc(g);
        const float DT = g.dt, DH = g.dh;
        const float dhi = DT / DH;
        const int slot = ti.slot;
        const bool surf = EDGE && fsurf && q.j == 1;
        float vxx[V], vyx[V], vxy[V], vyy[V], sx[V], sy[V];  // sx, sy: the surface's zero-started differences
        {
            XWin<FDOH, V> w;
            w.load(t_vx + (q.jj + P::H) * P::BW, c0);
#pragma unroll
            for (int e = 0; e < V; e++) vxx[e] = xbwd(hc, w, e) * dhi;
            if (surf) {
#pragma unroll
                for (int e = 0; e < V; e++) sx[e] = xbwd<true>(hc, w, e);
            }
            w.load(t_vy + (q.jj + P::H) * P::BW, c0);
#pragma unroll
            for (int e = 0; e < V; e++) vyx[e] = xfwd(hc, w, e) * dhi;
        }
        ydiff<true, false, false, P>(hc, t_vx, q.jj, c0, vxy);
        ydiff<false, false, false, P>(hc, t_vy, q.jj, c0, vyy);
        if (surf) ydiff<false, false, false, P, true>(hc, t_vy, q.jj, c0, sy);
        const float *in = pl + q.jj * kTileX + q.c;
        auto ld = [&](int k) { return ldv<V>(in + k * P::PLS); };
        const FV<V> sxx0 = ld(0), syy0 = ld(1), sxy0 = ld(2), fipjp = ld(3), f = ld(4), gg = ld(5);
        release_stage(empty);
#pragma unroll
        for (int e = 0; e < V; e++) vxy[e] *= dhi, vyy[e] *= dhi;
        float o[3][V];
        if (QUIRK) {
#pragma unroll
            for (int e = 0; e < V; e++) {
                const float fi = fipjp.v[e] * DT, ff = f.v[e] * DT, gd = gg.v[e] * DT;
                o[2][e] = sxy0.v[e] + (fi * (vxy[e] + vyx[e]));
                o[0][e] = (float)((D)sxx0.v[e] + ((D)(gd * (vxx[e] + vyy[e])) - ((D)2 * (D)ff * (D)vyy[e])));
                o[1][e] = (float)((D)syy0.v[e] + ((D)(gd * (vxx[e] + vyy[e])) - ((D)2 * (D)ff * (D)vxx[e])));
            }
        } else {
            if (EDGE) {
                cpml_x<V>(g, M, pt, S.psix[X_VXX] + slot * S.psix_slot, pre.x0, q, false, vxx);
                cpml_x<V>(g, M, pt, S.psix[X_VYX] + slot * S.psix_slot, pre.x1, q, true, vyx);
                cpml_y<V>(g, pt, S.psiy[Y_VYY] + slot * S.psiy_slot, pre.y0, q, false, vyy);
                cpml_y<V>(g, pt, S.psiy[Y_VXY] + slot * S.psiy_slot, pre.y1, q, true, vxy);
            }
#pragma unroll
            for (int e = 0; e < V; e++) {
                o[2][e] = sxy0.v[e] + fipjp.v[e] * (vyx[e] + vxy[e]);
                o[0][e] = (float)((D)sxx0.v[e] + ((D)(gg.v[e] * (vxx[e] + vyy[e])) + ((D)2 * (D)f.v[e] * (D)vxx[e])));
                o[1][e] = (float)((D)syy0.v[e] + ((D)(gg.v[e] * (vxx[e] + vyy[e])) + ((D)2 * (D)f.v[e] * (D)vyy[e])));
            }
        }
        if (EDGE) {
            if (fps && q.j >= src_j0 && q.j <= src_j1) {
                SxxSyy v{};
#pragma unroll
                for (int e = 0; e < V; e++) v.xx[e] = o[0][e], v.yy[e] = o[1][e];
                v = psource_row(g, src, slot, nt, q, v);
#pragma unroll
                for (int e = 0; e < V; e++) o[0][e] = v.xx[e], o[1][e] = v.yy[e];
            }
            if (surf) {
                SurfVals<0, V> r;
#pragma unroll
                for (int e = 0; e < V; e++)
                    r.xx[e] = o[0][e], r.yy[e] = o[1][e], r.vxx[e] = sx[e], r.vyy[e] = sy[e], r.p[0][e] = r.q[0][e] = 0.0f;
                r = surface_row<0, V>(g, S, M, pt, q, slot, ti.model(), r);
#pragma unroll
                for (int e = 0; e < V; e++) o[0][e] = r.xx[e], o[1][e] = r.yy[e];
            }
        }
        const RowOut<EDGE, V> out(g, S, slot, q);
        out.put(S.off[P_SXX], o[0]);
        out.put(S.off[P_SYY], o[1]);
        out.put(S.off[P_SXY], o[2]);
        if (so.base) {
            snap<EDGE, V>(g, so, slot, q, tm.snap_comp[P_SXX], o[0]);
            snap<EDGE, V>(g, so, slot, q, tm.snap_comp[P_SYY], o[1]);
            snap<EDGE, V>(g, so, slot, q, tm.snap_comp[P_SXY], o[2]);
        }
    }
};

// ---------------------------------------------------------------------------
// velocity, P-SV (src/update_v_PML.c:161-252; 10/12 reference branches
// :466-528 when QUIRK) and acoustic (src/update_v_acoustic_PML.c:72-148,
// default :396-409 when QUIRK; AC).  halo: sxx syy sxy (acoustic: sp);
// plain: vx vy rip rjp [+ vxp1 vyp1 in the adjoint].  SW: 0 forward,
// 1 adjoint; P1: this forward step forms vxp1/vyp1 for a snapshot (written to
// the snapshot when the launch stores one, else to the state).
template <int FDOH, int TY, int NST, bool QUIRK, int SW, bool P1, bool AC, bool SMALL = false>
struct OpVPsv {
    static constexpr int V = SMALL ? 2 : cells_v(FDOH);
    static constexpr bool EARLY = false;
    static constexpr int DEP_TILES = FDOH <= 2 && !AC ? kDepTiles : INT_MAX;
    static constexpr int NH_ = AC ? 1 : 3;
    static constexpr int NP_ = (SW == 1 && !QUIRK) ? 6 : 4;
    static constexpr bool CPML = !QUIRK, MIRROR = true;
    using P = Pipe<FDOH, TY, NH_, NP_, NST, SMALL ? 2 : vblocks(FDOH), V>;
    IFOS_OP_MEMBERS
    // boxes of consecutive planes: their number, planes of box k, whether they are model planes
    static constexpr int NG = NP_ / 2;
    __host__ __device__ static constexpr int gd(int k) { return 2 + 0 * k; }
    __host__ __device__ static constexpr bool gm(int k) { return k == 1; }
    void planes(int &hz, int (&gz)[NG]) const {  // first planes of the boxes, in slot 0 and model 0
        hz = tm.pid[AC ? P_SP : P_SXX];
        gz[0] = tm.pid[P_VX];
        gz[1] = tm.mid[M_RIP];
        if (NG > 2) gz[2 % NG] = tm.pid[P_VXP1];
    }
    struct Pre {
        Psi<V> x0, x1, y0, y1;
        RecIdx rec;
    };
    __device__ __forceinline__ void prefetch(const TileInfo &ti, Pre &pre) const {
        const Lane q = Lane::of<true, V>(g, ti);
        if (rec_mode && q.j >= rec_j0 && q.j <= rec_j1) pre.rec = rec_lookup(g, rec, rec_j0 == rec_j1, ti.slot, q);
        else pre.rec = RecIdx{{-1, -1, -1, -1}};
        if (!CPML) return;
        psi_x<V>(g, S.psix[X_SXX] + ti.slot * S.psix_slot, q, pre.x0);
        if (!AC) psi_x<V>(g, S.psix[X_SXY] + ti.slot * S.psix_slot, q, pre.x1);
        psi_y<V>(g, S.psiy[Y_SYY] + ti.slot * S.psiy_slot, q, pre.y0);
        if (!AC) psi_y<V>(g, S.psiy[Y_SXY] + ti.slot * S.psiy_slot, q, pre.y1);
    }
    template <bool EDGE>
    __device__ __forceinline__ void rows(const TileInfo &ti, Pre &pre, const ProfTab &pt, const float *h,
                                         const float *pl, uint64_t *empty) const {
        const Lane q = Lane::of<EDGE, V>(g, ti);
        // P-SV: sxx, syy, sxy boxes; acoustic: the sp box serves as all three
        const float *t_sxx = h, *t_syy = AC ? h : h + P::BOXS, *t_sxy = AC ? h : h + 2 * P::BOXS;
        const int c0 = P::XH + q.c, slot = ti.slot;
        const Hc<FDOH> hc(g);
        const bool mir = EDGE && g.free_surf && ti.j0 == 1;
        // P-SV: sxx_x, syy_y, sxy_x, sxy_y; acoustic: sp_x, sp_y
        float a_x[V], a_y[V], b_x[V], b_y[V];
        {
            XWin<FDOH, V> w;
            w.load(t_sxx + (q.jj + P::H) * P::BW, c0);
#pragma unroll
            for (int e = 0; e < V; e++) a_x[e] = xfwd<QUIRK && AC>(hc, w, e);
        }
        ydiff_fs<true, EDGE, false, P, QUIRK && AC>(hc, t_syy, q.jj, c0, mir, a_y);
        if (!AC) {
            XWin<FDOH, V> w;
            w.load(t_sxy + (q.jj + P::H) * P::BW, c0);
            if (!QUIRK) {
#pragma unroll
                for (int e = 0; e < V; e++) b_x[e] = xbwd(hc, w, e);
                ydiff_fs<false, EDGE, true, P>(hc, t_sxy, q.jj, c0, mir, b_y);
            } else {
                // one written-out sum per component (src/update_v_PML.c:469-490)
#pragma unroll
                for (int m = 1; m <= FDOH; m++) {
                    const FV<V> a = EDGE && mir ? ldy<true, true, P, V>(t_sxy, q.jj, c0, m - 1)
                                             : ldy<false, true, P, V>(t_sxy, q.jj, c0, m - 1);
                    const FV<V> b = EDGE && mir ? ldy<true, true, P, V>(t_sxy, q.jj, c0, -m)
                                             : ldy<false, true, P, V>(t_sxy, q.jj, c0, -m);
#pragma unroll
                    for (int e = 0; e < V; e++) {
                        a_x[e] += hc.w[m] * (a.v[e] - b.v[e]);
                        a_y[e] += hc.w[m] * (w.v[XWin<FDOH, V>::XB + e + m - 1] - w.v[XWin<FDOH, V>::XB + e - m]);
                    }
                }
            }
        }
        const float *in = pl + q.jj * kTileX + q.c;
        auto ld = [&](int k) { return ldv<V>(in + k * P::PLS); };
        const FV<V> vxo = ld(0), vyo = ld(1), rip = ld(2), rjp = ld(3);
        FV<V> px{}, py{};
        if (NP_ > 4) px = ld(4 % NP_), py = ld(5 % NP_);
        release_stage(empty);
        const float DT = g.dt, DH = g.dh;
        float o[4][V];
        if (QUIRK) {
            const float dtdh = DT * DT / DH;
#pragma unroll
            for (int e = 0; e < V; e++) {
                o[0][e] = vxo.v[e] + a_x[e] * dtdh * rip.v[e];
                o[1][e] = vyo.v[e] + a_y[e] * dtdh * rjp.v[e];
            }
        } else {
            if (EDGE) {
                cpml_x<V>(g, M, pt, S.psix[X_SXX] + slot * S.psix_slot, pre.x0, q, true, a_x);
                cpml_y<V>(g, pt, S.psiy[Y_SYY] + slot * S.psiy_slot, pre.y0, q, true, a_y);
                if (!AC) {
                    cpml_x<V>(g, M, pt, S.psix[X_SXY] + slot * S.psix_slot, pre.x1, q, false, b_x);
                    cpml_y<V>(g, pt, S.psiy[Y_SXY] + slot * S.psiy_slot, pre.y1, q, false, b_y);
                }
            }
            float fx[V], fy[V];
#pragma unroll
            for (int e = 0; e < V; e++) {
                // P-SV: x force sxx_x + sxy_y, y force sxy_x + syy_y; acoustic: sp_x, sp_y
                const float x = AC ? (a_x[e]) : (a_x[e] + b_y[e]), y = AC ? (a_y[e]) : (b_x[e] + a_y[e]);
                if (SW == 0) {
                    if (P1) {
                        o[2][e] = rip.v[e] * x;
                        o[3][e] = rjp.v[e] * y;
                    }
                } else {
                    o[2][e] = px.v[e] + vxo.v[e] * DT;
                    o[3][e] = py.v[e] + vyo.v[e] * DT;
                }
                fx[e] = DT * rip.v[e] * x;
                fy[e] = DT * rjp.v[e] * y;
            }
            if (SW == 0 && P1) {
                div_dh(g, o[2]);
                div_dh(g, o[3]);
            }
            div_dh(g, fx);
            div_dh(g, fy);
#pragma unroll
            for (int e = 0; e < V; e++) {
                o[0][e] = vxo.v[e] + fx[e];
                o[1][e] = vyo.v[e] + fy[e];
            }
        }
        if (EDGE && q.nv > 0) {
            if (any_receiver(pre.rec)) {
                SxxSyy v{};
#pragma unroll
                for (int e = 0; e < V; e++) v.xx[e] = o[0][e], v.yy[e] = o[1][e];
                v = rec_row(g, rec, rec_mode, slot, nt, pre.rec, v);
#pragma unroll
                for (int e = 0; e < V; e++) o[0][e] = v.xx[e], o[1][e] = v.yy[e];
            }
            if (probe && q.j == g.ny / 2) {  // the instability probe of the driver (src/IFOS2D.c:1660-1672)
                const int at = g.nx / 2 - q.i;
#pragma unroll
                for (int e = 0; e < V; e++)
                    if (e == at && e < q.nv && isnan(o[1][e])) atomicExch(bad, 1);
            }
        }
        const RowOut<EDGE, V> out(g, S, slot, q);
        out.put(S.off[P_VX], o[0]);
        out.put(S.off[P_VY], o[1]);
        if (!QUIRK && (SW == 1 || (P1 && !so.base))) {
            out.put(S.off[P_VXP1], o[2]);
            out.put(S.off[P_VYP1], o[3]);
        }
        if (!QUIRK && SW == 0 && P1 && so.base) {
            snap<EDGE, V>(g, so, slot, q, tm.snap_comp[P_VXP1], o[2]);
            snap<EDGE, V>(g, so, slot, q, tm.snap_comp[P_VYP1], o[3]);
        }
    }
};

// velocity, SH (src/update_v_PML_SH.c:61-297, CPML on every order);
// halo: sxz syz; plain: vz rjp; writes vz and vzp1 = previous vz
template <int FDOH, int TY, int NST>
struct OpVSh {
    static constexpr int V = kCells;
    static constexpr bool EARLY = false;
    static constexpr int DEP_TILES = INT_MAX;
    static constexpr int NH_ = 2, NP_ = 2;
    static constexpr bool CPML = true, MIRROR = true;
    using P = Pipe<FDOH, TY, NH_, NP_, NST, vblocks(FDOH), V>;
    IFOS_OP_MEMBERS
    // boxes of consecutive planes: their number, planes of box k, whether they are model planes
    static constexpr int NG = 2;
    __host__ __device__ static constexpr int gd(int k) { return 1 + 0 * k; }
    __host__ __device__ static constexpr bool gm(int k) { return k == 1; }
    void planes(int &hz, int (&gz)[NG]) const {  // first planes of the boxes, in slot 0 and model 0
        hz = tm.pid[P_SXZ];
        gz[0] = tm.pid[P_VZ];
        gz[1] = tm.mid[M_RJP];
    }
    struct Pre {
        Psi<V> x0, y0;
        RecIdx rec;
    };
    __device__ __forceinline__ void prefetch(const TileInfo &ti, Pre &pre) const {
        const Lane q = Lane::of<true, V>(g, ti);
        if (rec_mode && q.j >= rec_j0 && q.j <= rec_j1) pre.rec = rec_lookup(g, rec, rec_j0 == rec_j1, ti.slot, q);
        else pre.rec = RecIdx{{-1, -1, -1, -1}};
        if (!CPML) return;
        psi_x<V>(g, S.psix[X_SXZ] + ti.slot * S.psix_slot, q, pre.x0);
        psi_y<V>(g, S.psiy[Y_SYZ] + ti.slot * S.psiy_slot, q, pre.y0);
    }
    template <bool EDGE>
    __device__ __forceinline__ void rows(const TileInfo &ti, Pre &pre, const ProfTab &pt, const float *h,
                                         const float *pl, uint64_t *empty) const {
        const Lane q = Lane::of<EDGE, V>(g, ti);
        const int c0 = P::XH + q.c, slot = ti.slot;
        const Hc<FDOH> hc(g);
        float sxz_x[V], syz_y[V];
        {
            XWin<FDOH, V> w;
            w.load(h + (q.jj + P::H) * P::BW, c0);
#pragma unroll
            for (int e = 0; e < V; e++) sxz_x[e] = xbwd(hc, w, e);
        }
        ydiff_fs<true, EDGE, false, P>(hc, h + P::BOXS, q.jj, c0, g.free_surf && ti.j0 == 1, syz_y);
        const float *in = pl + q.jj * kTileX + q.c;
        const FV<V> vz = ldv<V>(in), rjp = ldv<V>(in + P::PLS);
        release_stage(empty);
        if (EDGE) {
            cpml_x<V>(g, M, pt, S.psix[X_SXZ] + slot * S.psix_slot, pre.x0, q, false, sxz_x);
            cpml_y<V>(g, pt, S.psiy[Y_SYZ] + slot * S.psiy_slot, pre.y0, q, true, syz_y);
        }
        float f[V], o[V];
#pragma unroll
        for (int e = 0; e < V; e++) f[e] = rjp.v[e] * g.dt * (sxz_x[e] + syz_y[e]);
        div_dh(g, f);
#pragma unroll
        for (int e = 0; e < V; e++) o[e] = vz.v[e] + f[e];
        if (EDGE && q.nv > 0) {
            const bool force = fvs && q.j >= src_j0 && q.j <= src_j1;
            if (force || any_receiver(pre.rec)) {
                Cells4 v{}, r{};
#pragma unroll
                for (int e = 0; e < V; e++) v.v[e] = o[e], r.v[e] = rjp.v[e];
                if (force) v = force_row_sh(g, src, slot, nt, q, r, v);
                if (any_receiver(pre.rec)) v = rec_row1<false>(g, rec, rec_mode, slot, nt, pre.rec, v);
#pragma unroll
                for (int e = 0; e < V; e++) o[e] = v.v[e];
            }
            if (probe && q.j == g.ny / 2) {
                const int at = g.nx / 2 - q.i;
#pragma unroll
                for (int e = 0; e < V; e++)
                    if (e == at && e < q.nv && isnan(o[e])) atomicExch(bad, 1);
            }
        }
        const RowOut<EDGE, V> out(g, S, slot, q);
        out.put(S.off[P_VZP1], vz.v);
        out.put(S.off[P_VZ], o);
        if (so.base) snap<EDGE, V>(g, so, slot, q, tm.snap_comp[P_VZP1], vz.v);
    }
};

// stress, SH elastic / viscoelastic (src/update_s_elastic_PML_SH.c,
// src/update_s_visc_PML_SH.c); halo: vz; plain: sxz syz [t[LL] o[LL]] and the
// coefficients (elastic: uipjp f; visco: fipjp f mu muipjp); writes sxz syz [t o]
template <int FDOH, int TY, int LL, int NST>
struct OpSSh {
    static constexpr int V = kCells;
    static constexpr bool EARLY = false;
    static constexpr int DEP_TILES = INT_MAX;
    static constexpr int NH_ = 1, NP_ = LL ? 2 + 2 * LL + 4 : 4, L1 = LL > 0 ? LL : 1;
    static constexpr bool CPML = true, MIRROR = false;
    using P = Pipe<FDOH, TY, NH_, NP_, NST, LL ? 3 : sblocks(FDOH), V>;
    IFOS_OP_MEMBERS
    // boxes of consecutive planes: their number, planes of box k, whether they are model planes
    static constexpr int NG = LL ? 5 : 2;
    __host__ __device__ static constexpr int gd(int k) { return k == 0 ? 2 : (!LL ? 2 : (k == 1 ? 2 * LL : (k == 2 ? 2 : 1))); }
    __host__ __device__ static constexpr bool gm(int k) { return k >= (LL ? 2 : 1); }
    void planes(int &hz, int (&gz)[NG]) const {  // first planes of the boxes, in slot 0 and model 0
        hz = tm.pid[P_VZ];
        gz[0] = tm.pid[P_SXZ];
        gz[1] = LL ? tm.mem_pid[MEM_T] : tm.mid[M_UIPJP];
        if (LL) gz[2 % NG] = tm.mid[M_FIPJPV], gz[3 % NG] = tm.mid[M_MUR], gz[4 % NG] = tm.mid[M_MUIPJPR];
    }
    struct Pre {
        Psi<V> x0, y0;
    };
    __device__ __forceinline__ void prefetch(const TileInfo &ti, Pre &pre) const {
        if (!CPML) return;
        const Lane q = Lane::of<true, V>(g, ti);
        psi_x<V>(g, S.psix[X_VZX] + ti.slot * S.psix_slot, q, pre.x0);
        psi_y<V>(g, S.psiy[Y_VZY] + ti.slot * S.psiy_slot, q, pre.y0);
    }
    template <bool EDGE>
    __device__ __forceinline__ void rows(const TileInfo &ti, Pre &pre, const ProfTab &pt, const float *h,
                                         const float *pl, uint64_t *empty) const {
        const Lane q = Lane::of<EDGE, V>(g, ti);
        const int c0 = P::XH + q.c, slot = ti.slot;
        const Hc<FDOH> hc(g);
        const float DT = g.dt, DH = g.dh;
        const float dhi = LL ? (float)(1.0 / (double)DH) : DT / DH, dthalbe = (float)((double)DT / 2.0);
        float vzx[V], vzy[V];
        {
            XWin<FDOH, V> w;
            w.load(h + (q.jj + P::H) * P::BW, c0);
#pragma unroll
            for (int e = 0; e < V; e++) vzx[e] = xfwd(hc, w, e) * dhi;
        }
        ydiff<false, false, false, P>(hc, h, q.jj, c0, vzy);
#pragma unroll
        for (int e = 0; e < V; e++) vzy[e] *= dhi;
        if (EDGE) {
            cpml_x<V>(g, M, pt, S.psix[X_VZX] + slot * S.psix_slot, pre.x0, q, true, vzx);
            cpml_y<V>(g, pt, S.psiy[Y_VZY] + slot * S.psiy_slot, pre.y0, q, false, vzy);
        }
        const float *in = pl + q.jj * kTileX + q.c;
        auto ld = [&](int k) { return ldv<V>(in + k * P::PLS); };
        const RowOut<EDGE, V> out(g, S, slot, q);
        const FV<V> s0 = ld(0), s1 = ld(1);
        float o[2][V];
        if (LL == 0) {
            const FV<V> fi = ld(2 % NP_), f = ld(3 % NP_);
            release_stage(empty);
#pragma unroll
            for (int e = 0; e < V; e++) {
                o[0][e] = s0.v[e] + (fi.v[e] * vzx[e]);
                o[1][e] = s1.v[e] + (f.v[e] * vzy[e]);
            }
        } else {
            constexpr int CO = 2 + 2 * LL;
            FV<V> mt[L1], mo[L1];
#pragma unroll
            for (int l = 0; l < LL; l++) mt[l] = ld(2 + l), mo[l] = ld(2 + LL + l);
            const FV<V> fipjp = ld(CO), f = ld(CO + 1), mu = ld(CO + 2), muij = ld(CO + 3);
            release_stage(empty);
            FV<V> ts = FV<V>::of(g.taus0), tsij = FV<V>::of(g.tausipjp0);
            if (M.m[M_TAUS]) {
                const long long at = (long long)ti.model() * M.model_stride + (min(q.j, g.ny) - 1 + HY) * g.pitch +
                                     (q.nv ? q.i - 1 + HX : 0);
                ts = ldv<V>(M.m[M_TAUS] + at);
                tsij = ldv<V>(M.m[M_TAUSIPJP] + at);
            }
            float sumo[V] = {}, sumt[V] = {};
#pragma unroll
            for (int e = 0; e < V; e++) {
#pragma unroll
                for (int l = 0; l < LL; l++) {
                    sumo[e] += mo[l].v[e];
                    sumt[e] += mt[l].v[e];
                }
                o[0][e] = s0.v[e] + ((fipjp.v[e] * vzx[e]) + (dthalbe * sumo[e]));
                o[1][e] = s1.v[e] + ((f.v[e] * vzy[e]) + (dthalbe * sumt[e]));
                sumo[e] = sumt[e] = 0;
            }
#pragma unroll
            for (int l = 0; l < LL; l++) {
                const float eta = g.eta[l + 1];
#pragma unroll
                for (int e = 0; e < V; e++) {
                    const float dip = muij.v[e] * eta * tsij.v[e], dd = mu.v[e] * eta * ts.v[e];
                    const float oo = g.bip[l + 1] * (mo[l].v[e] * g.cip[l + 1] - (dip * vzx[e]));
                    const float tt = g.bjm[l + 1] * (mt[l].v[e] * g.cjm[l + 1] - (dd * vzy[e]));
                    mo[l].v[e] = oo;
                    mt[l].v[e] = tt;
                    sumt[e] += tt;
                    sumo[e] += oo;
                }
                out.put(S.mem_off[MEM_T] + l * g.plane, mt[l].v);
                out.put(S.mem_off[MEM_O] + l * g.plane, mo[l].v);
            }
#pragma unroll
            for (int e = 0; e < V; e++) {
                o[0][e] = o[0][e] + (dthalbe * sumo[e]);
                o[1][e] = o[1][e] + (dthalbe * sumt[e]);
            }
        }
        if (EDGE && fsurf && q.j == 1) {  // src/surface_elastic_PML.c, SH: syz = 0
#pragma unroll
            for (int e = 0; e < V; e++) o[1][e] = 0.0f;
        }
        out.put(S.off[P_SXZ], o[0]);
        out.put(S.off[P_SYZ], o[1]);
        if (so.base) {
            snap<EDGE, V>(g, so, slot, q, tm.snap_comp[P_SXZ], o[0]);
            snap<EDGE, V>(g, so, slot, q, tm.snap_comp[P_SYZ], o[1]);
        }
    }
};

// pressure, acoustic (src/update_p_PML.c:55-273; default :275-287 when QUIRK)
// halo: vx vy; plain: sp g (reference 10/12 branch: vp); writes sp
template <int FDOH, int TY, int NST, bool QUIRK>
struct OpPAc {
    static constexpr int V = kCells;
    static constexpr bool EARLY = false;
    static constexpr int DEP_TILES = INT_MAX;
    static constexpr int NH_ = 2, NP_ = 2;
    static constexpr bool CPML = !QUIRK, MIRROR = false;
    using P = Pipe<FDOH, TY, NH_, NP_, NST, sblocks(FDOH), V>;
    IFOS_OP_MEMBERS
    // boxes of consecutive planes: their number, planes of box k, whether they are model planes
    static constexpr int NG = 2;
    __host__ __device__ static constexpr int gd(int k) { return 1 + 0 * k; }
    __host__ __device__ static constexpr bool gm(int k) { return k == 1; }
    void planes(int &hz, int (&gz)[NG]) const {  // first planes of the boxes, in slot 0 and model 0
        hz = tm.pid[P_VX];
        gz[0] = tm.pid[P_SP];
        gz[1] = tm.mid[QUIRK ? M_VP : M_GAC];
    }
    struct Pre {
        Psi<V> x0, y0;
        RecIdx rec;
    };
    __device__ __forceinline__ void prefetch(const TileInfo &ti, Pre &pre) const {
        const Lane q = Lane::of<true, V>(g, ti);
        if (rec_mode && q.j >= rec_j0 && q.j <= rec_j1) pre.rec = rec_lookup(g, rec, rec_j0 == rec_j1, ti.slot, q);
        else pre.rec = RecIdx{{-1, -1, -1, -1}};
        if (!CPML) return;
        psi_x<V>(g, S.psix[X_VXX] + ti.slot * S.psix_slot, q, pre.x0);
        psi_y<V>(g, S.psiy[Y_VYY] + ti.slot * S.psiy_slot, q, pre.y0);
    }
    template <bool EDGE>
    __device__ __forceinline__ void rows(const TileInfo &ti, Pre &pre, const ProfTab &pt, const float *h,
                                         const float *pl, uint64_t *empty) const {
        const Lane q = Lane::of<EDGE, V>(g, ti);
        const int c0 = P::XH + q.c, slot = ti.slot;
        const Hc<FDOH> hc(g);
        const float DT = g.dt, DH = g.dh;
        const float dhi = DT / DH;
        float vxx[V], vyy[V], o[V];
        {
            XWin<FDOH, V> w;
            w.load(h + (q.jj + P::H) * P::BW, c0);
#pragma unroll
            for (int e = 0; e < V; e++) vxx[e] = xbwd<QUIRK>(hc, w, e);
        }
        ydiff<false, false, false, P, QUIRK>(hc, h + P::BOXS, q.jj, c0, vyy);
        const float *in = pl + q.jj * kTileX + q.c;
        const FV<V> sp = ldv<V>(in), gg = ldv<V>(in + P::PLS);
        release_stage(empty);
        if (QUIRK) {
#pragma unroll
            for (int e = 0; e < V; e++) {
                const float gd = gg.v[e] * DT;
                o[e] = sp.v[e] + (gd * (vxx[e] + vyy[e])) * dhi;
            }
        } else {
#pragma unroll
            for (int e = 0; e < V; e++) vxx[e] = vxx[e] * dhi, vyy[e] = vyy[e] * dhi;
            if (EDGE) {
                cpml_x<V>(g, M, pt, S.psix[X_VXX] + slot * S.psix_slot, pre.x0, q, false, vxx);
                cpml_y<V>(g, pt, S.psiy[Y_VYY] + slot * S.psiy_slot, pre.y0, q, false, vyy);
            }
#pragma unroll
            for (int e = 0; e < V; e++) o[e] = sp.v[e] + gg.v[e] * (vxx[e] + vyy[e]);
        }
        if (EDGE && q.nv > 0) {
            // sources or adjoint sources, then the free surface, then the receivers
            const bool source = fps && q.j >= src_j0 && q.j <= src_j1, surface = fsurf && q.j == 1;
            if (source || surface || any_receiver(pre.rec)) {
                Cells4 v{};
#pragma unroll
                for (int e = 0; e < V; e++) v.v[e] = o[e];
                if (source) v = psource_row_p(g, src, slot, nt, q, v);
                if (rec_mode == 2 && any_receiver(pre.rec)) v = rec_row1<true>(g, rec, 2, slot, nt, pre.rec, v);
                if (surface) v = Cells4{};
                if (rec_mode == 1 && any_receiver(pre.rec)) v = rec_row1<true>(g, rec, 1, slot, nt, pre.rec, v);
#pragma unroll
                for (int e = 0; e < V; e++) o[e] = v.v[e];
            }
        }
        RowOut<EDGE, V>(g, S, slot, q).put(S.off[P_SP], o);
        if (so.base) snap<EDGE, V>(g, so, slot, q, tm.snap_comp[P_SP], o);
    }
};
// pressure, viscoacoustic with LL relaxation mechanisms
// (src/update_p_visc_PML.c:61-146 at FDORDER 2, with CPML; :148-182 for every
// other order: sums from zero and no CPML, hence Z0 and no strip path)
// halo: vx vy; plain: sp p[LL] g pi; writes sp p[LL].  Non-uniform taup is
// read from HBM.
template <int FDOH, int TY, int LL, int NST>
struct OpPVisc {
    static constexpr int V = kCells;
    static constexpr bool EARLY = false;
    static constexpr int DEP_TILES = INT_MAX;
    static constexpr bool Z0 = FDOH != 1, CPML = !Z0, MIRROR = false;
    static constexpr int NH_ = 2, NP_ = 3 + LL;
    using P = Pipe<FDOH, TY, NH_, NP_, NST, 3, V>;
    IFOS_OP_MEMBERS
    // boxes of consecutive planes: their number, planes of box k, whether they are model planes
    static constexpr int NG = 3;
    __host__ __device__ static constexpr int gd(int k) { return k == 0 ? 1 : (k == 1 ? LL : 2); }
    __host__ __device__ static constexpr bool gm(int k) { return k == 2; }
    void planes(int &hz, int (&gz)[NG]) const {  // first planes of the boxes, in slot 0 and model 0
        hz = tm.pid[P_VX];
        gz[0] = tm.pid[P_SP];
        gz[1] = tm.mem_pid[MEM_P];
        gz[2] = tm.mid[M_GV];
    }
    struct Pre {
        Psi<V> x0, y0;
        RecIdx rec;
    };
    __device__ __forceinline__ void prefetch(const TileInfo &ti, Pre &pre) const {
        const Lane q = Lane::of<true, V>(g, ti);
        if (rec_mode && q.j >= rec_j0 && q.j <= rec_j1) pre.rec = rec_lookup(g, rec, rec_j0 == rec_j1, ti.slot, q);
        else pre.rec = RecIdx{{-1, -1, -1, -1}};
        if (!CPML) return;
        psi_x<V>(g, S.psix[X_VXX] + ti.slot * S.psix_slot, q, pre.x0);
        psi_y<V>(g, S.psiy[Y_VYY] + ti.slot * S.psiy_slot, q, pre.y0);
    }
    template <bool EDGE>
    __device__ __forceinline__ void rows(const TileInfo &ti, Pre &pre, const ProfTab &pt, const float *h,
                                         const float *pl, uint64_t *empty) const {
        const Lane q = Lane::of<EDGE, V>(g, ti);
        const int c0 = P::XH + q.c, slot = ti.slot;
        const Hc<FDOH> hc(g);
        const float DT = g.dt, DH = g.dh;
        const float dhi = (float)(1.0 / (double)DH), dthalbe = (float)((double)DT / 2.0);
        float vxx[V], vyy[V], o[V];
        {
            XWin<FDOH, V> w;
            w.load(h + (q.jj + P::H) * P::BW, c0);
#pragma unroll
            for (int e = 0; e < V; e++) vxx[e] = xbwd<Z0>(hc, w, e) * dhi;
        }
        ydiff<false, false, false, P, Z0>(hc, h + P::BOXS, q.jj, c0, vyy);
#pragma unroll
        for (int e = 0; e < V; e++) vyy[e] *= dhi;
        const float *in = pl + q.jj * kTileX + q.c;
        auto ld = [&](int k) { return ldv<V>(in + k * P::PLS); };
        FV<V> mp[LL];
#pragma unroll
        for (int l = 0; l < LL; l++) mp[l] = ld(1 + l);
        const FV<V> sp = ld(0), gg = ld(1 + LL), pi = ld(2 + LL);
        release_stage(empty);
        if (EDGE && CPML) {
            cpml_x<V>(g, M, pt, S.psix[X_VXX] + slot * S.psix_slot, pre.x0, q, false, vxx);
            cpml_y<V>(g, pt, S.psiy[Y_VYY] + slot * S.psiy_slot, pre.y0, q, false, vyy);
        }
        FV<V> tp = FV<V>::of(g.taup0);
        if (M.m[M_TAUP])
            tp = ldv<V>(M.m[M_TAUP] + (long long)ti.model() * M.model_stride + (min(q.j, g.ny) - 1 + HY) * g.pitch +
                      (q.nv ? q.i - 1 + HX : 0));
        const RowOut<EDGE, V> out(g, S, slot, q);
        float sump[V] = {};
#pragma unroll
        for (int e = 0; e < V; e++) {
#pragma unroll
            for (int l = 0; l < LL; l++) sump[e] += mp[l].v[e];
            o[e] = sp.v[e] + ((gg.v[e] * (vxx[e] + vyy[e])) + (dthalbe * sump[e]));
            sump[e] = 0;
        }
#pragma unroll
        for (int l = 0; l < LL; l++) {
#pragma unroll
            for (int e = 0; e < V; e++) {
                const float ee = pi.v[e] * g.eta[l + 1] * tp.v[e];  // e of src/prepare_update_p.c:62
                const float pp = g.bjm[l + 1] * (mp[l].v[e] * g.cjm[l + 1] - (ee * (vxx[e] + vyy[e])));
                mp[l].v[e] = pp;
                sump[e] += pp;
            }
            out.put(S.mem_off[MEM_P] + l * g.plane, mp[l].v);
        }
#pragma unroll
        for (int e = 0; e < V; e++) o[e] = o[e] + (dthalbe * sump[e]);
        if (EDGE && q.nv > 0) {
            // sources or adjoint sources, then the free surface, then the receivers
            const bool source = fps && q.j >= src_j0 && q.j <= src_j1, surface = fsurf && q.j == 1;
            if (source || surface || any_receiver(pre.rec)) {
                Cells4 v{};
#pragma unroll
                for (int e = 0; e < V; e++) v.v[e] = o[e];
                if (source) v = psource_row_p(g, src, slot, nt, q, v);
                if (rec_mode == 2 && any_receiver(pre.rec)) v = rec_row1<true>(g, rec, 2, slot, nt, pre.rec, v);
                if (surface) v = Cells4{};
                if (rec_mode == 1 && any_receiver(pre.rec)) v = rec_row1<true>(g, rec, 1, slot, nt, pre.rec, v);
#pragma unroll
                for (int e = 0; e < V; e++) o[e] = v.v[e];
            }
        }
        out.put(S.off[P_SP], o);
        if (so.base) snap<EDGE, V>(g, so, slot, q, tm.snap_comp[P_SP], o);
    }
};
#undef IFOS_OP_MEMBERS

// Blocks per SM for the register budget: as many as the shared-memory ring
// allows (227 KB per SM), at most the op's BLOCK_CAP.
template <typename P>
constexpr int ring_blocks() {
    constexpr int b = (int)(232448 / (P::bytes() + 1024 + 2 * kTileBatch * sizeof(TileInfo) + 6 * (kProfX + kProfY) * 4 + 128));
    return b < 1 ? 1 : (b > P::BLOCK_CAP ? P::BLOCK_CAP : b);
}

// the kernel: one Op per launch, persistent over all tiles of all slots
template <typename Op>
__global__ void __launch_bounds__(Op::P::THREADS, ring_blocks<typename Op::P>())
    kp_stencil(const __grid_constant__ KMaps maps, const __grid_constant__ TileWalk walk, const __grid_constant__ Op op,
               int *err) {
    run_pipeline<typename Op::P>(op.g, maps, walk, op, err);
}

}  // namespace ifos
