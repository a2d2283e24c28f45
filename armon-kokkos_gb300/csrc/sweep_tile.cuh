// sweep_tile.cuh -- the axis pass with one thread per position: a block takes a tile (a few lines by a
// stretch of positions, halo included), every thread computes each stage at its own position, and
// the stages hand their values to the neighbouring positions through shared memory.
//
// Same stage functions on the same operands as the marches (sweep.cuh, sweep_split.cuh), so the
// results are the same bits.
//
// Why tiles.  A march owns a segment of a line per thread: its positions run one after the other
// (~1600 dependent instructions each), its pipeline keeps ~75 FP64 values alive (250 registers, 8
// warps per SM), and in the X pass its warp loads touch 32 rows.  A tile's thread keeps one position,
// and only a stage's operands are alive at once, so more warps share an SM, a pass over a small
// domain lasts as long as one position's chain, and both axes read consecutive addresses.
//
// What bounds it.  FP64 where every position is computed (2048x2048 moving flow): the FP64 pipe, 76 %
// busy with ~106 operations a position on 24 warps per SM (a march's 8 to 12 warps left it 60-75 %
// busy in each of two launches): 0.94 ms an X pass; 24 cycles 78.2 ms with marches, 45.9 ms now.  FP32
// there: instruction issue, 70 % busy, 0.14 ms.  A uniform fluid with fronts (4096x4096 circular Sod):
// a block's own chain of scan, stores and computed stretches (30 000 cycles each), three blocks per
// SM; 0.55 ms a pass at cycles 180-200, against 1.1 ms.  Small domains: one position's ~3000
// dependent instructions, 16 us a pass (96x64: 40 us a cycle, 546 us with marches).
// Where it loses to marches: planar fronts.  Every line along one holds a state of its own, which a march
// streams; a scan knows two states and computes the rest (solver.cu planar_test, batch.cu wants_tiles).
// Looking for runs of any state in units that are not all idle made planar fronts 1.3 to 1.6 times
// faster in FP64 and the 4096x4096 circular Sod 20 to 30 % slower (code size), and was dropped.
// Measured and dropped: 64 registers and four blocks per SM in FP64 (spills; +4 to +20 %), products on
// the integer pipes (dense 5 % faster at best, fronts 15-40 % slower), the quotients of a stage in one
// straight-line group (+7 to +10 %: more code), cells of the next unit asked for in L2 (+8 %),
// batches of eight cells in a scan (+4 %).
//
// Tile geometry.  X pass: a tile is tile_lines rows by tile_width positions, thread = row * tile_width +
// position, so a warp reads a stretch of a row.  Y pass: tile_lines columns by tile_width positions,
// thread = position * tile_lines + column; the neighbours along the axis are tile_lines threads away.
// tile_width = tile_len + 2 H positions (H = the stencil reach, 4 for GAD + second order), of which
// the inner tile_len are stored.
//
// Units and dispatch.  Blocks stay resident; a block takes units of consecutive tiles, the first by its
// index and the following ones from a ticket counter, so that tiles that cost more (fronts) spread
// over the blocks by themselves.  The first tile_big units hold kTileUnit tiles, the rest one each,
// so that the launch ends evenly.
//
// Exact reuse (SweepArgs::reuse).  A position whose window (H positions on either side) holds equal
// cells, bit for bit, has results that depend on that cell's state alone.  A block keeps two such
// states with their results, recorded by the thread at the middle of a computed stretch when its
// window is uniform.  Once it keeps one it scans a unit before computing: every cell is loaded (the
// loads of a batch issued together) and compared with the kept states, eight-position chunks whose
// windows all hold a kept state get its results, and what is left becomes stretches (a line's
// consecutive chunks) in a list.  The block computes the list packed, several stretches side by side
// in its threads, so that a thin front costs its own positions and not whole tiles.  A unit without
// a uniform chunk is computed as tiles, and a block that keeps no state does not scan.
// The results of the states a pass keeps are what its uniform regions hold next, so they are left as
// hints: the next pass's blocks start by evaluating them (a window of equal cells, and the positions
// next to either wall), and so know the resting regions, walls included, from their first unit.
// A hint only proposes a state; cells take its results when they equal it bit for bit.
#pragma once

#include "sweep.cuh"

namespace armon {

constexpr int kTileThreads = 256;
constexpr int kTileWarps = kTileThreads / 32;
constexpr int kTileSlots = 15;
constexpr int kTileList = 512;        // stretches the list can hold (at most 128 per scan, 32 left over)

#ifndef ARMON_TILE_MIN_BLOCKS
#define ARMON_TILE_MIN_BLOCKS 3
#endif
#ifndef ARMON_TILE_MIN_BLOCKS_F32
#define ARMON_TILE_MIN_BLOCKS_F32 4
#endif
template <class T> constexpr int tile_min_blocks() { return sizeof(T) == 8 ? ARMON_TILE_MIN_BLOCKS : ARMON_TILE_MIN_BLOCKS_F32; }

// A kept state: the cell, its p and c, the results of a position inside a run of it, and the results of
// the H <= 4 positions next to a wall (low side, high side) when the run reaches it.
enum : int { kRunRho, kRunUa, kRunUo, kRunE, kRunP, kRunC, kRunOut, kRunWall = kRunOut + 4, kRunValues = kRunWall + 32 };

// Consecutive owned positions of a line waiting to be computed.
struct Stretch {
    int32_t line;
    int32_t start_len;    // first position (below 2^23) << 8 | positions (at most 248)
};

template <class T>
struct TileShared {
    // Slots between the stages (a barrier after each stage's writes; a slot is only rewritten after a
    // barrier that follows its last reads, the next tile's stages included):
    //   cell products      rc, rcu, p, ua, dm                9-13
    //   face differences   au, bu, ap, bp                    5-8
    //   fluxes             u*, p*, p* u*, dt u*              0-3
    //   Lagrangian cells   rho, rho ua, rho uo, rho E, W     4-8
    //   their differences  four, and the width sum           9-13
    //   advection fluxes   four                              0, 1, 2, 14
    T ex[kTileSlots][kTileThreads];
    T c[kTileThreads];                // sound speed of the position, for dt_CFL
    T kept[2][kRunValues];
    DtAcc acc[kTileThreads];
    Stretch list[kTileList];          // a ring: entries head .. tail - 1
    uint32_t match[2][2][kTileWarps][kTileWarps];   // [unit parity][kept state]: see scan_rows / scan_columns
    uint32_t head;
    uint32_t tail[2];                 // [unit parity]
    int uniform[2];                   // [unit parity]: the unit holds a uniform chunk
    int valid[2];                     // bit 0: the state is kept; bit 1: with its walls
    int turn;                         // the kept state to replace next
    int claims;                       // states recorded so far
    int next[2];                      // [unit parity]: the block's next unit
};

// The place of thread tid among packed stretches: the first stretch whose threads (sum(j): those of the
// stretches up to j) end past it, k, and its position there, q.  False for a thread that stands for
// none: behind the `take` stretches that fit, or behind the last of all 32, which the search's five
// steps also give k = 31 (32 stretches of fewer than eight threads leave such threads: a segment's
// last few cells with a stencil reach of two or three).  sum and need are the block's shuffles, or arrays on the host.
#pragma nv_exec_check_disable
template <class Sum, class Need>
__host__ __device__ __forceinline__ bool pack_place(int tid, int take, Sum sum, Need need, int& k, int& q)
{
    k = 0;
    for (int o = 16; o > 0; o >>= 1) {
        const int v = sum(k + o - 1);
        if (v <= tid) k += o;
    }
    const int threads = need(k);
    q = tid - (sum(k) - threads);
    return k < take && q < threads;
}

// The tiles of one unit of one domain.  SCAN: its units may be scanned (AxisGeom::tile_scan); without it
// the pass is its stages alone, half the code.
template <class T, int SCHEME, int PROJ, bool SCAN>
struct TilePass {
    static constexpr bool kGAD = SCHEME == 1;
    static constexpr bool kE2 = PROJ == 2;
    static constexpr int H = 2 + (kGAD ? 1 : 0) + (kE2 ? 1 : 0);
    static constexpr int kLagLo = kGAD ? 2 : 1;      // first position with a Lagrangian cell

    const SweepArgs<T>& A;
    TileShared<T>& sh;
    int axis = 0, src = 0;
    T dt{};
    bool last = false, pcg = false;
    int tile_q = 0, tile_l = 0;       // the thread's position and line in a tile
    int parity = 0;
    bool hints = false;               // the hinted states are still to be evaluated
    uint32_t counted = 0;             // kept states whose speeds this thread has added (a bit each)

    struct Spot {                     // the thread's place
        int hint;                     // the hinted state the thread stands for, -1 for a cell
        int q, t, width;              // position in the stretch (halo included), along the axis; positions of the stretch
        int64_t base;                 // index of position 0 of the line
        bool in;
    };

    __device__ __forceinline__ TilePass(const SweepArgs<T>& a, TileShared<T>& s) : A(a), sh(s) {}

    // Reads the domain's step state; false when this pass has nothing to do.
    __device__ __forceinline__ bool start(int pass, bool last_pass, bool reports)
    {
        const StepState st = *A.state;
        const CycleDt cd = cycle_time_step(st, A.cfg);
        if (!cd.run) return false;
        if (cd.invalid) {
            if (last_pass && reports) A.state->status = STATUS_INVALID_DT;
            return false;
        }
        double factor;
        split_axis(A.cfg.splitting, st.cycle, pass, &axis, &factor);
        dt = T(cd.current * factor);
        src = (int)(((int64_t)st.cycle * A.npass + pass + st.buf_base) & 1);
        last = last_pass;
        counted = 0;
        pcg = A.write_eos > 0 || (last_pass && A.write_eos == 0);
        const AxisGeom<T>& g = A.geom[axis];
        const int tid = threadIdx.x;
        if (axis == 0) {
            tile_l = tid / g.tile_width;
            tile_q = tid - tile_l * g.tile_width;
        } else {
            tile_q = tid / g.tile_lines;
            tile_l = tid - tile_q * g.tile_lines;
        }
        hints = SCAN && A.reuse && g.tile_scan && A.sw >= H &&
                (__ldcg(&A.hints->valid[src][0]) | __ldcg(&A.hints->valid[src][1])) != 0;
        return true;
    }

    // Segment and line group of a tile: along rows (X) consecutive tiles follow the line, along
    // columns (Y) they lie side by side.
    __device__ __forceinline__ void place(const AxisGeom<T>& g, int tile, int& seg, int& grp) const
    {
        if (axis == 0) { grp = tile / g.tile_segs; seg = tile - grp * g.tile_segs; }
        else { seg = tile / g.tile_groups; grp = tile - seg * g.tile_groups; }
    }
    __device__ __forceinline__ Spot tile_spot(const AxisGeom<T>& g, int tile) const
    {
        int seg, grp;
        place(g, tile, seg, grp);
        const int a0 = seg * g.tile_len;
        Spot p;
        p.hint = -1;
        p.q = tile_q;
        p.width = min(g.n, a0 + g.tile_len) - a0 + 2 * H;
        p.t = a0 - H + tile_q;
        const int line = grp * g.tile_lines + tile_l;
        p.in = tile_q < p.width && tile_l < g.tile_lines && line < g.nlines;
        p.base = A.origin + (int64_t)line * g.lstride;
        return p;
    }
    // position t -> the cell read there: itself (real, or an untouched ghost past the mirrored band:
    // stale), or the mirror of a real cell (side 1: low, 2: high); the same rule as the marches'
    __device__ __forceinline__ bool source(int n, int t, int& m, int& side) const
    {
        m = t;
        side = 0;
        if (t < 0) {
            if (t < -A.sw) return true;
            m = -1 - t;
            side = 1;
        } else if (t >= n) {
            if (t >= n + A.sw) return true;
            m = 2 * n - 1 - t;
            side = 2;
        }
        return false;
    }
    __device__ __forceinline__ void mirror(const AxisGeom<T>& g, CellIn<T>& c, int side) const
    {
        if (side) {
            if (g.f_unit) {
                const uint32_t b = side == 1 ? 0 : 2;
                c.ua = qneg_if(c.ua, (g.fneg >> b) & 1u);
                c.uo = qneg_if(c.uo, (g.fneg >> (b + 1)) & 1u);
            } else {
                c.ua = c.ua * (side == 1 ? g.fa_lo : g.fa_hi);
                c.uo = c.uo * (side == 1 ? g.fo_lo : g.fo_hi);
            }
        }
    }
    __device__ __forceinline__ void load(int64_t i, CellIn<T>& c) const
    {
        T* const* in = A.buf[src];
        c.rho = in[0][i];
        c.ua = in[1 + axis][i];
        c.uo = in[2 - axis][i];
        c.E = in[3][i];
    }
    __device__ __forceinline__ bool same_as_kept(const CellIn<T>& c, int e) const
    {
        const T* k = sh.kept[e];
        return same_bits(c.rho, k[kRunRho]) & same_bits(c.ua, k[kRunUa]) & same_bits(c.uo, k[kRunUo]) &
               same_bits(c.E, k[kRunE]);
    }

    // Whether a loaded cell equals a kept state, read from shared memory each time (a state held in
    // registers over a scan's loop costs 8 or 16 of them, and the loop's loads in flight spill).
    static __device__ __forceinline__ bool same_cell(const T (&c)[4], const T* k)
    {
        return same_bits(c[0], k[kRunRho]) & same_bits(c[1], k[kRunUa]) & same_bits(c[2], k[kRunUo]) & same_bits(c[3], k[kRunE]);
    }

    // The unit's tiles.  `after`, run by thread 0, gives the block's next unit, which is returned;
    // when there is none (>= total), what the list still holds is computed too.
    template <class After>
    __device__ __forceinline__ int unit(int u, int total, After after)
    {
        const AxisGeom<T>& g = A.geom[axis];
        int tile = u < g.tile_big ? u * kTileUnit : g.tile_big * kTileUnit + (u - g.tile_big);
        // (a batch's domains have as many units as their larger axis: those past the axis's own are empty)
        const int end = u < g.tile_big ? tile + kTileUnit : u < g.tile_units ? tile + 1 : tile;
        int next = total;
        bool fetch = true;
        do {
            parity ^= 1;
            if (threadIdx.x == 0) {
                if (fetch) sh.next[parity] = after();
                sh.tail[parity] = sh.tail[parity ^ 1];
                sh.uniform[parity ^ 1] = 0;     // read before the last barrier, set after the next
            }
            const int v0 = sh.valid[0], v1 = sh.valid[1], claims = sh.claims;
            int seen = claims;
            // the same for every thread: a barrier follows each of their writes
            const bool waiting = hints;      // only the hinted states this time
            bool evaluate = hints;
            hints = false;
            const bool scan = SCAN && g.tile_scan && (v0 | v1) && !evaluate && tile < end;
            // a block that keeps no state yet takes a tile at a time, to scan the rest once it does
            int nk = evaluate ? 0 : scan || !SCAN || !g.tile_scan ? end - tile : min(1, end - tile);
            int k = 0;
            if (scan) {
                if (axis == 0) scan_rows(g, tile, nk, v0, v1);
                else scan_columns(g, tile, nk, v0, v1);
                __syncthreads();
                if (sh.uniform[parity]) {
                    k = nk;
                    if (axis == 0) fill_rows(g, tile, nk);
                    else fill_columns(g, tile, nk);
                }
            }
            __syncthreads();
            if (fetch) next = sh.next[parity];
            fetch = false;
            const bool all = next >= total && tile + nk >= end && !evaluate;
            // the hinted states, the tiles, or the list's stretches, packed
            for (;;) {
                Spot p;
                int ds = 1, centre = -1;
                if (SCAN && evaluate) {
                    p = hint_spot(g);
                } else if (k < nk) {
                    if (scan && seen != claims) {   // a state more is kept: scan the rest again
                        nk = k;
                        continue;
                    }
                    p = tile_spot(g, tile + k);
                    if (axis != 0) ds = g.tile_lines;
                    centre = (p.width / 2) * ds;      // the middle of the tile's first line
                    k++;
                } else if (!SCAN || waiting || !pack(all && tile + nk >= end, p, centre)) {
                    break;
                }
                seen = compute(g, p, ds, centre);
                evaluate = false;
            }
            tile += nk;
        } while (tile < end);
        return next;
    }

    // ---- scan ----
    // Ghosts (whose mirrored velocities differ from a state at rest by the sign of zero) match a state
    // that is kept with its walls' results.
    // Rows: warp w takes the unit's tile w, its positions 32 at a time; match[state][w][i] is the ballot
    // of positions 32 i .. 32 i + 31 of the tile (positions past its end count as matching).
    __device__ __forceinline__ void scan_rows(const AxisGeom<T>& g, int tile0, int nk, int v0, int v1)
    {
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if (w >= nk) return;
        int seg, grp;
        place(g, tile0 + w, seg, grp);
        if (grp >= g.nlines) return;
        const int a0 = seg * g.tile_len;
        const int width = min(g.n, a0 + g.tile_len) - a0 + 2 * H;
        // positions [lo, lo + real) of the tile are cells; the ones past its end match, ghosts as the state allows
        const int lo = max(0, H - a0), real = min(width, g.n - a0 + H) - lo;
        T* const* in = A.buf[src];
        const int64_t i0 = A.origin + (int64_t)grp * g.lstride + (a0 - H) + lane;
        const T *rho = in[0] + i0, *ua = in[1 + axis] + i0, *uo = in[2 - axis] + i0, *E = in[3] + i0;
        const T *k0 = sh.kept[0], *k1 = sh.kept[1];
        constexpr int kBatch = 4;
#pragma unroll 1
        for (int i0 = 0; i0 < kTileWarps; i0 += kBatch) {
            T c[kBatch][4] = {};
#pragma unroll
            for (int i = 0; i < kBatch; i++) {
                if ((unsigned)(32 * (i0 + i) + lane - lo) < (unsigned)real) {
                    c[i][0] = rho[32 * i]; c[i][1] = ua[32 * i]; c[i][2] = uo[32 * i]; c[i][3] = E[32 * i];
                }
            }
#pragma unroll
            for (int i = 0; i < kBatch; i++) {
                const int q = 32 * (i0 + i) + lane;
                const bool cell = (unsigned)(q - lo) < (unsigned)real;
                const uint32_t b0 = __ballot_sync(0xffffffffu, (cell & same_cell(c[i], k0) & (v0 != 0)) | (!cell & ((q >= width) | (v0 > 1))));
                uint32_t b1 = 0;
                if (v1 && b0 != 0xffffffffu)
                    b1 = __ballot_sync(0xffffffffu, (cell & same_cell(c[i], k1)) | (!cell & ((q >= width) | (v1 > 1))));
                if (lane == 0) {
                    sh.match[parity][0][w][i0 + i] = b0;
                    sh.match[parity][1][w][i0 + i] = b1;
                }
            }
            rho += 32 * kBatch; ua += 32 * kBatch; uo += 32 * kBatch; E += 32 * kBatch;
        }
        __syncwarp();
        if (__any_sync(0xffffffffu, chunk_state(w, lane) >= 0 && 8 * lane < width - 2 * H) && lane == 0)
            sh.uniform[parity] = 1;
    }
    // The kept state of chunk j (owned positions 8 j .. 8 j + 7) of warp w's tile, -1 when its windows do
    // not all hold one: they lie in positions 8 j .. 8 j + 15 of the tile.
    __device__ __forceinline__ int chunk_state(int w, int j) const
    {
        if (j >= 31) return -1;
        const uint16_t b0 = window16(&sh.match[parity][0][w][0], j), b1 = window16(&sh.match[parity][1][w][0], j);
        return b0 == 0xffffu ? 0 : b1 == 0xffffu ? 1 : -1;
    }
    static __device__ __forceinline__ uint16_t window16(const uint32_t* words, int j)
    {
        const unsigned char* b = reinterpret_cast<const unsigned char*>(words);
        return (uint16_t)(b[j] | (b[j + 1] << 8));
    }
    __device__ __forceinline__ void fill_rows(const AxisGeom<T>& g, int tile0, int nk)
    {
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if (w >= nk) return;
        int seg, grp;
        place(g, tile0 + w, seg, grp);
        if (grp >= g.nlines) return;
        const int a0 = seg * g.tile_len;
        const int len = min(g.n, a0 + g.tile_len) - a0;
        const int e = chunk_state(w, lane);
        const uint32_t live = __ballot_sync(0xffffffffu, 8 * lane < len);
        const uint32_t idle0 = __ballot_sync(0xffffffffu, e == 0), idle1 = __ballot_sync(0xffffffffu, e == 1);
        push(live & ~(idle0 | idle1), grp, a0, len);
        const int64_t base = A.origin + (int64_t)grp * g.lstride + a0;
        const int whole = live == (idle0 & live) ? 0 : live == (idle1 & live) ? 1 : -1;
        if (whole >= 0 && !pcg && a0 >= H && a0 + len <= g.n - H) {
            // the whole tile, away from the walls
            const T* kv = sh.kept[whole];
            const T o0 = kv[kRunOut], o1 = kv[kRunOut + 1], o2 = kv[kRunOut + 2], o3 = kv[kRunOut + 3];
            T* const* out = A.buf[src ^ 1];
            T *rho = out[0] + base + lane, *ua = out[1 + axis] + base + lane, *uo = out[2 - axis] + base + lane, *E = out[3] + base + lane;
#pragma unroll
            for (int i = 0; i < kTileWarps; i++) {
                if (32 * i + lane < len) { rho[32 * i] = o0; ua[32 * i] = o1; uo[32 * i] = o2; E[32 * i] = o3; }
            }
            count_kept(whole);
            return;
        }
        for (int o = lane; o < len; o += 32) {
            const int j = o >> 3;
            if ((idle0 >> j) & 1u) store_kept(g, base + o, a0 + o, 0);
            else if ((idle1 >> j) & 1u) store_kept(g, base + o, a0 + o, 1);
        }
    }
    // Appends the runs of a line's chunks in `todo` (bit j: chunk j, at a0 + 8 j) to the list; runs one
    // idle chunk apart are joined (they share their halos).  Every lane of a warp has the same mask.
    __device__ __forceinline__ void push(uint32_t todo, int line, int a0, int len)
    {
        todo |= (todo << 1) & (todo >> 1);
        const int lane = threadIdx.x & 31;
        if (((todo >> lane) & 1u) && (lane == 0 || !((todo >> (lane - 1)) & 1u))) push_run(todo >> lane, lane, line, a0, len);
    }
    __device__ __forceinline__ void push_run(uint32_t mask, int j, int line, int a0, int len)
    {
        const int chunks = __ffs((int)~mask) - 1;            // ones at the low end (mask has at most 31)
        list(line, a0 + 8 * j, min(8 * chunks, len - 8 * j));
    }
    __device__ __forceinline__ void list(int line, int start, int cells)
    {
        const uint32_t at = atomicAdd(&sh.tail[parity], 1u);
        sh.list[at % kTileList] = Stretch{line, (start << 8) | cells};
    }
    // The results of position t, at index i, of a run of kept state e.
    __device__ __forceinline__ void store_kept(const AxisGeom<T>& g, int64_t i, int t, int e)
    {
        const T* kv = sh.kept[e];
        const bool wall = t < H || t >= g.n - H;
        const T* o = kv + (!wall ? (int)kRunOut : t < H ? kRunWall + 4 * t : kRunWall + 16 + 4 * (t - (g.n - H)));
        T* const* out = A.buf[src ^ 1];
        out[0][i] = o[0];
        out[1 + axis][i] = o[1];
        out[2 - axis][i] = o[2];
        out[3][i] = o[3];
        if (pcg) {
            A.pmat[i] = kv[kRunP];
            A.cmat[i] = kv[kRunC];
            A.gmat[i] = (1 + A.gamma) / 2;
        }
        if (wall) {
            if (last) add_dt(o, kv[kRunC]);
        } else {
            count_kept(e);
        }
    }
    // A run of kept state e has been stored: its speeds count once.
    __device__ __forceinline__ void count_kept(int e)
    {
        if (last && !((counted >> e) & 1u)) {
            counted |= 1u << e;
            add_dt(sh.kept[e] + kRunOut, sh.kept[e][kRunC]);
        }
    }
    // dt_CFL of the state after this pass, with c from this pass's EOS
    __device__ __forceinline__ void add_dt(const T* o, T c)
    {
        if (axis == 0) sh.acc[threadIdx.x].add(o[1], o[2], c);
        else sh.acc[threadIdx.x].add(o[2], o[1], c);
    }
    // The evaluation of the hinted states: per state, threads for a position inside a run of it (a
    // window of 2 H + 1 cells) and for the H positions next to either wall.
    __device__ __forceinline__ Spot hint_spot(const AxisGeom<T>& g) const
    {
        constexpr int kPlain = 2 * H + 1, kSide = 3 * H, kAll = kPlain + 2 * kSide;
        const int tid = threadIdx.x;
        const int r = tid % kAll;
        Spot p;
        p.hint = tid / kAll;
        p.in = p.hint < 2 && __ldcg(&A.hints->valid[src][min(p.hint, 1)]);
        p.base = 0;
        if (r < kPlain) { p.q = r; p.width = kPlain; p.t = g.n / 2; }
        else if (r < kPlain + kSide) { p.q = r - kPlain; p.width = kSide; p.t = p.q - H; }
        else { p.q = r - kPlain - kSide; p.width = kSide; p.t = g.n - 2 * H + p.q; }
        return p;
    }
    // Columns: the unit's nk tiles are `cols` columns of one segment; thread f takes column f % cols and
    // the eight positions 8 (f / cols) .. of the segment (halo included), and bit f of match[state][0]
    // says whether they all match.  Chunk j of a column is uniform when bits j cols + column and
    // (j + 1) cols + column are set.
    __device__ __forceinline__ void scan_columns(const AxisGeom<T>& g, int tile0, int nk, int v0, int v1)
    {
        const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
        int seg, grp;
        place(g, tile0, seg, grp);
        const int cols = nk * g.tile_lines;
        const int j = tid / cols;
        const int line = grp * g.tile_lines + tid - j * cols;
        const int a0 = seg * g.tile_len;
        const int width = min(g.n, a0 + g.tile_len) - a0 + 2 * H;
        // positions [lo, lo + real) of the segment are cells
        const int lo = max(0, H - a0), real = min(width, g.n - a0 + H) - lo;
        T* const* in = A.buf[src];
        const int64_t i0 = A.origin + (int64_t)line * g.lstride + (int64_t)(a0 - H + 8 * j) * g.s;
        const T *rho = in[0] + i0, *ua = in[1 + axis] + i0, *uo = in[2 - axis] + i0, *E = in[3] + i0;
        const T *k0 = sh.kept[0], *k1 = sh.kept[1];
        constexpr int kBatch = 4;
        bool m0 = v0 != 0, m1 = v1 != 0;
        const bool live = line < g.nlines && 8 * j < width;
        if (live) {
#pragma unroll 1
            for (int q0 = 8 * j; q0 < 8 * j + 8; q0 += kBatch) {
                T c[kBatch][4] = {};      // (left unset, they would be carried from batch to batch)
#pragma unroll
                for (int i = 0; i < kBatch; i++) {
                    if ((unsigned)(q0 + i - lo) < (unsigned)real) { c[i][0] = *rho; c[i][1] = *ua; c[i][2] = *uo; c[i][3] = *E; }
                    rho += g.s; ua += g.s; uo += g.s; E += g.s;
                }
#pragma unroll
                for (int i = 0; i < kBatch; i++) {
                    const bool cell = (unsigned)(q0 + i - lo) < (unsigned)real, out = q0 + i >= width;
                    m0 = m0 & ((cell & same_cell(c[i], k0)) | (!cell & (out | (v0 > 1))));
                    m1 = m1 & ((cell & same_cell(c[i], k1)) | (!cell & (out | (v1 > 1))));
                }
            }
        }
        const uint32_t b0 = __ballot_sync(0xffffffffu, m0), b1 = __ballot_sync(0xffffffffu, m1);
        if (lane == 0) {
            sh.match[parity][0][0][w] = b0;
            sh.match[parity][1][0][w] = b1;
        }
        __syncthreads();
        if (__any_sync(0xffffffffu, live && 8 * j < width - 2 * H && column_state(tid, cols) >= 0) && lane == 0)
            sh.uniform[parity] = 1;
    }
    // The kept state of the chunk that begins with thread f's positions, -1 when its windows do not all
    // hold one.  (A segment's last chunk may lack positions past its halo: they would match.)
    __device__ __forceinline__ int column_state(int f, int cols) const
    {
        const int h = f + cols;
        const bool past = h >= kTileThreads;
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const uint32_t* m = &sh.match[parity][e][0][0];
            if (((m[f >> 5] >> (f & 31)) & 1u) && (past || ((m[(h & 255) >> 5] >> (h & 31)) & 1u))) return e;
        }
        return -1;
    }
    __device__ __forceinline__ void fill_columns(const AxisGeom<T>& g, int tile0, int nk)
    {
        const int tid = threadIdx.x;
        int seg, grp;
        place(g, tile0, seg, grp);
        const int cols = nk * g.tile_lines;
        const int j = tid / cols;
        const int line = grp * g.tile_lines + tid - j * cols;
        if (line >= g.nlines) return;
        const int a0 = seg * g.tile_len;
        const int len = min(g.n, a0 + g.tile_len) - a0;
        const int end = min(8 * j + 8, len);
        const int e = 8 * j < len ? column_state(tid, cols) : -1;
        if (e >= 0 && !pcg && a0 >= H && a0 + len <= g.n - H) {
            // away from the walls
            const T* kv = sh.kept[e];
            const T o0 = kv[kRunOut], o1 = kv[kRunOut + 1], o2 = kv[kRunOut + 2], o3 = kv[kRunOut + 3];
            T* const* out = A.buf[src ^ 1];
            const int64_t i0 = A.origin + (int64_t)line * g.lstride + (int64_t)(a0 + 8 * j) * g.s;
            T *rho = out[0] + i0, *ua = out[1 + axis] + i0, *uo = out[2 - axis] + i0, *E = out[3] + i0;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (8 * j + i < end) { *rho = o0; *ua = o1; *uo = o2; *E = o3; }
                rho += g.s; ua += g.s; uo += g.s; E += g.s;
            }
            count_kept(e);
        } else if (e >= 0) {
            for (int o = 8 * j; o < end; o++)
                store_kept(g, A.origin + (int64_t)line * g.lstride + (int64_t)(a0 + o) * g.s, a0 + o, e);
        }
        // a run's first thread lists it; runs one chunk apart are joined, as push does
        const auto todo = [&](int k) { return k >= 0 && 8 * k < len && column_state(tid + (k - j) * cols, cols) < 0; };
        if (8 * j < len && e < 0 && !todo(j - 1) && !todo(j - 2)) {
            int k = j + 1;
            for (;;) {
                if (todo(k)) k++;
                else if (todo(k + 1)) k += 2;
                else break;
            }
            list(line, a0 + 8 * j, min(8 * k, len) - 8 * j);
        }
    }

    // ---- packed stretches ----
    // The thread's place among the list's next stretches, as many as fit in the block; false when the
    // list is empty or (unless `all`) would leave a quarter of the threads idle.
    __device__ __forceinline__ bool pack(bool all, Spot& p, int& centre)
    {
        const int tid = threadIdx.x, lane = tid & 31;
        const uint32_t head = sh.head;
        const int left = (int)(sh.tail[parity] - head);
        if (left == 0) return false;
        // every warp packs for itself: inclusive sums of the next 32 stretches' threads
        Stretch s{0, 0};
        int need = 1 << 20;
        if (lane < left) {
            s = sh.list[(head + lane) % kTileList];
            need = (s.start_len & 255) + 2 * H;
        }
        int sum = need;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += v;
        }
        const int take = __popc(__ballot_sync(0xffffffffu, sum <= kTileThreads));
        if (!all && take == left && __shfl_sync(0xffffffffu, sum, take - 1) < kTileThreads * 3 / 4) return false;
        int k;
        p.in = pack_place(tid, take, [&](int j) { return __shfl_sync(0xffffffffu, sum, j); },
                          [&](int j) { return __shfl_sync(0xffffffffu, need, j); }, k, p.q);
        const int line = __shfl_sync(0xffffffffu, s.line, k);
        const int sl = __shfl_sync(0xffffffffu, s.start_len, k);
        p.hint = -1;
        p.width = (sl & 255) + 2 * H;
        p.t = (sl >> 8) - H + p.q;
        p.base = A.origin + (int64_t)line * A.geom[axis].lstride;
        centre = (__shfl_sync(0xffffffffu, s.start_len, 0) & 255) / 2 + H;
        __syncthreads();         // before sh.head or the entries are written again
        if (tid == 0) sh.head = head + take;
        return true;
    }

    // ---- compute ----
    // The kept-state slot that the centre thread's state may take, -1 when it should not be recorded:
    // its window is not real and uniform, or the state is kept already.  Run by the centre's warp.
    __device__ __forceinline__ int claim_slot(const AxisGeom<T>& g, const Spot& p, const CellIn<T>& c, int centre)
    {
        const int lane = threadIdx.x & 31, from = centre & 31;
        const int tc = __shfl_sync(0xffffffffu, p.t, from);
        const int in = __shfl_sync(0xffffffffu, (int)p.in, from);
        if (!in || tc - H < 0 || tc + H >= g.n) return -1;
        const int64_t bc = __shfl_sync(0xffffffffu, (long long)p.base, from);
        CellIn<T> u;
        u.rho = __shfl_sync(0xffffffffu, c.rho, from);
        u.ua = __shfl_sync(0xffffffffu, c.ua, from);
        u.uo = __shfl_sync(0xffffffffu, c.uo, from);
        u.E = __shfl_sync(0xffffffffu, c.E, from);
        bool same = true;
        if (lane <= 2 * H) {
            CellIn<T> o;
            load(bc + (int64_t)(tc - H + lane) * g.s, o);
            same = same_state(o, u);
        }
        if (!__all_sync(0xffffffffu, same)) return -1;
        const int v0 = sh.valid[0], v1 = sh.valid[1];
        if ((v0 && same_as_kept(u, 0)) || (v1 && same_as_kept(u, 1))) return -1;
        const int s = !v0 ? 0 : !v1 ? 1 : sh.turn;
        __syncwarp();
        if (lane == 0) {
            sh.valid[s] = 0;
            sh.turn = s ^ 1;
            sh.claims++;
        }
        __syncwarp();
        return s;
    }

    // The stages at the thread's position; ds threads between neighbouring positions.  The centre
    // thread records its state when it can.  Returns sh.claims as every thread of the block sees it: read
    // between the barrier that follows this call's claim and the ones before the next call's.  (Nothing
    // else that a claim writes, sh.turn and sh.kept among it, may decide a branch between two calls: the
    // centre's warp may be in the next one already, and warps that disagree meet different barriers.)
    __device__ __forceinline__ int compute(const AxisGeom<T>& g, const Spot& p, const int ds, const int centre)
    {
        const int tid = threadIdx.x;
        const T dx = g.dx;
        const int q = p.q, width = p.width;
        const bool on = p.in;
        const bool own = on && q >= H && q < width - H;
        T* X = &sh.ex[0][tid];
#define ARMON_X(slot) X[(slot) * kTileThreads]
#define ARMON_AT(slot, off) X[(slot) * kTileThreads + (off)]
        int rec = -1;

        // ---- cell: load, mirror, EOS ----
        CellIn<T> c{};
        if (on) {
            int m, side;
            const bool stale = source(g.n, p.t, m, side);
            const int64_t i = p.base + (int64_t)m * g.s;
            if (SCAN && p.hint >= 0) {
                const T* v = A.hints->v[src][p.hint];
                c.rho = __ldcg(v);
                c.ua = __ldcg(v + 1 + axis);
                c.uo = __ldcg(v + 2 - axis);
                c.E = __ldcg(v + 3);
            } else {
                load(i, c);
            }
            mirror(g, c, side);
            if (stale) {
                c.p = A.pmat[i];
                c.c = A.cmat[i];
            } else {
                eos(c, A.gamma, A.gamma - 1);
                if (pcg && own && p.hint < 0) {
                    A.pmat[i] = c.p;
                    A.cmat[i] = c.c;
                    A.gmat[i] = (1 + A.gamma) / 2;
                }
            }
            c.rc = qmul<1>(c.rho, c.c);
            c.rcu = qmul<1>(c.rc, c.ua);
            c.dm = mul_dx(c.rho, g);
            ARMON_X(9) = c.rc;
            ARMON_X(10) = c.rcu;
            ARMON_X(11) = c.p;
            ARMON_X(12) = c.ua;
            ARMON_X(13) = c.dm;
            sh.c[tid] = c.c;
        }
        if (SCAN && A.reuse && g.tile_scan) {
            if (p.hint >= 0) {
                if (on && q == H && width == 2 * H + 1) rec = p.hint;
            } else if ((tid >> 5) == (centre >> 5)) {
                rec = claim_slot(g, p, c, centre);
                if (tid != centre) rec = -1;
            }
            if (rec >= 0) {
                T* const rv = sh.kept[rec];
                rv[kRunRho] = c.rho; rv[kRunUa] = c.ua; rv[kRunUo] = c.uo; rv[kRunE] = c.E;
                rv[kRunP] = c.p; rv[kRunC] = c.c;
            }
        }
        __syncthreads();
        const int claims = sh.claims;

        // ---- Godunov face q (between positions q - 1 and q) ----
        God<T> G{};
        GadDiff<T> D{};
        if (on && q >= 1) {
            CellIn<T> cl{};
            cl.rc = ARMON_AT(9, -ds);
            cl.rcu = ARMON_AT(10, -ds);
            cl.p = ARMON_AT(11, -ds);
            cl.ua = ARMON_AT(12, -ds);
            G = godunov(cl, c);
            if (kGAD) {
                D = gad_diff(G, cl, c);
                ARMON_X(5) = D.au;
                ARMON_X(6) = D.bu;
                ARMON_X(7) = D.ap;
                ARMON_X(8) = D.bp;
            }
        }
        if (kGAD) __syncthreads();

        // ---- flux at face q ----
        Flux<T> F{};
        if (on && (kGAD ? (q >= 2 && q <= width - 2) : q >= 1)) {
            if (kGAD) {
                GadDiff<T> Dm{}, Dp{};
                Dm.bu = ARMON_AT(6, -ds);
                Dm.bp = ARMON_AT(8, -ds);
                Dp.au = ARMON_AT(5, ds);
                Dp.ap = ARMON_AT(7, ds);
                F = gad(G, Dm, D, Dp, ARMON_AT(13, -ds), c.dm, A.limiter, dt);
            } else {
                F.us = G.us;
                F.ps = G.ps;
            }
            F.psus = qmul<4>(F.ps, F.us);
            F.dtus = qmul<4>(dt, F.us);
            ARMON_X(0) = F.us;
            ARMON_X(1) = F.ps;
            ARMON_X(2) = F.psus;
            ARMON_X(3) = F.dtus;
        }
        __syncthreads();

        // ---- Lagrangian cell q (faces q and q + 1) ----
        Lag<T> L{};
        const bool has_lag = on && q >= kLagLo && q <= width - 1 - kLagLo;
        if (has_lag) {
            Flux<T> F1{};
            F1.us = ARMON_AT(0, ds);
            F1.ps = ARMON_AT(1, ds);
            F1.psus = ARMON_AT(2, ds);
            L = lagrange(c, F, F1, dt, dx);
            ARMON_X(4) = L.rho;
            ARMON_X(5) = L.rua;
            ARMON_X(6) = L.ruo;
            ARMON_X(7) = L.rE;
            ARMON_X(8) = L.W;
        }
        __syncthreads();

        // ---- differences of adjacent Lagrangian cells, which two faces share ----
        if (kE2) {
            if (has_lag && q >= kLagLo + 1) {
                Lag<T> Lm{};
                Lm.rho = ARMON_AT(4, -ds);
                Lm.rua = ARMON_AT(5, -ds);
                Lm.ruo = ARMON_AT(6, -ds);
                Lm.rE = ARMON_AT(7, -ds);
                const Adv<T> d = lag_diff(Lm, L);
                ARMON_X(9) = d.r;
                ARMON_X(10) = d.ra;
                ARMON_X(11) = d.ro;
                ARMON_X(12) = d.rE;
                ARMON_X(13) = ARMON_AT(8, -ds) + L.W;
            }
            __syncthreads();
        }

        // ---- advection flux at face q ----
        Adv<T> a{};
        if (on && q >= H && q <= width - H) {
            const T disp = F.dtus;
            const bool up = qgt0(disp);
            const int o = up ? -ds : 0;       // the upwind cell
            if (kE2) {
                const T Dx = qneg_if(dx + (up ? qneg_if(ARMON_AT(3, -ds), true) : ARMON_AT(3, ds)), up);
                const Adv<T> u0{ARMON_AT(4, o), ARMON_AT(5, o), ARMON_AT(6, o), ARMON_AT(7, o)};
                const Adv<T> dm{ARMON_AT(9, o), ARMON_AT(10, o), ARMON_AT(11, o), ARMON_AT(12, o)};
                const int o1 = o + ds;
                const Adv<T> dp{ARMON_AT(9, o1), ARMON_AT(10, o1), ARMON_AT(11, o1), ARMON_AT(12, o1)};
                a = advect2_upwind(disp, Dx, ARMON_AT(8, o), u0, dm, dp, ARMON_AT(13, o), ARMON_AT(13, o1));
            } else {
                a.r = qmul<6>(disp, ARMON_AT(4, o));
                a.ra = qmul<6>(disp, ARMON_AT(5, o));
                a.ro = qmul<6>(disp, ARMON_AT(6, o));
                a.rE = qmul<6>(disp, ARMON_AT(7, o));
            }
            ARMON_X(0) = a.r;
            ARMON_X(1) = a.ra;
            ARMON_X(2) = a.ro;
            ARMON_X(14) = a.rE;
        }
        if (rec >= 0) sh.valid[rec] = p.hint >= 0 ? 3 : 1;    // its results follow; they are read after the next unit's first barrier
        __syncthreads();

        // ---- projection of cell q (src/kernels/euler_projection.cpp:36-46) ----
        if (own) {
            const T dXr = qmul<7>(L.W, L.rho);
            T o[4];
            o[0] = div_dx(dXr - (ARMON_AT(0, ds) - a.r), g);
            const T ra = div_dx(qmul<7>(dXr, L.ua) - (ARMON_AT(1, ds) - a.ra), g);
            const T ro = div_dx(qmul<7>(dXr, L.uo) - (ARMON_AT(2, ds) - a.ro), g);
            const T rE = div_dx(qmul<7>(dXr, L.E) - (ARMON_AT(14, ds) - a.rE), g);
            const auto inv_rho = qrecip_at<8>(o[0]);
            o[1] = qdiv_at<8>(ra, inv_rho);
            o[2] = qdiv_at<8>(ro, inv_rho);
            o[3] = qdiv_at<8>(rE, inv_rho);
            if (!SCAN || p.hint < 0) {
                const int64_t i = p.base + (int64_t)p.t * g.s;
                T* const* out = A.buf[src ^ 1];
                out[0][i] = o[0];
                out[1 + axis][i] = o[1];
                out[2 - axis][i] = o[2];
                out[3][i] = o[3];
                if (last) add_dt(o, sh.c[tid]);
            } else if (rec < 0) {
                T* const wv = sh.kept[p.hint] + (p.t < H ? kRunWall + 4 * p.t : kRunWall + 16 + 4 * (p.t - (g.n - H)));
                wv[0] = o[0]; wv[1] = o[1]; wv[2] = o[2]; wv[3] = o[3];
            }
            if (rec >= 0) {
                T* const rv = sh.kept[rec];
                rv[kRunOut] = o[0]; rv[kRunOut + 1] = o[1]; rv[kRunOut + 2] = o[2]; rv[kRunOut + 3] = o[3];
                // a run of this state is one of its results for the next pass
                TileHints<T>* h = A.hints;
                T* v = h->v[src ^ 1][rec];
                v[0] = o[0];
                v[1 + axis] = o[1];
                v[2 - axis] = o[2];
                v[3] = o[3];
                h->valid[src ^ 1][rec] = 1;
            }
        }
#undef ARMON_X
#undef ARMON_AT
        return claims;
    }
};

// Adds the block's dt maxima to the domain's (max_x, max_y of its state).  Every thread calls it.
template <class T>
__device__ __forceinline__ void tile_flush(TileShared<T>& sh, StepState* state)
{
    __shared__ unsigned long long red[2];
    const int tid = threadIdx.x;
    if (tid < 2) red[tid] = 0;
    __syncthreads();
    DtAcc acc = sh.acc[tid];
    acc.finish();
    for (int o = 16; o > 0; o >>= 1)
        acc.merge(__shfl_xor_sync(0xffffffffu, acc.ax, o), __shfl_xor_sync(0xffffffffu, acc.ay, o));
    if ((tid & 31) == 0) {
        // maxima of non-negative, non-NaN values: the order of the bit patterns
        atomicMax(&red[0], (unsigned long long)__double_as_longlong(acc.ax));
        atomicMax(&red[1], (unsigned long long)__double_as_longlong(acc.ay));
    }
    __syncthreads();
    if (tid == 0) {
        if (red[0] > __ldcg((const unsigned long long*)&state->max_x)) atomicMax((unsigned long long*)&state->max_x, red[0]);
        if (red[1] > __ldcg((const unsigned long long*)&state->max_y)) atomicMax((unsigned long long*)&state->max_y, red[1]);
    }
    sh.acc[tid].init();
}

// The end of a cycle for one domain: dt_CFL, time and cycle (run by one thread when every block of the
// launch has added its maxima).
static __device__ __forceinline__ void tile_commit(StepState* state, const StepConfig& cfg)
{
    StepState st;
    st.time = __ldcg(&state->time);
    st.current_dt = __ldcg(&state->current_dt);
    st.next_dt = __ldcg(&state->next_dt);
    st.raw_dt = __ldcg(&state->raw_dt);
    st.cycle = __ldcg(&state->cycle);
    st.status = __ldcg(&state->status);
    st.counter = 0;
    st.buf_base = __ldcg(&state->buf_base);
    const double ax = __longlong_as_double((long long)__ldcg((const unsigned long long*)&state->max_x));
    const double ay = __longlong_as_double((long long)__ldcg((const unsigned long long*)&state->max_y));
    const CycleDt cd = cycle_time_step(st, cfg);
    if (!cd.run || cd.invalid) return;
    st.raw_dt = dt_from_maxima(ax, ay, cfg.dt_dx, cfg.dt_dy);
    st.current_dt = cd.current;
    st.next_dt = cd.next;
    st.time += cd.current;
    st.cycle += 1;
    st.max_x = st.max_y = 0;
    *state = st;
}

// Whether this block is the launch's last to get here; resets the launch's counters then.
__device__ __forceinline__ bool tile_arrive(TileCtl* ctl)
{
    __shared__ int is_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        is_last = atomicAdd(&ctl->arrived, 1u) == gridDim.x - 1;
        __threadfence();
        if (is_last) {
            ctl->ticket = 0;
            ctl->arrived = 0;
            ctl->dealt = 0;
            __threadfence();
        }
    }
    __syncthreads();
    return is_last != 0;
}

// The hints this pass has used are written again by the next.
template <class T>
__device__ __forceinline__ void tile_clear_hints(const SweepArgs<T>& A, int src)
{
    A.hints->valid[src][0] = A.hints->valid[src][1] = 0;
}

template <class T>
__device__ __forceinline__ void tile_forget(TileShared<T>& sh)
{
    if (threadIdx.x == 0) {
        sh.valid[0] = sh.valid[1] = 0;
        sh.turn = sh.claims = 0;
        sh.head = sh.tail[0] = sh.tail[1] = 0;
        sh.uniform[0] = sh.uniform[1] = 0;
    }
}

// One domain.
template <class T, int SCHEME, int PROJ, bool SCAN>
__global__ void __launch_bounds__(kTileThreads, tile_min_blocks<T>())
tile_kernel(const __grid_constant__ SweepArgs<T> A, TileCtl* ctl, int last)
{
    __shared__ TileShared<T> sh;
    TilePass<T, SCHEME, PROJ, SCAN> P(A, sh);
    tile_forget(sh);
    sh.acc[threadIdx.x].init();
    const bool ran = P.start(A.pass, last != 0, blockIdx.x == 0 && threadIdx.x == 0);
    if (ran) {
        const int total = A.geom[P.axis].tile_units;
        __syncthreads();
        int u = blockIdx.x;
        while (u < total) {
            u = P.unit(u, total, [&]() {
                return total > (int)gridDim.x ? (int)(gridDim.x + atomicAdd(&ctl->ticket, 1u)) : total;
            });
        }
        if (last) tile_flush(sh, A.state);
    }
    if (tile_arrive(ctl) && threadIdx.x == 0) {
        if (ran) tile_clear_hints(A, P.src);
        if (last) tile_commit(A.state, A.cfg);
    }
}

// Many independent domains in one launch (batch.cu).  Blocks [first[d], first[d + 1]) start on domain d,
// in proportion to its cells, so that a block keeps the states of one domain; a domain's units beyond
// its blocks' first ones come from its own ticket counter.  A block that finds its domain's units
// taken is dealt the next of the domains that no block started on (`rest`, `nrest` of them), and when
// those are all under way joins the domain with the most units left, blocks starting their search
// apart so that domains with equally many left get one each.  The last block to finish commits every domain.
// A small domain is a few units, so with thousands of them the search would be most of a pass, and
// blocks that search at once would find the same domain: 8000 domains of 16 to 32 cells a side, 40
// cycles, take 40 ms in FP32 (190 in FP64), against 1238 (1162) when every domain was searched for and
// 80 (518) with marches.
template <class T, int SCHEME, int PROJ>
__global__ void __launch_bounds__(kTileThreads, tile_min_blocks<T>())
tile_batch_kernel(const SweepArgs<T>* __restrict__ doms, const int* __restrict__ first, const int* __restrict__ units,
                  const int* __restrict__ rest, int nrest, uint32_t* __restrict__ tickets, int ndom, int pass, TileCtl* ctl,
                  int last)
{
    __shared__ TileShared<T> sh;
    __shared__ __align__(16) SweepArgs<T> sA;
    __shared__ unsigned long long pick;
    const int tid = threadIdx.x;
    TilePass<T, SCHEME, PROJ, true> P(sA, sh);
    sh.acc[tid].init();
    int d = batch_domain_index(first, ndom, blockIdx.x);
    int u = (int)blockIdx.x - first[d];
    for (;;) {
        // the domain's arguments in shared memory: read once, and not aliased by the stores
        __syncthreads();
        {
            static_assert(sizeof(SweepArgs<T>) % 4 == 0, "word copy");
            const int* s = reinterpret_cast<const int*>(&doms[d]);
            int* t = reinterpret_cast<int*>(&sA);
            for (int w = tid; w < (int)(sizeof(SweepArgs<T>) / 4); w += kTileThreads) t[w] = s[w];
        }
        tile_forget(sh);
        __syncthreads();
        const int total = units[d];
        const int given = first[d + 1] - first[d];
        uint32_t* ticket = &tickets[d];
        if (u < total) {
            if (P.start(pass, last != 0, tid == 0)) {
                while (u < total)
                    u = P.unit(u, total, [&]() { return (int)(given + atomicAdd(ticket, 1u)); });
                if (last) tile_flush(sh, sA.state);
            } else if (tid == 0) {
                atomicMax(ticket, (uint32_t)total);      // nothing to do here: no block joins it
            }
        }
        // the next domain of the list
        __syncthreads();
        int dealt = nrest;
        if (nrest > 0) {
            if (tid == 0) pick = __ldcg(&ctl->dealt) < (uint32_t)nrest ? atomicAdd(&ctl->dealt, 1u) : (uint32_t)nrest;
            __syncthreads();
            dealt = (int)pick;
            __syncthreads();
        }
        if (dealt < nrest) {
            d = rest[dealt];
        } else {
            // the domain with the most units left, the first from `from` on among equals
            const int from = (int)((uint64_t)blockIdx.x * ndom / gridDim.x);
            if (tid == 0) pick = 0;
            __syncthreads();
            unsigned long long best = 0;
            for (int k = tid; k < ndom; k += kTileThreads) {
                const int left = units[k] - (first[k + 1] - first[k]) - (int)min(__ldcg(&tickets[k]), 0x3fffffffu);
                const int behind = k >= from ? k - from : k + ndom - from;
                if (left > 0) best = max(best, (unsigned long long)left << 32 | (unsigned)(ndom - behind));
            }
            if (best != 0) atomicMax(&pick, best);
            __syncthreads();
            if (pick == 0) break;
            d = from + ndom - (int)(uint32_t)pick;
            if (d >= ndom) d -= ndom;
            __syncthreads();
        }
        if (tid == 0) pick = atomicAdd(&tickets[d], 1u);
        __syncthreads();
        u = first[d + 1] - first[d] + (int)(uint32_t)pick;
    }
    if (tile_arrive(ctl)) {
        for (int k = tid; k < ndom; k += kTileThreads) {
            const SweepArgs<T>& A = doms[k];
            tickets[k] = 0;
            StepState st;
            st.time = __ldcg(&A.state->time);
            st.next_dt = __ldcg(&A.state->next_dt);
            st.raw_dt = __ldcg(&A.state->raw_dt);
            st.cycle = __ldcg(&A.state->cycle);
            st.status = __ldcg(&A.state->status);
            st.buf_base = __ldcg(&A.state->buf_base);
            const CycleDt cd = cycle_time_step(st, A.cfg);
            if (!cd.run || cd.invalid) continue;
            tile_clear_hints(A, (int)(((int64_t)st.cycle * A.npass + pass + st.buf_base) & 1));
            if (last) tile_commit(A.state, A.cfg);
        }
    }
}

}  // namespace armon
