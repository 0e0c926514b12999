// Work split and data movement of the flux passes (both precisions): a unit --
// a warp, or on small grids a block -- takes chunks of one or two scheduled
// tiles, stages a tile's rows in shared memory and computes its points four a
// warp round, eight lanes a point.
#pragma once

#include "batch.cuh"
#include "halo.cuh"

namespace lskum {

constexpr int LPP = 8;                       // lanes per point
constexpr int PPW = 32 / LPP;                // points per warp round
constexpr int FLUX_BLOCK = 128;              // four warps
constexpr int FLUX_WARPS = FLUX_BLOCK / 32;
constexpr int CHUNK_MAX = 2 * TILE;          // points of a chunk

// The small grids' D and I passes: a point's eight lanes leave their slots'
// fields in shared memory, SLOT_F elements a field and SLOT_P a point, so that
// a warp's stores and loads fall on distinct banks.
constexpr int SLOT_BLOCK = 128, SLOT_PTS = SLOT_BLOCK / LPP, SLOT_F = 9, SLOT_P = 68;
__device__ __forceinline__ int slot_point(const Sched &s, const SchedSmem &ss, int total, int vp) {
    return vp < total ? sched_point(s, ss, vp) : -1;
}

// Sum of v over the eight lanes of a point: component 2 (bit 2) + (bit 1) of
// the lane, in a fixed order.
__device__ __forceinline__ double reduce8(const double v[4], int lane) {
    const unsigned full = 0xffffffffu;
    const bool h4 = lane & 4, h2 = lane & 2;
    const double s0 = __shfl_xor_sync(full, h4 ? v[0] : v[2], 4);
    const double s1 = __shfl_xor_sync(full, h4 ? v[1] : v[3], 4);
    const double a0 = (h4 ? v[2] : v[0]) + s0, a1 = (h4 ? v[3] : v[1]) + s1;
    const double b = (h2 ? a1 : a0) + __shfl_xor_sync(full, h2 ? a0 : a1, 2);
    return b + __shfl_xor_sync(full, b, 1);
}

// A scheduled tile: its first point, the points in it (0: no such tile), and
// the numbers of its points up to which they are wall and outer points.
struct FluxTile {
    int i0 = 0, cnt = 0, wall = 0, outer = 0, tile = 0;
    __device__ __forceinline__ FluxTile() {}
    __device__ __forceinline__ FluxTile(const Sched &s, int ntiles, int v) {
        if (v >= ntiles) return;
        const TileRef t = sched_tile_global(s, v);
        i0 = t.base + t.j0;
        cnt = min(TILE, t.n - t.j0);
        wall = t.nw - t.j0;
        outer = t.nw + t.no - t.j0;
        tile = t.tile;
    }
    __device__ __forceinline__ int kind(int j) const {
        return j < wall ? KIND_WALL : (j < outer ? KIND_OUTER : KIND_INTERIOR);
    }
};

// The row indices of a tile's halo: lane l holds rows l and l + 32.
struct FluxHalo {
    int h0 = 0, hn = 0, k0 = 0, k1 = 0;  // hn 0: no tile, or not staged
    __device__ __forceinline__ void range(const Geom &g, const FluxTile &t) {
        h0 = hn = 0;
        if (t.cnt == 0) return;
        h0 = __ldg(g.hoff + t.tile);
        hn = __ldg(g.hoff + t.tile + 1);
    }
    // most: the rows shared memory holds
    __device__ __forceinline__ void rows(const Geom &g, int lane, int most) {
        hn = hn - h0 <= most ? hn - h0 : 0;
        k0 = lane < hn ? __ldg(g.hrow + h0 + lane) : 0;
        k1 = lane + 32 < hn ? __ldg(g.hrow + h0 + 32 + lane) : 0;
    }
    // row u (u / 32 the same for the whole warp)
    __device__ __forceinline__ int row(int u) const {
        return __shfl_sync(0xffffffffu, u < 32 ? k0 : k1, u & 31);
    }
};

// Copies NP 16-byte pieces of every halo row of an array with the NT threads
// of the unit, tid of them this one; whole warps.  HC: stride of the arrays.
template <int NP, int NT, int HC>
__device__ __forceinline__ void stage_rows(const void *src, const FluxHalo &x, double2 *dst,
                                           int tid) {
#pragma unroll
    for (int t = 0; t < (HALO_CAP * NP + NT - 1) / NT; ++t) {
        if (NT * t >= NP * x.hn) break;
        const int u = (NT / NP) * t + tid / NP, part = tid % NP;
        const int k = x.row(u);
        if (u < x.hn)
            halo_cp16(dst + part * HC + u,
                      static_cast<const char *>(src) + (size_t)(unsigned)(k * NP + part) * 16);
    }
}

// Copies what both precisions keep of the tile's own points: (nx, ny), the
// membership masks, the local rows and the stencil size.
struct FluxOwn {
    double2 nrm[TILE];
    uint4 mask[TILE];              // xpos, xneg, ypos, yneg
    unsigned char loc[TILE * 16];  // hloc rows (of up to 16 bytes)
    int nbhs[TILE];
    template <int NT>
    __device__ __forceinline__ void stage(const Geom &g, const FluxTile &t, int tid) {
        if (g.hkp <= 16 && tid < g.hkp / 8 * t.cnt)
            halo_cp8(loc + 8 * tid, g.hloc + (size_t)t.i0 * g.hkp + 8 * tid);
        if (tid < 2 * TILE) {
            const int j = tid % TILE;
            if (j < t.cnt) {
                double *d = reinterpret_cast<double *>(&mask[j]);
                if (tid < TILE) {
                    halo_cp16(&nrm[j], g.nrm + t.i0 + j);
                    halo_cp8(d, g.mx + t.i0 + j);
                } else {
                    halo_cp4(&nbhs[j], g.nbhs + t.i0 + j);
                    halo_cp8(d + 1, g.my + t.i0 + j);
                }
            }
        }
    }
    // local rows of slot r's neighbour and of point j (global index i) itself
    __device__ __forceinline__ void rows(const Geom &g, int i, int j, int r, int &lk,
                                         int &li) const {
        const unsigned char *gl = g.hloc + (size_t)i * g.hkp, *ml = loc + j * g.hkp;
        const bool in = g.hkp <= 16;
        lk = in ? ml[r] : __ldg(gl + r);
        li = in ? ml[g.hkp - 1] : __ldg(gl + g.hkp - 1);
    }
};

// A flux pass over chunks of `ct` (1 or 2) scheduled tiles.  coop = 0: a warp
// owns a chunk, computes its points four at a time and updates them with one
// lane each, with no block barrier.  coop = 1: the block's four warps share a
// chunk (each a quarter of its points) and its first warp updates it.  Both
// call the same functions on a point, so the split does not change a result.
// A tile never straddles two instances and its partial lands in slot
// (instance's first tile + tile number), summed over its 16 points in point
// order, so an instance's residual sums do not depend on the other instances
// or on the launch shape.
//
// A tile's rows come through shared memory: its halo (54 rows a 16-point tile
// of an O-grid, against 144 row reads) is copied with cp.async, the next
// tile's while this chunk's points are updated, the row indices a tile ahead.
//
// P: the pass.  P::Smem: the unit's shared memory, with ROWS halo rows and the
// chunk's flux residuals G.  stage<NT>(tile, halo, smem, tid); group(tile, j,
// halo rows, smem, G[j]): point j of the tile by eight lanes; update(i, kind,
// outer row, G[j]): its new state, returns its res_sqr term.
template <class P>
__device__ __forceinline__ void flux_pass(P &p, const Geom &g, const Sched &s,
                                          typename P::Smem *sm, double *res_part, int last, int ct,
                                          int coop) {
    const int live = __ldg(s.nact), ntiles = s.single ? s.one.ntiles : __ldg(s.pre + live);
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    typename P::Smem &m = sm[coop ? 0 : warp];
    constexpr int ROWS = P::Smem::ROWS;
    const int nchunks = (ntiles + ct - 1) / ct, pts = ct * TILE;
    const int jw = coop ? warp * PPW : 0, nj = coop ? PPW : TILE;  // the warp's points of a tile
    const int step = coop ? gridDim.x : gridDim.x * FLUX_WARPS;
    int ch = coop ? blockIdx.x : blockIdx.x * FLUX_WARPS + warp, u = 0;
    if (ch >= nchunks) return;  // (coop: the whole block)
    FluxTile cur(s, ntiles, ct * ch);
    FluxHalo hx;
    hx.range(g, cur);
    hx.rows(g, lane, ROWS);
    if (!live) return;  // (retired)
    auto stage = [&] {
        if (coop) p.template stage<FLUX_BLOCK>(cur, hx, m, threadIdx.x);
        else p.template stage<32>(cur, hx, m, lane);
    };
    auto sync = [&] {
        if (coop) __syncthreads();
        else __syncwarp();
    };
    stage();
    while (true) {
        const int hn = hx.hn, done = ct * ch;  // the chunk's first tile
        const bool end = u + 1 == ct;
        if (end) ch += step;
        // the tile after this one: its halo's range now, its row indices once
        // that has come (after the first round)
        const FluxTile nxt(s, ntiles, end ? ct * ch : done + u + 1);
        hx.range(g, nxt);
        halo_wait();
        sync();
        for (int rnd = 0; rnd < nj; rnd += PPW) {
            const int j = jw + rnd + lane / LPP;
            p.group(cur, j, hn, m, m.G[u * TILE + j]);
            if (rnd == 0) hx.rows(g, lane, ROWS);
        }
        sync();
        // the next tile's rows are on their way while this chunk is updated
        cur = nxt;
        stage();
        u = end ? 0 : u + 1;
        if (!end) continue;
        // the chunk's state updates, one point per lane
        if (!coop || warp == 0) {
            const int v = done + lane / TILE;
            const bool tile = lane < pts && v < ntiles;
            const TileRef t = sched_tile_global(s, tile ? v : done);
            const int j = t.j0 + (lane % TILE);
            double rs = 0.0;
            if (tile && j < t.n) {
                const int kind =
                    j < t.nw ? KIND_WALL : (j < t.nw + t.no ? KIND_OUTER : KIND_INTERIOR);
                rs = p.update(t.base + j, kind, t.obc_off + j - t.nw, m.G[lane]);
            }
            if (last) {
                m.G[lane][0] = rs;
                __syncwarp();
                if ((lane % TILE) == 0 && tile) {
                    double acc = 0.0;
                    for (int q = 0; q < TILE; ++q) acc = acc + m.G[lane + q][0];
                    res_part[t.tile] = acc;
                }
            }
        }
        if (ch >= nchunks) break;
    }
}

}  // namespace lskum
