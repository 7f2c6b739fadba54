// jp_cells.cu -- device cell-list build and pair-tile list (replaces md_run celprp/celpar/
// cutoff: src_md_run/celprp.f90:2-175, celpar.f90:2-244, cutoff.f90:2-505).
//
// Pipeline (every UPDATE steps, all replicas in one pass):
//   1. k_cell_key      radix binning: wrapped position -> fine cell -> Morton key per replica
//   2. scan            counting-sort offsets (deterministic exclusive scan)
//   3. k_scatter       atoms to their bins; blocks per column
//   4. k_fill_slots    compact order -> 32-atom blocks padded per replica
//   5. k_block_setup   per-block bounding box, frame origin, block-local coordinates
//   6. k_block_list    one thread block per i-block: bounding-box tests of the later blocks,
//                      the exact 32x32 interaction mask of the survivors (r^2 <= (rc+1.5)^2 at
//                      build time, cutatm `dd .le. rlim2`, minus 1-2/1-3/1-4 partners,
//                      cutoff.f90:50-96), and the pair records of its two halves.
#include "jp_common.cuh"
#include "jp_kernels.h"

namespace jp {

// Binning: atoms go to xy columns of edge ~(32/density)^(1/3) (~6.8 A for water) and,
// inside a column, to 0.25 A z bins.  The key orders atoms by (replica, column, z), so each
// column's atoms are z-sorted and a column cut into runs of 32 gives near-cubic blocks.
__global__ void k_cell_key(DevPtrs P, int natom) {
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= natom) return;
  const Rep& R = P.reps[P.rep_of[a]];
  int c[3];
  bool out = false;
  for (int k = 0; k < 3; ++k) {
    const double x = P.x[3 * a + k];
    out |= R.free_bnd && !(x >= R.win_lo[k] && x <= R.win_hi[k]);
    const double w = x - R.box[k] * floor(x * R.invbox[k]);
    int q = (int)(w / R.cell[k]);
    c[k] = q < 0 ? 0 : (q >= R.grid[k] ? R.grid[k] - 1 : q);
  }
  if (out) atomicOr(P.status, ERR_FREE_WINDOW);
  const unsigned key = (unsigned)(R.key0 + (c[1] * R.grid[0] + c[0]) * R.grid[2] + c[2]);
  P.key[a] = key;
  P.rank[a] = atomicAdd(&P.hist[key], 1);
}

// an atom to its place of its bin; and the blocks each column needs: ceil(atoms in column / 32)
__global__ void k_scatter(DevPtrs P, int natom, int ncol) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a < natom) P.sorted[P.hist_scan[P.key[a]] + P.rank[a]] = a;
  if (a >= ncol) return;
  const Rep& R = P.reps[P.col_rep[a]];
  const int k0 = R.key0 + (a - R.col0) * R.grid[2];
  const int n = P.hist_scan[k0 + R.grid[2]] - P.hist_scan[k0];
  P.col_nb[a] = (n + kTile - 1) / kTile;
}

// what a list build starts from: empty bins and slots, no records, no block extents (a small
// system's build is a chain of launches of 2-4 us each: with this for six memsets and a launch,
// with the sort within bins, the column counts and the exclusion slots inside their
// neighbours' launches, 2,200 atoms took 80 us instead of 104, 22,700 atoms 118 instead of 141)
__global__ void k_list_reset(DevPtrs P, int nkeys, int nslot, int nrep, int dummy_type, int hbond) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i <= nkeys) P.hist[i] = 0;
  if (i < nslot) {
    P.satom[i] = -1;
    P.styp[i] = dummy_type;
  }
  if (i < 3 * nrep) P.rep_hmax[i] = 0.f;
  if (i < 3) P.nctiles[i] = 0;
  if (i == 0) *P.ext_pos = 0;
  if (i == 0 && hbond) *P.ntiles = 0;
}

// sorted position -> slot: block = replica's first block + blocks of the columns before this
// one (a column never shares a block with another), lane = rank inside the column
__global__ void k_fill_slots(DevPtrs P, int natom) {
  const int pos = blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= natom) return;
  const int a = P.sorted[pos];
  const Rep& R = P.reps[P.rep_of[a]];
  const int col = R.col0 + ((int)P.key[a] - R.key0) / R.grid[2];
  const int kcol = R.key0 + (col - R.col0) * R.grid[2];
  // within a bin (a few atoms) by ascending atom index, so that the order does not depend on the
  // arrival that k_cell_key counted
  const int bin = (int)P.key[a], b0 = P.hist_scan[bin], b1 = b0 + P.hist[bin];
  int place = b0;
  for (int q = b0; q < b1; ++q) place += P.sorted[q] < a ? 1 : 0;
  const int rank = place - P.hist_scan[kcol];
  const int blk = R.blk0 + (P.col_blk[col] - P.col_blk[R.col0]) + rank / kTile;
  const int slot = blk * kTile + (rank % kTile);
  P.slot_of[a] = slot;
  P.satom[slot] = a;
  P.styp[slot] = P.typ[a];
}

// one warp per block; the blocks from nsetup on: the slot of every exclusion partner (lets the
// tile build clear excluded pairs per partner instead of searching the partner list per pair)
__global__ void k_block_setup(DevPtrs P, int nblk, double qscale, int nsetup, int natom) {
  if ((int)blockIdx.x >= nsetup) {
    const int a = (blockIdx.x - nsetup) * blockDim.x + threadIdx.x;
    if (a < natom)
      for (int p = P.excl_ptr[a]; p < P.excl_ptr[a + 1]; ++p) P.excl_slot[p] = P.slot_of[P.excl_idx[p]];
    return;
  }
  // largest extents and replica of the thread block's warps: one atomic per replica among them
  // (with one per warp the blocks of 64 replicas waited for each other: a list build of theirs
  // took 2,364 us, and 2,303 so)
  __shared__ float s_h[kSetupWarps][3];
  __shared__ int s_rep[kSetupWarps];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int blk = blockIdx.x * kSetupWarps + w;
  if (lane == 0) s_rep[w] = -1;
  if (blk < nblk) {
    const int slot = blk * kTile + lane;
    const int a = P.satom[slot];
    const int r = P.blk_rep[blk];
    const Rep& R = P.reps[r];
    const int ty = P.styp[slot];
    const unsigned lj = __ballot_sync(0xffffffffu, a >= 0 && !P.lj_free[ty & kTypeMask]);
    const unsigned cls = __ballot_sync(0xffffffffu, a >= 0 && ((ty >> 30) & 1));
    if (lane == 0) P.blk_kind[blk] = make_uint2(lj, cls);
    double x[3] = {0, 0, 0}, img[3] = {0, 0, 0};
    double lo[3], hi[3], ref[3];
    for (int k = 0; k < 3; ++k) {
      if (a >= 0) {
        x[k] = P.x[3 * a + k];
        img[k] = floor(x[k] * R.invbox[k]);
        lo[k] = hi[k] = x[k] - R.box[k] * img[k];
      } else {
        lo[k] = 1e300;
        hi[k] = -1e300;
      }
    }
    for (int o = 16; o > 0; o >>= 1)
      for (int k = 0; k < 3; ++k) {
        lo[k] = fmin(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
        hi[k] = fmax(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
      }
    for (int k = 0; k < 3; ++k) ref[k] = 0.5 * (lo[k] + hi[k]);
    if (lane == 0) {
      P.blk_ref[3 * blk + 0] = ref[0];
      P.blk_ref[3 * blk + 1] = ref[1];
      P.blk_ref[3 * blk + 2] = ref[2];
      P.blk_ctr[blk] = make_float4((float)ref[0], (float)ref[1], (float)ref[2], 0.f);
      // an empty block (capacity not used this rebuild) gets a -inf extent: it never passes
      // the bounding-box test
      P.blk_half[blk] = make_float4((float)(0.5 * (hi[0] - lo[0])) + 1e-4f,
                                    (float)(0.5 * (hi[1] - lo[1])) + 1e-4f,
                                    (float)(0.5 * (hi[2] - lo[2])) + 1e-4f, 0.f);
      if (lo[0] <= hi[0]) {
        s_rep[w] = r;
        for (int k = 0; k < 3; ++k) s_h[w][k] = (float)(0.5 * (hi[k] - lo[k]));
      }
    }
    if (a >= 0) {
      double o[3];
      for (int k = 0; k < 3; ++k) {
        o[k] = ref[k] + R.box[k] * img[k];
        P.off[3 * a + k] = o[k];
      }
      const float q = (float)((double)qscale * P.chg[a]);
      P.pos_f[a] = make_float4((float)(x[0] - o[0]), (float)(x[1] - o[1]), (float)(x[2] - o[2]), q);
    }
  }
  __syncthreads();
  if (w == 0 && lane < kSetupWarps) {
    const unsigned all = (1u << kSetupWarps) - 1u;
    const int r = s_rep[lane];
    const unsigned same = __match_any_sync(all, r);
    for (int k = 0; k < 3; ++k) {   // (non-negative floats order like their bit patterns)
      const unsigned h = __reduce_max_sync(same, r >= 0 ? __float_as_uint(s_h[lane][k]) : 0u);
      if (r >= 0 && lane == __ffs(same) - 1) atomicMax(reinterpret_cast<int*>(&P.rep_hmax[3 * r + k]), (int)h);
    }
  }
}

// ---- pair list: one thread block per i-block ---------------------------------------------------
// k_block_list does everything that belongs to one 32-atom i-block: the bounding-box test of
// the later blocks of its replica, the exact 32x32 interaction mask of every survivor, and the
// pair records of its two halves.  The masks and what belongs to a tile stay in shared memory
// (in global memory beyond kTileCache tiles), and a unit's records are placed by one atomic
// counter: which records stand where varies from run to run, what a record holds does not, and
// the sums of the pair kernels do not depend on it.
// Before, a warp scanned 32 candidates one after the other, and eleven more launches (three
// scans of per-chunk counts, tile emit, unit counts, their scan, record index, record emit)
// passed the tiles on through memory.  A whole list build, before and now: 64 replicas 4,380 and
// 2,303 us, 99,200 atoms 534 and 344, 22,700 atoms 216 and 118, 2,200 atoms 196 and 80.  Its
// shared memory counts: 4.6 KB more a block took 64 replicas 170 us longer.
//
// Pair record: a half block (16 i atoms: rows 0-15 or 16-31 of an i-block, unit u = 2 i-block +
// half) with 32 j entries, the j atoms of that block's tiles that at least one of the 16 i
// atoms lists, by kind (below) and in tile order (ascending j block, ascending slot).
// A 32 x 32 tile of two blocks holds ~26 % listed pairs at the md_run list radius; keeping only the j atoms a half
// block lists raises that to ~55 %, because 16 atoms span a smaller volume than 32 (within the
// cut-off: 32 % of the slots with whole blocks, 39 % with half blocks), and the pair kernels'
// work per pair falls in proportion.  Each entry carries its tile's image shift (into the i
// block's frame) and its atom, with the atom's type beside it; the mask of i atom l (0..15)
// has bit k = entry (l + k) & 15 and bit 16 + k = entry 16 + ((l + k) & 15).

// The four kinds of entries (0 .. 3), in their order in the first half of a block (in the second
// half the other way round, so that a unit ends with the kind that the next one begins with): with
// an LJ term, without, and the same two, without first, of the entries that make a record take per-pair
// images or ALSD classes.  The pair kernels leave the LJ term out over eight entries of a
// warp's records that have none (in waters two thirds of the entries), and few records mix
// the forms.  Pair kernel (eight warps a block, an i atom's 32 terms in one sum) with entries
// in tile order and so: 64 replicas (883,000 atoms) 1,345 and 1,290 us, 99,200 atoms 181 and
// 166, 22,700 atoms 54 and 51.  With the LJ order alone the entries of image tiles, scattered
// over more records, cost 64 replicas more than it gave (1,480 us).
constexpr int kListWarps = 8;     // warps of a block, at most
constexpr int kTileListImg = 1 << 30, kTilePairImg = 1 << 29, kTileBlock = kTilePairImg - 1;   // BlkTile.j
constexpr int kSegment = 512;     // candidate blocks tested at a time
constexpr int kTileCache = 96;    // tiles of an i-block kept in shared memory (water: 65 on average)
constexpr int kNarrowTiles = 256; // tiles of an i-block whose entries go in 16 bits (which hold 2,048;
                                  // cut-offs that list more than 256 blocks are rare, and a system
                                  // of 8,000 atoms without a cut-off then meets both forms)
constexpr int kWindow = 40;       // records of a half emitted at a time (water: 27 on average)

struct __align__(16) ListShared {
  double x[kTile], y[kTile], z[kTile];     // the i block, wrapped
  union {
    // a candidate's live j atoms, compacted, two per element: x, x', y, y' and z, z', mask bits
    struct {
      float4 xy[kListWarps][kTile / 2], zb[kListWarps][kTile / 2];
    } l;
    // afterwards, entry -> tile << 5 | j lane of each half's window (beyond kNarrowTiles tiles in
    // 32 bits, half the window)
    unsigned short e16[2][kWindow * 32];
    unsigned e32[2][kWindow * 16];
  };
  unsigned ball[kSegment / 32];            // survivors of the bounding-box test
  unsigned excl[kSegment / 32];            // blocks that hold an exclusion partner
  int carry[8];                            // entries by half and kind
  int first[2][4];                         // a half's first entry of each kind
  int base[2];                             // of the records at the start and at the end
  int nimg;                                // ALSD: records at the start whose pairs take their own images
  // ALSD: which of a window's records hold a class but BB, and each one's place
  unsigned char rcls[2 * kWindow];
  size_t rpos[2 * kWindow];
  BlkTile tile[kTileCache];
};

// 1-2/1-3/1-4 partners (cutoff.f90:50-96) of this lane's i atom that sit in block bj out of its
// mask row: lane l sees slot bj * 32 + ((l + k) & 31) at bit k
__device__ __forceinline__ unsigned drop_excluded(const DevPtrs& P, int bj, int lane, int ai, unsigned mask) {
  if (ai >= 0)
    for (int p = P.excl_ptr[ai]; p < P.excl_ptr[ai + 1]; ++p) {
      const int sp = P.excl_slot[p];
      if ((sp >> 5) == bj) mask &= ~(1u << (((sp & 31) - lane) & 31));
    }
  return mask;
}

// (the two FP64 forms are out of line and take plain pointers: a reference to the kernel's
// parameter block would have it copied to local memory)
// General form of a tile's mask in FP64, per-pair minimum image: lane = i atom, bit k = j lane
// (lane + k) & 31.  CMM: level-1 cells ci / cj (packed 0-based x | y << 8 | z << 16, -1 = off the
// grid); neighbours (neartb.f90 first table) set mask and mel, cells up to idelay apart with
// r^2 < rc2 at the rebuild (neartb.f90:330-370, the LJ-only table) set mask only
template <bool CMM>
__device__ __noinline__ unsigned tile_mask(const int* satom, const double* x, const int* cmm_cell, const Rep& R, int bi,
                                           int bj, int lane, int ai, double rlim2, double rc2, unsigned& mel) {
  const int aj = satom[bj * kTile + lane];
  double xi = 0, yi = 0, zi = 0, xj = 0, yj = 0, zj = 0;
  int ci = -1, cj = -1;
  if (ai >= 0) {
    xi = x[3 * ai]; yi = x[3 * ai + 1]; zi = x[3 * ai + 2];
    if (CMM) ci = cmm_cell[ai];
  }
  if (aj >= 0) {
    xj = x[3 * aj]; yj = x[3 * aj + 1]; zj = x[3 * aj + 2];
    if (CMM) cj = cmm_cell[aj];
  }
  unsigned mask = 0;
  mel = 0;
  const double bx = R.box[0], by = R.box[1], bz = R.box[2];
  const double ibx = R.invbox[0], iby = R.invbox[1], ibz = R.invbox[2];
  const int idelay = R.idelay;
  for (int k = 0; k < 32; ++k) {
    const int src = (lane + k) & 31;
    const double xk = __shfl_sync(0xffffffffu, xj, src);
    const double yk = __shfl_sync(0xffffffffu, yj, src);
    const double zk = __shfl_sync(0xffffffffu, zj, src);
    const int ak = __shfl_sync(0xffffffffu, aj, src);
    const int ck = CMM ? __shfl_sync(0xffffffffu, cj, src) : 0;
    if (ai < 0 || ak < 0) continue;
    if (bj == bi && (k == 0 || k > 16 || (k == 16 && lane >= 16))) continue;
    int cheb = 0;
    if (CMM) {
      if (ci < 0 || ck < 0) continue;
      cheb = max(abs((ci & 255) - (ck & 255)),
                 max(abs(((ci >> 8) & 255) - ((ck >> 8) & 255)), abs((ci >> 16) - (ck >> 16))));
      if (cheb <= 1) {
        mask |= 1u << k;
        mel |= 1u << k;
        continue;
      }
      if (!(idelay > 1 && cheb <= idelay)) continue;
    }
    double dx = xi - xk, dy = yi - yk, dz = zi - zk;
    dx -= bx * anint(dx * ibx);
    dy -= by * anint(dy * iby);
    dz -= bz * anint(dz * ibz);
    const double d2 = dx * dx + dy * dy + dz * dz;
    if (CMM ? d2 < rc2 : d2 <= rlim2) mask |= 1u << k;
  }
  return mask;
}

// The FP64 form where the tile's image serves every listed pair (no CMM): lane = j atom; the i block is read from shared
// memory one atom per step (a broadcast) and a ballot gives that i atom's row of the tile at
// once; lane i keeps row i.  Coordinates are wrapped (x - box floor(x / box)) and the tile's
// image is the block references' minimum image n.
__device__ __noinline__ unsigned tile_row_fast(const int* satom, const double* xm, const double* blk_ref, const Rep& R,
                                               int bi, int bj, int lane, int ai, const ListShared& S,
                                               double rlim2) {
  const int aj = satom[bj * kTile + lane];
  double xj = 0.0, yj = 0.0, zj = 0.0;
  if (aj >= 0) {
    double w[3];
    for (int k = 0; k < 3; ++k) {
      const double x = xm[3 * aj + k];
      const double n = anint((blk_ref[3 * bi + k] - blk_ref[3 * bj + k]) * R.invbox[k]);
      w[k] = (x - R.box[k] * floor(x * R.invbox[k])) + R.box[k] * n;
    }
    xj = w[0]; yj = w[1]; zj = w[2];
  }
  unsigned row = 0;
#pragma unroll 8
  for (int i = 0; i < kTile; ++i) {
    const double dx = S.x[i] - xj, dy = S.y[i] - yj, dz = S.z[i] - zj;
    const bool in = aj >= 0 && dx * dx + dy * dy + dz * dz <= rlim2;
    const unsigned b = __ballot_sync(0xffffffffu, in);
    if (lane == i) row = b;
  }
  return ai >= 0 ? row : 0u;
}

// The exact list radius decides in FP64, but almost every pair is far from it: the mask is
// first built in FP32 on coordinates relative to the i block's reference (|x| <~ 25 A, so
// d^2 is good to ~3e-4 A^2), and a tile with any pair within `band` of rlim^2 is redone in
// FP64; the FP32 mask is returned only where every decision is certain, so the list is the
// FP64 list.  `unsure` is warp-uniform.
// Lane = i atom (xi, in its block's frame).  A j atom in the i frame is its block-local position
// pj (relative to its block's reference in the wrapped frame) plus c, block bj's reference
// shifted by the tiles' image into the i block's frame.  Only the j atoms within the list
// radius of the i block's bounding box (half extents hi; with a margin of 1e-4 rlim^2 +
// 1e-3 A^2, far wider than `band` and the FP32 rounding) can be listed, and the loop takes only
// them: compacted in shared memory with their mask bits, two per pass in packed arithmetic.
// (With a j atom a lane and the i atoms in the loop every pass also needed a ballot and a
// select per row: 24 instructions for two atoms, so 17.)
// PIMG (two blocks nearly half a small box apart): the tile's image is not every pair's, so each
// pair takes its own minimum image in FP32 and no j atom is culled.  Decided per tile: with one
// rule per replica from its largest block, boxes up to 51 A imaged every pair.
template <bool PIMG>
__device__ __forceinline__ unsigned tile_row_f32(const Rep& R, float3 c, float4 hi, int lane, float3 xi, bool ireal,
                                                 float4 pj, bool jreal, ListShared& S, float rlim2f, float band,
                                                 bool& unsure) {
  const unsigned full = 0xffffffffu;
  const int w = threadIdx.x >> 5;
  const float rx = pj.x + c.x, ry = pj.y + c.y, rz = pj.z + c.z;
  bool lv = jreal;
  if (!PIMG) {
    const float gx = fmaxf(fabsf(rx) - hi.x, 0.f);
    const float gy = fmaxf(fabsf(ry) - hi.y, 0.f);
    const float gz = fmaxf(fabsf(rz) - hi.z, 0.f);
    lv = lv && fmaf(gx, gx, fmaf(gy, gy, gz * gz)) <= rlim2f * 1.0001f + 1e-3f;
  }
  const unsigned live = __ballot_sync(full, lv);
  const int nlive = __popc(live);
  __syncwarp();   // the previous tile's passes are done with the compacted atoms
  {
    float* xy = reinterpret_cast<float*>(S.l.xy[w]);
    float* zb = reinterpret_cast<float*>(S.l.zb[w]);
    if (lv) {
      const int t = __popc(live & ((1u << lane) - 1u));
      const int o = 4 * (t >> 1) + (t & 1);
      xy[o] = rx;
      xy[o + 2] = ry;
      zb[o] = rz;
      zb[o + 2] = __uint_as_float(1u << lane);
    }
    if (lane == 0 && (nlive & 1)) {   // the odd one's partner lists nothing: no comparison holds for a NaN
      const int o = 4 * (nlive >> 1) + 1;
      xy[o] = xy[o + 2] = zb[o] = __int_as_float(0x7fffffff);
      zb[o + 2] = 0.f;
    }
  }
  __syncwarp();
  const float bx = (float)R.box[0], by = (float)R.box[1], bz = (float)R.box[2];
  const float ibx = (float)R.invbox[0], iby = (float)R.invbox[1], ibz = (float)R.invbox[2];
  const float2 nx = make_float2(-xi.x, -xi.x), ny = make_float2(-xi.y, -xi.y), nz = make_float2(-xi.z, -xi.z);
  const float2 ml = make_float2(-rlim2f, -rlim2f);
  unsigned row = 0;
  bool u = false;
#pragma unroll 4
  for (int q = 0; 2 * q < nlive; ++q) {   // warp-uniform
    const float4 xy = S.l.xy[w][q], zb = S.l.zb[w][q];
    float2 dx = __fadd2_rn(make_float2(xy.x, xy.y), nx);
    float2 dy = __fadd2_rn(make_float2(xy.z, xy.w), ny);
    float2 dz = __fadd2_rn(make_float2(zb.x, zb.y), nz);
    if (PIMG) {
      dx.x = fmaf(-bx, rintf(dx.x * ibx), dx.x);
      dx.y = fmaf(-bx, rintf(dx.y * ibx), dx.y);
      dy.x = fmaf(-by, rintf(dy.x * iby), dy.x);
      dy.y = fmaf(-by, rintf(dy.y * iby), dy.y);
      dz.x = fmaf(-bz, rintf(dz.x * ibz), dz.x);
      dz.y = fmaf(-bz, rintf(dz.y * ibz), dz.y);
    }
    // d^2 - rlim^2 has the sign of the comparison (a difference rounds to zero only if it is)
    const float2 e = __fadd2_rn(__ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz))), ml);
    u |= fabsf(e.x) < band;
    u |= fabsf(e.y) < band;
    if (e.x <= 0.f) row |= __float_as_uint(zb.z);
    if (e.y <= 0.f) row |= __float_as_uint(zb.w);
  }
  unsure = __any_sync(full, u && ireal);
  return ireal ? row : 0u;
}

// where tile c of i-block b keeps its mask rows and its record
__device__ __forceinline__ BlkTile& blk_tile(const DevPtrs& P, ListShared& S, long long t0, int c) {
  return c < kTileCache ? S.tile[c] : P.blk_tiles[t0 + c];
}

// 16 mask rows (64 bytes) of a half block's record slots: every slot contributes, per row, the
// bit of its j lane (stored rotated: bit k of row ri is j lane (ri + k) & 31), one ballot a row;
// lane r keeps row r
__device__ __forceinline__ unsigned record_rows(const unsigned* rows, bool live, int jl, int h, int lane) {
  unsigned cur = 0u;
  uint4 m[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) m[q] = live ? reinterpret_cast<const uint4*>(rows)[q] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const unsigned v[4] = {m[q].x, m[q].y, m[q].z, m[q].w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int r = 4 * q + k;
      const unsigned row = __ballot_sync(0xffffffffu, (v[k] >> ((jl - kHalf * h - r) & 31)) & 1u);
      if (lane == r) cur = row;
    }
  }
  return cur;
}

// count_only: as far as the records per unit (the block-shape tuner needs no more); keep: leave
// the masks in global memory and list the tiles (the H-bond list reads them); split_cls (ALSD,
// mixed path): records with a cluster atom go to the top end of the record arrays, downwards,
// as their pairs take class weights and class energies in a launch of their own
template <bool CMM>
__global__ void __launch_bounds__(32 * kListWarps, CMM ? 3 : 4) k_block_list(DevPtrs P, int bi0, double rlim2, float rlimf,
                                                                             double rc2, int dummy_type, int count_only,
                                                                             int keep, int apart) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  ListShared& S = *reinterpret_cast<ListShared*>(s_dyn);
  unsigned* s_mask = reinterpret_cast<unsigned*>(s_dyn + sizeof(ListShared));   // [kTileCache][32], CMM: twice
  const unsigned full = 0xffffffffu;
  const int bi = bi0 + blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int ai = P.satom[bi * kTile + lane];
  // a block fills from its first slot: this one is not used by the present sort
  if (!__any_sync(full, ai >= 0)) {
    if (threadIdx.x < 2) P.ct_cnt[2 * bi + threadIdx.x] = 0;
    return;
  }
  const int rep = P.blk_rep[bi];
  const Rep& R = P.reps[rep];
  const long long t0 = P.blk_tile0[bi];
  const float rlim2f = (float)rlim2;
  // the FP32 mask's uncertainty band: every coordinate tile_row_f32 works with is below
  // M = rlim + 3 h_max in magnitude (h_max: the replica's largest block half extent) and
  // carries at most 2.5 roundings of 2^-24 M, a difference one more, so |error of d^2| <=
  // 2 sqrt(3) rlim 5 2^-24 M + 3 2^-24 rlim^2; pairs within 4 times that of rlim^2 are
  // decided in FP64 (about 1.5e-3 A^2 for water blocks at rc = 12 A)
  const float hm = fmaxf(P.rep_hmax[3 * rep], fmaxf(P.rep_hmax[3 * rep + 1], P.rep_hmax[3 * rep + 2]));
  // (with per-pair images, in a box below twice that, the coordinates before imaging reach the
  // box edge)
  const float lmax = (float)fmax(R.box[0], fmax(R.box[1], R.box[2]));
  const float mb = (0.5f * lmax > rlimf + 2.f * hm ? rlimf : fmaxf(rlimf, lmax)) + 3.f * hm;
  const float band = 4.f * 5.9604645e-8f * (17.33f * rlimf * mb + 3.f * rlimf * rlimf);
  float3 xi = make_float3(0.f, 0.f, 0.f);   // this lane's i atom relative to its block's reference
  if (!CMM) {   // the i block, wrapped, for the broadcast reads of the FP64 form
    double q[3] = {0.0, 0.0, 0.0};
    for (int k = 0; k < 3; ++k)
      if (ai >= 0) {
        const double x = P.x[3 * ai + k];
        q[k] = x - R.box[k] * floor(x * R.invbox[k]);
      }
    if (w == 0) {
      S.x[lane] = q[0];
      S.y[lane] = q[1];
      S.z[lane] = q[2];
    }
    xi = make_float3((float)(q[0] - P.blk_ref[3 * bi]), (float)(q[1] - P.blk_ref[3 * bi + 1]),
                     (float)(q[2] - P.blk_ref[3 * bi + 2]));
  }
  const float4 ci = P.blk_ctr[bi], hi = P.blk_half[bi];
  const float bx = (float)R.box[0], by = (float)R.box[1], bz = (float)R.box[2];
  const float ibx = (float)R.invbox[0], iby = (float)R.invbox[1], ibz = (float)R.invbox[2];
  const int ncand = R.blk0 + R.nblk - bi;   // later blocks of the replica, itself included
  auto mask_rows = [&](int c, bool el) -> unsigned* {
    if (c < kTileCache && !keep) return s_mask + (size_t)(el ? kTileCache + c : c) * 32;
    return (el ? P.tmp_masks_el : P.tmp_masks) + (size_t)(t0 + c) * 32;
  };

  int nt = 0;   // tiles so far
  for (int seg = 0; seg < ncand; seg += kSegment) {
    const int nb = min(kSegment, ncand - seg);
    for (int k = threadIdx.x; k < kSegment / 32; k += blockDim.x) S.ball[k] = S.excl[k] = 0u;
    __syncthreads();
    // bounding boxes, 32 candidates a warp at once
    for (int g = w; 32 * g < nb; g += nw) {
      const int bj = bi + seg + 32 * g + lane;
      bool cand = false;
      if (32 * g + lane < nb) {
        const float4 cj = P.blk_ctr[bj], hj = P.blk_half[bj];
        float dx = ci.x - cj.x, dy = ci.y - cj.y, dz = ci.z - cj.z;
        dx -= bx * rintf(dx * ibx);
        dy -= by * rintf(dy * iby);
        dz -= bz * rintf(dz * ibz);
        const float gx = fmaxf(fabsf(dx) - hi.x - hj.x, 0.f);
        const float gy = fmaxf(fabsf(dy) - hi.y - hj.y, 0.f);
        const float gz = fmaxf(fabsf(dz) - hi.z - hj.z, 0.f);
        cand = gx * gx + gy * gy + gz * gz <= rlimf * rlimf * 1.0001f + 1e-3f;
      }
      const unsigned ball = __ballot_sync(full, cand);
      if (lane == 0) S.ball[g] = ball;
    }
    // blocks of the segment that hold an exclusion partner of the i block (partners by atom,
    // the atoms' lists spread over the warps)
    for (int i = w; i < kTile; i += nw) {
      const int a = __shfl_sync(full, ai, i);
      if (a < 0) continue;
      for (int p = P.excl_ptr[a] + lane; p < P.excl_ptr[a + 1]; p += 32) {
        const int rel = (P.excl_slot[p] >> 5) - bi - seg;
        if (rel >= 0 && rel < nb) atomicOr(&S.excl[rel >> 5], 1u << (rel & 31));
      }
    }
    __syncthreads();
    // the survivors in order, each with its block reference in the i block's frame
    int n = 0;
    for (int g = 0; 32 * g < nb; ++g) {
      const unsigned ball = S.ball[g];
      if (g % nw == w && ((ball >> lane) & 1u)) {
        BlkTile& T = blk_tile(P, S, t0, nt + n + __popc(ball & ((1u << lane) - 1u)));
        const int bj = bi + seg + 32 * g + lane;
        // Per axis a pair's separation in the tile's image is at most |c| + h_i + h_j, so in any
        // other image it is at least the box edge minus that.  The tile's image serves every
        // listed pair if that is beyond the list radius; it serves every pair the kernels meet
        // until the next build if, with 2 A for the atoms' motion, it is beyond the cut-off
        // (CMM, no cut-off: beyond the farthest near-field pair)
        const float4 hj = P.blk_half[bj];
        const uint2 kind = P.blk_kind[bj];
        const float hh[3] = {hi.x + hj.x, hi.y + hj.y, hi.z + hj.z};
        const float rk = CMM ? rlimf : (float)sqrt(rc2);
        float c[3];
        int img = 0;
        for (int k = 0; k < 3; ++k) {
          const double d = P.blk_ref[3 * bi + k] - P.blk_ref[3 * bj + k];
          c[k] = (float)(R.box[k] * anint(d * R.invbox[k]) - d);
          const float other = (float)R.box[k] - (fabsf(c[k]) + hh[k]);
          if (!(other > rlimf + 0.01f)) img |= kTileListImg;
          if (!(other > rk + 2.f)) img |= kTilePairImg;
        }
        T.j = bj | img;
        T.lj = kind.x;
        T.sp = (img & kTilePairImg) ? 0xffffffffu : kind.y;
        T.cx = c[0]; T.cy = c[1]; T.cz = c[2];
      }
      n += __popc(ball);
    }
    __syncthreads();
    // one warp a tile: its mask, and the j lanes some i atom of each half lists.  The next
    // tile's j atoms are gathered before this one's pairs
    int an = -1;
    float4 pn = make_float4(0.f, 0.f, 0.f, 0.f);
    auto gather = [&](int c) {
      an = c < nt + n ? P.satom[(blk_tile(P, S, t0, c).j & kTileBlock) * kTile + lane] : -1;
      if (an >= 0) pn = P.pos_f[an];
    };
    if (!CMM) gather(nt + w);
    for (int c = nt + w; c < nt + n; c += nw) {
      BlkTile& T = blk_tile(P, S, t0, c);
      const int bj = T.j & kTileBlock;
      const bool fast = !CMM && !(T.j & kTileListImg);
      unsigned mask = 0, mel = 0;
      bool unsure = true;
      if (!CMM) {
        const float3 cc = make_float3(T.cx, T.cy, T.cz);
        const bool jreal = an >= 0;
        const float4 pj = pn;
        gather(c + nw);
        const unsigned row =
            fast ? tile_row_f32<false>(R, cc, hi, lane, xi, ai >= 0, pj, jreal, S, rlim2f, band, unsure)
                 : tile_row_f32<true>(R, cc, hi, lane, xi, ai >= 0, pj, jreal, S, rlim2f, band, unsure);
        if (!unsure) mask = __funnelshift_r(row, row, lane);
      }
      if (unsure) {
        if (fast) {
          const unsigned row = tile_row_fast(P.satom, P.x, P.blk_ref, R, bi, bj, lane, ai, S, rlim2);
          mask = __funnelshift_r(row, row, lane);
        } else {
          mask = tile_mask<CMM>(P.satom, P.x, P.cmm_cell, R, bi, bj, lane, ai, rlim2, rc2, mel);
        }
      }
      if (bj == bi) mask &= lane < 16 ? 0x1fffeu : 0xfffeu;   // each unordered pair once, no self pair
      const int rel = bj - bi - seg;
      if ((S.excl[rel >> 5] >> (rel & 31)) & 1u) mask = drop_excluded(P, bj, lane, ai, mask);
      mask_rows(c, false)[lane] = mask;
      if (CMM) mask_rows(c, true)[lane] = mel & mask;
      const unsigned rowj = __funnelshift_l(mask, mask, lane);
      const unsigned o0 = __reduce_or_sync(full, lane < kHalf ? rowj : 0u);
      const unsigned o1 = __reduce_or_sync(full, lane < kHalf ? 0u : rowj);
      if (lane == 0) {
        T.occ[0] = o0;
        T.occ[1] = o1;
        if (keep && !count_only && (o0 | o1)) {
          const int t = atomicAdd(P.ntiles, 1);
          P.tiles[t] = make_int2(bi, bj);
          P.tile_src[t] = t0 + c;
        }
      }
    }
    nt += n;
    __syncthreads();
  }

  // entries of each half and kind, a warp a sum: exclusive sums over the tiles
  for (int key = w; key < 8; key += nw) {
    const int h = key >> 2, k = key & 3;
    int sum = 0;
    for (int c0 = 0; c0 < nt; c0 += 32) {
      const bool in = c0 + lane < nt;
      BlkTile& T = blk_tile(P, S, t0, min(c0 + lane, nt - 1));
      const int n = in ? __popc(T.occ[h] & (k & 2 ? T.sp : ~T.sp) & (k == 0 || k == 3 ? T.lj : ~T.lj)) : 0;
      int s = n;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(full, s, o);
        if (lane >= o) s += y;
      }
      if (in) T.eoff[h][k] = sum + s - n;
      sum += __shfl_sync(full, s, 31);
    }
    if (lane == 0) S.carry[key] = sum;
  }
  __syncthreads();
  const int E[2] = {S.carry[0] + S.carry[1] + S.carry[2] + S.carry[3], S.carry[4] + S.carry[5] + S.carry[6] + S.carry[7]};
  if (threadIdx.x < 8) {   // half h: kinds 0 1 2 3, or 3 2 1 0
    const int h = threadIdx.x >> 2, k = threadIdx.x & 3;
    int f = 0;
    for (int q = 0; q < 4; ++q)
      if (h ? q > k : q < k) f += S.carry[4 * h + q];
    S.first[h][k] = f;
  }
  const int nr0 = (E[0] + 31) >> 5, nr1 = (E[1] + 31) >> 5;
  if (threadIdx.x == 0) {
    P.ct_cnt[2 * bi] = nr0;
    P.ct_cnt[2 * bi + 1] = nr1;
  }
  if (count_only) return;
  const bool split_cls = apart == kApartCls;
  // records of each half at the array's end (kApartImg)
  int na0 = 0, na1 = 0;
  if (apart == kApartImg) {
    na0 = S.carry[2] + S.carry[3] > 0 ? nr0 - ((S.carry[0] + S.carry[1]) >> 5) : 0;
    na1 = (S.carry[6] + S.carry[7] + 31) >> 5;
  }
  if (threadIdx.x == 0) S.nimg = 0;
  if (threadIdx.x < 2 && !split_cls) {
    const int na = na0 + na1;
    S.base[threadIdx.x] = atomicAdd(&P.nctiles[threadIdx.x], threadIdx.x ? na : nr0 + nr1 - na);
  }

  const bool wide = nt > kNarrowTiles;
  const int win = wide ? kWindow / 2 : kWindow;
  auto entry = [&](int h, int e) { return wide ? S.e32[h][e] : (unsigned)S.e16[h][e]; };
  // the records, `win` of each half at a time: every tile spreads its entries over the
  // window's list, then a warp takes a record, lane p slot p
  for (int w0 = 0; w0 < max(nr0, nr1); w0 += win) {
    __syncthreads();
    for (int c = w; c < nt; c += nw) {
      const BlkTile& T = blk_tile(P, S, t0, c);
      const bool sp = (T.sp >> lane) & 1u, lj = (T.lj >> lane) & 1u;
      const int k = sp ? (lj ? 3 : 2) : (lj ? 0 : 1);
      const unsigned same = (sp ? T.sp : ~T.sp) & (lj ? T.lj : ~T.lj) & ((1u << lane) - 1u);   // of this kind, before
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const unsigned occ = T.occ[h];
        const int e = S.first[h][k] + T.eoff[h][k] + __popc(occ & same) - 32 * w0;
        if (((occ >> lane) & 1u) && e >= 0 && e < 32 * win) {
          if (wide) S.e32[h][e] = ((unsigned)c << 5) | lane;
          else S.e16[h][e] = (unsigned short)((c << 5) | lane);
        }
      }
    }
    __syncthreads();
    const int m0 = max(0, min(win, nr0 - w0)), m1 = max(0, min(win, nr1 - w0));
    if (split_cls) {
      for (int q = w; q < m0 + m1; q += nw) {
        const int h = q < m0 ? 0 : 1, r = q < m0 ? q : q - m0;
        int ty = 0;
        if (32 * (w0 + r) + lane < E[h]) {
          const unsigned v = entry(h, 32 * r + lane);
          ty = P.styp[(blk_tile(P, S, t0, (int)(v >> 5)).j & kTileBlock) * kTile + (int)(v & 31u)];
        }
        if (lane < kHalf) ty |= P.styp[bi * kTile + kHalf * h + lane];
        const bool cls = __any_sync(full, (ty >> 30) & 1);
        if (lane == 0) S.rcls[q] = cls ? 1 : 0;
      }
      __syncthreads();
      if (w == 0) {   // places of the window's records in their two sequences
        int n[2] = {0, 0};
        for (int pass = 0; pass < 2; ++pass) {
          int b[2] = {0, 0};
          if (pass) {
            if (lane < 2) b[0] = atomicAdd(&P.nctiles[lane], lane ? n[1] : n[0]);
            b[1] = __shfl_sync(full, b[0], 1);
            b[0] = __shfl_sync(full, b[0], 0);
            n[0] = n[1] = 0;
          }
          for (int q0 = 0; q0 < m0 + m1; q0 += 32) {
            const bool in = q0 + lane < m0 + m1;
            const bool cls = in && S.rcls[q0 + lane];
            const unsigned mc = __ballot_sync(full, cls), mp = __ballot_sync(full, in && !cls);
            const unsigned below = (1u << lane) - 1u;
            if (pass && in)
              S.rpos[q0 + lane] = cls ? P.rec_cap - 1 - (size_t)(b[1] + n[1] + __popc(mc & below))
                                      : (size_t)(b[0] + n[0] + __popc(mp & below));
            n[0] += __popc(mp);
            n[1] += __popc(mc);
          }
        }
      }
      __syncthreads();
    }
    for (int q = w; q < m0 + m1; q += nw) {
      const int h = q < m0 ? 0 : 1, r = q < m0 ? q : q - m0;   // record r of the window of half h
      size_t ct;
      if (split_cls) ct = S.rpos[q];
      else if (h == 0)
        ct = w0 + r < nr0 - na0 ? (size_t)(S.base[0] + w0 + r)
                                : P.rec_cap - 1 - (size_t)(S.base[1] + w0 + r - (nr0 - na0));
      else
        ct = w0 + r < na1 ? P.rec_cap - 1 - (size_t)(S.base[1] + na0 + w0 + r)
                          : (size_t)(S.base[0] + nr0 - na0 + w0 + r - na1);
      const bool live = 32 * (w0 + r) + lane < E[h];
      const unsigned v = live ? entry(h, 32 * r + lane) : 0u;
      const int c = (int)(v >> 5), jl = (int)(v & 31u);
      float4 ent = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
      int ty = dummy_type;
      bool img = false, has_lj = false;
      if (live) {
        const BlkTile& T = blk_tile(P, S, t0, c);
        has_lj = (T.lj >> jl) & 1u;
        img = (T.j & kTilePairImg) != 0;
        const int slot = (T.j & kTileBlock) * kTile + jl;
        ent = make_float4(-T.cx, -T.cy, -T.cz, __int_as_float(P.satom[slot]));
        ty = P.styp[slot];
      }
      P.ct_j[ct * 32 + lane] = ent;
      P.ct_ty[ct * 32 + lane] = type_half(ty);
      const unsigned cur = record_rows(mask_rows(c, false) + kHalf * h, live, jl, h, lane);
      if (lane < kHalf) P.ct_mask[ct * kHalf + lane] = record_row(cur, lane);
      if (CMM) {
        const unsigned cel = record_rows(mask_rows(c, true) + kHalf * h, live, jl, h, lane);
        if (lane < kHalf) P.ct_mask_el[ct * kHalf + lane] = record_row(cel, lane);
      }
      const bool any_img = __any_sync(full, img);
      const unsigned lj = __ballot_sync(full, has_lj);
      int fl = any_img ? kRecImg : 0;
#pragma unroll
      for (int g = 0; g < 4; ++g) fl |= ((lj >> (8 * g)) & 0xffu) ? 0 : 1 << (kRecFree + g);
      if (lane == 0) P.ct_blk[ct] = (2 * bi + h) | fl;
      if (lane == 0 && split_cls && any_img && !S.rcls[q]) atomicAdd(&S.nimg, 1);
    }
  }
  if (split_cls) {
    __syncthreads();
    if (threadIdx.x == 0 && S.nimg > 0) atomicAdd(&P.nctiles[2], S.nimg);
  }
}

static size_t list_smem(bool cmm) { return sizeof(ListShared) + (size_t)kTileCache * 128 * (cmm ? 2 : 1); }

void init_block_list() {
  cudaFuncSetAttribute(k_block_list<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)list_smem(false));
  cudaFuncSetAttribute(k_block_list<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)list_smem(true));
}

void launch_block_list(const DevPtrs& P, int bi0, int nblk, int nsm, double rlim2, float rlimf, double rc2, bool cmm,
                       int dummy_type, bool count_only, bool keep, int apart, cudaStream_t st) {
  // eight warps a block where the blocks fill the chip a few times at most (each i-block's tiles in
  // fewer rounds), four where they fill it often and eight mostly wait for each other.  A build
  // with eight and with four: 816 blocks 111 and 160 us, 1,482 blocks 162 and 184, 2,288 blocks
  // 233 and 231, 3,383 blocks 343 and 330, 64 replicas (some 28,000 blocks) 2,447 and 2,310
  const int nt = 32 * (nblk < 16 * nsm ? 8 : 4);
  if (cmm)
    k_block_list<true><<<nblk, nt, list_smem(true), st>>>(P, bi0, rlim2, rlimf, rc2, dummy_type, count_only, keep, apart);
  else
    k_block_list<false><<<nblk, nt, list_smem(false), st>>>(P, bi0, rlim2, rlimf, rc2, dummy_type, count_only, keep, apart);
}

// ---- deterministic exclusive scan (3 passes) --------------------------------------------
__global__ void k_scan_block_sums(const int* in, int n, int* bsum) {
  __shared__ int sh[1024];
  int i = blockIdx.x * 1024 + threadIdx.x;
  int v = i < n ? in[i] : 0;
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = 512; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) bsum[blockIdx.x] = sh[0];
}

// single block: exclusive scan of nb block sums (any nb)
__global__ void k_scan_small(int* bsum, int nb) {
  __shared__ int sh[1024];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int b0 = 0; b0 < nb; b0 += 1024) {
    int i = b0 + threadIdx.x;
    int v = i < nb ? bsum[i] : 0;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
      int t = threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
      __syncthreads();
      sh[threadIdx.x] += t;
      __syncthreads();
    }
    if (i < nb) bsum[i] = carry + sh[threadIdx.x] - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry += sh[1023];
    __syncthreads();
  }
}

__global__ void k_scan_final(const int* in, int n, const int* bsum, int* out, int* total) {
  __shared__ int sh[1024];
  int i = blockIdx.x * 1024 + threadIdx.x;
  int v = i < n ? in[i] : 0;
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    int t = threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
    __syncthreads();
    sh[threadIdx.x] += t;
    __syncthreads();
  }
  if (i < n) out[i] = bsum[blockIdx.x] + sh[threadIdx.x] - v;
  if (i == n - 1 && total) *total = bsum[blockIdx.x] + sh[threadIdx.x];
}

// one block for up to kScanOneMax values: thread t sums its run of consecutive values, the
// 1024 run sums are scanned with warp shuffles, and each thread writes its run's prefixes
constexpr int kScanOneMax = 1 << 13;   // above it the three-pass scan is faster

__global__ void __launch_bounds__(1024) k_scan_one(const int* in, int n, int* out, int* total) {
  __shared__ int wsum[32];
  const unsigned full = 0xffffffffu;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int per = (n + 1023) / 1024;
  const int b = min(t * per, n), e = min(b + per, n);
  int s = 0;
  for (int i = b; i < e; ++i) s += in[i];
  int x = s;   // inclusive scan of the run sums: within the warp, then over the warps
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(full, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int w = wsum[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(full, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  int run = x - s + (wid > 0 ? wsum[wid - 1] : 0);
  for (int i = b; i < e; ++i) {
    const int v = in[i];
    out[i] = run;
    run += v;
  }
  if (t == 0 && total) *total = wsum[31];
}

int scan_exclusive(const int* in, int* out, int n, int* scratch, int* total, cudaStream_t st) {
  if (n <= kScanOneMax) {
    k_scan_one<<<1, 1024, 0, st>>>(in, n, out, total);
    return 1;
  }
  int nb = (n + 1023) / 1024;
  k_scan_block_sums<<<nb, 1024, 0, st>>>(in, n, scratch);
  k_scan_small<<<1, 1024, 0, st>>>(scratch, nb);
  k_scan_final<<<nb, 1024, 0, st>>>(in, n, scratch, out, total);
  return 3;
}

}  // namespace jp
