// jp_pair.cu -- zero-dipole (ZD) cut-off Coulomb + Lennard-Jones pair kernels.
//
// Replaces enear_ZD_{redu,high,doub}_PB (src_md_run/enear.f90:2-593, lines tagged #ZD #PB):
//   co   = [r <= rc]                                  (enear.f90:134, sign(0.5,dd2i-irlim2)+.5)
//   E_el += qi qj co (1/r + b r^2 - z)                 (enear.f90:138-141)
//   E_lj += co (C12/r^12 - C6/r^6)                      (enear.f90:199-210)
//   dE/dxi = -d [qi qj co (1/r^3 - f) + co (12 C12/r^12 - 6 C6/r^6)/r^2],  d = xi - xj
// with q = charge * sqrt(332.06378/eps) (chgmod, inpcls.f90:215-227), b = 1/(2 rc^3),
// f = 1/rc^3, z = 1.5/rc (incel.f90:655-658).
//
// Work unit: a pair record (jp_cells.cu) = half an i-block (16 cell-sorted atoms) and 32 j
// entries (j atoms with at least one listed pair in the half block, each with the image
// shift of its block) with an interaction mask fixed at list-build time.  Newton's third
// law: each unordered pair is evaluated once.
//
// Mixed path, k_pair_packed (plain and ALSD contexts): a warp takes four consecutive records,
// eight lanes each; a lane holds two i atoms (l and l + 8 of its record) and meets one j entry
// per step, two pairs in packed FP32x2 arithmetic.  k_pair_mixed (CMM and partial McMD): two
// records, a half-warp each, one i atom a lane, the two entries of a step in scalar
// arithmetic.  FP32 pair arithmetic on block-local coordinates (|x| < ~30 A), every step of a
// record branch-free (a pair outside the mask or the cut-off contributes an exact zero);
// an i atom's forces summed over eight entries and a j atom's over the record's i atoms in FP32,
// energies in FP32 over 4 steps then in FP64, all added as 64-bit fixed point (2^-32 kcal/mol/A)
// with integer atomics -- order independent, so results are bit-identical run to run.  Warps take short runs of consecutive record groups,
// the first by their own index and the next from a global counter, so all finish together
// whatever their records hold.  A warp keeps two groups in flight ahead of the one it
// computes: the bulk-copy engine (cp.async.bulk, completion on an mbarrier) brings the
// entries and masks of the group after next into shared memory, and the gathers of the next
// group's j atoms are issued before the current group's arithmetic.
// FP64 path: the same records in FP64 with FP64 force atomics (k_pair_fp64q; k_pair_fp64 with
// classes and CMM).
#include <algorithm>
#include <vector>

#include "jp_kernels.h"

namespace jp {

// Six warps a block, two blocks an SM: 168 registers a thread, which the packed kernel's sums
// need.  With eight warps (128 registers) they spilled: 64 replicas (883,000 atoms) 1,390 us, so
// 1,307, 99,200 atoms 174 and 163, 2,200 atoms 21 and 17.  The FP64 kernels keep eight (ALSD
// replicas of 36,500 atoms 255 us, with six 289; 270,000 atoms 673 and 696).
constexpr int kPairWarps = 6, kPairThreads = 32 * kPairWarps;
constexpr int kFp64Warps = 8, kFp64Threads = 32 * kFp64Warps;
constexpr long long kCopyWaitCycles = 2000000000LL;

// ---- bulk copies into shared memory (TMA engine, no tensor map) -------------------------
__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(unsigned long long* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// arm the barrier for `bytes` of incoming copies and start one copy of `bytes` (a multiple
// of 16, both addresses 16-byte aligned) from global to shared memory
__device__ __forceinline__ void mbar_expect(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// the shared-memory buffer is about to be overwritten by the async proxy after generic reads
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// wait for phase `parity` of the barrier, at most `limit` SM cycles; false on timeout
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, long long limit) {
  const long long t0 = clock64();
  for (;;) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > limit) return false;
  }
}

// the same for a whole warp, one answer: after a wait that ran out in some lanes alone these would
// leave the loop, and the others would wait for them in its next warp collective without end
__device__ __forceinline__ bool mbar_wait_warp(unsigned long long* bar, unsigned parity, long long limit) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, limit));
}

// each lane group's energies (ELE15, VDW15; ALSD class AA / AB, BB the rest) and pair count
// into the slots of its replica: 64-bit fixed point, summed per record, so the totals do not
// depend on which warp took which record (the kernels claim their records dynamically).  The
// W-lane groups of a warp may work for different replicas: the sums stay inside each group.
template <int W>
__device__ __forceinline__ void flush_fix(const DevPtrs& P, int rep, long long eel, long long elj,
                                          long long eaa, long long eab, long long npair, bool count,
                                          bool alsd) {
  for (int o = W / 2; o > 0; o >>= 1) {
    eel += __shfl_xor_sync(0xffffffffu, eel, o);
    elj += __shfl_xor_sync(0xffffffffu, elj, o);
    if (alsd) {
      eaa += __shfl_xor_sync(0xffffffffu, eaa, o);
      eab += __shfl_xor_sync(0xffffffffu, eab, o);
    }
    if (count) npair += __shfl_xor_sync(0xffffffffu, npair, o);
  }
  if ((threadIdx.x & (W - 1)) == 0 && rep >= 0) {
    atomic_add_ll(&P.ene_fix[rep * 16 + JP_E_ELE15], eel);
    atomic_add_ll(&P.ene_fix[rep * 16 + JP_E_VDW15], elj);
    if (alsd) {
      atomic_add_ll(&P.ene_cls[rep * 4 + 0], eaa);
      atomic_add_ll(&P.ene_cls[rep * 4 + 1], eab);
      atomic_add_ll(&P.ene_cls[rep * 4 + 2], eel + elj - eaa - eab);
    }
    if (count) atomicAdd(reinterpret_cast<unsigned long long*>(&P.pair_cnt[rep]),
                         static_cast<unsigned long long>(npair));
  }
}

// Per-warp shared memory of k_pair_mixed: two bulk-copy buffers (entries and masks of a
// record pair: record 0 in entries 0-31 and masks 0-15, record 1 in 32-63 and 16-31) and the
// staged j atoms of the pair being computed.  Half-warp h stages its record at [32 h, 32 h +
// 32): lane l's entries a = l and b = 16 + l side by side, stored twice (at 32 h + l and
// 32 h + l + 16) so that step k reads slot 32 h + l + k at a constant offset.
struct __align__(16) MixStage {
  float4 ent[2][64];
  unsigned msk[2][32];
  unsigned msk_el[2][32];
  float4 p2[64];      // x_a, x_b, y_a, y_b
  float4 q2[64];      // z_a, z_b, q_a, q_b
  int2 t2[64];        // their LJ type words
  unsigned long long bar[2];
};

// rsqrt.approx without the IEEE-mode denormal fix-up: its argument is a squared distance of
// a listed pair (far above the FP32 denormal range) or a masked slot's 1 or 1e30
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Nearest integer of v (ties to even, as rintf) for |v| < 2^22, on the FMA pipe: adding and
// subtracting 1.5 * 2^23 rounds v at the unit place in round-to-nearest-even (the explicit
// _rn adds are never contracted or reassociated).  The minimum-image multiples are a few
// units at most.
__device__ __forceinline__ float2 rint2(float2 v) {
  const float2 m = make_float2(12582912.f, 12582912.f), nm = make_float2(-12582912.f, -12582912.f);
  return __fadd2_rn(__fadd2_rn(v, m), nm);
}

__device__ __forceinline__ float rint1(float v) {
  return __fadd_rn(__fadd_rn(v, 12582912.f), -12582912.f);
}

// The last flush of a block's warps: their sums are added in shared memory first and reach the
// slots as one atomic per block and slot.  Every warp of a single-system launch adds to the
// same two addresses, and L2 takes atomics on one address one after the other: with one pair
// of them per lane group (19,000 atomics) a launch on 24,000 atoms took 59.1 us, so 52.0.
// Called by all threads of the block.
template <int W, int WARPS>
__device__ __forceinline__ void flush_block(const DevPtrs& P, int rep, long long eel, long long elj, long long eaa,
                                            long long eab, long long npair, bool count, bool cls) {
  __shared__ long long s_sum[WARPS][5];
  __shared__ int s_rep[WARPS];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int r = __reduce_max_sync(full, rep);
  if (!__all_sync(full, rep < 0 || rep == r)) {   // lane groups of several replicas
    flush_fix<W>(P, rep, eel, elj, eaa, eab, npair, count, cls);
    r = -1;
  }
  for (int o = 16; o > 0; o >>= 1) {
    eel += __shfl_xor_sync(full, eel, o);
    elj += __shfl_xor_sync(full, elj, o);
    if (cls) {
      eaa += __shfl_xor_sync(full, eaa, o);
      eab += __shfl_xor_sync(full, eab, o);
    }
    if (count) npair += __shfl_xor_sync(full, npair, o);
  }
  if (lane == 0) {
    s_rep[warp] = r;
    s_sum[warp][0] = eel;
    s_sum[warp][1] = elj;
    s_sum[warp][2] = count ? npair : 0;
    s_sum[warp][3] = eaa;
    s_sum[warp][4] = eab;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 0; w < WARPS; ++w) {
      const int rw = s_rep[w];
      if (rw < 0) continue;
      long long a = 0, b = 0, n = 0, ca = 0, cb = 0;   // the warps of this replica, taken together
      for (int v = w; v < WARPS; ++v)
        if (s_rep[v] == rw) {
          a += s_sum[v][0];
          b += s_sum[v][1];
          n += s_sum[v][2];
          ca += s_sum[v][3];
          cb += s_sum[v][4];
          s_rep[v] = -1;
        }
      atomic_add_ll(&P.ene_fix[rw * 16 + JP_E_ELE15], a);
      atomic_add_ll(&P.ene_fix[rw * 16 + JP_E_VDW15], b);
      if (cls) {
        if (ca) atomic_add_ll(&P.ene_cls[rw * 4 + 0], ca);
        if (cb) atomic_add_ll(&P.ene_cls[rw * 4 + 1], cb);
        atomic_add_ll(&P.ene_cls[rw * 4 + 2], a + b - ca - cb);
      }
      if (count) atomic_add_ll(&P.pair_cnt[rw], n);
    }
  }
}

// ---- packed kernel: four records a warp, eight lanes and two i atoms a lane -----------------
// In ALSD contexts the records that hold a cluster atom stand apart (k_block_list) and take a
// launch of their own with class weights and class energies (CLS); the others take the plain
// kernel.  Both forms in one kernel, chosen per group, spilled the class state and ran the rare
// form's instructions through the others' cache (32 replicas of 9,100 atoms with four cluster
// residues each: 897 us with the classes in every record, 717 chosen per group, 573 so).
// Per-warp shared memory: two bulk-copy buffers (entries, their atoms and types, and masks of a
// record group: record q in entries 32 q and masks 16 q), and the staged j atoms of the group
// being computed.  The position of entry 8 g + e of record q is staged twice, at 64 q + 16 g + e
// and 8 further on, so that step k of group g reads slot 64 q + 16 g + l + k at a constant
// offset (l: lane in the record); its type moves from lane to lane instead (a shuffle costs
// the pipe what a 4-byte read does).
struct __align__(16) QuadStage {
  float4 ent[2][128];
  unsigned short ty[2][128];
  unsigned msk[2][64];
  float4 p[256];            // x, y, z in the i block's frame, scaled charge
  int2 at[4 * 36];          // (atom, type word) of entry 8 g + e at 36 q + 8 g + e
  // of each record's replica: box edges and their inverses (per-pair images), class weights
  // BB, AB, AA (ALSD); read where a group needs them, which spares registers in the others
  float rep[4][12];
  unsigned long long bar[2];
};

// a group's sums over its entries, (i atom, i atom + 8) side by side, into the lane's fixed-point
// forces; a value outside the fixed-point range (2^24 kcal/mol/A) or not finite is reported
__device__ __noinline__ void report_force(unsigned* status, float2 x, float2 y, float2 z) {
  to_fix_f(x.x, status); to_fix_f(x.y, status);
  to_fix_f(y.x, status); to_fix_f(y.y, status);
  to_fix_f(z.x, status); to_fix_f(z.y, status);
}

__device__ __forceinline__ float max_nan(float a, float b) {   // NaN if either is
  float m;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
  return m;
}

__device__ __forceinline__ void add_forces(unsigned* status, float2 x, float2 y, float2 z, long long (&ga)[3],
                                           long long (&gb)[3]) {
  const float m = max_nan(max_nan(max_nan(fabsf(x.x), fabsf(x.y)), max_nan(fabsf(y.x), fabsf(y.y))),
                          max_nan(fabsf(z.x), fabsf(z.y)));
  if (!(m < 16777216.f)) report_force(status, x, y, z);
  const float2 k = make_float2(4294967296.f, 4294967296.f);
  x = __fmul2_rn(x, k);
  y = __fmul2_rn(y, k);
  z = __fmul2_rn(z, k);
  ga[0] += __float2ll_rn(x.x);
  gb[0] += __float2ll_rn(x.y);
  ga[1] += __float2ll_rn(y.x);
  gb[1] += __float2ll_rn(y.y);
  ga[2] += __float2ll_rn(z.x);
  gb[2] += __float2ll_rn(z.y);
}

// what the inner loop reads of a lane's replica and classes
struct PackedArgs {
  float2 nx, ny, nz, qi;                 // minus the two i positions, their charges
  unsigned ma, mb;                       // their mask words (step_mask order)
  float rc2, zb, zf, zc;
  // ALSD classes (CLS): cluster bits of the entries (step order) and of the i atoms, class
  // weights of a pair with a plain (0) or a cluster (1) entry
  unsigned jc;
  bool ca, cb;
  float2 w0, w1;
};

// One record: four groups of eight entries; at step k of group g lane l meets entry
// 8 g + ((l + k) & 7) with its two i atoms, the pairs side by side in packed FP32x2 arithmetic
// (Blackwell's FFMA2 / FADD2 / FMUL2).  A pair outside the mask or the cut-off takes r^2 = 1e30
// (its r^-6 = 1e-90 is zero in FP32) and a zero charge product, so it contributes an exact
// zero without a branch.  The j-force accumulator moves one lane a step (from lane src = l + 1
// of the record) and after a group's eight steps lane l holds entry (l + 7) & 7, whose atom it
// adds to.  LJ from (-6 C6, 12 C12): with p = 12 C12 r^-6 the force factor is (p - 6 C6) r^-8
// and six times the energy (p / 2 - 6 C6) r^-6.
// Why two i atoms a lane: the shared-memory and shuffle pipe (one 128-byte wavefront a cycle
// per SM) bounds the loop.  A step of 64 pairs reads one j position (4 wavefronts), one type
// (1), one LJ record (4) and shuffles one force (3): 12, where one i atom and two entries a
// lane took 20 (two positions, two forces); without the LJ term (LJ = false) it is 7.  Measured
// on 64 replicas (883,000 atoms): 1,612 us with one i atom a lane, 1,494 so, 1,346 with images
// by tile and 1,290 with the groups without an LJ term; on 99,200 atoms 190, 179, 180 and 165,
// on 22,700 atoms 59, 52, 54 and 51 (the third with the positions by atom), each with the i
// atoms' sums over a record's 32 terms.
// The i atoms' sums: a group's eight entries stand close together and are of one kind (hydrogens,
// say), so their forces on an atom mostly have one sign and a sum of many of them is large
// before the other kind takes it back.  So four terms, plus four, then into fixed point: the
// forces' error against FP64 (RMS, relative, mean of 27 systems of 2,100 to 15,300 atoms) is
// 1.016e-6; 1.018e-6 with one i atom a lane and 16 terms a sum, 1.023e-6 with eight terms in a
// row, 1.043e-6 with those groups added in FP32 (64 replicas 1,365 us, 99,200 atoms 171, 22,700
// atoms 52; in this form 1,307, 163 and 50).  58 % of the issue slots and 65 % of that pipe are
// busy, the FMA pipe 42 %.
// Half or quarter groups as work units of small lists measured slower (the per-record work).
template <bool MINIMG, bool COUNT, bool TRI, bool CLS, bool LJ>
__device__ __forceinline__ void group_packed(const DevPtrs& P, const QuadStage& S, const float2* __restrict__ s_lj,
                                              const float4* __restrict__ s_lj3, int rowa, int rowb,
                                             const PackedArgs& A, int g, int sp, int st, int sat, int src,
                                             long long (&gia)[3], long long (&gib)[3], double& te, double& tl,
                                             int& tn, double& ea, double& eb) {
  const unsigned full = 0xffffffffu;
  const float2 zb2 = make_float2(A.zb, A.zb), mzc = make_float2(-A.zc, -A.zc), mzf = make_float2(-A.zf, -A.zf);
  const float2 half2 = make_float2(0.5f, 0.5f);
  float bx = 0.f, by = 0.f, bz = 0.f, ibx = 0.f, iby = 0.f, ibz = 0.f;
  if (MINIMG) {
    const float* rp = S.rep[(threadIdx.x & 31) >> 3];
    bx = rp[0]; by = rp[1]; bz = rp[2];
    ibx = rp[3]; iby = rp[4]; ibz = rp[5];
  }
  const float4* __restrict__ pp = S.p + sp + 16 * g;
  int tj = LJ ? S.at[st + 8 * g].y : 0;
  if (CLS && LJ) tj &= kTypeMask;
  const unsigned ma = A.ma >> (8 * g), mb = A.mb >> (8 * g);
  const unsigned jc = CLS ? A.jc >> (8 * g) : 0u;
  float2 fx = make_float2(0.f, 0.f), fy = fx, fz = fx, hx = fx, hy = fx, hz = fx;   // minus the i forces
  float gx = 0.f, gy = 0.f, gz = 0.f;   // minus the j force of the entry this lane meets
  float2 te4 = make_float2(0.f, 0.f), tl4 = te4;
  float ea4 = 0.f, eb4 = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float4 j = pp[k];
    float2 dx = __fadd2_rn(make_float2(j.x, j.x), A.nx);   // x_j - x_i
    float2 dy = __fadd2_rn(make_float2(j.y, j.y), A.ny);
    float2 dz = __fadd2_rn(make_float2(j.z, j.z), A.nz);
    if (MINIMG) {
      dx = __ffma2_rn(make_float2(-bx, -bx), rint2(__fmul2_rn(dx, make_float2(ibx, ibx))), dx);
      dy = __ffma2_rn(make_float2(-by, -by), rint2(__fmul2_rn(dy, make_float2(iby, iby))), dy);
      dz = __ffma2_rn(make_float2(-bz, -bz), rint2(__fmul2_rn(dz, make_float2(ibz, ibz))), dz);
    }
    const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
    const bool ia = ((ma >> k) & 1u) && r2.x <= A.rc2;
    const bool ib = ((mb >> k) & 1u) && r2.y <= A.rc2;
    const float2 rinv = make_float2(rsqrt_ftz(ia ? r2.x : 1e30f), rsqrt_ftz(ib ? r2.y : 1e30f));
    const float2 r2i = __fmul2_rn(rinv, rinv);
    float2 r6 = make_float2(0.f, 0.f), m6 = r6, p12 = r6;   // -6 C6, 12 C12
    if (LJ) {
      r6 = __fmul2_rn(__fmul2_rn(r2i, r2i), r2i);
      if (TRI) {
        const float4 lj = s_lj3[rowa + tj];
        m6 = make_float2(lj.x, lj.y);
        p12 = make_float2(lj.z, lj.w);
      } else {
        const float2 lja = s_lj[rowa + tj], ljb = s_lj[rowb + tj];
        m6 = make_float2(lja.x, ljb.x);
        p12 = make_float2(lja.y, ljb.y);
      }
    }
    const float2 qf = __fmul2_rn(A.qi, make_float2(j.w, j.w));
    const float2 qq = make_float2(ia ? qf.x : 0.f, ib ? qf.y : 0.f);
    const float2 p = __fmul2_rn(p12, r6);
    const float2 h = __ffma2_rn(p, half2, m6);
    const float2 c = __fadd2_rn(rinv, __ffma2_rn(zb2, r2, mzc));
    const float2 fc = __ffma2_rn(rinv, r2i, mzf);
    float2 fs = LJ ? __ffma2_rn(qq, fc, __fmul2_rn(__fadd2_rn(p, m6), __fmul2_rn(r6, r2i))) : __fmul2_rn(qq, fc);
    if (CLS) {   // the pair's class from the number of cluster atoms in it
      const float2 eel = __fmul2_rn(qq, c), elj = LJ ? __fmul2_rn(h, r6) : make_float2(0.f, 0.f);
      te4 = __fadd2_rn(te4, eel);
      if (LJ) tl4 = __fadd2_rn(tl4, elj);
      const bool cj = ((jc >> k) & 1u) != 0u;
      const float2 e2 = LJ ? __ffma2_rn(elj, make_float2(1.f / 6.f, 1.f / 6.f), eel) : eel;
      ea4 += (cj && A.ca ? e2.x : 0.f) + (cj && A.cb ? e2.y : 0.f);
      eb4 += (cj != A.ca ? e2.x : 0.f) + (cj != A.cb ? e2.y : 0.f);
      fs = __fmul2_rn(fs, cj ? A.w1 : A.w0);
    } else {
      te4 = __ffma2_rn(qq, c, te4);
      if (LJ) tl4 = __ffma2_rn(h, r6, tl4);
    }
    fx = __ffma2_rn(dx, fs, fx);
    fy = __ffma2_rn(dy, fs, fy);
    fz = __ffma2_rn(dz, fs, fz);
    gx = fmaf(dx.y, fs.y, fmaf(dx.x, fs.x, gx));
    gy = fmaf(dy.y, fs.y, fmaf(dy.x, fs.x, gy));
    gz = fmaf(dz.y, fs.y, fmaf(dz.x, fs.x, gz));
    if (COUNT) tn += (ia ? 1 : 0) + (ib ? 1 : 0);
    if (k < 7) {
      gx = __shfl_sync(full, gx, src);
      gy = __shfl_sync(full, gy, src);
      gz = __shfl_sync(full, gz, src);
      if (LJ) tj = __shfl_sync(full, tj, src);
    }
    if (k == 3) {   // i forces: four terms plus four
      hx = fx; hy = fy; hz = fz;
      fx = fy = fz = make_float2(0.f, 0.f);
    }
    if (k == 3 || k == 7) {   // energies: FP32 over 4 steps, then FP64
      te += (double)te4.x + (double)te4.y;
      if (LJ) tl += (double)tl4.x + (double)tl4.y;
      te4 = tl4 = make_float2(0.f, 0.f);
      if (CLS) {
        ea += (double)ea4;
        eb += (double)eb4;
        ea4 = eb4 = 0.f;
      }
    }
  }
  add_forces(P.status, __fadd2_rn(fx, hx), __fadd2_rn(fy, hy), __fadd2_rn(fz, hz), gia, gib);
  const int aj = S.at[sat + 8 * g].x;
  if (aj >= 0 && (gx != 0.f || gy != 0.f || gz != 0.f)) {
    atomic_add_ll(&P.frc[3 * aj + 0], to_fix_f(-gx, P.status));
    atomic_add_ll(&P.frc[3 * aj + 1], to_fix_f(-gy, P.status));
    atomic_add_ll(&P.frc[3 * aj + 2], to_fix_f(-gz, P.status));
  }
}

// ljg: bit g set if some entry 8 g .. 8 g + 7 of the warp's four records has an LJ term
template <bool MINIMG, bool COUNT, bool TRI, bool CLS>
__device__ __forceinline__ void record_packed(const DevPtrs& P, const QuadStage& S, const float2* __restrict__ s_lj,
                                              const float4* __restrict__ s_lj3, int rowa, int rowb,
                                              const PackedArgs& A, unsigned ljg, int sp, int st, int sat, int src,
                                              long long (&gia)[3], long long (&gib)[3], double& te, double& tl,
                                              int& tn, double& ea, double& eb) {
  // in the groups' order whatever the neighbouring records are (the sums must not depend on
  // where a record stands); a run of groups of one form is a loop of its own
  int g = 0;
#pragma unroll 1
  do {
#pragma unroll 1
    for (; (ljg >> g) & 1u; ++g)
      group_packed<MINIMG, COUNT, TRI, CLS, true>(P, S, s_lj, s_lj3, rowa, rowb, A, g, sp, st, sat, src, gia, gib, te,
                                                  tl, tn, ea, eb);
#pragma unroll 1
    for (; g < 4 && !((ljg >> g) & 1u); ++g)
      group_packed<MINIMG, COUNT, TRI, CLS, false>(P, S, s_lj, s_lj3, rowa, rowb, A, g, sp, st, sat, src, gia, gib, te,
                                                   tl, tn, ea, eb);
  } while (g < 4);
}

// what a lane gathers for a record group before computing it: the positions (in their own
// blocks' frames, with the charge) of entries 8 g + l of its record, and its record's unit
// (-1: none)
struct Gather4 {
  float4 p[4];
  int unit;
};

// dynamic shared memory of the packed kernel: the stages, then the LJ table -- type triples
// (i type, i type, j type) up to kTriMaxTypes types, where two blocks still fit an SM
// (85 KB of stages + 28 KB of table each), type pairs above (two 8-byte reads a step)
constexpr int kTriMaxTypes = 12;
__host__ __device__ constexpr bool lj_tri(int nt1) { return nt1 <= kTriMaxTypes; }
__host__ __device__ constexpr size_t lj_bytes(int nt1) {
  return lj_tri(nt1) ? (size_t)nt1 * nt1 * nt1 * 16 : ((size_t)nt1 * nt1 * 8 + 15) / 16 * 16;
}
constexpr size_t kPackedStageBytes = sizeof(QuadStage) * kPairWarps;

// CLS: every record with class weights and energies; without it cls_sum adds the energies to class
// BB.  which: the records at the start of the arrays (1), at their end (2), or both (3), those at
// the end first.  Without classes these are the records whose pairs take their own images: the
// two image forms' code does not fit the instruction cache together, and with both kinds of
// records in turn 200 replicas in boxes of 28 A took 1,134 us, 20 in boxes of 39 A 275; with one
// kind after the other 697 and 210.
template <bool COUNT, bool CLS, bool TRI>
__global__ void __launch_bounds__(kPairThreads, CLS ? 1 : 2) k_pair_packed(DevPtrs P, ZdConst z, int which, int cls_sum) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  __shared__ unsigned long long s_tab_bar;
  const unsigned full = 0xffffffffu;
  QuadStage& S = reinterpret_cast<QuadStage*>(s_dyn)[threadIdx.x >> 5];
  const float2* s_lj = reinterpret_cast<const float2*>(s_dyn + kPackedStageBytes);
  const float4* s_lj3 = reinterpret_cast<const float4*>(s_dyn + kPackedStageBytes);
  const int lane = threadIdx.x & 31;
  const int qd = lane >> 3, lp = lane & 7;              // record of the group, lane inside it
  const int sp = 64 * qd + lp, sta = 36 * qd + lp;      // this lane's staging slots
  const int sat = 36 * qd + ((lp + 7) & 7);
  const int src = (lane & 24) | ((lp + 1) & 7);         // rotation: from the next lane of the record
  for (int k = lp; k < 12; k += 8) S.rep[qd][k] = k < 6 ? 0.f : 1.f;   // a record group past the list
  if (lane == 0) {
    mbar_init(&S.bar[0]);
    mbar_init(&S.bar[1]);
  }
  if (threadIdx.x == 0) {
    mbar_init(&s_tab_bar);
    mbar_expect(&s_tab_bar, (unsigned)lj_bytes(z.nt1));
    bulk_load(s_dyn + kPackedStageBytes, P.lj_tab, (unsigned)lj_bytes(z.nt1), &s_tab_bar);
  }
  __syncthreads();
  // records at the arrays' start and end; the record groups at the end come first, downwards
  const int T0 = which & 1 ? P.nctiles[0] : 0, T1 = which & 2 ? P.nctiles[1] : 0;
  const int U1 = (T1 + 3) >> 2;
  // the first record of group t's copies
  auto rec0 = [&](int t) { return t < U1 ? P.rec_cap - 4 * (size_t)(t + 1) : 4 * (size_t)(t - U1); };
  // every pair takes its own image: after replaced coordinates (below), or where most records need
  // it and the others cannot stand apart (the ALSD records without classes): one form's code
  const bool all_img = (*P.ext_pos & kExtImg) != 0 || 2 * (long long)P.nctiles[2] > T0;
  const int TU = U1 + ((T0 + 3) >> 2);   // record groups: a warp's work units
  // a 2.5-KiB copy lands in microseconds; the bound (about a second of SM clock) only ends
  // the wait on a broken device, and it is not the integrator's adjustable barrier bound:
  // a block must never leave with one of its copies still in flight
  const long long wlim = kCopyWaitCycles;
  unsigned phase = 0u, pend = 0u;   // per buffer: barrier parity to wait for; copy in flight
  bool ok = true;

  // record groups are claimed in runs of `run` consecutive ones: the records of a unit are
  // consecutive, so a run mostly keeps its i atoms; the run is short enough that every warp
  // still gets several.  A warp's first run goes by its index, without the counter's latency;
  // a list that these runs cover makes no claim at all.
  const int gw = blockIdx.x * kPairWarps + (threadIdx.x >> 5), nw = gridDim.x * kPairWarps;
  const int run = max(1, min(8, TU / (nw * 8)));
  int run_next = min(gw * run, TU), run_end = min(run_next + run, TU);
  auto claim = [&]() {
    if (run_next >= run_end) {
      if (nw * run >= TU) return TU;
      int t = 0;
      if (lane == 0) t = atomicAdd(&P.tile_ctr[which == 2 ? 1 : 0], run);
      t = __shfl_sync(full, t, 0) + nw * run;
      run_next = t;
      run_end = min(t + run, TU);
    }
    return run_next < run_end ? run_next++ : TU;
  };
  // the entries, types and masks of group t's four records into buffer b (up to three past
  // the last record of the sequence lie inside the arrays: read, never used)
  auto issue = [&](int t, int b) {
    if (lane == 0) {
      const size_t r0 = rec0(t);
      fence_proxy_async();
      mbar_expect(&S.bar[b], 2560u);
      bulk_load(S.ent[b], P.ct_j + r0 * 32, 2048u, &S.bar[b]);
      bulk_load(S.ty[b], P.ct_ty + r0 * 32, 256u, &S.bar[b]);
      bulk_load(S.msk[b], P.ct_mask + r0 * kHalf, 256u, &S.bar[b]);
    }
    pend |= 1u << b;
  };
  // group t's copy has landed in buffer b: start the gathers of this lane's four entries
  auto fetch = [&](int t, int b, Gather4& G) {
    if (!mbar_wait_warp(&S.bar[b], (phase >> b) & 1u, wlim)) {
      ok = false;
      atomicOr(P.status, ERR_TIMEOUT);
      return;
    }
    phase ^= 1u << b;
    pend &= ~(1u << b);
    const bool valid = t < U1 ? 4 * t + 3 - qd < T1 : 4 * (t - U1) + qd < T0;
    G.unit = valid ? P.ct_blk[rec0(t) + qd] : -1;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int aj = valid ? __float_as_int(S.ent[b][32 * qd + 8 * g + lp].w) : -1;
      G.p[g] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (aj >= 0) G.p[g] = P.pos_f[aj];
    }
  };

  PackedArgs A;
  A.rc2 = (float)z.rc2; A.zb = (float)z.bcoeff; A.zf = (float)z.fcoeff; A.zc = (float)z.zcore;
  A.nx = A.ny = A.nz = A.qi = make_float2(0.f, 0.f);
  A.jc = 0u;
  A.ca = A.cb = false;
  A.w0 = A.w1 = make_float2(1.f, 1.f);   // set where a record holds classes
  int cur_unit = -2, cur_rep = -1, rep = -1, aia = -1, aib = -1, tia = z.nt1 - 1, tib = tia;
  long long gia[3] = {0, 0, 0}, gib[3] = {0, 0, 0};
  long long eel = 0, elj = 0, eaa = 0, eab = 0;
  long long npair = 0;
  auto flush_i = [&]() {
    if (aia >= 0 && (gia[0] | gia[1] | gia[2]))
      for (int k = 0; k < 3; ++k) atomic_add_ll(&P.frc[3 * aia + k], gia[k]);
    if (aib >= 0 && (gib[0] | gib[1] | gib[2]))
      for (int k = 0; k < 3; ++k) atomic_add_ll(&P.frc[3 * aib + k], gib[k]);
    for (int k = 0; k < 3; ++k) gia[k] = gib[k] = 0;
  };
  // Where a warp's runs are short, a unit's records go to many warps and all add to the same i
  // atoms at once: the four lane groups' sums are then added first if they are of one unit
  // (called by all lanes; mine: the lane's unit ends).  9,300 atoms inside their cut-off 137 us
  // without and 97 with it, 48,000 atoms 97 and 90; with longer runs it costs (64 replicas 1,310
  // and 1,323 us).
  const bool merge = run <= 2;
  auto merge_i = [&](bool mine) {
    const int u0 = __shfl_sync(full, cur_unit, 0);   // by every lane, whatever its `mine`
    if (!__all_sync(full, mine && cur_unit == u0)) return;
    for (int o = 8; o < 32; o <<= 1)
      for (int k = 0; k < 3; ++k) {
        gia[k] += __shfl_xor_sync(full, gia[k], o);
        gib[k] += __shfl_xor_sync(full, gib[k], o);
      }
    if (qd != 0)
      for (int k = 0; k < 3; ++k) gia[k] = gib[k] = 0;
  };

  int t = claim(), tn = TU;
  Gather4 G;
  if (t < TU) {
    issue(t, 0);
    tn = claim();
    if (tn < TU) issue(tn, 1);
    fetch(t, 0, G);
  }
  if (!mbar_wait_warp(&s_tab_bar, 0u, wlim)) {
    ok = false;
    atomicOr(P.status, ERR_TIMEOUT);
  }
  int b = 0;
  while (t < TU && ok) {
    // this lane's four entries into the stage, twice
    __syncwarp();
    unsigned jc = 0u;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      // buffer b still holds this group's entries, types and masks (a record past the last one:
      // no atom, the zero dummy type).  The shift into the i block's frame waits
      // until here, as nothing may use a gather's result before the last group's arithmetic
      const float4 e = S.ent[b][32 * qd + 8 * g + lp];
      const float4 q = make_float4(G.p[g].x - e.x, G.p[g].y - e.y, G.p[g].z - e.z, G.p[g].w);
      S.p[sp + 16 * g] = q;
      S.p[sp + 16 * g + 8] = q;
      const int2 ta = G.unit >= 0 ? make_int2(__float_as_int(e.w), type_word(S.ty[b][32 * qd + 8 * g + lp]))
                                  : make_int2(-1, z.nt1 - 1);
      S.at[sta + 8 * g] = ta;
      if (CLS) jc |= ((__ballot_sync(full, (ta.y >> 30) & 1) >> (8 * qd)) & 0xffu) << (8 * g);
    }
    const int unit = G.unit >= 0 ? G.unit & kRecUnit : -1;
    A.ma = unit >= 0 ? step_mask(S.msk[b][16 * qd + lp], lp) : 0u;
    A.mb = unit >= 0 ? step_mask(S.msk[b][16 * qd + 8 + lp], lp + 8) : 0u;
    // the lane's i atoms: a new unit flushes the last one's forces and loads the new atoms
    if (merge && __any_sync(full, unit != cur_unit)) merge_i(unit != cur_unit);
    if (unit != cur_unit) {
      flush_i();
      cur_unit = unit;
      if (unit >= 0) {
        const int si = unit * kHalf + lp;
        aia = P.satom[si];
        aib = P.satom[si + 8];
        const float4 pa = aia >= 0 ? P.pos_f[aia] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 pb = aib >= 0 ? P.pos_f[aib] : make_float4(0.f, 0.f, 0.f, 0.f);
        A.nx = make_float2(-pa.x, -pb.x);
        A.ny = make_float2(-pa.y, -pb.y);
        A.nz = make_float2(-pa.z, -pb.z);
        A.qi = make_float2(pa.w, pb.w);
        tia = P.styp[si];
        tib = P.styp[si + 8];
        rep = P.blk_rep[unit >> 1];
      } else {
        A.nx = A.ny = A.nz = A.qi = make_float2(0.f, 0.f);
        tia = tib = z.nt1 - 1;
        aia = aib = -1;
      }
    }
    // a new replica in any record: every record's energies go to its replica so far
    if (__any_sync(full, rep != cur_rep)) {
      flush_fix<8>(P, cur_rep, eel, elj, eaa, eab, npair, COUNT, CLS || cls_sum);
      eel = elj = eaa = eab = 0;
      npair = 0;
      if (rep != cur_rep) {
        cur_rep = rep;
        const Rep& R = P.reps[rep];
        if (lp < 6) S.rep[qd][lp] = (float)(lp < 3 ? R.box[lp] : R.invbox[lp - 3]);
        if (CLS && lp < 3) S.rep[qd][6 + lp] = (float)cls_weight(R, P.lam[2 * rep], 2 - lp);
      }
    }
    // Per-pair minimum image is needed only where a pair within the cut-off can have another image
    // than its tile's: the list build flags the records with such a tile (k_block_list).
    // Coordinates replaced without a build since may have moved farther than its margin: then
    // every pair takes its own, unless no box of the context can need it (k_update_pos).  One
    // form for the whole warp.
    const bool wmi = all_img || __any_sync(full, G.unit >= 0 && (G.unit & kRecImg));
    // (a record past the last one, -1, has every flag set)
    const unsigned ljg = (~__reduce_and_sync(full, (unsigned)G.unit) >> kRecFree) & 0xfu;
    __syncwarp();
    // buffer b is free again: the group after next goes into it; the next group's gathers
    // are issued before this group's arithmetic
    int t2 = TU;
    if (tn < TU) {
      t2 = claim();
      if (t2 < TU) issue(t2, b);
    }
    if (tn < TU) fetch(tn, b ^ 1, G);
    double te = 0.0, tl = 0.0;
    int tn_pairs = 0;
    const int ka = CLS ? (tia & kTypeMask) : tia, kb = CLS ? (tib & kTypeMask) : tib;
    const int rowa = TRI ? (ka * z.nt1 + kb) * z.nt1 : ka * z.nt1, rowb = kb * z.nt1;
    double ea = 0.0, eb = 0.0;
    if (CLS) {
      const float f0 = S.rep[qd][6], f1 = S.rep[qd][7], f2 = S.rep[qd][8];
      A.ca = ((tia >> 30) & 1) != 0;
      A.cb = ((tib >> 30) & 1) != 0;
      A.jc = byte_rotr(jc, lp);
      A.w0 = make_float2(A.ca ? f1 : f0, A.cb ? f1 : f0);
      A.w1 = make_float2(A.ca ? f2 : f1, A.cb ? f2 : f1);
    }
    // (classes: with per-pair images always, which change nothing where they are not needed)
    if (CLS || wmi)
      record_packed<true, COUNT, TRI, CLS>(P, S, s_lj, s_lj3, rowa, rowb, A, ljg, sp, sta, sat, src, gia, gib, te, tl,
                                           tn_pairs, ea, eb);
    else
      record_packed<false, COUNT, TRI, CLS>(P, S, s_lj, s_lj3, rowa, rowb, A, ljg, sp, sta, sat, src, gia, gib, te, tl,
                                            tn_pairs, ea, eb);
    if (CLS) {
      eaa += to_fix(ea, kEneScale, P.status);
      eab += to_fix(eb, kEneScale, P.status);
    }
    eel += to_fix(te, kEneScale, P.status);
    elj += to_fix(tl * (1.0 / 6.0), kEneScale, P.status);
    if (COUNT) npair += tn_pairs;
    t = tn;
    tn = t2;
    b ^= 1;
  }
  if (merge) merge_i(true);
  flush_i();
  flush_block<8, kPairWarps>(P, cur_rep, eel, elj, eaa, eab, npair, COUNT, CLS || cls_sum);
  // a copy still in flight (only after a timed-out wait) must land before the block exits
  for (int k = 0; k < 2; ++k)
    if ((pend >> k) & 1u) mbar_wait(&S.bar[k], (phase >> k) & 1u, wlim);
}

// what a lane gathers for a record pair before computing it: its two j entries a = l and
// b = 16 + l of its record (position in the i block's frame with the charge, type word,
// atom), its mask rows and its record's unit (-1: no record)
struct Gather {
  float4 pa, pb;
  int ta, tb, aa, ab;
  unsigned m, me;
  int unit;
};

// One pair in the scalar form, branch-free like the packed step: d = x_i - x_j, and the
// force scalar fs (F = -fs d on the i atom) and energies, all zero outside the mask (`bit`)
// or the cut-off.  CMM: the Coulomb term only where `elbit` is set.
template <bool MINIMG, bool CMM>
__device__ __forceinline__ void pair_scalar(float4 pi, float xj, float yj, float zj, float qj, float2 lj,
                                            bool bit, bool elbit, float bx, float by, float bz, float ibx,
                                            float iby, float ibz, float rc2, float zb, float zf, float zc,
                                            float& dx, float& dy, float& dz, float& fs, float& eel,
                                            float& elj, bool& in) {
  dx = pi.x - xj;
  dy = pi.y - yj;
  dz = pi.z - zj;
  if (MINIMG) {
    dx = fmaf(-bx, rint1(dx * ibx), dx);
    dy = fmaf(-by, rint1(dy * iby), dy);
    dz = fmaf(-bz, rint1(dz * ibz), dz);
  }
  const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  in = bit && r2 <= rc2;
  const float rinv = rsqrt_ftz(in ? r2 : 1.f);
  const float r2inv = rinv * rinv;
  const float r6inv = r2inv * r2inv * r2inv;
  const float qq = (CMM ? elbit : true) ? pi.w * qj : 0.f;
  const float v1 = lj.x * r6inv;
  const float v2 = lj.y * r6inv * r6inv;
  const float e1 = qq * (rinv + fmaf(zb, r2, -zc));
  const float e2 = v2 - v1;
  const float f = fmaf(qq, fmaf(rinv, r2inv, -zf), fmaf(12.f, v2, -6.f * v1) * r2inv);
  fs = in ? f : 0.f;
  eel = in ? e1 : 0.f;
  elj = in ? e2 : 0.f;
}

// One record in the scalar form (CMM and partial-McMD variants): at step k (k < 16) lane l of
// the half-warp meets entries a = (l + k) & 15 and b = 16 + a, staged at sidx + k (sidx =
// 32 h + l), one after the other.  The j-force accumulators of a and b move one lane per step
// (from lane src = l + 1 of the same half); after 16 steps lane l holds those of entries l and
// 16 + l.  SPLIT (partial McMD): the pair's class from the regions of its atoms (bit cj of
// trow: class 1), the class-1 forces in accumulators of their own (fi[3..5], gj[6..11],
// rotated like the others) and the class-1 energy in ea.  CMM: no cut-off (rc2 is huge) and
// the Coulomb term only for the pairs of `me`.  gj[0..5]: entries a and b.
template <bool MINIMG, bool COUNT, bool CMM, bool SPLIT>
__device__ __forceinline__ void tile_scalar(const MixStage& S, const float2* __restrict__ s_lj, int row,
                                            float4 pi, unsigned m, unsigned me, int sidx, int src, float bx,
                                            float by, float bz, float ibx, float iby, float ibz, float rc2,
                                            float zb, float zf, float zc, float (&fi)[6], float (&gj)[12],
                                            double& te, double& tl, int& tn, unsigned trow, double& ea) {
  const unsigned full = 0xffffffffu;
  constexpr int NG = SPLIT ? 12 : 6;
#pragma unroll 1
  for (int k0 = 0; k0 < 16; k0 += 4) {
    float te4 = 0.f, tl4 = 0.f, ea4 = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 a = S.p2[sidx + k0 + k];
      const float4 b = S.q2[sidx + k0 + k];
      const int2 t = S.t2[sidx + k0 + k];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int tj = e ? t.y : t.x;
        const int sh = k0 + k + 16 * e;
        const float2 lj = s_lj[row + (SPLIT ? (tj & kTypeMask) : tj)];
        float dx, dy, dz, fs, eel, elj;
        bool in;
        pair_scalar<MINIMG, CMM>(pi, e ? a.y : a.x, e ? a.w : a.z, e ? b.y : b.x, e ? b.w : b.z, lj,
                                 ((m >> sh) & 1u) != 0u, ((me >> sh) & 1u) != 0u, bx, by, bz, ibx, iby, ibz,
                                 rc2, zb, zf, zc, dx, dy, dz, fs, eel, elj, in);
        te4 += eel;
        tl4 += elj;
        float fs1 = 0.f;
        if (SPLIT) {
          const bool c1 = ((trow >> ((tj >> kRegionShift) & 3)) & 1u) != 0u;
          ea4 += c1 ? eel + elj : 0.f;
          fs1 = c1 ? fs : 0.f;
          fs -= fs1;
        }
        const float fx = dx * fs, fy = dy * fs, fz = dz * fs;
        fi[0] -= fx; fi[1] -= fy; fi[2] -= fz;
        gj[3 * e + 0] += fx; gj[3 * e + 1] += fy; gj[3 * e + 2] += fz;
        if (SPLIT) {
          const float hx = dx * fs1, hy = dy * fs1, hz = dz * fs1;
          fi[3] -= hx; fi[4] -= hy; fi[5] -= hz;
          gj[6 + 3 * e + 0] += hx; gj[6 + 3 * e + 1] += hy; gj[6 + 3 * e + 2] += hz;
        }
        if (COUNT) tn += (in && (CMM ? ((me >> sh) & 1u) != 0u : true)) ? 1 : 0;
      }
#pragma unroll
      for (int q = 0; q < NG; ++q) gj[q] = __shfl_sync(full, gj[q], src);
    }
    te += (double)te4;
    tl += (double)tl4;
    if (SPLIT) ea += (double)ea4;
  }
}

template <bool COUNT, bool CMM, bool SPLIT>
__global__ void __launch_bounds__(kPairThreads, 2)
k_pair_mixed(DevPtrs P, ZdConst z) {
  extern __shared__ float2 s_lj[];
  __shared__ MixStage s_stage[kPairWarps];
  const unsigned full = 0xffffffffu;
  const int nlj = z.nt1 * z.nt1;
  for (int i = threadIdx.x; i < nlj; i += blockDim.x) s_lj[i] = P.lj_f[i];
  const int lane = threadIdx.x & 31;
  const int hw = lane >> 4, lp = lane & (kHalf - 1);   // half-warp, lane inside it
  const int sidx = 32 * hw + lp;                        // this lane's staging slot
  const int src = ((lp + 1) & (kHalf - 1)) | (hw << 4); // rotation: from the next lane of the half
  MixStage& S = s_stage[threadIdx.x >> 5];
  if (lane == 0) {
    mbar_init(&S.bar[0]);
    mbar_init(&S.bar[1]);
  }
  __syncthreads();
  const int T = *P.nctiles;         // records
  const int TU = (T + 1) >> 1;      // record pairs: a warp's work units
  // a 1.2-KiB copy lands in microseconds; the bound (about a second of SM clock) only ends
  // the wait on a broken device, and it is not the integrator's adjustable barrier bound:
  // a block must never leave with one of its copies still in flight
  const long long wlim = kCopyWaitCycles;
  const float rc2 = (float)z.rc2, zb = (float)z.bcoeff, zf = (float)z.fcoeff, zc = (float)z.zcore;
  const unsigned txb = CMM ? 1280u : 1152u;
  unsigned phase = 0u, pend = 0u;   // per buffer: barrier parity to wait for; copy in flight
  bool ok = true;

  // record pairs are claimed in runs of `run` consecutive ones: the records of a unit are
  // consecutive, so a run mostly keeps its i atoms (no reload, no i-force flush between
  // records); the run is short enough that every warp still gets several (8 per warp at most
  // of the total, 1 to 16 pairs)
  const int run = max(1, min(16, TU / (int)(gridDim.x * kPairWarps * 8)));
  int run_next = 0, run_end = 0;
  auto claim = [&]() {
    if (run_next >= run_end) {
      int t = 0;
      if (lane == 0) t = atomicAdd(P.tile_ctr, run);
      t = __shfl_sync(full, t, 0);
      run_next = t;
      run_end = min(t + run, TU);
    }
    return run_next < run_end ? run_next++ : TU;
  };
  // the entries and masks of records 2t and 2t + 1 into buffer b (one past the last record
  // is padding inside the arrays: read, never used)
  auto issue = [&](int t, int b) {
    if (lane == 0) {
      fence_proxy_async();
      mbar_expect(&S.bar[b], txb);
      bulk_load(S.ent[b], P.ct_j + (size_t)t * 64, 1024u, &S.bar[b]);
      bulk_load(S.msk[b], P.ct_mask + (size_t)t * 32, 128u, &S.bar[b]);
      if (CMM) bulk_load(S.msk_el[b], P.ct_mask_el + (size_t)t * 32, 128u, &S.bar[b]);
    }
    pend |= 1u << b;
  };
  auto gather1 = [&](float4 e, bool valid, float4& p, int& ty, int& at) {
    at = valid ? __float_as_int(e.w) : -1;
    if (at >= 0) {
      const float4 q = P.pos_f[at];
      p = make_float4(q.x - e.x, q.y - e.y, q.z - e.z, q.w);   // into the i block's frame
      ty = P.typ[at];
    } else {
      p = make_float4(0.f, 0.f, 0.f, 0.f);
      ty = z.nt1 - 1;   // the zero dummy type
    }
  };
  // pair t's copy has landed in buffer b: start the gathers of this lane's two entries
  auto fetch = [&](int t, int b, Gather& G) {
    if (!mbar_wait_warp(&S.bar[b], (phase >> b) & 1u, wlim)) {
      ok = false;
      atomicOr(P.status, ERR_TIMEOUT);
      return;
    }
    phase ^= 1u << b;
    pend &= ~(1u << b);
    const int rec = 2 * t + hw;
    const bool valid = rec < T;
    G.m = valid ? S.msk[b][lane] : 0u;
    G.me = CMM && valid ? S.msk_el[b][lane] : 0u;
    G.unit = valid ? P.ct_blk[rec] & kRecUnit : -1;
    gather1(S.ent[b][32 * hw + lp], valid, G.pa, G.ta, G.aa);
    gather1(S.ent[b][32 * hw + kHalf + lp], valid, G.pb, G.tb, G.ab);
  };

  int cur_unit = -2, cur_rep = -1, rep = -1, ai = -1, ti = 0;
  float4 pi = make_float4(0.f, 0.f, 0.f, 0.f);
  long long gix = 0, giy = 0, giz = 0;
  long long gix1 = 0, giy1 = 0, giz1 = 0;   // partial McMD: class-1 i forces
  long long eel = 0, elj = 0, eaa = 0;
  long long npair = 0;
  bool mi = false;
  float bx = 0.f, by = 0.f, bz = 0.f, ibx = 0.f, iby = 0.f, ibz = 0.f;
  unsigned tab = 0u;

  int t = claim(), tn = TU;
  Gather G;
  if (t < TU) {
    issue(t, 0);
    tn = claim();
    if (tn < TU) issue(tn, 1);
    fetch(t, 0, G);
  }
  int b = 0;
  while (t < TU && ok) {
    // this lane's two entries into the stage, twice
    __syncwarp();
    {
      const float4 p2 = make_float4(G.pa.x, G.pb.x, G.pa.y, G.pb.y);
      const float4 q2 = make_float4(G.pa.z, G.pb.z, G.pa.w, G.pb.w);
      const int2 t2 = make_int2(G.ta, G.tb);
      S.p2[sidx] = p2;
      S.p2[sidx + kHalf] = p2;
      S.q2[sidx] = q2;
      S.q2[sidx + kHalf] = q2;
      S.t2[sidx] = t2;
      S.t2[sidx + kHalf] = t2;
    }
    const unsigned m = G.m, me = G.me;
    const int aa = G.aa, ab = G.ab, unit = G.unit;
    // the lane's i atom: a new unit flushes the last one's force and loads the new atom
    if (unit != cur_unit) {
      if (ai >= 0 && (gix | giy | giz)) {
        atomic_add_ll(&P.frc[3 * ai + 0], gix);
        atomic_add_ll(&P.frc[3 * ai + 1], giy);
        atomic_add_ll(&P.frc[3 * ai + 2], giz);
      }
      if (SPLIT && ai >= 0 && (gix1 | giy1 | giz1)) {
        atomic_add_ll(&P.frc1[3 * ai + 0], gix1);
        atomic_add_ll(&P.frc1[3 * ai + 1], giy1);
        atomic_add_ll(&P.frc1[3 * ai + 2], giz1);
      }
      gix = giy = giz = 0;
      gix1 = giy1 = giz1 = 0;
      cur_unit = unit;
      if (unit >= 0) {
        const int si = (unit >> 1) * kTile + (unit & 1) * kHalf + lp;
        ti = P.styp[si];
        ai = P.satom[si];
        pi = ai >= 0 ? P.pos_f[ai] : make_float4(0.f, 0.f, 0.f, 0.f);
        rep = P.blk_rep[unit >> 1];
      } else {
        pi = make_float4(0.f, 0.f, 0.f, 0.f);
        ti = z.nt1 - 1;
        ai = -1;
      }
    }
    // a new replica in either half: both halves' energies go to their replicas so far
    if (__any_sync(full, rep != cur_rep)) {
      flush_fix<16>(P, cur_rep, eel, elj, eaa, 0, npair, COUNT, SPLIT);
      eel = elj = eaa = 0;
      npair = 0;
      if (rep != cur_rep) {
        cur_rep = rep;
        const Rep& R = P.reps[rep];
        bx = (float)R.box[0]; by = (float)R.box[1]; bz = (float)R.box[2];
        ibx = (float)R.invbox[0]; iby = (float)R.invbox[1]; ibz = (float)R.invbox[2];
        if (SPLIT) tab = R.split ? R.cls_tab : 0u;
        // Per-pair minimum image is needed only where a pair within the cut-off can have
        // another image than its tile's.  Per axis the tile's image puts the two block
        // references at most box/2 apart, and a pair's separation differs from theirs by at
        // most h_i + h_j <= 2 h_max plus the atoms' motion since the build (2 A margin), so
        // in the tile's image |d| <= box/2 + 2 h_max + 2; in any other image |d| >= box - rc.
        // Both hold at once only if box/2 <= rc + 2 h_max + 2.  CMM (no cut-off): the
        // farthest near-field pair rlim in place of rc, with twice the block margin.
        mi = false;
        for (int k = 0; k < 3; ++k) {
          const double h = (double)P.rep_hmax[3 * rep + k];
          const double reach = CMM ? z.rlim + 4.0 * h : sqrt(z.rc2) + 2.0 * h;
          if (0.5 * R.box[k] < reach + 2.0) mi = true;
        }
      }
    }
    const bool wmi = __any_sync(full, mi);   // one image form for the whole warp
    __syncwarp();
    // buffer b is free again: the pair after next goes into it; the next pair's gathers
    // are issued before this pair's arithmetic
    int t2 = TU;
    if (tn < TU) {
      t2 = claim();
      if (t2 < TU) issue(t2, b);
    }
    Gather Gn;
    if (tn < TU) fetch(tn, b ^ 1, Gn);
    double te = 0.0, tl = 0.0, ea = 0.0;
    int tn_pairs = 0;
    const int row = (SPLIT ? (ti & kTypeMask) : ti) * z.nt1;
    float fi6[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float gj[12] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const unsigned trow = SPLIT ? tab >> (3 * ((ti >> kRegionShift) & 3)) : 0u;
    if (wmi)
      tile_scalar<true, COUNT, CMM, SPLIT>(S, s_lj, row, pi, m, me, sidx, src, bx, by, bz, ibx, iby, ibz, rc2, zb,
                                           zf, zc, fi6, gj, te, tl, tn_pairs, trow, ea);
    else
      tile_scalar<false, COUNT, CMM, SPLIT>(S, s_lj, row, pi, m, me, sidx, src, bx, by, bz, ibx, iby, ibz, rc2,
                                            zb, zf, zc, fi6, gj, te, tl, tn_pairs, trow, ea);
    auto add_j = [&](long long* f, int aj, float3 g) {
      if (aj >= 0 && (g.x != 0.f || g.y != 0.f || g.z != 0.f)) {
        atomic_add_ll(&f[3 * aj + 0], to_fix_f(g.x, P.status));
        atomic_add_ll(&f[3 * aj + 1], to_fix_f(g.y, P.status));
        atomic_add_ll(&f[3 * aj + 2], to_fix_f(g.z, P.status));
      }
    };
    add_j(P.frc, aa, make_float3(gj[0], gj[1], gj[2]));
    add_j(P.frc, ab, make_float3(gj[3], gj[4], gj[5]));
    gix += to_fix_f(fi6[0], P.status);
    giy += to_fix_f(fi6[1], P.status);
    giz += to_fix_f(fi6[2], P.status);
    eel += to_fix(te, kEneScale, P.status);
    elj += to_fix(tl, kEneScale, P.status);
    if (SPLIT) {
      add_j(P.frc1, aa, make_float3(gj[6], gj[7], gj[8]));
      add_j(P.frc1, ab, make_float3(gj[9], gj[10], gj[11]));
      gix1 += to_fix_f(fi6[3], P.status);
      giy1 += to_fix_f(fi6[4], P.status);
      giz1 += to_fix_f(fi6[5], P.status);
      eaa += to_fix(ea, kEneScale, P.status);
    }
    if (COUNT) npair += tn_pairs;
    t = tn;
    tn = t2;
    G = Gn;
    b ^= 1;
  }
  if (ai >= 0 && (gix | giy | giz)) {
    atomic_add_ll(&P.frc[3 * ai + 0], gix);
    atomic_add_ll(&P.frc[3 * ai + 1], giy);
    atomic_add_ll(&P.frc[3 * ai + 2], giz);
  }
  if (SPLIT && ai >= 0 && (gix1 | giy1 | giz1)) {
    atomic_add_ll(&P.frc1[3 * ai + 0], gix1);
    atomic_add_ll(&P.frc1[3 * ai + 1], giy1);
    atomic_add_ll(&P.frc1[3 * ai + 2], giz1);
  }
  flush_fix<16>(P, cur_rep, eel, elj, eaa, 0, npair, COUNT, SPLIT);
  // a copy still in flight (only after a timed-out wait) must land before the block exits
  for (int k = 0; k < 2; ++k)
    if ((pend >> k) & 1u) mbar_wait(&S.bar[k], (phase >> k) & 1u, wlim);
}

// ---- FP64 kernel of the plain contexts ---------------------------------------------------------
// Four records a warp, eight lanes each, two i atoms a lane, as k_pair_packed, in FP64.  The FP64
// pipe bounds it (a warp instruction every 2.2 cycles of a scheduler), so the step holds
// nothing that can be done once per atom or by fewer instructions:
//  - Images.  Every atom is taken in its image nearest to the i block's reference.  A pair
//    within the cut-off then is in the right image if box/2 exceeds the cut-off plus the i
//    block's half extent plus the atoms' motion since the build (2 A): the j atom's image
//    within the cut-off of the i atom lies within half a box of the reference on every axis.
//    Else (a small box, or coordinates replaced without a build) each pair takes its own.
//  - 1/r by rsqrt_h3; the cut-off test on r^2 itself; LJ from (-6 C6, 12 C12) as in record_packed.
//  - Branch-free: a pair outside the mask or the cut-off has zero charge product and r^-1 = 0.
// On 22,700 atoms 144 us with one i atom a lane and an image, a division and a square root per
// pair, 93 with rsqrt() and the images per atom, 83 so (the FP64 pipe busy half the time), 72
// with the LJ term left out where a record group has none.
struct __align__(16) QuadStageD {
  double2 pxy[256], pzq[256];   // entry 8 g + e of record q at 64 q + 16 g + e, and 8 further on
  int2 at[4 * 36];              // (atom, type) of entry 8 g + e at 36 q + 8 g + e
};

// d's image nearest to zero (adding and subtracting 1.5 * 2^52 rounds to the nearest integer)
__device__ __forceinline__ double near_image(double d, double box, double inv) {
  const double n = __dadd_rn(__dadd_rn(d * inv, 6755399441055744.0), -6755399441055744.0);
  return fma(-box, n, d);
}

// 1/sqrt(x) from the hardware's approximation (on normal numbers within 2^-20.03, measured over
// 2^31 values of each of three ranges) by rsqrt_step; its largest error there was 1.27 x 2^-53
__device__ __forceinline__ double rsqrt_h3(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return rsqrt_step(x, y);
}

template <bool MINIMG, bool COUNT, bool LJ>
__device__ __forceinline__ void group_fp64(const DevPtrs& P, const QuadStageD& S, const double2* __restrict__ s_lj,
                                           int rowa, int rowb, const double (&xa)[4], const double (&xb)[4],
                                           unsigned ma, unsigned mb, int g, const double (&box)[3], const double (&inv)[3],
                                           double rc2, double zb, double zf, double zc, int sp, int st, int sat,
                                           int src, double (&fa)[3], double (&fb)[3], double& te, double& tl,
                                           int& tn) {
  const unsigned full = 0xffffffffu;
  const double2* __restrict__ pxy = S.pxy + sp + 16 * g;
  const double2* __restrict__ pzq = S.pzq + sp + 16 * g;
  int tj = LJ ? S.at[st + 8 * g].y : 0;
  double gx = 0.0, gy = 0.0, gz = 0.0;   // minus the j force of the entry this lane meets
#pragma unroll 2
  for (int k = 0; k < 8; ++k) {
    const double2 jxy = pxy[k], jzq = pzq[k];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const double* xi = e ? xb : xa;
      double dx = jxy.x - xi[0], dy = jxy.y - xi[1], dz = jzq.x - xi[2];   // x_j - x_i
      if (MINIMG) {
        dx = near_image(dx, box[0], inv[0]);
        dy = near_image(dy, box[1], inv[1]);
        dz = near_image(dz, box[2], inv[2]);
      }
      const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
      const bool in = (((e ? mb : ma) >> (8 * g + k)) & 1u) && r2 <= rc2;
      const double ri = in ? rsqrt_h3(r2) : 0.0;
      const double qq = in ? xi[3] * jzq.y : 0.0;
      const double r2i = ri * ri;
      te = fma(qq, ri + fma(zb, r2, -zc), te);
      double fs = qq * fma(ri, r2i, -zf);
      if (LJ) {
        const double2 lj = s_lj[(e ? rowb : rowa) + tj];   // -6 C6, 12 C12
        const double r6 = r2i * r2i * r2i, p = lj.y * r6;
        tl = fma(fma(p, 0.5, lj.x), r6, tl);
        fs = fma(p + lj.x, r6 * r2i, fs);
      }
      double* fi = e ? fb : fa;
      fi[0] = fma(dx, fs, fi[0]);
      fi[1] = fma(dy, fs, fi[1]);
      fi[2] = fma(dz, fs, fi[2]);
      gx = fma(dx, fs, gx);
      gy = fma(dy, fs, gy);
      gz = fma(dz, fs, gz);
      if (COUNT) tn += in ? 1 : 0;
    }
    if (k < 7) {
      gx = __shfl_sync(full, gx, src);
      gy = __shfl_sync(full, gy, src);
      gz = __shfl_sync(full, gz, src);
      if (LJ) tj = __shfl_sync(full, tj, src);
    }
  }
  const int aj = S.at[sat + 8 * g].x;
  if (aj >= 0 && (gx != 0.0 || gy != 0.0 || gz != 0.0)) {
    atomicAdd(&P.grd[3 * aj + 0], -gx);
    atomicAdd(&P.grd[3 * aj + 1], -gy);
    atomicAdd(&P.grd[3 * aj + 2], -gz);
  }
}

// (ljg as in record_packed)
template <bool MINIMG, bool COUNT>
__device__ __forceinline__ void record_fp64(const DevPtrs& P, const QuadStageD& S, const double2* __restrict__ s_lj,
                                            int rowa, int rowb, const double (&xa)[4], const double (&xb)[4],
                                            unsigned ma, unsigned mb, unsigned ljg, const double (&box)[3],
                                            const double (&inv)[3], double rc2, double zb, double zf, double zc, int sp,
                                            int st, int sat, int src, double (&fa)[3], double (&fb)[3], double& te,
                                            double& tl, int& tn) {
  int g = 0;
#pragma unroll 1
  do {
#pragma unroll 1
    for (; (ljg >> g) & 1u; ++g)
      group_fp64<MINIMG, COUNT, true>(P, S, s_lj, rowa, rowb, xa, xb, ma, mb, g, box, inv, rc2, zb, zf, zc, sp, st, sat,
                                      src, fa, fb, te, tl, tn);
#pragma unroll 1
    for (; g < 4 && !((ljg >> g) & 1u); ++g)
      group_fp64<MINIMG, COUNT, false>(P, S, s_lj, rowa, rowb, xa, xb, ma, mb, g, box, inv, rc2, zb, zf, zc, sp, st, sat,
                                       src, fa, fb, te, tl, tn);
  } while (g < 4);
}

template <bool COUNT>
__global__ void __launch_bounds__(kFp64Threads, 2) k_pair_fp64q(DevPtrs P, ZdConst z) {
  extern __shared__ __align__(16) unsigned char s_dynd[];
  const unsigned full = 0xffffffffu;
  QuadStageD& S = reinterpret_cast<QuadStageD*>(s_dynd)[threadIdx.x >> 5];
  double2* s_lj = reinterpret_cast<double2*>(s_dynd + sizeof(QuadStageD) * kFp64Warps);
  for (int i = threadIdx.x; i < z.nt1 * z.nt1; i += blockDim.x) {
    const double2 c = P.lj_d[i];
    s_lj[i] = make_double2(-6.0 * c.x, 12.0 * c.y);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, qd = lane >> 3, lp = lane & 7;
  const int sp = 64 * qd + lp, sta = 36 * qd + lp, sat = 36 * qd + ((lp + 7) & 7);
  const int src = (lane & 24) | ((lp + 1) & 7);
  const int T = P.nctiles[0];
  const bool ext = *P.ext_pos != 0;
  const int TU = (T + 3) >> 2;
  const int gw = blockIdx.x * kFp64Warps + (threadIdx.x >> 5), nw = gridDim.x * kFp64Warps;
  int cur_unit = -2, cur_rep = -1, rep = -1, aia = -1, aib = -1, tia = z.nt1 - 1, tib = tia;
  double xa[4] = {0, 0, 0, 0}, xb[4] = {0, 0, 0, 0}, fa[3] = {0, 0, 0}, fb[3] = {0, 0, 0};
  double box[3] = {0, 0, 0}, inv[3] = {0, 0, 0}, ref[3] = {0, 0, 0};
  long long eel = 0, elj = 0, npair = 0;
  bool mi = false;
  auto flush_i = [&]() {
    if (aia >= 0)
      for (int k = 0; k < 3; ++k) atomicAdd(&P.grd[3 * aia + k], fa[k]);
    if (aib >= 0)
      for (int k = 0; k < 3; ++k) atomicAdd(&P.grd[3 * aib + k], fb[k]);
    for (int k = 0; k < 3; ++k) fa[k] = fb[k] = 0.0;
  };
  auto take = [&](int a, double (&x)[4]) {   // an atom in its image nearest to the i block's reference
    x[0] = x[1] = x[2] = x[3] = 0.0;
    if (a < 0) return;
    const double4 p = P.pos_d[a];
    x[0] = near_image(p.x - ref[0], box[0], inv[0]);
    x[1] = near_image(p.y - ref[1], box[1], inv[1]);
    x[2] = near_image(p.z - ref[2], box[2], inv[2]);
    x[3] = p.w;
  };
  // the first group by the warp's index, the others from the counter
  for (int t = gw; t < TU;) {
    const int rec = 4 * t + qd;
    const bool valid = rec < T;
    const int word = valid ? P.ct_blk[rec] : -1, unit = valid ? word & kRecUnit : -1;
    const unsigned ljg = (~__reduce_and_sync(full, (unsigned)word) >> kRecFree) & 0xfu;
    int aj[4], ty[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const size_t o = (size_t)rec * 32 + 8 * g + lp;
      aj[g] = valid ? __float_as_int(P.ct_j[o].w) : -1;
      ty[g] = valid ? type_word(P.ct_ty[o]) : z.nt1 - 1;
    }
    const unsigned ma = valid ? step_mask(P.ct_mask[(size_t)rec * kHalf + lp], lp) : 0u;
    const unsigned mb = valid ? step_mask(P.ct_mask[(size_t)rec * kHalf + lp + 8], lp + 8) : 0u;
    if (unit != cur_unit) {
      flush_i();
      cur_unit = unit;
      aia = aib = -1;
      tia = tib = z.nt1 - 1;
      if (unit >= 0) {
        const int si = unit * kHalf + lp, bi = unit >> 1;
        aia = P.satom[si];
        aib = P.satom[si + 8];
        tia = P.styp[si];
        tib = P.styp[si + 8];
        rep = P.blk_rep[bi];
        const Rep& R = P.reps[rep];
        const float4 h = P.blk_half[bi];
        const double hh[3] = {(double)h.x, (double)h.y, (double)h.z}, rc = sqrt(z.rc2);
        mi = ext;
        for (int k = 0; k < 3; ++k) {
          box[k] = R.box[k];
          inv[k] = R.invbox[k];
          ref[k] = P.blk_ref[3 * bi + k];
          if (!(0.5 * box[k] > rc + hh[k] + 2.0)) mi = true;
        }
      }
      take(aia, xa);
      take(aib, xb);
    }
    if (__any_sync(full, rep != cur_rep)) {
      flush_fix<8>(P, cur_rep, eel, elj, 0, 0, npair, COUNT, false);
      eel = elj = npair = 0;
      cur_rep = rep;
    }
    __syncwarp();   // the last group's steps are done with the stage
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      double x[4];
      take(aj[g], x);
      const double2 xy = make_double2(x[0], x[1]), zq = make_double2(x[2], x[3]);
      S.pxy[sp + 16 * g] = xy;
      S.pxy[sp + 16 * g + 8] = xy;
      S.pzq[sp + 16 * g] = zq;
      S.pzq[sp + 16 * g + 8] = zq;
      S.at[sta + 8 * g] = make_int2(aj[g], ty[g]);
    }
    __syncwarp();
    double te = 0.0, tl = 0.0;
    int tn = 0;
    if (__any_sync(full, mi))
      record_fp64<true, COUNT>(P, S, s_lj, tia * z.nt1, tib * z.nt1, xa, xb, ma, mb, ljg, box, inv, z.rc2, z.bcoeff,
                               z.fcoeff, z.zcore, sp, sta, sat, src, fa, fb, te, tl, tn);
    else
      record_fp64<false, COUNT>(P, S, s_lj, tia * z.nt1, tib * z.nt1, xa, xb, ma, mb, ljg, box, inv, z.rc2, z.bcoeff,
                                z.fcoeff, z.zcore, sp, sta, sat, src, fa, fb, te, tl, tn);
    if (COUNT) npair += tn;
    eel += to_fix(te, kEneScale, P.status);
    elj += to_fix(tl * (1.0 / 6.0), kEneScale, P.status);
    t = TU;
    if (nw < TU) {
      if (lane == 0) t = atomicAdd(P.tile_ctr, 1) + nw;
      t = __shfl_sync(full, t, 0);
    }
  }
  flush_i();
  flush_block<8, kFp64Warps>(P, cur_rep, eel, elj, 0, 0, npair, COUNT, false);
}

// Per-warp shared memory of k_pair_fp64 (classes, CMM): each half-warp's record, entries a and b
// of every lane, twice (see MixStage).
struct __align__(16) F64Stage {
  double4 pa[64], pb[64];
  int2 t[64];
};

template <bool COUNT, bool ALSD, bool CMM, bool SPLIT = false>
__global__ void __launch_bounds__(kFp64Threads)
k_pair_fp64(DevPtrs P, ZdConst z) {
  extern __shared__ double2 s_ljd[];
  __shared__ F64Stage s_stage[kFp64Warps];
  const unsigned full = 0xffffffffu;
  const int nlj = z.nt1 * z.nt1;
  for (int i = threadIdx.x; i < nlj; i += blockDim.x) s_ljd[i] = P.lj_d[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int hw = lane >> 4, lp = lane & (kHalf - 1);
  const int sidx = 32 * hw + lp;
  const int src = ((lp + 1) & (kHalf - 1)) | (hw << 4);
  F64Stage& S = s_stage[threadIdx.x >> 5];
  const int T = *P.nctiles;
  const int TU = (T + 1) >> 1;
  const double irlim2 = 1.0 / z.rc2;
  int cur_unit = -2, cur_rep = -1, rep = -1, ai = -1, ti = 0;
  double4 pi = make_double4(0, 0, 0, 0);
  double gix = 0, giy = 0, giz = 0;
  double gix1 = 0, giy1 = 0, giz1 = 0;            // partial McMD: class-1 i forces
  long long eel = 0, elj = 0, eaa = 0, eab = 0;   // fixed point, per record
  long long npair = 0;
  double bx = 0, by = 0, bz = 0, ibx = 0, iby = 0, ibz = 0;
  double f0 = 1.0, f1 = 1.0, f2 = 1.0;
  unsigned tab = 0u;
  auto flush_i = [&]() {
    if (ai >= 0) {
      atomicAdd(&P.grd[3 * ai + 0], gix);
      atomicAdd(&P.grd[3 * ai + 1], giy);
      atomicAdd(&P.grd[3 * ai + 2], giz);
      if (SPLIT) {
        atomicAdd(&P.grd1[3 * ai + 0], gix1);
        atomicAdd(&P.grd1[3 * ai + 1], giy1);
        atomicAdd(&P.grd1[3 * ai + 2], giz1);
      }
    }
    gix = giy = giz = 0;
    gix1 = giy1 = giz1 = 0;
  };
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(P.tile_ctr, 1);
    t = __shfl_sync(full, t, 0);
    if (t >= TU) break;
    const int rec = 2 * t + hw;
    const bool valid = rec < T;
    const int unit = valid ? P.ct_blk[rec] & kRecUnit : -1;
    if (unit != cur_unit) {
      flush_i();
      cur_unit = unit;
      if (unit >= 0) {
        const int si = (unit >> 1) * kTile + (unit & 1) * kHalf + lp;
        ti = P.styp[si];
        ai = P.satom[si];
        pi = ai >= 0 ? P.pos_d[ai] : make_double4(0, 0, 0, 0);
        rep = P.blk_rep[unit >> 1];
      } else {
        pi = make_double4(0, 0, 0, 0);
        ti = z.nt1 - 1;
        ai = -1;
      }
    }
    if (__any_sync(full, rep != cur_rep)) {
      flush_fix<16>(P, cur_rep, eel, elj, eaa, eab, npair, COUNT, ALSD || SPLIT);
      eel = elj = eaa = eab = 0;
      npair = 0;
      if (rep != cur_rep) {
        cur_rep = rep;
        const Rep& R = P.reps[rep];
        bx = R.box[0]; by = R.box[1]; bz = R.box[2];
        ibx = R.invbox[0]; iby = R.invbox[1]; ibz = R.invbox[2];
        if (ALSD) {
          f0 = cls_weight(R, P.lam[2 * rep], 2);
          f1 = cls_weight(R, P.lam[2 * rep], 1);
          f2 = cls_weight(R, P.lam[2 * rep], 0);
        }
        if (SPLIT) tab = R.split ? R.cls_tab : 0u;
      }
    }
    const unsigned m = valid ? P.ct_mask[(size_t)rec * kHalf + lp] : 0u;
    const unsigned me = CMM && valid ? P.ct_mask_el[(size_t)rec * kHalf + lp] : 0u;
    int aj[2], tjv[2];
    double4 pj[2];
    for (int e = 0; e < 2; ++e) {
      const size_t o = (size_t)rec * 32 + kHalf * e + lp;
      aj[e] = valid ? __float_as_int(P.ct_j[o].w) : -1;
      tjv[e] = valid ? type_word(P.ct_ty[o]) : z.nt1 - 1;
      pj[e] = aj[e] >= 0 ? P.pos_d[aj[e]] : make_double4(0.0, 0.0, 0.0, 0.0);
    }
    __syncwarp();
    S.pa[sidx] = pj[0];
    S.pa[sidx + kHalf] = pj[0];
    S.pb[sidx] = pj[1];
    S.pb[sidx + kHalf] = pj[1];
    S.t[sidx] = make_int2(tjv[0], tjv[1]);
    S.t[sidx + kHalf] = make_int2(tjv[0], tjv[1]);
    __syncwarp();
    const int row = ((ALSD || SPLIT) ? (ti & kTypeMask) : ti) * z.nt1;
    const int ci = ALSD ? ((ti >> 30) & 1) : 0;
    const unsigned trow = SPLIT ? tab >> (3 * ((ti >> kRegionShift) & 3)) : 0u;
    constexpr int NG = SPLIT ? 12 : 6;
    double gj[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};   // entries a, b; class 1 a, b
    int tn = 0;
    double te = 0.0, tl = 0.0, ta = 0.0, tb = 0.0;   // this record's energies
#pragma unroll 2
    for (int k = 0; k < kHalf; ++k) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int sh = k + kHalf * e;
        if ((m >> sh) & 1u) {
          const double4 q = e ? S.pb[sidx + k] : S.pa[sidx + k];
          const int tj = e ? S.t[sidx + k].y : S.t[sidx + k].x;
          double dx = pi.x - q.x, dy = pi.y - q.y, dz = pi.z - q.z;
          dx -= bx * anint(dx * ibx);
          dy -= by * anint(dy * iby);
          dz -= bz * anint(dz * ibz);
          const double dd2 = dx * dx + dy * dy + dz * dz;
          const double dd2i = 1.0 / dd2;
          if (dd2i - irlim2 >= 0.0) {
            const double ddi = sqrt(dd2i);
            const double dd6i = dd2i * dd2i * dd2i;
            const bool elp = CMM ? ((me >> sh) & 1u) != 0u : true;
            const double ee = elp ? pi.w * q.w : 0.0;
            const double epair = ee * (ddi + z.bcoeff * dd2 - z.zcore);
            te += epair;
            const double2 lj = s_ljd[row + ((ALSD || SPLIT) ? (tj & kTypeMask) : tj)];
            const double v1 = lj.x * dd6i;
            const double v2 = lj.y * dd6i * dd6i;
            tl += -v1 + v2;
            double cc = ee * (dd2i * ddi - z.fcoeff) + (-6.0 * v1 + 12.0 * v2) * dd2i;
            bool c1 = false;
            if (SPLIT) {   // partial McMD: class 1 by the regions of the two atoms
              c1 = ((trow >> ((tj >> kRegionShift) & 3)) & 1u) != 0u;
              if (c1) ta += epair + (-v1 + v2);
            } else if (ALSD) {
              const int na = ci + ((tj >> 30) & 1);
              if (na == 2) { ta += epair + (-v1 + v2); cc *= f2; }
              else if (na == 1) { tb += epair + (-v1 + v2); cc *= f1; }
              else cc *= f0;
            }
            const double fx = dx * cc, fy = dy * cc, fz = dz * cc;
            if (SPLIT && c1) {
              gix1 -= fx; giy1 -= fy; giz1 -= fz;
              gj[6 + 3 * e] += fx; gj[7 + 3 * e] += fy; gj[8 + 3 * e] += fz;
            } else {
              gix -= fx; giy -= fy; giz -= fz;
              gj[3 * e] += fx; gj[1 + 3 * e] += fy; gj[2 + 3 * e] += fz;
            }
            if (COUNT && elp) ++tn;
          }
        }
      }
#pragma unroll
      for (int q = 0; q < NG; ++q) gj[q] = __shfl_sync(full, gj[q], src);
    }
    for (int e = 0; e < 2; ++e) {
      if (aj[e] >= 0 && (gj[3 * e] != 0.0 || gj[1 + 3 * e] != 0.0 || gj[2 + 3 * e] != 0.0)) {
        atomicAdd(&P.grd[3 * aj[e] + 0], gj[3 * e]);
        atomicAdd(&P.grd[3 * aj[e] + 1], gj[1 + 3 * e]);
        atomicAdd(&P.grd[3 * aj[e] + 2], gj[2 + 3 * e]);
      }
      if (SPLIT && aj[e] >= 0 && (gj[6 + 3 * e] != 0.0 || gj[7 + 3 * e] != 0.0 || gj[8 + 3 * e] != 0.0)) {
        atomicAdd(&P.grd1[3 * aj[e] + 0], gj[6 + 3 * e]);
        atomicAdd(&P.grd1[3 * aj[e] + 1], gj[7 + 3 * e]);
        atomicAdd(&P.grd1[3 * aj[e] + 2], gj[8 + 3 * e]);
      }
    }
    if (COUNT) npair += tn;
    eel += to_fix(te, kEneScale, P.status);
    elj += to_fix(tl, kEneScale, P.status);
    if (ALSD || SPLIT) { eaa += to_fix(ta, kEneScale, P.status); eab += to_fix(tb, kEneScale, P.status); }
  }
  flush_i();
  flush_fix<16>(P, cur_rep, eel, elj, eaa, eab, npair, COUNT, ALSD || SPLIT);
}

// The packed kernels' stages and tables take more than the default 48 KiB of dynamic shared memory.
// The limit belongs to the function on its device, not to a context, so every context raises it
// to the same value, all that the device allows: with the context's own size there, one of
// fewer types created later lowered it below what an earlier context launches with.
// Resident blocks of the kernel an SM, 0 if `bytes` do not fit.
template <class Kernel>
static int raise_smem_limit(Kernel kernel, int threads, int bytes) {
  int dev = 0, optin = 0, per = 0;
  cudaFuncAttributes fa{};
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaFuncGetAttributes(&fa, kernel) != cudaSuccess)
    return 0;
  const int limit = optin - (int)fa.sharedSizeBytes;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) != cudaSuccess) return 0;
  if (bytes > limit ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, bytes) != cudaSuccess)
    return 0;
  return per;
}

template <bool TRI>
static int packed_blocks_per_sm(int bytes) {
  const int per = raise_smem_limit(k_pair_packed<false, false, TRI>, kPairThreads, bytes);
  raise_smem_limit(k_pair_packed<true, false, TRI>, kPairThreads, bytes);
  raise_smem_limit(k_pair_packed<false, true, TRI>, kPairThreads, bytes);
  raise_smem_limit(k_pair_packed<true, true, TRI>, kPairThreads, bytes);
  return per;
}

// the LJ table of the packed kernel as it lies in shared memory: per type pair (-6 C6, 12 C12),
// or per type triple (i, i', j) those of (i, j) and (i', j) side by side
void pack_lj_table(const float2* lj, int nt1, std::vector<float>& out) {
  out.assign(lj_bytes(nt1) / sizeof(float), 0.f);
  size_t o = 0;
  if (!lj_tri(nt1)) {
    for (int i = 0; i < nt1 * nt1; ++i) {
      out[o++] = -6.f * lj[i].x;
      out[o++] = 12.f * lj[i].y;
    }
    return;
  }
  for (int a = 0; a < nt1; ++a)
    for (int b = 0; b < nt1; ++b)
      for (int j = 0; j < nt1; ++j) {
        const float2 pa = lj[a * nt1 + j], pb = lj[b * nt1 + j];
        out[o++] = -6.f * pa.x;
        out[o++] = -6.f * pb.x;
        out[o++] = 12.f * pa.y;
        out[o++] = 12.f * pb.y;
      }
}

static size_t fp64q_bytes(int nt1) { return sizeof(QuadStageD) * kFp64Warps + sizeof(double2) * nt1 * nt1; }

int pair_blocks_per_sm(bool fp64, bool packed, int nt1) {
  int per = 0;
  if (fp64 && packed) {
    const int bytes = (int)fp64q_bytes(nt1);
    per = raise_smem_limit(k_pair_fp64q<false>, kFp64Threads, bytes);
    raise_smem_limit(k_pair_fp64q<true>, kFp64Threads, bytes);
  } else if (fp64) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pair_fp64<false, true, false>, kFp64Threads,
                                                  sizeof(double2) * nt1 * nt1);
  } else if (packed) {
    const int bytes = (int)(kPackedStageBytes + lj_bytes(nt1));
    per = lj_tri(nt1) ? packed_blocks_per_sm<true>(bytes) : packed_blocks_per_sm<false>(bytes);
  } else {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pair_mixed<false, true, false>, kPairThreads,
                                                  sizeof(float2) * nt1 * nt1);
  }
  // (tables that fit no block: the first evaluation's launch is refused and says so)
  if (per <= 0) cudaGetLastError();
  return per > 0 ? per : 1;
}

template <bool COUNT>
static void launch_mixed(const DevPtrs& P, const ZdConst& z, int nb, bool alsd, bool every_cls, bool split,
                         cudaStream_t st) {
  const size_t sh = sizeof(float2) * z.nt1 * z.nt1, shp = kPackedStageBytes + lj_bytes(z.nt1);
  const bool tri = lj_tri(z.nt1);
  if (split) k_pair_mixed<COUNT, false, true><<<nb, kPairThreads, sh, st>>>(P, z);
  else if (z.cmm) k_pair_mixed<COUNT, true, false><<<nb, kPairThreads, sh, st>>>(P, z);
  else {
    // the records with cluster atoms, and under every_cls the others too, by class
    auto plain = tri ? k_pair_packed<COUNT, false, true> : k_pair_packed<COUNT, false, false>;
    auto cls = tri ? k_pair_packed<COUNT, true, true> : k_pair_packed<COUNT, true, false>;
    if (alsd) cls<<<nb, kPairThreads, shp, st>>>(P, z, 2, 0);
    (every_cls ? cls : plain)<<<nb, kPairThreads, shp, st>>>(P, z, alsd ? 1 : 3, alsd ? 1 : 0);
  }
}

void launch_pair_mixed(const DevPtrs& P, const ZdConst& z, int nb, bool count, bool alsd, bool every_cls,
                       bool split, cudaStream_t st) {
  if (count) launch_mixed<true>(P, z, nb, alsd, every_cls, split, st);
  else launch_mixed<false>(P, z, nb, alsd, every_cls, split, st);
}

void launch_pair_fp64(const DevPtrs& P, const ZdConst& z, int nb, bool count, bool alsd, bool split,
                      cudaStream_t st) {
  const size_t sh = sizeof(double2) * z.nt1 * z.nt1;
  if (split) {
    if (count) k_pair_fp64<true, true, false, true><<<nb, kFp64Threads, sh, st>>>(P, z);
    else k_pair_fp64<false, true, false, true><<<nb, kFp64Threads, sh, st>>>(P, z);
  } else if (z.cmm) {
    if (count) k_pair_fp64<true, false, true><<<nb, kFp64Threads, sh, st>>>(P, z);
    else k_pair_fp64<false, false, true><<<nb, kFp64Threads, sh, st>>>(P, z);
  } else if (alsd) {
    if (count) k_pair_fp64<true, true, false><<<nb, kFp64Threads, sh, st>>>(P, z);
    else k_pair_fp64<false, true, false><<<nb, kFp64Threads, sh, st>>>(P, z);
  } else {
    if (count) k_pair_fp64q<true><<<nb, kFp64Threads, fp64q_bytes(z.nt1), st>>>(P, z);
    else k_pair_fp64q<false><<<nb, kFp64Threads, fp64q_bytes(z.nt1), st>>>(P, z);
  }
}

// kernel positions from the master coordinates (after an external coordinate change).  The
// records' image flags don't hold until the next build: kExtPos, and kExtImg if per-pair images
// can then be needed in the box of some replica.  Per axis a tile's image puts the two block
// references at most box/2 apart, and a pair's separation differs from theirs by at most h_i + h_j
// <= 2 h_max plus 2 A of motion, so in the tile's image |d| <= box/2 + 2 h_max + 2; in any other
// image |d| >= box - rc; both hold at once only if box/2 <= rc + 2 h_max + 2.  One answer for the
// whole context: with one per replica both image forms of the packed kernel stood in the
// instruction cache at once, and 64 replicas with boxes on both sides of that line took 1,920 us
// a launch with 883,000 atoms and 2,647 with 1.06 M, where all in one form take 1,484 and 1,763.
__global__ void k_update_pos(DevPtrs P, int natom, int nrep, int fp64, double qscale, double rc) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a < nrep) {
    const Rep& R = P.reps[a];
    int f = kExtPos;
    for (int k = 0; k < 3; ++k)
      if (0.5 * R.box[k] < rc + 2.0 * (double)P.rep_hmax[3 * a + k] + 2.0) f |= kExtImg;
    atomicOr(P.ext_pos, f);
  }
  if (a >= natom) return;
  const double x[3] = {P.x[3 * a], P.x[3 * a + 1], P.x[3 * a + 2]};
  if (fp64) {
    P.pos_d[a] = make_double4(x[0], x[1], x[2], qscale * P.chg[a]);
    return;
  }
  // an atom put into another periodic image since the list build keeps to its block: its frame
  // origin moves along, so that the FP32 position stays small
  const Rep& R = P.reps[P.rep_of[a]];
  float q[3];
  for (int k = 0; k < 3; ++k) {
    const double d = x[k] - P.off[3 * a + k], n = anint(d * R.invbox[k]);
    q[k] = (float)(d - R.box[k] * n);
    if (n != 0.0) P.off[3 * a + k] += R.box[k] * n;
  }
  P.pos_f[a] = make_float4(q[0], q[1], q[2], (float)(qscale * P.chg[a]));
}

void launch_update_pos(const DevPtrs& P, int natom, int nrep, bool fp64, double qscale, double rc, cudaStream_t st) {
  k_update_pos<<<(std::max(natom, nrep) + 255) / 256, 256, 0, st>>>(P, natom, nrep, fp64 ? 1 : 0, qscale, rc);
}

}  // namespace jp
