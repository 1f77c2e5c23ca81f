// fos_ilut.cu -- dual-threshold incomplete LU (ILUT) on the device.
//
// The reference's ILU class (numerics/sparse.f90:52-63,334-392) factors a CSR matrix with
// SPARSKIT's ilut (ITSOL/ilut.f:38-382) and applies it with lusol (:2272-2320).  Here the
// same algorithm runs one warp per row:
//
//   factor  blocks of five consecutive rows are claimed in increasing order from an atomic
//           ticket, a warp a row; the rows of a block hand over to one another in shared
//           memory, the others through global memory.  A row's working
//           copy (L part, U part, and a column -> position hash) lives in shared memory;
//           its L entries are eliminated in increasing column order, each waiting (bounded
//           spin) until the pivot row's own warp has published it.  A warp only waits on
//           rows whose tickets were taken before its own, by warps that are running, so the
//           wait always ends.  Every floating-point operation of a row is the one ilut
//           performs, in the same order, with the FMA contraction ilut does not have
//           written out (__dmul_rn / __dsub_rn): given the same CSR the factors are
//           bit-identical to SPARSKIT's.  Fill-in positions follow ilut's append order
//           (ballot prefix counts), and the quick-split is ilut's, swap for swap, run by the
//           whole warp.
//   solve   the forward and backward sweeps of lusol, groups of five rows or single rows claimed
//           level by level of their graph, each unknown published by its own store and polled by
//           the groups that read it; the row sums are fixed-order warp reductions.
//
// Storage: every row owns lfil slots for L and lfil for U (ilut keeps at most lfil L and
// lfil - 1 off-diagonal U entries per row), so the factor storage never runs out (the
// reference's -2 / -3); rows longer than the shared-memory working capacity are redone
// with a larger capacity.
#include <algorithm>
#include <climits>
#include <cstring>
#include <string>
#include <vector>

#include "fos_internal.h"
#include "fos_device.cuh"

struct fos_ilut {
  int n = 0, lfil = 0, device = 0;
  int* d_Lcol = nullptr;
  double* d_Lval = nullptr;
  int* d_Lcnt = nullptr;
  int* d_Ucol = nullptr;
  double* d_Uval = nullptr;
  int* d_Ucnt = nullptr;
  double* d_dinv = nullptr;
  int* d_done = nullptr;   // factor: epoch of the factorisation that published the row
  double* d_z = nullptr;   // forward-sweep result (kPending before each solve)
  int* d_levL = nullptr;   // level of every row in the L graph, published by the factor
  int* d_permF = nullptr;  // row groups or rows by forward / backward level: the solves' claim order
  int* d_permB = nullptr;
  int nlevF = 0, nlevB = 0;  // levels of the L and U graphs of rows
  int perF = 0, perB = 0;    // rows that a warp of the forward / backward sweep takes at a time
  int swF = 0, swB = 0;      // and levels of the graph of these
  int* d_ctr = nullptr;    // [0] factor ticket [1] forward [2] backward [3] error [4] error row
                           // [5] malformed row [6] most levels [7] groups done [8] most levels in
                           // the stored columns
  int* h_ctr = nullptr;    // pinned copy
  int fepoch = 0;
  int cap = 256;           // working-row capacity (entries of L and of U)
  long spin_limit = 0;     // polls of one dependency wait before giving up (0: kSpinLimit)
  int withhold = -1;       // failure injection: a row that is never published (-1: none)
  bool factored = false;
  long launches = 0;
  ~fos_ilut();
};

fos_ilut::~fos_ilut() {
  void* p[] = {d_Lcol, d_Lval, d_Lcnt, d_Ucol, d_Uval, d_Ucnt, d_dinv, d_done, d_z,
               d_levL, d_permF, d_permB, d_ctr};
  for (void* q : p)
    if (q) cudaFree(q);
  if (h_ctr) cudaFreeHost(h_ctr);
}

namespace {

constexpr int kWarps = 4;                 // the capacity limit is that of four rows in a CTA
#ifndef FOS_ILUT_WARPS
#define FOS_ILUT_WARPS 5
#endif
constexpr int kMaxWarps = FOS_ILUT_WARPS;  // rows of a CTA where they fit
constexpr long kSpinLimit = 1L << 23;     // polls of a dependency flag before giving up
__device__ __forceinline__ unsigned long long timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned long long ld_level(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
constexpr int kCtr = 9;                   // words of d_ctr
constexpr int kErrCapacity = -1, kErrZeroRow = -5, kErrTimeout = -6, kErrSlow = -7;

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The rows a warp knows to be published: bit l of mask is row base + l.
struct Known {
  int base;
  unsigned mask;
  __device__ __forceinline__ bool has(int j) const {
    const unsigned d = (unsigned)(j - base);
    return d < 32u && (mask >> d & 1u);
  }
};
// The warp spins until row j < top is published (flag >= epoch), looking at the 32 rows from j on:
// the pivots that follow are mostly among them and need no look of their own.  False when the
// limit ran out or another warp already gave up (the error word is set), so no wait outlives a
// failure.  The lanes' acquires, ordered before the others' reads by the syncwarp, come after
// the publishing warps' releases.
__device__ __forceinline__ bool wait_row(const int* flag, int j, int top, int epoch, int* ctr,
                                         long spin, int lane, Known& known) {
  for (long it = 0; it < spin; it++) {
    const bool mine = j + lane < top && ld_acquire(flag + j + lane) >= epoch;
    const unsigned m = __ballot_sync(~0u, mine);
    if (m & 1u) {
      known.base = j;
      known.mask = m;
      __syncwarp();
      return true;
    }
    if ((it & 15) == 15) {
      if (__any_sync(~0u, *(volatile int*)(ctr + 3) == kErrTimeout)) return false;
      __nanosleep(32);
    }
  }
  atomicCAS(ctr + 3, 0, kErrTimeout);
  return false;
}
// The wait for a row that a warp of this CTA publishes in shared memory
__device__ __forceinline__ bool wait_local(const int* flag, int* ctr, long spin) {
  for (long it = 0; it < spin; it++) {
    const int f = *(const volatile int*)flag;
    if (__all_sync(~0u, f != 0)) {
      __threadfence_block();
      return true;
    }
    if ((it & 1023) == 1023 && __any_sync(~0u, *(volatile int*)(ctr + 3) == kErrTimeout)) return false;
  }
  atomicCAS(ctr + 3, 0, kErrTimeout);
  return false;
}

// |v| > t by integer comparison (an FP64 one takes the FP64 pipe, and these stand on the chain of
// rows): bits of numbers without a sign order as the numbers do, and a NaN's are above infinity's.
// t as the bits to compare with: those of a negative t, which every |v| exceeds, are a negative
// integer; -0.0 counts as 0, and nothing exceeds a NaN.
__device__ __forceinline__ long long threshold_bits(double t) {
  const long long c = __double_as_longlong(t), mag = c & 0x7fffffffffffffffll;
  return mag > 0x7ff0000000000000ll ? LLONG_MAX : mag == 0 ? 0 : c;
}
__device__ __forceinline__ long long abs_bits(double v) {
  return __double_as_longlong(v) & 0x7fffffffffffffffll;
}
__device__ __forceinline__ bool abs_above(double v, long long t) {
  const long long b = abs_bits(v);
  return b <= 0x7ff0000000000000ll && b > t;
}
// |v| <= t; false for NaN
__device__ __forceinline__ bool abs_within(double v, double t) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
  const unsigned long long c = (unsigned long long)__double_as_longlong(t);
  return c <= 0x7ff0000000000000ull ? b <= c : fabs(v) <= t;
}
__device__ __forceinline__ void set_error(int* ctr, int code, int row) {
  if (atomicCAS(ctr + 3, 0, code) == 0) ctr[4] = row;
}

// column -> position hash of a working row; L positions are stored as ~pos
__device__ __forceinline__ unsigned hslot(int key, unsigned mask) {
  return ((unsigned)key * 2654435761u) & mask;
}
__device__ __forceinline__ bool hfind(const int* hkey, const int* hpos, unsigned mask, int key,
                                      int& pos, unsigned& slot) {
  unsigned s = hslot(key, mask);
  for (;;) {
    const int k = hkey[s];
    if (k == key) { pos = hpos[s]; slot = s; return true; }
    if (k < 0) return false;
    s = (s + 1) & mask;
  }
}
__device__ __forceinline__ void hinsert(int* hkey, int* hpos, unsigned mask, int key, int pos) {
  unsigned s = hslot(key, mask);
  for (;;) {
    const int prev = atomicCAS(hkey + s, -1, key);
    if (prev < 0 || prev == key) { hpos[s] = pos; return; }
    s = (s + 1) & mask;
  }
}

__device__ __forceinline__ unsigned lanes_below(int lane) { return (1u << lane) - 1u; }

// SPARSKIT qsplit (ilut.f:2376-2434): the ncut largest |a| first, by the warp, every element where
// the sequential routine leaves it.  A pass over [first, last] with key |a(first)| walks
// j = first + 1, ... and swaps element j to the end of the larger ones when it is larger.  In
// slots t = j - first: the larger elements end up in order in slots 1, 2, ...; the others form a
// queue behind them whose front goes to slot t whenever x_t is larger.  So with c_t the number of
// larger elements before t, slot t receives x_t, or for a larger x_t what slot c_t + 1 held, and
// the final content of a slot is found by following those links back to a smaller element.  sa,
// si, src: scratch of n.  One lane took 20 us for a row whose U part outgrew lfil, on the chain of
// rows.  Up to 65 elements the links come from the ballots of the comparisons, without scratch.
// passes over at most 65 elements
__device__ __forceinline__ void qsplit_tail(double* a, int* ind, int first, int last, int cut,
                                            int lane) {
  for (;;) {
    const double key = a[first];
    const int m = last - first, t0 = 1 + lane, t1 = 33 + lane;  // the lane's two slots
    const double w0 = t0 <= m ? a[first + t0] : 0.0, w1 = t1 <= m ? a[first + t1] : 0.0;
    const int i0 = t0 <= m ? ind[first + t0] : 0, i1 = t1 <= m ? ind[first + t1] : 0;
    const int ikey = ind[first];
    const long long akey = abs_bits(key);
    const bool g0 = t0 <= m && abs_above(w0, akey), g1 = t1 <= m && abs_above(w1, akey);
    const unsigned long long G = (unsigned long long)__ballot_sync(~0u, g0) |
                                 (unsigned long long)__ballot_sync(~0u, g1) << 32;  // bit t - 1
    const int larger = __popcll(G);
    auto before = [&](int t) { return __popcll(G & ((1ull << (t - 1)) - 1ull)); };
    auto source = [&](int t) {  // the slot whose element ends up in slot t > larger
      while (G >> (t - 1) & 1ull) t = before(t) + 1;
      return t;
    };
    double r0 = 0.0, r1 = 0.0;
    int k0 = 0, k1 = 0;
    if (t0 > larger && t0 <= m) { const int q = source(t0); r0 = a[first + q]; k0 = ind[first + q]; }
    if (t1 > larger && t1 <= m) { const int q = source(t1); r1 = a[first + q]; k1 = ind[first + q]; }
    __syncwarp();
    // larger elements in order to slots 1 ..., the last of them to the pivot's place, which goes
    // to slot `larger`; then the others
    if (g0) { const int d = before(t0) + 1, e = first + (d == larger ? 0 : d); a[e] = w0; ind[e] = i0; }
    if (g1) { const int d = before(t1) + 1, e = first + (d == larger ? 0 : d); a[e] = w1; ind[e] = i1; }
    if (t0 > larger && t0 <= m) { a[first + t0] = r0; ind[first + t0] = k0; }
    if (t1 > larger && t1 <= m) { a[first + t1] = r1; ind[first + t1] = k1; }
    if (lane == 0) { a[first + larger] = key; ind[first + larger] = ikey; }
    __syncwarp();
    const int mid = first + larger;
    if (mid == cut) return;
    if (mid > cut) last = mid - 1; else first = mid + 1;
  }
}
__device__ __forceinline__ void qsplit(double* a, int* ind, int n, int ncut, double* sa, int* si,
                                       int* src, int lane) {
  int first = 0, last = n - 1;
  const int cut = ncut - 1;
  if (cut < first || cut > last) return;
  if (last - first <= 64) {
    qsplit_tail(a, ind, first, last, cut, lane);
    return;
  }
  for (;;) {
    const long long key = abs_bits(a[first]);
    const int m = last - first;
    int larger = 0;
    for (int t0 = 1; t0 <= m; t0 += 32) {
      const int t = t0 + lane;
      double v = 0.0;
      bool g = false;
      if (t <= m) {
        v = a[first + t];
        g = abs_above(v, key);
        sa[t] = v;
        si[t] = ind[first + t];
      }
      const unsigned bg = __ballot_sync(~0u, g);
      if (t <= m) src[t] = g ? larger + __popc(bg & lanes_below(lane)) + 1 : t;
      larger += __popc(bg);
    }
    __syncwarp();
    for (int t = 1 + lane; t <= m; t += 32) {
      if (abs_above(sa[t], key)) {
        a[first + src[t]] = sa[t];
        ind[first + src[t]] = si[t];
      }
      if (t > larger) {
        int q = t;
        while (src[q] != q) q = src[q];
        a[first + t] = sa[q];
        ind[first + t] = si[q];
      }
    }
    __syncwarp();
    const int mid = first + larger;
    if (lane == 0) {
      const double v = a[mid]; a[mid] = a[first]; a[first] = v;
      const int i = ind[mid]; ind[mid] = ind[first]; ind[first] = i;
    }
    __syncwarp();
    if (mid == cut) return;
    if (mid > cut) last = mid - 1; else first = mid + 1;
    if (last - first <= 64) {
      qsplit_tail(a, ind, first, last, cut, lane);
      return;
    }
  }
}

// One row per warp, the rows of a CTA consecutive; shared memory per warp: lval, uval [cap]
// doubles, lcol, ucol [cap] ints, hash keys and positions [4 cap] ints (56 cap bytes).  At most
// 2 cap keys go into the hash, so at least half of its slots stay empty and every probe
// sequence ends.
// What bounds it is the chain of rows (nearly every row of the Euler P reads the row just
// above): from a row's last update to the next row's.  Rows of one CTA hand over in shared memory
// (pivot, U part and flag); only the first of them waits for another CTA's release through the L2.
// A finished row's first 64 U entries, pivot and count are read at once.  P of 20,160 tetrahedra
// (100,800 rows), factored and applied: 182 ms before the hand-over and the warp's quick-split, 50.5
// now (with the sweeps' orders and both sweeps, 4.0 ms).
struct IlutShared {
  int group;
  int flag[kMaxWarps], cnt[kMaxWarps], lev[kMaxWarps];  // a finished row: set last, U entries, level
  double dinv[kMaxWarps];
};

__global__ void __launch_bounds__(32 * kMaxWarps, 1) k_ilut_factor(
    int n, const int* __restrict__ ia, const int* __restrict__ ja, const double* __restrict__ a,
    int lfil, double droptol, int cap, int epoch, int* __restrict__ Lcol,
    double* __restrict__ Lval, int* __restrict__ Lcnt, int* __restrict__ Ucol,
    double* __restrict__ Uval, int* __restrict__ Ucnt, double* __restrict__ dinv,
    int* __restrict__ levL, int* __restrict__ done, int* __restrict__ ctr, long spin,
    int withhold) {
  pdl_entry();
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned hmask = 4u * cap - 1u;
  __shared__ IlutShared sh;
  const int nw = blockDim.x >> 5;
  unsigned char* base = smem + (size_t)wid * 56 * cap;
  double* lval = reinterpret_cast<double*>(base);
  double* uval = lval + cap;
  int* lcol = reinterpret_cast<int*>(uval + cap);
  int* ucol = lcol + cap;
  int* hkey = ucol + cap;
  int* hpos = hkey + 4 * cap;
  const size_t slot = (size_t)(lfil > 0 ? lfil : 1);
  for (;;) {
    __syncthreads();  // the rows of the last group have been read
    if (threadIdx.x == 0) sh.group = atomicAdd(ctr, 1);
    if (lane == 0) sh.flag[wid] = 0;
    __syncthreads();
    const int g0 = sh.group * nw;  // the group's first row
    const int ii = g0 + wid;
    if (g0 >= n) return;
    if (ii >= n) continue;
    for (int k = lane; k < 4 * cap; k += 32) hkey[k] = -1;
    const int j1 = ia[ii], j2 = ia[ii + 1];
    double tnorm = 0.0;
    if (lane == 0)
      for (int k = j1; k < j2; k++) tnorm += fabs(a[k]);
    tnorm = __shfl_sync(~0u, tnorm, 0);
    bool ok = true;
    int lenl = 0, lenu = 1, len = 0;
    if (tnorm == 0.0) {
      if (lane == 0) set_error(ctr, kErrZeroRow, ii);
      ok = false;
    }
    tnorm = tnorm / (double)(j2 - j1);
    const long long thr = threshold_bits(__dmul_rn(droptol, tnorm));
    __syncwarp();
    if (ok) {
      // unpack: L in CSR order, U with the diagonal first, then CSR order
      if (lane == 0) {
        ucol[0] = ii;
        uval[0] = 0.0;
        hinsert(hkey, hpos, hmask, ii, 0);
      }
      __syncwarp();
      for (int c = j1; c < j2; c += 32) {
        const int k = c + lane;
        const bool valid = k < j2;
        const int col = valid ? ja[k] : 0;
        const double v = valid ? a[k] : 0.0;
        const bool isL = valid && col < ii, isU = valid && col > ii;
        const unsigned bl = __ballot_sync(~0u, isL), bu = __ballot_sync(~0u, isU);
        if (isL || isU) {
          const int p = isL ? lenl + __popc(bl & lanes_below(lane)) : lenu + __popc(bu & lanes_below(lane));
          if (p < cap) {
            if (isL) { lcol[p] = col; lval[p] = v; hinsert(hkey, hpos, hmask, col, ~p); }
            else { ucol[p] = col; uval[p] = v; hinsert(hkey, hpos, hmask, col, p); }
          }
        }
        if (valid && col == ii) uval[0] = v;
        lenl += __popc(bl);
        lenu += __popc(bu);
        __syncwarp();
      }
      if (lenl > cap || lenu > cap) ok = false;
    }
    // elimination of the L entries in increasing column order (ilut.f:150-226); lev = the
    // largest L-graph level among the rows of stored multipliers (a superset of the kept
    // ones, so 1 + lev is a valid level for the sweeps' claim order)
    int jj = 0, lev = 0;
    Known known = {0, 0u};
    // the U row of the pivot expected next (jp, -1: none): its first 64 entries, two to a lane,
    // its pivot, count and level
    int jp = -1, pc0 = 0, pc1 = 0, pn = 0, plev = 0;
    double pd = 0.0, pv0 = 0.0, pv1 = 0.0;
    auto fetch = [&](int j) {
      const int* uc = Ucol + (size_t)j * slot;
      const double* uv = Uval + (size_t)j * slot;
      jp = j;
      pd = dinv[j];
      pn = Ucnt[j];
      plev = levL[j];
      if (lane < (int)slot) { pc0 = uc[lane]; pv0 = uv[lane]; }  // (entries past the count unused)
      if (lane + 32 < (int)slot) { pc1 = uc[lane + 32]; pv1 = uv[lane + 32]; }
    };
    while (ok && jj < lenl) {
      // the smallest remaining column, and the next one as far as it is known now
      int m1 = INT_MAX, m2 = INT_MAX, k1 = 0;
      for (int k = jj + lane; k < lenl; k += 32) {
        const int cl = lcol[k];
        if (cl < m1) { m2 = m1; m1 = cl; k1 = k; }
        else if (cl < m2) m2 = cl;
      }
      const int jrow = __reduce_min_sync(~0u, m1);
      const unsigned who = __ballot_sync(~0u, m1 == jrow);
      const int k = __shfl_sync(~0u, k1, __ffs(who) - 1);
      const int jnext = __reduce_min_sync(~0u, m1 == jrow ? m2 : m1);
      if (k != jj) {  // swap entries jj and k, their hash positions looked up by two lanes
        const int cj = lcol[jj];
        const double vj = lval[jj], vk = lval[k];
        __syncwarp();
        if (lane < 2) {
          int pos;
          unsigned sl;
          hfind(hkey, hpos, hmask, lane == 0 ? jrow : cj, pos, sl);
          const int to = lane == 0 ? jj : k;
          hpos[sl] = ~to;
          lcol[to] = lane == 0 ? jrow : cj;
          lval[to] = lane == 0 ? vk : vj;
        }
      }
      __syncwarp();
      const bool local = jrow >= g0;
      const double lj = lval[jj];
      double dj, v0, v1;
      int ulen, lv, c0, c1;
      const int* uc;
      const double* uv;
      if (local) {  // a row of this CTA: in the shared memory of its warp
        const int w = jrow - g0;
        if (!wait_local(sh.flag + w, ctr, spin)) { ok = false; break; }
        dj = *(volatile double*)(sh.dinv + w);
        ulen = *(volatile int*)(sh.cnt + w);
        lv = *(volatile int*)(sh.lev + w);
        unsigned char* ob = smem + (size_t)w * 56 * cap;
        uv = reinterpret_cast<double*>(ob) + cap + 1;
        uc = reinterpret_cast<int*>(ob + 16 * (size_t)cap) + cap + 1;
        c0 = uc[lane];  // (cap >= 256: in the arrays; entries past ulen unused)
        v0 = uv[lane];
        c1 = uc[lane + 32];
        v1 = uv[lane + 32];
      } else {
        uc = Ucol + (size_t)jrow * slot;
        uv = Uval + (size_t)jrow * slot;
        if (jp != jrow) {
          if (!known.has(jrow) && !wait_row(done, jrow, g0, epoch, ctr, spin, lane, known)) {
            ok = false;
            break;
          }
          fetch(jrow);
        }
        dj = pd; ulen = pn; lv = plev;
        c0 = pc0; c1 = pc1; v0 = pv0; v1 = pv1;
        jp = -1;
      }
      // on its way while this pivot is worked off; a fill-in may come before it, then it is unused
      if (jnext < g0 && known.has(jnext)) fetch(jnext);
      const double fact = __dmul_rn(lj, dj);
      if (abs_within(fact, droptol)) { jj++; __syncwarp(); continue; }
      lev = max(lev, lv);
      // row update, 64 entries at a time: a row's columns are distinct, so the second 32 are
      // looked up before the first 32 append their fill-ins; positions go in ilut's order
      for (int c = 0; c < ulen; c += 64) {
        if (c > 0) {
          if (c + lane < ulen) { c0 = uc[c + lane]; v0 = uv[c + lane]; }
          if (c + 32 + lane < ulen) { c1 = uc[c + 32 + lane]; v1 = uv[c + 32 + lane]; }
        }
        const bool in0 = c + lane < ulen, in1 = c + 32 + lane < ulen;
        int p0 = 0, p1 = 0;
        unsigned sl;
        const bool f0 = in0 && hfind(hkey, hpos, hmask, c0, p0, sl);
        const bool f1 = in1 && hfind(hkey, hpos, hmask, c1, p1, sl);
        const double s0 = __dmul_rn(fact, v0), s1 = __dmul_rn(fact, v1);
        __syncwarp();
        auto update = [&](bool found, int pos, double sv) {
          if (found) {
            double* t = pos >= 0 ? uval + pos : lval + ~pos;
            *t = __dsub_rn(*t, sv);
          }
        };
        update(f0, p0, s0);
        update(f1, p1, s1);
        auto append = [&](bool fill, int j, double sv) {
          const unsigned bu = __ballot_sync(~0u, fill && j >= ii);
          const unsigned bl = __ballot_sync(~0u, fill && j < ii);
          if (fill) {
            if (j >= ii) {
              const int q = lenu + __popc(bu & lanes_below(lane));
              if (q < cap) { ucol[q] = j; uval[q] = -sv; hinsert(hkey, hpos, hmask, j, q); }
            } else {
              const int q = lenl + __popc(bl & lanes_below(lane));
              if (q < cap) { lcol[q] = j; lval[q] = -sv; hinsert(hkey, hpos, hmask, j, ~q); }
            }
          }
          lenu += __popc(bu);
          lenl += __popc(bl);
        };
        append(in0 && !f0, c0, s0);
        append(in1 && !f1, c1, s1);
        __syncwarp();
      }
      if (lenl > cap || lenu > cap) { ok = false; break; }
      if (lane == 0) { lval[len] = fact; lcol[len] = jrow; }
      len++;
      jj++;
      __syncwarp();
    }
    if (!ok) {
      if (lane == 0) {
        if (lenl > cap || lenu > cap) set_error(ctr, kErrCapacity, ii);
        Lcnt[ii] = 0;
        Ucnt[ii] = 0;
        dinv[ii] = 0.0;
        levL[ii] = 1;
        sh.cnt[wid] = 0;
        sh.dinv[wid] = 0.0;
        sh.lev[wid] = 1;
        __threadfence();
        if (ii != withhold) {
          *(volatile int*)(sh.flag + wid) = 1;
          st_release(done + ii, epoch);
        }
      }
      __syncwarp();
      continue;
    }
    // U part first (the rows below wait for it): drop |w| <= droptol * tnorm keeping the
    // order, keep the largest (ilut.f:258-287), publish U and the inverted pivot
    double w0 = uval[0];
    if (abs_within(w0, 0.0)) w0 = __dmul_rn(__dadd_rn(0.0001, droptol), tnorm);
    const double di = 1.0 / w0;
    int cnt = 0;
    for (int c = 1; c < lenu; c += 64) {  // (64 at a time: one wait on the reads, one on the writes)
      const int a0 = c + lane, a1 = c + 32 + lane;
      const double x0 = a0 < lenu ? uval[a0] : 0.0, x1 = a1 < lenu ? uval[a1] : 0.0;
      const int q0 = a0 < lenu ? ucol[a0] : 0, q1 = a1 < lenu ? ucol[a1] : 0;
      const bool keep0 = a0 < lenu && abs_above(x0, thr), keep1 = a1 < lenu && abs_above(x1, thr);
      const unsigned b0 = __ballot_sync(~0u, keep0), b1 = __ballot_sync(~0u, keep1);
      const int d0 = 1 + cnt + __popc(b0 & lanes_below(lane));
      const int d1 = 1 + cnt + __popc(b0) + __popc(b1 & lanes_below(lane));
      __syncwarp();
      if (keep0) { uval[d0] = x0; ucol[d0] = q0; }
      if (keep1) { uval[d1] = x1; ucol[d1] = q1; }
      cnt += __popc(b0) + __popc(b1);
      __syncwarp();
    }
    const int lenu2 = cnt + 1;
    const int keepu = min(lenu2, lfil);
    // (the hash is done with: its room holds the scratch of the quick-splits)
    double* sa = reinterpret_cast<double*>(hkey);
    int* si = reinterpret_cast<int*>(sa + cap);
    qsplit(uval + 1, ucol + 1, lenu2 - 1, keepu, sa, si, si + cap, lane);
    __syncwarp();
    const int nu = max(keepu - 1, 0);
    if (lane == 0) {  // for the rows of this CTA (the U part is in place, ordered by the syncwarp)
      sh.dinv[wid] = di;
      sh.cnt[wid] = nu;
      sh.lev[wid] = lev + 1;
      __threadfence_block();
      if (ii != withhold) *(volatile int*)(sh.flag + wid) = 1;
    }
    for (int k = lane; k < nu; k += 32) {
      Ucol[(size_t)ii * slot + k] = ucol[1 + k];
      Uval[(size_t)ii * slot + k] = uval[1 + k];
    }
    if (lane == 0) {
      dinv[ii] = di;
      Ucnt[ii] = nu;
      levL[ii] = lev + 1;
    }
    __threadfence();
    __syncwarp();
    if (lane == 0 && ii != withhold) st_release(done + ii, epoch);
    // L part afterwards, off the rows-below path: the lfil largest multipliers (:236-254);
    // only the sweeps read it, after this kernel
    const int keepl = min(len, lfil);
    qsplit(lval, lcol, len, keepl, sa, si, si + cap, lane);
    __syncwarp();
    for (int k = lane; k < keepl; k += 32) {
      Lcol[(size_t)ii * slot + k] = lcol[k];
      Lval[(size_t)ii * slot + k] = lval[k];
    }
    if (lane == 0) Lcnt[ii] = keepl;
    __syncwarp();
  }
}

// The sweeps publish each solved unknown by its own 64-bit store: the output vectors start
// filled with kPending, a signalling-NaN pattern that no arithmetic produces (results that
// would carry it are stored as the canonical NaN), and a row polls the unknowns it reads
// until they stop being kPending.  One L2 round trip per dependency, no flags, no fences.
constexpr unsigned long long kPending = 0x7ff4deadbeefcafeull;
// warps of a sweep: about kLookahead levels' worth of rows in flight.  More only add warps
// that spin on unknowns many levels ahead and load L2 with their polls.
#ifndef FOS_ILUT_LOOKAHEAD
#define FOS_ILUT_LOOKAHEAD 2
#endif
constexpr int kLookahead = FOS_ILUT_LOOKAHEAD;
#ifndef FOS_ILUT_MIN_WARPS
#define FOS_ILUT_MIN_WARPS 304
#endif

__device__ __forceinline__ double ld_poll(const double* p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_publish(double* p, double v) {
  if (__double_as_longlong(v) == (long long)kPending) v = __longlong_as_double(0x7ff8000000000000ll);
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ bool pending(double v) {
  return __double_as_longlong(v) == (long long)kPending;
}
__global__ void k_fill_pending(long n, double* __restrict__ x) {
  pdl_entry();
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = __longlong_as_double((long long)kPending);
}

// One sweep of lusol, a warp per group of kG consecutive rows (kGroup, or 1: see one_at_a_time):
//   forward (ilut.f:2300-2305):  z_i = y_i - sum_k L_ik z_k into z (kPending on entry), and x_i set
//     to kPending for the backward sweep (x may be y: a group reads its own y_i only)
//   backward (:2309-2315):       x_i = dinv_i (z_i - sum_k U_ik x_k) into x (kPending on entry)
// Groups are claimed in order of their level in the graph of groups (perm): the groups in flight
// are mostly independent, and a group's dependencies have lower levels, hence earlier claims
// (rows of a group are consecutive, so a group only reads groups on one side of it).  The lanes
// go over the entries of all rows of the group at once, all loads in flight together; entries
// inside the group are set aside and solved in registers afterwards.  What bounds a sweep is the
// chain of dependencies, and the unknowns of one cell are a chain of five: a row at a time each
// link took an L2 round trip, its polls and a five-step sum (2.1 us; 0.75 now, with kG = 1); in
// groups the five cost 2.2 (both sweeps of 100,800 rows of the Euler P: 17.5 ms before, 4.0 now).  A wait that ran out makes the row NaN, so
// the failure reaches callers that only look at the result (the Krylov driver's non-finite checks)
// as well as fos_ilut_status.
constexpr int kGroup = 5;

template <bool kBwd, int kG>
__global__ void __launch_bounds__(256) k_ilut_sweep(int n, int lfil, const int* __restrict__ col,
                                                    const double* __restrict__ val,
                                                    const int* __restrict__ cnt,
                                                    const double* __restrict__ dinv,
                                                    const int* __restrict__ perm,
                                                    const double* rhs, double* out, double* clear,
                                                    int* __restrict__ ctr, long spin,
                                                    int withhold) {
  pdl_entry();
  // the entries between rows of the warp's group (kPending, no number that is stored: no entry; a
  // stored zero counts, its product with an unknown that is not finite is a NaN)
  __shared__ double in_group[8][kG][kG];
  const int lane = threadIdx.x & 31;
  double (*cg)[kG] = in_group[threadIdx.x >> 5];
  const size_t slot = (size_t)(lfil > 0 ? lfil : 1);
  const int ng = (n + kG - 1) / kG;
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(ctr + (kBwd ? 2 : 1), 1);
    t = __shfl_sync(~0u, t, 0);
    if (t >= ng) return;
    const int r0 = perm[t] * kG, nr = min(kG, n - r0);
    const double own = lane < nr ? rhs[r0 + lane] : 0.0;  // before the polls: its load overlaps them
    const double di = kBwd && lane < nr ? dinv[r0 + lane] : 1.0;
    if (lane < kG * kG)
      cg[lane / kG][lane % kG] = __longlong_as_double((long long)kPending);
    __syncwarp();
    const int cl = lane < nr ? cnt[r0 + lane] : 0;
    const int longest = __reduce_max_sync(~0u, cl);
    constexpr int kAcc = kG == 1 ? 1 : 8;
    double acc[kAcc];
#pragma unroll
    for (int r = 0; r < kAcc; r++) acc[r] = 0.0;
    bool ok = true;
    for (int k0 = 0; k0 < longest; k0 += 64) {
      int j[2][kG];
      double a[2][kG], v[2][kG];
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int r = 0; r < kG; r++) {
          const int k = k0 + 32 * h + lane;
          const bool in = r < nr && k < __shfl_sync(~0u, cl, r);
          j[h][r] = in ? col[(size_t)(r0 + r) * slot + k] : -1;
          a[h][r] = in ? val[(size_t)(r0 + r) * slot + k] : 0.0;
        }
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int r = 0; r < kG; r++) {
          const int q = j[h][r];
          if (q >= r0 && q < r0 + nr) {
            cg[r][q - r0] = a[h][r];
            a[h][r] = 0.0;
            j[h][r] = -1;
          }
          v[h][r] = j[h][r] >= 0 ? ld_poll(out + j[h][r]) : 0.0;
        }
      // bounded spin over all of them together: every round asks for what is still missing, so
      // a group's unknowns that were published together cost its readers one round trip.  The
      // error word is looked at every 64 rounds only.
      for (long it = 0;; it++) {
        bool wait = false;
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int r = 0; r < kG; r++) wait |= pending(v[h][r]);
        if (!__any_sync(~0u, wait)) break;
        if (it >= spin) {
          atomicCAS(ctr + 3, 0, kErrTimeout);
          ok = false;
          break;
        }
        if ((it & 63) == 63) {
          if (__any_sync(~0u, *(volatile int*)(ctr + 3) == kErrTimeout)) { ok = false; break; }
          __nanosleep(32);
        }
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int r = 0; r < kG; r++)
            if (pending(v[h][r])) v[h][r] = ld_poll(out + j[h][r]);
      }
      if (!ok) break;
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int r = 0; r < kG; r++) acc[r] = fma(a[h][r], v[h][r], acc[r]);
    }
    if (!ok) {
#pragma unroll
      for (int r = 0; r < kG; r++) acc[r] = __longlong_as_double(0x7ff8000000000000ll);
    }
    double sums;  // row r's in lane 4 r
    if constexpr (kG == 1) {
      sums = acc[0];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sums += __shfl_xor_sync(~0u, sums, o);
    } else {
      sums = warp_sum8(acc, lane);
    }
    __syncwarp();
    // the group's own triangle, by every lane
    double w[kG];
#pragma unroll
    for (int i = 0; i < kG; i++) {
      const int r = kBwd ? kG - 1 - i : i;
      double s = __shfl_sync(~0u, own, r) - __shfl_sync(~0u, sums, 4 * r);
#pragma unroll
      for (int q = 0; q < kG; q++)
        if (kBwd ? q > r : q < r) {
          const double e = cg[r][q];
          if (!pending(e)) s = fma(-e, w[q], s);
        }
      w[r] = kBwd ? s * __shfl_sync(~0u, di, r) : s;
      if (!kBwd && r0 + r == withhold)  // (its readers in the group are left without it too)
        w[r] = __longlong_as_double(0x7ff8000000000000ll);
      else if (lane == r && r < nr)
        st_publish(out + r0 + r, w[r]);
    }
    if (!kBwd && lane < nr) clear[r0 + lane] = __longlong_as_double((long long)kPending);
    __syncwarp();
  }
}

// Levels of the graph of row groups: 1 + the largest level among the other groups that a group's
// stored entries read.  The sweeps' own scheme with integers: a warp per group, claimed in the
// natural order of the sweep, which every dependency respects; a row publishes one word (0: not
// yet), its group's level in the low half and its own level in the graph of rows in the high half.
// ctr[8]: the most levels of a row; ctr[6]: the same, for L of levL, where the factor kernel counted the
// multipliers that the quick-split dropped too.
// A link of the chain of groups takes 0.5-0.75 us here, and 100,800 rows of the Euler P 0.6 ms for both
// orders, 8 ms from the columns on the host; but 20,000 groups that are one chain take 15 ms, on
// the host 1.7.  So the kernel has the time that the host would take (budget_ns): beyond it, or when
// the groups done after a quarter of it foretell that, the warps leave (kErrSlow) and the host
// counts.
template <bool kBwd>
__global__ void __launch_bounds__(256) k_ilut_levels(int n, int lfil, const int* __restrict__ col,
                                                     const int* __restrict__ cnt,
                                                     const int* __restrict__ levL,
                                                     unsigned long long* pub, int* __restrict__ lev,
                                                     int* __restrict__ ctr, long spin, int withhold,
                                                     unsigned long long budget_ns) {
  pdl_entry();
  const unsigned long long t0 = timer_ns();
  const int lane = threadIdx.x & 31;
  const size_t slot = (size_t)(lfil > 0 ? lfil : 1);
  const int ng = (n + kGroup - 1) / kGroup;
  int most = 0, rows = 0;  // the warp's part of ctr[6] and ctr[8]
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(ctr + (kBwd ? 2 : 1), 1);
    t = __shfl_sync(~0u, t, 0);
    if (t >= ng) break;
    const int g = kBwd ? ng - 1 - t : t, r0 = g * kGroup, nr = min(kGroup, n - r0);
    const int cl = lane < nr ? cnt[r0 + lane] : 0;
    const int longest = __reduce_max_sync(~0u, cl);
    int mx = 0, row[kGroup];
    unsigned own[kGroup];  // the entries inside the group, a bit each
#pragma unroll
    for (int r = 0; r < kGroup; r++) row[r] = 0, own[r] = 0u;
    for (int k0 = 0; k0 < longest; k0 += 64) {
      int j[2][kGroup];
      unsigned long long v[2][kGroup];
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int r = 0; r < kGroup; r++) {
          const int k = k0 + 32 * h + lane;
          const bool in = r < nr && k < __shfl_sync(~0u, cl, r);
          j[h][r] = in ? col[(size_t)(r0 + r) * slot + k] : -1;
        }
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int r = 0; r < kGroup; r++) {
          const int q = j[h][r];
          if (q >= r0 && q < r0 + nr) {
            own[r] |= 1u << (q - r0);
            j[h][r] = -1;
          }
          v[h][r] = j[h][r] >= 0 ? ld_level(pub + j[h][r]) : 0ull;
        }
      for (long it = 0;; it++) {
        bool wait = false;
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int r = 0; r < kGroup; r++) wait |= j[h][r] >= 0 && v[h][r] == 0ull;
        if (!__any_sync(~0u, wait)) break;
        if (it >= spin) {
          atomicCAS(ctr + 3, 0, kErrTimeout);
          return;
        }
        if ((it & 63) == 63) {
          const unsigned long long t = timer_ns() - t0, done = *(volatile unsigned*)(ctr + 7);
          if (__any_sync(~0u, t > budget_ns / 4 && t * ng > budget_ns * done))
            atomicCAS(ctr + 3, 0, kErrSlow);
          if (__any_sync(~0u, *(volatile int*)(ctr + 3) != 0)) return;
          __nanosleep(32);
        }
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int r = 0; r < kGroup; r++)
            if (j[h][r] >= 0 && v[h][r] == 0ull) v[h][r] = ld_level(pub + j[h][r]);
      }
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int r = 0; r < kGroup; r++) {
          mx = max(mx, (int)(unsigned)v[h][r]);
          row[r] = max(row[r], (int)(v[h][r] >> 32));
        }
    }
    mx = __reduce_max_sync(~0u, mx) + 1;
#pragma unroll
    for (int i = 0; i < kGroup; i++) {
      const int r = kBwd ? kGroup - 1 - i : i;
      const unsigned in = __reduce_or_sync(~0u, own[r]);
      int l = __reduce_max_sync(~0u, row[r]);
#pragma unroll
      for (int q = 0; q < kGroup; q++)
        if ((kBwd ? q > r : q < r) && (in >> q & 1u)) l = max(l, row[q]);
      row[r] = l + 1;
    }
#pragma unroll
    for (int r = 0; r < kGroup; r++) rows = max(rows, row[r]);  // (1 for a row past the end)
    most = kBwd ? rows : max(most, lane < nr ? levL[r0 + lane] : 0);
#pragma unroll
    for (int r = 0; r < kGroup; r++)
      if (lane == r && r < nr && r0 + r != withhold)
        asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(pub + r0 + r),
                     "l"((unsigned long long)row[r] << 32 | (unsigned)mx)
                     : "memory");
    if (lane == 0) {
      lev[g] = mx;
      atomicAdd(ctr + 7, 1);
    }
  }
  most = __reduce_max_sync(~0u, most);
  if (lane == 0) {  // (once a warp: once a group they cost 0.2 ms a sweep with 83,000 groups)
    atomicMax(ctr + 6, most);
    atomicMax(ctr + 8, rows);
  }
}

// CSR sanity before the factor kernel indexes with it: ia[0] = 0, ia non-decreasing, every
// column in [0, n); bad[0] = 1 + first failing row
__global__ void k_ilut_check(int n, const int* __restrict__ ia, const int* __restrict__ ja,
                             int* __restrict__ bad) {
  pdl_entry();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int b = ia[i], e = ia[i + 1];
  bool ok = b >= 0 && e >= b && (i > 0 || b == 0);
  if (ok)
    for (int k = b; k < e; k++) {
      const int j = ja[k];
      if (j < 0 || j >= n) { ok = false; break; }
    }
  if (!ok) atomicMin(bad, i + 1);
}

int grid_for(const void* kernel, int threads, size_t smem, long rows_per_cta, long n) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem);
  const long need = (n + rows_per_cta - 1) / rows_per_cta;
  return (int)std::max(1L, std::min(need, (long)std::max(per, 1) * sms));
}

template <typename T>
int alloc(T** p, size_t count) {
  if (cudaMalloc((void**)p, std::max<size_t>(count, 1) * sizeof(T)) != cudaSuccess) {
    fos_set_error("fos_ilut: cudaMalloc failed");
    return -100;
  }
  return 0;
}

}  // namespace

extern "C" int fos_ilut_create(fos_ilut** out, int n, int lfil) {
  if (!out || n <= 0) {
    fos_set_error("fos_ilut_create: bad arguments");
    return -1;
  }
  if (lfil < 0) {  // ilut.f:998, ierr = -4
    fos_set_error("fos_ilut_create: lfil < 0");
    return -4;
  }
  fos_ilut* f = new fos_ilut();
  f->n = n;
  f->lfil = std::min(lfil, n - 1);  // initILU, sparse.f90:341
  cudaGetDevice(&f->device);
  const size_t slots = (size_t)n * (size_t)std::max(f->lfil, 1);
  int rc = 0;
  rc = rc ? rc : alloc(&f->d_Lcol, slots);
  rc = rc ? rc : alloc(&f->d_Lval, slots);
  rc = rc ? rc : alloc(&f->d_Ucol, slots);
  rc = rc ? rc : alloc(&f->d_Uval, slots);
  rc = rc ? rc : alloc(&f->d_Lcnt, n);
  rc = rc ? rc : alloc(&f->d_Ucnt, n);
  rc = rc ? rc : alloc(&f->d_dinv, n);
  rc = rc ? rc : alloc(&f->d_done, n);
  rc = rc ? rc : alloc(&f->d_z, n);
  rc = rc ? rc : alloc(&f->d_levL, n);
  rc = rc ? rc : alloc(&f->d_permF, n);
  rc = rc ? rc : alloc(&f->d_permB, n);
  rc = rc ? rc : alloc(&f->d_ctr, kCtr);
  if (!rc && cudaMallocHost((void**)&f->h_ctr, kCtr * sizeof(int)) != cudaSuccess) {
    fos_set_error("fos_ilut_create: cudaMallocHost failed");
    rc = -100;
  }
  if (!rc) {
    if (cudaMemset(f->d_done, 0, sizeof(int) * n) != cudaSuccess) {
      fos_set_error("fos_ilut_create: cudaMemset failed");
      rc = -100;
    }
  }
  if (rc) {
    delete f;
    return rc;
  }
  *out = f;
  return 0;
}

extern "C" void fos_ilut_destroy(fos_ilut* f) { delete f; }

// The levels of k_ilut_levels on the host, from the stored columns (fetched in chunks of rows in the
// sweep's order, so host memory stays small): lev by group, row by row, *most as in ctr[6].
static int levels_on_host(fos_ilut* f, bool bwd, const int* d_col, const int* d_cnt, int* lev,
                          std::vector<int>& row, int* most, cudaStream_t s) {
  const int n = f->n;
  const size_t slot = (size_t)std::max(f->lfil, 1);
  std::fill(lev, lev + (n + kGroup - 1) / kGroup, 1);
  if (!bwd) {
    row.resize(n);
    FOS_CUDA(cudaMemcpyAsync(row.data(), f->d_levL, sizeof(int) * n, cudaMemcpyDeviceToHost, s));
    FOS_CUDA(cudaStreamSynchronize(s));
    *most = *std::max_element(row.begin(), row.end());
  }
  row.assign(n, 1);
  const int chunk = (int)std::min<size_t>(n, std::max<size_t>(1, (size_t)(16u << 20) / (slot * sizeof(int))));
  std::vector<int> cnt(chunk), col(slot * chunk);
  for (int done = 0; done < n; done += chunk) {
    const int m = std::min(chunk, n - done), lo = bwd ? n - done - m : done;
    FOS_CUDA(cudaMemcpyAsync(cnt.data(), d_cnt + lo, sizeof(int) * m, cudaMemcpyDeviceToHost, s));
    FOS_CUDA(cudaMemcpyAsync(col.data(), d_col + slot * lo, sizeof(int) * slot * m,
                             cudaMemcpyDeviceToHost, s));
    FOS_CUDA(cudaStreamSynchronize(s));
    for (int k = 0; k < m; k++) {  // the rows that row i reads are final
      const int i = bwd ? lo + m - 1 - k : lo + k, g = i / kGroup;
      const int* c = col.data() + slot * (i - lo);
      for (int e = 0; e < cnt[i - lo]; e++) {
        const int q = c[e] / kGroup;
        if (q != g) lev[g] = std::max(lev[g], lev[q] + 1);
        row[i] = std::max(row[i], row[c[e]] + 1);
      }
    }
  }
  if (bwd) *most = *std::max_element(row.begin(), row.end());
  return 0;
}

// Whether a sweep takes its rows one at a time: by what the two take, from the levels of their graphs.
// A chain of 20,000 rows (4,000 groups) takes 30.0 ms with rows and 17.3 with groups, both sweeps, so a
// level of rows costs 0.75 us and one of groups 2.2; and every row that is claimed 0.6 ns more than
// its share of a group (50,000 rows of a diagonal: 92 and 50 us).  Groups win where the rows of a
// group hang together (the unknowns of a cell), rows where a group waits for the latest of rows that
// do not: 27x28x29 cells of a 7-point stencil with 5 entries a row have 274 and 219 levels of rows
// and 3,150 of groups, 0.45 and 13.7 ms; with 700 and 3,330 1.2 and 14.7; 150x151 cells of a 5-point
// one with 900 and 330 1.32 and 1.46, with 2,000 and 625 3.3 and 2.6.
static bool one_at_a_time(int n, int rows, int groups) {
  return 0.77 * rows + 6.2e-4 * n < 2.2 * groups + 0.5;
}

// Claim orders of the two sweeps: groups of kGroup rows, or rows, sorted (stably) by their level.
static int solve_orders(fos_ilut* f, cudaStream_t s) {
  const int n = f->n, ng = (n + kGroup - 1) / kGroup;
  std::vector<int> lev, row, perm;
  std::vector<unsigned long long> pub;
  // what the host takes for an order: 100,000 rows of 8 slots 1.7 ms, 14,000 of 50 1.5.  (A row that
  // is withheld is waited for until the limit on the polls.)
  const unsigned long long host_ns = 50000ull + 5ull * n + 2ull * n * std::max(f->lfil, 1);
  const unsigned long long budget = f->withhold >= 0 ? ~0ull : host_ns;
  auto order = [&](auto kernel, const int* d_col, const int* d_cnt, int* d_perm, int* per, int* nlev,
                   int* nlev_rows) -> int {
    lev.resize(ng);
    row.clear();
    FOS_CUDA(cudaMemsetAsync(f->d_ctr, 0, kCtr * sizeof(int), s));
    FOS_CUDA(cudaMemsetAsync(f->d_z, 0, sizeof(double) * n, s));  // (refilled before every solve)
    kernel<<<grid_for((const void*)kernel, 256, 0, 8, std::min(ng, 2432)), 256, 0, s>>>(
        n, f->lfil, d_col, d_cnt, f->d_levL, reinterpret_cast<unsigned long long*>(f->d_z), d_perm,
        f->d_ctr, f->spin_limit > 0 ? f->spin_limit : kSpinLimit, f->withhold, budget);
    f->launches++;
    FOS_CUDA(cudaGetLastError());
    FOS_CUDA(cudaMemcpyAsync(lev.data(), d_perm, sizeof(int) * ng, cudaMemcpyDeviceToHost, s));
    FOS_CUDA(cudaMemcpyAsync(f->h_ctr, f->d_ctr, kCtr * sizeof(int), cudaMemcpyDeviceToHost, s));
    FOS_CUDA(cudaStreamSynchronize(s));
    if (f->h_ctr[3] == kErrSlow) {
      if (int rc = levels_on_host(f, d_perm == f->d_permB, d_col, d_cnt, lev.data(), row, f->h_ctr + 6, s))
        return rc;
      f->h_ctr[8] = *std::max_element(row.begin(), row.end());
    } else if (f->h_ctr[3]) {
      fos_set_error("fos_ilut_factor_dev: a dependency wait ran out");
      return -6;
    }
    *nlev_rows = f->h_ctr[6];
    *per = kGroup;
    if (one_at_a_time(n, f->h_ctr[8], *std::max_element(lev.begin(), lev.end()))) {
      *per = 1;
      if (row.empty()) {  // the rows' levels are where they were published
        pub.resize(n);
        row.resize(n);
        FOS_CUDA(cudaMemcpyAsync(pub.data(), f->d_z, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
        FOS_CUDA(cudaStreamSynchronize(s));
        for (int i = 0; i < n; i++) row[i] = (int)(pub[i] >> 32);
      }
      lev.swap(row);
    }
    const int m = (int)lev.size(), nl = *std::max_element(lev.begin(), lev.end());
    std::vector<int> start(nl + 2, 0);
    perm.resize(m);
    for (int g = 0; g < m; g++) start[lev[g] + 1]++;
    for (int l = 0; l <= nl; l++) start[l + 1] += start[l];
    for (int g = 0; g < m; g++) perm[start[lev[g]]++] = g;
    FOS_CUDA(cudaMemcpyAsync(d_perm, perm.data(), sizeof(int) * m, cudaMemcpyHostToDevice, s));
    FOS_CUDA(cudaStreamSynchronize(s));
    *nlev = nl;
    return 0;
  };
  if (int rc = order(k_ilut_levels<false>, f->d_Lcol, f->d_Lcnt, f->d_permF, &f->perF, &f->swF, &f->nlevF))
    return rc;
  return order(k_ilut_levels<true>, f->d_Ucol, f->d_Ucnt, f->d_permB, &f->perB, &f->swB, &f->nlevB);
}

int fos_ilut_factor_on(fos_ilut* f, const int* ia, const int* ja, const double* a,
                       double droptol, cudaStream_t s) {
  if (!f || !ia || !ja || !a) {
    fos_set_error("fos_ilut_factor_dev: bad arguments");
    return -1;
  }
  int dev = 0, smem_max = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  {
    const int big = INT_MAX;
    FOS_CUDA(cudaMemcpyAsync(f->d_ctr + 5, &big, sizeof(int), cudaMemcpyHostToDevice, s));
    k_ilut_check<<<(f->n + 255) / 256, 256, 0, s>>>(f->n, ia, ja, f->d_ctr + 5);
    f->launches++;
    FOS_CUDA(cudaGetLastError());
    FOS_CUDA(cudaMemcpyAsync(f->h_ctr + 5, f->d_ctr + 5, sizeof(int), cudaMemcpyDeviceToHost, s));
    FOS_CUDA(cudaStreamSynchronize(s));
    if (f->h_ctr[5] != INT_MAX) {
      fos_set_error("fos_ilut_factor_dev: malformed CSR at row " + std::to_string(f->h_ctr[5]));
      return -1;
    }
  }
  f->factored = false;  // until the factors and the sweeps' orders are complete
  for (;;) {
    const size_t row_smem = (size_t)56 * f->cap;
    if (kWarps * row_smem > (size_t)smem_max) {
      fos_set_error("fos_ilut_factor_dev: a row outgrew the largest working capacity (" +
                    std::to_string(f->cap / 2) + " entries of L and of U)");
      return -1;
    }
    const int rows = (int)std::min<size_t>(FOS_ILUT_WARPS, ((size_t)smem_max - 1024) / row_smem);
    const size_t smem = rows * row_smem;
    // (the same value for every object and capacity: another thread may set it before this launch)
    FOS_CUDA(cudaFuncSetAttribute(k_ilut_factor, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  smem_max - 1024));
    FOS_CUDA(cudaMemsetAsync(f->d_ctr, 0, 5 * sizeof(int), s));
    f->fepoch++;
    const int grid = grid_for((const void*)k_ilut_factor, 32 * rows, smem, rows, f->n);
    k_ilut_factor<<<grid, 32 * rows, smem, s>>>(f->n, ia, ja, a, f->lfil, droptol, f->cap, f->fepoch,
                                                f->d_Lcol, f->d_Lval, f->d_Lcnt, f->d_Ucol,
                                                f->d_Uval, f->d_Ucnt, f->d_dinv, f->d_levL,
                                                f->d_done, f->d_ctr,
                                                f->spin_limit > 0 ? f->spin_limit : kSpinLimit,
                                                f->withhold);
    f->launches++;
    FOS_CUDA(cudaGetLastError());
    FOS_CUDA(cudaMemcpyAsync(f->h_ctr, f->d_ctr, 5 * sizeof(int), cudaMemcpyDeviceToHost, s));
    FOS_CUDA(cudaStreamSynchronize(s));
    const int err = f->h_ctr[3], row = f->h_ctr[4];
    if (err == kErrCapacity) {  // a row outgrew the working copy: redo with twice the room
      f->cap *= 2;
      continue;
    }
    if (err == 0) {
      if (int rc = solve_orders(f, s)) return rc;
      f->factored = true;
    }
    if (err == kErrZeroRow) {
      fos_set_error("fos_ilut_factor_dev: zero row " + std::to_string(row + 1));
      return -5;
    }
    if (err == kErrTimeout) {
      fos_set_error("fos_ilut_factor_dev: a dependency wait ran out");
      return -6;
    }
    return 0;
  }
}

int fos_ilut_solve_on(fos_ilut* f, const double* y, double* x, cudaStream_t s) {
  if (!f || !y || !x || !f->factored) {
    fos_set_error("fos_ilut_solve_dev: bad arguments or no factorisation");
    return -1;
  }
  FOS_CUDA(cudaMemsetAsync(f->d_ctr, 0, 4 * sizeof(int), s));
  const long spin = f->spin_limit > 0 ? f->spin_limit : kSpinLimit;
  k_fill_pending<<<(f->n + 255) / 256, 256, 0, s>>>(f->n, f->d_z);
  // groups in flight: kLookahead levels of the average width, at least one CTA per SM
  auto sweep = [&](auto kernel, int per, int nlev, const int* col, const double* val, const int* cnt,
                   const int* perm, const double* rhs, double* out, double* clear, int withhold) {
    const int ng = (f->n + per - 1) / per;
    const long width = (ng + std::max(nlev, 1) - 1) / std::max(nlev, 1);
    const long warps = std::max((long)FOS_ILUT_MIN_WARPS, kLookahead * width);
    const int grid = std::min(grid_for((const void*)kernel, 256, 0, 8, ng), (int)((warps + 7) / 8));
    kernel<<<grid, 256, 0, s>>>(f->n, f->lfil, col, val, cnt, f->d_dinv, perm, rhs, out, clear,
                                f->d_ctr, spin, withhold);
  };
  sweep(f->perF == 1 ? k_ilut_sweep<false, 1> : k_ilut_sweep<false, kGroup>, f->perF, f->swF, f->d_Lcol,
        f->d_Lval, f->d_Lcnt, f->d_permF, y, f->d_z, x, f->withhold);
  sweep(f->perB == 1 ? k_ilut_sweep<true, 1> : k_ilut_sweep<true, kGroup>, f->perB, f->swB, f->d_Ucol,
        f->d_Uval, f->d_Ucnt, f->d_permB, f->d_z, x, nullptr, -1);
  f->launches += 3;
  FOS_CUDA(cudaGetLastError());
  return 0;
}

extern "C" int fos_ilut_factor_dev(fos_ilut* f, const int* ia, const int* ja, const double* a,
                                   double droptol, void* stream) {
  return fos_ilut_factor_on(f, ia, ja, a, droptol, (cudaStream_t)stream);
}

extern "C" int fos_ilut_solve_dev(fos_ilut* f, const double* y, double* x, void* stream) {
  return fos_ilut_solve_on(f, y, x, (cudaStream_t)stream);
}

// Failure injection for tests: the wait limit and a row that is never published.
extern "C" int fos_ilut_set_wait_limit(fos_ilut* f, long polls, int withhold_row) {
  if (!f || withhold_row < -1 || withhold_row >= f->n) {
    fos_set_error("fos_ilut_set_wait_limit: bad arguments");
    return -1;
  }
  f->spin_limit = polls > 0 ? polls : 0;
  f->withhold = withhold_row;
  return 0;
}

// Solve status after the stream has drained: 0, or -6 when a dependency wait ran out.
extern "C" int fos_ilut_status(fos_ilut* f) {
  if (!f) return -1;
  int h = 0;
  FOS_CUDA(cudaMemcpy(&h, f->d_ctr + 3, sizeof(int), cudaMemcpyDeviceToHost));
  if (h == kErrTimeout) {
    fos_set_error("fos_ilut: a dependency wait ran out");
    return -6;
  }
  return 0;
}

// The factors in SPARSKIT's MSR layout on the host (1-based values, as ilut returns them):
// alu(1:n) the inverted diagonal, jlu(1) = n + 2, row i = its L then its U entries from
// ju(i).  Returns the used length of alu/jlu (jlu(n+1) - 1), or < 0.
extern "C" long fos_ilut_copy(const fos_ilut* f, double* alu, int* jlu, int* ju, long iwk) {
  if (!f || !f->factored) {
    fos_set_error("fos_ilut_copy: no factorisation");
    return -1;
  }
  const int n = f->n;
  const size_t slot = (size_t)std::max(f->lfil, 1);
  std::vector<int> lc(n), uc(n);
  if (cudaMemcpy(lc.data(), f->d_Lcnt, sizeof(int) * n, cudaMemcpyDeviceToHost) != cudaSuccess ||
      cudaMemcpy(uc.data(), f->d_Ucnt, sizeof(int) * n, cudaMemcpyDeviceToHost) != cudaSuccess) {
    fos_set_error("fos_ilut_copy: cudaMemcpy failed");
    return -100;
  }
  long total = n + 1;
  for (int i = 0; i < n; i++) total += lc[i] + uc[i];
  if (!alu || !jlu || !ju) return total;
  if (iwk < total) {
    fos_set_error("fos_ilut_copy: iwk too small");
    return -2;
  }
  std::vector<int> col(slot * n);
  std::vector<double> val(slot * n), dv(n);
  if (cudaMemcpy(dv.data(), f->d_dinv, sizeof(double) * n, cudaMemcpyDeviceToHost) != cudaSuccess) {
    fos_set_error("fos_ilut_copy: cudaMemcpy failed");
    return -100;
  }
  for (int i = 0; i < n; i++) alu[i] = dv[i];
  alu[n] = 0.0;
  long q = n + 1;  // 0-based position of the next entry (1-based n + 2)
  jlu[0] = n + 2;
  if (cudaMemcpy(col.data(), f->d_Lcol, sizeof(int) * slot * n, cudaMemcpyDeviceToHost) != cudaSuccess ||
      cudaMemcpy(val.data(), f->d_Lval, sizeof(double) * slot * n, cudaMemcpyDeviceToHost) != cudaSuccess) {
    fos_set_error("fos_ilut_copy: cudaMemcpy failed");
    return -100;
  }
  std::vector<int> ucol(slot * n);
  std::vector<double> uval(slot * n);
  if (cudaMemcpy(ucol.data(), f->d_Ucol, sizeof(int) * slot * n, cudaMemcpyDeviceToHost) != cudaSuccess ||
      cudaMemcpy(uval.data(), f->d_Uval, sizeof(double) * slot * n, cudaMemcpyDeviceToHost) != cudaSuccess) {
    fos_set_error("fos_ilut_copy: cudaMemcpy failed");
    return -100;
  }
  for (int i = 0; i < n; i++) {
    for (int k = 0; k < lc[i]; k++, q++) {
      alu[q] = val[(size_t)i * slot + k];
      jlu[q] = col[(size_t)i * slot + k] + 1;
    }
    ju[i] = (int)(q + 1);
    for (int k = 0; k < uc[i]; k++, q++) {
      alu[q] = uval[(size_t)i * slot + k];
      jlu[q] = ucol[(size_t)i * slot + k] + 1;
    }
    jlu[i + 1] = (int)(q + 1);
  }
  return q;
}

extern "C" int fos_ilut_info(const fos_ilut* f, long* out) {
  if (!f || !out) return -1;
  out[0] = f->n;
  out[1] = f->lfil;
  out[2] = f->cap;
  out[3] = f->launches;
  out[4] = f->nlevF;
  out[5] = f->nlevB;
  return 0;
}

// ---------------------------------------------------------------- the Euler preconditioner
// With FOS_PREC_ILUT, pset factors the scalar P = I - gamma diag(1/v) J with ILUT instead of
// block ILU(0), the way fopbc wires its ILU class (modPbc.f90:676-711: COO -> setCOO ->
// fact(droptol) -> lusol).  P is laid out in the ILU position order, unknown 5p + a for
// component a of the cell at position p, each row's columns ascending (blocks by position,
// components within a block).  psol permutes r into that order, solves, and permutes back.
namespace {

__global__ void k_pcsr_rows(int nC, const int* __restrict__ prow, int* __restrict__ ia) {
  pdl_entry();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r > 5 * nC) return;
  if (r == 5 * nC) { ia[r] = 25 * prow[nC]; return; }
  const int p = r / 5, a = r - 5 * p;
  ia[r] = 25 * prow[p] + 5 * a * (prow[p + 1] - prow[p]);
}

__global__ void k_pcsr_cols(int nC, const int* __restrict__ prow, const int* __restrict__ pcol,
                            int* __restrict__ ja) {
  pdl_entry();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= 5 * nC) return;
  const int p = r / 5, a = r - 5 * p, s0 = prow[p], nb = prow[p + 1] - s0;
  int* dst = ja + 25 * (size_t)s0 + 5 * a * nb;
  for (int s = 0; s < nb; s++)
    for (int b = 0; b < 5; b++) dst[5 * s + b] = 5 * pcol[s0 + s] + b;
}

// P entries as the oracle forms them: (1 on the diagonal) - (gamma / v) J, no contraction
template <typename TJ>
__global__ void k_pcsr_vals(int nC, const int* __restrict__ prow, const int* __restrict__ pdiag,
                            const int* __restrict__ ord, const double* __restrict__ vol,
                            double gamma, const TJ* __restrict__ J, double* __restrict__ A) {
  pdl_entry();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= 5 * nC) return;
  const int p = r / 5, a = r - 5 * p, s0 = prow[p], nb = prow[p + 1] - s0;
  const double sc = gamma / vol[ord[p]];
  double* dst = A + 25 * (size_t)s0 + 5 * a * nb;
  for (int s = 0; s < nb; s++)
    for (int b = 0; b < 5; b++) {
      const double d = (s0 + s == pdiag[p] && a == b) ? 1.0 : 0.0;
      dst[5 * s + b] = __dsub_rn(d, __dmul_rn(sc, (double)J[25 * (size_t)(s0 + s) + 5 * a + b]));
    }
}

__global__ void k_ilut_in(int nC, const int* __restrict__ ipos, const double* __restrict__ r,
                          double* __restrict__ x) {
  pdl_entry();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nC) return;
  const size_t q = 5 * (size_t)ipos[i];
#pragma unroll
  for (int a = 0; a < 5; a++) x[q + a] = r[(size_t)a * nC + i];
}

__global__ void k_ilut_out(int nC, const int* __restrict__ ipos, const double* __restrict__ x,
                           double* __restrict__ z) {
  pdl_entry();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nC) return;
  const size_t q = 5 * (size_t)ipos[i];
#pragma unroll
  for (int a = 0; a < 5; a++) z[(size_t)a * nC + i] = x[q + a];
}

inline int blocks(long n, int t = 256) { return (int)((n + t - 1) / t); }

}  // namespace

int fos_ilut_ctx_factor(fos_ctx* c, double gamma) {
  const int nC = c->nC, n = 5 * nC;
  if (!c->has_jac) {
    fos_set_error("ILUT: no Jacobian assembled");
    return -1;
  }
  if (c->ilut && c->ilut->lfil != std::min(c->ilut_lfil, n - 1)) {
    fos_ilut_destroy(c->ilut);
    c->ilut = nullptr;
  }
  if (!c->d_pia) {
    const size_t nnz = 25 * (size_t)c->nnzb;
    if (nnz > (size_t)INT_MAX) {
      fos_set_error("ILUT: P has more than 2^31 - 1 entries");
      return -2;
    }
    FOS_CUDA(cudaMalloc((void**)&c->d_pia, sizeof(int) * (n + 1)));
    FOS_CUDA(cudaMalloc((void**)&c->d_pja, sizeof(int) * nnz));
    FOS_CUDA(cudaMalloc((void**)&c->d_pa, sizeof(double) * nnz));
    FOS_CUDA(cudaMalloc((void**)&c->d_vol, sizeof(double) * nC));
    FOS_CUDA(cudaMalloc((void**)&c->d_ilut_x, sizeof(double) * n));
    FOS_CUDA(cudaMemcpy(c->d_vol, c->h_vol.data(), sizeof(double) * nC, cudaMemcpyHostToDevice));
    fos_launch(c, k_pcsr_rows, blocks(n + 1), 256, nC, (const int*)c->d_prow, c->d_pia);
    fos_launch(c, k_pcsr_cols, blocks(n), 256, nC, (const int*)c->d_prow, (const int*)c->d_pcol,
               c->d_pja);
  }
  if (!c->ilut)
    if (int rc = fos_ilut_create(&c->ilut, n, c->ilut_lfil)) return rc;
  if (c->flags & FOS_ILU_FP32)
    fos_launch(c, k_pcsr_vals<float>, blocks(n), 256, nC, (const int*)c->d_prow,
               (const int*)c->d_pdiag, (const int*)c->d_ord, (const double*)c->d_vol, gamma,
               (const float*)c->d_Jraw, c->d_pa);
  else
    fos_launch(c, k_pcsr_vals<double>, blocks(n), 256, nC, (const int*)c->d_prow,
               (const int*)c->d_pdiag, (const int*)c->d_ord, (const double*)c->d_vol, gamma,
               (const double*)c->d_Jraw, c->d_pa);
  FOS_LAUNCH_CHECK();
  const long before = c->ilut->launches;
  const int rc = fos_ilut_factor_on(c->ilut, c->d_pia, c->d_pja, c->d_pa, c->ilut_droptol,
                                    c->stream);
  c->n_launch += c->ilut->launches - before;
  c->has_factor = rc == 0;
  c->ilu_ierr = rc == -5 ? 1 : 0;
  return rc == -5 ? 0 : rc;  // a zero row is reported like a zero pivot (recoverable)
}

int fos_ilut_ctx_apply(fos_ctx* c, const double* r, double* z) {
  if (!c->ilut || !c->has_factor) {
    fos_set_error("ILUT: no factorisation");
    return -1;
  }
  fos_launch(c, k_ilut_in, blocks(c->nC), 256, c->nC, (const int*)c->d_ipos, r, c->d_ilut_x);
  const long before = c->ilut->launches;
  if (int rc = fos_ilut_solve_on(c->ilut, c->d_ilut_x, c->d_ilut_x, c->stream)) return rc;
  c->n_launch += c->ilut->launches - before;
  fos_launch(c, k_ilut_out, blocks(c->nC), 256, c->nC, (const int*)c->d_ipos,
             (const double*)c->d_ilut_x, z);
  FOS_LAUNCH_CHECK();
  return 0;
}

extern "C" int fos_ctx_set_ilut(fos_ctx* c, int lfil, double droptol) {
  if (!c || lfil < 0 || !(droptol >= 0.0)) {
    fos_set_error("fos_ctx_set_ilut: bad arguments (lfil >= 0, droptol >= 0)");
    return -1;
  }
  c->ilut_lfil = lfil;
  c->ilut_droptol = droptol;
  c->has_factor = false;
  return 0;
}
