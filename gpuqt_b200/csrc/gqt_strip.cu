// The strip moment loop of the FP64 form (sm_100a): several Chebyshev steps per launch.
//
// One step per launch moves T_{k-1}, T_{k-2}, left and T_k once per step: 75 bytes per
// site at z = 3, which bounds k_step on lattices beyond L2, and on smaller ones every
// step pays a launch (about 2.4 us for 0.3 us of work on 65,536 sites). Here a block
// marches down a strip of the lattice, E columns wide, and computes S steps at once:
// group j of its warps computes step j, two lines behind group j - 1, from the lines of
// step j - 1 that shared memory keeps in a ring. The input lines (T_{k-1}, T_{k-2} and
// the sites' records) arrive by bulk copies several lines ahead; only the last two steps'
// lines go back to HBM, so it sees about 96 bytes per site per S steps. The strip's outer
// columns and the segment's first and last lines are computed by each block that needs
// them.
//
// Per element the arithmetic is k_step's (ExactArith, neighbours in ELL order), so every
// T_k is bit-identical to the step loop's. Where every hopping of the operator is real
// the products with their zero imaginary parts are left out: adding such a product changes
// no value (only, on exact zeros, a sign; and where a vector has overflowed to infinity,
// the step at which it turns to NaN). The moments are the same compensated sums over the
// sites in another fixed order.
//
// What bounds it: instruction issue and the serial chain of a line, not HBM. On graphene
// 2,097,152 sites (3 steps of 128 columns, 65 us per launch of 3 steps, 35 % of DRAM
// throughput) a cell takes about 160 instructions of which 48 are FP64, and shared memory
// runs at 72 %. us per step, step loop first: 28.1 -> 20.3 direct, 13.0 -> 10.0 per moment
// of a symmetric set (two moments a step); the table at strip_geometry has the other sizes.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "gqt_forms_impl.cuh"
#include "gqt_strip.h"

namespace gqt {

namespace {

constexpr int kStripThreads = 384;  // most computing threads of a block: steps x columns
constexpr int kStripBlocks = 2;     // blocks per SM (72 registers a thread)
// Most dynamic shared memory of a block, with which two fit an SM.
constexpr size_t kStripSmem = (113 << 10) - 2048;
// Lines of a vector ring: an iteration reads lines q - 2 .. q + 1 of a step's ring and
// writes q + 2; input line q replaces q - 6, whose last reader is iteration q - 5, and is
// copied from then on, two iterations before its first reader.
constexpr int kRing = 6;
constexpr int kFirstLines = 5;  // input lines copied before the first iteration
// Lines of the record ring: 2 steps + 1 are in use at a time.
__host__ __device__ constexpr int rec_ring(int steps) { return steps <= 3 ? 8 : 16; }
constexpr int kMaxReach = 8;            // |c0| of an offset
constexpr int kGuard = kMaxReach * 16;  // bytes before and after the rings

// A launch: strips of b0 sites (E columns with the halo) in segments of b1 lines.
struct StripArgs {
  int d1, h0;          // sites per line, columns an offset reaches
  int steps, levels;   // steps of the geometry; of this launch
  int cols;            // E
  int b0, b1, strips;
  int lines;           // of the lattice
  int patterns;
  const int* __restrict__ pat;      // per pattern: length, then per entry packed (c0, c1)
  const double2* __restrict__ hop;  // per pattern: its hoppings
  const uint4* __restrict__ rec;    // per site: potential, 16 * pattern
  unsigned* err;                    // set when a wait for an input line ran out
  double* slab;
  size_t stride;
  unsigned* counter;
};

// Shared-memory tables of the row patterns. Offsets: per pattern Z byte offsets of the
// neighbours from the site's own place (PAD: then the row length), in three versions: the
// own line first in the ring (the line before is then kRing - 1 lines on), last, or
// neither. Hoppings: per pattern Z values (REAL: real parts).
template <int Z, bool REAL, bool PAD>
struct StripTables {
  static constexpr int kInts = Z + (PAD ? 1 : 0) <= 4 ? 4 : 8;
  static constexpr int kOffBytes = kInts * 4;                            // a multiple of 16
  static constexpr int kHopBytes = (Z + 1) / 2 * 2 * (REAL ? 8 : 16);    // a multiple of 16
};

// lane keeps a or b by one of its index bits and receives its partner's other one
__device__ __forceinline__ CSum give_take(const CSum& a, const CSum& b, int bit)
{
  const bool hi = (threadIdx.x & bit) != 0;
  CSum keep = hi ? b : a;
  const CSum give = hi ? a : b;
  csum_merge(keep, shfl_xor(give, bit));
  return keep;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, unsigned bytes,
                                          uint32_t bar)
{
  asm volatile(
    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
      "r"(dst),
    "l"(src), "r"(bytes), "r"(bar)
    : "memory");
}

// Bounded wait for phase `parity` of a barrier: false when it ran out, after 2^18 tries of
// about 4 us each (B200, a phase that does not complete), about a second. (No suspend-time
// hint: with one the compiler adds a sleep of its length to the loop; square 256^2 ran 4 %
// slower.)
__device__ __forceinline__ bool bounded_wait(uint32_t bar, unsigned parity)
{
  for (int it = 0; it < (1 << 18); ++it) {
    unsigned ok;
    asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
    if (ok)
      return true;
  }
  return false;
}

// Shared-memory accesses by 32-bit address (a pointer that alternates between the two
// vector buffers would be accessed as a generic one).
__device__ __forceinline__ double2 lds2(uint32_t a)
{
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ int4 lds4(uint32_t a)
{
  int4 v;
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(a));
  return v;
}
// a site's record: potential and 16 * pattern
__device__ __forceinline__ void lds_rec(uint32_t a, double& pot, int& pat)
{
  asm volatile("{\n\t.reg .b64 t;\n\t"
               "ld.shared.v2.b64 {%0, t}, [%2];\n\t"
               "cvt.u32.u64 %1, t;\n\t}"
               : "=d"(pot), "=r"(pat)
               : "r"(a));
}
template <int N>
__device__ __forceinline__ void lds_ints(uint32_t a, int (&v)[N])
{
#pragma unroll
  for (int k = 0; k < N; k += 4) {
    const int4 q = lds4(a + 4 * k);
    v[k] = q.x;
    v[k + 1] = q.y;
    v[k + 2] = q.z;
    v[k + 3] = q.w;
  }
}
__device__ __forceinline__ void sts2(uint32_t a, double2 v)
{
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y));
}

template <int Z, int DOT, bool REAL, bool PAD>
__global__ void __launch_bounds__(kStripThreads + 32, kStripBlocks)
  k_strip(Op op, StripArgs sa, const double2* __restrict__ p2, const double2* __restrict__ p1,
          double2* __restrict__ o2, double2* __restrict__ o1, const double2* __restrict__ left)
{
  using A = ExactArith;
  using Tab = StripTables<Z, REAL, PAD>;
  constexpr int kSums = DOT == kDotPair ? 2 : 1;
  extern __shared__ __align__(128) unsigned char strip_smem[];
  const int S = sa.steps, E = sa.cols, E16 = E * 16;
  // rings: T_{k-2}, T_{k-1}, then steps 1 .. S - 1; records; offset tables; hoppings
  const uint32_t s_base = smem_addr(strip_smem);
  const uint32_t s_ring = s_base + kGuard;
  const uint32_t ring_bytes = kRing * E16, rec_bytes = rec_ring(S) * E16;
  const uint32_t s_rec = s_ring + (S + 1) * ring_bytes + kGuard;
  const uint32_t s_off = s_rec + rec_bytes;
  const uint32_t off_bytes = sa.patterns * Tab::kOffBytes;
  const uint32_t s_hop = s_off + 3 * off_bytes;
  __shared__ __align__(8) uint64_t full[kRing];
  __shared__ double sums[kStripThreads / 32][kSums * 4];

  const int tid = threadIdx.x;
  for (int k = tid; k < 3 * sa.patterns; k += blockDim.x) {
    const int v = k / sa.patterns, p = k - v * sa.patterns;
    int* off = reinterpret_cast<int*>(strip_smem + (s_off - s_base) + k * Tab::kOffBytes);
    for (int m = 0; m < Z; ++m) {
      const int w = sa.pat[p * (Z + 1) + 1 + m];
      const int c0 = (signed char)(w & 255);
      int c1 = (signed char)((w >> 8) & 255);
      if (v == 1 && c1 < 0)
        c1 += kRing;
      if (v == 2 && c1 > 0)
        c1 -= kRing;
      off[m] = (c1 * E + c0) * 16;
    }
    if constexpr (PAD)
      off[Tab::kInts - 1] = sa.pat[p * (Z + 1)];
  }
  for (int k = tid; k < sa.patterns * Z; k += blockDim.x) {
    const int p = k / Z, m = k - p * Z;
    unsigned char* to = strip_smem + (s_hop - s_base) + p * Tab::kHopBytes;
    const double2 h = sa.hop[k];
    if constexpr (REAL)
      reinterpret_cast<double*>(to)[m] = h.x;
    else
      reinterpret_cast<double2*>(to)[m] = h;
  }
  // The gathers of a strip's outermost columns reach past the ring (values nobody uses):
  // guards and rings start at zero, so that these are ordinary numbers, and every record
  // names a pattern whatever happens to a copy.
  for (uint32_t k = tid; k < (s_off - s_base) / 16; k += blockDim.x)
    reinterpret_cast<double2*>(strip_smem)[k] = make_double2(0.0, 0.0);
  if (tid == 0) {
    for (int k = 0; k < kRing; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(full + k)), "r"(1)
                   : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();

  const int n = op.n;
  const int strip = blockIdx.x % sa.strips, seg = blockIdx.x / sa.strips;
  const int a0 = strip * sa.b0, r0 = seg * sa.b1;
  const int s0 = min(sa.b0, sa.d1 - a0);    // this strip's sites per line
  const int L = min(sa.b1, sa.lines - r0);  // this segment's lines
  const int H0 = S * sa.h0;
  const int inputs = L + 2 * S;             // input line q is lattice line r0 - S + q
  const int total = L + 2 * S + sa.levels - 3;  // iterations
  const int computing = (int)blockDim.x - 32;
  pdl_wait();  // the vectors are the previous launch's

  // The last warp copies the input lines; the others compute. (A computing warp that also
  // issued the copies was the one all others waited for: 22.7 us per step on graphene
  // 2,097,152 sites against 20.3.)
  if (tid >= computing) {
    const bool copier = tid == computing;  // (all its lanes take every barrier together)
    int issued = 0;
    uint32_t slot = 0, rslot = 0;
    int g = (int)((((long long)(r0 - S) * sa.d1 + a0 - H0) % n + n) % n);
    auto load_line = [&] {
      const uint32_t bar = smem_addr(full + issued % kRing);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                   "r"(3 * E16)
                   : "memory");
      // a line that reaches the lattice's end goes on at its start (more than once where E
      // exceeds a small lattice)
      uint32_t at = 0;
      int from = g;
      for (int rest = E; rest > 0;) {
        const int run = min(rest, n - from);
        bulk_copy(s_ring + ring_bytes + slot + at, p1 + from, run * 16, bar);
        bulk_copy(s_ring + slot + at, p2 + from, run * 16, bar);
        bulk_copy(s_rec + rslot + at, sa.rec + from, run * 16, bar);
        at += run * 16;
        rest -= run;
        from = 0;
      }
      ++issued;
      slot = slot + E16 == ring_bytes ? 0 : slot + E16;
      rslot = rslot + E16 == rec_bytes ? 0 : rslot + E16;
      g += sa.d1;
      if (g >= n)
        g -= n;
    };
    if (copier)
      while (issued < kFirstLines && issued < inputs)
        load_line();
    __syncwarp();
    for (int i = 0; i < total; ++i) {
      __syncthreads();
      if (copier && issued < inputs)
        load_line();
      __syncwarp();
    }
    pdl_trigger();
    // every copy has landed before the block leaves
    if (copier)
      for (int w = max(0, issued - kRing); w < issued; ++w)
        bounded_wait(smem_addr(full + w % kRing), (unsigned)(w / kRing) & 1u);
    __syncwarp();
    __syncthreads();
    return;
  }

  // This thread's step and column.
  const int j = tid / E + 1, c = tid % E;
  const bool mine = (unsigned)(c - H0) < (unsigned)s0;
  // the ring of T_{j-1}; T_j goes to the next ring, T_{j-2} is in the one before
  const uint32_t ring_from = s_ring + j * ring_bytes + c * 16;
  double2* const og = j == sa.levels ? o1 : (j == sa.levels - 1 ? o2 : nullptr);
  const bool keep = j < S, store = og != nullptr && mine;
  CSum re[kSums], im[kSums];
#pragma unroll
  for (int k = 0; k < kSums; ++k)
    re[k] = im[k] = CSum{0.0, 0.0};
  // this step's iterations
  const int first = 3 * (j - 1), last = j <= sa.levels ? L + 2 * S + j - 3 : first;
  // the division's constants stay in registers
  double emax = op.emax, inv_emax = op.inv_emax;
  unsigned div_span = op.div_span;
  asm volatile("" : "+d"(emax), "+d"(inv_emax), "+r"(div_span));
  int i = 0;
  for (; i < first && i < total; ++i)
    __syncthreads();
  // The next input line has landed; after a wait that ran out the block goes on without
  // waiting (on old lines, in bounds) and the host reports the error (gqt_moments_check).
  bool ok = true;
  uint32_t wait_bar = smem_addr(full);
  unsigned wait_phase = 0;
  auto landed = [&] {
    if (ok && !bounded_wait(wait_bar, wait_phase)) {
      ok = false;
      atomicOr(sa.err, kStripWait);
    }
    wait_bar += 8;
    if (wait_bar == smem_addr(full + kRing)) {
      wait_bar = smem_addr(full);
      wait_phase ^= 1u;
    }
  };
  if (first < last) {
    if (j == 1) {
      landed();
      landed();
      landed();
    }
    int q = j;                                   // this step's line: i + 1 - 2 (j - 1)
    int g = (r0 - S + q) * sa.d1 + a0 - H0 + c;  // its site
    uint32_t slot = (q % kRing) * E16, rslot = (q % rec_ring(S)) * E16;
    // what the next line needs early: its record, offsets and left
    struct Ahead {
      double pv;
      int pat;
      int off[Tab::kInts];
      double2 l;
    };
    auto fetch = [&](Ahead& a, uint32_t sl, uint32_t rs, int line, int site) {
      lds_rec(s_rec + c * 16 + rs, a.pv, a.pat);
      const uint32_t tab = sl == 0 ? s_off + off_bytes
                                   : (sl == ring_bytes - E16 ? s_off + 2 * off_bytes : s_off);
      lds_ints<Tab::kInts>(tab + a.pat * (Tab::kOffBytes / 16), a.off);
      if constexpr (DOT == kDotLeft) {
        if ((unsigned)(line - S) < (unsigned)L && mine)
          a.l = left[site];
      }
    };
    // One line: this step's values at line q, from `a`; fetches line q + 1's into `b`.
    auto line = [&](const Ahead& a, Ahead& b) {
      const uint32_t own = ring_from + slot;
      const double2 xx = lds2(own);
      double2 y[Z], h[Z];
#pragma unroll
      for (int m = 0; m < Z; ++m)
        y[m] = lds2(own + a.off[m]);
      const uint32_t hp = s_hop + a.pat * (Tab::kHopBytes / 16);
#pragma unroll
      for (int m = 0; m < Z; m += REAL ? 2 : 1) {
        const double2 t = lds2(hp + m * (REAL ? 8 : 16));
        if constexpr (REAL) {
          h[m].x = t.x;
          if (m + 1 < Z)
            h[m + 1].x = t.y;
        } else {
          h[m] = t;
        }
      }
      const double2 y0 = lds2(own - ring_bytes);
      const uint32_t ns = slot + E16 == ring_bytes ? 0 : slot + E16;
      const uint32_t nr = rslot + E16 == rec_bytes ? 0 : rslot + E16;
      fetch(b, ns, nr, q + 1, g + sa.d1);
      double tr = A::mul(a.pv, xx.x), ti = A::mul(a.pv, xx.y);
#pragma unroll
      for (int m = 0; m < Z; ++m) {
        if (PAD && m >= a.off[Tab::kInts - 1])
          continue;
        if constexpr (REAL) {
          tr = A::add(tr, A::mul(h[m].x, y[m].x));
          ti = A::add(ti, A::mul(h[m].x, y[m].y));
        } else {
          tr = A::add(tr, A::cre(h[m].x, h[m].y, y[m].x, y[m].y));
          ti = A::add(ti, A::cim(h[m].x, h[m].y, y[m].x, y[m].y));
        }
      }
      if (max(A::div_key(tr), A::div_key(ti)) >= div_span) {
        tr = A::divide_any(tr, op);
        ti = A::divide_any(ti, op);
      } else {
        tr = A::divide(tr, emax, inv_emax);
        ti = A::divide(ti, emax, inv_emax);
      }
      const double2 o = make_double2(A::two_x_minus(tr, y0.x), A::two_x_minus(ti, y0.y));
      if (keep)
        sts2(own + ring_bytes, o);
      if ((unsigned)(q - S) < (unsigned)L) {  // a line of the segment
        if (store)
          og[g] = o;
        // (columns outside the strip sum values nobody uses: dropped below)
        if constexpr (DOT == kDotPair) {
          dot_term_self(re[0], o);
          dot_term(re[kSums - 1], im[kSums - 1], o, xx);
        } else {
          dot_term(re[0], im[0], o, a.l);
        }
      }
      slot = ns;
      rslot = nr;
      ++q;
      g += sa.d1;
      // every line written is visible, and every line read may be replaced
      __syncthreads();
      ++i;
      if (j == 1 && i < last)
        landed();
    };
    Ahead a{}, b{};
    fetch(a, slot, rslot, q, g);
    while (i + 1 < last) {  // two lines a turn: what is fetched ahead needs no moves
      line(a, b);
      line(b, a);
    }
    if (i < last)
      line(a, b);
  }
  for (; i < total; ++i)
    __syncthreads();
  pdl_trigger();
  // Block partials of every step, in the layout of the deferred steps: [block][sums][4].
#pragma unroll
  for (int k = 0; k < kSums; ++k) {
    if (!mine)
      re[k] = im[k] = CSum{0.0, 0.0};
    CSum s = give_take(re[k], im[k], 16);
#pragma unroll
    for (int w = 8; w >= 1; w >>= 1)
      csum_merge(s, shfl_xor(s, w));
    if ((tid & 15) == 0) {
      double* d = &sums[tid >> 5][k * 4 + (tid & 16 ? 2 : 0)];
      d[0] = s.s;
      d[1] = s.c;
    }
  }
  __syncthreads();
  const int per = E / 32;  // warps of a step
  for (int k = tid; k < sa.levels * kSums * 2; k += computing) {
    const int lv = k / (kSums * 2), f = k % (kSums * 2);
    CSum a{0.0, 0.0};
    for (int w = lv * per; w < (lv + 1) * per; ++w)
      csum_merge(a, CSum{sums[w][f * 2], sums[w][f * 2 + 1]});
    double* dst = sa.slab + (size_t)lv * sa.stride + (size_t)blockIdx.x * kSums * 4 + f * 2;
    dst[0] = a.s;
    dst[1] = a.c;
  }
  if (blockIdx.x == 0 && tid == 0)
    sa.counter[1] = gridDim.x;
}

// Each site's record: its potential and 16 times its row pattern.
__global__ void __launch_bounds__(kBlock) k_strip_rec(const double* __restrict__ pot,
                                                      const uint8_t* __restrict__ pid, int n,
                                                      uint4* __restrict__ out)
{
  for (int i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) {
    const double v = pot[i];
    out[i] = make_uint4((unsigned)__double2loint(v), (unsigned)__double2hiint(v),
                        (unsigned)pid[i] * 16u, 0u);
  }
}

size_t table_bytes(int patterns, int z, bool real, bool pad)
{
  const size_t off = z + (pad ? 1 : 0) <= 4 ? 16 : 32;
  return patterns * (3 * off + (size_t)(z + 1) / 2 * 2 * (real ? 8 : 16));
}

// d = c1 * d1 + c0 (mod n) with |c1| <= 1 and the smallest |c0|; false above kMaxReach.
bool split_offset(long long d, long long n, long long d1, int& c0, int& c1)
{
  long long best = kMaxReach + 1;
  for (int q = -1; q <= 1; ++q) {
    if (q && !d1)
      continue;
    long long r = (d - q * d1) % n;
    if (r > n / 2)
      r -= n;
    if (r < -(n / 2))
      r += n;
    const long long a = std::llabs(r);
    if (a < best) {
      best = a;
      c0 = (int)r;
      c1 = q;
    }
  }
  return best <= kMaxReach;
}

// Time of a step of the step loop, us (a symmetric set's gives two moments), on rows of z:
// it depends on the sites alone. B200, coded operator, at these numbers of sites; beyond the
// last in proportion.
double step_loop_us(int n, int z, bool pair)
{
  constexpr int kPoints = 8;
  static const double kSites[kPoints] = {20e3, 65e3, 160e3, 450e3, 1.05e6, 1.35e6, 2.1e6, 4e6};
  static const double kTime[2][3][kPoints] = {
    // direct, rows of 3, 4 and 6
    {{2.18, 2.75, 3.95, 6.3, 11.4, 14.4, 28.0, 53.5},
     {2.20, 2.83, 3.85, 6.4, 11.6, 14.3, 28.1, 51.1},
     {2.20, 2.72, 3.95, 7.3, 14.5, 19.5, 36.6, 65.6}},
    // symmetric
    {{2.55, 3.25, 4.70, 7.3, 12.7, 15.2, 22.7, 45.0},
     {2.55, 3.55, 4.70, 7.8, 13.3, 15.9, 24.6, 49.4},
     {2.55, 3.28, 4.60, 8.4, 15.5, 18.8, 34.4, 64.6}}};
  const double* t = kTime[pair][z == 3 ? 0 : z == 4 ? 1 : 2];
  if (n >= kSites[kPoints - 1])
    return t[kPoints - 1] * n / kSites[kPoints - 1];
  int k = 1;
  while (n > kSites[k])
    ++k;
  const double f = std::max(0.0, (n - kSites[k - 1]) / (kSites[k] - kSites[k - 1]));
  return t[k - 1] + f * (t[k] - t[k - 1]);
}

// The same of the strip loop: iterations times the time of one (steps x columns cells; a
// lattice of few columns, or one that leaves few of a strip's columns after the halo, takes
// more of them), and the launch. B200, 927 lattices of 624 to 4 million sites, 10 to 2,000
// columns, reach 1 to 8, full and short rows, real and complex hoppings: within 10 % but for
// a few of less than 3,000 sites or 20 columns (20 %).
double strip_loop_us(const StripGeo& g, int n, int z, bool real, bool pad, bool pair)
{
  static const double kLine[2][3][4] = {
    // columns 32, 64, 96, 128; complex hoppings, rows of 3, 4 and 6
    {{0.68, 0.94, 1.10, 1.10}, {0.68, 0.80, 0.92, 0.92}, {0.74, 0.92, 1.02, 1.05}},
    // real
    {{0.66, 0.71, 0.77, 0.73}, {0.65, 0.75, 0.80, 0.81}, {0.73, 0.78, 0.95, 0.98}}};
  const double line = kLine[real][z == 3 ? 0 : z == 4 ? 1 : 2][g.cols / 32 - 1] +
                      (pad ? 0.05 : 0.0) + (pair ? 0.03 : 0.0);
  const double launch = 0.5 + (pair ? 1.0 : 0.0) + (n >= 1400000 ? 6.0 : g.cols == 128 ? 1.5 : 0.0);
  return (launch + line * (g.b1 + 3 * (g.steps - 1))) / g.steps;
}

}  // namespace

StripLattice strip_lattice(int n, const int* delta, int count, int* packed)
{
  auto fits = [&](long long d1, StripLattice& L) {
    L = StripLattice{};
    for (int k = 0; k < count; ++k) {
      int c0 = 0, c1 = 0;
      if (!split_offset(delta[k], n, d1, c0, c1))
        return false;
      packed[k] = (c0 & 255) | (c1 & 255) << 8;
      L.h0 = std::max(L.h0, std::abs(c0));
    }
    L.d1 = (int)d1;
    L.lines = (int)(n / d1);
    return true;
  };
  // Offsets beyond the in-line reach lie near the line length.
  std::vector<long long> far, cand;
  for (int k = 0; k < count; ++k)
    if (std::llabs(delta[k]) > kMaxReach)
      far.push_back(std::llabs(delta[k]));
  std::sort(far.begin(), far.end());
  far.erase(std::unique(far.begin(), far.end()), far.end());
  if (far.size() > 64)
    return {};
  for (long long f : far)
    for (int k = -kMaxReach; k <= kMaxReach; ++k)
      if (f + k > kMaxReach && 2 * (f + k) <= n && n % (f + k) == 0)
        cand.push_back(f + k);
  std::sort(cand.begin(), cand.end());
  cand.erase(std::unique(cand.begin(), cand.end()), cand.end());
  // the smallest in-line reach, then the shortest line
  StripLattice best, L;
  for (long long d1 : cand)
    if (fits(d1, L) && (!best.d1 || L.h0 < best.h0))
      best = L;
  if (best.d1)
    fits(best.d1, L);  // packed, again
  return best;
}

// Steps and columns by the lattice's size. A launch takes (lines of a segment + 3 (steps -
// 1)) iterations of about 0.55 us (vectors in L2) to 0.9 us (in HBM) after some 3.5 us:
// small lattices want many steps per launch, large ones wide strips, whose halo columns
// cost least, and few lines lost at a segment's ends. B200, us per step, direct / per
// moment of a symmetric set, step loop first:
//   square 100 x 90       2.11 / 1.39   6 steps of 32: 1.84 / 0.95   of 64: 1.87 / 0.97
//   square 256 x 256      2.77 / 1.84   6 of 64: 2.41 / 1.26   4 of 96: 2.54 / 1.36
//   square 400 x 380      3.72 / 2.42   6 of 64: 3.17 / 1.65   4 of 96: 3.28 / 1.72
//   square 640 x 700      6.20 / 3.96   6 of 64: 5.78 / 3.03   4 of 96: 5.46 / 2.90
//   square 1000 x 1001    11.4 / 6.83   4 of 96: 10.8 / 5.62   3 of 128: 11.2 / 5.70
//   graphene 2,097,152    28.1 / 13.0   4 of 96: 21.2 / 10.6   3 of 128: 21.1 / 10.0
//   square 2000 x 2000    51.5 / 25.6   4 of 96: 37.5 / 18.7   3 of 128: 37.1 / 17.5
StripGeo strip_geometry(const gqt_ham* h, int patterns)
{
  const StripLattice& L = h->strip;
  static const int kShapes[][2] = {{6, 32}, {6, 64}, {4, 96}, {3, 128}};
  const int first = h->n < 20000 ? 0 : h->n < 300000 ? 1 : h->n < 1400000 ? 2 : 3;
  const int sms = device_info().sms;
  const size_t tables = table_bytes(patterns, h->z, h->real_hop, h->strip_pad);
  for (int k = first; k < 4; ++k) {
    StripGeo g;
    g.steps = kShapes[k][0];
    g.cols = kShapes[k][1];
    // at least half the columns are the strip's own
    const int room = g.cols - 2 * g.steps * L.h0;
    if (2 * room < g.cols)
      continue;
    g.strips = (L.d1 + room - 1) / room;
    g.b0 = (L.d1 + g.strips - 1) / g.strips;
    g.smem = (size_t)((g.steps + 1) * kRing + rec_ring(g.steps)) * g.cols * 16 + 2 * kGuard +
             tables;
    if (g.smem > kStripSmem)
      continue;
    // one wave of two blocks per SM
    const int segs = std::min(L.lines, sms * kStripBlocks / g.strips);
    if (segs < 1)
      continue;
    g.b1 = (L.lines + segs - 1) / segs;
    g.grid = g.strips * ((L.lines + g.b1 - 1) / g.b1);
    // long lines leave short segments, most of whose iterations the ends take
    if (h->n >= 300000 && g.b1 < 3 * (g.steps - 1))
      continue;
    return g;
  }
  return {};
}

// The loops that run in strips, bit 0 the direct one, bit 1 the symmetric one: those whose
// strips are expected to take no longer than the step loop, give or take the 2.5 % at which as
// many lattices are decided wrongly one way as the other. Of the 927 lattices, direct and
// symmetric, 10 run 3 to 11 % slower so than step by step (none slower than the step loop was
// before programmatic launches), and for 7 a gain of 5 to 13 % is left. Without the
// comparison, us a step in strips / step by step: thin lattices 184 / 28 (square 210,000 x
// 10), 39 / 7.8 (60,000 x 10); slabs 24.2 / 14.7 (cubic 420 x 420 x 6); long reaches 16.3 /
// 11.1 (rows of four, 6 columns, 1000 x 1001); graphene with complex hoppings 18.8 / 14.5
// (600 x 580).
int strip_loops(const gqt_ham* h, const StripGeo& g)
{
  int loops = 0;
  for (int pair = 0; g.steps && pair < 2; ++pair)
    if (strip_loop_us(g, h->n, h->z, h->real_hop, h->strip_pad, pair) <=
        1.025 * step_loop_us(h->n, h->z, pair))
      loops |= 1 << pair;
  return loops;
}

bool strip_possible(gqt_ham* h)
{
  h->strip_pad = h->uniform ? 0 : 1;
  return strip_loops(h, strip_geometry(h, 1)) != 0;
}

gqt_status strip_upload(gqt_ham* h, const RowPatterns& rp, const std::vector<int>& packed,
                        const std::vector<double2>& hop)
{
  const int z = h->z, np = (int)rp.len.size();
  const StripGeo geo = strip_geometry(h, np);
  h->strip_loops = strip_loops(h, geo);
  if (!h->strip_loops)
    return GQT_OK;
  h->strip_patterns = np;
  // one allocation: the patterns' hoppings, their lengths and offsets, the sites' patterns
  const size_t hops = (size_t)np * z * sizeof(double2), ints = (size_t)np * (z + 1) * sizeof(int);
  std::vector<unsigned char> table(hops + ints);
  double2* const th = reinterpret_cast<double2*>(table.data());
  int* const tp = reinterpret_cast<int*>(table.data() + hops);
  for (int k = 0; k < np; ++k) {
    tp[k * (z + 1)] = rp.len[k];
    for (int m = 0; m < z; ++m) {
      const int c = rp.code[(size_t)k * z + m];
      tp[k * (z + 1) + 1 + m] = packed[c];
      th[k * z + m] = hop[c];
    }
  }
  unsigned char* dev = nullptr;
  if (cudaMalloc(&dev, table.size() + (size_t)h->n) != cudaSuccess) {
    cudaGetLastError();  // no memory for them: step by step
    h->strip_loops = 0;
    return GQT_OK;
  }
  h->strip_hop = reinterpret_cast<double2*>(dev);
  h->strip_pat = reinterpret_cast<int*>(dev + hops);
  h->strip_site = dev + table.size();
  GQT_CUDA(cudaMemcpy(dev, table.data(), table.size(), cudaMemcpyHostToDevice));
  GQT_CUDA(cudaMemcpy(h->strip_site, rp.site.data(), (size_t)h->n, cudaMemcpyHostToDevice));
  h->strip_geo = geo;
  return GQT_OK;
}

gqt_status strip_records(const gqt_ham* h)
{
  if (h->strip_rec)
    return GQT_OK;
  uint4* rec = nullptr;
  GQT_CUDA(cudaMalloc(&rec, (size_t)h->n * sizeof(uint4)));
  const int grid = std::min((h->n + kBlock - 1) / kBlock, max_grid());
  k_strip_rec<<<grid, kBlock, 0, stream()>>>(h->pot, h->strip_site, h->n, rec);
  count_launches(1);
  const cudaError_t e = cudaStreamSynchronize(stream());
  if (e != cudaSuccess) {
    cudaFree(rec);
    return cuda_fail(e, "records of the strip loop", __FILE__, __LINE__);
  }
  h->strip_rec = rec;
  return GQT_OK;
}

gqt_status strip_steps(const gqt_ham* h, const Op& op, bool pair, int levels, const double2* p2,
                       const double2* p1, double2* o2, double2* o1, const double2* left,
                       double* slab, size_t stride, unsigned* counter)
{
  const StripGeo& geo = h->strip_geo;
  StripArgs sa{};
  sa.d1 = h->strip.d1;
  sa.h0 = h->strip.h0;
  sa.steps = geo.steps;
  sa.levels = levels;
  sa.cols = geo.cols;
  sa.b0 = geo.b0;
  sa.b1 = geo.b1;
  sa.strips = geo.strips;
  sa.lines = h->strip.lines;
  sa.patterns = h->strip_patterns;
  sa.pat = h->strip_pat;
  sa.hop = h->strip_hop;
  sa.rec = h->strip_rec;
  sa.err = h->stage_err;
  sa.slab = slab;
  sa.stride = stride;
  sa.counter = counter;
  auto go = [&](auto* kernel) -> gqt_status {
    // (the same limit for every lattice: one of its own would take the room from a larger
    // lattice's launch that another thread is about to make)
    GQT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kStripSmem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(geo.grid);
    cfg.blockDim = dim3(geo.steps * geo.cols + 32);
    cfg.dynamicSmemBytes = geo.smem;
    cfg.stream = stream();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GQT_CUDA(cudaLaunchKernelEx(&cfg, kernel, op, sa, p2, p1, o2, o1, left));
    count_launches(1);
    return GQT_OK;
  };
  auto pick = [&](auto zc, auto dc) -> gqt_status {
    constexpr int Z = decltype(zc)::value;
    constexpr int D = decltype(dc)::value;
    if (h->strip_pad)
      return h->real_hop ? go(k_strip<Z, D, true, true>) : go(k_strip<Z, D, false, true>);
    return h->real_hop ? go(k_strip<Z, D, true, false>) : go(k_strip<Z, D, false, false>);
  };
  auto with_dot = [&](auto zc) -> gqt_status {
    return pair ? pick(zc, std::integral_constant<int, kDotPair>{})
                : pick(zc, std::integral_constant<int, kDotLeft>{});
  };
  switch (h->z) {
    case 3:
      return with_dot(std::integral_constant<int, 3>{});
    case 4:
      return with_dot(std::integral_constant<int, 4>{});
    case 6:
      return with_dot(std::integral_constant<int, 6>{});
    default:
      return fail(GQT_ERR_STATE, "strip loop: rows of %d entries", h->z);
  }
}

}  // namespace gqt
