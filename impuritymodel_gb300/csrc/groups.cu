// Operator application to single product states in one pass (edgpu_apply_groups*): H|b> of every
// input state, merged, filtered and in upstream's order (finite.applyOp with {b: 1},
// impurityModel/ed/finite.py:1301-1511), the same bits as edgpu_apply_columns.
//
// Two terms of an operator lead from one state to the same output exactly when they create and
// annihilate the same orbitals, so which emissions merge is a property of the operator: its terms
// are sorted once per operator into groups of equal (created, annihilated) sets (apply_plan_kernel).
// Per state, a lane then takes a whole group: it tests the flipped orbitals once, adds the group's
// terms in term order (each term left with at most two spectator orbitals to test) and has the
// merged output; no emission buffer, no hash of output states, no W-word keys.  The fermionic sign
// is the parity of the occupied orbitals below each flipped orbital, read as a bit of the state's
// running parity, times a sign per term that does not depend on the state.
//
// Against the two-pass form (a count and a fill launch that each did all of the work; per state an
// emission buffer with an O(m^2) ordered merge, ~19 dependent reads for every basis lookup, a
// double-precision hypot per output) the application launches of the 316-orbital photoemission
// sector's construction (462 120 states, 2542 terms) take 3.4 ms instead of 71.  What the one pass is
// made of there: some 80 candidate groups a state tested against occupations and restrictions (61
// of them hops out of a full bath that the restrictions drop; the counts of all restrictions change by
// bit-sliced sums), ~8 that survive, finished 32 at a time.
//
// Diagonal sums (some 600 valid terms a state in term order, one dependent FP64 add each, ~64 cycles)
// run a state per lane in other warps than the off-diagonal outputs, so that the chain is the launch's
// latency only once; the outputs go to an arena in the order the states finish, and
// edgpu_apply_groups_gather moves them to their rows once the row offsets are known.
#include "common.cuh"

namespace edgpu {
namespace {

constexpr int kPlanThreads = 1024;
constexpr int kPlanMaxTerms = 8192;  // sorted in one CTA's shared memory
constexpr int kNoKey = 1024;         // bucket of the groups that create nothing
constexpr int kDiagKey = 1025;       // bucket of the terms that map a state onto itself
constexpr int kNever = 2047;         // terms that vanish on every state
constexpr int kBuckets = 1026;
constexpr uint32_t kNone = 0x7FF;    // absent orbital entry

// The operator sorted into groups.  gkey: four 11-bit entries (orbital << 1 | created), orbitals
// ascending, kNone past the last, above them the bucket (lowest created orbital).
struct Plan {
  int* head;        // [0]: groups
  int* bptr;        // [kBuckets + 1] first group of each bucket
  uint64_t* gkey;   // [G]
  uint16_t* gptr;   // [G + 1] first term of each group
  uint32_t* desc;   // [T] spectators and signs
  uint16_t* term;   // [T] index in the operator
  double* re;       // [T] coefficients with the state-independent sign
  double* im;       // [T]
};

// desc: orbital, required occupation and presence of two spectators; sign bit of a zero imaginary part
constexpr uint32_t kReq1 = 1u << 10, kHas1 = 1u << 11, kReq2 = 1u << 22, kHas2 = 1u << 23, kImNeg = 1u << 25;

__host__ __device__ inline size_t plan_bytes(int T) {
  return 64 + sizeof(int) * (size_t)(kBuckets + 2) + (size_t)T * (8 + 4 + 2 + 2 + 16) + 64;
}

__host__ __device__ inline Plan plan_at(void* base, int T) {
  Plan p;
  unsigned char* b = reinterpret_cast<unsigned char*>(base);
  p.gkey = reinterpret_cast<uint64_t*>(b);
  p.re = reinterpret_cast<double*>(p.gkey + T);
  p.im = p.re + T;
  p.desc = reinterpret_cast<uint32_t*>(p.im + T);
  p.bptr = reinterpret_cast<int*>(p.desc + T);
  p.head = p.bptr + kBuckets + 1;
  p.term = reinterpret_cast<uint16_t*>(p.head + 1);
  p.gptr = p.term + T;
  return p;
}

// One term taken apart: what it needs of a state, what it flips, its sign up to the parity below
// the flipped orbitals.  False when no state survives it, or one of its orbitals is none of the
// state's n_orb.
__device__ bool parse_term(uint64_t ops, int n_orb, uint64_t& key, uint32_t& desc, bool& negative) {
  int orb[4];
  bool initial[4], now[4];
  int n = 0;
  negative = false;
#pragma unroll
  for (int k = 3; k >= 0; --k) {  // right to left
    const uint32_t op = (uint32_t)(ops >> (16 * k)) & 0xFFFFu;
    if (!(op & 0x8000u)) continue;
    const int o = (int)(op & 0x3FFu);
    const bool cre = (op & 0x4000u) != 0;
    if (o >= n_orb) return false;
    int at = -1;
    for (int q = 0; q < n; ++q) {
      if (orb[q] == o) at = q;
      if (orb[q] < o && now[q] != initial[q]) negative = !negative;  // flipped since, and counted
    }
    if (at < 0) {
      at = n++;
      orb[at] = o;
      initial[at] = now[at] = !cre;
    }
    if (now[at] == cre) return false;
    now[at] = cre;
  }
  for (int a = 1; a < n; ++a)  // by orbital
    for (int b = a; b > 0 && orb[b] < orb[b - 1]; --b) {
      const int o = orb[b];
      const bool i0 = initial[b], w0 = now[b];
      orb[b] = orb[b - 1], initial[b] = initial[b - 1], now[b] = now[b - 1];
      orb[b - 1] = o, initial[b - 1] = i0, now[b - 1] = w0;
    }
  int bucket = kNoKey, flips = 0, spect = 0;
  key = 0;
  desc = 0;
  for (int q = 0; q < n; ++q) {
    if (now[q] != initial[q]) {
      if (now[q] && bucket == kNoKey) bucket = orb[q];
      key |= (uint64_t)((orb[q] << 1) | (now[q] ? 1 : 0)) << (33 - 11 * flips);
      ++flips;
    } else {
      const uint32_t d = (uint32_t)orb[q] | (initial[q] ? kReq1 : 0u) | kHas1;
      desc |= spect ? d << 12 : d;
      ++spect;
    }
  }
  for (int q = flips; q < 4; ++q) key |= (uint64_t)kNone << (33 - 11 * q);
  if (flips == 0) bucket = kDiagKey;
  key |= (uint64_t)bucket << 44;
  return true;
}

// One CTA: terms sorted by (bucket, flips, term index) with a bitonic network, cut into groups.
__global__ void __launch_bounds__(kPlanThreads) apply_plan_kernel(const uint64_t* __restrict__ ops,
                                                                  const double2* __restrict__ coeff, int T, int N,
                                                                  int n_orb, void* plan) {
  extern __shared__ __align__(16) unsigned char sm[];
  uint64_t* key = reinterpret_cast<uint64_t*>(sm);
  uint32_t* idx = reinterpret_cast<uint32_t*>(key + N);
  __shared__ int wsum[32];
  const Plan p = plan_at(plan, T);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int t = tid; t < N; t += kPlanThreads) {
    uint64_t k = ~0ull;
    if (t < T) {
      uint32_t d;
      bool neg;
      if (!parse_term(ops[t], n_orb, k, d, neg)) k = (uint64_t)kNever << 44;
    }
    key[t] = k;
    idx[t] = (uint32_t)t;
  }
  __syncthreads();
  for (int size = 2; size <= N; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int t = tid; t < (N >> 1); t += kPlanThreads) {
        const int lo = 2 * t - (t & (stride - 1)), hi = lo + stride;
        const uint64_t a = key[lo], b = key[hi];
        const bool above = a > b || (a == b && idx[lo] > idx[hi]);
        if (above == ((lo & size) == 0)) {
          key[lo] = b;
          key[hi] = a;
          const uint32_t i = idx[lo];
          idx[lo] = idx[hi];
          idx[hi] = i;
        }
      }
      __syncthreads();
    }
  }
  // groups: heads counted in chunks of consecutive positions per thread
  const int chunk = (N + kPlanThreads - 1) / kPlanThreads, q0 = tid * chunk;
  int heads = 0;
  for (int q = q0; q < q0 + chunk && q < N; ++q)
    heads += (key[q] >> 44) < kNever && (q == 0 || key[q] != key[q - 1]);
  int incl = heads;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int t = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    wsum[lane] = t;
  }
  __syncthreads();
  const int G = wsum[31];
  int g = (warp ? wsum[warp - 1] : 0) + incl - heads;  // groups before this thread's chunk
  for (int q = q0; q < q0 + chunk && q < N; ++q) {
    const uint64_t k = key[q];
    const int bucket = (int)(k >> 44);
    if (bucket >= kNever) {
      if (q == 0 || (key[q - 1] >> 44) < kNever) p.gptr[G] = (uint16_t)q;  // end of the last group
      continue;
    }
    if (q == 0 || k != key[q - 1]) {
      const int before = q == 0 ? -1 : (int)(key[q - 1] >> 44);
      for (int b = before + 1; b <= bucket; ++b) p.bptr[b] = g;
      p.gkey[g] = k & ((1ull << 44) - 1);
      p.gptr[g] = (uint16_t)q;
      ++g;
    }
    const bool last = q + 1 == N || (key[q + 1] >> 44) >= kNever;
    if (last) {
      for (int b = bucket + 1; b <= kBuckets; ++b) p.bptr[b] = G;
      if (q + 1 == N) p.gptr[G] = (uint16_t)N;
    }
    const int t = (int)idx[q];
    uint64_t kk;
    uint32_t d;
    bool neg;
    parse_term(ops[t], n_orb, kk, d, neg);
    double2 c = coeff[t];
    long long cr = __double_as_longlong(c.x), ci = __double_as_longlong(c.y);
    if (neg) {
      cr ^= (long long)(1ull << 63);
      ci ^= (long long)(1ull << 63);
    }
    if (ci < 0) d |= kImNeg;
    p.desc[q] = d;
    p.term[q] = (uint16_t)t;
    p.re[q] = __longlong_as_double(cr);
    p.im[q] = __longlong_as_double(ci);
  }
  if (tid == 0) {
    p.head[0] = G;
    if (G == 0) {
      for (int b = 0; b <= kBuckets; ++b) p.bptr[b] = 0;
      p.gptr[0] = 0;
    }
  }
}

// Whether any coefficient has an imaginary part, and the largest orbital of any slot in use (-1: none): one
// launch for some 18 tensor operations on every call with a caller's own tables (torch.ops.edgpu.build_csr of
// 1 to 700 states: 410-500 us by two passes, 560-590 with the tensor operations, 290-330 so).
__global__ void __launch_bounds__(kPlanThreads) term_info_kernel(const uint64_t* __restrict__ ops,
                                                                 const double2* __restrict__ coeff, int T,
                                                                 int32_t* __restrict__ info) {
  __shared__ int top[kPlanThreads / 32];
  int cplx = 0, orb = -1;
  for (int t = threadIdx.x; t < T; t += kPlanThreads) {
    cplx |= coeff[t].y != 0.0;
    const uint64_t o = ops[t];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t op = (uint32_t)(o >> (16 * k)) & 0xFFFFu;
      if (op & 0x8000u) orb = max(orb, (int)(op & 0x3FFu));
    }
  }
  orb = __reduce_max_sync(0xffffffffu, orb);
  if ((threadIdx.x & 31) == 0) top[threadIdx.x >> 5] = orb;
  cplx = __syncthreads_or(cplx);
  if (threadIdx.x >= 32) return;
  orb = __reduce_max_sync(0xffffffffu, top[threadIdx.x]);
  if (threadIdx.x == 0) {
    info[0] = cplx != 0;
    info[1] = orb;
  }
}

// Outputs of a state in the arena, in upstream's order of first occurrence.
struct Entry {
  uint64_t key;   // flipped orbitals (Plan::gkey)
  double re, im;
  int first;      // term index of the first contribution
  int idx;        // basis index or -1
};

struct GroupParams {
  const uint64_t* states;
  int64_t n;
  void* plan;
  int T;
  Restr restr;
  double weight_min;
  const uint64_t* basis;
  int64_t n_basis;
  const int32_t* table;  // hash of the basis (null: binary search)
  uint64_t table_mask;
  int filter;
  int64_t* counts;       // [n], zeroed
  int64_t* start;        // [n] first arena entry of a state
  double2* dval;         // [n] diagonal output
  int2* dinfo;           // [n] its first term (-1: none kept) and basis index
  Entry* arena;          // null: counts only
  int64_t arena_cap;
  unsigned long long* cursor;
  int cap;               // outputs per state that a warp's buffer holds
  int plan_in_smem;
  int32_t* status;
};

template <int W>
__device__ __forceinline__ int64_t group_find(const GroupParams& p, const uint64_t (&s)[W]) {
  if (!p.table) return find_state<W>(p.basis, p.n_basis, s);
  return hash_find<W>(p.basis, p.table, p.table_mask, s);
}

// |v|^2 as CPython computes it; hypot(x, 0) is |x|
__device__ __forceinline__ double abs2_fast(double re, double im) {
  return im == 0.0 ? __dmul_rn(re, re) : abs2_py(re, im);
}

// s with the orbitals of key flipped
template <int W>
__device__ __forceinline__ void flip_state(uint64_t (&s)[W], uint64_t key) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t e = (uint32_t)(key >> (33 - 11 * k)) & kNone;
    if (e == kNone) break;
    const int o = (int)(e >> 1);
    const uint64_t m = 1ull << (63 - (o & 63));
#pragma unroll
    for (int q = 0; q < W; ++q)
      if (q == (o >> 6)) s[q] ^= m;
  }
}

// bit of orbital o in words where orbital i is bit 63 - i % 64 of word i / 64, as 32-bit halves
__device__ __forceinline__ uint32_t orbital_bit(const uint32_t* half, int stride, int o) {
  // little-endian halves of a word: the high one second
  return (half[((o >> 5) ^ 1) * stride] >> (31 - (o & 31))) & 1u;
}

// Shared copy of the plan's arrays (or the global ones when they do not fit).
struct View {
  const uint64_t* gkey;
  const double *re, *im;
  const uint32_t* desc;
  const int* bptr;
  const uint16_t *term, *gptr;
};

constexpr int kCandidates = 64;  // groups a warp holds back until 32 lanes are full

template <bool CPLX>
__host__ __device__ inline size_t view_bytes(int T) {
  return (size_t)T * (8 + 8 + (CPLX ? 8 : 0) + 4 + 2 + 2) + sizeof(int) * (size_t)(kBuckets + 2) + 64;
}

// States whose candidates a warp finishes together: a code is slot << 13 | group (kPlanMaxTerms groups and
// terms).  A
// state of the photoemission sector has some ten, a third of the lanes that finish them: the construction of
// the sector (462 120 states) takes 6.4 -> 5.65 ms.
constexpr int kBatch = 4;

template <int W, bool CPLX>
__host__ __device__ inline size_t group_warp_bytes(int cap, int batch) {
  const size_t out = (size_t)cap * (8 + (CPLX ? 8 : 0) + 4 + 2 + 2);
  const size_t diag = sizeof(uint32_t) * 2 * W * 32;
  return ((out > diag ? out : diag) + 16 * (size_t)W * batch + 2 * kCandidates + 15) & ~(size_t)15;
}

// Restrictions whose count may change by -2 .. 2 from a state's, one bit each.
struct Slack {
  unsigned ok[5];
};

// Whether the flips of key keep every restriction: the changes of all counts at once, bit-sliced
// (at most two orbitals created and two annihilated; others are checked on the output state).
__device__ __forceinline__ bool restr_delta_ok(const Slack& s, const uint16_t* member, uint64_t key, bool& sliced) {
  unsigned p1 = 0, p2 = 0, q1 = 0, q2 = 0, over = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t e = (uint32_t)(key >> (33 - 11 * k)) & kNone;
    if (e == kNone) break;
    const unsigned m = member[e >> 1];
    if (e & 1u) {
      over |= p2 & m;
      p2 ^= p1 & m;
      p1 ^= m;
    } else {
      over |= q2 & m;
      q2 ^= q1 & m;
      q1 ^= m;
    }
  }
  sliced = over == 0;
  const unsigned p = p1 | p2, q = q1 | q2;
  const unsigned bad = ((p2 & ~q) & ~s.ok[4]) | (((p1 & ~q) | (p2 & q1)) & ~s.ok[3]) |
                       (((~p & ~q) | (p1 & q1) | (p2 & q2)) & ~s.ok[2]) | (((q1 & ~p) | (q2 & p1)) & ~s.ok[1]) |
                       ((q2 & ~p) & ~s.ok[0]);
  return bad == 0;
}

// The diagonal output of one state per thread; halves: its words in shared memory, [2 W][stride].
template <int W, bool CPLX>
__device__ void diagonal(const GroupParams& p, const View& v, int64_t j, uint32_t* half, int stride) {
  uint64_t s[W];
  load_state<W>(p.states + j * W, s);
  int64_t idx = -1;
  bool want = restr_ok<W>(p.restr, s);
  if (want && p.filter != EDGPU_FILTER_NONE) {
    idx = group_find<W>(p, s);
    want = p.filter == EDGPU_FILTER_IN_BASIS ? idx >= 0 : idx < 0;
  }
#pragma unroll
  for (int q = 0; q < W; ++q) {
    half[(2 * q) * stride] = (uint32_t)s[q];
    half[(2 * q + 1) * stride] = (uint32_t)(s[q] >> 32);
  }
  double re = 0.0, im = 0.0;
  int first = -1;
  bool neg0 = true, started = false;
  const int g = v.bptr[kDiagKey];
  if (want && v.bptr[kDiagKey + 1] > g) {
    // the tests of eight terms run side by side; only the additions follow one another
    constexpr int U = 8;
    const int q1 = v.gptr[g + 1];
    for (int q0 = v.gptr[g]; q0 < q1; q0 += U) {
      unsigned valid = 0, neg = 0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t d = v.desc[q0 + u < q1 ? q0 + u : q1 - 1];
        bool ok = q0 + u < q1;
        if (d & kHas1) ok = ok && orbital_bit(half, stride, d & 0x3FFu) == ((d & kReq1) ? 1u : 0u);
        if (d & kHas2) ok = ok && orbital_bit(half, stride, (d >> 12) & 0x3FFu) == ((d & kReq2) ? 1u : 0u);
        valid |= (ok ? 1u : 0u) << u;
        neg |= ((d & kImNeg) ? 1u : 0u) << u;
      }
      if (!valid) continue;
      neg0 = neg0 && (valid & ~neg) == 0;
      if (first < 0) first = v.term[q0 + __ffs(valid) - 1];
      double x[U], z[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        x[u] = v.re[q0 + u < q1 ? q0 + u : q1 - 1];
        if (CPLX) z[u] = v.im[q0 + u < q1 ? q0 + u : q1 - 1];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!((valid >> u) & 1u)) continue;
        re = started ? __dadd_rn(re, x[u]) : x[u];
        if (CPLX) im = started ? __dadd_rn(im, z[u]) : z[u];
        started = true;
      }
    }
  }
  if (!CPLX) im = neg0 ? -0.0 : 0.0;
  const bool keep = first >= 0 && abs2_fast(re, im) >= p.weight_min;
  if (keep) atomicAdd(reinterpret_cast<unsigned long long*>(p.counts + j), 1ull);
  if (p.arena) {
    p.dval[j] = make_double2(re, im);
    p.dinfo[j] = make_int2(keep ? first : -1, (int)idx);
  }
}

template <int W, bool CPLX, int NB>
__global__ void __launch_bounds__(1024) apply_groups_kernel(GroupParams p) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint16_t member[64 * W];  // restrictions that count an orbital
  static_assert(EDGPU_MAX_RESTRICTIONS <= 16, "one bit per restriction");
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const Plan pl = plan_at(p.plan, p.T);
  View v{pl.gkey, pl.re, pl.im, pl.desc, pl.bptr, pl.term, pl.gptr};
  size_t off = 0;
  if (p.plan_in_smem) {
    const int T = p.T;
    uint64_t* gk = reinterpret_cast<uint64_t*>(smem);
    double* re = reinterpret_cast<double*>(gk + T);
    double* im = re + T;
    uint32_t* de = reinterpret_cast<uint32_t*>(CPLX ? im + T : im);
    int* bp = reinterpret_cast<int*>(de + T);
    uint16_t* te = reinterpret_cast<uint16_t*>(bp + kBuckets + 1);
    uint16_t* gp = te + T;
    const int G = pl.head[0], nt = pl.gptr[G];
    for (int q = threadIdx.x; q < nt; q += blockDim.x) {
      re[q] = pl.re[q];
      if (CPLX) im[q] = pl.im[q];
      de[q] = pl.desc[q];
      te[q] = pl.term[q];
    }
    for (int q = threadIdx.x; q < G; q += blockDim.x) gk[q] = pl.gkey[q];
    for (int q = threadIdx.x; q <= G; q += blockDim.x) gp[q] = pl.gptr[q];
    for (int q = threadIdx.x; q <= kBuckets; q += blockDim.x) bp[q] = pl.bptr[q];
    v = View{gk, re, im, de, bp, te, gp};
    off = (view_bytes<CPLX>(T) + 15) & ~(size_t)15;
  }
  for (int o = threadIdx.x; o < 64 * W; o += blockDim.x) {
    unsigned m = 0;
    for (int k = 0; k < p.restr.n; ++k) m |= (unsigned)((p.restr.mask[k][o >> 6] >> (63 - (o & 63))) & 1ull) << k;
    member[o] = (uint16_t)m;
  }
  __syncthreads();
  unsigned char* mine = smem + off + group_warp_bytes<W, CPLX>(p.cap, NB) * warp;
  // per state of the batch: its words, and the parity of the occupied orbitals before each orbital
  uint64_t* const states = reinterpret_cast<uint64_t*>(mine);
  double* bre = reinterpret_cast<double*>(states + 2 * W * NB);
  double* bim = bre + p.cap;
  int* bidx = reinterpret_cast<int*>(CPLX ? bim + p.cap : bim);
  uint16_t* bfirst = reinterpret_cast<uint16_t*>(bidx + p.cap);
  uint16_t* bgroup = bfirst + p.cap;
  uint16_t* cand = reinterpret_cast<uint16_t*>(mine + group_warp_bytes<W, CPLX>(p.cap, NB) - 2 * kCandidates);

  // off-diagonal outputs of the states j0, j0 + stride, ... by the whole warp: at most `batch` of them, fewer
  // once they fill the lanes; returns how many, 0 when their outputs are more than the scratch holds
  auto off_diagonal = [&](int64_t j0, int64_t stride, int batch) -> int {
    int m = 0;   // kept outputs (warp-uniform, as nc)
    int nc = 0;  // candidate groups held back
    // merged value, filters and the kept output of a candidate, one per lane; code < 0: none
    auto finish = [&](int code) {
      const int g = NB == 1 || code < 0 ? code : code & 0x1fff;
      const uint64_t* occ = states + 2 * W * (NB == 1 || code < 0 ? 0 : code >> 13);
      const uint32_t* occ32 = reinterpret_cast<const uint32_t*>(occ);
      const uint32_t* below32 = reinterpret_cast<const uint32_t*>(occ + W);
      bool keep = false;
      double re = 0.0, im = 0.0;
      int first = -1;
      int64_t idx = -1;
      if (g >= 0) {
        const uint64_t key = v.gkey[g];
        uint32_t par = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t e = (uint32_t)(key >> (33 - 11 * k)) & kNone;
          if (e != kNone) par ^= orbital_bit(below32, 1, (int)(e >> 1));
        }
        bool neg0 = true;
        const int q1 = v.gptr[g + 1];
        for (int q = v.gptr[g]; q < q1; ++q) {
          const uint32_t d = v.desc[q];
          if ((d & kHas1) && orbital_bit(occ32, 1, (int)(d & 0x3FFu)) != ((d & kReq1) ? 1u : 0u)) continue;
          double x = v.re[q];
          if (par) x = __longlong_as_double(__double_as_longlong(x) ^ (long long)(1ull << 63));
          double z = 0.0;
          if (CPLX) {
            z = v.im[q];
            if (par) z = __longlong_as_double(__double_as_longlong(z) ^ (long long)(1ull << 63));
          }
          if (first < 0) {
            re = x;
            im = z;
            first = v.term[q];
          } else {
            re = __dadd_rn(re, x);
            if (CPLX) im = __dadd_rn(im, z);
          }
          // real operator: the sum of signed zeros is -0 only when all of them are
          if (!CPLX) neg0 = neg0 && (((d & kImNeg) != 0) != (par != 0));
        }
        if (first >= 0) {
          if (!CPLX) im = neg0 ? -0.0 : 0.0;
          keep = abs2_fast(re, im) >= p.weight_min;
          if (keep && p.filter != EDGPU_FILTER_NONE) {
            uint64_t s[W];
#pragma unroll
            for (int q = 0; q < W; ++q) s[q] = occ[q];
            flip_state<W>(s, key);
            idx = group_find<W>(p, s);
            keep = p.filter == EDGPU_FILTER_IN_BASIS ? idx >= 0 : idx < 0;
          }
        }
      }
      const unsigned b = __ballot_sync(FULL, keep);
      if (keep) {
        const int at = m + __popc(b & ((1u << lane) - 1u));
        if (at < p.cap) {
          bre[at] = re;
          if (CPLX) bim[at] = im;
          bfirst[at] = (uint16_t)(first | (code & 0x6000));  // slot << 13 | first term
          bgroup[at] = (uint16_t)(g | (!CPLX && __double_as_longlong(im) < 0 ? 0x8000 : 0));
          bidx[at] = (int)idx;
        }
      }
      m += __popc(b);
    };
    int done = 0;
    for (; done < (NB > 1 ? batch : 1) && j0 + done * stride < p.n && (done == 0 || m + nc < 32); ++done) {
      const int slot = NB > 1 ? done : 0;
      const int64_t j = j0 + slot * stride;
      uint64_t* const occ = states + 2 * W * slot;
      const uint32_t* const occ32 = reinterpret_cast<const uint32_t*>(occ);
      {
        const uint64_t x = lane < W ? p.states[j * W + lane] : 0ull;
        const unsigned odd = __ballot_sync(FULL, __popcll(x) & 1);
        uint64_t y = x >> 1;
        y ^= y >> 1;
        y ^= y >> 2;
        y ^= y >> 4;
        y ^= y >> 8;
        y ^= y >> 16;
        y ^= y >> 32;
        if (__popc(odd & ((1u << lane) - 1u)) & 1) y = ~y;
        if (lane < W) {
          occ[lane] = x;
          occ[W + lane] = y;
        }
      }
      __syncwarp();
      Slack slack;
      {
        int c = 0;
        if (lane < p.restr.n)
#pragma unroll
          for (int q = 0; q < W; ++q) c += __popcll(occ[q] & p.restr.mask[lane][q]);
#pragma unroll
        for (int d = 0; d < 5; ++d) {
          const bool ok = lane >= p.restr.n || (c + d - 2 >= p.restr.lo[lane] && c + d - 2 <= p.restr.hi[lane]);
          slack.ok[d] = __ballot_sync(FULL, ok);
        }
      }
      // which groups can act on the state at all: flipped orbitals and restrictions
      auto consider = [&](int g) {
        bool ok = g >= 0;
        if (ok) {
          const uint64_t key = v.gkey[g];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t e = (uint32_t)(key >> (33 - 11 * k)) & kNone;
            if (e != kNone && orbital_bit(occ32, 1, (int)(e >> 1)) == (e & 1u)) ok = false;
          }
          if (ok && p.restr.n > 0) {
            bool sliced;
            ok = restr_delta_ok(slack, member, key, sliced);
            if (!sliced) {
              uint64_t s[W];
#pragma unroll
              for (int q = 0; q < W; ++q) s[q] = occ[q];
              flip_state<W>(s, key);
              ok = restr_ok<W>(p.restr, s);
            }
          }
        }
        const unsigned b = __ballot_sync(FULL, ok);
        if (!b) return;
        if (ok) cand[nc + __popc(b & ((1u << lane) - 1u))] = (uint16_t)(g | slot << 13);
        nc += __popc(b);
        __syncwarp();
        if (nc >= 32) {
          nc -= 32;
          finish(cand[nc + lane]);
          __syncwarp();
        }
      };
      // the buckets of 32 orbitals at a time: the empty ones' group ranges laid end to end
      for (int c = 0; c < 2 * W; ++c) {
        const int o = 32 * c + lane;
        int lo = 0, len = 0;
        if (!orbital_bit(occ32, 1, o)) {
          lo = v.bptr[o];
          len = v.bptr[o + 1] - lo;
        }
        if (!__ballot_sync(FULL, len > 0)) continue;
        int end = len;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int y = __shfl_up_sync(FULL, end, d);
          if (lane >= d) end += y;
        }
        const int total = __shfl_sync(FULL, end, 31);
        for (int k0 = 0; k0 < total; k0 += 32) {
          const int k = k0 + lane;
          int at = 0;  // first range that ends after k
#pragma unroll
          for (int step = 16; step > 0; step >>= 1) {
            const int e = __shfl_sync(FULL, end, at + step - 1);
            if (e <= k) at += step;
          }
          const int rlo = __shfl_sync(FULL, lo, at), rend = __shfl_sync(FULL, end, at), rlen = __shfl_sync(FULL, len, at);
          consider(k < total ? rlo + (k - (rend - rlen)) : -1);
        }
      }
      for (int g0 = v.bptr[kNoKey]; g0 < v.bptr[kNoKey + 1]; g0 += 32)
        consider(g0 + lane < v.bptr[kNoKey + 1] ? g0 + lane : -1);
    }
    if (nc > 0) finish(lane < nc ? (int)cand[lane] : -1);
    __syncwarp();
    if (m > p.cap) return 0;
    // the states' entries one after another in the arena, each state's in term order
    unsigned long long at0 = 0;
    if (lane == 0 && m > 0 && p.arena) at0 = atomicAdd(p.cursor, (unsigned long long)m);
    at0 = __shfl_sync(FULL, at0, 0);
    int before = 0;
    for (int slot = 0; slot < (NB > 1 ? done : 1); ++slot) {
      int ms = NB == 1 || done == 1 ? m : 0;
      for (int k0 = 0; NB > 1 && done > 1 && k0 < m; k0 += 32)
        ms += __popc(__ballot_sync(FULL, k0 + lane < m && bfirst[k0 + lane] >> 13 == slot));
      if (lane == 0) {
        const int64_t j = j0 + slot * stride;
        if (ms > 0) atomicAdd(reinterpret_cast<unsigned long long*>(p.counts + j), (unsigned long long)ms);
        if (p.arena) p.start[j] = (int64_t)at0 + before;
      }
      before += ms;
    }
    if (p.arena && (int64_t)at0 + m <= p.arena_cap) {
      for (int k = lane; k < m; k += 32) {
        const int f = bfirst[k];
        int rank = 0;
        for (int e = 0; e < m; ++e) rank += bfirst[e] < f;
        Entry en;
        en.key = v.gkey[bgroup[k] & 0x7fff];
        en.re = bre[k];
        en.im = CPLX ? bim[k] : (bgroup[k] & 0x8000 ? -0.0 : 0.0);
        en.first = f & 0x1fff;
        en.idx = bidx[k];
        p.arena[at0 + rank] = en;
      }
    }
    __syncwarp();
    return done;
  };

  // Off-diagonal states from the first warp on, chunks of 32 diagonals from the last one back; every
  // other warp takes its diagonals first, so that their FP64 chains run beside the integer work of
  // the others.
  const int64_t nw = (int64_t)gridDim.x * warps, w0 = (int64_t)blockIdx.x * warps + warp;
  const int64_t chunks = (p.n + 31) / 32;
  for (int pass = 0; pass < 2; ++pass) {
    if ((pass ^ (warp & 1)) != 0) {
      for (int64_t c = nw - 1 - w0; c < chunks; c += nw) {
        const int64_t j = 32 * c + lane;
        if (j < p.n) diagonal<W, CPLX>(p, v, j, reinterpret_cast<uint32_t*>(bre) + lane, 32);
        __syncwarp();
      }
    } else {
      for (int64_t j = w0; j < p.n;) {
        int done = off_diagonal(j, nw, NB);
        if (NB > 1 && done == 0) done = off_diagonal(j, nw, 1);
        if (done == 0 && lane == 0) atomicExch(p.status, (int32_t)EDGPU_ERR_OVERFLOW);
        j += nw * max(done, 1);
      }
    }
  }
}

struct GatherParams {
  const uint64_t* states;
  int64_t n;
  const int64_t* offsets;
  const int64_t* start;
  const double2* dval;
  const int2* dinfo;
  const Entry* arena;
  uint64_t* out_states;
  int64_t* out_index;
  int32_t* out_col;
  double2* out_vals;
  double* out_real;
  int conj_vals;
};

// Rows of the result from the arena, a warp per state, the diagonal output at its place among the
// first term indices.
template <int W>
__global__ void __launch_bounds__(256) apply_gather_kernel(GatherParams p) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; j < p.n; j += nw) {
    const int64_t o0 = p.offsets[j];
    const int2 di = p.dinfo[j];
    const int m = (int)(p.offsets[j + 1] - o0) - (di.x >= 0 ? 1 : 0);
    if (m == 0 && di.x < 0) continue;
    const int64_t at0 = m > 0 ? p.start[j] : 0;
    auto put = [&](int64_t o, uint64_t key, double re, double im, int idx) {
      if (p.out_states) {
        uint64_t s[W];
        load_state<W>(p.states + j * W, s);
        flip_state<W>(s, key);
        store_state<W>(p.out_states + o * W, s);
      }
      if (p.out_index) p.out_index[o] = idx;
      if (p.out_col) p.out_col[o] = idx;
      if (p.conj_vals) im = __longlong_as_double(__double_as_longlong(im) ^ (long long)(1ull << 63));
      if (p.out_vals) p.out_vals[o] = make_double2(re, im);
      if (p.out_real) p.out_real[o] = re;
    };
    int before = 0;  // outputs ahead of the diagonal one
    for (int k0 = 0; k0 < m; k0 += 32) {
      const int k = k0 + lane;
      bool ahead = false;
      if (k < m) {
        const Entry e = p.arena[at0 + k];
        ahead = di.x >= 0 && e.first < di.x;
        put(o0 + k + (di.x >= 0 && !ahead ? 1 : 0), e.key, e.re, e.im, e.idx);
      }
      before += __popc(__ballot_sync(0xffffffffu, ahead));
    }
    if (di.x >= 0 && lane == 0) {
      const double2 d = p.dval[j];
      put(o0 + before, ~0ull, d.x, d.y, di.y);
    }
  }
}

template <int W, bool CPLX>
int launch_groups(GroupParams& p, cudaStream_t s) {
  const size_t limit = 218 * 1024;
  const size_t view = (view_bytes<CPLX>(p.T) + 15) & ~(size_t)15;
  size_t per_warp = group_warp_bytes<W, CPLX>(p.cap, 1);
  // a state per warp: few states in small blocks over all SMs, many in blocks of up to 32 warps that
  // share one copy of the plan (read from global memory where not even 8 warps fit beside it)
  int warps = 32;
  while (warps > 4 && (int64_t)warps * grid_cap() > p.n) warps >>= 1;
  while (warps > 1 && per_warp * warps > limit) warps >>= 1;
  if (per_warp * warps > limit) return EDGPU_ERR_ARG;
  while (warps > 8 && view + per_warp * warps > limit) warps >>= 1;
  p.plan_in_smem = view + per_warp * warps <= limit;
  // Candidates of several states finished together where restrictions leave a state few of them, every
  // warp has as many states and the room is there without giving up warps or the plan's copy.  Without
  // restrictions a state fills the lanes by itself: 60 000 states of 87 outputs take 1.45 ms in batches and
  // 1.34 one by one.
  const size_t wide = group_warp_bytes<W, CPLX>(p.cap, kBatch);
  const bool batch = p.restr.n > 0 && p.n >= (int64_t)kBatch * warps * grid_cap() &&
                     (p.plan_in_smem ? view : 0) + wide * warps <= limit;
  if (batch) per_warp = wide;
  const size_t smem = (p.plan_in_smem ? view : 0) + per_warp * warps;
  auto kern = batch ? apply_groups_kernel<W, CPLX, kBatch> : apply_groups_kernel<W, CPLX, 1>;
  int per_sm = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * warps, smem) != cudaSuccess || per_sm < 1)
    return EDGPU_ERR_CUDA;
  int64_t blocks = (p.n + (p.n + 31) / 32 + warps - 1) / warps;
  const int64_t cap = (int64_t)grid_cap() * per_sm;
  if (blocks > cap) blocks = cap;
  kern<<<(unsigned)blocks, 32 * warps, smem, s>>>(p);
  note_launch();
  return check_launch();
}

}  // namespace
}  // namespace edgpu

using namespace edgpu;

extern "C" int edgpu_apply_groups_max_terms(void) { return kPlanMaxTerms; }

extern "C" size_t edgpu_apply_plan_bytes(int n_terms) { return n_terms < 0 ? 0 : plan_bytes(n_terms); }

extern "C" int edgpu_apply_plan(int n_words, const edgpu_terms* terms, void* plan, size_t bytes, void* stream) {
  if (!terms || !plan || terms->n_terms < 1 || terms->n_terms > kPlanMaxTerms || !terms->ops || !terms->coeff)
    return EDGPU_ERR_ARG;
  if (n_words < 1 || n_words > EDGPU_MAX_WORDS || (reinterpret_cast<uintptr_t>(plan) & 15)) return EDGPU_ERR_ARG;
  if (bytes < plan_bytes(terms->n_terms)) return EDGPU_ERR_WORKSPACE;
  int N = 32;
  while (N < terms->n_terms) N <<= 1;
  const size_t smem = (size_t)N * 12;
  if (cudaFuncSetAttribute(apply_plan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return EDGPU_ERR_CUDA;
  apply_plan_kernel<<<1, kPlanThreads, smem, (cudaStream_t)stream>>>(
      terms->ops, reinterpret_cast<const double2*>(terms->coeff), terms->n_terms, N, 64 * n_words, plan);
  note_launch();
  return check_launch();
}

extern "C" int edgpu_term_info(const edgpu_terms* terms, int32_t* info, void* stream) {
  if (!terms || !info || terms->n_terms < 1 || !terms->ops || !terms->coeff) return EDGPU_ERR_ARG;
  term_info_kernel<<<1, kPlanThreads, 0, (cudaStream_t)stream>>>(
      terms->ops, reinterpret_cast<const double2*>(terms->coeff), terms->n_terms, info);
  note_launch();
  return check_launch();
}

extern "C" size_t edgpu_apply_groups_workspace(int64_t n_states) {
  if (n_states < 0) return 0;
  return (sizeof(int64_t) + sizeof(double2) + sizeof(int2)) * (size_t)n_states + 512;
}

extern "C" size_t edgpu_apply_groups_entry_bytes(void) { return sizeof(Entry); }

namespace {
struct GroupSpace {
  double2* dval;
  int64_t* start;
  int2* dinfo;
};

GroupSpace group_space(void* ws, int64_t n) {
  unsigned char* b = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ws) + 255) & ~(uintptr_t)255);
  GroupSpace g;
  g.dval = reinterpret_cast<double2*>(b);
  g.start = reinterpret_cast<int64_t*>(g.dval + n);
  g.dinfo = reinterpret_cast<int2*>(g.start + n);
  return g;
}
}  // namespace

extern "C" int edgpu_apply_groups(int n_words, const uint64_t* states, int64_t n_states, const void* plan, int n_terms,
                                  int real_terms, const edgpu_restrictions* restr, double weight_min,
                                  const uint64_t* basis, int64_t n_basis, const int32_t* table, int64_t table_size,
                                  int filter, int64_t* info_counts, void* arena, int64_t arena_entries,
                                  int scratch_entries, void* workspace, size_t workspace_bytes, void* stream) {
  if (n_states < 1 || !states || !info_counts || !plan || !workspace) return EDGPU_ERR_ARG;
  if (n_terms < 1 || n_terms > kPlanMaxTerms) return EDGPU_ERR_ARG;
  if (filter != EDGPU_FILTER_NONE && filter != EDGPU_FILTER_IN_BASIS && filter != EDGPU_FILTER_NOT_IN_BASIS)
    return EDGPU_ERR_ARG;
  if (filter != EDGPU_FILTER_NONE && (!basis || n_basis < 0 || n_basis >= (1ll << 31))) return EDGPU_ERR_ARG;
  if (table && (table_size < 2 * n_basis || (table_size & (table_size - 1)))) return EDGPU_ERR_ARG;
  if (restr && (restr->n < 0 || restr->n > EDGPU_MAX_RESTRICTIONS)) return EDGPU_ERR_ARG;
  if (n_words < 1 || n_words > EDGPU_MAX_WORDS) return EDGPU_ERR_ARG;
  if (arena && arena_entries < 1) return EDGPU_ERR_ARG;
  if (workspace_bytes < edgpu_apply_groups_workspace(n_states)) return EDGPU_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  const GroupSpace sp = group_space(workspace, n_states);
  GroupParams p{};
  p.states = states;
  p.n = n_states;
  p.plan = const_cast<void*>(plan);
  p.T = n_terms;
  p.restr = make_restr(restr);
  p.weight_min = weight_min;
  p.basis = basis;
  p.n_basis = n_basis;
  p.table = table;
  p.table_mask = table ? (uint64_t)table_size - 1 : 0;
  p.filter = filter;
  p.status = reinterpret_cast<int32_t*>(info_counts);
  p.cursor = reinterpret_cast<unsigned long long*>(info_counts + 1);
  p.counts = info_counts + 2;
  p.start = sp.start;
  p.dval = sp.dval;
  p.dinfo = sp.dinfo;
  p.arena = reinterpret_cast<Entry*>(arena);
  p.arena_cap = arena_entries;
  p.cap = scratch_entries > 0 ? scratch_entries : 256;
  if (cudaMemsetAsync(info_counts, 0, sizeof(int64_t) * (size_t)(n_states + 2), s) != cudaSuccess)
    return EDGPU_ERR_CUDA;
  EDGPU_DISPATCH_W(n_words, return real_terms ? launch_groups<W, false>(p, s) : launch_groups<W, true>(p, s));
  return EDGPU_ERR_ARG;
}

extern "C" int edgpu_apply_groups_gather(int n_words, const uint64_t* states, int64_t n_states,
                                         const int64_t* offsets, const void* arena, uint64_t* out_states,
                                         int64_t* out_index, int32_t* out_col, double* out_vals, double* out_real,
                                         int conj_vals, void* workspace, size_t workspace_bytes, void* stream) {
  if (n_states < 1 || !states || !offsets || !arena || !workspace) return EDGPU_ERR_ARG;
  if (n_words < 1 || n_words > EDGPU_MAX_WORDS) return EDGPU_ERR_ARG;
  if (workspace_bytes < edgpu_apply_groups_workspace(n_states)) return EDGPU_ERR_WORKSPACE;
  const GroupSpace sp = group_space(workspace, n_states);
  GatherParams p{};
  p.states = states;
  p.n = n_states;
  p.offsets = offsets;
  p.start = sp.start;
  p.dval = sp.dval;
  p.dinfo = sp.dinfo;
  p.arena = reinterpret_cast<const Entry*>(arena);
  p.out_states = out_states;
  p.out_index = out_index;
  p.out_col = out_col;
  p.out_vals = reinterpret_cast<double2*>(out_vals);
  p.out_real = out_real;
  p.conj_vals = conj_vals;
  int64_t blocks = (n_states + 7) / 8;
  const int64_t cap = (int64_t)grid_cap() * 16;
  if (blocks > cap) blocks = cap;
  EDGPU_DISPATCH_W(n_words, {
    apply_gather_kernel<W><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(p);
    note_launch();
  });
  return check_launch();
}
