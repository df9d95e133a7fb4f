// fec_pairgather.cu -- the gather of element matrices stored as symmetric halves
// (KE_PAIRS) by output entry instead of by node.
//
// Two nodes n <= m share a block of nine entries in every element that has both.
// The plan lists, for every such node pair, where those blocks are, in increasing
// element order; a thread adds a row (three entries) of one pair over its list -- the
// same additions in the same order as the per-node gathers (fec_kernels.cuh), so
// bitwise their results -- and stores it at its two places, columns (n, k) and rows
// (m, i), columns (m, i) and row (n, k).  Every stored block is read once (the
// per-node gathers read it for both nodes), nothing goes through shared memory, and
// the loads of a thread do not depend on one another.  Nodes with Dirichlet dofs need
// no path of their own.  The plan is the mesh's: only the pairs' row offsets follow the
// Dirichlet dofs (offsets_kernel).
//
// Bound: latency and issue, then DRAM.  A hex8 node of a box has 14 pairs with lists
// of 8, 4, 2 or 1; the pairs of GROUP consecutive nodes are ordered by the length of
// their lists, so that the lanes of a warp have the same (in node order a warp runs
// its longest list, and an entry per thread, not a row, spends most of its
// instructions on addresses: 1,014 warp instructions a node, 4.48 ms at 128^3). A plane of
// that mesh does not stay in L2 between the two times a column is written: 1.6 ns a node
// against 1.25 at 61 x 53 x 47.
#include <type_traits>
#include "fec_launch.h"
#include "fec_pattern.h"

namespace fec {
namespace {

constexpr int WPB = 4;      // warps per CTA of the plan kernel
// Places of a node's hash table (its neighbours m >= n): 128 unless a node has more (warps of
// 512 leave an SM a third of its warps: 48^3 165 us to fill instead of 86)
constexpr int GROUP = 8;    // nodes whose pairs are ordered together (8: 128^3 3.40 ms; 32: 3.49, 128: 3.53)
constexpr int CLASSES = 64; // list lengths told apart

// One warp per node n: its elements' nodes m >= n, told apart by their place in a hash table.
// FILL = false: how many pairs and list entries n has; FILL = true: writes
// them.  flags[0]: a node with too many neighbours or elements; flags[1]: a node of this
// block shared with another.  Nothing here depends on the Dirichlet dofs.
struct PlanArgs {
  int64_t nn, elem_start, ne, conn_off;
  int A;
  bool shared;                     // several blocks: nodes may be shared
  const int64_t* nadj_ptr;
  const uint32_t* nadj;
  const int32_t* conn;
  int32_t *nslot, *nlist;          // per node (FILL = false)
  const int64_t *slot0, *list0;    // their exclusive sums (FILL = true)
  int4* slots;                     // n, m, first list entry, row offsets (offsets_kernel)
  uint32_t* count;                 // list entries of a slot | n's and m's places in that element << 16, << 24
  uint32_t* list;                  // (element * pairs + pair) << 1 | transposed
  int* flags;
};

__device__ __forceinline__ bool owned(const PlanArgs& a, int64_t n) {
  const int64_t p0 = a.nadj_ptr[n], p1 = a.nadj_ptr[n + 1];
  return p1 > p0 && int64_t(a.nadj[p0] >> 5) >= a.elem_start && int64_t(a.nadj[p1 - 1] >> 5) < a.elem_start + a.ne;
}

template <bool FILL, int MAXT>
__global__ void __launch_bounds__(WPB * 32) plan_kernel(PlanArgs a) {
  // a place: a neighbour, its list entries so far, and which of the CHUNK elements at hand have it
  __shared__ int32_t s_key[WPB][MAXT];
  __shared__ uint32_t s_in[WPB][MAXT];
  __shared__ uint16_t s_cnt[WPB][MAXT], s_at[WPB][FILL ? MAXT : 1], s_rank[WPB][FILL ? MAXT : 1];
  __shared__ int2 s_pair[WPB][FILL ? MAXT : 1];  // the neighbours; their list entries, places << 16
  constexpr int CHUNK = 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t n = int64_t(blockIdx.x) * WPB + warp;
  if (n >= a.nn) return;
  int32_t* key = s_key[warp];
  uint32_t* in = s_in[warp];
  uint16_t* cnt = s_cnt[warp];
  const int64_t p0 = a.nadj_ptr[n], p1 = a.nadj_ptr[n + 1], cand = (p1 - p0) * a.A;
  bool use = p1 > p0 && (!a.shared || owned(a, n));
  if (use && cand > 65535) {
    if (lane == 0) a.flags[0] = 1;
    use = false;
  }
  if (!use) {
    if (!FILL && lane == 0) a.nslot[n] = a.nlist[n] = 0;
    return;
  }
  int T = 32;  // no more places than candidates
  while (T < MAXT && T < cand) T <<= 1;
  for (int i = lane; i < T; i += 32) {
    key[i] = -1;
    cnt[i] = 0;
    in[i] = 0;
  }
  __syncwarp();
  // the place of m, taken if it has none; -1 where the table is full
  auto place = [&](int32_t m) {
    unsigned h = uint32_t(m) * 2654435761u >> 16;
    for (int tries = 0; tries < T; ++tries, ++h) {
      const int i = int(h & unsigned(T - 1));
      const int32_t was = atomicCAS(&key[i], -1, m);
      if (was == -1 || was == m) return i;
    }
    return -1;
  };
  // f(element of the chunk, local element, local nodes of n and m, m): the lanes take the
  // nodes of the chunk's elements, all at once
  const unsigned by_A = 65536u / unsigned(a.A) + 1u;  // i / A = i by_A >> 16 for i < 32 * 27
  auto nodes = [&](int64_t q, auto f) {
    const int ne = int(p1 - q < CHUNK ? p1 - q : CHUNK);
    for (int i = lane; i < ne * a.A; i += 32) {
      const int j = int(unsigned(i) * by_A >> 16), b = i - j * a.A;
      const uint32_t packed = a.nadj[q + j];
      const int64_t le = int64_t(packed >> 5) - a.elem_start;
      const int32_t m = a.conn[a.conn_off + le * a.A + b];
      f(j, le, int(packed & 31u), b, m);
    }
  };
  // which elements of the chunk have m (an element's nodes are distinct)
  auto mark = [&](int64_t q) {
    nodes(q, [&](int j, int64_t, int, int, int32_t m) {
      if (!FILL && a.shared && !owned(a, m)) a.flags[1] = 1;
      if (m < n) return;
      const int i = place(m);
      if (i >= 0)
        atomicOr(&in[i], 1u << j);
      else
        a.flags[0] = 1;
    });
    __syncwarp();
  };
  auto next = [&](uint16_t* to) {  // ... counted, and cleared for the next chunk
    for (int i = lane; i < T; i += 32) {
      to[i] = uint16_t(to[i] + __popc(in[i]));
      in[i] = 0;
    }
    __syncwarp();
  };
  const bool once = p1 - p0 <= CHUNK;
  for (int64_t q = p0; q < p1; q += CHUNK) {
    mark(q);
    if (!once) next(cnt);
  }
  if (once) {
    for (int i = lane; i < T; i += 32) cnt[i] = uint16_t(__popc(in[i]));
    __syncwarp();
  }
  int slots = 0, entries = 0;
  for (int i0 = 0; i0 < T; i0 += 32) {
    const int i = i0 + lane, c = cnt[i];
    const unsigned mask = __ballot_sync(0xffffffffu, c > 0);
    if (FILL && c > 0) s_pair[warp][slots + __popc(mask & ((1u << lane) - 1u))] = make_int2(key[i], c | i << 16);
    slots += __popc(mask);
    entries += c;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) entries += __shfl_xor_sync(0xffffffffu, entries, o);
  if (!FILL) {
    if (lane == 0) {
      a.nslot[n] = slots;
      a.nlist[n] = entries;
    }
    return;
  }
  __syncwarp();
  // pairs and list entries of the neighbours before each (ascending: rows of a column, and
  // element nodes, are)
  uint16_t* at = s_at[warp];
  for (int e = lane; e < slots; e += 32) {
    const int2 own = s_pair[warp][e];
    int rank = 0, before = 0;
#pragma unroll 4
    for (int j = 0; j < slots; ++j) {
      const int2 o = s_pair[warp][j];
      if (o.x < own.x) {
        ++rank;
        before += o.y & 0xffff;
      }
    }
    s_rank[warp][own.y >> 16] = uint16_t(rank);
    at[own.y >> 16] = uint16_t(before);
  }
  __syncwarp();
  const int np = a.A * (a.A + 1) / 2;
  for (int64_t q = p0; q < p1; q += CHUNK) {
    if (!once) mark(q);
    nodes(q, [&](int j, int64_t le, int la, int lb, int32_t m) {
      const int i = m >= n ? place(m) : -1;
      if (i < 0) return;  // (a full table: the plan is not used)
      const int x = la < lb ? la : lb, y = la < lb ? lb : la;
      const uint32_t first = in[i] & ((1u << j) - 1u);
      const int64_t t = a.list0[n] + at[i] + __popc(first);
      const int64_t block = le * np + x * (2 * a.A - x + 1) / 2 + y - x;
      a.list[t] = uint32_t(block) << 1 | (la > lb ? 1u : 0u);
      if (first == 0 && cnt[i] != 0) {  // the pair's first element (t is its first list entry)
        const int64_t s = a.slot0[n] + s_rank[warp][i];
        a.slots[s] = make_int4(int(n), m, int(uint32_t(t)), 0);
        a.count[s] = uint32_t(cnt[i]) | uint32_t(la) << 16 | uint32_t(lb) << 24;
      }
    });
    __syncwarp();
    if (q + CHUNK < p1) {
      for (int i = lane; i < T; i += 32)
        if (in[i]) cnt[i] = 0;  // its slot is written
      __syncwarp();
      next(at);
    }
  }
}

// The slots of GROUP consecutive nodes by descending list length (a CTA per group).
__global__ void __launch_bounds__(256) order_kernel(int64_t nn, const int64_t* slot0, const int4* in,
                                                    const uint32_t* cin, int4* out, uint32_t* cout) {
  __shared__ int hist[CLASSES];
  const int64_t n0 = int64_t(blockIdx.x) * GROUP, n1 = n0 + GROUP < nn ? n0 + GROUP : nn;
  const int64_t s0 = slot0[n0], s1 = slot0[n1];
  auto cls = [](uint32_t v) {
    const int c = int(v & 0xffffu);
    return c < CLASSES ? CLASSES - 1 - c : 0;
  };
  for (int i = threadIdx.x; i < CLASSES; i += 256) hist[i] = 0;
  __syncthreads();
  for (int64_t s = s0 + threadIdx.x; s < s1; s += 256) atomicAdd(&hist[cls(cin[s])], 1);
  __syncthreads();
  if (threadIdx.x == 0) {
    int sum = 0;
    for (int i = 0; i < CLASSES; ++i) {
      const int h = hist[i];
      hist[i] = sum;
      sum += h;
    }
  }
  __syncthreads();
  for (int64_t s = s0 + threadIdx.x; s < s1; s += 256) {
    const int64_t at = s0 + atomicAdd(&hist[cls(cin[s])], 1);
    out[at] = in[s];
    cout[at] = cin[s];
  }
}

// The row offsets of a slot's m in n's columns and of n in m's, by the pattern at hand: from
// the element map at the pair's first element.
__global__ void __launch_bounds__(256) offsets_kernel(GatherArgs g, int4* slots, const uint32_t* count,
                                                      const uint32_t* list, int64_t nslots, int block) {
  const int64_t s = int64_t(blockIdx.x) * 256 + threadIdx.x;
  if (s >= nslots) return;
  const BlockInfo& B = g.blk[block];
  const int A = B.nnpe;
  const uint32_t c = count[s], la = c >> 16 & 0xffu, lb = c >> 24;
  const uint32_t le = (list[uint32_t(slots[s].z)] >> 1) / uint32_t(A * (A + 1) / 2);
  const uint16_t* ep = g.epos + B.epos_off + int64_t(le) * A * A;
  slots[s].w = int(uint32_t(ep[la * A + lb]) | uint32_t(ep[lb * A + la]) << 16);
}

// Row k of pair slot s per thread (85 slots a CTA); the first nbr CTAs form the residual.
constexpr int SLOTS = 85;
__global__ void __launch_bounds__(256) pair_gather_kernel(GatherArgs g, PairPlan plan, int block, unsigned nbr) {
  if (blockIdx.x < nbr) {
    residual_gather_entry<float2, 3>(g, int64_t(blockIdx.x) * 256 + threadIdx.x);
    return;
  }
  const int sl = int(threadIdx.x) / 3, k = int(threadIdx.x) - 3 * sl;
  const int64_t s = int64_t(blockIdx.x - nbr) * SLOTS + sl;
  if (sl >= SLOTS || s >= plan.nslots) return;
  const int4 r = __ldg(plan.slots + s);
  int left = int(__ldg(plan.count + s) & 0xffffu);
  const uint32_t* lp = plan.list + uint32_t(r.z);
  const unsigned un = g.umask[r.x], um = g.umask[r.y];
  const int64_t cn = g.col_base[r.x], cm = g.col_base[r.y];
  const int Ln = g.col_len[r.x], Lm = g.col_len[r.y];
  const float2* Ke = static_cast<const float2*>(g.Ke) + g.blk[block].ke_off;
  float2 acc[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
  auto add = [&](auto num) {  // the next `num` elements, loads first
    constexpr int N = decltype(num)::value;
    uint32_t at[N];
    float2 v[N][3];
#pragma unroll
    for (int c = 0; c < N; ++c) at[c] = __ldg(lp + c);
#pragma unroll
    for (int c = 0; c < N; ++c) {
      const bool tr = at[c] & 1u;
      const float2* e = Ke + int64_t(at[c] >> 1) * 9 + (tr ? k : 3 * k);
      const int d = tr ? 3 : 1;
#pragma unroll
      for (int i = 0; i < 3; ++i) v[c][i] = __ldg(e + i * d);
    }
#pragma unroll
    for (int c = 0; c < N; ++c)
#pragma unroll
      for (int i = 0; i < 3; ++i) acc[i] = GatherAcc::plus(acc[i], v[c][i]);
    lp += N;
    left -= N;
  };
  while (left >= 4) add(std::integral_constant<int, 4>());
  if (left >= 2) add(std::integral_constant<int, 2>());
  if (left >= 1) add(std::integral_constant<int, 1>());
  if (!((un >> k) & 1u)) return;
  const int kk = __popc(un & ((1u << k) - 1u));
  double* col = g.nzval + cn + int64_t(kk) * Ln + (r.w & 0xffff);
  double* row = g.nzval + cm + int(uint32_t(r.w) >> 16) + kk;
  int ii = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if ((um >> i) & 1u) {
      const double v = GatherAcc::value(acc[i]);
      col[ii] = v;
      if (r.x != r.y) row[int64_t(ii) * Lm] = v;
      ++ii;
    }
}

}  // namespace

static PlanArgs plan_args(const GatherArgs& g, int block, int64_t ne, int* flags) {
  PlanArgs a{};
  const BlockInfo& B = g.blk[block];
  a.nn = g.nn;
  a.elem_start = B.elem_start;
  a.ne = ne;
  a.conn_off = B.conn_off;
  a.A = B.nnpe;
  a.shared = g.nblocks > 1;
  a.nadj_ptr = g.nadj_ptr;
  a.nadj = g.nadj;
  a.conn = g.conn;
  a.flags = flags;
  return a;
}

cudaError_t pair_plan_count(const GatherArgs& g, int block, int64_t ne, int32_t* nslot, int32_t* nlist, int* flags,
                            bool wide, cudaStream_t s) {
  PlanArgs a = plan_args(g, block, ne, flags);
  a.nslot = nslot;
  a.nlist = nlist;
  const unsigned grid = unsigned((g.nn + WPB - 1) / WPB);
  if (wide)
    plan_kernel<false, 512><<<grid, WPB * 32, 0, s>>>(a);
  else
    plan_kernel<false, 128><<<grid, WPB * 32, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t pair_plan_fill(const GatherArgs& g, int block, int64_t ne, const int64_t* slot0, const int64_t* list0,
                           void* unordered, void* slots, uint32_t* count2, uint32_t* count, uint32_t* list, int* flags,
                           bool wide, cudaStream_t s) {
  PlanArgs a = plan_args(g, block, ne, flags);
  a.slot0 = slot0;
  a.list0 = list0;
  a.slots = static_cast<int4*>(unordered);
  a.count = count2;
  a.list = list;
  const unsigned grid = unsigned((g.nn + WPB - 1) / WPB);
  if (wide)
    plan_kernel<true, 512><<<grid, WPB * 32, 0, s>>>(a);
  else
    plan_kernel<true, 128><<<grid, WPB * 32, 0, s>>>(a);
  order_kernel<<<unsigned((g.nn + GROUP - 1) / GROUP), 256, 0, s>>>(g.nn, slot0, a.slots, count2,
                                                                     static_cast<int4*>(slots), count);
  return cudaGetLastError();
}

cudaError_t pair_plan_offsets(const GatherArgs& g, int block, const PairPlan& plan, cudaStream_t s) {
  offsets_kernel<<<unsigned((plan.nslots + 255) / 256), 256, 0, s>>>(g, plan.slots, plan.count, plan.list, plan.nslots,
                                                                     block);
  return cudaGetLastError();
}

cudaError_t launch_pair_gather(const GatherArgs& g, int block, const PairPlan& plan, cudaStream_t s, int* launches) {
  const int64_t nodes = g.nodes ? g.nnodes : g.nn;
  const int64_t nbr = g.R_u ? (nodes * 3 + 255) / 256 : 0, nbk = (plan.nslots + SLOTS - 1) / SLOTS;
  if (nbr + nbk == 0) return cudaSuccess;
  if (nbr + nbk > int64_t(0x7fffffff)) return cudaErrorInvalidValue;
  pair_gather_kernel<<<unsigned(nbr + nbk), 256, 0, s>>>(g, plan, block, unsigned(nbr));
  ++*launches;
  return cudaGetLastError();
}

}  // namespace fec
