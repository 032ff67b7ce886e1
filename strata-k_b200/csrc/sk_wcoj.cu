// sk_wcoj.cu — worst-case-optimal counting joins on a device CSR.
//
// The count aggregate  n(count<X>) :- e(X,Y), e(Y,Z), e(X,Z)  counts the body
// bindings (strata-eval/src/naive.rs:300-391, fold_aggregate Count :391).
// With out(x) the sorted successors of x in the set e, the bindings are
//     Σ_{(X,Y) ∈ e} |out(X) ∩ out(Y)|,
// a leapfrog of two sorted lists per edge.  The reference runs one thread per
// edge with a serial merge over an id-oriented CSR built on the host
// (strata-gpu/src/wcoj.rs:27-43, 99-131).  Here the CSR is built on the device
// (radix sort + run reduction + offsets) and one warp owns a source vertex X:
// it stages out(X) in shared memory, expands the concatenation of out(Y) over
// Y ∈ out(X) with a warp scan so the 32 lanes stream the successor lists with
// coalesced loads, and probes each candidate Z in the staged list.
//
// Graphs with many candidates per edge take the hub-row plan instead
// (k_tri_edges below): vertices are relabelled by descending degree, the part
// of out(x) among the first T labels becomes a T-bit row, and an edge (X, Y)
// is one AND + popcount of two rows plus a short search of the rest.
#include "sk_ops.cuh"
#include "sk_prims.cuh"
#include "sk_rel.cuh"

#include <type_traits>

namespace sk {
namespace {

constexpr int TC_WARPS = 8;
constexpr int TC_NT = TC_WARPS * 32;
constexpr uint32_t TC_STAGE = 1024;  // successor entries staged per warp

__device__ __forceinline__ bool bsearch_u32(const uint32_t* a, uint32_t n, uint32_t x) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo < n && a[lo] == x;
}

__global__ void __launch_bounds__(TC_NT)
    k_tri_count(const uint32_t* __restrict__ off, const uint32_t* __restrict__ nbr, uint64_t n_nodes,
                uint32_t* counter, unsigned long long* total, uint32_t u_lo, uint32_t u_hi) {
  __shared__ uint32_t s_list[TC_WARPS][TC_STAGE];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long count = 0;
  while (true) {
    uint32_t u = 0;
    if (lane == 0) u = u_lo + atomicAdd(counter, 1u);
    u = __shfl_sync(kFull, u, 0);
    if (u >= u_hi || u >= n_nodes) break;
    const uint32_t a0 = off[u], du = off[u + 1] - a0;
    if (du == 0) continue;
    const bool staged = du <= TC_STAGE;
    if (staged) {
      for (uint32_t k = lane; k < du; k += 32) s_list[warp][k] = nbr[a0 + k];
    }
    __syncwarp();
    const uint32_t* A = staged ? s_list[warp] : nbr + a0;
    for (uint32_t c = 0; c < du; c += 32) {
      const uint32_t i = c + lane;
      const bool valid = i < du;
      const uint32_t v = valid ? A[i] : 0u;
      const uint64_t dv = (valid && v < n_nodes) ? (uint64_t)(off[v + 1] - off[v]) : 0ull;
      const uint32_t sv = (valid && v < n_nodes) ? off[v] : 0u;
      const uint64_t incl = warp_incl_sum(dv);
      const uint64_t D = __shfl_sync(kFull, incl, 31);
      for (uint64_t base = 0; base < D; base += 32) {
        const uint64_t j = base + lane;
        const bool ok = j < D;
        // owner lane t = number of lanes whose inclusive prefix is <= j
        int t = 0;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
          const uint64_t val = __shfl_sync(kFull, incl, t + s - 1);
          if (val <= j) t += s;
        }
        const uint64_t ex_t = __shfl_sync(kFull, incl - dv, t & 31);
        const uint32_t sv_t = __shfl_sync(kFull, sv, t & 31);
        if (ok) {
          const uint32_t w = nbr[sv_t + (j - ex_t)];
          if (bsearch_u32(A, du, w)) count++;
        }
      }
    }
    __syncwarp();
  }
  count = warp_sum(count);
  if (lane == 0 && count) atomicAdd(total, count);
}

// Filtered probe (default).  Most candidates Z of a warp's expansion are not
// in out(X): the warp also sets one bit per out(X) entry in a small
// shared-memory bitmap (hash of Z, 16 bits per entry up to 8,192 bits, so a
// non-member passes with probability <= 1 - e^(-1/16) ~ 6 %, a member always),
// answers most candidates with one shared-memory load, and queues the ones
// that pass; whenever 32 are queued the whole warp binary-searches them
// together, so the searches run without idle lanes.  Exact: the bitmap has no
// false negatives and every queued candidate is searched once.
constexpr uint32_t TF_WORDS = 256;  // 8,192-bit filter per warp
constexpr uint32_t TF_MIN = 8;      // out-degree from which the filter pays for its setup

__device__ __forceinline__ uint32_t tf_hash(uint32_t z, int lg) { return (z * 0x85EBCA77u) >> (32 - lg); }

__global__ void __launch_bounds__(TC_NT)
    k_tri_count_filt(const uint32_t* __restrict__ off, const uint32_t* __restrict__ nbr, uint64_t n_nodes,
                     uint32_t* counter, unsigned long long* total, uint32_t u_lo, uint32_t u_hi) {
  __shared__ uint32_t s_list[TC_WARPS][TC_STAGE];
  __shared__ uint32_t s_filt[TC_WARPS][TF_WORDS];
  __shared__ uint32_t s_q[TC_WARPS][64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = lanemask_lt();
  uint32_t* q = s_q[warp];
  uint32_t* F = s_filt[warp];
  unsigned long long count = 0;
  while (true) {
    uint32_t u = 0;
    if (lane == 0) u = u_lo + atomicAdd(counter, 1u);
    u = __shfl_sync(kFull, u, 0);
    if (u >= u_hi || u >= n_nodes) break;
    const uint32_t a0 = off[u], du = off[u + 1] - a0;
    if (du == 0) continue;
    const bool staged = du <= TC_STAGE;
    const bool filt = staged && du >= TF_MIN;
    // filter size: 16 bits per entry, 512 .. 8,192 bits
    int lg = 9;
    while (filt && lg < 13 && (1u << lg) < 16u * du) lg++;
    if (staged) {
      for (uint32_t k = lane; k < du; k += 32) s_list[warp][k] = nbr[a0 + k];
    }
    if (filt) {
      for (uint32_t k = lane; k < (1u << (lg - 5)); k += 32) F[k] = 0u;
      __syncwarp();
      for (uint32_t k = lane; k < du; k += 32) {
        const uint32_t h = tf_hash(s_list[warp][k], lg);
        atomicOr(&F[h >> 5], 1u << (h & 31));
      }
    }
    __syncwarp();
    const uint32_t* A = staged ? s_list[warp] : nbr + a0;
    uint32_t qn = 0;  // queued candidates (uniform)
    for (uint32_t c = 0; c < du; c += 32) {
      const uint32_t i = c + lane;
      const bool valid = i < du;
      const uint32_t v = valid ? A[i] : 0u;
      const uint32_t dv = (valid && v < n_nodes) ? off[v + 1] - off[v] : 0u;
      const uint32_t sv = (valid && v < n_nodes) ? off[v] : 0u;
      const uint32_t incl = warp_incl_sum(dv);
      const uint32_t ex = incl - dv;
      const uint32_t D = __shfl_sync(kFull, incl, 31);
      for (uint32_t base = 0; base < D; base += 32) {
        const uint32_t j = base + lane;
        const bool ok = j < D;
        // owner lane t = number of lanes whose inclusive prefix is <= j
        int t = 0;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
          const uint32_t val = __shfl_sync(kFull, incl, t + s - 1);
          if (val <= j) t += s;
        }
        const uint32_t ex_t = __shfl_sync(kFull, ex, t);
        const uint32_t sv_t = __shfl_sync(kFull, sv, t);
        const uint32_t w = ok ? nbr[sv_t + (j - ex_t)] : 0u;
        if (!filt) {
          if (ok && bsearch_u32(A, du, w)) count++;
          continue;
        }
        const uint32_t h = tf_hash(w, lg);
        const bool pass = ok && ((F[h >> 5] >> (h & 31)) & 1u);
        const unsigned bal = __ballot_sync(kFull, pass);
        if (pass) q[qn + __popc(bal & lt)] = w;
        qn += __popc(bal);
        __syncwarp();
        if (qn >= 32) {
          if (bsearch_u32(A, du, q[lane])) count++;
          __syncwarp();
          if ((uint32_t)lane + 32 < qn) q[lane] = q[lane + 32];
          qn -= 32;
          __syncwarp();
        }
      }
    }
    if (qn > 0 && (uint32_t)lane < qn && bsearch_u32(A, du, q[lane])) count++;
    __syncwarp();
  }
  count = warp_sum(count);
  if (lane == 0 && count) atomicAdd(total, count);
}

// ---- hub rows ----------------------------------------------------------------
// What bounds the probing kernels above is the candidates: Σ_{(X,Y)} |out(Y)|
// is 30 G on R-MAT-22 (450 per edge), each costing about one lane-clock.  Most
// of those candidates are the same few thousand vertices: with labels by
// descending in-degree, the first 8,192 labels hold 97 % of the candidates of
// R-MAT-20.  So out(x) is split at label T:
//   hub part   labels < T: a T-bit row for vertices with more than 32 of them
//              ("dense"), else the sorted list itself (at most one per lane);
//   the rest   labels >= T: the sorted list.
// |out(X) ∩ out(Y)| = hub part + rest, and per edge
//   dense, dense    AND + popcount of the rows, Q = T / 4,096 uint4 a lane,
//                   cut at the shorter row's last label;
//   sparse, dense   one lane per listed label tests its bit of the row;
//   sparse, sparse  every lane compares its label with the other list's;
//   rest            X's list as a hashed bitmap in shared memory (built once
//                   per run of edges of one X), Y's list streamed past it; the
//                   few entries that pass are queued and binary-searched 32
//                   at a time (searching every entry of the shorter list in
//                   the longer one made the kernel 21.4 ms:
//                   its 32 scattered loads a step fill the L1 pipe).
// A warp owns a span of consecutive edges of the sorted edge list, so a vertex of any
// degree is spread over many warps.  Measured on one B200, R-MAT-22 with 16
// edges a node: 12.5 ms
// (dense pairs 4.4, sparse 1.7, rest 6.4) against 95.2 ms of k_tri_count_filt;
// T = 8,192 against 16,384: 12.5 / 14.7 ms (wider rows cost the dense pairs
// more than they save the rest).
constexpr uint32_t kHubNone = 0xffffffffu;
constexpr uint32_t kHubSparse = 32;  // hub labels up to which the list is kept (one per lane)

// Degrees over every step-th row of the raw columns (repeats included: the
// labels only decide how the work is laid out, never the result).  The sample
// is at least two rows per vertex; all 67 M rows of R-MAT-22 took 0.91 ms, most
// of it same-address atomics.  dout may equal din (undirected); self-loops do
// not count there.
__global__ void k_hub_degree(const uint32_t* __restrict__ x, const uint32_t* __restrict__ y, uint64_t n, uint32_t step,
                             uint32_t* din, uint32_t* dout, int undirected) {
  for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * step; i < n;
       i += (uint64_t)gridDim.x * blockDim.x * step) {
    const uint32_t a = x[i], b = y[i];
    if (undirected && a == b) continue;
    atomicAdd(&dout[a], 1u);
    atomicAdd(&din[b], 1u);
  }
}

// out[0] = Σ_v in(v)·out(v), the candidates of the probing plan; out[1] = the
// rows whose Y has at least `heavy` in-edges.
__global__ void k_hub_candidates(const uint32_t* __restrict__ din, const uint32_t* __restrict__ dout, uint64_t n_nodes,
                                 uint32_t heavy, unsigned long long* out) {
  unsigned long long s = 0, h = 0;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n_nodes; v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t d = din[v];
    s += (unsigned long long)d * dout[v];
    h += d >= heavy ? d : 0u;
  }
  s = warp_sum(s);
  h = warp_sum(h);
  if ((threadIdx.x & 31) == 0) {
    if (s) atomicAdd(&out[0], s);
    if (h) atomicAdd(&out[1], h);
  }
}

__global__ void k_hub_sort_keys(const uint32_t* __restrict__ deg, uint64_t n_nodes, uint32_t* __restrict__ keys,
                                uint32_t* __restrict__ ids) {
  const uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n_nodes) return;
  keys[v] = ~deg[v];  // ascending keys = descending degree
  ids[v] = (uint32_t)v;
}

__global__ void k_hub_labels(const uint32_t* __restrict__ order, uint64_t n_nodes, uint32_t* __restrict__ label) {
  const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n_nodes) label[order[r]] = (uint32_t)r;
}

// Labelled edge keys: (label(x) << bits) | label(y) as given, or (undirected)
// from the larger label, the lower degree, to the smaller; self-loops become
// the all-ones key, which no real edge can take and which sorts last.
template <class K>
__global__ void k_hub_pack(const uint32_t* __restrict__ x, const uint32_t* __restrict__ y, uint64_t n,
                           const uint32_t* __restrict__ label, int bits, int undirected, K* __restrict__ keys) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t a = label[x[i]], b = label[y[i]];
  const K sent = (K)((K(1) << bits) - 1);
  if (!undirected) keys[i] = (K)(((K)a << bits) | b);
  else if (a == b) keys[i] = (K)((sent << bits) | sent);
  else keys[i] = a > b ? (K)(((K)a << bits) | b) : (K)(((K)b << bits) | a);
}

// Per vertex {CSR start, degree, hub count | (128-label blocks used << 16), row slot or none}.
__global__ void k_hub_meta(const uint32_t* __restrict__ off, const uint32_t* __restrict__ nbr, uint64_t n_nodes,
                           uint32_t T, uint4* __restrict__ meta, uint32_t* n_dense) {
  const uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  uint4 mt = make_uint4(0u, 0u, 0u, kHubNone);
  bool dense = false;
  if (u < n_nodes) {
    const uint32_t a = off[u], d = off[u + 1] - a;
    uint32_t lo = 0, hi = d;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (nbr[a + mid] < T) lo = mid + 1; else hi = mid;
    }
    dense = lo > kHubSparse;
    mt.x = a;
    mt.y = d;
    mt.z = lo | (lo ? ((nbr[a + lo - 1] >> 7) + 1) << 16 : 0u);
  }
  const unsigned bal = __ballot_sync(kFull, dense);
  uint32_t base = 0;
  if (lane == 0 && bal) base = atomicAdd(n_dense, (uint32_t)__popc(bal));
  base = __shfl_sync(kFull, base, 0);
  if (dense) mt.w = base + __popc(bal & lanemask_lt());
  if (u < n_nodes) meta[u] = mt;
}

// The dense vertices' rows, a warp per `per` vertices, built in shared memory.
template <int Q>
__global__ void __launch_bounds__(TC_NT) k_hub_rows(const uint32_t* __restrict__ nbr, const uint4* __restrict__ meta,
                                                    uint64_t n_nodes, uint32_t per, uint32_t n_rows,
                                                    uint4* __restrict__ rows) {
  __shared__ uint4 s_row[TC_WARPS][Q * 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* w = reinterpret_cast<uint32_t*>(s_row[warp]);
  const uint64_t nw = (uint64_t)gridDim.x * TC_WARPS;
  for (uint64_t g = (uint64_t)blockIdx.x * TC_WARPS + warp; g * per < n_nodes; g += nw) {
    const uint64_t u = g * per + lane;
    const uint4 mine =
        (uint32_t)lane < per && u < n_nodes ? meta[u] : make_uint4(0u, 0u, 0u, kHubNone);
    for (unsigned dm = __ballot_sync(kFull, mine.w < n_rows); dm; dm &= dm - 1) {
      const int t = __ffs(dm) - 1;
      const uint32_t a = __shfl_sync(kFull, mine.x, t), h = __shfl_sync(kFull, mine.z, t) & 0xffffu;
      const uint32_t slot = __shfl_sync(kFull, mine.w, t);
#pragma unroll
      for (int q = 0; q < Q; q++) s_row[warp][q * 32 + lane] = make_uint4(0u, 0u, 0u, 0u);
      __syncwarp();
      for (uint32_t k = lane; k < h; k += 32) {
        const uint32_t z = nbr[a + k];  // < T by the split
        atomicOr(&w[z >> 5], 1u << (z & 31));
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < Q; q++) rows[(uint64_t)slot * (Q * 32) + q * 32 + lane] = s_row[warp][q * 32 + lane];
      __syncwarp();
    }
  }
}

// Σ over the edges (X, Y) of |out(X) ∩ out(Y)|; with `orig`, only X whose
// original id lies in [x_lo, x_hi).
template <class K, int Q>
__global__ void __launch_bounds__(TC_NT, 4)
    k_tri_edges(const K* __restrict__ keys, uint64_t m, int bits, uint32_t span, const uint32_t* __restrict__ nbr,
                const uint4* __restrict__ meta, const uint4* __restrict__ rows, const uint32_t* __restrict__ orig,
                uint32_t x_lo, uint32_t x_hi, unsigned long long* total) {
  __shared__ __align__(16) uint32_t s_filt[TC_WARPS][TF_WORDS];
  __shared__ uint32_t s_q[TC_WARPS][64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = lanemask_lt();
  uint32_t* F = s_filt[warp];
  uint32_t* q = s_q[warp];
  const uint64_t nw = (uint64_t)gridDim.x * TC_WARPS;
  const K mask = (K)((K(1) << bits) - 1);
  const uint32_t* rows32 = reinterpret_cast<const uint32_t*>(rows);
  unsigned long long count = 0;
  uint32_t cur = kHubNone;  // the X whose row is in ra
  uint4 ra[Q];
  uint32_t fx = kHubNone, fn = 0, qn = 0;  // CSR start and length of the filter's list, queued entries
  for (uint64_t g = ((uint64_t)blockIdx.x * TC_NT + threadIdx.x) >> 5; g * span < m; g += nw) {
    const uint64_t e1 = (g + 1) * span < m ? (g + 1) * span : m;
    for (uint64_t e0 = g * span; e0 < e1; e0 += 32) {
      const uint64_t e = e0 + lane;
      uint4 a = make_uint4(0u, 0u, 0u, kHubNone), b = a;
      if (e < e1) {
        const K k = keys[e];
        const uint32_t u = (uint32_t)(k >> bits), v = (uint32_t)(k & mask);
        bool in = true;
        if (orig) {
          const uint32_t o = orig[u];
          in = o >= x_lo && o < x_hi;
        }
        if (in) {
          a = meta[u];
          b = meta[v];
        }
      }
      const uint32_t ha = a.z & 0xffffu, hb = b.z & 0xffffu;
      const bool da = a.w != kHubNone, db = b.w != kHubNone;
      uint32_t c = 0;
      // dense, dense: four rows of the Y side in flight; the X side changes
      // rarely (edges are sorted by X) and stays in registers
      unsigned md = __ballot_sync(kFull, da && db);
      const uint32_t lim = (a.z >> 16) < (b.z >> 16) ? (a.z >> 16) : (b.z >> 16);  // 128-label blocks both can share
      while (md) {
        constexpr int U = 4;
        uint4 rb[U][Q];
        uint32_t sa[U];
#pragma unroll
        for (int j = 0; j < U; j++) {
          const bool live = md != 0;
          const int t = live ? __ffs(md) - 1 : 0;
          md &= md - 1;
          sa[j] = __shfl_sync(kFull, a.w, t);
          const uint32_t sb = __shfl_sync(kFull, b.w, t);
          const uint32_t lm = live ? __shfl_sync(kFull, lim, t) : 0u;
          if (!live) sa[j] = kHubNone;
#pragma unroll
          for (int q = 0; q < Q; q++) {
            rb[j][q] = make_uint4(0u, 0u, 0u, 0u);
            if ((uint32_t)(q * 32 + lane) < lm) rb[j][q] = rows[(uint64_t)sb * (Q * 32) + q * 32 + lane];
          }
        }
#pragma unroll
        for (int j = 0; j < U; j++) {
          if (sa[j] == kHubNone) break;
          if (sa[j] != cur) {
            cur = sa[j];
#pragma unroll
            for (int q = 0; q < Q; q++) ra[q] = rows[(uint64_t)cur * (Q * 32) + q * 32 + lane];
          }
#pragma unroll
          for (int q = 0; q < Q; q++)
            c += __popc(ra[q].x & rb[j][q].x) + __popc(ra[q].y & rb[j][q].y) + __popc(ra[q].z & rb[j][q].z) +
                 __popc(ra[q].w & rb[j][q].w);
        }
      }
      // one side dense: one lane per label of the sparse side's list
      const uint32_t l_off = da ? b.x : a.x, l_h = da ? hb : ha, d_slot = da ? a.w : b.w;
      for (unsigned m1 = __ballot_sync(kFull, da != db && l_h != 0); m1;) {
        constexpr int U = 4;
        uint32_t z[U], sl[U];
        bool on[U];
#pragma unroll
        for (int j = 0; j < U; j++) {
          const bool live = m1 != 0;
          const int t = live ? __ffs(m1) - 1 : 0;
          m1 &= m1 - 1;
          const uint32_t o = __shfl_sync(kFull, l_off, t), h = __shfl_sync(kFull, l_h, t);
          sl[j] = __shfl_sync(kFull, d_slot, t);
          on[j] = live && (uint32_t)lane < h;
          z[j] = on[j] ? nbr[o + lane] : 0u;
        }
#pragma unroll
        for (int j = 0; j < U; j++)
          if (on[j]) c += (rows32[(uint64_t)sl[j] * (Q * 128) + (z[j] >> 5)] >> (z[j] & 31)) & 1u;
      }
      // both sparse: the lists in registers, the shorter one broadcast
      for (unsigned m2 = __ballot_sync(kFull, !da && !db && ha != 0 && hb != 0); m2; m2 &= m2 - 1) {
        const int t = __ffs(m2) - 1;
        const uint32_t oa = __shfl_sync(kFull, a.x, t), na = __shfl_sync(kFull, ha, t);
        const uint32_t ob = __shfl_sync(kFull, b.x, t), nb = __shfl_sync(kFull, hb, t);
        const uint32_t za = (uint32_t)lane < na ? nbr[oa + lane] : kHubNone;
        const uint32_t zb = (uint32_t)lane < nb ? nbr[ob + lane] : kHubNone;
        const uint32_t zl = na > nb ? za : zb, zs = na > nb ? zb : za, ns = na > nb ? nb : na;
        for (uint32_t k = 0; k < ns; k++) c += zl == __shfl_sync(kFull, zs, (int)k) ? 1u : 0u;
      }
      // labels from T on: X's list as a filter, Y's lists streamed past it
      const uint32_t la = a.y - ha, lb = b.y - hb;
      const uint32_t ra0 = a.x + ha, rb0 = b.x + hb;
      for (unsigned m3 = __ballot_sync(kFull, la != 0 && lb != 0); m3;) {
        const int t0 = __ffs(m3) - 1;
        const uint32_t x0 = __shfl_sync(kFull, ra0, t0);
        if (x0 != fx) {  // a new X: finish the queue against the old list, rebuild the filter
          if ((uint32_t)lane < qn && bsearch_u32(nbr + fx, fn, q[lane])) c++;
          qn = 0;
          fx = x0;
          fn = __shfl_sync(kFull, la, t0);
          __syncwarp();
          reinterpret_cast<uint4*>(F)[lane] = make_uint4(0u, 0u, 0u, 0u);
          reinterpret_cast<uint4*>(F)[lane + 32] = make_uint4(0u, 0u, 0u, 0u);
          __syncwarp();
          for (uint32_t k = lane; k < fn; k += 32) {
            const uint32_t z = nbr[fx + k];
            atomicOr(&F[(z >> 5) & (TF_WORDS - 1)], 1u << (z & 31));
          }
          __syncwarp();
        }
        // this X's edges: their lists as one stream of 32-entry pieces, four in flight
        unsigned same = m3 & __ballot_sync(kFull, ra0 == fx);
        m3 &= ~same;
        uint32_t o = 0, n = 0;  // the rest of the list being streamed
        while (n != 0 || same != 0) {
          constexpr int U = 4;
          uint32_t z[U];
          bool ok[U];
#pragma unroll
          for (int j = 0; j < U; j++) {
            if (n == 0 && same != 0) {
              const int t = __ffs(same) - 1;
              same &= same - 1;
              o = __shfl_sync(kFull, rb0, t);
              n = __shfl_sync(kFull, lb, t);
            }
            ok[j] = (uint32_t)lane < n;
            z[j] = ok[j] ? nbr[o + lane] : 0u;
            const uint32_t took = n < 32 ? n : 32;
            o += took;
            n -= took;
          }
#pragma unroll
          for (int j = 0; j < U; j++) {
            const bool pass = ok[j] && ((F[(z[j] >> 5) & (TF_WORDS - 1)] >> (z[j] & 31)) & 1u);
            const unsigned bal = __ballot_sync(kFull, pass);
            if (bal == 0) continue;
            if (pass) q[qn + __popc(bal & lt)] = z[j];
            qn += __popc(bal);
            __syncwarp();
            if (qn >= 32) {
              if (bsearch_u32(nbr + fx, fn, q[lane])) c++;
              __syncwarp();
              if ((uint32_t)lane + 32 < qn) q[lane] = q[lane + 32];
              qn -= 32;
              __syncwarp();
            }
          }
        }
      }
      count += c;
    }
  }
  if ((uint32_t)lane < qn && bsearch_u32(nbr + fx, fn, q[lane])) count++;
  count = warp_sum(count);
  if (lane == 0 && count) atomicAdd(total, count);
}

// Hash-probe variant (STRATA_KNOB_TRI_PROBE = 1; measured slower than the
// binary search on R-MAT-22, which stays the default: the 8 KB table per warp
// cuts residency to 24 warps per SM and the probe loop diverges).  The warp
// builds an open-addressing set of out(X) in
// its shared-memory table (size the next power of two >= 2·d+(X), at most
// TH_TAB, so at least half the slots stay empty and every probe chain ends at
// an empty slot), then streams the successor lists of Y ∈ out(X) exactly as
// above and answers each membership test with ~1-2 table reads instead of a
// ~log2(d+(X))-step binary search.  A vertex whose out-list does not fit
// falls back to the binary search over its list in global memory.
constexpr uint32_t TH_TAB = 2048;
constexpr uint32_t kEmpty = 0xffffffffu;

__device__ __forceinline__ uint32_t tri_hash(uint32_t z, int lg) { return (z * 0x9E3779B1u) >> (32 - lg); }

__global__ void __launch_bounds__(TC_NT)
    k_tri_count_hash(const uint32_t* __restrict__ off, const uint32_t* __restrict__ nbr, uint64_t n_nodes,
                     uint32_t* counter, unsigned long long* total, uint32_t u_lo, uint32_t u_hi) {
  extern __shared__ __align__(16) uint32_t s_tab[];  // TC_WARPS * TH_TAB
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* tab = s_tab + warp * TH_TAB;
  unsigned long long count = 0;
  while (true) {
    uint32_t u = 0;
    if (lane == 0) u = u_lo + atomicAdd(counter, 1u);
    u = __shfl_sync(kFull, u, 0);
    if (u >= u_hi || u >= n_nodes) break;
    const uint32_t a0 = off[u], du = off[u + 1] - a0;
    if (du == 0) continue;
    const bool hashed = du <= TH_TAB / 2;
    int lg = 5;
    while (hashed && (1u << lg) < 2 * du) lg++;
    const uint32_t tmask = (1u << lg) - 1;
    if (hashed) {
      for (uint32_t k = lane; k <= tmask; k += 32) tab[k] = kEmpty;
      __syncwarp();
      for (uint32_t k = lane; k < du; k += 32) {
        const uint32_t z = nbr[a0 + k];
        uint32_t slot = tri_hash(z, lg);
        // at most tmask+1 steps: the table is at most half full
        for (uint32_t step = 0; step <= tmask; step++) {
          const uint32_t prev = atomicCAS(&tab[slot], kEmpty, z);
          if (prev == kEmpty || prev == z) break;
          slot = (slot + 1) & tmask;
        }
      }
      __syncwarp();
    }
    for (uint32_t c = 0; c < du; c += 32) {
      const uint32_t i = c + lane;
      const bool valid = i < du;
      const uint32_t v = valid ? nbr[a0 + i] : 0u;
      const uint32_t dv = (valid && v < n_nodes) ? off[v + 1] - off[v] : 0u;
      const uint32_t sv = (valid && v < n_nodes) ? off[v] : 0u;
      const uint32_t incl = warp_incl_sum(dv);
      const uint32_t ex = incl - dv;
      const uint32_t D = __shfl_sync(kFull, incl, 31);
      for (uint32_t base = 0; base < D; base += 32) {
        const uint32_t j = base + lane;
        int t = 0;
#pragma unroll
        for (int st = 16; st > 0; st >>= 1) {
          const uint32_t val = __shfl_sync(kFull, incl, t + st - 1);
          if (val <= j) t += st;
        }
        const uint32_t ex_t = __shfl_sync(kFull, ex, t);
        const uint32_t sv_t = __shfl_sync(kFull, sv, t);
        if (j < D) {
          const uint32_t w = nbr[sv_t + (j - ex_t)];
          if (hashed) {
            uint32_t slot = tri_hash(w, lg);
            for (uint32_t step = 0; step <= tmask; step++) {
              const uint32_t x = tab[slot];
              if (x == w) { count++; break; }
              if (x == kEmpty) break;
              slot = (slot + 1) & tmask;
            }
          } else if (bsearch_u32(nbr + a0, du, w)) {
            count++;
          }
        }
      }
    }
    __syncwarp();
  }
  count = warp_sum(count);
  if (lane == 0 && count) atomicAdd(total, count);
}

// K4 on a degree-oriented DAG, one warp per lowest-rank vertex u.  A 4-clique
// a < b < c < d (rank order) is counted exactly once, at u = a, v = b, w = c,
// z = d: the warp stages out(u) in shared memory, and for each v ∈ out(u)
// builds the common-successor set C(u,v) = out(u) ∩ out(v) as a sorted list
// in shared memory (the lanes stream out(v) with coalesced loads, probe the
// staged out(u), and a ballot compacts the hits in order).  Then every
// w ∈ C(u,v) expands its out-list with the same warp-cooperative expansion
// as the triangle count (a warp scan over the 32 lanes' degrees, owner lane
// found by a shuffle search) and each entry z is probed in C(u,v).
//   count(u) = Σ_{v ∈ out(u)} Σ_{w ∈ C(u,v)} |out(w) ∩ C(u,v)|.
// A launch handles the vertices whose out-degree lies in (d_lo, d_hi]; `cap`
// (≥ d_hi, a multiple of 32) sizes the two per-warp lists in dynamic shared
// memory: one launch with a small cap and 8 warps per block for the bulk of
// the vertices, one with the largest out-degree as cap for the rest.
__global__ void k_k4_warp(const uint32_t* __restrict__ off, const uint32_t* __restrict__ nbr, uint64_t n_nodes,
                          uint32_t d_lo, uint32_t d_hi, uint32_t cap, uint32_t* counter,
                          unsigned long long* total) {
  extern __shared__ __align__(16) uint32_t s_k4[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* A = s_k4 + (size_t)warp * 2 * cap;  // out(u), staged
  uint32_t* CL = A + cap;                       // C(u, v), sorted
  unsigned long long count = 0;
  while (true) {
    uint32_t u = 0;
    if (lane == 0) u = atomicAdd(counter, 1u);
    u = __shfl_sync(kFull, u, 0);
    if (u >= n_nodes) break;
    const uint32_t a0 = off[u], du = off[u + 1] - a0;
    if (du <= d_lo || du > d_hi || du < 3) continue;
    for (uint32_t k = lane; k < du; k += 32) A[k] = nbr[a0 + k];
    __syncwarp();
    for (uint32_t i = 0; i < du; i++) {  // v = A[i] (lists are in id order, not rank order)
      const uint32_t v = A[i];
      if (v >= n_nodes) continue;
      const uint32_t v0 = off[v], dv = off[v + 1] - v0;
      uint32_t nc = 0;
      for (uint32_t c = 0; c < dv; c += 32) {
        const bool valid = c + lane < dv;
        const uint32_t z = valid ? nbr[v0 + c + lane] : 0u;
        const bool hit = valid && bsearch_u32(A, du, z);
        const unsigned bal = __ballot_sync(kFull, hit);
        const uint32_t pos = nc + __popc(bal & lanemask_lt());
        if (hit && pos < cap) CL[pos] = z;  // distinct successors: nc <= du <= cap
        nc += __popc(bal);
      }
      __syncwarp();
      nc = min(nc, cap);
      if (nc < 2) continue;
      for (uint32_t c = 0; c < nc; c += 32) {
        const bool valid = c + lane < nc;
        const uint32_t w = valid ? CL[c + lane] : 0u;
        const bool inr = valid && w < n_nodes;
        const uint32_t sw = inr ? off[w] : 0u;
        const uint32_t dw = inr ? off[w + 1] - sw : 0u;
        const uint32_t incl = warp_incl_sum(dw);
        const uint32_t ex = incl - dw;
        const uint32_t D = __shfl_sync(kFull, incl, 31);
        for (uint32_t base = 0; base < D; base += 32) {
          const uint32_t j = base + lane;
          int t = 0;
#pragma unroll
          for (int st = 16; st > 0; st >>= 1) {
            const uint32_t val = __shfl_sync(kFull, incl, t + st - 1);
            if (val <= j) t += st;
          }
          const uint32_t ex_t = __shfl_sync(kFull, ex, t);
          const uint32_t sw_t = __shfl_sync(kFull, sw, t);
          if (j < D && bsearch_u32(CL, nc, nbr[sw_t + (j - ex_t)])) count++;
        }
      }
      __syncwarp();
    }
    __syncwarp();
  }
  count = warp_sum(count);
  if (lane == 0 && count) atomicAdd(total, count);
}

__global__ void k_max_outdeg(const uint32_t* __restrict__ off, uint64_t n_nodes, unsigned int* out) {
  unsigned int m = 0;
  for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n_nodes; u += (uint64_t)gridDim.x * blockDim.x)
    m = max(m, off[u + 1] - off[u]);
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(kFull, m, o));
  if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

// Canonical undirected edge key (min << b) | max; self-loops become the key
// (2^b-1, 2^b-1), which no real edge can take and which sorts last.
template <class K>
__global__ void k_canon(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, uint64_t n, int bits,
                        K* __restrict__ keys) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t x = a[i], y = b[i];
  const K lo = x < y ? x : y, hi = x < y ? y : x;
  const K sent = (K)((K(1) << bits) - 1);
  keys[i] = (x == y) ? (K)((sent << bits) | sent) : (K)((lo << bits) | hi);
}

template <class K>
__global__ void k_degree(const K* __restrict__ keys, uint64_t m, int bits, uint32_t* __restrict__ deg) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const K k = keys[i];
  const K mask = (K)((K(1) << bits) - 1);
  atomicAdd(&deg[(uint64_t)(k >> bits)], 1u);
  atomicAdd(&deg[(uint64_t)(k & mask)], 1u);
}

// Orient each undirected edge from lower to higher (degree, id) rank.
template <class K>
__global__ void k_orient(K* __restrict__ keys, uint64_t m, int bits, const uint32_t* __restrict__ deg) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const K k = keys[i];
  const K mask = (K)((K(1) << bits) - 1);
  const K x = k >> bits, y = k & mask;
  const uint32_t dx = deg[(uint64_t)x], dy = deg[(uint64_t)y];
  const bool x_first = dx < dy || (dx == dy && x < y);
  keys[i] = x_first ? (K)((x << bits) | y) : (K)((y << bits) | x);
}

__global__ void k_sum_sq_deg(const uint32_t* __restrict__ off, uint64_t n_nodes, unsigned long long* out) {
  unsigned long long acc = 0;
  for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n_nodes; u += (uint64_t)gridDim.x * blockDim.x) {
    const unsigned long long d = off[u + 1] - off[u];
    acc += d * d;
  }
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd(out, acc);
}

__global__ void k_max_u64(const uint64_t* __restrict__ a, uint64_t n, unsigned long long* out) {
  unsigned long long m = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    m = a[i] > m ? a[i] : m;
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long t = __shfl_xor_sync(kFull, m, o);
    m = t > m ? t : m;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

__global__ void k_intern_map(const uint64_t* __restrict__ keys, uint64_t n, const uint64_t* __restrict__ table,
                             uint64_t m, uint32_t* __restrict__ ids) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  ids[i] = (uint32_t)lower_bound_dev(table, 0, m, keys[i]);
}

inline unsigned blocks(uint64_t n, int nt = 256) { return (unsigned)ceil_div(n ? n : 1, nt); }
inline unsigned grid_of(strata_ctx* ctx, uint64_t n) {  // grid-stride kernels
  return (unsigned)std::min<uint64_t>(blocks(n), (uint64_t)ctx->num_sms * 16);
}

// Σ over oriented edges (u, v) of d+(u) + d+(v): the successor-list entries
// the triangle count streams (its algorithmic bytes; profiling only).
template <class K>
__global__ void k_tri_list_sum(const K* __restrict__ keys, uint64_t m, int bits, const uint32_t* __restrict__ off,
                               uint64_t n_nodes, unsigned long long* out) {
  unsigned long long s = 0;
  const K mask = (K)((K(1) << bits) - 1);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t u = (uint64_t)(keys[i] >> bits), v = (uint64_t)(keys[i] & mask);
    if (u < n_nodes) s += off[u + 1] - off[u];
    if (v < n_nodes) s += off[v + 1] - off[v];
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(out, s);
}

// Sort + dedup packed keys in `keys` (n), result in out (returns count).
// `vary`: the bits in which they may differ (sk_ops.cuh).
template <class K>
uint64_t sort_unique(strata_ctx* ctx, DBuf<K>& keys, uint64_t n, int bits, uint64_t vary, DBuf<K>& out) {
  DBuf<K> alt(ctx, n + 1);
  K* kp = keys.p;
  K* ka = alt.p;
  uint32_t* vp = nullptr;
  uint32_t* va = nullptr;
  radix_sort<K, uint32_t>(ctx, &kp, &ka, &vp, &va, false, n, bits, vary);
  out.reserve(n + 1);
  DBuf<uint64_t> cnt(ctx, 1);
  reduce_runs<K, int32_t, false>(ctx, kp, nullptr, n, out.p, nullptr, cnt.p);
  uint64_t r;
  read_u64(ctx, cnt.p, &r, 1);
  return r;
}

// The count of sorted unique keys without the self-loops' all-ones key, which sorts last.
template <class K>
uint64_t drop_loops(strata_ctx* ctx, const DBuf<K>& keys, uint64_t m, int bits) {
  if (!m) return 0;
  K last;
  SK_CUDA(cudaMemcpyAsync(&last, keys.p + (m - 1), sizeof(K), cudaMemcpyDeviceToHost, ctx->stream));
  SK_CUDA(cudaStreamSynchronize(ctx->stream));
  const K sent = (K)((K(1) << bits) - 1);
  return last == (K)((sent << bits) | sent) ? m - 1 : m;
}

// Count via the warp-per-vertex kernel over a CSR built from sorted unique keys.
template <class K>
uint64_t tri_from_sorted(strata_ctx* ctx, const K* keys, uint64_t m, int bits, uint64_t n_nodes, uint64_t u_lo = 0,
                         uint64_t u_hi = ~0ull) {
  if (u_hi > n_nodes) u_hi = n_nodes;
  if (u_lo >= u_hi) return 0;
  DBuf<uint32_t> off(ctx, n_nodes + 1), nbr(ctx, m + 1);
  build_csr<K>(ctx, keys, m, bits, n_nodes, off.p, nbr.p);
  DBuf<uint64_t> acc(ctx, 3);  // count, vertex counter, list-entry sum
  SK_CUDA(cudaMemsetAsync(acc.p, 0, 24, ctx->stream));
  const unsigned grid = (unsigned)std::min<uint64_t>(ceil_div(n_nodes, TC_WARPS), (uint64_t)ctx->num_sms * 8);
  const int kh = kprof_begin(ctx, K_TRI_COUNT);
  if (ctx->tune_tri_probe == 0 || ctx->tune_tri_probe == 3) {
    k_tri_count_filt<<<grid ? grid : 1, TC_NT, 0, ctx->stream>>>(off.p, nbr.p, n_nodes,
                                                                 reinterpret_cast<uint32_t*>(acc.p + 1),
                                                                 reinterpret_cast<unsigned long long*>(acc.p),
                                                                 (uint32_t)u_lo, (uint32_t)u_hi);
  } else if (ctx->tune_tri_probe == 2) {
    k_tri_count<<<grid ? grid : 1, TC_NT, 0, ctx->stream>>>(off.p, nbr.p, n_nodes,
                                                            reinterpret_cast<uint32_t*>(acc.p + 1),
                                                            reinterpret_cast<unsigned long long*>(acc.p),
                                                            (uint32_t)u_lo, (uint32_t)u_hi);
  } else {
    const size_t smem = (size_t)TC_WARPS * TH_TAB * sizeof(uint32_t);
    SK_CUDA(cudaFuncSetAttribute(k_tri_count_hash, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_tri_count_hash<<<grid ? grid : 1, TC_NT, smem, ctx->stream>>>(off.p, nbr.p, n_nodes,
                                                                     reinterpret_cast<uint32_t*>(acc.p + 1),
                                                                     reinterpret_cast<unsigned long long*>(acc.p),
                                                                     (uint32_t)u_lo, (uint32_t)u_hi);
  }
  // Algorithmic bytes: every out-list once per incident oriented edge plus the
  // edge list and offsets, 4 B·Σ(d+(u)+d+(v)) + 8 B·M + 4 B·(N+1); the sum is
  // counted on the device after the timed launch when profiling.
  kprof_end(ctx, kh, 8 * m + 4 * (n_nodes + 1));
  after_launch(ctx, "k_tri_count");
  if (ctx->profiling && m) {
    k_tri_list_sum<K><<<(unsigned)std::min<uint64_t>(blocks(m), (uint64_t)ctx->num_sms * 8), 256, 0, ctx->stream>>>(
        keys, m, bits, off.p, n_nodes, reinterpret_cast<unsigned long long*>(acc.p + 2));
    after_launch(ctx, "k_tri_list_sum");
  }
  SK_CUDA(cudaMemcpyAsync(ctx->h_scalar, acc.p, 24, cudaMemcpyDeviceToHost, ctx->stream));
  sync_and_check(ctx);
  const uint64_t r = ctx->h_scalar[0];
  if (ctx->profiling) kprof_add_last(ctx, K_TRI_COUNT, 4 * ctx->h_scalar[2]);
  kprof_collect(ctx);
  return r;
}

// ---- hub-row plan, host side ---------------------------------------------------
// Where the plan applies (one B200, us a call, hub rows against probing):
//   pattern   172 k edges with 53 candidates each 353 / 373, 259 k with 40
//             374 / 319, 1 M with 62 559 / 656, 4.2 M with 95 1,192 / 2,211,
//             67 M with 450 18,900 / 101,000
//   both      without skew the labels beyond the rows dominate: uniform graphs
//             of 4.2 M edges with 11 candidates 1,057 / 674, 12.6 M with 32
//             3,236 / 2,167
//   undirected  the labels also save a sort: 15 k edges 327 / 303, 40 k 343 /
//             365, 172 k 470 / 624, 4.2 M 4,797 / 6,468
// so: from 2^18 directed and 2^15 undirected edges on, with at least 48
// candidates an edge (directed), and with the rows covering the columns: few
// enough vertices, or a quarter of the edges ending in vertices of at least
// eight times the mean in-degree.
constexpr uint64_t kHubMinDirected = 1ull << 18, kHubMinUndirected = 1ull << 15;
constexpr uint64_t kHubMinCandidates = 48;
// Undirected graphs without skew take the labels for the sort they save (one
// of the edges instead of two) while the sort of the ids costs less: up to
// eight ids an edge.  Uniform graphs of 600 k edges over as many vertices, us a
// call, labels / none: 0.6 M ids 1,280 / 1,363, 4.8 M 4,167 / 4,201, 9.6 M
// 7,469 / 7,414; 4 M edges, 32 M ids 26,309 / 26,041, 100 M 73,298 / 71,894.
// With skew the rows pay at any width (40 k edges over 10^8 ids 4,771 / 65,681).
constexpr uint64_t kHubSortIds = 8;
constexpr uint64_t kHubMaxNodes = 1ull << 27;  // above, the per-vertex tables outgrow their use

// Device bytes the plan needs beside the edge keys (an upper bound on the rows).
inline uint64_t hub_bytes(uint64_t n, uint64_t n_nodes, int q) {
  return n_nodes * (6 * 4 + 16) + (n / (kHubSparse + 1) + 1) * (uint64_t)q * 512 + (1ull << 20);
}

// Stride of the degree sample.
inline uint32_t hub_step(uint64_t n, uint64_t n_nodes) {
  return (uint32_t)std::max<uint64_t>(1, n / std::max<uint64_t>(1ull << 17, 2 * n_nodes));
}

inline int hub_q(uint64_t n_nodes) { return n_nodes <= 4096 ? 1 : 2; }

// The plan applies: default probe, sizes in range, and its memory within the
// context's cap.  Without a cap the device may still be too full for it: then
// its first allocation to fail ends it and the edges are probed instead.
inline bool hub_fits(strata_ctx* ctx, uint64_t n, uint64_t n_min, uint64_t n_nodes, size_t key_bytes) {
  if (ctx->tune_tri_probe != 0 || n < n_min || n_nodes > kHubMaxNodes) return false;
  return !ctx->cap || ctx->in_use + n * (3 * key_bytes + 4) + hub_bytes(n, n_nodes, hub_q(n_nodes)) <= ctx->cap;
}

// Sampled degrees (step rows apart) and what they say of the graph: candidates
// and heavy rows as k_hub_candidates counts them.
struct HubSample {
  uint32_t step;
  uint64_t rows, candidates, heavy;
  bool covered(uint64_t n_nodes) const { return n_nodes <= hub_q(n_nodes) * 4096ull || heavy * 4 >= rows; }
};
HubSample hub_sample(strata_ctx* ctx, const uint32_t* x, const uint32_t* y, uint64_t n, uint64_t n_nodes,
                     bool undirected, DBuf<uint32_t>& deg) {
  // din, then dout (directed), then the two sums
  const uint64_t half = (n_nodes + 3) & ~3ull, words = half * (undirected ? 1 : 2);
  deg.reserve(words + 4);
  SK_CUDA(cudaMemsetAsync(deg.p, 0, (words + 4) * 4, ctx->stream));
  uint32_t* din = deg.p;
  uint32_t* dout = undirected ? deg.p : deg.p + half;
  auto* sums = reinterpret_cast<unsigned long long*>(deg.p + words);
  HubSample r{hub_step(n, n_nodes), 0, 0, 0};
  r.rows = ceil_div(n, r.step);
  k_hub_degree<<<grid_of(ctx, r.rows), 256, 0, ctx->stream>>>(x, y, n, r.step, din, dout, undirected ? 1 : 0);
  after_launch(ctx, "k_hub_degree");
  const uint64_t ends = undirected ? 2 * r.rows : r.rows;
  k_hub_candidates<<<grid_of(ctx, n_nodes), 256, 0, ctx->stream>>>(
      din, dout, n_nodes, (uint32_t)std::min<uint64_t>(8 * ceil_div(ends, n_nodes), 0xffffffffull), sums);
  after_launch(ctx, "k_hub_candidates");
  uint64_t h[2];
  read_u64(ctx, reinterpret_cast<const uint64_t*>(sums), h, 2);
  r.candidates = h[0];
  r.heavy = undirected ? h[1] / 2 : h[1];
  return r;
}

// Labels by descending degree: label[v], and (optional) order[label] = v.
void hub_labels(strata_ctx* ctx, const uint32_t* deg, uint64_t n_nodes, DBuf<uint32_t>& label, DBuf<uint32_t>* order) {
  DBuf<uint32_t> k(ctx, n_nodes), ka(ctx, n_nodes), id(ctx, n_nodes), ia(ctx, n_nodes);
  k_hub_sort_keys<<<blocks(n_nodes), 256, 0, ctx->stream>>>(deg, n_nodes, k.p, id.p);
  after_launch(ctx, "k_hub_sort_keys");
  uint32_t *kp = k.p, *kalt = ka.p, *vp = id.p, *valt = ia.p;
  radix_sort<uint32_t, uint32_t>(ctx, &kp, &kalt, &vp, &valt, true, n_nodes, 32, kSortLook);
  label.reserve(n_nodes);
  k_hub_labels<<<blocks(n_nodes), 256, 0, ctx->stream>>>(vp, n_nodes, label.p);
  after_launch(ctx, "k_hub_labels");
  if (order) *order = vp == id.p ? std::move(id) : std::move(ia);
}

// Count over sorted unique labelled keys.
template <class K>
uint64_t hub_count(strata_ctx* ctx, const K* keys, uint64_t m, int bits, uint64_t n_nodes, const uint32_t* orig,
                   uint32_t x_lo, uint32_t x_hi) {
  DBuf<uint32_t> off(ctx, n_nodes + 1), nbr(ctx, m + 1);
  build_csr<K>(ctx, keys, m, bits, n_nodes, off.p, nbr.p);
  DBuf<uint64_t> acc(ctx, 2);  // count, dense vertices
  SK_CUDA(cudaMemsetAsync(acc.p, 0, 16, ctx->stream));
  DBuf<uint4> meta(ctx, n_nodes);
  const int q = hub_q(n_nodes);
  k_hub_meta<<<blocks(n_nodes), 256, 0, ctx->stream>>>(off.p, nbr.p, n_nodes, (uint32_t)q * 4096u, meta.p,
                                                       reinterpret_cast<uint32_t*>(acc.p + 1));
  after_launch(ctx, "k_hub_meta");
  uint64_t nd = 0;
  read_u64(ctx, acc.p + 1, &nd, 1);
  DBuf<uint4> rows(ctx, nd * (uint64_t)q * 32 + 1);
  auto run = [&](auto qt) {
    constexpr int Q = decltype(qt)::value;
    if (nd) {
      // few vertices a warp while the grid is not full, else a lane each
      const uint32_t per = n_nodes >= (uint64_t)ctx->num_sms * 8 * TC_NT ? 32 : 2;
      const unsigned rg = (unsigned)std::min<uint64_t>(ceil_div(n_nodes, per * TC_WARPS), (uint64_t)ctx->num_sms * 8);
      k_hub_rows<Q><<<rg, TC_NT, 0, ctx->stream>>>(nbr.p, meta.p, n_nodes, per, (uint32_t)nd, rows.p);
      after_launch(ctx, "k_hub_rows");
    }
    // consecutive edges a warp takes at a time: as many as leave eight turns per resident warp
    const uint64_t warps = (uint64_t)ctx->num_sms * 4 * TC_WARPS;
    const uint32_t span = 32 * (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(16, m / (warps * 32 * 8)));
    const unsigned g = (unsigned)std::min<uint64_t>(ceil_div(m, (uint64_t)span * TC_WARPS), (uint64_t)ctx->num_sms * 4);
    const int kh = kprof_begin(ctx, K_TRI_COUNT);
    k_tri_edges<K, Q><<<g, TC_NT, 0, ctx->stream>>>(keys, m, bits, span, nbr.p, meta.p, rows.p, orig, x_lo, x_hi,
                                                    reinterpret_cast<unsigned long long*>(acc.p));
    kprof_end(ctx, kh, m * sizeof(K) + n_nodes * 16 + nd * (uint64_t)Q * 512 + 4 * m);  // keys, meta, rows, lists once
    after_launch(ctx, "k_tri_edges");
  };
  if (q == 1) run(std::integral_constant<int, 1>{});
  else run(std::integral_constant<int, 2>{});
  SK_CUDA(cudaMemcpyAsync(ctx->h_scalar, acc.p, 8, cudaMemcpyDeviceToHost, ctx->stream));
  sync_and_check(ctx);
  const uint64_t r = ctx->h_scalar[0];
  kprof_collect(ctx);
  return r;
}

// The ids of two edge columns: bits of the largest, one past it, and the bits
// in which the packed keys may differ.
struct Ids {
  int bits;
  uint64_t n_nodes;
  uint32_t vx, vy;    // bits in which the ids of a column differ
  uint32_t any, hole; // of both columns together; the bits not set in all of them
  bool loops;
  uint64_t pattern() const { return (uint64_t)vx << bits | vy; }
  // either column's id in either half; a self-loop's key is all ones
  uint64_t undirected(bool with_loops) const {
    const uint64_t v = with_loops && loops ? hole & ((1ull << bits) - 1) : any;
    return v << bits | v;
  }
};

Ids id_space(strata_ctx* ctx, const uint32_t* a, const uint32_t* b, uint64_t n) {
  const ColScan c = col_scan(ctx, a, b, n);
  const uint32_t m = std::max(c.a.max, c.b.max);
  const uint32_t hole = c.a.none | c.b.none;
  return Ids{std::max(1, bits_for(m)), (uint64_t)m + 1, c.a.vary(), c.b.vary(), (c.a.some | c.b.some) & hole, hole,
             c.loops};
}

template <class K>
uint64_t pattern_impl(strata_ctx* ctx, const uint32_t* x, const uint32_t* y, uint64_t n, const Ids& I,
                      uint64_t u_lo = 0, uint64_t u_hi = ~0ull) {
  const int b = I.bits;
  const uint64_t n_nodes = I.n_nodes;
  if (u_hi > n_nodes) u_hi = n_nodes;
  if (u_lo >= u_hi) return 0;
  DBuf<K> keys(ctx, n + 1), uniq;
  uniq.ctx = ctx;
  if (hub_fits(ctx, n, kHubMinDirected, n_nodes, sizeof(K))) {
    bool counted = false;
    uint64_t r = 0;
    const bool had = with_memory([&] {
      DBuf<uint32_t> deg;
      deg.ctx = ctx;
      const HubSample hs = hub_sample(ctx, x, y, n, n_nodes, false, deg);
      const double cand = (double)hs.candidates * hs.step * hs.step;
      if (cand < (double)kHubMinCandidates * (double)n || !hs.covered(n_nodes)) return;
      const bool whole = u_lo == 0 && u_hi == n_nodes;
      DBuf<uint32_t> label, order;
      label.ctx = order.ctx = ctx;
      hub_labels(ctx, deg.p, n_nodes, label, whole ? nullptr : &order);
      k_hub_pack<K><<<blocks(n), 256, 0, ctx->stream>>>(x, y, n, label.p, b, 0, keys.p);
      after_launch(ctx, "k_hub_pack");
      const uint64_t m = sort_unique<K>(ctx, keys, n, 2 * b, kSortAll, uniq);
      r = hub_count<K>(ctx, uniq.p, m, b, n_nodes, whole ? nullptr : order.p, (uint32_t)u_lo, (uint32_t)u_hi);
      counted = true;
    });
    if (had && counted) return r;
    uniq.release();
  }
  pack_pairs<K, int32_t, false>(ctx, x, y, nullptr, nullptr, n, b, keys.p, nullptr);
  const uint64_t m = sort_unique<K>(ctx, keys, n, 2 * b, I.pattern(), uniq);
  return tri_from_sorted<K>(ctx, uniq.p, m, b, n_nodes, u_lo, u_hi);
}

// Canonicalize, dedup, drop self-loops, orient by (degree, id).  Leaves the
// oriented sorted keys in `out` and returns their count.
template <class K>
uint64_t oriented_edges(strata_ctx* ctx, const uint32_t* a, const uint32_t* b, uint64_t n, const Ids& I,
                        bool by_degree, DBuf<K>& out) {
  const int bits = I.bits;
  const uint64_t n_nodes = I.n_nodes;
  DBuf<K> keys(ctx, n + 1), uniq;
  uniq.ctx = ctx;
  k_canon<K><<<blocks(n), 256, 0, ctx->stream>>>(a, b, n, bits, keys.p);
  after_launch(ctx, "k_canon");
  const uint64_t m = drop_loops<K>(ctx, uniq, sort_unique<K>(ctx, keys, n, 2 * bits, I.undirected(true), uniq), bits);
  if (!by_degree || m == 0) {
    out = std::move(uniq);
    return m;
  }
  DBuf<uint32_t> deg(ctx, n_nodes + 1);
  SK_CUDA(cudaMemsetAsync(deg.p, 0, (n_nodes + 1) * 4, ctx->stream));
  k_degree<K><<<blocks(m), 256, 0, ctx->stream>>>(uniq.p, m, bits, deg.p);
  after_launch(ctx, "k_degree");
  k_orient<K><<<blocks(m), 256, 0, ctx->stream>>>(uniq.p, m, bits, deg.p);
  after_launch(ctx, "k_orient");
  DBuf<K> alt(ctx, m + 1);
  K* kp = uniq.p;
  K* ka = alt.p;
  uint32_t* vp = nullptr;
  uint32_t* va = nullptr;
  radix_sort<K, uint32_t>(ctx, &kp, &ka, &vp, &va, false, m, 2 * bits, I.undirected(false));
  if (kp == uniq.p) out = std::move(uniq);
  else out = std::move(alt);
  return m;
}

template <class K>
uint64_t tri_undirected_impl(strata_ctx* ctx, const uint32_t* a, const uint32_t* b, uint64_t n, const Ids& I) {
  const int bits = I.bits;
  const uint64_t n_nodes = I.n_nodes;
  DBuf<K> ori;
  ori.ctx = ctx;
  if (hub_fits(ctx, n, kHubMinUndirected, n_nodes, sizeof(K))) {
    // Any total order of the vertices counts each triangle of the simple
    // graph once; the labels are one, so a single sort orients and dedups.
    bool counted = false;
    uint64_t r = 0;
    const bool had = with_memory([&] {
      DBuf<uint32_t> deg, label;
      deg.ctx = label.ctx = ctx;
      const HubSample hs = hub_sample(ctx, a, b, n, n_nodes, true, deg);
      if (!hs.covered(n_nodes) && n_nodes > kHubSortIds * n) return;
      counted = true;
      hub_labels(ctx, deg.p, n_nodes, label, nullptr);
      DBuf<K> keys(ctx, n + 1);
      k_hub_pack<K><<<blocks(n), 256, 0, ctx->stream>>>(a, b, n, label.p, bits, 1, keys.p);
      after_launch(ctx, "k_hub_pack");
      const uint64_t m = drop_loops<K>(ctx, ori, sort_unique<K>(ctx, keys, n, 2 * bits, kSortAll, ori), bits);
      if (m == 0) return;
      r = hs.covered(n_nodes) ? hub_count<K>(ctx, ori.p, m, bits, n_nodes, nullptr, 0, 0)
                              : tri_from_sorted<K>(ctx, ori.p, m, bits, n_nodes);
    });
    if (had && counted) return r;
    ori.release();
  }
  const uint64_t m = oriented_edges<K>(ctx, a, b, n, I, true, ori);
  if (m == 0) return 0;
  return tri_from_sorted<K>(ctx, ori.p, m, bits, n_nodes);
}

template <class K>
uint64_t k4_impl(strata_ctx* ctx, const uint32_t* a, const uint32_t* b, uint64_t n, const Ids& I) {
  const int bits = I.bits;
  const uint64_t n_nodes = I.n_nodes;
  DBuf<K> ori;
  ori.ctx = ctx;
  const uint64_t m = oriented_edges<K>(ctx, a, b, n, I, true, ori);
  if (m == 0) return 0;
  DBuf<uint32_t> off(ctx, n_nodes + 1), nbr(ctx, m + 1);
  build_csr<K>(ctx, ori.p, m, bits, n_nodes, off.p, nbr.p);
  DBuf<uint64_t> acc(ctx, 3);  // count, two vertex counters, largest out-degree
  SK_CUDA(cudaMemsetAsync(acc.p, 0, 24, ctx->stream));
  unsigned int* maxdeg = reinterpret_cast<unsigned int*>(acc.p + 2);
  k_max_outdeg<<<(unsigned)std::min<uint64_t>(blocks(n_nodes), (uint64_t)ctx->num_sms * 8), 256, 0, ctx->stream>>>(
      off.p, n_nodes, maxdeg);
  after_launch(ctx, "k_max_outdeg");
  uint64_t md;
  read_u64(ctx, acc.p + 2, &md, 1);
  md &= 0xffffffffull;
  // Shared memory of one warp: two lists of `cap` ids.
  constexpr uint32_t kSmallCap = 512;
  constexpr size_t kSmemLimit = 200 * 1024;
  const uint32_t big_cap = (uint32_t)ceil_div(std::max<uint64_t>(md, 1), 32) * 32;
  if ((size_t)big_cap * 8 > kSmemLimit)
    fail(STRATA_E_UNSUPPORTED, "4-clique count: an oriented out-degree above 25,600 does not fit shared memory");
  const uint64_t grid_cap = (uint64_t)ctx->num_sms * 8;
  auto launch = [&](uint32_t d_lo, uint32_t d_hi, uint32_t cap, int warps, uint32_t* counter) {
    const size_t smem = (size_t)warps * 2 * cap * 4;
    allow_smem(k_k4_warp, kSmemLimit);
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(n_nodes, warps), grid_cap));
    k_k4_warp<<<grid, warps * 32, smem, ctx->stream>>>(off.p, nbr.p, n_nodes, d_lo, d_hi, cap, counter,
                                                       reinterpret_cast<unsigned long long*>(acc.p));
    after_launch(ctx, "k_k4_warp");
  };
  uint32_t* counters = reinterpret_cast<uint32_t*>(acc.p + 1);
  launch(0, kSmallCap, kSmallCap, 8, counters);
  if (md > kSmallCap) {
    const int warps = (int)std::max<size_t>(1, std::min<size_t>(8, kSmemLimit / ((size_t)big_cap * 8)));
    launch(kSmallCap, (uint32_t)md, big_cap, warps, counters + 1);
  }
  SK_CUDA(cudaMemcpyAsync(ctx->h_scalar, acc.p, 8, cudaMemcpyDeviceToHost, ctx->stream));
  sync_and_check(ctx);
  return ctx->h_scalar[0];
}

template <class K>
uint64_t bpi_impl(strata_ctx* ctx, const uint32_t* a, const uint32_t* b, uint64_t n, const Ids& I) {
  const int bits = I.bits;
  const uint64_t n_nodes = I.n_nodes;
  DBuf<K> ori;
  ori.ctx = ctx;
  const uint64_t m = oriented_edges<K>(ctx, a, b, n, I, false, ori);
  if (m == 0) return 0;
  DBuf<uint32_t> off(ctx, n_nodes + 1), nbr(ctx, m + 1);
  build_csr<K>(ctx, ori.p, m, bits, n_nodes, off.p, nbr.p);
  DBuf<uint64_t> acc(ctx, 1);
  SK_CUDA(cudaMemsetAsync(acc.p, 0, 8, ctx->stream));
  k_sum_sq_deg<<<blocks(n_nodes), 256, 0, ctx->stream>>>(off.p, n_nodes, reinterpret_cast<unsigned long long*>(acc.p));
  after_launch(ctx, "k_sum_sq_deg");
  uint64_t r;
  read_u64(ctx, acc.p, &r, 1);
  return r;
}

}  // namespace

uint64_t count_triangle_pattern(strata_ctx* ctx, const uint32_t* x, const uint32_t* y, uint64_t n) {
  reset_status(ctx);
  if (n == 0) return 0;
  const Ids I = id_space(ctx, x, y, n);
  if (2 * I.bits <= 32) return pattern_impl<uint32_t>(ctx, x, y, n, I);
  return pattern_impl<uint64_t>(ctx, x, y, n, I);
}

uint64_t count_triangle_pattern_range(strata_ctx* ctx, const uint32_t* x, const uint32_t* y, uint64_t n,
                                      uint64_t u_lo, uint64_t u_hi) {
  reset_status(ctx);
  if (n == 0 || u_lo >= u_hi) return 0;
  const Ids I = id_space(ctx, x, y, n);
  if (2 * I.bits <= 32) return pattern_impl<uint32_t>(ctx, x, y, n, I, u_lo, u_hi);
  return pattern_impl<uint64_t>(ctx, x, y, n, I, u_lo, u_hi);
}

uint64_t count_triangles_undirected(strata_ctx* ctx, const uint32_t* a, const uint32_t* b, uint64_t n) {
  reset_status(ctx);
  if (n == 0) return 0;
  const Ids I = id_space(ctx, a, b, n);
  if (2 * I.bits <= 32) return tri_undirected_impl<uint32_t>(ctx, a, b, n, I);
  return tri_undirected_impl<uint64_t>(ctx, a, b, n, I);
}

uint64_t count_4cliques_undirected(strata_ctx* ctx, const uint32_t* a, const uint32_t* b, uint64_t n) {
  reset_status(ctx);
  if (n == 0) return 0;
  const Ids I = id_space(ctx, a, b, n);
  if (2 * I.bits <= 32) return k4_impl<uint32_t>(ctx, a, b, n, I);
  return k4_impl<uint64_t>(ctx, a, b, n, I);
}

uint64_t binary_plan_intermediate(strata_ctx* ctx, const uint32_t* a, const uint32_t* b, uint64_t n) {
  reset_status(ctx);
  if (n == 0) return 0;
  const Ids I = id_space(ctx, a, b, n);
  if (2 * I.bits <= 32) return bpi_impl<uint32_t>(ctx, a, b, n, I);
  return bpi_impl<uint64_t>(ctx, a, b, n, I);
}

uint64_t intern_terms(strata_ctx* ctx, const uint64_t* keys, uint64_t n, uint32_t* ids) {
  reset_status(ctx);
  if (n == 0) return 0;
  DBuf<uint64_t> mx(ctx, 1);
  SK_CUDA(cudaMemsetAsync(mx.p, 0, 8, ctx->stream));
  k_max_u64<<<(unsigned)std::min<uint64_t>(ceil_div(n, 256), (uint64_t)ctx->num_sms * 8), 256, 0, ctx->stream>>>(
      keys, n, reinterpret_cast<unsigned long long*>(mx.p));
  after_launch(ctx, "k_max_u64");
  uint64_t maxk;
  read_u64(ctx, mx.p, &maxk, 1);
  DBuf<uint64_t> copy(ctx, n + 1), table;
  table.ctx = ctx;
  SK_CUDA(cudaMemcpyAsync(copy.p, keys, n * 8, cudaMemcpyDeviceToDevice, ctx->stream));
  const uint64_t m = sort_unique<uint64_t>(ctx, copy, n, std::max(1, bits_for(maxk)), kSortLook, table);
  k_intern_map<<<blocks(n), 256, 0, ctx->stream>>>(keys, n, table.p, m, ids);
  after_launch(ctx, "k_intern_map");
  sync_and_check(ctx);
  return m;
}

}  // namespace sk
