// sk_bitset.cu — bit-parallel semi-naive transitive closure, one instance or
// a batch of independent instances.
//
// The program is   path(X,Y) :- edge(X,Y).   path(X,Z) :- edge(X,Y), path(Y,Z).
// evaluated semi-naively exactly as the interpreter does
// (strata-eval/src/seminaive.rs:29-106, 192-209): the bootstrap round derives
// Δ0 = edge, then every round derives
//     Δ'(X, ·) = ( ∪_{Y ∈ out(X)} Δ(Y, ·) ) ∖ path(X, ·),   path ∪= Δ'
// until Δ' is empty.  Here each relation row is a bit row over the Z domain,
// so one OR of a 128-bit word joins 128 Δ tuples at once, the AND-NOT is the
// dedup and Δ-difference, and the popcount of the new bits is |Δ'|.  Rounds,
// Δ sets and the final relation are those of the tuple plans.
//
// Layout (per instance i): rows X ∈ [0, n_rows), each row W4 = ceil(n_cols /
// 128) uint4 words; three matrices (path F, Δ and Δ' double-buffered), an
// out-edge CSR with local ids, and for Δ and Δ' a summary: per row and block of
// 32 words a mask of its nonzero words, stored block by block
// (sum_base + block * n_rows + row).  A Δ word is read only where its summary
// bit is set, so zero words are neither written nor cleared between rounds.
// All instances of a wave share one pool; instance i starts at vec_base[i]
// and row_base[i].
//
// Work split.  Rows of at most 16 words share a warp (L = next power of two
// >= W4 lanes per row, a unit is 32 / L rows).  Wider rows are cut into
// blocks of 32 words, one uint4 a lane: a unit is one warp over one block of
// a strip of up to 16 rows, the blocks outermost.  So at any time the resident
// warps read one or two blocks of Δ (26 MB each at 50,000 nodes), which stay
// in L2 for all the rows that join them, and one unit's metadata, CSR
// offsets, neighbour ids and summaries are read once for its strip.
// Per round one persistent kernel strides its warps over the units of all
// active instances of the wave; its last block does the bookkeeping (the unit
// prefix over active instances), and the host replays a captured CUDA graph of
// R rounds until no instance is active — one launch per semi-naive round for
// the whole batch, no host round trip inside the graph.  A single closure
// launches its rounds directly (instantiating a graph costs more than it
// saves there).
//
// What bounds the round: the latency of the Δ loads and, at 40 % of the issue
// slots, the instructions around them (DRAM at 50 %); the word summaries and
// blocks took the DRAM bytes of a dense round at 50,000 nodes and 5 edges a
// node from about 2.6 to 1.6 GB, reading the strip's edges as one list (eight
// Δ words and the ending rows' path words in flight) the rest.  Measured on
// one B200 against the form with a byte flag per row and whole rows per warp:
// that closure 6.7 -> 4.5 ms, 192 ER instances of up to 50,000 nodes (rounds
// alone) 88.4 -> 70.3 ms.  Three blocks an SM of up to 85 registers: four of
// 64 spill and lose 5 %, six with four words in flight 12 %.
//
// Summary per instance: |path| and  fp = Σ_{(X,Z) ∈ path} mix64(X) · c^Z
// (mod 2^64, c = 0x9E3779B97F4A7C15), computed from the bit rows one 32-bit
// word at a time with byte tables.
#include "sk_ops.cuh"
#include "sk_prims.cuh"
#include "sk_rel.cuh"

#include <algorithm>
#include <cstring>
#include <vector>

namespace sk {
namespace {

constexpr int BS_NT = 256;
constexpr uint64_t kPolyC = 0x9e3779b97f4a7c15ull;

// Device view of a wave (all pointers into fixed buffers of the call).
struct BsView {
  // per instance of the wave
  const uint32_t* n_rows;
  const uint32_t* n_cols;
  const uint32_t* w4;
  const uint32_t* rpu;    // rows per unit
  const uint8_t* lshift;  // log2(lanes per row)
  const uint64_t* row_base;
  const uint64_t* vec_base;
  const uint64_t* sum_base;
  const uint64_t* eoff;   // first edge in wave order (n + 1)
  const uint64_t* ebase;  // first edge in the input columns
  const uint64_t* fprefix;  // units of the summary kernel (n + 1)
  uint64_t* delta;   // |Δ'| of the current round
  uint64_t* total;   // |path| so far
  uint64_t* counts;  // summary kernel's |path| and fingerprint
  uint64_t* fps;
  uint32_t* rounds;
  uint8_t* active;
  // active list and unit prefix (rebuilt by bs_book)
  uint32_t* act;
  uint64_t* uprefix;
  uint32_t* n_act;   // [0] active instances, [1] an edge endpoint was out of range
  uint64_t* u_total;
  uint32_t* ticket;  // blocks of the running round that are done
  uint32_t n_inst;
  // CSR over global rows, local neighbour ids
  const uint64_t* off;
  const uint32_t* nbr;
  // matrices and summaries
  uint4* F;
  uint4* D0;
  uint4* D1;
  uint32_t* s0;
  uint32_t* s1;
  unsigned long long* bytes;  // algorithmic bytes of the rounds (profiling), or null
};

__device__ __forceinline__ uint32_t popc4(const uint4& a) {
  return __popc(a.x) + __popc(a.y) + __popc(a.z) + __popc(a.w);
}
__device__ __forceinline__ bool any4(const uint4& a) { return (a.x | a.y | a.z | a.w) != 0u; }
__device__ __forceinline__ void or4(uint4& a, const uint4& d) {
  a.x |= d.x;
  a.y |= d.y;
  a.z |= d.z;
  a.w |= d.w;
}

// Slot k of unit u in [lo, n): uprefix[k] <= u < uprefix[k + 1].
__device__ __forceinline__ uint32_t unit_owner(const uint64_t* uprefix, uint32_t lo, uint32_t n, uint64_t u) {
  uint32_t hi = n;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (uprefix[mid] <= u) lo = mid; else hi = mid;
  }
  return lo;
}

// After a round (or the bootstrap): close finished instances, add |Δ'| to
// |path|, rebuild the active list and its unit prefix.  One block.
__device__ void bs_book(const BsView& v, int count_round) {
  __shared__ uint64_t s_scan[BS_NT / 32 + 1];
  __shared__ uint64_t s_carry[2];
  if (threadIdx.x == 0) s_carry[0] = s_carry[1] = 0;
  __syncthreads();
  for (uint32_t base = 0; base < v.n_inst; base += BS_NT) {
    const uint32_t i = base + threadIdx.x;
    uint64_t units = 0, act = 0;
    if (i < v.n_inst && v.active[i]) {
      const uint64_t d = __ldcg(reinterpret_cast<const unsigned long long*>(&v.delta[i]));
      v.delta[i] = 0;
      if (count_round) v.rounds[i]++;
      if (d == 0) {
        v.active[i] = 0;
      } else {
        v.total[i] += d;
        act = 1;
        const uint32_t r = v.rpu[i];
        units = (v.n_rows[i] + r - 1) / r;
        if (v.lshift[i] == 5) units *= (v.w4[i] + 31) / 32;
      }
    }
    uint64_t tot_a, tot_u;
    const uint64_t ex_a = block_excl_sum<BS_NT>(act, s_scan, &tot_a);
    const uint64_t ex_u = block_excl_sum<BS_NT>(units, s_scan, &tot_u);
    if (act) {
      v.act[s_carry[0] + ex_a] = i;
      v.uprefix[s_carry[0] + ex_a] = s_carry[1] + ex_u;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      s_carry[0] += tot_a;
      s_carry[1] += tot_u;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    v.uprefix[s_carry[0]] = s_carry[1];
    *v.n_act = (uint32_t)s_carry[0];
    *v.u_total = s_carry[1];
  }
}

__global__ void __launch_bounds__(BS_NT) k_bs_book(BsView v) { bs_book(v, 0); }

// Algorithmic bytes of one lane, counted in profiling runs: Δ words read, path
// words read, path and Δ' words written.
template <bool ON>
struct BsMoved {
  uint32_t d = 0, f = 0, w = 0;
  __device__ void delta(bool x) { if (ON) d += x ? 1u : 0u; }
  __device__ void path() { if (ON) f++; }
  __device__ void write() { if (ON) w++; }
  __device__ unsigned long long bytes() const { return 16ull * d + 16ull * f + 32ull * w; }
};

// The new words of one row word: acc ∖ path, path updated.
__device__ __forceinline__ uint4 bs_new_word(const uint4& acc, uint4 f, uint4* fp) {
  const uint4 nw = make_uint4(acc.x & ~f.x, acc.y & ~f.y, acc.z & ~f.z, acc.w & ~f.w);
  if (any4(nw)) {
    or4(f, nw);
    *fp = f;
  }
  return nw;
}

// One semi-naive round over every active instance of the wave.  Reads Δ from
// (D_PAR, s_PAR), writes Δ' to the other buffer pair and updates F.
template <int PAR, bool PROF>
__global__ void __launch_bounds__(BS_NT, 3) k_bs_round(BsView v) {
  const uint32_t n_act = *v.n_act;
  const uint64_t U = *v.u_total;
  const uint4* __restrict__ Dc = PAR ? v.D1 : v.D0;
  uint4* __restrict__ Dn = PAR ? v.D0 : v.D1;
  const uint32_t* __restrict__ sc = PAR ? v.s1 : v.s0;
  uint32_t* __restrict__ sn = PAR ? v.s0 : v.s1;
  __shared__ uint4 s_ent[BS_NT / 32][32];
  __shared__ uint32_t s_seen[BS_NT / 32][16];
  const int lane = threadIdx.x & 31;
  uint4* ent = s_ent[threadIdx.x >> 5];        // edges with a non-empty Δ block: Δ row, summary, row of the strip
  uint32_t* seen_of = s_seen[threadIdx.x >> 5];  // per row of the strip: the words any of its edges has
  const uint64_t nwarps = (uint64_t)gridDim.x * (BS_NT / 32);
  BsMoved<PROF> mv;
  unsigned long long moved = 0;
  uint32_t k = 0;
  uint64_t k_end = 0;
  for (uint64_t u = ((uint64_t)blockIdx.x * BS_NT + threadIdx.x) >> 5; u < U; u += nwarps) {
    if (u >= k_end) {
      k = unit_owner(v.uprefix, k, n_act, u);
      k_end = v.uprefix[k + 1];
    }
    const uint32_t i = v.act[k];
    const uint32_t n = v.n_rows[i], W = v.w4[i], R = v.rpu[i];
    const int ls = v.lshift[i];
    const uint64_t rb = v.row_base[i], vb = v.vec_base[i], sb = v.sum_base[i];
    const uint32_t ul = (uint32_t)(u - v.uprefix[k]);
    uint32_t cnt = 0;
    if (ls < 5) {
      // lane group `sub` owns row X, its lane sl the row's word sl
      const uint32_t lpr = 1u << ls, sub = (uint32_t)lane >> ls, sl = (uint32_t)lane & (lpr - 1);
      const uint32_t X = ul * (32u >> ls) + sub;
      const bool valid = X < n;
      const uint64_t e0 = valid ? v.off[rb + X] : 0, e1 = valid ? v.off[rb + X + 1] : 0;
      uint4 acc = make_uint4(0u, 0u, 0u, 0u);
      for (uint64_t e = e0; e < e1; e += 4) {
        uint32_t y[4], sm[4];
#pragma unroll
        for (int q = 0; q < 4; q++) y[q] = e + q < e1 ? v.nbr[e + q] : 0xffffffffu;
#pragma unroll
        for (int q = 0; q < 4; q++) sm[q] = y[q] < n ? sc[sb + y[q]] : 0u;
        uint4 d[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const bool on = (sm[q] >> sl) & 1u;
          d[q] = on ? Dc[vb + (uint64_t)y[q] * W + sl] : make_uint4(0u, 0u, 0u, 0u);
          mv.delta(on);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) or4(acc, d[q]);
      }
      uint4 nw = make_uint4(0u, 0u, 0u, 0u);
      if (any4(acc)) {
        uint4* fp = v.F + vb + (uint64_t)X * W + sl;
        nw = bs_new_word(acc, *fp, fp);
        mv.path();
      }
      const bool has = any4(nw);
      if (has) {
        Dn[vb + (uint64_t)X * W + sl] = nw;
        cnt = popc4(nw);
        mv.write();
      }
      const unsigned bal = __ballot_sync(kFull, has);
      if (valid && sl == 0) sn[sb + X] = (bal >> (sub << ls)) & ((1u << lpr) - 1u);
      if (PROF && valid && sl == 0) moved += (e1 - e0) * 8ull + 4ull;
    } else {
      const uint32_t strips = (n + R - 1) / R;
      const uint32_t cb = ul / strips, x0 = (ul - cb * strips) * R;
      const uint32_t rows = n - x0 < R ? n - x0 : R;
      const uint32_t c = cb * 32 + lane;  // this lane's word (summary bits exist only below W)
      const uint32_t* __restrict__ sblk = sc + sb + (uint64_t)cb * n;
      uint32_t* __restrict__ snblk = sn + sb + (uint64_t)cb * n + x0;
      const uint4* __restrict__ dcol = Dc + vb + c;
      uint4* __restrict__ frow = v.F + vb + (uint64_t)x0 * W + c;
      uint4* __restrict__ drow = Dn + vb + (uint64_t)x0 * W + c;
      // CSR offsets of the strip, one a lane (rows <= 16)
      const uint64_t eb = v.off[rb + x0];
      const uint32_t eo = (uint32_t)lane <= rows ? (uint32_t)(v.off[rb + x0 + lane] - eb) : 0xffffffffu;
      const uint32_t* __restrict__ nb = v.nbr + eb;
      uint32_t mine = 0;  // lane r: the summary of row r's new words
      // row r done: its new words are acc outside the path word f
      auto finish = [&](uint32_t r, const uint4& acc, const uint4& f, uint32_t seen) {
        uint4 nw = make_uint4(0u, 0u, 0u, 0u);
        if ((seen >> lane) & 1u) nw = bs_new_word(acc, f, frow + (uint64_t)r * W);
        const bool has = any4(nw);
        if (has) {
          drow[(uint64_t)r * W] = nw;
          cnt += popc4(nw);
          mv.write();
        }
        const unsigned bal = __ballot_sync(kFull, has);
        if ((uint32_t)lane == r) mine = bal;
      };
      for (uint32_t r0 = 0; r0 < rows;) {
        // whole rows of at most 32 edges together
        const uint32_t p0 = __shfl_sync(kFull, eo, (int)r0);
        const uint32_t r1 = r0 + __popc(__ballot_sync(kFull, (uint32_t)lane > r0 && (uint32_t)lane <= rows && eo - p0 <= 32u));
        if (r1 == r0) {  // one row of more than 32 edges: its windows in turn
          const uint32_t end = __shfl_sync(kFull, eo, (int)r0 + 1);
          uint4 acc = make_uint4(0u, 0u, 0u, 0u), f = acc;
          uint32_t seen = 0;
          for (uint32_t pos = p0; pos < end; pos += 32) {
            const uint32_t y = pos + lane < end ? nb[pos + lane] : 0xffffffffu;
            const uint32_t sm = y < n ? sblk[y] : 0u;
            for (unsigned on = __ballot_sync(kFull, sm != 0u); on;) {
              uint4 d[8];
#pragma unroll
              for (int q = 0; q < 8; q++) {
                const int t = on ? __ffs(on) - 1 : 0;
                const uint32_t yt = __shfl_sync(kFull, y, t), st = on ? __shfl_sync(kFull, sm, t) : 0u;
                on &= on - 1;
                seen |= st;
                d[q] = make_uint4(0u, 0u, 0u, 0u);
                if ((st >> lane) & 1u) {
                  d[q] = dcol[(uint64_t)yt * W];
                  mv.delta(true);
                }
              }
#pragma unroll
              for (int q = 0; q < 8; q++) or4(acc, d[q]);
            }
          }
          if ((seen >> lane) & 1u) {
            f = frow[(uint64_t)r0 * W];
            mv.path();
          }
          finish(r0, acc, f, seen);
          r0++;
          continue;
        }
        const uint32_t ne = __shfl_sync(kFull, eo, (int)r1) - p0;
        const uint32_t y = (uint32_t)lane < ne ? nb[p0 + lane] : 0xffffffffu;
        const uint32_t sm = y < n ? sblk[y] : 0u;
        // the row of this lane's edge: the last one that starts at or before it
        uint32_t row = 0;
#pragma unroll
        for (uint32_t st = 8; st > 0; st >>= 1) {
          const uint32_t o = __shfl_sync(kFull, eo, (int)(row + st));
          if (row + st < r1 && o <= p0 + lane) row += st;
        }
        // the edges whose Δ block is not empty, compacted: N entries, `endm`
        // those that end their row
        const bool act = sm != 0u;
        const unsigned A = __ballot_sync(kFull, act);
        const uint32_t N = __popc(A), ci = __popc(A & lanemask_lt());
        const unsigned above = A & ~(lanemask_lt() | (1u << lane));
        const uint32_t next_row = __shfl_sync(kFull, row, above ? __ffs(above) - 1 : 0);
        const bool last = act && (above == 0u || next_row != row);
        const unsigned endm = __reduce_or_sync(kFull, last ? 1u << ci : 0u);
        if (lane < 16) seen_of[lane] = 0u;
        __syncwarp();
        if (act) {
          ent[ci] = make_uint4(y, sm, row, 0u);
          atomicOr(&seen_of[row], sm);
        }
        __syncwarp();
        // eight entries at a time, at most three row ends among them: their Δ
        // words and the ending rows' path words are in flight together
        uint4 acc = make_uint4(0u, 0u, 0u, 0u);
        for (uint32_t j = 0; j < N;) {
          uint32_t nq = N - j < 8 ? N - j : 8;
          unsigned ends = (endm >> j) & ((1u << nq) - 1u);
          if (__popc(ends) > 3) {
            const unsigned e3 = ends & (ends - 1) & ((ends & (ends - 1)) - 1);  // without the first two
            nq = __ffs(e3);
            ends &= (1u << nq) - 1u;
          }
          uint4 d[8];
#pragma unroll
          for (int q = 0; q < 8; q++) {
            d[q] = make_uint4(0u, 0u, 0u, 0u);
            if ((uint32_t)q < nq) {
              const uint4 en = ent[j + q];
              if ((en.y >> lane) & 1u) {
                d[q] = dcol[(uint64_t)en.x * W];
                mv.delta(true);
              }
            }
          }
          uint4 f[3];
          uint32_t fr[3], fs[3];
          unsigned left = ends;
#pragma unroll
          for (int t = 0; t < 3; t++) {
            f[t] = make_uint4(0u, 0u, 0u, 0u);
            fr[t] = fs[t] = 0u;
            if (left) {
              fr[t] = ent[j + __ffs(left) - 1].z;
              fs[t] = seen_of[fr[t]];
              left &= left - 1;
              if ((fs[t] >> lane) & 1u) {
                f[t] = frow[(uint64_t)fr[t] * W];
                mv.path();
              }
            }
          }
          int t = 0;
#pragma unroll
          for (int q = 0; q < 8; q++) {
            or4(acc, d[q]);
            if ((ends >> q) & 1u) {
              finish(t == 0 ? fr[0] : t == 1 ? fr[1] : fr[2], acc, t == 0 ? f[0] : t == 1 ? f[1] : f[2],
                     t == 0 ? fs[0] : t == 1 ? fs[1] : fs[2]);
              t++;
              acc = make_uint4(0u, 0u, 0u, 0u);
            }
          }
          j += nq;
        }
        __syncwarp();  // the entries are rewritten for the next rows
        r0 = r1;
      }
      if ((uint32_t)lane < rows) snblk[lane] = mine;
      if (PROF && (uint32_t)lane == rows) moved += eo * 8ull + rows * 12ull;
    }
    cnt = warp_sum(cnt);
    if (lane == 0 && cnt) atomicAdd(reinterpret_cast<unsigned long long*>(&v.delta[i]), (unsigned long long)cnt);
  }
  if (PROF) {
    moved = warp_sum(moved + mv.bytes());
    if (lane == 0 && moved) atomicAdd(v.bytes, moved);
  }
  // the last block to finish does the bookkeeping (no block waits)
  __shared__ bool s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(v.ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (threadIdx.x == 0) *v.ticket = 0;
  bs_book(v, 1);
}

// Instance of a wave-local edge index (edge offsets relative to the wave).
__device__ __forceinline__ uint32_t edge_owner(const uint64_t* eoff, uint32_t n_inst, uint64_t g) {
  uint32_t lo = 0, hi = n_inst;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (eoff[mid] <= g) lo = mid; else hi = mid;
  }
  return lo;
}

// Out-degree per global row.
__global__ void k_bs_degree(const uint32_t* __restrict__ src, const uint32_t* __restrict__ dst, uint64_t m, BsView v,
                            uint32_t* deg) {
  for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < m; g += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = edge_owner(v.eoff, v.n_inst, g);
    const uint64_t e = v.ebase[i] + (g - v.eoff[i]);
    const uint32_t x = src[e], y = dst[e];
    if (x >= v.n_rows[i] || y >= v.n_cols[i]) {
      v.n_act[1] = 1u;  // an edge endpoint outside its instance's nodes
      continue;
    }
    atomicAdd(&deg[v.row_base[i] + x], 1u);
  }
}

// Exclusive scan of u32 degrees into u64 offsets: per-tile sums, one-block
// scan of the sums, then the write.
constexpr uint32_t SC_TILE = 2048;
__global__ void __launch_bounds__(BS_NT) k_bs_tile_sums(const uint32_t* __restrict__ deg, uint64_t n,
                                                        uint64_t* __restrict__ sums) {
  __shared__ uint64_t s_red[BS_NT / 32];
  uint64_t s = 0;
  const uint64_t b = (uint64_t)blockIdx.x * SC_TILE;
  for (uint32_t j = threadIdx.x; j < SC_TILE; j += BS_NT)
    if (b + j < n) s += deg[b + j];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint64_t t = 0;
    for (int w = 0; w < BS_NT / 32; w++) t += s_red[w];
    sums[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(BS_NT) k_bs_tile_write(const uint32_t* __restrict__ deg, uint64_t n,
                                                         const uint64_t* __restrict__ sums, uint64_t* __restrict__ off) {
  __shared__ uint64_t s_scan[BS_NT / 32 + 1];
  __shared__ uint64_t s_carry;
  if (threadIdx.x == 0) s_carry = sums[blockIdx.x];
  __syncthreads();
  const uint64_t b = (uint64_t)blockIdx.x * SC_TILE;
  for (uint32_t j0 = 0; j0 < SC_TILE; j0 += BS_NT) {
    const uint64_t r = b + j0 + threadIdx.x;
    const uint64_t d = r < n ? deg[r] : 0;
    uint64_t tot;
    const uint64_t ex = block_excl_sum<BS_NT>(d, s_scan, &tot);
    if (r < n) off[r] = s_carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) s_carry += tot;
    __syncthreads();
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) off[n] = s_carry;
}

// Scatter edges into the CSR (order within a row is free: the round ORs; deg
// counts each row's free places down) and seed path = Δ0 = edge bits with
// their summary, counting distinct edges per instance.
__global__ void k_bs_seed(const uint32_t* __restrict__ src, const uint32_t* __restrict__ dst, uint64_t m, BsView v,
                          uint32_t* deg, uint32_t* nbr) {
  const int lane = threadIdx.x & 31;
  for (uint64_t g0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull; g0 < m;
       g0 += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t g = g0 + lane;
    uint32_t fresh = 0, i = 0xffffffffu;
    if (g < m) {
      i = edge_owner(v.eoff, v.n_inst, g);
      const uint64_t e = v.ebase[i] + (g - v.eoff[i]);
      const uint32_t x = src[e], y = dst[e];
      if (x < v.n_rows[i] && y < v.n_cols[i]) {
        const uint64_t row = v.row_base[i] + x;
        nbr[v.off[row] + (atomicSub(&deg[row], 1u) - 1u)] = y;
        uint32_t* Fw = reinterpret_cast<uint32_t*>(v.F + v.vec_base[i] + (uint64_t)x * v.w4[i]);
        const uint32_t bit = 1u << (y & 31);
        const uint32_t old = atomicOr(&Fw[y >> 5], bit);
        fresh = (old & bit) ? 0u : 1u;
        const uint32_t c = y >> 7;
        if (fresh) atomicOr(&v.s0[v.sum_base[i] + (uint64_t)(c >> 5) * v.n_rows[i] + x], 1u << (c & 31));
      }
    }
    // per-instance distinct-edge counts (warp-aggregated when the warp is one instance)
    const uint32_t i0 = __shfl_sync(kFull, i, 0);
    if (__all_sync(kFull, i == i0 || i == 0xffffffffu)) {
      const uint32_t c = warp_sum(fresh);
      if (lane == 0 && c && i0 != 0xffffffffu)
        atomicAdd(reinterpret_cast<unsigned long long*>(&v.delta[i0]), (unsigned long long)c);
    } else if (fresh) {
      atomicAdd(reinterpret_cast<unsigned long long*>(&v.delta[i]), 1ull);
    }
  }
}

// Δ0's nonzero words: every edge copies its (finished) path word.
__global__ void k_bs_delta0(const uint32_t* __restrict__ src, const uint32_t* __restrict__ dst, uint64_t m, BsView v) {
  for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < m; g += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = edge_owner(v.eoff, v.n_inst, g);
    const uint64_t e = v.ebase[i] + (g - v.eoff[i]);
    const uint32_t x = src[e], y = dst[e];
    if (x >= v.n_rows[i] || y >= v.n_cols[i]) continue;
    const uint64_t w = v.vec_base[i] + (uint64_t)x * v.w4[i] + (y >> 7);
    v.D0[w] = v.F[w];
  }
}

// |path| and Σ mix64(X) · c^Z per instance from the final bit rows.
// tpw[w] = c^(32 w); tables tb[b][v] = Σ_{j ∈ bits(v)} c^(8 b + j).  Bound by
// the integer work per 32-bit word (192 ER instances, 4.8 GB of rows: 3.4 ms).
__global__ void __launch_bounds__(BS_NT) k_bs_final(BsView v, const uint64_t* __restrict__ tpw,
                                                    const uint64_t* __restrict__ tb_g) {
  __shared__ uint64_t tb[4][256];
  for (int t = threadIdx.x; t < 1024; t += BS_NT) (&tb[0][0])[t] = tb_g[t];
  __syncthreads();
  const uint64_t U = v.fprefix[v.n_inst];
  const int lane = threadIdx.x & 31;
  const uint64_t nwarps = (uint64_t)gridDim.x * (BS_NT / 32);
  uint32_t i = 0;
  for (uint64_t u = ((uint64_t)blockIdx.x * BS_NT + threadIdx.x) >> 5; u < U; u += nwarps) {
    i = unit_owner(v.fprefix, i, v.n_inst, u);
    const uint32_t n = v.n_rows[i], W = v.w4[i];
    const int ls = v.lshift[i];
    const uint32_t lpr = 1u << ls, sub = (uint32_t)lane >> ls, sl = (uint32_t)lane & (lpr - 1);
    const uint64_t X = (u - v.fprefix[i]) * (32u >> ls) + sub;
    uint64_t cnt = 0, poly = 0;
    if (X < n) {
      const uint4* row = v.F + v.vec_base[i] + X * W;
      for (uint32_t c0 = sl; c0 < W; c0 += 4 * lpr) {
        uint4 w4[4];  // four words in flight
#pragma unroll
        for (int q = 0; q < 4; q++) {
          w4[q] = make_uint4(0u, 0u, 0u, 0u);
          if (c0 + q * lpr < W) w4[q] = __ldcs(&row[c0 + q * lpr]);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const uint32_t wd[4] = {w4[q].x, w4[q].y, w4[q].z, w4[q].w};
          if (!any4(w4[q])) continue;
          const uint64_t* pw = tpw + 4 * (uint64_t)(c0 + q * lpr);
#pragma unroll
          for (int h = 0; h < 4; h++) {
            const uint32_t x = wd[h];
            cnt += __popc(x);
            poly += pw[h] * (tb[0][x & 255] + tb[1][(x >> 8) & 255] + tb[2][(x >> 16) & 255] + tb[3][x >> 24]);
          }
        }
      }
      // splitmix64 finalizer of X
      uint64_t z = X + kPolyC;
      z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
      z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
      z ^= z >> 31;
      poly *= z;
    }
    cnt = warp_sum(cnt);
    poly = warp_sum(poly);
    if (lane == 0) {
      if (cnt) atomicAdd(reinterpret_cast<unsigned long long*>(&v.counts[i]), (unsigned long long)cnt);
      if (poly) atomicAdd(reinterpret_cast<unsigned long long*>(&v.fps[i]), (unsigned long long)poly);
    }
  }
}

inline uint32_t lanes_shift(uint32_t w4) {
  int s = 0;
  while (s < 5 && (1u << s) < w4) s++;
  return (uint32_t)s;
}

// Fixed buffers of one call, sized for the largest wave.  Everything kept per
// instance lives in one block, which one copy fills (and zeroes) per wave.
struct BsBuffers {
  DBuf<uint64_t> inst, off, sums, bytes;
  DBuf<uint32_t> deg, nbr, s0, s1;
  DBuf<uint4> F, D0, D1;
  std::vector<uint64_t> host;  // the block as the next wave starts
  uint32_t n = 0;              // instances the block holds
  // 64-bit arrays (n + 1 entries each), then 32-bit, then bytes
  enum { ROW_BASE, VEC_BASE, SUM_BASE, EOFF, EBASE, FPREFIX, UPREFIX, DELTA, TOTAL, COUNTS, FPS, SCALARS, N64 };
  enum { N_ROWS, N_COLS, W4, RPU, ACT, ROUNDS, N32 };
  enum { LSHIFT, ACTIVE, N8 };
  explicit BsBuffers(strata_ctx* c) {
    for (auto* b : {&inst, &off, &sums, &bytes}) b->ctx = c;
    for (auto* b : {&deg, &nbr, &s0, &s1}) b->ctx = c;
    F.ctx = D0.ctx = D1.ctx = c;
  }
  uint64_t s64() const { return n + 1; }
  uint64_t s32() const { return (n + 2) & ~1ull; }   // entries, 8-byte multiples
  uint64_t s8() const { return (n + 8) & ~7ull; }
  uint64_t words() const { return N64 * s64() + N32 * s32() / 2 + N8 * s8() / 8; }
  uint64_t* p64(uint64_t* b, int k) const { return b + k * s64(); }
  uint32_t* p32(uint64_t* b, int k) const { return reinterpret_cast<uint32_t*>(b + N64 * s64()) + k * s32(); }
  uint8_t* p8(uint64_t* b, int k) const {
    return reinterpret_cast<uint8_t*>(b + N64 * s64() + N32 * s32() / 2) + k * s8();
  }
  void reserve_inst(uint32_t max_n) {
    n = std::max<uint32_t>(max_n, 3);  // SCALARS holds three words
    inst.reserve(words());
    host.assign(words(), 0);
  }
  BsView view(bool profile, uint32_t n_inst) {
    uint64_t* b = inst.p;
    BsView v{};
    v.n_rows = p32(b, N_ROWS);
    v.n_cols = p32(b, N_COLS);
    v.w4 = p32(b, W4);
    v.rpu = p32(b, RPU);
    v.lshift = p8(b, LSHIFT);
    v.row_base = p64(b, ROW_BASE);
    v.vec_base = p64(b, VEC_BASE);
    v.sum_base = p64(b, SUM_BASE);
    v.eoff = p64(b, EOFF);
    v.ebase = p64(b, EBASE);
    v.fprefix = p64(b, FPREFIX);
    v.delta = p64(b, DELTA);
    v.total = p64(b, TOTAL);
    v.counts = p64(b, COUNTS);
    v.fps = p64(b, FPS);
    v.rounds = p32(b, ROUNDS);
    v.active = p8(b, ACTIVE);
    v.act = p32(b, ACT);
    v.uprefix = p64(b, UPREFIX);
    v.n_act = reinterpret_cast<uint32_t*>(p64(b, SCALARS));
    v.u_total = p64(b, SCALARS) + 1;
    v.ticket = reinterpret_cast<uint32_t*>(p64(b, SCALARS) + 2);
    v.n_inst = n_inst;
    v.off = off.p;
    v.nbr = nbr.p;
    v.F = F.p;
    v.D0 = D0.p;
    v.D1 = D1.p;
    v.s0 = s0.p;
    v.s1 = s1.p;
    v.bytes = profile ? reinterpret_cast<unsigned long long*>(bytes.p) : nullptr;
    return v;
  }
};

struct InstSpec {
  uint32_t rows, cols;
  uint64_t e0, e1;  // edge range in the input arrays
};

inline uint64_t inst_w4(const InstSpec& s) { return std::max<uint64_t>(1, ceil_div(s.cols, 128)); }
inline uint64_t inst_vecs(const InstSpec& s) { return (uint64_t)s.rows * inst_w4(s); }
// Matrices, row and edge arrays: what the size rules (8 GB, one instance per
// budget) go by.
inline uint64_t inst_bytes(const InstSpec& s) {
  return 3 * inst_vecs(s) * 16 + (uint64_t)s.rows * (2 + 4 + 16) + (s.e1 - s.e0) * 4 + 64;
}
// What an instance takes: also the Δ summaries of rows wider than 32 words
// (inst_bytes has room for narrower ones).
inline uint64_t wave_bytes(const InstSpec& s) {
  return inst_bytes(s) + (uint64_t)s.rows * 8 * (ceil_div(inst_w4(s), 32) - 1);
}

struct BsResult {
  std::vector<uint64_t> counts, fps, totals;
  std::vector<uint32_t> rounds;
  uint64_t waves = 0, graph_launches = 0, round_launches = 0, bytes = 0;
  uint32_t rounds_max = 0;
};

// Host tables of the fingerprint: c^(32 w) for w < words, and the byte tables.
void poly_tables(uint64_t words, std::vector<uint64_t>& tpw, std::vector<uint64_t>& tb) {
  tpw.resize(std::max<uint64_t>(words, 1));
  uint64_t c32 = 1;
  for (int j = 0; j < 32; j++) c32 *= kPolyC;
  uint64_t a = 1;
  for (uint64_t w = 0; w < tpw.size(); w++) {
    tpw[w] = a;
    a *= c32;
  }
  uint64_t pw[32];
  pw[0] = 1;
  for (int j = 1; j < 32; j++) pw[j] = pw[j - 1] * kPolyC;
  tb.assign(1024, 0);
  for (int b = 0; b < 4; b++)
    for (int x = 0; x < 256; x++) {
      uint64_t s = 0;
      for (int j = 0; j < 8; j++)
        if (x >> j & 1) s += pw[8 * b + j];
      tb[b * 256 + x] = s;
    }
}

int round_grid(strata_ctx* ctx) {
  int per_sm = 0;
  check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bs_round<0, false>, BS_NT, 0), "occupancy");
  if (ctx->tune_bs_blocks > 0) per_sm = std::min(per_sm, ctx->tune_bs_blocks);
  return std::max(1, per_sm) * ctx->num_sms;
}

// Rows per unit of an instance of rows wider than 16 words: as many (up to 16)
// as leave each resident warp two units, so that one unit's metadata serves
// several rows without leaving warps idle on a small instance.
inline uint32_t strip_rows(uint64_t rows, uint64_t w4, uint64_t warps) {
  uint32_t r = 1;
  while (r < 16 && rows * ((w4 + 31) / 32) / (2 * r) >= 2 * warps) r *= 2;
  return r;
}

// Run the instances as waves within `budget` bytes.  Mode 0: graph-replayed
// batched rounds; 1: one instance per launch, host-driven rounds; 2: batched,
// the rounds launched in groups of R without a graph.  F of the last wave is
// left in `bufs`.
void bs_run(strata_ctx* ctx, const std::vector<InstSpec>& spec, const uint32_t* d_src, const uint32_t* d_dst,
            int mode, uint64_t budget, BsBuffers& B, BsResult& R, bool want_fp) {
  const uint32_t n_inst = (uint32_t)spec.size();
  R.counts.assign(n_inst, 0);
  R.fps.assign(n_inst, 0);
  R.totals.assign(n_inst, 0);
  R.rounds.assign(n_inst, 0);
  // order: largest first (mode 0 packs waves; mode 1 runs one at a time)
  std::vector<uint32_t> order(n_inst);
  for (uint32_t i = 0; i < n_inst; i++) order[i] = i;
  std::stable_sort(order.begin(), order.end(),
                   [&](uint32_t a, uint32_t b) { return inst_vecs(spec[a]) > inst_vecs(spec[b]); });
  std::vector<std::pair<uint32_t, uint32_t>> waves;  // ranges of `order`
  {
    uint32_t a = 0;
    while (a < n_inst) {
      if (inst_bytes(spec[order[a]]) > budget) fail(STRATA_E_OOM, "one instance's bit matrices exceed the memory budget");
      uint64_t bytes = wave_bytes(spec[order[a]]);
      uint32_t b = a + 1;
      if (mode != 1)
        for (; b < n_inst && bytes + wave_bytes(spec[order[b]]) <= budget; b++) bytes += wave_bytes(spec[order[b]]);
      waves.push_back({a, b});
      a = b;
    }
  }
  // size the fixed buffers for the largest wave
  uint64_t max_rows = 1, max_vecs = 1, max_sums = 1, max_edges = 1, max_w32 = 1;
  uint32_t max_n = 1;
  for (auto& w : waves) {
    uint64_t rows = 0, vecs = 0, sums = 0, edges = 0;
    for (uint32_t k = w.first; k < w.second; k++) {
      const InstSpec& s = spec[order[k]];
      rows += s.rows;
      vecs += inst_vecs(s);
      sums += s.rows * ceil_div(inst_w4(s), 32);
      edges += s.e1 - s.e0;
      max_w32 = std::max<uint64_t>(max_w32, 4 * inst_w4(s));
    }
    max_rows = std::max(max_rows, rows);
    max_vecs = std::max(max_vecs, vecs);
    max_sums = std::max(max_sums, sums);
    max_edges = std::max(max_edges, edges);
    max_n = std::max(max_n, w.second - w.first);
  }
  B.reserve_inst(max_n);
  B.deg.reserve(max_rows + 1);
  B.off.reserve(max_rows + 1);
  B.sums.reserve(ceil_div(max_rows + 1, SC_TILE) + 2);
  B.nbr.reserve(max_edges);
  B.s0.reserve(max_sums);
  B.s1.reserve(max_sums);
  B.F.reserve(max_vecs);
  B.D0.reserve(max_vecs);
  B.D1.reserve(max_vecs);
  B.bytes.reserve(1);
  DBuf<uint64_t> d_tpw, d_tb;
  d_tpw.ctx = d_tb.ctx = ctx;
  if (want_fp) {
    std::vector<uint64_t> tpw, tb;
    poly_tables(max_w32, tpw, tb);
    d_tpw.reserve(max_w32);
    d_tb.reserve(1024);
    SK_CUDA(cudaMemcpyAsync(d_tpw.p, tpw.data(), tpw.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
    SK_CUDA(cudaMemcpyAsync(d_tb.p, tb.data(), 1024 * 8, cudaMemcpyHostToDevice, ctx->stream));
  }
  const bool profile = ctx->profiling;
  if (profile) SK_CUDA(cudaMemsetAsync(B.bytes.p, 0, 8, ctx->stream));
  const int grid = round_grid(ctx);
  const uint64_t warps = (uint64_t)grid * (BS_NT / 32);
  const int R_group = ctx->tune_bs_graph_rounds > 0 ? ctx->tune_bs_graph_rounds : 8;
  auto round = [&](const BsView& v, int par) {
    auto* kern = par == 0 ? (profile ? k_bs_round<0, true> : k_bs_round<0, false>)
                          : (profile ? k_bs_round<1, true> : k_bs_round<1, false>);
    kern<<<grid, BS_NT, 0, ctx->stream>>>(v);
  };

  // The graph of R_group rounds (even, so buffer parity is the same at every
  // replay) over the fixed buffers, captured once per call.
  cudaGraphExec_t exec = nullptr;
  uint32_t graph_n_inst = 0;
  auto capture = [&](const BsView& v) {
    if (exec && graph_n_inst == v.n_inst) return;
    if (exec) cudaGraphExecDestroy(exec);
    exec = nullptr;
    cudaGraph_t g;
    SK_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    for (int r = 0; r < R_group; r++) round(v, r & 1);
    SK_CUDA(cudaStreamEndCapture(ctx->stream, &g));
    SK_CUDA(cudaGraphInstantiate(&exec, g, 0));
    cudaGraphDestroy(g);
    graph_n_inst = v.n_inst;
  };

  for (auto& w : waves) {
    const uint32_t nw = w.second - w.first;
    uint64_t* h = B.host.data();
    std::fill(B.host.begin(), B.host.end(), 0);
    uint64_t rows = 0, vecs = 0, sums = 0, edges = 0, units = 0;
    for (uint32_t k = 0; k < nw; k++) {
      const InstSpec& s = spec[order[w.first + k]];
      const uint32_t w4 = (uint32_t)inst_w4(s), ls = lanes_shift(w4);
      B.p32(h, B.N_ROWS)[k] = s.rows;
      B.p32(h, B.N_COLS)[k] = s.cols;
      B.p32(h, B.W4)[k] = w4;
      B.p32(h, B.RPU)[k] = ls < 5 ? 32u >> ls : strip_rows(s.rows, w4, warps);
      B.p8(h, B.LSHIFT)[k] = (uint8_t)ls;
      B.p8(h, B.ACTIVE)[k] = 1;
      B.p64(h, B.ROW_BASE)[k] = rows;
      B.p64(h, B.VEC_BASE)[k] = vecs;
      B.p64(h, B.SUM_BASE)[k] = sums;
      B.p64(h, B.EOFF)[k] = edges;
      B.p64(h, B.EBASE)[k] = s.e0;
      B.p64(h, B.FPREFIX)[k] = units;
      rows += s.rows;
      vecs += inst_vecs(s);
      sums += s.rows * ceil_div(w4, 32);
      edges += s.e1 - s.e0;
      units += ceil_div(s.rows, 32u >> ls);
    }
    B.p64(h, B.EOFF)[nw] = edges;
    B.p64(h, B.FPREFIX)[nw] = units;
    const BsView v = B.view(profile, nw);
    SK_CUDA(cudaMemcpyAsync(B.inst.p, h, B.words() * 8, cudaMemcpyHostToDevice, ctx->stream));
    SK_CUDA(cudaMemsetAsync(B.deg.p, 0, (rows + 1) * 4, ctx->stream));
    SK_CUDA(cudaMemsetAsync(B.s0.p, 0, sums * 4, ctx->stream));
    SK_CUDA(cudaMemsetAsync(B.F.p, 0, vecs * 16, ctx->stream));
    const unsigned eg = (unsigned)std::min<uint64_t>(ceil_div(std::max<uint64_t>(edges, 1), 256), ctx->num_sms * 16ull);
    if (edges) {
      k_bs_degree<<<eg, 256, 0, ctx->stream>>>(d_src, d_dst, edges, v, B.deg.p);
      after_launch(ctx, "k_bs_degree");
    }
    const uint64_t tiles = ceil_div(rows + 1, SC_TILE);
    k_bs_tile_sums<<<(unsigned)tiles, BS_NT, 0, ctx->stream>>>(B.deg.p, rows, B.sums.p);
    after_launch(ctx, "k_bs_tile_sums");
    scan_tile_sums(ctx, B.sums.p, tiles);
    k_bs_tile_write<<<(unsigned)tiles, BS_NT, 0, ctx->stream>>>(B.deg.p, rows, B.sums.p, B.off.p);
    after_launch(ctx, "k_bs_tile_write");
    if (edges) {
      k_bs_seed<<<eg, 256, 0, ctx->stream>>>(d_src, d_dst, edges, v, B.deg.p, B.nbr.p);
      after_launch(ctx, "k_bs_seed");
      k_bs_delta0<<<eg, 256, 0, ctx->stream>>>(d_src, d_dst, edges, v);
      after_launch(ctx, "k_bs_delta0");
    }
    k_bs_book<<<1, BS_NT, 0, ctx->stream>>>(v);
    after_launch(ctx, "k_bs_book");
    // rounds: the host looks at the active count after every group
    const int kh = kprof_begin(ctx, K_BS_ROUND);
    auto active = [&]() {
      SK_CUDA(cudaMemcpyAsync(ctx->h_scalar, v.n_act, 8, cudaMemcpyDeviceToHost, ctx->stream));
      SK_CUDA(cudaStreamSynchronize(ctx->stream));
      if ((uint32_t)(ctx->h_scalar[0] >> 32)) {
        if (exec) cudaGraphExecDestroy(exec);
        fail(STRATA_E_INVALID, "an edge endpoint lies outside its instance's nodes");
      }
      return (uint32_t)ctx->h_scalar[0];
    };
    if (mode == 0) {
      if (active()) {
        capture(v);
        do {
          SK_CUDA(cudaGraphLaunch(exec, ctx->stream));
          R.graph_launches++;
          R.round_launches += R_group;
          ctx->launches += (uint64_t)R_group;
        } while (active());
      }
    } else {
      const int group = mode == 1 ? 1 : R_group;
      int par = 0;
      bool more = mode == 2 || active();  // mode 2: the first group runs before the first look
      while (more) {
        for (int r = 0; r < group; r++, par ^= 1) {
          round(v, par);
          after_launch(ctx, "k_bs_round");
          R.round_launches++;
        }
        more = active() != 0;
      }
    }
    kprof_end(ctx, kh, 0);
    if (want_fp) {
      k_bs_final<<<grid, BS_NT, 0, ctx->stream>>>(v, d_tpw.p, d_tb.p);
      after_launch(ctx, "k_bs_final");
    }
    SK_CUDA(cudaMemcpyAsync(h, B.inst.p, B.words() * 8, cudaMemcpyDeviceToHost, ctx->stream));
    sync_and_check(ctx);
    const uint64_t *c = B.p64(h, B.COUNTS), *f = B.p64(h, B.FPS), *t = B.p64(h, B.TOTAL);
    const uint32_t* r = B.p32(h, B.ROUNDS);
    for (uint32_t k = 0; k < nw; k++) {
      const uint32_t i = order[w.first + k];
      R.counts[i] = want_fp ? c[k] : t[k];
      R.fps[i] = f[k];
      R.totals[i] = t[k];
      R.rounds[i] = r[k];
      R.rounds_max = std::max(R.rounds_max, r[k]);
      if (want_fp && c[k] != t[k]) fail(STRATA_E_CUDA, "bit-row popcount disagrees with the summed Δ sizes");
    }
    R.waves++;
  }
  if (profile) {
    uint64_t b = 0;
    read_u64(ctx, B.bytes.p, &b, 1);
    R.bytes = b;
    kprof_add_last(ctx, K_BS_ROUND, b);
  }
  if (exec) cudaGraphExecDestroy(exec);
}

// ---- one rank's share of a sharded closure ---------------------------------
// The rank owns path rows X ∈ [lo, lo + rows) (local row x = X - lo), each W4
// uint4 words over the Z domain.  A round reads Δ(Y) of every node from the
// gathered matrix Dfull (all ranks' slices of the previous round, rank r's
// slice = rows [r·per, r·per + per)) with its byte flags ffull, and writes
// Δ'(X) of its own rows into Dmine / fmine:
//     Δ'(X) = ( ∪_{Y ∈ out(X)} Δ(Y) ) ∖ path(X),   path(X) ∪= Δ'(X)
// the same round as k_bs_round, one warp per unit of 32 / L rows.
struct ShardView {
  uint32_t rows, n, W;
  int ls;                // log2(lanes per row)
  const uint64_t* off;   // rows + 1, local rows
  const uint32_t* nbr;   // global neighbour ids
  uint4* F;              // rows × W
  unsigned long long* delta;
  unsigned long long* bytes;  // algorithmic bytes (as k_bs_round counts them), or null
};

__global__ void __launch_bounds__(BS_NT) k_shard_round(ShardView v, const uint4* __restrict__ Dfull,
                                                       const uint8_t* __restrict__ ffull, uint4* __restrict__ Dmine,
                                                       uint8_t* __restrict__ fmine) {
  const int lane = threadIdx.x & 31;
  const int ls = v.ls;
  const uint32_t lpr = 1u << ls, sub = (uint32_t)lane >> ls, sl = (uint32_t)lane & (lpr - 1);
  const unsigned smask = ls == 5 ? 0xffffffffu : (((1u << lpr) - 1u) << (sub << ls));
  const uint32_t W = v.W;
  const uint64_t units = ((uint64_t)v.rows + (32u >> ls) - 1) / (32u >> ls);
  const uint64_t nwarps = (uint64_t)gridDim.x * (BS_NT / 32);
  uint64_t cnt = 0;
  unsigned long long moved = 0;
  for (uint64_t u = ((uint64_t)blockIdx.x * BS_NT + threadIdx.x) >> 5; u < units; u += nwarps) {
    const uint64_t x = u * (32u >> ls) + sub;
    const bool valid = x < v.rows;
    const uint64_t e0 = valid ? v.off[x] : 0, e1 = valid ? v.off[x + 1] : 0;
    bool any_y = false;
    for (uint64_t e = e0 + sl; e < e1; e += lpr) {
      const uint32_t y = v.nbr[e];
      if (y < v.n && ffull[y]) any_y = true;
    }
    const unsigned bal_y = __ballot_sync(kFull, any_y);  // every lane takes part
    const bool row_has = valid && (bal_y & smask) != 0u;
    bool row_any = false;
    if (valid) {
      uint32_t active_edges = 0, acc_words = 0;
      for (uint32_t c = sl; c < W; c += lpr) {
        uint4 nw = make_uint4(0u, 0u, 0u, 0u);
        if (row_has) {
          uint4 acc = make_uint4(0u, 0u, 0u, 0u);
          active_edges = 0;
          for (uint64_t e = e0; e < e1; e += 4) {
            uint32_t y[4];
            bool on[4];
#pragma unroll
            for (int q = 0; q < 4; q++) y[q] = e + q < e1 ? v.nbr[e + q] : 0xffffffffu;
#pragma unroll
            for (int q = 0; q < 4; q++) on[q] = y[q] < v.n && ffull[y[q]] != 0;
            uint4 d[4];
#pragma unroll
            for (int q = 0; q < 4; q++) d[q] = on[q] ? Dfull[(uint64_t)y[q] * W + c] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int q = 0; q < 4; q++) {
              acc.x |= d[q].x;
              acc.y |= d[q].y;
              acc.z |= d[q].z;
              acc.w |= d[q].w;
              active_edges += on[q] ? 1u : 0u;
            }
          }
          if (any4(acc)) {
            acc_words++;
            uint4* fp = v.F + x * W + c;
            uint4 f = *fp;
            nw = make_uint4(acc.x & ~f.x, acc.y & ~f.y, acc.z & ~f.z, acc.w & ~f.w);
            if (any4(nw)) {
              *fp = make_uint4(f.x | nw.x, f.y | nw.y, f.z | nw.z, f.w | nw.w);
              cnt += popc4(nw);
              row_any = true;
            }
          }
        }
        Dmine[x * W + c] = nw;  // rows without Δ' are cleared too
      }
      if (v.bytes && row_has) {
        // this lane's words: Δ rows read, Δ' written, path read (and written
        // where bits are new); its share of the edge list and flags
        const uint64_t lw = (W > sl) ? (W - sl + lpr - 1) / lpr : 0;
        moved += lw * 16ull * (active_edges + 1) + acc_words * 32ull + (sl == 0 ? (e1 - e0) * 5ull : 0ull);
      }
    }
    const unsigned bal = __ballot_sync(kFull, row_any);
    if (valid && sl == 0) fmine[x] = (bal & smask) != 0u ? 1 : 0;
  }
  cnt = warp_sum(cnt);
  if (lane == 0 && cnt) atomicAdd(v.delta, (unsigned long long)cnt);
  if (v.bytes) {
    moved = warp_sum(moved);
    if (lane == 0 && moved) atomicAdd(v.bytes, moved);
  }
}

// Local out-degrees of the rank's rows; endpoints outside [0, n) set *bad.
__global__ void k_shard_degree(const uint32_t* __restrict__ src, const uint32_t* __restrict__ dst, uint64_t m,
                               uint32_t n, uint32_t lo, uint32_t hi, uint64_t* deg, uint32_t* bad) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t a = src[e], b = dst[e];
    if (a >= n || b >= n) {
      atomicOr(bad, 1u);
      continue;
    }
    if (a >= lo && a < hi) atomicAdd(reinterpret_cast<unsigned long long*>(&deg[a - lo]), 1ull);
  }
}

// CSR fill (neighbour order within a row is free: the round ORs them) and
// the seed: path(X) = Δ0(X) = the out-neighbour bits of X.
__global__ void k_shard_fill(const uint32_t* __restrict__ src, const uint32_t* __restrict__ dst, uint64_t m,
                             uint32_t n, uint32_t lo, uint32_t hi, uint32_t W, const uint64_t* __restrict__ off,
                             uint32_t* cursor, uint32_t* nbr, uint32_t* F, uint32_t* Dmine, uint8_t* fmine) {
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t a = src[e], b = dst[e];
    if (a >= n || b >= n || a < lo || a >= hi) continue;
    const uint32_t x = a - lo;
    nbr[off[x] + atomicAdd(&cursor[x], 1u)] = b;
    const uint64_t wd = (uint64_t)x * W * 4 + (b >> 5);
    atomicOr(&F[wd], 1u << (b & 31));
    atomicOr(&Dmine[wd], 1u << (b & 31));
    fmine[x] = 1;
  }
}

__global__ void k_shard_popc(const uint4* __restrict__ F, uint64_t words, unsigned long long* out) {
  uint64_t c = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (uint64_t)gridDim.x * blockDim.x)
    c += popc4(F[i]);
  c = warp_sum(c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, (unsigned long long)c);
}

// |path| and Σ mix64(X)·c^Z of the rank's rows (global X = lo + x); one warp
// per row.
__global__ void __launch_bounds__(BS_NT) k_shard_summary(const uint4* __restrict__ F, uint32_t rows, uint32_t W,
                                                         uint32_t lo, const uint64_t* __restrict__ tpw,
                                                         const uint64_t* __restrict__ tb_g, unsigned long long* out) {
  __shared__ uint64_t tb[4][256];
  for (int t = threadIdx.x; t < 1024; t += BS_NT) (&tb[0][0])[t] = tb_g[t];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint64_t nwarps = (uint64_t)gridDim.x * (BS_NT / 32);
  for (uint64_t x = ((uint64_t)blockIdx.x * BS_NT + threadIdx.x) >> 5; x < rows; x += nwarps) {
    uint64_t cnt = 0, poly = 0;
    for (uint32_t c = lane; c < W; c += 32) {
      const uint4 q = F[x * W + c];
      const uint32_t wd[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int h = 0; h < 4; h++) {
        const uint32_t w = wd[h];
        if (!w) continue;
        cnt += __popc(w);
        const uint64_t t = tb[0][w & 255] + tb[1][(w >> 8) & 255] + tb[2][(w >> 16) & 255] + tb[3][w >> 24];
        poly += tpw[4 * (uint64_t)c + h] * t;
      }
    }
    cnt = warp_sum(cnt);
    poly = warp_sum(poly);
    if (lane == 0) {
      uint64_t z = (uint64_t)lo + x + kPolyC;  // splitmix64 finalizer of the global X
      z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
      z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
      z ^= z >> 31;
      if (cnt) atomicAdd(&out[0], (unsigned long long)cnt);
      if (poly) atomicAdd(&out[1], (unsigned long long)(poly * z));
    }
  }
}

uint64_t bs_budget(strata_ctx* ctx, uint64_t need) {
  uint64_t b = device_budget(ctx, 0.7, need);
  if (ctx->cap && ctx->cap > ctx->in_use) b = std::min<uint64_t>(b, ctx->cap - ctx->in_use);
  if (ctx->tune_bs_budget_mb > 0) b = std::min<uint64_t>(b, (uint64_t)ctx->tune_bs_budget_mb << 20);
  return b;
}

}  // namespace

// Batched driver (instances described on the host, edges on the device).
void tc_bool_batch(strata_ctx* ctx, uint32_t n_inst, const uint32_t* nodes, const uint64_t* edge_off,
                   const uint32_t* d_src, const uint32_t* d_dst, int mode, uint64_t* counts, uint64_t* fps,
                   uint32_t* rounds, strata_batch_stats* st) {
  if (st) std::memset(st, 0, sizeof(*st));
  reset_status(ctx);
  if (mode != 0 && mode != 1) fail(STRATA_E_INVALID, "mode must be 0 (batched) or 1 (one instance per launch)");
  std::vector<InstSpec> spec(n_inst);
  for (uint32_t i = 0; i < n_inst; i++) {
    if (edge_off[i + 1] < edge_off[i]) fail(STRATA_E_INVALID, "edge offsets must be non-decreasing");
    spec[i] = InstSpec{nodes[i], nodes[i], edge_off[i], edge_off[i + 1]};
  }
  const uint64_t l0 = ctx->launches;
  cudaEvent_t e0, e1;
  check_cuda(cudaEventCreate(&e0), "cudaEventCreate");
  check_cuda(cudaEventCreate(&e1), "cudaEventCreate");
  check_cuda(cudaEventRecord(e0, ctx->stream), "cudaEventRecord");
  uint64_t need = 0;  // of all instances in one wave
  for (auto& i : spec) need += wave_bytes(i);
  const uint64_t budget = bs_budget(ctx, need);  // the waves are sized from what this context can reuse
  release_all_cached(ctx);
  BsBuffers B(ctx);
  BsResult R;
  try {
    bs_run(ctx, spec, d_src, d_dst, mode, budget, B, R, true);
  } catch (...) {
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    throw;
  }
  check_cuda(cudaEventRecord(e1, ctx->stream), "cudaEventRecord");
  sync_and_check(ctx);
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  kprof_collect(ctx);
  for (uint32_t i = 0; i < n_inst; i++) {
    if (counts) counts[i] = R.counts[i];
    if (fps) fps[i] = R.fps[i];
    if (rounds) rounds[i] = R.rounds[i];
  }
  if (st) {
    st->instances = n_inst;
    st->waves = R.waves;
    st->graph_launches = R.graph_launches;
    st->round_launches = R.round_launches;
    st->rounds_max = R.rounds_max;
    uint64_t tot = 0;
    for (auto c : R.counts) tot += c;
    st->result_tuples = tot;
    st->device_ms = ms;
    st->round_bytes = R.bytes;
    st->launches = ctx->launches - l0;
  }
}

// Single-instance Bool TC on bit rows: the relation comes back sorted by
// (X, Z) through the bitmap compaction.  Returns false when the bit matrices
// do not fit (the caller falls back to another plan).
bool tc_bool_bitset_fits(strata_ctx* ctx, uint64_t n_src, uint64_t n_dst, uint64_t m) {
  const InstSpec s{(uint32_t)n_src, (uint32_t)n_dst, 0, m};
  // asked for by name (plan 3), the rounds are tried up to the size rule itself
  const uint64_t need = ctx->plan == 3 ? inst_bytes(s) : wave_bytes(s);
  return n_src < (1ull << 32) && n_dst < (1ull << 32) && inst_bytes(s) <= (8ull << 30) && need <= bs_budget(ctx, need);
}

// ---- one small closure in one block --------------------------------------------
// A graph of a few hundred nodes: the edge CSR, path, Δ and Δ' bit rows fit one
// block's shared memory, so every round is a pass over them between two block
// barriers, and the sorted relation is written straight from the final rows.
// The general form spends 0.6 ms on such a graph in launches and waits; this is
// bound by the rounds' shared-memory reads (300 nodes, 701 edges, 14 rounds:
// 49 us on one B200, the call from host columns 639 -> 308 us).
constexpr int SM_NT = 1024;
constexpr uint64_t kSmallEdges = 16384, kSmallSmem = 226 * 1024;

inline uint64_t small_smem(uint64_t rows, uint64_t w, uint64_t m) {
  return 3 * rows * w * 4 + 2 * (rows + 1) * 4 + m * 2 + 16;
}

__global__ void __launch_bounds__(SM_NT) k_bs_small(const uint32_t* __restrict__ src, const uint32_t* __restrict__ dst,
                                                    uint32_t m, uint32_t rows, uint32_t cols, int b1,
                                                    uint32_t* __restrict__ out, uint64_t* res) {
  extern __shared__ __align__(16) uint32_t s_raw32[];
  __shared__ uint32_t s_scan[SM_NT / 32 + 1];
  const uint32_t W = (cols + 31) / 32, N = rows * W;
  uint32_t* F = s_raw32;
  uint32_t* D0 = F + N;
  uint32_t* D1 = D0 + N;
  uint32_t* off = D1 + N;        // rows + 1
  uint32_t* deg = off + rows + 1;  // rows + 1
  uint16_t* nbr = reinterpret_cast<uint16_t*>(deg + rows + 1);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (uint32_t i = tid; i < N; i += SM_NT) F[i] = 0u;
  for (uint32_t i = tid; i <= rows; i += SM_NT) deg[i] = 0u;
  __syncthreads();
  for (uint32_t e = tid; e < m; e += SM_NT) {
    const uint32_t x = src[e], y = dst[e];
    if (x >= rows || y >= cols) continue;
    atomicAdd(&deg[x], 1u);
    atomicOr(&F[x * W + (y >> 5)], 1u << (y & 31));
  }
  __syncthreads();
  uint32_t carry = 0;
  for (uint32_t b = 0; b < rows; b += SM_NT) {  // exclusive scan of the degrees
    const uint32_t d = b + tid < rows ? deg[b + tid] : 0u;
    uint32_t tot;
    const uint32_t ex = block_excl_sum<SM_NT>(d, s_scan, &tot);
    if (b + tid < rows) off[b + tid] = carry + ex;
    carry += tot;
  }
  if (tid == 0) off[rows] = carry;
  for (uint32_t i = tid; i < N; i += SM_NT) D0[i] = F[i];
  __syncthreads();
  for (uint32_t e = tid; e < m; e += SM_NT) {
    const uint32_t x = src[e], y = dst[e];
    if (x >= rows || y >= cols) continue;
    nbr[off[x] + atomicSub(&deg[x], 1u) - 1u] = (uint16_t)y;
  }
  __syncthreads();
  // a round adds a path length, so there are at most rows + 1 of them
  uint32_t rounds = 0;
  for (bool more = true; more && rounds <= rows + 1;) {
    bool any = false;
    for (uint32_t i = tid; i < N; i += SM_NT) {
      const uint32_t x = i / W, w = i - x * W, e1 = off[x + 1];
      uint32_t acc = 0;
      for (uint32_t e = off[x]; e < e1; e++) {
        const uint32_t y = nbr[e];
        if (y < rows) acc |= D0[y * W + w];
      }
      const uint32_t f = F[i], nw = acc & ~f;
      F[i] = f | nw;
      D1[i] = nw;
      any |= nw != 0u;
    }
    more = __syncthreads_or(any);
    uint32_t* t = D0;
    D0 = D1;
    D1 = t;
    rounds++;
  }
  // rows' sizes, their scan (deg now holds first ordinals), then the keys
  for (uint32_t x = warp; x < rows; x += SM_NT / 32) {
    uint32_t c = 0;
    for (uint32_t w = lane; w < W; w += 32) c += __popc(F[x * W + w]);
    c = warp_sum(c);
    if (lane == 0) deg[x] = c;
  }
  __syncthreads();
  carry = 0;
  for (uint32_t b = 0; b < rows; b += SM_NT) {
    const uint32_t d = b + tid < rows ? deg[b + tid] : 0u;
    uint32_t tot;
    const uint32_t ex = block_excl_sum<SM_NT>(d, s_scan, &tot);
    if (b + tid < rows) deg[b + tid] = carry + ex;
    carry += tot;
  }
  __syncthreads();
  for (uint32_t x = warp; x < rows; x += SM_NT / 32) {
    uint32_t at = deg[x];
    for (uint32_t w = 0; w < W; w++) {
      const uint32_t v = F[x * W + w];
      if ((v >> lane) & 1u) out[at + __popc(v & lanemask_lt())] = (x << b1) | (w * 32 + lane);
      at += __popc(v);
    }
  }
  if (tid == 0) {
    res[0] = carry;
    res[1] = rounds;
  }
}

bool tc_bool_small_fits(strata_ctx* ctx, uint64_t n_src, uint64_t n_dst, uint64_t m) {
  const uint64_t w = ceil_div(n_dst, 32);
  if (n_src > 1024 || n_dst > 1024 || m > kSmallEdges || small_smem(n_src, w, m) > kSmallSmem) return false;
  return !ctx->cap || ctx->in_use + 2 * size_class(n_src * n_dst * 4 + 64) <= ctx->cap;
}

uint64_t tc_bool_small(strata_ctx* ctx, const uint32_t* d_src, const uint32_t* d_dst, uint64_t m, uint64_t n_src,
                       uint64_t n_dst, int b1, DBuf<uint32_t>& out, uint64_t* rounds) {
  out.reserve(n_src * n_dst + 1);
  DBuf<uint64_t> res(ctx, 2);
  const size_t smem = small_smem(n_src, ceil_div(n_dst, 32), m);
  allow_smem(k_bs_small, kSmallSmem);
  k_bs_small<<<1, SM_NT, smem, ctx->stream>>>(d_src, d_dst, (uint32_t)m, (uint32_t)n_src, (uint32_t)n_dst, b1, out.p,
                                              res.p);
  after_launch(ctx, "k_bs_small");
  SK_CUDA(cudaMemcpyAsync(ctx->h_scalar, res.p, 16, cudaMemcpyDeviceToHost, ctx->stream));
  sync_and_check(ctx);
  *rounds = ctx->h_scalar[1];
  const uint64_t n = ctx->h_scalar[0];
  if (n_src * n_dst > 2 * n + 4096) {  // the relation keeps a buffer of its own size
    DBuf<uint32_t> fit(ctx, n + 1);
    if (n) SK_CUDA(cudaMemcpyAsync(fit.p, out.p, n * 4, cudaMemcpyDeviceToDevice, ctx->stream));
    out = std::move(fit);
  }
  return n;
}

template <class K>
uint64_t tc_bool_bitset(strata_ctx* ctx, const uint32_t* d_src, const uint32_t* d_dst, uint64_t m, uint64_t n_src,
                        uint64_t n_dst, int b1, DBuf<K>& out, uint64_t* rounds, uint64_t* round_bytes) {
  std::vector<InstSpec> spec{InstSpec{(uint32_t)n_src, (uint32_t)n_dst, 0, m}};
  BsBuffers B(ctx);
  BsResult R;
  bs_run(ctx, spec, d_src, d_dst, 2, UINT64_MAX, B, R, false);
  *rounds = R.rounds[0];
  *round_bytes = R.bytes;
  const uint64_t n = R.totals[0];
  const uint64_t w4 = inst_w4(spec[0]);
  const DenseLayout lay = dense_layout(b1, n_src, w4 * 128, false);
  out.reserve(n + 1);
  DBuf<uint64_t> states(ctx, dense_marks_states(lay.entries));
  const uint64_t got = dense_marks_compact<K, false, int32_t>(ctx, reinterpret_cast<uint32_t*>(B.F.p), lay, nullptr, out.p,
                                                     nullptr, n + 1, states.p);
  if (got != n) fail(STRATA_E_CUDA, "bit-row compaction count disagrees with the summed Δ sizes");
  return n;
}

// ---- sharded closure: one rank's share ------------------------------------
void tc_shard_init(strata_ctx* ctx, strata_tc_shard* sh, uint32_t n, const uint32_t* d_src, const uint32_t* d_dst,
                   uint64_t m, uint32_t rank, uint32_t world) {
  sh->n = n;
  sh->rank = rank;
  sh->world = world;
  sh->per = (uint32_t)ceil_div(n, world);
  sh->lo = std::min<uint64_t>((uint64_t)rank * sh->per, n);
  sh->hi = std::min<uint64_t>((uint64_t)sh->lo + sh->per, n);
  sh->w4 = (uint32_t)std::max<uint64_t>(1, ceil_div(n, 128));
  const uint32_t rows = sh->hi - sh->lo;
  sh->off.ctx = sh->nbr.ctx = sh->F.ctx = sh->acc.ctx = ctx;
  sh->acc.reserve(4);
  sh->off.reserve((uint64_t)rows + 2);
  SK_CUDA(cudaMemsetAsync(sh->off.p, 0, ((uint64_t)rows + 2) * 8, ctx->stream));
  SK_CUDA(cudaMemsetAsync(sh->acc.p, 0, 4 * 8, ctx->stream));
  const unsigned g = (unsigned)std::min<uint64_t>(ceil_div(m ? m : 1, BS_NT), (uint64_t)ctx->num_sms * 8);
  uint32_t* bad = reinterpret_cast<uint32_t*>(sh->acc.p + 3);
  k_shard_degree<<<g, BS_NT, 0, ctx->stream>>>(d_src, d_dst, m, n, sh->lo, sh->hi, sh->off.p, bad);
  after_launch(ctx, "k_shard_degree");
  scan_tile_sums(ctx, sh->off.p, rows);  // off[rows] = the rank's edges
  uint64_t edges, flag;
  read_u64(ctx, sh->off.p + rows, &edges, 1);
  read_u64(ctx, reinterpret_cast<const uint64_t*>(sh->acc.p + 3), &flag, 1);
  if ((uint32_t)flag) fail(STRATA_E_INVALID, "an edge endpoint is outside [0, n_nodes)");
  sh->n_edges = edges;
  sh->nbr.reserve(edges + 1);
  sh->F.reserve((uint64_t)sh->per * sh->w4 + 1);
  sh->src = d_src;
  sh->dst = d_dst;
  sh->m = m;
}

uint64_t tc_shard_seed(strata_ctx* ctx, strata_tc_shard* sh, uint4* Dmine, uint8_t* fmine) {
  const uint64_t vecs = (uint64_t)sh->per * sh->w4;
  SK_CUDA(cudaMemsetAsync(sh->F.p, 0, vecs * 16, ctx->stream));
  SK_CUDA(cudaMemsetAsync(Dmine, 0, vecs * 16, ctx->stream));
  SK_CUDA(cudaMemsetAsync(fmine, 0, sh->per, ctx->stream));
  DBuf<uint32_t> cursor(ctx, (uint64_t)(sh->hi - sh->lo) + 1);
  SK_CUDA(cudaMemsetAsync(cursor.p, 0, ((uint64_t)(sh->hi - sh->lo) + 1) * 4, ctx->stream));
  const unsigned g = (unsigned)std::min<uint64_t>(ceil_div(sh->m ? sh->m : 1, BS_NT), (uint64_t)ctx->num_sms * 8);
  k_shard_fill<<<g, BS_NT, 0, ctx->stream>>>(sh->src, sh->dst, sh->m, sh->n, sh->lo, sh->hi, sh->w4, sh->off.p,
                                             cursor.p, sh->nbr.p, reinterpret_cast<uint32_t*>(sh->F.p),
                                             reinterpret_cast<uint32_t*>(Dmine), fmine);
  after_launch(ctx, "k_shard_fill");
  SK_CUDA(cudaMemsetAsync(sh->acc.p, 0, 8, ctx->stream));
  k_shard_popc<<<(unsigned)std::min<uint64_t>(ceil_div(vecs ? vecs : 1, BS_NT), (uint64_t)ctx->num_sms * 8), BS_NT, 0,
                 ctx->stream>>>(sh->F.p, vecs, sh->acc.p);
  after_launch(ctx, "k_shard_popc");
  uint64_t c;
  read_u64(ctx, reinterpret_cast<const uint64_t*>(sh->acc.p), &c, 1);
  sync_and_check(ctx);
  // The rounds read only nbr / F: drop the caller's columns, which need not
  // outlive this call.
  sh->src = sh->dst = nullptr;
  sh->seeded = true;
  return c;  // |Δ0| of the rank's rows (distinct edges)
}

uint64_t tc_shard_round(strata_ctx* ctx, strata_tc_shard* sh, const uint4* Dfull, const uint8_t* ffull, uint4* Dmine,
                        uint8_t* fmine) {
  ShardView v{};
  v.rows = sh->hi - sh->lo;
  v.n = sh->n;
  v.W = sh->w4;
  v.ls = (int)lanes_shift(sh->w4);
  v.off = sh->off.p;
  v.nbr = sh->nbr.p;
  v.F = sh->F.p;
  v.delta = sh->acc.p;
  v.bytes = ctx->profiling ? sh->acc.p + 1 : nullptr;
  SK_CUDA(cudaMemsetAsync(sh->acc.p, 0, 16, ctx->stream));
  const uint64_t units = ceil_div((uint64_t)v.rows, 32u >> v.ls);
  int kh = -1;
  if (units) {
    const unsigned g = (unsigned)std::min<uint64_t>(ceil_div(units, BS_NT / 32), (uint64_t)ctx->num_sms * 8);
    kh = kprof_begin(ctx, K_SHARD_ROUND);
    k_shard_round<<<g, BS_NT, 0, ctx->stream>>>(v, Dfull, ffull, Dmine, fmine);
    kprof_end(ctx, kh, 0);
    after_launch(ctx, "k_shard_round");
  }
  uint64_t c[2];
  read_u64(ctx, reinterpret_cast<const uint64_t*>(sh->acc.p), c, 2);
  sync_and_check(ctx);
  if (kh >= 0) ctx->krecs[kh].bytes = c[1];
  return c[0];
}

void tc_shard_summary(strata_ctx* ctx, strata_tc_shard* sh, uint64_t* count, uint64_t* fp) {
  std::vector<uint64_t> tpw, tb;
  poly_tables((uint64_t)sh->w4 * 4, tpw, tb);
  DBuf<uint64_t> d_tpw(ctx, tpw.size()), d_tb(ctx, 1024);
  SK_CUDA(cudaMemcpyAsync(d_tpw.p, tpw.data(), tpw.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
  SK_CUDA(cudaMemcpyAsync(d_tb.p, tb.data(), 1024 * 8, cudaMemcpyHostToDevice, ctx->stream));
  SK_CUDA(cudaMemsetAsync(sh->acc.p, 0, 16, ctx->stream));
  const uint32_t rows = sh->hi - sh->lo;
  if (rows) {
    const unsigned g = (unsigned)std::min<uint64_t>(ceil_div(rows, BS_NT / 32), (uint64_t)ctx->num_sms * 8);
    k_shard_summary<<<g, BS_NT, 0, ctx->stream>>>(sh->F.p, rows, sh->w4, sh->lo, d_tpw.p, d_tb.p, sh->acc.p);
    after_launch(ctx, "k_shard_summary");
  }
  uint64_t h[2];
  read_u64(ctx, reinterpret_cast<const uint64_t*>(sh->acc.p), h, 2);
  sync_and_check(ctx);
  *count = h[0];
  *fp = h[1];
}

// ---- sparse Δ exchange -------------------------------------------------------
// When a round's Δ' is sparse, the ranks exchange only its nonzero 128-bit
// words: each rank packs (global word index, low 64 bits, high 64 bits)
// triples of its slice, the triples of all ranks are gathered, and every rank
// rebuilds the full Δ and its row flags from them.  The bytes on the wire are
// 24 per nonzero word instead of the whole slice.

// Nonzero words of the slice, written at claimed slots below `cap`; *count
// receives the total (which may exceed cap).
__global__ void k_shard_pack(const uint4* __restrict__ D, uint64_t words, uint64_t row0_word, uint64_t cap,
                             long long* __restrict__ out, unsigned long long* count) {
  const int lane = threadIdx.x & 31;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < words; base += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t w = base + threadIdx.x;
    uint4 q = make_uint4(0u, 0u, 0u, 0u);
    if (w < words) q = D[w];
    const bool nz = any4(q);
    const unsigned bal = __ballot_sync(kFull, nz);
    if (!bal) continue;
    unsigned long long first = 0;
    if (lane == 0) first = atomicAdd(count, (unsigned long long)__popc(bal));
    first = __shfl_sync(kFull, first, 0);
    if (nz) {
      const uint64_t slot = first + __popc(bal & lanemask_lt());
      if (slot < cap) {
        out[3 * slot] = (long long)(row0_word + w);
        out[3 * slot + 1] = (long long)(((uint64_t)q.y << 32) | q.x);
        out[3 * slot + 2] = (long long)(((uint64_t)q.w << 32) | q.z);
      }
    }
  }
}

// Scatter gathered triples into the (cleared) full Δ; entries with index -1
// are padding, indexes past the matrix are skipped and flagged.
__global__ void k_shard_unpack(const long long* __restrict__ in, uint64_t n, uint4* __restrict__ D, uint64_t words,
                               uint32_t W, uint8_t* __restrict__ flags, uint32_t* status) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const long long idx = in[3 * i];
    if (idx < 0) continue;
    if ((uint64_t)idx >= words) {
      atomicOr(status, ST_BOUNDS);
      continue;
    }
    const uint64_t lo = (uint64_t)in[3 * i + 1], hi = (uint64_t)in[3 * i + 2];
    D[idx] = make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
    flags[(uint64_t)idx / W] = 1;
  }
}

uint64_t tc_shard_pack(strata_ctx* ctx, strata_tc_shard* sh, const uint4* Dmine, int64_t* out, uint64_t cap) {
  const uint64_t per = sh->per;
  const uint64_t words = per * sh->w4;
  DBuf<uint64_t> cnt(ctx, 1);
  SK_CUDA(cudaMemsetAsync(cnt.p, 0, 8, ctx->stream));
  if (cap) SK_CUDA(cudaMemsetAsync(out, 0xff, cap * 24, ctx->stream));  // padding: index -1
  if (words) {
    const unsigned g = (unsigned)std::min<uint64_t>(ceil_div(words, 256), (uint64_t)ctx->num_sms * 8);
    k_shard_pack<<<g, 256, 0, ctx->stream>>>(Dmine, words, (uint64_t)sh->rank * per * sh->w4, cap,
                                             reinterpret_cast<long long*>(out),
                                             reinterpret_cast<unsigned long long*>(cnt.p));
    after_launch(ctx, "k_shard_pack");
  }
  uint64_t c;
  read_u64(ctx, cnt.p, &c, 1);
  sync_and_check(ctx);
  return c;
}

void tc_shard_unpack(strata_ctx* ctx, strata_tc_shard* sh, const int64_t* in, uint64_t n, uint4* Dfull,
                     uint8_t* ffull) {
  const uint64_t rows = (uint64_t)sh->per * sh->world, words = rows * sh->w4;
  SK_CUDA(cudaMemsetAsync(Dfull, 0, words * 16, ctx->stream));
  SK_CUDA(cudaMemsetAsync(ffull, 0, rows, ctx->stream));
  if (n) {
    const unsigned g = (unsigned)std::min<uint64_t>(ceil_div(n, 256), (uint64_t)ctx->num_sms * 8);
    k_shard_unpack<<<g, 256, 0, ctx->stream>>>(reinterpret_cast<const long long*>(in), n, Dfull, words, sh->w4,
                                               ffull, ctx->d_status);
    after_launch(ctx, "k_shard_unpack");
  }
  sync_and_check(ctx);
}

template uint64_t tc_bool_bitset<uint32_t>(strata_ctx*, const uint32_t*, const uint32_t*, uint64_t, uint64_t,
                                           uint64_t, int, DBuf<uint32_t>&, uint64_t*, uint64_t*);
template uint64_t tc_bool_bitset<uint64_t>(strata_ctx*, const uint32_t*, const uint32_t*, uint64_t, uint64_t,
                                           uint64_t, int, DBuf<uint64_t>&, uint64_t*, uint64_t*);

}  // namespace sk
