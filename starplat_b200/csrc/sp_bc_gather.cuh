// Multi-source Brandes without atomics on path counts (included by sp_bc.cu): the default
// form of sp_bc, sp_bfs_sigma and sp_bc_graphs.
//
// A batch's sources share every pass over the edges: per vertex, a 64-bit mask says for
// which sources it sits in a level, and a row of SW doubles holds their values. Both
// directions are the same gather: an entry (v, m) of level d walks v's edges, and where a
// neighbour w is in the neighbouring level for some of m's sources (mask & m), it adds
// w's row for them:
//   forward   sigma[v] = sum over in-neighbours w of level d - 1 of sigma[w]
//   backward  delta[v] = sigma[v] * sum over out-neighbours w of level d + 1 of q[w],
//             q = (1 + delta) / sigma
// The forward sweep used to push sigma with FP64 atomics (8.7 of 17.3 ms for 64 sources of
// R-MAT 20, against 4.1 ms for the gathering backward sweep). Now an entry's edges are
// walked once for both things the forward sweep needs of them: sigma from level d - 1, and
// the sources that reach a neighbour first at level d + 1 (64-bit atomicOr on masks).
//
// Layout. A row belongs to a group of LPE = SW / 4 lanes, four sources each, and a group
// works on its own entry, so a warp has 32 / LPE entries at once (with a warp per entry, 1000
// ER graphs of degree 20 took twice as long) and asks only for sectors that hold a source
// (about 9 of 64 sources are active per neighbour on R-MAT 20). The neighbours that matter
// are compacted in shared memory, and their rows come there asynchronously, RING ahead, so
// that what is in flight costs no registers. q overwrites sigma, which nobody reads once v's
// dependency is final: one row per vertex is all the state (512 bytes for 64 sources, where
// sigma, q and delta took 1280), and delta goes to BC as soon as it is known, in FP64.
//
// A level costs one team barrier for its walk and one for the masks of the next; entries
// above hub_deg edges are listed as hub_chunk-edge pieces when their level is formed (the
// list is kept for the backward sweep), and their partial sums meet in an FP64 scratch.
//
// Push form and this: R-MAT 20, 256 sources 71.2 -> 23.5 ms; 1000 ER graphs, 16 sources each
// 81.7 -> 33.3 ms (as one graph instead of a CTA per graph: with a CTA per graph this form
// took 67 ms); 20 ER graphs of up to 50 thousand vertices, 40 sources each 57 -> 1.9 ms; a
// 300 x 300 grid, one source 9.4 -> 6.3 ms. Slower than the push form: strips of many narrow
// levels, a team each (20 of 300 x 5 vertices 2.0 -> 2.5 ms, two of 1500 x 4 6.5 -> 11.4), as a
// level's walk is a longer chain here.
// What bounds it is the latency of masks and rows (issue 35 % active, L2 75 % hits, 9 GB of
// DRAM traffic a batch on R-MAT 20, far from its rate).
#pragma once

#include "sp_internal.cuh"

namespace sp {
namespace bc {

// What the forward sweep asks of a neighbour, in one 32-byte sector (three arrays cost an
// L2 sector each per edge): the sources that have reached the vertex up to the level being
// walked, those that reach it next, and its masks in the last even and odd level it was in.
// A level's mask is overwritten by that of the next level of the same parity, not cleared:
// a stale one belongs to sources that have the vertex two or more levels further up than
// the walk looks for, and no edge joins levels that far apart.
struct __align__(32) Masks {
  unsigned long long seen, nxt, lev[2];
};

struct Gather {
  const int32_t* off;   // out-edges of this graph (global edge indices)
  const int32_t* adj;
  const int32_t* roff;  // in-edges; the same arrays when sym
  const int32_t* radj;
  int sym;
  int vbase;            // first vertex id of this graph in adj
  int V;
  double* row;          // [V][SW] sigma, then q
  double* dacc;         // [V][SW] partial sums of split entries, zero between uses
  Masks* mask;          // [V]
  unsigned long long* back;      // [2][bstride] backward sweep: masks of the levels, by d & 1
  int bstride;
  int32_t* flv;         // [cap] vertices of the level lists
  unsigned long long* flm;       // [cap] their masks
  int cap;
  int* lo;              // [maxd + 2] level starts
  int maxd;
  int* cnt;             // entries appended
  double* bc;           // [V]
  int* err;             // this team's own: 1 a list is full, 2 too deep, 3 barrier timeout
  // entries with more than hub_deg edges, as pieces {vertex, entry, first edge, end}; pcap = 0:
  // none split.
  // [0] by out-edges, kept for all levels (plo / hlo: level starts); [1] by in-edges, for
  // the current level of a directed graph (two halves in turn).
  int hub_deg, hub_chunk;
  int pcap, hcap;
  int4* piece;          // [pcap]
  int32_t* hub;         // [hcap] split entries
  int* plo;             // [maxd + 2]
  int* hlo;             // [maxd + 2]
  int4* rpiece;         // [2][pcap]
  int32_t* rhub;        // [2][hcap]
  int* pc;              // counters: [0] pieces, [1] hubs, [2 + k] rpieces, [4 + k] rhubs of half k
};

constexpr int ORDER_MAX = 8192;  // k_order_sources: most sources of a call that are put in order
// Tuned on R-MAT 20 (64 sources a batch) / 1000 ER graphs of 16 sources, 4 CTAs of 256 threads
// (64 registers) an SM: RING 4 and UE 4 24.9 / 34.7 ms; RING 3 24.8 / 35.1; UE 2 24.9 / 39.3,
// UE 6 27.9 / 45.0, UE 8 31.9 / 38.3; 3 CTAs, RING 6 26.0 / 33.0; 5 CTAs (48 registers) 26.1 / 53.
// Rows loaded to registers instead, two at a time, took 28.9 / 44.2.
constexpr int RING = 4;           // rows on their way to shared memory per lane
constexpr int UE = 4;             // edges per lane of a group at a time

// Per-warp scratch in shared memory: each group's neighbours that matter.
struct Picked {
  double2 ring[RING][2][32];
  unsigned long long m[32 * UE];
  int32_t w[32 * UE];
};

__device__ __forceinline__ int ld_now(const int* p) { return *(const volatile int*)p; }

// 32 bytes at once (a sector, one request)
__device__ __forceinline__ Masks ld_masks(const Masks* p) {
  Masks x;
  asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];"
               : "=l"(x.seen), "=l"(x.nxt), "=l"(x.lev[0]), "=l"(x.lev[1])
               : "l"(p)
               : "memory");
  return x;
}
// Lane sl of a group of SW / 4 holds the sources 2 sl, 2 sl + 1 and SW / 2 + 2 sl, + 1 of a
// row: two 16-byte pieces, each next to its neighbour lanes', so that a request covers whole
// sectors. The two bits of each in a mask:
template <int SW>
__device__ __forceinline__ unsigned own_bits(unsigned long long m, int sl) {
  return ((unsigned)(m >> (2 * sl)) & 3u) | (((unsigned)(m >> (SW / 2 + 2 * sl)) & 3u) << 2);
}
// element j (0 .. 3) of the lane's part of a row
template <int SW>
__device__ __forceinline__ int own_at(int sl, int j) {
  return (j >> 1) * (SW / 2) + 2 * sl + (j & 1);
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// Adds the rows of a group's n picked neighbours to this lane's four sources; most = the
// largest n of the warp's groups. ring: RING neighbours per lane are on their way to shared
// memory at any time.
template <int SW>
__device__ __forceinline__ void gather_picked(const double* __restrict__ rows, const unsigned long long* pm,
                                              const int32_t* pw, int n, int most, int sl, double2 (*ring)[2][32],
                                              double (&acc)[4]) {
  const int lane = threadIdx.x & 31;
  const double* mine = rows + 2 * sl;
  unsigned nib[RING];
  auto issue = [&](int t, int u) {
    nib[u] = 0;
    if (t < n) {
      nib[u] = own_bits<SW>(pm[t], sl);
      const double* r = mine + (size_t)pw[t] * SW;
      if (nib[u] & 3u) cp_async16(&ring[u][0][lane], r);
      if (nib[u] & 12u) cp_async16(&ring[u][1][lane], r + SW / 2);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int u = 0; u < RING; ++u) issue(u, u);
  for (int t = 0; t < most; t += RING) {
#pragma unroll
    for (int u = 0; u < RING; ++u) {
      if (t + u >= most) break;
      asm volatile("cp.async.wait_group %0;" ::"n"(RING - 1) : "memory");
      if (nib[u] & 3u) {
        const double2 a = ring[u][0][lane];
        if (nib[u] & 1u) acc[0] += a.x;
        if (nib[u] & 2u) acc[1] += a.y;
      }
      if (nib[u] & 12u) {
        const double2 b = ring[u][1][lane];
        if (nib[u] & 4u) acc[2] += b.x;
        if (nib[u] & 8u) acc[3] += b.y;
      }
      issue(t + u + RING, u);
    }
  }
}

// sigma of entry (v, m): lane sl of its group has four sources.
template <int SW>
__device__ __forceinline__ void put_sigma(const Gather& G, int v, unsigned long long m, int sl,
                                          const double (&acc)[4]) {
  const unsigned nib = own_bits<SW>(m, sl);
  double* r = G.row + (size_t)v * SW + 2 * sl;
  if ((nib & 3u) == 3u)
    *reinterpret_cast<double2*>(r) = make_double2(acc[0], acc[1]);
  else if (nib & 3u)
    r[(nib >> 1) & 1u] = (nib & 1u) ? acc[0] : acc[1];
  if ((nib & 12u) == 12u)
    *reinterpret_cast<double2*>(r + SW / 2) = make_double2(acc[2], acc[3]);
  else if (nib & 12u)
    r[SW / 2 + ((nib >> 3) & 1u)] = (nib & 4u) ? acc[2] : acc[3];
}

// Dependency of entry (v, m) from the sum of its successors' q: q of v in sigma's place,
// and the dependencies of all its sources to BC. Called by whole warps (m = 0: no entry).
template <int SW>
__device__ __forceinline__ void put_delta(const Gather& G, int v, unsigned long long m, int sl,
                                          const double (&acc)[4]) {
  double sum = 0.0;
  const unsigned nib = own_bits<SW>(m, sl);
  double* r = G.row + (size_t)v * SW;
  // every load before the first store, which the compiler could not move them across
  double s[4], before = 0.0;
#pragma unroll
  for (int j = 0; j < 4; ++j) s[j] = (nib >> j) & 1u ? r[own_at<SW>(sl, j)] : 1.0;
  if (sl == 0 && m) before = G.bc[v];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if ((nib >> j) & 1u) {
      const double d = s[j] * acc[j];
      r[own_at<SW>(sl, j)] = (1.0 + d) / s[j];
      sum += d;
    }
#pragma unroll
  for (int o = SW / 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (sl == 0 && sum != 0.0) G.bc[v] = before + sum;
}

template <int SW>
__device__ __forceinline__ void add_partial(const Gather& G, int v, unsigned long long m, int sl,
                                            const double (&acc)[4]) {
  const unsigned nib = own_bits<SW>(m, sl);
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (((nib >> j) & 1u) && acc[j] != 0.0) atomicAdd(G.dacc + (size_t)v * SW + own_at<SW>(sl, j), acc[j]);
}

template <int SW>
__device__ __forceinline__ void take_partial(const Gather& G, int v, unsigned long long m, int sl,
                                             double (&acc)[4]) {
  const unsigned nib = own_bits<SW>(m, sl);
  double* r = G.dacc + (size_t)v * SW;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if ((nib >> j) & 1u) {
      acc[j] = r[own_at<SW>(sl, j)];
      r[own_at<SW>(sl, j)] = 0.0;
    }
}

// Entry i (vertex v, edges [b, b + d)) as pieces, for the lanes that want it. Called by a
// whole warp.
__device__ __forceinline__ void list_pieces(const Gather& G, bool want, int i, int v, int b, int d, int4* piece,
                                            int32_t* hub, int* pc, int* hc) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned all = __ballot_sync(FULL, want);
  if (!all) return;
  const int np = want ? (d + G.hub_chunk - 1) / G.hub_chunk : 0;
  int inc = np;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(FULL, inc, o);
    if (lane >= o) inc += t;
  }
  int p = 0, h = 0;
  if (lane == 31) {
    p = atomicAdd(pc, inc);
    h = atomicAdd(hc, __popc(all));
    if (h > G.hcap - __popc(all) || (unsigned)p > (unsigned)max(0, G.pcap - inc)) atomicExch(G.err, 1);
  }
  p = __shfl_sync(FULL, p, 31) + inc - np;
  h = __shfl_sync(FULL, h, 31) + __popc(all & ((1u << lane) - 1u));
  if (want && h < G.hcap) hub[h] = i;
  for (unsigned todo = all; todo; todo &= todo - 1) {
    const int l = __ffs(todo) - 1;
    const int ei = __shfl_sync(FULL, i, l), ev = __shfl_sync(FULL, v, l), eb = __shfl_sync(FULL, b, l);
    const int ed = __shfl_sync(FULL, d, l), ep = __shfl_sync(FULL, p, l), en = __shfl_sync(FULL, np, l);
    for (int k = lane; k < en; k += 32)
      if ((unsigned)(ep + k) < (unsigned)G.pcap)
        piece[ep + k] = make_int4(ev, ei, eb + k * G.hub_chunk, eb + min(ed, (k + 1) * G.hub_chunk));
  }
}

// One walk of a level: its entries [b, e) (those of at most hub_deg edges) and the pieces
// [p0, p1) of the others, a group of LPE lanes each, over the rows of off / adj.
//   pull      sum the rows of the neighbours whose mask in the neighbouring level (of parity
//             par) meets the entry's: FWD, path counts; otherwise q, for the entry's
//             dependencies. Pieces add theirs to the scratch.
//   discover  neighbours that a source has not seen get it in nxt, and are appended to the
//             level list the first time.
//   own       the entries' masks are set (parity par ^ 1).
// The next item's vertex and mask are loaded ahead.
template <int SW, bool FWD>
__device__ __noinline__ void sweep(const Gather& G, const int32_t* __restrict__ off, const int32_t* __restrict__ adj,
                                   int b, int e, const int4* piece, int p0, int p1, int par, bool own, bool pull,
                                   bool discover, int gw, int nw, Picked& pk) {
  const unsigned FULL = 0xffffffffu;
  constexpr int LPE = SW / 4, EPS = 32 / LPE;
  if (gw * EPS >= e - b + (p1 - p0)) return;  // no item for this warp
  const int lane = threadIdx.x & 31, g = lane / LPE, sl = lane % LPE;
  const unsigned lt = (1u << lane) - 1u;
  const unsigned group = (LPE == 32 ? FULL : (1u << (LPE & 31)) - 1u) << (g * LPE);
  const int n = e - b, total = n + (p1 - p0), vbase = G.vbase, step = nw * EPS;
  const int hub_deg = G.pcap ? G.hub_deg : INT32_MAX;
  const int32_t* flv = G.flv + b;
  const unsigned long long* flm = G.flm;
  Masks* mask = G.mask;
  const unsigned long long* level = G.back + (size_t)par * G.bstride;
  const double* rows = G.row;
  unsigned long long* pm = pk.m + g * LPE * UE;
  int32_t* pw = pk.w + g * LPE * UE;
  piece += p0 - n;
  int v1 = 0, b1 = 0, e1 = 0;
  unsigned long long m1 = 0;
  // loads of item x that need no other (a piece's entry stands in m1)
  auto ahead = [&](int x) {
    if (x < n) {
      v1 = flv[x];
      m1 = flm[b + x];
    } else if (x < total) {
      const int4 q = piece[x];
      v1 = q.x;
      m1 = (unsigned long long)q.y;
      b1 = q.z;
      e1 = q.w;
    }
  };
  ahead(gw * EPS + g);
  for (int x0 = gw * EPS; x0 < total; x0 += step) {
    const int x = x0 + g;
    int v = v1, eb = b1, ee = e1;
    unsigned long long m = m1;
    if (x < n) {
      eb = off[v];
      ee = off[v + 1];
    } else if (x < total) {
      m = flm[m];
    }
    ahead(x + step);
    if (x < n) {
      if (own && sl == 0) {
        if (FWD)
          mask[v].lev[par ^ 1] = m;
        else
          G.back[(size_t)(par ^ 1) * G.bstride + v] = m;
      }
      if (ee - eb > hub_deg) m = 0;  // its pieces do the work
    }
    if (x >= total || m == 0) {
      m = 0;
      ee = eb;
    }
    double acc[4] = {0, 0, 0, 0};
    const int rounds = __reduce_max_sync(FULL, (ee - eb + LPE * UE - 1) / (LPE * UE));
    for (int r = 0; r < rounds; ++r) {
      int w[UE];
      unsigned long long s[UE];
#pragma unroll
      for (int f = 0; f < UE; ++f) {
        const int j = eb + (r * UE + f) * LPE + sl;
        w[f] = j < ee ? adj[j] - vbase : -1;
      }
      if (FWD) {
        unsigned long long q[UE];
#pragma unroll
        for (int f = 0; f < UE; ++f) {
          s[f] = q[f] = 0ull;
          if (w[f] >= 0) {
            const Masks k = ld_masks(mask + w[f]);
            if (pull) s[f] = m & (par ? k.lev[1] : k.lev[0]);
            if (discover) q[f] = m & ~k.seen;
            if ((q[f] & ~k.nxt) == 0ull) q[f] = 0ull;  // there already: no atomic
          }
        }
        unsigned fresh = 0;
#pragma unroll
        for (int f = 0; f < UE; ++f)
          if (q[f] && atomicOr(&mask[w[f]].nxt, q[f]) == 0ull) fresh |= 1u << f;
        if (__any_sync(FULL, fresh)) {
          int at = 0, all = 0;
#pragma unroll
          for (int f = 0; f < UE; ++f) {
            const unsigned bal = __ballot_sync(FULL, (fresh >> f) & 1u);
            at += __popc(bal & lt);
            all += __popc(bal);
          }
          int base = 0;
          if (lane == 0) base = atomicAdd(G.cnt, all);
          at += __shfl_sync(FULL, base, 0);
#pragma unroll
          for (int f = 0; f < UE; ++f)
            if ((fresh >> f) & 1u) {
              if (at < G.cap)
                G.flv[at] = w[f];
              else
                atomicExch(G.err, 1);
              ++at;
            }
        }
      } else {
#pragma unroll
        for (int f = 0; f < UE; ++f) s[f] = pull && w[f] >= 0 ? m & level[w[f]] : 0ull;
      }
      if (pull) {
        int np = 0;  // of this group
#pragma unroll
        for (int f = 0; f < UE; ++f) {
          const unsigned bal = __ballot_sync(FULL, s[f] != 0ull) & group;
          if (s[f]) {
            const int p = np + __popc(bal & lt);
            pw[p] = w[f];
            pm[p] = s[f];
          }
          np += __popc(bal);
        }
        const int most = __reduce_max_sync(FULL, np);
        if (most) {
          __syncwarp();
          gather_picked<SW>(rows, pm, pw, np, most, sl, pk.ring, acc);
          __syncwarp();
        }
      }
    }
    if (FWD && !pull) continue;
    if (x >= n) {
      if (m) add_partial<SW>(G, v, m, sl, acc);
      m = 0;
    }
    if (FWD)
      put_sigma<SW>(G, v, m, sl, acc);
    else
      put_delta<SW>(G, v, m, sl, acc);
  }
}

// One batch of nsrc sources (local ids, distinct), by a team of whole warps; S gives its
// barrier and thread ranks. Source k has column k (nsrc <= SW), or cols[k] < SW, where two
// sources of one column are in different components (graphs of a disjoint union). lvl_out / sig_out: forward only, levels and path counts of
// every (source, vertex), source-major. G lies in shared memory.
template <int SW, class S>
__device__ bool gather_batch(const Gather& G, const int32_t* srcs, const int32_t* cols, int nsrc, S& sync,
                             Picked& pk, int32_t* lvl_out = nullptr, double* sig_out = nullptr) {
  constexpr int LPE = SW / 4, EPS = 32 / LPE;
  const int gt = sync.tid(), nt = sync.nthreads();
  const int lane = threadIdx.x & 31;
  const int gw = gt >> 5, nw = nt >> 5;
  if (gt == 0) {
    G.lo[0] = 0;
    G.lo[1] = nsrc;
    *G.cnt = nsrc;
    if (G.pcap) {
      for (int k = 0; k < 6; ++k) G.pc[k] = 0;
      G.plo[0] = G.hlo[0] = 0;
    }
  }
  for (int k = gt; k < nsrc; k += nt) {
    const int v = srcs[k], j = cols ? cols[k] : k;
    G.flv[k] = v;
    G.flm[k] = 1ull << j;
    G.row[(size_t)v * SW + j] = 1.0;
    G.mask[v].seen = 1ull << j;
  }
  if (!sync.sync()) return false;
  if (G.pcap) {  // the sources' pieces
    for (int k0 = gw * 32; k0 < nsrc; k0 += nw * 32) {
      const int k = k0 + lane;
      const int v = k < nsrc ? srcs[k] : 0;
      const int b = G.off[v], d = G.off[v + 1] - b;
      list_pieces(G, k < nsrc && d > G.hub_deg, k, v, b, d, G.piece, G.hub, G.pc, G.pc + 1);
    }
    if (!sync.sync()) return false;
  }
  // ---- forward
  // A level's counters are read once per CTA: while every warp of the grid read them (six
  // loads of one sector by 4,700 warps), they took a quarter of a deep graph's time (levels of
  // a 300 x 300 grid from one source 7.4 ms, 5.6 without).
  __shared__ int s_now[5];
  int d = 0, p0 = 0, h0 = 0, b = 0, e = nsrc;
  while (b != e) {
    if (d + 2 > G.maxd) {
      if (gt == 0) atomicExch(G.err, 2);
      return false;
    }
    int p1 = 0, h1 = 0, rp1 = 0, rh1 = 0;
    const int half = d & 1;
    if (G.pcap) {
      const int k = threadIdx.x;
      if (k < 4) s_now[k] = ld_now(G.pc + (k < 2 ? k : 2 * k - 2 + half));
      __syncthreads();
      p1 = min(s_now[0], G.pcap);
      h1 = min(s_now[1], G.hcap);
      rp1 = min(s_now[2], G.pcap);
      rh1 = min(s_now[3], G.hcap);
      if (gt == 0) {
        G.plo[d + 1] = p1;
        G.hlo[d + 1] = h1;
      }
    }
    const int par = (d & 1) ^ 1;  // of the level above
    sweep<SW, true>(G, G.off, G.adj, b, e, G.piece, p0, p1, par, true, G.sym && d > 0, true, gw, nw, pk);
    if (!G.sym && d > 0)
      sweep<SW, true>(G, G.roff, G.radj, b, e, G.rpiece + (size_t)half * G.pcap, 0, rp1, par, false, true, false,
                          gw, nw, pk);
    if (!sync.sync()) return false;
    // the next level's masks and pieces, and the path counts of this level's split entries
    if (threadIdx.x == 0) s_now[4] = ld_now(G.cnt);
    __syncthreads();
    const int c = min(s_now[4], G.cap);
    if (gt == 0) G.lo[d + 2] = c;
    if (G.pcap && !G.sym && gt == 0) G.pc[2 + half] = G.pc[4 + half] = 0;  // read by all before the barrier
    for (int i0 = e + gw * 32; i0 < c; i0 += nw * 32) {
      const int k = i0 + lane;
      const int w = k < c ? G.flv[k] : 0;
      if (k < c) {
        const Masks x = ld_masks(G.mask + w);
        G.flm[k] = x.nxt;
        *reinterpret_cast<ulonglong2*>(G.mask + w) = make_ulonglong2(x.seen | x.nxt, 0ull);  // seen, nxt
      }
      if (G.pcap) {
        const int ob = G.off[w], od = G.off[w + 1] - ob;
        list_pieces(G, k < c && od > G.hub_deg, k, w, ob, od, G.piece, G.hub, G.pc, G.pc + 1);
        if (!G.sym) {
          const int ib = G.roff[w], id = G.roff[w + 1] - ib;
          list_pieces(G, k < c && id > G.hub_deg, k, w, ib, id, G.rpiece + (size_t)(half ^ 1) * G.pcap,
                      G.rhub + (size_t)(half ^ 1) * G.hcap, G.pc + 2 + (half ^ 1), G.pc + 4 + (half ^ 1));
        }
      }
    }
    if (G.pcap && d > 0) {
      const int n = G.sym ? h1 - h0 : rh1;
      const int32_t* hub = G.sym ? G.hub + h0 : G.rhub + (size_t)half * G.hcap;
      for (int k = gw * EPS + lane / LPE; k < n; k += nw * EPS) {
        const int w = G.flv[hub[k]];
        const unsigned long long mk = G.flm[hub[k]];
        double acc[4] = {0, 0, 0, 0};
        take_partial<SW>(G, w, mk, lane % LPE, acc);
        put_sigma<SW>(G, w, mk, lane % LPE, acc);
      }
    }
    if (!sync.sync()) return false;
    p0 = p1;
    h0 = h1;
    b = e;
    e = c;
    ++d;
  }
  const int D = d;  // levels 0 .. D - 1
  if (lvl_out) {
    for (int i = gt; i < G.lo[D]; i += nt) {
      const int v = G.flv[i];
      const unsigned long long mk = G.flm[i];
      int lev = 0;
      while (G.lo[lev + 1] <= i) ++lev;
      for (int k = 0; k < nsrc; ++k)
        if ((mk >> k) & 1ull) {
          lvl_out[(size_t)k * G.V + v] = lev;
          sig_out[(size_t)k * G.V + v] = G.row[(size_t)v * SW + k];
        }
    }
  }
  // ---- backward, with masks of its own, which start and end at zero (the forward sweep's
  // hold levels above, which edges do reach)
  for (d = lvl_out ? 0 : D - 1; d >= 1; --d) {
    const bool last = d + 1 == D;  // nothing below: no edges to walk (level D has no masks)
    const int q0 = G.pcap && !last ? G.plo[d] : 0, q1 = G.pcap && !last ? G.plo[d + 1] : 0;
    sweep<SW, false>(G, G.off, G.adj, G.lo[d], G.lo[d + 1], G.piece, q0, q1, (d & 1) ^ 1, true, !last, false, gw,
                         nw, pk);
    const int nh = G.pcap ? G.hlo[d + 1] - G.hlo[d] : 0;
    if (!sync.sync()) return false;
    if (nh > 0) {  // the same for the whole team
      const int32_t* hub = G.hub + G.hlo[d];
      for (int k0 = gw * EPS; k0 < nh; k0 += nw * EPS) {
        const int k = k0 + lane / LPE;
        const int w = k < nh ? G.flv[hub[k]] : 0;
        const unsigned long long mk = k < nh ? G.flm[hub[k]] : 0ull;
        double acc[4] = {0, 0, 0, 0};
        take_partial<SW>(G, w, mk, lane % LPE, acc);
        put_delta<SW>(G, w, mk, lane % LPE, acc);
      }
      if (!sync.sync()) return false;
    }
  }
  // ---- the masks back to zero
  for (int v = gt; v < G.V; v += nt) {
    Masks z;
    z.seen = z.nxt = z.lev[0] = z.lev[1] = 0ull;
    G.mask[v] = z;
    G.back[v] = G.back[G.bstride + v] = 0ull;
  }
  // a full list (err 1) truncated this batch: the whole team reads its flag after its last
  // barrier. No other team has the same word, so nothing writes it after that barrier and
  // all leave together: a CTA that stayed would wait for, or read the shared memory of, one
  // that has left.
  if (!sync.sync()) return false;
  return ld_now(G.err) == 0;
}

// Sources of a call in descending out-degree (ties in the caller's order), so that a
// batch's sources reach most vertices at the same level: a vertex is then listed in fewer
// levels and the sources active on an edge share sectors. R-MAT 18, 256 sources in four
// batches: 390 against 512 thousand entries and 7.9 against 10.6 M gathered neighbours a
// batch. One thread per source, n compares each.
__global__ void k_order_sources(const int32_t* __restrict__ off, const int32_t* __restrict__ srcs, int n,
                                int32_t* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int s = srcs[i], d = off[s + 1] - off[s];
  int r = 0;
  for (int j = 0; j < n; ++j) {
    const int t = srcs[j], dj = off[t + 1] - off[t];
    r += dj > d || (dj == d && j < i);
  }
  out[r] = s;
}

}  // namespace bc
}  // namespace sp
