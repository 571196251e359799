// Triangle counting on symmetric graphs, in rank order (included by sp_tc.cu).
//
// Vertices are numbered by degree, largest first (rank 0 is the largest hub), and
// N+(u) = the neighbours of u of smaller rank, sorted. A triangle x < v < u (ranks) is
// found once, from its edge (u, v): x is in N+(v) and in the part of N+(u) before v. So v
// is the anchor: N+(v) is staged in shared memory, and for each neighbour u > v the
// prefix of N+(u) before v is looked up in it. Streaming prefixes costs
// sum d+(u) (d+(u) - 1) / 2 lookups, where streaming the whole N+ of each of an anchor's
// neighbours of higher degree (k_tc_warp, k_tc_bitmap) costs sum over edges of d+(v):
// R-MAT 20 1.23 against 4.42 billion, R-MAT 16 33 against 95 million, ER 2^20 of degree
// 32 152 against 178 million. Choosing the shorter of both per edge would save another
// 0.5 % on R-MAT and 8 % on ER.
//
// The lookups want one shared-memory load each. Hubs have the smallest ranks, so a bitmap
// of the first B ranks holds 99 % of what is looked up on R-MAT 20; ranks from B on go to
// a second, hashed bitmap, whose hits are checked in N+(v). That is 4 KB per warp, so a
// warp works alone, without block barriers, with 40 to 48 warps on an SM.
//
// A call, before (k_tc_bitmap_cta, k_tc_warp) and now: R-MAT 16 168 -> 64 us, R-MAT 20
// 21.0 -> 0.91 ms, ER 2^20 of degree 32 0.97 -> 0.50; per-vertex counts of R-MAT 18
// 11.1 -> 0.37 ms (a global atomic per triangle corner before). Making the plan takes 1.4
// ms on R-MAT 20, 1.0 for the other kernels' plan.
#pragma once
#include <cub/cub.cuh>

#include "sp_internal.cuh"

namespace sp {
namespace tcr {

constexpr int B = 16384;          // ranks with a bit of their own
constexpr int BITS = 14;          // log2 B
constexpr int WORDS = 2 * B / 32; // exact bits, then hashed bits
// Counting: 8 warps a CTA, 5 CTAs (33 KB of shared memory each) an SM; CU windows (32
// vectors of 4 elements) whose loads are in flight together.
// R-MAT 20: 0.91 ms at 2 windows and 5 CTAs, 0.95 at 4 and 4, 0.93 at 2 and 6 (spills);
// ER 2^20 of degree 8: 0.25 ms at 2 windows, 0.39 at 3. What bounds it is issue (60 %
// active on R-MAT 16: about 45 instructions per window of 128 elements) and the bank
// conflicts of the lookups; loading the next item ahead cost registers and time.
constexpr int CW = 8, CMINB = 5, CU = 2;
// Per-vertex counts: 24 warps a CTA share a histogram of the PH smallest ranks' counts,
// which most hits add to; 2 CTAs (111 KB) an SM. R-MAT 18 0.36 ms; 16 warps with 12288
// counters (one CTA an SM) 0.60, 20 with 6144 0.35, but 1.69 against 1.64 on R-MAT 20.
constexpr int PW = 24, PMINB = 2, PH = 3072, PU = 1;
constexpr int STRIPES = 32;       // item counters, 128 bytes apart
constexpr int RUN_MAX = 8;        // items taken at once, at most (16 runs a warp, or single items)
constexpr int CHUNK_MAX = 128;    // prefixes per work item (a multiple of 32)

// Rows of oadj start at multiples of 4 and are padded with -1, so a prefix is read in
// 16-byte vectors without a check of its end: what follows it in the row is v and larger
// ranks, which N+(v) does not hold.
// A work item is up to `chunk` tasks of one anchor v: {first task, tasks, first vector of
// N+(v) in oadj, its length}, and itemv = v. Task {first vector, vectors} is the prefix of N+(u)
// before v, for one neighbour u > v (tu).
struct Args {
  const int32_t* __restrict__ oadj;
  const int2* __restrict__ tasks;
  const int32_t* __restrict__ tu;
  const int4* __restrict__ items;
  const int32_t* __restrict__ itemv;
  const int32_t* __restrict__ n_items;
  int part, nparts;    // this part's items: part, part + nparts, ...
  unsigned long long* total;
  unsigned int* next;  // per stripe (every 32nd): runs handed out beyond each warp's first
  int* cf;             // PV: counts by rank
};

__device__ __forceinline__ unsigned hashed(unsigned x) { return B + ((x * 2654435761u) >> (32 - BITS)); }
__device__ __forceinline__ unsigned bit_of(unsigned x) { return x < B ? x : hashed(x); }

__device__ __forceinline__ bool in_list(const int32_t* __restrict__ a, int n, int x) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int m = (lo + hi) >> 1;
    if (a[m] < x) lo = m + 1; else hi = m;
  }
  return lo < n && a[lo] == x;
}

// The tasks [tb, te) of one item, whose anchor's list is own[0 .. n). Their vectors are
// flattened over the warp's lanes: of each 32 tasks, lane i holds one that starts at
// position excl_i, and in a window of 32 positions the starts are one bit each (a warp
// reduction), so a lane's owner is the number of starts up to it: no search, and every
// lane works whatever the lengths. COLD: N+(v) may hold ranks of B and above; otherwise
// what is read from B on shares the bit B, which is never set.
template <bool PV, bool COLD, int U>
__device__ __forceinline__ unsigned item_tasks(const Args& a, int tb, int te, const int32_t* __restrict__ own,
                                               int n, const unsigned* bm, int* s_off, int* hist, unsigned& hits_v) {
  const unsigned FULL = 0xffffffffu;
  const int lane = lane_id();
  const unsigned le = 0xffffffffu >> (31 - lane);
  const int4* __restrict__ rows = reinterpret_cast<const int4*>(a.oadj);
  unsigned cnt = 0;
  for (int g = tb; g < te; g += 32) {
    const int2 t = g + lane < te ? a.tasks[g + lane] : make_int2(0, 0);
    int inc = t.y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL, inc, o);
      if (lane >= o) inc += y;
    }
    const int total = __shfl_sync(FULL, inc, 31);
    const int excl = inc - t.y;
    const unsigned nz = __ballot_sync(FULL, t.y > 0);
    if (t.y > 0) s_off[__popc(nz & (le >> 1))] = t.x - excl;
    __syncwarp();
    int base = -1;       // the last task that starts before the window
    unsigned mine = 0;   // PV: hits in this lane's task
    const bool on = t.y > 0;
    // Q windows from w0 on; a single one is worked on alone (most of a low-degree graph's)
    auto windows = [&](auto q_const, int w0) {
      constexpr int Q = decltype(q_const)::value;
      int4 x[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const unsigned d = (unsigned)(excl - (w0 + 32 * q));
        const unsigned m = __reduce_or_sync(FULL, on && d < 32u ? 1u << d : 0u);
        const int task = base + __popc(m & le);
        base += __popc(m);
        const int pos = w0 + 32 * q + lane;
        x[q] = pos < total ? __ldg(rows + (s_off[task] + pos)) : make_int4(-1, -1, -1, -1);
      }
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        unsigned hits = 0;  // PV: one bit per element
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const unsigned e = (unsigned)(k == 0 ? x[q].x : k == 1 ? x[q].y : k == 2 ? x[q].z : x[q].w);
          const unsigned b = COLD ? bit_of(e) : min(e, (unsigned)B);
          unsigned hit = (bm[b >> 5] >> (b & 31u)) & 1u;
          if (COLD && hit && e >= B) hit = in_list(own, n, (int)e);
          if (PV)
            hits |= hit << k;
          else
            cnt += hit;
        }
        if (PV && __any_sync(FULL, hits)) {
          const int lo = max(excl - (w0 + 32 * q), 0), hi = min(inc - (w0 + 32 * q), 32);
          const unsigned seg = lo < hi ? (FULL << lo) & (FULL >> (32 - hi)) : 0u;  // the lanes of this lane's task
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            mine += __popc(__ballot_sync(FULL, (hits >> k) & 1u) & seg);
            if ((hits >> k) & 1u) {
              const int e = k == 0 ? x[q].x : k == 1 ? x[q].y : k == 2 ? x[q].z : x[q].w;
              if (e < PH)
                atomicAdd(hist + e, 1);
              else
                atomicAdd(a.cf + e, 1);
            }
          }
        }
      }
    };
    int w0 = 0;
    for (; total - w0 > 32; w0 += 32 * U) windows(std::integral_constant<int, U>{}, w0);
    if (w0 < total) windows(std::integral_constant<int, 1>{}, w0);
    if (PV && mine) {
      atomicAdd(a.cf + a.tu[g + lane], (int)mine);
      hits_v += mine;
    }
    __syncwarp();
  }
  return cnt;
}

template <bool PV, int NW, int MINB, int U>
__global__ void __launch_bounds__(NW * 32, MINB) k_count(Args a) {
  extern __shared__ unsigned s_dyn[];
  const int lane = lane_id(), w = warp_id();
  unsigned* bm = s_dyn + w * WORDS;
  int* s_off = (int*)(s_dyn + NW * WORDS) + w * 32;
  int* hist = (int*)(s_dyn + NW * (WORDS + 32));
  for (int i = lane; i < WORDS; i += 32) bm[i] = 0u;
  if (PV) {
    for (int i = threadIdx.x; i < PH; i += NW * 32) hist[i] = 0;
    __syncthreads();
  }
  __syncwarp();
  unsigned long long cnt = 0;
  const int nwarps = gridDim.x * NW;
  const int all = *a.n_items;
  const int n_mine = all > a.part ? (all - a.part + a.nparts - 1) / a.nparts : 0;
  // Items are taken in runs of consecutive ones (whose lists and tasks share lines), dealt
  // in STRIPES interleaved stripes, each with a counter that its warps ask one run ahead.
  // One counter for single items would bound a graph of many small anchors, at 1.35 G
  // increments a second: ER 2^20 of degree 32 (972 thousand items) 726 us, now 500; ER
  // 70,000 of degree 16 (65 thousand items) 67 us, now 44.
  const int run = min(RUN_MAX, max(1, n_mine / (nwarps * 16)));
  const int gwarp = blockIdx.x * NW + w, stripes = min(STRIPES, nwarps);
  const int c = gwarp % stripes, mates = (nwarps - c + stripes - 1) / stripes;
  int it = gwarp * run, end = min(it + run, n_mine), nxt = 0;
  if (lane == 0) nxt = (c + (mates + (int)atomicAdd(a.next + 32 * c, 1u)) * stripes) * run;
  while (it < n_mine) {
    const int i = a.part + it * a.nparts;
    const int4 item = a.items[i];
    const int v = a.itemv[i];
    const int32_t* __restrict__ own = a.oadj + 4ll * item.z;
    const int n = item.w, tb = item.x, te = item.x + item.y;
    for (int j = lane; j < n; j += 32) {
      const unsigned b = bit_of((unsigned)own[j]);
      atomicOr(&bm[b >> 5], 1u << (b & 31u));
    }
    __syncwarp();
    unsigned hv = 0;
    if (v <= B)  // N+(v) holds ranks below v
      cnt += item_tasks<PV, false, U>(a, tb, te, own, n, bm, s_off, hist, hv);
    else
      cnt += item_tasks<PV, true, U>(a, tb, te, own, n, bm, s_off, hist, hv);
    if (PV) {
      hv = __reduce_add_sync(0xffffffffu, hv);
      if (lane == 0 && hv) atomicAdd(a.cf + v, (int)hv);
    }
    for (int j = lane; j < n; j += 32) bm[bit_of((unsigned)own[j]) >> 5] = 0u;
    __syncwarp();
    if (++it == end) {
      it = __shfl_sync(0xffffffffu, nxt, 0);
      end = min(it + run, n_mine);
      if (lane == 0 && it < n_mine) nxt = (c + (mates + (int)atomicAdd(a.next + 32 * c, 1u)) * stripes) * run;
    }
  }
  if (PV) {
    __syncthreads();
    for (int i = threadIdx.x; i < PH; i += NW * 32)
      if (hist[i]) atomicAdd(a.cf + i, hist[i]);
  } else {
    cnt = warp_sum(cnt);
    if (lane == 0 && cnt) atomicAdd(a.total, cnt);
  }
}

constexpr size_t smem_bytes(int nw, bool pv) { return sizeof(int) * ((size_t)nw * (WORDS + 32) + (pv ? PH : 0)); }

// counts by rank -> by vertex
__global__ void k_by_vertex(int V, const int32_t* __restrict__ order, const int* __restrict__ cf,
                            int* __restrict__ out) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < V; k += gridDim.x * blockDim.x) out[order[k]] = cf[k];
}

// ---- the plan
__global__ void k_deg_keys(int V, const int32_t* __restrict__ off, unsigned maxdeg, unsigned* __restrict__ key,
                           int32_t* __restrict__ id) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    key[v] = maxdeg - (unsigned)(off[v + 1] - off[v]);
    id[v] = v;
  }
}

__global__ void k_rank(int V, const int32_t* __restrict__ order, int32_t* __restrict__ rank) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < V; k += gridDim.x * blockDim.x) rank[order[k]] = k;
}

// Edge-parallel passes over the CSR: a block takes EDGE_TILE consecutive entries, a thread
// four of them (adj is 256-byte aligned), whose rows it finds by one binary search between
// the tile's first and last row and steps of one. A search per entry took 0.27 + 0.30 ms
// for the two passes over 33.5 M entries, this 0.21 + 0.27.
template <class F>
__device__ __forceinline__ void edge_quads(int V, long long E, const int32_t* __restrict__ off,
                                           const int32_t* __restrict__ adj, F&& f) {
  static_assert(EDGE_TILE == 4 * 256, "four entries per thread of 256");
  __shared__ int s_v[2];
  for (long long t0 = (long long)blockIdx.x * EDGE_TILE; t0 < E; t0 += (long long)gridDim.x * EDGE_TILE) {
    const long long t1 = t0 + EDGE_TILE < E ? t0 + EDGE_TILE : E;
    if (threadIdx.x < 2) s_v[threadIdx.x] = edge_source(off, 0, V, threadIdx.x == 0 ? t0 : t1 - 1);
    __syncthreads();
    const long long i0 = t0 + 4 * (int)threadIdx.x;
    if (i0 < t1) {
      const int4 q = *reinterpret_cast<const int4*>(adj + i0);  // buffers carry 16 spare bytes
      const int u[4] = {q.x, q.y, q.z, q.w};
      const int n = (int)(t1 - i0 < 4 ? t1 - i0 : 4);
      int v = edge_source(off, s_v[0], s_v[1] + 1, i0), row[4];
      long long next = off[v + 1];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (k < n)
          while (i0 + k >= next) next = off[++v + 1];
        row[k] = v;
      }
      f(i0, n, row, u);
    }
    __syncthreads();
  }
}

// keep[i] = 1 when entry i (v -> u) has v as its anchor: rank v < rank u.
__global__ void __launch_bounds__(256) k_keep(int V, long long E, const int32_t* __restrict__ off,
                                              const int32_t* __restrict__ adj, const int32_t* __restrict__ rank,
                                              unsigned char* __restrict__ keep) {
  edge_quads(V, E, off, adj, [&](long long i0, int n, const int (&row)[4], const int (&u)[4]) {
    int ru[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) ru[k] = k < n ? rank[u[k]] : -1;
    uchar4 c;
    c.x = rank[row[0]] < ru[0];
    c.y = rank[row[1]] < ru[1];
    c.z = rank[row[2]] < ru[2];
    c.w = rank[row[3]] < ru[3];
    *reinterpret_cast<uchar4*>(keep + i0) = c;  // past E, where keep has room: 0
  });
  if (E % 4 == 0 && blockIdx.x == 0 && threadIdx.x == 0) keep[E] = 0;  // the scan's last entry
}

// Per rank: its tasks as an anchor (x), the length of its row N+ (y), the row's vectors (z)
// and its work items (w; none without a row of its own). Entry V is 0. The row's length is
// what the anchor's part and a self-loop leave of the degree, so one scan gives every
// position before the rows are sorted (searched for in the sorted rows, with scans of their
// own, they took 30 us more of a first call).
__global__ void k_row_sizes(int V, const int32_t* __restrict__ off, const int32_t* __restrict__ adj,
                            const int32_t* __restrict__ pos, const int32_t* __restrict__ rank, int chunk,
                            int4* __restrict__ size) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v <= V; v += gridDim.x * blockDim.x) {
    if (v == V) {
      size[V] = make_int4(0, 0, 0, 0);
      continue;
    }
    const int b = off[v], e = off[v + 1], t = pos[e] - pos[b];
    const int d = e - b - t - (in_list(adj + b, e - b, v) ? 1 : 0);
    size[rank[v]] = make_int4(t, d, (d + 3) / 4, d > 0 ? (t + chunk - 1) / chunk : 0);
  }
}

struct Plus4 {
  __host__ __device__ __forceinline__ int4 operator()(const int4& a, const int4& b) const {
    return make_int4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
  }
};

// Task p of anchor v: tu[p] = u, ta[p] = v, id[p] = p (in ascending v). After the last of them,
// keys that sort behind every rank. start: the scanned sizes.
__global__ void __launch_bounds__(256) k_emit(int V, long long E, const int32_t* __restrict__ off,
                                              const int32_t* __restrict__ adj, const int32_t* __restrict__ rank,
                                              const unsigned char* __restrict__ keep, const int32_t* __restrict__ pos,
                                              const int4* __restrict__ start, int mcap, int32_t* __restrict__ tu,
                                              int32_t* __restrict__ ta, int32_t* __restrict__ id) {
  edge_quads(V, E, off, adj, [&](long long i0, int n, const int (&row)[4], const int (&u)[4]) {
    const uchar4 c = *reinterpret_cast<const uchar4*>(keep + i0);
    const unsigned char kc[4] = {c.x, c.y, c.z, c.w};
    int at = pos[i0];  // kept entries before entry i0 + k
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k >= n || !kc[k]) continue;
      const int r = rank[row[k]];
      const int p = start[r].x + (at - pos[off[row[k]]]);
      tu[p] = rank[u[k]];
      ta[p] = r;
      id[p] = p;
      ++at;
    }
  });
  for (int p = start[V].x + blockIdx.x * 256 + threadIdx.x; p < mcap; p += gridDim.x * 256) {
    tu[p] = -1;
    id[p] = p;
  }
}

// The tasks stably sorted by u are the rows N+(u), each ascending: entry e of the sorted
// order is task sp[e], whose anchor is the element, and whose prefix is what stands
// before it in its row. A prefix has at most
// sqrt(2 m) < 2^16 elements, so its vectors go to their task as 2 bytes: the scattered
// writes stay in L2 (whole 8-byte tasks: 0.68 ms for 16.8 M, now 0.24 and 0.09 in k_tasks).
__global__ void k_rows(int V, const int32_t* __restrict__ su, const int32_t* __restrict__ sp,
                       const int32_t* __restrict__ ta, const int4* __restrict__ start, int32_t* __restrict__ oadj,
                       unsigned short* __restrict__ nvec) {
  const int m = start[V].x;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m; e += gridDim.x * blockDim.x) {
    const int p = sp[e], u = su[e];
    const int4 s = start[u];
    const int before = e - s.y;
    long long at = 4ll * s.z + before;
    oadj[at] = ta[p];
    if (e + 1 == start[u + 1].y)
      while (++at & 3) oadj[at] = -1;
    nvec[p] = (unsigned short)((before + 3) / 4);
  }
}

// The tasks, the work items of every anchor, and their number.
__global__ void k_tasks(int V, const int32_t* __restrict__ tu, const int4* __restrict__ start,
                        const unsigned short* __restrict__ nvec, int chunk, int2* __restrict__ tasks,
                        int4* __restrict__ items, int32_t* __restrict__ itemv, int32_t* __restrict__ n_items) {
  const int m = start[V].x, t0 = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  for (int p = t0; p < m; p += nt) tasks[p] = make_int2(start[tu[p]].z, nvec[p]);
  for (int v = t0; v < V; v += nt) {
    const int4 s = start[v], e = start[v + 1];
    for (int k = s.w, t = s.x; k < e.w; ++k, t += chunk) {
      items[k] = make_int4(t, min(chunk, e.x - t), s.z, e.y - s.y);
      itemv[k] = v;
    }
    if (v == V - 1) *n_items = e.w;
  }
}

struct Plus {
  __host__ __device__ __forceinline__ int32_t operator()(int32_t x, int32_t y) const { return x + y; }
};

constexpr int OUT_ITEMS = 16 + 16 * STRIPES;  // 8-byte words before it are cleared by each call

struct Plan {
  Arena mem;
  dspan<int32_t> order, oadj, tu, itemv;
  dspan<int2> tasks;
  dspan<int4> items;
  dspan<unsigned long long> out;  // [0] count, [16 ..] the item counters, [OUT_ITEMS] (int32) the items
  dspan<int> cf;                  // counts by rank
  int items_max = 0;              // at most this many items
  bool built = false;
};

inline int bits_for(unsigned x) {  // bits of values up to x
  int b = 1;
  while (b < 32 && (x >> b)) ++b;
  return b;
}

inline int build(sp_graph* g, Plan& P) {
  if (P.built) return SP_OK;
  cudaStream_t s = g->stream;
  const int V = g->V;
  const long long E = g->E;
  const long long mcap = E / 2;  // each edge is there in both directions
  const int chunk = (int)std::min<long long>(
      CHUNK_MAX, std::max<long long>(32, mcap / ((long long)num_sms() * CW * CMINB * 4) / 32 * 32));
  const int vbits = bits_for((unsigned)std::max(1, V - 1));
  const int dbits = bits_for((unsigned)std::max(1, g->max_out_deg));
  // what the build alone needs, in one block
  Arena tmp;
  dspan<unsigned> key, skey;
  dspan<int32_t> id, rank, pos, ta, tid, su, sp;
  dspan<int4> size, start;
  dspan<unsigned char> keep, cubt;
  dspan<unsigned short> nvec;
  size_t t1 = 0, t2 = 0, t3 = 0, t4 = 0;
  SP_CHECK_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, t1, (unsigned*)nullptr, (unsigned*)nullptr,
                                                (int32_t*)nullptr, (int32_t*)nullptr, V, 0, dbits, s));
  SP_CHECK_CUDA(cub::DeviceScan::ExclusiveScan(nullptr, t2, (unsigned char*)nullptr, (int32_t*)nullptr, Plus{},
                                               (int32_t)0, (int)(E + 1), s));
  SP_CHECK_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, t3, (int32_t*)nullptr, (int32_t*)nullptr, (int32_t*)nullptr,
                                                (int32_t*)nullptr, (int)mcap, 0, vbits, s));
  SP_CHECK_CUDA(cub::DeviceScan::ExclusiveScan(nullptr, t4, (int4*)nullptr, (int4*)nullptr, Plus4{},
                                               make_int4(0, 0, 0, 0), V + 1, s));
  tmp.want(key, V);
  tmp.want(skey, V);
  tmp.want(id, V);
  tmp.want(rank, V);
  tmp.want(size, V + 1);
  tmp.want(start, V + 1);
  tmp.want(keep, E + 4);
  tmp.want(nvec, mcap);
  tmp.want(pos, E + 1);
  tmp.want(ta, mcap);
  tmp.want(tid, mcap);
  tmp.want(su, mcap);
  tmp.want(sp, mcap);
  tmp.want(cubt, std::max({t1, t2, t3, t4}));
  SP_TRY(tmp.commit());
  P.mem.want(P.order, V);
  P.mem.want(P.oadj, (size_t)mcap + 3 * (size_t)std::min<long long>(V, mcap));
  P.mem.want(P.tu, mcap);
  P.mem.want(P.tasks, mcap);
  const long long imax = mcap / chunk + std::min<long long>(V, mcap);  // an anchor has a list, so an edge
  P.mem.want(P.items, imax);
  P.mem.want(P.itemv, imax);
  P.mem.want(P.out, OUT_ITEMS + 1);
  P.mem.want(P.cf, V);
  if (const int st = P.mem.commit()) {
    P.mem.reqs.clear();
    P.mem.size = 0;
    return st;
  }
  const int vg = std::max(1, std::min((V + 256) / 256, num_sms() * 8));
  const int eg = (int)std::max<long long>(1, std::min<long long>((E + EDGE_TILE - 1) / EDGE_TILE, num_sms() * 8));
  k_deg_keys<<<vg, 256, 0, s>>>(V, g->off.p, (unsigned)std::max(1, g->max_out_deg), key.p, id.p);
  SP_CHECK_LAUNCH();
  SP_CHECK_CUDA(cub::DeviceRadixSort::SortPairs(cubt.p, t1, key.p, skey.p, id.p, P.order.p, V, 0, dbits, s));
  k_rank<<<vg, 256, 0, s>>>(V, P.order.p, rank.p);
  SP_CHECK_LAUNCH();
  if (E > 0) {
    k_keep<<<eg, 256, 0, s>>>(V, E, g->off.p, g->adj.p, rank.p, keep.p);
    SP_CHECK_LAUNCH();
  } else {
    SP_CHECK_CUDA(cudaMemsetAsync(keep.p, 0, 1, s));
  }
  SP_CHECK_CUDA(cub::DeviceScan::ExclusiveScan(cubt.p, t2, keep.p, pos.p, Plus{}, (int32_t)0, (int)(E + 1), s));
  k_row_sizes<<<vg, 256, 0, s>>>(V, g->off.p, g->adj.p, pos.p, rank.p, chunk, size.p);
  SP_CHECK_LAUNCH();
  SP_CHECK_CUDA(cub::DeviceScan::ExclusiveScan(cubt.p, t4, size.p, start.p, Plus4{}, make_int4(0, 0, 0, 0), V + 1, s));
  // the tasks: mcap, less the self-loops' entries
  const int mg = (int)std::max<long long>(1, std::min<long long>((std::max<long long>(mcap, V) + 255) / 256, num_sms() * 8));
  if (mcap > 0) {
    k_emit<<<eg, 256, 0, s>>>(V, E, g->off.p, g->adj.p, rank.p, keep.p, pos.p, start.p, (int)mcap, P.tu.p, ta.p,
                              tid.p);
    SP_CHECK_LAUNCH();
    SP_CHECK_CUDA(cub::DeviceRadixSort::SortPairs(cubt.p, t3, P.tu.p, su.p, tid.p, sp.p, (int)mcap, 0, vbits, s));
    k_rows<<<mg, 256, 0, s>>>(V, su.p, sp.p, ta.p, start.p, P.oadj.p, nvec.p);
    SP_CHECK_LAUNCH();
  }
  k_tasks<<<mg, 256, 0, s>>>(V, P.tu.p, start.p, nvec.p, chunk, P.tasks.p, P.items.p, P.itemv.p,
                             (int32_t*)(P.out.p + OUT_ITEMS));
  SP_CHECK_LAUNCH();
  g_launches += 4;  // the scans and sorts
  P.items_max = (int)std::min<long long>(imax, INT32_MAX);
  P.built = true;
  return SP_OK;
}

}  // namespace tcr
}  // namespace sp
