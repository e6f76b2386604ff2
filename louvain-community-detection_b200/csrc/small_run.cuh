// small_run.cuh -- the remaining levels of a small single graph in one
// launch (included by move.cu, inside its anonymous namespace).
//
// A small level's pass is a chain of up to nine dependent launches (bucket
// steps, modularity) of 4-9 us each whatever its size, and a level costs two
// host waits and about forty more launches for its set-up and contraction.
// Here one thread-block cluster runs every level to the end of the run
// (main.cu:43-48): set-up, the pass loop (modularity.cu:466-508) and the
// contraction (aggregation.cu:387-462).  What bounds it is latency (an L2
// round trip costs 700 cycles and more), so the community state is replicated
// in every block's shared memory, beside the rows of the block's own vertices
// (v % blocks == rank) as far as they fit.  A block decides for its vertices
// and writes their proposals into every block's shared memory; after the
// step's one cluster barrier every block applies all of the step's moves to
// its own copy.  (With the state in L2, a step at 1,000 vertices took 5 us.)
// The decisions are the bodies of the standalone kernels.  The contraction
// renumbers and groups members in every block redundantly, merges a community
// per warp or block in a shared table and takes its staging ranges from a
// bump counter: two barriers.
//
// Every block takes the same branches around barriers: what decides them
// (class counts, sums, Q) is computed by each block from the same values.

constexpr int kSmallThreads = 1024;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmallCtas = 16;
constexpr uint32_t kSmallWarpMerge = 128;  // entries of a community merged by a warp
// Dynamic shared memory for levels of up to cap vertices on `ctas` blocks:
// tables (kSmallArena), the state (tot, comm, sz, k, cdeg, prop_all, cls),
// row offsets, this block's class lists and proposals; what is left up to
// kSmallSmem holds entries of its rows (8 bytes each).
constexpr uint32_t kSmallArena = 4096u * (uint32_t)kSlotBytes;
constexpr uint32_t kSmallSmem = 216u * 1024;
__host__ __device__ constexpr uint32_t small_own(uint32_t cap, uint32_t ctas) {
  return (cap + ctas - 1) / ctas;
}
__host__ __device__ constexpr uint32_t small_fixed(uint32_t cap, uint32_t ctas) {
  return kSmallArena + 29 * cap + 8 * (cap + 2) + 8 * small_own(cap, ctas) + 64;
}
static_assert(kSmallMaxN <= 2048 && kBlockTabSmem <= (int)kSmallArena &&
                  kSmallWarps * 128 * kSlotBytes <= (int)kSmallArena &&
                  small_fixed(kSmallMaxN, 8) + 64 * 1024 <= kSmallSmem,
              "tables of 2 cap slots fit the arena; rows have 64 KB and more");

struct SmallCtx {
  PassDesc D;       // as the move bodies read it: state and rows in shared memory
  LevelView G;      // the level's CSR in global memory
  LevelScalars sc;
  double red[kSmallWarps][3];
  double shares[2][kSmallCtas][3];  // written by every block (alternating)
  unsigned long long scan[33];
  uint32_t cls_all[kClasses + 1];   // the level's class counts
  uint32_t cls_own[kClasses + 1];   // this block's
  uint32_t cursor[kClasses + 1];
  uint32_t bump;
  uint32_t row_cursor;
};
struct SmallMem {  // dynamic shared memory
  unsigned char* arena;
  double* tot;
  uint64_t* off;
  uint32_t *comm, *sz, *cdeg, *order, *prop, *prop_all;
  float* k;
  uint32_t* col;  // [ent] entries of the block's own rows
  float* w;
  unsigned char* cls;
  uint32_t ent;
};

__device__ __forceinline__ void small_sync(uint32_t ctas) {
  if (ctas == 1) {
    __syncthreads();
  } else {
    asm volatile(
        "barrier.cluster.arrive.release;\n\t"
        "barrier.cluster.wait.acquire;" ::: "memory");
  }
}

// Stores into the same place of block `r`'s shared memory.
__device__ __forceinline__ uint32_t small_remote(const void* p, uint32_t r) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;"
      : "=r"(a)
      : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(r));
  return a;
}
__device__ __forceinline__ void small_store(uint32_t a, uint32_t x) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(x) : "memory");
}
__device__ __forceinline__ void small_store(uint32_t a, double x) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(x) : "memory");
}

// This block's sums of three values into every block's shares[rank].
__device__ __forceinline__ void small_share(SmallCtx& S, uint32_t buf, double a, double b,
                                            double c, uint32_t rank, uint32_t ctas) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  a = group_sum<32>(a);
  b = group_sum<32>(b);
  c = group_sum<32>(c);
  if (lane == 0) {
    S.red[wib][0] = a;
    S.red[wib][1] = b;
    S.red[wib][2] = c;
  }
  __syncthreads();
  if (wib == 0) {
    a = group_sum<32>(S.red[lane][0]);
    b = group_sum<32>(S.red[lane][1]);
    c = group_sum<32>(S.red[lane][2]);
    if (ctas == 1) {
      if (lane == 0) {
        S.shares[buf][0][0] = a;
        S.shares[buf][0][1] = b;
        S.shares[buf][0][2] = c;
      }
    } else if ((uint32_t)lane < ctas) {
      const uint32_t p = small_remote(&S.shares[buf][rank][0], lane);
      small_store(p, a);
      small_store(p + 8, b);
      small_store(p + 16, c);
    }
  }
}

// The blocks' shares added, the same tree in every warp of every block.
__device__ __forceinline__ double small_gather(const SmallCtx& S, uint32_t buf, int k,
                                               uint32_t ctas) {
  const uint32_t i = threadIdx.x & (kSmallCtas - 1);  // both halves of a warp alike
  return group_sum<kSmallCtas>(i < ctas ? S.shares[buf][i][k] : 0.0);
}

// Classes of all vertices, singleton communities, this block's class lists,
// and its rows in shared memory (M.off, M.col, M.w) when they fit: returns
// whether they do.  A row's bounds sit at M.off[v] and M.off[v + 1] as in a
// CSR; with more than one block v + 1 is another block's vertex.
__device__ __noinline__ bool small_classes(SmallCtx& S, const SmallMem& M, const LevelView& G,
                                           uint32_t rank, uint32_t ctas) {
  const uint32_t n = G.n;
  const uint64_t* off = G.off;
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  if (tid <= kClasses) S.cls_all[tid] = S.cls_own[tid] = 0u;
  if (tid == 0) S.row_cursor = 0u;
  __syncthreads();
  for (uint32_t b = 0; b < n; b += kSmallThreads) {  // block-uniform
    const uint32_t v = b + tid;
    int c = 0;
    if (v < n) {
      c = move_class_of_degree(off[v + 1] - off[v]);
      M.cls[v] = (unsigned char)c;
      M.comm[v] = v;
      M.sz[v] = 1u;
    }
    const bool own = v % ctas == rank;
    for (int q = 1; q <= 8; q++) {
      const unsigned all = __ballot_sync(kFull, c == q);
      const unsigned mine = __ballot_sync(kFull, c == q && own);
      if (lane == 0 && all) atomicAdd(&S.cls_all[q], (uint32_t)__popc(all));
      if (lane == 0 && mine) atomicAdd(&S.cls_own[q], (uint32_t)__popc(mine));
    }
  }
  __syncthreads();
  if (tid == 0) {
    uint32_t run = 0;
    for (int q = 1; q <= 8; q++) {
      S.D.A.P.cls_start[q] = S.cursor[q] = run;
      run += S.cls_own[q];
    }
  }
  __syncthreads();
  // the own vertices 32 to a warp: class lists and local row bounds
  const uint32_t own_n = n > rank ? (n - rank + ctas - 1) / ctas : 0u;
  for (uint32_t i0 = (tid >> 5) * 32; i0 < own_n; i0 += kSmallThreads) {
    const uint32_t i = i0 + lane, v = i * ctas + rank;
    uint64_t s = 0;
    uint32_t d = 0;
    if (i < own_n) {
      s = off[v];
      d = (uint32_t)(off[v + 1] - s);
      const int c = M.cls[v];
      if (c) M.order[atomicAdd(&S.cursor[c], 1u)] = v;
    }
    uint32_t incl = d;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, incl, o);
      if (lane >= (uint32_t)o) incl += y;
    }
    uint32_t base = 0;
    if (lane == 31) base = atomicAdd(&S.row_cursor, incl);
    base = __shfl_sync(kFull, base, 31);
    if (i < own_n) {  // one block: its rows lie as they do in the CSR
      const uint64_t ls = ctas == 1 ? s : base + incl - d;
      M.off[v] = ls;
      M.off[v + 1] = ls + d;
    }
  }
  __syncthreads();
  return S.row_cursor <= M.ent;
}

// Row sums of this block's vertices into k_out (global), with the weight of
// their self-loops; the rows themselves into shared memory when they fit.
// G lanes per row.
template <int G>
__device__ __noinline__ void small_rows(const LevelView& L, const SmallMem& M, bool fits,
                                        float* k_out, uint32_t rank, uint32_t ctas, double& msum,
                                        double& asq, double& self) {
  const uint32_t n = L.n;
  const int gl = threadIdx.x & (G - 1);
  constexpr uint32_t per = kSmallThreads / G;
  for (uint32_t i0 = 0; i0 * ctas < n; i0 += per) {  // block-uniform
    const uint32_t r = (i0 + threadIdx.x / G) * ctas + rank;
    double x = 0.0, sl = 0.0;
    if (r < n) {
      const uint64_t s = L.off[r], ls = M.off[r];
      const uint32_t d = (uint32_t)(L.off[r + 1] - s);
      for (uint32_t j0 = gl; j0 < d; j0 += 4 * G) {
        uint32_t c[4];
        float w[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const uint32_t j = j0 + q * G;
          c[q] = j < d ? L.col[s + j] : kEmptyKey;
          w[q] = j < d ? L.w[s + j] : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
          if (c[q] == kEmptyKey) continue;
          x += (double)w[q];
          if (c[q] == r) sl += (double)w[q];
          if (fits) {
            M.col[ls + j0 + q * G] = c[q];
            M.w[ls + j0 + q * G] = w[q];
          }
        }
      }
    }
    x = group_sum<G>(x);
    self += sl;
    if (r < n && gl == 0) {
      const float kf = (float)x;
      k_out[r] = kf;
      msum += (double)kf;
      asq += (double)kf * (double)kf;
    }
  }
}

template <int G, int MODE>
__device__ __noinline__ void small_lanes(const PassDesc* D, int cls, unsigned char* smem) {
  small_body<G, MODE, kSmallThreads>(
      D, cls, 0, 1, reinterpret_cast<double(*)[32]>(smem),
      reinterpret_cast<uint32_t(*)[64]>(smem + kSmallWarps * 32 * sizeof(double)));
}
// The table phases add in FP64 whatever the weights: a level of this size has
// few rows for them.
template <int T, int MAXW, int MODE>
__device__ __noinline__ void small_warp(const PassDesc* D, int cls, unsigned char* smem,
                                        uint32_t warps) {
  warp_rows<T, MAXW, MODE, double, true>(D, cls, 0, 1, smem, StepIO{}, warps);
}
template <int MODE>
__device__ __noinline__ void small_block(const PassDesc* D, int cls, unsigned char* smem) {
  __shared__ typename BestOf<ModeOf<MODE>::kPrec>::T rb[kSmallWarps];
  __shared__ double ro[kSmallWarps];
  __shared__ uint16_t claims[kSmallWarps * claim_list(kHubSmemMaxDeg, kSmallThreads)];
  block_rows<MODE, double, kSmallThreads, kHubSmemSlots, (int)kHubSmemMaxDeg>(
      D, cls, 0, 1, smem, rb, ro, claims, StepIO{});
}

// One vertex's move into this block's copy of the state.  The lanes moving
// into (out of) the community of the warp's first mover add as one: many
// vertices joining one community would otherwise queue on one slot's FP64
// compare-and-swap.  Called by whole warps.
__device__ __forceinline__ void small_apply(const SmallMem& M, bool mv, uint32_t v, uint32_t oc,
                                            uint32_t nc) {
  const int lane = threadIdx.x & 31;
  const unsigned any = __ballot_sync(kFull, mv);
  if (!any) return;
  const double kv = mv ? (double)M.k[v] : 0.0;
  if (mv) M.comm[v] = nc;
  const int lead = __ffs(any) - 1;
#pragma unroll
  for (int side = 0; side < 2; side++) {
    const uint32_t c = side ? nc : oc;
    const double x = side ? kv : -kv;
    const uint32_t one = side ? 1u : 0xFFFFFFFFu;
    const uint32_t cl = __shfl_sync(kFull, c, lead);
    const unsigned m = __ballot_sync(kFull, mv && c == cl);
    if (__popc(m) > 1) {
      const double y = group_sum<32>((m >> lane & 1u) ? x : 0.0);
      if (lane == lead) {
        atomicAdd(&M.sz[cl], one * (uint32_t)__popc(m));
        atomicAdd(&M.tot[cl], y);
      }
    }
    if (mv && !(__popc(m) > 1 && (m >> lane & 1u))) {
      atomicAdd(&M.sz[c], one);
      atomicAdd(&M.tot[c], x);
    }
  }
}

// This block's shares of the intra-community weight (its vertices' rows) and
// of the squared totals.
template <int G>
__device__ __noinline__ void small_q_share(const LevelView& L, uint32_t rank, uint32_t ctas,
                                           double& intra, double& asq) {
  const uint32_t n = L.n;
  const int gl = threadIdx.x & (G - 1);
  constexpr uint32_t per = kSmallThreads / G;
  double a = 0.0, b = 0.0;
  for (uint32_t i = threadIdx.x / G; i * ctas + rank < n; i += per) {
    const uint32_t r = i * ctas + rank;
    const uint64_t s = L.off[r], e = L.off[r + 1];
    const uint32_t c = L.comm[r];
#pragma unroll 4
    for (uint64_t j = s + gl; j < e; j += G)
      if (L.comm[L.col[j]] == c) a += (double)L.w[j];
  }
  for (uint32_t c = threadIdx.x * ctas + rank; c < n; c += kSmallThreads * ctas) {
    const double x = L.tot[c];
    b += x * x;
  }
  intra = a;
  asq = b;
}

// One community's member rows into a table: nthr threads from tid, eight
// lanes per member row; entries inside the community summed in registers.
// cnew: new id of every vertex.
__device__ __forceinline__ void small_merge_rows(const LevelView& L, const uint32_t* cnew,
                                                 const uint32_t* members, uint32_t msz,
                                                 uint32_t cn, uint32_t tid, uint32_t nthr,
                                                 uint32_t* keys, double* vals, uint32_t mask,
                                                 double& hot, bool& hot_seen) {
  const uint32_t gl = tid & 7;
  for (uint32_t i = tid >> 3; i < msz; i += nthr >> 3) {
    const uint32_t v = members[i];
    const uint64_t s = L.off[v], e = L.off[v + 1];
#pragma unroll 2
    for (uint64_t j = s + gl; j < e; j += 8) {
      const uint32_t key = cnew[L.col[j]];
      const double w = (double)L.w[j];
      if (key == cn) {
        hot += w;
        hot_seen = true;
      } else {
        atomicAdd(&vals[table_insert(keys, mask, key, L.sc)], w);
      }
    }
  }
}

// Contracts the level's communities into CSR buffer `next`; the new vertex
// and entry counts to every thread.  Afterwards M.comm holds every vertex's
// new id and the rest of the state is scratch.
__device__ __noinline__ void small_contract(const SmallRunArgs& A, SmallCtx& S, const SmallMem& M,
                                            uint32_t rank, uint32_t ctas, int next,
                                            uint32_t n_first, uint32_t bump, uint32_t* new_n_out,
                                            uint64_t* new_e_out) {
  const LevelView& L = S.G;
  const uint32_t n = L.n;
  const uint32_t tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const uint32_t gt = rank * kSmallThreads + tid, gn = ctas * kSmallThreads;
  uint32_t* new_id = reinterpret_cast<uint32_t*>(M.tot);  // [n] by old id
  uint32_t* mstart = new_id + n;                          // [n] by new id
  uint32_t* members = reinterpret_cast<uint32_t*>(M.k);   // [n]
  uint32_t* cursor = reinterpret_cast<uint32_t*>(M.arena);
  unsigned long long carry = 0;
  for (uint32_t b = 0; b < n; b += kSmallThreads) {  // block-uniform
    const uint32_t c = b + tid;
    const uint32_t sz = c < n ? M.sz[c] : 0u;
    unsigned long long total;
    const unsigned long long pre =
        block_exclusive_scan<unsigned long long>(sz ? (1ull << 32) | sz : 0ull, S.scan, &total) +
        carry;
    if (c < n) {
      new_id[c] = (uint32_t)(pre >> 32);
      if (sz) mstart[pre >> 32] = (uint32_t)pre;
      cursor[c] = 0u;
      M.cdeg[c] = 0u;
    }
    carry += total;
  }
  const uint32_t new_n = (uint32_t)(carry >> 32);
  __syncthreads();
  for (uint32_t v = tid; v < n; v += kSmallThreads) {
    const uint32_t nid = new_id[M.comm[v]];
    M.comm[v] = nid;
    members[mstart[nid] + atomicAdd(&cursor[nid], 1u)] = v;
    atomicAdd(&M.cdeg[nid], (uint32_t)(L.off[v + 1] - L.off[v]));
  }
  __syncthreads();
  for (uint32_t v = gt; v < n_first; v += gn) A.map[v] = M.comm[A.map[v]];
  const uint32_t* cnew = M.comm;
  auto members_of = [&](uint32_t cn) {
    return (cn + 1 < new_n ? mstart[cn + 1] : n) - mstart[cn];
  };
  // communities above kSmallWarpMerge entries: a block each
  {
    const uint32_t slots = kSmallArena / kSlotBytes;
    double* vals = reinterpret_cast<double*>(M.arena);
    uint32_t* keys = reinterpret_cast<uint32_t*>(M.arena + sizeof(double) * slots);
    for (uint32_t cn = rank; cn < new_n; cn += ctas) {
      const uint32_t total = M.cdeg[cn];
      if (total <= kSmallWarpMerge) continue;  // block-uniform
      const uint32_t tv = table_size_for(min(total, new_n), slots);
      for (uint32_t i = tid; i < tv; i += kSmallThreads) {
        keys[i] = kEmptyKey;
        vals[i] = 0.0;
      }
      if (tid == 0) S.bump = atomicAdd(&A.counters[bump], total);
      __syncthreads();
      double hot = 0.0;
      bool hot_seen = false;
      small_merge_rows(L, cnew, members + mstart[cn], members_of(cn), cn, tid, kSmallThreads, keys,
                       vals, tv - 1, hot, hot_seen);
      __syncwarp();
      hot = group_sum<32>(hot);
      if (__any_sync(kFull, hot_seen) && lane == 0)
        atomicAdd(&vals[table_insert(keys, tv - 1, cn, L.sc)], hot);
      __syncthreads();
      const uint32_t seg = S.bump;
      uint32_t cnt = 0;
      for (uint32_t i0 = 0; i0 < tv; i0 += kSmallThreads) {  // block-uniform
        const uint32_t i = i0 + tid;
        const uint32_t key = i < tv ? keys[i] : kEmptyKey;
        unsigned long long tot;
        const uint32_t pos = cnt + (uint32_t)block_exclusive_scan<unsigned long long>(
                                       key != kEmptyKey ? 1ull : 0ull, S.scan, &tot);
        if (key != kEmptyKey) {
          A.tcol[seg + pos] = key;
          A.tw[seg + pos] = (float)vals[i];
        }
        cnt += (uint32_t)tot;
      }
      if (tid == 0) {
        A.new_deg[cn] = cnt;
        A.seg[cn] = seg;
      }
      __syncthreads();
    }
  }
  // the others: a warp each
  const uint32_t nw = min((uint32_t)kSmallWarps, kSmallArena / (256u * kSlotBytes));
  if (wib < nw) {
    double* vals = reinterpret_cast<double*>(M.arena) + wib * 256;
    uint32_t* keys = reinterpret_cast<uint32_t*>(M.arena + sizeof(double) * 256 * nw) + wib * 256;
    for (uint32_t cn = rank * nw + wib; cn < new_n; cn += ctas * nw) {
      const uint32_t total = M.cdeg[cn];
      if (total > kSmallWarpMerge) continue;  // warp-uniform
      const uint32_t tv = table_size_for(total, 256u);
      for (uint32_t i = lane; i < tv; i += 32) {
        keys[i] = kEmptyKey;
        vals[i] = 0.0;
      }
      uint32_t seg = 0;
      if (lane == 0) seg = atomicAdd(&A.counters[bump], total);
      seg = __shfl_sync(kFull, seg, 0);
      __syncwarp();  // the table is clear
      double hot = 0.0;
      bool hot_seen = false;
      small_merge_rows(L, cnew, members + mstart[cn], members_of(cn), cn, lane, 32, keys, vals,
                       tv - 1, hot, hot_seen);
      __syncwarp();
      hot = group_sum<32>(hot);
      if (__any_sync(kFull, hot_seen) && lane == 0)
        vals[table_insert(keys, tv - 1, cn, L.sc)] += hot;
      __syncwarp();
      uint32_t cnt = 0;
      for (uint32_t i0 = 0; i0 < tv; i0 += 32) {
        const uint32_t key = keys[i0 + lane];
        const unsigned b = __ballot_sync(kFull, key != kEmptyKey);
        if (key != kEmptyKey) {
          const uint32_t pos = cnt + __popc(b & ((1u << lane) - 1u));
          A.tcol[seg + pos] = key;
          A.tw[seg + pos] = (float)vals[i0 + lane];
        }
        cnt += __popc(b);
      }
      if (lane == 0) {
        A.new_deg[cn] = cnt;
        A.seg[cn] = seg;
      }
      __syncwarp();
    }
  }
  small_sync(ctas);
  if (gt == 0) A.counters[bump ^ 1u] = 0u;  // the next contraction's
  // new offsets, by every block; then the rows, dealt to all warps
  uint32_t new_e = 0;
  for (uint32_t b = 0; b < new_n; b += kSmallThreads) {
    const uint32_t c = b + tid;
    const unsigned long long x = c < new_n ? (unsigned long long)__ldcg(&A.new_deg[c]) : 0ull;
    unsigned long long total;
    const uint32_t pre =
        (uint32_t)block_exclusive_scan<unsigned long long>(x, S.scan, &total) + new_e;
    if (c < new_n) mstart[c] = pre;
    new_e += (uint32_t)total;
  }
  __syncthreads();
  uint64_t* off = A.c_off[next];
  uint32_t* col = A.c_col[next];
  float* w = A.c_w[next];
  for (uint32_t r = rank * kSmallWarps + wib; r < new_n; r += ctas * kSmallWarps) {
    const uint32_t dst = mstart[r], src = (uint32_t)__ldcg(&A.seg[r]);
    const uint32_t cnt = (r + 1 < new_n ? mstart[r + 1] : new_e) - dst;
    if (lane == 0) off[r] = dst;
#pragma unroll 4
    for (uint32_t j = lane; j < cnt; j += 32) {
      col[dst + j] = __ldcg(&A.tcol[src + j]);
      w[dst + j] = __ldcg(&A.tw[src + j]);
    }
  }
  if (gt == 0) off[new_n] = new_e;
  small_sync(ctas);
  *new_n_out = new_n;
  *new_e_out = new_e;
}

template <int MODE>
__global__ void __launch_bounds__(kSmallThreads, 1)
    small_run_kernel(const __grid_constant__ SmallRunArgs A, uint32_t cap) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(16) unsigned char ctx_raw[sizeof(SmallCtx)];
  SmallCtx& S = *reinterpret_cast<SmallCtx*>(ctx_raw);
  const uint32_t rank = blockIdx.x, ctas = gridDim.x, tid = threadIdx.x;
  const uint32_t gt = rank * kSmallThreads + tid;
  const bool lead = gt == 0;
  uint32_t n = A.L.n;
  uint64_t e = A.e_dev ? *A.e_dev : A.e;
  const uint32_t n_first = n;
  int cur = A.cur;
  SmallRunResult* R = A.res;
  // refused before anything is touched: uniform over the cluster
  if (e > A.e_max || n > cap) {
    if (lead) {
      R->status = kSmallRefused;
      R->levels = 0;
      R->contracted = 0;
      R->n = n;
      R->e = e;
      R->cur = cur;
    }
    return;
  }
  SmallMem M;
  {
    unsigned char* p = smem;
    M.arena = p;
    p += kSmallArena;
    M.tot = reinterpret_cast<double*>(p);
    p += 8 * cap;
    M.off = reinterpret_cast<uint64_t*>(p);
    p += 8 * (cap + 2);
    M.ent = (kSmallSmem - small_fixed(cap, ctas)) / 8;
    M.col = reinterpret_cast<uint32_t*>(p);  // 16-byte aligned, as the row loads like it
    p += 4 * (M.ent & ~3u);
    M.w = reinterpret_cast<float*>(p);
    p += 4 * (M.ent & ~3u);
    M.ent &= ~3u;
    M.comm = reinterpret_cast<uint32_t*>(p);
    p += 4 * cap;
    M.sz = reinterpret_cast<uint32_t*>(p);
    p += 4 * cap;
    M.k = reinterpret_cast<float*>(p);
    p += 4 * cap;
    M.cdeg = reinterpret_cast<uint32_t*>(p);
    p += 4 * cap;
    M.prop_all = reinterpret_cast<uint32_t*>(p);
    p += 4 * cap;
    const uint32_t own = small_own(cap, ctas);
    M.order = reinterpret_cast<uint32_t*>(p);
    p += 4 * own;
    M.prop = reinterpret_cast<uint32_t*>(p);
    p += 4 * own;
    M.cls = p;
  }
  if (gt < 2) A.counters[gt] = 0u;
  for (uint32_t v = gt; v < n; v += ctas * kSmallThreads) A.map[v] = v;
  if (tid == 0) {
    S.D.L = A.L;
    S.D.L.k = M.k;
    S.D.L.comm = M.comm;
    S.D.L.comm_sz = M.sz;
    S.D.L.tot = M.tot;
    S.D.L.sc = &S.sc;
    S.G = A.L;
    S.G.sc = &S.sc;
    S.D.act_cnt = S.cls_own;
    S.D.A.order = M.order;
    S.D.prop = M.prop;
    S.D.comm_start = nullptr;
    S.sc.error = 0u;
  }
  small_sync(ctas);  // every block runs before another writes to its memory
  uint32_t levels = 0, status = kSmallMore, contracted = 0;
  double q_run = 0.0;
  uint32_t buf = 0;  // shares alternate: a block may still read the last ones
  for (;;) {
    unsigned long long t0 = 0, t1 = 0;
    if (lead) t0 = global_ns();
    if (tid == 0) {
      S.D.L.n = S.G.n = n;
      S.G.off = cur < 0 ? A.L.off : A.c_off[cur];
      S.G.col = cur < 0 ? A.L.col : A.c_col[cur];
      S.G.w = cur < 0 ? A.L.w : A.c_w[cur];
    }
    __syncthreads();
    const bool fits = small_classes(S, M, S.G, rank, ctas);
    if (tid == 0) {
      S.D.L.off = fits ? M.off : S.G.off;
      S.D.L.col = fits ? M.col : S.G.col;
      S.D.L.w = fits ? M.w : S.G.w;
    }
    if (S.cls_all[8] || levels == kSmallLevels) {  // a row too long for the block table
      status = kSmallMore;
      break;
    }
    const bool wide = e > 24ull * n;  // lanes per row
    double x = 0.0, y = 0.0, z = 0.0;
    if (wide) small_rows<32>(S.G, M, fits, A.L.k, rank, ctas, x, y, z);
    else small_rows<8>(S.G, M, fits, A.L.k, rank, ctas, x, y, z);
    small_share(S, buf, x, y, z, rank, ctas);
    small_sync(ctas);
    const double m = small_gather(S, buf, 0, ctas) / 2.0;
    const double asq0 = small_gather(S, buf, 1, ctas), intra0 = small_gather(S, buf, 2, ctas);
    buf ^= 1u;
    const double q_start = m > 0.0 ? intra0 / (2.0 * m) - asq0 / (4.0 * m * m) : 0.0;
    for (uint32_t v = tid; v < n; v += kSmallThreads) {
      const float kf = __ldcg(&A.L.k[v]);
      M.k[v] = kf;
      M.tot[v] = (double)kf;
    }
    if (tid == 0) {
      const float mf = (float)m;
      S.sc.m64 = m;
      S.sc.m = mf;
      S.sc.den = __fmul_rn(__fmul_rn(2.0f, mf), mf);
    }
    __syncthreads();
    if (lead) t1 = global_ns();
    double q = q_start, q_before = q_start;
    uint32_t passes = 0;
    bool first_fail = !(m > 0.0);
    if (m > 0.0) {
      double q_prev = q_start;
      const uint32_t w512 = min((uint32_t)kSmallWarps, kSmallArena / (512u * kSlotBytes));
      for (;;) {
#pragma unroll 1
        for (int b = 1; b <= kBuckets; b++) {
          if (!S.cls_all[b]) continue;  // uniform over the cluster
          // a warp per vertex only where blocks would take several each
          const bool blk = b == 7 || (b >= 5 && S.cls_own[b] <= 2);
          if (blk) small_block<MODE>(&S.D, b, M.arena);
          else if (b == 1) small_lanes<4, MODE>(&S.D, b, M.arena);
          else if (b == 2) small_lanes<8, MODE>(&S.D, b, M.arena);
          else if (b == 3) small_lanes<16, MODE>(&S.D, b, M.arena);
          else if (b == 4) small_lanes<32, MODE>(&S.D, b, M.arena);
          else if (b == 5) small_warp<128, 3, MODE>(&S.D, b, M.arena, kSmallWarps);
          else small_warp<512, 10, MODE>(&S.D, b, M.arena, w512);
          __syncthreads();  // every decision of this block is in prop
          const uint32_t s0 = S.D.A.P.cls_start[b], cnt = S.cls_own[b];
          if (ctas == 1) {
            for (uint32_t i0 = 0; i0 < cnt; i0 += kSmallThreads) {
              const uint32_t i = i0 + tid;
              uint32_t v = 0, oc = 0, nc = 0;
              if (i < cnt) {
                v = M.order[s0 + i];
                nc = M.prop[s0 + i];
                oc = M.comm[v];
              }
              small_apply(M, nc != oc, v, oc, nc);
            }
          } else {  // a thread per (own vertex, block)
            const uint32_t to = tid % ctas;
            const uint32_t dst = small_remote(M.prop_all, to);
            for (uint32_t i = tid / ctas; i < cnt; i += kSmallThreads / ctas)
              small_store(dst + 4 * M.order[s0 + i], M.prop[s0 + i]);
            small_sync(ctas);
            for (uint32_t v0 = 0; v0 < n; v0 += kSmallThreads) {
              const uint32_t v = v0 + tid;
              uint32_t oc = 0, nc = 0;
              if (v < n && M.cls[v] == b) {
                nc = M.prop_all[v];
                oc = M.comm[v];
              }
              small_apply(M, nc != oc, v, oc, nc);
            }
          }
          __syncthreads();
        }
        double in = 0.0, sq2 = 0.0;
        if (wide) small_q_share<32>(S.D.L, rank, ctas, in, sq2);
        else small_q_share<8>(S.D.L, rank, ctas, in, sq2);
        small_share(S, buf, in, sq2, 0.0, rank, ctas);
        small_sync(ctas);
        q_before = q_prev;
        q = small_gather(S, buf, 0, ctas) / (2.0 * m) -
            small_gather(S, buf, 1, ctas) / (4.0 * m * m);
        buf ^= 1u;
        // stop rule of modularity.cu:501-508 / louvian.py:91-99
        passes++;
        if (passes == 1 && q - q_prev < A.min_gain) first_fail = true;
        const bool cont = q - q_prev >= A.min_gain && passes < A.max_passes;
        q_prev = q;
        if (!cont) break;
      }
    } else {
      q = q_before = 0.0;
    }
    q_run = first_fail ? q_before : q;
    if (lead) {
      SmallLevel& l = R->level[levels];
      l.n = n;
      l.e = e;
      l.passes = passes;
      l.q_start = q_start;
      l.q_end = q;
      l.t_start = t0;
      l.t_ready = t1;
      l.t_moved = l.t_done = global_ns();
    }
    levels++;
    if (first_fail || A.move_only) {  // the level's state is the caller's
      if (first_fail) status = kSmallFirstFail;
      for (uint32_t v = gt; v < n; v += ctas * kSmallThreads) {
        A.L.comm[v] = M.comm[v];
        A.L.comm_sz[v] = M.sz[v];
        A.L.tot[v] = M.tot[v];
      }
      break;
    }
    uint32_t new_n = 0;
    uint64_t new_e = 0;
    const int next = cur == 0 ? 1 : 0;
    small_contract(A, S, M, rank, ctas, next, n_first, contracted & 1u, &new_n, &new_e);
    contracted++;
    cur = next;
    if (lead) R->level[levels - 1].t_done = global_ns();
    const bool same = new_n == n;
    n = new_n;
    e = new_e;
    if (same || (A.max_levels && levels >= A.max_levels)) {
      status = kSmallMerged0;
      break;
    }
  }
  if (tid == 0 && S.sc.error) atomicExch(&A.L.sc->error, S.sc.error);
  small_sync(ctas);  // no block leaves while another may still write to it
  if (lead) {
    R->status = status;
    R->levels = levels;
    R->contracted = contracted;
    R->n = n;
    R->e = e;
    R->cur = cur;
    R->q = q_run;
  }
}
