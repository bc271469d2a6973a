// Batch-shared one-label distance search.
//
// The unbounded queries of one batch call need the distances from each of their groups
// to every vertex (below a cutoff).  Searching query by query reads the graph's edges and
// one random 32-byte distance row per relaxation, once per query; the relaxation rate is
// then bound by the device's random-access rate.  Here the distinct groups of all the
// batch's unbounded queries (up to BS_COLS of them) are searched together: one distance
// table of V rows x Gp columns (column c = the c-th group), one announcement bit per
// (vertex, column), and a relaxation of edge (v, u) serves every column whose distance
// at v improved in the previous step, reading u's row as one contiguous span (lanes of a
// warp take its 32-byte sectors) instead of one random row per query.
//
// Cutoffs: a query's distances are needed exactly only up to its search cutoff (its star
// bound x cut_pm / 1000).  Column c keeps the largest cutoff of the queries that use it;
// stars are found while the search runs (before each relax step, k_bs_scan sums each
// query's columns at every announced vertex) and the cutoffs only decrease, so every distance at
// most a column's final cutoff is exact (every prefix of its shortest path stayed below
// it) and every other one is only known to exceed it.  A query then takes the smallest
// final cutoff of its columns as its own `cut` (distances above it are clamped to cut + 1
// by every bound), at least as strong as its own search would have reached.
//
// Hop-bounded queries of one bound D (1 <= D <= KMAX) share a search the same way over
// D tables: table h holds d^{<=h}, the cheapest paths of at most h edges (table D is the
// distance table, 1..D-1 the hop budgets).  One step is one round: round r (r >= 1)
// first copies table r into table r+1 (a coalesced pass, so that table r+1 starts from
// the paths of at most r edges), then relaxes the edges of the vertices whose table r
// row improved in round r-1 (round 0: the members, distance 0) from table r into table
// r+1 alone.  Table r is final while round r reads it, so no snapshot is needed, and
// the result is the per-query rounds'.  Stars come from tables r with 2r <= D (trees of
// diameter <= D), as in the per-query search.
//
// The last rounds pull.  Table h bounds the states of height D - h only, and those hang at
// vertices within D - h edges of their query's members: table D is read at the members
// themselves, table D-1 at their neighbours.  So the last round (and, from D = 4 on, the
// one before it) takes each such vertex and the sectors of the queries that may have a state
// there, and looks at its own edges, instead of pushing along the edges of everything within
// D - 1 (D - 2) edges of a member, which is the whole graph.  Elsewhere these tables hold
// upper bounds that no state reads (and are zero at members only, like the others).  The
// bits to pull at come with the search: the members, and what round 0 announced.
// 32 queries with D = 3/4/5 over 1M vertices relax 410 M sectors instead of 1303 M (search
// 15.4 to 6.2 ms), the 4M-vertex batch 3.1 G instead of 5.3 G.
//
// Edge classes (unbounded searches): the edges are relaxed light ones first, to a fixpoint,
// and only then the heavier ones, from every vertex whose distances changed since its
// heavier edges were last relaxed.  A relaxation is bound by the random row it reads, and
// label-correcting steps over all edges repeat most of them: a vertex improves a few
// columns at a time, step after step, and its heavy edges run before the cutoffs are
// known.  The light fixpoint is a small share of the edges, settles nearly every distance
// and finds the stars, so a heavy edge is relaxed about once, for all columns of a sector
// together, against nearly final cutoffs.  Any order ends at the same distances.  On 32
// queries of k = 5/7 over 141k vertices 464 M sectors are relaxed instead of 1013 M (search
// 8.4 to 6.5 ms), on the 4M-vertex batch 5.3 G instead of 7.6 G (82 to 70 ms).  The light
// steps are more and smaller, so a search over few columns or edges runs in one class: a
// lone query takes 6.5 ms in one class and 8.9 ms in two at 4M vertices
// (Runner::search_classes).
//
// Per step, two launches: k_bs_scan turns the announcement bits of the step's class into
// relax items of at most BS_CHUNK edges (a hub's range spread over many warps) and finds
// the stars at the announced vertices, its last block lowers the cutoffs; k_bs_relax
// relaxes the items, its last block chooses the next step's class or ends the search.
#pragma once
#include "gst_device.cuh"

namespace gst {

constexpr int BS_COLS = 256;   // columns (distinct groups) of one shared search, at most
constexpr int BS_MAXQ = MAXB;  // queries of one shared search, at most
// The search finds distances up to here only: the relax kernel compares signed words, a cutoff
// plus one among them.
constexpr uint32_t BS_DIST_MAX = 0x7FFFFFFEu;

struct BsCtx {
  uint32_t* dist;       // V x Gp distances, row v at dist + v * Gp
  uint32_t* fm[2];      // V x Wm announcement words (bit c: column c improved at v)
  uint32_t* later;      // V x Wm, two classes: columns whose heavy edges wait
  uint32_t ncls;        // edge classes: 1, or 2 (light edges, heavy edges)
  const uint32_t* cend; // V, two classes: the end of v's light edges in its list
  uint32_t cls;         // class of the current step
  uint32_t have;        // later is not empty
  uint32_t arrived;     // blocks of the current launch that are done (see last_block)
  uint32_t* am;         // V x Wm: v's active columns in the current step (scan -> relax)
  uint2* items;         // relax items of the current step: {v, chunk}; whole chunks from the
                        // front, the lists' ends (shorter ones) from the back
  uint32_t item_cap;
  uint32_t chunk;       // edges per item, at most
  uint32_t n_items[2];  // whole and short items of the current step (appended by the scan)
  unsigned long long work[2];  // their (edge, active sector) pairs
  uint32_t next[2];     // items of each taken from the counter in the relax step
  uint32_t Gp, Wm;      // columns (a multiple of 8), mask words per vertex
  uint32_t in;          // fm[in] is scanned this step; fm[in ^ 1] takes its announcements
  uint32_t ann;         // the relax step announced something
  uint32_t done, steps, max_steps, error;
  uint32_t far;         // some distance may be beyond BS_DIST_MAX (k_bs_far)
  uint32_t cut_pm;      // query cutoff: star x cut_pm / 1000
  uint32_t D;           // 0: unbounded distances; else the hop bound (rounds 0..D-1)
  uint32_t round;       // hop-bounded: the current round
  uint32_t pull;        // hop-bounded: the first round that pulls
  uint32_t* near[2];    // hop-bounded: V x Wm, columns with a member at the vertex (0), or at
                        // it or a neighbour (1)
  uint32_t colsec[BS_COLS];  // per column: the sectors of the queries that use it
  uint32_t* tab[KMAX + 1];  // hop-bounded: tab[h] = d^{<=h} (V x Gp), tab[D] = dist
  uint32_t nq;          // queries
  uint32_t qk[BS_MAXQ];
  uint16_t qcol[BS_MAXQ][KMAX];  // columns of each query's groups
  uint32_t star[BS_MAXQ];        // best star found per query (a feasible cost)
  uint32_t cutc[BS_COLS];        // per column: its distance cutoff
  unsigned long long st_relax;   // target-row sectors read (edges x active lanes)
};
constexpr uint32_t BS_ERR_ITEMS = 1, BS_ERR_STEPS = 2;

// First and one-past-last edge of v's weight-sorted list in the current class.
__device__ __forceinline__ void class_range(const BsCtx* b, uint32_t cls, uint32_t v, int64_t deg,
                                            int64_t* lo, int64_t* hi) {
  const int64_t light = b->ncls > 1u ? (int64_t)__ldg(&b->cend[v]) : deg;
  *lo = cls ? light : 0;
  *hi = cls ? deg : light;
}

// Seeds: column c's members at distance 0, announced (blockIdx.y = column).
__global__ void k_bs_seed(BsCtx* b, DevGraph G, const int64_t* grp_ptr, const int32_t* members,
                          const int32_t* col_gid, int ncols) {
  const int c = blockIdx.y;
  if (c >= ncols) return;
  const int32_t g = col_gid[c];
  const uint32_t Gp = b->Gp, Wm = b->Wm;
  for (int64_t j = grp_ptr[g] + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < grp_ptr[g + 1];
       j += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t v = (uint32_t)members[j];
    if (v >= G.V) continue;
    atomicMin(&(b->D ? b->tab[1] : b->dist)[(uint64_t)v * Gp + c], 0u);
    const uint64_t word = (uint64_t)v * Wm + (c >> 5);
    if (G.beg[v + 1] > G.beg[v]) atomicOr(&b->fm[b->in][word], 1u << (c & 31));
    for (int i = 0; i < 2; i++)
      if (b->near[i]) atomicOr(&b->near[i][word], 1u << (c & 31));
  }
}

// Column cutoffs from the query stars (the last block of a scan).
__device__ __forceinline__ void bs_lower_cutoffs(BsCtx* b, uint32_t* s_cut) {
  for (uint32_t c = threadIdx.x; c < BS_COLS; c += blockDim.x) s_cut[c] = 0u;
  __syncthreads();
  for (uint32_t x = threadIdx.x; x < b->nq * KMAX; x += blockDim.x) {
    const uint32_t q = x / KMAX, i = x % KMAX;
    if (i >= b->qk[q]) continue;
    const uint32_t st = __ldcg(&b->star[q]);
    const uint64_t cut = st == COST_INF ? COST_INF : (uint64_t)st * b->cut_pm / 1000u;
    // a used column's cutoff is stored plus one, below: 0 marks an unused column
    atomicMax(&s_cut[b->qcol[q][i]], cut >= COST_INF ? COST_INF : (uint32_t)cut + 1u);
  }
  __syncthreads();
  for (uint32_t c = threadIdx.x; c < b->Gp; c += blockDim.x)
    if (s_cut[c] && s_cut[c] != COST_INF) b->cutc[c] = min(b->cutc[c], s_cut[c] - 1u);
}

// Scan: every vertex announced for the step's class gets its active columns (moved to am,
// and on to the next class's waiting columns) and its relax items: one per chunk of the
// edges it has in the class.  Then its stars: each query's columns summed at the vertex
// (the query's k shortest paths from there form a connected subgraph covering every group,
// a feasible cost); hop-bounded from table r with 2r <= D only (a tree of diameter <= D).
// A star found here lowers the cutoffs that this very step relaxes against.  One lane per
// (vertex, query).  VPT neighbouring vertices per thread: with four, their words come in
// Wm 16-byte loads issued together, which is all a step that announces few vertices does
// (large graphs); with one, the stars of a small graph spread over four times the warps.
// PULL: a pulling round, whose items are the vertices of near[D - 1 - r] with the sectors of
// the queries that may have a state there.
template <int VPT, bool PULL>
__global__ void __launch_bounds__(256, 4) k_bs_scan(BsCtx* b, DevGraph G) {
  __shared__ uint32_t s_star[BS_MAXQ];
  __shared__ uint32_t s_cut[BS_COLS];
  __shared__ uint16_t s_col[BS_MAXQ][KMAX];
  __shared__ uint32_t s_k[BS_MAXQ];
  __shared__ uint32_t s_sec[PULL ? BS_COLS : 1];  // colsec
  __shared__ uint32_t s_v[256 / 32][32];  // per warp: the announced vertices
  __shared__ uint32_t s_sum[2][256 / 32], s_work[2][256 / 32], s_base[2];
  if (b->done) return;
  const uint32_t Wm = b->Wm, cls = b->cls, Gp = b->Gp, nq = b->nq, D = b->D, r = b->round;
  const uint32_t chunk = b->chunk, cap = b->item_cap;
  const bool two = b->ncls > 1u;
  uint32_t* from = PULL ? b->near[D - 1u - r] : cls ? b->later : b->fm[b->in];
  // where the announced columns are kept for later: a light step's for the heavy class, what
  // round 0 of a hop-bounded search announced for the round that pulls at the neighbours
  uint32_t* keep = D ? (r == 1u ? b->near[1] : nullptr) : two && cls == 0u ? b->later : nullptr;
  uint32_t* am = b->am;
  uint2* items = b->items;
  const uint32_t* cend = b->cend;
  // Every improved distance is announced to the light class, and on to the heavy one.  With
  // two classes the light scans, of which there are many, look for stars only at the
  // vertices of highest degree (the lowest ids), where the best ones are, and the heavy
  // scans everywhere: with all vertices in the light ones too the searches of 32 queries take
  // 3 to 7 % longer (k = 5: 75.7 to 81.2 ms over 4.6M vertices, 19.6 to 20.7 over 1.1M), with a
  // quarter of them up to 3 % (78.1, 19.9), with a 64th the same as with a sixteenth (75.6, 19.4).
  const bool stars = D == 0u || (r >= 1u && 2u * r <= D);
  const int64_t star_end = !D && cls == 0u && b->ncls > 1u ? (G.V + 15) / 16 : G.V;
  const uint32_t* tab = D ? b->tab[r] : b->dist;
  if constexpr (PULL)
    for (uint32_t c = threadIdx.x; c < BS_COLS; c += blockDim.x) s_sec[c] = b->colsec[c];
  for (uint32_t q = threadIdx.x; q < BS_MAXQ; q += blockDim.x) {
    s_star[q] = COST_INF;
    s_k[q] = q < nq ? b->qk[q] : 0u;
#pragma unroll
    for (int i = 0; i < KMAX; i++) s_col[q][i] = q < nq ? b->qcol[q][i] : 0u;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  uint32_t more = 0;
  const int64_t spans = (G.V + VPT - 1) / VPT;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < spans;
       base += (int64_t)gridDim.x * blockDim.x) {
    const int64_t first = (base + threadIdx.x) * VPT;
    uint32_t hit = 0;  // bit i: vertex first + i is announced
    uint32_t cnt = 0;  // its active sectors, in byte i
    // (loads before stores throughout: the stores may alias them for the compiler, and one
    // access after the other made a scan of 4.6M announced vertices 1.1 ms long, 0.15 now)
    if (base + threadIdx.x < spans) {
      if constexpr (PULL) {
        for (int i = 0; i < VPT; i++) {
          uint32_t needed = 0;
          if (first + i < G.V)
            for (uint32_t w = 0; w < Wm; w++)
              for (uint32_t x = __ldcg(&from[(first + i) * Wm + w]); x; x &= x - 1u)
                needed |= s_sec[w * 32u + (uint32_t)__ffs(x) - 1u];
          if (!needed) continue;
          hit |= 1u << i;
          cnt |= (uint32_t)__popc(needed) << (8 * i);
          for (uint32_t w = 0; w < Wm; w++) {  // the needed sectors, all their columns
            const uint32_t x = (needed >> (4u * w)) & 0xFu;
            am[(first + i) * Wm + w] = ((x & 1u) | (x & 2u) << 7 | (x & 4u) << 14 | (x & 8u) << 21) * 0xFFu;
          }
        }
      } else if constexpr (VPT == 4) {
        uint4* f4 = (uint4*)(from + first * Wm);
        uint4* a4 = (uint4*)(am + first * Wm);
        uint4* k4 = keep ? (uint4*)(keep + first * Wm) : nullptr;
        uint32_t some = 0;
        for (uint32_t w = 0; w < Wm; w++) {  // (cached loads: a line serves several of them)
          const uint4 x = f4[w];
          some |= x.x | x.y | x.z | x.w;
        }
        for (uint32_t w0 = 0; some && w0 < Wm; w0 += 4) {
          uint4 x[4], y[4];
          bool on[4];
#pragma unroll
          for (uint32_t j = 0; j < 4; j++)
            x[j] = w0 + j < Wm ? f4[w0 + j] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
          for (uint32_t j = 0; j < 4; j++) {
            on[j] = (x[j].x | x[j].y | x[j].z | x[j].w) != 0u;
            y[j] = on[j] && k4 ? k4[w0 + j] : make_uint4(0u, 0u, 0u, 0u);
          }
#pragma unroll
          for (uint32_t j = 0; j < 4; j++) {
            if (w0 + j < Wm) a4[w0 + j] = x[j];
            if (!on[j]) continue;
            f4[w0 + j] = make_uint4(0u, 0u, 0u, 0u);
            if (k4) k4[w0 + j] = make_uint4(x[j].x | y[j].x, x[j].y | y[j].y, x[j].z | y[j].z, x[j].w | y[j].w);
            const uint32_t c[4] = {x[j].x, x[j].y, x[j].z, x[j].w};
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) {
              const uint32_t at = (4u * (w0 + j) + i) / Wm;  // the word's vertex
              const uint32_t n = ((c[i] & 0xFFu) != 0u) + ((c[i] & 0xFF00u) != 0u) +
                                 ((c[i] & 0xFF0000u) != 0u) + (c[i] >> 24 != 0u);
              hit |= (c[i] != 0u) << at;
              cnt += n << (8u * at);
            }
          }
        }
      } else {
        uint32_t x[BS_COLS / 32], y[BS_COLS / 32];
#pragma unroll
        for (uint32_t w = 0; w < BS_COLS / 32; w++) {
          x[w] = w < Wm ? __ldcg(&from[first * Wm + w]) : 0u;
          hit |= x[w] != 0u;
        }
        if (hit) {
#pragma unroll
          for (uint32_t w = 0; w < BS_COLS / 32; w++) y[w] = keep && w < Wm ? keep[first * Wm + w] : 0u;
#pragma unroll
          for (uint32_t w = 0; w < BS_COLS / 32; w++)
            if (w < Wm) {
              am[first * Wm + w] = x[w];
              from[first * Wm + w] = 0u;
              if (keep) keep[first * Wm + w] = x[w] | y[w];
              cnt += ((x[w] & 0xFFu) != 0u) + ((x[w] & 0xFF00u) != 0u) + ((x[w] & 0xFF0000u) != 0u) +
                     (x[w] >> 24 != 0u);
            }
        }
      }
    }
    if (!__syncthreads_or(hit != 0u)) continue;
    more |= hit && two && cls == 0u;
    uint32_t whole[VPT], rest[VPT], nw = 0, nr = 0, ww = 0, wr = 0;
    int64_t bg[VPT + 1];
    uint32_t light[VPT];
    if (hit) {
#pragma unroll
      for (int i = 0; i <= VPT; i++) bg[i] = first + i <= G.V ? G.beg[first + i] : 0;
#pragma unroll
      for (int i = 0; i < VPT; i++) light[i] = two && first + i < G.V ? __ldg(&cend[first + i]) : 0u;
    }
#pragma unroll
    for (int i = 0; i < VPT; i++) {
      whole[i] = rest[i] = 0u;
      if (!((hit >> i) & 1u)) continue;
      const uint32_t deg = (uint32_t)(bg[i + 1] - bg[i]), sectors = (cnt >> (8 * i)) & 0xFFu;
      const uint32_t edges = !two ? deg : cls ? deg - light[i] : light[i];
      whole[i] = edges / chunk;
      rest[i] = edges % chunk != 0u;
      nw += whole[i];
      nr += rest[i];
      ww += whole[i] * sectors;
      wr += edges % chunk * sectors;
    }
    // one reservation per block and list: a per-warp one made the counters the hottest
    // address of the step
    const uint32_t sw = warp_incl_scan(nw), sr = warp_incl_scan(nr);
    ww = __reduce_add_sync(0xffffffffu, ww);
    wr = __reduce_add_sync(0xffffffffu, wr);
    if (lane == 31) {
      s_sum[0][wib] = sw;
      s_sum[1][wib] = sr;
      s_work[0][wib] = ww;
      s_work[1][wib] = wr;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
      uint32_t tot = 0;
      unsigned long long work = 0;
      for (uint32_t w = 0; w < blockDim.x / 32; w++) {
        const uint32_t x = s_sum[threadIdx.x][w];
        s_sum[threadIdx.x][w] = tot;
        tot += x;
        work += (unsigned long long)s_work[threadIdx.x][w] * (threadIdx.x == 0 ? chunk : 1u);
      }
      s_base[threadIdx.x] = tot ? atomicAdd(&b->n_items[threadIdx.x], tot) : 0u;
      if (work) atomicAdd(&b->work[threadIdx.x], work);
    }
    __syncthreads();
    uint32_t tw = s_base[0] + s_sum[0][wib] + sw - nw, tr = s_base[1] + s_sum[1][wib] + sr - nr;
    // (by its size, V + E / chunk, the array holds every item of both lists)
    if (tw + nw + tr + nr > cap) atomicOr(&b->error, BS_ERR_ITEMS);
#pragma unroll
    for (int i = 0; i < VPT; i++) {
      // a hub's items (hundreds) are written by the whole warp
      uint32_t hubs = __ballot_sync(0xffffffffu, whole[i] > 16u);
      while (hubs) {
        const int src = __ffs(hubs) - 1;
        hubs &= hubs - 1u;
        const uint32_t n = __shfl_sync(0xffffffffu, whole[i], src), t = __shfl_sync(0xffffffffu, tw, src);
        const uint32_t v = __shfl_sync(0xffffffffu, (uint32_t)(first + i), src);
        for (uint32_t j = (uint32_t)lane; j < n; j += 32)
          if (t + j < cap) items[t + j] = make_uint2(v, j);
      }
      if (whole[i] <= 16u)
        for (uint32_t j = 0; j < whole[i]; j++)
          if (tw + j < cap) items[tw + j] = make_uint2((uint32_t)(first + i), j);
      tw += whole[i];
      if (rest[i]) {
        if (tr < cap) items[cap - 1u - tr] = make_uint2((uint32_t)(first + i), whole[i]);
        tr++;
      }
    }
#pragma unroll
    for (int i = 0; i < VPT; i++) {
      const uint32_t ann = __ballot_sync(0xffffffffu, (hit >> i) & 1u);
      if (!stars || !ann || (base + (threadIdx.x & ~31u)) * VPT >= star_end) continue;
      if ((hit >> i) & 1u) s_v[wib][__popc(ann & ((1u << lane) - 1u))] = (uint32_t)(first + i);
      __syncwarp();
      for (uint32_t p = (uint32_t)lane; p < __popc(ann) * nq; p += 32) {
        const uint32_t a = nq == 1u ? p : p / nq, q = p - a * nq, k = s_k[q];
        const uint32_t* row = tab + (uint64_t)s_v[wib][a] * Gp;
        uint64_t sum = 0;
#pragma unroll
        for (uint32_t t = 0; t < KMAX; t++) sum += t < k ? row[s_col[q][t]] : 0u;
        if (sum < (uint64_t)s_star[q]) atomicMin(&s_star[q], (uint32_t)sum);
      }
      __syncwarp();
    }
  }
  if (__any_sync(0xffffffffu, more != 0u) && lane == 0) b->have = 1u;
  __syncthreads();
  for (uint32_t q = threadIdx.x; q < nq; q += blockDim.x)
    if (s_star[q] < __ldcg(&b->star[q])) atomicMin(&b->star[q], s_star[q]);
  if (!last_block(&b->arrived)) return;
  if (stars) bs_lower_cutoffs(b, s_cut);
  if (threadIdx.x == 0 && cls) b->have = 0u;  // this scan took them all
}

// The next step (the last block of a relax launch): announced vertices first, else the
// heavy edges that wait; without any the search is done.  Hop-bounded: D rounds.
__device__ __forceinline__ void bs_advance(BsCtx* b) {
  const uint32_t cls = b->D || __ldcg(&b->ann) ? 0u : 1u;
  if (__ldcg(&b->error) || (b->D ? b->round + 1u >= b->D : cls && !__ldcg(&b->have))) {
    b->done = 1u;
  } else if (++b->steps > b->max_steps) {
    b->error |= BS_ERR_STEPS;
    b->done = 1u;
  } else {
    b->cls = cls;
    if (cls == 0u) b->in ^= 1u;
    b->ann = 0u;
    for (int i = 0; i < 2; i++) {
      b->n_items[i] = b->next[i] = 0u;
      b->work[i] = 0ull;
    }
    b->round++;
  }
}

// Relax.  A warp takes up to 32 items at a time and lists their units, the (item, active
// 8-column sector) pairs; 32 units form a window.  Lane t loads the distances of unit t's
// sector, stages them in shared memory and plans the item's edges (those light enough for
// some of its columns).  Then the window's work, every (edge, sector) pair of its items, is
// spread over all lanes: item by item, edge by edge, the sectors of one edge on neighbouring
// lanes, so that a target's row is read as one contiguous span.  One item per warp left most
// of it idle in the light classes, whose items have a few edges each behind a chain of
// dependent loads; fixed shares of the items left most warps waiting for the few that held
// the hubs, so the warps take items from a counter, the whole chunks
// first.  In one class, against one item per warp in fixed shares: 23 to 9 ms of relax steps
// for three lone queries over 4M vertices, 3.9 to 2.7 ms over 141k; 77 to 74 ms for the
// 4M-vertex batch, whose items are wide (57 ms with the two classes).  Two pairs per lane
// and four blocks per SM: three pairs in 80 registers and three blocks take 10 % longer on
// the batches, five blocks spill.
// The test of a sector is two instructions per column: with the sector's -d and cutoff + 1,
// some column improves over the edge's weight w iff max_i(min(target_i, cutoff_i + 1) - d_i) > w.
constexpr int BS_U = 2;        // (edge, sector) pairs per lane in flight
constexpr uint32_t BS_TAKE = 1024;  // pairs per take, about
constexpr uint32_t BS_LIST = 256;   // units per take, at most
struct __align__(16) BsUnit {  // one unit of a window
  int nd[8];                   // -distance per column (inactive: -INT_MAX); pulling: the
                               // target's distances, at most cutoff + 1
  uint32_t sec;                // the sector
  uint32_t at;                 // pulling: the target's row, in sectors
  uint32_t pad[2];             // 48-byte stride: eight lanes' 16-byte loads hit 32 banks
};
struct __align__(16) BsWork {  // one item of a window with work
  int64_t eb;                  // its first edge
  uint32_t start;              // its first pair in the window
  uint32_t unit;               // its first unit | its units c << 5 | ceil(2^16 / c) << 11: a
                               // pair's edge is (pair * that) >> 16, exact below 2^11 pairs
};
// PULL: the items are targets; a pair reads the neighbour's row and lowers the item's.
// in_loop: the launch is the last node of a graph loop over the steps, which it ends.
template <bool PULL>
__global__ void __launch_bounds__(256, 4) k_bs_relax(BsCtx* b, DevGraph G, cudaGraphConditionalHandle loop,
                                                  int in_loop) {
  // (shared memory is kept small: what it leaves to the L1 serves the edge lists)
  __shared__ __align__(16) int s_c1[BS_COLS / 8][12];  // per sector and column: cutoff + 1
  __shared__ BsUnit s_unit[256 / 32][32];              // per warp: the window's units
  __shared__ BsWork s_work[256 / 32][32];              // per warp: the window's items
  __shared__ uint16_t s_list[256 / 32][BS_LIST];       // per warp: lane of the item << 5 | sector
  if (b->done) return;
  const uint32_t Gp = b->Gp, Wm = b->Wm, nsec = Gp / 8u;
  for (uint32_t c = threadIdx.x; c < BS_COLS; c += blockDim.x)
    s_c1[c >> 3][c & 7u] = c < Gp ? (int)(min(b->cutc[c], BS_DIST_MAX) + 1u) : 0;
  __syncthreads();
  // hop-bounded round r: sources in table r (the members at 0 for r = 0), targets in
  // table r + 1; a round announces only to a next one that pushes
  const uint32_t D = b->D, r = b->round, cls = b->cls, chunk_edges = b->chunk, cap = b->item_cap;
  const bool over = (D && r >= D) || b->error;  // past the last round: nothing to relax
  const uint32_t pushes = D ? b->pull : 0u;     // the rounds that announce for a next one
  const uint32_t* src_tab = D ? (r ? b->tab[min(r, D)] : nullptr) : b->dist;
  uint32_t* dst_tab = D ? b->tab[min(r + 1u, D)] : b->dist;
  const bool extend = D == 0u || r + 1u < pushes;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  // neighbouring takes go to different blocks: the first ones hold the hubs' chunks
  const uint32_t wid = (uint32_t)wib * gridDim.x + blockIdx.x;
  uint32_t* fo = b->fm[b->in ^ 1u];
  unsigned long long relaxed = 0;
  uint32_t any = 0;
  for (int kind = 0; kind < 2 && !over; kind++) {
   const uint32_t n = b->n_items[kind];
   // about BS_TAKE pairs, and no more than spreads the step over all warps
   const uint32_t per = n ? (uint32_t)((unsigned long long)BS_TAKE * n / max(b->work[kind], 1ull)) : 0u;
   const uint32_t take =
       max(1u, min(min(min(32u, BS_LIST / nsec), per), (n + warps - 1u) / warps));
   // A warp's first take is its own share where the step is small (no contention for the
   // counter when most warps have nothing to do); else all come from the counter, so that
   // no share waits for a warp that is still at work on the whole chunks.
   const bool shares = kind ? n <= warps * take && b->n_items[0] <= warps / 8u : true;
   const uint32_t taken = shares ? warps * take : 0u;
   uint32_t base = wid * take;
   if (!shares) {
     if (lane == 0) base = atomicAdd(&b->next[kind], take);
     base = __shfl_sync(0xffffffffu, base, 0);
   }
   while (base < n) {
    // the items' active sectors, listed in item order
    uint2 item = make_uint2(0u, 0u);
    uint32_t sectors = 0;
    if ((uint32_t)lane < take && base + lane < n) {
      item = b->items[kind ? cap - 1u - (base + lane) : base + lane];
      for (uint32_t w = 0; w < Wm; w++) {
        const uint32_t x = __ldcg(&b->am[(uint64_t)item.x * Wm + w]);
#pragma unroll
        for (int j = 0; j < 4; j++)
          if ((x >> (8 * j)) & 0xFFu) sectors |= 1u << (4 * w + j);
      }
    }
    const uint32_t uscan = warp_incl_scan((uint32_t)__popc(sectors));
    const uint32_t units = __shfl_sync(0xffffffffu, uscan, 31);
    uint32_t at = uscan - (uint32_t)__popc(sectors);
    for (uint32_t m = sectors; m; m &= m - 1u) s_list[wib][at++] = (uint16_t)(lane << 5 | (__ffs(m) - 1));
    __syncwarp();
    for (uint32_t u0 = 0; u0 < units; u0 += 32) {
      const uint32_t live = min(32u, units - u0);
      const uint32_t ent = s_list[wib][u0 + min((uint32_t)lane, live - 1u)];
      const uint32_t sec = ent & 31u, own = ent >> 5;
      const uint32_t v = __shfl_sync(0xffffffffu, item.x, (int)own);
      const uint32_t chunk = __shfl_sync(0xffffffffu, item.y, (int)own);
      const uint32_t m = (__ldcg(&b->am[(uint64_t)v * Wm + (sec >> 2)]) >> ((sec & 3u) * 8u)) & 0xFFu;
      uint4 da = make_uint4(0, 0, 0, 0), db = da;  // round 0: the members themselves
      if (PULL || src_tab) {
        const uint4* src = (const uint4*)&(PULL ? dst_tab : src_tab)[(uint64_t)v * Gp + sec * 8];
        da = __ldcg(src);
        db = __ldcg(src + 1);
      }
      const int64_t b0 = G.beg[v], b1 = G.beg[v + 1];
      int64_t lo, hi;
      class_range(b, cls, v, b1 - b0, &lo, &hi);
      const uint32_t dv[8] = {da.x, da.y, da.z, da.w, db.x, db.y, db.z, db.w};
      BsUnit x;
      int wl = 0;  // heaviest edge some column of the unit may still take
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int c1 = s_c1[sec][i];
        if (PULL) {
          x.nd[i] = (int)min(dv[i], (uint32_t)c1);
          wl = max(wl, x.nd[i] - 1);
        } else {
          const bool on = ((m >> i) & 1u) && dv[i] < (uint32_t)c1 - 1u;
          x.nd[i] = on ? -(int)dv[i] : -0x7FFFFFFF;
          wl = max(wl, c1 + x.nd[i] - 1);
        }
      }
      x.sec = sec;
      x.at = v * nsec + sec;
      s_unit[wib][lane] = x;
      // the units of one item are neighbours: `lead` its first lane in the window, `cnt`
      // their number; the item's edges up to the largest limit among them
      uint32_t cnt = 1;
      bool lead = (uint32_t)lane < live;
      if (Gp > 8u) {
        const uint32_t prev = __shfl_up_sync(0xffffffffu, own, 1);
        lead = lead && (lane == 0 || prev != own);
        const uint32_t heads = __ballot_sync(0xffffffffu, lead);
        const uint32_t above = lane == 31 ? 0u : heads >> (lane + 1);
        const uint32_t end = above ? (uint32_t)(lane + __ffs(above)) : live;
        cnt = end > (uint32_t)lane ? end - lane : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_down_sync(0xffffffffu, wl, o);
          if ((uint32_t)(lane + o) < end) wl = max(wl, y);
        }
      }
      int64_t eb = 0;
      uint32_t work = 0;
      if (lead && wl > 0) {
        const int64_t e0 = lo + (int64_t)chunk * chunk_edges;
        const int64_t e1 = min(min(hi, count_upto(G, v, b1 - b0, (uint32_t)wl)), e0 + chunk_edges);
        if (e1 > e0) work = (uint32_t)(e1 - e0) * cnt;
        eb = b0 + e0;
      }
      const uint32_t scan = warp_incl_scan(work);
      const uint32_t tot = __shfl_sync(0xffffffffu, scan, 31);
      const uint32_t start = scan - work;
      // the items with work, in order; a pair's item follows from the starts below it
      const uint32_t busy = __ballot_sync(0xffffffffu, work != 0u);
      if (work) s_work[wib][__popc(busy & ((1u << lane) - 1u))] = BsWork{eb, start, (uint32_t)lane | cnt << 5 | ((0xFFFFu + cnt) / cnt) << 11};
      relaxed += tot;
      __syncwarp();
      const uint32_t mark = work ? start : 0xFFFFFFFFu;
      uint32_t before = 0;  // items that start before this round's pairs
      for (uint32_t j0 = 0; j0 < tot; j0 += 32 * BS_U) {
        uint32_t tu[BS_U], un[BS_U], at[BS_U];
        int tw[BS_U];
        uint4 ra[BS_U], rb[BS_U];
        bool ok[BS_U];
#pragma unroll
        for (int y = 0; y < BS_U; y++) {
          const uint32_t jb = j0 + (uint32_t)y * 32u, j = jb + lane;
          const uint32_t starts = __reduce_or_sync(0xffffffffu, mark - jb < 32u ? 1u << (mark - jb) : 0u);
          const uint32_t o = before + __popc(starts & (0xFFFFFFFFu >> (31 - lane))) - 1u;
          before += __popc(starts);
          const BsWork q = s_work[wib][o];
          ok[y] = j < tot;
          const uint32_t loc = ok[y] ? j - q.start : 0u;
          uint32_t e = loc, su = 0;
          if (Gp > 8u) {
            e = (loc * (q.unit >> 11)) >> 16;
            su = loc - e * ((q.unit >> 5) & 63u);
          }
          un[y] = (q.unit & 31u) + su;
          const int2 ed = ok[y] ? G.wedges[q.eb + e] : make_int2(0, 0);
          tu[y] = (uint32_t)ed.x;
          tw[y] = ed.y;
          ok[y] = ok[y] && tu[y] < G.V;
        }
#pragma unroll
        for (int y = 0; y < BS_U; y++) {
          at[y] = tu[y] * nsec + s_unit[wib][un[y]].sec;
          ra[y] = rb[y] = make_uint4(0, 0, 0, 0);
          if (ok[y]) {
            const uint4* row = (const uint4*)((PULL ? src_tab : dst_tab) + (uint64_t)at[y] * 8u);
            ra[y] = __ldcg(row);
            rb[y] = __ldcg(row + 1);
          }
        }
#pragma unroll
        for (int y = 0; y < BS_U; y++) {
          if (!ok[y]) continue;
          const BsUnit& q = s_unit[wib][un[y]];
          [[maybe_unused]] const int* c1 = s_c1[q.sec];
          const int w = tw[y];
          const uint32_t du[8] = {ra[y].x, ra[y].y, ra[y].z, ra[y].w, rb[y].x, rb[y].y, rb[y].z, rb[y].w};
          int best = -0x7FFFFFFF;
          if constexpr (PULL) {
            BsUnit& t = s_unit[wib][un[y]];
#pragma unroll
            for (int i = 0; i < 8; i++) best = max(best, t.nd[i] - (int)min(du[i], 0x7FFFFFFFu));
            if (best <= w) continue;
#pragma unroll
            for (int i = 0; i < 8; i++) {
              const uint32_t nd = du[i] + (uint32_t)w;
              if (du[i] < 0x7F000000u && nd < (uint32_t)t.nd[i]) {
                atomicMin(&t.nd[i], (int)nd);
                atomicMin(dst_tab + (uint64_t)t.at * 8u + i, nd);
              }
            }
          } else {
#pragma unroll
            for (int i = 0; i < 8; i++)
              best = __viaddmax_s32((int)min(du[i], (uint32_t)c1[i]), q.nd[i], best);
            if (best <= w) continue;
            uint32_t imp = 0, ann = 0;
#pragma unroll
            for (int i = 0; i < 8; i++)
              imp |= (int)min(du[i], (uint32_t)c1[i]) + q.nd[i] > w ? 1u << i : 0u;
            for (; imp; imp &= imp - 1u) {
              const int i = __ffs(imp) - 1;
              const int nd = w - q.nd[i];
              atomicMin(dst_tab + (uint64_t)at[y] * 8u + i, (uint32_t)nd);
              if (extend && nd + 1 < c1[i]) ann |= 1u << i;
            }
            if (ann) {
              const uint32_t col = q.sec * 8u;
              atomicOr(&fo[(uint64_t)tu[y] * Wm + (col >> 5)], ann << (col & 31u));
              any = 1u;
            }
          }
        }
      }
      __syncwarp();
    }
    if (lane == 0) base = taken + atomicAdd(&b->next[kind], take);
    base = __shfl_sync(0xffffffffu, base, 0);
   }
  }
  any = __reduce_or_sync(0xffffffffu, any);
  if (lane == 0 && any) b->ann = 1u;
  if (lane == 0 && relaxed) atomicAdd(&b->st_relax, relaxed);  // the same in every lane
  if (last_block(&b->arrived) && threadIdx.x == 0) {
    bs_advance(b);
    if (in_loop) cudaGraphSetConditional(loop, b->done ? 0u : 1u);
  }
}

// Whether a distance of the table (n words) exceeds `most`, so that a path over one edge more
// may have been too heavy for the search.
__global__ void k_bs_far(BsCtx* b, int64_t n, uint32_t most) {
  bool found = false;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t d = __ldcs(b->dist + i);
    found = found || (d > most && d != COST_INF);
  }
  if (found) b->far = 1u;
}

// Hop-bounded tables (n4 = V x Gp / 4 uint4 per table).  Before round r >= 1:
// table r + 1 := table r.
__global__ void k_bs_copy(BsCtx* b, int64_t n4) {
  if (b->done || b->round == 0u || b->round >= b->D) return;
  const uint4* src = (const uint4*)b->tab[b->round];
  uint4* dst = (uint4*)b->tab[b->round + 1u];
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n4;
       i += (int64_t)gridDim.x * blockDim.x)
    __stcs(dst + i, __ldcs(src + i));
}

}  // namespace gst
