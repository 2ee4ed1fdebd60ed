// edm_dyn.cuh — dynamics kernels (one BD step of DynamicsEngine.step,
// ed_mrdt/dynamics.py:2150-2465) for all replicas of an engine.
//
// Layout.  Every step the particles of every replica are counting-sorted into
// "slots" by a key: the reference cell cx*ny + cy of alive particles
// (dynamics.py:176-196: cx = int(x/cell_sx) clamped), and one extra bucket
// (key nx*ny) holding every particle that is not alive.  Replica r owns slots
// [particle_offset, +n_particles) and sort buckets [cell_offset, +nx*ny+1).
// Non-alive particles never take part in a pair computation
// (dynamics.py:680-681, 767-768, 850-851), so keeping them out of the cells
// leaves the neighbour sweeps with alive particles only; their reference
// cell is still stored per slot.  Slot arrays: position (float64 absolute, or
// float32 offset inside the cell), the cell, one flag byte (species |
// alive<<7) and the particle id.  Id-indexed arrays (bond partner, dye,
// photophysical state) do not move.
//
// Order independence.  The slot order inside a bucket comes from atomics and
// is not deterministic; nothing downstream depends on it:
//  - pair forces are summed per particle in the reference's own pair order
//    (its (j, i) pairs by ascending j, then its (i, j) pairs by neighbour-cell
//    ordinal and descending j; WCA terms before harmonic terms), recovered
//    from particle ids and cells;
//  - every random draw is keyed by particle ids, not by storage position;
//  - reaction passes are set-valued (catalysis) or per particle; the two
//    order-dependent rules (binding's greedy pair order, the recruitment cap
//    in index order) are resolved on small candidate lists sorted by the
//    reference's order key.
#pragma once

#include <type_traits>

#include "edm_common.cuh"

namespace edm {

constexpr int kBlock = 256;
constexpr int kSweepChunk = 128;  // slots per warp in the flag sweeps (4 per lane)
constexpr int kMaxPP = 32;        // recruitment-candidate, detachment and conversion passes per step
constexpr int kRecCap = 128;
constexpr int kBindCap = 512;

struct DevState {
  void* pos_pre;      // double2 (f64) or float2 (f32 offsets), slot order, before the move
  void* pos_post;     // same, after the move
  // f32 path: the float32 remainder of each offset (offset = hi + lo, hi in
  // pos_*); range tests read hi alone, exact arithmetic reads both
  short2* lo_pre;
  short2* lo_post;
  int32_t* cell_pre;  // reference cell of each slot, before the move
  int32_t* cell_post;
  const uint8_t* flags_old;
  uint8_t* flags;     // slot flags of the current step
  const int32_t* ids_old;
  int32_t* ids;       // global particle id of each slot, the top bit set in a tracked one
  int32_t* slot_of_id;  // slot of each tracked particle (a dye carrier; with binding, every one)
  int32_t* bond;      // id-indexed, global id or -1
  int32_t* cell_start;   // sort-bucket starts [n_buckets + 1]
  int32_t* cell_cursor;
  int32_t* cnt_next;     // bucket counts for the next step's sort
  int32_t* grid_cnt;     // density-grid counts (snapshot of the current pass)
  int32_t* grid_delta;   // pending changes of the current pass
  const double* hill;
  // draw thresholds: a keyed draw u = m 2^-53 with m >= the threshold is
  // rejected by its pass whatever the grid counts (threshold = ceil(b 2^53),
  // b = prob times the largest Hill factor of each rule of the pass)
  const uint64_t* pass_thr;  // [R][kMaxPP] per-particle passes, in schedule order
  const uint64_t* cat_thr;   // [R][EDM_MAX_CAT] catalytic passes
  int64_t* counters;     // [R][EDM_NCOUNTERS]
  uint32_t* status;
  const int64_t* d_step;
  // candidate buffers
  int32_t* rec_count;    // [R]
  int32_t* rec_id;       // [R][kRecCap] local id
  int32_t* rec_slot;     // [R][kRecCap]
  double* rec_xy;        // [R][kRecCap][2]
  int32_t* bind_count;   // [R]
  int64_t* bind_key;     // [R][kBindCap]
  int32_t* bind_ab;      // [R][kBindCap][2] local ids (a = reactant A role, b = B role)
  // complexes that dissociate in the binding pass (slot, partner's slot), replica
  // r's from its particle_offset up; from its last particle down the odd ones,
  // whose partner is alive or bound to another (no binding leaves one so, but a
  // state may hold one)
  int2* dis;
  int32_t* dis_count;    // [binding reactions][R][2]
  // catalytic contacts of the step: (enzyme slot, substrate-capable slot),
  // contact_cap per reaction.  With rep_contacts each replica has its own part
  // of the reaction's array, rep_contacts per particle and kRepContactsExtra, and
  // its own counts (k_react takes a replica per block); 0: one list per reaction
  // serves all replicas.
  int2* contacts;
  int32_t* contact_count;  // [EDM_MAX_CAT], or [R][EDM_MAX_CAT]
  int64_t contact_cap;      // per catalytic reaction
  int rep_contacts;
  const int64_t* rep_first;  // [R + 1] first slot of each replica
  const int32_t* chunk_rep;  // replica of the first slot of each kSweepChunk-slot chunk
  // slots that left their sort bucket's neighbourhood after the sort this step
  // (recruited, or placed by dissociation): per replica at particle_offset
  int32_t* moved;
  int32_t* moved_count;  // [R]
  // particles whose keyed draws pass some per-particle pass's bound this step:
  // (slot, bit mask of those passes, replica, local id); pl_index[slot] = its
  // entry.  With rep_pl replica r's entries start at its particle_offset.
  int4* pl;
  int32_t* pl_count;  // [1], or [R]
  int32_t* pl_index;
  int rep_pl;
  // per species: the density grids (bit g) that sense it in some replica
  uint32_t sensor_grids[EDM_MAX_SPECIES];
  // the contact search's sweepers (slot, replica) of this step (k_sweep_list)
  int2* sw_list;
  int32_t* sw_count;
  // per global grid cell: the adaptation field w (float64, on the adaptation
  // grid's cells) and the local-recruitment CDF (on a feedback grid's cells)
  double* adapt_w;
  double* local_cdf;
  int n_rep;
  int64_t n_slots;
};

// Tracked particles keep their entry of slot_of_id current through every sort.
// Nothing reads the others' entries, and their scattered 4-byte writes over the
// whole map were a fifth of the sort's time.
constexpr int32_t kTracked = (int32_t)0x80000000;
__device__ __forceinline__ int slot_id(const DevState& st, int64_t s) { return st.ids[s] & ~kTracked; }

// Particles a per-particle pass visits: the species set mask[1] of alive
// particles and mask[0] of particles that are not alive.
struct Match {
  uint32_t mask[2];
};
__device__ __forceinline__ bool matches(uint8_t f, const Match& m) {
  return ((fl_alive(f) ? m.mask[1] : m.mask[0]) >> fl_species(f)) & 1u;
}

// Flag sweep with warp-local compaction: each warp reads the flags of its
// kSweepChunk slots (4 per lane, one 32-bit load), gathers the matching
// slots in its shared-memory list (ballot + popc, no block barrier), then
// runs body(replica, slot) on them with every lane busy.  Launch with
// blockDim == kBlock and ceil(n_slots / (4*kBlock)) blocks.
template <typename Body>
__device__ __forceinline__ void sweep4(const DevState& st, const Match& m, Body body) {
  __shared__ int32_t list[kBlock / 32][kSweepChunk];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31)) * 4;
  if (w0 >= st.n_slots) return;  // whole warps only
  const int64_t s0 = w0 + (int64_t)lane * 4;
  uchar4 f4 = make_uchar4(0, 0, 0, 0);
  if (s0 < st.n_slots) f4 = *reinterpret_cast<const uchar4*>(st.flags + s0);
  const uint8_t f[4] = {f4.x, f4.y, f4.z, f4.w};
  const unsigned below = (1u << lane) - 1u;
  int n = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const bool hit = s0 + k < st.n_slots && matches(f[k], m);
    const unsigned bits = __ballot_sync(0xffffffffu, hit);
    if (hit) list[wid][n + __popc(bits & below)] = (int32_t)(s0 + k);
    n += __popc(bits);
  }
  __syncwarp();
  if (n == 0) return;
  const int r0 = st.chunk_rep[w0 / kSweepChunk];
  for (int q = lane; q < n; q += 32) {
    const int64_t s = list[wid][q];
    int r = r0;
    while (r + 1 < st.n_rep && st.rep_first[r + 1] <= s) ++r;
    body(r, s);
  }
}

// One atomicAdd per group of lanes adding 1 to the same address; returns
// the value each lane would have got from its own atomicAdd(addr, 1).
__device__ __forceinline__ int atomic_inc_aggregated(int32_t* addr) {
  const unsigned act = __activemask();
  const unsigned peers = __match_any_sync(act, (unsigned long long)(uintptr_t)addr);
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(peers) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(addr, __popc(peers));
  base = __shfl_sync(peers, base, leader);
  return base + __popc(peers & ((1u << lane) - 1u));
}

// ---- replica geometry --------------------------------------------------------
// The box side and the pair-list cutoff are read from the parameter block
// where they are used (rare branches), so they hold no registers meanwhile.
// Slot, particle and bucket offsets fit 32 bits (slot indices are int32).
struct Geo {
  const EdmDynParams* prm;
  int nx, ny, px, py;
  double sx, sy;
  float sxf, syf, inv_ny;
  int cbase, poff;
  int grave;  // bucket of non-alive particles
  __device__ __forceinline__ double Lx() const { return prm->Lx; }
  __device__ __forceinline__ double Ly() const { return prm->Ly; }
  __device__ __forceinline__ double cutoff_sq() const { return prm->cutoff_sq; }
  __device__ __forceinline__ explicit Geo(const EdmDynParams& p)
      : prm(&p), nx(p.nx), ny(p.ny), px(p.periodic_x), py(p.periodic_y),
        sx(p.cell_sx), sy(p.cell_sy), sxf((float)p.cell_sx),
        syf((float)p.cell_sy), inv_ny(0.0f), cbase((int)p.cell_offset), poff((int)p.particle_offset),
        grave(p.nx * p.ny) {
#ifdef __CUDA_ARCH__  // device-only intrinsic: the reciprocal without a division's slow path
    inv_ny = __frcp_rn((float)p.ny);
#endif
  }
};

// Asks for the lines of a replica's parameters that a step's kernels read
// whatever they do (its head, its grids, its key), by the block's first
// threads, before pdl_enter().
__device__ __forceinline__ void prefetch_params(const EdmDynParams& p) {
  const int t = threadIdx.x;
  if (t < 4) prefetch_l1(reinterpret_cast<const char*>(&p) + 128 * t);
  else if (t == 4) prefetch_l1(&p.seed);
  else if (t == 5) prefetch_l1(&p.grid[0]);
  else if (t == 6) prefetch_l1(&p.n_bind);
}

// Cell key c = cx * ny + cy -> (cx, cy) without an integer division: the
// float quotient (c + 0.5) / ny is within one of cx for any c < 2^24 and the
// remainder check corrects it, so the result is exact.
__device__ __forceinline__ void split_cell(int c, const Geo& g, int& cx, int& cy) {
  int q = __float2int_rz(((float)c + 0.5f) * g.inv_ny);
  int r = c - q * g.ny;
  if (r < 0) {
    --q;
    r += g.ny;
  } else if (r >= g.ny) {
    ++q;
    r -= g.ny;
  }
  cx = q;
  cy = r;
}

// float32 path: a cell offset o (float64) is stored as hi = its float32
// rounding, clamped into [0, cell side), and lo = o - hi as an int16 count of
// the quantum q = 2^(e - 37), 2^e <= side < 2^(e + 1).  |o - hi| stays within
// 1.5 float32 ulps of the side, 3 * 2^13 q, so lo fits, and hi + lo q is
// within q / 2 of o (3e-13 µm for a 0.165 µm cell).  The scalings by q are
// exact.
__device__ __forceinline__ int lo_exponent(float side_f) {
  return (int)((__float_as_uint(side_f) >> 23) & 0xFFu) - 127 - 37;
}
__device__ __forceinline__ double pow2(int e) { return __longlong_as_double((long long)(1023 + e) << 52); }
__device__ __forceinline__ double lo_value(short l, float side_f) { return (double)l * pow2(lo_exponent(side_f)); }
__device__ __forceinline__ void split_offset(double o, float side_f, float& hi, short& lo) {
  float h = (float)o;
  if (!(h >= 0.0f)) h = 0.0f;
  else if (h >= side_f) h = __int_as_float(__float_as_int(side_f) - 1);  // largest float below the side
  hi = h;
  int q = __double2int_rn((o - (double)h) * pow2(-lo_exponent(side_f)));
  q = q > 32767 ? 32767 : (q < -32767 ? -32767 : q);
  lo = (short)q;
}

// Absolute position of a slot (float64); lo is the f32 path's remainder array.
template <bool F64>
__device__ __forceinline__ void abs_pos(const void* pos, const short2* lo, const int32_t* cell, int64_t s,
                                        const Geo& g, double& x, double& y) {
  if constexpr (F64) {
    const double2 v = ((const double2*)pos)[s];
    x = v.x;
    y = v.y;
  } else {
    const float2 v = ((const float2*)pos)[s];
    const short2 l = lo[s];
    int cx, cy;
    split_cell(cell[s], g, cx, cy);
    x = __dadd_rn(__dmul_rn((double)cx, g.sx), __dadd_rn((double)v.x, lo_value(l.x, g.sxf)));
    y = __dadd_rn(__dmul_rn((double)cy, g.sy), __dadd_rn((double)v.y, lo_value(l.y, g.syf)));
  }
}

// Reference minimum-image separation (dynamics.py:199-216) of absolute points.
__device__ __forceinline__ double min_image_sq(double x1, double y1, double x2, double y2, const Geo& g,
                                               double& dx, double& dy) {
  dx = x1 - x2;
  dy = y1 - y2;
  if (g.px) {
    if (dx > 0.5 * g.Lx()) dx -= g.Lx();
    else if (dx < -0.5 * g.Lx()) dx += g.Lx();
  }
  if (g.py) {
    if (dy > 0.5 * g.Ly()) dy -= g.Ly();
    else if (dy < -0.5 * g.Ly()) dy += g.Ly();
  }
  return dx * dx + dy * dy;
}

// float32 separation of two cell-relative points, i in cell (cxi, cyi), j in
// cell key cj.
__device__ __forceinline__ float rel_sq_f32_xy(int cxi, int cyi, float2 oi, int cj, float2 oj, const Geo& g,
                                               float& dx, float& dy) {
  int cxj, cyj;
  split_cell(cj, g, cxj, cyj);
  int dcx = cxi - cxj, dcy = cyi - cyj;
  if (g.px) {
    if (2 * dcx > g.nx) dcx -= g.nx;
    else if (2 * dcx < -g.nx) dcx += g.nx;
  }
  if (g.py) {
    if (2 * dcy > g.ny) dcy -= g.ny;
    else if (2 * dcy < -g.ny) dcy += g.ny;
  }
  dx = __fmaf_rn((float)dcx, g.sxf, oi.x - oj.x);
  dy = __fmaf_rn((float)dcy, g.syf, oi.y - oj.y);
  return __fmaf_rn(dx, dx, dy * dy);
}

// float32 separation of two cell-relative points (cells ci, cj).
__device__ __forceinline__ float rel_sq_f32(int ci, float2 oi, int cj, float2 oj, const Geo& g, float& dx,
                                            float& dy) {
  int cxi, cyi;
  split_cell(ci, g, cxi, cyi);
  return rel_sq_f32_xy(cxi, cyi, oi, cj, oj, g, dx, dy);
}

// Squared separation of slots a and b in the given position array.
template <bool F64>
__device__ __forceinline__ double sep_sq(const void* pos, const int32_t* cell, int64_t a, int64_t b,
                                         const Geo& g) {
  if constexpr (F64) {
    const double2 pa = ((const double2*)pos)[a], pb = ((const double2*)pos)[b];
    double dx, dy;
    return min_image_sq(pa.x, pa.y, pb.x, pb.y, g, dx, dy);
  } else {
    float dx, dy;
    return (double)rel_sq_f32(cell[a], ((const float2*)pos)[a], cell[b], ((const float2*)pos)[b], g, dx, dy);
  }
}

// Replica r and slot s of this thread (block table of kBlock-slot tiles).
struct Tile {
  int r;
  int64_t s;
};
__device__ __forceinline__ Tile tile_of(const int2* blk) {
  const int2 b = blk[blockIdx.x];
  Tile t;
  t.r = b.x;
  t.s = (int64_t)(uint32_t)b.y + threadIdx.x;
  return t;
}

// Visit the slots of the 3x3 neighbour cells of cell c: f(slot, ordinal,
// dcx, dcy), ordinal = (dcx + 1) * 3 + (dcy + 1) as in dynamics.py:243-260.
// The cells of one neighbour column are consecutive sort buckets, so each
// column is one slot run (two where the column wraps in y); a slot's dcy
// follows from its bucket (its pre-move cell).
template <typename F>
__device__ __forceinline__ void for_neighbour_slots_box(const Geo& g, const DevState& st, int c, int dxlo, int dxhi,
                                                        int dylo, int dyhi, F f) {
  int cx, cy;
  split_cell(c, g, cx, cy);
  // rows cy+dylo .. cy+dyhi (dylo <= 0 <= dyhi) as one or two runs
  int ya0 = cy + dylo, yb0 = cy + dyhi, ya1 = 0, yb1 = -1;
  if (!g.py) {
    ya0 = ya0 < 0 ? 0 : ya0;
    yb0 = yb0 >= g.ny ? g.ny - 1 : yb0;
  } else if (ya0 < 0) {
    ya0 = 0;
    ya1 = yb1 = g.ny - 1;
  } else if (yb0 >= g.ny) {
    yb0 = g.ny - 1;
    ya1 = yb1 = 0;
  }
  for (int dcx = dxlo; dcx <= dxhi; ++dcx) {
    int ncx = cx + dcx;
    if (g.px) ncx = ncx < 0 ? ncx + g.nx : (ncx >= g.nx ? ncx - g.nx : ncx);
    else if (ncx < 0 || ncx >= g.nx) continue;
    const int col = ncx * g.ny;
    for (int run = 0; run < 2; ++run) {
      const int ya = run == 0 ? ya0 : ya1, yb = run == 0 ? yb0 : yb1;
      if (yb < ya) break;
      const int j0 = st.cell_start[g.cbase + col + ya], j1 = st.cell_start[g.cbase + col + yb + 1];
      for (int j = j0; j < j1; ++j) {
        int dcy = st.cell_pre[j] - col - cy;
        dcy = dcy > 1 ? dcy - g.ny : (dcy < -1 ? dcy + g.ny : dcy);
        f(j, (dcx + 1) * 3 + (dcy + 1), dcx, dcy);
      }
    }
  }
}

template <typename F>
__device__ __forceinline__ void for_neighbour_slots(const Geo& g, const DevState& st, int c, F f) {
  for_neighbour_slots_box(g, st, c, -1, 1, -1, 1, f);
}

// ---- density grids -----------------------------------------------------------
// int(x / s) as the reference computes it (a rounded float64 quotient,
// truncated), without the division when it cannot matter: the product x * inv
// lies within a few ulps of the quotient, so when it is farther than 1e-6
// from an integer both truncate to the same value; closer than that (about
// one call in 10^6) the quotient itself is taken.
__device__ __forceinline__ int grid_index(double x, double s, double inv) {
  const double q = x * inv;
  const double f = q - floor(q);
  return (f > 1e-6 && f < 1.0 - 1e-6) ? (int)q : (int)__ddiv_rn(x, s);
}

__device__ __forceinline__ int64_t grid_cell_of(const EdmGrid& G, double x, double y) {
  const int gx = clampi(grid_index(x, G.sx, G.inv_sx), G.nx);
  const int gy = clampi(grid_index(y, G.sy, G.inv_sy), G.ny);
  return G.offset + (int64_t)gx * G.ny + gy;
}

// Density of a grid cell holding k particles: the reference's k-fold
// sequential float64 sum of inv_area (dynamics.py:1685-1703).
__device__ __forceinline__ double kfold_density(int k, double inv_area) {
  double rho = 0.0;
  for (int i = 0; i < k; ++i) rho = __dadd_rn(rho, inv_area);
  return rho;
}

// Adaptation factor 1/(1 + (w/K)^n) of catalytic feedback rule `rule` at
// (x, y) (dynamics.py:1077-1083): w is read as adaptation_field[gx, gy] with
// the feedback grid's (gx, gy), i.e. at flat index gx * ny_adapt + gy of the
// adaptation grid (the host rejects grids where that leaves the array); w = 0
// without a PIP3 grid.
__device__ __forceinline__ double adapt_factor(const EdmDynParams& p, const double* __restrict__ w_all, int rule,
                                               double x, double y) {
  const EdmGrid& G = p.grid[p.rule[rule].grid];
  const int gx = clampi(grid_index(x, G.sx, G.inv_sx), G.nx);
  const int gy = clampi(grid_index(y, G.sy, G.inv_sy), G.ny);
  double w = 0.0;
  if (p.adapt_grid >= 0) {
    const EdmGrid& A = p.grid[p.adapt_grid];
    w = w_all[A.offset + (int64_t)gx * A.ny + gy];
  }
  if (p.adapt_K > 0) return __ddiv_rn(1.0, __dadd_rn(1.0, pow(__ddiv_rn(w, p.adapt_K), p.adapt_n)));
  return 1.0;
}

// Where a pass's grid changes go until the merge before the next pass that
// reads the grids: an array of pending changes per cell ...
struct DeltaArray {
  int32_t* delta;
  __device__ __forceinline__ void add(int64_t cell, int d) const { atomicAdd(&delta[cell], d); }
};
// ... or, for a block that has the replica to itself, a short list in shared
// memory (the array takes what finds it full).
constexpr int kDeltaList = 512;
struct DeltaList {
  int64_t* cell;
  int* d;
  int* n;
  int32_t* delta;
  __device__ __forceinline__ void add(int64_t c, int change) const {
    const int k = atomicAdd(n, 1);
    if (k < kDeltaList) {
      cell[k] = c;
      d[k] = change;
    } else {
      atomicAdd(&delta[c], change);
    }
  }
};

// Add d to every grid counting species sp, at (x, y).
template <typename Sink>
__device__ __forceinline__ void grid_add(const EdmDynParams& p, const Sink& sink, int sp, double x, double y, int d) {
  for (int g = 0; g < p.n_grids; ++g) {
    if (p.grid[g].sensor == sp) sink.add(grid_cell_of(p.grid[g], x, y), d);
  }
}

__device__ __forceinline__ double rule_factor(const EdmDynParams& p, int rule, const DevState& st, double x,
                                              double y) {
  const EdmRule& R = p.rule[rule];
  const int k = st.grid_cnt[grid_cell_of(p.grid[R.grid], x, y)];
  return hill_of(R, st.hill, k, st.status);
}

// Grid bookkeeping of a particle changing (species, alive) at one position.
template <typename Sink>
__device__ __forceinline__ void grid_change(const EdmDynParams& p, const Sink& sink, int sp_old, bool alive_old,
                                            int sp_new, bool alive_new, double x, double y) {
  if (alive_old) grid_add(p, sink, sp_old, x, y, -1);
  if (alive_new) grid_add(p, sink, sp_new, x, y, +1);
}

// Record a slot placed away from its sort bucket after this step's sort.
__device__ __forceinline__ void note_moved(const DevState& st, int r, const EdmDynParams& p, int64_t slot) {
  const int k = atomicAdd(&st.moved_count[r], 1);
  if (k < p.n_particles) st.moved[p.particle_offset + k] = (int32_t)slot;
}

// Next step's bucket counts when a particle changes bucket.
__device__ __forceinline__ void rebucket(const DevState& st, const Geo& g, int from, int to) {
  if (from == to) return;
  atomicAdd(&st.cnt_next[g.cbase + from], -1);
  atomicAdd(&st.cnt_next[g.cbase + to], 1);
}

// =============================================================================
// Sort: exclusive scan of the bucket counts, scatter into slots.
// =============================================================================
constexpr int kScanThreads = 512;
constexpr int kScanItems = 4;  // one int4 per thread: a warp touches 512 contiguous bytes
constexpr int kScanTile = kScanThreads * kScanItems;

// The kScanItems counts at [base, base + 4) (zero past n); arrays are
// 16-byte aligned and base is a multiple of 4.
__device__ __forceinline__ int4 load4(const int32_t* __restrict__ a, int64_t base, int64_t n) {
  if (base + 3 < n) return *reinterpret_cast<const int4*>(a + base);
  int4 v = make_int4(0, 0, 0, 0);
  if (base < n) v.x = a[base];
  if (base + 1 < n) v.y = a[base + 1];
  if (base + 2 < n) v.z = a[base + 2];
  return v;
}
__device__ __forceinline__ void store4(int32_t* __restrict__ a, int64_t base, int64_t n, int4 v) {
  if (base + 3 < n) {
    *reinterpret_cast<int4*>(a + base) = v;
    return;
  }
  if (base < n) a[base] = v.x;
  if (base + 1 < n) a[base + 1] = v.y;
  if (base + 2 < n) a[base + 2] = v.z;
}

// The same for the part of [i, i + 4) that lies in [lo, hi), i a multiple of 4.
__device__ __forceinline__ int4 load4_in(const int32_t* a, int64_t i, int64_t lo, int64_t hi) {
  if (i >= lo && i + 3 < hi) return *reinterpret_cast<const int4*>(a + i);
  int4 v = make_int4(0, 0, 0, 0);
  if (i >= lo && i < hi) v.x = a[i];
  if (i + 1 >= lo && i + 1 < hi) v.y = a[i + 1];
  if (i + 2 >= lo && i + 2 < hi) v.z = a[i + 2];
  if (i + 3 >= lo && i + 3 < hi) v.w = a[i + 3];
  return v;
}
__device__ __forceinline__ void store4_in(int32_t* a, int64_t i, int64_t lo, int64_t hi, int4 v) {
  if (i >= lo && i + 3 < hi) {
    *reinterpret_cast<int4*>(a + i) = v;
    return;
  }
  if (i >= lo && i < hi) a[i] = v.x;
  if (i + 1 >= lo && i + 1 < hi) a[i + 1] = v.y;
  if (i + 2 >= lo && i + 2 < hi) a[i + 2] = v.z;
  if (i + 3 >= lo && i + 3 < hi) a[i + 3] = v.w;
}

__device__ __forceinline__ int block_exclusive_scan(int v, int& total) {
  __shared__ int warp_sums[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[wid] = x;
  __syncthreads();
  if (wid == 0) {
    const int nw = blockDim.x >> 5;
    int w = lane < nw ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < nw) warp_sums[lane] = w;
  }
  __syncthreads();
  const int base = wid > 0 ? warp_sums[wid - 1] : 0;
  total = warp_sums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return base + x - v;
}

// Buffers the step clears before its kernels use them (density grids and
// their deltas, the placed-after-sort and contact counters, the draw and
// dissociation list lengths): cleared by the first scan kernel instead of one memset each.
struct StepZero {
  static constexpr int kCount = 7;
  int32_t* p[kCount];
  int64_t n[kCount];
};

__global__ void k_scan_reduce(const int32_t* __restrict__ cnt, int64_t n, int32_t* __restrict__ bsum, StepZero z) {
  for (int k = 0; k < StepZero::kCount; ++k)
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < z.n[k]; i += (int64_t)gridDim.x * blockDim.x)
      z.p[k][i] = 0;
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  const int4 c = load4(cnt, base, n);
  const int v = c.x + c.y + c.z + c.w;
  int total;
  block_exclusive_scan(v, total);
  if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}

// The whole scan in one launch for systems of small replicas, a block each (a
// replica's slots are contiguous, so its bucket starts count from its first
// slot): the block holds its counts in registers, a warp 128 of them per round.
// One launch of latency instead of three: a 5,000-slot system's scan 10.5 to 8 us,
// its whole step 25.0 to 23.7, one of 13,600 slots 27.5 to 27.1, 100 replicas of
// 538,000 65.1 to 64.2.  At 15,700 slots in one replica the two are even (29.8 and
// 29.7 us in float64, 27.1 and 27.7 in float32), with six rounds instead of four
// 22,900 slots take 33.0 us against 31.4 tiled: the line lies between.  With more
// replicas than SMs the blocks take turns and the gain is gone as well (scans of
// 16.0 and 16.0 us at 296 replicas, 17.6 against 15.1 at 600).
constexpr int kSmallScanRounds = 4;
constexpr int kSmallScan = 1024 * 4 * kSmallScanRounds - 4;
__global__ void __launch_bounds__(1024) k_scan_replica(const EdmDynParams* __restrict__ P, int32_t* cnt,
                                                     int32_t* __restrict__ start, int32_t* __restrict__ cursor,
                                                     StepZero z) {
  __shared__ int warp_sum[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const EdmDynParams& p = P[blockIdx.x];
  const int64_t lo = p.cell_offset, hi = lo + (int64_t)p.nx * p.ny + 1, first = lo & ~(int64_t)3;
  const int slot0 = (int)p.particle_offset;
  pdl_enter();
  for (int k = 0; k < StepZero::kCount; ++k)
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < z.n[k]; i += (int64_t)gridDim.x * blockDim.x)
      z.p[k][i] = 0;
  // warp w takes the rounds' 128-cell stretches one after another
  const int rounds = (int)((hi - first + 4095) / 4096);
  const int64_t w0 = first + (int64_t)wid * rounds * 128 + lane * 4;
  int4 v[kSmallScanRounds];
  int sum = 0;
#pragma unroll
  for (int k = 0; k < kSmallScanRounds; ++k) {
    v[k] = k < rounds ? load4_in(cnt, w0 + k * 128, lo, hi) : make_int4(0, 0, 0, 0);
    sum += v[k].x + v[k].y + v[k].z + v[k].w;
  }
  sum = __reduce_add_sync(0xffffffffu, sum);
  if (lane == 0) warp_sum[wid] = sum;
  __syncthreads();
  int run = slot0 + __reduce_add_sync(0xffffffffu, lane < wid ? warp_sum[lane] : 0);
#pragma unroll
  for (int k = 0; k < kSmallScanRounds; ++k) {
    if (k >= rounds) break;
    const int4 c = v[k];
    const int mine = c.x + c.y + c.z + c.w;
    int x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const int at = run + x - mine;
    const int64_t i = w0 + k * 128;
    const int4 st4 = make_int4(at, at + c.x, at + c.x + c.y, at + c.x + c.y + c.z);
    store4_in(start, i, lo, hi, st4);
    store4_in(cursor, i, lo, hi, st4);
    store4_in(cnt, i, lo, hi, make_int4(0, 0, 0, 0));
    run += __shfl_sync(0xffffffffu, x, 31);
  }
  // start[n]: the end of the last replica's last bucket
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) start[hi] = slot0 + (int)p.n_particles;
}

__global__ void k_scan_bsum(int32_t* __restrict__ bsum, int nb) {
  pdl_enter();
  int carry = 0;
  for (int off = 0; off < nb; off += blockDim.x) {
    const int i = off + threadIdx.x;
    const int v = i < nb ? bsum[i] : 0;
    int total;
    const int ex = block_exclusive_scan(v, total);
    if (i < nb) bsum[i] = carry + ex;
    carry += total;
  }
}

__global__ void k_scan_down(int32_t* __restrict__ cnt, int64_t n, const int32_t* __restrict__ bsum,
                            int32_t* __restrict__ start, int32_t* __restrict__ cursor) {
  pdl_enter();
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  const int4 c = load4(cnt, base, n);
  int total;
  const int run = block_exclusive_scan(c.x + c.y + c.z + c.w, total) + bsum[blockIdx.x];
  const int4 st4 = make_int4(run, run + c.x, run + c.x + c.y, run + c.x + c.y + c.z);
  store4(start, base, n, st4);
  store4(cursor, base, n, st4);
  store4(cnt, base, n, make_int4(0, 0, 0, 0));
  // the thread holding element n-1 writes the sentinel start[n]
  if (base < n && base + kScanItems >= n) start[n] = run + c.x + c.y + c.z + c.w;
  if (n == 0 && blockIdx.x == 0 && threadIdx.x == 0) start[0] = 0;
}

// A tile of one replica's slots: [first, end), the replica's first bucket and
// its last one (non-alive particles).  A kernel that takes these from the tile
// reads the slots' data one round trip earlier than through the replica's
// parameter block.
struct SlotTile {
  int32_t first, end, bucket0, grave;
};

// The counting sort's permutation.  Its time is the chain of round trips a
// warp makes (tile, slot, bucket cursor, stores) and its scattered stores, not
// the cursor atomics: ranks taken in the move instead of cursors measured the
// same.  So every load of a slot is issued before its cursor atomic (78 to 68
// us for 4.7M slots) and only tracked particles update slot_of_id (68 to 53).
// SPT tiles per block put SPT slots' loads and atomics in flight per thread.
template <bool F64, int BS, int SPT>
__global__ void __launch_bounds__(BS) k_scatter(const SlotTile* __restrict__ tiles, int ntiles, DevState st) {
  using Pos = typename std::conditional<F64, double2, float2>::type;
  int src[SPT], cl[SPT], id[SPT], dst[SPT], grave[SPT], bucket0[SPT];
  uint8_t fl[SPT];
  Pos pos[SPT];
  short2 lo[SPT];
#pragma unroll
  for (int k = 0; k < SPT; ++k) {
    src[k] = -1;
    const int tile = (int)blockIdx.x * SPT + k;
    if (tile >= ntiles) continue;
    const SlotTile t = tiles[tile];
    const int s = t.first + (int)threadIdx.x;
    if (s >= t.end) continue;
    src[k] = s;
    bucket0[k] = t.bucket0;
    grave[k] = t.grave;
  }
  pdl_enter();
#pragma unroll
  for (int k = 0; k < SPT; ++k) {
    const int s = src[k];
    if (s < 0) continue;
    cl[k] = st.cell_post[s];
    fl[k] = st.flags_old[s];
    id[k] = st.ids_old[s];
    pos[k] = ((const Pos*)st.pos_post)[s];
    if constexpr (!F64) lo[k] = st.lo_post[s];
  }
#pragma unroll
  for (int k = 0; k < SPT; ++k) {
    if (src[k] < 0) continue;
    // alive particles mostly have a cell to themselves: a plain atomic; the
    // non-alive ones all share their replica's last bucket: aggregated per warp
    dst[k] = fl_alive(fl[k]) ? atomicAdd(&st.cell_cursor[bucket0[k] + cl[k]], 1)
                             : atomic_inc_aggregated(&st.cell_cursor[grave[k]]);
  }
#pragma unroll
  for (int k = 0; k < SPT; ++k) {
    if (src[k] < 0) continue;
    const int d = dst[k];
    ((Pos*)st.pos_pre)[d] = pos[k];
    if constexpr (!F64) st.lo_pre[d] = lo[k];
    st.cell_pre[d] = cl[k];
    st.flags[d] = fl[k];
    st.ids[d] = id[k];
    if (id[k] & kTracked) st.slot_of_id[id[k] & ~kTracked] = d;
  }
}

// =============================================================================
// Forces + Ermak–McCammon move (dynamics.py:440-519, 665-816, 323-406).
// =============================================================================

// Enumerate the pair-force terms of slot s; pass `emit(key, fx, fy)`.
constexpr int kForceCand = 2;  // float32 force candidates listed per sweep

template <bool F64, typename Emit>
__device__ __forceinline__ void for_each_force_term(const EdmDynParams& p, const Geo& g, const DevState& st,
                                                    int64_t s, int sp, int id, Emit emit, int2* cand = nullptr,
                                                    int cand_stride = 0) {
  double xi = 0, yi = 0;
  float2 oi = make_float2(0.f, 0.f);
  if constexpr (F64) {
    const double2 v = ((const double2*)st.pos_pre)[s];
    xi = v.x;
    yi = v.y;
  } else {
    oi = ((const float2*)st.pos_pre)[s];
  }
  // pairs beyond both the pair-list cutoff and every potential's range carry no force
  const double range_sq = p.force_range_sq < g.cutoff_sq() ? p.force_range_sq : g.cutoff_sq();
  const float range_sqf = (float)range_sq * 1.0001f;
  // Only neighbour cells within that range of the particle can hold a force
  // partner (a partner in a skipped column or row is farther than its offset
  // to the cell side, itself beyond the range), so the sweep skips the others.
  // Range <= cutoff <= cell side keeps every partner inside the 3x3 block.
  const int c_pre = st.cell_pre[s];
  double ox, oy;
  if constexpr (F64) {
    int cx, cy;
    split_cell(c_pre, g, cx, cy);
    ox = xi - (double)cx * g.sx;
    oy = yi - (double)cy * g.sy;
  } else {
    ox = (double)oi.x;
    oy = (double)oi.y;
  }
  const double reach = p.force_reach;  // sqrt(range_sq) * 1.0001 + 1e-9, from the host
  const int dxlo = ox < reach ? -1 : 0, dxhi = ox > g.sx - reach ? 1 : 0;
  const int dylo = oy < reach ? -1 : 0, dyhi = oy > g.sy - reach ? 1 : 0;
  auto term = [&](int j, int ordinal, int dcx, int dcy) {
    {
      if (j == s) return;
      double dx, dy, dsq;
      if constexpr (F64) {
        const double2 v = ((const double2*)st.pos_pre)[j];
        dsq = min_image_sq(xi, yi, v.x, v.y, g, dx, dy);
        if (!(dsq < range_sq)) return;
      } else {
        // float32 range test (with a 1e-4 relative margin) on every
        // neighbour; the few pairs inside it get their separation in float64
        // from (cell, offset): the float32 sum below rounds at the ulp of a
        // cell side, a large fraction of |dx| for nearly coincident pairs
        const float2 oj = ((const float2*)st.pos_pre)[j];
        const float fdx = __fmaf_rn(-(float)dcx, g.sxf, oi.x - oj.x);
        const float fdy = __fmaf_rn(-(float)dcy, g.syf, oi.y - oj.y);
        const float fdsq = __fmaf_rn(fdx, fdx, fdy * fdy);
        if (!(fdsq < range_sqf)) return;
        const short2 li = st.lo_pre[s], lj = st.lo_pre[j];
        dx = (double)(-dcx) * g.sx +
             (((double)oi.x - (double)oj.x) + (double)((int)li.x - (int)lj.x) * pow2(lo_exponent(g.sxf)));
        dy = (double)(-dcy) * g.sy +
             (((double)oi.y - (double)oj.y) + (double)((int)li.y - (int)lj.y) * pow2(lo_exponent(g.syf)));
        dsq = dx * dx + dy * dy;
        if (!(dsq < range_sq)) return;
      }
      const uint8_t fj = st.flags[j];
      if (!fl_alive(fj)) return;
      const int spj = fl_species(fj);
      const double sig = p.sigma[sp * EDM_MAX_SPECIES + spj];
      if (!(sig > 0.0)) return;
      const int idj = slot_id(st, j) - (int)g.poff;
      const uint64_t order = idj < id ? (uint64_t)idj
                                      : ((1ull << 60) | ((uint64_t)ordinal << 32) | (uint64_t)(0xFFFFFFFFu - (uint32_t)idj));
      // The pair force itself is float64 on both paths: a pair inside force
      // range is rare (a few per thousand particles at the membrane
      // densities), and a capped move takes the direction of this force.
      if (p.use_wca) {
        const double eps = p.eps[sp * EDM_MAX_SPECIES + spj];
        if (eps > 0.0) {
          const double rcut2 = sig * sig * 1.2599210498948732;
          if (dsq < rcut2 && dsq >= 1e-30) {
            const double inv_r2 = 1.0 / dsq;
            const double s2 = sig * sig * inv_r2;
            const double s6 = s2 * s2 * s2;
            const double s12 = s6 * s6;
            double f = 24.0 * eps * (2.0 * s12 - s6) * inv_r2;
            const double fmax = 2400.0 * eps / (sig * sig);
            if (f > fmax) f = fmax;
            emit(order, f * dx, f * dy);
          }
        }
      }
      if (p.use_harmonic) {
        const double k = p.kharm[sp * EDM_MAX_SPECIES + spj];
        if (k > 0.0) {
          const double s2 = sig * sig;
          if (dsq < s2 && dsq >= 1e-30) {
            const double r = sqrt(dsq);
            const double f = k * (sig - r) / r;
            emit(order | (1ull << 62), f * dx, f * dy);
          }
        }
      }
    }
  };
  if constexpr (F64) {
    for_neighbour_slots_box(g, st, c_pre, dxlo, dxhi, dylo, dyhi, term);
  } else {
    // The sweep only lists the neighbours that pass the float32 range test
    // (rarely any) in cand[0], cand[cand_stride], ...; their float64
    // separation and force follow after it, so the sweep's loop does not
    // hold the float64 pair code's registers.  More than kForceCand of them
    // take further sweeps, each listing the next kForceCand in sweep order.
    for (int done = 0;; done += kForceCand) {
      int found = 0, kept = 0;
      for_neighbour_slots_box(g, st, c_pre, dxlo, dxhi, dylo, dyhi, [&](int j, int ordinal, int dcx, int dcy) {
        if (j == s) return;
        const float2 oj = ((const float2*)st.pos_pre)[j];
        const float fdx = __fmaf_rn(-(float)dcx, g.sxf, oi.x - oj.x);
        const float fdy = __fmaf_rn(-(float)dcy, g.syf, oi.y - oj.y);
        if (!(__fmaf_rn(fdx, fdx, fdy * fdy) < range_sqf)) return;
        const int rank = found++;
        if (rank >= done && rank < done + kForceCand) cand[(kept++) * cand_stride] = make_int2(j, ordinal);
      });
      for (int k = 0; k < kept; ++k) {
        const int2 e = cand[k * cand_stride];
        term(e.x, e.y, e.y / 3 - 1, e.y % 3 - 1);
      }
      if (found <= done + kForceCand) break;
    }
  }
}

// D(x) and grad D at an absolute position (dynamics.py:440-519; sine-x field).
__device__ __forceinline__ void dfield(const EdmDynParams& p, int sp, double x, double y, double& D, double& gx,
                                       double& gy) {
  const double base = p.D_base[sp];
  double factor = 1.0, gfx = 0.0, gfy = 0.0;
  if (p.dfield == EDM_DFIELD_REGIONS) {
    for (int reg = 0; reg < p.n_regions; ++reg) {
      const double dxc = x - p.reg_cx[reg], dyc = y - p.reg_cy[reg];
      const double dsq = dxc * dxc + dyc * dyc;
      const double d = dsq > 1e-30 ? sqrt(dsq) : 1e-15;
      const double arg = (d - p.reg_r[reg]) / p.smooth_w;
      double sig, dsig;
      if (arg > 100.0) {
        sig = 0.0;
        dsig = 0.0;
      } else if (arg < -100.0) {
        sig = 1.0;
        dsig = 0.0;
      } else {
        const double ea = exp(arg);
        const double den = 1.0 + ea;
        sig = 1.0 / den;
        dsig = -ea / (den * den * p.smooth_w);
      }
      const double local = 1.0 + (p.reg_f[reg] - 1.0) * sig;
      if (sig > 0.01) {
        factor = local;
        const double inv_d = 1.0 / d;
        gfx = (p.reg_f[reg] - 1.0) * dsig * dxc * inv_d;
        gfy = (p.reg_f[reg] - 1.0) * dsig * dyc * inv_d;
        break;
      }
    }
    D = base * factor;
    gx = base * gfx;
    gy = base * gfy;
  } else if (p.dfield == EDM_DFIELD_SINE_X) {
    const double w = 2.0 * 3.141592653589793 / p.sine_wavelength;
    const double ph = w * x;
    double sn, cs;
    sincos(ph, &sn, &cs);
    D = base * (1.0 + p.sine_amp * sn);
    gx = base * p.sine_amp * w * cs;
    gy = 0.0;
  } else {
    D = base * factor;
    gx = base * gfx;
    gy = base * gfy;
  }
}

// dfield out of line, for the float32 move: most systems have no D(x) field,
// and the field's float64 code would otherwise share the move's registers.
__device__ __noinline__ void dfield_call(const EdmDynParams& p, int sp, double x, double y, double& D, double& gx,
                                         double& gy) {
  dfield(p, sp, x, y, D, gx, gy);
}

// BS threads per block over tiles of BS slots; MINB resident blocks per SM
// requested from the register allocator (1 = no constraint).
template <bool F64, int BS, int MINB>
__global__ void __launch_bounds__(BS, MINB) k_move(const EdmDynParams* __restrict__ P, const int2* __restrict__ blk,
                                                 DevState st) {
  const Tile t = tile_of(blk);
  const EdmDynParams& p = P[t.r];
  const int64_t s = t.s;
  prefetch_params(p);
  const Geo g(p);
  const bool in = s < p.particle_offset + p.n_particles;
  pdl_enter();
  if (!in) return;
  const uint8_t f = st.flags[s];
  const int c = st.cell_pre[s];
  if (!fl_alive(f)) {  // dead / dormant particles do not move (dynamics.py:360)
    if constexpr (F64) {
      ((double2*)st.pos_post)[s] = ((const double2*)st.pos_pre)[s];
    } else {
      ((float2*)st.pos_post)[s] = ((const float2*)st.pos_pre)[s];
      st.lo_post[s] = st.lo_pre[s];
    }
    st.cell_post[s] = c;
    atomic_inc_aggregated(&st.cnt_next[g.cbase + g.grave]);
    return;
  }
  const int sp = fl_species(f);
  // the float32 path reads its id and the step index after the force sweep,
  // which needs neither, so that they hold no registers during it
  int id = 0;
  int64_t step = 0;
  if constexpr (F64) {
    id = slot_id(st, s) - (int)g.poff;
    step = *st.d_step;
  }

  // Pair forces.  The float64 path sums them in the reference's accumulation
  // order (a sum of two terms is the same either way, so only three or more
  // terms are re-summed in order).  The float32 path sums them in 2^-20
  // fixed point, exact and independent of the sweep order, so runs repeat
  // bit for bit.
  double Fx = 0.0, Fy = 0.0;
  long long qx = 0, qy = 0;
  int nterms = 0;
  __shared__ int2 cand_smem[F64 ? 1 : kForceCand * BS];
  for_each_force_term<F64>(p, g, st, s, sp, id, [&](uint64_t, double fx, double fy) {
    ++nterms;
    if constexpr (F64) {
      Fx += fx;
      Fy += fy;
    } else {
      qx += __double2ll_rn(fx * 0x1p20);
      qy += __double2ll_rn(fy * 0x1p20);
    }
  }, cand_smem + threadIdx.x, BS);
  if constexpr (F64) {
    if (nterms > 2) {
      Fx = 0.0;
      Fy = 0.0;
      uint64_t last = 0;
      bool first = true;
      for (int k = 0; k < nterms; ++k) {
        uint64_t best = ~0ull;
        double bx = 0.0, by = 0.0;
        for_each_force_term<F64>(p, g, st, s, sp, id, [&](uint64_t key, double fx, double fy) {
          if ((first || key > last) && key < best) {
            best = key;
            bx = fx;
            by = fy;
          }
        });
        Fx += bx;
        Fy += by;
        last = best;
        first = false;
      }
    }
  } else if (nterms > 0) {  // most particles have no partner in force range
    Fx = (double)qx * 0x1p-20;
    Fy = (double)qy * 0x1p-20;
  }

  double x = 0.0, y = 0.0;
  // the float32 path needs the absolute position here only for a D(x) field
  if (F64 || p.dfield != EDM_DFIELD_NONE) abs_pos<F64>(st.pos_pre, st.lo_pre, st.cell_pre, s, g, x, y);
  double Di, gDx, gDy;
  if constexpr (F64) {
    dfield(p, sp, x, y, Di, gDx, gDy);
  } else if (p.dfield == EDM_DFIELD_NONE) {
    Di = p.D_base[sp];
    gDx = gDy = 0.0;
  } else {
    dfield_call(p, sp, x, y, Di, gDx, gDy);
  }
  const double dt = p.dt;
  int newc;
  if constexpr (F64) {
    const U2 z = normal2(p.seed, step, EDM_S_BD_NORMAL, (uint64_t)id);
    const double sn = sqrt(2.0 * Di * dt);
    double dxt = gDx * dt, dyt = gDy * dt;
    dxt += sn * z.u0;
    dyt += sn * z.u1;
    dxt += Di * Fx * dt;
    dyt += Di * Fy * dt;
    const double dr2 = dxt * dxt + dyt * dyt;
    if (dr2 > p.max_disp_sq) {
      const double scale = p.max_disp / sqrt(dr2);
      dxt *= scale;
      dyt *= scale;
    }
    x += dxt;
    y += dyt;
    if (g.px) x = py_fmod(x, g.Lx());
    else if (x < 0.0) x = -x;
    else if (x >= g.Lx()) x = 2.0 * g.Lx() - x;
    if (g.py) y = py_fmod(y, g.Ly());
    else if (y < 0.0) y = -y;
    else if (y >= g.Ly()) y = 2.0 * g.Ly() - y;
    if (!isfinite(x) || !isfinite(y)) set_status(st.status, EDM_STATUS_NONFINITE);
    ((double2*)st.pos_post)[s] = make_double2(x, y);
    newc = cell_index(x, g.sx, g.nx) * g.ny + cell_index(y, g.sy, g.ny);
  } else {
    id = slot_id(st, s) - (int)g.poff;
    step = *st.d_step;
    float z0, z1;
    normal2_f32(p.seed, step, EDM_S_BD_NORMAL, (uint64_t)id, z0, z1);
    const float Dif = (float)Di, dtf = (float)dt;
    const float sn = sqrtf(2.0f * Dif * dtf);
    float dxt = __fmaf_rn(sn, z0, __fmaf_rn((float)gDx, dtf, Dif * (float)Fx * dtf));
    float dyt = __fmaf_rn(sn, z1, __fmaf_rn((float)gDy, dtf, Dif * (float)Fy * dtf));
    const float dr2 = __fmaf_rn(dxt, dxt, dyt * dyt);
    double ddx = (double)dxt, ddy = (double)dyt;
    if (dr2 > (float)(p.max_disp_sq * 0.999)) {
      // at (or within rounding of) the displacement cap the move keeps only
      // its direction: form and cap it in float64 as dynamics.py:378-385 do
      ddx = gDx * dt;
      ddy = gDy * dt;
      const double sn64 = sqrt(2.0 * Di * dt);
      ddx += sn64 * (double)z0;
      ddy += sn64 * (double)z1;
      ddx += Di * Fx * dt;
      ddy += Di * Fy * dt;
      const double d2 = ddx * ddx + ddy * ddy;
      if (d2 > p.max_disp_sq) {
        const double scale = p.max_disp / sqrt(d2);
        ddx *= scale;
        ddy *= scale;
      }
    }
    // the new offset in float64 from hi + lo, carried into the next cell
    // against the float64 cell side, then stored as hi + lo again
    const float2 oh = ((const float2*)st.pos_pre)[s];
    const short2 ol = st.lo_pre[s];
    int cx, cy;
    split_cell(c, g, cx, cy);
    double ax = ((double)oh.x + lo_value(ol.x, g.sxf)) + ddx;
    double ay = ((double)oh.y + lo_value(ol.y, g.syf)) + ddy;
    if (!(ax >= 0.0 && ax < g.sx)) {
      const int k = (int)floor(ax / g.sx);
      cx += k;
      ax -= (double)k * g.sx;
    }
    if (!(ay >= 0.0 && ay < g.sy)) {
      const int k = (int)floor(ay / g.sy);
      cy += k;
      ay -= (double)k * g.sy;
    }
    if (g.px) {  // |cx| stays within 64 cells of the box: a few wraps at most
      while (cx >= g.nx) cx -= g.nx;
      while (cx < 0) cx += g.nx;
    } else if (cx < 0 || cx >= g.nx) {  // reflecting wall, in float64
      double bx = (double)cx * g.sx + ax;
      if (bx < 0.0) bx = -bx;
      else if (bx >= g.Lx()) bx = 2.0 * g.Lx() - bx;
      cx = cell_index(bx, g.sx, g.nx);
      ax = bx - (double)cx * g.sx;
    }
    if (g.py) {
      while (cy >= g.ny) cy -= g.ny;
      while (cy < 0) cy += g.ny;
    } else if (cy < 0 || cy >= g.ny) {
      double by = (double)cy * g.sy + ay;
      if (by < 0.0) by = -by;
      else if (by >= g.Ly()) by = 2.0 * g.Ly() - by;
      cy = cell_index(by, g.sy, g.ny);
      ay = by - (double)cy * g.sy;
    }
    if (!isfinite(ax) || !isfinite(ay)) set_status(st.status, EDM_STATUS_NONFINITE);
    float2 o;
    short2 l;
    split_offset(ax, g.sxf, o.x, l.x);
    split_offset(ay, g.syf, o.y, l.y);
    ((float2*)st.pos_post)[s] = o;
    st.lo_post[s] = l;
    newc = cx * g.ny + cy;
    x = (double)cx * g.sx + ax;
    y = (double)cy * g.sy + ay;
  }
  st.cell_post[s] = newc;
  atomicAdd(&st.cnt_next[g.cbase + newc], 1);  // result unused: a fire-and-forget reduction
  // grid_add over only the grids that can sense this species (most species have none)
  for (uint32_t gm = st.sensor_grids[sp]; gm; gm &= gm - 1) {
    const int gi = __ffs(gm) - 1;
    if (p.grid[gi].sensor == sp) atomicAdd(&st.grid_cnt[grid_cell_of(p.grid[gi], x, y)], 1);
  }
}

// =============================================================================
// Reactions.
// =============================================================================

// Catalytic contacts (pairs of the reference's pre-move pair list, dynamics.py
// :219-278, in post-move contact).  During the catalytic passes enzymes keep
// their species and nobody moves or dies, so pass c needs the pairs (enzyme
// of species E_c, partner) within c's contact radius whose partner holds c's
// substrate S_c when pass c runs:
// * direct pairs, whose partner holds S_c at the step start, are found by
//   one sweep after the move, from the rarer side of each reaction: the
//   alive particles of the sweeping species (E_c or S_c) visit their
//   neighbour cells for the other species.  Both distance tests are
//   symmetric in the two particles (the float32 differences change sign
//   exactly), so either side finds the same pairs.  A particle that a
//   dissociation of the step woke lies in the bucket of the non-alive ones,
//   where no neighbour sweep meets it: woken_contacts looks from it for the
//   sweepers around the cell it was sorted from;
// * late pairs, whose partner an earlier catalytic pass of the step turns
//   into S_c, are few: the pass that converts a particle looks up its
//   enzymes of the later reactions at once (late_contacts).
// A pair is filed only when its keyed draw for the pass lies below the pass's
// threshold (the pass rejects it otherwise).  A pair can be filed twice (a
// partner converted away and back); the passes accept a substrate once, so
// duplicates change nothing.
struct CatLists {
  // byte [sweeper species][other species]: the reactions whose direct pairs
  // the first sweeps for among the second
  uint32_t rx_of[EDM_MAX_SPECIES * EDM_MAX_SPECIES / 4];
  uint32_t partners[EDM_MAX_SPECIES];  // species the sweeper species looks for
  uint32_t from_enzyme;                // reactions swept from the enzyme side
  uint32_t woken;                      // a dissociation can wake a species that sweeps look for: bit 0; among those
                                       // a sweeping one: bit 1
};
static_assert(EDM_MAX_CAT <= 8, "rx_of holds a reaction set per byte");

// Whether pass c's keyed draw for the pair of local ids (a, b) of replica r
// lies below the pass's threshold.  The pass rejects the pair otherwise,
// whatever the state, so a pair whose draw fails is not filed.
__device__ __forceinline__ bool cat_draw_passes(const EdmDynParams& p, const DevState& st, int r, int c, int a,
                                                int b, int64_t step) {
  const uint32_t lo = a < b ? a : b, hi = a < b ? b : a;
  return draw_u53(p.seed, step, EDM_S_CAT + c, lo, hi) < st.cat_thr[(int64_t)r * EDM_MAX_CAT + c];
}

// Neighbour sweep of one slot by G lanes (G divides 32, one group of G lanes
// per slot; every lane of the warp calls it, `have` false for a group without
// a slot).  The alive slots of the 3x3 block around cell c are three
// consecutive runs, one per neighbour column (and three more where the block
// wraps in y); the group's lanes take consecutive slots of the runs laid end
// to end, so neighbouring lanes read neighbouring addresses and a lane is idle
// only in the last round.  f(j, valid, column, col + cy) is called by the
// whole warp, column = dcx + 1; the slot's row offset is
// row_offset(cell_pre[j] - (col + cy), g).
template <int G, typename F>
__device__ __forceinline__ void for_neighbour_slots_grouped(const Geo& g, const DevState& st, int c, bool have, F f) {
  const int lane = threadIdx.x & (G - 1);
  int cx, cy;
  split_cell(c, g, cx, cy);
  int ya = cy - 1, yb = cy + 1, wrapped = -1;  // the row that wraps in y
  if (ya < 0) {
    ya = 0;
    wrapped = g.ny - 1;
  } else if (yb >= g.ny) {
    yb = g.ny - 1;
    wrapped = 0;
  }
  if (!have || !g.py) wrapped = -1;
  for (int part = 0; part < 2; ++part) {
    int lo[3], len[3], base[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      int ncx = cx + d - 1;
      bool in = have;
      if (g.px) ncx = ncx < 0 ? ncx + g.nx : (ncx >= g.nx ? ncx - g.nx : ncx);
      else in = in && ncx >= 0 && ncx < g.nx;
      lo[d] = len[d] = 0;
      base[d] = ncx * g.ny + cy;
      if (in) {
        const int32_t* b = st.cell_start + g.cbase + ncx * g.ny;
        lo[d] = b[ya];
        len[d] = b[yb + 1] - lo[d];
      }
    }
    const int n0 = len[0], n1 = n0 + len[1], n = n1 + len[2];
    lo[1] -= n0;
    lo[2] -= n1;
    const int most = __reduce_max_sync(0xffffffffu, n);
    for (int q0 = 0; q0 < most; q0 += G) {
      const int q = q0 + lane;
      const bool a1 = q >= n0, a2 = q >= n1;
      f(q + (a2 ? lo[2] : (a1 ? lo[1] : lo[0])), q < n, a2 ? 2 : (a1 ? 1 : 0), a2 ? base[2] : (a1 ? base[1] : base[0]));
    }
    if (!__any_sync(0xffffffffu, wrapped >= 0)) break;
    have = wrapped >= 0;  // the second part: the wrapped row alone
    ya = yb = wrapped >= 0 ? wrapped : 0;
    wrapped = -1;
  }
}

__device__ __forceinline__ int row_offset(int d, const Geo& g) {
  return d > 1 ? d - g.ny : (d < -1 ? d + g.ny : d);
}

// The alive-or-not species matches among the BLK * SPT slots from s0 (below
// end), gathered in the block's shared list in any order.
template <int BLK, int SPT>
__device__ __forceinline__ void gather_matching(const DevState& st, const Match& m, int64_t s0, int64_t end,
                                                int32_t* list, int& n_list) {
  uint8_t f[SPT];
#pragma unroll
  for (int k = 0; k < SPT; ++k) {
    const int64_t s = s0 + k * BLK + threadIdx.x;
    f[k] = s < end ? st.flags[s] : (uint8_t)0;
  }
  const int lane = threadIdx.x & 31;
  unsigned hits = 0;
#pragma unroll
  for (int k = 0; k < SPT; ++k)
    if (s0 + k * BLK + threadIdx.x < end && matches(f[k], m)) hits |= 1u << k;
  // one shared atomic per warp: lane l's hits go after those of the lanes below
  const int mine = __popc(hits);
  int upto = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += y;
  }
  const int total = __shfl_sync(0xffffffffu, upto, 31);
  if (total == 0) return;
  int at = 0;
  if (lane == 0) at = atomicAdd(&n_list, total);
  at = __shfl_sync(0xffffffffu, at, 0) + upto - mine;
  for (; hits; hits &= hits - 1) list[at++] = (int32_t)(s0 + (__ffs(hits) - 1) * BLK + threadIdx.x);
}

// Where replica r's listed contacts go.
constexpr int kRepContactsExtra = 4096;
struct ContactOut {
  int2* list;      // reaction c's part starts at list + c * stride
  int64_t stride;
  int64_t cap;
  int32_t* count;  // [EDM_MAX_CAT]
  uint32_t* status;
  __device__ __forceinline__ void file(int c, int e, int sub) const {
    const int q = atomicAdd(&count[c], 1);
    if (q < cap) list[(int64_t)c * stride + q] = make_int2(e, sub);
    else set_status(status, EDM_STATUS_CONTACT_CAP);
  }
};
__device__ __forceinline__ ContactOut contact_out(const DevState& st, const EdmDynParams& p, int r) {
  ContactOut o{st.contacts, st.contact_cap, st.contact_cap, st.contact_count, st.status};
  if (st.rep_contacts) {
    const int64_t off = (int64_t)st.rep_contacts * p.particle_offset + (int64_t)kRepContactsExtra * r;
    o.list += off;
    o.cap = r + 1 < st.n_rep ? (int64_t)st.rep_contacts * p.n_particles + kRepContactsExtra : st.contact_cap - off;
    o.count += (int64_t)r * EDM_MAX_CAT;
  }
  return o;
}

// A warp's pairs (sweeper, neighbour, replica) that passed the pre-move test
// of the sweep.  About one neighbour in six does, so the rest of the work
// (post-move contact, keyed draw, listing) is done 32 pairs at a time with
// every lane busy.
struct ContactQueue {
  int2 pair[64];
  int32_t rep[64];
};

// The first k <= 32 pairs of the queue: the post-move contact radius of each
// reaction the pair meets, then the reaction's keyed draw; the pairs below
// the pass's threshold are listed.
template <bool F64>
__device__ __forceinline__ void finish_contacts(const EdmDynParams* __restrict__ P, const DevState& st,
                                                const CatLists& L, const uint8_t* rx_of, const ContactQueue& Q,
                                                int k) {
  const int lane = threadIdx.x & 31;
  if (lane >= k) return;
  const int2 sj = Q.pair[lane];
  const int r = Q.rep[lane];
  const EdmDynParams& p = P[r];
  const Geo g(p);
  uint32_t bits = rx_of[fl_species(st.flags[sj.x]) * EDM_MAX_SPECIES + fl_species(st.flags[sj.y])];
  const int ids = slot_id(st, sj.x) - g.poff, idj = slot_id(st, sj.y) - g.poff;
  // the sweeper first, as the pre-move test (both differences change sign
  // exactly when the pair is swept from its other side)
  const double d2 = sep_sq<F64>(st.pos_post, st.cell_post, sj.x, sj.y, g);
  for (; bits; bits &= bits - 1) {
    const int c = __ffs(bits) - 1;
    if (d2 > p.cat[c].contact_sq) continue;
    if (!cat_draw_passes(p, st, r, c, ids, idj, *st.d_step)) continue;
    const bool from_enzyme = (L.from_enzyme >> c) & 1u;
    contact_out(st, p, r).file(c, from_enzyme ? sj.x : sj.y, from_enzyme ? sj.y : sj.x);
  }
}

// Adds the pair (s, j) of replica r to the warp's queue in the lanes with `hit`
// (every lane of the warp calls it); 32 waiting pairs are finished at once.
template <bool F64>
__device__ __forceinline__ void queue_contact(const EdmDynParams* __restrict__ P, const DevState& st,
                                              const CatLists& L, const uint8_t* rx_of, bool hit, int s, int j, int r,
                                              ContactQueue& Q, int& queued) {
  const int lane = threadIdx.x & 31;
  const unsigned who = __ballot_sync(0xffffffffu, hit);
  if (!who) return;
  if (hit) {
    const int at = queued + __popc(who & ((1u << lane) - 1u));
    Q.pair[at] = make_int2(s, j);
    Q.rep[at] = r;
  }
  queued += __popc(who);
  __syncwarp();
  if (queued < 32) return;  // at most 31 + 32 wait here
  finish_contacts<F64>(P, st, L, rx_of, Q, 32);
  __syncwarp();
  queued -= 32;
  if (lane < queued) {
    const int2 e = Q.pair[32 + lane];
    const int32_t k = Q.rep[32 + lane];
    Q.pair[lane] = e;
    Q.rep[lane] = k;
  }
  __syncwarp();
}

// Sweeper s of replica r (one per group of G lanes, `have` false for a group
// without one) against its neighbour slots: alive, of a species it sweeps
// for, within the pre-move cutoff.  The pairs go to the warp's queue, `queued`
// of them wait there.
template <bool F64, int G>
__device__ __forceinline__ void contact_sweep(const EdmDynParams* __restrict__ P, const DevState& st,
                                              const CatLists& L, const uint8_t* rx_of, int r, int s, bool have,
                                              ContactQueue& Q, int& queued) {
  const EdmDynParams& p = P[r];
  const Geo g(p);
  const uint32_t pmask = L.partners[fl_species(st.flags[s])];
  const int c_pre = st.cell_pre[s];
  float2 oi = make_float2(0.f, 0.f);
  double2 xi = make_double2(0.0, 0.0);
  // a float is below the float64 bound exactly when it is below the smallest
  // float at or above it: the float32 path compares in float32
  const float cutoff_f = __double2float_ru(p.cutoff_sq);
  if constexpr (F64) xi = ((const double2*)st.pos_pre)[s];
  else oi = ((const float2*)st.pos_pre)[s];
  for_neighbour_slots_grouped<G>(g, st, c_pre, have, [&](int j, bool valid, int column, int base) {
    bool hit = false;
    if (valid) {
      const uint8_t fj = st.flags[j];
      if constexpr (F64) {
        const double2 v = ((const double2*)st.pos_pre)[j];
        double dx, dy;
        hit = fl_alive(fj) && ((pmask >> fl_species(fj)) & 1u) && j != s &&
              min_image_sq(xi.x, xi.y, v.x, v.y, g, dx, dy) < g.cutoff_sq();
      } else {
        const float2 o = ((const float2*)st.pos_pre)[j];
        const int dcy = row_offset(st.cell_pre[j] - base, g);
        // j sits in the neighbour cell at (column - 1, dcy)
        const float fdx = __fmaf_rn(-(float)(column - 1), g.sxf, oi.x - o.x);
        const float fdy = __fmaf_rn(-(float)dcy, g.syf, oi.y - o.y);
        hit = fl_alive(fj) && ((pmask >> fl_species(fj)) & 1u) && j != s &&
              __fmaf_rn(fdx, fdx, fdy * fdy) < cutoff_f;
      }
    }
    queue_contact<F64>(P, st, L, rx_of, hit, s, j, r, Q, queued);
  });
}

// The contacts that the neighbour sweeps cannot meet: particles that this step's
// binding passes woke (st.moved; nobody else has been placed yet), as the
// neighbour of a sweeper.  The warp's groups of G lanes take a woken particle
// each, part `part` of `parts` of the replica's, and walk the sweepers among its
// neighbours and, where a woken particle can be one, among the woken.  One that
// was alive before as well is met twice, which a pass does not mind.
template <bool F64, int G>
__device__ __noinline__ void woken_contacts(const EdmDynParams* __restrict__ P, const DevState& st, const CatLists& L,
                                            const uint8_t* rx_of, int r, int part, int parts, ContactQueue& Q) {
  const EdmDynParams& p = P[r];
  const Geo g(p);
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int32_t* woken = st.moved + p.particle_offset;
  const int n = min(st.moved_count[r], (int)p.n_particles);
  int queued = 0;
  for (int t0 = (part * warps + (threadIdx.x >> 5)) * (32 / G); t0 < n; t0 += parts * warps * (32 / G)) {
    const int t = t0 + lane / G;
    const int w = woken[t < n ? t : t0];
    const uint8_t fw = st.flags[w];
    const bool have = t < n && fl_alive(fw);
    auto meets = [&](int j) {
      const uint8_t fj = st.flags[j];
      return fl_alive(fj) && j != w && rx_of[fl_species(fj) * EDM_MAX_SPECIES + fl_species(fw)] != 0 &&
             sep_sq<F64>(st.pos_pre, st.cell_pre, j, w, g) < g.cutoff_sq();
    };
    for_neighbour_slots_grouped<G>(g, st, st.cell_pre[w], have, [&](int j, bool valid, int, int) {
      queue_contact<F64>(P, st, L, rx_of, valid && meets(j), j, w, r, Q, queued);
    });
    if (!(L.woken & 2u)) continue;
    for (int k0 = 0; k0 < n; k0 += G) {
      const int k = k0 + (lane & (G - 1));
      const int j = woken[min(k, n - 1)];
      queue_contact<F64>(P, st, L, rx_of, have && k < n && meets(j), j, w, r, Q, queued);
    }
  }
  finish_contacts<F64>(P, st, L, rx_of, Q, queued);
}

// ---- per-particle passes: recruitment candidates, detachments, conversions ----
// Each decides for one particle from its flags, its keyed draw u, and (only
// when u is below the pass's threshold, pass_thr) its position and the grid
// counts.  One sweep before the first of these passes (k_pass_draws) draws,
// for every particle, the passes whose match holds its state; the few
// particles with some draw below its threshold go to a list, and the passes
// visit only that list.  A pass that changes a listed particle's state
// (detachment, conversion, recruitment) draws at once the later passes that
// match the new state.  A particle left off the list for a pass would be
// rejected by it, so skipping it changes nothing.
enum GroupPass : int8_t { kGroupRecruit = 0, kGroupDetach = 1, kGroupConvert = 2 };
struct DrawPlan {
  Match any;                           // states that some pass matches
  uint32_t reach[2][EDM_MAX_SPECIES];  // passes matching (alive, species), from the sweep on
  uint32_t after[kMaxPP];              // passes after pass k matching the state pass k leaves
  int8_t kind[kMaxPP];                 // GroupPass of each per-particle pass
  int8_t index[kMaxPP];                // its exchange or conversion
  int n;
};

__device__ __forceinline__ int pass_stream(int kind, int idx) {
  return kind == kGroupRecruit ? EDM_S_EX_ACCEPT + 4 * idx
                               : (kind == kGroupDetach ? EDM_S_EX_DETACH + 4 * idx : EDM_S_CONV + idx);
}

// Bits of the passes in `todo` whose keyed draw for local id `id` lies below
// the pass's threshold (the others reject the particle).
__device__ __forceinline__ uint32_t draw_passes(const DevState& st, const DrawPlan* __restrict__ D, uint64_t seed,
                                                int r, int id, int64_t step, uint32_t todo) {
  uint32_t bits = 0;
  for (; todo; todo &= todo - 1) {
    const int k = __ffs(todo) - 1;
    const uint64_t m = draw_u53(seed, step, pass_stream(D->kind[k], D->index[k]), (uint64_t)id, 0);
    if (m < st.pass_thr[(int64_t)r * kMaxPP + k]) bits |= 1u << k;
  }
  return bits;
}

// The draw sweep's work for one slot of replica r: its passes' draws, and its
// list entry when one lies below its threshold.
__device__ __forceinline__ void draw_slot(const EdmDynParams& p, const DevState& st, const DrawPlan* __restrict__ D,
                                          int r, int64_t s) {
  const uint8_t f = st.flags[s];
  const int sp = fl_species(f);
  const uint32_t todo = sp < EDM_MAX_SPECIES ? D->reach[fl_alive(f) ? 1 : 0][sp] : 0u;
  const int id = slot_id(st, s) - (int)p.particle_offset;
  const uint32_t bits = draw_passes(st, D, p.seed, r, id, *st.d_step, todo);
  if (bits) {
    const int q = st.rep_pl ? (int)p.particle_offset + atomicAdd(&st.pl_count[r], 1) : atomicAdd(st.pl_count, 1);
    st.pl[q] = make_int4((int)s, (int)bits, r, id);
    st.pl_index[s] = q;
  }
}

// Contact search of the step.  What bounds it is the chain of round trips to
// L2 (sweeper, bucket bounds, neighbours, their post-move positions) and the
// instructions per neighbour, not bytes: groups of G lanes take one sweeper
// each and its neighbour slots G at a time, so a group's chain is a few rounds
// long whatever the runs' lengths, and the pairs beyond the pre-move test are
// finished 32 at a time.  A lane per sweeper and column, walking slot by
// slot, chained three dependent loads per neighbour with 12 of 32 lanes
// active: 25 us per step for a 5,000-slot system and 56 us for 464,000 slots
// (float64), against 14 and 26 us here; for 4.7M slots 63 us, against 54 us
// with the pairs' draws taken too.  64 registers without spills at 4 blocks per
// SM beat 5, 6 and 8 blocks with spills (42.6 / 48.3 / 50 / 60 us at 1.86M
// slots).  G follows the neighbours per sweeper, nine cells' occupancy (4
// lanes at one particle per cell, 54 against 61 us with 8; 8 to 16 at four):
// the autotuner chooses it.
//
// k_contacts: a block takes a tile of BLK * SPT slots of one replica and
// gathers its sweepers in shared memory.  One launch and one block's chain:
// the form for systems that do not fill the chip.  With a draw plan D as many
// blocks again take the tiles' draws (the draw sweep, k_pass_draws, beside the
// search without a stream of its own); with WOKEN blocks beyond those, woken_parts
// per replica, take the woken particles.  A form of its own: with the branch and
// its call in the only one, 24 replicas without binding took 40.8 us a step, 40.65
// without.
template <bool F64, int BLK, int SPT, int G, int MINB, bool WOKEN>
__global__ void __launch_bounds__(BLK, MINB) k_contacts(const EdmDynParams* __restrict__ P,
                                                      const int2* __restrict__ blk, int ntiles,
                                                      const __grid_constant__ DevState st, Match m,
                                                      const __grid_constant__ CatLists L,
                                                      const DrawPlan* __restrict__ D, Match any, int woken_parts) {
  __shared__ int32_t list[BLK * SPT];
  __shared__ ContactQueue queue[BLK / 32];
  __shared__ uint32_t rx_of[EDM_MAX_SPECIES * EDM_MAX_SPECIES / 4];
  __shared__ int n_list;
  if (const int woken = (int)blockIdx.x - (D ? 2 * ntiles : ntiles); WOKEN && woken >= 0) {
    if (threadIdx.x < EDM_MAX_SPECIES * EDM_MAX_SPECIES / 4) rx_of[threadIdx.x] = L.rx_of[threadIdx.x];
    pdl_enter();
    __syncthreads();
    woken_contacts<F64, G>(P, st, L, (const uint8_t*)rx_of, woken / woken_parts, woken % woken_parts, woken_parts,
                           queue[threadIdx.x >> 5]);
    return;
  }
  const bool draws = (int)blockIdx.x >= ntiles;
  const int2 b = blk[draws ? (int)blockIdx.x - ntiles : (int)blockIdx.x];
  const int64_t end = P[b.x].particle_offset + P[b.x].n_particles;
  prefetch_params(P[b.x]);
  pdl_enter();
  if (threadIdx.x == 0) n_list = 0;
  if (threadIdx.x < EDM_MAX_SPECIES * EDM_MAX_SPECIES / 4) rx_of[threadIdx.x] = L.rx_of[threadIdx.x];
  __syncthreads();
  gather_matching<BLK, SPT>(st, draws ? any : m, (int64_t)(uint32_t)b.y, end, list, n_list);
  __syncthreads();
  if (draws) {
    for (int t = threadIdx.x; t < n_list; t += BLK) draw_slot(P[b.x], st, D, b.x, list[t]);
    return;
  }
  const int sweepers = n_list, lane = threadIdx.x & 31;
  ContactQueue& Q = queue[threadIdx.x >> 5];
  int queued = 0;
  for (int t0 = (threadIdx.x >> 5) * (32 / G); t0 < sweepers; t0 += BLK / G) {  // whole warps
    const int t = t0 + lane / G;
    contact_sweep<F64, G>(P, st, L, (const uint8_t*)rx_of, b.x, list[t < sweepers ? t : t0], t < sweepers, Q, queued);
  }
  finish_contacts<F64>(P, st, L, (const uint8_t*)rx_of, Q, queued);
}

// The sweepers of the step as one global list of (slot, replica), tile by
// tile, for k_contacts_list.
constexpr int kSweepSlots = 16;  // per thread
__global__ void __launch_bounds__(kBlock) k_sweep_list(const EdmDynParams* __restrict__ P,
                                                       const int2* __restrict__ blk, DevState st, Match m) {
  __shared__ int32_t list[kBlock * kSweepSlots];
  __shared__ int n_list, at;
  const int2 b = blk[blockIdx.x];
  const int64_t end = P[b.x].particle_offset + P[b.x].n_particles;
  if (threadIdx.x == 0) n_list = 0;
  pdl_enter();
  __syncthreads();
  gather_matching<kBlock, kSweepSlots>(st, m, (int64_t)(uint32_t)b.y, end, list, n_list);
  __syncthreads();
  const int n = n_list;
  if (n == 0) return;
  if (threadIdx.x == 0) at = atomicAdd(st.sw_count, n);
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += kBlock) st.sw_list[at + k] = make_int2(list[k], b.x);
}

// The same sweep over the global list, one wave of sweep_blocks blocks (those
// beyond take the woken particles): no per-tile
// prologue and every group has a sweeper until the list ends, which pays when
// the sweepers outnumber the chip's groups several times.
template <bool F64, int G, int MINB, bool WOKEN>
__global__ void __launch_bounds__(kBlock, MINB) k_contacts_list(const EdmDynParams* __restrict__ P,
                                                              const __grid_constant__ DevState st,
                                                              const __grid_constant__ CatLists L, int sweep_blocks,
                                                              int woken_parts) {
  __shared__ ContactQueue queue[kBlock / 32];
  __shared__ uint32_t rx_of[EDM_MAX_SPECIES * EDM_MAX_SPECIES / 4];
  if (threadIdx.x < EDM_MAX_SPECIES * EDM_MAX_SPECIES / 4) rx_of[threadIdx.x] = L.rx_of[threadIdx.x];
  pdl_enter();
  __syncthreads();
  if (WOKEN && (int)blockIdx.x >= sweep_blocks) {
    const int woken = (int)blockIdx.x - sweep_blocks;
    woken_contacts<F64, G>(P, st, L, (const uint8_t*)rx_of, woken / woken_parts, woken % woken_parts, woken_parts,
                           queue[threadIdx.x >> 5]);
    return;
  }
  const int n = *st.sw_count, lane = threadIdx.x & 31;
  const int stride = sweep_blocks * (kBlock / G);
  ContactQueue& Q = queue[threadIdx.x >> 5];
  int queued = 0;
  int t0 = (int)(blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5)) * (32 / G);
  if (t0 >= n) return;
  int2 e = st.sw_list[min(t0 + lane / G, n - 1)];
  while (t0 < n) {  // whole warps; the next sweeper is read while this one is swept
    const bool have = t0 + lane / G < n;
    const int2 cur = e;
    t0 += stride;
    if (t0 < n) e = st.sw_list[min(t0 + lane / G, n - 1)];
    contact_sweep<F64, G>(P, st, L, (const uint8_t*)rx_of, cur.y, cur.x, have, Q, queued);
  }
  finish_contacts<F64>(P, st, L, (const uint8_t*)rx_of, Q, queued);
}

// Late pairs of particle j, which a catalytic pass has just turned into the
// substrate of the later reactions `late`: its alive neighbours of those
// reactions' enzyme species passing the tests an enzyme-side sweep makes
// (j seen from enzyme e at the opposite cell offset, the same float32
// expressions), appended to the reactions' lists.
template <bool F64>
__device__ __forceinline__ void late_contacts(const EdmDynParams& p, const Geo& g, const DevState& st, int r,
                                           int64_t j, int id_j, int64_t step, uint32_t late,
                                           const ContactOut& out) {
  uint32_t emask = 0;
  for (uint32_t b = late; b; b &= b - 1) emask |= 1u << p.cat[__ffs(b) - 1].enzyme;
  for_neighbour_slots(g, st, st.cell_pre[j], [&](int e, int, int dcx, int dcy) {
    if (e == j) return;
    const uint8_t fe = st.flags[e];
    const int spe = fl_species(fe);
    if (!fl_alive(fe) || !((emask >> spe) & 1u)) return;
    double d2;
    if constexpr (F64) {
      if (!(sep_sq<F64>(st.pos_pre, st.cell_pre, e, j, g) < g.cutoff_sq())) return;
      d2 = sep_sq<F64>(st.pos_post, st.cell_post, e, j, g);
    } else {
      const float2 oe = ((const float2*)st.pos_pre)[e], oj = ((const float2*)st.pos_pre)[j];
      const float fdx = __fmaf_rn(-(float)(-dcx), g.sxf, oe.x - oj.x);
      const float fdy = __fmaf_rn(-(float)(-dcy), g.syf, oe.y - oj.y);
      if (!((double)__fmaf_rn(fdx, fdx, fdy * fdy) < g.cutoff_sq())) return;
      d2 = sep_sq<F64>(st.pos_post, st.cell_post, e, j, g);
    }
    for (uint32_t b = late; b; b &= b - 1) {
      const int c = __ffs(b) - 1;
      if (spe != p.cat[c].enzyme || d2 > p.cat[c].contact_sq) continue;
      if (!cat_draw_passes(p, st, r, c, slot_id(st, e) - (int)g.poff, id_j, step)) continue;
      out.file(c, e, (int)j);
    }
  });
}

// And those of its neighbours among the particles woken in the step, which the
// cells do not hold.
template <bool F64>
__device__ __forceinline__ void late_woken_contacts(const EdmDynParams& p, const Geo& g, const DevState& st, int r,
                                                 int64_t j, int id_j, int64_t step, uint32_t late,
                                                 const ContactOut& out) {
  uint32_t enzymes = 0, woken = 0;
  for (uint32_t b = late; b; b &= b - 1) enzymes |= 1u << p.cat[__ffs(b) - 1].enzyme;
  for (int b = 0; b < p.n_bind; ++b) woken |= enzymes & (1u << p.bind[b].rb);
  if (!woken) return;
  const int n = min(st.moved_count[r], (int)p.n_particles);
  for (int k = 0; k < n; ++k) {
    const int e = st.moved[p.particle_offset + k];
    const uint8_t fe = st.flags[e];
    const int spe = fl_species(fe);
    if (e == j || !fl_alive(fe) || !((woken >> spe) & 1u)) continue;
    if (!(sep_sq<F64>(st.pos_pre, st.cell_pre, e, j, g) < g.cutoff_sq())) continue;
    const double d2 = sep_sq<F64>(st.pos_post, st.cell_post, e, j, g);
    for (uint32_t b = late; b; b &= b - 1) {
      const int c = __ffs(b) - 1;
      if (spe != p.cat[c].enzyme || d2 > p.cat[c].contact_sq) continue;
      if (!cat_draw_passes(p, st, r, c, slot_id(st, e) - (int)g.poff, id_j, step)) continue;
      out.file(c, e, (int)j);
    }
  }
}

// Catalytic pass c (dynamics.py:825-983) over its contact list: the set of
// substrates with at least one accepted (enzyme, substrate) pair converts.
// Every listed pair is alive, has the pass's enzyme, is within its contact
// radius and has its draw below the pass's threshold; the partner's current
// species and the exact probability are left to test.
// `late`: the later reactions whose substrate is this pass's product.
template <bool F64, bool WOKEN, typename Sink>
__device__ __forceinline__ void catalytic_pair(const EdmDynParams& p, const DevState& st, int r, int cidx,
                                               uint32_t late, int2 es, const Sink& sink, const ContactOut& out) {
  const uint8_t fs = st.flags[es.y];
  const EdmCat& C = p.cat[cidx];
  if (!fl_alive(fs) || fl_species(fs) != C.substrate) return;
  const Geo g(p);
  const int ide = slot_id(st, es.x) - g.poff, ids = slot_id(st, es.y) - g.poff;
  const uint32_t lo = ide < ids ? ide : ids, hi = ide < ids ? ids : ide;
  const uint64_t m = draw_u53(p.seed, *st.d_step, EDM_S_CAT + cidx, lo, hi);
  if (m >= st.cat_thr[(int64_t)r * EDM_MAX_CAT + cidx]) return;
  const double u = __dmul_rn(__ull2double_rn(m), 0x1p-53);
  double xs, ys;
  abs_pos<F64>(st.pos_post, st.lo_post, st.cell_post, es.y, g, xs, ys);
  double peff = C.prob;
  if (C.rule >= 0) peff = C.prob * rule_factor(p, C.rule, st, xs, ys);
  if (C.rule >= 0 && ((p.adapt_cat_mask >> cidx) & 1)) peff = peff * adapt_factor(p, st.adapt_w, C.rule, xs, ys);
  if (u < peff && cas_u8(&st.flags[es.y], fs, fl_make(C.product, true))) {
    atomic_add_i64(&st.counters[(int64_t)r * EDM_NCOUNTERS + EDM_C_CATALYTIC], 1);
    grid_change(p, sink, C.substrate, true, C.product, true, xs, ys);
    if (late) {
      late_contacts<F64>(p, g, st, r, es.y, ids, *st.d_step, late, out);
      if constexpr (WOKEN) late_woken_contacts<F64>(p, g, st, r, es.y, ids, *st.d_step, late, out);
    }
  }
}

// One pass over one list for all replicas, for systems whose lists are long.
template <bool F64, bool WOKEN>
__global__ void __launch_bounds__(kBlock, 4) k_catalytic(const EdmDynParams* __restrict__ P, DevState st, int cidx,
                                                       uint32_t late) {
  pdl_enter();
  const int n = st.contact_count[cidx];
  const int lim = (int64_t)n < st.contact_cap ? n : (int)st.contact_cap;
  const int2* list = st.contacts + (int64_t)cidx * st.contact_cap;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < lim; q += (int64_t)gridDim.x * blockDim.x) {
    const int2 es = list[q];
    int r = st.chunk_rep[es.x / kSweepChunk];
    while (r + 1 < st.n_rep && st.rep_first[r + 1] <= es.x) ++r;
    catalytic_pair<F64, WOKEN>(P[r], st, r, cidx, late, es, DeltaArray{st.grid_delta}, contact_out(st, P[r], r));
  }
}

__global__ void __launch_bounds__(kBlock, 8) k_pass_draws(const EdmDynParams* __restrict__ P, DevState st,
                                                       const DrawPlan* __restrict__ D, Match any) {
  pdl_enter();
  sweep4(st, any, [&](int r, int64_t s) { draw_slot(P[r], st, D, r, s); });
}

// Puts particle `id` of replica r (in `slot`), recruited by exchange e, at (x, y).  It is
// alive from here on, so the passes after this one that match it (`after`) get
// their draws now, in its list entry (entry(q) = entry q of the list; it
// exists: the particle was listed for this exchange's candidates).
template <bool F64, typename Sink, typename Entry>
__device__ __forceinline__ void place_recruit(const EdmDynParams& p, const Geo& g, const DevState& st, int r, int e,
                                              int id, int64_t slot, double x, double y, const Sink& sink,
                                              const DrawPlan* __restrict__ D, uint32_t after, Entry entry) {
  const EdmExch& X = p.exch[e];
  const int cxn = cell_index(x, g.sx, g.nx), cyn = cell_index(y, g.sy, g.ny);
  const int newc = cxn * g.ny + cyn;
  if constexpr (F64) {
    ((double2*)st.pos_post)[slot] = make_double2(x, y);
  } else {
    float2 o;
    short2 l;
    split_offset(x - (double)cxn * g.sx, g.sxf, o.x, l.x);
    split_offset(y - (double)cyn * g.sy, g.syf, o.y, l.y);
    ((float2*)st.pos_post)[slot] = o;
    st.lo_post[slot] = l;
  }
  st.cell_post[slot] = newc;
  rebucket(st, g, g.grave, newc);
  st.flags[slot] = fl_make(X.species, true);
  note_moved(st, r, p, slot);
  grid_add(p, sink, X.species, x, y, 1);
  if (after) {
    const uint32_t bits = draw_passes(st, D, p.seed, r, id, *st.d_step, after);
    int4* q = entry(st.pl_index[slot]);
    if (q && q->x == (int)slot) q->y |= (int)bits;
    else set_status(st.status, EDM_STATUS_RECRUIT_CAP);  // cannot happen: see above
  }
}

// Apply the first max_recruits accepted candidates in particle order.
template <bool F64>
__global__ void k_recruit_apply(const EdmDynParams* __restrict__ P, int n_rep, DevState st, int e,
                                const DrawPlan* __restrict__ D,
                                uint32_t after) {
  pdl_enter();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n_rep) return;
  const EdmDynParams& p = P[r];
  const EdmExch& X = p.exch[e];
  int n = st.rec_count[r];
  if (n > kRecCap) n = kRecCap;
  st.rec_count[r] = 0;
  if (n == 0) return;
  int32_t* ids = st.rec_id + (int64_t)r * kRecCap;
  int32_t* slots = st.rec_slot + (int64_t)r * kRecCap;
  double* xy = st.rec_xy + (int64_t)r * kRecCap * 2;
  for (int a = 1; a < n; ++a) {  // insertion sort by particle index
    const int id = ids[a], slot = slots[a];
    const double x = xy[2 * a], y = xy[2 * a + 1];
    int b = a - 1;
    while (b >= 0 && ids[b] > id) {
      ids[b + 1] = ids[b];
      slots[b + 1] = slots[b];
      xy[2 * (b + 1)] = xy[2 * b];
      xy[2 * (b + 1) + 1] = xy[2 * b + 1];
      --b;
    }
    ids[b + 1] = id;
    slots[b + 1] = slot;
    xy[2 * (b + 1)] = x;
    xy[2 * (b + 1) + 1] = y;
  }
  const Geo g(p);
  const int take = n < X.max_recruits ? n : X.max_recruits;
  for (int a = 0; a < take; ++a)
    place_recruit<F64>(p, g, st, r, e, ids[a], slots[a], xy[2 * a], xy[2 * a + 1], DeltaArray{st.grid_delta}, D, after,
                       [&](int q) { return q >= 0 && q < *st.pl_count ? st.pl + q : (int4*)nullptr; });
  atomic_add_i64(&st.counters[(int64_t)r * EDM_NCOUNTERS + EDM_C_RECRUITED], take);
}

// Candidates of one replica's recruitment: [kRecCap] ids, slots and positions.
struct RecruitList {
  int32_t* count;
  int32_t* id;
  int32_t* slot;
  double* xy;
};

// Recruitment candidate of exchange e (dynamics.py:1229-1458): a dormant
// particle of the species whose keyed draw accepts at the keyed position.
// The per-particle passes below run on listed particles only.
__device__ __forceinline__ void recruit_candidate(const EdmDynParams& p, const DevState& st, const RecruitList& out,
                                                  int id, int64_t slot, int e) {
  const EdmExch& X = p.exch[e];
  const int64_t step = *st.d_step;
  const double ua = uniform1(p.seed, step, EDM_S_EX_ACCEPT + 4 * e, (uint64_t)id, 0);
  double cx, cy;
  if (X.local_recruit) {  // density-biased position (dynamics.py:1115-1217)
    const EdmGrid& G = p.grid[p.rule[X.rule_on].grid];
    const double rl = uniform1(p.seed, step, EDM_S_EX_LOC + 4 * e, (uint64_t)id, 0);
    const U2 off = normal2(p.seed, step, EDM_S_EX_OFFSET + e, (uint64_t)id);
    const double* cdf = st.local_cdf + G.offset;
    int lo = 0, hi = G.nx * G.ny - 1;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (cdf[mid] < rl) lo = mid + 1;
      else hi = mid;
    }
    const int gx = lo / G.ny, gy = lo - gx * G.ny;
    cx = py_fmod(__dadd_rn(__dmul_rn(__dadd_rn((double)gx, 0.5), G.sx), __dmul_rn(off.u0, p.recruit_sigma)), p.Lx);
    cy = py_fmod(__dadd_rn(__dmul_rn(__dadd_rn((double)gy, 0.5), G.sy), __dmul_rn(off.u1, p.recruit_sigma)), p.Ly);
  } else {
    const U2 up = uniform2(p.seed, step, EDM_S_EX_POS + 4 * e, (uint64_t)id, 0);
    cx = up.u0 * p.Lx;
    cy = up.u1 * p.Ly;
  }
  double peff = X.prob_on;
  if (X.rule_on >= 0 && X.rule_on2 >= 0) {
    peff = X.prob_on * rule_factor(p, X.rule_on, st, cx, cy) * rule_factor(p, X.rule_on2, st, cx, cy);
  } else if (X.rule_on >= 0) {
    peff = X.prob_on * rule_factor(p, X.rule_on, st, cx, cy);
  }
  if (ua < peff) {
    const int k = atomicAdd(out.count, 1);
    if (k < kRecCap) {
      out.id[k] = id;
      out.slot[k] = (int32_t)slot;
      out.xy[2 * k] = cx;
      out.xy[2 * k + 1] = cy;
    } else {
      set_status(st.status, EDM_STATUS_RECRUIT_CAP);
    }
  }
}

// Position of slot s after the move, fetched once for the passes that need it.
template <bool F64>
struct LazyPos {
  bool have = false;
  double x = 0.0, y = 0.0;
  __device__ __forceinline__ void get(const DevState& st, int64_t s, const Geo& g) {
    if (!have) abs_pos<F64>(st.pos_post, st.lo_post, st.cell_post, s, g, x, y);
    have = true;
  }
};

// Detachment of exchange e (dynamics.py:1461-1555) of the alive particle in
// slot s; returns its flags afterwards.
template <bool F64, typename Sink>
__device__ __forceinline__ uint8_t detach_one(const EdmDynParams& p, const Geo& g, const DevState& st, int r,
                                              int64_t s, int id, LazyPos<F64>& pos, int e, uint8_t f,
                                              const Sink& sink) {
  const EdmExch& X = p.exch[e];
  const double u = uniform1(p.seed, *st.d_step, EDM_S_EX_DETACH + 4 * e, (uint64_t)id, 0);
  pos.get(st, s, g);
  double peff = X.prob_off;
  if (X.rule_off >= 0) peff = X.prob_off * rule_factor(p, X.rule_off, st, pos.x, pos.y);
  if (u < peff) {
    f = fl_make(X.species, false);
    st.flags[s] = f;
    rebucket(st, g, st.cell_post[s], g.grave);
    atomic_add_i64(&st.counters[(int64_t)r * EDM_NCOUNTERS + EDM_C_DETACHED], 1);
    grid_add(p, sink, X.species, pos.x, pos.y, -1);
  }
  return f;
}

// Unimolecular conversion v (dynamics.py:1565-1657) of the alive particle in
// slot s; returns its flags afterwards.
template <bool F64, typename Sink>
__device__ __forceinline__ uint8_t convert_one(const EdmDynParams& p, const Geo& g, const DevState& st, int r,
                                               int64_t s, int id, LazyPos<F64>& pos, int v, uint8_t f,
                                               const Sink& sink) {
  const EdmConv& V = p.conv[v];
  const double u = uniform1(p.seed, *st.d_step, EDM_S_CONV + v, (uint64_t)id, 0);
  pos.get(st, s, g);
  double peff = V.prob;
  if (V.rule >= 0) peff = V.prob * rule_factor(p, V.rule, st, pos.x, pos.y);
  if (u < peff) {
    f = fl_make(V.to, true);
    st.flags[s] = f;
    atomic_add_i64(&st.counters[(int64_t)r * EDM_NCOUNTERS + EDM_C_CONVERTED], 1);
    grid_change(p, sink, V.from, true, V.to, true, pos.x, pos.y);
  }
  return f;
}

// A run of consecutive per-particle passes over the listed particles.  Each
// of these passes decides for a particle from its own flags, position and
// keyed draws and from the grid counts, which no pass of the run changes
// (their grid changes go to the delta grid), and a particle's flags change
// only in its own passes.  So taking every listed particle through the run's
// passes in order gives the result of the passes one after another.
constexpr int kMaxGroup = 16;
struct PassGroup {
  Match m[kMaxGroup];      // particles each pass visits
  int8_t kind[kMaxGroup];  // GroupPass
  int8_t index[kMaxGroup]; // exchange or conversion index
  int8_t pp[kMaxGroup];    // the pass's bit in the list entries
  uint32_t bits;           // union of the passes' bits
  int n;
};

// Takes the particle of list entry e through the run's passes; returns the
// entry's pass bits afterwards (a state change adds those of later passes).
template <bool F64, typename Sink>
__device__ __forceinline__ uint32_t run_passes(const EdmDynParams& p, const DevState& st, const PassGroup& sg,
                                               const DrawPlan* __restrict__ D, int4 e, const RecruitList& rec,
                                               const Sink& sink) {
  uint32_t bits = (uint32_t)e.y;
  if (!(bits & sg.bits)) return bits;
  const int64_t s = e.x;
  const int r = e.z, id = e.w;
  const Geo g(p);
  uint8_t f = st.flags[s];
  LazyPos<F64> pos;  // these passes move no particle
  for (int k = 0; k < sg.n; ++k) {
    const int pk = sg.pp[k];
    if (!((bits >> pk) & 1u) || !matches(f, sg.m[k])) continue;
    const int kind = sg.kind[k], idx = sg.index[k];
    if (kind == kGroupRecruit) {
      recruit_candidate(p, st, rec, id, s, idx);
      continue;
    }
    const uint8_t f0 = f;
    f = kind == kGroupDetach ? detach_one<F64>(p, g, st, r, s, id, pos, idx, f, sink)
                             : convert_one<F64>(p, g, st, r, s, id, pos, idx, f, sink);
    if (f != f0) bits |= draw_passes(st, D, p.seed, r, id, *st.d_step, D->after[pk] & ~bits);
  }
  return bits;
}

template <bool F64>
__global__ void __launch_bounds__(kBlock) k_particle_passes(const EdmDynParams* __restrict__ P, DevState st,
                                                            const PassGroup* __restrict__ G,
                                                            const DrawPlan* __restrict__ D) {
  pdl_enter();
  const int n = *st.pl_count;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    const int4 e = st.pl[q];
    const int64_t at = (int64_t)e.z * kRecCap;
    const RecruitList rec{st.rec_count + e.z, st.rec_id + at, st.rec_slot + at, st.rec_xy + 2 * at};
    const uint32_t bits = run_passes<F64>(P[e.z], st, *G, D, e, rec, DeltaArray{st.grid_delta});
    if (bits != (uint32_t)e.y) st.pl[q].y = (int)bits;
  }
}

// Whether the complex of local id `id` of reaction b dissociates in this step
// (dynamics.py:609-654).
__device__ __forceinline__ bool dissociates(const EdmDynParams& p, const DevState& st, int b, int id) {
  return uniform1(p.seed, *st.d_step, EDM_S_DISSOC + 2 * b, (uint64_t)id, 0) < p.bind[b].prob_dissoc;
}

// Lists the candidate of particles id and idj (unlike, of the reaction's two
// species, id's the one swept from; in contact before and after the move) when
// idj is unbound and the pair's draw says so; offset(): the cell offset from id's
// slot to idj's.
template <typename Offset>
__device__ __forceinline__ void list_candidate(const EdmDynParams& p, const Geo& g, const DevState& st, int r, int b,
                                               int id, int idj, bool swept_ra, Offset offset) {
  if (st.bond[g.poff + idj] >= 0) return;
  const int lo = id < idj ? id : idj, hi = id < idj ? idj : id;
  const double u = uniform1(p.seed, *st.d_step, EDM_S_BIND + 2 * b, (uint64_t)lo, (uint64_t)hi);
  if (!(u < p.bind[b].prob_bind)) return;
  int2 d = offset();
  if (lo != id) d.x = -d.x, d.y = -d.y;
  const int ordinal = (d.x + 1) * 3 + d.y + 1;
  const int k = atomicAdd(&st.bind_count[r], 1);
  if (k < kBindCap) {
    st.bind_key[(int64_t)r * kBindCap + k] =
        ((int64_t)lo << 36) | ((int64_t)ordinal << 32) | (int64_t)(0xFFFFFFFFu - (uint32_t)hi);
    st.bind_ab[((int64_t)r * kBindCap + k) * 2] = swept_ra ? id : idj;
    st.bind_ab[((int64_t)r * kBindCap + k) * 2 + 1] = swept_ra ? idj : id;
  } else {
    set_status(st.status, EDM_STATUS_BIND_CAP);
  }
}

// Binding candidates whose unswept particle an earlier reaction of the step woke
// (see woken_contacts): from the woken particle to the swept species m among its
// neighbours and among the woken.  Of a homodimer's pairs the woken one's own
// sweep has those with a higher partner in the cells.
template <bool F64, int G>
__device__ __noinline__ void woken_candidates(const EdmDynParams& p, const DevState& st, const Match& m, int r, int b,
                                              int part, int parts) {
  const Geo g(p);
  const EdmBind& B = p.bind[b];
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int32_t* woken = st.moved + p.particle_offset;
  const int n = min(st.moved_count[r], (int)p.n_particles);
  const int swept = (m.mask[1] >> B.ra) & 1u ? B.ra : B.rb, other = swept == B.ra ? B.rb : B.ra;
  for (int t0 = (part * warps + (threadIdx.x >> 5)) * (32 / G); t0 < n; t0 += parts * warps * (32 / G)) {
    const int t = t0 + lane / G;
    const int w = woken[t < n ? t : t0], idw = slot_id(st, w) - g.poff;
    const bool have = t < n && st.flags[w] == fl_make(other, true) && st.bond[g.poff + idw] < 0;
    auto meet = [&](int j) {
      if (j == w || st.flags[j] != fl_make(swept, true)) return;
      if (!(sep_sq<F64>(st.pos_pre, st.cell_pre, j, w, g) < g.cutoff_sq())) return;
      if (sep_sq<F64>(st.pos_post, st.cell_post, j, w, g) > B.contact_sq) return;
      const int idj = slot_id(st, j) - g.poff;
      if (swept == other && idj > idw) return;
      if (st.bond[g.poff + idj] >= 0) return;
      list_candidate(p, g, st, r, b, idj, idw, swept == B.ra, [&] {
        int xj, yj, xw, yw;
        split_cell(st.cell_pre[j], g, xj, yj);
        split_cell(st.cell_pre[w], g, xw, yw);
        const int dx = xw - xj, dy = yw - yj;
        return make_int2(dx > 1 ? dx - g.nx : (dx < -1 ? dx + g.nx : dx), dy > 1 ? dy - g.ny : (dy < -1 ? dy + g.ny : dy));
      });
    };
    for_neighbour_slots_grouped<G>(g, st, st.cell_pre[w], have, [&](int j, bool valid, int, int) {
      if (valid) meet(j);
    });
    for (int k = lane & (G - 1); have && k < n; k += G) meet(woken[k]);
  }
}

// Binding candidates of reaction b (dynamics.py:528-606): pairs (i < j)
// passing every test of the pass-start state, keyed by the reference's pair
// order (i, neighbour-cell ordinal seen from i, descending j).  Swept from one
// of the two species (both distance tests are symmetric in the particles), a
// tile of BLK * SPT slots per block, G lanes per sweeper, as the contact search;
// with both species swept slot by slot in a lane each the pass was 36 us for a
// 13,900-slot sensor membrane.  The tile's complexes draw for their dissociation
// on the way (st.dis).  With WOKEN blocks beyond the tiles, woken_parts per replica,
// take the woken particles (a form of its own: the sensor membrane takes 45.7 us a
// step with it where none can wake, 45.1 without).
template <bool F64, int BLK, int SPT, int G, bool WOKEN>
__global__ void __launch_bounds__(BLK) k_bind_candidates(const EdmDynParams* __restrict__ P,
                                                         const int2* __restrict__ blk, int ntiles,
                                                         const __grid_constant__ DevState st,
                                                         const __grid_constant__ Match m, int b, int woken_parts) {
  __shared__ int32_t list[BLK * SPT];
  __shared__ int n_list;
  if (WOKEN && (int)blockIdx.x >= ntiles) {
    const int woken = (int)blockIdx.x - ntiles;
    pdl_enter();
    woken_candidates<F64, G>(P[woken / woken_parts], st, m, woken / woken_parts, b, woken % woken_parts, woken_parts);
    return;
  }
  const int2 tile = blk[blockIdx.x];
  const int r = tile.x;
  const EdmDynParams& p = P[r];
  const int64_t end = p.particle_offset + p.n_particles;
  prefetch_params(p);
  if (threadIdx.x == 0) n_list = 0;
  pdl_enter();
  __syncthreads();
  gather_matching<BLK, SPT>(st, m, (int64_t)(uint32_t)tile.y, end, list, n_list);
  __syncthreads();
  const int sweepers = n_list, lane = threadIdx.x & 31;
  const uint8_t complex = fl_make(p.bind[b].product, true);
  for (int k = threadIdx.x; k < BLK * SPT; k += BLK) {
    const int64_t s = (int64_t)(uint32_t)tile.y + k;
    if (s >= end || st.flags[s] != complex) continue;
    const int id = slot_id(st, s) - (int)p.particle_offset;
    const int partner = st.bond[p.particle_offset + id];
    if (partner < 0 || !dissociates(p, st, b, id)) continue;
    const int sj = st.slot_of_id[partner], back = st.bond[partner];
    const int odd = fl_alive(st.flags[sj]) || back != p.particle_offset + id ? 1 : 0;
    const int q = atomicAdd(&st.dis_count[(b * st.n_rep + r) * 2 + odd], 1);
    st.dis[odd ? end - 1 - q : p.particle_offset + q] = make_int2((int)s, sj);
  }
  if (sweepers == 0) return;
  const EdmBind& B = p.bind[b];
  const Geo g(p);
  for (int t0 = (threadIdx.x >> 5) * (32 / G); t0 < sweepers; t0 += BLK / G) {  // whole warps
    const int t = t0 + lane / G;
    const int s = list[t < sweepers ? t : t0];
    const int other = fl_species(st.flags[s]) == B.ra ? B.rb : B.ra;
    const int id = slot_id(st, s) - g.poff;
    const bool have = t < sweepers && st.bond[g.poff + id] < 0;
    for_neighbour_slots_grouped<G>(g, st, st.cell_pre[s], have, [&](int j, bool valid, int column, int base) {
      if (!valid || j == s) return;
      const uint8_t fj = st.flags[j];
      if (!fl_alive(fj) || fl_species(fj) != other) return;
      if (!(sep_sq<F64>(st.pos_pre, st.cell_pre, s, j, g) < g.cutoff_sq())) return;
      if (sep_sq<F64>(st.pos_post, st.cell_post, s, j, g) > B.contact_sq) return;
      const int idj = slot_id(st, j) - g.poff;
      if (B.ra == B.rb && idj < id) return;  // seen from the other particle
      list_candidate(p, g, st, r, b, id, idj, other == B.rb,
                     [&] { return make_int2(column - 1, row_offset(st.cell_pre[j] - base, g)); });
    });
  }
}

// Dissociation of the complex in slot s, its partner in slot sj, of reaction b.
// Odd: the partner may be alive (and the complex itself), else it is dormant.
// The binding passes change the grid counts at once: none of them reads them.
template <bool F64, bool Odd>
__device__ __forceinline__ void dissociate_one(const EdmDynParams& p, const Geo& g, const DevState& st, int r, int b,
                                               int64_t s, int64_t sj) {
  const EdmBind& B = p.bind[b];
  const DeltaArray sink{st.grid_cnt};
  double x, y;
  abs_pos<F64>(st.pos_post, st.lo_post, st.cell_post, s, g, x, y);
  int from = g.grave;
  if constexpr (Odd) {
    const uint8_t fj = s == sj ? fl_make(B.ra, true) : st.flags[sj];
    if (fl_alive(fj)) {  // an alive partner is counted where it stands
      double xj, yj;
      abs_pos<F64>(st.pos_post, st.lo_post, st.cell_post, sj, g, xj, yj);
      grid_add(p, sink, fl_species(fj), xj, yj, -1);
      from = st.cell_post[sj];
    }
  }
  st.flags[s] = fl_make(B.ra, true);
  st.flags[sj] = fl_make(B.rb, true);
  const int newc = st.cell_post[s];
  if constexpr (F64) {
    ((double2*)st.pos_post)[sj] = ((const double2*)st.pos_post)[s];
  } else {
    ((float2*)st.pos_post)[sj] = ((const float2*)st.pos_post)[s];
    st.lo_post[sj] = st.lo_post[s];
  }
  rebucket(st, g, from, newc);
  st.cell_post[sj] = newc;
  note_moved(st, r, p, sj);
  st.bond[slot_id(st, s)] = -1;
  st.bond[slot_id(st, sj)] = -1;
  grid_change(p, sink, B.product, true, B.ra, true, x, y);
  grid_add(p, sink, B.rb, x, y, +1);
  atomic_add_i64(&st.counters[(int64_t)r * EDM_NCOUNTERS + EDM_C_DISSOC], 1);
}

// The dissociations of a replica that holds odd complexes, by one block: in
// particle order, one after the other, each by the state the earlier ones left,
// as the reference's loop (dynamics.py:609-654).  Complexes that share a partner
// both dissociate and the last one places it; one whose partner is a complex
// itself may end that one's bond.  Taken side by side, two of them would take the
// shared partner out of its bucket twice, and the next sort would write past the
// bucket.  Lists: n plain and n_odd odd entries of st.dis, and n_fresh of the
// pass's new complexes.  Rare, so no faster than one dissociation at a time.
template <bool F64>
__device__ __noinline__ void dissociate_in_order(const EdmDynParams& p, const DevState& st, int r, int b, int n,
                                                 int n_odd, int2* fresh, int n_fresh) {
  const Geo g(p);
  int2* plain = st.dis + p.particle_offset;
  int2* odd = st.dis + p.particle_offset + p.n_particles - 1;
  const int total = n + n_odd + n_fresh;
  auto at = [&](int q) -> int2& {
    return q < n ? plain[q] : (q < n + n_odd ? *(odd - (q - n)) : fresh[q - n - n_odd]);
  };
  for (int q = threadIdx.x; q < total; q += blockDim.x) at(q).x = slot_id(st, at(q).x);
  __syncthreads();
  // bitonic merges with every comparison ascending: positions past the end need no partner
  for (int64_t k = 2; k < 2 * (int64_t)total; k <<= 1)
    for (int64_t j = k - 1; j > 0; j = j == k - 1 ? k >> 2 : j >> 1) {
      for (int q = threadIdx.x; q < total; q += blockDim.x) {
        const int64_t o = q ^ j;
        if (o <= q || o >= total) continue;
        const int2 lo = at(q), hi = at((int)o);
        if (lo.x <= hi.x) continue;
        at(q) = hi;
        at((int)o) = lo;
      }
      __syncthreads();
    }
  if (threadIdx.x != 0) return;
  for (int q = 0; q < total; ++q) {
    const int id = at(q).x, s = st.slot_of_id[id], partner = st.bond[id];
    if (partner < 0 || st.flags[s] != fl_make(p.bind[b].product, true)) continue;
    dissociate_one<F64, true>(p, g, st, r, b, s, st.slot_of_id[partner]);
  }
}

// Reaction b after its candidates, 1 + `parts` blocks per replica.  The first
// applies the replica's candidates in pair order, each unless an earlier one took
// one of its particles, and dissociates the new complexes whose draw says so; the
// others dissociate the listed ones, which neither a candidate nor another entry
// touches (their particles were bound to one another, the partner dormant, at the
// pass's start).  With an odd entry (DevState::dis) the first block takes all of
// them after its candidates, in order.  What bounds it is round trips, so
// the candidates' state is fetched for all at once and their order settled in
// shared memory, where a candidate waits only for earlier ones that share a
// particle with it.  One thread per replica taking one candidate after the other,
// a sweep over all slots for the dissociations and a merge of the grid changes
// were three launches: 26 us against 10 for 13,900 slots, 167 against 19 for
// 714,000 (150 candidates a step).
constexpr int kBindThreads = 256;
template <bool F64>
__global__ void __launch_bounds__(kBindThreads, 4) k_bind_apply(const EdmDynParams* __restrict__ P,
                                                           const __grid_constant__ DevState st, int b, int parts) {
  __shared__ int64_t key[kBindCap];
  __shared__ int2 pair[kBindCap];  // in pair order
  __shared__ int8_t state[kBindCap];
  __shared__ int2 fresh[kBindCap];  // new complexes that dissociate
  __shared__ int n_fresh, n_bound;
  enum { kOpen, kTaken, kRejected };
  const int r = blockIdx.x / (1 + parts), part = blockIdx.x % (1 + parts), tid = threadIdx.x;
  const EdmDynParams& p = P[r];
  prefetch_params(p);
  pdl_enter();
  const EdmBind& B = p.bind[b];
  const Geo g(p);
  const int2 listed = ((const int2*)st.dis_count)[b * st.n_rep + r];  // plain, odd
  if (part > 0) {
    if (listed.y > 0) return;
    for (int q = (part - 1) * kBindThreads + tid; q < listed.x; q += parts * kBindThreads) {
      const int2 e = st.dis[g.poff + q];
      dissociate_one<F64, false>(p, g, st, r, b, e.x, e.y);
    }
    return;
  }
  const int n = min(st.bind_count[r], kBindCap);
  if (n == 0 && listed.y == 0) return;
  for (int i = tid; i < n; i += kBindThreads) key[i] = st.bind_key[(int64_t)r * kBindCap + i];
  if (tid == 0) n_fresh = n_bound = 0;
  __syncthreads();
  if (tid == 0) st.bind_count[r] = 0;
  for (int i = tid; i < n; i += kBindThreads) {
    const int2 ab = ((const int2*)st.bind_ab)[(int64_t)r * kBindCap + i];
    int rank = 0;
    for (int j = 0; j < n; ++j) rank += key[j] < key[i] || (key[j] == key[i] && j < i);
    pair[rank] = ab;
    const uint8_t fa = st.flags[st.slot_of_id[g.poff + ab.x]], fb = st.flags[st.slot_of_id[g.poff + ab.y]];
    const bool free = st.bond[g.poff + ab.x] < 0 && st.bond[g.poff + ab.y] < 0;
    state[rank] = free && fa == fl_make(B.ra, true) && fb == fl_make(B.rb, true) ? kOpen : kRejected;
  }
  __syncthreads();
  for (bool open = true; open;) {  // the first open candidate is settled in every round
    open = false;
    for (int i = tid; i < n; i += kBindThreads) {
      if (((volatile int8_t*)state)[i] != kOpen) continue;
      const int2 ab = pair[i];
      int8_t now = kTaken;
      for (int j = 0; j < i && now != kRejected; ++j) {
        const int2 o = pair[j];
        if (o.x != ab.x && o.x != ab.y && o.y != ab.x && o.y != ab.y) continue;
        const int8_t other = ((volatile int8_t*)state)[j];
        if (other == kTaken) now = kRejected;
        else if (other == kOpen) now = kOpen;
      }
      if (now == kOpen) open = true;
      else ((volatile int8_t*)state)[i] = now;
    }
    open = __syncthreads_or(open);
  }
  for (int i = tid; i < n; i += kBindThreads) {
    if (state[i] != kTaken) continue;
    const int a = pair[i].x, bb = pair[i].y;
    const int64_t sa = st.slot_of_id[g.poff + a], sb = st.slot_of_id[g.poff + bb];
    double xa, ya, xb, yb;
    abs_pos<F64>(st.pos_post, st.lo_post, st.cell_post, sa, g, xa, ya);
    abs_pos<F64>(st.pos_post, st.lo_post, st.cell_post, sb, g, xb, yb);
    st.flags[sa] = fl_make(B.product, true);
    st.flags[sb] = fl_make(B.rb, false);
    rebucket(st, g, st.cell_post[sb], g.grave);
    st.bond[g.poff + a] = (int32_t)(g.poff + bb);
    st.bond[g.poff + bb] = (int32_t)(g.poff + a);
    grid_change(p, DeltaArray{st.grid_cnt}, B.ra, true, B.product, true, xa, ya);
    grid_change(p, DeltaArray{st.grid_cnt}, B.rb, true, B.rb, false, xb, yb);
    atomicAdd(&n_bound, 1);
    if (dissociates(p, st, b, a)) fresh[atomicAdd(&n_fresh, 1)] = make_int2((int)sa, (int)sb);
  }
  __syncthreads();
  if (tid == 0) atomic_add_i64(&st.counters[(int64_t)r * EDM_NCOUNTERS + EDM_C_BINDINGS], n_bound);
  if (listed.y > 0) {
    dissociate_in_order<F64>(p, st, r, b, listed.x, listed.y, fresh, n_fresh);
    return;
  }
  for (int q = tid; q < n_fresh; q += kBindThreads) dissociate_one<F64, false>(p, g, st, r, b, fresh[q].x, fresh[q].y);
}

// Adaptation field update w += dt/tau_w (rho_PIP3 - w) on every cell of each
// replica's adaptation grid (dynamics.py:1093-1112, 2227-2242); block row =
// replica.
__global__ void k_adapt(const EdmDynParams* __restrict__ P, const int32_t* __restrict__ cnt,
                        double* __restrict__ w) {
  pdl_enter();
  const EdmDynParams& p = P[blockIdx.y];
  if (p.adapt_grid < 0) return;
  const EdmGrid& A = p.grid[p.adapt_grid];
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < A.nx * A.ny; c += gridDim.x * blockDim.x) {
    const int64_t i = A.offset + c;
    const double rho = kfold_density(cnt[i], p.adapt_inv_area);
    w[i] = __dadd_rn(w[i], __dmul_rn(p.adapt_inv_tau, __dadd_rn(rho, -w[i])));
  }
}

// Local-recruitment CDF of exchange e of one replica, by one block:
// cumulative max(density, 0.01) over the feedback grid's cells in (gx, gy)
// order, summed sequentially as the reference does, then divided by the total
// (dynamics.py:2356-2371).  The block computes the densities of kCdfTile cells
// in shared memory and one thread adds them; it holds the next eight cells in
// registers while it adds eight, so the chain is one dependent add per cell
// (k_react of a 42,900-slot wave system with 900 cells 23.3 to 21.9 us).
constexpr int kCdfTile = 512;
__device__ __forceinline__ void local_cdf_of(const EdmDynParams& p, const int32_t* cnt, double* cdf_all, int e,
                                             double* tile) {
  constexpr int kAhead = 8;
  const EdmExch& X = p.exch[e];
  if (!X.local_recruit || X.rule_on < 0) return;
  const EdmRule& R = p.rule[X.rule_on];
  const EdmGrid& G = p.grid[R.grid];
  const int n = G.nx * G.ny;
  double* cdf = cdf_all + G.offset;
  double total = 0.0;
  for (int c0 = 0; c0 < n; c0 += kCdfTile) {
    const int m = n - c0 < kCdfTile ? n - c0 : kCdfTile;
    __syncthreads();
    for (int c = threadIdx.x; c < kCdfTile; c += blockDim.x) {
      double v = 0.0;  // past the last cell: adding it changes no sum
      if (c < m) {
        const double rho = kfold_density(cnt[G.offset + c0 + c], R.inv_area);
        v = rho > 0.01 ? rho : 0.01;
      }
      tile[c] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double v[kAhead], next[kAhead];
#pragma unroll
      for (int k = 0; k < kAhead; ++k) next[k] = tile[k];
      for (int c = 0; c < m; c += kAhead) {
#pragma unroll
        for (int k = 0; k < kAhead; ++k) v[k] = next[k];
        const int ahead = c + kAhead < kCdfTile ? c + kAhead : c;
#pragma unroll
        for (int k = 0; k < kAhead; ++k) next[k] = tile[ahead + k];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
          total = __dadd_rn(total, v[k]);
          tile[c + k] = total;
        }
      }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < m; c += blockDim.x) cdf[c0 + c] = tile[c];
  }
  __syncthreads();
  if (threadIdx.x == 0) tile[0] = total;
  __syncthreads();
  total = tile[0];
  for (int c = threadIdx.x; c < n; c += blockDim.x)
    cdf[c] = total > 0 ? __ddiv_rn(cdf[c], total) : __ddiv_rn((double)c + 1.0, (double)n);
}

__global__ void k_local_cdf(const EdmDynParams* __restrict__ P, const int32_t* cnt, double* cdf_all, int e) {
  pdl_enter();
  __shared__ double tile[kCdfTile];
  local_cdf_of(P[blockIdx.x], cnt, cdf_all, e, tile);
}

// grid_cnt += grid_delta; grid_delta = 0
__global__ void k_grid_merge(int32_t* __restrict__ cnt, int32_t* __restrict__ delta, int64_t n) {
  pdl_enter();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int d = delta[i];
    if (d) {
      cnt[i] += d;
      delta[i] = 0;
    }
  }
}

// ---- the passes after the contact search, one block per replica ---------------
// The catalytic passes, the runs of per-particle passes, the recruitment
// applies, the local-recruitment CDFs and the grid merges between them touch
// one replica's data only, and their lists are short (only pairs and
// particles whose draw lies below the pass's threshold).  So one block takes
// its replica through all of them with a barrier between two passes instead of
// a launch: as separate launches each pass cost 2.5 to 7 us however short its
// list.  The replica's parameters, list entries, counts and grid changes sit in
// shared memory, which leaves the round trips to the particles themselves.
constexpr int kReactThreads = 512;
constexpr int kReactPasses = 48;
constexpr int kReactGroups = 8;
constexpr int kReactList = 512;  // list entries held in shared memory
enum ReactKind : int8_t { kReactCatalytic, kReactGroup, kReactRecruit, kReactCdf, kReactMerge };
struct ReactPlan {
  int8_t kind[kReactPasses];
  int8_t index[kReactPasses];    // reaction, group or exchange
  uint32_t more[kReactPasses];   // catalytic: later reactions; recruit: later passes; CDF: its candidates' pass
  int n, n_groups;
};

template <bool F64, bool WOKEN>
__global__ void __launch_bounds__(kReactThreads) k_react(const EdmDynParams* __restrict__ P, DevState st,
                                                       const __grid_constant__ ReactPlan plan,
                                                       const PassGroup* __restrict__ groups,
                                                       const DrawPlan* __restrict__ D, int64_t* step,
                                                       unsigned* ticket) {
  static_assert(sizeof(EdmDynParams) % 16 == 0 && sizeof(PassGroup) % 4 == 0, "copied in words");
  __shared__ __align__(16) uint8_t par[sizeof(EdmDynParams)];
  __shared__ __align__(16) uint8_t grp[kReactGroups * sizeof(PassGroup)];
  __shared__ int4 entry[kReactList];
  __shared__ int64_t delta_cell[kDeltaList];
  __shared__ int delta_d[kDeltaList];
  __shared__ double rec_xy[2 * kRecCap];
  __shared__ double tile[kCdfTile];
  __shared__ int32_t rec_id[kRecCap], rec_slot[kRecCap], n_contact[EDM_MAX_CAT], n_rec;
  __shared__ int n_delta;
  const int r = blockIdx.x, tid = threadIdx.x;
  for (int k = tid; k < (int)(sizeof(EdmDynParams) / 16); k += blockDim.x)
    ((uint4*)par)[k] = ((const uint4*)(P + r))[k];
  for (int k = tid; k < plan.n_groups * (int)(sizeof(PassGroup) / 4); k += blockDim.x)
    ((uint32_t*)grp)[k] = ((const uint32_t*)groups)[k];
  const int64_t poff = P[r].particle_offset;
  pdl_enter();
  if (tid < EDM_MAX_CAT) n_contact[tid] = st.rep_contacts ? st.contact_count[(int64_t)r * EDM_MAX_CAT + tid] : 0;
  if (tid == 0) n_rec = n_delta = 0;
  const int n_listed = st.pl_count[r];
  for (int q = tid; q < n_listed && q < kReactList; q += blockDim.x) entry[q] = st.pl[poff + q];
  __syncthreads();
  const EdmDynParams& p = *reinterpret_cast<const EdmDynParams*>(par);
  const DeltaList sink{delta_cell, delta_d, &n_delta, st.grid_delta};
  ContactOut out = contact_out(st, p, r);
  out.count = n_contact;
  const RecruitList rec{&n_rec, rec_id, rec_slot, rec_xy};
  auto entry_at = [&](int q) -> int4* {  // entry q of the replica's list
    return q < kReactList ? entry + q : st.pl + poff + q;
  };
  for (int i = 0; i < plan.n; ++i) {
    const int idx = plan.index[i];
    switch (plan.kind[i]) {
      case kReactCatalytic: {
        const int n = n_contact[idx] < out.cap ? n_contact[idx] : (int)out.cap;
        for (int q = tid; q < n; q += blockDim.x)
          catalytic_pair<F64, WOKEN>(p, st, r, idx, plan.more[i], out.list[(int64_t)idx * out.stride + q], sink, out);
        break;
      }
      case kReactGroup: {
        const PassGroup& sg = reinterpret_cast<const PassGroup*>(grp)[idx];
        for (int q = tid; q < n_listed; q += blockDim.x) {
          int4* e = entry_at(q);
          const int4 v = *e;
          const uint32_t bits = run_passes<F64>(p, st, sg, D, v, rec, sink);
          if (bits != (uint32_t)v.y) e->y = (int)bits;
        }
        break;
      }
      case kReactRecruit: {  // the first max_recruits candidates in particle order
        const int n = n_rec < kRecCap ? n_rec : kRecCap;
        if (n == 0) break;
        const int cap = p.exch[idx].max_recruits, take = n < cap ? n : cap;
        for (int a = tid; a < n; a += blockDim.x) {
          const int id = rec_id[a];
          int rank = 0;
          for (int b = 0; b < n; ++b) rank += rec_id[b] < id;
          if (rank < take)
            place_recruit<F64>(p, Geo(p), st, r, idx, id, rec_slot[a], rec_xy[2 * a], rec_xy[2 * a + 1], sink, D,
                               plan.more[i],
                               [&](int q) {
                                 const int k = q - (int)poff;
                                 return k >= 0 && k < n_listed ? entry_at(k) : (int4*)nullptr;
                               });
        }
        __syncthreads();
        if (tid == 0) {
          n_rec = 0;
          atomic_add_i64(&st.counters[(int64_t)r * EDM_NCOUNTERS + EDM_C_RECRUITED], take);
        }
        break;
      }
      case kReactCdf: {
        // only the candidates of the pass that follows read it, and most steps
        // of a small system have none (a 42,900-slot wave system 21.9 to 16.4 us)
        bool mine = false;
        for (int q = tid; q < n_listed; q += blockDim.x) mine |= ((uint32_t)entry_at(q)->y & plan.more[i]) != 0;
        if (__syncthreads_or(mine)) local_cdf_of(p, st.grid_cnt, st.local_cdf, idx, tile);
        break;
      }
      case kReactMerge: {
        const int n = n_delta;
        for (int k = tid; k < n && k < kDeltaList; k += blockDim.x) atomicAdd(&st.grid_cnt[delta_cell[k]], delta_d[k]);
        if (n > kDeltaList && p.n_grids > 0) {  // the changes that found the list full
          const EdmGrid& last = p.grid[p.n_grids - 1];  // a replica's grids are contiguous
          for (int64_t at = p.grid[0].offset + tid; at < last.offset + (int64_t)last.nx * last.ny; at += blockDim.x) {
            const int d = st.grid_delta[at];
            if (d) {
              atomicAdd(&st.grid_cnt[at], d);
              st.grid_delta[at] = 0;
            }
          }
        }
        __syncthreads();
        if (tid == 0) n_delta = 0;
        break;
      }
    }
    __syncthreads();
  }
  // the last block to finish moves the step index on
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(ticket, 1u) == gridDim.x - 1) {
      *ticket = 0;
      *step += 1;
    }
  }
}

__global__ void k_step_inc(int64_t* step) {
  pdl_enter();
  *step += 1;
}

}  // namespace edm
