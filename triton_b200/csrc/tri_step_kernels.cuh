// tri_step_kernels.cuh -- the fused time-step kernels of the domain path.
//
// One time step of the reference (triton_simulate.h:191-346) becomes, on the
// domain's stream:
//   k_flux_update   fluxes + conserved update + Manning friction + runoff
//                   (kernels_flux.h, kernels_state.h, kernels.h:103-152)
//   k_forcing       point inflows (kernels.h:51-84), open-boundary ghosts
//                   (kernels.h:437-512) and external boundary cells
//                   (kernels.h:237-424), only where there are any
//   k_post          wet/dry masks + max depth (kernels_wetdry.h:25-93) fused
//                   with the NEXT step's CFL dt and its min reduction
//                   (kernels.h:167-212); moves the clock on
// The flux kernel's blocks begin with the step's clock work: dt policy
// (compute_global_dt :202-226), runoff row and hydrograph bracket (:246-285),
// step events.
// Every kernel reads the step's parameters from the device clock, so a
// sequence of steps needs no host round trip and can be captured in a graph.
#pragma once

#include "tri_common.cuh"
#include "tri_bulk.cuh"
#include "tri_face.cuh"
#include "tri_step_launch.h"
#include "tri_types.cuh"

namespace tri {

template <typename T>
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------
// The per-step scalar work of the reference host loop.  begin_step only reads
// the clock: in the single-domain step one thread of every flux block runs it
// (about a microsecond before the block's first tile, against 3.3 us for a
// launch of its own), block 0 leaves the outcome in c->now for the post kernel.
// ---------------------------------------------------------------------------
__device__ __forceinline__ StepNow begin_step(const DevClock* __restrict__ c) {
  StepNow n;
  n.active = !(c->halt || c->steps >= c->limit);
  const double t0 = c->simtime;
  double dt;
  if (!c->time_increment_fixed) {
    // compute_global_dt: dry fallback, then clamp to the next print time
    const unsigned long long key0 = c->dt_key[0], key1 = c->dt_key[1];  // both, not one behind rd
    dt = dt_of_key(c->rd ? key1 : key0, c->cfl_a);
    if (dt >= kMaxValue - 1.0) dt = c->init_dt;
    const double tp = c->print_interval * (c->print_id + 1);
    if (t0 + dt > tp) dt = tp - t0;
  } else {
    dt = c->time_step;
  }
  n.dt = dt;
  n.rdt = 1.0 / dt;
  n.t_step = t0;
  n.step = c->it_count + 1;
  n.runoff_row = c->runoff_row;
  if (n.active && c->nroff > 0) {
    const int last = c->roff_rows - 1;
    if (t0 > c->roff_t[last]) {
      n.runoff_row = last;
    } else if (n.runoff_row + 1 <= last && t0 > c->roff_t[n.runoff_row + 1]) {
      n.runoff_row++;
    }
  }
  n.src_idx_low = n.src_idx_high = c->src_idx_low;
  if (n.active && c->nsrc > 0) {
    int lo = c->src_idx_low, hi = c->hyg_rows - 1;
    bool found = false;
    for (int i = lo; i < hi; i++) {
      if (c->hyg_t[i + 1] > t0) {
        lo = i;
        hi = i + 1;
        found = true;
        break;
      }
    }
    if (!found) lo = hi;
    n.src_idx_low = lo;
    n.src_idx_high = hi;
  }
  n.src = c->cur;
  n.dst = c->cur ^ 1;
  n.wr = c->rd ^ 1;
  const double t1 = t0 + dt;
  n.t_end = t1;
  int ev = 0;
  if (c->it_print > 0 && n.step % c->it_print == 0) ev |= TRI_EV_LOG;
  if (c->time_series && t1 - c->last_obs_time >= c->print_observation) ev |= TRI_EV_OBS;
  if (t1 >= c->print_interval * (c->print_id + 1)) ev |= TRI_EV_PRINT;
  if (!(t1 < c->sim_duration)) ev |= TRI_EV_END;
  n.events = ev;
  return n;
}

// The clock moves on by the step c->now (one thread).  Returns true when the
// step raised an event (the domain halts after it).
__device__ __forceinline__ bool end_step(DevClock* __restrict__ c) {
  const StepNow& n = c->now;
  c->global_dt = n.dt;
  c->it_count = n.step;
  c->runoff_row = n.runoff_row;
  c->src_idx_low = n.src_idx_low;
  c->tile_next = 0;
  c->cur = n.dst;
  c->rd = n.wr;
  c->dt_key[n.wr ^ 1] = kDtKeyInf;  // the next step's slot
  c->simtime = n.t_end;
  c->average_dt += n.dt;
  c->steps++;
  if (n.events) {
    c->halt = 1;
    c->events = n.events;
    *c->host_halt = 1;  // the host reads it behind an event recorded after this kernel
    return true;
  }
  return false;
}

// ---------------------------------------------------------------------------
// Forcing that writes into single cells of the destination buffer after their
// flux update: point sources, open-boundary ghosts, external boundary cells,
// in the reference's order.  One launch for all of it: a warp applies the items
// of one flux tile (TileForcing; no item touches another tile's cells), where
// a launch per kind and conflict-free wave took 4 to 8 us each, several a step.
// (Applied by the flux kernel's own warps, at the end of each tile, it cost
// every tile registers: bowl 2048^2 FP64 99.7 -> 102.6 us, a 24-member FP32
// ensemble step 259 -> 270 us.)
// ---------------------------------------------------------------------------
// Point source `id` (compute_flow, kernels.h:51-84).
template <typename T>
__device__ __forceinline__ void source_apply(DevClock* __restrict__ clk, const StepNow& now, const StateBufs<T>& sb,
                                             const ForcingDev<T>& f, T dx, int id) {
  const int lo = now.src_idx_low, hi = now.src_idx_high;
  const T dt = T(now.dt), simtime = T(now.t_step);
  T* h = sb.H(now.dst);
  const T flo = f.hyg_v[(size_t)lo * f.nsrc + id], fhi = f.hyg_v[(size_t)hi * f.nsrc + id];
  const T tlo = T(f.hyg_t[lo]), thi = T(f.hyg_t[hi]);
  T flow;
  if (lo == hi) {
    flow = flo;
  } else {
    const T td = simtime - tlo, td2 = thi - tlo;
    flow = flo + (((fhi - flo) * td) / td2);
  }
  const int sid = f.src_cells[id];
  T hij = h[sid];
  const T hs = (flow * dt) / (dx * dx);
  hij += hs;
  h[sid] = hij;
  atomicAdd(&clk->acc_step[kAccSources], (double)hs);
}

// Final values of copy_info_to_exterior_boundaries_west_east followed by
// _north_south (kernels.h:437-512) in state buffer d, item k of max(rows, cols): ghost columns
// take the adjacent interior column (rows 1..rows-2), ghost rows take the
// adjacent interior row, corners the diagonal interior cell.
template <typename T>
__device__ __forceinline__ void open_bc_item(int d, const StateBufs<T>& sb, int rows, int cols, int k) {
  T* h = sb.H(d);
  T* qx = sb.QX(d);
  T* qy = sb.QY(d);
  auto cp = [&](size_t g, size_t i) {
    h[g] = h[i];
    qx[g] = qx[i];
    qy[g] = qy[i];
  };
  if (k < rows) {
    const int r = k;
    if (r >= 1 && r <= rows - 2) {
      cp((size_t)r * cols, (size_t)r * cols + 1);
      cp((size_t)r * cols + cols - 1, (size_t)r * cols + cols - 2);
    }
  }
  if (k < cols) {
    const int cc = k;
    const int ci = cc == 0 ? 1 : (cc == cols - 1 ? cols - 2 : cc);
    cp((size_t)cc, (size_t)cols + ci);
    cp((size_t)(rows - 1) * cols + cc, (size_t)(rows - 2) * cols + ci);
  }
}

// The same for the ghosts next to one flux tile (rows r0..r1, columns from c0
// on), by the warp that owns it.
template <typename T>
__device__ __forceinline__ void open_bc_tile(int d, const StateBufs<T>& sb, int rows, int cols, int r0, int r1,
                                             int c0, int lane) {
  T* h = sb.H(d);
  T* qx = sb.QX(d);
  T* qy = sb.QY(d);
  auto cp = [&](size_t g, size_t i) {
    h[g] = h[i];
    qx[g] = qx[i];
    qy[g] = qy[i];
  };
  const int c1 = min(c0 + kStripCols - 1, cols - 2);
  for (int r = r0 + lane; r <= r1; r += 32) {
    if (c0 == 1) cp((size_t)r * cols, (size_t)r * cols + 1);
    if (c1 == cols - 2) cp((size_t)r * cols + cols - 1, (size_t)r * cols + cols - 2);
  }
  // ghost rows; a corner takes the diagonal interior cell
  const int ca = c0 == 1 ? 0 : c0, cz = c1 == cols - 2 ? cols - 1 : c1;
  for (int c = ca + lane; c <= cz; c += 32) {
    const int ci = min(max(c, 1), cols - 2);
    if (r0 == 1) cp((size_t)c, (size_t)cols + ci);
    if (r1 == rows - 2) cp((size_t)(rows - 1) * cols + c, (size_t)(rows - 2) * cols + ci);
  }
}

// compute_extbc_values for one boundary cell (kernels.h:254-420), single rank.
template <typename T>
__device__ __forceinline__ void extbc_apply(DevClock* __restrict__ clk, const StepNow& now, const StateBufs<T>& sb,
                                            const BedMap<T>& bed, const T* __restrict__ n2, int id,
                                            const ForcingDev<T>& f, int rows, int cols) {
  const T* __restrict__ var1 = f.bc_v1;
  const T* __restrict__ var2 = f.bc_v2;
  const int d = now.dst;
  T* h = sb.H(d);
  T* qx = sb.QX(d);
  T* qy = sb.QY(d);
  const T dt = T(now.dt);
  const T simtime = T(now.t_step);
  const int ii = f.bc_cells[id];
  const int bt = f.bc_types[id];
  const int s0 = f.bc_start[id];
  const int ix = ii / cols, iy = ii % cols;
  const bool top = (ix == 1), btm = (ix == rows - 2), lt = (iy == 1), rt = (iy == cols - 2);
  if (!(top || lt || rt || btm)) return;
  bool corner = false;
  int ib = ii, ibc = ii;
  T f0 = T(1), f1 = T(0), f2 = T(0);
  if (lt) {
    ib = ii - 1;
    f1 = T(-1);
    f2 = T(0);
  }
  if (rt) {
    ib = ii + 1;
    f1 = T(1);
    f2 = T(0);
  }
  if (top) {
    ib = ii - cols;
    f1 = T(0);
    f2 = T(1);
    if (lt) {
      corner = true;
      ibc = ii - 1;
      f2 = T(0);
    }
    if (rt) {
      corner = true;
      ibc = ii + 1;
      f2 = T(0);
    }
  }
  if (btm) {
    ib = ii + cols;
    f1 = T(0);
    f2 = T(-1);
    if (lt) {
      corner = true;
      ibc = ii - 1;
      f2 = T(0);
    }
    if (rt) {
      corner = true;
      ibc = ii + 1;
      f2 = T(0);
    }
  }
  T hij = h[ii], qxij = qx[ii], qyij = qy[ii];
  if (bt == 0) {
    h[ib] = hij;
    qx[ib] = qxij;
    qy[ib] = qyij;
    if (corner) {
      h[ibc] = hij;
      qx[ibc] = qxij;
      qy[ibc] = qyij;
    }
    return;
  }
  if (bt == 1) {
    const T lvar = T(0.5) * (simtime + simtime + dt);
    int lo = 0, hi = f.bc_nrows[id] - 1;
    if (lvar < var1[s0]) {
      lo = 0;
      hi = 0;
    } else if (lvar > var1[hi + s0]) {
      lo = hi;
    } else {
      lo = 0;  // a non-monotone table leaves the reference's index unset; clamp to row 0
      for (int i = 0; i < hi; i++) {
        if (var1[i + s0] <= lvar && var1[i + 1 + s0] > lvar) {
          lo = i;
          hi = i + 1;
          break;
        }
      }
    }
    T aux;
    if (lo == hi) {
      aux = var2[lo + s0];
    } else {
      const T td = lvar - var1[lo + s0];
      const T td2 = var1[hi + s0] - var1[lo + s0];
      aux = var2[lo + s0] + (((var2[hi + s0] - var2[lo + s0]) * td) / td2);
    }
    if (sizeof(T) == 8) {
      hij = dev_fmax(aux - (T)bed.absolute(ii, ix, iy), T(0));
    } else {  // FP32 form: level minus bed in FP64, then rounded
      hij = (T)fmax((double)aux - bed.absolute(ii, ix, iy), 0.0);
    }
    atomicAdd(&clk->acc_step[kAccExtbc], (double)hij - (double)h[ii]);
  } else {
    const T aux = var1[s0];
    T vel = T(0);
    if (bt == 2) vel = dev_sqrt(aux * hij * dev_cbrt(hij) / dev_fmax(n2[ii], T(1e-6)));
    if (bt == 3) vel = aux * dev_sqrt(T(kGravity) * hij);
    qxij = hij * vel;
    qyij = hij * vel;
  }
  h[ib] = hij * f0;
  qx[ib] = qxij * f1;
  qy[ib] = qyij * f2;
  h[ii] = hij * f0;
  qx[ii] = qxij * f1;
  qy[ii] = qyij * f2;
  if (corner) {
    h[ibc] = hij * f0;
    qx[ibc] = qxij * f1;
    qy[ibc] = qyij * f2;
  }
}

// Applies the forcing of list entry k's tile (whole warp).
template <typename T>
__device__ __forceinline__ void tile_forcing(DevClock* clk, const StepNow& now, const StateBufs<T>& sb,
                                             const BedMap<T>& bed, const T* __restrict__ n2, const ForcingDev<T>& f,
                                             const TileForcing& tf, bool open, T dx, int rows, int cols, int rb,
                                             int tile, int k, int lane) {
  int g = tf.group_of[k];
  const int gz = tf.group_of[k + 1];
  for (bool edges = open; g < gz || edges; g++) {
    const int a = g < gz ? tf.item_of[g] : 0, z = g < gz ? tf.item_of[g + 1] : 0;
    if (edges && (g >= gz || tf.items[a] < 0)) {  // after the sources, before the boundary cells
      const int ns = (cols - 2 + kStripCols - 1) / kStripCols;
      const int c0 = 1 + (tile % ns) * kStripCols, r0 = 1 + (tile / ns) * rb, r1 = min(r0 + rb - 1, rows - 2);
      open_bc_tile<T>(now.dst, sb, rows, cols, r0, r1, c0, lane);
      edges = false;
      __syncwarp();
    }
    for (int i = a + lane; i < z; i += 32) {
      const int id = tf.items[i];
      if (id >= 0)
        source_apply<T>(clk, now, sb, f, dx, id);
      else
        extbc_apply<T>(clk, now, sb, bed, n2, -1 - id, f, rows, cols);
    }
    __syncwarp();
  }
}

template <typename T>
__global__ void __launch_bounds__(128) k_forcing(DevClock* __restrict__ clk, const __grid_constant__ StateBufs<T> sb,
                                                 const __grid_constant__ BedMap<T> bed, const T* __restrict__ n2,
                                                 const __grid_constant__ ForcingDev<T> f,
                                                 const __grid_constant__ TileForcing tf, bool open, T dx, int rows,
                                                 int cols, int rb) {
  pdl_wait();
  pdl_trigger();
  const int k = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (k >= tf.count || !clk->now.active) return;
  tile_forcing<T>(clk, clk->now, sb, bed, n2, f, tf, open, dx, rows, cols, rb, tf.tiles[k], k, threadIdx.x & 31);
}

// The same for the tiles of all members of a batch (tiles over all members).
template <typename T>
__global__ void __launch_bounds__(128) k_batch_forcing(const MemberDev<T>* __restrict__ mem,
                                                       const int32_t* __restrict__ tile_member,
                                                       const __grid_constant__ TileForcing tf) {
  pdl_wait();
  pdl_trigger();
  const int k = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (k >= tf.count) return;
  const int tile = tf.tiles[k];
  const MemberDev<T>& M = mem[tile_member[tile]];
  if (!M.clk->now.active) return;
  tile_forcing<T>(M.clk, M.clk->now, M.sb, M.bed, M.n2, M.f, tf, M.open != 0, M.dx, M.rows, M.cols, M.rb,
                  tile - (int)M.tile_begin, k, threadIdx.x & 31);
}

// ---------------------------------------------------------------------------
// k_flux_update: fluxes + conserved update + friction + runoff.
//
// Work unit: a tile of one warp = a strip of 30 interior columns and rb rows.
// Lane l holds column c = c0-1+l: lanes 1..30 own interior columns, lanes 0
// and 31 are the west/east halo columns.  The warp marches down its rows
// keeping the previous row in registers, so every x face and y face of the
// strip is evaluated once (plus one halo y row per tile and one halo x face
// per row); neighbours are exchanged with shuffles, there is no block-level
// synchronisation.  Warps fetch tiles from a per-step counter (the dry part of
// a domain costs far less than the wet part, so static tiling leaves SMs idle).
//   y face (r, r-1): owner row r, north neighbour row r-1 (kernels_flux.h:359-360)
//   x face (c-1, c): owner column c-1, east neighbour c   (kernels_flux.h:76-77)
// A row's update runs once its south face (computed with the next row) is
// known: h = hn - (xE+yN) - (xW+yS), i.e. hn - rhsh0 - rhsh1 with the
// reference's rhs0 = flux_x part + flux_y part (kernels_state.h:65).
// Ghost cells are copied from the source to the destination buffer so both
// ping-pong buffers keep the boundary state the reference keeps in place.
// ---------------------------------------------------------------------------
// rhs contributions collected for one cell before its south face is known.
// The owner parts of its east and north faces are summed at once, in the
// reference's order (flux_x writes rhs*0, flux_y adds to it):
// r = e + n; the west face's neighbour part w waits for the south face's s
// (rhs*1 = w + s).  Six values carried per lane instead of nine.
template <typename T>
struct RowParts {
  T r0, r1, r2;  // east + north owner parts
  T w0, w1, w2;  // west face, neighbour part (flux_x rhs*1)
  T an;          // FP32 form: |e0| + |n0|, for the noise test of the depth update
};

// A friction quotient's dividend that div_line takes: 0 (of either sign) or at
// least 2^-200 (a transverse discharge can decay to any size), which over a
// friction term of 2^760 at most leaves a normal quotient.
__device__ __forceinline__ bool line_dividend(double a) {
  const uint32_t hi = (uint32_t)__double2hiint(a) & 0x7FFFFFFFu;
  return hi >= (1023u - 200u) << 20 || (hi | (uint32_t)__double2loint(a)) == 0u;
}

// LINE (FP64): the straight-line forms; *odd is set where they do not hold.
template <typename T, bool LINE>
__device__ __forceinline__ void update_cell(const CellQ<T>& c, const RowParts<T>& p, T s0, T s1, T s2, T n2v, T dt,
                                            T hextra, T& ho, T& qxo, T& qyo, double& clip, uint32_t rnd, bool& odd) {
  constexpr bool L64 = LINE && sizeof(T) == 8;
  const T E12 = eps12<T>();
  const T G = T(kGravity);
  const T hn = c.h;
  T hij;
  if (sizeof(T) == 8) {
    const T rh1 = p.w0 + s0;
    hij = hn - p.r0 - rh1;
    clip = hij < T(0) ? -(double)hij : 0.0;
  } else {
    // FP32 form: the depth change is summed in FP64 and rounded
    // stochastically (unbiased).  Rounded to nearest, a deep cell drops every
    // inflow below half its ulp while the thin cell it came from loses it
    // exactly, so runoff draining from films into channels would vanish
    // (1.4e-5 of the volume over 2 h of rain on a 2048^2 watershed).  A
    // result within the rounding noise of its terms is zero, as FP32
    // arithmetic would give it: noise must not leave water on a cell that
    // drained, or the cell counts as wet.
    const float parts = p.r0 + (p.w0 + s0);
    float lo;
    const float hs = sr_add(hn, -parts, rnd, &lo);
    const float noise = float(kNoise32) * (hn + p.an + dev_fabs(p.w0) + dev_fabs(s0));
    if (__fadd_rn(hn, -parts) <= noise) {
      clip = -((double)__fadd_rn(hn, -parts) + (double)lo);  // removed (noise) or clipped to zero: accounted
      hij = T(0);
    } else {
      clip = 0.0;
      hij = hs;
    }
  }
  T qxij, qyij;
  if (hij < T(0)) hij = T(0);
  if (hij < hextra) {
    qxij = T(0);
    qyij = T(0);
  } else {
    const T rx1 = p.w1 + s1;
    const T ry1 = p.w2 + s2;
    const T mx = c.qx - p.r1 - rx1;
    const T my = c.qy - p.r2 - ry1;
    T mxx, myy;
    mul2(mx, my, mx, my, &mxx, &myy);
    const T mm = mxx + myy;
    T modM;
    if constexpr (L64) {  // a square below 1e-30 is no flow either way
      odd |= ((uint32_t)__double2hiint(mm) & 0x7FFFFFFFu) > (1023u + 600u) << 20;
      const double ms = mm > 1e-30 ? mm : 1e-30;
      modM = sqrt_line(ms, rsqrt_line(ms));
    } else {
      modM = dev_sqrt(mm);
    }
    if (L64 && n2v > E12 && hn >= hextra && modM > E12) {
      // dividend of the friction term: 2^-300 .. 2^60 keeps it, its reciprocal
      // and its square root normal for every regular depth (2^-700 .. 2^234 as den)
      const double num = dt * G * n2v * modM, den = hn * hn * dev_cbrt(hn);
      odd |= (uint32_t)__double2hiint(num) - ((1023u - 300u) << 20) > (360u << 20);
      const double tt = div_line(num, den, recip_line(den));
      const double t4 = T(1) + T(4) * tt;
      const double sq = sqrt_line(t4, rsqrt_line(t4));
      const double rtt = recip_line(tt);
      const double ax = T(-0.5) * (mx - mx * sq), ay = T(-0.5) * (my - my * sq);
      qxij = div_line(ax, tt, rtt);
      qyij = div_line(ay, tt, rtt);
      if (!line_dividend(ax)) qxij = div_rare(ax, tt);
      if (!line_dividend(ay)) qyij = div_rare(ay, tt);
    } else if (!L64 && n2v > E12 && hn >= hextra && modM > E12) {
      const T tt = fdiv(dt * G * n2v * modM, hn * hn * dev_cbrt(hn));
      const T sq = dev_sqrt(T(1) + T(4) * tt);
      if (sizeof(T) == 8) {  // the reference's expression (kernels_state.h:86-96), bit for bit
        const T rtt = recip(tt);
        qxij = div_shared(T(-0.5) * (mx - mx * sq), tt, rtt);
        qyij = div_shared(T(-0.5) * (my - my * sq), tt, rtt);
      } else {
        // FP32 form: -(m - m*s)/(2t) with s = sqrt(1 + 4t) equals
        // 2m/(1 + s), without the cancellation of 1 - s: where t is small
        // (deep, fast channel flow) 1 - s keeps only a few FP32 bits, and the
        // rounding of s alone moved the friction-corrected discharge by up to
        // 1e-3 of itself each step, one way (the 512^2 6 h watershed then
        // ponded up to 0.97 m away from the FP64 run).
        const T k = recip(T(1) + sq);
        T mx2, my2;
        mul2(T(2), T(2), mx, my, &mx2, &my2);
        mul2(k, k, mx2, my2, &qxij, &qyij);
      }
    } else {
      qxij = mx;
      qyij = my;
    }
  }
  ho = hij;
  qxo = qxij;
  qyo = qyij;
}

template <typename T>
__device__ __forceinline__ T shfl_up1(T v) {
  return __shfl_up_sync(0xffffffffu, v, 1);
}
template <typename T>
__device__ __forceinline__ T shfl_down1(T v) {
  return __shfl_down_sync(0xffffffffu, v, 1);
}


// Everything one tile of the flux kernel needs: the domain's arrays and the
// running step's constants (from its clock).
template <typename T>
struct FluxCtx {
  DevClock* clk;
  const T* hi;
  const T* qxi;
  const T* qyi;
  T* ho;
  T* qxo;
  T* qyo;
  BedMap<T> bed;
  const T* n2;
  const int32_t* zone;
  const T* rates;
  int rows, cols, rb, nstrips;
  int nroff, roff_rows, roff_row;
  uint32_t step;  // it_count of the running step (seeds the FP32 form's rounding of runoff)
  StepK<T> K;
  // Dry-tile skipping (null: every tile is computed).  tz_src[t] / tz_dst[t]:
  // tile t of the source / destination buffer holds only zero bits in h, qx
  // and qy; tpin[t]: tile t is never skipped (a later kernel of the step
  // writes into it: sources, external boundary cells, open boundaries).
  const uint8_t* tz_src;
  uint8_t* tz_dst;
  const uint8_t* tpin;
};

template <typename T>
__device__ __forceinline__ FluxCtx<T> flux_ctx(DevClock* clk, const StepNow& now, const StateBufs<T>& sb,
                                               const BedMap<T>& bed, const T* n2, const int32_t* zone, const T* rates,
                                               int rows, int cols, int rb, T dx, T rdx, T hextra) {
  FluxCtx<T> X;
  X.clk = clk;
  X.hi = sb.H(now.src);
  X.qxi = sb.QX(now.src);
  X.qyi = sb.QY(now.src);
  X.ho = sb.H(now.dst);
  X.qxo = sb.QX(now.dst);
  X.qyo = sb.QY(now.dst);
  X.bed = bed;
  X.n2 = n2;
  X.zone = zone;
  X.rates = rates;
  X.rows = rows;
  X.cols = cols;
  X.rb = rb;
  X.nstrips = (cols - 2 + kStripCols - 1) / kStripCols;
  X.nroff = clk->nroff;
  X.roff_rows = clk->roff_rows;
  X.roff_row = now.runoff_row;
  X.step = (uint32_t)now.step;
  X.K = step_k<T>(dx, T(now.dt), rdx, T(now.rdt), hextra);
  X.tz_src = nullptr;
  X.tz_dst = nullptr;
  X.tpin = nullptr;
  return X;
}

// The same with the tile flags: [2][tiles] by buffer, then [tiles] pinned.
template <typename T, bool kSkip>
__device__ __forceinline__ FluxCtx<T> flux_ctx_tiles(DevClock* clk, const StepNow& now, const StateBufs<T>& sb,
                                                     const BedMap<T>& bed, const T* n2, const int32_t* zone,
                                                     const T* rates, int rows, int cols, int rb, T dx, T rdx,
                                                     T hextra, uint8_t* tflag) {
  FluxCtx<T> X = flux_ctx<T>(clk, now, sb, bed, n2, zone, rates, rows, cols, rb, dx, rdx, hextra);
  const size_t ntiles = (size_t)X.nstrips * (size_t)((rows - 2 + rb - 1) / rb);
  if (kSkip) X.tz_src = tflag + (size_t)now.src * ntiles;
  X.tz_dst = tflag + (size_t)now.dst * ntiles;
  X.tpin = tflag + 2 * ntiles;
  return X;
}

// Zero bits (+0): a tile is skipped only where every value it would write
// is +0 already, so skipping is exact.
__device__ __forceinline__ bool nonzero_bits(double v) { return __double_as_longlong(v) != 0; }
__device__ __forceinline__ bool nonzero_bits(float v) { return __float_as_uint(v) != 0u; }

// A tile whose cells and whose four neighbour tiles' cells hold only +0 in
// the source buffer computes exactly +0 everywhere (every face is dry-dry and
// contributes nothing; no runoff on such a domain), and if its cells in the
// destination buffer hold +0 already (it was all-zero two steps ago), it has
// nothing to write.  Called by lane 0, which takes the tiles.
template <typename T>
__device__ __forceinline__ bool tile_skippable(const FluxCtx<T>& X, unsigned tile) {
  if (X.tz_src == nullptr) return false;
  const int ns = X.nstrips, nty = (X.rows - 2 + X.rb - 1) / X.rb;
  const int sx = (int)(tile % ns), ry = (int)(tile / ns);
  if (!(X.tz_src[tile] & X.tz_dst[tile]) || X.tpin[tile]) return false;
  if (sx > 0 && !(X.tz_src[tile - 1])) return false;
  if (sx < ns - 1 && !(X.tz_src[tile + 1])) return false;
  if (ry > 0 && !(X.tz_src[tile - ns])) return false;
  if (ry < nty - 1 && !(X.tz_src[tile + ns])) return false;
  return true;
}

// The same pointer, opaque to the compiler: values read through it cannot be
// taken from an earlier read through the original.
template <typename P>
__device__ __forceinline__ const P* launder_ptr(const P* p) {
  const P* q;
  asm volatile("mov.b64 %0, %1;" : "=l"(q) : "l"(p));
  return q;
}

// A piece of work of one warp: rows r0..r1 of strip sx, tile 'tile' or part of it.
struct FluxUnit {
  unsigned tile;
  int sx, r0, r1;
};
__device__ __forceinline__ FluxUnit whole_tile(unsigned tile, int rows, int nstrips, int rb) {
  FluxUnit u;
  u.tile = tile;
  u.sx = (int)(tile % (unsigned)nstrips);
  u.r0 = 1 + (int)(tile / (unsigned)nstrips) * rb;
  u.r1 = min(u.r0 + rb - 1, rows - 2);
  return u;
}

// The last tiles of a launch, as many as it has warps (`split`), are taken in
// parts of 4 or (tiles above 8 rows) 8 rows, so that the warps end together: unit
// n of tiles - split + split * parts.  Rain on 1531x2049, FP64: step 181 -> 175
// us (8 rows, parts of 4); a 24-member FP32 ensemble 239 -> 232 us (16 rows,
// parts of 8; 235 with parts of 4, which repeat more rows of faces).
__device__ __forceinline__ int part_rows(int rb) { return rb > 8 ? 8 : 4; }
__device__ __forceinline__ unsigned tile_parts(int rb) { return (unsigned)((rb + part_rows(rb) - 1) / part_rows(rb)); }
// Tile of unit n; *part: which part of it (-1: all).
__device__ __forceinline__ unsigned unit_tile(unsigned n, unsigned ntiles, unsigned split, int rb, int* part) {
  const unsigned whole = ntiles - split, parts = tile_parts(rb);
  if (n < whole) {
    *part = -1;
    return n;
  }
  const unsigned v = n - whole;
  *part = (int)(v % parts);
  return whole + v / parts;
}
__device__ __forceinline__ void take_part(FluxUnit* u, int part, int rb) {
  if (part < 0) return;
  u->r0 += part * part_rows(rb);
  u->r1 = min(u->r1, u->r0 + part_rows(rb) - 1);
}

// Whether any lane's column h (row stride `cols`) holds a 0 in rows r .. z.
template <typename T>
__device__ __noinline__ bool column_dry(const T* h, int cols, int r, int z) {
  bool dry = false;
  for (; r <= z; ++r) dry |= h[(size_t)r * cols] == T(0);
  return __any_sync(0xffffffffu, dry);
}

// One warp tile: strip sx (30 interior columns), rows r0..r1.  kTrack:
// record in X.tz_dst whether the tile wrote only +0 (dry-tile skipping; the
// kernels of domains that cannot skip are built without it).  kReload: the
// context (in shared memory) is read again every row, where each value is
// used, instead of being held in registers across the row loop; the batched
// kernels' member parameters are not kernel parameters, and holding them
// spilled (FP32 batched ensemble at 8 blocks per SM: 252 bytes of spill
// stores, 20 with the reads; 25.5 against 23.8 G cell-updates/s at the best
// launch shape).  The single-domain kernel keeps kReload off: its context
// comes from kernel parameters, which the compiler reads at each use.
//
// kLine (FP64): the tile is computed with the straight-line forms, which hold
// for regular cells; where a lane meets another kind of cell, the whole tile
// returns false without having added to the accounts or its dry flag, and
// the caller computes it again with the guarded forms (the tile only reads
// the source buffer, so it can be repeated).
template <typename T, bool kTrack, bool kReload, bool kLine>
__device__ __forceinline__ bool flux_tile_form(const FluxCtx<T>& X0, FluxUnit u, int lane) {
  bool odd = false;  // this lane met a cell that is not regular
  const FluxCtx<T>& X = kReload ? *launder_ptr(&X0) : X0;
  const int rows = X.rows, cols = X.cols;
  const T hextra = X.K.hextra;
  const int c = u.sx * kStripCols + lane;  // = c0 - 1 + lane with c0 = 1 + 30*sx
  const int r0 = u.r0, r1 = u.r1;
  const bool incol = c < cols;
  const bool mid = (lane >= 1 && lane <= kStripCols);
  const bool upd = mid && c >= 1 && c <= cols - 2;
  const bool gcol = incol && (c == 0 || c == cols - 1);  // ghost column owned by this lane
  const bool owner = incol && (mid || gcol);
  double acc_b = 0.0, acc_r = 0.0, acc_c = 0.0;  // FP64 volume accounts in both forms
  const double sxq = (double)X.K.dt / (double)X.K.dx;  // dt/dx of the boundary discharges

  bool wrote_nonzero = false;  // any value this lane writes is not +0
  auto copy_ghost = [&](const FluxCtx<T>& Z, int r) {
    const T* __restrict__ hi = Z.hi;
    const T* __restrict__ qxi = Z.qxi;
    const T* __restrict__ qyi = Z.qyi;
    T* __restrict__ ho = Z.ho;
    T* __restrict__ qxo = Z.qxo;
    T* __restrict__ qyo = Z.qyo;
    const size_t id = (size_t)r * Z.cols + c;
    if (kTrack) {
      const T gh = hi[id];
      ho[id] = gh;
      const T gqx = qxi[id];
      qxo[id] = gqx;
      const T gqy = qyi[id];
      qyo[id] = gqy;
      wrote_nonzero |= nonzero_bits(gh) | nonzero_bits(gqx) | nonzero_bits(gqy);
    } else {
      ho[id] = hi[id];
      qxo[id] = qxi[id];
      qyo[id] = qyi[id];
    }
  };

  // with a threshold of zero or less a dry cell has velocities, 0/0 (looked for
  // here: a test in the row loop costs every other domain up to 1 %)
  if (kLine && !(hextra > T(0)) && column_dry<T>(X.hi + c, cols, r0 - 1, incol ? r1 + 1 : r0 - 2)) return false;

  // raw values of the next row are loaded one iteration ahead
  T lh = T(0), lqx = T(0), lqy = T(0), lz = T(0);
  auto fetch = [&](const FluxCtx<T>& Z, int r) {
    if (incol) {
      const size_t id = (size_t)r * Z.cols + c;
      lh = Z.hi[id];
      lqx = Z.qxi[id];
      lqy = Z.qyi[id];
      lz = Z.bed.z[id];  // FP32 form: the offset from the base of the cell's tile
    }
  };
  fetch(X, r0 - 1);
  if (kLine) odd = !regular_cell(lh, lqx, lqy);
  CellQ<T> prev = make_cell<T, kLine>(lh, lqx, lqy, lz, X.K);
  if (r0 - 1 == 0 && owner) copy_ghost(X, 0);
  fetch(X, r0);
  // FP32 form: base level of the bed tile of this lane's column minus that of
  // the column to the west, for the tile row of row r (0 within a tile)
  double dzx = 0.0;
  const bool crossx = sizeof(T) == 4 && incol && lane >= 1 && (c & 31) == 0;
  auto base_step = [&](const FluxCtx<T>& Z, int r) {
    if (crossx) dzx = Z.bed.base_at(r, c) - Z.bed.base_at(r, c - 1);
  };
  base_step(X, r0);
  RowParts<T> pp;
  pp.r0 = pp.r1 = pp.r2 = pp.w0 = pp.w1 = pp.w2 = pp.an = T(0);
  T pn2 = T(0);  // Manning of the previous row's cell

  for (int r = r0; r <= r1 + 1; ++r) {
    // the context is read where it is used, so with kReload none of it is
    // held across the face computations
    const FluxCtx<T>& XL = kReload ? *launder_ptr(&X0) : X0;
    if (kLine) odd |= !regular_cell(lh, lqx, lqy);
    const CellQ<T> cur = make_cell<T, kLine>(lh, lqx, lqy, lz, XL.K);
    T cn2 = T(0);
    if (r <= r1) {
      if (upd) cn2 = XL.n2[(size_t)r * XL.cols + c];
      fetch(XL, r + 1);  // r1 + 1 <= rows - 1
    }
    // (no row below the last cell of the grid's last tile: r1 + 1 <= rows - 1)
    bool crossy = false;  // FP32 form: a bed tile row begins here
    double dzy = 0.0;
    if (sizeof(T) == 4 && (r & 31) == 0) {
      crossy = true;
      if (incol) dzy = XL.bed.base_at(r - 1, c) - XL.bed.base_at(r, c);
      base_step(XL, r);
    }
    // every lane forms its faces (those that no cell takes are not used):
    // a branch around them would end the block the compiler schedules in
    const FaceOut<T> Y = face_flux<T, false, kLine>(cur, prev, XL.K, crossy, dzy);
    if (r - 1 >= r0 && upd) {
      const FluxCtx<T>& XU = kReload ? *launder_ptr(&X0) : X0;
      const int cols = XU.cols;
      const T dt = XU.K.dt, hextra = XU.K.hextra;
      const size_t id = (size_t)(r - 1) * cols + c;
      T hn, qn, vn;
      double clip;
      update_cell<T, kLine>(prev, pp, Y.b0, Y.b1, Y.b2, pn2, dt, hextra, hn, qn, vn, clip,
                            cell_hash((uint32_t)id, 2u * XU.step), odd);
      // Inflow through the south face of a cell of the last interior row
      // (the other boundary faces are counted where their parts are
      // formed, below), and the depth the update clipped back to zero.
      if (r - 1 == XU.rows - 2) acc_b += sxq * (double)prev.qy - (double)Y.b0;
      acc_c += clip;
      if (XU.nroff > 0) {  // update_runoff (kernels.h:128-149)
        const T h0 = hn;
        // with one zone its rate, without the zone map
        const T net = XU.rates[(size_t)(XU.nroff > 1 ? XU.zone[id] : 0) * XU.roff_rows + XU.roff_row];
        if (sizeof(T) == 8) {
          hn += net * dt;
        } else if (net != T(0)) {
          // FP32 form: uniform rain adds the same increment to every cell of
          // a zone, so rounding h + r*dt to nearest would round the same way
          // in every cell of a binade; the FP64 sum is rounded
          // stochastically instead (unbiased), deterministic in (cell, step)
          float lo;
          hn = sr_add(hn, net * dt, cell_hash((uint32_t)id, 2u * XU.step + 1u), &lo);
        }
        if (hn < hextra) {
          if (hn < T(0)) hn = T(0);
          qn = T(0);
          vn = T(0);
        }
        acc_r += (double)hn - (double)h0;
      }
      T* __restrict__ ho = XU.ho;
      T* __restrict__ qxo = XU.qxo;
      T* __restrict__ qyo = XU.qyo;
      ho[id] = hn;
      qxo[id] = qn;
      qyo[id] = vn;
      if (kTrack) wrote_nonzero |= nonzero_bits(hn) | nonzero_bits(qn) | nonzero_bits(vn);
    }
    if (r > r1) {
      if (r == XL.rows - 1 && owner) copy_ghost(XL, r);
      break;
    }
    // x faces of row r: lane l evaluates the face between lanes l-1 and l
    CellQ<T> left;
    left.h = shfl_up1(cur.h);
    left.qx = shfl_up1(cur.qx);
    left.qy = shfl_up1(cur.qy);
    left.z = shfl_up1(cur.z);
    left.sq = shfl_up1(cur.sq);
    left.u = shfl_up1(cur.u);
    left.v = shfl_up1(cur.v);
    left.hd = shfl_up1(cur.hd);
    const FaceOut<T> Xf = face_flux<T, true, kLine>(left, cur, XL.K, crossx, dzx);
    const T e0 = shfl_down1(Xf.a0), e1 = shfl_down1(Xf.a1), e2 = shfl_down1(Xf.a2);
    if (upd) {
      // Inflow through faces shared with ghost cells, in depth units.  The
      // update is in fluctuation form, so the mass flux through a face of
      // boundary cell i is F(Q_i).n plus the fluctuation it receives there:
      // west / south faces dt/dx*q - b, east / north faces -(a + dt/dx*q).
      if (c == 1) acc_b += sxq * (double)cur.qx - (double)Xf.b0;
      if (c == XL.cols - 2) acc_b -= (double)e0 + sxq * (double)cur.qx;
      if (r == 1) acc_b -= (double)Y.a0 + sxq * (double)cur.qy;
    }
    pp.r0 = e0 + Y.a0;
    pp.r1 = e1 + Y.a1;
    pp.r2 = e2 + Y.a2;
    pp.w0 = Xf.b0;
    pp.w1 = Xf.b1;
    pp.w2 = Xf.b2;
    if (sizeof(T) == 4) pp.an = dev_fabs(e0) + dev_fabs(Y.a0);
    pn2 = cn2;
    if (gcol) copy_ghost(XL, r);
    prev = cur;
  }
  if (kLine && __any_sync(0xffffffffu, odd)) return false;
  acc_b = warp_sum<T>(acc_b);
  acc_r = warp_sum<T>(acc_r);
  acc_c = warp_sum<T>(acc_c);
  if (lane == 0) {
    if (acc_b != 0.0) atomicAdd(&X.clk->acc_step[kAccBoundary], acc_b);
    if (acc_r != 0.0) atomicAdd(&X.clk->acc_step[kAccRunoff], acc_r);
    if (acc_c != 0.0) atomicAdd(&X.clk->acc_step[kAccClip], acc_c);
  }
  if (kTrack) {
    const bool nz = __any_sync(0xffffffffu, wrote_nonzero);
    if (lane == 0) X.tz_dst[u.tile] = (!nz && !X.tpin[u.tile]) ? 1 : 0;
  }
  return true;
}

// The guarded forms, out of line: a tile with extreme values is rare.  The
// single-domain kernel's context is formed again from the kernel parameters
// (a context that the call took by reference would live in local memory).
template <typename T>
__device__ __noinline__ void flux_tile_guarded_ctx(const FluxCtx<T>* X, FluxUnit u, int lane) {
  flux_tile_form<T, false, true, false>(*X, u, lane);
}
template <typename T, bool kSkip>
__device__ __noinline__ void flux_tile_guarded(DevClock* clk, const StepNow* now, const StateBufs<T>* sb,
                                               const BedMap<T>* bed, const T* n2, const int32_t* zone, const T* rates,
                                               int rows, int cols, int rb, T dx, T rdx, T hextra, uint8_t* tflag,
                                               FluxUnit u, int lane) {
  flux_tile_form<T, kSkip, false, false>(
      flux_ctx_tiles<T, kSkip>(clk, *now, *sb, *bed, n2, zone, rates, rows, cols, rb, dx, rdx, hextra, tflag), u,
      lane);
}

// A unit of a batch member, its context in shared memory.
template <typename T>
__device__ __forceinline__ void flux_tile_member(const FluxCtx<T>& X, FluxUnit u, int lane) {
  if (!flux_tile_form<T, false, true, sizeof(T) == 8>(X, u, lane)) flux_tile_guarded_ctx<T>(&X, u, lane);
}

// kSkip: the domain can have dry tiles (no runoff) and skips them.
template <typename T, int MINB, bool kSkip>
__global__ void __launch_bounds__(128, MINB)
    k_flux_update(DevClock* __restrict__ clk, const __grid_constant__ StateBufs<T> sb,
                  const __grid_constant__ BedMap<T> bed, const T* __restrict__ n2, const int32_t* __restrict__ zone,
                  const T* __restrict__ rates, int rows, int cols, int rb, T dx, T rdx, T hextra,
                  uint8_t* __restrict__ tflag) {
  __shared__ StepNow s_now;
  pdl_wait();
  if (threadIdx.x == 0) {
    s_now = begin_step(clk);
    if (blockIdx.x == 0) clk->now = s_now;
  }
  __syncthreads();
  if (!s_now.active) return;
  const FluxCtx<T> X = flux_ctx_tiles<T, kSkip>(clk, s_now, sb, bed, n2, zone, rates, rows, cols, rb, dx, rdx, hextra,
                                                tflag);
  const int lane = threadIdx.x & 31;
  const unsigned ntiles = (unsigned)X.nstrips * (unsigned)((rows - 2 + rb - 1) / rb);
  // a dry-tile flag has one writer: where dry tiles are skipped, tiles stay whole
  const unsigned split = kSkip ? 0u : min(ntiles, gridDim.x * 4u);
  const unsigned nunits = ntiles - split + split * tile_parts(rb);
  unsigned skipped = 0;  // interior cells of the tiles this warp skipped (lane 0)
  while (true) {
    unsigned n = 0;  // lane 0 takes the next unit; bit 31: skip it (tiles < 2^31)
    if (lane == 0) {
      n = atomicAdd(&clk->tile_next, 1u);
      if (kSkip && n < ntiles && tile_skippable<T>(X, n)) {
        const FluxUnit u = whole_tile(n, rows, X.nstrips, rb);
        skipped += (unsigned)((u.r1 - u.r0 + 1) * min(kStripCols, cols - 2 - u.sx * kStripCols));
        n |= 0x80000000u;
      }
    }
    n = __shfl_sync(0xffffffffu, n, 0);
    if ((n & 0x7FFFFFFFu) >= nunits) break;
    if (kSkip && (n >> 31)) continue;
    int part = -1;
    const unsigned tile = kSkip ? n : unit_tile(n, ntiles, split, rb, &part);
    FluxUnit u = whole_tile(tile, rows, X.nstrips, rb);
    take_part(&u, part, rb);
    if (u.r0 > u.r1) continue;  // the grid's last tile row can be short
    if (!flux_tile_form<T, kSkip, false, sizeof(T) == 8>(X, u, lane))
      flux_tile_guarded<T, kSkip>(clk, &s_now, &sb, &bed, n2, zone, rates, rows, cols, rb, dx, rdx, hextra, tflag, u,
                                  lane);
  }
  pdl_trigger();  // no tile left for this warp
  if (kSkip && lane == 0 && skipped)  // spread over the slots: one address would serialize the atomics
    atomicAdd(&clk->skipped[0][(blockIdx.x * 4 + (threadIdx.x >> 5)) % kSkipSlots], (unsigned long long)skipped);
}

// Kahan fold of the step's volume terms into the domain's totals.
__device__ __forceinline__ void fold_accounts(DevClock* __restrict__ clk) {
  for (int k = 0; k < kAccTerms; k++) {
    const double y = clk->acc_step[k] - clk->acc_comp[k];
    const double t = clk->acc_sum[k] + y;
    clk->acc_comp[k] = (t - clk->acc_sum[k]) - y;
    clk->acc_sum[k] = t;
    clk->acc_step[k] = 0.0;
  }
}

// Wave speed of a wet cell (compute_dt_and_sqrt, kernels.h:167-187).  FP64:
// the reference's denominator, bit for bit, straight-line where the cell's
// values are in the range of those forms.  FP32 form: in FP32 (its maximum and
// the dt are FP64).
__device__ __forceinline__ double wave_speed(double h, double qx, double qy) {
  const double q = fmax(fabs(qx), fabs(qy));
  if (regular_cell(h, q, q)) {
    const double y = rsqrt_line(h);
    return div_line(q, h, recip_line(h, y * y)) + kSqrtG * sqrt_line(h, y);
  }
  return q / h + kSqrtG * fmax(sqrt(h), 0.0);
}
__device__ __forceinline__ float wave_speed(float h, float qx, float qy) {
  const float maxu = fdiv(dev_fmax(dev_fabs(qx), dev_fabs(qy)), h);
  return maxu + float(kSqrtG) * dev_fmax(dev_sqrt(h), 0.0f);
}

// ---------------------------------------------------------------------------
// Staged wet-dry/dt, the wet-dry item of the single-launch batch mode: one block per band of WetStage<T>::kBand rows x
// kWetCols columns.  The block stages, in shared memory, its rows of h and
// the bed with a halo row above and below, and its rows of qx, qy and the
// maximum depth, each row from column c0-1 to c0+kWetCols (clipped to the
// grid) with one bulk asynchronous copy (cp.async.bulk: rounded out to
// 16-byte boundaries, which every field's kFieldPad allows at its end).  All
// copies are issued at once, in groups of kStageGroupRows output rows, each
// group completing on its own mbarrier: a thread walking its column down the band
// starts on the first two rows while the later rows are still in flight, so
// a block's loads overlap its own arithmetic even when every block of a wave
// starts at the same moment.  The FP32 form turns a staged bed offset into a
// level relative to the block's reference as it reads it (its tile's delta,
// added in registers), so no pass over shared memory and no block barrier
// sits between the copies and the arithmetic.
// ---------------------------------------------------------------------------
template <typename T>
struct WetStage {
  static constexpr int kBand = kStageBand<T>;                        // rows per block
  static constexpr int kVec = 16 / (int)sizeof(T);                   // elements per 16 bytes
  static constexpr int kCap = kWetCols + 2 + 2 * (kVec - 1);         // elements per row buffer
  static constexpr int kHRows = kBand + 2;                           // h and bed rows (with halos)
  static constexpr int kRows = 2 * kHRows + 3 * kBand;               // + qx, qy, max depth rows
  static constexpr size_t kData = (size_t)kRows * kCap * sizeof(T);
  // copy groups of kGR output rows: group 0 = h and bed staged rows
  // 0..kGR+1 and band rows 0..kGR-1 of qx, qy, max depth; group g > 0 = h and
  // bed staged rows g*kGR+2..g*kGR+kGR+1 and band rows g*kGR..g*kGR+kGR-1
  static constexpr int kGR = kStageGroupRows<T>;
  static constexpr int kGroups = kBand / kGR;
  static constexpr int kFirst = 2 * (kGR + 2) + 3 * kGR, kNext = 5 * kGR;
  static constexpr size_t kBarBytes = (8 * kGroups + 15) / 16 * 16;
  // FP32 form: the staged rows span at most 2 x 6 bed tiles of 32 x 32
  // (kBand + 2 <= 32 rows, kWetCols + 2 <= 5 * 32 + 2 columns)
  static constexpr int kTileCols = 6, kTileSlots = 2 * kTileCols;
  static constexpr size_t kBytes = kData + kBarBytes + 4 * kHRows + 4 * kTileSlots;  // + row offsets, tiles
};
static_assert(kStageBand<double> % kStageGroupRows<double> == 0 && kStageBand<float> % kStageGroupRows<float> == 0,
              "bands are whole copy groups");
static_assert(WetStage<double>::kFirst + (WetStage<double>::kGroups - 1) * WetStage<double>::kNext ==
                  WetStage<double>::kRows, "copy groups cover the staged rows");
static_assert(WetStage<float>::kFirst + (WetStage<float>::kGroups - 1) * WetStage<float>::kNext ==
                  WetStage<float>::kRows, "copy groups cover the staged rows");
static_assert(WetStage<float>::kBand + 2 <= 32, "staged rows span at most two bed tile rows");

// Gives up on a block whose copies did not land: reports it, waits (bounded)
// once more on every group from 'from' on so no copy still writes this
// block's shared memory when it exits.
template <int kGroups>
__device__ __forceinline__ void stage_abandon(DevClock* clk, uint64_t* bar, int from) {
  atomicExch(&clk->status, kStatusStageTimeout);
  for (int g = from; g < kGroups; ++g) mbar_wait(&bar[g], 0);
}

// Test hook (one thread of one block): a bounded wait on a barrier whose
// phase can never complete (its arrival count is met, but it expects 16 bytes
// that no copy delivers, and no copy is ever issued on it).  The wait gives up
// after clk->wait_test polls and records a device status as a stage timeout
// does, so the host's handling of a wait that gave up can be tested without
// disturbing any real copy.
static __device__ __noinline__ void wait_test(DevClock* clk) {
  __shared__ __align__(8) uint64_t bar;
  mbar_init(&bar, 1);
  mbar_arrive_expect_tx(&bar, 16);
  if (!mbar_wait(&bar, 0, clk->wait_test)) atomicExch(&clk->status, kStatusTestWait);
}

template <typename T>
__device__ __forceinline__ unsigned long long wetdry_staged(DevClock* __restrict__ clk, const StateBufs<T>& sb,
                                                            const BedMap<T>& bed, T* __restrict__ maxh, int rows,
                                                            int cols, T hextra, float* __restrict__ arrival,
                                                            float arrival_depth, int bx, int by, T* stage) {
  using S = WetStage<T>;
  constexpr bool kF32 = sizeof(T) == 4;
  const int buf = clk->now.dst;
  T* __restrict__ qx = sb.QX(buf);
  T* __restrict__ qy = sb.QY(buf);
  const T E12 = eps12<T>();
  const int tid = threadIdx.x, lane = tid & 31;
  const int c0 = bx * kWetCols;
  const int ra = by * S::kBand;
  const int rz = min(ra + S::kBand - 1, rows - 1);
  const int cl = max(c0 - 1, 0), ce = min(c0 + kWetCols + 1, cols);  // staged columns [cl, ce)
  unsigned char* tail = reinterpret_cast<unsigned char*>(stage) + S::kData;
  uint64_t* bar = reinterpret_cast<uint64_t*>(tail);
  // offs[j]: column c of staged row ra-1+j sits at buffer index c + offs[j]
  int* offs = reinterpret_cast<int*>(tail + S::kBarBytes);
  // FP32 form: per bed tile the staged rows touch, its base minus the
  // block's reference level
  float* tdel = reinterpret_cast<float*>(offs + S::kHRows);
  const int rlo = max(ra - 1, 0), rhi = min(rz + 1, rows - 1);
  const int tr0 = rlo >> 5, tc0 = cl >> 5;
  if (tid < S::kGroups) mbar_init(&bar[tid], 1);
  if (tid < S::kHRows) {
    const int64_t r = (int64_t)(ra - 1 + tid);
    offs[tid] = (int)(r * cols - ((r * cols + cl) & ~(int64_t)(S::kVec - 1)));
  }
  if (kF32 && tid >= 32 && tid < 32 + S::kTileSlots) {
    const int s = tid - 32, tr = tr0 + s / S::kTileCols, tc = tc0 + s % S::kTileCols;
    if (tr <= (rhi >> 5) && tc <= ((ce - 1) >> 5))
      tdel[s] = (float)(bed.base_at(tr << 5, tc << 5) - bed.ref_of(ra, min(c0, cols - 1)));
  }
  __syncthreads();
  if (tid < 32) {
    for (int i = lane; i < S::kRows; i += 32) {
      // copy i -> group g, field f (0 h, 1 bed, 2 qx, 3 qy, 4 max depth) and
      // q: staged row (h, bed; global row ra-1+q) or band row (global ra+q)
      int g, f, q;
      if (i < S::kFirst) {
        g = 0;
        if (i < 2 * (S::kGR + 2)) {
          f = i / (S::kGR + 2);
          q = i % (S::kGR + 2);
        } else {
          f = 2 + (i - 2 * (S::kGR + 2)) / S::kGR;
          q = (i - 2 * (S::kGR + 2)) % S::kGR;
        }
      } else {
        const int t = (i - S::kFirst) % S::kNext;
        g = 1 + (i - S::kFirst) / S::kNext;
        if (t < 2 * S::kGR) {
          f = t / S::kGR;
          q = g * S::kGR + 2 + t % S::kGR;
        } else {
          f = 2 + (t - 2 * S::kGR) / S::kGR;
          q = g * S::kGR + (t - 2 * S::kGR) % S::kGR;
        }
      }
      int r, slot;
      const T* src;
      if (f < 2) {
        r = ra - 1 + q;
        if (r < 0 || r > rows - 1) continue;
        slot = f * S::kHRows + q;
        src = f == 0 ? (const T*)sb.H(buf) : (const T*)bed.z;
      } else {
        r = ra + q;
        if (r > rz) continue;
        slot = 2 * S::kHRows + (f - 2) * S::kBand + q;
        src = f == 2 ? (const T*)qx : (f == 3 ? (const T*)qy : (const T*)maxh);
      }
      const int64_t e0 = ((int64_t)r * cols + cl) & ~(int64_t)(S::kVec - 1);
      const int64_t e1 = ((int64_t)r * cols + ce + S::kVec - 1) & ~(int64_t)(S::kVec - 1);
      const uint32_t bytes = (uint32_t)((e1 - e0) * (int64_t)sizeof(T));
      mbar_expect_tx(&bar[g], bytes);
      bulk_g2s(stage + (size_t)slot * S::kCap, src + e0, bytes, &bar[g]);
    }
    __syncwarp();
    if (lane == 0)
      for (int g = 0; g < S::kGroups; ++g) mbar_arrive(&bar[g]);
  }
  const T* sh = stage;
  const T* sz = stage + (size_t)S::kHRows * S::kCap;
  const T* sqx = stage + (size_t)2 * S::kHRows * S::kCap;
  const T* sqy = sqx + (size_t)S::kBand * S::kCap;
  const T* smh = sqy + (size_t)S::kBand * S::kCap;
  const int c = c0 + tid;
  const bool incol = c < cols;
  const bool intcol = c >= 1 && c <= cols - 2;
  // FP32 form: tile deltas of columns c-1, c, c+1 in tile rows 0 and 1
  // (where a delta is zero the level is the offset itself, up to the sign of a
  // zero, which no comparison below sees)
  T dw0 = T(0), dw1 = T(0), dc0 = T(0), dc1 = T(0), de0 = T(0), de1 = T(0);
  if (kF32 && intcol) {
    const int tw = ((c - 1) >> 5) - tc0, tc = (c >> 5) - tc0, te = ((c + 1) >> 5) - tc0;
    dw0 = (T)tdel[tw];
    dc0 = (T)tdel[tc];
    de0 = (T)tdel[te];
    if ((rhi >> 5) > tr0) {
      dw1 = (T)tdel[S::kTileCols + tw];
      dc1 = (T)tdel[S::kTileCols + tc];
      de1 = (T)tdel[S::kTileCols + te];
    }
  }
  const float simtime_now = (float)clk->now.t_end;
  // largest wave speed of the thread's cells (NaN speeds left out, as
  // speed_key does); one key at the end equals the minimum of per-cell keys
  T dmax = T(-1);
  if (incol) {
    // bed level of the thread's column at staged row j (buffer offset oj)
    auto zlev = [&](int j, int oj) -> T {
      T v = sz[j * S::kCap + c + oj];
      if (kF32) v += (((ra - 1 + j) >> 5) > tr0) ? dc1 : dc0;
      return v;
    };
    int om = offs[0], o = offs[1];
    T zm = T(0), z0 = T(0);
#pragma unroll
    for (int jq = 0; jq < S::kBand; ++jq) {
      const int r = ra + jq;
      if (r > rz) break;
      if (jq % S::kGR == 0 && !mbar_wait(&bar[jq / S::kGR], 0)) {
        stage_abandon<S::kGroups>(clk, bar, jq / S::kGR);
        return kDtKeyInf;
      }
      const int j = jq + 1;
      const int op = offs[j + 1];
      if (jq == 0) {
        zm = zlev(0, om);
        z0 = zlev(1, o);
      }
      const T zp = zlev(j + 1, op);
      const size_t id = (size_t)r * cols + c;
      const T* hrow = sh + j * S::kCap + o;
      const T hij = hrow[c];
      T qxv = sqx[jq * S::kCap + c + o], qyv = sqy[jq * S::kCap + c + o];
      if (intcol && r >= 1 && r <= rows - 2) {
        if (hij > hextra) {
          const T he = hrow[c + 1], hw = hrow[c - 1];
          const T hm = sh[(j - 1) * S::kCap + c + om];
          const T hp = sh[(j + 1) * S::kCap + c + op];
          const T* zrow = sz + j * S::kCap + o;
          T ze = zrow[c + 1], zw = zrow[c - 1];
          if (kF32) {
            const bool t1 = (r >> 5) > tr0;
            ze += t1 ? de1 : de0;
            zw += t1 ? dw1 : dw0;
          }
          if ((hij + z0 < ze && he < E12) || (hij + z0 < zw && hw < E12)) {
            qxv = T(0);
            qx[id] = T(0);
          }
          if ((hij + z0 < zm && hm < E12) || (hij + z0 < zp && hp < E12)) {
            qyv = T(0);
            qy[id] = T(0);
          }
        }
        if (hij > smh[jq * S::kCap + c + o]) maxh[id] = hij;
        if (arrival != nullptr && hij > arrival_depth && !(arrival[id] < 3.0e38f)) arrival[id] = simtime_now;
      }
      if (hij > hextra) dmax = dev_fmax(dmax, wave_speed(hij, qxv, qyv));
      zm = z0;
      z0 = zp;
      om = o;
      o = op;
    }
  }
  return dmax >= T(0) ? speed_key((double)dmax) : kDtKeyInf;
}

// Block minimum of the threads' keys, folded into *slot with one atomic.
__device__ __forceinline__ void block_min_into(unsigned long long key, unsigned long long* slot) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
    key = other < key ? other : key;
  }
  __shared__ unsigned long long s_min[kWetCols / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) s_min[warp] = key;
  __syncthreads();
  if (threadIdx.x == 0) {
    key = s_min[0];
    for (int w = 1; w < kWetCols / 32; w++) key = s_min[w] < key ? s_min[w] : key;
    // most blocks cannot lower the slot: read it first, then one atomic
    if (key < kDtKeyInf && key < *reinterpret_cast<volatile unsigned long long*>(slot)) atomicMin(slot, key);
  }
}

// The CFL dt of the current state, ghosts included (compute_dt_and_sqrt runs
// over rows*cols), into the slot the next step reads.
template <typename T>
__global__ void __launch_bounds__(kWetCols) k_initial_dt(DevClock* __restrict__ clk, StateBufs<T> sb, int64_t n,
                                                         T hextra) {
  const T* __restrict__ h = sb.H(clk->cur);
  const T* __restrict__ qx = sb.QX(clk->cur);
  const T* __restrict__ qy = sb.QY(clk->cur);
  T dmax = T(-1);
  for (int64_t i = (int64_t)blockIdx.x * kWetCols + threadIdx.x; i < n; i += (int64_t)gridDim.x * kWetCols) {
    const T hv = h[i];
    if (hv > hextra) dmax = dev_fmax(dmax, wave_speed(hv, qx[i], qy[i]));
  }
  block_min_into(dmax >= T(0) ? speed_key((double)dmax) : kDtKeyInf, &clk->dt_key[clk->rd]);
}

// ---------------------------------------------------------------------------
// The post kernel: wet/dry masks, max depth and the CFL dt, tile by tile of the
// flux kernel's tiles; the end of the step.
//
// A warp walks a tile as the flux kernel does: lane l holds column c0-1+l, the
// rows come one after the other with the next row's loads in flight, east and
// west neighbours by shuffle.  Ghost cells belong to the tiles at the grid's
// edge (the reference's dt covers rows*cols).  It is a stream of 40 B (FP64) or
// 20 B a cell read and 8 or 4 written where a max depth rises, so what counts is
// loads in flight: no staging through shared memory, no block barrier, and as
// many warps as registers allow.
// A dry tile (flagged all +0 by the flux kernel in the step's destination
// buffer) has no wet cell: nothing to mask and no wave speed, and nothing to
// record while no max depth is negative and the arrival depth is not.
// ---------------------------------------------------------------------------
template <typename T>
struct PostArgs {
  const T* h;
  T* qx;
  T* qy;
  const T* z;  // FP32 form: offsets from the bed tiles' bases
  BedMap<T> bed;
  T* maxh;
  float* arrival;
  float arrival_depth, t_end;
  int rows, cols, rb;
  T hextra;
};

template <typename T>
__device__ __forceinline__ PostArgs<T> post_args(const StepNow& now, const StateBufs<T>& sb, const BedMap<T>& bed,
                                                 T* maxh, float* arrival, float arrival_depth, int rows, int cols,
                                                 int rb, T hextra) {
  PostArgs<T> P;
  P.h = sb.H(now.dst);
  P.qx = sb.QX(now.dst);
  P.qy = sb.QY(now.dst);
  P.z = bed.z;
  P.bed = bed;
  P.maxh = maxh;
  P.arrival = arrival;
  P.arrival_depth = arrival_depth;
  P.t_end = (float)now.t_end;
  P.rows = rows;
  P.cols = cols;
  P.rb = rb;
  P.hextra = hextra;
  return P;
}

// One tile (whole warp): returns the largest wave speed of dmax and the lane's
// cells.  The kernels take the tiles last first: the flux kernel has just
// written the last ones, and what of them is in L2 is read before it is evicted
// (rain on 1531x2049, FP64: step 193.2 -> 190.4 us).
template <typename T>
__device__ __forceinline__ T post_tile(const PostArgs<T>& P, unsigned tile, int lane, T dmax) {
  constexpr bool kF32 = sizeof(T) == 4;
  const T E12 = eps12<T>();
  const int rows = P.rows, cols = P.cols;
  const unsigned ns = (unsigned)(cols - 2 + kStripCols - 1) / kStripCols;
  const int sx = (int)(tile % ns), ry = (int)(tile / ns);
  const int c = sx * kStripCols + lane;
  const bool incol = c < cols;
  const bool upd = lane >= 1 && lane <= kStripCols && c <= cols - 2;  // an interior column of this tile
  const bool own = upd || (incol && (c == 0 || c == cols - 1));       // or a ghost column
  const int r0 = 1 + ry * P.rb, r1 = min(r0 + P.rb - 1, rows - 2);
  const int ra = r0 == 1 ? 0 : r0, rz = r1 == rows - 2 ? rows - 1 : r1;
  // FP32 form: bed levels relative to a reference per 128 columns and bed tile
  // row (deltas of the bed tiles of columns c-1, c, c+1), so that a difference
  // of levels keeps FP32 accuracy on high terrain
  T dw = T(0), dc = T(0), de = T(0);
  double ref = 0.0;
  auto deltas = [&](int r) {
    if (kF32 && upd) {
      ref = P.bed.base_at(r, c & ~(kWetCols - 1));
      dw = (T)(P.bed.base_at(r, c - 1) - ref);
      dc = (T)(P.bed.base_at(r, c) - ref);
      de = (T)(P.bed.base_at(r, c + 1) - ref);
    }
  };
  struct Row {
    T h, z, qx, qy, m;
  };
  const T* __restrict__ hp = P.h;
  const T* __restrict__ zp = P.z;
  const T* __restrict__ mp = P.maxh;
  // row r's values; of the row below the tile only the depth and the bed
  auto load = [&](int r) {
    Row w;
    w.h = w.z = w.qx = w.qy = w.m = T(0);
    const size_t id = (size_t)r * cols + c;
    if (incol && r <= rz + 1 && r < rows) {
      w.h = hp[id];
      w.z = zp[id];
    }
    if (own && r <= rz) {
      w.qx = P.qx[id];
      w.qy = P.qy[id];
      if (upd && r >= 1 && r <= rows - 2) w.m = mp[id];
    }
    return w;
  };
  T hn = T(0), zn = T(0);  // the row above
  if (ra > 0 && incol) {
    const size_t id = (size_t)(ra - 1) * cols + c;
    hn = hp[id];
    zn = zp[id];
  }
  // two rows of loads in flight
  Row cur = load(ra), nxt = load(ra + 1);
  deltas(ra);
  for (int r = ra; r <= rz; ++r) {
    const Row nx2 = load(r + 2);
    if (kF32 && r > ra && (r & 31) == 0) deltas(r);
    const T he = __shfl_down_sync(0xffffffffu, cur.h, 1), hw = __shfl_up_sync(0xffffffffu, cur.h, 1);
    T ze = __shfl_down_sync(0xffffffffu, cur.z, 1), zw = __shfl_up_sync(0xffffffffu, cur.z, 1);
    const size_t id = (size_t)r * cols + c;
    const bool wet = cur.h > P.hextra;
    T qx = cur.qx, qy = cur.qy;
    if (upd && r >= 1 && r <= rows - 2) {
      if (wet && (he < E12 || hw < E12 || hn < E12 || nxt.h < E12)) {  // a dry neighbour may stop the flow
        T zc = cur.z, zu = zn, zd = nxt.z;
        if (kF32) {
          zc += dc;
          ze += de;
          zw += dw;
          zu += (r & 31) == 0 ? (T)(P.bed.base_at(r - 1, c) - ref) : dc;
          zd += (r & 31) == 31 ? (T)(P.bed.base_at(r + 1, c) - ref) : dc;
        }
        const T level = cur.h + zc;
        if ((level < ze && he < E12) || (level < zw && hw < E12)) {
          qx = T(0);
          P.qx[id] = T(0);
        }
        if ((level < zu && hn < E12) || (level < zd && nxt.h < E12)) {
          qy = T(0);
          P.qy[id] = T(0);
        }
      }
      if (cur.h > cur.m) P.maxh[id] = cur.h;
      if (P.arrival != nullptr && cur.h > P.arrival_depth && !(P.arrival[id] < 3.0e38f)) P.arrival[id] = P.t_end;
    }
    if (own && wet) dmax = dev_fmax(dmax, wave_speed(cur.h, qx, qy));
    hn = cur.h;
    zn = cur.z;
    cur = nxt;
    nxt = nx2;
  }
  return dmax;
}

// Interior cells of a tile.
__device__ __forceinline__ unsigned tile_cells(unsigned tile, int rows, int cols, int rb) {
  const unsigned ns = (unsigned)(cols - 2 + kStripCols - 1) / kStripCols;
  const int sx = (int)(tile % ns), r0 = 1 + (int)(tile / ns) * rb;
  return (unsigned)((min(r0 + rb - 1, rows - 2) - r0 + 1) * min(kStripCols, cols - 2 - sx * kStripCols));
}

// tflag: the flux kernel's tile flags where dry tiles are skipped, else null.
template <typename T>
__global__ void __launch_bounds__(kWetCols, PostBlocks<T>::v)
    k_post(DevClock* __restrict__ clk, const __grid_constant__ StateBufs<T> sb, const __grid_constant__ BedMap<T> bed,
           T* __restrict__ maxh, int rows, int cols, T hextra, float* __restrict__ arrival, float arrival_depth,
           const uint8_t* __restrict__ tflag, const int32_t* __restrict__ maxh_neg, int rb, unsigned ntiles) {
  pdl_wait();
  pdl_trigger();
  const bool skips = tflag != nullptr && *maxh_neg == 0;
  if (!clk->now.active) return;
  const int lane = threadIdx.x & 31;
  const unsigned warps = gridDim.x * (kWetCols / 32);
  const PostArgs<T> P = post_args<T>(clk->now, sb, bed, maxh, arrival, arrival_depth, rows, cols, rb, hextra);
  const uint8_t* flags = nullptr;
  if (skips) flags = tflag + (size_t)clk->now.dst * ntiles;
  T dmax = T(-1);
  unsigned skipped = 0;  // interior cells of the tiles this lane found dry
  // the warp's tiles are t, t + warps, ...; 32 of them are looked at at once
  for (unsigned t = blockIdx.x * (kWetCols / 32) + (threadIdx.x >> 5); t < ntiles; t += 32 * warps) {
    const uint64_t mine = t + (uint64_t)lane * warps;
    bool todo = mine < ntiles;
    if (todo && flags != nullptr && flags[ntiles - 1 - mine]) {
      todo = false;
      skipped += tile_cells(ntiles - 1 - (unsigned)mine, rows, cols, rb);
    }
    for (unsigned left = __ballot_sync(0xffffffffu, todo); left != 0; left &= left - 1)
      dmax = post_tile<T>(P, ntiles - 1 - (t + (unsigned)(__ffs(left) - 1) * warps), lane, dmax);
  }
  skipped = __reduce_add_sync(0xffffffffu, skipped);
  if (lane == 0 && skipped)
    atomicAdd(&clk->skipped[1][(blockIdx.x * 4 + (threadIdx.x >> 5)) % kSkipSlots], (unsigned long long)skipped);
  block_min_into(dmax >= T(0) ? speed_key((double)dmax) : kDtKeyInf, &clk->dt_key[clk->now.wr]);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (clk->wait_test) wait_test(clk);
    fold_accounts(clk);
    end_step(clk);  // writes nothing that the other blocks read
  }
}

// ===========================================================================
// Batched ensembles: one launch per kernel type advances every member of a
// batch by one of its own steps (each member keeps its own clock and dt).
// Members are described in device memory (MemberDev); the flux kernel's warps
// take tiles from one queue over all members' tiles, the post kernel's
// blocks are a concatenation of every member's blocks.
// ===========================================================================
// The first step's clocks of an advance; later ones are run by the post kernel.
template <typename T>
__global__ void k_batch_clock(const MemberDev<T>* __restrict__ mem, int nm, BatchCtl* __restrict__ ctl) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m == 0) ctl->tile_next = 0;
  if (m < nm) mem[m].clk->now = begin_step(mem[m].clk);
}

template <typename T>
__device__ __forceinline__ FluxCtx<T> member_ctx(const MemberDev<T>& M) {
  return flux_ctx<T>(M.clk, M.clk->now, M.sb, M.bed, M.n2, M.zone, M.rates, M.rows, M.cols, M.rb, M.dx, M.rdx, M.hextra);
}

template <typename T, int MINB>
__global__ void __launch_bounds__(128, MINB) k_batch_flux(const MemberDev<T>* __restrict__ mem,
                                                          const int32_t* __restrict__ tile_member,
                                                          BatchCtl* __restrict__ ctl, uint32_t ntiles) {
  __shared__ FluxCtx<T> s_ctx[4];  // the member context of each warp's tile
  const int lane = threadIdx.x & 31;
  pdl_wait();
  const int rb = mem[0].rb;
  const unsigned split = min(ntiles, gridDim.x * 4u), nunits = ntiles - split + split * tile_parts(rb);
  while (true) {
    unsigned n = 0;
    if (lane == 0) n = atomicAdd(&ctl->tile_next, 1u);
    n = __shfl_sync(0xffffffffu, n, 0);
    if (n >= nunits) break;
    int part;
    const unsigned tile = unit_tile(n, ntiles, split, rb, &part);
    const MemberDev<T>& M = mem[tile_member[tile]];
    if (!M.clk->now.active) continue;
    FluxUnit u = whole_tile(tile - M.tile_begin, M.rows, (M.cols - 2 + kStripCols - 1) / kStripCols, rb);
    take_part(&u, part, rb);
    if (u.r0 > u.r1) continue;
    __syncwarp();  // the warp's previous unit no longer reads its context
    FluxCtx<T>& X = s_ctx[threadIdx.x >> 5];
    if (lane == 0) X = member_ctx<T>(M);
    __syncwarp();
    flux_tile_member<T>(X, u, lane);
  }
  pdl_trigger();
}

// The post kernel of every member: block b serves member post_member[b], whose
// warps share the member's tiles.  A member's last block folds its volume
// accounts and runs its clock for the next step, which the other members'
// blocks hide (a kernel for all clocks took 6 to 7 us a step).
template <typename T>
__global__ void __launch_bounds__(kWetCols, PostBlocks<T>::batch)
    k_batch_post(const MemberDev<T>* __restrict__ mem, const int32_t* __restrict__ post_member,
                 BatchCtl* __restrict__ ctl) {
  pdl_wait();
  pdl_trigger();
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->tile_next = 0;  // this step's flux launch is done
  const unsigned b = gridDim.x - 1 - blockIdx.x;  // last members first, see post_tile
  const MemberDev<T>& M = mem[post_member[b]];
  DevClock* clk = M.clk;
  if (!clk->now.active) return;
  const PostArgs<T> P = post_args<T>(clk->now, M.sb, M.bed, M.maxh, M.arrival, M.arrival_depth, M.rows, M.cols, M.rb,
                                     M.hextra);
  const unsigned warps = M.post_count * (kWetCols / 32), ntiles = M.tile_end - M.tile_begin;
  T dmax = T(-1);
  for (unsigned t = (b - M.post_begin) * (kWetCols / 32) + (threadIdx.x >> 5); t < ntiles; t += warps)
    dmax = post_tile<T>(P, ntiles - 1 - t, threadIdx.x & 31, dmax);
  block_min_into(dmax >= T(0) ? speed_key((double)dmax) : kDtKeyInf, &clk->dt_key[clk->now.wr]);
  if (threadIdx.x == 0) {  // block_min_into's atomic was this thread's
    __threadfence();
    if (atomicAdd(&clk->post_done, 1u) == M.post_count - 1) {
      __threadfence();
      clk->post_done = 0;
      fold_accounts(clk);
      if (end_step(clk)) atomicAdd(&ctl->halted, 1);
      clk->now = begin_step(clk);
    }
  }
}

// ===========================================================================
// Single-launch batches: k_batch_steps advances every member of a batch by
// `nsteps` of its own time steps in ONE launch.  Blocks stay resident and take
// work items from a ticket counter in a fixed order; per batched step s:
//   nm clock items (one per member), then the flux tiles of all members in
//   groups of four (one per warp), then nm forcing items (a member's point
//   sources, open-edge ghosts and external-boundary cells, wave by wave), then
//   the wet-dry/dt blocks of all members.
// An item waits only for items of its own member with lower tickets (flux
// tiles for the member's clock of step s, forcing for all its flux tiles of
// step s, wet-dry blocks for its forcing of step s, the clock of step s+1 for
// all its wet-dry blocks of step s), counted in MemberProgress.  Lower
// tickets were taken by blocks that are running, so the lowest unfinished
// ticket can always proceed and every wait ends: members advance without a
// barrier across members or across the grid, and the tail of one phase
// overlaps the next phase of members that are ahead.  Waits are bounded
// (kStepWaitPolls); one that gives up records a status, and the others then
// give up at once.  A producer publishes as a grid barrier does: a block (or
// warp) barrier, then one thread's gpu-scope fence and increment; a consumer
// polls with one thread's acquire load, then a block (or warp) barrier (and
// a proxy fence before bulk copies).  A block takes its next ticket while
// its current item runs, and acquires a (member, step) dependency once for
// consecutive items of the same kind.
// ===========================================================================
template <typename T>
__device__ __forceinline__ void forcing_block(const MemberDev<T>& M) {
  DevClock* clk = M.clk;
  for (int w = 0; w < M.src_nw; ++w) {
    for (int i = M.src_woff[w] + (int)threadIdx.x; i < M.src_woff[w + 1]; i += blockDim.x)
      source_apply<T>(clk, clk->now, M.sb, M.f, M.dx, M.src_order[i]);
    __syncthreads();
  }
  if (M.open) {
    const int n = max(M.rows, M.cols);
    for (int k = threadIdx.x; k < n; k += blockDim.x) open_bc_item<T>(clk->now.dst, M.sb, M.rows, M.cols, k);
    __syncthreads();
  }
  for (int w = 0; w < M.bc_nw; ++w) {
    for (int i = M.bc_woff[w] + (int)threadIdx.x; i < M.bc_woff[w + 1]; i += blockDim.x)
      extbc_apply<T>(clk, clk->now, M.sb, M.bed, M.n2, M.bc_order[i], M.f, M.rows, M.cols);
    __syncthreads();
  }
}

// Bounded wait until *counter >= target (acquire).  A wait that gives up
// records the status; once any wait of the launch has given up, the others
// give up at once instead of waiting out their own limit.
__device__ __forceinline__ void steps_wait(const uint32_t* counter, uint32_t target, BatchCtl* ctl,
                                           uint32_t polls = kStepWaitPolls) {
  for (uint32_t it = 0; it < polls; ++it) {
    if (ld_acquire_u32(counter) >= target) return;
    if (*reinterpret_cast<volatile int32_t*>(&ctl->status) != 0) return;
    if (it > 32) __nanosleep(128);
  }
  atomicExch(&ctl->status, kStatusStepWait);
}

// Publishes a block's item: after a block barrier (every thread's writes of
// the item happen before it), one thread makes them visible at gpu scope
// (a cumulative fence) and counts the item; the pattern of a grid barrier.
__device__ __forceinline__ void publish_block(uint32_t* counter) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(counter, 1u);
  }
}

// Thread 0 waits for *counter >= target (acquire); the block barrier after
// it orders every thread's later reads after what the producers published.
__device__ __forceinline__ void acquire_block(const uint32_t* counter, uint32_t target, BatchCtl* ctl) {
  if (threadIdx.x == 0) steps_wait(counter, target, ctl);
  __syncthreads();
}

// The kinds of block item.  The clock, forcing and wet-dry items are compiled
// out of line, so their registers are allocated apart from the flux tile's
// (the persistent loop keeps only a few values live across the calls).
// *seen caches the last (member, step) whose clock this warp has acquired:
// consecutive tiles of one member and step wait once.
template <typename T>
__device__ __forceinline__ void steps_flux_item(const MemberDev<T>* __restrict__ mem,
                                                const int32_t* __restrict__ tile_member, uint32_t ntiles,
                                                uint32_t r, uint32_t s, BatchCtl* __restrict__ ctl,
                                                MemberProgress* __restrict__ prog, uint32_t* seen_m,
                                                uint32_t* seen_s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t tile = 4u * r + (uint32_t)warp;  // one tile per warp
  if (tile >= ntiles) return;
  const int m = tile_member[tile];
  const MemberDev<T>& M = mem[m];
  if (*seen_m != (uint32_t)m || *seen_s != s) {
    if (lane == 0) steps_wait(&prog[m].clock, s + 1, ctl);
    __syncwarp();
    *seen_m = (uint32_t)m;
    *seen_s = s;
  }
  if (M.clk->now.active) {
    __shared__ FluxCtx<T> s_ctx[4];  // the member context of each warp's tile, reread every row
    if (lane == 0)
      s_ctx[warp] = member_ctx<T>(M);
    __syncwarp();
    flux_tile_member<T>(s_ctx[warp],
                        whole_tile(tile - M.tile_begin, M.rows, (M.cols - 2 + kStripCols - 1) / kStripCols, M.rb),
                        lane);
  }
  __syncwarp();
  if (lane == 0) {
    __threadfence();
    atomicAdd(&prog[m].flux, 1u);
  }
}

template <typename T>
__device__ __noinline__ void steps_clock_item(const MemberDev<T>& M, uint32_t m, uint32_t s,
                                              BatchCtl* __restrict__ ctl, MemberProgress* __restrict__ prog) {
  // test hook (tri_batch_set_wait_test): the first clock item waits for a
  // count no item ever reaches, bounded by ctl->wait_test polls, so the
  // handling of a wait that gave up can be tested with nothing else wrong
  if (ctl->wait_test != 0 && m == 0 && s == 0) steps_wait(&prog[0].clock, 0xFFFFFFFFu, ctl, ctl->wait_test);
  steps_wait(&prog[m].wet, s * M.wet_count, ctl);
  M.clk->now = begin_step(M.clk);
  if (M.clk->now.active && end_step(M.clk)) atomicAdd(&ctl->halted, 1);
  __threadfence();
  atomicAdd(&prog[m].clock, 1u);
}

template <typename T>
__device__ __noinline__ void steps_forcing_item(const MemberDev<T>& M, uint32_t m, uint32_t s,
                                                BatchCtl* __restrict__ ctl, MemberProgress* __restrict__ prog) {
  acquire_block(&prog[m].flux, (s + 1) * (M.tile_end - M.tile_begin), ctl);
  if (M.clk->now.active) forcing_block<T>(M);
  publish_block(&prog[m].forcing);
}

// Returns true when the block must take no further item (a copy group of
// its staging never completed, so its shared memory may still be written).
// The forcing of (member, step) is acquired once per block: consecutive
// bands of one member and step do not wait again.
template <typename T>
__device__ __noinline__ bool steps_wet_item(const MemberDev<T>* __restrict__ mem,
                                            const int32_t* __restrict__ wet_member, uint32_t r, uint32_t s,
                                            BatchCtl* __restrict__ ctl, MemberProgress* __restrict__ prog,
                                            unsigned char* smem, uint32_t* seen_m, uint32_t* seen_s) {
  using S = WetStage<T>;
  const int m = wet_member[r];
  const MemberDev<T>& M = mem[m];
  if (*seen_m != (uint32_t)m || *seen_s != s) {
    acquire_block(&prog[m].forcing, s + 1, ctl);
    *seen_m = (uint32_t)m;
    *seen_s = s;
  }
  DevClock* clk = M.clk;
  bool broken = false;
  if (clk->now.active) {
    fence_proxy_async_global();  // the bulk copies read what other blocks wrote
    const uint32_t local = r - M.wet_begin;
    if (local == 0 && threadIdx.x == 0) fold_accounts(clk);
    const unsigned long long key =
        wetdry_staged<T>(clk, M.sb, M.bed, M.maxh, M.rows, M.cols, M.hextra, M.arrival, M.arrival_depth,
                         (int)(local % M.wet_nbx), (int)(local / M.wet_nbx), reinterpret_cast<T*>(smem));
    block_min_into(key, &clk->dt_key[clk->now.wr]);
    broken = __syncthreads_or(clk->status == kStatusStageTimeout) != 0;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + S::kData);
    if (!broken && threadIdx.x < S::kGroups) mbar_inval(&bar[threadIdx.x]);
  }
  publish_block(&prog[m].wet);
  return broken;
}

// The next ticket is taken while the current item runs (its atomic's latency
// hidden); a block then holds two tickets, but its next one is higher than
// its current one, so the lowest unfinished ticket is always a current item
// and can proceed.
template <typename T, int MINB>
__global__ void __launch_bounds__(128, MINB)
    k_batch_steps(const MemberDev<T>* __restrict__ mem, int nm, const int32_t* __restrict__ tile_member,
                  uint32_t ntiles, const int32_t* __restrict__ wet_member, uint32_t nwet, int nsteps,
                  BatchCtl* __restrict__ ctl, MemberProgress* __restrict__ prog) {
  extern __shared__ __align__(128) unsigned char wet_smem[];
  __shared__ uint32_t s_ticket[2];
  const uint32_t nflux = (ntiles + 3) / 4;
  const uint32_t per_step = 2u * (uint32_t)nm + nflux + nwet;
  const uint32_t total = per_step * (uint32_t)nsteps;
  if (threadIdx.x == 0) s_ticket[0] = atomicAdd(&ctl->ticket, 1u);
  __syncthreads();
  uint32_t fm = 0xFFFFFFFFu, fs = 0, wm = 0xFFFFFFFFu, ws = 0;  // last acquired (member, step) per kind
  for (int cur = 0;; cur ^= 1) {
    const uint32_t t = s_ticket[cur];
    if (t >= total) return;
    if (threadIdx.x == 0) s_ticket[cur ^ 1] = atomicAdd(&ctl->ticket, 1u);
    const uint32_t s = t / per_step;
    uint32_t r = t - s * per_step;
    if (r < (uint32_t)nm) {  // clock of member r, step s
      if (threadIdx.x == 0) steps_clock_item<T>(mem[r], r, s, ctl, prog);
    } else if ((r -= (uint32_t)nm) < nflux) {
      steps_flux_item<T>(mem, tile_member, ntiles, r, s, ctl, prog, &fm, &fs);
    } else if ((r -= nflux) < (uint32_t)nm) {
      steps_forcing_item<T>(mem[r], r, s, ctl, prog);
    } else {
      r -= (uint32_t)nm;
      if (steps_wet_item<T>(mem, wet_member, r, s, ctl, prog, wet_smem, &wm, &ws)) return;
    }
    __syncthreads();  // the item is finished by every thread; the next ticket is visible
  }
}

}  // namespace tri
