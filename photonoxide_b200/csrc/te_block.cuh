// Several 2D TE steps in one launch (included by batch.cu): a CTA takes a tile of a grid with HALO
// places around it, holds its E_x, E_y, H_z and cb in registers (a lane four places of R rows of a
// warp) and its CPML psi in shared memory, takes up to HALO steps, each of which spoils one place
// more of the halo's rim, and writes the tile's own places back. So the fields cross memory once
// for HALO steps, where a step a launch reads and writes 32 bytes a cell each time; and a step
// costs two barriers, an exchange of one row a warp and the arithmetic, not a launch and its
// loads. Each value's arithmetic is te_step_kernel's, operation for operation (a halo place is
// computed by every CTA that holds it, to the same bits), so the results are the same bits.
//
// The step's code stays short: with the CPML's updates unrolled into every row it ran at a third of
// the issue rate, waiting for instructions more than for anything else (no-instruction stalls 3.0 of
// 10.6 cycles an instruction), so they are loops of one copy each over rows laid in shared memory.
//
// Sources, monitored values and the adjoint's curls are few places of few tiles: a tile that has
// some lays its new fields out in shared memory once a half-step, where a thread per source adds,
// a thread per item reads, and the lanes take their values back.
#pragma once

namespace pxb {

// A value recorded after each step: its place in the tile's region, its component (0 E_x, 1 E_y, 2
// H_z, 3 a component that stays zero), and where it goes: ring column `col`, or (col < 0) probe
// `probe` of the instance's record row.
struct TeRec {
  int local, comp;
  long long col;
  int probe, pad;
};
// A design value whose curl is kept after each step (te_design_kernel): component and number.
struct TeDesign {
  int local, comp;
  long long d;
};

template <typename T>
struct BlockArgs {
  const int *hbucket, *ebucket;  // per tile: its sources on H_z and on E, halo places included
  const Group *hgroups, *egroups;
  const Entry *entries;
  const double *waves_h, *waves_e;  // the chunk's, 2 x nwaves a step
  int nwaves;
  const int *hrecs, *erecs;  // per tile: its recorded values of H_z and of the others
  const TeRec *hrec, *erec;
  T *ring;
  long long nring;
  const int *dbucket;  // per tile: its design values; null without a design
  const TeDesign *design;
  T *K;
  long long k_first, ndesign;
  int record;  // 0: no values recorded
  int ahead;   // the tile a CTA after this one's SM takes next, about: its rows are brought into L2
};

constexpr int BW = 128;  // places along x of a tile's region: four a lane

template <typename T, int NW, int R>
__host__ __device__ constexpr size_t block_smem_values() {
  // psi (H_z along x and y, E_y along x, E_x along y), the two arrays values are laid out in, the
  // exchanged rows, the x CPML's b and a and kappa/h along x, the same along y
  return (size_t)6 * NW * R * BW + (2 * NW + 1) * BW + 6 * BW + 8 * NW * R;
}

// A slab's psi at four places: psi <- b psi + a (d/h) where `in`; u, in the differences' place, is
// what the field's update takes: sign psi, or elsewhere a zero that leaves the field as it is (H
// subtracts dt u: +0; E adds cb u: -0).
template <typename T>
__device__ __forceinline__ void block_psi(T *psi, T *diff_u, const V4<T> &b, const V4<T> &a, T h, T inv,
                                          double rd, int fast, T sign, T nothing, int in) {
  V4<T> old = ldv(psi);
  const V4<T> diff = ldv(diff_u);
  T d[4], u[4];
  div4_by_step(diff.v, d, h, inv, rd, fast);
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const T nw = b.v[j] * old.v[j] + a.v[j] * d[j];
    u[j] = in >> j & 1 ? sign * nw : nothing;
    if (in >> j & 1) old.v[j] = nw;
  }
  stv(psi, old.v);
  stv(diff_u, u);
}

// A warp's places in an x slab, shared out: the few lanes that hold some (`lanes`; `in` which of a
// lane's four) times the warp's rows, an item a lane at a time, rather than row after row by those
// lanes alone (a row's psi is a chain of some 300 cycles however few lanes take it). f(row, holder,
// its `in`) for each item in the grid.
template <int R, typename F>
__device__ __forceinline__ void block_x_items(unsigned lanes, int in, int flags, int lane, F f) {
  const int n = __popc(lanes), first = n ? __ffs(lanes) - 1 : 0;
  const bool run = (lanes >> first) == (n < 32 ? (1u << n) - 1u : ~0u);  // one run of lanes
#pragma unroll 1
  for (int base = 0; base < n * R; base += 32) {
    const int it = base + lane, r = it / n, k = it - r * n;
    const bool valid = it < n * R;
    const int holder = !valid ? lane : run ? first + k : (int)__fns(lanes, 0, k + 1);
    const int its = __shfl_sync(0xffffffffu, in, holder);
    if (valid && (flags >> (4 * r) & 1)) f(r, holder, its);
  }
}

// g wrapped into 0 .. n-1 (from any number of periods away), or -1 beyond a wall.
__host__ __device__ __forceinline__ int wrap_any(int g, int n, int periodic) {
  if (g >= 0 && g < n) return g;
  if (!periodic) return -1;
  while (g < 0) g += n;
  while (g >= n) g -= n;
  return g;
}

template <typename T, int NW, int R, int HALO>
__global__ void __launch_bounds__(NW * 32, 1)
    te_block_kernel(const TeInst<T> *__restrict__ insts, const int *__restrict__ tile_inst,
                    BlockArgs<T> B, int m0, int count, int launch) {
  constexpr int ROWS = NW * R, OWNX = BW - 2 * HALO, OWNY = ROWS - 2 * HALO, AREA = ROWS * BW;
  constexpr int THREADS_ = NW * 32;
  static_assert(HALO % 4 == 0 && OWNY > 0, "whole vectors of halo, and rows of its own");
  extern __shared__ __align__(16) unsigned char block_raw[];
  T *psi_hx = reinterpret_cast<T *>(block_raw), *psi_hy = psi_hx + AREA, *psi_ex = psi_hy + AREA,
    *psi_ey = psi_ex + AREA;
  T *pub = psi_ey + AREA;            // [2][AREA]
  T *row_h = pub + 2 * AREA;         // [NW][BW]: each warp's last row of H_z
  T *row_e = row_h + NW * BW;        // [NW + 1][BW]: each warp's first row of E_x
  T *xco = row_e + (NW + 1) * BW;    // [6][BW]: the x CPML's b, a for H_z, then for E_y; fh, fe
  T *yco = xco + 6 * BW;             // [ROWS][8]: the y CPML's b, a for H_z, b, a for E_x; fh, fe
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int tile = blockIdx.x;
  const TeInst<T> &I = insts[tile_inst[tile]];
  const int lt = tile - I.tile0;
  const int X0 = (lt % I.tiles_x) * OWNX - HALO, Y0 = (lt / I.tiles_x) * OWNY - HALO;
  const int nx = I.nx, ny = I.ny, low_x = I.low_x, low_y = I.low_y;
  const long long N = I.N;
  const int cur = (I.parity + launch) & 1, pcur = (I.psi_parity + launch) & 1;
  const T dt = I.dt;
  const T *ein = I.e[cur], *hin = I.h[cur] + 2 * N, *pin = I.psi_h[cur];
  const T *pein = pcur ? I.psi_e2 : I.psi_e;
  const bool vec = (nx & 3) == 0;

  // -- the lane's places along x (the same for every row) and the warp's rows
  const int xb = X0 + 4 * lane;
  int okx = 0, inhx = 0, inex = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int m = wrap_any(xb + j, nx, I.px);
    if (m < 0) continue;
    okx |= 1 << j;
    if (!I.px) {
      const int side = m < low_x ? 0 : 1;
      if (in_slab(I.hx[side], m)) inhx |= 1 << j;
      if (in_slab(I.ex[side], m)) inex |= 1 << j;
    }
  }
  const bool whole = vec && okx == 15;  // four places of a row are one aligned vector
  const int slots = w * R * BW + 4 * lane;  // the lane's first place of the warp's first row
  // where the lane's places are in a row
  int off[4];
#pragma unroll
  for (int j = 0; j < 4; j++) off[j] = max(wrap_any(xb + j, nx, I.px), 0);
  // the lane's four values of row my (zero where a place is not in the grid)
  auto get = [&](const T *__restrict__ f, int my, T v[4]) {
    const T *row = f + (long long)(my < 0 ? 0 : my) * nx;
    if (whole) {
      V4<T> q = {{T(0), T(0), T(0), T(0)}};
      if (my >= 0) q = ldv(row + off[0]);
#pragma unroll
      for (int j = 0; j < 4; j++) v[j] = q.v[j];
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++) v[j] = my >= 0 && (okx >> j & 1) ? row[off[j]] : T(0);
    }
  };
  T ex[R][4], ey[R][4], hz[R][4], cbx[R][4], cby[R][4];
  int flags = 0;  // a row r: bit 4r in the grid, 4r+1 in H_z's y CPML, 4r+2 in E_x's
  bool held = false;  // a value the update sets to zero (cb 0: a wall, a conductor, beyond the grid)
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int my = wrap_any(Y0 + w * R + r, ny, I.py);
    get(ein, my, ex[r]);
    get(ein + N, my, ey[r]);
    get(hin, my, hz[r]);
    get(I.cb, my, cbx[r]);
    get(I.cb + N, my, cby[r]);
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
#pragma unroll
    for (int j = 0; j < 4; j++) held = held || cbx[r][j] == T(0) || cby[r][j] == T(0);
    const int my = wrap_any(Y0 + w * R + r, ny, I.py);
    if (my < 0) continue;
    flags |= 1 << (4 * r);
    T p[4];
    auto keep = [&](T *to, const T *from, int in) {  // psi of the lane's places in a slab
#pragma unroll
      for (int j = 0; j < 4; j++) p[j] = in >> j & 1 ? from[j] : T(0);
      stv(to + slots + r * BW, p);
    };
    if (inhx | inex) {
      T q[4], o[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int m = xb + j;  // (no slab along a periodic x)
        const SlabEntry &s = I.hx[m < low_x ? 0 : 1], &t = I.ex[m < low_x ? 0 : 1];
        q[j] = inhx >> j & 1 ? pin[s.psi + (long long)my * s.pw + (m - s.pf)] : T(0);
        o[j] = inex >> j & 1 ? pein[t.psi + (long long)my * t.pw + (m - t.pf)] : T(0);
      }
      keep(psi_hx, q, inhx);
      keep(psi_ex, o, inex);
    }
    if (!I.py) {
      const int side = my < low_y ? 0 : 1;
      const SlabEntry &s = I.hy[side], &t = I.ey[side];
      T q[4];
      if (in_slab(s, my)) {
        flags |= 2 << (4 * r);
        get(pin + s.psi + (long long)(my - s.from) * I.pitch, 0, q);
        keep(psi_hy, q, okx);
      }
      if (in_slab(t, my)) {
        flags |= 4 << (4 * r);
        get(pein + t.psi + (long long)(my - t.from) * I.pitch, 0, q);
        keep(psi_ey, q, okx);
      }
    }
  }
  // the CPMLs' coefficients at the region's places and rows
  for (int q = threadIdx.x; q < BW; q += THREADS_) {
    const int m = wrap_any(X0 + q, nx, I.px);
    T c[4] = {T(0), T(0), T(0), T(0)};
    if (m >= 0 && !I.px) {
      const SlabEntry &s = I.hx[m < low_x ? 0 : 1], &t = I.ex[m < low_x ? 0 : 1];
      if (in_slab(s, m)) c[0] = I.coefs[s.coef + m - s.from], c[1] = I.coefs[s.coef + s.count + m - s.from];
      if (in_slab(t, m)) c[2] = I.coefs[t.coef + m - t.from], c[3] = I.coefs[t.coef + t.count + m - t.from];
    }
    for (int k = 0; k < 4; k++) xco[k * BW + q] = c[k];
    xco[4 * BW + q] = m >= 0 ? I.fh[m] : T(0);
    xco[5 * BW + q] = m >= 0 ? I.fe[m] : T(0);
  }
  for (int q = threadIdx.x; q < ROWS; q += THREADS_) {
    const int m = wrap_any(Y0 + q, ny, I.py);
    T c[4] = {T(0), T(0), T(0), T(0)};
    if (m >= 0 && !I.py) {
      const SlabEntry &s = I.hy[m < low_y ? 0 : 1], &t = I.ey[m < low_y ? 0 : 1];
      if (in_slab(s, m)) c[0] = I.coefs[s.coef + m - s.from], c[1] = I.coefs[s.coef + s.count + m - s.from];
      if (in_slab(t, m)) c[2] = I.coefs[t.coef + m - t.from], c[3] = I.coefs[t.coef + t.count + m - t.from];
    }
    stv(yco + 8 * q, c);
    yco[8 * q + 4] = m >= 0 ? I.fh[nx + m] : T(0);
    yco[8 * q + 5] = m >= 0 ? I.fe[nx + m] : T(0);
  }
  for (int q = threadIdx.x; q < BW; q += THREADS_) row_e[NW * BW + q] = T(0);
  // a region that reaches beyond a wall keeps its places there at zero
  const bool edge = (!I.px && (X0 < 0 || X0 + BW > nx)) || (!I.py && (Y0 < 0 || Y0 + ROWS > ny));
  const int hg0 = B.hbucket[tile], hg1 = B.hbucket[tile + 1];
  const int eg0 = B.ebucket[tile], eg1 = B.ebucket[tile + 1];
  const int hr0 = B.record ? B.hrecs[tile] : 0, hr1 = B.record ? B.hrecs[tile + 1] : 0;
  const int er0 = B.record ? B.erecs[tile] : 0, er1 = B.record ? B.erecs[tile + 1] : 0;
  const int d0 = B.dbucket ? B.dbucket[tile] : 0, d1 = B.dbucket ? B.dbucket[tile + 1] : 0;
  const bool lay_h = hg1 > hg0 || hr1 > hr0 || d1 > d0, lay_e = eg1 > eg0 || er1 > er0;
  if (HALO == 4 && tile + B.ahead < (int)gridDim.x) {
    // one CTA an SM loads, steps and stores in turn; the next one's rows, a 128-byte line a lane
    // (2400 x 2400 places, both in one call: 34.5 -> 29.8 us a step; six grids of 1.29 M cells in
    // all, two tiles an SM or fewer: 17.6 -> 18.0)
    const TeInst<T> &Q = insts[tile_inst[tile + B.ahead]];
    const int t = tile + B.ahead - Q.tile0;
    const int x0 = max((t % Q.tiles_x) * OWNX - HALO, 0), x1 = min((t % Q.tiles_x) * OWNX - HALO + BW, Q.nx);
    const int y0 = (t / Q.tiles_x) * OWNY - HALO + w * R, c = (Q.parity + launch) & 1;
    constexpr int LINE = 128 / (int)sizeof(T), LINES = BW / LINE + 1;
#pragma unroll 1
    for (int q = lane; q < 5 * R * LINES; q += 32) {
      const int a = q / (R * LINES), y = y0 + q / LINES % R, x = min(x0 + q % LINES * LINE, x1 - 1);
      const T *f = a < 2 ? Q.e[c] + a * Q.N : a == 2 ? Q.h[c] + 2 * Q.N : Q.cb + (a - 3) * Q.N;
      if (y >= 0 && y < Q.ny)
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(f + (long long)y * Q.nx + x));
    }
  }
  const T *ca = I.ca;
  const T sx = I.sx, sy = I.sy, inv_sx = I.inv_sx, inv_sy = I.inv_sy;
  const int fast_x = I.fast_x, fast_y = I.fast_y;
  stv(row_e + w * BW + 4 * lane, ex[0]);
  const bool any_held = __syncthreads_or(held);
  // whether the warp has a slab's places, and the lanes that have an x slab's
  const unsigned lanes_h = __ballot_sync(0xffffffffu, inhx != 0), lanes_e = __ballot_sync(0xffffffffu, inex != 0);
  const bool slab_h = __any_sync(0xffffffffu, inhx != 0 || (flags & 0x2222)),
             slab_e = __any_sync(0xffffffffu, inex != 0 || (flags & 0x4444));

  for (int s = 0; s < count; s++) {
    const int m = m0 + s;
    // -- H_z (src/fdtd/kernel/reference.rs:14-56 with E_z, H_x, H_y zero)
    {
      const V4<T> exn = ldv(row_e + (w + 1) * BW + 4 * lane), fhx = ldv(xco + 4 * BW + 4 * lane);
#pragma unroll
      for (int r = 0; r < R; r++) {
        const T eyn = __shfl_down_sync(0xffffffffu, ey[r][0], 1);
        const T fhy = yco[8 * (w * R + r) + 4];
        T dx[4], dy[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          dx[j] = (j < 3 ? ey[r][j < 3 ? j + 1 : 3] : eyn) - ey[r][j];
          dy[j] = (r + 1 < R ? ex[r + 1 < R ? r + 1 : r][j] : exn.v[j]) - ex[r][j];
          hz[r][j] = hz[r][j] - dt * (dx[j] * fhx.v[j] - dy[j] * fhy);
        }
        if (slab_h) {  // for the CPML below
          stv(pub + slots + r * BW, dx);
          stv(pub + AREA + slots + r * BW, dy);
        }
      }
    }
    if (slab_h) {
      // the CPML: H_z along x (+), then along y (-); the lane's rows one after another, in one copy
      // of the code (see above), through its own places of `pub`
#pragma unroll 1
      for (int r = 0; r < R; r++) {
        T *d = pub + slots + r * BW;
        if (flags >> (4 * r) & 2) {
          const T b = yco[8 * (w * R + r)], a = yco[8 * (w * R + r) + 1];
          const V4<T> bb = {{b, b, b, b}}, aa = {{a, a, a, a}};
          block_psi<T>(psi_hy + slots + r * BW, d + AREA, bb, aa, sy, inv_sy, I.rd_y, fast_y, T(-1), T(0),
                       okx);
        }
      }
      __syncwarp();
      block_x_items<R>(lanes_h, inhx, flags, lane, [&](int r, int q, int in) {
        const int at = (w * R + r) * BW + 4 * q;
        block_psi<T>(psi_hx + at, pub + at, ldv(xco + 4 * q), ldv(xco + BW + 4 * q), sx, inv_sx, I.rd_x,
                     fast_x, T(1), T(0), in);
      });
      __syncwarp();
#pragma unroll
      for (int r = 0; r < R; r++) {
        if (inhx && (flags >> (4 * r) & 1)) {
          const V4<T> u = ldv(pub + slots + r * BW);
#pragma unroll
          for (int j = 0; j < 4; j++) hz[r][j] = hz[r][j] - dt * u.v[j];
        }
        if (flags >> (4 * r) & 2) {
          const V4<T> u = ldv(pub + AREA + slots + r * BW);
#pragma unroll
          for (int j = 0; j < 4; j++) hz[r][j] = hz[r][j] - dt * u.v[j];
        }
      }
    }
    if (edge) {
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (!(flags >> (4 * r) & okx >> j & 1)) hz[r][j] = T(0);
    }
    if (lay_h) {
#pragma unroll
      for (int r = 0; r < R; r++) stv(pub + slots + r * BW, hz[r]);
      __syncthreads();
      if (hg1 > hg0) {
        // the magnetic sources (src/fdtd.rs:1348-1359), each value's entries in CPU order
        const double *wave = B.waves_h + 2LL * m * B.nwaves;
        for (int g = hg0 + threadIdx.x; g < hg1; g += THREADS_) {
          const Group gr = B.hgroups[g];
          T v = pub[gr.local];
          for (int q = gr.first; q < gr.first + gr.count; q++)
            v = apply_h<T>(v, B.entries[q], wave, dt);
          pub[gr.local] = v;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; r++) {
          const V4<T> q = ldv(pub + slots + r * BW);
#pragma unroll
          for (int j = 0; j < 4; j++) hz[r][j] = q.v[j];
        }
      }
      for (int q = hr0 + threadIdx.x; q < hr1; q += THREADS_) {
        const TeRec it = B.hrec[q];
        if (it.col >= 0) B.ring[(long long)m * B.nring + it.col] = pub[it.local];
        else I.rows[(long long)m * I.nprobes + it.probe] = (double)pub[it.local];
      }
      for (int q = d0 + threadIdx.x; q < d1; q += THREADS_) {
        // the curl E's update multiplies by cb (te_design_kernel)
        const TeDesign it = B.design[q];
        const int x = X0 + it.local % BW, y = Y0 + it.local / BW;
        const T h = pub[it.local];
        T curl;
        if (it.comp == 0) curl = (h - pub[it.local - BW]) * I.fe[nx + wrap_any(y, ny, I.py)];
        else curl = T(0) - (h - pub[it.local - 1]) * I.fe[wrap_any(x, nx, I.px)];
        B.K[(I.first + m - B.k_first) * B.ndesign + it.d] = curl;
      }
    }
    stv(row_h + w * BW + 4 * lane, hz[R - 1]);
    __syncthreads();
    // -- E_x, E_y (reference.rs:58-99): back differences of the new H_z
    if (ca || any_held) {
      // ca E: ca 0 where cb is and 1 elsewhere (1 x E is E: nothing to do), or, where the grid has
      // one of its own, read again each step (no room to keep it)
#pragma unroll 1
      for (int r = 0; r < R && ca; r++) {
        T a[4];
        const int my = wrap_any(Y0 + w * R + r, ny, I.py);
        get(ca, my, a);
        stv(pub + slots + r * BW, a);
        get(ca + N, my, a);
        stv(pub + AREA + slots + r * BW, a);
      }
#pragma unroll
      for (int r = 0; r < R; r++) {
        if (ca) {
          const V4<T> a = ldv(pub + slots + r * BW), b = ldv(pub + AREA + slots + r * BW);
#pragma unroll
          for (int j = 0; j < 4; j++) ex[r][j] = a.v[j] * ex[r][j], ey[r][j] = b.v[j] * ey[r][j];
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++) {
            if (cbx[r][j] == T(0)) ex[r][j] = T(0) * ex[r][j];
            if (cby[r][j] == T(0)) ey[r][j] = T(0) * ey[r][j];
          }
        }
      }
    }
    {
      const V4<T> fex = ldv(xco + 5 * BW + 4 * lane);
      V4<T> hp = {{T(0), T(0), T(0), T(0)}};
      if (w > 0) hp = ldv(row_h + (w - 1) * BW + 4 * lane);
#pragma unroll
      for (int r = 0; r < R; r++) {
        const T hl = __shfl_up_sync(0xffffffffu, hz[r][3], 1);
        const T fey = yco[8 * (w * R + r) + 5];
        T dx[4], dy[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          dx[j] = hz[r][j] - (j > 0 ? hz[r][j > 0 ? j - 1 : 0] : hl);
          dy[j] = hz[r][j] - (r > 0 ? hz[r > 0 ? r - 1 : 0][j] : hp.v[j]);
          // curl_x = dyHz fey - dzHy fez and curl_y = dzHx fez - dxHz fex, with dzHy = dzHx = +0
          const T c0 = dy[j] * fey, c1 = T(0) - dx[j] * fex.v[j];
          ex[r][j] = ex[r][j] + cbx[r][j] * c0;
          ey[r][j] = ey[r][j] + cby[r][j] * c1;
        }
        if (slab_e) {
          stv(pub + slots + r * BW, dx);
          stv(pub + AREA + slots + r * BW, dy);
        }
      }
    }
    if (slab_e) {
      // the CPML: E_x along y (+), E_y along x (-)
#pragma unroll 1
      for (int r = 0; r < R; r++) {
        T *d = pub + slots + r * BW;
        if (flags >> (4 * r) & 4) {
          const T b = yco[8 * (w * R + r) + 2], a = yco[8 * (w * R + r) + 3];
          const V4<T> bb = {{b, b, b, b}}, aa = {{a, a, a, a}};
          block_psi<T>(psi_ey + slots + r * BW, d + AREA, bb, aa, sy, inv_sy, I.rd_y, fast_y, T(1), T(-0.0),
                       okx);
        }
      }
      __syncwarp();
      block_x_items<R>(lanes_e, inex, flags, lane, [&](int r, int q, int in) {
        const int at = (w * R + r) * BW + 4 * q;
        block_psi<T>(psi_ex + at, pub + at, ldv(xco + 2 * BW + 4 * q), ldv(xco + 3 * BW + 4 * q), sx,
                     inv_sx, I.rd_x, fast_x, T(-1), T(-0.0), in);
      });
      __syncwarp();
#pragma unroll
      for (int r = 0; r < R; r++) {
        if (flags >> (4 * r) & 4) {
          const V4<T> u = ldv(pub + AREA + slots + r * BW);
#pragma unroll
          for (int j = 0; j < 4; j++) ex[r][j] = ex[r][j] + cbx[r][j] * u.v[j];
        }
        if (inex && (flags >> (4 * r) & 1)) {
          const V4<T> u = ldv(pub + slots + r * BW);
#pragma unroll
          for (int j = 0; j < 4; j++) ey[r][j] = ey[r][j] + cby[r][j] * u.v[j];
        }
      }
    }
    if (edge) {
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (!(flags >> (4 * r) & okx >> j & 1)) ex[r][j] = ey[r][j] = T(0);
    }
    if (lay_e) {
      // (the barrier above: every thread is done with H_z's layout)
#pragma unroll
      for (int r = 0; r < R; r++) {
        stv(pub + slots + r * BW, ex[r]);
        stv(pub + AREA + slots + r * BW, ey[r]);
      }
      __syncthreads();
      if (eg1 > eg0) {
        // the electric currents (src/fdtd.rs:1375-1387)
        const double *wave = B.waves_e + 2LL * m * B.nwaves;
        for (int g = eg0 + threadIdx.x; g < eg1; g += THREADS_) {
          const Group gr = B.egroups[g];
          const int x = wrap_any(X0 + gr.local % BW, nx, I.px), y = wrap_any(Y0 + gr.local / BW, ny, I.py);
          T *at = pub + gr.comp * AREA + gr.local;
          T v = *at;
          const T cbv = I.cb[gr.comp * N + (long long)y * nx + x];
          for (int q = gr.first; q < gr.first + gr.count; q++)
            v = apply_e<T>(v, B.entries[q], wave, cbv);
          *at = v;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; r++) {
          const V4<T> q = ldv(pub + slots + r * BW), o = ldv(pub + AREA + slots + r * BW);
#pragma unroll
          for (int j = 0; j < 4; j++) ex[r][j] = q.v[j], ey[r][j] = o.v[j];
        }
      }
      for (int q = er0 + threadIdx.x; q < er1; q += THREADS_) {
        const TeRec it = B.erec[q];
        const T v = it.comp < 2 ? pub[it.comp * AREA + it.local] : T(0);
        if (it.col >= 0) B.ring[(long long)m * B.nring + it.col] = v;
        else I.rows[(long long)m * I.nprobes + it.probe] = (double)v;
      }
    }
    stv(row_e + w * BW + 4 * lane, ex[0]);
    __syncthreads();
  }

  // -- the tile's own places to the other copies
  T *eout = I.e[1 - cur], *hout = I.h[1 - cur] + 2 * N, *pout = I.psi_h[1 - cur];
  T *peout = pcur ? I.psi_e : I.psi_e2;
  if (4 * lane < HALO || 4 * lane >= BW - HALO) return;
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int row = w * R + r, y = Y0 + row;
    if (row < HALO || row >= ROWS - HALO || y >= ny) continue;  // an own row's place is in the grid
    const long long at = (long long)y * nx;
    auto put = [&](T *f, const T v[4]) {
      if (vec) {
        if (xb < nx) stv(f + at + xb, v);
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (xb + j < nx) f[at + xb + j] = v[j];
      }
    };
    put(eout, ex[r]);
    put(eout + N, ey[r]);
    put(hout, hz[r]);
    if ((inhx | inex) != 0) {
      const V4<T> q = ldv(psi_hx + slots + r * BW), o = ldv(psi_ex + slots + r * BW);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int m = xb + j;
        const SlabEntry &a = I.hx[m < low_x ? 0 : 1], &b = I.ex[m < low_x ? 0 : 1];
        if (inhx >> j & 1) pout[a.psi + (long long)y * a.pw + (m - a.pf)] = q.v[j];
        if (inex >> j & 1) peout[b.psi + (long long)y * b.pw + (m - b.pf)] = o.v[j];
      }
    }
    if (flags >> (4 * r) & 6) {
      const int side = y < low_y ? 0 : 1;
      const SlabEntry &a = I.hy[side], &b = I.ey[side];
      const V4<T> q = ldv(psi_hy + slots + r * BW), o = ldv(psi_ey + slots + r * BW);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (xb + j >= nx) continue;
        if (flags >> (4 * r) & 2) pout[a.psi + (long long)(y - a.from) * I.pitch + xb + j] = q.v[j];
        if (flags >> (4 * r) & 4) peout[b.psi + (long long)(y - b.from) * I.pitch + xb + j] = o.v[j];
      }
    }
  }
}

}  // namespace pxb
