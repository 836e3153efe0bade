// Several steps of the TE step's transpose in one launch (included by batch.cu): te_block_kernel's
// tile, a CTA with HALO places around its own, for te_adjoint_kernel's arithmetic, operation for
// operation. The adjoint fields and cb are in registers and psi~ in shared memory; each step first adds
// the objective's derivatives to the values that the transforms record and keeps E~ at the design's
// values. What bounds the steps one by one is latency: a step of a 240 x 180 grid took three launches,
// 21 us (te_inject_kernel and te_grad_kernel 4 us each, te_adjoint_kernel 12).
#pragma once

namespace pxb {

// A field value that the transforms record, in a tile's region: its place, its component (0 E_x, 1
// E_y, 2 H_z) and its transform values first .. first + count - 1 of the table of amounts.
struct AdjOwner {
  int local, comp, first, count;
};

template <typename T>
struct AdjTables {
  const int *obucket, *dbucket;  // per tile: its owners (E's, then H's from omid on), its design values
  const int *omid;
  const AdjOwner *owner;
  const TeDesign *design;
  const T *amount;  // [step of the segment][norder]
  long long norder;
  T *kept;  // [step of the segment][ndesign]: E~ there
  long long ndesign;
  int tiles_x;
};

// A slab's psi~ at four places: its total (what later steps carried, `sign` times this step's use of
// it added), the field's share (a/h) total in the use's place, and psi~ <- b total.
template <typename T>
__device__ __forceinline__ void adjoint_psi(T *psi, T *use, const V4<T> &b, const V4<T> &ah, T sign,
                                            int in) {
  V4<T> old = ldv(psi);
  const V4<T> used = ldv(use);
  T share[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const T total = sign > T(0) ? old.v[j] + used.v[j] : old.v[j] - used.v[j];
    share[j] = ah.v[j] * total;
    if (in >> j & 1) old.v[j] = b.v[j] * total;
  }
  stv(psi, old.v);
  stv(use, share);
}

// Steps m0, m0 - 1, ... of a segment, `count` (<= HALO) of them.
template <typename T, int NW, int R, int HALO>
__global__ void __launch_bounds__(NW * 32, 1)
    te_adjoint_block_kernel(const TeInst<T> *__restrict__ insts, AdjState<T> A, AdjTables<T> B, int m0,
                            int count) {
  constexpr int ROWS = NW * R, OWNX = BW - 2 * HALO, OWNY = ROWS - 2 * HALO, AREA = ROWS * BW;
  constexpr int THREADS_ = NW * 32;
  extern __shared__ __align__(16) unsigned char block_raw[];
  T *psi_hx = reinterpret_cast<T *>(block_raw), *psi_hy = psi_hx + AREA, *psi_ex = psi_hy + AREA,
    *psi_ey = psi_ex + AREA;
  T *pub = psi_ey + AREA;          // [2][AREA]
  T *row_h = pub + 2 * AREA;       // [NW][BW]: each warp's last row of H~
  T *row_e = row_h + NW * BW;      // [NW + 1][BW]: each warp's first row of cb (kappa/h) E~_x
  T *xco = row_e + (NW + 1) * BW;  // [6][BW]: the x CPML's b, a/h for H_z, then for E_y; fh, fe
  T *yco = xco + 6 * BW;           // [ROWS][8]: the y CPML's b, a/h for H_z, for E_x; fh, fe
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int tile = blockIdx.x;
  const TeInst<T> &I = insts[0];
  const int X0 = (tile % B.tiles_x) * OWNX - HALO, Y0 = (tile / B.tiles_x) * OWNY - HALO;
  const int nx = I.nx, ny = I.ny, low_x = I.low_x, low_y = I.low_y;
  const long long N = I.N;
  const T dt = I.dt;
  const T *eb = A.e[A.cur], *hb = A.h[A.cur], *pei = A.pe[A.cur], *phi = A.ph[A.cur];
  const bool vec = (nx & 3) == 0;
  const int xb = X0 + 4 * lane;
  int okx = 0, inhx = 0, inex = 0, off[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int m = wrap_any(xb + j, nx, I.px);
    off[j] = max(m, 0);
    if (m < 0) continue;
    okx |= 1 << j;
    if (!I.px) {
      const int side = m < low_x ? 0 : 1;
      if (in_slab(I.hx[side], m)) inhx |= 1 << j;
      if (in_slab(I.ex[side], m)) inex |= 1 << j;
    }
  }
  const bool whole = vec && okx == 15;
  const int slots = w * R * BW + 4 * lane;
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
  // a row r: bit 4r in the grid, 4r+1 in H_z's y CPML, 4r+2 in E_x's (and the rows after and before
  // the warp's, for the neighbours' shares)
  int flags = 0;
  auto row_flags = [&](int row) {
    const int my = wrap_any(Y0 + row, ny, I.py);
    if (my < 0) return 0;
    int f = 1;
    if (!I.py) {
      const int side = my < low_y ? 0 : 1;
      if (in_slab(I.hy[side], my)) f |= 2;
      if (in_slab(I.ey[side], my)) f |= 4;
    }
    return f;
  };
  bool held = false;
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int my = wrap_any(Y0 + w * R + r, ny, I.py);
    get(eb, my, ex[r]);
    get(eb + N, my, ey[r]);
    get(hb, my, hz[r]);
    get(I.cb, my, cbx[r]);
    get(I.cb + N, my, cby[r]);
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
#pragma unroll
    for (int j = 0; j < 4; j++) held = held || cbx[r][j] == T(0) || cby[r][j] == T(0);
    const int my = wrap_any(Y0 + w * R + r, ny, I.py);
    const int f = row_flags(w * R + r);
    flags |= f << (4 * r);
    if (my < 0) continue;
    T q[4], o[4];
    if (inhx | inex) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int m = xb + j;  // (no slab along a periodic x)
        const SlabEntry &s = I.hx[m < low_x ? 0 : 1], &t = I.ex[m < low_x ? 0 : 1];
        q[j] = inhx >> j & 1 ? phi[s.psi + (long long)my * s.pw + (m - s.pf)] : T(0);
        o[j] = inex >> j & 1 ? pei[t.psi + (long long)my * t.pw + (m - t.pf)] : T(0);
      }
      stv(psi_hx + slots + r * BW, q);
      stv(psi_ex + slots + r * BW, o);
    }
    if (f & 6) {
      const int side = my < low_y ? 0 : 1;
      const SlabEntry &s = I.hy[side], &t = I.ey[side];
      if (f & 2) {
        get(phi + s.psi + (long long)(my - s.from) * I.pitch, 0, q);
        stv(psi_hy + slots + r * BW, q);
      }
      if (f & 4) {
        get(pei + t.psi + (long long)(my - t.from) * I.pitch, 0, q);
        stv(psi_ey + slots + r * BW, q);
      }
    }
  }
  const int after = row_flags(w * R + R), before = row_flags(w * R - 1);
  for (int q = threadIdx.x; q < BW; q += THREADS_) {
    const int m = wrap_any(X0 + q, nx, I.px);
    T c[4] = {T(0), T(0), T(0), T(0)};
    if (m >= 0 && !I.px) {
      const SlabEntry &s = I.hx[m < low_x ? 0 : 1], &t = I.ex[m < low_x ? 0 : 1];
      if (in_slab(s, m)) c[0] = coef_b(I, s, m), c[1] = coef_a(I, s, m) / I.sx;
      if (in_slab(t, m)) c[2] = coef_b(I, t, m), c[3] = coef_a(I, t, m) / I.sx;
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
      if (in_slab(s, m)) c[0] = coef_b(I, s, m), c[1] = coef_a(I, s, m) / I.sy;
      if (in_slab(t, m)) c[2] = coef_b(I, t, m), c[3] = coef_a(I, t, m) / I.sy;
    }
    stv(yco + 8 * q, c);
    yco[8 * q + 4] = m >= 0 ? I.fh[nx + m] : T(0);
    yco[8 * q + 5] = m >= 0 ? I.fe[nx + m] : T(0);
  }
  for (int q = threadIdx.x; q < BW; q += THREADS_) row_e[NW * BW + q] = T(0);
  const bool edge = (!I.px && (X0 < 0 || X0 + BW > nx)) || (!I.py && (Y0 < 0 || Y0 + ROWS > ny));
  const int o0 = B.obucket[tile], o1 = B.obucket[tile + 1], om = B.omid[tile];
  const int d0 = B.dbucket[tile], d1 = B.dbucket[tile + 1];
  const T *ca = I.ca;
  const int nexte = __shfl_down_sync(0xffffffffu, inex, 1), prevh = __shfl_up_sync(0xffffffffu, inhx, 1);
  const bool any_held = __syncthreads_or(held);
  const bool slab_h = __any_sync(0xffffffffu, inhx != 0 || (flags & 0x2222)),
             slab_e = __any_sync(0xffffffffu, inex != 0 || (flags & 0x4444));
  const bool tile_slab = __syncthreads_or(slab_h || slab_e);
  const unsigned lanes_h = __ballot_sync(0xffffffffu, inhx != 0), lanes_e = __ballot_sync(0xffffffffu, inex != 0);

  for (int s = 0; s < count; s++) {
    const int m = m0 - s;
    const T *amount = B.amount + m * B.norder;
    if (o1 > o0 || d1 > d0) {
      // the objective's derivatives (te_inject_kernel), each value's in value order; E~ at the design
#pragma unroll
      for (int r = 0; r < R; r++) {
        stv(pub + slots + r * BW, ex[r]);
        stv(pub + AREA + slots + r * BW, ey[r]);
      }
      __syncthreads();
      for (int q = o0 + threadIdx.x; q < om; q += THREADS_) {
        const AdjOwner it = B.owner[q];
        T v = pub[it.comp * AREA + it.local];
        for (int k = it.first; k < it.first + it.count; k++) v = v + amount[k];
        pub[it.comp * AREA + it.local] = v;
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < R; r++) {
        const V4<T> q = ldv(pub + slots + r * BW), o = ldv(pub + AREA + slots + r * BW);
#pragma unroll
        for (int j = 0; j < 4; j++) ex[r][j] = q.v[j], ey[r][j] = o.v[j];
      }
      for (int q = d0 + threadIdx.x; q < d1; q += THREADS_) {
        const TeDesign it = B.design[q];
        B.kept[(long long)m * B.ndesign + it.d] = pub[it.comp * AREA + it.local];
      }
      if (o1 > om) {
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; r++) stv(pub + slots + r * BW, hz[r]);
        __syncthreads();
        for (int q = om + threadIdx.x; q < o1; q += THREADS_) {
          const AdjOwner it = B.owner[q];
          T v = pub[it.local];
          for (int k = it.first; k < it.first + it.count; k++) v = v + amount[k];
          pub[it.local] = v;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; r++) {
          const V4<T> q = ldv(pub + slots + r * BW);
#pragma unroll
          for (int j = 0; j < 4; j++) hz[r][j] = q.v[j];
        }
      }
      __syncthreads();  // `pub` is laid out anew below
    }
    // -- the E slabs' psi~: E_x += cb (+psi') along y, E_y += cb (-psi') along x
    if (slab_e) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        T p[4], q[4];
#pragma unroll
        for (int j = 0; j < 4; j++) p[j] = cbx[r][j] * ex[r][j], q[j] = cby[r][j] * ey[r][j];
        stv(pub + AREA + slots + r * BW, p);
        stv(pub + slots + r * BW, q);
      }
#pragma unroll 1
      for (int r = 0; r < R; r++) {
        T *d = pub + slots + r * BW;
        if (flags >> (4 * r) & 4) {
          const T b = yco[8 * (w * R + r) + 2], a = yco[8 * (w * R + r) + 3];
          const V4<T> bb = {{b, b, b, b}}, aa = {{a, a, a, a}};
          adjoint_psi<T>(psi_ey + slots + r * BW, d + AREA, bb, aa, T(1), okx);
        }
      }
      __syncwarp();
      block_x_items<R>(lanes_e, inex, flags, lane, [&](int r, int q, int in) {
        const int at = (w * R + r) * BW + 4 * q;
        adjoint_psi<T>(psi_ex + at, pub + at, ldv(xco + 2 * BW + 4 * q), ldv(xco + 3 * BW + 4 * q), T(-1),
                       in);
      });
    }
    const V4<T> fex = ldv(xco + 5 * BW + 4 * lane);
    {
      const T fey = yco[8 * w * R + 5];
      T p[4];
#pragma unroll
      for (int j = 0; j < 4; j++) p[j] = cbx[0][j] * fey * ex[0][j];
      stv(row_e + w * BW + 4 * lane, p);
    }
    __syncthreads();
    // -- H~ of the step's new H_z: E_x(x, y) read it with cb fey(y), E_x(x, y+1) with -cb fey(y+1),
    // E_y(x, y) with -cb fex(x), E_y(x+1, y) with +cb fex(x+1); then the slabs, along y and along x
#pragma unroll
    for (int r = 0; r < R; r++) {
      const T fey = yco[8 * (w * R + r) + 5], feyn = yco[8 * min(w * R + r + 1, ROWS - 1) + 5];
      V4<T> next = ldv(row_e + (w + 1) * BW + 4 * lane);
      if (r + 1 < R) {
#pragma unroll
        for (int j = 0; j < 4; j++) next.v[j] = cbx[r + 1 < R ? r + 1 : r][j] * feyn * ex[r + 1 < R ? r + 1 : r][j];
      }
      T px[4];
#pragma unroll
      for (int j = 0; j < 4; j++) px[j] = cby[r][j] * fex.v[j] * ey[r][j];
      const T pn = __shfl_down_sync(0xffffffffu, px[0], 1);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        T acc = hz[r][j] + cbx[r][j] * fey * ex[r][j] - px[j];
        acc = acc - next.v[j];
        acc = acc + (j < 3 ? px[j < 3 ? j + 1 : 3] : pn);
        hz[r][j] = acc;
      }
    }
    if (tile_slab) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        if (flags >> (4 * r) & 4) {
          const V4<T> q = ldv(pub + AREA + slots + r * BW);
#pragma unroll
          for (int j = 0; j < 4; j++) hz[r][j] = hz[r][j] + q.v[j];
        }
        if (((r + 1 < R ? flags >> (4 * (r + 1)) : after) & 4) && w * R + r + 1 < ROWS &&
            (flags >> (4 * r) & 1)) {
          const V4<T> q = ldv(pub + AREA + slots + (r + 1) * BW);
#pragma unroll
          for (int j = 0; j < 4; j++) hz[r][j] = hz[r][j] - q.v[j];
        }
        const V4<T> t = ldv(pub + slots + r * BW);
        const T tn = __shfl_down_sync(0xffffffffu, t.v[0], 1);
        if (flags >> (4 * r) & 1) {
#pragma unroll
          for (int j = 0; j < 4; j++) {
            if (inex >> j & 1) hz[r][j] = hz[r][j] + t.v[j];
            if (j < 3 ? inex >> (j + 1) & 1 : nexte & 1) hz[r][j] = hz[r][j] - (j < 3 ? t.v[j < 3 ? j + 1 : 3] : tn);
          }
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
    if (tile_slab) __syncthreads();  // every warp is done with `pub`
    // -- the H slabs' psi~: H_z -= dt (+psi') along x, H_z -= dt (-psi') along y
    if (slab_h) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        T p[4];
#pragma unroll
        for (int j = 0; j < 4; j++) p[j] = dt * hz[r][j];
        stv(pub + AREA + slots + r * BW, p);
        stv(pub + slots + r * BW, p);
      }
#pragma unroll 1
      for (int r = 0; r < R; r++) {
        T *d = pub + slots + r * BW;
        if (flags >> (4 * r) & 2) {
          const T b = yco[8 * (w * R + r)], a = yco[8 * (w * R + r) + 1];
          const V4<T> bb = {{b, b, b, b}}, aa = {{a, a, a, a}};
          adjoint_psi<T>(psi_hy + slots + r * BW, d + AREA, bb, aa, T(1), okx);
        }
      }
      __syncwarp();
      block_x_items<R>(lanes_h, inhx, flags, lane, [&](int r, int q, int in) {
        const int at = (w * R + r) * BW + 4 * q;
        adjoint_psi<T>(psi_hx + at, pub + at, ldv(xco + 4 * q), ldv(xco + BW + 4 * q), T(-1), in);
      });
    }
    stv(row_h + w * BW + 4 * lane, hz[R - 1]);
    __syncthreads();
    // -- E~ of the values before the step: H_z(x, y) read E_x(x, y) with -dt fhy(y) and E_y(x, y)
    // with +dt fhx(x); H_z(x, y-1) read E_x(x, y) with +dt fhy(y-1); H_z(x-1, y) E_y(x, y) with
    // -dt fhx(x-1); then the slabs
    const V4<T> fhx = ldv(xco + 4 * BW + 4 * lane);
    V4<T> hp = {{T(0), T(0), T(0), T(0)}};
    if (w > 0) hp = ldv(row_h + (w - 1) * BW + 4 * lane);
#pragma unroll
    for (int r = 0; r < R; r++) {
      const T fhy = yco[8 * (w * R + r) + 4], fhyp = yco[8 * max(w * R + r - 1, 0) + 4];
      T a[4], b[4];
      if (ca) {
        const int my = wrap_any(Y0 + w * R + r, ny, I.py);
        get(ca, my, a);
        get(ca + N, my, b);
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++) {
          a[j] = any_held && cbx[r][j] == T(0) ? T(0) : T(1);
          b[j] = any_held && cby[r][j] == T(0) ? T(0) : T(1);
        }
      }
      T g[4];
#pragma unroll
      for (int j = 0; j < 4; j++) g[j] = dt * fhx.v[j] * hz[r][j];
      const T gp = __shfl_up_sync(0xffffffffu, g[3], 1);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        T ax = a[j] * ex[r][j] - dt * fhy * hz[r][j];
        T ay = b[j] * ey[r][j] + g[j];
        ax = ax + dt * fhyp * (r > 0 ? hz[r > 0 ? r - 1 : 0][j] : hp.v[j]);
        ay = ay - (j > 0 ? g[j > 0 ? j - 1 : 0] : gp);
        ex[r][j] = ax;
        ey[r][j] = ay;
      }
    }
    if (tile_slab) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        if (flags >> (4 * r) & 2) {
          const V4<T> q = ldv(pub + AREA + slots + r * BW);
#pragma unroll
          for (int j = 0; j < 4; j++) ex[r][j] = ex[r][j] - q.v[j];
        }
        if (((r > 0 ? flags >> (4 * (r > 0 ? r - 1 : 0)) : before) & 2) && w * R + r > 0 &&
            (flags >> (4 * r) & 1)) {
          const V4<T> q = ldv(pub + AREA + slots + (r - 1) * BW);
#pragma unroll
          for (int j = 0; j < 4; j++) ex[r][j] = ex[r][j] + q.v[j];
        }
        const V4<T> t = ldv(pub + slots + r * BW);
        const T tp = __shfl_up_sync(0xffffffffu, t.v[3], 1);
        if (flags >> (4 * r) & 1) {
#pragma unroll
          for (int j = 0; j < 4; j++) {
            if (inhx >> j & 1) ey[r][j] = ey[r][j] - t.v[j];
            if (j > 0 ? inhx >> (j - 1) & 1 : prevh >> 3 & 1) ey[r][j] = ey[r][j] + (j > 0 ? t.v[j > 0 ? j - 1 : 0] : tp);
          }
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
    __syncthreads();
  }

  // -- the tile's own places to the other copies
  T *eo = A.e[1 - A.cur], *ho = A.h[1 - A.cur], *peo = A.pe[1 - A.cur], *pho = A.ph[1 - A.cur];
  if (4 * lane < HALO || 4 * lane >= BW - HALO) return;
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int row = w * R + r, y = Y0 + row;
    if (row < HALO || row >= ROWS - HALO || y >= ny) continue;
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
    put(eo, ex[r]);
    put(eo + N, ey[r]);
    put(ho, hz[r]);
    if ((inhx | inex) != 0) {
      const V4<T> q = ldv(psi_hx + slots + r * BW), o = ldv(psi_ex + slots + r * BW);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int m = xb + j;
        const SlabEntry &a = I.hx[m < low_x ? 0 : 1], &b = I.ex[m < low_x ? 0 : 1];
        if (inhx >> j & 1) pho[a.psi + (long long)y * a.pw + (m - a.pf)] = q.v[j];
        if (inex >> j & 1) peo[b.psi + (long long)y * b.pw + (m - b.pf)] = o.v[j];
      }
    }
    if (flags >> (4 * r) & 6) {
      const int side = y < low_y ? 0 : 1;
      const SlabEntry &a = I.hy[side], &b = I.ey[side];
      const V4<T> q = ldv(psi_hy + slots + r * BW), o = ldv(psi_ey + slots + r * BW);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (xb + j >= nx) continue;
        if (flags >> (4 * r) & 2) pho[a.psi + (long long)(y - a.from) * I.pitch + xb + j] = q.v[j];
        if (flags >> (4 * r) & 4) peo[b.psi + (long long)(y - b.from) * I.pitch + xb + j] = o.v[j];
      }
    }
  }
}

// The segment's amounts: dJ/dF of each transform value in the owners' order at each of its steps
// (te_inject_kernel's sum over the frequencies).
template <typename T>
__global__ void te_amount_kernel(const TeInst<T> *insts, const long long *order, long long norder,
                                 const double *phase, const double *grad_sums, int steps, T *amount) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= norder * steps) return;
  const TeInst<T> &I = insts[0];
  const long long q = t % norder, m = t / norder;
  const long long v = order[q];
  const SeriesDev s = I.series[I.value_series[v]];
  const long long o = v - s.value0;
  const double *ph = phase + 2 * (m * I.nslots + s.slot0);
  double x = 0.0;
  for (int k = 0; k < s.nf; k++) {
    const double *gs = grad_sums + 2 * (s.sum0 + (long long)k * s.volume + o);
    x += gs[0] * ph[2 * k] + gs[1] * ph[2 * k + 1];
  }
  amount[t] = (T)x;
}

// dJ/dcb at each design value += E~ x curl over the segment's steps, from the last (te_grad_kernel).
template <typename T>
__global__ void te_grad_sum_kernel(long long n, const T *kept, const T *K, int steps, double *grad) {
  const long long d = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= n) return;
  double g = grad[d];
#pragma unroll 8
  for (int m = steps - 1; m >= 0; m--) g += (double)kept[m * n + d] * (double)K[m * n + d];
  grad[d] = g;
}

}  // namespace pxb
