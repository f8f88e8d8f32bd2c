// kernels_resident_exact.cuh -- resident reverse loop of the exact discrete
// adjoint (FP32, pressure receivers): the recursion of kernels_exact.cuh with
// lp, lu, lw and the sum gA in registers, on the tiles, bands and halos of
// kernels_resident.cuh.
//
// The transposed stencils read products coefficient * field, so those are what
// moves: B lu and B lw between the phases, A lp after the pressure phase, and
// across a band edge three columns of A lp, from which the edge threads
// recompute the ghost columns' lu.  lp is zero outside S1's range and lw outside
// S4's rows, so no product of the sums needs a test: what the transposes leave
// out adds c * 0.  The mirror row's m belongs to the thread that holds rows F and
// F+1; lw~ = lw + m is formed when m is, so both gathers read it, except after a
// launch's last step, which leaves lw and m apart in memory as the step kernels
// do.
#pragma once
#include "kernels_exact.cuh"
#include "kernels_resident.cuh"

namespace swit {

__device__ __forceinline__ void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// lp from B lu (x-neighbours in the edge arrays) and B lw; gA -= lp D.  p comes scaled, with the adjoint
// sources added.
template <int TX>
__device__ __forceinline__ void xtile_p(const Tile<TX>& T, const ResPlan& r, float (&p)[TX][4], const float (&u)[TX][4],
                                        const float (&w)[TX][4], float (&gA)[TX][4], float c1, float c2) {
  const int lane = threadIdx.x & 31;
  float um2[4], um1[4], up1[4], e1[TX], e2[TX], e6[TX], bu[TX][4];
  lds4(T.e - kEdge * r.nq + 3, um2);
  lds4(T.e - kEdge * r.nq + 4, um1);
  lds4(T.e + kEdge * r.nq + 5, up1);
  zrow_get<TX>(r, -1, 3, e1);
  zrow_get<TX>(r, -1, 4, e2);
  zrow_get<TX>(r, 1, 5, e6);
  float bw[TX][4];
#pragma unroll
  for (int c = 0; c < TX; ++c) {
    float b[4];
    lds4(r.oC + (2 * TX + 1) * threadIdx.x + TX + c, b);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      bu[c][j] = b[j] * u[c][j];
      bw[c][j] = b[j] * w[c][j];
    }
  }
#pragma unroll
  for (int c = 0; c < TX; ++c) {
    float z[7], D[4];  // B lw at rows -2 .. 4
    lds4(r.oD + c * r.nA + threadIdx.x, D);
    z[0] = __shfl_up_sync(0xffffffffu, bw[c][2], 1);
    z[1] = __shfl_up_sync(0xffffffffu, bw[c][3], 1);
    z[6] = __shfl_down_sync(0xffffffffu, bw[c][0], 1);
    z[0] = lane == 0 ? e2[c] : z[0];
    z[1] = lane == 0 ? e1[c] : z[1];
    z[6] = lane == 31 ? e6[c] : z[6];
#pragma unroll
    for (int j = 0; j < 4; ++j) z[2 + j] = bw[c][j];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float l1 = c >= 1 ? bu[c >= 1 ? c - 1 : 0][j] : um1[j];
      const float l2 = c >= 2 ? bu[c >= 2 ? c - 2 : 0][j] : (c == 1 ? um1[j] : um2[j]);
      const float r1 = c + 1 < TX ? bu[c + 1 < TX ? c + 1 : 0][j] : up1[j];
      float a = p[c][j];
      a = a - c1 * l1;
      a = a + c1 * bu[c][j];
      a = a - c2 * l2;
      a = a + c2 * r1;
      a = a - c1 * z[j + 1];
      a = a + c1 * z[j + 2];
      a = a - c2 * z[j];
      sub_if(bit_at(T.f, kP + j), p[c][j], a, -(c2 * z[j + 3]));
      if (j == 2) sub_if(T.f & kTopFs, p[c][j], p[c][j], c2 * z[j + 1]);  // the mirror of S3
      gA[c][j] = gA[c][j] - p[c][j] * D[j];
    }
  }
}

// lw from A lp.
template <int TX>
__device__ __forceinline__ void xtile_w(const Tile<TX>& T, const ResPlan& r, int tt0, const float (&al)[TX][4],
                                        float (&w)[TX][4], float c1, float c2) {
  const int lane = threadIdx.x & 31;
  float fz[4], e0[TX], e5[TX], e6[TX];
  lds4(T.rf + 1, fz);
  zrow_get<TX>(r, -1, 0, e0);
  zrow_get<TX>(r, 1, 1, e5);
  zrow_get<TX>(r, 1, 2, e6);
#pragma unroll
  for (int c = 0; c < TX; ++c) {
    const float fx = col_factor<TX>(T, r, tt0, c).x;
    float z[7];  // A lp at rows -1 .. 5
    z[0] = __shfl_up_sync(0xffffffffu, al[c][3], 1);
    z[5] = __shfl_down_sync(0xffffffffu, al[c][0], 1);
    z[6] = __shfl_down_sync(0xffffffffu, al[c][1], 1);
    z[0] = lane == 0 ? e0[c] : z[0];
    z[5] = lane == 31 ? e5[c] : z[5];
    z[6] = lane == 31 ? e6[c] : z[6];
#pragma unroll
    for (int j = 0; j < 4; ++j) z[1 + j] = al[c][j];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float a = fminf(fx, fz[j]) * w[c][j];
      a = a - c1 * z[j + 1];
      a = a + c1 * z[j + 2];
      a = a - c2 * z[j];
      sub_if(bit_at(T.f, kW + j), w[c][j], a, -(c2 * z[j + 3]));
    }
  }
}

// lu from A lp (x-neighbours in the edge arrays).
template <int TX>
__device__ __forceinline__ void xtile_u(const Tile<TX>& T, const ResPlan& r, int tt0, const float (&al)[TX][4],
                                        float (&u)[TX][4], float c1, float c2) {
  float pm1[4], pp1[4], pp2[4], fz[4];
  lds4(T.rf, fz);
  lds4(T.e - kEdge * r.nq + 2, pm1);
  lds4(T.e + kEdge * r.nq, pp1);
  lds4(T.e + kEdge * r.nq + 1, pp2);
#pragma unroll
  for (int c = 0; c < TX; ++c) {
    const float fx = col_factor<TX>(T, r, tt0, c).y;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float l1 = c >= 1 ? al[c >= 1 ? c - 1 : 0][j] : pm1[j];
      const float r1 = c + 1 < TX ? al[c + 1 < TX ? c + 1 : 0][j] : pp1[j];
      const float r2 = c + 2 < TX ? al[c + 2 < TX ? c + 2 : 0][j] : (c + 1 < TX ? pp1[j] : pp2[j]);
      float a = fminf(fx, fz[j]) * u[c][j];
      a = a - c1 * al[c][j];
      a = a + c1 * r1;
      a = a - c2 * l1;
      a = a + c2 * r2;
      u[c][j] = a;
    }
  }
}

// Edges of B lu and B lw within the band.
template <int TX>
__device__ __forceinline__ void xpublish_uw(const Tile<TX>& T, const ResPlan& r, const float (&u)[TX][4],
                                            const float (&w)[TX][4]) {
  float b[TX][4], v[TX][4];
#pragma unroll
  for (int c = 0; c < TX; ++c) lds4(r.oC + (2 * TX + 1) * threadIdx.x + TX + c, b[c]);
#pragma unroll
  for (int c = 0; c < TX; ++c)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[c][j] = b[c][j] * w[c][j];
      b[c][j] = b[c][j] * u[c][j];
    }
  publish_uw<TX>(T, r, b, v);
}

// Ghost lu of one column (state) and its product with B (slot).
__device__ __forceinline__ void ghost_xu(int state, int slot, int coef, int fac, float c1, float c2, const float* l1,
                                         const float* a0, const float* r1, const float* r2) {
  float u[4], b[4], f[4], v[4];
  lds4(state, u);
  lds4(coef, b);
  lds4(fac, f);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a = f[j] * u[j];
    a = a - c1 * a0[j];
    a = a + c1 * r1[j];
    a = a - c2 * l1[j];
    a = a + c2 * r2[j];
    u[j] = a;
    v[j] = b[j] * a;
  }
  res_sm[state] = mk4(u);
  res_sm[slot] = mk4(v);
}

// As edge_recv, of A lp.
template <int TX>
__device__ __forceinline__ void xedge_recv(const Tile<TX>& T, const ResPlan& r, unsigned gu, bool& dead,
                                           const float (&al)[TX][4], unsigned tag, float c1, float c2) {
  if (!(T.f & (kLeft | kRight))) return;
  const int nq = r.nq, k = opaque(T.k), g = r.oG + kEdge * k, st = r.oGR + kRow * k;
  const int e = opaque(T.e), el = e - kEdge * nq, er = e + kEdge * nq;
  Halo h;
  if (T.f & kLeft) {  // columns ix0-3, ix0-2, ix0-1
    halo_wait(halo_from<TX>(T, r, 0, tag, true), tag, r, dead, h);
    res_sm[el + 2] = mk4(h.c);
    if (gu & 1u) ghost_xu(st, el + 3, g, g + 3, c1, c2, h.a, h.b, h.c, al[0]);
    if (gu & 2u) ghost_xu(st + 1, el + 4, g + 1, g + 4, c1, c2, h.b, h.c, al[0], al[1]);
  }
  if (T.f & kRight) {  // columns ix0+TX .. ix0+TX+2
    halo_wait(halo_from<TX>(T, r, 0, tag, false), tag, r, dead, h);
    res_sm[er] = mk4(h.a);
    res_sm[er + 1] = mk4(h.b);
    if (gu & 4u) ghost_xu(st + 2, er + 5, g + 2, g + 5, c1, c2, al[TX - 1], h.a, h.b, h.c);
  }
}

// Steps it1 .. it0 of shots shot0 + block / C.  D of a step: float4 [column][row tile], as the
// forward loop stored it (whatever its columns per thread); a thread fetches its own a step ahead, 16 bytes
// per column, consecutive in a warp.  384 threads of 168 registers, for four 16-value arrays.
//
// Bound by the dependent chain of a step, and on a full device by issue.  10 shots 241x121, per step, against
// the kernels of kernels_exact.cuh: forward keeping D 1.95, reverse 2.59 us, together 18.8 -> 4.5 us (gradient
// of 1200 steps 22.5 -> 5.3 ms); 20 shots 481x141: 5.7 and 9.9 us.
template <int TX, int MAXT>
__global__ void __launch_bounds__(MAXT, 1)
    k_xadj_res(const __grid_constant__ Grid<float> g, const __grid_constant__ ResPlan r,
               const __grid_constant__ Sources src, const __grid_constant__ Receivers rec, XAdj<float> x, int it1, int it0,
               int shot0) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int b = blockIdx.x % r.C, s = shot0 + blockIdx.x / r.C;
  const int per = r.nt_tiles / r.C, rem = r.nt_tiles % r.C;
  const int tt0 = b * per + min(b, rem), n = per + (b < rem ? 1 : 0);
  const int fs = g.fs, NX = g.NX, NZ = g.NZ, nq = r.nq;
  const float c1 = g.c1, c2 = g.c2;
  int* s_cnt = reinterpret_cast<int*>(res_sm + r.oEnt);  // receiver entries
  int* s_ig = s_cnt + 4;
  int* s_code = s_ig + r.ent_cap;

  for (int i = tid; i < r.smem / 16; i += nthr) res_sm[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  factor_setup(g, r, tt0 * TX + 1);
  __syncthreads();
  Tile<TX> T;
  tile_setup<TX, kResFwd>(T, g, r, tid, tt0, n, 0, nq, 0, b > 0, b < r.C - 1);
  const size_t off = (size_t)s * g.FSZ;
  const bool live = T.f & kLive;
  const int iz0 = row0<TX>(T, r, fs);
  float p[TX][4], u[TX][4], w[TX][4], gA[TX][4], m[TX];
  tile_load<TX>(g.A, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, p);
  tile_load<TX>(g.B, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, u);
#pragma unroll
  for (int c = 0; c < TX; ++c) {
    res_sm[r.oC + (2 * TX + 1) * tid + c] = mk4(p[c]);
    res_sm[r.oC + (2 * TX + 1) * tid + TX + c] = mk4(u[c]);
  }
  tile_load<TX>(x.lp + off, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, p);
  tile_load<TX>(x.lu + off, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, u);
  tile_load<TX>(x.lw + off, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, w);
  tile_load<TX>(x.gA + off, g.LD, T.ix0, iz0, live, fs + 1, NZ - 2, 3, NX - 2, gA);
#pragma unroll
  for (int c = 0; c < TX; ++c) {
    m[c] = (T.f & kTopFs) && T.ix0 + c <= NX ? x.m[((size_t)s * 2 + (it1 & 1)) * NX + T.ix0 + c - 1] : 0.f;
    add_if(T.f & kTopFs, w[c][1], m[c]);
  }
  const unsigned gu = ghost_setup<TX, kResFwd>(T, g, r, x.lu + off);
#pragma unroll
  for (int q = 0; q < 3; ++q)
    if (T.f & (q < 2 ? kLeft : kRight)) {
      const int slot = q < 2 ? T.e - kEdge * nq + 3 + q : T.e + kEdge * nq + 5;
      float v[4], a[4];
      lds4(slot, v);
      lds4(r.oG + kEdge * T.k + q, a);
      res_sm[r.oGR + kRow * T.k + q] = mk4(v);
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = a[j] * v[j];
      res_sm[slot] = mk4(v);
    }
  const RecTile R = rec_setup<TX>(T, g, r, rec, s, s_cnt, s_ig, s_code);
  int isrc = -1;  // the source point, where S1 updates it
  {
    const int cx = src.isx[s] - T.ix0, jz = src.isz[s] - iz0;
    if (live && cx >= 0 && cx < TX && jz >= 0 && jz < 4 && bit_at(T.f, kP + jz) && src.isx[s] >= 3 &&
        src.isx[s] <= NX - 2)
      isrc = 4 * cx + jz;
  }
  xpublish_uw<TX>(T, r, u, w);
  __syncthreads();
  const int nrec = s_cnt[0];
  const float4* dsave = reinterpret_cast<const float4*>(x.dsave);
  const int dat = (T.ix0 - 1) * nq + T.k;
  // inputs of a step: its adjoint sources (entries without a receiver, the padding of a tile's, repeat
  // receiver 0: never read) and D
  auto prefetch = [&](int it) {
    const size_t so = opaque(s);
    const float* at = x.adj_t + (so * g.nt + (it - 1)) * g.ngmax;
    float* box = res_smf() + 4 * (r.oBox + (it & 1) * r.box);
    for (int i = tid; i < nrec; i += nthr) cp4(box + i, at + s_ig[i]);
    const float4* d = dsave + (so * g.snt + (it - g.sit0)) * (g.SL / 4) + dat;
    if (T.f & kLive)
#pragma unroll
      for (int c = 0; c < TX; ++c) cp16(res_sm + r.oD + c * r.nA + tid, d + c * nq);
  };
  prefetch(it1);
  cp_wait();
  if (__any_sync(0xffffffffu, (T.f & (kLeft | kRight | kEnds)) || isrc >= 0 || R.n > 0)) T.f |= kRare;
  __syncthreads();
  bool dead = false;

  for (int it = it1; it >= it0; --it) {
    // ---- pressure phase
    {
      float fz[4];
      lds4(T.rf, fz);
#pragma unroll
      for (int c = 0; c < TX; ++c) {
        const float fx = col_factor<TX>(T, r, tt0, c).x;
#pragma unroll
        for (int j = 0; j < 4; ++j) p[c][j] = fminf(fx, fz[j]) * p[c][j];
      }
    }
    if ((T.f & kRare) && R.n) {
      const int val = r.oBox + (it & 1) * r.box;
      if (R.row >= 0) {
        if (bit_at(T.f, kP + R.row)) rec_add_line<TX, false>(R, p, val, 1.f);
      } else {
#pragma unroll 1
        for (int i = 0; i < R.n; ++i) {
          const int code = s_code[R.base + i];
          if (bit_at(T.f, kP + (code & 3))) add_at<TX, false>(p, code, res_smf()[4 * val + R.base + i]);
        }
      }
    }
    __syncwarp();
    xtile_p<TX>(T, r, p, u, w, gA, c1, c2);
    if (T.f & kRare) {
      if (isrc >= 0) {
        float a = 0.f;
#pragma unroll
        for (int c = 0; c < TX; ++c)
#pragma unroll
          for (int j = 0; j < 4; ++j) a = isrc == 4 * c + j ? p[c][j] : a;
        x.gsrc[(size_t)s * g.nt + (it - 1)] = g.dt * a;
      }
      if (T.f & kEnds) zero_cols<TX>(T.ix0, p, 3, NX - 2);
    }
    float al[TX][4];
#pragma unroll
    for (int c = 0; c < TX; ++c) {
      lds4(r.oC + (2 * TX + 1) * threadIdx.x + c, al[c]);
#pragma unroll
      for (int j = 0; j < 4; ++j) al[c][j] = al[c][j] * p[c][j];
    }
    if (T.f & kRare) edge_send<TX>(T, r, 0, al, (unsigned)it);
    publish_p<TX>(T, r, al);
    if (it > it0) prefetch(it - 1);  // the thread's D is read, the other box is free
    __syncthreads();
    // ---- velocity phase
    xtile_w<TX>(T, r, tt0, al, w, c1, c2);
    if (T.f & kRare) xedge_recv<TX>(T, r, gu, dead, al, (unsigned)it, c1, c2);
    __syncwarp();
    xtile_u<TX>(T, r, tt0, al, u, c1, c2);
    if ((T.f & kRare) && (T.f & kEnds)) zero_cols<TX>(T.ix0, u, 2, NX - 2);
#pragma unroll
    for (int c = 0; c < TX; ++c) {
      m[c] = c2 * al[c][2];
      add_if(it > it0 ? T.f & kTopFs : 0u, w[c][1], m[c]);
    }
    if (it > it0) {
      xpublish_uw<TX>(T, r, u, w);
      cp_wait();
      __syncthreads();
    }
  }
  tile_store<TX>(x.lp + off, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, p);
  tile_store<TX>(x.lu + off, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, u);
  tile_store<TX>(x.lw + off, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, w);
  tile_store<TX>(x.gA + off, g.LD, T.ix0, iz0, live, fs + 1, NZ - 2, 3, NX - 2, gA);
  if (T.f & kTopFs) {
#pragma unroll
    for (int c = 0; c < TX; ++c)
      if (T.ix0 + c <= NX) x.m[((size_t)s * 2 + ((it0 - 1) & 1)) * NX + T.ix0 + c - 1] = m[c];
  }
}

}  // namespace swit
