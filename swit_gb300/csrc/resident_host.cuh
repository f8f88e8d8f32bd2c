// resident_host.cuh -- split, shared memory and launches of the resident time
// loops (kernels_resident.cuh).  Included by engine.cu only.
#pragma once

// One direction's launch: the kernel instance (columns per thread tile, threads
// it is compiled for), its split and the shots of one launch.
struct ResLoop {
  bool ok = false;
  int tx = 0, maxt = 0;
  int shots = 0;  // per launch, at most
  double us = 0.0;  // estimated microseconds per time step of all shots
  swit::ResPlan r{};
};

namespace {

using ResFwdFn = void (*)(Grid<float>, ResPlan, Sources, Receivers, const float*, float*, float*, float*, float*,
                          float*, float4*, int, int, int);
using ResBwdFn = void (*)(Grid<float>, ResPlan, Sources, Receivers, const float*, const float*, float*, float*, float*,
                          float*, float*, float*, float*, float*, float*, const float*, int, int, int);

using ResXadjFn = void (*)(Grid<float>, ResPlan, Sources, Receivers, XAdj<float>, int, int, int);

enum ResKind { kResLoopFwd, kResLoopBwd, kResLoopXadj };

struct ResInst {
  int tx, maxt;
  ResFwdFn f, fd;  // forward; the one that keeps D of every step for the exact adjoint
  ResBwdFn b;
  ResXadjFn x;
  const void* any() const { return f ? (const void*)f : (b ? (const void*)b : (const void*)x); }
};
inline const ResInst* res_instances(ResKind kind, int& n) {
  static const ResInst F[] = {{4, 512, k_fwd_res<4, 512, false>, k_fwd_res<4, 512, true>, nullptr, nullptr},
                              {8, 384, k_fwd_res<8, 384, false>, k_fwd_res<8, 384, true>, nullptr, nullptr}};
  static const ResInst B[] = {{4, 512, nullptr, nullptr, k_bwd_res<4, 512>, nullptr},
                              {4, 384, nullptr, nullptr, k_bwd_res<4, 384>, nullptr}};
  static const ResInst X[] = {{4, 384, nullptr, nullptr, nullptr, k_xadj_res<4, 384>}};
  n = kind == kResLoopXadj ? 1 : 2;
  return kind == kResLoopFwd ? F : (kind == kResLoopBwd ? B : X);
}

// Split of a shot into bands of at most `tiles` column tiles, with the shared memory of a block.
inline ResPlan res_plan(const swit_engine* e, ResKind kind, int tx, int tiles) {
  const bool bwd = kind == kResLoopBwd;
  ResPlan r{};
  r.negz = -0.0f;
  r.nt_tiles = (e->NX + tx - 1) / tx;
  r.C = (r.nt_tiles + tiles - 1) / tiles;
  const int widest = (r.nt_tiles + r.C - 1) / r.C;
  r.W = widest * tx;
  r.m0 = e->L / tx;
  r.m1 = (e->L + e->nx - 1) / tx;
  // a band reaches the strip columns of both sides only if it is nearly as wide as the interior; with 4 columns
  // per thread there is room for both, and a constant index (481x141: 14.1 against 14.3 us per step)
  r.nside = tx == 4 || r.W + 8 >= e->nx ? 6 : 3;
  if (bwd) {
    r.kr = (e->fs - 2 + 3) / 4;  // rows from fs-1-4 kr <= 1
    r.nq = (e->NZ - (e->fs - 1 - 4 * r.kr) + 1 + 3) / 4;
    r.nqr = (e->nz + 1 + 3) / 4;  // rows fs-1 .. fs+nz-1
    // the widest reconstruction part of a band
    int nr = 0;
    const int per = r.nt_tiles / r.C, rem = r.nt_tiles % r.C;
    for (int b = 0; b < r.C; ++b) {
      const int t0 = b * per + std::min(b, rem), n = per + (b < rem ? 1 : 0);
      nr = std::max(nr, std::min(t0 + n - 1, r.m1) - std::max(t0, r.m0) + 1);
    }
    r.nR = round_up(nr * r.nqr, 32);
  } else {
    r.nq = (e->NZ - (e->fs - 1) + 1 + 3) / 4;  // rows fs-1 .. NZ
  }
  r.nA = round_up(widest * r.nq, 32);
  r.ns = (widest + 2) * r.nq;
  const int iz0 = e->fs - 1 - 4 * r.kr;  // first row
  r.jz = (e->L + e->nz - iz0) & 3;
  // receiver entries of the fullest band of any shot
  int cap = 4;
  const int per = r.nt_tiles / r.C, rem = r.nt_tiles % r.C;
  for (int s = 0; s < e->ns; ++s) {
    const int* cp = &e->colptr[(size_t)s * (e->NX + 2)];
    for (int b = 0; b < r.C; ++b) {
      const int t0 = b * per + std::min(b, rem), n = per + (b < rem ? 1 : 0);
      const int x0 = 1 + t0 * tx, x1 = std::min(e->NX, (t0 + n) * tx);
      // a tile's entries start at a multiple of 4: at most 3 unused for every tile that has any
      const int n_ent = cp[x1 + 1] - cp[x0];
      cap = std::max(cap, n_ent + 3 * std::min(n_ent, n * r.nq));
    }
  }
  r.ent_cap = round_up(cap, 4);
  int o = 0;
  auto take = [&](int float4s) {
    const int at = o;
    o += float4s;
    return at;
  };
  r.oC = take((2 * tx + 1) * (r.nA + r.nR));
  r.oE = take(kEdge * r.ns);
  r.oG = take(kEdge * r.nq);
  r.oZ = take(((r.nA + r.nR) / 32 + 2) * 6 * tx / 4);
  r.oR = take(kRow * r.nq);
  r.oX = take((r.W + 1) / 2);
  if (bwd) {
    r.oER = take(kEdge * r.ns);
    r.oGR = take(kEdge * r.nq);
    r.oR1 = take(kRow * r.nq);
    r.oD = take((tx + 1) * r.ns);
    r.box = 2 * r.W + 6 * r.nqr + r.ent_cap / 4;
    r.oBox = take(2 * r.box);
    r.oEnt = take(1 + r.ent_cap / 2);  // counters, receivers, codes
    r.oList = take((6 * r.W + 6 * e->nz + r.ent_cap + 1) / 2);
  } else if (kind == kResLoopXadj) {
    r.oGR = take(kRow * r.nq);  // lu of the ghost columns
    r.oD = take(tx * r.nA);
    r.box = r.ent_cap / 4;
    r.oBox = take(2 * r.box);
    r.oEnt = take(1 + r.ent_cap / 2);
  } else {
    r.oStage = take(6 * r.W);
    r.oS = take(r.nside * r.nq);
    r.oEnt = take(1 + (2 * r.ent_cap + r.W + 3) / 4);  // counters, receivers, codes, columns
    r.oList = take((10 * r.W + r.nside * e->nz + 1) / 2);
  }
  r.smem = 16 * o;
  return r;
}

// Estimated microseconds of one time step of a launch whose fullest SM holds `bpsm` blocks, fitted to
// measured steps (GB300, 11 grids of 60x40 to 700x40 and 401x151 in bands of 1 to 10 column tiles, 1 to 15
// warps per block): a fixed part, the dependent chain of a step (updates, barriers, halo), and a part by the
// warps that share the SM.  Bands of one column tile exchange both edges in the same threads, and in bands of
// two every thread has an edge (forward of 101x51: 2.00 us with one tile, 2.06 with two, 1.64 with three);
// a shot in one band exchanges nothing.  The reverse loop's 128-register instance pays for its spills; the
// forward's with 8 columns per thread holds half as many points again per SM and is taken where that saves
// launches (10 shots 801x301: 9.7 against 11.0 us per step in 2 and 4 launches; 49 shots 481x141: 17.9
// against 14.2) or nothing else fits (2001x601).
inline double res_step_us(const ResPlan& r, ResKind kind, int maxt, int bpsm, int tiles) {
  const double warps = bpsm * ((r.nA + r.nR) / 32);
  const double edge[3][2] = {{0.40, 0.33}, {0.50, 0.20}, {0.50, 0.37}};
  const double t = kind == kResLoopFwd   ? 1.5 + (maxt < 512 ? 0.28 : 0.09) * warps
                   : kind == kResLoopBwd ? 1.95 + (maxt > 384 ? 0.23 : 0.095) * warps
                                         : 1.85 + 0.11 * warps;
  return t + (r.C == 1 ? -0.3 : (tiles <= 2 ? edge[kind][tiles - 1] : 0.0));
}

// The fastest split by estimate among those whose blocks are co-resident.
inline void res_choose(const swit_engine* e, ResKind kind, ResLoop& out) {
  int dev = 0, sms = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return;
  int want = 0;  // column tiles per band instead of the estimate's choice, e.g. to test a split
  if (const char* v = std::getenv(kind != kResLoopFwd ? "SWIT_RES_BWD_TILES" : "SWIT_RES_FWD_TILES")) want = std::atoi(v);
  int cols = 0;  // columns per thread, likewise
  if (const char* v = std::getenv("SWIT_RES_FWD_COLS")) cols = kind == kResLoopFwd ? std::atoi(v) : 0;
  int ninst = 0;
  const ResInst* I = res_instances(kind, ninst);
  double best = 0.0;
  for (int i = 0; i < ninst; ++i) {
    if (cols && I[i].tx != cols) continue;
    const int all = (e->NX + I[i].tx - 1) / I[i].tx;
    int lastC = -1;
    for (int tiles = 1; tiles <= all; ++tiles) {
      if (want && tiles != std::min(want, all)) continue;
      ResPlan r = res_plan(e, kind, I[i].tx, tiles);
      if (r.C == lastC) continue;
      lastC = r.C;
      if (r.nA + r.nR > I[i].maxt) break;
      if (r.smem > optin) continue;
      const void* f = e->exact && kind == kResLoopFwd ? (const void*)I[i].fd : I[i].any();
      int occ = 0;
      if (cudaFuncSetAttribute(I[i].any(), cudaFuncAttributeMaxDynamicSharedMemorySize, optin) != cudaSuccess ||
          cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin) != cudaSuccess ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, f, r.nA + r.nR, r.smem) != cudaSuccess) {
        cudaGetLastError();
        continue;
      }
      const int fit = occ * sms / r.C;
      if (fit < 1) continue;
      const int waves = (e->ns + fit - 1) / fit;
      const int shots = (e->ns + waves - 1) / waves;
      const int bpsm = (shots * r.C + sms - 1) / sms;
      const double t = waves * res_step_us(r, kind, I[i].maxt, bpsm, (r.nt_tiles + r.C - 1) / r.C);
      if (!out.ok || t < best) {
        best = t;
        out.ok = true;
        out.tx = I[i].tx;
        out.maxt = I[i].maxt;
        out.shots = shots;
        out.us = t;
        out.r = r;
      }
    }
  }
}

// Packets of a full launch, and the stop word's behind them: with it in front, 16 or 128 bytes into the
// allocation, some loops took 7 to 14 % longer (forward step of 2 shots 172x52 1.80 against 1.58 us).
inline size_t res_halo_packets(const ResLoop& l) {
  return l.ok ? (size_t)l.shots * l.r.C * 2 * 2 * 2 * 4 * l.r.nq : 0;
}

inline const ResInst& res_inst(ResKind kind, const ResLoop& l) {
  int n = 0;
  const ResInst* I = res_instances(kind, n);
  for (int i = 0; i < n; ++i)
    if (I[i].tx == l.tx && I[i].maxt == l.maxt) return I[i];
  return I[0];
}

// Launch configuration of `shots` shots; the packets' tags and the stop word start from zero.
inline cudaLaunchConfig_t res_config(const ResLoop& l, int shots, cudaStream_t st, cudaLaunchAttribute* at) {
  cudaMemsetAsync(l.r.halo, 0, (l.r.stop + 1) * sizeof(uint4), st);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(shots * l.r.C);
  cfg.blockDim = dim3(l.r.nA + l.r.nR);
  cfg.dynamicSmemBytes = l.r.smem;
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

inline cudaEvent_t res_event() {
  cudaEvent_t x = nullptr;
  cudaEventCreate(&x);
  return x;
}

// Steps lo .. hi of shots s0 .. s0+nb-1, one launch after another (a launch fills the device); ev: events
// around every launch, for profiling.
inline void res_forward(swit_engine* e, const ResLoop& l, bool store, int s0, int nb, cudaStream_t st, int lo, int hi,
                        std::vector<cudaEvent_t>* ev = nullptr) {
  if (lo > hi) return;
  const bool save = store && e->exact;  // the strip buffer holds D
  const ResFwdFn f = save ? res_inst(kResLoopFwd, l).fd : res_inst(kResLoopFwd, l).f;
  for (int s = s0; s < s0 + nb; s += l.shots) {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = res_config(l, std::min(l.shots, s0 + nb - s), st, at);
    if (ev) cudaEventRecord(ev->emplace_back(res_event()), st);
    cudaLaunchKernelEx(&cfg, f, make_grid<float>(e), l.r, make_src(e), make_rec(e), (const float*)e->src,
                       (float*)e->p, (float*)e->u, (float*)e->w, (float*)e->seis_t,
                       store && !save ? (float*)e->strips : (float*)nullptr,
                       save ? (float4*)e->strips : (float4*)nullptr, lo, hi, s);
    if (ev) cudaEventRecord(ev->emplace_back(res_event()), st);
  }
}

inline void res_backward(swit_engine* e, const ResLoop& l, int s0, int nb, cudaStream_t st, int hi, int lo,
                         std::vector<cudaEvent_t>* ev = nullptr) {
  if (lo > hi) return;
  const ResBwdFn f = res_inst(kResLoopBwd, l).b;
  for (int s = s0; s < s0 + nb; s += l.shots) {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = res_config(l, std::min(l.shots, s0 + nb - s), st, at);
    if (ev) cudaEventRecord(ev->emplace_back(res_event()), st);
    cudaLaunchKernelEx(&cfg, f, make_grid<float>(e), l.r, make_src(e), make_rec(e), (const float*)e->src,
                       (const float*)e->adj_t, (float*)e->pb, (float*)e->ub, (float*)e->wb, (float*)e->pe,
                       (float*)e->ue, (float*)e->we, (float*)e->dg, (float*)e->dfw, (float*)e->dbk,
                       (const float*)e->strips, hi, lo, s);
    if (ev) cudaEventRecord(ev->emplace_back(res_event()), st);
  }
}

inline void res_xadj(swit_engine* e, const ResLoop& l, const XAdj<float>& x, int s0, int nb, cudaStream_t st, int hi,
                     int lo) {
  if (lo > hi) return;
  const ResXadjFn f = res_inst(kResLoopXadj, l).x;
  for (int s = s0; s < s0 + nb; s += l.shots) {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = res_config(l, std::min(l.shots, s0 + nb - s), st, at);
    cudaLaunchKernelEx(&cfg, f, make_grid<float>(e), l.r, make_src(e), make_rec(e), x, hi, lo, s);
  }
}

}  // namespace
