// resident_host.cuh -- split, shared memory and launches of the resident time
// loops (kernels_resident.cuh).  Included by engine.cu only.
#pragma once

// One direction's launch: the kernel instance (columns per thread tile, threads
// it is compiled for), its split and the shots of one launch.
struct ResLoop {
  bool ok = false;
  bool alone = false;  // runs where the engine runs by itself
  int tx = 0, maxt = 0;
  int shots = 0;  // per launch, at most
  double us = 0.0;  // estimated microseconds per time step of all shots, launches included
  swit::ResPlan r{};
};

namespace {

using ResFwdFn = void (*)(Grid<float>, ResPlan, Sources, Receivers, const float*, float*, float*, float*, float*,
                          float*, float4*, int, int, int);
using ResBwdFn = void (*)(Grid<float>, ResPlan, Sources, Receivers, const float*, const float*, float*, float*, float*,
                          float*, float*, float*, float*, float*, float*, const float*, int, int, int);

using ResXadjFn = void (*)(Grid<float>, ResPlan, Sources, Receivers, XAdj<float>, int, int, int);

// A saving forward keeps the strips, or the divergence for the exact adjoint.
enum ResKind { kResLoopFwd, kResLoopSave, kResLoopBwd, kResLoopXadj };

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
  return kind <= kResLoopSave ? F : (kind == kResLoopBwd ? B : X);
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
  // per thread there is room for both, and a constant index
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

// Estimated microseconds of one time step of a launch whose fullest SM holds `bpsm` blocks: the dependent chain
// of a step (updates, barriers, halo), a part for every warp of the SM and one for every warp of a scheduler, by
// instance and by how a shot is split: one band, which exchanges nothing, and bands of one tile (both edges in
// the same threads), of two (every thread has an edge) and of more.  Fitted to 10,400 measured loops (GB300,
// 1,400 problems of 61x41 to 2000x1000, every width of band): 7 % rms.  E.g.
// forward of 49 shots 481x141 in 5 launches (15 warps) 12.4 estimated and measured, saving 14.6 and 14.8,
// reverse in 13 launches 35.3 and 35.5; forward of one shot 2001x601 (8 columns, 133 bands of two tiles, 11
// warps) 5.2 and 5.2, saving 5.9 and 5.7.
inline double res_step_us(const ResPlan& r, ResKind kind, bool exact, int tx, int maxt, int bpsm) {
  struct Cost {
    double a, warp, sched, least;
  };
  static const Cost
      fwd4[4] = {{0.52, 0.080, 0.110, 0.0}, {1.61, 0.046, 0.174, 0.0}, {1.53, 0.045, 0.172, 0.0}, {1.25, 0.034, 0.182, 0.0}},
      fwd8[4] = {{1.40, 0.050, 0.500, 0.0}, {2.15, 0.335, 0.000, 3.2}, {0.95, 0.390, 0.000, 3.4}, {1.60, 0.130, 0.370, 2.9}},
      save4[4] = {{1.20, 0.090, 0.110, 0.0}, {1.95, 0.040, 0.230, 0.0}, {1.86, 0.050, 0.190, 0.0}, {1.56, 0.047, 0.164, 0.0}},
      save8[4] = {{1.47, 0.200, 0.310, 0.0}, {3.00, 0.335, 0.000, 4.0}, {1.75, 0.380, 0.000, 4.1}, {2.60, 0.150, 0.180, 3.6}},
      bwd384[4] = {{1.60, 0.057, 0.114, 0.0}, {2.19, 0.120, 0.069, 0.0}, {1.64, 0.087, 0.112, 0.0}, {1.69, 0.057, 0.114, 0.0}},
      bwd512[4] = {{3.80, 0.088, 0.000, 0.0}, {3.80, 0.088, 0.000, 0.0}, {3.80, 0.088, 0.000, 0.0}, {3.80, 0.088, 0.000, 0.0}},
      xadj[4] = {{1.50, 0.014, 0.257, 0.0}, {2.37, 0.014, 0.286, 0.0}, {2.41, 0.031, 0.158, 0.0}, {1.93, 0.014, 0.257, 0.0}};
  const bool strips = kind == kResLoopSave && !exact;  // keeping D costs the forward next to nothing
  const Cost* c = kind == kResLoopXadj  ? xadj
                  : kind == kResLoopBwd ? (maxt > 384 ? bwd512 : bwd384)  // 512 threads: 128 registers, spills
                  : tx == 8             ? (strips ? save8 : fwd8)
                                        : (strips ? save4 : fwd4);
  c += r.C == 1 ? 0 : std::min((r.nt_tiles + r.C - 1) / r.C, 3);
  const int warps = bpsm * ((r.nA + r.nR) / 32);
  const double t = std::max(c->least, c->a + c->warp * warps + c->sched * ((warps + 3) / 4));
  return tx == 8 && bpsm > 1 ? 1.1 * t : t;
}
constexpr double kResLaunchUs = 20.0;  // a launch's memset, state in and out, tables

// Estimated microseconds of one time step of all shots on the vec kernels, in the engine's batches and
// branches: per launch of a branch the chain of its two kernels, per point the throughput, less of it where the
// state in flight outgrows its share of L2.  Fitted to the loops of 425 engines, 61x41 to 2001x2337: 6 to
// 8 % rms.  E.g. forward of 1 and 3 shots 2001x601 9.0 and 17.9 estimated, 8.5 and 19.2 measured; 23 shots
// 587x238 23.4 and 24.9, reverse 50.9 and 51.1.
inline double vec_step_us(const swit_engine* e, ResKind kind) {
  const bool fwd = kind <= kResLoopSave, xadj = kind == kResLoopXadj;
  const double pml = 1e-6 * e->NX * e->NZ, inner = 1e-6 * e->nx * e->nz;
  const double pts = kind == kResLoopBwd ? pml + inner : 1e-6 * e->NX * (e->nz + e->L);
  const int batch = fwd ? e->fbatch : e->batch, nl = (e->ns + batch - 1) / batch;
  const int br = std::min(fwd ? e->fbranches : e->branches, nl);
  const double rounds = 0.5 * ((nl + br - 1) / br + (double)nl / br);  // the last one may leave branches idle
  const double shot = kind == kResLoopBwd ? 12.0 * pml + 24.0 * inner : (xadj ? 20.0 : 12.0) * pml;  // MB
  const double mb = br * batch * shot + 20.0 * pml, launch = std::min(1.0, batch * pts / 0.3);
  const double all = e->ns * pts;
  if (xadj) return rounds * (7.0 + 0.8 * launch) + all * (6.7 + std::min(4.0, 0.040 * std::max(0.0, mb - 36.0)));
  if (!fwd)  // both wavefields in the interior, the adjoint alone outside it
    return rounds * (8.5 + 1.25 * launch) + e->ns * (5.5 * inner + 6.3 * (pml - inner)) +
           all * std::min(4.5, 0.031 * std::max(0.0, mb - 74.0));
  return rounds * ((kind == kResLoopSave ? 5.7 : 5.3) + 0.8 * launch) +
         all * ((e->ns <= 2 ? 2.05 : 2.5) + std::min(6.0, 0.012 * std::max(0.0, mb - 60.0)));
}

// Whether a split is set by the environment (column tiles per band; columns per thread), e.g. to test it.
inline int res_forced_tiles(ResKind kind) {
  const char* v = std::getenv(kind > kResLoopSave ? "SWIT_RES_BWD_TILES" : "SWIT_RES_FWD_TILES");
  return v ? std::atoi(v) : 0;
}
inline int res_forced_cols(ResKind kind) {
  const char* v = kind > kResLoopSave ? nullptr : std::getenv("SWIT_RES_FWD_COLS");
  return v ? std::atoi(v) : 0;
}
inline bool res_forced(ResKind kind) { return res_forced_tiles(kind) || res_forced_cols(kind); }

// The fastest split by estimate among those whose blocks are co-resident, for launches of `steps` steps.  A
// multi-instance engine's launches share the device, so there a split that takes fewer SMs may be slower by itself
// (reverse loops of 3, 1 and 2 shots up to 288x138: in bands that add up to 187 blocks they overlap, 3.0 ms a
// gradient, 232 blocks do not, 4.0 ms; gradients of 505 sets of 3 to 7 problems in the mean 2.5 % faster with a
// weight of 0.4 than of 0.1).
inline void res_choose(const swit_engine* e, ResKind kind, int steps, bool multi, ResLoop& out) {
  int dev = 0, sms = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return;
  const int want = res_forced_tiles(kind), cols = res_forced_cols(kind);
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
      const void* f = e->exact && kind == kResLoopSave ? (const void*)I[i].fd : I[i].any();
      int occ = 0;
      if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin) != cudaSuccess ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, f, r.nA + r.nR, r.smem) != cudaSuccess) {
        cudaGetLastError();
        continue;
      }
      const int fit = occ * sms / r.C;
      if (fit < 1) continue;
      const int waves = (e->ns + fit - 1) / fit;
      const int shots = (e->ns + waves - 1) / waves;
      const int bpsm = (shots * r.C + sms - 1) / sms;
      const double t = waves * (res_step_us(r, kind, e->exact, I[i].tx, I[i].maxt, bpsm) + kResLaunchUs / steps);
      const double cost = multi ? t * (1.0 + 0.4 * std::min(1.0, (double)shots * r.C / sms)) : t;
      if (!out.ok || cost < best) {
        best = cost;
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
