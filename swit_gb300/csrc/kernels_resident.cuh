// kernels_resident.cuh -- persistent time loops with the wavefields in registers
// (FP32).
//
// What bounds the step kernels of kernels_vec.cuh is moving the fields through
// L2 and L1 every step (about 26 flops per 32 bytes) and two dependent launches
// per step.  Here one cooperative launch runs the whole time loop of a wave of
// shots: every thread keeps the wavefields of a tile of 4 rows x TX columns in
// registers, a block owns a band of whole columns of one shot, and only tile
// edges move: along z by warp shuffles, along x through shared memory, between
// bands through L2.
//
// Rows.  Tiles are aligned to the free surface: row fs-1 is row 0 of its tile,
// so both mirrors, p(fs-1) = -p(fs+1) and w(fs-1) = w(fs), stay inside one
// thread for every npml.  The threads of a role number its tiles column tile by
// column tile, row tile fastest, so lanes are neighbours in z; the rows next to
// a warp's ends come through shared memory.
//
// Bands.  Only the pressure crosses a band edge, once per step: three columns
// each way as four 16-byte packets per row tile, each {tag, 3 values} written
// and polled with single 128-bit accesses, so a packet whose tag matches is
// complete and needs no fence (0.34 us between two blocks of a die, 0.69 us
// across dies).  It is sent as soon as the band's edge tiles have updated p and
// awaited after w, which needs no neighbour.  The u values the pressure phase
// reads beyond the edge (two columns on the left, one on the right) are
// recomputed from that halo by the edge threads, the same operations on the
// same values as in the neighbour.  A packet slot is reused two steps later; the
// neighbour can only be that far ahead after every thread of this block has left
// the phase that reads it.  Every poll is bounded; a thread that gives up
// records it in the engine's error word, which stays until a call reports it, and
// in the launch's stop word, at which the other threads soon give up too; it does
// not wait again.
//
// Damping.  The reference's profile is damp(max(iX, iZ)) with iX, iZ the cell
// numbers from the inner edges and damp non-decreasing, and rounding is
// monotone, so a factor 1 - kappa is the smaller of a column's and a row's:
// p: min(fx, fz), u: min(fxu, fz), w: min(fx, fzw), where fxu (fzw) averages two
// neighbouring columns (rows) -- neighbouring cell numbers differ by one, so
// iX is never strictly between those of two rows.  Tiles away from the sides,
// where fx = 1, take the minimum all the same: a second copy of the updates
// without it cost more in the instruction cache than the minimum does (49 shots
// 481x141: 14.1 against 13.2 us per forward step, 37.4 against 35.2 per reverse
// step).
//
// Update ranges.  Every point of a tile is updated; what the reference never
// updates is put right afterwards: the few of those values that a later update
// reads hold their initial zero (predicated rows, zero_cols), and everything the
// reconstruction does not update is re-inserted from the strips.
//
// Registers and instructions are what limits these kernels, so a thread keeps
// its fields, one word of flags and a few indices; strides are kernel
// parameters, and all roles run the same update code (two copies of it per block
// did not fit the instruction cache: 3.0 stalls per issue against 0.4).
//
// Every scalar expression is the one of kernels.cuh (fdcore.f90 order, no FMA):
// results are bit-identical to the other kernels and the oracle.
#pragma once
#include "kernels.cuh"

namespace swit {

enum { kResFwd = 0, kResAdj = 1, kResRec = 2 };
constexpr unsigned kResWaitLimit = 1u << 22;  // polls of one halo wait
constexpr int kResErr = 0x200;                // error word of a halo wait that gave up

// Split of a shot over its bands and threads, and the float4 indices of the
// shared-memory arrays.  Filled on the host (res_plan).  A slot numbers the row
// tiles of the band's column tiles: slot = column tile * nq + row tile.
struct ResPlan {
  int nt_tiles;  // column tiles of a shot
  int C;         // bands (blocks) per shot; band b has nt_tiles / C tiles, the first nt_tiles % C one more
  int nA, nR;    // threads (whole warps) of the forward or adjoint role, of the reconstruction
  int nq, nqr;   // row tiles of the forward or adjoint role, of the reconstruction
  int kr;        // row tile at the free surface (rows fs-1 ..), the reconstruction's first
  int m0, m1;    // first and last column tile with interior columns
  int ent_cap;   // receiver entries a band may hold
  int W;         // columns of the widest band
  int ns;        // slots: (tiles of the widest band + 2) nq
  int jz;        // row nz within its tile
  int nside;     // side arrays a band may hold: 6, or the 3 of one side
  float negz;    // -0 (see f2)
  unsigned wait; // polls before a halo wait gives up
  uint4* halo;   // packets: [block][role][side][parity][packet][row tile]; then the stop word
  int stop;      // packets before the stop word
  int* err;      // the engine's error word
  // A thread's data lies together at an odd stride of float4: addresses are a base and a constant, and the
  // 16-byte accesses of a warp are free of bank conflicts.
  int oC;        // coefficients of a thread: p update [TX], u, w updates [TX]; stride 2 TX + 1
  int oE, oER;   // edges of a slot, by role: pL0 pL1 pR uR0 uR1 uL; stride kEdge
  int oG, oGR;   // ghost columns of a row tile, by role: 3 coefficients, 3 factors; stride kEdge
  int oZ;        // rows next to every warp's ends, [warps + 2][6 TX floats]
  int oR, oR1;   // row factors fz, fzw of a row tile; the same, all 1; stride kRow
  int oX;        // column factors, float2 [W]
  int oD;        // adjoint -> reconstruction, [TX] of a slot; stride TX + 1
  int oStage;    // forward: staged rows, [6][W]
  int oS;        // forward: side columns, [nside][nq]
  int oEnt;      // receiver entries
  int oList;     // values moved every step, int2
  int oBox, box; // reverse: inputs of a step (strips, side columns, adjoint sources), [2 steps][box]
  int smem;      // bytes
};

constexpr int kEdge = 7, kRow = 3;

extern __shared__ __align__(16) float4 res_sm[];
__device__ __forceinline__ float* res_smf() { return reinterpret_cast<float*>(res_sm); }
__device__ __forceinline__ float4 mk4(const float* v) { return make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void lds4(int i, float* v) {
  const float4 t = res_sm[i];
  v[0] = t.x;
  v[1] = t.y;
  v[2] = t.z;
  v[3] = t.w;
}

// Predicated forms: what only some lanes of a warp do -- edges, special rows -- costs an issue slot each
// this way; as branches, which the compiler makes of it, they were a third of a step's latency.
// Their addresses are one register and constants: left to itself the compiler keeps every address of the
// loop in a register, and spills.
__device__ __forceinline__ unsigned res_addr(int i) { return (unsigned)__cvta_generic_to_shared(res_sm) + 16u * i; }
__device__ __forceinline__ int opaque(int x) {
  asm volatile("" : "+r"(x));
  return x;
}
__device__ __forceinline__ void sts4_if(bool on, int i, const float* v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q st.shared.v4.f32 [%1], {%2, %3, %4, %5};\n\t}" ::"r"(
                   (unsigned)on),
               "r"(res_addr(i)), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
               : "memory");
}
// a, b, c (d) to float4 i, i+1, ..
__device__ __forceinline__ void sts3x4_if(bool on, int i, const float* a, const float* b, const float* c) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q st.shared.v4.f32 [%1], {%2, %3, %4, %5};\n\t"
      "@q st.shared.v4.f32 [%1 + 16], {%6, %7, %8, %9};\n\t@q st.shared.v4.f32 [%1 + 32], {%10, %11, %12, %13};\n\t}" ::"r"(
          (unsigned)on),
      "r"(res_addr(i)), "f"(a[0]), "f"(a[1]), "f"(a[2]), "f"(a[3]), "f"(b[0]), "f"(b[1]), "f"(b[2]), "f"(b[3]),
      "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3])
      : "memory");
}
__device__ __forceinline__ void sts4x4_if(bool on, int i, const float* a, const float* b, const float* c,
                                          const float* d) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q st.shared.v4.f32 [%1], {%2, %3, %4, %5};\n\t"
      "@q st.shared.v4.f32 [%1 + 16], {%6, %7, %8, %9};\n\t@q st.shared.v4.f32 [%1 + 32], {%10, %11, %12, %13};\n\t"
      "@q st.shared.v4.f32 [%1 + 48], {%14, %15, %16, %17};\n\t}" ::"r"((unsigned)on),
      "r"(res_addr(i)), "f"(a[0]), "f"(a[1]), "f"(a[2]), "f"(a[3]), "f"(b[0]), "f"(b[1]), "f"(b[2]), "f"(b[3]),
      "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]), "f"(d[0]), "f"(d[1]), "f"(d[2]), "f"(d[3])
      : "memory");
}
// Rows 1 .. 3 of a, b, c, d from float4 i, i+1, ..
__device__ __forceinline__ void lds4x3_if(bool on, int i, float* a, float* b, float* c, float* d) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t.reg .f32 t;\n\tsetp.ne.u32 q, %12, 0;\n\t"
      "@q ld.shared.v4.f32 {t, %0, %1, %2}, [%13];\n\t@q ld.shared.v4.f32 {t, %3, %4, %5}, [%13 + 16];\n\t"
      "@q ld.shared.v4.f32 {t, %6, %7, %8}, [%13 + 32];\n\t@q ld.shared.v4.f32 {t, %9, %10, %11}, [%13 + 48];\n\t}"
      : "+f"(a[1]), "+f"(a[2]), "+f"(a[3]), "+f"(b[1]), "+f"(b[2]), "+f"(b[3]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]),
        "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"((unsigned)on), "r"(res_addr(i))
      : "memory");
}
// a, b, c, d from component k of float4 i, i+1, ..
__device__ __forceinline__ void lds4x1_if(bool on, int i, int k, float& a, float& b, float& c, float& d) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %4, 0;\n\t@q ld.shared.f32 %0, [%5];\n\t@q ld.shared.f32 %1, [%5 + 16];\n\t"
      "@q ld.shared.f32 %2, [%5 + 32];\n\t@q ld.shared.f32 %3, [%5 + 48];\n\t}"
      : "+f"(a), "+f"(b), "+f"(c), "+f"(d)
      : "r"((unsigned)on), "r"(res_addr(i) + 4u * k)
      : "memory");
}
__device__ __forceinline__ void stg4_if(unsigned on, float4* p, const float* v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q st.global.v4.f32 [%1], {%2, %3, %4, %5};\n\t}" ::"r"(on),
               "l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
               : "memory");
}
// v = a - b, v = v + a.
__device__ __forceinline__ void sub_if(unsigned on, float& v, float a, float b) {
  asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q sub.rn.f32 %0, %1, %2;\n\t}" : "+f"(v) : "f"(a), "f"(b), "r"(on));
}
__device__ __forceinline__ void add_if(unsigned on, float& v, float a) {
  asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q add.rn.f32 %0, %0, %1;\n\t}" : "+f"(v) : "f"(a), "r"(on));
}
__device__ __forceinline__ void mov_if(unsigned on, float& v, float a) {
  asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q mov.f32 %0, %1;\n\t}" : "+f"(v) : "f"(a), "r"(on));
}

// ---------------------------------------------------------------------------
// 128-bit packets through L2.
__device__ __forceinline__ void pkt_put(uint4* p, unsigned tag, float a, float b, float c) {
  asm volatile(
      "{\n\t.reg .b128 v;\n\t.reg .b64 lo, hi;\n\tmov.b64 lo, {%1, %2};\n\tmov.b64 hi, {%3, %4};\n\t"
      "mov.b128 v, {lo, hi};\n\tst.relaxed.gpu.global.b128 [%0], v;\n\t}" ::"l"(p),
      "r"(tag), "f"(a), "f"(b), "f"(c)
      : "memory");
}
// Three columns of one row tile.
__device__ __forceinline__ void halo_put(uint4* p, int nq, unsigned tag, const float* a, const float* b,
                                         const float* c) {
  pkt_put(p, tag, a[0], a[1], a[2]);
  pkt_put(p + nq, tag, a[3], b[0], b[1]);
  pkt_put(p + 2 * nq, tag, b[2], b[3], c[0]);
  pkt_put(p + 3 * nq, tag, c[1], c[2], c[3]);
}
// The four packets of a row tile as loaded.
struct Halo {
  unsigned t[4];
  float a[4], b[4], c[4];
};
// Issues the loads; what they bring is looked at later (halo_wait).
__device__ __forceinline__ void halo_issue(const uint4* p, int nq, Halo& h) {
  auto get = [&](const uint4* q, unsigned& t, float& x, float& y, float& z) {
    asm volatile(
        "{\n\t.reg .b128 v;\n\t.reg .b64 lo, hi;\n\tld.relaxed.gpu.global.b128 v, [%4];\n\tmov.b128 {lo, hi}, v;\n\t"
        "mov.b64 {%0, %1}, lo;\n\tmov.b64 {%2, %3}, hi;\n\t}"
        : "=r"(t), "=f"(x), "=f"(y), "=f"(z)
        : "l"(q)
        : "memory");
  };
  get(p, h.t[0], h.a[0], h.a[1], h.a[2]);
  get(p + nq, h.t[1], h.a[3], h.b[0], h.b[1]);
  get(p + 2 * nq, h.t[2], h.b[2], h.b[3], h.c[0]);
  get(p + 3 * nq, h.t[3], h.c[1], h.c[2], h.c[3]);
}
__device__ __forceinline__ bool halo_here(const Halo& h, unsigned tag) {
  return h.t[0] == tag && h.t[1] == tag && h.t[2] == tag && h.t[3] == tag;
}
// Loads until the packets are those of the tag.
__device__ __forceinline__ void halo_wait(const uint4* p, unsigned tag, const ResPlan& r, bool& dead, Halo& h) {
  for (unsigned n = 0;; ++n) {
    halo_issue(p, r.nq, h);
    if (halo_here(h, tag) || dead) return;
    int* stop = reinterpret_cast<int*>(r.halo + r.stop);
    if (n >= r.wait || ((n & 255u) == 255u && *(volatile int*)stop != 0)) {
      atomicExch(stop, 1);
      atomicCAS(r.err, 0, kResErr);
      dead = true;
    }
  }
}

__device__ __forceinline__ void cp4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// ---------------------------------------------------------------------------
// Flags of a thread's tile.  kRare is uniform over the warp.
enum : unsigned {
  kLive = 1u << 0,   // holds a tile
  kAdj = 1u << 1,    // adjoint role (reverse kernel)
  kRare = 1u << 3,   // the warp has band edges, columns to zero, side strips, the source or scattered receivers
  kEnds = 1u << 4,   // the tile has columns to zero
  kLeft = 1u << 5,   // at the band's left edge, and a neighbour band exists
  kRight = 1u << 6,  // at its right edge
  kTop = 1u << 7,    // the tile at the free surface (rows fs-1 .. fs+2)
  kStrip = 1u << 8,  // the tile has a side-strip column
  kImg = 1u << 9,    // adjoint tile with a reconstruction partner
  kB0 = 1u << 10,    // holds row nz of the interior
  kB1 = 1u << 11,    // holds row nz-1
  kRec = 1u << 12,   // has scattered receivers
  kTopFs = 1u << 13, // kTop, and there is a free surface
};
constexpr int kP = 16;     // 4 bits: rows of p the phase updates
constexpr int kW = 20;     // 4 bits: rows of w
constexpr int kRows = 24;  // 4 bits: rows on the interior
__device__ __forceinline__ unsigned bit_at(unsigned f, int b) { return f & (1u << b); }

template <int TX>
struct Tile {
  unsigned f;   // flags
  int slot, k;  // slot of the edge arrays, row tile (of the forward or adjoint role)
  int ix0;      // first column (PML grid, 1-based)
  int e;        // edges of the slot; its neighbours' are kEdge nq away
  int rf;       // row factors of this row tile
};
// Row 0 of a tile.
template <int TX>
__device__ __forceinline__ int row0(const Tile<TX>& T, const ResPlan& r, int fs) {
  return fs - 1 + 4 * (T.k - r.kr);
}

// Rows next to a warp's tiles, TX floats each.  Of p: 0 lane 31 row 3, 1 lane 0 row 0, 2 lane 0
// row 1; of w: 3 lane 31 row 3, 4 lane 31 row 2, 5 lane 0 row 0.  Warp w's are at (w + 1) 6 TX / 4.
template <int TX>
__device__ __forceinline__ void zrow_put(bool on, const ResPlan& r, int a, const float (&f)[TX][4], int j) {
  const int z = r.oZ + opaque((threadIdx.x >> 5) + 1) * (6 * TX / 4) + a * TX / 4;
#pragma unroll
  for (int c = 0; c < TX; c += 4) {
    const float v[4] = {f[c][j], f[c + 1][j], f[c + 2][j], f[c + 3][j]};
    sts4_if(on, z + c / 4, v);
  }
}
template <int TX>
__device__ __forceinline__ void zrow_get(const ResPlan& r, int warp, int a, float (&v)[TX]) {
  const int z = r.oZ + ((threadIdx.x >> 5) + 1 + warp) * (6 * TX / 4) + a * TX / 4;
#pragma unroll
  for (int c = 0; c < TX; c += 4) lds4(z + c / 4, v + c);
}

__device__ __forceinline__ float f_one(float d, float dt) { return 1.0f - d * dt; }
__device__ __forceinline__ float f_two(float d0, float d1, float dt) { return 1.0f - 0.5f * (d0 + d1) * dt; }
template <int TX>
__device__ __forceinline__ float2 col_factor(const Tile<TX>& T, const ResPlan& r, int tt0, int c) {
  return reinterpret_cast<const float2*>(res_sm + r.oX)[T.ix0 - 1 - tt0 * TX + c];
}

// Two FP32 operations per instruction (f32x2), each rounded as the scalar one.  Products are fma(x, y, -0)
// with a -0 the compiler cannot see, for ptxas contracts a packed product and a following packed sum even
// under --fmad=false; differences are fma(b, -1, a).  Rows j, j+1 of a column pair up without moves in the
// x-differences and the products, so u is packed in every loop (forward step of 49 shots 481x141 with
// strips 16.6 -> 16.2 us, of one shot 101x51 2.09 -> 1.98 us).  The operands of z-differences straddle
// pairs: w's stay scalar and only its products and sums are packed, in the reverse loop (38.0 -> 37.6 us,
// one shot 2.66 -> 2.42 us; in the forward loop it costs, 1.98 -> 2.08 us).  p, mostly z- and x-differences
// of separate arrays, is scalar: its moves cost more than the sums save (14.8 against 14.3 us).
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// The updates of a tile, the same code for every role: f := factor f - coef D (the reconstruction, which
// adds without damping, has row factor 1 and negated coefficients: the same values; its last column's u, the
// one interior value with a column factor below 1, is never read).
//
// p from u (x-neighbours in the edge arrays) and w.
// SAVE: D of the tile to save[column of the tile * nq].
template <int TX, bool SAVE = false>
__device__ __forceinline__ void tile_p(const Tile<TX>& T, const ResPlan& r, int tt0, float (&p)[TX][4],
                                       const float (&u)[TX][4], const float (&w)[TX][4], float c1, float c2,
                                       float4* save = nullptr) {
  const int lane = threadIdx.x & 31;
  float um2[4], um1[4], up1[4], fz[4], e1[TX], e2[TX], e6[TX];
  lds4(T.rf, fz);
  lds4(T.e - kEdge * r.nq + 3, um2);
  lds4(T.e - kEdge * r.nq + 4, um1);
  lds4(T.e + kEdge * r.nq + 5, up1);
  zrow_get<TX>(r, -1, 3, e1);
  zrow_get<TX>(r, -1, 4, e2);
  zrow_get<TX>(r, 1, 5, e6);
#pragma unroll
  for (int c = 0; c < TX; ++c) {
    float a[4];
    lds4(r.oC + (2 * TX + 1) * threadIdx.x + c, a);
    const float fx = col_factor<TX>(T, r, tt0, c).x;
    float z[7];  // w at rows -2 .. 4
    z[0] = __shfl_up_sync(0xffffffffu, w[c][2], 1);
    z[1] = __shfl_up_sync(0xffffffffu, w[c][3], 1);
    z[6] = __shfl_down_sync(0xffffffffu, w[c][0], 1);
    z[0] = lane == 0 ? e2[c] : z[0];
    z[1] = lane == 0 ? e1[c] : z[1];
    z[6] = lane == 31 ? e6[c] : z[6];
#pragma unroll
    for (int j = 0; j < 4; ++j) z[2 + j] = w[c][j];
    float d[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float l1 = c >= 1 ? u[c >= 1 ? c - 1 : 0][j] : um1[j];
      const float l2 = c >= 2 ? u[c >= 2 ? c - 2 : 0][j] : (c == 1 ? um1[j] : um2[j]);
      const float r1 = c + 1 < TX ? u[c + 1 < TX ? c + 1 : 0][j] : up1[j];
      const float D = c1 * (u[c][j] - l1 + z[j + 2] - z[j + 1]) + c2 * (r1 - l2 + z[j + 3] - z[j]);
      sub_if(bit_at(T.f, kP + j), p[c][j], fminf(fx, fz[j]) * p[c][j], a[j] * D);
      d[j] = D;
    }
    if constexpr (SAVE) stg4_if(T.f & kLive, save + c * r.nq, d);
  }
}

// w from p.
template <int TX, bool PACK>
__device__ __forceinline__ void tile_w(const Tile<TX>& T, const ResPlan& r, int tt0, const float (&p)[TX][4],
                                       float (&w)[TX][4], float c1, float c2) {
  const int lane = threadIdx.x & 31;
  float fz[4], e0[TX], e5[TX], e6[TX];
  lds4(T.rf + 1, fz);
  zrow_get<TX>(r, -1, 0, e0);
  zrow_get<TX>(r, 1, 1, e5);
  zrow_get<TX>(r, 1, 2, e6);
  const f2 Z = pk(r.negz, r.negz), C1 = pk(c1, c1), C2 = pk(c2, c2);
#pragma unroll
  for (int c = 0; c < TX; ++c) {
    float a[4];
    lds4(r.oC + (2 * TX + 1) * threadIdx.x + TX + c, a);
    const float fx = col_factor<TX>(T, r, tt0, c).x;
    float z[7];  // p at rows -1 .. 5
    z[0] = __shfl_up_sync(0xffffffffu, p[c][3], 1);
    z[5] = __shfl_down_sync(0xffffffffu, p[c][0], 1);
    z[6] = __shfl_down_sync(0xffffffffu, p[c][1], 1);
    z[0] = lane == 0 ? e0[c] : z[0];
    z[5] = lane == 31 ? e5[c] : z[5];
    z[6] = lane == 31 ? e6[c] : z[6];
#pragma unroll
    for (int j = 0; j < 4; ++j) z[1 + j] = p[c][j];
    if constexpr (!PACK) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float D = c1 * (z[j + 2] - z[j + 1]) + c2 * (z[j + 3] - z[j]);
        sub_if(bit_at(T.f, kW + j), w[c][j], fminf(fx, fz[j]) * w[c][j], a[j] * D);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        const f2 d1 = pk(z[j + 2] - z[j + 1], z[j + 3] - z[j + 2]), d2 = pk(z[j + 3] - z[j], z[j + 4] - z[j + 1]);
        const f2 D = add2(fma2(C1, d1, Z), fma2(C2, d2, Z));
        const f2 S = fma2(pk(a[j], a[j + 1]), D, Z);
        const f2 F = pk(fminf(fx, fz[j]), fminf(fx, fz[j + 1]));
        const f2 Q = fma2(F, pk(w[c][j], w[c][j + 1]), Z);
        float s0, s1, q0, q1;
        upk(S, s0, s1);
        upk(Q, q0, q1);
        sub_if(bit_at(T.f, kW + j), w[c][j], q0, s0);
        sub_if(bit_at(T.f, kW + j + 1), w[c][j + 1], q1, s1);
      }
    }
  }
}

// u from p (x-neighbours in the edge arrays).
template <int TX>
__device__ __forceinline__ void tile_u(const Tile<TX>& T, const ResPlan& r, int tt0, const float (&p)[TX][4],
                                       float (&u)[TX][4], float c1, float c2) {
  float pm1[4], pp1[4], pp2[4], fz[4];
  lds4(T.rf, fz);
  lds4(T.e - kEdge * r.nq + 2, pm1);
  lds4(T.e + kEdge * r.nq, pp1);
  lds4(T.e + kEdge * r.nq + 1, pp2);
  const f2 Z = pk(r.negz, r.negz), M = pk(-1.f, -1.f), C1 = pk(c1, c1), C2 = pk(c2, c2);
#pragma unroll
  for (int c = 0; c < TX; ++c) {
    float a[4];
    lds4(r.oC + (2 * TX + 1) * threadIdx.x + TX + c, a);
    const float fx = col_factor<TX>(T, r, tt0, c).y;
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
      auto P = [&](int k) {
        const float* q = k < 0 ? pm1 : (k < TX ? p[k < 0 || k >= TX ? 0 : k] : (k == TX ? pp1 : pp2));
        return pk(q[j], q[j + 1]);
      };
      const f2 d1 = fma2(P(c), M, P(c + 1)), d2 = fma2(P(c - 1), M, P(c + 2));
      const f2 D = add2(fma2(C1, d1, Z), fma2(C2, d2, Z));
      const f2 S = fma2(pk(a[j], a[j + 1]), D, Z);
      const f2 F = pk(fminf(fx, fz[j]), fminf(fx, fz[j + 1]));
      const f2 U = fma2(S, M, fma2(F, pk(u[c][j], u[c][j + 1]), Z));
      upk(U, u[c][j], u[c][j + 1]);
    }
  }
}

// Zeroes the columns a phase must not have changed and a later update reads: 1, 2, NX-1, NX of p, 1 and
// from NX-1 of u (rows: p and w are not updated outside their ranges, of u no such row is read).
template <int TX>
__device__ __forceinline__ void zero_cols(int ix0, float (&f)[TX][4], int lo, int hi) {
#pragma unroll
  for (int c = 0; c < TX; ++c)
    if (ix0 + c < lo || ix0 + c > hi) {
#pragma unroll
      for (int j = 0; j < 4; ++j) f[c][j] = 0.f;
    }
}

// Publishes the edges of p / of u and w within the band.
template <int TX>
__device__ __forceinline__ void publish_p(const Tile<TX>& T, const ResPlan& r, const float (&p)[TX][4]) {
  const int lane = threadIdx.x & 31;
  sts3x4_if(T.f & kLive, T.e, p[0], p[1], p[TX - 1]);
  zrow_put<TX>(lane == 31, r, 0, p, 3);
  zrow_put<TX>(lane == 0, r, 1, p, 0);
  zrow_put<TX>(lane == 0, r, 2, p, 1);
}
template <int TX>
__device__ __forceinline__ void publish_uw(const Tile<TX>& T, const ResPlan& r, const float (&u)[TX][4],
                                           const float (&w)[TX][4]) {
  const int lane = threadIdx.x & 31;
  sts3x4_if(T.f & kLive, T.e + 3, u[TX - 2], u[TX - 1], u[0]);
  zrow_put<TX>(lane == 31, r, 3, w, 3);
  zrow_put<TX>(lane == 31, r, 4, w, 2);
  zrow_put<TX>(lane == 0, r, 5, w, 0);
}

// ---------------------------------------------------------------------------
// Band edges.  Packets towards the left neighbour of (block, role): [parity][packet][row tile], those
// towards the right one kHaloSide row tiles further.
constexpr int kHaloSide = 8, kHaloRole = 16, kHaloBlock = 32;
template <int TX>
__device__ __forceinline__ uint4* halo_at(const Tile<TX>& T, const ResPlan& r, int role, unsigned tag) {
  return r.halo + (opaque(blockIdx.x * kHaloBlock + role * kHaloRole) + (int)(tag & 1u) * 4) * r.nq + T.k;
}

// Sends the edge columns of p (tag: the step they belong to).
template <int TX>
__device__ __forceinline__ void edge_send(const Tile<TX>& T, const ResPlan& r, int role, const float (&p)[TX][4],
                                          unsigned tag) {
  if (!(T.f & (kLeft | kRight))) return;
  uint4* o = halo_at<TX>(T, r, role, tag);
  if (T.f & kLeft) halo_put(o, r.nq, tag, p[0], p[1], p[2]);
  if (T.f & kRight) halo_put(o + kHaloSide * r.nq, r.nq, tag, p[TX - 3], p[TX - 2], p[TX - 1]);
}

// Ghost u of one column: the neighbour's own update of it.
__device__ __forceinline__ void ghost_u(int slot, int coef, int fac, float c1, float c2, const float* l1,
                                        const float* p0, const float* r1, const float* r2) {
  float u[4], a[4], f[4];
  lds4(slot, u);
  lds4(coef, a);
  lds4(fac, f);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float D = c1 * (r1[j] - p0[j]) + c2 * (r2[j] - l1[j]);
    u[j] = f[j] * u[j] - a[j] * D;
  }
  res_sm[slot] = mk4(u);
}

// Packets for this tile: from the left neighbour's right side, or the right one's left side.
template <int TX>
__device__ __forceinline__ const uint4* halo_from(const Tile<TX>& T, const ResPlan& r, int role, unsigned tag, bool left) {
  return halo_at<TX>(T, r, role, tag) + (left ? kHaloSide - kHaloBlock : kHaloBlock) * r.nq;
}
// The reverse loop issues the loads for a tile at one edge before it updates w: by then the packets have
// mostly arrived, and their latency (about 650 cycles) is covered (49 shots 481x141: 41.0 -> 39.1 us per
// step).  The forward gets to that point too early for that: 14.2 against 15.5 us.
template <int TX>
__device__ __forceinline__ void edge_issue(const Tile<TX>& T, const ResPlan& r, int role, unsigned tag, Halo& h) {
  if ((T.f & kRare) && (T.f & (kLeft | kRight))) halo_issue(halo_from<TX>(T, r, role, tag, T.f & kLeft), r.nq, h);
}

// Waits for the halo of p, puts its columns into the ghost slots of the edge
// arrays and updates the ghost u.  gu: ghost columns whose u is updated (bits 0,
// 1: left, 2: right); ghosts: the role's ghost tables; EARLY: h holds loads issued for the left edge, or for
// the right one where that is the tile's only one.
template <int TX, bool EARLY>
__device__ __forceinline__ void edge_recv(const Tile<TX>& T, const ResPlan& r, int role, int ghosts, unsigned gu,
                                          bool& dead, const float (&p)[TX][4], unsigned tag, float c1, float c2,
                                          Halo& h) {
  if (!(T.f & (kLeft | kRight))) return;
  const int nq = r.nq, g = ghosts + kEdge * opaque(T.k), e = opaque(T.e), el = e - kEdge * nq, er = e + kEdge * nq;
  if (T.f & kLeft) {  // columns ix0-3, ix0-2, ix0-1
    if (!EARLY || !halo_here(h, tag)) halo_wait(halo_from<TX>(T, r, role, tag, true), tag, r, dead, h);
    res_sm[el + 2] = mk4(h.c);
    if (gu & 1u) ghost_u(el + 3, g, g + 3, c1, c2, h.a, h.b, h.c, p[0]);
    if (gu & 2u) ghost_u(el + 4, g + 1, g + 4, c1, c2, h.b, h.c, p[0], p[1]);
  }
  if (T.f & kRight) {  // columns ix0+TX .. ix0+TX+2
    if (!EARLY || (T.f & kLeft) || !halo_here(h, tag))
      halo_wait(halo_from<TX>(T, r, role, tag, false), tag, r, dead, h);
    res_sm[er] = mk4(h.a);
    res_sm[er + 1] = mk4(h.b);
    if (gu & 4u) ghost_u(er + 5, g + 2, g + 5, c1, c2, p[TX - 1], h.a, h.b, h.c);
  }
}

// ---------------------------------------------------------------------------
// Rows [lo, hi] of a tile as bits.
__device__ __forceinline__ unsigned row_bits(int iz0, int lo, int hi) {
  unsigned m = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (iz0 + j >= lo && iz0 + j <= hi) m |= 1u << j;
  return m;
}

// Global <-> tile, points of the given range; zero outside it.
template <int TX>
__device__ __forceinline__ void tile_load(const float* f, int LD, int ix0, int iz0, bool live, int zlo, int zhi,
                                          int xlo, int xhi, float (&v)[TX][4]) {
#pragma unroll
  for (int c = 0; c < TX; ++c)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int ix = ix0 + c, iz = iz0 + j;
      v[c][j] = live && ix >= xlo && ix <= xhi && iz >= zlo && iz <= zhi ? f[(size_t)(ix - 1) * LD + iz - 1] : 0.f;
    }
}
template <int TX>
__device__ __forceinline__ void tile_store(float* f, int LD, int ix0, int iz0, bool live, int zlo, int zhi, int xlo,
                                           int xhi, const float (&v)[TX][4]) {
#pragma unroll
  for (int c = 0; c < TX; ++c)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int ix = ix0 + c, iz = iz0 + j;
      if (live && ix >= xlo && ix <= xhi && iz >= zlo && iz <= zhi) f[(size_t)(ix - 1) * LD + iz - 1] = v[c][j];
    }
}

// Damping of the 1-D profiles: by the cell number from the inner edge, 0 inside.
__device__ __forceinline__ float damp_1d(const float* damp, int i, int L, int N) {
  if (i < 1 || i > N) return 0.f;
  if (i <= L) return damp[L - i + 1];
  if (i >= N - L + 1) return damp[i - (N - L)];
  return 0.f;
}
// Row and column factors of the band whose first column is ix0.
__device__ __forceinline__ void factor_setup(const Grid<float>& g, const ResPlan& r, int ix0) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  for (int i = tid; i < 4 * r.nq; i += nthr) {
    const int iz = g.fs - 1 - 4 * r.kr + i;
    const float d0 = damp_1d(g.damp, iz, g.L, g.NZ), d1 = damp_1d(g.damp, iz + 1, g.L, g.NZ);
    const int at = 4 * kRow * (i >> 2) + (i & 3);
    res_smf()[4 * r.oR + at] = f_one(d0, g.dt);
    res_smf()[4 * r.oR + at + 4] = f_two(d0, d1, g.dt);
    if (r.nR) res_smf()[4 * r.oR1 + at] = res_smf()[4 * r.oR1 + at + 4] = 1.f;
  }
  for (int i = tid; i < r.W; i += nthr) {
    const float d0 = damp_1d(g.damp, ix0 + i, g.L, g.NX), d1 = damp_1d(g.damp, ix0 + i + 1, g.L, g.NX);
    reinterpret_cast<float2*>(res_sm + r.oX)[i] = make_float2(f_one(d0, g.dt), f_two(d0, d1, g.dt));
  }
}

// A thread's tile: thread t of a role whose n column tiles start at tile tt of the shot (column tile
// xoff of the band), nq row tiles each from row tile k0.
template <int TX, int ROLE>
__device__ __forceinline__ void tile_setup(Tile<TX>& T, const Grid<float>& g, const ResPlan& r, int t, int tt, int n,
                                           int xoff, int nq, int k0, bool lband, bool rband) {
  const bool live = t < n * nq;
  const int xt = live ? t / nq : 0;
  T.k = live ? k0 + t - xt * nq : k0;
  T.slot = ((live ? xoff + xt : 0) + 1) * r.nq + T.k;  // threads without a tile read inside the arrays too
  T.e = (ROLE == kResRec ? r.oER : r.oE) + kEdge * T.slot;
  T.rf = (ROLE == kResRec ? r.oR1 : r.oR) + kRow * T.k;
  T.ix0 = 1 + (tt + xt) * TX;
  const int NX = g.NX, NZ = g.NZ, L = g.L, fs = g.fs, iz0 = row0<TX>(T, r, fs);
  const bool strip = live && (T.ix0 <= L + 2 || T.ix0 + TX - 1 >= NX - L - 1);
  unsigned f = live ? kLive : 0u;
  auto holds = [&](int iz) { return live && iz >= iz0 && iz < iz0 + 4; };
  if (live && xt == 0 && lband) f |= kLeft;
  if (live && xt == n - 1 && rband) f |= kRight;
  if (strip) f |= kStrip;
  if (live && T.k == r.kr) f |= kTop;
  if (live && T.k == r.kr && g.fs_flag == 1) f |= kTopFs;
  if (holds(L + g.nz)) f |= kB0;
  if (holds(L + g.nz - 1)) f |= kB1;
  f |= row_bits(iz0, L + 1, L + g.nz) << kRows;
  if (ROLE == kResRec) {
    f |= 255u << kP;
  } else {
    if (ROLE == kResAdj) f |= kAdj;
    f |= row_bits(iz0, ROLE == kResFwd ? fs + 1 : 3, NZ - 2) << kP | row_bits(iz0, ROLE == kResFwd ? fs : 2, NZ - 2) << kW;
    if (live && (T.ix0 < 3 || T.ix0 + TX - 1 > NX - 2)) f |= kEnds;
  }
  T.f = live ? f : f & kAdj;
}

// Ghost tables of an edge thread: coefficient and damping factor of u at the
// ghost columns, and the ghost u of the state the loop starts from.  Returns the
// ghost columns to update (bits 0..2) and those the strips S2 / S5 replace (bits 4.., 8..).
template <int TX, int ROLE>
__device__ __forceinline__ unsigned ghost_setup(const Tile<TX>& T, const Grid<float>& g, const ResPlan& r,
                                                const float* u) {
  unsigned gu = 0u;
  const int gc = (ROLE == kResRec ? r.oGR : r.oG) + kEdge * T.k, iz0 = row0<TX>(T, r, g.fs);
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (!(T.f & (q < 2 ? kLeft : kRight))) continue;
    const int ix = q == 0 ? T.ix0 - 2 : (q == 1 ? T.ix0 - 1 : T.ix0 + TX);
    const int lo = ROLE == kResRec ? g.L + 2 : 2, hi = ROLE == kResRec ? g.L + g.nx - 2 : g.NX - 2;
    float a[4], f[4], v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int iz = iz0 + j;
      const bool in = ix >= 1 && ix <= g.NX && iz >= 1 && iz <= g.NZ;
      const size_t k = in ? (size_t)(ix - 1) * g.LD + iz - 1 : 0;
      a[j] = in ? (ROLE == kResAdj ? g.A[k] : (ROLE == kResRec ? -g.B[k] : g.B[k])) : 0.f;
      const float d = in ? damp_at(g.damp, iz, ix, g.L, g.NX, g.NZ) : 0.f;
      f[j] = ROLE == kResRec ? 1.f
                             : f_two(d, in && ix + 1 <= g.NX ? damp_at(g.damp, iz, ix + 1, g.L, g.NX, g.NZ) : d, g.dt);
      v[j] = in ? u[k] : 0.f;
    }
    if (ix >= lo && ix <= hi) gu |= 1u << q;
    if (ROLE == kResRec && ix == g.L + 1) gu |= 16u << q;
    if (ROLE == kResRec && ix == g.NX - g.L - 1) gu |= 256u << q;
    res_sm[gc + q] = mk4(a);
    res_sm[gc + 3 + q] = mk4(f);
    res_sm[q < 2 ? T.e - kEdge * r.nq + 3 + q : T.e + kEdge * r.nq + 5] = mk4(v);
  }
  return gu;
}

// ---------------------------------------------------------------------------
// f[code] += a (SUB: -=), code = 4 column + row.
template <int TX, bool SUB>
__device__ __forceinline__ void add_at(float (&f)[TX][4], int code, float a) {
#pragma unroll
  for (int c = 0; c < TX; ++c)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float v = SUB ? f[c][j] - a : f[c][j] + a;
      f[c][j] = code == 4 * c + j ? v : f[c][j];
    }
}
// Row j (0..3, run time) of a tile's column.
__device__ __forceinline__ float row_of(const float (&f)[4], int j) {
  return j == 0 ? f[0] : (j == 1 ? f[1] : (j == 2 ? f[2] : f[3]));
}

// Receiver entries of a tile are [base, base+n) of the band's list, ordered by node (column, then
// row) and, at one node, in receiver order.  row: the tile has exactly one receiver per column, all
// on that row and with consecutive numbers from ig0 (a receiver line); -1: general.
struct RecTile {
  int base, n, row, ig0;
};
// The forward records the tiles at the free surface with at most one receiver per column through the
// staged rows: s_col[c] = 4 receiver + row of the tile's column c, -1: none.
template <int TX>
__device__ __forceinline__ RecTile rec_setup(const Tile<TX>& T, const Grid<float>& g, const ResPlan& r,
                                             const Receivers& rec, int s, int* cnt, int* s_ig, int* s_code,
                                             int* s_col = nullptr) {
  RecTile R{0, 0, -1, 0};
  bool single = true;
  const int iz0 = row0<TX>(T, r, g.fs);
  if ((T.f & kLive) && iz0 + 3 >= rec.zlo[s] && iz0 <= rec.zhi[s]) {
    const int* cp = rec.colptr + (size_t)s * (g.NX + 2);
    for (int pass = 0; pass < 2; ++pass) {
      int n = 0, row = -1;
      bool line = true;
      for (int c = 0; c < TX; ++c) {
        const int ix = T.ix0 + c;
        int here = 0;
        if (ix <= g.NX)
          for (int j = 0; j < 4; ++j)
            for (int e = cp[ix]; e < cp[ix + 1]; ++e)
              if (rec.zrow[e] == iz0 + j) {
                if (pass) {
                  s_ig[R.base + n] = rec.ig[e];
                  s_code[R.base + n] = 4 * c + j;
                }
                if (row < 0) {
                  row = j;
                  R.ig0 = rec.ig[e] - c;
                }
                if (row != j || rec.ig[e] != R.ig0 + c) line = false;
                ++n;
                ++here;
              }
        if (here != 1) line = false;
        if (here > 1) single = false;
      }
      if (pass == 0) {
        R.n = n;
        R.row = line ? row : -1;
        if (n) R.base = atomicAdd(cnt, (n + 3) & ~3);
      } else if (s_col && (T.f & kTop) && single) {
        for (int i = 0; i < n; ++i) s_col[s_code[R.base + i] >> 2] = 4 * s_ig[R.base + i] + (s_code[R.base + i] & 3);
        R.n = 0;
      }
    }
  }
  return R;
}
// Values of the tile's receiver nodes to the step's traces.
template <int TX>
__device__ __forceinline__ void rec_take(const RecTile& R, const float (&f)[TX][4], const int* s_ig, const int* s_code,
                                         float* __restrict__ out) {
  if (R.row >= 0) {
#pragma unroll
    for (int c = 0; c < TX; ++c) out[R.ig0 + c] = row_of(f[c], R.row);
    return;
  }
#pragma unroll 1
  for (int n = 0; n < R.n; ++n) {
    const int code = s_code[R.base + n];
    float v = 0.f;
#pragma unroll
    for (int c = 0; c < TX; ++c)
#pragma unroll
      for (int j = 0; j < 4; ++j) v = code == 4 * c + j ? f[c][j] : v;
    out[s_ig[R.base + n]] = v;
  }
}
// f += dt * value (SUB: -=) at the tile's receiver nodes, in receiver order; s_val 16-byte aligned.
template <int TX, bool SUB>
__device__ __forceinline__ void rec_add_line(const RecTile& R, float (&f)[TX][4], int val, float dt) {
#pragma unroll
  for (int c = 0; c < TX; c += 4) {
    float v[4];
    lds4(val + (R.base + c) / 4, v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float a = SUB ? -(dt * v[i]) : dt * v[i];
#pragma unroll
      for (int j = 0; j < 4; ++j) add_if(R.row == j, f[c + i][j], a);
    }
  }
}
template <int TX, bool SUB>
__device__ __forceinline__ void rec_add(const RecTile& R, float (&f)[TX][4], const int* s_code, const float* s_val,
                                        float dt) {
#pragma unroll 1
  for (int n = 0; n < R.n; ++n) add_at<TX, SUB>(f, s_code[R.base + n], dt * s_val[R.base + n]);
}

// The columns of a tile -> consecutive float4.
template <int TX>
__device__ __forceinline__ void put_cols(bool on, int i, const float (&f)[TX][4]) {
  i = opaque(i);
#pragma unroll
  for (int c = 0; c < TX; c += 4) sts4x4_if(on, i + c, f[c], f[c + 1], f[c + 2], f[c + 3]);
}

// A band's list of single values that move between shared memory and the traces or strips of a step:
// {float index in shared memory, offset in the step's strips, or ~offset in its traces}.
__device__ __forceinline__ int2* res_list(const ResPlan& r) { return reinterpret_cast<int2*>(res_sm + r.oList); }
// Appends n items (whole warp; item i by lane i mod 32).
template <class F>
__device__ __forceinline__ void list_append(const ResPlan& r, int* cnt, int n, F&& item) {
  const int lane = threadIdx.x & 31;
  int at = 0;
  if (lane == 0) at = atomicAdd(cnt, n);
  at = __shfl_sync(0xffffffffu, at, 0);
  for (int i = lane; i < n; i += 32) res_list(r)[at + i] = item(i);
}

// ---------------------------------------------------------------------------
// Forward loop, steps it0 .. it1 (fdcore.f90:75-160) of shots shot0 + block / C.
//
// Bound by the dependent chain of a step (about 1.4 us: updates, two barriers, the halo) and, with 16 warps
// on an SM, by issue (2.2 instructions per cycle and SM, 940 per warp and step of which 455 are the
// stencil's): 512 threads of 128 registers hold as many points as the register file, so a launch takes as
// many shots as the device holds.  Measured against the vec kernels: 49 shots 481x141, nt 2000, misfit only
// 56.4 -> 25.7 ms; one shot 101x51, nt 600: 3.1 -> 0.93 ms.
template <int TX, int MAXT, bool SAVE>
__global__ void __launch_bounds__(MAXT, 1)
    k_fwd_res(const __grid_constant__ Grid<float> g, const __grid_constant__ ResPlan r,
              const __grid_constant__ Sources src, const __grid_constant__ Receivers rec, const float* __restrict__ s_fwd,
              float* __restrict__ P, float* __restrict__ U, float* __restrict__ W_, float* __restrict__ seis_t,
              float* __restrict__ strips, float4* __restrict__ dsave, int it0, int it1, int shot0) {
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31;
  const int b = blockIdx.x % r.C, s = shot0 + blockIdx.x / r.C;
  const int per = r.nt_tiles / r.C, rem = r.nt_tiles % r.C;
  const int tt0 = b * per + min(b, rem), n = per + (b < rem ? 1 : 0);
  const int fs = g.fs, L = g.L, NX = g.NX, NZ = g.NZ, nq = r.nq;
  const float c1 = g.c1, c2 = g.c2;
  int* s_cnt = reinterpret_cast<int*>(res_sm + r.oEnt);  // receiver entries
  int* s_ig = s_cnt + 4;
  int* s_code = s_ig + r.ent_cap;
  int* s_col = s_code + r.ent_cap;  // [W]

  for (int i = tid; i < r.smem / 16; i += nthr) res_sm[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  factor_setup(g, r, tt0 * TX + 1);
  for (int i = tid; i < r.W; i += nthr) s_col[i] = -1;
  __syncthreads();
  Tile<TX> T;
  tile_setup<TX, kResFwd>(T, g, r, tid, tt0, n, 0, nq, 0, b > 0, b < r.C - 1);
  const int xl = T.ix0 - 1 - tt0 * TX;  // first column within the band
  const size_t off = (size_t)s * g.FSZ;
  float p[TX][4], u[TX][4], w[TX][4];
  {
    const int iz0 = row0<TX>(T, r, fs);
    const bool live = T.f & kLive;
    tile_load<TX>(g.A, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, p);
    tile_load<TX>(g.B, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, u);
#pragma unroll
    for (int c = 0; c < TX; ++c) {
      res_sm[r.oC + (2 * TX + 1) * tid + c] = mk4(p[c]);
      res_sm[r.oC + (2 * TX + 1) * tid + TX + c] = mk4(u[c]);
    }
    tile_load<TX>(P + off, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, p);
    tile_load<TX>(U + off, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, u);
    tile_load<TX>(W_ + off, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, w);
  }
  const unsigned gu = ghost_setup<TX, kResFwd>(T, g, r, U + off);
  const RecTile R = rec_setup<TX>(T, g, r, rec, s, s_cnt, s_ig, s_code, s_col + xl);
  // the source point, if it is in this tile
  int isrc = -1;
  {
    const int cx = src.isx[s] - T.ix0, jz = src.isz[s] - row0<TX>(T, r, fs);
    if ((T.f & kLive) && cx >= 0 && cx < TX && jz >= 0 && jz < 4) isrc = 4 * cx + jz;
  }
  float snext = isrc >= 0 ? s_fwd[(size_t)s * (g.nt + 1) + it0 - 1] : 0.f;
  publish_uw<TX>(T, r, u, w);
  __syncthreads();

  // Traces and strips: the tiles that hold recorded rows stage whole columns in shared memory at the
  // end of a step -- p, u, w at the free surface, p at row nz, p and w at row nz - 1, the side columns --
  // and the block writes the values out by its list in the next step, while its halo is under way.
  auto side_at = [&](int a) { return TX == 4 || a < 3 ? a : a - 6 + r.nside; };
  {
    const StripOff o = strip_offsets(g.nx, g.nz);
    const int jx0 = tt0 * TX + 1 - L;
    const int flo = max(0, 1 - jx0), fn = max(0, min(n * TX, g.nx - jx0 + 1) - flo);
    for (int a = tid >> 5; a < 16; a += nthr >> 5) {
      if (a == 0) {
        for (int c = lane; c < n * TX; c += 32) {
          const int q = s_col[c];
          if (q >= 0)
            res_list(r)[atomicAdd(s_cnt + 1, 1)] =
                make_int2(4 * (r.oStage + rec.comp * r.W + c) + (q & 3), ~(q >> 2));
        }
      } else if (strips && a < 10) {
        // B0, B1 (p), B2 (w); T0, T1, T2 (p), T3, T4 (u), T5 (w): rows fs .. of the top tile
        const int q = a - 1;
        const int row = q < 3 ? (q == 1 && r.jz ? 3 : 3 + q) : (q < 6 ? 0 : (q < 8 ? 1 : 2));
        const int j = q < 1 ? (g.nz & 3) : (q < 3 ? ((g.nz - 1) & 3) : (q < 6 ? q - 2 : (q < 8 ? q - 5 : 1)));
        const int from = 4 * (r.oStage + row * r.W + flo) + j;
        const int to = (q < 3 ? q * g.nx : o.T0 + (q - 3) * g.nx) + jx0 + flo - 1;
        list_append(r, s_cnt + 1, fn, [&](int i) { return make_int2(from + 4 * i, to + i); });
      } else if (strips) {
        const int q = a - 10;  // S0 .. S5, if this band has the column
        const int ix = q < 3 ? (q == 1 ? L + 2 : L + 1) : (q == 3 ? NX - L : NX - L - 1);
        if (ix > tt0 * TX && ix <= (tt0 + n) * TX)
          list_append(r, s_cnt + 1, g.nz,
                      [&](int i) { return make_int2(4 * (r.oS + side_at(q) * nq) + i + 1, o.S0 + q * g.nz + i); });
      }
    }
  }
  __syncthreads();
  const int nlist = s_cnt[1];
  // (forward of 49 shots 481x141 without strips, staging p alone: 13.2 -> 12.4 us per step)
  auto stage = [&]() {
    put_cols<TX>(T.f & kTop, r.oStage + xl, p);
    if (!strips && rec.comp == 0) return;
    put_cols<TX>(T.f & kTop, r.oStage + r.W + xl, u);
    put_cols<TX>(T.f & kTop, r.oStage + 2 * r.W + xl, w);
    if (!strips) return;
    put_cols<TX>(T.f & kB0, r.oStage + 3 * r.W + xl, p);
    if (r.jz == 0) put_cols<TX>(T.f & kB1, r.oStage + 4 * r.W + xl, p);  // else rows nz-1 and nz share a tile
    put_cols<TX>(T.f & kB1, r.oStage + 5 * r.W + xl, w);
    if ((T.f & (kRare | kStrip)) == (kRare | kStrip)) {
#pragma unroll
      for (int c = 0; c < TX; ++c) {
        const int ix = T.ix0 + c;
        // with nx >= 8 the four columns are distinct
        const int a = ix == L + 1 ? 0 : (ix == L + 2 ? 1 : (ix == NX - L ? 3 : (ix == NX - L - 1 ? 4 : -1)));
        if (a >= 0) res_sm[r.oS + side_at(a) * nq + T.k] = mk4(p[c]);
        if (a == 0 || a == 4) res_sm[r.oS + side_at(a == 0 ? 2 : 5) * nq + T.k] = mk4(u[c]);
      }
    }
  };
  auto flush = [&](int it) {
    const size_t so = opaque(s);
    float* bs = strips + (so * g.snt + (it - g.sit0)) * g.SL;
    float* tr = seis_t + (so * g.nt + (it - 1)) * g.ngmax;
    for (int i = tid; i < nlist; i += nthr) {
      const int2 q = res_list(r)[i];
      *(q.y < 0 ? tr + ~q.y : bs + q.y) = res_smf()[q.x];
    }
  };
  bool dead = false;
  const bool rare = __any_sync(0xffffffffu, (T.f & (kLeft | kRight | kEnds | kStrip)) || isrc >= 0 || R.n > 0);
  if (rare) T.f |= kRare;

  for (int it = it0; it <= it1; ++it) {
    // ---- pressure phase
    float4* save = nullptr;
    if constexpr (SAVE)
      save = dsave + ((size_t)opaque(s) * g.snt + (it - g.sit0)) * (g.SL / 4) + (T.ix0 - 1) * nq + T.k;
    tile_p<TX, SAVE>(T, r, tt0, p, u, w, c1, c2, save);
    if (T.f & kRare) {
      if (T.f & kEnds) zero_cols<TX>(T.ix0, p, 3, NX - 2);
      if (isrc >= 0) {
        add_at<TX, false>(p, isrc, g.dt * snext);
        snext = s_fwd[(size_t)s * (g.nt + 1) + (it < it1 ? it : it - 1)];
      }
    }
#pragma unroll
    for (int c = 0; c < TX; ++c) mov_if(T.f & kTopFs, p[c][0], -p[c][2]);
    if (T.f & kRare) edge_send<TX>(T, r, 0, p, (unsigned)it);
    publish_p<TX>(T, r, p);
    if (it > it0) flush(it - 1);
    __syncthreads();
    // ---- velocity phase
    tile_w<TX, false>(T, r, tt0, p, w, c1, c2);
#pragma unroll
    for (int c = 0; c < TX; ++c) mov_if(T.f & kTopFs, w[c][0], w[c][1]);
    if (T.f & kRare) {
      Halo h;
      edge_recv<TX, false>(T, r, 0, r.oG, gu, dead, p, (unsigned)it, c1, c2, h);
    }
    __syncwarp();
    tile_u<TX>(T, r, tt0, p, u, c1, c2);
    if ((T.f & kRare) && (T.f & kEnds)) zero_cols<TX>(T.ix0, u, 2, NX - 2);
    publish_uw<TX>(T, r, u, w);
    stage();
    if ((T.f & kRare) && R.n) {
      float* out = seis_t + ((size_t)s * g.nt + (it - 1)) * g.ngmax;
      if (rec.comp == 0) rec_take<TX>(R, p, s_ig, s_code, out);
      if (rec.comp == 1) rec_take<TX>(R, u, s_ig, s_code, out);
      if (rec.comp == 2) rec_take<TX>(R, w, s_ig, s_code, out);
    }
    __syncthreads();
  }
  flush(it1);
  const int iz0 = row0<TX>(T, r, fs);
  const bool live = T.f & kLive;
  tile_store<TX>(P + off, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, p);
  tile_store<TX>(U + off, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, u);
  tile_store<TX>(W_ + off, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, w);
}

// ---------------------------------------------------------------------------
// What the reconstruction of a band re-inserts at one step (the strips of the
// step before): per column {-, T0, T1, T2} and {B0, B1, B2, -}, and the six side
// arrays of bands at (or next to) the sides (row jz at float jz); then the
// step's adjoint sources.  Two boxes by step parity.
__device__ __forceinline__ int box_at(const ResPlan& r, int it) { return r.oBox + (it & 1) * r.box; }
__device__ __forceinline__ int strip_t(const ResPlan& r, int it) { return box_at(r, it); }
__device__ __forceinline__ int strip_b(const ResPlan& r, int it) { return box_at(r, it) + r.W; }
__device__ __forceinline__ int strip_s(const ResPlan& r, int it, int a) { return box_at(r, it) + 2 * r.W + a * r.nqr; }
__device__ __forceinline__ int box_adj(const ResPlan& r, int it) { return box_at(r, it) + 2 * r.W + 6 * r.nqr; }
// Replaces the rows of column f that lie on the interior by side array a.
template <int TX>
__device__ __forceinline__ void insert_row(bool on, int at, int k, float (&f)[TX][4], int j) {
#pragma unroll
  for (int c = 0; c < TX; c += 4) lds4x1_if(on, at + c, k, f[c][j], f[c + 1][j], f[c + 2][j], f[c + 3][j]);
}
// Row nz falls on the same row J of its tile in every column: a constant of the launch.
#define SWIT_RES_ROW(j, call)                     \
  if ((j) == 0) {                                 \
    constexpr int J = 0;                          \
    call;                                         \
  } else if ((j) == 1) {                          \
    constexpr int J = 1;                          \
    call;                                         \
  } else if ((j) == 2) {                          \
    constexpr int J = 2;                          \
    call;                                         \
  } else {                                        \
    constexpr int J = 3;                          \
    call;                                         \
  }
template <int TX>
__device__ __forceinline__ void side_insert(const Tile<TX>& T, const ResPlan& r, int it, int a, float (&f)[4]) {
  float v[4];
  lds4(strip_s(r, it, a) + opaque(T.k) - r.kr, v);
#pragma unroll
  for (int j = 0; j < 4; ++j) f[j] = (T.f >> (kRows + j)) & 1u ? v[j] : f[j];
}

// Reverse loop, steps it1 .. it0 (solver.f90:230-253), of shots shot0 + block /
// C: the first nA threads run the adjoint (fdcore.f90:293-375), the others the
// reconstruction (fdcore.f90:202-289) on the same band, so each keeps three
// fields and the sums of one side; the image needs one value per point from one
// to the other, pb(t+1) - pb(t), through shared memory.
//
// Five 16-value arrays and the rest need more registers than 128: 384 threads of 168 are faster on a full
// device than 512 of 128, which spill (49 shots 481x141: 3.1 against 4.4 us per step and launch, 13 and 10
// launches, before later steps).  Measured against the vec kernels: reverse step of 49 shots 481x141
// 59.8 -> 34.1 us, of 5 shots 201x101 11.2 -> 2.4 us.
template <int TX, int MAXT>
__global__ void __launch_bounds__(MAXT, 1)
    k_bwd_res(const __grid_constant__ Grid<float> g, const __grid_constant__ ResPlan r,
              const __grid_constant__ Sources src, const __grid_constant__ Receivers rec, const float* __restrict__ s_fwd,
              const float* __restrict__ adj_t, float* __restrict__ PB, float* __restrict__ UB, float* __restrict__ WB,
              float* __restrict__ PE, float* __restrict__ UE, float* __restrict__ WE, float* __restrict__ DG,
              float* __restrict__ DFW, float* __restrict__ DBK, const float* __restrict__ strips, int it1, int it0,
              int shot0) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int b = blockIdx.x % r.C, s = shot0 + blockIdx.x / r.C;
  const int per = r.nt_tiles / r.C, rem = r.nt_tiles % r.C;
  const int tt0 = b * per + min(b, rem), n = per + (b < rem ? 1 : 0);
  const int fs = g.fs, L = g.L, NX = g.NX, NZ = g.NZ;
  const float c1 = g.c1, c2 = g.c2;
  // column tiles of the reconstruction in this band
  const int q0 = max(tt0, r.m0), q1 = min(tt0 + n - 1, r.m1);
  const int xoff = q0 - tt0, nr = q1 >= q0 ? q1 - q0 + 1 : 0;
  int* s_cnt = reinterpret_cast<int*>(res_sm + r.oEnt);  // receiver entries
  int* s_ig = s_cnt + 4;
  int* s_code = s_ig + r.ent_cap;

  for (int i = tid; i < r.smem / 16; i += nthr) res_sm[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  factor_setup(g, r, tt0 * TX + 1);
  __syncthreads();
  Tile<TX> T;
  const bool adj0 = tid < r.nA;  // role, uniform over a warp
  if (adj0)
    tile_setup<TX, kResAdj>(T, g, r, tid, tt0, n, 0, r.nq, 0, b > 0, b < r.C - 1);
  else
    tile_setup<TX, kResRec>(T, g, r, tid - r.nA, q0, nr, xoff, r.nqr, r.kr, xoff == 0 && tt0 > r.m0,
                            q1 == tt0 + n - 1 && q1 < r.m1);
  float p[TX][4], u[TX][4], w[TX][4];
  float s1[TX][4], s2[TX][4];  // adjoint: sum of pb^2, pb before the update; reconstruction: image, sum of pf^2
  const size_t off = (size_t)s * g.FSZ;
  unsigned gu;
  RecTile R{0, 0, -1, 0};
  int isrc = -1;  // source subtraction point, if it is in this tile
  {
    const int iz0 = row0<TX>(T, r, fs);
    const bool live = T.f & kLive;
    tile_load<TX>(adj0 ? g.A : g.B, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, p);
    tile_load<TX>(adj0 ? g.B : g.A, g.LD, T.ix0, iz0, live, 1, NZ, 1, NX, u);
#pragma unroll
    for (int c = 0; c < TX; ++c) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        p[c][j] = adj0 ? p[c][j] : -p[c][j];
        u[c][j] = adj0 ? u[c][j] : -u[c][j];
      }
      res_sm[r.oC + (2 * TX + 1) * tid + TX + c] = mk4(p[c]);
      res_sm[r.oC + (2 * TX + 1) * tid + c] = mk4(u[c]);
    }
    const int z0 = adj0 ? 1 : L + 1, z1 = adj0 ? NZ : L + g.nz, x0 = adj0 ? 1 : L + 1, x1 = adj0 ? NX : L + g.nx;
    tile_load<TX>((adj0 ? PB : PE) + off, g.LD, T.ix0, iz0, live, z0, z1, x0, x1, p);
    tile_load<TX>((adj0 ? UB : UE) + off, g.LD, T.ix0, iz0, live, z0, z1, x0, x1, u);
    tile_load<TX>((adj0 ? WB : WE) + off, g.LD, T.ix0, iz0, live, z0, z1, x0, x1, w);
    tile_load<TX>((adj0 ? DBK : DG) + off, g.LD, T.ix0, iz0, live, L + 1, L + g.nz, L + 1, L + g.nx, s1);
    tile_load<TX>(DFW + off, g.LD, T.ix0, iz0, live && !adj0, L + 1, L + g.nz, L + 1, L + g.nx, s2);
    if (adj0) {
      gu = ghost_setup<TX, kResAdj>(T, g, r, UB + off);
      R = rec_setup<TX>(T, g, r, rec, s, s_cnt, s_ig, s_code);
      // one value per point goes to the reconstruction's tile in the same slot
      const int xr = (T.ix0 - 1) / TX - q0, kq = T.k - r.kr;
      const bool img = live && xr >= 0 && xr < nr && kq >= 0 && kq < r.nqr;
      if (img) T.f |= kImg;
      if (R.n > 0 && R.row < 0) T.f |= kRec;
    } else {
      gu = ghost_setup<TX, kResRec>(T, g, r, UE + off);
      const int cx = src.risx[s] + L - T.ix0, jz = src.risz[s] + L - iz0;
      if (live && src.risx[s] > 0 && cx >= 0 && cx < TX && jz >= 0 && jz < 4) isrc = 4 * cx + jz;
    }
  }
  float snext = isrc >= 0 ? s_fwd[(size_t)s * (g.nt + 1) + it1] : 0.f;
  const int role = adj0 ? 0 : 1;
  edge_send<TX>(T, r, role, p, (unsigned)(it1 + 1));
  publish_p<TX>(T, r, p);
  publish_uw<TX>(T, r, u, w);
  __syncthreads();
  // Inputs of step it, fetched a step ahead by the adjoint threads: adjoint sources; strips of step it-1,
  // the side arrays in bands with (or next to) columns L+1, L+2 / NX-L-1, NX-L.
  {
    const StripOff o = strip_offsets(g.nx, g.nz);
    const int jx0 = tt0 * TX + 1 - L, lo = max(0, 1 - jx0), fn = nr ? max(0, min(n * TX, g.nx - jx0 + 1) - lo) : 0;
    const int xa = tt0 * TX + 1 - 3, xb = (tt0 + n) * TX + 3;
    for (int a = tid >> 5; a < 13; a += nthr >> 5) {
      if (a < 6) {
        const int to = 4 * ((a < 3 ? r.W : 0) + lo) + (a < 3 ? a : a - 2);
        const int from = (a < 3 ? a * g.nx : o.T0 + (a - 3) * g.nx) + jx0 + lo - 1;
        list_append(r, s_cnt + 1, fn, [&](int i) { return make_int2(to + 4 * i, from + i); });
      } else if (a < 12) {
        if (nr && (a < 9 ? (xa <= L + 2 && xb >= L + 1) : (xa <= NX - L && xb >= NX - L - 1)))
          list_append(r, s_cnt + 1, g.nz, [&](int i) {
            return make_int2(4 * (2 * r.W + (a - 6) * r.nqr) + 1 + i, o.S0 + (a - 6) * g.nz + i);
          });
      } else {
        // entries without a receiver (the padding of a tile's entries) repeat receiver 0: never read
        list_append(r, s_cnt + 1, s_cnt[0],
                    [&](int i) { return make_int2(4 * (2 * r.W + 6 * r.nqr) + i, ~s_ig[i]); });
      }
    }
  }
  __syncthreads();
  const int nlist = s_cnt[1];
  auto prefetch = [&](int it) {
    const size_t so = opaque(s);
    const float* at = adj_t + (so * g.nt + (it - 1)) * g.ngmax;
    const float* bs = strips + (so * g.snt + (it - 1 - g.sit0)) * g.SL;
    float* box = res_smf() + 4 * box_at(r, it);
    for (int i = tid; i < nlist; i += r.nA) {
      const int2 q = res_list(r)[i];
      cp4(box + q.x, q.y < 0 ? at + ~q.y : bs + q.y);
    }
  };
  const bool rare = __any_sync(0xffffffffu, (T.f & (kLeft | kRight | kEnds | kStrip | kRec)) || isrc >= 0 || gu);
  if (rare) T.f |= kRare;
  if (T.f & kAdj) {
    prefetch(it1);
    cp_wait();
  }
  __syncthreads();
  auto image = [&]() {  // the step before: image and illumination of the reconstruction
#pragma unroll
    for (int c = 0; c < TX; ++c) {
      float d[4];
      lds4(r.oD + (TX + 1) * T.slot + c, d);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s1[c][j] = s1[c][j] + p[c][j] * d[j];
        s2[c][j] = s2[c][j] + p[c][j] * p[c][j];
      }
    }
  };
  bool dead = false;

  for (int it = it1; it >= it0; --it) {
    // ---- velocity phase
    if (!(T.f & kAdj) && it < it1) image();
    Halo h;
    edge_issue<TX>(T, r, role, (unsigned)(it + 1), h);
    tile_w<TX, true>(T, r, tt0, p, w, c1, c2);
    if (T.f & kAdj) {
      // outside the update range of w both rows are never read
#pragma unroll
      for (int c = 0; c < TX; ++c) mov_if(T.f & kTopFs, w[c][0], w[c][1]);
      if (it > it0) prefetch(it - 1);
    } else {
      const int at = strip_b(r, it) + opaque(T.ix0) - 1 - tt0 * TX;
      SWIT_RES_ROW(r.jz, insert_row<TX>(T.f & kB1, at, 2, w, (J + 3) & 3))
    }
    if (T.f & kRare) {
      edge_recv<TX, true>(T, r, role, role ? r.oGR : r.oG, gu, dead, p, (unsigned)(it + 1), c1, c2, h);
      if (gu >> 4) {  // ghost columns jx = 1 and nx-1 of the reconstruction
#pragma unroll
        for (int q = 0; q < 3; ++q)
          if ((gu >> q) & 0x110u) {
            const int slot = q < 2 ? T.e - kEdge * r.nq + 3 + q : T.e + kEdge * r.nq + 5;
            float v[4];
            lds4(slot, v);
            side_insert<TX>(T, r, it, (gu >> q) & 16u ? 2 : 5, v);
            res_sm[slot] = mk4(v);
          }
      }
    }
    __syncwarp();
    tile_u<TX>(T, r, tt0, p, u, c1, c2);
    if (T.f & kRare) {
      if (T.f & kEnds) zero_cols<TX>(T.ix0, u, 2, NX - 2);
      if ((T.f & (kStrip | kAdj)) == kStrip) {
#pragma unroll
        for (int c = 0; c < TX; ++c) {
          const int ix = T.ix0 + c;
          if (ix == L + 1 || ix == NX - L - 1) side_insert<TX>(T, r, it, ix == L + 1 ? 2 : 5, u[c]);
        }
      }
    }
    publish_uw<TX>(T, r, u, w);
    __syncthreads();
    // ---- pressure phase
    if (T.f & kAdj) {
#pragma unroll
      for (int c = 0; c < TX; ++c)
#pragma unroll
        for (int j = 0; j < 4; ++j) s2[c][j] = p[c][j];
    } else if ((T.f & kRare) && isrc >= 0) {
      add_at<TX, true>(p, isrc, g.dt * snext);
      snext = s_fwd[(size_t)s * (g.nt + 1) + it - 1];
    }
    tile_p<TX>(T, r, tt0, p, u, w, c1, c2);
    if (T.f & kAdj) {
      if ((T.f & kRare) && (T.f & kEnds)) zero_cols<TX>(T.ix0, p, 3, NX - 2);
      if (rec.comp == 0) {
        rec_add_line<TX, false>(R, p, box_adj(r, it), g.dt);
        if ((T.f & kRare) && (T.f & kRec)) rec_add<TX, false>(R, p, s_code, res_smf() + 4 * box_adj(r, it), g.dt);
      }
#pragma unroll
      for (int c = 0; c < TX; ++c) mov_if(T.f & kTop, p[c][0], -p[c][2]);
    } else {
      // re-insert in the reference's order: bottom, sides, top.  Every pressure the reference does not
      // update is re-inserted, and no update that survives reads a velocity it does not update, apart
      // from the re-inserted ones (w row nz-1, u columns 1 and nx-1): no update range is tested.
      const int xl = opaque(T.ix0) - 1 - tt0 * TX;
      const int at = strip_b(r, it) + xl;
      SWIT_RES_ROW(r.jz, insert_row<TX>(T.f & kB0, at, 0, p, J); insert_row<TX>(T.f & kB1, at, 1, p, (J + 3) & 3))
      if ((T.f & kRare) && (T.f & kStrip)) {
#pragma unroll
        for (int c = 0; c < TX; ++c) {
          const int ix = T.ix0 + c;
          // with nx >= 8 the four columns are distinct
          const int a = ix == L + 1 ? 0 : (ix == L + 2 ? 1 : (ix == NX - L ? 3 : (ix == NX - L - 1 ? 4 : -1)));
          if (a >= 0) side_insert<TX>(T, r, it, a, p[c]);
        }
      }
#pragma unroll
      for (int c = 0; c < TX; c += 4) lds4x3_if(T.f & kTop, strip_t(r, it) + xl + c, p[c], p[c + 1], p[c + 2], p[c + 3]);
    }
    if (T.f & kRare)     edge_send<TX>(T, r, role, p, (unsigned)it);
    publish_p<TX>(T, r, p);
    if (T.f & kAdj) {
#pragma unroll
      for (int c = 0; c < TX; ++c)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s2[c][j] = s2[c][j] - p[c][j];
          s1[c][j] = s1[c][j] + p[c][j] * p[c][j];
        }
      put_cols<TX>(T.f & kImg, r.oD + (TX + 1) * T.slot, s2);
      // vz receivers: the adjoint source changes w after the pressure phase (vx: not on this path)
      if (rec.comp == 2) {
        rec_add_line<TX, true>(R, w, box_adj(r, it), g.dt);
        if ((T.f & kRare) && (T.f & kRec)) rec_add<TX, true>(R, w, s_code, res_smf() + 4 * box_adj(r, it), g.dt);
      }
    }
    if (T.f & kAdj) cp_wait();
    __syncthreads();
  }
  const bool adj = T.f & kAdj, live = T.f & kLive;
  if (!adj) image();
  const int iz0 = row0<TX>(T, r, fs);
  const int z0 = adj ? 1 : L + 1, z1 = adj ? NZ : L + g.nz, x0 = adj ? 1 : L + 1, x1 = adj ? NX : L + g.nx;
  tile_store<TX>((adj ? PB : PE) + off, g.LD, T.ix0, iz0, live, z0, z1, x0, x1, p);
  tile_store<TX>((adj ? UB : UE) + off, g.LD, T.ix0, iz0, live, z0, z1, x0, x1, u);
  tile_store<TX>((adj ? WB : WE) + off, g.LD, T.ix0, iz0, live, z0, z1, x0, x1, w);
  tile_store<TX>((adj ? DBK : DG) + off, g.LD, T.ix0, iz0, live, L + 1, L + g.nz, L + 1, L + g.nx, s1);
  tile_store<TX>(DFW + off, g.LD, T.ix0, iz0, live && !adj, L + 1, L + g.nz, L + 1, L + g.nx, s2);
}

}  // namespace swit
