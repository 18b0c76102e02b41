// k_resident.cu -- the IRLS + CG solve with a field's state resident on chip.
//
// Same iteration as k_solver.cu (VariationalRefine, hvd-core/src/engine/
// variational.cpp:198-556, with the single-reduction recurrence described
// there) for fields that fit in the SMs' tensor and shared memory. The
// streaming kernel moves ~82 B of HBM or L2 per pixel in every CG iteration
// and passes the phases of a lone field through a work queue; here a gang of
// CTAs takes a whole field, each CTA keeps one tile of it (a 64-column strip
// x up to 112 rows) for the entire solve -- g, q and chi, which only their own
// thread touches, in tensor memory; d, its luma part and the weights, which
// neighbours read, in shared memory -- and an iteration exchanges only the
// tile edges' q and the CTA's partial sums.
//
//  * Exchange: every word another CTA needs is published as a 16-byte slot
//    {8 bytes of data, 8 bytes of tag} by one 128-bit store and polled by one
//    128-bit load (both relaxed, gpu scope, single-copy atomic), the tag
//    naming the field and the exchange. Data and flag arrive together: no
//    fence, no flag round trip, one L2 latency per iteration. Edge slots
//    rotate over three sets: a CTA that publishes exchange n + 3 has either
//    every CTA's partial sums of a CG sweep after n, or (in the reweight and
//    gradient exchanges of an outer pass, which carry no sums) has polled all
//    four neighbours' exchange n + 1 or n + 2, which they published after
//    consuming n. Sum slots alternate by sweep: sweep n + 2 is published with
//    all of n + 1's sums in hand, whose owners had consumed n.
//  * Reduction: each CTA publishes six FP64 partials and sums all CTAs' in a
//    fixed order itself, so every CTA holds the same alpha and beta without a
//    broadcast, and the result does not depend on timing.
//  * Halo pixels: one thread per edge pixel keeps the neighbour's g and d and
//    repeats its update from the published q.
//  * Gangs: a batch runs as `gangs` fields at a time, each on sm_count / gangs
//    CTAs; a gang's first CTA fetches its next field when all have finished
//    with the last one.
//
// All waits are bounded: SolverArgs::phase_wait_limit polls for what another CTA
// publishes next. A CTA that has no tile of its gang's field waits for the
// whole field: one such limit for each of the field's exchanges, looking at the
// error flag after each. A CTA that gives up sets that flag and leaves, and its
// peers follow by their own limits. The launch is cooperative, so all CTAs are
// co-resident.
//
// Per-pixel arithmetic, its order and the FP32 row terms of the inner
// products are those of k_solver.cu; only the order of the FP64 additions
// differs.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <functional>
#include <vector>

#include "hvdg_common.cuh"
#include "k_solver.h"

namespace hvdg {

namespace {

constexpr int kRT = 512;             // threads per CTA
constexpr int kRW = kRT / 32;        // warps
constexpr int kMaxRows = 112;        // tile rows: seven per warp
constexpr int kSideCap = 112;        // side slots per column (>= kMaxRows, multiple of 16)
constexpr int kOutSlots = 2 * kStrip + 2 * kSideCap;
constexpr int kSets = 3;             // edge slot sets
constexpr int kHaloThreads = kOutSlots;  // thread t < 352 owns one possible halo pixel
constexpr int kRedWarp0 = kHaloThreads / 32;  // warps 11..15 collect the sums
constexpr int kNV = 6;               // H, <g,d>, <g,q>, <q,q>, <g,g>, and ||g_0||^2 at k = 0
// Sum slots: one 128-byte line of eight slots per CTA, written by one store
// instruction, in four copies, each polled by a quarter of the CTAs. Polling
// traffic on the lines is what an exchange waits for: a reader polls a line's
// first slot alone and takes the others once it has arrived.
constexpr int kLine = 8, kRep = 4;
constexpr int kMaxCtas = 160;        // CTAs of a gang (five slots per collecting lane)
static_assert(kHaloThreads % 32 == 0 && kRW - kRedWarp0 == 5, "five collecting warps");

struct __align__(16) Slot {
  unsigned long long lo, hi;
};
constexpr uint32_t kSetBytes = sizeof(Slot) * kOutSlots;

// Exchange memory: per CTA three sets of edge slots, then per gang the sum slots
// ([set][copy][CTA][value]), then a fetch slot per gang and a done counter per CTA.
__host__ __device__ constexpr size_t edge_bytes() { return sizeof(Slot) * kSets * kOutSlots; }
__host__ __device__ constexpr size_t red_bytes() { return sizeof(Slot) * 2 * kLine * kRep; }

__device__ __forceinline__ void st_slot(Slot* p, unsigned long long lo, unsigned long long hi) {
  asm volatile(
      "{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p),
      "l"(lo), "l"(hi)
      : "memory");
}
__device__ __forceinline__ void ld_slot(const Slot* p, unsigned long long& lo,
                                        unsigned long long& hi) {
  asm volatile(
      "{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
      : "=l"(lo), "=l"(hi)
      : "l"(p)
      : "memory");
}
__device__ __forceinline__ unsigned long long pack2(float2 v) {
  return (unsigned long long)__float_as_uint(v.x) |
         ((unsigned long long)__float_as_uint(v.y) << 32);
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  return make_float2(__uint_as_float((unsigned)v), __uint_as_float((unsigned)(v >> 32)));
}
// The roundings of the streaming kernel, spelled out so that the two agree bit
// for bit: which products are rounded (the fluxes: they are carried or
// shuffled) and which share a fused multiply-add. Factors of 2 are exact and
// move freely.
__device__ __forceinline__ float2 scale_rn(float2 v, float s) {
  return make_float2(__fmul_rn(v.x, s), __fmul_rn(v.y, s));
}
__device__ __forceinline__ float mix(float x, float m2h, float y, float m2v) {
  return __fmaf_rn(x, m2h, __fmul_rn(y, m2v));
}
// Re[u c]
__device__ __forceinline__ float re_rn(float2 u, float2 c) {
  return __fmaf_rn(u.x, c.x, -__fmul_rn(u.y, c.y));
}

__device__ __forceinline__ float dot_yx(float2 a, float2 b) {
  return __fmaf_rn(a.y, b.y, __fmul_rn(a.x, b.x));
}
__device__ __forceinline__ float norm_yx(float2 a) { return dot_yx(a, a); }
__device__ __forceinline__ float norm_xy(float2 a) {
  return __fmaf_rn(a.x, a.x, __fmul_rn(a.y, a.y));
}
__device__ __forceinline__ float curv_sum(float luma, float wh, float nh, float wv, float nv) {
  return __fmaf_rn(wv, nv, __fmaf_rn(wh, nh, luma));
}

// g^2 + eps^2, and m^2 + k g^2 + eps_c^2
__device__ __forceinline__ float edge_y(float g, float e2) {
  return __fadd_rn(__fmul_rn(g, g), e2);
}
__device__ __forceinline__ float edge_c(float m, float k, float g, float ec2) {
  return __fadd_rn(__fmaf_rn(__fmul_rn(k, g), g, __fmul_rn(m, m)), ec2);
}

// What the sums decide, published to the CTA by one warp.
struct Scalars {
  float alpha, beta;
  int pending, stop;
  double tol2, thr_abs;  // exit thresholds: relative to ||g_0||^2, absolute
  long long limits;      // wait limits that the fetch of the next field may take
};

struct ResidentArgs {
  int gangs, ctas, rows;
};

// Shared memory of a tile, as 32-bit shared addresses. Two row arrays, so that
// the unrolled rows of a warp address everything by immediate offsets from two
// lane bases:
//  * U block r + 1 holds row r of u (d; chi in the R and G phases) with the
//    column right of the strip, its luma part y, and the column left of the
//    strip (luma part, horizontal weights, u); blocks 0 and rows + 1 are the
//    rows above and below the tile.
//  * W block r holds the weights (wx, wy, wcx, wcy) of each lane's even and odd
//    pixel, the line phasor (sw Lx, sw Ly, Lx, Ly) with sw the V-switch
//    sense, and (kNbr) the neighbour data term.
constexpr uint32_t kUB = 800;
constexpr uint32_t kUR = 512, kY = 520, kYR = 776, kYL = 780, kWL = 784, kUL = 792;
constexpr uint32_t kWb = 512, kLn = 1024, kM = 1040;
template <bool kNbr>
struct Smem {
  static constexpr uint32_t kWB = kNbr ? 1808 : 1040;
  uint32_t u, w, wtop;  // wtop: 64 x (wy, wcy) of the row above the tile
  double* part;         // kNV x warps
  double* res;          // kNV x collecting warps
  Scalars* sc;
  int* word;            // [0]: a wait ran out, [1..2]: next field
  static constexpr size_t bytes(int rows) {
    return (size_t)(rows + 2) * kUB + (size_t)rows * kWB + kStrip * 8 +
           sizeof(double) * (kRW + 5) * kNV + sizeof(Scalars) + 16;
  }
  __device__ Smem(char* p, int rows) {
    u = smem_u32(p);
    p += (rows + 2) * kUB;
    w = smem_u32(p);
    p += rows * kWB;
    wtop = smem_u32(p);
    p += kStrip * 8;
    part = reinterpret_cast<double*>(p);
    p += sizeof(double) * kRW * kNV;
    res = reinterpret_cast<double*>(p);
    p += sizeof(double) * kNV * 5;
    sc = reinterpret_cast<Scalars*>(p);
    p += sizeof(Scalars);
    word = reinterpret_cast<int*>(p);
  }
};

// The tallest tile: kMaxRows, or what fits shared memory beside the fixed part
// (the neighbour terms take 12 bytes more per pixel: 87 rows).
constexpr size_t kSmemMax = 232448;
template <bool kNbr>
constexpr int tallest_tile() {
  int rows = kMaxRows;
  while (Smem<kNbr>::bytes(rows) > kSmemMax) --rows;
  return rows;
}
// Rows per warp of the tallest tile: launch_resident has an instance for each
// count up to these.
constexpr int kMaxNr = 7, kMaxNrNbr = 6;
static_assert(tallest_tile<false>() <= kMaxNr * kRW && tallest_tile<true>() <= kMaxNrNbr * kRW,
              "an instance for the tallest tile");

__device__ __forceinline__ float4 lds4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a)
               : "memory");
  return v;
}
__device__ __forceinline__ float2 lds2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts4(uint32_t a, float4 v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z),
               "f"(v.w)
               : "memory");
}
__device__ __forceinline__ void sts2(uint32_t a, float2 v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void sts1(uint32_t a, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
// an address the compiler keeps instead of computing it again from the lane
__device__ __forceinline__ uint32_t keep(uint32_t a) {
  asm volatile("" : "+r"(a));
  return a;
}

// A tile's place in its field and this thread's part of it.
struct Tile {
  int x0, y0, rows;     // first column / row, rows of the tile
  int rb, nrow;         // this warp's first row and row count
  bool up, down, left, right;  // neighbouring tiles
  bool pub_up;          // this warp holds the tile's first row, wanted above
  int pub_down;         // its row that is the tile's last one, wanted below, or -1
  int side;             // this lane's first side slot, or -1
  int xa, xb;
  bool va, vb, ia, ib;  // pixels inside the field; with a right neighbour
  float2 Pa, Pb;        // column phasors
};

// A predicated store, so that the lanes of a warp stay together (branches around
// the stores, and __syncwarp after them in every row, cost 0.1 to 0.3 us a sweep).
__device__ __forceinline__ void st_slot_if(bool p, Slot* out, float2 v, unsigned long long tag) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 d;\n .reg .b128 t;\n setp.ne.s32 p, %4, 0;\n"
      " mov.b64 d, {%1, %2};\n mov.b128 t, {d, %3};\n"
      " @p st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(out),
      "f"(v.x), "f"(v.y), "l"(tag), "r"((int)p)
      : "memory");
}

// Publish row i (of nrow) of a warp: the tile's first and last rows go whole
// to the neighbours above and below, lane 0 and lane 31 carry the side columns.
__device__ __forceinline__ void publish_row(const Tile& t, Slot* out, int lane, int i,
                                            unsigned long long tag, float2 a, float2 b) {
  if (i == 0 && t.pub_up) {
    st_slot_if(t.va, out + 2 * lane, a, tag);
    st_slot_if(t.vb, out + 2 * lane + 1, b, tag);
  }
  if (i == t.pub_down) {
    st_slot_if(t.va, out + kStrip + 2 * lane, a, tag);
    st_slot_if(t.vb, out + kStrip + 2 * lane + 1, b, tag);
  }
  st_slot_if(t.side >= 0, out + t.side + i, lane == 0 ? a : b, tag);
}

__device__ __forceinline__ bool poll_slot(const Slot* p, unsigned long long tag,
                                          unsigned long long& lo, long long limit) {
  unsigned long long hi;
  long long n = 0;
  for (;;) {
    ld_slot(p, lo, hi);
    if (hi == tag) return true;
    if (++n > limit) return false;
  }
}

// Tensor memory as a second register file: what a thread alone reads and writes
// -- g, q and chi of its two pixels in each row, four words each -- moved by
// one instruction per row (the whole warp at once: __syncwarp before it where
// lanes may have parted) and waited for where it is used. With g and q in
// registers (56 of 128 at seven rows) and chi in shared memory the sweep
// spilled, and took 5.4 us at 61 rows, 7.5 at 81 and 8.6 at 97; this takes 4.6,
// 5.4 and 6.0, and the shared memory freed holds 112 rows instead of 97.
constexpr uint32_t kTg = 0, kTq = 4, kTc = 8, kTRow = 12;
__device__ __forceinline__ void tmem_st4(uint32_t a, float2 u, float2 v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a),
               "r"(__float_as_uint(u.x)), "r"(__float_as_uint(u.y)), "r"(__float_as_uint(v.x)),
               "r"(__float_as_uint(v.y))
               : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t a, float2& u, float2& v) {
  uint32_t r0, r1, r2, r3;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(a)
               : "memory");
  u = make_float2(__uint_as_float(r0), __uint_as_float(r1));
  v = make_float2(__uint_as_float(r2), __uint_as_float(r3));
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// the values of a load are there only after the wait
__device__ __forceinline__ void tmem_arrived(float2& u, float2& v) {
  asm volatile("" : "+f"(u.x), "+f"(u.y), "+f"(v.x), "+f"(v.y)::"memory");
}

// This warp's rows: its first row's U and W blocks, and this lane's places in
// them.
struct Rows {
  uint32_t u, ul, yl, w, wl;
  template <bool kNbr>
  __device__ Rows(const Smem<kNbr>& M, int rb, int lane) {
    u = M.u + (rb + 1) * kUB;
    w = M.w + rb * Smem<kNbr>::kWB;
    ul = keep(u + 16 * lane);
    yl = keep(u + kY + 8 * lane);
    wl = keep(w + 16 * lane);
  }
};

// c = L P, or -conj(L P) on a switched line (s = (sw Lx, sw Ly, Lx, Ly))
__device__ __forceinline__ float2 car_rn(float4 s, float2 P) {
  return make_float2(__fmaf_rn(s.x, P.x, -__fmul_rn(s.y, P.y)),
                     __fmaf_rn(s.z, P.y, __fmul_rn(s.w, P.x)));
}

// Row state carried down a warp's rows: u (d, or chi in the gradient) and its
// luma part at this lane's pixels, and the vertical fluxes from the row above.
struct Carry {
  float2 ua, ub;
  float ya, yb;
  float aya, ayb;
  float2 bya, byb;
};

// The differences and weights of a row, for the curvature.
struct RowDiff {
  float4 wa, wb;
  float dxya, dxyb, dyya, dyyb;
  float axa, axb, aya, ayb;
  float2 dxua, dxub, dyua, dyub;
};

// This warp's first row, and the vertical fluxes into it. Outside the field
// u, y and the weights are zero in shared memory, and so are the weights of
// differences that leave it, so no row or column needs a test.
template <bool kNbr>
__device__ __forceinline__ void carry_init(const Smem<kNbr>& M, const Rows& R, int rb, int lane,
                                           Carry& c) {
  const float4 c4 = lds4(R.ul);
  const float2 cy = lds2(R.yl);
  const float4 p4 = lds4(R.ul - kUB);
  const float2 py = lds2(R.yl - kUB);
  float2 wpa, wpb;
  if (rb > 0) {
    const float4 w0 = lds4(R.wl - Smem<kNbr>::kWB), w1 = lds4(R.wl - Smem<kNbr>::kWB + kWb);
    wpa = make_float2(w0.y, w0.w);
    wpb = make_float2(w1.y, w1.w);
  } else {
    const float4 w = lds4(M.wtop + 16 * lane);
    wpa = make_float2(w.x, w.y);
    wpb = make_float2(w.z, w.w);
  }
  c.ua = make_float2(c4.x, c4.y);
  c.ub = make_float2(c4.z, c4.w);
  c.ya = cy.x;
  c.yb = cy.y;
  c.aya = __fmul_rn(wpa.x, c.ya - py.x);
  c.ayb = __fmul_rn(wpb.x, c.yb - py.y);
  c.bya = scale_rn(csub(c.ua, make_float2(p4.x, p4.y)), wpa.y);
  c.byb = scale_rn(csub(c.ub, make_float2(p4.z, p4.w)), wpb.y);
}

// Row i of the operator: -2 (ax(x-1) - ax + ay(y-1) - ay) conj(c)
// + 2 (mu_h (..) + mu_v (..)), m2h = 2 mu_h and m2v = 2 mu_v; moves the carry
// to the next row.
template <bool kI, bool kNbr>
__device__ __forceinline__ void stencil_row(const Rows& R, int i, int lane, float2 ca, float2 cb,
                                            float m2h, float m2v, Carry& c, RowDiff& d, float2& oa,
                                            float2& ob) {
  const float4 n4 = lds4(R.ul + (i + 1) * kUB);
  const float2 ny = lds2(R.yl + (i + 1) * kUB);
  d.wa = lds4(R.wl + i * Smem<kNbr>::kWB);
  d.wb = lds4(R.wl + i * Smem<kNbr>::kWB + kWb);
  const float2 ur = lds2(R.u + i * kUB + kUR), yrl = lds2(R.u + i * kUB + kYR);
  const float4 wul = lds4(R.u + i * kUB + kWL);
  const float2 nua = make_float2(n4.x, n4.y), nub = make_float2(n4.z, n4.w);
  const float ys = __shfl_down_sync(0xffffffffu, c.ya, 1);
  const float2 us = make_float2(__shfl_down_sync(0xffffffffu, c.ua.x, 1),
                                __shfl_down_sync(0xffffffffu, c.ua.y, 1));
  const float y_r = lane == 31 ? yrl.x : ys;
  const float2 u_r = lane == 31 ? ur : us;
  d.dxya = c.yb - c.ya;
  d.dxyb = y_r - c.yb;
  d.dxua = csub(c.ub, c.ua);
  d.dxub = csub(u_r, c.ub);
  d.axa = __fmul_rn(d.wa.x, d.dxya);
  d.axb = __fmul_rn(d.wb.x, d.dxyb);
  const float2 bxb = scale_rn(d.dxub, d.wb.z);
  const float axs = __shfl_up_sync(0xffffffffu, d.axb, 1);
  const float2 bxs = make_float2(__shfl_up_sync(0xffffffffu, bxb.x, 1),
                                 __shfl_up_sync(0xffffffffu, bxb.y, 1));
  const float axl = lane == 0 ? __fmul_rn(wul.x, c.ya - yrl.y) : axs;
  const float2 bxl = lane == 0 ? scale_rn(csub(c.ua, make_float2(wul.z, wul.w)), wul.y) : bxs;
  d.dyya = ny.x - c.ya;
  d.dyyb = ny.y - c.yb;
  d.dyua = csub(nua, c.ua);
  d.dyub = csub(nub, c.ub);
  d.aya = __fmul_rn(d.wa.y, d.dyya);
  d.ayb = __fmul_rn(d.wb.y, d.dyyb);
  const float2 bya = scale_rn(d.dyua, d.wa.w), byb = scale_rn(d.dyub, d.wb.w);
  const float ima = 2.f * ((axl - d.axa) + (c.aya - d.aya));
  const float imb = 2.f * ((d.axa - d.axb) + (c.ayb - d.ayb));
  // horizontal chroma flux differences: in the CG sweep the even pixel's flux
  // is fused into both
  float2 ha, hb;
  if (kI) {
    ha = make_float2(__fmaf_rn(-d.wa.z, d.dxua.x, bxl.x), __fmaf_rn(-d.wa.z, d.dxua.y, bxl.y));
    hb = make_float2(__fmaf_rn(d.wa.z, d.dxua.x, -bxb.x), __fmaf_rn(d.wa.z, d.dxua.y, -bxb.y));
  } else {
    const float2 bxa = scale_rn(d.dxua, d.wa.z);
    ha = csub(bxl, bxa);
    hb = csub(bxa, bxb);
  }
  oa = make_float2(__fmaf_rn(-ima, ca.x, mix(ha.x, m2h, c.bya.x - bya.x, m2v)),
                   __fmaf_rn(ima, ca.y, mix(ha.y, m2h, c.bya.y - bya.y, m2v)));
  ob = make_float2(__fmaf_rn(-imb, cb.x, mix(hb.x, m2h, c.byb.x - byb.x, m2v)),
                   __fmaf_rn(imb, cb.y, mix(hb.y, m2h, c.byb.y - byb.y, m2v)));
  c.ua = nua;
  c.ub = nub;
  c.ya = ny.x;
  c.yb = ny.y;
  c.aya = d.aya;
  c.ayb = d.ayb;
  c.bya = bya;
  c.byb = byb;
}

// Six per-lane values summed over the warp, folding two values into one
// register at each of the first steps: eight FP64 shuffles instead of thirty.
// Lane l ends with the sum of value `which`.
__device__ __forceinline__ void warp_sum6(const double v[kNV], int lane, double& out, int& which) {
  const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
  // step 1: lanes < 16 keep values 0, 2, 4; the others 1, 3, 5
  double a[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const double keep = h16 ? v[2 * j + 1] : v[2 * j];
    const double give = h16 ? v[2 * j] : v[2 * j + 1];
    a[j] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
  }
  // step 2: bit 3 clear keeps a[0] and a[2], set keeps a[1]
  const double keep = h8 ? a[1] : a[0], give = h8 ? a[0] : a[1];
  double b0 = keep + __shfl_xor_sync(0xffffffffu, give, 8);
  double b1 = a[2] + __shfl_xor_sync(0xffffffffu, a[2], 8);
  // step 3: bit 2 clear keeps b0, set keeps b1
  const double k2 = h4 ? b1 : b0, g2 = h4 ? b0 : b1;
  double c = k2 + __shfl_xor_sync(0xffffffffu, g2, 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  out = c;
  which = (h4 ? 4 : h8 ? 2 : 0) + (h16 ? 1 : 0);
}

// n / d to within a rounding or two of FP64, for the scalar step's critical
// path (the FP64 division measured 408 cycles there): Newton's
// iteration for the reciprocal from a single-precision seed, then one residual
// correction of the quotient. Outside the seed's range, the division itself.
__device__ __forceinline__ double quotient(double n, double d) {
  const bool in_range = fabs(d) > 1e-30 && fabs(d) < 1e30;
  if (!__all_sync(__activemask(), in_range)) return n / d;
  double r = (double)__fdividef(1.0f, (float)d);
  r = fma(r, fma(-d, r, 1.0), r);
  r = fma(r, fma(-d, r, 1.0), r);
  const double q = n * r;
  return fma(fma(-d, q, n), r, q);
}

// Waits for a gang's fetch `ord` or a later one (-> {field, fetch}; {-1, ord} when
// the wait ran out): `limits` times `limit` polls, the error flag looked at after
// each. A call, so that this cold loop leaves the registers of the sweep alone
// (64 mixed fields: 34.6 ms with it in line, 34.4 so).
__device__ __noinline__ int2 wait_fetch(const Slot* fetch, int ord, long long limit,
                                        long long limits, const int* err) {
  for (; limits > 0; --limits) {
    for (long long n = 0; n <= limit; ++n) {
      unsigned long long lo, hi;
      ld_slot(fetch, lo, hi);
      if (hi >= (unsigned long long)ord) return make_int2((int)lo, (int)hi);
    }
    if (ld_acquire(err) != 0) break;
  }
  return make_int2(-1, ord);
}

template <int NR, bool kNbr>
__global__ void __launch_bounds__(kRT, 1)
    k_resident(const __grid_constant__ SolverArgs A, const ResidentArgs R) {
  extern __shared__ __align__(16) char resident_smem[];
  const Smem<kNbr> M(resident_smem, R.rows);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int gang = blockIdx.x / R.ctas, cta = blockIdx.x % R.ctas;
  char* const xb = static_cast<char*>(A.xchg);
  const int n_cta = R.gangs * R.ctas;
  // byte offsets into the exchange memory, so that one register each suffices
  const uint32_t my_edges = (uint32_t)edge_bytes() * blockIdx.x;
  // reduction slots of the gang: [set][copy][cta][value]
  const uint32_t red = (uint32_t)edge_bytes() * n_cta + (uint32_t)red_bytes() * gang * R.ctas;
  Slot* const fetch = reinterpret_cast<Slot*>(xb + (edge_bytes() + red_bytes()) * n_cta) + gang;
  int* const done = reinterpret_cast<int*>(
                        reinterpret_cast<Slot*>(xb + (edge_bytes() + red_bytes()) * n_cta) +
                        R.gangs) + gang * R.ctas;
  const float2 z = make_float2(0.f, 0.f);
  // tensor memory: a warp's lane quarter is its number modulo 4, the four warps
  // of a quarter follow one another in columns, a row takes kTRow of them
  constexpr uint32_t kNeed = NR * kTRow * (kRW / 4);
  constexpr uint32_t kCols = kNeed <= 64 ? 64 : kNeed <= 128 ? 128 : kNeed <= 256 ? 256 : 512;
  static_assert(kNeed <= 512, "columns of the SM's tensor memory");
  if (wid == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(M.word + 3)),
                 "r"(kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) M.word[0] = 0;
  __syncthreads();
  const uint32_t tbase = (uint32_t)M.word[3];
  const uint32_t tm = tbase + ((uint32_t)(wid & 3) << 21) + (uint32_t)(wid >> 2) * (NR * kTRow);
  int prev_parts = 0;  // CTAs of the gang's previous field (first CTA only)
  for (int ord = 0;; ++ord) {
    int idx = gang;
    if (ord > 0) {
      if (A.n_fields <= R.gangs) break;
      if (cta == 0) {
        // every CTA of the previous field is through with its slots
        if (tid < prev_parts) {
          long long n = 0;
          while (ld_acquire(done + tid) < ord)
            if (++n > A.phase_wait_limit) {
              M.word[0] = 1;
              break;
            }
        }
        __syncthreads();
        if (tid == 0) {
          M.word[1] = M.word[0] ? A.n_fields : R.gangs + (int)atomicAdd(A.queue, 1ULL);
          M.word[2] = ord;
          __threadfence();
          st_slot(fetch, (unsigned long long)M.word[1], (unsigned long long)ord);
        }
      } else if (tid == 0) {
        // the tag may be ahead: a CTA that a field has no tile for may find
        // the fetch after it
        const int2 next = wait_fetch(fetch, ord, A.phase_wait_limit, M.sc->limits, A.err);
        if (next.x < 0) M.word[0] = 1;
        M.word[1] = next.x;
        M.word[2] = next.y;
      }
      __syncthreads();
      idx = M.word[1];
      ord = M.word[2];
      __syncthreads();
      if (M.word[0]) {
        if (tid == 0) atomicOr(A.err, 1);
        break;
      }
    }
    if (idx >= A.n_fields) break;
    const int fi = __ldg(A.order + idx);
    const FieldDesc& f = A.fields[fi];
    const int fh = f.h, fw = f.w, pitch = f.pitch;
    const int ns = (fw + kStrip - 1) / kStrip;
    int nv = min(R.ctas / ns, (fh + kRW - 1) / kRW);
    const int trows = (fh + nv - 1) / nv;
    nv = (fh + trows - 1) / trows;
    const int parts = ns * nv;
    prev_parts = parts;
    if (cta >= parts) {
      if (tid == 0) M.sc->limits = 1 + f.n_outer * (f.n_inner + 3LL);
      continue;
    }
    Tile t;
    {
      const int v = cta / ns, s = cta - v * ns;
      t.x0 = s * kStrip;
      t.y0 = v * trows;
      t.rows = min(trows, fh - t.y0);
      t.up = v > 0;
      t.down = t.y0 + t.rows < fh;
      t.left = s > 0;
      t.right = s + 1 < ns;
      const int q = t.rows / kRW, rem = t.rows - q * kRW;
      t.rb = wid * q + min(wid, rem);
      t.nrow = q + (wid < rem ? 1 : 0);
      t.pub_up = t.up && t.rb == 0 && t.nrow > 0;
      t.pub_down = t.down && t.nrow > 0 && t.rb + t.nrow == t.rows ? t.nrow - 1 : -1;
      t.side = lane == 0 && t.left    ? 2 * kStrip + t.rb
               : lane == 31 && t.right ? 2 * kStrip + kSideCap + t.rb
                                       : -1;
      t.xa = t.x0 + 2 * lane;
      t.xb = t.xa + 1;
      t.va = t.xa < fw;
      t.vb = t.xb < fw;
      t.ia = t.xa < fw - 1;
      t.ib = t.xb < fw - 1;
      const float2* P = A.col_phasor + f.col_off;
      t.Pa = t.va ? __ldg(P + t.xa) : z;
      t.Pb = t.vb ? __ldg(P + t.xb) : z;
    }
    const int64_t base = f.px_off;
    const float4* const LP = A.line_phasor + f.line_off + t.y0;
    const float mu_h = f.mu_h, mu_v = f.mu_v;
    const bool fixed_w = (f.adj_flags & kAdjFixedW) != 0;
    const bool ext_b = (f.adj_flags & kAdjExtB) != 0;
    const bool has_nbr = kNbr && f.has_nbr;
    const int n_inner = f.n_inner, n_outer = f.n_outer;
    if (tid == 0) {
      const double tol = (double)f.cg_tol;
      M.sc->tol2 = tol * tol;
      M.sc->thr_abs = 1e-10 * (double)fh * (double)fw;
      M.sc->limits = 1;
    }

    // this thread's halo pixel: thread t < 64 above, < 128 below the tile, then
    // the left column, then the right one
    bool hrole = false;
    float2 hc = z, hg = z, hd = z;
    float hS = 0.f;
    uint32_t hsrc = 0;           // the neighbour's slot of set 0
    uint32_t hu = 0, hyp = 0;    // where its d and luma part go in shared memory
    if (tid < kHaloThreads) {
      int hx = 0, hy = 0, nb = 0, sl = 0;
      if (tid < kStrip) {
        hrole = t.up && t.x0 + tid < fw;
        hx = t.x0 + tid;
        hy = t.y0 - 1;
        nb = -ns;
        sl = kStrip + tid;
        hu = M.u + 8 * tid;
        hyp = M.u + kY + 4 * tid;
      } else if (tid < 2 * kStrip) {
        const int j = tid - kStrip;
        hrole = t.down && t.x0 + j < fw;
        hx = t.x0 + j;
        hy = t.y0 + t.rows;
        nb = ns;
        sl = j;
        hu = M.u + (t.rows + 1) * kUB + 8 * j;
        hyp = M.u + (t.rows + 1) * kUB + kY + 4 * j;
      } else if (tid < 2 * kStrip + kSideCap) {
        const int r = tid - 2 * kStrip;
        hrole = t.left && r < t.rows;
        hx = t.x0 - 1;
        hy = t.y0 + r;
        nb = -1;
        sl = 2 * kStrip + kSideCap + r;
        hu = M.u + (r + 1) * kUB + kUL;
        hyp = M.u + (r + 1) * kUB + kYL;
      } else {
        const int r = tid - 2 * kStrip - kSideCap;
        hrole = t.right && r < t.rows;
        hx = t.x0 + kStrip;
        hy = t.y0 + r;
        nb = 1;
        sl = 2 * kStrip + r;
        hu = M.u + (r + 1) * kUB + kUR;
        hyp = M.u + (r + 1) * kUB + kYR;
      }
      if (hrole) {
        const float4 L = __ldg(A.line_phasor + f.line_off + hy);
        const float sw = L.z < 0.f ? -1.f : 1.f;
        hc = car_rn(make_float4(sw * L.x, sw * L.y, L.x, L.y),
                    __ldg(A.col_phasor + f.col_off + hx));
        hS = __ldcg(A.S + base + (int64_t)hy * pitch + hx);
        hsrc = (uint32_t)edge_bytes() * (blockIdx.x + nb) + (uint32_t)sizeof(Slot) * sl;
      }
    }

    const float m2h = 2.f * mu_h, m2v = 2.f * mu_v;
    // zero everything the stencil reads outside the field; line phasors; the
    // field's chi from its plane
    for (int k = tid; k < (t.rows + 2) * (int)(kUB / 16); k += kRT)
      sts4(M.u + 16 * k, make_float4(0.f, 0.f, 0.f, 0.f));
    if (tid < kStrip) sts2(M.wtop + 8 * tid, z);
    if (tid < t.rows) {
      const float4 L = __ldg(LP + tid);
      const float sw = L.z < 0.f ? -1.f : 1.f;
      sts4(M.w + tid * Smem<kNbr>::kWB + kLn, make_float4(sw * L.x, sw * L.y, L.x, L.y));
    }
    const Rows rw(M, t.rb, lane);
    constexpr uint32_t WB = Smem<kNbr>::kWB;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      if (i >= t.nrow) break;
      float4 v = __ldcg(reinterpret_cast<const float4*>(
          A.X[0] + base + (int64_t)(t.y0 + t.rb + i) * pitch + t.xa));
      if (!t.va) v.x = v.y = 0.f;
      if (!t.vb) v.z = v.w = 0.f;
      tmem_st4(tm + kTRow * i + kTc, make_float2(v.x, v.y), make_float2(v.z, v.w));
    }
    tmem_wait_st();
    __syncthreads();
    const unsigned long long tag_hi = (unsigned long long)(ord + 1) << 32;
    unsigned ex = 0;  // exchanges of this field so far
    int set = 0;      // ex % kSets
    int rset_i = 0;   // CG sweeps so far, modulo 2
    float alpha = 0.f, beta = 0.f;
    int pending = 0, iters = 0;
    bool bad = false;

    for (int outer = 0; outer < n_outer && !bad; ++outer) {
      // ---- R: apply the pending step; chi and its luma residual into u, y ----
      ++ex;
      set = set == kSets - 1 ? 0 : set + 1;
      {
        Slot* out = reinterpret_cast<Slot*>(xb + my_edges + set * kSetBytes);
        const unsigned long long tag = tag_hi | ex;
        __syncwarp();
#pragma unroll 1
        for (int i = 0; i < t.nrow; ++i) {
          float2 xa, xb2;
          tmem_ld4(tm + kTRow * i + kTc, xa, xb2);
          tmem_wait_ld();
          tmem_arrived(xa, xb2);
          if (pending) {
            const float4 d4 = lds4(rw.ul + i * kUB);
            xa = cadd(xa, cscale(make_float2(d4.x, d4.y), alpha));
            xb2 = cadd(xb2, cscale(make_float2(d4.z, d4.w), alpha));
            tmem_st4(tm + kTRow * i + kTc, xa, xb2);
          }
          const float4 L = lds4(rw.w + i * WB + kLn);
          const float2 s2 = __ldcg(reinterpret_cast<const float2*>(
              A.S + base + (int64_t)(t.y0 + t.rb + i) * pitch + t.xa));
          const float ya = t.va ? s2.x - re_rn(xa, car_rn(L, t.Pa)) : 0.f;
          const float yb = t.vb ? s2.y - re_rn(xb2, car_rn(L, t.Pb)) : 0.f;
          sts4(rw.ul + i * kUB, make_float4(xa.x, xa.y, xb2.x, xb2.y));
          sts2(rw.yl + i * kUB, make_float2(ya, yb));
          publish_row(t, out, lane, i, tag, xa, xb2);
        }
        tmem_wait_st();
        if (hrole) {
          unsigned long long lo;
          if (!poll_slot(reinterpret_cast<const Slot*>(xb + hsrc + set * kSetBytes), tag, lo,
                         A.phase_wait_limit))
            M.word[0] = 1;
          const float2 hx = unpack2(lo);
          sts2(hu, hx);
          sts1(hyp, hS - re_rn(hx, hc));
        }
      }
      pending = 0;
      __syncthreads();
      // ---- weights (lagged diffusivity), neighbour data term ----
      ++ex;
      set = set == kSets - 1 ? 0 : set + 1;
      {
        Slot* out = reinterpret_cast<Slot*>(xb + my_edges + set * kSetBytes);
        const unsigned long long tag = tag_hi | ex;
        const float eps = f.eps, epsc = f.eps_c, k = f.k_coupling;
        const float e2 = eps * eps, ec2 = epsc * epsc;
#pragma unroll 1
        for (int i = 0; i < t.nrow; ++i) {
          const int r = t.rb + i;
          const int64_t o = (int64_t)(t.y0 + r) * pitch + t.xa;
          float4 wa, wb;
          if (fixed_w) {
            wa = __ldcg(A.W + base + o);
            wb = __ldcg(A.W + base + o + 1);
          } else {
            const bool hn = t.y0 + r + 1 < fh;
            const float4 c4 = lds4(rw.ul + i * kUB), n4 = lds4(rw.ul + (i + 1) * kUB);
            const float2 cy = lds2(rw.yl + i * kUB), ny = lds2(rw.yl + (i + 1) * kUB);
            const float2 ca = make_float2(c4.x, c4.y), cb = make_float2(c4.z, c4.w);
            const float2 na = make_float2(n4.x, n4.y), nb = make_float2(n4.z, n4.w);
            float y_r = __shfl_down_sync(0xffffffffu, cy.x, 1);
            float2 x_r = make_float2(__shfl_down_sync(0xffffffffu, ca.x, 1),
                                     __shfl_down_sync(0xffffffffu, ca.y, 1));
            if (lane == 31) {
              y_r = lds2(rw.u + i * kUB + kYR).x;
              x_r = lds2(rw.u + i * kUB + kUR);
            }
            const float gxa = t.ia ? cy.y - cy.x : 0.f;
            const float gxb = t.ib ? y_r - cy.y : 0.f;
            const float gya = hn ? ny.x - cy.x : 0.f;
            const float gyb = hn ? ny.y - cy.y : 0.f;
            const float2 dxa = t.ia ? csub(cb, ca) : z;
            const float2 dxb = t.ib ? csub(x_r, cb) : z;
            const float2 dya = hn ? csub(na, ca) : z;
            const float2 dyb = hn ? csub(nb, cb) : z;
            wa.x = eps / sqrtf(edge_y(gxa, e2));
            wa.y = eps / sqrtf(edge_y(gya, e2));
            wa.z = epsc / sqrtf(edge_c(sqrtf(norm_xy(dxa)), k, gxa, ec2));
            wa.w = epsc / sqrtf(edge_c(sqrtf(norm_xy(dya)), k, gya, ec2));
            wb.x = eps / sqrtf(edge_y(gxb, e2));
            wb.y = eps / sqrtf(edge_y(gyb, e2));
            wb.z = epsc / sqrtf(edge_c(sqrtf(norm_xy(dxb)), k, gxb, ec2));
            wb.w = epsc / sqrtf(edge_c(sqrtf(norm_xy(dyb)), k, gyb, ec2));
            if (has_nbr) {
              // robust neighbour weights, prior renormalisation and the
              // pointwise data term (variational.cpp:452-516)
              const float nu = f.nu, et2 = f.eps_t * f.eps_t;
              float psa = 1.f, psb = 1.f;
              float4 Ma = make_float4(0.f, 0.f, 0.f, 0.f), Mb = Ma;
              float2 ba = z, bb = z;
              for (int j = 0; j < f.n_nbr; ++j) {
                const float4* NB = A.nbr + f.nbr_off + (int64_t)j * f.plane_px;
                const float4 pa = __ldcg(NB + o);
                const float4 pb = __ldcg(NB + o + 1);
                const float rta = pa.x + (ca.x * pa.y - ca.y * pa.z);
                const float rtb = pb.x + (cb.x * pb.y - cb.y * pb.z);
                const float wta = pa.w * et2 / (rta * rta + et2);
                const float wtb = pb.w * et2 / (rtb * rtb + et2);
                psa += nu * wta * (pa.y * pa.y + pa.z * pa.z);
                psb += nu * wtb * (pb.y * pb.y + pb.z * pb.z);
                const float sa = 2.f * nu * wta, sb = 2.f * nu * wtb;
                Ma.x += sa * pa.y * pa.y;
                Ma.y -= sa * pa.y * pa.z;
                Ma.z += sa * pa.z * pa.z;
                Mb.x += sb * pb.y * pb.y;
                Mb.y -= sb * pb.y * pb.z;
                Mb.z += sb * pb.z * pb.z;
                ba.x += sa * pa.x * pa.y;
                ba.y -= sa * pa.x * pa.z;
                bb.x += sb * pb.x * pb.y;
                bb.y -= sb * pb.x * pb.z;
              }
              wa.x *= psa; wa.y *= psa; wa.z *= psa; wa.w *= psa;
              wb.x *= psb; wb.y *= psb; wb.z *= psb; wb.w *= psb;
              if (!t.va) Ma = make_float4(0.f, 0.f, 0.f, 0.f);
              if (!t.vb) Mb = make_float4(0.f, 0.f, 0.f, 0.f);
              const uint32_t mr = rw.w + i * WB + kM + 8 * lane;
              sts2(mr, make_float2(Ma.x, Mb.x));
              sts2(mr + 256, make_float2(Ma.y, Mb.y));
              sts2(mr + 512, make_float2(Ma.z, Mb.z));
              float2* Bp = A.B + base + o;
              if (t.va) __stcg(Bp, ba);
              if (t.vb) __stcg(Bp + 1, bb);
            }
            if (A.keep_w) {
              if (t.va) __stcg(A.W + base + o, wa);
              if (t.vb) __stcg(A.W + base + o + 1, wb);
            }
          }
          // differences that leave the field do not exist: zero weights
          if (!t.ia) wa.x = wa.z = 0.f;
          if (!t.ib) wb.x = wb.z = 0.f;
          if (!t.va || t.y0 + r + 1 >= fh) wa.y = wa.w = 0.f;
          if (!t.vb || t.y0 + r + 1 >= fh) wb.y = wb.w = 0.f;
          sts4(rw.wl + i * WB, wa);
          sts4(rw.wl + i * WB + kWb, wb);
          if (r == t.rows - 1 && t.down) {
            if (t.va) st_slot(out + kStrip + 2 * lane, pack2(make_float2(wa.y, wa.w)), tag);
            if (t.vb) st_slot(out + kStrip + 2 * lane + 1, pack2(make_float2(wb.y, wb.w)), tag);
          }
          if (lane == 31 && t.right)
            st_slot(out + 2 * kStrip + kSideCap + r, pack2(make_float2(wb.x, wb.z)), tag);
        }
        // the row above's vertical weights, the left column's horizontal ones
        if (hrole && (tid < kStrip || (tid >= 2 * kStrip && tid < 2 * kStrip + kSideCap))) {
          unsigned long long lo;
          if (!poll_slot(reinterpret_cast<const Slot*>(xb + hsrc + set * kSetBytes), tag, lo,
                         A.phase_wait_limit))
            M.word[0] = 1;
          const float2 w2 = unpack2(lo);
          sts2(tid < kStrip ? M.wtop + 8 * tid : M.u + (tid - 2 * kStrip + 1) * kUB + kWL, w2);
        }
      }
      __syncthreads();
      // ---- G: the gradient at chi into tensor memory ----
      ++ex;
      set = set == kSets - 1 ? 0 : set + 1;
      double pgg0 = 0.0;
      {
        Slot* out = reinterpret_cast<Slot*>(xb + my_edges + set * kSetBytes);
        const unsigned long long tag = tag_hi | ex;
        Carry c;
        __syncwarp();
        if (t.nrow > 0) carry_init(M, rw, t.rb, lane, c);
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          if (i >= t.nrow) break;
          const float4 L = lds4(rw.w + i * WB + kLn);
          const float2 cua = c.ua, cub = c.ub;
          RowDiff d;
          float2 oa, ob;
          stencil_row<false, kNbr>(rw, i, lane, car_rn(L, t.Pa), car_rn(L, t.Pb), m2h, m2v, c, d,
                                   oa, ob);
          if (has_nbr) {
            const uint32_t mr = rw.w + i * WB + kM + 8 * lane;
            const float2 m0 = lds2(mr), m1 = lds2(mr + 256), m2 = lds2(mr + 512);
            oa.x += m0.x * cua.x + m1.x * cua.y;
            oa.y += m1.x * cua.x + m2.x * cua.y;
            ob.x += m0.y * cub.x + m1.y * cub.y;
            ob.y += m1.y * cub.x + m2.y * cub.y;
          }
          if (has_nbr || ext_b) {
            const float4 b4 = __ldcg(reinterpret_cast<const float4*>(
                A.B + base + (int64_t)(t.y0 + t.rb + i) * pitch + t.xa));
            oa = cadd(oa, make_float2(b4.x, b4.y));
            ob = cadd(ob, make_float2(b4.z, b4.w));
          }
          if (!t.va) oa = z;
          if (!t.vb) ob = z;
          tmem_st4(tm + kTRow * i + kTg, oa, ob);
          pgg0 += (double)cnorm(oa) + (double)cnorm(ob);
          publish_row(t, out, lane, i, tag, oa, ob);
        }
        tmem_wait_st();
        if (hrole) {
          unsigned long long lo;
          if (!poll_slot(reinterpret_cast<const Slot*>(xb + hsrc + set * kSetBytes), tag, lo,
                         A.phase_wait_limit))
            M.word[0] = 1;
          hg = unpack2(lo);
          hd = make_float2(-hg.x, -hg.y);
        }
      }
      __syncthreads();
      bad = M.word[0] != 0;
      if (bad) break;
      // ---- CG ----
      double gg0 = 0.0;
      for (int k = 0; k < n_inner; ++k) {
        const bool first = k == 0;
        // the pending step and the new direction, own pixels then halo
        __syncwarp();
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          if (i >= t.nrow) break;
          float2 ua, ub, gka, gkb;
          tmem_ld4(tm + kTRow * i + kTg, gka, gkb);
          if (first) {
            tmem_wait_ld();
            tmem_arrived(gka, gkb);
            ua = make_float2(-gka.x, -gka.y);
            ub = make_float2(-gkb.x, -gkb.y);
          } else {
            float2 qka, qkb, xa, xb2;
            tmem_ld4(tm + kTRow * i + kTq, qka, qkb);
            tmem_ld4(tm + kTRow * i + kTc, xa, xb2);
            const float4 d4 = lds4(rw.ul + i * kUB);
            const float2 doa = make_float2(d4.x, d4.y), dob = make_float2(d4.z, d4.w);
            tmem_wait_ld();
            tmem_arrived(gka, gkb);
            tmem_arrived(qka, qkb);
            tmem_arrived(xa, xb2);
            tmem_st4(tm + kTRow * i + kTc, cadd(xa, cscale(doa, alpha)),
                     cadd(xb2, cscale(dob, alpha)));
            gka = cadd(gka, cscale(qka, alpha));
            gkb = cadd(gkb, cscale(qkb, alpha));
            tmem_st4(tm + kTRow * i + kTg, gka, gkb);
            ua = cadd(make_float2(-gka.x, -gka.y), cscale(doa, beta));
            ub = cadd(make_float2(-gkb.x, -gkb.y), cscale(dob, beta));
          }
          const float4 L = lds4(rw.w + i * WB + kLn);
          sts4(rw.ul + i * kUB, make_float4(ua.x, ua.y, ub.x, ub.y));
          sts2(rw.yl + i * kUB,
               make_float2(-re_rn(ua, car_rn(L, t.Pa)), -re_rn(ub, car_rn(L, t.Pb))));
        }
        tmem_wait_st();
        if (hrole) {
          sts2(hu, hd);
          sts1(hyp, -re_rn(hd, hc));
        }
        __syncthreads();
        // ---- q = A d, the curvature and the inner products ----
        ++ex;
        set = set == kSets - 1 ? 0 : set + 1;
        Slot* out = reinterpret_cast<Slot*>(xb + my_edges + set * kSetBytes);
        const unsigned long long tag = tag_hi | ex;
        double pv[kNV] = {0.0, 0.0, 0.0, 0.0, 0.0, pgg0};
        pgg0 = 0.0;
        {
          Carry c;
          __syncwarp();
          if (t.nrow > 0) carry_init(M, rw, t.rb, lane, c);
#pragma unroll
          for (int i = 0; i < NR; ++i) {
            if (i >= t.nrow) break;
            const float4 L = lds4(rw.w + i * WB + kLn);
            const float2 cua = c.ua, cub = c.ub;
            float2 gka, gkb;
            tmem_ld4(tm + kTRow * i + kTg, gka, gkb);
            RowDiff d;
            float2 oa, ob;
            stencil_row<true, kNbr>(rw, i, lane, car_rn(L, t.Pa), car_rn(L, t.Pb), m2h, m2v, c, d,
                                    oa, ob);
            float rH = 0.f;
            if (has_nbr) {
              const uint32_t mr = rw.w + i * WB + kM + 8 * lane;
              const float2 m0 = lds2(mr), m1 = lds2(mr + 256), m2 = lds2(mr + 512);
              oa.x += m0.x * cua.x + m1.x * cua.y;
              oa.y += m1.x * cua.x + m2.x * cua.y;
              ob.x += m0.y * cub.x + m1.y * cub.y;
              ob.y += m1.y * cub.x + m2.y * cub.y;
              rH += 0.5f * (m0.x * cua.x * cua.x + 2.f * m1.x * cua.x * cua.y +
                            m2.x * cua.y * cua.y);
              rH += 0.5f * (m0.y * cub.x * cub.x + 2.f * m1.y * cub.x * cub.y +
                            m2.y * cub.y * cub.y);
            }
            // a pixel's curvature terms ((w Dx Y) Dx Y + ... + mu_v wcy |Dy u|^2) and
            // the inner products; all zero outside the field
            rH += curv_sum(__fmaf_rn(d.axa, d.dxya, __fmul_rn(d.aya, d.dyya)),
                           __fmul_rn(mu_h, d.wa.z), norm_xy(d.dxua), __fmul_rn(mu_v, d.wa.w),
                           norm_yx(d.dyua));
            rH += curv_sum(__fmaf_rn(d.ayb, d.dyyb, __fmul_rn(d.axb, d.dxyb)),
                           __fmul_rn(mu_h, d.wb.z), norm_xy(d.dxub), __fmul_rn(mu_v, d.wb.w),
                           norm_xy(d.dyub));
            tmem_wait_ld();
            tmem_arrived(gka, gkb);
            pv[0] += (double)rH;
            pv[1] += (double)(dot_yx(gka, cua) + dot_yx(gkb, cub));
            pv[2] += (double)(dot_yx(gka, oa) + dot_yx(gkb, ob));
            pv[3] += (double)(norm_yx(oa) + norm_yx(ob));
            pv[4] += (double)(norm_yx(gka) + norm_yx(gkb));
            tmem_st4(tm + kTRow * i + kTq, oa, ob);
            publish_row(t, out, lane, i, tag, oa, ob);
          }
        }
        tmem_wait_st();
        // ---- the CTA's sums ----
        {
          double v;
          int which;
          warp_sum6(pv, lane, v, which);
          if ((lane & 3) == 0) M.part[which * kRW + wid] = v;
        }
        __syncthreads();
        rset_i ^= 1;
        Slot* const rset = reinterpret_cast<Slot*>(xb + red) + rset_i * kRep * kLine * R.ctas;
        if (wid == kRW - 1) {
          // lane 4 v + j adds four warps' sums of value v, its quad the sixteen;
          // it then writes slot v of copy j
          const int v = lane >> 2;
          double a = 0.0;
          if (v < kNV) {
            const double2* pp = reinterpret_cast<const double2*>(M.part + lane * 4);
            const double2 p0 = pp[0], p1 = pp[1];
            a = (p0.x + p0.y) + (p1.x + p1.y);
          }
          a += __shfl_xor_sync(0xffffffffu, a, 1);
          a += __shfl_xor_sync(0xffffffffu, a, 2);
          st_slot(rset + ((lane & 3) * R.ctas + cta) * kLine + v,
                  (unsigned long long)__double_as_longlong(a), tag);
        }
        // ---- collect: edge q's (threads < 352), sums (warps 11..15) ----
        float2 hq = z;
        if (hrole) {
          unsigned long long lo;
          if (!poll_slot(reinterpret_cast<const Slot*>(xb + hsrc + set * kSetBytes), tag, lo,
                         A.phase_wait_limit))
            M.word[0] = 1;
          hq = unpack2(lo);
        }
        if (wid >= kRedWarp0) {
          const int src = tid - kHaloThreads;
          double sv[kNV] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
          if (src < parts) {
            const Slot* line = rset + ((cta & (kRep - 1)) * R.ctas + src) * kLine;
            unsigned long long lo[kNV], hi[kNV];
            bool ok = poll_slot(line, tag, lo[0], A.phase_wait_limit);
            long long n = 0;
            for (;;) {
              bool all = true;
#pragma unroll
              for (int j = 1; j < kNV; ++j) ld_slot(line + j, lo[j], hi[j]);
#pragma unroll
              for (int j = 1; j < kNV; ++j) all &= hi[j] == tag;
              if (all || !ok) break;
              if (++n > A.phase_wait_limit) ok = false;
            }
            if (!ok) M.word[0] = 1;
#pragma unroll
            for (int j = 0; j < kNV; ++j) sv[j] = __longlong_as_double((long long)lo[j]);
          }
          __syncwarp();
          {
            double v;
            int which;
            warp_sum6(sv, lane, v, which);
            if ((lane & 3) == 0) M.res[which * 5 + wid - kRedWarp0] = v;
          }
          // the five collecting warps meet, one of them does the scalar step
          // (variational.cpp:519-549; k_solver.cu complete_phase)
          asm volatile("bar.sync 1, 160;" ::: "memory");
          if (wid == kRedWarp0) {
            const double* rp = M.res + min(lane, kNV - 1) * 5;
            const double tot = ((rp[0] + rp[1]) + (rp[2] + rp[3])) + rp[4];
            const double H = __shfl_sync(0xffffffffu, tot, 0), gd = __shfl_sync(0xffffffffu, tot, 1),
                         gq = __shfl_sync(0xffffffffu, tot, 2), qq = __shfl_sync(0xffffffffu, tot, 3),
                         ggk = __shfl_sync(0xffffffffu, tot, 4),
                         g0 = __shfl_sync(0xffffffffu, tot, 5);
            if (first) gg0 = g0;
            // both quotients at once: alpha's on lane 0, 1 / ||g||^2 on lane 1
            const double quo = quotient(lane == 1 ? 1.0 : -0.5 * gd,
                                        lane == 1 ? fmax(ggk, 1e-30) : H);
            const double inv = __shfl_sync(0xffffffffu, quo, 1);
            if (lane == 0) {
              const double thr_rel = M.sc->tol2 * gg0, thr_abs = M.sc->thr_abs;
              const float al = (float)quo;
              const double a = (double)al, gn = ggk + 2.0 * a * gq + a * a * qq;
              const double bound = 1e-5 * (ggk + 2.0 * fabs(a * gq) + a * a * qq);
              // the norm measured by this sweep ends the pass with chi final; a
              // predicted one with its step pending
              const bool done_now = (!first && (ggk < thr_rel || ggk < thr_abs)) || H <= 1e-12;
              M.sc->alpha = done_now ? 0.f : al;
              M.sc->beta = done_now ? 0.f : (float)(gn * inv);
              M.sc->pending = !done_now;
              M.sc->stop = done_now || gn + bound < thr_rel || gn + bound < thr_abs;
            }
          }
        }
        __syncthreads();
        bad = M.word[0] != 0;
        if (bad) break;
        alpha = M.sc->alpha;
        beta = M.sc->beta;
        pending = M.sc->pending;
        iters += pending;
        if (M.sc->stop) break;
        if (hrole) {
          hg = cadd(hg, cscale(hq, alpha));
          hd = cadd(make_float2(-hg.x, -hg.y), cscale(hd, beta));
        }
      }
      // u and y are rewritten by the next pass; every thread is past its
      // reads of them (the barrier after the sums). No wait of the next pass may
      // run out before all have read that none had: the warps leave (and free the
      // tensor memory) together or not at all.
      __syncthreads();
    }
    if (bad) {
      if (tid == 0) atomicOr(A.err, 1);
      break;
    }
    // ---- F: apply the pending step, luma = S - Re[chi c], outputs ----
#pragma unroll 1
    for (int i = 0; i < t.nrow; ++i) {
      const int r = t.rb + i, y = t.y0 + r;
      const int64_t o = (int64_t)y * pitch + t.xa;
      float2 xa, xb2;
      __syncwarp();
      tmem_ld4(tm + kTRow * i + kTc, xa, xb2);
      tmem_wait_ld();
      tmem_arrived(xa, xb2);
      if (pending) {
        const float4 d4 = lds4(rw.ul + i * kUB);
        xa = cadd(xa, cscale(make_float2(d4.x, d4.y), alpha));
        xb2 = cadd(xb2, cscale(make_float2(d4.z, d4.w), alpha));
      }
      const float4 L = lds4(rw.w + i * WB + kLn);
      const float2 s2 = __ldcg(reinterpret_cast<const float2*>(A.S + base + o));
      const float ya = s2.x - re_rn(xa, car_rn(L, t.Pa));
      const float yb = s2.y - re_rn(xb2, car_rn(L, t.Pb));
      if (t.va && t.vb) {
        __stcg(reinterpret_cast<float4*>(A.X[0] + base + o), make_float4(xa.x, xa.y, xb2.x, xb2.y));
        __stcg(reinterpret_cast<float2*>(A.Y + base + o), make_float2(ya, yb));
      } else if (t.va) {
        __stcg(A.X[0] + base + o, xa);
        __stcg(A.Y + base + o, ya);
      }
      // the caller's buffers promise no alignment beyond a float's
      const int64_t od = (int64_t)y * fw + t.xa;
      if (f.out_c) {
        float* oc = reinterpret_cast<float*>(f.out_c) + 2 * od;
        const uintptr_t ac = reinterpret_cast<uintptr_t>(oc);
        if (t.va && t.vb && (ac & 15) == 0) {
          __stcs(reinterpret_cast<float4*>(oc), make_float4(xa.x, xa.y, xb2.x, xb2.y));
        } else if ((ac & 7) == 0) {
          if (t.va) __stcs(reinterpret_cast<float2*>(oc), xa);
          if (t.vb) __stcs(reinterpret_cast<float2*>(oc) + 1, xb2);
        } else {
          if (t.va) {
            __stcs(oc, xa.x);
            __stcs(oc + 1, xa.y);
          }
          if (t.vb) {
            __stcs(oc + 2, xb2.x);
            __stcs(oc + 3, xb2.y);
          }
        }
      }
      if (f.out_y) {
        if (t.va && t.vb && ((reinterpret_cast<uintptr_t>(f.out_y + od) & 7) == 0)) {
          __stcs(reinterpret_cast<float2*>(f.out_y + od), make_float2(ya, yb));
        } else {
          if (t.va) __stcs(f.out_y + od, ya);
          if (t.vb) __stcs(f.out_y + od + 1, yb);
        }
      }
    }
    if (cta == 0 && tid == 0) A.ctl[fi].cg_iters = iters;
    // this CTA has consumed every slot of the field; shared memory is free too
    __syncthreads();
    if (tid == 0) st_release(done + cta, ord + 1);
  }
  __syncthreads();
  __syncwarp();
  if (wid == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase),
                 "r"(kCols));
}

template <bool kNbr, int... NR>
cudaError_t configure() {
  cudaError_t e = cudaSuccess;
  ((e = e != cudaSuccess ? e
                         : cudaFuncSetAttribute(k_resident<NR, kNbr>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)kSmemMax)),
   ...);
  return e;
}

template <int NR, bool kNbr>
cudaError_t launch_one(const SolverArgs& a, const ResidentPlan& p, cudaStream_t st) {
  const size_t smem = Smem<kNbr>::bytes(p.rows);
  SolverArgs sa = a;
  ResidentArgs ra;
  ra.gangs = p.gangs;
  ra.ctas = p.ctas;
  ra.rows = p.rows;
  void* params[] = {&sa, &ra};
  return cudaLaunchCooperativeKernel((const void*)k_resident<NR, kNbr>, dim3(p.gangs * p.ctas),
                                     dim3(kRT), params, smem, st);
}

}  // namespace

cudaError_t configure_resident_kernels() {
  const cudaError_t e = configure<false, 1, 2, 3, 4, 5, kMaxNr>();
  return e != cudaSuccess ? e : configure<true, 1, 2, 3, 5, kMaxNrNbr>();
}

size_t resident_xchg_bytes(int sm_count) {
  // edge and reduction slots per CTA, a fetch slot per gang, a counter per CTA
  return (edge_bytes() + red_bytes()) * (size_t)sm_count + sizeof(Slot) * sm_count +
         sizeof(int) * sm_count;
}

ResidentPlan plan_resident(const SolveShape* shapes, int n, bool nbr, bool diag, int sm_count) {
  ResidentPlan best;
  if (diag || n <= 0) return best;
  const int max_rows = nbr ? tallest_tile<true>() : tallest_tile<false>();
  double best_t = 0.0;
  std::vector<double> cost(n), load;
  for (int g = 1; g <= std::min(n, sm_count); ++g) {
    const int c = std::min(sm_count / g, kMaxCtas);
    int rows = 0;
    bool fits = true;
    for (int i = 0; i < n && fits; ++i) {
      const int ns = (shapes[i].w + kStrip - 1) / kStrip;
      if (c / ns < 1) {
        fits = false;
        break;
      }
      const int nv = std::min(c / ns, (shapes[i].h + kRW - 1) / kRW);
      const int tr = (shapes[i].h + nv - 1) / nv;
      rows = std::max(rows, tr);
      fits = tr <= max_rows;
      // a sweep costs its exchange plus its rows (us, measured: 3.6 at 21 rows, 4.1 at
      // 41, 4.6 at 61, 5.4 at 81, 6.0 at 97)
      const double sweep = 3.0 + 0.033 * tr;
      cost[i] = shapes[i].n_outer * (shapes[i].n_inner + 3.0) * sweep + 5.0;
    }
    if (!fits) break;
    // the gangs take the fields heaviest first, each the next when it is free
    std::sort(cost.begin(), cost.end(), [](double x, double y) { return x > y; });
    load.assign(g, 0.0);
    for (double t : cost) {
      std::pop_heap(load.begin(), load.end(), std::greater<double>());
      load.back() += t;
      std::push_heap(load.begin(), load.end(), std::greater<double>());
    }
    const double t = *std::max_element(load.begin(), load.end());
    if (best.gangs == 0 || t < best_t) {
      best_t = t;
      best.gangs = g;
      best.ctas = c;
      best.rows = rows;
    }
  }
  best.us = best_t;
  if (best.gangs) best.nr = (best.rows + kRW - 1) / kRW;
  return best;
}

cudaError_t launch_resident(const SolverArgs& a, const ResidentPlan& p, bool nbr,
                            cudaStream_t st) {
  if (nbr) {
    if (p.nr <= 1) return launch_one<1, true>(a, p, st);
    if (p.nr <= 2) return launch_one<2, true>(a, p, st);
    if (p.nr <= 3) return launch_one<3, true>(a, p, st);
    if (p.nr <= 5) return launch_one<5, true>(a, p, st);
    if (p.nr <= kMaxNrNbr) return launch_one<kMaxNrNbr, true>(a, p, st);
    return cudaErrorInvalidValue;
  }
  if (p.nr <= 1) return launch_one<1, false>(a, p, st);
  if (p.nr <= 2) return launch_one<2, false>(a, p, st);
  if (p.nr <= 3) return launch_one<3, false>(a, p, st);
  if (p.nr <= 4) return launch_one<4, false>(a, p, st);
  if (p.nr <= 5) return launch_one<5, false>(a, p, st);
  if (p.nr <= kMaxNr) return launch_one<kMaxNr, false>(a, p, st);
  return cudaErrorInvalidValue;
}

}  // namespace hvdg
