// Red/black SOR with a domain's lambda resident in shared memory: one
// cooperative launch runs a whole solve (start stage, pre-phase, reference
// loop with its stopping rules) of every domain of a list.
//
// A domain is cut into nty x ntz tiles (full x rows, ty rows, tz planes), one
// per CTA of a group; the CTAs of a group advance one domain together, the
// groups of a launch take domains from a queue. A tile's lambda (both colours)
// stays in shared memory from the first iteration to the last, with the wall
// mask and as much of R as fits beside it (the rest streams from L2). The
// streaming sweeps (qesb_sor_zm.cuh) move 17 B per cell and iteration through
// HBM or L2 and pay two launches an iteration; here an iteration costs
// shared-memory reads, arithmetic and the exchange of the tiles' faces.
//
// Half-sweep. Every warp updates its share of the tile and publishes the cells
// of the tile's faces as it stores them; then the threads collect the
// neighbours' faces into the halo around the tile, and one CTA barrier ends the
// half-sweep. A published cell is 8 bytes: the value and the half-sweep's
// number, so the reader polls the data itself and no fence, flag or barrier lies
// between a store and its use. A slot of colour c is written again two
// half-sweeps later; its writer has then used a face that the reader published
// after reading the slot, so nothing unread is lost.
//
// Compute. A lane updates 4 cells of a row and marches along y, so the rows
// below and above rotate through registers and a plane's coefficients stay
// there. A warp's lanes cover planes of one parity: the x parity of the row is
// then the same in every lane, and the west/east neighbours are fixed
// registers. Here all cells are taken as open on every face; the few that are
// not (beside walls) have been updated before, from a list, a cell per lane, and
// keep what they hold: a city's row of 128 cells nearly always meets a wall, and
// selecting six coefficients for every cell of it tripled the instructions. The
// row code has no divergent branch: those cost more than its sums.
//
// Measured (B200, us an iteration of one domain, against the fastest streaming
// shape): 40 x 40 x 20 5.6 (8.6), 100 x 100 x 50 7.2 (12.7), 200 x 180 x 60 10.2
// (18.6), 256 x 256 x 64 13.7 (21.0). A half-sweep of the last takes about 7 us;
// the FP32 operations of its rows alone would take 0.9. 16 warps an SM issue in 47 %
// of the cycles (rows: fixed and shared-memory latency); a third of their time is
// the CTA barriers and the loads of faces and of streamed R: 47 KB in and out of L2
// per CTA and the wait for the slowest neighbour. Small domains are all latency:
// two exchanges of about 1.2 us each.
//
// The kernel sits at the limit of 128 registers a thread: code added beside the
// rows (two more slots of the window rule by remainder, the alias path in the
// wall-mask kernel) has cost 4 % at 100 x 100 x 50.
//
// FULL: every cell has its own six coefficients (no wall mask): they stream from
// L2, 28 B a cell with omega / (their sum), while lambda still stays here. An
// iteration of 151 x 133 x 61 takes 12 us, with the four launches of the
// streaming loop (both colours, mirror, poll; 68 B a cell) 33.
//
// The arithmetic is the other sweeps' (Solver_CPU_RB.cpp:118-125, the same
// operation order), so results are bit-identical. The ground mirror
// lambda(k=0) <- lambda(k=1) of every iteration (Solver_CPU_RB.cpp:155-162)
// is one more store: a cell of plane 1 is written below itself too, where only
// its own next update reads it. Plane 0 of the array is written once, after the
// launch (k_res_to_pad).
//
// Stopping. max|dlambda| of an iteration is exact in FP64 (err[it]). The loop
// condition of Solver_CPU_RB.cpp:106 must be decided before the next red
// half-sweep overwrites lambda. A red cell that changed by more than tol proves
// that the iteration does not stop; any CTA's proof lets every CTA go on. Only
// iterations without one (near the end) meet at a barrier to read the full
// maximum. A NaN proves nothing, so it ends the loop once it has reached every
// tile, or at itermax; the iteration reported is the first whose maximum is NaN.
#include <cuda_runtime.h>

#include "qesb_sor_res.cuh"

namespace qesb {

constexpr int kResWalls = 512;  // wall cells of a colour in shared memory
constexpr int kResSegs = 32;    // most runs of rows
constexpr float kResTinyF = 1.40129846e-45f;  // the smallest positive (subnormal) float

__device__ __forceinline__ void res_arrive(unsigned long long *p)
{
  asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(p) : "memory");
}
__device__ __forceinline__ unsigned long long res_load(const unsigned long long *p)
{
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned res_load32(const unsigned *p)
{
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool res_fault(ResCtl *ctl) { return *reinterpret_cast<volatile int *>(&ctl->fault) != 0; }
// Waits (bounded) until *p >= want; false when it gave up or another CTA did.
__device__ __forceinline__ bool res_wait(const unsigned long long *p, unsigned long long want, uint32_t limit,
                                         ResCtl *ctl)
{
  for (uint32_t n = 0; n < limit; ++n) {
    if (res_load(p) >= want) return true;
    if ((n & 1023u) == 1023u && res_fault(ctl)) return false;
  }
  atomicExch(&ctl->fault, 1);
  return false;
}

// The same for the group's next domain. A CTA that has no tile of the current
// one waits here for as long as its solve lasts: the count starts again whenever
// that solve's iteration number (beat, null before the first domain) has moved.
__device__ __forceinline__ bool res_wait_next(const unsigned long long *p, unsigned long long want, const unsigned *beat,
                                              uint32_t limit, ResCtl *ctl)
{
  unsigned seen = 0;
  for (uint32_t n = 0; n < limit; ++n) {
    if (res_load(p) >= want) return true;
    if (beat) {
      const unsigned b = *reinterpret_cast<const volatile unsigned *>(beat);
      if (b != seen) {
        seen = b;
        n = 0;
      }
    }
    if ((n & 1023u) == 1023u && res_fault(ctl)) return false;
  }
  atomicExch(&ctl->fault, 1);
  return false;
}

__device__ __forceinline__ float max_nan(float a, float b)
{
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// compile-time x parity
template <int V>
struct ResPar {
  static constexpr int v = V;
};

extern __shared__ __align__(128) unsigned char res_sm[];  // all offsets below are bytes

template <class T>
__device__ __forceinline__ T &sm(int off) { return *reinterpret_cast<T *>(res_sm + off); }
// a group of 4 cells
__device__ __forceinline__ float4 lds4(int off) { return sm<float4>(off); }
__device__ __forceinline__ void sts4(int off, float4 v) { sm<float4>(off) = v; }

// A CTA's tile and its shared memory, fixed for a domain.
struct ResTile {
  int X, Y, Z, PQ;
  int P, PS, CP;    // bytes per shared row, plane and colour
  int nq4, ty, tz, j0, k0;
  int tym, tzm;     // the domain's largest tile
  unsigned magic, epoch;
  unsigned base0;   // common face mask of the first plane (the others': 63)
  int rp;           // planes of R held in shared memory (the first rp)
  bool pubS, pubN, pubB, pubT;  // a neighbour reads row 0 / row ty - 1 / plane 0 / plane tz - 1
  long CS;
  int own;          // [2][tz + 2][ty + 2][P] lambda with a halo of one; here: cell (k, j) = (0, 0) of colour 0
  int wls;          // [2][kResWalls] wall cells, two words each (the rest of the list stays in global memory)
  int kp;           // [2][tz][ty][P] bytes: 0xff: the rows keep the cell (a wall or boundary cell)
  int xt;           // [2 (tz + ty) nq4] the halo's groups: {place in the exchange slots, place in the tile}
  int xn;           // how many of them a neighbour feeds
  int rs;           // [2][rp][ty][P]
  int cf;           // [tz][8]: e f g h m n, omega / (their sum), 1 - omega
  int inv;          // [tz][64]
  // tasks: 32 lanes' columns (planes of one parity x groups of 4 cells) over one of nseg runs of rows
  int lanes[2], chunks[2], nseg, ntask;
  unsigned segmagic;  // ceil(2^32 / nseg)
  bool split;         // a colour row spans tasks
  float *lam;
  const float *R;
  const uint8_t *mask;
  const float *co;  // full coefficients, or null
  __device__ __forceinline__ long gidx(int c, int k, int j, int q4) const
  {
    return c * CS + ((long)(k0 + k) * Y + (j0 + j)) * PQ + 4 * q4;
  }
  __device__ __forceinline__ int at(int c, int k, int j, int q4) const { return own + c * CP + k * PS + j * P + 16 * q4; }
  __device__ __forceinline__ int row_of(int x) const { return nq4 == 1 ? x : (int)__umulhi((unsigned)x, magic); }
};

// A thread's running max|dlambda| of the current iteration.
struct ResMax {
  float thr;    // largest change seen by the warp (rounded), at least the smallest subnormal
  double dmax;  // this thread's exact maximum among the cells that reached it
};

// A plane's coefficients: e f g h m n, omega / (their sum), 1 - omega.
struct ResCoef {
  float e, f, g, h, m, n, inv, c1;
};

// 4 cells of a row whose x parity is I0 (cell u is i = 2 (4*q4 + u) + I0) with the plane's coefficients: C the
// other colour's cells of the row at the same places, `edge` the one before (I0 = 0) or after (I0 = 1) them.
template <int I0>
__device__ __forceinline__ float4 res_row(const ResCoef &K, float4 C, float edge, float4 N, float4 S, float4 T,
                                          float4 B, float4 O, float4 R)
{
  const float x0 = I0 ? C.x : edge, x1 = I0 ? C.y : C.x, x2 = I0 ? C.z : C.y, x3 = I0 ? C.w : C.z, x4 = I0 ? edge : C.w;
  auto cell = [&](float xe, float xw, float yn, float ys, float zt, float zb, float r, float o) {
    return K.inv * (K.e * xe + K.f * xw + K.g * yn + K.h * ys + K.m * zt + K.n * zb - r) + K.c1 * o;
  };
  return make_float4(cell(x1, x0, N.x, S.x, T.x, B.x, R.x, O.x), cell(x2, x1, N.y, S.y, T.y, B.y, R.y, O.y),
                     cell(x3, x2, N.z, S.z, T.z, B.z, R.z, O.z), cell(x4, x3, N.w, S.w, T.w, B.w, R.w, O.w));
}

// publishes a group of 4 cells: each with the half-sweep's number
__device__ __forceinline__ void res_publish(ulonglong2 *d, unsigned mark, float4 v)
{
  const float m = __uint_as_float(mark);
  asm volatile("{.reg .b64 a, b; mov.b64 a, {%1, %3}; mov.b64 b, {%2, %3}; st.relaxed.gpu.global.v2.b64 [%0], {a, b};}" ::"l"(d), "f"(v.x), "f"(v.y), "f"(m) : "memory");
  asm volatile("{.reg .b64 a, b; mov.b64 a, {%1, %3}; mov.b64 b, {%2, %3}; st.relaxed.gpu.global.v2.b64 [%0], {a, b};}" ::"l"(d + 1), "f"(v.z), "f"(v.w), "f"(m) : "memory");
}
// a where the byte b (0 .. 3) of m is 0xff, else v
template <int B>
__device__ __forceinline__ float res_pick(uint32_t m, float a, float v)
{
  const uint32_t k = __byte_perm(m, 0, 0x1111u * B);  // the byte four times
  return __uint_as_float((__float_as_uint(a) & k) | (__float_as_uint(v) & ~k));
}

// The same with each cell's own coefficients: at q = 0 .. 6 the split arrays of e f g h m n and omega / (their sum)
// lie cs floats apart.
template <int I0>
__device__ __forceinline__ float4 res_row_full(const float *q, long cs, float c1, float4 C, float edge, float4 N, float4 S,
                                               float4 T, float4 B, float4 O, float4 R)
{
  auto ld = [&](int i) { return __ldg(reinterpret_cast<const float4 *>(q + i * cs)); };
  const float4 e = ld(0), f = ld(1), g = ld(2), h = ld(3), m = ld(4), n = ld(5), v = ld(6);
  const float x0 = I0 ? C.x : edge, x1 = I0 ? C.y : C.x, x2 = I0 ? C.z : C.y, x3 = I0 ? C.w : C.z, x4 = I0 ? edge : C.w;
  return make_float4(
      v.x * (e.x * x1 + f.x * x0 + g.x * N.x + h.x * S.x + m.x * T.x + n.x * B.x - R.x) + c1 * O.x,
      v.y * (e.y * x2 + f.y * x1 + g.y * N.y + h.y * S.y + m.y * T.y + n.y * B.y - R.y) + c1 * O.y,
      v.z * (e.z * x3 + f.z * x2 + g.z * N.z + h.z * S.z + m.z * T.z + n.z * B.z - R.z) + c1 * O.z,
      v.w * (e.w * x4 + f.w * x3 + g.w * N.w + h.w * S.w + m.w * T.w + n.w * B.w - R.w) + c1 * O.w);
}

__device__ __forceinline__ void res_exact(ResMax &mx, float a, float b)
{
  const double y = fabs((double)a - (double)b);
  if (y > mx.dmax || y != y) mx.dmax = y;
}
// A change d that reaches the warp's largest so far? The rounded difference is
// monotone in the exact one, so the exact maximum is among the cells whose
// rounded difference is the largest. All lanes; true: the lane's cells are to be
// looked at in FP64.
__device__ __forceinline__ bool res_reaches(ResMax &mx, float d)
{
  if (!__any_sync(0xffffffffu, !(d < mx.thr))) return false;
  mx.thr = fmaxf(mx.thr, __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(d == d ? d : 0.0f))));
  return !(d < mx.thr);
}

// One task: the lanes' columns of colour c over a run of rows. xb: this CTA's exchange slots of colour c.
template <bool FULL>
__device__ __forceinline__ void res_task(const ResTile &t, const short *segs, int task, int c, ulonglong2 *xb,
                                         unsigned mark, ResMax &mx)
{
  const int lane = threadIdx.x & 31;
  const int ch = t.nseg == 1 ? task : (int)__umulhi((unsigned)task, t.segmagic), seg = task - ch * t.nseg;
  const int p = ch >= t.chunks[0];
  const int idx = (ch - (p ? t.chunks[0] : 0)) * 32 + lane;
  const bool ok = idx < t.lanes[p];
  const int x = ok ? idx : 0;
  const int kk = t.row_of(x), q4 = x - kk * t.nq4, k = p + 2 * kk;
  const int ja = segs[seg], jb = segs[seg + 1];
  const int jS = t.pubS ? 0 : -1, jN = t.pubN ? t.ty - 1 : -1, PQ = t.PQ;  // rows a neighbour reads
  const int P = t.P, PS = t.PS;
  int o = t.at(c, k, ja, q4);                     // own cells
  const int dx = c ? -t.CP : t.CP;                // own -> other colour
  const bool rres = __all_sync(0xffffffffu, k < t.rp);  // R from shared memory
  const int rrow = (c * t.tz + k) * t.ty + ja;
  int ko = t.kp + 4 * (rrow * t.nq4 + q4);        // keep bytes
  const int kd = 4 * t.nq4;
  int rx = t.rs + (rrow - c * (t.tz - t.rp) * t.ty) * P + 16 * q4;  // R in shared memory: [2][rp][ty][P]
  const float *gR = t.R + t.gidx(c, k, ja, q4);
  ResCoef K;
  const float *gC = nullptr;
  long cs = 0;
  if (FULL) {
    gC = t.co + t.gidx(c, k, ja, q4);
    cs = 2 * t.CS;
    K.c1 = sm<float>(t.cf + 28);
  } else {
    K = sm<ResCoef>(t.cf + 32 * k);
    if (k == 0 && t.base0 == 31u) K.n = 0.0f;
  }
  const bool ground = ok && t.k0 == 1 && k == 0;
  const bool pB = ok && t.pubB && k == 0, pT = ok && t.pubT && k == t.tz - 1;
  const bool anyp = __any_sync(0xffffffffu, pB || pT), split = t.split;
  const uint32_t out = ok ? 0u : 0xffffffffu;     // lanes without a column keep everything
  float4 S = lds4(o + dx - P), C = lds4(o + dx), Rn = C;
  if (!rres) Rn = __ldg(reinterpret_cast<const float4 *>(gR));
  const int par = __shfl_sync(0xffffffffu, (c + t.j0 + ja + t.k0 + k) & 1, 0);  // of row ja, the same in every lane
  auto publish = [&](int j, float4 V) {
    ulonglong2 *d = xb + 2 * (2 * t.tzm * t.nq4 + j * t.nq4 + q4);
    if (pB) res_publish(d, mark, V);
    if (pT) res_publish(d + 2 * t.tym * t.nq4, mark, V);
    if (j == jS && ok) res_publish(xb + 2 * (k * t.nq4 + q4), mark, V);
    if (j == jN && ok) res_publish(xb + 2 * ((t.tzm + k) * t.nq4 + q4), mark, V);
  };
  auto update = [&](auto tag, float4 C_, float4 N_, float4 S_, int o_, float4 R_, uint32_t km, float4 &O_, int dc = 0) {
    constexpr int I0 = decltype(tag)::v;
    const float4 T = lds4(o_ + dx + PS), B = lds4(o_ + dx - PS);
    O_ = lds4(o_);
    // from the next lane, or from shared memory where the row goes on in another task
    float edge = I0 ? __shfl_down_sync(0xffffffffu, C_.x, 1) : __shfl_up_sync(0xffffffffu, C_.w, 1);
    if (split) {
      const float e = sm<float>(o_ + dx + (I0 ? 16 : -4));
      edge = lane == (I0 ? 31 : 0) ? e : edge;
    }
    float4 V = FULL ? res_row_full<I0>(gC + dc, cs, K.c1, C_, edge, N_, S_, T, B, O_, R_)
                    : res_row<I0>(K, C_, edge, N_, S_, T, B, O_, R_);
    V.x = res_pick<0>(km, O_.x, V.x);
    V.y = res_pick<1>(km, O_.y, V.y);
    V.z = res_pick<2>(km, O_.z, V.z);
    V.w = res_pick<3>(km, O_.w, V.w);
    return V;
  };
  auto change = [&](float4 V, float4 O_) {
    return max_nan(max_nan(fabsf(V.x - O_.x), fabsf(V.y - O_.y)), max_nan(fabsf(V.z - O_.z), fabsf(V.w - O_.w)));
  };
  auto exact = [&](float4 V, float4 O_) {
    res_exact(mx, V.x, O_.x), res_exact(mx, V.y, O_.y);
    res_exact(mx, V.z, O_.z), res_exact(mx, V.w, O_.w);
  };
  auto rows2 = [&](int j, auto tag) {
    constexpr int I0 = decltype(tag)::v;
    const float4 N0 = lds4(o + dx + P), N1 = lds4(o + dx + 2 * P);
    float4 R0 = Rn, R1;
    if (rres) {
      R0 = lds4(rx);
      R1 = lds4(rx + P);
    } else {
      R1 = __ldg(reinterpret_cast<const float4 *>(gR + PQ));
      gR += 2 * PQ;
      if (j + 2 < jb) Rn = __ldg(reinterpret_cast<const float4 *>(gR));
    }
    const uint32_t k0 = sm<uint32_t>(ko) | out, k1 = sm<uint32_t>(ko + kd) | out;
    float4 O0, O1;
    const float4 V0 = update(ResPar<I0>{}, C, N0, S, o, R0, k0, O0);
    const float4 V1 = update(ResPar<1 - I0>{}, N0, N1, C, o + P, R1, k1, O1, PQ);
    if (ok) {
      sts4(o, V0);
      sts4(o + P, V1);
    }
    if (ground) {  // the ground mirror: the cell below, of the other colour
      sts4(o + dx - PS, V0);
      sts4(o + dx - PS + P, V1);
    }
    if (anyp || j == jS) publish(j, V0);
    if (anyp || j + 1 == jN) publish(j + 1, V1);
    if (res_reaches(mx, max_nan(change(V0, O0), change(V1, O1)))) {
      exact(V0, O0);
      exact(V1, O1);
    }
    S = N0;
    C = N1;
    o += 2 * P;
    rx += 2 * P;
    ko += 2 * kd;
    if (FULL) gC += 2 * PQ;
  };
  auto row1 = [&](int j, auto tag) {
    constexpr int I0 = decltype(tag)::v;
    const float4 N = lds4(o + dx + P);
    float4 R = Rn, O;
    if (rres) R = lds4(rx);
    const float4 V = update(ResPar<I0>{}, C, N, S, o, R, sm<uint32_t>(ko) | out, O);
    if (ok) sts4(o, V);
    if (ground) sts4(o + dx - PS, V);
    if (anyp || j == jS || j == jN) publish(j, V);
    if (res_reaches(mx, change(V, O))) exact(V, O);
  };
  int j = ja;
  if (par) {
#pragma unroll 1
    for (; j + 1 < jb; j += 2) rows2(j, ResPar<1>{});
    if (j < jb) row1(j, ResPar<1>{});
  } else {
#pragma unroll 1
    for (; j + 1 < jb; j += 2) rows2(j, ResPar<0>{});
    if (j < jb) row1(j, ResPar<0>{});
  }
}

// A wall cell of the tile: x = its shared-memory place / 4 | face mask << 16 | plane << 22, y = R (float bits). Its
// new value goes into the tile; the row that holds it publishes and mirrors it. Lanes without one (on = false)
// take part in the warp's votes.
__device__ __forceinline__ void res_wall(const ResTile &t, uint2 w, bool on, int c, ResMax &mx)
{
  float nv = 0.0f, ov = 0.0f;
  if (on) {
    const int o = (int)(w.x & 0xffffu) * 4, k = (int)(w.x >> 22), P = t.P, PS = t.PS;
    const unsigned m_ = (w.x >> 16) & 63u;
    const int j = t.row_of((o - t.at(c, k, 0, 0)) >> 4);
    const int I0 = (c + t.j0 + j + t.k0 + k) & 1;
    const int x = o + (c ? -t.CP : t.CP);
    const float4 a = sm<float4>(t.cf + 32 * k);
    const float4 b = sm<float4>(t.cf + 32 * k + 16);
    const float e = (m_ & 1u) ? a.x : 0.0f, f = (m_ & 2u) ? a.y : 0.0f, g = (m_ & 4u) ? a.z : 0.0f;
    const float h = (m_ & 8u) ? a.w : 0.0f, m = (m_ & 16u) ? b.x : 0.0f, n = (m_ & 32u) ? b.y : 0.0f;
    ov = sm<float>(o);
    nv = sm<float>(t.inv + 256 * k + 4 * m_) *
             (e * sm<float>(x + 4 * I0) + f * sm<float>(x + 4 * I0 - 4) + g * sm<float>(x + P) + h * sm<float>(x - P) +
              m * sm<float>(x + PS) + n * sm<float>(x - PS) - __uint_as_float(w.y)) +
         b.w * ov;
    sm<float>(o) = nv;
  }
  if (res_reaches(mx, fabsf(nv - ov))) res_exact(mx, nv, ov);
}

template <bool FULL>
__global__ void __launch_bounds__(kResMaxThreads, 1) k_sor_res(ResArgs a)
{
  __shared__ unsigned long long s_err[2];  // CTA's exact max|dlambda| (double bits), by iteration parity
  __shared__ unsigned s_thr[2];            // its rounded value so far (float bits)
  __shared__ int s_cert;                   // number of the last iteration of which this CTA has posted a proof
  __shared__ int s_go, s_bad;              // the group: proven not to stop; a wait gave up
  __shared__ double s_val, s_win;
  __shared__ unsigned long long s_slot, s_target, s_narr;  // s_target, s_narr: counts of barrier and red arrivals
  __shared__ ResTile t;
  __shared__ ResPhase F;                   // the current phase
  __shared__ float s_ctol;
  __shared__ short s_seg[kResSegs + 1];    // the runs' first rows
  __shared__ int s_nw[2];                  // wall cells of each colour
  __shared__ const unsigned *s_idle;       // the current domain's iteration number, where this CTA has no tile of it
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, NT = blockDim.x, NW = NT >> 5;
  const int rank = blockIdx.x % a.gsz, grp = blockIdx.x / a.gsz;
  const uint32_t limit = a.wait_limit ? a.wait_limit : kResWaitLimit;
  unsigned serial = 0;
  if (tid == 0) {
    s_bad = 0;
    s_idle = nullptr;
  }
  for (;;) {
    // the group's next domain
    __syncthreads();
    if (tid == 0) {
      unsigned long long v;
      if (rank == 0) {
        v = ((unsigned long long)(serial + 1) << 32) | (unsigned)atomicAdd(&a.ctl->queue, 1);
        if (a.gsz > 1) asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(a.slot + grp), "l"(v) : "memory");
      } else {
        if (!res_wait_next(a.slot + grp, (unsigned long long)(serial + 1) << 32, s_idle, limit, a.ctl)) s_bad = 1;
        v = res_load(a.slot + grp);
      }
      s_slot = v;
      s_err[0] = s_err[1] = 0;
      s_cert = 0;
    }
    __syncthreads();
    if (s_bad) return;
    serial = (unsigned)(s_slot >> 32);
    const int di = (int)(unsigned)s_slot;
    if (di >= a.n) return;
    const ResDomain &D = a.dom[di];
    const int nty = D.nty, tiles = nty * D.ntz;
    ResSync *sy = D.sync;
    if (tid == 0) s_idle = rank >= tiles ? &sy->beat : nullptr;
    if (rank >= tiles) continue;
    if (tid == 0) {
      s_target = s_narr = 0;
      t.tym = D.tym;
      t.tzm = D.tzm;
      t.epoch = D.epoch;
      t.X = D.X;
      t.Y = D.Y;
      t.Z = D.Z;
      t.PQ = D.PQ;
      t.CS = D.CS;
      t.nq4 = D.nq4;
      t.magic = D.magic;
      t.lam = D.lam;
      t.R = D.R;
      t.mask = D.mask;
      t.co = D.co;
      const int jt = rank % nty, kt = rank / nty;
      t.j0 = 1 + (int)((long)(D.Y - 2) * jt / nty);
      t.ty = 1 + (int)((long)(D.Y - 2) * (jt + 1) / nty) - t.j0;
      t.k0 = 1 + (int)((long)(D.Z - 2) * kt / D.ntz);
      t.tz = 1 + (int)((long)(D.Z - 2) * (kt + 1) / D.ntz) - t.k0;
      t.pubS = jt > 0;
      t.pubN = jt < nty - 1;
      t.pubB = kt > 0;
      t.pubT = kt < D.ntz - 1;
      t.P = 16 * t.nq4;
      t.PS = (t.ty + 2) * t.P;
      t.CP = (t.tz + 2) * t.PS;
      int p = 0;
      t.cf = p;
      p += t.tz * 32;
      t.inv = p;
      p += t.tz * 256;
      t.own = p + t.PS + t.P;
      p += 2 * t.CP;
      t.wls = p;
      p += 16 * kResWalls;
      t.kp = p;
      p += (8 * t.tz * t.ty * t.nq4 + 15) / 16 * 16;  // every region starts on 16 bytes
      t.xt = p;
      p += 16 * (t.tz + t.ty) * t.nq4;
      t.rs = p;
      t.rp = min(t.tz, (4 * a.smem_floats - p) / (2 * t.ty * t.P));
      for (int q = 0; q < 2; ++q) {
        t.lanes[q] = (t.tz - q + 1) / 2 * t.nq4;
        t.chunks[q] = (t.lanes[q] + 31) / 32;
      }
      // runs of rows: the fewest row steps (and four of a task's start) on the busiest warp
      const int ch = t.chunks[0] + t.chunks[1];
      int best = 1 << 30;
      for (int n = 1; n <= min(t.ty, kResSegs); ++n) {
        const int cost = (ch * n + NW - 1) / NW * ((t.ty + n - 1) / n + 4);
        if (cost < best) {
          best = cost;
          t.nseg = n;
        }
      }
      t.ntask = ch * t.nseg;
      t.segmagic = (unsigned)(((1ull << 32) + t.nseg - 1) / t.nseg);
      t.split = t.nq4 % 32 != 0 ? t.lanes[0] > 32 : t.nq4 > 32;
      for (int n = 0; n <= t.nseg; ++n) s_seg[n] = (short)(t.ty * n / t.nseg);
      s_nw[0] = s_nw[1] = 0;
    }
    __syncthreads();
    const int cols = t.ty * t.nq4;
    // exchange slots of colour c of the group's CTA r
    auto slots = [&](int c, int r) { return a.xbuf + ((long)(2 * grp + c) * a.gsz + r) * a.xstride * 2; };
    // the halo's groups that a neighbour feeds: where they come from (colour 0's slots, in groups) and go to
    if (tid == 0) t.xn = 0;
    __syncthreads();
    int2 *xt = &sm<int2>(t.xt);
    {
      const int nr = t.tz * t.nq4;
      for (int i = tid; i < 2 * (nr + cols); i += NT) {
        int side, o;
        if (i < 2 * nr) side = i >= nr, o = i - side * nr;
        else side = 2 + (i - 2 * nr >= cols), o = i - 2 * nr - (side - 2) * cols;
        if (!(side == 0 ? t.pubN : side == 1 ? t.pubS : side == 2 ? t.pubT : t.pubB)) continue;
        const int r = t.row_of(o), q4 = o - r * t.nq4;
        const int q = side == 0 ? rank + 1 : side == 1 ? rank - 1 : side == 2 ? rank + nty : rank - nty;
        const int base = side == 0 ? 0 : side == 1 ? t.tzm * t.nq4 : side == 2 ? 2 * t.tzm * t.nq4 : (2 * t.tzm + t.tym) * t.nq4;
        xt[atomicAdd(&t.xn, 1)] = make_int2(q * a.xstride + base + o,
                                            side < 2 ? t.at(0, r, side ? -1 : t.ty, q4) : t.at(0, side == 2 ? t.tz : -1, r, q4));
      }
    }
    // Collects the neighbours' faces of colour c and half-sweep `mark` into the halo, as they arrive. Thread 0
    // also learns (certs > 0: the iteration's number) whether the iteration is proven not to stop: by any CTA,
    // or by none once all have reported.
    auto collect = [&](int c, unsigned mark, unsigned certs) {
      const ulonglong2 *base = slots(c, 0);
      const int to = c * t.CP, tot = t.xn;
      bool cert = tid == 0 && certs != 0;
      constexpr int U = 2;  // groups a thread asks for at once
      for (int i0 = tid; i0 < tot || cert; i0 += U * NT) {
        const ulonglong2 *src[U];
        int dst[U];
        unsigned pend = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = i0 + u * NT;
          int2 e = make_int2(0, 0);
          if (i < tot) {
            e = xt[i];
            pend |= 1u << u;
          }
          src[u] = base + 2 * e.x;
          dst[u] = to + e.y;
        }
        for (uint32_t n = 0; pend || cert; ++n) {
          if (n >= limit || ((n & 1023u) == 1023u && res_fault(a.ctl))) {
            atomicExch(&a.ctl->fault, 1);
            s_bad = 1;
            return;
          }
          ulonglong2 v[U], w[U];
          unsigned proof = 0;  // asked for together with the faces
          if (cert) asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(proof) : "l"(&sy->cert) : "memory");
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (pend >> u & 1u) {
              asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v[u].x), "=l"(v[u].y) : "l"(src[u]) : "memory");
              asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(w[u].x), "=l"(w[u].y) : "l"(src[u] + 1) : "memory");
            }
          if (cert) {
            if (proof >= certs) {
              s_go = 1;
              cert = false;
            } else if (res_load(&sy->arr) >= s_narr) {
              s_go = res_load32(&sy->cert) >= certs;
              cert = false;
            }
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (pend >> u & 1u) {
              const unsigned f = (unsigned)(v[u].x >> 32) ^ mark, h = (unsigned)(v[u].y >> 32) ^ mark;
              const unsigned x = (unsigned)(w[u].x >> 32) ^ mark, y = (unsigned)(w[u].y >> 32) ^ mark;
              if ((f | h | x | y) == 0u) {
                sts4(dst[u], make_float4(__uint_as_float((unsigned)v[u].x), __uint_as_float((unsigned)v[u].y),
                                         __uint_as_float((unsigned)w[u].x), __uint_as_float((unsigned)w[u].y)));
                pend &= ~(1u << u);
              }
            }
        }
      }
    };
    // The plane's common open faces: all six, but on the plane above the ground the face below is closed wherever
    // the ground is solid (counted on one row: either choice gives the same results).
    {
      int open = 0, closed = 0;
      if (!FULL && t.k0 == 1)
        for (int q = tid; q < t.X / 2; q += NT) {
          const unsigned m = __ldg(t.mask + t.gidx(0, 0, t.ty / 2, 0) + q);
          open += m == 63u;
          closed += m == 31u;
        }
      const int n = __syncthreads_count(closed > open) - __syncthreads_count(open > closed);
      if (tid == 0) t.base0 = n > 0 ? 31u : 63u;
    }
    __syncthreads();
    // the tile's lambda with its halo, the resident planes of R, which cells the rows leave out
    auto swalls = [&](int c) { return &sm<uint2>(t.wls) + c * kResWalls; };
    // the tile's part of the domain's lists: tiles of a layer of planes side by side
    const long w0 = (long)t.P / 4 * ((long)(t.k0 - 1) * (t.Y - 2) + (long)(t.j0 - 1) * t.tz);
    for (int c = 0; c < 2; ++c) {
      const int rows = t.ty + 2;
      for (int i = tid; i < (t.tz + 2) * rows * t.nq4; i += NT) {
        const int r = t.row_of(i), q4 = i - r * t.nq4, k = r / rows - 1, j = r % rows - 1;
        sts4(t.at(c, k, j, q4), __ldcg(reinterpret_cast<const float4 *>(t.lam + t.gidx(c, k, j, q4))));
      }
      // and the list of the wall cells: those whose open faces are not their plane's common ones
      for (int i = tid; i < t.tz * cols; i += NT) {
        const int r = t.row_of(i), q4 = i - r * t.nq4, k = r / t.ty, j = r - k * t.ty;
        const long g = t.gidx(c, k, j, q4);
        const float4 R = __ldg(reinterpret_cast<const float4 *>(t.R + g));
        if (k < t.rp) sts4(t.rs + c * t.rp * t.ty * t.P + 16 * i, R);
        const uint32_t m = FULL ? 0x3f3f3f3fu : __ldg(reinterpret_cast<const uint32_t *>(t.mask + g));
        const float rv[4] = {R.x, R.y, R.z, R.w};
        const int I0 = (c + t.j0 + j + t.k0 + k) & 1;
        uint32_t keep = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int x = 2 * (4 * q4 + u) + I0;
          const unsigned mu = (m >> (8 * u)) & 63u;
          if (x < 1 || x > t.X - 2) {
            keep |= 0xffu << (8 * u);
          } else if (!FULL && mu != (k == 0 ? t.base0 : 63u)) {
            keep |= 0xffu << (8 * u);
            const int at = atomicAdd(&s_nw[c], 1);
            const uint2 w = make_uint2((unsigned)(t.at(c, k, j, q4) / 4 + u) | mu << 16 | (unsigned)k << 22, __float_as_uint(rv[u]));
            if (at < kResWalls) swalls(c)[at] = w;
            else __stcg(D.walls[c] + w0 + at, w);
          }
        }
        sm<uint32_t>(t.kp + 4 * (c * t.tz * cols + i)) = keep;
      }
    }
    __syncthreads();
    // meets the group's other CTAs (thread 0): everything the CTA stored before the last CTA barrier is
    // visible to them, and theirs to this thread
    auto meet = [&]() {
      if (tiles > 1) {
        res_arrive(&sy->bar);
        s_target += tiles;
        if (!res_wait(&sy->bar, s_target, limit, a.ctl)) s_bad = 1;
      }
    };
    if (FULL && D.alias) {
      // every CTA has read its part of the start: the CTA clears its slots of what lies there (lambda, or an earlier
      // solve's words, which carry the same marks), before any neighbour asks for them
      if (tid == 0) meet();
      __syncthreads();
      if (s_bad) return;
      for (int c = 0; c < 2; ++c)
        for (int i = tid; i < 2 * a.xstride; i += NT) slots(c, rank)[i] = make_ulonglong2(0, 0);
      __syncthreads();
      if (tid == 0) meet();
      __syncthreads();
      if (s_bad) return;
    }
    unsigned iters = 0;  // iterations of all phases
    bool dead = false;
    for (int ph = 0; ph < D.nph && !dead; ++ph) {
      if (tid == 0) {
        F = D.ph[ph];
        s_ctol = (float)(F.tol * (1.0 + 1e-6));  // a rounded change above it is a change above tol
        s_thr[0] = s_thr[1] = 0;
      }
      __syncthreads();
      for (int i = tid; !FULL && i < t.tz * 64; i += NT) sm<float>(t.inv + 4 * i) = __ldg(F.inv + (long)t.k0 * 64 + i);
      for (int i = tid; i < t.tz * 8; i += NT) {
        const int k = t.k0 + (i >> 3), q = i & 7;
        if (FULL) sm<float>(t.cf + 4 * i) = F.c1;
        else sm<float>(t.cf + 4 * i) = q < 6 ? __ldg(D.val + q * t.Z + k)
                                        : (q == 6 ? __ldg(F.inv + (long)k * 64 + (i < 8 ? t.base0 : 63u)) : F.c1);
      }
      __syncthreads();
      // the window rule's snapshot: the tile's cells and, below plane 1, the ground plane's
      auto window = [&](bool check) {
        double dm = 0.0;
        auto cmp = [&](float p, float q) {
          const double y = fabs((double)p - (double)q);
          if (y > dm || y != y) dm = y;
        };
        const int kb = t.k0 == 1 ? -1 : 0;
        for (int c = 0; c < 2; ++c)
          for (int i = tid; i < (t.tz - kb) * cols; i += NT) {
            const int r = t.row_of(i), q4 = i - r * t.nq4, kr = r / t.ty, j = r - kr * t.ty, k = kr + kb;
            const float4 v = lds4(t.at(c, k, j, q4));
            float4 *sp = reinterpret_cast<float4 *>(D.snap + t.gidx(c, k, j, q4));
            if (check) {
              const float4 o = *sp;
              if (k >= 0) {
                cmp(v.x, o.x), cmp(v.y, o.y), cmp(v.z, o.z), cmp(v.w, o.w);
              } else {
                const int I0 = (c + t.j0 + j + t.k0 + k) & 1;
                const float vv[4] = {v.x, v.y, v.z, v.w}, oo[4] = {o.x, o.y, o.z, o.w};
                for (int u = 0; u < 4; ++u) {
                  const int x = 2 * (4 * q4 + u) + I0;
                  if (x >= 1 && x <= t.X - 2) cmp(vv[u], oo[u]);
                }
              }
            }
            *sp = v;
          }
        return warp_max_d(dm);
      };
      if (F.wK > 0) window(false);  // the first window starts from lambda as the loop begins
      int left = F.wK, it = 0, windows = 0, converged = 0, nan = 0;
      double wdrift = 0.0;
      bool done = false;
      ResMax mx{kResTinyF, 0.0};
      while (!done) {
        const int par = it & 1;
        ++iters;
        mx.thr = kResTinyF;
        mx.dmax = 0.0;
        for (int c = 0; c < 2; ++c) {
          const unsigned mark = t.epoch + 2 * iters + c;
          const bool ask = !(F.tol < 0.0);  // a tolerance below zero is never met
          if (c == 1 && tid == 0) {
            s_thr[par ^ 1] = 0;
            if (tiles > 1 && ask) {
              res_arrive(&sy->arr);  // the CTA's proof, if it has one, was posted before the last CTA barrier
              s_narr += tiles;
            } else {
              s_go = !ask || s_cert == (int)iters;
            }
          }
          ulonglong2 *xb = slots(c, rank);
          if (!FULL && s_nw[c]) {
            for (int b = warp * 32; b < s_nw[c]; b += NT) {
              const int i = b + lane;
              const bool on = i < s_nw[c];
              uint2 w = make_uint2(0, 0);
              if (on) w = i < kResWalls ? swalls(c)[i] : __ldcg(D.walls[c] + w0 + i);
              res_wall(t, w, on, c, mx);
            }
            __syncthreads();
          }
          for (int task = warp; task < t.ntask; task += NW) {
            res_task<FULL>(t, s_seg, task, c, xb, mark, mx);
            if (lane == 0) atomicMax(&s_thr[par], __float_as_uint(mx.thr));
            mx.thr = fmaxf(mx.thr, __uint_as_float(*reinterpret_cast<volatile unsigned *>(&s_thr[par])));
          }
          if (c == 0) {
            if (lane == 0 && mx.thr > s_ctol && mx.thr > kResTinyF && atomicExch(&s_cert, (int)iters) != (int)iters && tiles > 1)
              atomicMax(&sy->cert, iters);
          } else {
            const double v = warp_max_d(mx.dmax);
            if (lane == 0 && v != 0.0) atomicMax(&s_err[par], (unsigned long long)__double_as_longlong(v));
          }
          if (tiles > 1) collect(c, mark, c == 1 && ask ? iters : 0u);
          __syncthreads();
          if (s_bad) return;
        }
        // the iteration's maximum, then the loop condition (Solver_CPU_RB.cpp:106)
        const bool go = s_go != 0;
        if (tid == 0) {
          const unsigned long long v = s_err[par];
          if (v) atomicMax(reinterpret_cast<unsigned long long *>(F.err + it), v);
          s_err[par] = 0;
          if (rank == 0) *reinterpret_cast<volatile unsigned *>(&sy->beat) = iters;
          if (!go) {
            meet();
            s_val = *reinterpret_cast<volatile double *>(F.err + it);
          }
        }
        if (!go) {
          __syncthreads();
          if (s_bad) return;
          const double e = s_val;
          if (isnan(e)) {
            nan = 1;
            done = true;
          } else if (!(e > F.tol)) {
            converged = 1;
            done = true;
          }
        }
        ++it;
        if (it >= F.itermax) done = true;
        if (!done && F.wK > 0 && --left == 0) {
          // window rule: FP64 max|lambda - snapshot|, the snapshot takes lambda's values
          left = F.wK;
          const double dm = window(true);
          if (tid == 0) s_win = 0.0;
          __syncthreads();
          if (lane == 0 && dm != 0.0)
            atomicMax(reinterpret_cast<unsigned long long *>(&s_win), (unsigned long long)__double_as_longlong(dm));
          __syncthreads();
          if (tid == 0) {
            if (s_win != 0.0) atomic_max_nonneg(&sy->wacc[windows & 3], s_win);
            meet();
            s_win = *reinterpret_cast<volatile double *>(&sy->wacc[windows & 3]);
            // the slot after the next: its last readers arrived at this barrier, its next writers leave the next one
            if (rank == 0) *reinterpret_cast<volatile double *>(&sy->wacc[(windows & 3) ^ 2]) = 0.0;
          }
          __syncthreads();
          if (s_bad) return;
          wdrift = s_win;
          ++windows;
          if (isnan(wdrift)) {
            nan = 1;
            done = true;
          } else if (wdrift <= D.wtol) {
            converged = 2;
            done = true;
          }
        }
      }
      // every CTA's last maximum is in err before the first CTA reads it
      if (tid == 0) {
        meet();
        s_val = *reinterpret_cast<volatile double *>(F.err + it - 1);
      }
      __syncthreads();
      if (s_bad) return;
      if (isnan(s_val)) nan = 1;
      dead = nan;
      if (tid == 0 && rank == 0) {
        SolveState *st = F.st;
        if (isnan(s_val))  // the first iteration with a NaN
          while (it > 1 && isnan(*reinterpret_cast<volatile double *>(F.err + it - 2))) --it;
        st->done = 1;
        st->it = it;
        st->converged = nan ? 0 : converged;
        st->nan = nan;
        st->residual = s_val;
        st->wdrift = wdrift;
        st->t_done = global_ns();
      }
      __syncthreads();  // s_val is read before the next phase writes it
    }
    // lambda back to global memory
    for (int c = 0; c < 2; ++c)
      for (int i = tid; i < t.tz * cols; i += NT) {
        const int r = t.row_of(i), q4 = i - r * t.nq4, k = r / t.ty, j = r - k * t.ty;
        *reinterpret_cast<float4 *>(t.lam + t.gidx(c, k, j, q4)) = lds4(t.at(c, k, j, q4));
      }
  }
}

cudaError_t res_launch(const ResArgs &a, bool full, int groups, int threads, cudaStream_t s)
{
  const size_t smem = sizeof(float) * (size_t)a.smem_floats;
  void (*const fn)(ResArgs) = full ? k_sor_res<true> : k_sor_res<false>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  ResArgs b = a;
  void *args[] = {&b};
  return cudaLaunchCooperativeKernel((const void *)fn, dim3(groups * a.gsz), dim3(threads), args, smem, s);
}

}  // namespace qesb
