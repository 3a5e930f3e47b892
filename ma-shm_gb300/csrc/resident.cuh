// Stepping with the elements resident on the chip: all steps of an
// advance in one cooperative launch, for plans whose element state fits into
// the shared memory of the GPU (flat shells on any mesh, 3D solids of box
// elements; both precisions).
//
// The two-kernel general step and the strip sweep both bring every node value
// from memory in every step, and meet at a kernel boundary once or twice per
// step; on a plate of a few hundred to a few thousand elements that costs far
// more than the element work.  Here each CTA keeps u_n, d_n = u_n - u_{n-1} (FP64:
// u_{n-1}) and the force of its own elements' nodes in shared memory for the whole
// advance (a node shared by several elements is kept, and updated, by each of
// them), so that a step moves only the forces of shared nodes:
//   1. K_e u_n of the CTA's elements, in passes of `epass` elements;
//   2. the forces of element nodes that other CTAs hold copies of go to an
//      exchange buffer (L2) as 8-byte words that each carry the step's tag;
//   3. each record that the CTA needs from others is read into shared memory,
//      by one thread, as soon as its words carry the tag;
//   4. every copy of a node sums the copies' forces in basket order (so all
//      copies compute the same bits) and updates u.
// There is no device-wide barrier, no fence and no separate flag between
// steps: a CTA waits only for the forces it reads.  Two exchange buffers,
// alternating by step, are enough: a CTA writes a record of step n + 2 after
// it has read the step n + 1 records of every CTA it shares nodes with, which
// those write after they have read its records of step n.  Tags are never
// reused, so nothing is cleared between launches.
//
// State.  In FP32 the update d_{n+1} = k1 d_n - k2 F / M, u_{n+1} = u_n + d_{n+1}
// keeps the increment instead of u_{n-1}: the rounding of u then stays a rounding
// of u, where u + k1 (u - u_{n-1}) turns it into a velocity that every later step
// integrates.  FP32 errors against 64 bits fall accordingly, and velocity and
// acceleration frames, a1 (d_{n+1} + d_n) and a0 (d_{n+1} - d_n), lose no digits to
// cancellation.  The plan keeps d between launches, so that advancing in pieces
// gives the bits of one advance, and hands it out as u_{n-1} = u - d in FP64, which
// has every bit of both (res_coarse), so that a state that was read and set
// again steps on with the same bits.  In FP64, where u - d has no wider type to be
// exact in, the second value is u_{n-1} itself, as in the other kernels.
//
// Element cores.  FP64: elements that are axis-aligned rectangles with constant
// laminate commute with the reflections of the reference square: with
// S-values (sums and differences of the four mirror nodes) as unknowns, the
// antisymmetric 6x6 derivative matrix splits into two 3x3 blocks that map even
// to odd and odd to even, the resultants act inside one parity sector, and a
// derivative costs 3 multiply-adds per value instead of 6.  All constants of
// an element (derivative blocks scaled by 2/ax and 2/ay, laminate times
// quadrature weight) come from a table with one entry per (ax, ay, laminate),
// so the count is about 4 900 floating-point operations per element against
// 8 700 of the direct form.  FP64 runs at 2 operations per clock and SM on this
// GPU, so in FP64 this count is the time.  The 3D solid's boxes are treated the
// same way in xi and eta, with the three zeta layers as they are (about 9 600
// against 17 600 operations).  Other shell elements, and all elements in FP32,
// use the direct form.  FP32 is not bound by its operations (20x20 plate 2.7 us a
// step by sectors, 2.6 direct; 80x80 10.0 and 9.3), and sums of mirror nodes carry
// the rounding of a large value at one corner of an element to the others, which shows
// ahead of a wave front, where displacements are orders below the source's: 12x12x8
// solid after 80 steps 9.0e-6 from 64 bits by sectors, 3.0e-6 direct (6.1e-6 by the
// element and node kernels).  FP64 loses nothing by sectors there: against 80-bit
// arithmetic the same solid is 1.7e-13 off (1.8e-13 by the element and node kernels), a
// 24x24 plate 3.6e-15 (4.0e-15 by the structured kernel, 7.1e-14 by the general ones).
#pragma once
#include "shell_element.cuh"
#include "shell_structured_f32.cuh"  // packed FP32 arithmetic
#include "solid_element.cuh"

namespace shm {

constexpr int RES_OWNER = 1 << 30, RES_HAS_OUT = 1 << 29, RES_FORCED = 1 << 28, RES_NODE = RES_FORCED - 1;
// 16-bit codes of a node's copies, up to eight: offset of F in the CTA's shared
// memory (its own state, or a record read from another CTA); no further copy;
// more than eight copies, in the node's list
constexpr unsigned RES_NONE = 0xffff, RES_LIST = 0xfffe;

// Element cores.  NF fields, NODES nodes per element; STAGE values of staging and
// RED of sensor partial sums per element in a pass; CLASS values per table
// entry; EPASS elements of a pass at most, on THREADS threads; ctas() the CTAs per
// SM that the registers are limited for (a shell's eight warps: 80 registers a thread
// in FP32, 128 in FP64).  Rectangles and boxes by sector are FP64's, solid nodes FP32's.
struct ShellRect {
  // 5 fields by sector, later the sector forces, and 8 resultants
  static constexpr int NF = 5, NODES = NPE, STAGE = 13 * NPE, RED = NPE, EPASS = 7;
  static constexpr int CLASS = 36 + 21 * 9;  // derivative blocks, laminate x weight
  static constexpr int THREADS = 256;
  static constexpr int ctas(size_t) { return 2; }
};
struct ShellQuad {
  static constexpr int NF = 5, NODES = NPE, STAGE = 10 * NPE, RED = NPE, EPASS = 7;  // 10 fluxes
  static constexpr int CLASS = 0, CLASS32 = 28;  // FP32: the laminate as 12 pairs and 3 shear values
  static constexpr int THREADS = 256;
  static constexpr int ctas(size_t value) { return value == 4 ? 3 : 2; }
};
struct SolidBox {
  // 3 fields by sector, later the sector forces, and 6 stresses
  static constexpr int NF = 3, NODES = S_NPE, STAGE = 9 * S_NPE, RED = 0, EPASS = 4;
  static constexpr int CLASS = 45 + 13 * 27;  // derivative blocks, zeta derivatives, stiffness x weight
  static constexpr int THREADS = 448;
  static constexpr int ctas(size_t) { return 1; }
};
struct SolidNodes {
  // 8 planes of stresses
  static constexpr int NF = 3, NODES = S_NPE, STAGE = 8 * S_NPE, RED = 0, EPASS = 4;
  static constexpr int CLASS = 4 + 13;  // 2/a of the three directions, Jacobian determinant; stiffness
  static constexpr int THREADS = 448;
  static constexpr int ctas(size_t) { return 2; }
};
// Layout of an element's state: u, d and F of its nodes, field by field.  FP32
// shells keep (u, phi_x) and (v, phi_y) in pairs -- the two members of a pair see
// the same derivatives and pair up in the resultants -- so that shared-memory
// accesses move 8 or 16 bytes and the arithmetic is packed FP32x2; w follows
// alone, in F with an empty partner so that a copy's three parts are equally
// spaced.  (Bound by shared-memory wavefronts on full SMs: 80x80 jittered quads
// 10.7 us a step with one value at a time, 9.2 in pairs; 20x20 2.7 and 2.5.)
template <typename T, class C> struct ResLay {
  static constexpr bool PAIRS = sizeof(T) == 4 && C::NF == 5;
  static constexpr int N = C::NODES, NF = C::NF;
  static constexpr int PITCH = PAIRS ? 2 : 1;            // between nodes in F
  static constexpr int PARTS = PAIRS ? 3 : NF;           // of F, PITCH values each
  static constexpr int UB = NF * N, FB = PARTS * PITCH * N;
  // values per element; pairs: 8 mod 32, so that consecutive elements start in
  // other banks (80x80 jittered quads 9.5 us a step without, 9.2 with)
  static constexpr int SS = 2 * UB + FB + (PAIRS ? 8 : 0);
  static_assert(!PAIRS || SS % 32 == 8, "element stride");
  __device__ static __forceinline__ void ld_u(const T* b, int n, T (&v)[NF]) {
    if constexpr (PAIRS) {
      const float2 p = *reinterpret_cast<const float2*>(b + 2 * n), q = *reinterpret_cast<const float2*>(b + 2 * N + 2 * n);
      v[0] = p.x; v[1] = p.y; v[2] = q.x; v[3] = q.y;
      v[4] = b[4 * N + n];
    } else {
#pragma unroll
      for (int f = 0; f < NF; ++f) v[f] = b[f * N + n];
    }
  }
  __device__ static __forceinline__ void st_u(T* b, int n, const T (&v)[NF]) {
    if constexpr (PAIRS) {
      *reinterpret_cast<float2*>(b + 2 * n) = make_float2(v[0], v[1]);
      *reinterpret_cast<float2*>(b + 2 * N + 2 * n) = make_float2(v[2], v[3]);
      b[4 * N + n] = v[4];
    } else {
#pragma unroll
      for (int f = 0; f < NF; ++f) b[f * N + n] = v[f];
    }
  }
  // F at q, its parts d apart
  __device__ static __forceinline__ void ld_f(const T* q, int d, T (&v)[NF]) {
    if constexpr (PAIRS) {
      const float2 x = *reinterpret_cast<const float2*>(q), y = *reinterpret_cast<const float2*>(q + d);
      v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
      v[4] = q[2 * d];
    } else {
#pragma unroll
      for (int f = 0; f < NF; ++f) v[f] = q[f * d];
    }
  }
  __device__ static __forceinline__ void st_f(T* q, int d, const T (&v)[NF]) {
    if constexpr (PAIRS) {
      *reinterpret_cast<float2*>(q) = make_float2(v[0], v[1]);
      *reinterpret_cast<float2*>(q + d) = make_float2(v[2], v[3]);
      q[2 * d] = v[4];
    } else {
#pragma unroll
      for (int f = 0; f < NF; ++f) q[f * d] = v[f];
    }
  }
};
// which of the three update coefficients a field has: shells (u, v), (phi_x,
// phi_y), w; solids (u, v), -, w
template <class C> __host__ __device__ constexpr int res_coef(int f) { return C::NF == 5 ? (f == 4 ? 2 : f & 1) : (f == 2 ? 2 : 0); }
// FP32: the second value of the state is the increment d (FP64: u_{n-1})
template <typename T> constexpr bool RES_INC = sizeof(T) == 4;
// d without the bits that u - d has no room for in FP64: where |d| < 2^-25 |u|, d is
// rounded to a multiple of 2^-50 |u| or finer (2^-26 of u's own rounding)
__device__ __forceinline__ float res_coarse(float d, float u) {
  const float c = u * 0x1p-25f;
  return fabsf(d) < fabsf(c) ? __fsub_rn(__fadd_rn(d, c), c) : d;
}

// exchange record: NF values in 8-byte words of 4 bytes payload and the tag, two
// words a piece
template <typename T, class C> __host__ __device__ constexpr int res_pieces() { return (C::NF * (int)sizeof(T) / 4 + 1) / 2; }

template <typename T> struct ResArgs {
  int fen, epc, epass, ncta, nn_first, nft;
  int64_t nnode_pad;
  T* UA;
  T* UB;
  T* dinc;                         // [NF][nnode_pad] second values left by the previous launch
  int dvalid;                      // (0: the state was set otherwise, in UA and UB)
  const int2* __restrict__ meta;   // [fen][NODES] node | owner; list start
  const uint4* __restrict__ codes; // [fen][NODES] codes of the node's copies in basket order
  const int* __restrict__ lists;   // per node with excitation or more copies: counts of the copies listed and
                                   // of the excitation entries, the copies' offsets, the entries
  const int* __restrict__ exp_ptr; // [ncta + 1] records that a CTA writes
  const int* __restrict__ exp_off; // offset of F in the CTA's state, per record
  const int* __restrict__ imp_ptr; // [ncta + 1] records that a CTA reads
  const int* __restrict__ imp_rec; // their numbers
  int maximp;                      // most records a CTA reads
  uint4* xch;                      // [2][nrec][pieces]
  int nrec;
  unsigned tag0;                   // the launch's first tag
  unsigned* abortw;                // tag0 of a launch that gave up
  int spin;
  // elements
  const int* __restrict__ cls;     // class of each element
  const T* __restrict__ table;     // [nclass][CLASS]
  const T* __restrict__ geo;       // ShellQuad: [fen][5][36]
  const int* __restrict__ emat;    // (per-element arrays in the resident order)
  const T* __restrict__ mat;
  const T* __restrict__ ekeep;
  const T* __restrict__ km;        // [fen][NODES][4] k2 / M of (u, v), of (phi_x, phi_y) and of w; owner, has-outputs, forced bits
  T k1[3];                         // of (u, v), (phi_x, phi_y), w
  // excitation and outputs
  const int* __restrict__ fq_field;
  const int* __restrict__ fq_scen;
  const double* __restrict__ fq_val;
  const double* __restrict__ st;
  const int* __restrict__ out_start;  // [fen][NODES] into out_list (read where RES_HAS_OUT is set)
  const int* __restrict__ out_list;   // count, outputs
  const int* __restrict__ out_field;
  double* displ;
  int nslot;
  const int* __restrict__ esens;
  double* vsum;
  SensorConst<T> sc;
  FrameSpec fs;
  T* frames;
  PressureArgs<T> pr;
  T a0, a1, blowup;
  int* flag;
  const int* d_base;
  // states kept: u after step i of the launch at keep_u + i * keep_stride (null: none);
  // end: UA, UB and dinc take the last state
  T* keep_u;
  int64_t keep_stride;
  bool end;
  // adjoint: the forward states that the launch's steps meet, last first -- the
  // states at um + i * keep_stride for i = nsteps - 2 .. 0, then um0
  const T* um;
  const T* um0;
  const T* __restrict__ keep;      // stiffness factors (ekeep is all ones)
  double* gpart;                   // [fen][NODES] sums of (K_e^0 lambda)_n' u_n
  const double* asig;              // [nout][nft] residuals in reversed time
};

template <typename T, class C>
__host__ __device__ constexpr size_t res_smem_bytes(int epc, int epass, int maximp) {
  return sizeof(uint4) * C::NODES * (size_t)epc +
         sizeof(T) * ((size_t)epc * ResLay<T, C>::SS + (size_t)epass * (C::STAGE + C::RED) +
                      (size_t)ResLay<T, C>::PARTS * ResLay<T, C>::PITCH * maximp);
}

// Pieces are written and read at GPU scope as pairs of 8-byte words; each word
// carries the tag, so it does not matter whether the pair is seen at once.
__device__ __forceinline__ void st_piece(uint4* p, unsigned a, unsigned b, unsigned tag) {
  asm volatile(
      "{\n .reg .b64 lo, hi;\n mov.b64 lo, {%1, %3};\n mov.b64 hi, {%2, %3};\n"
      " st.relaxed.gpu.global.v2.b64 [%0], {lo, hi};\n}\n" ::"l"(p),
      "r"(a), "r"(b), "r"(tag)
      : "memory");
}
__device__ __forceinline__ uint4 ld_piece(const uint4* p) {
  uint4 v;
  asm volatile(
      "{\n .reg .b64 lo, hi;\n ld.relaxed.gpu.global.v2.b64 {lo, hi}, [%4];\n"
      " mov.b64 {%0, %1}, lo;\n mov.b64 {%2, %3}, hi;\n}\n"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p)
      : "memory");
  return v;
}
__device__ __forceinline__ void ld4(const float* p, float (&v)[4]) {
  const float4 q = __ldg(reinterpret_cast<const float4*>(p));
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void ld4(const double* p, double (&v)[4]) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(p)), b = __ldg(reinterpret_cast<const double2*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ int res_bits(float v) { return __float_as_int(v); }
__device__ __forceinline__ int res_bits(double v) { return __double2loint(v); }
__device__ __forceinline__ unsigned res_word(const float* v, int w) { return __float_as_uint(v[w]); }
__device__ __forceinline__ unsigned res_word(const double* v, int w) {
  return (unsigned)((w & 1) ? __double2hiint(v[w / 2]) : __double2loint(v[w / 2]));
}
template <int NF, typename T> __device__ __forceinline__ void xch_store(uint4* p, const T (&F)[NF], unsigned tag) {
  constexpr int NW = NF * (int)sizeof(T) / 4;
#pragma unroll
  for (int q = 0; q < (NW + 1) / 2; ++q) st_piece(p + q, res_word(F, 2 * q), 2 * q + 1 < NW ? res_word(F, 2 * q + 1) : 0u, tag);
}
template <int NF, int P> __device__ __forceinline__ void xch_unpack(const uint4 (&p)[P], float (&v)[NF]) {
#pragma unroll
  for (int f = 0; f < NF; ++f) v[f] = __uint_as_float(f & 1 ? p[f / 2].z : p[f / 2].x);
}
template <int NF, int P> __device__ __forceinline__ void xch_unpack(const uint4 (&p)[P], double (&v)[NF]) {
#pragma unroll
  for (int f = 0; f < NF; ++f) v[f] = __hiloint2double((int)p[f].z, (int)p[f].x);
}

// K_e u of the pass's elements [e0, e0 + ne), all kept in `state` (u at 0,
// F at 10*36 of each element); every thread of the CTA calls it.
__device__ __forceinline__ void res_pass_rect(const ResArgs<double>& a, double* state, double* stage, double* vred, int e0,
                                              int ne, int nn) {
  using T = double;
  const int t = threadIdx.x, nt = blockDim.x;
  constexpr int ST = ShellRect::STAGE, RES_STATE = ResLay<T, ShellRect>::SS;
  // nodal values to parity sectors: S[px + 2 py](i, k) over the four mirror nodes
  for (int w = t; w < 45 * ne; w += nt) {
    const int le = w / 45, r = w % 45, f = r / 9, m = r % 9, i = m % 3, k = m / 3;
    const T* u = state + le * RES_STATE + f * NPE;
    const T A = u[k * 6 + i], B = u[k * 6 + 5 - i], C = u[(5 - k) * 6 + i], D = u[(5 - k) * 6 + 5 - i];
    T* s = stage + le * ST + f * NPE + m;
    const T ab = A + B, am = A - B, cd = C + D, cm = C - D;
    s[0] = ab + cd;
    s[9] = am + cm;
    s[18] = ab - cd;
    s[27] = am - cm;
  }
  __syncthreads();
  const int le = t / NPE, n = t % NPE;
  const bool act = t < NPE * ne;
  const int s = n / 9, m = n % 9, i = m % 3, k = m / 3;
  const int px = s & 1, py = s >> 1;
  const int e = e0 + le;
  T* sg = stage + le * ST;
  T* sr = sg + 5 * NPE;
  const T* tab = nullptr;
  if (act) {
    tab = a.table + (int64_t)a.cls[e] * ShellRect::CLASS;
    // rows of the derivative blocks into this sector: from the odd values
    // (block B) for an even result, from the even ones (block A) for an odd
    const T* mx = tab + (px ? 0 : 9) + 3 * i;
    const T* my = tab + 18 + (py ? 0 : 9) + 3 * k;
    const T x0 = mx[0], x1 = mx[1], x2 = mx[2], y0 = my[0], y1 = my[1], y2 = my[2];
    const T* gx = sg + (s ^ 1) * 9 + 3 * k;   // xi lines of the mirrored sector
    const T* gy = sg + (s ^ 2) * 9 + i;       // eta lines
    auto dxi = [&](int f, T c) { const T* p = gx + f * NPE; return fma(x2, p[2], fma(x1, p[1], fma(x0, p[0], c))); };
    auto det = [&](int f, T c) { const T* p = gy + f * NPE; return fma(y2, p[6], fma(y1, p[3], fma(y0, p[0], c))); };
    auto dxi0 = [&](int f) { const T* p = gx + f * NPE; return fma(x2, p[2], fma(x1, p[1], x0 * p[0])); };
    auto det0 = [&](int f) { const T* p = gy + f * NPE; return fma(y2, p[6], fma(y1, p[3], y0 * p[0])); };
    const T* own = sg + s * 9 + m;
    const T ex = dxi0(0), ey = det0(2), gxy = dxi(2, det0(0));
    const T kx = dxi0(1), ky = det0(3), kxy = dxi(3, det0(1));
    const T gyz = det(4, own[3 * NPE]), gxz = dxi(4, own[NPE]);
    if (a.nslot > 0 && s == 0)  // the even-even sector holds the sums over mirror nodes
      vred[le * NPE + m] = a.sc.k0 * (a.sc.e31 * (ex + a.sc.hh * kx) + a.sc.e32 * (ey + a.sc.hh * ky));
    const T* L = tab + 36 + m;  // coefficient q at L[9 q]: a11 a12 a16 a22 a26 a66 a44 a45 a55 b.. d..
    auto l = [&](int q) { return L[9 * q]; };
    T* r = sr + n;
    r[0 * NPE] = fma(l(11), kxy, fma(l(10), ky, fma(l(9), kx, fma(l(2), gxy, fma(l(1), ey, l(0) * ex)))));
    r[1 * NPE] = fma(l(13), kxy, fma(l(12), ky, fma(l(10), kx, fma(l(4), gxy, fma(l(3), ey, l(1) * ex)))));
    r[2 * NPE] = fma(l(14), kxy, fma(l(13), ky, fma(l(11), kx, fma(l(5), gxy, fma(l(4), ey, l(2) * ex)))));
    r[3 * NPE] = fma(l(17), kxy, fma(l(16), ky, fma(l(15), kx, fma(l(11), gxy, fma(l(10), ey, l(9) * ex)))));
    r[4 * NPE] = fma(l(19), kxy, fma(l(18), ky, fma(l(16), kx, fma(l(13), gxy, fma(l(12), ey, l(10) * ex)))));
    r[5 * NPE] = fma(l(20), kxy, fma(l(19), ky, fma(l(17), kx, fma(l(14), gxy, fma(l(13), ey, l(11) * ex)))));
    r[6 * NPE] = fma(l(7), gxz, l(6) * gyz);  // Qy
    r[7 * NPE] = fma(l(8), gxz, l(7) * gyz);  // Qx
  }
  __syncthreads();
  if (act) {
    // transposed blocks: an even force from the odd fluxes through A', an odd
    // one from the even fluxes through B'
    const T* mx = tab + (px ? 9 : 0) + i;
    const T* my = tab + 18 + (py ? 9 : 0) + k;
    const T x0 = mx[0], x1 = mx[3], x2 = mx[6], y0 = my[0], y1 = my[3], y2 = my[6];
    const T* gx = sr + (s ^ 1) * 9 + 3 * k;
    const T* gy = sr + (s ^ 2) * 9 + i;
    auto both = [&](int rx, int ry, T c) {
      const T *p = gx + rx * NPE, *q = gy + ry * NPE;
      c = fma(x2, p[2], fma(x1, p[1], fma(x0, p[0], c)));
      return fma(y2, q[6], fma(y1, q[3], fma(y0, q[0], c)));
    };
    auto both0 = [&](int rx, int ry) {
      const T *p = gx + rx * NPE, *q = gy + ry * NPE;
      const T c = fma(x2, p[2], fma(x1, p[1], x0 * p[0]));
      return fma(y2, q[6], fma(y1, q[3], fma(y0, q[0], c)));
    };
    const T keep = a.ekeep[e];
    T* o = sg + n;  // (the sector values were last read before the barrier)
    o[0 * NPE] = keep * both0(0, 2);
    o[1 * NPE] = keep * both(3, 5, sr[7 * NPE + n]);  // + Qx into phi_x
    o[2 * NPE] = keep * both0(2, 1);
    o[3 * NPE] = keep * both(5, 4, sr[6 * NPE + n]);  // + Qy into phi_y
    o[4 * NPE] = keep * both0(7, 6);
    if (a.nslot > 0 && n == 0) {
      const int slot = a.esens[e];
      if (slot >= 0) {
        double v = 0.0;
        for (int q = 0; q < 9; ++q) v += (double)vred[le * NPE + q];
        a.vsum[(int64_t)slot * a.nft + (nn - 1)] = v;
      }
    }
  }
  __syncthreads();
  // sector forces back to the nodes (the factor 1/4 is in the laminate table)
  for (int w = t; w < 45 * ne; w += nt) {
    const int l2 = w / 45, r = w % 45, f = r / 9, mm = r % 9, ii = mm % 3, kk = mm / 3;
    const T* q = stage + l2 * ST + f * NPE + mm;
    const T ee = q[0], oe = q[9], eo = q[18], oo = q[27];
    const T p0 = ee + eo, p1 = oe + oo, m0 = ee - eo, m1 = oe - oo;
    T* F = state + l2 * RES_STATE + (10 + f) * NPE;
    F[kk * 6 + ii] = p0 + p1;
    F[kk * 6 + 5 - ii] = p0 - p1;
    F[(5 - kk) * 6 + ii] = m0 + m1;
    F[(5 - kk) * 6 + 5 - ii] = m0 - m1;
  }
  __syncthreads();
}

// six consecutive values from an even index, as three pairs
__device__ __forceinline__ void ld_line(const float* p, float (&o)[NP]) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const float2 v = reinterpret_cast<const float2*>(p)[q];
    o[2 * q] = v.x;
    o[2 * q + 1] = v.y;
  }
}
__device__ __forceinline__ void ld_line(const double* p, double (&o)[NP]) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const double2 v = reinterpret_cast<const double2*>(p)[q];
    o[2 * q] = v.x;
    o[2 * q + 1] = v.y;
  }
}

__device__ __forceinline__ void res_pass_general(const ResArgs<double>& a, double* state, double* stage, double* vred,
                                                 const double* sD, int e0, int ne, int nn) {
  using T = double;
  const int t = threadIdx.x;
  constexpr int ST = ShellQuad::STAGE, RES_STATE = ResLay<T, ShellQuad>::SS;
  const int le = t / NPE, n = t % NPE, i = n % NP, k = n / NP;
  const bool act = t < NPE * ne;
  const int e = e0 + le;
  T* u = state + le * RES_STATE;
  T* sg = stage + le * ST;
  T sx = T(0), sy = T(0);  // pointwise shear terms
  if (act) {
    T dx[5], de[5];
    {
      T Di[NP], Dk[NP];
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        Di[q] = sD[i * NP + q];
        Dk[q] = sD[k * NP + q];
      }
#pragma unroll
      for (int f = 0; f < 5; ++f) {
        T x = T(0), y = T(0), ln[NP];
        ld_line(u + f * NPE + k * NP, ln);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          x = fma(Di[q], ln[q], x);
          y = fma(Dk[q], u[f * NPE + q * NP + i], y);
        }
        dx[f] = x;
        de[f] = y;
      }
    }
    const T* g = a.geo + (int64_t)e * 5 * NPE + n;
    const T i11 = g[0], i12 = g[NPE], i21 = g[2 * NPE], i22 = g[3 * NPE];
    const T W = g[4 * NPE] * a.ekeep[e];
    T gx[5], gy[5];
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      gx[f] = fma(de[f], i21, dx[f] * i11);
      gy[f] = fma(de[f], i22, dx[f] * i12);
    }
    const T* L = a.mat + (int64_t)a.emat[e] * MAT_STRIDE_DEV;
    const T ex = gx[0], ey = gy[2], gxy = gy[0] + gx[2];
    const T kx = gx[1], ky = gy[3], kxy = gy[1] + gx[3];
    const T gyz = u[3 * NPE + n] + gy[4], gxz = u[NPE + n] + gx[4];
    if (a.nslot > 0) {  // invJ12 / invJ21 as the reference has them (main_flat_shell.m:691-692)
      const T dux = dx[0] * i11 + de[0] * i12, dfxx = dx[1] * i11 + de[1] * i12;
      const T dvy = dx[2] * i21 + de[2] * i22, dfyy = dx[3] * i21 + de[3] * i22;
      vred[le * NPE + n] = a.sc.k0 * (a.sc.e31 * (dux + a.sc.hh * dfxx) + a.sc.e32 * (dvy + a.sc.hh * dfyy));
    }
    const T Nxx = L[0] * ex + L[1] * ey + L[2] * gxy + L[9] * kx + L[10] * ky + L[11] * kxy;
    const T Nyy = L[1] * ex + L[3] * ey + L[4] * gxy + L[10] * kx + L[12] * ky + L[13] * kxy;
    const T Nxy = L[2] * ex + L[4] * ey + L[5] * gxy + L[11] * kx + L[13] * ky + L[14] * kxy;
    const T Mxx = L[9] * ex + L[10] * ey + L[11] * gxy + L[15] * kx + L[16] * ky + L[17] * kxy;
    const T Myy = L[10] * ex + L[12] * ey + L[13] * gxy + L[16] * kx + L[18] * ky + L[19] * kxy;
    const T Mxy = L[11] * ex + L[13] * ey + L[14] * gxy + L[17] * kx + L[19] * ky + L[20] * kxy;
    const T Qy = L[6] * gyz + L[7] * gxz, Qx = L[7] * gyz + L[8] * gxz;
    const T w11 = W * i11, w12 = W * i12, w21 = W * i21, w22 = W * i22;
    const T Sx[5] = {Nxx, Mxx, Nxy, Mxy, Qx}, Sy[5] = {Nxy, Mxy, Nyy, Myy, Qy};
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      sg[f * NPE + n] = fma(w12, Sy[f], w11 * Sx[f]);
      sg[(5 + f) * NPE + i * NP + k] = fma(w22, Sy[f], w21 * Sx[f]);  // (eta lines contiguous)
    }
    sx = W * Qx;
    sy = W * Qy;
  }
  __syncthreads();
  if (act) {
    T Di[NP], Dk[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      Di[q] = sD[q * NP + i];
      Dk[q] = sD[q * NP + k];
    }
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      T F = f == 1 ? sx : f == 3 ? sy : T(0), lx[NP], le_[NP];
      ld_line(sg + f * NPE + k * NP, lx);
      ld_line(sg + (5 + f) * NPE + i * NP, le_);
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        F = fma(Di[q], lx[q], F);
        F = fma(Dk[q], le_[q], F);
      }
      u[(10 + f) * NPE + n] = F;
    }
    if (a.nslot > 0 && n == 0) {
      const int slot = a.esens[e];
      if (slot >= 0) {
        double v = 0.0;
        for (int q = 0; q < NPE; ++q) v += (double)vred[le * NPE + q];
        a.vsum[(int64_t)slot * a.nft + (nn - 1)] = v;
      }
    }
  }
  __syncthreads();
}

// --- FP32 shells in pairs ------------------------------------------------------
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ const float2* as2(const float* p) { return reinterpret_cast<const float2*>(p); }

// staging of an element: xi fluxes of (u, phi_x), (v, phi_y), w at 0, 72, 144 in
// node order, eta fluxes at 180, 252, 324 eta-major
__device__ __forceinline__ void res_pass_quad2(const ResArgs<float>& a, float* state, float* stage, float* vred,
                                               const float* sD, int e0, int ne, int nn) {
  using LY = ResLay<float, ShellQuad>;
  const int t = threadIdx.x;
  constexpr int ST = ShellQuad::STAGE;
  const int le = t / NPE, n = t % NPE, i = n % NP, k = n / NP;
  const bool act = t < NPE * ne;
  const int e = e0 + le;
  float* u = state + le * LY::SS;
  float* sg = stage + le * ST;
  auto line2 = [](const float* p, float2 (&o)[NP]) {  // six consecutive pairs, 16-byte aligned
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const float4 v = reinterpret_cast<const float4*>(p)[q];
      o[2 * q] = make_float2(v.x, v.y);
      o[2 * q + 1] = make_float2(v.z, v.w);
    }
  };
  float sx = 0.f, sy = 0.f;
  if (act) {
    float Di[NP], Dk[NP];
    ld_line(sD + i * NP, Di);
    ld_line(sD + k * NP, Dk);
    float2 dx[2], de[2];
#pragma unroll
    for (int pl = 0; pl < 2; ++pl) {
      float2 ln[NP], x, y;
      line2(u + pl * 72 + 12 * k, ln);
      const float2* col = as2(u + pl * 72) + i;
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        x = q == 0 ? mul2(bc2(Di[0]), ln[0]) : fma2(bc2(Di[q]), ln[q], x);
        y = q == 0 ? mul2(bc2(Dk[0]), col[0]) : fma2(bc2(Dk[q]), col[q * NP], y);
      }
      dx[pl] = x;
      de[pl] = y;
    }
    float wx = 0.f, wy = 0.f;
    {
      float ln[NP];
      ld_line(u + 144 + k * NP, ln);
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        wx = fmaf(Di[q], ln[q], wx);
        wy = fmaf(Dk[q], u[144 + q * NP + i], wy);
      }
    }
    const float* g = a.geo + (int64_t)e * 5 * NPE + n;
    const float i11 = g[0], i12 = g[NPE], i21 = g[2 * NPE], i22 = g[3 * NPE];
    const float W = g[4 * NPE] * a.ekeep[e];
    const float2 gxU = fma2(de[0], bc2(i21), mul2(dx[0], bc2(i11))), gyU = fma2(de[0], bc2(i22), mul2(dx[0], bc2(i12)));
    const float2 gxV = fma2(de[1], bc2(i21), mul2(dx[1], bc2(i11))), gyV = fma2(de[1], bc2(i22), mul2(dx[1], bc2(i12)));
    const float2 E3 = add2(gyU, gxV);
    const float gyz = u[72 + 2 * n + 1] + fmaf(wy, i22, wx * i12), gxz = u[2 * n + 1] + fmaf(wy, i21, wx * i11);
    if (a.nslot > 0) {  // invJ12 / invJ21 as the reference has them (main_flat_shell.m:691-692)
      const float2 sxU = fma2(de[0], bc2(i12), mul2(dx[0], bc2(i11))), syV = fma2(de[1], bc2(i22), mul2(dx[1], bc2(i21)));
      vred[le * NPE + n] = a.sc.k0 * (a.sc.e31 * (sxU.x + a.sc.hh * sxU.y) + a.sc.e32 * (syV.x + a.sc.hh * syV.y));
    }
    const float* tab = a.table + (int64_t)a.emat[e] * ShellQuad::CLASS32;
    const float2* L = as2(tab);
    auto row = [&](int q0, int q1, int q2) {
      float2 R = mul2(L[q0], bc2(gxU.x));
      R = fma2(L[q1], bc2(gyV.x), R);
      R = fma2(L[q2], bc2(E3.x), R);
      R = fma2(L[6 + q0], bc2(gxU.y), R);
      R = fma2(L[6 + q1], bc2(gyV.y), R);
      return fma2(L[6 + q2], bc2(E3.y), R);
    };
    const float2 XX = row(0, 1, 2), YY = row(1, 3, 4), XY = row(2, 4, 5);
    const float Qy = fmaf(tab[25], gxz, tab[24] * gyz), Qx = fmaf(tab[26], gxz, tab[25] * gyz);
    const float w11 = W * i11, w12 = W * i12, w21 = W * i21, w22 = W * i22;
    const int nT = i * NP + k;
    reinterpret_cast<float2*>(sg)[n] = fma2(bc2(w12), XY, mul2(bc2(w11), XX));
    reinterpret_cast<float2*>(sg + 72)[n] = fma2(bc2(w12), YY, mul2(bc2(w11), XY));
    sg[144 + n] = fmaf(w12, Qy, w11 * Qx);
    reinterpret_cast<float2*>(sg + 180)[nT] = fma2(bc2(w22), XY, mul2(bc2(w21), XX));
    reinterpret_cast<float2*>(sg + 252)[nT] = fma2(bc2(w22), YY, mul2(bc2(w21), XY));
    sg[324 + nT] = fmaf(w22, Qy, w21 * Qx);
    sx = W * Qx;
    sy = W * Qy;
  }
  __syncthreads();
  if (act) {
    float Ti[NP], Tk[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      Ti[q] = sD[q * NP + i];
      Tk[q] = sD[q * NP + k];
    }
    float F[5];
#pragma unroll
    for (int pl = 0; pl < 2; ++pl) {
      float2 lx[NP], ly[NP], c = make_float2(0.f, pl ? sy : sx);
      line2(sg + pl * 72 + 12 * k, lx);
      line2(sg + 180 + pl * 72 + 12 * i, ly);
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        c = fma2(bc2(Ti[q]), lx[q], c);
        c = fma2(bc2(Tk[q]), ly[q], c);
      }
      F[2 * pl] = c.x;
      F[2 * pl + 1] = c.y;
    }
    float lx[NP], ly[NP], c = 0.f;
    ld_line(sg + 144 + k * NP, lx);
    ld_line(sg + 324 + i * NP, ly);
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      c = fmaf(Ti[q], lx[q], c);
      c = fmaf(Tk[q], ly[q], c);
    }
    F[4] = c;
    LY::st_f(u + 2 * LY::UB + 2 * n, 2 * NPE, F);
    if (a.nslot > 0 && n == 0) {
      const int slot = a.esens[e];
      if (slot >= 0) {
        double v = 0.0;
        for (int q = 0; q < NPE; ++q) v += (double)vred[le * NPE + q];
        a.vsum[(int64_t)slot * a.nft + (nn - 1)] = v;
      }
    }
  }
  __syncthreads();
}

// 3D solid boxes: node (i, k) of layer z at 36 z + 6 k + i, sector value s(i, k)
// of layer z at 36 z + 9 s + 3 k + i.  A xi derivative flips the sector's xi
// parity, an eta derivative its eta parity, a zeta derivative neither.
__device__ __forceinline__ void res_pass_solid(const ResArgs<double>& a, double* state, double* stage, int e0, int ne) {
  using T = double;
  const int t = threadIdx.x, nt = blockDim.x;
  constexpr int ST = SolidBox::STAGE, SS = ResLay<T, SolidBox>::SS, N = S_NPE;
  for (int w = t; w < 81 * ne; w += nt) {
    const int le = w / 81, r = w % 81, fz = r / 9, m = r % 9, i = m % 3, k = m / 3;  // fz = 3 field + layer
    const T* u = state + le * SS + fz * 36;
    const T A = u[k * 6 + i], B = u[k * 6 + 5 - i], C = u[(5 - k) * 6 + i], D = u[(5 - k) * 6 + 5 - i];
    T* s = stage + le * ST + fz * 36 + m;
    const T ab = A + B, am = A - B, cd = C + D, cm = C - D;
    s[0] = ab + cd;
    s[9] = am + cm;
    s[18] = ab - cd;
    s[27] = am - cm;
  }
  __syncthreads();
  const int le = t / N, n = t % N;
  const bool act = t < N * ne;
  const int z = n / 36, q36 = n % 36, s = q36 / 9, m = q36 % 9, i = m % 3, k = m / 3;
  const int px = s & 1, py = s >> 1;
  const int e = e0 + le;
  T* sg = stage + le * ST;
  T* sr = sg + 3 * N;
  const T* tab = nullptr;
  const int ox = z * 36 + (s ^ 1) * 9 + 3 * k, oy = z * 36 + (s ^ 2) * 9 + i, oz = s * 9 + m;
  if (act) {
    tab = a.table + (int64_t)a.cls[e] * SolidBox::CLASS;
    const T* mx = tab + (px ? 0 : 9) + 3 * i;
    const T* my = tab + 18 + (py ? 0 : 9) + 3 * k;
    const T* mz = tab + 36 + 3 * z;
    const T x0 = mx[0], x1 = mx[1], x2 = mx[2], y0 = my[0], y1 = my[1], y2 = my[2], z0 = mz[0], z1 = mz[1], z2 = mz[2];
    auto dx = [&](int f, T c) { const T* p = sg + f * N + ox; return fma(x2, p[2], fma(x1, p[1], fma(x0, p[0], c))); };
    auto dz = [&](int f, T c) { const T* p = sg + f * N + oz; return fma(z2, p[72], fma(z1, p[36], fma(z0, p[0], c))); };
    auto dx0 = [&](int f) { const T* p = sg + f * N + ox; return fma(x2, p[2], fma(x1, p[1], x0 * p[0])); };
    auto dy0 = [&](int f) { const T* p = sg + f * N + oy; return fma(y2, p[6], fma(y1, p[3], y0 * p[0])); };
    auto dz0 = [&](int f) { const T* p = sg + f * N + oz; return fma(z2, p[72], fma(z1, p[36], z0 * p[0])); };
    // strains_spec_p.m: xx yy zz xy yz xz
    const T Exx = dx0(0), Eyy = dy0(1), Ezz = dz0(2), Exy = dx(1, dy0(0)), Eyz = dz(1, dy0(2)), Exz = dz(0, dx0(2));
    const T* L = tab + 45 + z * 9 + m;  // coefficient q at L[27 q]: D11 D12 D13 D14 D22 D23 D24 D33 D34 D44 D55 D56 D66
    auto l = [&](int q) { return L[27 * q]; };
    T* r = sr + n;
    r[0 * N] = fma(l(3), Exy, fma(l(2), Ezz, fma(l(1), Eyy, l(0) * Exx)));  // Sxx
    r[1 * N] = fma(l(6), Exy, fma(l(5), Ezz, fma(l(4), Eyy, l(1) * Exx)));  // Syy
    r[2 * N] = fma(l(8), Exy, fma(l(7), Ezz, fma(l(5), Eyy, l(2) * Exx)));  // Szz
    r[3 * N] = fma(l(9), Exy, fma(l(8), Ezz, fma(l(6), Eyy, l(3) * Exx)));  // Sxy
    r[4 * N] = fma(l(11), Exz, l(10) * Eyz);                                // Syz
    r[5 * N] = fma(l(12), Exz, l(11) * Eyz);                                // Sxz
  }
  __syncthreads();
  if (act) {
    const T* mx = tab + (px ? 9 : 0) + i;
    const T* my = tab + 18 + (py ? 9 : 0) + k;
    const T* mz = tab + 36 + z;
    const T x0 = mx[0], x1 = mx[3], x2 = mx[6], y0 = my[0], y1 = my[3], y2 = my[6], z0 = mz[0], z1 = mz[3], z2 = mz[6];
    auto sum = [&](int rx, int ry, int rz) {
      const T *p = sr + rx * N + ox, *q = sr + ry * N + oy, *r = sr + rz * N + oz;
      T c = fma(x2, p[2], fma(x1, p[1], x0 * p[0]));
      c = fma(y2, q[6], fma(y1, q[3], fma(y0, q[0], c)));
      return fma(z2, r[72], fma(z1, r[36], fma(z0, r[0], c)));
    };
    const T keep = a.ekeep[e];
    T* o = sg + n;  // (the sector values were last read before the barrier)
    o[0 * N] = keep * sum(0, 3, 5);
    o[1 * N] = keep * sum(3, 1, 4);
    o[2 * N] = keep * sum(5, 4, 2);
  }
  __syncthreads();
  for (int w = t; w < 81 * ne; w += nt) {
    const int l2 = w / 81, r = w % 81, fz = r / 9, mm = r % 9, ii = mm % 3, kk = mm / 3;
    const T* q = stage + l2 * ST + fz * 36 + mm;
    const T ee = q[0], oe = q[9], eo = q[18], oo = q[27];
    const T p0 = ee + eo, p1 = oe + oo, m0 = ee - eo, m1 = oe - oo;
    T* F = state + l2 * SS + 6 * N + fz * 36;
    F[kk * 6 + ii] = p0 + p1;
    F[kk * 6 + 5 - ii] = p0 - p1;
    F[(5 - kk) * 6 + ii] = m0 + m1;
    F[(5 - kk) * 6 + 5 - ii] = m0 - m1;
  }
  __syncthreads();
}

// FP32 solids, a thread per node and derivatives from whole lines.  Staging of an
// element: Sxx, Sxy, Sxz, Syz, Szz in node order, Sxy, Syy, Syz with eta fastest,
// all times the quadrature weight.
__device__ __forceinline__ void res_pass_solid_nodes(const ResArgs<float>& a, float* state, float* stage, const float* sD,
                                                     int e0, int ne) {
  constexpr int N = S_NPE, SS = ResLay<float, SolidNodes>::SS;
  const int t = threadIdx.x, le = t / N, n = t % N;
  const bool act = t < N * ne;
  const int z = n / 36, m = n % 36, i = m % NP, k = m / NP;
  const int e = e0 + le;
  float* u = state + le * SS;
  float* sg = stage + le * SolidNodes::STAGE;
  const float* tab = nullptr;
  if (act) {
    tab = a.table + (int64_t)a.cls[e] * SolidNodes::CLASS;
    const float hx = tab[0], hy = tab[1], hz = tab[2];
    float gx[3], gy[3], gz[3];
    {
      float Di[NP], Dk[NP];
      ld_line(sD + i * NP, Di);
      ld_line(sD + k * NP, Dk);
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        const float* p = u + f * N;
        float ln[NP], x = 0.f, y = 0.f, q3 = 0.f;
        ld_line(p + z * 36 + k * NP, ln);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          x = fmaf(Di[q], ln[q], x);
          y = fmaf(Dk[q], p[z * 36 + q * NP + i], y);
        }
#pragma unroll
        for (int q = 0; q < S_NZ; ++q) q3 = fmaf(D3m<float>(z, q), p[q * 36 + m], q3);
        gx[f] = hx * x;
        gy[f] = hy * y;
        gz[f] = hz * q3;
      }
    }
    // strains_spec_p.m: xx yy zz xy yz xz
    const float Exx = gx[0], Eyy = gy[1], Ezz = gz[2], Exy = gy[0] + gx[1], Eyz = gy[2] + gz[1], Exz = gx[2] + gz[0];
    const float W = tab[3] * Wg<float>(i) * Wg<float>(k) * W3m<float>(z) * a.ekeep[e];
    const float* L = tab + 4;  // D11 D12 D13 D14 D22 D23 D24 D33 D34 D44 D55 D56 D66
    const int nT = z * 36 + i * NP + k;
    const float Sxx = fmaf(L[3], Exy, fmaf(L[2], Ezz, fmaf(L[1], Eyy, L[0] * Exx)));
    const float Syy = fmaf(L[6], Exy, fmaf(L[5], Ezz, fmaf(L[4], Eyy, L[1] * Exx)));
    const float Szz = fmaf(L[8], Exy, fmaf(L[7], Ezz, fmaf(L[5], Eyy, L[2] * Exx)));
    const float Sxy = W * fmaf(L[9], Exy, fmaf(L[8], Ezz, fmaf(L[6], Eyy, L[3] * Exx)));
    const float Syz = W * fmaf(L[11], Exz, L[10] * Eyz), Sxz = W * fmaf(L[12], Exz, L[11] * Eyz);
    sg[0 * N + n] = W * Sxx;
    sg[1 * N + n] = Sxy;
    sg[2 * N + n] = Sxz;
    sg[3 * N + n] = Syz;
    sg[4 * N + n] = W * Szz;
    sg[5 * N + nT] = Sxy;
    sg[6 * N + nT] = W * Syy;
    sg[7 * N + nT] = Syz;
  }
  __syncthreads();
  if (act) {
    float Ti[NP], Tk[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      Ti[q] = sD[q * NP + i];
      Tk[q] = sD[q * NP + k];
    }
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      float lx[NP], ly[NP], x = 0.f, y = 0.f, q3 = 0.f;
      ld_line(sg + f * N + z * 36 + k * NP, lx);        // Sxx Sxy Sxz
      ld_line(sg + (5 + f) * N + z * 36 + i * NP, ly);  // Sxy Syy Syz
      const float* p = sg + (2 + f) * N + m;            // Sxz Syz Szz
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        x = fmaf(Ti[q], lx[q], x);
        y = fmaf(Tk[q], ly[q], y);
      }
#pragma unroll
      for (int q = 0; q < S_NZ; ++q) q3 = fmaf(D3m<float>(q, z), p[q * 36], q3);
      u[(6 + f) * N + n] = fmaf(tab[2], q3, fmaf(tab[1], y, tab[0] * x));
    }
  }
  __syncthreads();
}

// kAdj: the adjoint of the same operator.  lambda in place of u, the residuals
// of the point outputs in place of the excitation, and between the element
// passes and the exchange each element's (K_e^0 lambda)' u_{n-1}: the passes run
// with a factor of one, each node's thread adds its product with the stored
// forward state to an FP64 sum of its own and then scales the force.  The next
// step's states are asked into L2 during the update.  A step costs 7 to 25 % more
// than a forward one: 2 x 20x20 quads FP64 20.6 us (forward 19.4; element and node
// kernels 88), 16 x 18x18 plates FP64 71 (66; 170), 60x60 plate FP32 7.0 (6.0; 14.6).
template <typename T, class C, bool kAdj>
__global__ void __launch_bounds__(C::THREADS, C::ctas(sizeof(T))) k_resident(ResArgs<T> a, int nsteps) {
  extern __shared__ __align__(16) unsigned char smraw[];
  using LY = ResLay<T, C>;
  constexpr int NF = C::NF, N = C::NODES, SS = LY::SS, P = res_pieces<T, C>();
  uint4* codes = reinterpret_cast<uint4*>(smraw);
  T* state = reinterpret_cast<T*>(codes + (size_t)a.epc * N);
  T* imp = state + (size_t)a.epc * SS;  // records read, laid out as F
  T* stage = imp + (size_t)(LY::PARTS * LY::PITCH) * a.maximp;
  T* vred = stage + (size_t)a.epass * C::STAGE;
  __shared__ __align__(16) T sD[NPE];
  __shared__ int s_go;
  const int t = threadIdx.x, nt = blockDim.x, cta = blockIdx.x;
  const int e0 = cta * a.epc, nel = min(a.epc, a.fen - e0);
  const int ntot = nel * N;
  const int2* __restrict__ meta = a.meta + (int64_t)e0 * N;
  const int nn0 = *a.d_base;
  if (t == 0) s_go = 1;
  if constexpr (std::is_same<C, ShellQuad>::value || std::is_same<C, SolidNodes>::value)
    for (int q = t; q < NPE; q += nt) sD[q] = Dm<T>(q / NP, q % NP);
  {
    const bool odd = ((nn0 - a.nn_first) & 1);
    const T* cur = odd ? a.UB : a.UA;
    const T* prev = odd ? a.UA : a.UB;
    for (int w = t; w < ntot; w += nt) {
      const int g = meta[w].x & RES_NODE;
      codes[w] = a.codes[(int64_t)e0 * N + w];
      T* s = state + (w / N) * SS;
      T u[NF], d[NF];
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        u[f] = cur[f * a.nnode_pad + g];
        const T second = (a.dvalid ? a.dinc : prev)[f * a.nnode_pad + g];
        d[f] = RES_INC<T> && !a.dvalid ? u[f] - second : second;
      }
      LY::st_u(s, w % N, u);
      LY::st_u(s + LY::UB, w % N, d);
    }
  }
  const int x0 = a.exp_ptr[cta], xn = a.exp_ptr[cta + 1] - x0;
  const int i0 = a.imp_ptr[cta], in = a.imp_ptr[cta + 1] - i0;
  bool bad = false;
  __syncthreads();
  for (int step = 0; step < nsteps; ++step) {
    const int nn = nn0 + step;
    const unsigned tag = a.tag0 + (unsigned)step;
    for (int p = 0; p < nel; p += a.epass) {
      const int ne = min(a.epass, nel - p);
      if constexpr (std::is_same<C, SolidBox>::value)
        res_pass_solid(a, state + (size_t)p * SS, stage, e0 + p, ne);
      else if constexpr (std::is_same<C, SolidNodes>::value)
        res_pass_solid_nodes(a, state + (size_t)p * SS, stage, sD, e0 + p, ne);
      else if constexpr (LY::PAIRS)
        res_pass_quad2(a, state + (size_t)p * SS, stage, vred, sD, e0 + p, ne, nn);
      else if constexpr (std::is_same<C, ShellRect>::value)
        res_pass_rect(a, state + (size_t)p * SS, stage, vred, e0 + p, ne, nn);
      else
        res_pass_general(a, state + (size_t)p * SS, stage, vred, sD, e0 + p, ne, nn);
    }
    if constexpr (kAdj) {
      const int left = nsteps - 2 - step;
      const T* um = left >= 0 ? a.um + left * a.keep_stride : a.um0;
      double* gp = a.gpart + (int64_t)e0 * N;
      for (int w = t; w < ntot; w += nt) {
        const T* ug = um + (meta[w].x & RES_NODE);
        T* fs = state + (w / N) * SS + 2 * LY::UB + LY::PITCH * (w % N);
        const T kp = a.keep[e0 + w / N];
        T F[NF], dot = T(0);
        LY::ld_f(fs, LY::PITCH * N, F);
#pragma unroll
        for (int f = 0; f < NF; ++f) {
          dot += F[f] * ug[f * a.nnode_pad];
          F[f] *= kp;
        }
        gp[w] += (double)dot;
        LY::st_f(fs, LY::PITCH * N, F);
      }
      __syncthreads();
    }
    uint4* const xb = a.xch + (size_t)(step & 1) * a.nrec * P;
    for (int w = t; w < xn; w += nt) {
      T F[NF];
      LY::ld_f(state + a.exp_off[x0 + w], LY::PITCH * N, F);
      xch_store<NF>(xb + (size_t)(x0 + w) * P, F, tag);
    }
    for (int w = t; w < in; w += nt) {
      const uint4* r = xb + (size_t)a.imp_rec[i0 + w] * P;
      uint4 p[P];
      bool ok = false;
      for (int it = 0; it < a.spin; ++it) {
        ok = true;
#pragma unroll
        for (int q = 0; q < P; ++q) p[q] = ld_piece(r + q);
#pragma unroll
        for (int q = 0; q < P; ++q) ok = ok && p[q].y == tag && p[q].w == tag;
        if (ok || ((it & 255) == 255 && *(volatile unsigned*)a.abortw == a.tag0)) break;
      }
      if (!ok) {  // the wait gave up: every CTA leaves after its step
        *(volatile unsigned*)a.abortw = a.tag0;
        atomicOr(a.flag, 2);
        s_go = 0;
      }
      T v[NF];
      xch_unpack<NF>(p, v);
      LY::st_f(imp + LY::PITCH * w, LY::PITCH * a.maximp, v);
    }
    __syncthreads();
    // update every copy of every node
    const bool frame = a.fs.frm_int > 0 && (nn % a.fs.frm_int) == 0;
    const bool guard = guard_step(a.fs, nn);
    const int imp_off = (int)(imp - state);
    for (int w = t; w < ntot; w += nt) {
      T km[4];
      ld4(a.km + ((int64_t)e0 * N + w) * 4, km);
      const int bits = res_bits(km[3]);
      const uint4 cd = codes[w];
      T* s = state + (w / N) * SS;
      T F[NF];
      auto add = [&](int q) {  // the force of the copy at offset q
        T v[NF];
        LY::ld_f(state + q, LY::PITCH * (q < imp_off ? N : a.maximp), v);
#pragma unroll
        for (int f = 0; f < NF; ++f) F[f] += v[f];
      };
      const unsigned c0 = cd.x & 0xffff;
      {
        const int q = c0 == RES_LIST ? a.lists[meta[w].y + 2] : (int)c0;
        LY::ld_f(state + q, LY::PITCH * (q < imp_off ? N : a.maximp), F);
      }
      if (c0 != RES_LIST) {
        if ((cd.x >> 16) != RES_NONE) {
          add(cd.x >> 16);
          if ((cd.y & 0xffff) != RES_NONE) {
            add(cd.y & 0xffff);
            if ((cd.y >> 16) != RES_NONE) {
              add(cd.y >> 16);
              const unsigned more[4] = {cd.z & 0xffff, cd.z >> 16, cd.w & 0xffff, cd.w >> 16};
              if (more[0] != RES_NONE) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                  if (more[q] != RES_NONE) add(more[q]);
              }
            }
          }
        }
      } else {
        const int* li = a.lists + meta[w].y;
        for (int q = 1; q < li[0]; ++q) add(li[2 + q]);
      }
      if constexpr (kAdj) {
        if (bits & RES_HAS_OUT) {
          const int* o = a.out_list + a.out_start[(int64_t)e0 * N + w];
          const int cnt = o[0];
          for (int q = 1; q <= cnt; ++q) {
            const int of = a.out_field[o[q]];
            const T v = (T)a.asig[(int64_t)o[q] * a.nft + (nn - 1)];
#pragma unroll
            for (int f = 0; f < NF; ++f) F[f] += f == of ? v : T(0);
          }
        }
      }
      if (!kAdj && (bits & RES_FORCED)) {
        const int* li = a.lists + meta[w].y;
        const int nc = li[0], nfc = li[1];
        for (int q = 0; q < nfc; ++q) {
          const int fq = li[2 + nc + q];
          const T v = (T)(-a.fq_val[fq] * a.st[(int64_t)a.fq_scen[fq] * a.nft + (nn - 1)]);
          const int ff = a.fq_field[fq];
#pragma unroll
          for (int f = 0; f < NF; ++f) F[f] += f == ff ? v : T(0);
        }
      }
      if constexpr (NF == 5 && !kAdj)
        if (a.pr.npf > 0) F[4] -= pressure_load(a.pr, nn, a.nnode_pad, (int64_t)(meta[w].x & RES_NODE));
      T u[NF], un[NF], d0[NF], d1[NF];
      LY::ld_u(s, w % N, u);
      LY::ld_u(s + LY::UB, w % N, d0);
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        const int c = res_coef<C>(f);
        if constexpr (RES_INC<T>) {
          d1[f] = fma(a.k1[c], d0[f], -km[c] * F[f]);
          un[f] = u[f] + d1[f];
          if (!kAdj) d1[f] = res_coarse(d1[f], un[f]);
        } else {  // d0 is u_{n-1}
          un[f] = fma(-km[c], F[f], fma(a.k1[c], u[f] - d0[f], u[f]));
          d1[f] = u[f];
        }
      }
      LY::st_u(s, w % N, un);
      LY::st_u(s + LY::UB, w % N, d1);
      constexpr int own_out = RES_OWNER | RES_HAS_OUT;
      if (!kAdj && (bits & own_out) == own_out) {  // displ(nn,:): the state at the start of the step
        const int* o = a.out_list + a.out_start[(int64_t)e0 * N + w];
        const int cnt = o[0];
        for (int q = 1; q <= cnt; ++q) {
          const int of = a.out_field[o[q]];
          T v = u[0];
#pragma unroll
          for (int f = 1; f < NF; ++f) v = of == f ? u[f] : v;
          a.displ[(int64_t)o[q] * a.nft + (nn - 1)] = (double)v;
        }
      }
      if ((frame || guard || kAdj || a.keep_u) && (bits & RES_OWNER)) {
        const int64_t g = meta[w].x & RES_NODE;
        if constexpr (kAdj) {
          const int left = nsteps - 3 - step;
          const T* um = left >= 0 ? a.um + left * a.keep_stride : a.um0;
#pragma unroll
          for (int f = 0; f < NF; ++f) asm volatile("prefetch.global.L2 [%0];" ::"l"(um + f * a.nnode_pad + g));
        } else if (a.keep_u) {
          T* k = a.keep_u + step * a.keep_stride + g;
#pragma unroll
          for (int f = 0; f < NF; ++f) k[f * a.nnode_pad] = un[f];
        }
#pragma unroll
        for (int f = 0; f < NF; ++f) {
          if (!kAdj && frame) {
            const int fc = nn / a.fs.frm_int - a.fs.fc0;
            if (fc >= 0 && fc < a.fs.nframes) {
              T* base = a.frames + (int64_t)fc * a.fs.nfields * a.nnode_pad + g;
              const int sU = a.fs.slot[f], sV = a.fs.slot[5 + f], sA = a.fs.slot[10 + f];
              if (sU >= 0) base[sU * a.nnode_pad] = u[f];
              if (sV >= 0) base[sV * a.nnode_pad] = a.a1 * (RES_INC<T> ? d1[f] + d0[f] : un[f] - d0[f]);
              if (sA >= 0) base[sA * a.nnode_pad] = a.a0 * (RES_INC<T> ? d1[f] - d0[f] : d0[f] - T(2) * u[f] + un[f]);
            }
          }
          if (guard && (!isfinite(un[f]) || (f == NF - 1 && u[f] > a.blowup))) bad = true;
        }
      }
    }
    __syncthreads();
    if (!s_go) break;
  }
  if (s_go && a.end) {  // the owners' copies are the state
    const bool odd = ((nn0 + nsteps - a.nn_first) & 1);
    T* cur = odd ? a.UB : a.UA;
    T* prev = odd ? a.UA : a.UB;
    for (int w = t; w < ntot; w += nt) {
      const int x = meta[w].x;
      if (!(x & RES_OWNER)) continue;
      const int g = x & RES_NODE;
      const T* s = state + (w / N) * SS;
      T u[NF], d[NF];
      LY::ld_u(s, w % N, u);
      LY::ld_u(s + LY::UB, w % N, d);
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        cur[f * a.nnode_pad + g] = u[f];
        prev[f * a.nnode_pad + g] = RES_INC<T> ? u[f] - d[f] : d[f];
        a.dinc[f * a.nnode_pad + g] = d[f];
      }
    }
  }
  if (bad) atomicOr(a.flag, 1);
}

// dJ/dd_e = -sum over steps and nodes of (K_e^0 lambda)' u_{n-1}, in the plan's order
__global__ void k_resident_grad(const double* __restrict__ gpart, const int* __restrict__ ord, int fen, int nodes,
                                double* grad) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= fen) return;
  double s = 0.0;
  for (int q = 0; q < nodes; ++q) s += gpart[(int64_t)r * nodes + q];
  grad[ord[r]] = -s;
}

}  // namespace shm
