// Device helpers shared by the plain and mixed step kernels.
#pragma once
#include <cuda_bf16.h>

#include "wf_device.cuh"

namespace wf {

constexpr double WF_PI = 3.14159265358979323846;
constexpr double MIN_PS_FOR_NBSEARCH = 1.e-6;  // Source/Domain.cpp:28
constexpr int BLOCK = 256;                      // threads of the per-particle kernels

__device__ __forceinline__ double col(const DevPtrs& P, int c, size_t N, int i) { return P.f[(size_t)c * N + i]; }
__device__ __forceinline__ double& colw(const DevPtrs& P, int c, size_t N, int i) { return P.f[(size_t)c * N + i]; }
__device__ __forceinline__ int icol(const DevPtrs& P, int c, size_t N, int i) { return P.i[(size_t)c * N + i]; }

// Counters of a search that begins, by the thread that decides it; without the
// Verlet-skin reuse every search re-sorts (with it, k_skin_check decides).
__device__ __forceinline__ void search_begin(const DevPtrs& P, const DomainConst& K) {
  StepState* s = P.st;
  s->pair_count = 0;
  s->contact_pair_count = 0;
  s->surface_count = 0;
  s->cp_count = 0;
  s->nan_count = 0;
  s->maxdisp2_bits = 0;
  s->nb_searches += 1;
  if (!K.skin_on) { s->search_full = 1; s->nb_full_searches += 1; }
}

// Deterministic block reduction (fixed shuffle tree, then fixed order across
// warps) of one value per thread; the result is valid in thread 0.
template <int OP>  // 0 sum, 1 max, 2 min
__device__ __forceinline__ double block_reduce(double v, double* sh) {
  for (int off = 16; off > 0; off >>= 1) {
    double o = __shfl_down_sync(0xffffffffu, v, off);
    v = (OP == 0) ? v + o : (OP == 1 ? fmax(v, o) : fmin(v, o));
  }
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    int nw = blockDim.x >> 5;
    double r = sh[0];
    for (int k = 1; k < nw; ++k) r = (OP == 0) ? r + sh[k] : (OP == 1 ? fmax(r, sh[k]) : fmin(r, sh[k]));
    v = r;
  }
  return v;
}

// Largest (MIN: smallest) value of a warp in every lane, NaN left out as fmax
// and fmin leave it out, by two 32-bit integer reductions of an order-keeping
// key instead of five FP64 maxima (an FP64 instruction takes 16 cycles of an SM).
template <bool MIN>
__device__ __forceinline__ double warp_extreme(double v) {
  unsigned long long k = (unsigned long long)__double_as_longlong(v);
  const bool nan = (k & 0x7fffffffffffffffull) > 0x7ff0000000000000ull;
  k = (k >> 63) ? ~k : k | 0x8000000000000000ull;  // ascending as unsigned
  if (MIN) k = ~k;
  if (nan) k = 0;  // unkeyed again a NaN, when every lane holds one
  const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32));
  const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32) == hi ? (unsigned)k : 0u);
  k = ((unsigned long long)hi << 32) | lo;
  if (MIN) k = ~k;
  k = (k >> 63) ? k & 0x7fffffffffffffffull : ~k;
  return __longlong_as_double((long long)k);
}

// Block reduction of NS sums and of an optional largest and smallest value with
// one barrier.  The sums share a warp's halves: two of them take the first
// addition in one instruction (lanes below 16 keep the first, the others the
// second), four of them the second one in one, so two to four sums cost six
// FP64 additions instead of five each; every sum's additions are those of
// block_reduce's tree in the same order.  Warps are added in their order.
// Sum q goes to out[q], then the largest and the smallest value (thread q
// writes out[q]).  sh: 6 * 32 doubles, free when it is called.
template <int NS, bool MAXMIN>
__device__ __forceinline__ void block_reduce_all(const double (&s)[NS], double mx0, double mx1, double mn, double* sh,
                                                 double* const* out) {
  static_assert(NS >= 2 && NS <= 4, "two to four sums");
  constexpr int NV = NS + 1 + (MAXMIN ? 2 : 0);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const bool up = l & 16, up8 = l & 8;
  auto fold = [](bool u, int off, double a, double b) {  // a's sum in the lower lanes of the pair, b's in the upper
    const double keep = u ? b : a, give = u ? a : b;
    return keep + __shfl_xor_sync(0xffffffffu, give, off);
  };
  double v = fold(up, 16, s[0], s[1]);
  if (NS > 2) {
    const double t = NS == 4 ? fold(up, 16, s[2], s[NS - 1]) : s[NS > 2 ? 2 : 0] + __shfl_xor_sync(0xffffffffu, s[NS > 2 ? 2 : 0], 16);
    v = fold(up8, 8, v, t);
  } else {
    v = v + __shfl_xor_sync(0xffffffffu, v, 8);
  }
  v = v + __shfl_xor_sync(0xffffffffu, v, 4);
  v = v + __shfl_xor_sync(0xffffffffu, v, 2);
  v = v + __shfl_xor_sync(0xffffffffu, v, 1);
  // lane 0: sum 0, lane 16: sum 1, lane 8: sum 2, lane 24: sum 3
  if (l == 0) sh[w] = v;
  if (l == 16) sh[32 + w] = v;
  if (NS > 2 && l == 8) sh[64 + w] = v;
  if (NS > 3 && l == 24) sh[96 + w] = v;
  const double a = warp_extreme<false>(mx0);
  if (l == 1) sh[NS * 32 + w] = a;
  if (MAXMIN) {
    const double b = warp_extreme<false>(mx1), c = warp_extreme<true>(mn);
    if (l == 2) sh[(NS + 1) * 32 + w] = b;
    if (l == 3) sh[(NS + 2) * 32 + w] = c;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    const int q = threadIdx.x, nw = blockDim.x >> 5;
    double r = sh[q * 32];
    for (int k = 1; k < nw; ++k) {
      const double o = sh[q * 32 + k];
      r = q < NS ? r + o : (MAXMIN && q == NS + 2 ? fmin(r, o) : fmax(r, o));
    }
    *out[q] = r;
  }
}

// FP32 <-> FP64 conversions of the mixed kernels on the integer pipe.  GB300
// runs a conversion on the FP64 pipe at 2 per clock and SM, as slow as an FP64
// add (`bench.py --pipe-rates` for the add; conversions measured 2.07), while
// integer instructions issue at 64 lanes per clock: the ten or so integer
// instructions below take a third of a conversion's time, and a split a
// seventh of its four FP64-pipe instructions.  The FP64 pipe was 58 % busy in
// the rate-stress kernel and 81 % in the kick, a third of it conversions.
// They round as the hardware does (to nearest even); values outside the
// normal range, other than zero, take the hardware's conversion.
__device__ __forceinline__ double f2d(float f) {
  const unsigned u = __float_as_uint(f), a = u & 0x7fffffffu;
  const bool normal = a - 0x00800000u < 0x7f000000u;
  if (normal || a == 0u) {  // exponent rebiased from 127 to 1023, mantissa shifted by 29
    const unsigned h = normal ? (a >> 3) + 0x38000000u : 0u;
    return __hiloint2double((int)(h | (u & 0x80000000u)), (int)(u << 29));
  }
  return (double)f;
}
__device__ __forceinline__ float d2f(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v), a = hi & 0x7fffffffu;
  const bool normal = a - 0x38100000u < 0x0fe00000u;  // 2^-126 <= |v| < 2^128
  if (normal || (a | lo) == 0u) {
    // round to nearest even at bit 29; a carry out of the mantissa raises the exponent
    const unsigned long long r = (((unsigned long long)a << 32) | lo) + 0x0fffffffu + ((lo >> 29) & 1u);
    const unsigned f = normal ? (unsigned)(r >> 29) - 0xc0000000u : 0u;
    return __uint_as_float(f | (hi & 0x80000000u));
  }
  return __double2float_rn(v);
}
// Float-float split of a double: hi = fl(v), lo = fl(v - hi).  This form is for
// ff_split3: it sets odd where v is neither zero nor in its range.
__device__ __forceinline__ void ff_split_int(double v, float& hi, float& lo, bool& odd) {
  const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v), a = h & 0x7fffffffu;
  const bool normal = a - 0x3b500000u < 0x0c800000u;  // 2^-74 <= |v| < 2^126: the remainder's last bit is a normal FP32 too
  odd = odd || !(normal || (a | l) == 0u);
  const unsigned lsb = (l >> 29) & 1u, sign = h & 0x80000000u;
  const unsigned long long r = (((unsigned long long)a << 32) | l) + 0x0fffffffu + lsb;
  hi = __uint_as_float((normal ? (unsigned)(r >> 29) - 0xc0000000u : 0u) | sign);
  // v - hi in units of the last place of v: the low 29 bits, less 2^29 where they rounded up
  const unsigned low = l & 0x1fffffffu, up = (low + 0x0fffffffu + lsb) & 0x20000000u;
  const unsigned scale = normal ? (((a >> 20) - 948u) << 23) | sign : 0u;  // 2^(exponent - 52)
  lo = (float)((int)low - (int)up) * __uint_as_float(scale);
}
__device__ __forceinline__ void ff_split(double v, float& hi, float& lo) {
  const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v), a = h & 0x7fffffffu;
  if (a - 0x3b500000u < 0x0c800000u) {  // 2^-74 <= |v| < 2^126: the remainder's last bit is a normal FP32 too
    const unsigned lsb = (l >> 29) & 1u, sign = h & 0x80000000u;
    const unsigned long long r = (((unsigned long long)a << 32) | l) + 0x0fffffffu + lsb;
    hi = __uint_as_float(((unsigned)(r >> 29) - 0xc0000000u) | sign);
    // v - hi in units of the last place of v: the low 29 bits, less 2^29 where they rounded up
    const unsigned low = l & 0x1fffffffu, up = (low + 0x0fffffffu + lsb) & 0x20000000u;
    const unsigned scale = (((a >> 20) - 948u) << 23) | sign;  // 2^(exponent - 52)
    lo = (float)((int)low - (int)up) * __uint_as_float(scale);
    return;
  }
  if ((a | l) == 0u) { hi = __uint_as_float(h); lo = 0.0f; return; }
  hi = __double2float_rn(v);
  lo = __double2float_rn(v - (double)hi);
}
// f() where c holds, behind a branch that a warp without such a lane takes.  A
// short body would be compiled to instructions predicated off, which still take
// their slots of the FP64 pipe; the count of this loop is hidden from the
// compiler.  No vote: the lanes here need not be together.
template <class F>
__device__ __forceinline__ void branch_over(bool c, F f) {
  int n = c ? 1 : 0;
  asm volatile("" : "+r"(n));
#pragma unroll 1
  while (n > 0) {
    f();
    --n;
    asm volatile("" : "+r"(n));
  }
}
// Three splits that share one branch over the conversions (the kick kernel,
// whose work this is: 37.5 -> 31.4 us at 982,072 particles, with contact 69 ->
// 59 us at 1,171,832; the rate-stress and density kernels lost more to the
// registers that grouping holds).
__device__ __forceinline__ void ff_split3(const double v[3], float hi[3], float lo[3]) {
  bool odd = false;
  for (int d = 0; d < 3; ++d) ff_split_int(v[d], hi[d], lo[d], odd);
  branch_over(odd, [&] {
    for (int d = 0; d < 3; ++d) {
      hi[d] = __double2float_rn(v[d]);
      lo[d] = __double2float_rn(v[d] - (double)hi[d]);
    }
  });
}
// Low-half group: x = (xlo0, xlo1), y = (xlo2, vlo0), z = (vlo1, vlo2) as bf16
// pairs (first value in the low 16 bits), w = a float.  A bf16 is the upper
// half of an FP32, so unpacking is a shift or a mask.
__device__ __forceinline__ unsigned short bf16_bits(float f) { return __bfloat16_as_ushort(__float2bfloat16_rn(f)); }
__device__ __forceinline__ float bf16_pair(float a, float b) {
  return __uint_as_float((unsigned)bf16_bits(a) | ((unsigned)bf16_bits(b) << 16));
}
__device__ __forceinline__ float bf16_first(float p) { return __uint_as_float(__float_as_uint(p) << 16); }
__device__ __forceinline__ float bf16_second(float p) { return __uint_as_float(__float_as_uint(p) & 0xffff0000u); }
__device__ __forceinline__ float4 lo_pack(const float xl[3], const float vl[3], float w) {
  return make_float4(bf16_pair(xl[0], xl[1]), bf16_pair(xl[2], vl[0]), bf16_pair(vl[1], vl[2]), w);
}
// v lo component d sits in 16-bit half 3 + d of the group.
__device__ __forceinline__ unsigned short* lo_v_half(float4* group, int d) {
  return reinterpret_cast<unsigned short*>(group) + 3 + d;
}

// Velocity component d of particle i into the current (next) float4 groups.
__device__ __forceinline__ float* rec_v_hi(float4* r, size_t N, int d) {  // r: the record's column base + i
  return d == 0 ? reinterpret_cast<float*>(r + (size_t)RC_XV * N) + 3 : reinterpret_cast<float*>(r + (size_t)RC_VW * N) + d - 1;
}
__device__ __forceinline__ void rec_set_v(const DevPtrs& P, size_t N, int i, int d, double v, bool next) {
  static_assert((int)RN_XV == (int)RC_XV && (int)RN_VW == (int)RC_VW && (int)RN_L == (int)RC_L, "same places in both records");
  float4* r = (next ? P.rn : P.rc) + i;
  float h, l;
  ff_split(v, h, l);
  *rec_v_hi(r, N, d) = h;
  *lo_v_half(r + (size_t)RC_L * N, d) = bf16_bits(l);
}

// The current velocity record of particle i from its three FP64 components
// (the other fields of the three groups carried over).
__device__ __forceinline__ void rec_set_v3(const DevPtrs& P, size_t N, int i, const double v[3]) {
  float4* r = P.rc + i;
  float h[3], l[3];
  ff_split3(v, h, l);
  *rec_v_hi(r, N, 0) = h[0];
  *reinterpret_cast<float2*>(r + (size_t)RC_VW * N) = make_float2(h[1], h[2]);
  *lo_v_half(r + (size_t)RC_L * N, 0) = bf16_bits(l[0]);
  reinterpret_cast<float*>(r + (size_t)RC_L * N)[2] = bf16_pair(l[1], l[2]);
}

// Batched domain: flag the particle's specimen as yielding once its plastic
// strain passes the rebuild threshold (Domain.cpp:28), the per-specimen form of
// the max-plastic-strain test of the rebuild schedule.
__device__ __forceinline__ void mark_yield(const DevPtrs& P, const DomainConst& K, size_t N, int i, double pl) {
  if (K.nspec > 0 && pl > MIN_PS_FOR_NBSEARCH) {
    SpecState* sp = P.sp + icol(P, I_SPEC, N, i);
    if (!sp->yielded_next) sp->yielded_next = 1;
  }
}

// Amplitude lookup (SPH::amplitude::getValAtTime, Source/Domain.h:69-89).
__device__ __forceinline__ double amp_value(const DomainTables* T, int amp_id, double t, bool* found) {
  for (int k = 0; k < T->namp; ++k) {
    if (T->amp[k].id != amp_id) continue;
    *found = true;
    const double* tt = T->amp_t + T->amp[k].offset;
    const double* vv = T->amp_v + T->amp[k].offset;
    int i = T->amp[k].n - 1;
    bool end = false;
    while (!end) { i--; if (i == 0 || t > tt[i]) end = true; }
    return vv[i] + (vv[i + 1] - vv[i]) / (tt[i + 1] - tt[i]) * (t - tt[i]);
  }
  return 0.0;
}

// The velocity the BCs of zone id impose at time t (GeneralAfter,
// WeldForm.cpp:51-120): each of the zone's BCs in the order added, a later one
// overriding an earlier; an amplitude BC applies only where its table covers
// t.  False when none applies.  k_bc applies this to its list of BC
// particles; the kick and drift kernels apply it to their own particle in
// place of the BC passes that would follow them.
__device__ __forceinline__ bool bc_velocity(const DomainTables* T, int id, double t, double v[3]) {
  int lo, hi;
  bc_range(T, id, lo, hi);
  bool hit = false;
  for (int r = lo; r < hi; ++r) {
    const BCDev& b = T->bc[T->bc_order[r]];
    if (b.value_type == 0) {
      hit = true;
      for (int d = 0; d < 3; ++d) v[d] = b.value[d];
    } else {
      bool found = false;
      double val = b.amp_factor * amp_value(T, b.amp_id, t, &found);
      if (found) {
        hit = true;
        for (int d = 0; d < 3; ++d) v[d] = val * b.value[d];
      }
    }
  }
  return hit;
}

// CalcConvHeat (Thermal.cpp:339-389, 3D; Fraser Eq. 3-121): a particle with
// Thermal_BC == TH_BC_CONVECTION exchanges heat with the ambient temperature
// T_inf through its contact area dS^2 = (m / rho)^(2/3):
// q_conv = rho h_conv dS^2 (T_inf - T) / m, at the step's updated density and
// temperature.  Other particles keep their q_conv (0 from the constructor).
__device__ __forceinline__ double conv_heat(const DevPtrs& P, size_t N, int i, double rho, double T) {
  if (P.i[(size_t)I_THBC * N + i] != 1) return col(P, C_QCONV, N, i);
  double m = col(P, C_MASS, N, i);
  double dS2 = pow(m / rho, 2.0 / 3.0);
  double q = rho * col(P, C_HCONV, N, i) * dS2 * (col(P, C_TINF, N, i) - T) / m;
  colw(P, C_QCONV, N, i) = q;
  return q;
}

// Johnson-Cook flow stress (Source/Material.cpp:6-25).
__device__ __forceinline__ double jc_yield(const MaterialDev& M, double strain, double strain_rate, double temp) {
  double T_h = (temp - M.T_t) / (M.T_m - M.T_t);
  double f = 1.0;
  if (strain_rate > M.eps_0) f = (1.0 + M.C * log(strain_rate / M.eps_0));
  return (M.A + M.B * pow(strain, M.n)) * f * (1.0 - pow(T_h, M.jm));
}
// Hollomon flow stress with plateau (Source/Material.cpp:59-64).
__device__ __forceinline__ double hollomon_yield(const MaterialDev& M, double strain) {
  if (strain + M.eps0 > M.eps1) return M.K * pow(strain + M.eps0, M.m);
  return M.sy0;
}

// Cubic-spline kernel W(q) (Functions.cpp:25-36, 3D) without its constant
// 1/(pi h^3): the tensile-instability term only uses ratios of W.
__device__ __forceinline__ double kernel_shape(double q) {
  if (q < 1.0) return 1.0 - (3.0 / 2.0) * q * q + (3.0 / 4.0) * q * q * q;
  else if (q < 2.0) return (1.0 / 4.0) * (2.0 - q) * (2.0 - q) * (2.0 - q);
  return 0.0;
}

// Symmetric 3x3 eigen-decomposition by cyclic Jacobi rotations (a published
// method; the reference calls GSL's gsl_eigen_symmv through Rotation,
// Functions.cpp:381-395).  s: xx yy zz xy xz yz.  Returns the eigenvalues in
// L and the eigenvectors as columns of V.  The sweep count is bounded.
__device__ __forceinline__ void eig_sym3(const double s[6], double L[3], double V[3][3]) {
  double a[3][3] = {{s[0], s[3], s[4]}, {s[3], s[1], s[5]}, {s[4], s[5], s[2]}};
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) V[r][c] = (r == c) ? 1.0 : 0.0;
  for (int sweep = 0; sweep < 50; ++sweep) {
    double off = a[0][1] * a[0][1] + a[0][2] * a[0][2] + a[1][2] * a[1][2];
    double diag = a[0][0] * a[0][0] + a[1][1] * a[1][1] + a[2][2] * a[2][2];
    if (off == 0.0 || off <= 1e-36 * diag) break;
    for (int e = 0; e < 3; ++e) {
      int p = e == 2 ? 1 : 0, q = e == 0 ? 1 : 2;
      if (a[p][q] == 0.0) continue;
      double theta = (a[q][q] - a[p][p]) / (2.0 * a[p][q]);
      double t = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
      double c = 1.0 / sqrt(t * t + 1.0), sn = t * c;
      for (int k = 0; k < 3; ++k) {
        double akp = a[k][p], akq = a[k][q];
        a[k][p] = c * akp - sn * akq;
        a[k][q] = sn * akp + c * akq;
      }
      for (int k = 0; k < 3; ++k) {
        double apk = a[p][k], aqk = a[q][k];
        a[p][k] = c * apk - sn * aqk;
        a[q][k] = sn * apk + c * aqk;
      }
      for (int k = 0; k < 3; ++k) {
        double vkp = V[k][p], vkq = V[k][q];
        V[k][p] = c * vkp - sn * vkq;
        V[k][q] = sn * vkp + c * vkq;
      }
    }
  }
  for (int k = 0; k < 3; ++k) L[k] = a[k][k];
}

// The same cyclic Jacobi iteration in FP32, for the mixed form, whose
// tensile-instability stress enters the FP32 pair terms: converged to FP32
// resolution (off-diagonal squares below 1e-14 of the diagonal's).  A rotation
// angle beyond FP32 range takes t = 1 / (2 theta).
__device__ __forceinline__ void eig_sym3f(const float s[6], float L[3], float V[3][3]) {
  float a[3][3] = {{s[0], s[3], s[4]}, {s[3], s[1], s[5]}, {s[4], s[5], s[2]}};
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) V[r][c] = (r == c) ? 1.0f : 0.0f;
  for (int sweep = 0; sweep < 20; ++sweep) {
    float off = a[0][1] * a[0][1] + a[0][2] * a[0][2] + a[1][2] * a[1][2];
    float diag = a[0][0] * a[0][0] + a[1][1] * a[1][1] + a[2][2] * a[2][2];
    if (off == 0.0f || off <= 1e-14f * diag) break;
    for (int e = 0; e < 3; ++e) {
      int p = e == 2 ? 1 : 0, q = e == 0 ? 1 : 2;
      if (a[p][q] == 0.0f) continue;
      float theta = (a[q][q] - a[p][p]) / (2.0f * a[p][q]);
      float t = fabsf(theta) > 1e15f ? 0.5f / theta
                                      : (theta >= 0.0f ? 1.0f : -1.0f) / (fabsf(theta) + sqrtf(theta * theta + 1.0f));
      float c = rsqrtf(t * t + 1.0f), sn = t * c;
      for (int k = 0; k < 3; ++k) {
        float akp = a[k][p], akq = a[k][q];
        a[k][p] = c * akp - sn * akq;
        a[k][q] = sn * akp + c * akq;
      }
      for (int k = 0; k < 3; ++k) {
        float apk = a[p][k], aqk = a[q][k];
        a[p][k] = c * apk - sn * aqk;
        a[q][k] = sn * apk + c * aqk;
      }
      for (int k = 0; k < 3; ++k) {
        float vkp = V[k][p], vkq = V[k][q];
        V[k][p] = c * vkp - sn * vkq;
        V[k][q] = sn * vkp + c * vkq;
      }
    }
  }
  for (int k = 0; k < 3; ++k) L[k] = a[k][k];
}

// Radial-return constitutive update of one particle, Particle::CalcStressStrain
// (Source/Particle.cpp:960-1067), on symmetric storage (xx yy zz xy xz yz).
// sr: strain rate (6), rr: rotation rate (xy xz yz of the antisymmetric part).
// Returns dep (plastic strain increment).
struct StressIO {
  double tau[6], sig[6], eps[6], epl[6], epli[6];
  double pressure, pl_strain, delta_pl_strain, sigmay, Ep, esr;
  double sc = 1.0, sy_new = 0.0;  // branch record: scale factor and the step's flow stress
};
__device__ __forceinline__ double stress_update(StressIO& s, const double sr[6], const double rr[3], double rho,
                                                double rho0, double Cs, double P0, double G, double T, int fail,
                                                int model, const MaterialDev* M, double dt) {
  s.pressure = P0 + (Cs * Cs) * (rho - rho0);  // EOS case 0, Functions.cpp:206-212
  // Full matrices: S (symmetric tau), W (antisymmetric rotation rate).
  double S[3][3] = {{s.tau[0], s.tau[3], s.tau[4]}, {s.tau[3], s.tau[1], s.tau[5]}, {s.tau[4], s.tau[5], s.tau[2]}};
  double W[3][3] = {{0.0, rr[0], rr[1]}, {-rr[0], 0.0, rr[2]}, {-rr[1], -rr[2], 0.0}};
  // SRT = S W^T, RS = W S; entries summed k = 2, 1, 0 (matvec.h Mult order).
  const int ui[6] = {0, 1, 2, 0, 0, 1}, uj[6] = {0, 1, 2, 1, 2, 2};
  double tr = sr[0] + sr[1] + sr[2];
  double s3 = 1.0 / 3.0 * tr;
  double twoG = 2.0 * G;
  double t6[6];
  for (int c = 0; c < 6; ++c) {
    int a = ui[c], b = uj[c];
    double srt = S[a][2] * W[b][2] + S[a][1] * W[b][1] + S[a][0] * W[b][0];
    double rs = W[a][2] * S[2][b] + W[a][1] * S[1][b] + W[a][0] * S[0][b];
    double dev = sr[c] - (c < 3 ? s3 : 0.0);
    t6[c] = dt * (twoG * dev + srt + rs) + s.tau[c];
  }
  double d01 = sr[0] - sr[1], d12 = sr[1] - sr[2], d20 = sr[2] - sr[0];
  s.esr = sqrt(0.5 * (d01 * d01 + d12 * d12 + d20 * d20) + 3.0 * (sr[3] * sr[3] + sr[5] * sr[5] + sr[4] * sr[4]));
  double dep = 0.0;
  if (fail == 1) {
    double J2 = 0.5 * (t6[0] * t6[0] + 2.0 * t6[3] * t6[3] + 2.0 * t6[4] * t6[4] + t6[1] * t6[1] +
                       2.0 * t6[5] * t6[5] + t6[2] * t6[2]);
    double sig_trial = sqrt(3.0 * J2);
    double ratio = s.sigmay / sig_trial;
    double sc = (1.0 < ratio) ? 1.0 : ratio;  // std::min(ratio, 1.0)
    for (int c = 0; c < 6; ++c) t6[c] = sc * t6[c];
    if (model == 1 && M) s.sigmay = hollomon_yield(*M, s.pl_strain);
    else if (model == 2 && M) s.sigmay = jc_yield(*M, s.pl_strain, s.esr, T);
    s.sc = sc;
    s.sy_new = s.sigmay;
    if (sig_trial > s.sigmay) {
      if (s.Ep < 0) s.Ep = M ? M->E : 0.0;
      dep = (sig_trial - s.sigmay) / (3. * G + s.Ep);
      s.pl_strain += dep;
      s.delta_pl_strain = dep;
      if (model == 0) s.sigmay += dep * s.Ep;
    }
  }
  for (int c = 0; c < 6; ++c) s.tau[c] = t6[c];
  for (int c = 0; c < 6; ++c) s.sig[c] = (c < 3 ? -s.pressure : 0.0) + t6[c];
  if (dep > 0.0) {
    double f = dep / s.sigmay;
    s.epli[0] = f * (s.sig[0] - 0.5 * (s.sig[1] + s.sig[2]));
    s.epli[1] = f * (s.sig[1] - 0.5 * (s.sig[0] + s.sig[2]));
    s.epli[2] = f * (s.sig[2] - 0.5 * (s.sig[0] + s.sig[1]));
    s.epli[3] = 1.5 * f * s.sig[3];
    s.epli[4] = 1.5 * f * s.sig[4];
    s.epli[5] = 1.5 * f * s.sig[5];
    for (int c = 0; c < 6; ++c) s.epl[c] = s.epl[c] + s.epli[c];
  }
  for (int c = 0; c < 6; ++c) s.eps[c] = dt * sr[c] + s.eps[c];
  return dep;
}

// Plastic work heat source (Particle::CalcPlasticWorkHeat, Particle.cpp:922-939):
// q = Sigma : (Strain_pl_incr / dt) with the off-diagonal pairs doubled.
__device__ __forceinline__ double plastic_heat_f(const double sig[6], const double epli[6], double f) {  // f = 1 / dt
  return sig[0] * (f * epli[0]) + 2.0 * sig[3] * (f * epli[3]) + 2.0 * sig[4] * (f * epli[4]) + sig[1] * (f * epli[1]) +
         2.0 * sig[5] * (f * epli[5]) + sig[2] * (f * epli[2]);
}
__device__ __forceinline__ double plastic_heat(const double sig[6], const double epli[6], double dt) {
  return plastic_heat_f(sig, epli, 1. / dt);
}

}  // namespace wf
