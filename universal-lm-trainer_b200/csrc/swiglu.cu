// SwiGLU gate of the feed-forward block (sm_100a), HBM-bound elementwise work.
//
// The reference computes  w2( silu(w1 x) * (w3 x) )  (train.py:1966-1975) with
// three PyTorch kernels in the forward (silu, mul) and five in the backward.  Here
// one kernel each way, over the two GEMM outputs a = w1 x and b = w3 x:
//   fwd:  y  = r(r(silu(a)) * b)
//   bwd:  db = r(dy * r(silu(a))),  da = r(r(dy * b) * silu'(a)),
//         silu'(a) = s (1 + a (1 - s)),  s = 1 / (1 + exp(-a)),
// where r() rounds to the tensors' dtype: the intermediate roundings are the ones
// eager PyTorch makes between its kernels (each kernel computes in fp32 and writes
// the tensor dtype).  fp32 results agree with the reference's path to the last bit except
// where exp() itself differs by an ulp; 16-bit results differ in the few roundings that an
// error of 2^-19 in s can flip (y over all values of a, b = 1: two of fp16, none of bf16).
// 16-byte vectors; bytes moved: fwd 3 per element pair (2 reads + 1 write) x elem size, bwd 5.
#include "common.cuh"

namespace ulm {
namespace {

constexpr int kThreads = 256;

template <typename T> struct VecN { static constexpr int N = 16 / sizeof(T); };

template <typename T>
__device__ __forceinline__ void unpack(const uint4& u, float (&f)[VecN<T>::N]) {
  if constexpr (sizeof(T) == 4) {
    const float* p = reinterpret_cast<const float*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = p[i];
  } else {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 t = Cvt<T>::unpack2(w[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
  }
}

template <typename T>
__device__ __forceinline__ uint4 pack(const float (&f)[VecN<T>::N]) {
  uint4 u;
  if constexpr (sizeof(T) == 4) {
    float* p = reinterpret_cast<float*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] = f[i];
  } else {
    uint32_t* w = reinterpret_cast<uint32_t*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = Cvt<T>::pack2(f[2 * i], f[2 * i + 1]);
  }
  return u;
}

template <typename T>
__device__ __forceinline__ float rnd(float v) { return Cvt<T>::to_f(Cvt<T>::from_f(v)); }

// s = sigmoid(a) and silu(a).  fp32 tensors: the forms ATen's kernels use.  16-bit tensors: one ex2 and one reciprocal
// on the special-function unit instead of expf and an IEEE division each: the divisions' fix-up code, not memory, was what
// the kernels waited for (see kVecs).  Relative error of s and u: 2^-19 for |a| <= 16, 2^-17 down to a = -88, below which s
// is 0 as in the divided form.  Over 0.4 G random values of each type and of deviation 0.3, 1 and 3, the rms error of y, da
// and db against float64 is that of the divided form within what so many roundings can show (1e-6 of itself, da of fp16
// 4e-6).  Newton steps that bring s and u to within an ulp of the divisions flip fewer roundings and cost 14 us of 66
// forward, 6 of 104 backward (32768 x 2048 bf16).
template <typename T>
__device__ __forceinline__ void sigmoid_silu(float a, float& s, float& u) {
  if constexpr (sizeof(T) == 4) {
    const float d = 1.f + expf(-a);
    s = 1.f / d;
    u = a / d;                                           // the form ATen's kernel uses
  } else {
    float e;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(a * -1.4426950408889634f));
    asm("rcp.approx.f32 %0, %1;" : "=f"(s) : "f"(1.f + e));   // no ftz: s goes down to 2^-128 before e overflows
    u = a * s;
  }
}

// 16-byte vectors per thread and tensor, all loaded before the first is worked on.  The grid covers the tensor once:
// what bounds the kernels is HBM, and the block scheduler keeps more loads in flight than a grid-stride loop.
// Measured at 32768 x 2048 bf16, before (expf, IEEE division, grid-stride) -> now: forward 83 -> 61 us (6.6 TB/s),
// backward 135 -> 100 us (6.7 TB/s).  One or four vectors forward, two backward: within 3 %.
template <typename T> constexpr int kVecsFwd = 2;
template <typename T> constexpr int kVecsBwd = 1;

// Where vector v of the gate's operands lies: a and b (da and db) are dense, or column blocks of a wider matrix (the two
// halves of one projection's output): rows of vpr vectors, `stride` vectors apart.
struct Rows { uint32_t vpr; int64_t stride; };
template <bool ROWS>
__device__ __forceinline__ int64_t operand_vec(int64_t v, const Rows& rw) {
  if constexpr (!ROWS) return v;
  const uint32_t u = (uint32_t)v, r = u / rw.vpr;        // fewer than 2^32 vectors (checked by the host)
  return (int64_t)r * rw.stride + (u - r * rw.vpr);
}

template <typename T, bool ROWS>
__global__ void __launch_bounds__(kThreads)
swiglu_fwd_kernel(const T* __restrict__ a, const T* __restrict__ b, T* __restrict__ y, int64_t nvec, int64_t n, const Rows rw) {
  constexpr int N = VecN<T>::N, K = kVecsFwd<T>;
  const int64_t v0 = (int64_t)blockIdx.x * (kThreads * K) + threadIdx.x;
  uint4 ra[K], rb[K];
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (v0 + k * kThreads < nvec) {
      const int64_t o = operand_vec<ROWS>(v0 + k * kThreads, rw);
      ra[k] = __ldg(reinterpret_cast<const uint4*>(a) + o);
      rb[k] = __ldg(reinterpret_cast<const uint4*>(b) + o);
    }
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (v0 + k * kThreads < nvec) {
      float fa[N], fb[N], fy[N];
      unpack<T>(ra[k], fa);
      unpack<T>(rb[k], fb);
#pragma unroll
      for (int i = 0; i < N; ++i) {
        float s, u;
        sigmoid_silu<T>(fa[i], s, u);
        fy[i] = rnd<T>(u) * fb[i];
      }
      reinterpret_cast<uint4*>(y)[v0 + k * kThreads] = pack<T>(fy);
    }
  // tail shorter than a vector
  if (blockIdx.x == 0 && threadIdx.x < (int)(n - nvec * N)) {
    const int64_t i = nvec * N + threadIdx.x;
    float s, u;
    sigmoid_silu<T>(Cvt<T>::to_f(a[i]), s, u);
    y[i] = Cvt<T>::from_f(rnd<T>(u) * Cvt<T>::to_f(b[i]));
  }
}

template <typename T>
__device__ __forceinline__ void bwd_one(float fa, float fb, float fg, float& da, float& db) {
  float s, u;
  sigmoid_silu<T>(fa, s, u);
  db = fg * rnd<T>(u);
  da = rnd<T>(fg * fb) * (s * (1.f + fa * (1.f - s)));
}

template <typename T, bool ROWS>
__global__ void __launch_bounds__(kThreads)
swiglu_bwd_kernel(const T* __restrict__ a, const T* __restrict__ b, const T* __restrict__ dy,
                  T* __restrict__ da, T* __restrict__ db, int64_t nvec, int64_t n, const Rows rw) {
  constexpr int N = VecN<T>::N, K = kVecsBwd<T>;
  const int64_t v0 = (int64_t)blockIdx.x * (kThreads * K) + threadIdx.x;
  uint4 ra[K], rb[K], rg[K];
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (v0 + k * kThreads < nvec) {
      const int64_t o = operand_vec<ROWS>(v0 + k * kThreads, rw);
      ra[k] = __ldg(reinterpret_cast<const uint4*>(a) + o);
      rb[k] = __ldg(reinterpret_cast<const uint4*>(b) + o);
      rg[k] = __ldg(reinterpret_cast<const uint4*>(dy) + v0 + k * kThreads);
    }
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (v0 + k * kThreads < nvec) {
      float fa[N], fb[N], fg[N], oa[N], ob[N];
      unpack<T>(ra[k], fa);
      unpack<T>(rb[k], fb);
      unpack<T>(rg[k], fg);
#pragma unroll
      for (int i = 0; i < N; ++i) bwd_one<T>(fa[i], fb[i], fg[i], oa[i], ob[i]);
      const int64_t o = operand_vec<ROWS>(v0 + k * kThreads, rw);
      reinterpret_cast<uint4*>(da)[o] = pack<T>(oa);
      reinterpret_cast<uint4*>(db)[o] = pack<T>(ob);
    }
  if (blockIdx.x == 0 && threadIdx.x < (int)(n - nvec * N)) {
    const int64_t i = nvec * N + threadIdx.x;
    float oa, ob;
    bwd_one<T>(Cvt<T>::to_f(a[i]), Cvt<T>::to_f(b[i]), Cvt<T>::to_f(dy[i]), oa, ob);
    da[i] = Cvt<T>::from_f(oa);
    db[i] = Cvt<T>::from_f(ob);
  }
}

unsigned grid_for(int64_t nvec, int per_thread) {
  const int64_t per = (int64_t)kThreads * per_thread, blocks = (nvec + per - 1) / per;
  return (unsigned)(blocks < 1 ? 1 : blocks);
}
bool too_many(int64_t n) { return n / 4 / kThreads > 0x7ffffff0LL; }      // blocks of the smallest launch per element

bool aligned16(const void* p) { return p && !(reinterpret_cast<uintptr_t>(p) & 15); }

// d == 0: dense operands; otherwise rows of d elements, `stride` elements apart (y and dy are dense either way)
int check_swiglu(const ulm_swiglu_args* p, int64_t d, int64_t stride, const char* who) {
  if (!p) return fail(ULM_ERR_ARG, "%s: null args", who);
  if (p->dtype != ULM_F16 && p->dtype != ULM_BF16 && p->dtype != ULM_F32) return fail(ULM_ERR_ARG, "%s: bad dtype", who);
  if (p->n < 0) return fail(ULM_ERR_ARG, "%s: negative size", who);
  if (too_many(p->n)) return fail(ULM_ERR_TOO_LARGE, "%s: too many elements", who);
  if (d) {
    const int64_t vec = p->dtype == ULM_F32 ? 4 : 8;
    if (d < 0 || d % vec || stride % vec || stride < d || p->n % d) return fail(ULM_ERR_ARG, "%s: rows and their stride must be whole 16-byte vectors", who);
    if (p->n / vec > 0xffffffffLL || d / vec > 0xffffffffLL) return fail(ULM_ERR_TOO_LARGE, "%s: too many elements", who);
  }
  return ULM_OK;
}

template <typename T>
void swiglu_launch(const ulm_swiglu_args* p, bool bwd, int64_t d, int64_t stride) {
  cudaStream_t st = (cudaStream_t)p->stream;
  const int64_t nvec = p->n / VecN<T>::N;
  const Rows rw{(uint32_t)(d / VecN<T>::N), stride / VecN<T>::N};
  const T *a = (const T*)p->a, *b = (const T*)p->b, *dy = (const T*)p->dy;
  T *y = (T*)p->y, *da = (T*)p->da, *db = (T*)p->db;
  const unsigned grid = grid_for(nvec, bwd ? kVecsBwd<T> : kVecsFwd<T>);
  if (bwd && d) swiglu_bwd_kernel<T, true><<<grid, kThreads, 0, st>>>(a, b, dy, da, db, nvec, p->n, rw);
  else if (bwd) swiglu_bwd_kernel<T, false><<<grid, kThreads, 0, st>>>(a, b, dy, da, db, nvec, p->n, rw);
  else if (d) swiglu_fwd_kernel<T, true><<<grid, kThreads, 0, st>>>(a, b, y, nvec, p->n, rw);
  else swiglu_fwd_kernel<T, false><<<grid, kThreads, 0, st>>>(a, b, y, nvec, p->n, rw);
}

int swiglu(const ulm_swiglu_args* p, bool bwd, int64_t d, int64_t stride, const char* who) {
  if (int rc = check_swiglu(p, d, stride, who)) return rc;
  if (p->n == 0) return ULM_OK;
  if (!aligned16(p->a) || !aligned16(p->b) || (bwd ? !aligned16(p->dy) || !aligned16(p->da) || !aligned16(p->db) : !aligned16(p->y)))
    return fail(ULM_ERR_ARG, "%s: %s must be non-null and 16-byte aligned", who, bwd ? "a, b, dy, da, db" : "a, b, y");
  if (p->dtype == ULM_F16) swiglu_launch<__half>(p, bwd, d, stride);
  else if (p->dtype == ULM_BF16) swiglu_launch<__nv_bfloat16>(p, bwd, d, stride);
  else swiglu_launch<float>(p, bwd, d, stride);
  return check_launch(who);
}

}  // namespace
}  // namespace ulm

extern "C" int ulm_swiglu_fwd(const ulm_swiglu_args* p) { return ulm::swiglu(p, false, 0, 0, "ulm_swiglu_fwd"); }
extern "C" int ulm_swiglu_bwd(const ulm_swiglu_args* p) { return ulm::swiglu(p, true, 0, 0, "ulm_swiglu_bwd"); }

extern "C" int ulm_swiglu_rows(const ulm_swiglu_args* p, int32_t backward, int64_t d, int64_t row_stride) {
  if (d <= 0) return ulm::fail(ULM_ERR_ARG, "ulm_swiglu_rows: d must be positive");
  return ulm::swiglu(p, backward != 0, d, row_stride, "ulm_swiglu_rows");
}
