// rowkernels.cuh -- the innermost-axis kernels of the GB300 hybrid
// convolution (complex rows and Hermitian rows), templated on the
// multiplier so that both the library's built-in multipliers and a
// caller's device functor (include/fftwpp_gb300_mult.cuh) are compiled into
// the row kernel itself: the multiply stays straight-line code on registers
// between the forward and inverse transforms, as FFTW++ calls its
// multiplier between them (Convolution::operate, convolve.h:1120-1135).
#pragma once

#include "kernels.cuh"

#include <algorithm>
#include <climits>
#include <cooperative_groups.h>
#include <type_traits>

namespace fgb {

// ---------------------------------------------------------------------------
// Multipliers (convolve.cc:26-110 and the 2D advection Jacobian), applied to
// the A values X[0..A-1] of one transformed slot; results overwrite
// X[0..B-1].  "Real" multipliers act lane-wise on the two doubles of a slot,
// which is how the reference applies them to its double-valued buffers
// (realMultBinary, convolve.cc:60-83).
template<typename T>
__device__ __forceinline__ void applyMult(int kind, cplx<T> *X, int A)
{
  switch(kind) {
    case MULT_BINARY:
      X[0]=cmul(X[0],X[1]);
      break;
    case MULT_REALBINARY:
      X[0]=mk(X[0].x*X[1].x,X[0].y*X[1].y);
      break;
    case MULT_CORRELATION:
      X[0]=cmulconj(X[0],X[1]);
      break;
    case MULT_REALJACOBIAN:
      X[0]=mk(fma(X[0].x,X[3].x,-X[1].x*X[2].x),
              fma(X[0].y,X[3].y,-X[1].y*X[2].y));
      break;
    case MULT_JACOBIAN:
      X[0]=cmul(X[0],X[3])-cmul(X[1],X[2]);
      break;
    case MULT_REALJACADJ: {
      // Inputs u0..u3 and the back-propagated field g; outputs the four
      // lane-wise partial products dJ/du_i * g of J = u0 u3 - u1 u2.
      cplx<T> g=X[4];
      cplx<T> u0=X[0], u1=X[1], u2=X[2], u3=X[3];
      X[0]=mk(g.x*u3.x,g.y*u3.y);
      X[1]=mk(-g.x*u2.x,-g.y*u2.y);
      X[2]=mk(-g.x*u1.x,-g.y*u1.y);
      X[3]=mk(g.x*u0.x,g.y*u0.y);
      break;
    }
    case MULT_DOT: {
      // Sum of A/2 binary products: X[0] = sum_k X[k] X[A/2+k].
      int K=A/2;
      cplx<T> s=cmul(X[0],X[K]);
      for(int k=1; k < K; ++k) s=s+cmul(X[k],X[K+k]);
      X[0]=s;
      break;
    }
    case MULT_REALDOT: {
      // The same on real data (two doubles per complex slot).
      int K=A/2;
      cplx<T> s=mk(X[0].x*X[K].x,X[0].y*X[K].y);
      for(int k=1; k < K; ++k)
        s=mk(fma(X[k].x,X[K+k].x,s.x),fma(X[k].y,X[K+k].y,s.y));
      X[0]=s;
      break;
    }
    default:
      break;
  }
}

// Compile-time input/output counts of the fixed-arity multipliers; the
// row kernels are instantiated per multiplier so that the fused multiply is
// straight-line code on registers (MULT_GENERIC: runtime kind and counts).
#define MULT_GENERIC (-1)
template<int K> struct MultArity {static const int A=0, B=0;};
template<> struct MultArity<MULT_BINARY> {static const int A=2, B=1;};
template<> struct MultArity<MULT_REALBINARY> {static const int A=2, B=1;};
template<> struct MultArity<MULT_REALJACOBIAN> {static const int A=4, B=1;};
template<> struct MultArity<MULT_REALJACADJ> {static const int A=5, B=4;};

// Values in and out of a multiplier type, 0 where they are known only at run
// time.
template<class Mul> struct MulArity;

// Multiply one transformed slot: the A values at X[sp(base+a*stride)] in,
// the B results back to X[sp(base+b*stride)].
template<int K, typename T>
__device__ __forceinline__ void multiplySlot(cplx<T> *X, int base, int stride,
                                             int A, int B, int kind)
{
  if constexpr(MultArity<K>::A > 0) {
    constexpr int KA=MultArity<K>::A, KB=MultArity<K>::B;
    cplx<T> v[KA];
#pragma unroll
    for(int a=0; a < KA; ++a) v[a]=nrm(X[sp(base+a*stride)]);
    applyMult(K,v,KA);
#pragma unroll
    for(int b=0; b < KB; ++b) X[sp(base+b*stride)]=v[b];
  } else {
    cplx<T> v[FGB_MAXA];
    for(int a=0; a < A; ++a) v[a]=nrm(X[sp(base+a*stride)]);
    applyMult(kind,v,A);
    for(int b=0; b < B; ++b) X[sp(base+b*stride)]=v[b];
  }
}

// The specialised instantiation serving a (mult, A, B), or MULT_GENERIC.
inline int multVariant(int mult, int A, int B)
{
  switch(mult) {
    case MULT_BINARY: return A == 2 && B == 1 ? MULT_BINARY : MULT_GENERIC;
    case MULT_REALBINARY:
      return A == 2 && B == 1 ? MULT_REALBINARY : MULT_GENERIC;
    case MULT_REALJACOBIAN:
      return A == 4 && B == 1 ? MULT_REALJACOBIAN : MULT_GENERIC;
    case MULT_REALJACADJ:
      return A == 5 && B == 4 ? MULT_REALJACADJ : MULT_GENERIC;
    default: return MULT_GENERIC;
  }
}

// ---------------------------------------------------------------------------
// The multiplier as a type parameter of the innermost-axis kernels.  A
// built-in multiplier K is BuiltinMult<K>; a caller's device functor F is
// UserMult<F> (include/fftwpp_gb300_mult.cuh), which also receives each
// slot's position on the padded grid.

template<int K> struct BuiltinMult {
  static constexpr bool positional=false;
  // A slot held in registers (fixed arity).
  template<typename T>
  __device__ __forceinline__ void slot(cplx<T> *v) const
  {
    applyMult(K,v,MultArity<K>::A);
  }
  template<typename T>
  __device__ __forceinline__ void operator()(cplx<T> *X, int base, int stride,
                                             int A, int B, int kind) const
  {
    multiplySlot<K>(X,base,stride,A,B,kind);
  }
};

// The position of a slot handed to a position-dependent multiplier: for
// every axis d (outermost first) the transformed index index[d], the
// position on the padded grid of axis d, 0 <= index[d] < size[d] (the
// padded length); on a real outer axis the frequency 0 <= index[0] <=
// size[0]/2.  These are the values the reference's Indices::index[] and
// fftBase::index(r, i) give a multiplier (convolve.h:48-82, 297-326).
struct Indices {
  int dim;
  int index[3];
  int size[3];
};

// Natural index of position p after a decimation-in-frequency transform
// (fftDIF) over the given radices: p = sum_s d_s n/(R_0...R_s) maps to
// k = d_0 + R_0 (d_1 + R_1 (d_2 + ...)).
template<typename R>
__device__ __forceinline__ int digitRev(int p, int n, int nst, const R *radix)
{
  int k=0, w=n, mul=1;
  for(int s=0; s < nst; ++s) {
    const int r=radix[s];
    w /= r;
    const int d=p/w;
    p -= d*w;
    k += d*mul;
    mul *= r;
  }
  return k;
}

__device__ __forceinline__ int outerAxisIndex(const IndexMap& im, int d,
                                              long long row)
{
  if(d == 0 && im.real0) return (int) row;
  const int m=im.m[d];
  const int r=(int) (row/m);
  int j=(int) (row-(long long) r*m);
  if(im.rev[d]) j=digitRev(j,m,im.nst[d],im.radix[d]);
  return im.q[d]*j+r;
}

// Indices of the outer axes of innermost-kernel row `row`; the caller
// fills in the inner entry.
__device__ __forceinline__ Indices outerIndices(const IndexMap& im,
                                                long long row)
{
  Indices ix;
  ix.dim=im.dim;
  for(int d=0; d < 3; ++d) {
    ix.size[d]=d < im.dim ? im.N[d] : 1;
    ix.index[d]=0;
  }
  if(im.dim == 2) ix.index[0]=outerAxisIndex(im,0,row);
  else if(im.dim == 3) {
    const long long r0=row/im.rowsY;
    ix.index[0]=outerAxisIndex(im,0,r0);
    ix.index[1]=outerAxisIndex(im,1,row-r0*im.rowsY);
  }
  return ix;
}

__device__ __forceinline__ double nrmS(double a) {return a;}
__device__ __forceinline__ float nrmS(float a) {return a;}
__device__ __forceinline__ ff nrmS(ff a) {return nrm(a);}

// A caller's functor F: static constexpr int A, B (values in, results out)
// and a device call operator template<class V> void operator()(V *v, const
// Indices& ix) const, V = cplx<T> on complex data and T on real data (a
// Hermitian innermost axis: one real value per grid point, as the reference
// presents double buffers to its real multipliers).
template<class F> struct UserMult {
  static constexpr bool positional=true;
  F f;
  // A slot held in registers; the two real grid points k and k+1 of one.
  template<typename T>
  __device__ __forceinline__ void slot(cplx<T> *v, const Indices& ix) const
  {
    f(v,ix);
  }
  template<typename T>
  __device__ __forceinline__ void slotReal(cplx<T> *v, Indices ix, int k) const
  {
    T u[F::A], w[F::A];
#pragma unroll
    for(int a=0; a < F::A; ++a) {
      u[a]=v[a].x;
      w[a]=v[a].y;
    }
    ix.index[ix.dim-1]=k;
    f(u,ix);
    ix.index[ix.dim-1]=k+1;
    f(w,ix);
#pragma unroll
    for(int b=0; b < F::B; ++b) v[b]=mk(u[b],w[b]);
  }
  template<typename T>
  __device__ __forceinline__ void at(cplx<T> *X, int base, int stride,
                                     const Indices& ix) const
  {
    cplx<T> v[F::A];
#pragma unroll
    for(int a=0; a < F::A; ++a) v[a]=nrm(X[sp(base+a*stride)]);
    f(v,ix);
#pragma unroll
    for(int b=0; b < F::B; ++b) X[sp(base+b*stride)]=v[b];
  }
};

template<int K> struct MulArity<BuiltinMult<K>> {
  static constexpr int A=MultArity<K>::A, B=MultArity<K>::B;
};
template<class F> struct MulArity<UserMult<F>> {
  static constexpr int A=F::A, B=F::B;
};

// One slot of a complex row: entry j of residue r (REV: j in the
// digit-reversed order of the row FFT) of row `row`.
template<class Mul, bool REV, typename T>
__device__ __forceinline__ void mulRowSlot(const Mul& mul, const RowPlan<T>& P,
                                           cplx<T> *X, int base, int stride,
                                           long long row, int j, int r)
{
  if constexpr(Mul::positional) {
    const int jn=REV ? digitRev(j,P.fp.n,P.fp.nst,P.fp.radix) : j;
    int k=P.q*jn+r;
    long long orow=row;
    if(P.im.longQ > 0) {               // long rows: column k1 of outer row
      orow=row/P.im.longQ;
      k=(int) (row-orow*P.im.longQ)+P.im.longQ*jn;
    }
    Indices ix=outerIndices(P.im,orow);
    ix.index[P.im.dim-1]=k;
    mul.at(X,base,stride,ix);
  } else {
    mul(X,base,stride,P.A,P.B,P.mult);
  }
}

// One slot of a fused row held in registers: entry p of the transform's
// digit-reversed order, of row `row`.
template<class Mul, typename T>
__device__ __forceinline__ void mulFusedSlot(const Mul& mul,
                                             const RowPlan<T>& P, cplx<T> *v,
                                             long long row, int p)
{
  if constexpr(Mul::positional) {
    const int jn=digitRev(p,P.fz.n,P.fz.nst,P.fz.radix);
    int k=jn;
    long long orow=row;
    if(P.im.longQ > 0) {                 // long rows: column k1 of outer row
      orow=row/P.im.longQ;
      k=(int) (row-orow*P.im.longQ)+P.im.longQ*jn;
    }
    Indices ix=outerIndices(P.im,orow);
    ix.index[P.im.dim-1]=k;
    mul.slot(v,ix);
  } else mul.slot(v);
}

// The same for a Hermitian row (real grid points 2t and 2t+1).
template<class Mul, typename T>
__device__ __forceinline__ void mulFusedSlot(const Mul& mul,
                                             const HermRowPlan<T>& P,
                                             cplx<T> *v, long long row, int p)
{
  if constexpr(Mul::positional) {
    const int tn=digitRev(p,P.fz.n,P.fz.nst,P.fz.radix);
    mul.slotReal(v,outerIndices(P.im,row),2*tn);
  } else mul.slot(v);
}

// ---------------------------------------------------------------------------
// FP64 values at the interface of the float-float mode.  The first kernel of
// a convolution reads the caller's FP64 arrays and the last one writes them
// (RowPlan::io64); complex FP64 and float-float elements are both 16 bytes,
// so offsets are unchanged.  The split avoids the FP64 pipe: hi keeps the
// leading 24 significand bits of x, lo the float nearest to the remaining
// 29, so hi + lo = x to 2^-48 relative; values outside [2^-70, 2^101)
// (zero, subnormals, huge values) take the FP64 conversion.
//
// Range guard: FP64 data span exponents far beyond a float's, so every
// input array a is scaled by an exact power of two 2^-sh[a] on the way in
// (its largest magnitude then lies in [1, 2)) and every output b by
// 2^sh[8+b] on the way out (ffScaleKernel in kernels.cu chooses them from
// the data and the multiplier).  Scaling by a power of two only moves the
// exponent, so it costs no accuracy.

__device__ __forceinline__ ff toFF(double x, int sh=0)
{
  unsigned long long b=(unsigned long long) __double_as_longlong(x);
  const int ef=(int) ((b >> 52) & 0x7ff);
  const int e=ef-1023-sh;
  if(ef == 0 || ef == 0x7ff || e < -70 || e > 100) {
    // keep 2^(e-52) a normal float: the FP64 conversion
    const double xs=sh ? scalbn(x,-sh) : x;
    float h=__double2float_rn(xs);
    return ff(h,__double2float_rn(xs-(double) h));
  }
  unsigned sign=(unsigned) (b >> 32) & 0x80000000u;
  float hi=__uint_as_float(sign | ((unsigned) (e+127) << 23) |
                           (unsigned) ((b >> 29) & 0x7fffffu));
  // The remaining 29 significand bits R as a float without an integer
  // conversion: R = 64 Ra + Rb, each part exact through the 2^23 bias,
  // rounded once by the multiply-add.
  unsigned R=(unsigned) (b & 0x1fffffffull);
  float ra=__fsub_rn(__uint_as_float(0x4b000000u | (R >> 6)),8388608.0f);
  float rb=__fsub_rn(__uint_as_float(0x4b000000u | (R & 63u)),8388608.0f);
  float lo=fmaf(ra,64.0f,rb);
  lo=__fmul_rn(lo,__uint_as_float((unsigned) (e-52+127) << 23)); // * 2^(e-52)
  lo=__uint_as_float(__float_as_uint(lo) | sign);
  return ffFast(hi,lo);
}

// f 2^sh widened to double exactly by moving its fields (the FP64 pipe only
// for subnormals, infinities, NaNs and results outside the double range).
__device__ __forceinline__ double widen(float f, int sh=0)
{
  unsigned u=__float_as_uint(f);
  unsigned ef=(u >> 23) & 0xffu;
  unsigned long long sign=(unsigned long long) (u & 0x80000000u) << 32;
  if((u & 0x7fffffffu) == 0) return __longlong_as_double((long long) sign);
  const int E=(int) ef+896+sh;
  if(ef == 0 || ef == 255 || E <= 0 || E >= 2047)
    return sh ? scalbn((double) f,sh) : (double) f;
  return __longlong_as_double((long long) (sign |
    ((unsigned long long) E << 52) |
    ((unsigned long long) (u & 0x7fffffu) << 29)));
}

__device__ __forceinline__ double fromFF(ff v, int sh=0)
{
  return widen(v.hi,sh)+widen(v.lo,sh);
}

// The range-guard exponent of input a (io < 8) or output io-8 of the
// float-float mode; 0 for the other modes or without a guard.
template<typename T>
__device__ __forceinline__ int ioShift(const int *sh, int io)
{
  if constexpr(std::is_same<T,ff>::value) return sh ? __ldg(sh+io) : 0;
  else return 0;
}

// Both components, out of line: the fused stages convert at dozens of
// places, and inlined there the conversion was most of their code.
static __device__ __noinline__ cplx<ff> toFF2(double2 d, int sh)
{
  return mk(toFF(d.x,sh),toFF(d.y,sh));
}

static __device__ __noinline__ double2 fromFF2(cplx<ff> v, int sh)
{
  return make_double2(fromFF(v.x,sh),fromFF(v.y,sh));
}

template<typename T>
__device__ __forceinline__ cplx<T> loadIO(const cplx<T> *p, bool f64,
                                          int sh=0)
{
  if constexpr(std::is_same<T,ff>::value)
    if(f64) return toFF2(*(const double2 *) p,sh);
  return *p;
}

template<typename T>
__device__ __forceinline__ T loadIOr(const T *p, bool f64, int sh=0)
{
  if constexpr(std::is_same<T,ff>::value)
    if(f64) return toFF(*(const double *) p,sh);
  return *p;
}

template<typename T>
__device__ __forceinline__ void storeIO(cplx<T> *p, cplx<T> v, bool f64,
                                        int sh=0)
{
  if constexpr(std::is_same<T,ff>::value) {
    if(f64) {
      *(double2 *) p=fromFF2(v,sh);
      return;
    }
  }
  *p=v;
}

template<typename T>
__device__ __forceinline__ void storeIOr(T *p, T v, bool f64, int sh=0)
{
  if constexpr(std::is_same<T,ff>::value) {
    if(f64) {
      *(double *) p=fromFF(v,sh);
      return;
    }
  }
  *p=v;
}

// Convert n elements staged in shared memory as FP64 (by cp.async) to
// float-float in place; each thread converts the elements it copied.
template<typename T>
__device__ __forceinline__ void convertStaged(cplx<T> *y, int i, int sh=0)
{
  if constexpr(std::is_same<T,ff>::value) {
    double2 d=*(double2 *) (y+i);
    y[i]=mk(toFF(d.x,sh),toFF(d.y,sh));
  }
}

// Exponent ((s-c) mod N)*r mod N of a residue twiddle (r < N; 32-bit
// arithmetic while the product fits).
__device__ __forceinline__ int twExp(int s, int c, int r, int N)
{
  int d=s-c;
  if(d < 0) d += N;
  if(N <= 65536) return (int) (((unsigned) d*(unsigned) r) % (unsigned) N);
  return (int) (((unsigned long long) d*(unsigned long long) r) %
                (unsigned long long) N);
}

// The exponent step m*r mod N between the terms s and s+m of a fold.
__device__ __forceinline__ int twStep(int m, int r, int N)
{
  return (int) (((unsigned long long) m*(unsigned long long) r) %
                (unsigned long long) N);
}

__device__ __forceinline__ int posmod(int a, int m)
{
  int r=a % m;
  return r < 0 ? r+m : r;
}

// ---------------------------------------------------------------------------
// Row kernel, complex data (fftPad / fftPadCentered along the contiguous
// axis): fold + pre-twiddle (forwardInner: Zetaqp/Zetaqm), m-point FFT, fused
// multiplier, inverse FFT, post-twiddle and accumulation over residues
// (backwardInner), normalisation (Convolution::normalize).
// Load of data another CTA of the same launch may have written: CG bypasses
// the (non-coherent) L1 with ld.global.cg.
template<bool CG>
__device__ __forceinline__ cplx<double> ldx(const cplx<double> *p)
{
  if(CG) {
    double2 v=__ldcg((const double2 *) p);
    return mk(v.x,v.y);
  }
  return *p;
}

template<bool CG>
__device__ __forceinline__ cplx<float> ldx(const cplx<float> *p)
{
  if(CG) {
    float2 v=__ldcg((const float2 *) p);
    return mk(v.x,v.y);
  }
  return *p;
}

template<bool CG>
__device__ __forceinline__ cplx<ff> ldx(const cplx<ff> *p)
{
  if(CG) {
    float4 v=__ldcg((const float4 *) p);
    return mk(ff(v.x,v.y),ff(v.z,v.w));
  }
  return *p;
}

// Asynchronous global->shared copy of one complex element (cp.async; the
// 16-byte form bypasses L1).  cpAsyncWait() waits for all of the thread's
// copies; a __syncthreads() must follow before other threads read them.
__device__ __forceinline__ void cpAsync(cplx<double> *dst,
                                        const cplx<double> *src)
{
  unsigned s=(unsigned) __cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n"
               :: "r"(s), "l"(src) : "memory");
}

__device__ __forceinline__ void cpAsync(cplx<ff> *dst, const cplx<ff> *src)
{
  unsigned s=(unsigned) __cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n"
               :: "r"(s), "l"(src) : "memory");
}

__device__ __forceinline__ void cpAsync(cplx<float> *dst,
                                        const cplx<float> *src)
{
  unsigned s=(unsigned) __cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n"
               :: "r"(s), "l"(src) : "memory");
}

__device__ __forceinline__ void cpAsyncWait()
{
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// Global loads a thread issues back to back in the row kernels' load loops
// (more bytes in flight per thread than one dependent load per iteration).
#define FGB_LOADS 4

// One group of P.rpc rows of the complex row convolution (all residues),
// using the block's shared memory.  The A x rpc input rows are transformed
// together as interleaved columns col = a*rpc + rho, so the B x rpc output
// columns are a contiguous prefix for the inverse transforms.  Every thread
// of the block calls it.
template<typename T, bool CG, class Mul, bool R16=false>
__device__ __forceinline__ void rowConvRow(const RowPlan<T>& P,
                                           long long group,
                                           unsigned char *smemRaw,
                                           const Mul& mul)
{
  const int A=P.A, B=P.B, L=P.L, m=P.m, N=P.N, c=P.cshift, R=P.rpc;
  const int ld=A*R, lb=B*R;
  cplx<T> *fin=(cplx<T> *) smemRaw;
  cplx<T> *acc=fin+ld*L;
  cplx<T> *x=acc+lb*L;
  cplx<T> *y=x+padded(m*ld);         // ping-pong buffer of the FP64 form
  const int tid=threadIdx.x, nthr=blockDim.x;
  const typename TwT<T>::type *tw=P.twN;
  const UDiv dL(L), dLd(ld);
  const UDiv dR(R);
  const long long row0=group*R;

  // The loads of FGB_LOADS iterations are issued before any is used.
  for(int i0=tid; i0 < ld*L; i0 += FGB_LOADS*nthr) {
    cplx<T> v[FGB_LOADS];
#pragma unroll
    for(int u=0; u < FGB_LOADS; ++u) {
      const int i=i0+u*nthr;
      v[u]=mk((T) 0,(T) 0);
      if(i >= ld*L) continue;
      int col=dL(i), s=i-col*L;
      int a=dR(col);
      long long row=row0+col-a*R;
      if(row < P.nrows) {
        long long off=row*P.rowStride+s;
        if(P.realIO)
          v[u]=mk(loadIOr((const T *) P.in[a]+off,P.io64 & 1,
                          ioShift<T>(P.ioShift,a)),(T) 0);
        else if(P.io64 & 1)
          v[u]=loadIO(P.in[a]+off,true,ioShift<T>(P.ioShift,a));
        else v[u]=ldx<CG>(P.in[a]+off);
      }
    }
#pragma unroll
    for(int u=0; u < FGB_LOADS; ++u)
      if(i0+u*nthr < ld*L) fin[i0+u*nthr]=v[u];
  }
  for(int i=tid; i < lb*L; i += nthr) acc[i]=mk((T) 0,(T) 0);
  __syncthreads();

  for(int r=0; r < P.q; ++r) {
    // Fold the data into one length-m block with the residue twiddles.
    for(int i=tid; i < m*ld; i += nthr) {
      int t=dLd(i), col=i-t*ld;
      int s0=posmod(t+c,m);
      cplx<T> sum=mk((T) 0,(T) 0);
      // The twiddle exponent advances by m r mod N from term to term.
      int e=r != 0 ? twExp(s0,c,r,N) : 0;
      const int de=r != 0 ? twStep(m,r,N) : 0;
      for(int s=s0; s < L; s += m) {
        cplx<T> v=fin[col*L+s];
        if(r != 0) {
          v=twmul<1>(v,tw[e]);
          e += de;
          if(e >= N) e -= N;
        }
        sum=accum(sum,v);
      }
      x[sp(i)]=sum;
    }
    __syncthreads();
    const cplx<T> *Z;
    if constexpr(inplaceFFT<T>()) {
      fftDIF<T,1,R16>(x,P.fp,ld,ld,tid,nthr);
      for(int i=tid; i < m*R; i += nthr) {
        int j=dR(i), rho=i-j*R;
        mulRowSlot<Mul,true>(mul,P,x,j*ld+rho,R,row0+rho,j,r);
      }
      __syncthreads();
      fftDIT<T,-1,R16>(x,P.fp,lb,ld,tid,nthr);
      Z=x;
    } else {
      cplx<T> *X=fftSmem<T,1>(x,y,P.fp,ld,ld,tid,nthr);
      cplx<T> *Y=X == x ? y : x;
      for(int i=tid; i < m*R; i += nthr) {
        int j=dR(i), rho=i-j*R;
        mulRowSlot<Mul,false>(mul,P,X,j*ld+rho,R,row0+rho,j,r);
      }
      __syncthreads();
      Z=fftSmem<T,-1>(X,Y,P.fp,lb,ld,tid,nthr);
    }
    for(int i=tid; i < lb*L; i += nthr) {
      int col=dL(i), s=i-col*L;
      int t=posmod(s-c,m);
      cplx<T> v=Z[sp(t*ld+col)];
      if(r != 0) v=twmul<-1>(v,tw[twExp(s,c,r,N)]);
      acc[i]=accum(acc[i],v);
    }
    __syncthreads();
  }
  for(int i=tid; i < lb*L; i += nthr) {
    int col=dL(i), s=i-col*L;
    int b=dR(col);
    long long row=row0+col-b*R;
    if(row >= P.nrows) continue;
    long long off=row*P.rowStride+s;
    const int sh=ioShift<T>(P.ioShift,8+b);
    if(P.realIO)
      storeIOr((T *) P.out[b]+off,acc[i].x*P.scale,P.io64 & 2,sh);
    else storeIO(P.out[b]+off,acc[i]*P.scale,P.io64 & 2,sh);
  }
  __syncthreads();
}

template<typename T, class Mul>
__global__ void __launch_bounds__(256)
rowConvKernel(const RowPlan<T> P, const Mul mul)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  const long long groups=(P.nrows+P.rpc-1)/P.rpc;
  for(long long g=blockIdx.x; g < groups; g += gridDim.x)
    rowConvRow<T,false,Mul>(P,g,smemRaw,mul);
}

// The same for FP32 plans with a radix-16 stage: the radix-16 code needs
// more registers, so only those plans launch it, capped at 85 registers a
// thread (three CTAs of 256 threads per SM).
template<typename T, class Mul>
__global__ void __launch_bounds__(256,3)
rowConvKernel16(const RowPlan<T> P, const Mul mul)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  const long long groups=(P.nrows+P.rpc-1)/P.rpc;
  for(long long g=blockIdx.x; g < groups; g += gridDim.x)
    rowConvRow<T,false,Mul,true>(P,g,smemRaw,mul);
}

// ---------------------------------------------------------------------------
// Fused rows (fft_fused.cuh): one residue, one fold.  A CTA's threads form
// teams of P.nteam-th parts; a team convolves whole rows on its own (its
// own A columns of shared memory, its own barriers), so the rows of a CTA
// do not wait for one another.

// Values a middle stage may hold in registers: R of each of the A inputs.
template<typename T, int A> __device__ constexpr bool fusedMiddle(int R)
{
  return R*A <= 20;
}

// The multiplier alone on every slot of a row (parts exchanged in the
// results).
template<typename T, class Mul, class Plan>
__device__ __forceinline__ void fusedMulSlots(const Plan& P, const Mul& mul,
                                              cplx<T> *x, int cs,
                                              long long row, int t, int nt)
{
  constexpr int KA=MulArity<Mul>::A, KB=MulArity<Mul>::B;
#pragma unroll 1
  for(int i=t; i < P.fz.n; i += nt) {
    cplx<T> *xi=x+spl(i,P.fz.lg);
    if constexpr(KA > 0) {
      cplx<T> v[KA];
#pragma unroll
      for(int c=0; c < KA; ++c) v[c]=nrm(xi[c*cs]);
      mulFusedSlot(mul,P,v,row,i);
#pragma unroll
      for(int c=0; c < KB; ++c) xi[c*cs]=swapXY(v[c]);
    } else {
      cplx<T> v[FGB_MAXA];
      for(int a=0; a < P.A; ++a) v[a]=nrm(xi[a*cs]);
      applyMult(P.mult,v,P.A);
      for(int b=0; b < P.B; ++b) xi[b*cs]=swapXY(v[b]);
    }
  }
}

// The last forward stage, the multiplier and the first inverse stage of one
// row: every butterfly of radix R holds R neighbouring slots of all A
// inputs, multiplies them in registers and transforms the B products back
// (parts exchanged).
template<typename T, int R, class Mul, class Plan>
__device__ __forceinline__ void fusedMulStage(const Plan& P, const Mul& mul,
                                              cplx<T> *x, int cs,
                                              long long row, int t, int nt)
{
  constexpr int A=MulArity<Mul>::A, B=MulArity<Mul>::B;
  typedef typename TwT<T>::type Tw;
  const FusedFFT& p=P.fz;
  const int nblk=p.n/R;
  const Tw *tw=(const Tw *) p.twb+(nblk-p.radix[0]);
#pragma unroll 1
  for(int b=t; b < nblk; b += nt) {
    cplx<T> *xq=x+spl(b*R,p.lg);
    cplx<T> a[A][R];
#pragma unroll
    for(int c=0; c < A; ++c)
#pragma unroll
      for(int r=0; r < R; ++r) a[c][r]=nrm(xq[c*cs+r]);
    inTwiddleDFT<T,R,A>(a,tw,b,nblk);
#pragma unroll
    for(int r=0; r < R; ++r) {
      cplx<T> v[A];
#pragma unroll
      for(int c=0; c < A; ++c) v[c]=nrm(a[c][r]);
      mulFusedSlot(mul,P,v,row,b*R+r);
#pragma unroll
      for(int c=0; c < B; ++c) a[c][r]=nrm(swapXY(v[c]));
    }
#pragma unroll
    for(int c=0; c < B; ++c) {
      Codelet<R,1,T>::run(a[c]);
#pragma unroll
      for(int r=0; r < R; ++r) xq[c*cs+r]=a[c][r];
    }
  }
}

// Everything between the first forward and the last inverse stage of a row
// whose A columns lie cs apart at x; ends synchronised.
template<typename T, bool WIDE, class Mul, class Plan>
__device__ __forceinline__ void fusedRowInner(const Plan& P, const Mul& mul,
                                              cplx<T> *x, int cs,
                                              long long row, int team, int t,
                                              int nt)
{
  constexpr int KA=MulArity<Mul>::A;
  const FusedFFT& p=P.fz;
  const int A=P.A, B=P.B;
  if constexpr(std::is_same<T,ff>::value) {
    runStages<T>(x,cs,A,B,p,0,1,team,t,nt,[&] {
        fusedMulSlots(P,mul,x,cs,row,t,nt);
      });
  } else {
    const int nblk=runFusedMiddle<T,WIDE>(x,cs,A,p,0,false,team,t,nt);
    teamSync(team,nt);
    bool fused=KA > 0;
    if constexpr(KA >= 4) {
      // A thread of the fused step takes A + B butterflies one after the
      // other; on rows with fewer butterflies than threads the three steps
      // spread them (FP64 Jacobian rows of 180 points).
      const int per=(nblk+nt-1)/nt;
      fused=per*(A+B) <= (A*nblk+nt-1)/nt+(B*nblk+nt-1)/nt+2;
    }
    if(fused) {
      if constexpr(KA > 0) switch(p.radix[p.nst-1]) {
        case 1: fusedMulStage<T,1>(P,mul,x,cs,row,t,nt); break;
        case 2: fusedMulStage<T,2>(P,mul,x,cs,row,t,nt); break;
        case 3: fusedMulStage<T,3>(P,mul,x,cs,row,t,nt); break;
        case 4: fusedMulStage<T,4>(P,mul,x,cs,row,t,nt); break;
        case 5:
          if constexpr(fusedMiddle<T,KA>(5))
            fusedMulStage<T,5>(P,mul,x,cs,row,t,nt);
          break;
        case 7:
          if constexpr(fusedMiddle<T,KA>(7))
            fusedMulStage<T,7>(P,mul,x,cs,row,t,nt);
          break;
        case 8:
          if constexpr(fusedMiddle<T,KA>(8))
            fusedMulStage<T,8>(P,mul,x,cs,row,t,nt);
          break;
        case 16:
          if constexpr(WIDE && fusedMiddle<T,KA>(16))
            fusedMulStage<T,16>(P,mul,x,cs,row,t,nt);
          break;
        default: break;
      }
    } else if constexpr(KA == 0 || KA >= 4) {
      // Arity known at run time (or as above): the three steps one after the
      // other.
      typedef typename TwT<T>::type Tw;
      const Tw *twb=(const Tw *) p.twb+(nblk-p.radix[0]);
      const Tw *twj=(const Tw *) p.twj;
      const int R=p.radix[p.nst-1];
      FGB_FUSED_SWITCH(R,(fusedStage<T,R_,WIDE>(x,cs,A,p,0,1,twb,nblk,false,t,
                                             nt)))
      teamSync(team,nt);
      fusedMulSlots(P,mul,x,cs,row,t,nt);
      teamSync(team,nt);
      FGB_FUSED_SWITCH(R,(fusedStage<T,R_,WIDE>(x,cs,B,p,0,1,twj,1,true,t,nt)))
    }
    runFusedMiddle<T,WIDE>(x,cs,B,p,0,true,team,t,nt);
    teamSync(team,nt);
  }
}

// One row of complex (or, realIO, real) data by a team.
template<typename T, bool CG, bool WIDE, class Mul>
__device__ __forceinline__ void fusedRow(const RowPlan<T>& P, const Mul& mul,
                                         cplx<T> *x, int cs, long long row,
                                         int team, int t, int nt)
{
  const int m=P.m, c=P.cshift;
  const int top=row < P.nrows ? P.L : 0;   // entries of a row that exists
  const long long off0=row*P.rowStride;
  const auto load=[&](int a, int) {
    const cplx<T> *f=P.in[a]+(P.realIO ? 0 : off0);
    const T *fr=(const T *) P.in[a]+off0;
    const int sh=ioShift<T>(P.ioShift,a);
    return [=,&P](int j) {
      int s=j+c;
      if(s >= m) s -= m;
      cplx<T> v=mk((T) 0,(T) 0);
      if(s < top) {
        if(P.realIO) v.x=loadIOr(fr+s,P.io64 & 1,sh);
        else if(P.io64 & 1) v=loadIO(f+s,true,sh);
        else v=ldx<CG>(f+s);
      }
      return v;
    };
  };
  const auto store=[&](int b, int) {
    cplx<T> *f=P.out[b]+(P.realIO ? 0 : off0);
    T *fr=(T *) P.out[b]+off0;
    const int sh=ioShift<T>(P.ioShift,8+b);
    return [=,&P](int j, cplx<T> v) {
      int s=j+c;
      if(s >= m) s -= m;
      if(s >= top) return;
      if(P.realIO) storeIOr(fr+s,v.x*P.scale,P.io64 & 2,sh);
      else storeIO(f+s,v*P.scale,P.io64 & 2,sh);
    };
  };
  // The staged form where the fused first stage would leave threads of the
  // team without a butterfly, and for FP64 rows of up to 128 points (512 rows
  // of 80 points 26 us fused, 19 staged; 6000 of 128 104 / 100; 512 of 160 25.9
  // / 26.1, 1536 of 192 60 / 65).  FP32 rows are faster fused throughout (441
  // of 80 points 9 us, 12 staged; 1536 of 360 13 / 19), but for the batched
  // launch, whose short problems have a whole CTA for one row.
  bool staged=P.A*(m/P.fz.radix[0]) < nt;
  if constexpr(std::is_same<T,double>::value) staged=staged || m <= 128;
  if constexpr(std::is_same<T,float>::value && !CG) staged=false;
  if(staged) {
    const ColumnMap cols(m);             // the staged form (runStages)
#pragma unroll 2
    for(int i=t; i < P.A*m; i += nt) {
      const int a=cols(i), j=i-a*m;
      x[a*cs+spl(j,P.fz.lg)]=load(a,0)(j);
    }
    runStages<T,WIDE>(x,cs,P.A,P.B,P.fz,0,0,team,t,nt,[&] {
        fusedMulSlots(P,mul,x,cs,row,t,nt);
      });
    for(int i=t; i < P.B*m; i += nt) {
      const int b=cols(i), j=i-b*m;
      store(b,0)(j,swapXY(x[b*cs+spl(j,P.fz.lg)]));
    }
  } else {
    runFusedFirst<T,WIDE>(x,cs,P.A,P.fz,0,t,nt,load);
    fusedRowInner<T,WIDE>(P,mul,x,cs,row,team,t,nt);
    runFusedLast<T,WIDE>(x,cs,P.B,P.fz,0,t,nt,store);
  }
  teamSync(team,nt);
}

template<typename T, class Mul, bool WIDE>
__device__ __forceinline__ void fusedRows(const RowPlan<T>& P, const Mul& mul,
                                          unsigned char *smemRaw)
{
  const int nt=blockDim.x/P.nteam;
  const int team=threadIdx.x/nt, t=threadIdx.x-team*nt;
  const int cs=fusedSpan(P.fz.n,P.fz.lg);
  cplx<T> *x=(cplx<T> *) smemRaw+team*P.A*cs;
  const long long groups=(P.nrows+P.rpc-1)/P.rpc;
  for(long long g=blockIdx.x; g < groups; g += gridDim.x)
    for(int rho=team; rho < P.rpc; rho += P.nteam)
      fusedRow<T,false,WIDE>(P,mul,x,cs,g*P.rpc+rho,team,t,nt);
}

template<typename T, class Mul>
__global__ void __launch_bounds__(256,fusedBlocks<T>())
rowFusedKernel(const RowPlan<T> P, const Mul mul)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  fusedRows<T,Mul,false>(P,mul,smemRaw);
}

// FP32 plans with a radix-16 stage.
template<typename T, class Mul>
__global__ void __launch_bounds__(256,fusedBlocks<T>())
rowFusedKernel16(const RowPlan<T> P, const Mul mul)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  fusedRows<T,Mul,true>(P,mul,smemRaw);
}

// ---------------------------------------------------------------------------
// Split rows: with few rows (RowPlan::split CTAs per row still fit the SMs) a
// cluster of P.split CTAs convolves each row, CTA r the residue r of the
// padded transform: it folds the data into a block of N/split points with
// the residue twiddles, transforms, multiplies and transforms back on its
// own; then every CTA adds a share of the outputs over the blocks of the
// cluster, read through distributed shared memory, with their
// post-twiddles.  A row alone is bound by the FP64 pipe and the latency of
// its one SM: one pair of 1024 points (2048 padded) took 66 us in FP64, 29
// split eight ways (rowSplit in engine.cu).
template<typename T, class Mul>
__global__ void __launch_bounds__(256,2)
rowSplitKernel(const RowPlan<T> P, const Mul mul)
{
  namespace cg=cooperative_groups;
  extern __shared__ __align__(16) unsigned char smemRaw[];
  cg::cluster_group cluster=cg::this_cluster();
  const int Q=P.split, r=(int) cluster.block_rank();
  const long long row=blockIdx.x/Q;
  const int L=P.L, c=P.cshift, N=P.N, m=P.fz.n;
  const int t=threadIdx.x, nt=blockDim.x;
  const int cs=fusedSpan(m,P.fz.lg);
  cplx<T> *x=(cplx<T> *) smemRaw;
  const typename TwT<T>::type *tw=P.twN;
  const long long off0=row*P.rowStride;
  const ColumnMap cols(m);
  const int step=twStep(m,r,N);
#pragma unroll 1
  for(int i=t; i < P.A*m; i += nt) {
    const int a=cols(i), j=i-a*m;
    const int sh=ioShift<T>(P.ioShift,a);
    cplx<T> sum=mk((T) 0,(T) 0);
    int s=posmod(j+c,m);
    int e=twExp(s,c,r,N);
#pragma unroll 4
    for(; s < L; s += m) {
      cplx<T> v=mk((T) 0,(T) 0);
      if(P.realIO)
        v.x=loadIOr((const T *) P.in[a]+off0+s,P.io64 & 1,sh);
      else v=loadIO(P.in[a]+off0+s,P.io64 & 1,sh);
      sum=accum(sum,twmul<1>(v,ldtw(tw+e)));
      e += step;
      if(e >= N) e -= N;
    }
    x[a*cs+spl(j,P.fz.lg)]=sum;
  }
  runStages<T>(x,cs,P.A,P.B,P.fz,0,0,0,t,nt,[&] {
      fusedMulSlots(P,mul,x,cs,row,t,nt);
    });
  cluster.sync();
  const int share=(L+Q-1)/Q, s0=r*share, n=max(0,min(L-s0,share));
#pragma unroll 1
  for(int i=t; i < P.B*n; i += nt) {
    const int b=i/n, s=s0+i-b*n;
    const int at=b*cs+spl(posmod(s-c,m),P.fz.lg);
    const int de=twExp(s,c,1,N);
    cplx<T> sum=mk((T) 0,(T) 0);
    int e=0;
#pragma unroll 4
    for(int k=0; k < Q; ++k) {
      const cplx<T> v=swapXY(cluster.map_shared_rank(x,k)[at]);
      sum=accum(sum,twmul<-1>(v,ldtw(tw+e)));
      e += de;
      if(e >= N) e -= N;
    }
    const int sh=ioShift<T>(P.ioShift,8+b);
    if(P.realIO)
      storeIOr((T *) P.out[b]+off0+s,sum.x*P.scale,P.io64 & 2,sh);
    else storeIO(P.out[b]+off0+s,sum*P.scale,P.io64 & 2,sh);
  }
  cluster.sync();                 // until the others have read this block
}

template<typename T, class Mul>
cudaError_t launchRowSplit(const RowPlan<T>& P, const Mul& mul, int threads,
                           size_t smem, cudaStream_t s)
{
  cudaError_t e=cudaSuccess;
  if(smem > 48*1024)
    e=cudaFuncSetAttribute(rowSplitKernel<T,Mul>,
                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int) smem);
  if(e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg={};
  cfg.gridDim=dim3((unsigned) (P.nrows*P.split));
  cfg.blockDim=dim3(threads);
  cfg.dynamicSmemBytes=smem;
  cfg.stream=s;
  cudaLaunchAttribute at[1];
  at[0].id=cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x=P.split;
  at[0].val.clusterDim.y=at[0].val.clusterDim.z=1;
  cfg.attrs=at;
  cfg.numAttrs=1;
  return cudaLaunchKernelEx(&cfg,rowSplitKernel<T,Mul>,P,mul);
}

// ---------------------------------------------------------------------------
// Row kernel, Hermitian data (fftPadHermitian along the contiguous axis,
// explicit padding to an even real length N): the H stored modes are packed
// into a length-N/2 complex sequence whose sign +1 FFT yields the N real
// physical values as (u[2t], u[2t+1]) pairs; the multiplier acts on those
// doubles; the sign -1 FFT of the packed product is unpacked into the H
// output modes (real-to-complex).
//
// The packing pairs k with Nh-k, and butterfly j of the first stage (inputs
// j + r m) holds exactly the partners of butterfly m-j, so one thread packs
// and transforms both; the unpacking does the same behind the last stage.

// Y[k] = S + i W_N^k D with S = Z[k] + conj Z[Nh-k], D = Z[k] -
// conj Z[Nh-k], and its partner Y[Nh-k] = conj(S) + i conj(W_N^k D) (since
// W_N^{Nh} = -1): one twiddle multiply for both.
template<typename T>
__device__ __forceinline__ void hermPack(cplx<T> zk, cplx<T> zc,
                                         typename TwT<T>::type w,
                                         cplx<T>& Y, cplx<T>& Yc)
{
  const cplx<T> b=conjg(zc);
  const cplx<T> S=zk+b;
  if constexpr(std::is_same<T,double>::value) {
    // FP64: S + (i D) W as four DFMAs, the partner as conj(2S - Y).
    const cplx<T> D=zk-b;
    Y=fmaTw<1>(S,mk(-D.y,D.x),w);
    Yc=mk(fma((T) 2,S.x,-Y.x),fma((T) -2,S.y,Y.y));
  } else {
    const cplx<T> Pw=twmul<1>(zk-b,w);
    Y=mk(S.x-Pw.y,S.y+Pw.x);
    Yc=mk(S.x+Pw.y,Pw.x-S.y);
  }
}

// V[k] = hs (s + Q) with s = Z[k] + conj Z[Nh-k], Q = W_N^{-k} (-i)(Z[k] -
// conj Z[Nh-k]), and V[Nh-k] = hs conj(s - Q); zm is Z[Nh-k] (Z[0] for
// k = 0).
template<typename T>
__device__ __forceinline__ void hermUnpack(cplx<T> zk, cplx<T> zm, T hs,
                                           typename TwT<T>::type w,
                                           cplx<T>& V, cplx<T>& Vc)
{
  const cplx<T> zb=conjg(zm);
  if constexpr(std::is_same<T,double>::value) {
    // FP64: hs sum, hs dd = 2 hs zk - hs sum, V = hs sum + hs Q as four
    // DFMAs, the partner as conj(2 hs sum - V).
    const cplx<T> hsum=(zk+zb)*hs;
    const T h2=hs+hs;
    const cplx<T> hdd=mk(fma(h2,zk.x,-hsum.x),fma(h2,zk.y,-hsum.y));
    V=fmaTw<-1>(hsum,mk(hdd.y,-hdd.x),w);
    Vc=mk(fma((T) 2,hsum.x,-V.x),fma((T) -2,hsum.y,V.y));
  } else {
    const cplx<T> sum=zk+zb, dd=zk-zb;
    const cplx<T> Q=twmul<-1>(mk(dd.y,-dd.x),w);
    V=(sum+Q)*hs;
    Vc=conjg(sum-Q)*hs;
  }
}

// First stage of a row's inputs (cs apart at x0): butterflies j and m-j, or
// 0 and m/2 (each its own partner; only 0 when m is odd), so ceil(m/2)
// threads' worth an input.
template<typename T, int R>
__device__ __forceinline__ void hermFirst(const HermRowPlan<T>& P, cplx<T> *x0,
                                          int cs, long long row, int t, int nt)
{
  const FusedFFT& p=P.fz;
  const int H=row < P.nrows ? P.H : 0, m=P.Nh/R;
  const StageMap map(R,m,p.lg,0);
  const bool even=m % 2 == 0;
  const ColumnMap cols((m+1)/2);
#pragma unroll 1
  for(int i=t; i < P.A*cols.per; i += nt) {
    const int c=cols(i), j=i-c*cols.per;
    cplx<T> *x=x0+c*cs;
    const cplx<T> *z=P.in[c]+row*P.rowStride;
    const int sh=ioShift<T>(P.ioShift,c);
    const int j2=j == 0 ? m/2 : m-j;
    cplx<T> a[R], b[R], u[R], v[R];
#pragma unroll
    for(int r=0; r < R; ++r) {
      const int k=j+r*m, k2=j2+r*m;
      a[r]=k < H ? loadIO(z+k,P.io64 & 1,sh) : mk((T) 0,(T) 0);
      b[r]=k2 < H ? loadIO(z+k2,P.io64 & 1,sh) : mk((T) 0,(T) 0);
    }
    if(j != 0) {
#pragma unroll
      for(int r=0; r < R; ++r)
        hermPack(a[r],b[R-1-r],ldtw(P.twN+j+r*m),u[r],v[R-1-r]);
    } else {
      cplx<T> dummy;
      a[0].y=(T) 0;
      hermPack(a[0],mk((T) 0,(T) 0),ldtw(P.twN),u[0],dummy);
#pragma unroll
      for(int r=1; r <= R/2; ++r)
        hermPack(a[r],a[R-r],ldtw(P.twN+r*m),u[r],
                 2*r == R ? dummy : u[R-r]);
#pragma unroll
      for(int r=0; r < (R+1)/2; ++r)
        hermPack(b[r],b[R-1-r],ldtw(P.twN+m/2+r*m),v[r],
                 2*r == R-1 ? dummy : v[R-1-r]);
    }
#pragma unroll
    for(int r=0; r < R; ++r) {
      u[r]=nrm(u[r]);
      v[r]=nrm(v[r]);
    }
    Codelet<R,1,T>::run(u);
    Codelet<R,1,T>::run(v);
    cplx<T> *xq=x+map.offset(j,0,0), *xr=x+map.offset(j2,0,0);
#pragma unroll
    for(int r=0; r < R; ++r) xq[r*map.step]=u[r];
    if(j != 0 || even) {
#pragma unroll
      for(int r=0; r < R; ++r) xr[r*map.step]=v[r];
    }
  }
}

// Last inverse stage of one output row, unpacked: the same pairs.
template<typename T, int R>
__device__ __forceinline__ void hermLast(const HermRowPlan<T>& P,
                                         const cplx<T> *x0, int cs,
                                         long long row, int t, int nt)
{
  const FusedFFT& p=P.fz;
  const int Nh=P.Nh, H=row < P.nrows ? P.H : 0, m=Nh/R;
  const StageMap map(R,m,p.lg,0);
  const bool even=m % 2 == 0;
  const T hs=(T) 0.5*P.scale;
  const ColumnMap cols((m+1)/2);
#pragma unroll 1
  for(int i=t; i < P.B*cols.per; i += nt) {
    const int c=cols(i), j=i-c*cols.per;
    const cplx<T> *x=x0+c*cs;
    cplx<T> *o=P.out[c]+row*P.rowStride;
    const int sh=ioShift<T>(P.ioShift,8+c);
    auto put=[&](int k, cplx<T> v) {
      if(k < H) storeIO(o+k,v,P.io64 & 2,sh);
    };
    cplx<T> a[1][R], b[1][R];
    const int j2=j == 0 ? m/2 : m-j;
    const cplx<T> *xq=x+map.offset(j,0,0), *xr=x+map.offset(j2,0,0);
#pragma unroll
    for(int r=0; r < R; ++r) {
      a[0][r]=nrm(xq[r*map.step]);
      b[0][r]=nrm(xr[r*map.step]);
    }
    const typename TwT<T>::type *tw=(const typename TwT<T>::type *) p.twj+
      (m-1);
    inTwiddleDFT<T,R,1>(a,tw,j,m);
    inTwiddleDFT<T,R,1>(b,tw,j2,m);
#pragma unroll
    for(int r=0; r < R; ++r) {
      a[0][r]=swapXY(a[0][r]);
      b[0][r]=swapXY(b[0][r]);
    }
    cplx<T> V, Vc;
    if(j != 0) {
#pragma unroll
      for(int r=0; r < R; ++r) {
        const int k=j+r*m;
        if(k >= H && Nh-k >= H) continue;
        hermUnpack(a[0][r],b[0][R-1-r],hs,ldtw(P.twN+k),V,Vc);
        put(k,V);
        put(Nh-k,Vc);
      }
    } else {
#pragma unroll
      for(int r=0; r <= R/2; ++r) {
        hermUnpack(a[0][r],a[0][(R-r)%R],hs,ldtw(P.twN+r*m),V,Vc);
        put(r*m,V);
        if(r > 0 && 2*r < R) put(Nh-r*m,Vc);
      }
      if(even) {
#pragma unroll
        for(int r=0; r < (R+1)/2; ++r) {
          const int k=m/2+r*m;
          hermUnpack(b[0][r],b[0][R-1-r],hs,ldtw(P.twN+k),V,Vc);
          put(k,V);
          if(2*r < R-1) put(Nh-k,Vc);
        }
      }
    }
  }
}

// The staged form (runStages) of a Hermitian row: the packing and unpacking
// one pair at a time.
template<typename T, bool WIDE, class Mul>
__device__ __forceinline__ void hermRowStaged(const HermRowPlan<T>& P,
                                              const Mul& mul, cplx<T> *x,
                                              int cs, long long row, int team,
                                              int t, int nt)
{
  const FusedFFT& p=P.fz;
  const int Nh=P.Nh, H=row < P.nrows ? P.H : 0;
  const ColumnMap cols(Nh/2+1);
#pragma unroll 2
  for(int i=t; i < P.A*cols.per; i += nt) {
    const int c=cols(i), k=i-c*cols.per, kk=Nh-k;
    const cplx<T> *z=P.in[c]+row*P.rowStride;
    const int sh=ioShift<T>(P.ioShift,c);
    cplx<T> a=mk((T) 0,(T) 0), b=a, Y, Yc;
    if(k < H) a=loadIO(z+k,P.io64 & 1,sh);
    if(kk < H) b=loadIO(z+kk,P.io64 & 1,sh);
    if(k == 0) a.y=(T) 0;
    hermPack(a,b,ldtw(P.twN+k),Y,Yc);
    x[c*cs+spl(k,p.lg)]=Y;
    if(k != 0 && 2*k != Nh) x[c*cs+spl(kk,p.lg)]=Yc;
  }
  runStages<T,WIDE>(x,cs,P.A,P.B,p,0,0,team,t,nt,[&] {
      fusedMulSlots(P,mul,x,cs,row,t,nt);
    });
  const T hs=(T) 0.5*P.scale;
#pragma unroll 1
  for(int i=t; i < P.B*cols.per; i += nt) {
    const int c=cols(i), k=i-c*cols.per, kk=k == 0 ? 0 : Nh-k;
    if(k >= H && kk >= H) continue;
    const cplx<T> zk=swapXY(x[c*cs+spl(k,p.lg)]);
    const cplx<T> zm=swapXY(x[c*cs+spl(kk,p.lg)]);
    cplx<T> *o=P.out[c]+row*P.rowStride, V, Vc;
    const int sh=ioShift<T>(P.ioShift,8+c);
    hermUnpack(zk,zm,hs,ldtw(P.twN+k),V,Vc);
    if(k < H) storeIO(o+k,V,P.io64 & 2,sh);
    if(kk > k && kk < H) storeIO(o+kk,Vc,P.io64 & 2,sh);
  }
}

// One slot t of a Hermitian row (real grid points 2t and 2t+1) in shared
// memory: the A values at X[sp(base+a*stride)] in, the B results back.
template<class Mul, typename T>
__device__ __forceinline__ void mulHermSlot(const Mul& mul,
                                            const HermRowPlan<T>& P,
                                            cplx<T> *X, int base, int stride,
                                            long long row, int t)
{
  if constexpr(Mul::positional) {
    constexpr int A=MulArity<Mul>::A, B=MulArity<Mul>::B;
    cplx<T> v[A];
#pragma unroll
    for(int a=0; a < A; ++a) v[a]=nrm(X[sp(base+a*stride)]);
    mul.slotReal(v,outerIndices(P.im,row),2*t);
#pragma unroll
    for(int b=0; b < B; ++b) X[sp(base+b*stride)]=v[b];
  } else mul(X,base,stride,P.A,P.B,P.mult);
}

// FP64 rows through the self-sorting transform (hermPingPong in engine.cu):
// the P.rpc rows of a group as interleaved columns col = a rpc + rho of two
// buffers, all threads on all of them, natural order throughout.  Every read
// of a group precedes its writes, so in = out is safe.
template<typename T, class Mul>
__global__ void __launch_bounds__(256)
hermRowPingPongKernel(const HermRowPlan<T> P, const Mul mul)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  const int H=P.H, Nh=P.Nh, R=P.rpc, ld=P.A*R, lb=P.B*R;
  cplx<T> *x=(cplx<T> *) smemRaw, *y=x+padded(Nh*ld);
  const int tid=threadIdx.x, nthr=blockDim.x;
  const UDiv dH(H), dLd(ld), dR(R);
  const int np=Nh/2+1;                 // k = 0 .. floor(Nh/2)
  const long long groups=(P.nrows+R-1)/R;
  for(long long g=blockIdx.x; g < groups; g += gridDim.x) {
    const long long row0=g*R;
    for(int i0=tid; i0 < np*ld; i0 += FGB_LOADS*nthr) {
      cplx<T> zk[FGB_LOADS], zc[FGB_LOADS];
#pragma unroll
      for(int u=0; u < FGB_LOADS; ++u) {
        const int i=i0+u*nthr, k=dLd(i), col=i-k*ld, a=dR(col), kk=Nh-k;
        const long long row=row0+col-a*R;
        const bool live=i < np*ld && row < P.nrows;
        zk[u]=zc[u]=mk((T) 0,(T) 0);
        if(live && k < H) zk[u]=P.in[a][row*P.rowStride+k];
        if(live && kk < H) zc[u]=P.in[a][row*P.rowStride+kk];
      }
#pragma unroll
      for(int u=0; u < FGB_LOADS; ++u) {
        const int i=i0+u*nthr;
        if(i >= np*ld) break;
        const int k=dLd(i), col=i-k*ld;
        cplx<T> Y, Yc;
        if(k == 0) zk[u].y=(T) 0;
        hermPack(zk[u],zc[u],ldtw(P.twN+k),Y,Yc);
        x[sp(i)]=Y;
        if(k != 0 && 2*k != Nh) x[sp((Nh-k)*ld+col)]=Yc;
      }
    }
    __syncthreads();
    cplx<T> *X=fftSmem<T,1>(x,y,P.fp,ld,ld,tid,nthr);
    cplx<T> *Y=X == x ? y : x;
    for(int i=tid; i < Nh*R; i += nthr) {
      const int t=dR(i), rho=i-t*R;
      mulHermSlot(mul,P,X,t*ld+rho,R,row0+rho,t);
    }
    __syncthreads();
    const cplx<T> *Z=fftSmem<T,-1>(X,Y,P.fp,lb,ld,tid,nthr);
    // When both k and Nh-k are stored modes the lower one writes both.
    const T hs=(T) 0.5*P.scale;
    for(int i=tid; i < lb*H; i += nthr) {
      const int col=dH(i), k=i-col*H, b=dR(col), kk=k == 0 ? 0 : Nh-k;
      const long long row=row0+col-b*R;
      const bool pair=k != 0 && kk < H && kk != k;
      if(row >= P.nrows || (pair && kk < k)) continue;
      cplx<T> V, Vc;
      hermUnpack(Z[sp(k*ld+col)],Z[sp(kk*ld+col)],hs,ldtw(P.twN+k),V,Vc);
      cplx<T> *o=P.out[b]+row*P.rowStride;
      o[k]=V;
      if(pair) o[kk]=Vc;
    }
    __syncthreads();
  }
}

// First radices of fused Hermitian rows (the two butterflies of a pair are
// in registers together).
#define FGB_HERM_SWITCH(R,CALL) \
  switch(R) { \
    case 1: {constexpr int R_=1; CALL;} break; \
    case 2: {constexpr int R_=2; CALL;} break; \
    case 3: {constexpr int R_=3; CALL;} break; \
    case 4: {constexpr int R_=4; CALL;} break; \
    case 5: {constexpr int R_=5; CALL;} break; \
    case 6: {constexpr int R_=6; CALL;} break; \
    case 7: {constexpr int R_=7; CALL;} break; \
    case 8: {constexpr int R_=8; CALL;} break; \
    default: break; \
  }

template<typename T, class Mul, bool WIDE, bool STAGED>
__device__ __forceinline__ void hermRows(const HermRowPlan<T>& P,
                                         const Mul& mul,
                                         unsigned char *smemRaw)
{
  const int nt=blockDim.x/P.nteam;
  const int team=threadIdx.x/nt, t=threadIdx.x-team*nt;
  const int cs=fusedSpan(P.Nh,P.fz.lg);
  cplx<T> *x=(cplx<T> *) smemRaw+team*P.A*cs;
  const long long groups=(P.nrows+P.rpc-1)/P.rpc;
  for(long long g=blockIdx.x; g < groups; g += gridDim.x)
    for(int rho=team; rho < P.rpc; rho += P.nteam) {
      const long long row=g*P.rpc+rho;
      if constexpr(STAGED) hermRowStaged<T,WIDE>(P,mul,x,cs,row,team,t,nt);
      else {
        const int R0=P.fz.radix[0];
        FGB_HERM_SWITCH(R0,(hermFirst<T,R_>(P,x,cs,row,t,nt)))
        fusedRowInner<T,WIDE>(P,mul,x,cs,row,team,t,nt);
        FGB_HERM_SWITCH(R0,(hermLast<T,R_>(P,x,cs,row,t,nt)))
      }
      teamSync(team,nt);
    }
}

template<typename T, class Mul>
__global__ void __launch_bounds__(256,fusedBlocks<T>())
hermRowStagedKernel(const HermRowPlan<T> P, const Mul mul)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  hermRows<T,Mul,std::is_same<T,float>::value,true>(P,mul,smemRaw);
}

// FP32, fused; WIDE: plans with a radix-16 stage.
template<typename T, class Mul, bool WIDE>
__global__ void __launch_bounds__(256,fusedBlocks<T>())
hermRowFusedKernel(const HermRowPlan<T> P, const Mul mul)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  hermRows<T,Mul,WIDE,false>(P,mul,smemRaw);
}

// ---------------------------------------------------------------------------
// Launchers of the row kernels for any multiplier type.

template<typename K>
inline cudaError_t setRowSmem(K kernel, size_t bytes)
{
  if(bytes > 48*1024)
    return cudaFuncSetAttribute(kernel,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int) bytes);
  return cudaSuccess;
}

template<typename T, class Mul>
cudaError_t launchRowWith(const RowPlan<T>& P, const Mul& mul, int threads,
                          long long grid, cudaStream_t s)
{
  if constexpr(!Mul::positional)
    if(P.split > 1)
      return launchRowSplit(P,mul,threads,
                            fusedRowSmem<T>(P.fz.n,P.fz.lg,P.A,1),s);
  const size_t sm=P.direct ? fusedRowSmem<T>(P.fz.n,P.fz.lg,P.A,P.nteam) :
    rowSmem<T>(P.L,P.m,P.A,P.B,P.rpc);
  const long long groups=(P.nrows+P.rpc-1)/P.rpc;
  grid=std::min(std::min(grid,groups),(long long) INT_MAX);
  if(grid < 1) return cudaSuccess;
  auto go=[&](auto kernel) {
    cudaError_t e=setRowSmem(kernel,sm);
    if(e != cudaSuccess) return e;
    kernel<<<(unsigned) grid,threads,sm,s>>>(P,mul);
    return cudaGetLastError();
  };
  if constexpr(std::is_same<T,float>::value) {
    if(P.direct && wideFused(P.fz)) return go(rowFusedKernel16<T,Mul>);
    if(!P.direct && hasWideRadix(P.fp)) return go(rowConvKernel16<T,Mul>);
  }
  if(P.direct) return go(rowFusedKernel<T,Mul>);
  return go(rowConvKernel<T,Mul>);
}

template<typename T, class Mul>
cudaError_t launchHermRowWith(const HermRowPlan<T>& P, const Mul& mul,
                              int threads, long long grid, cudaStream_t s)
{
  const size_t sm=P.pingpong ? hermRowSmem<T>(P.Nh,P.A,P.rpc) :
    fusedRowSmem<T>(P.fz.n,P.fz.lg,P.A,P.nteam);
  const long long groups=(P.nrows+P.rpc-1)/P.rpc;
  grid=std::min(std::min(grid,groups),(long long) INT_MAX);
  if(grid < 1) return cudaSuccess;
  auto go=[&](auto kernel) {
    cudaError_t e=setRowSmem(kernel,sm);
    if(e != cudaSuccess) return e;
    kernel<<<(unsigned) grid,threads,sm,s>>>(P,mul);
    return cudaGetLastError();
  };
  if constexpr(std::is_same<T,double>::value)
    if(P.pingpong) return go(hermRowPingPongKernel<T,Mul>);
  if constexpr(std::is_same<T,float>::value)
    if(!P.staged)
      return wideFused(P.fz) ? go(hermRowFusedKernel<T,Mul,true>) :
        go(hermRowFusedKernel<T,Mul,false>);
  return go(hermRowStagedKernel<T,Mul>);
}

} // namespace fgb
