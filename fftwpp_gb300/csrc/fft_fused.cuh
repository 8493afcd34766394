// fft_fused.cuh -- shared-memory transforms whose first and last stages run
// on values in registers, for the convolution kernels whose padded data are
// one fold long (explicit padding, or a residue block at least as long as
// the data).
//
// A kernel that loads into shared memory, transforms, multiplies, transforms
// back and stores passes every value through shared memory once for each
// of those steps.  Here the first forward stage takes its inputs from global
// memory, the last forward stage, the multiplier and the first inverse
// stage share one set of registers, and the last inverse stage hands its
// outputs to global memory: a three-stage transform and its inverse cross
// shared memory four times instead of eight, with four barriers instead of
// eight.
//
// Decimation.  With radices R_0 .. R_{k-1} and span m_s = n/(R_0 .. R_s), a
// forward stage s combines elements b R_s m_s + j + r m_s (r < R_s) of block
// b, after multiplying input r by W_{R_0..R_s}^{r rev(b)}, where rev(b) is
// the natural index of block b's digits.  (The common factor W^{j rev(b)} of
// the usual decimation in frequency is left to the later stages, which
// absorb it into theirs.)  Natural order in, mixed-radix digit-reversed
// order out, as fftDIF.  The twiddles depend on the block alone: the early
// stages have a handful, which a whole warp shares, and all columns of a
// tile and all inputs of a convolution use the same ones.  The inverse takes
// its stages in the opposite order with the twiddles W_{R m}^{-r j} on the
// inputs (decimation in time), so that both directions multiply before the
// butterfly and FP64 fuses the products into its additions.
//
// The inverse runs on values with their real and imaginary parts exchanged:
// exchanging them turns a conj(w) into a w and the sign -1 transform into
// the sign +1 one, so one piece of code serves the middle stages of both
// directions.  Code size matters: with separate inverse stages the
// float-float row kernel stalled on instruction fetch more than on anything
// else.
#pragma once

#include "fft_smem.cuh"

#include <vector>

namespace fgb {

#define FGB_FUSED_STAGES 12

// A transform of length n.  Its element j of column c lies at
// spl(j, lg) ld + c of shared memory for ld interleaved columns.
struct FusedFFT {
  int n, nst;
  int lg;                  // one pad element every 2^lg: the product of the
                           // last radices (fusedPadding), so that every
                           // stage's inputs lie at a fixed step
  int half;                // only the first half of the input is nonzero and
                           // only the first half of the output is wanted
                           // (radix[0] is even)
  unsigned char radix[FGB_FUSED_STAGES];
  const void *twb;         // block twiddles: stage s >= 1 with nblk blocks
                           // at nblk - R_0, entry (r-1) nblk + b
  const void *twj;         // inverse twiddles W_{R m}^{r j}: stage s at m - 1,
                           // entry (r-1) m + j
  const int4 *pairs;       // last-stage blocks paired for real data: (block,
                           // partner, rev(block)), ceil(nblk/2) entries
  const int *pos;          // position of natural index k after the last
                           // forward stage
  const int *rev;          // rev(b) of the last stage's blocks
};

// The same tables on the host (fusedHost in engine.cu), twiddles as exponents
// of W_n.
struct FusedHost {
  std::vector<long> block, inverse;
  std::vector<int4> pairs;
  std::vector<int> pos, rev;
};

// Whether a plan holds a radix-16 stage (its kernels need the WIDE form).
inline bool wideFused(const FusedFFT& p)
{
  for(int s=0; s < p.nst; ++s)
    if(p.radix[s] == 16) return true;
  return false;
}

// Padded position of element j, and the elements to allocate for n.
__host__ __device__ __forceinline__ int spl(int j, int lg) {return j+(j >> lg);}
__host__ __device__ __forceinline__ int fusedSpan(int n, int lg)
{
  return n+((n-1) >> lg);
}

// Synchronise the nt threads of a team: a team of up to a warp runs in step
// with its warp, at most four teams of several warps share a CTA (256
// threads), and their barriers are named by constants (a barrier number in
// a register would reserve all sixteen and allow four CTAs per SM).
__device__ __forceinline__ void teamSync(int team, int nt)
{
  if(nt <= 32) __syncwarp();
  else if(team == 0)
    asm volatile("bar.sync 1, %0;" :: "r"(nt) : "memory");
  else if(team == 1)
    asm volatile("bar.sync 2, %0;" :: "r"(nt) : "memory");
  else if(team == 2)
    asm volatile("bar.sync 3, %0;" :: "r"(nt) : "memory");
  else
    asm volatile("bar.sync 4, %0;" :: "r"(nt) : "memory");
}

template<typename T>
__device__ __forceinline__ cplx<T> swapXY(cplx<T> a) {return mk(a.y,a.x);}

__device__ __forceinline__ double2 ldtw(const double2 *p) {return __ldg(p);}
__device__ __forceinline__ float4 ldtw(const float4 *p) {return __ldg(p);}

// a w with w = exp(2 pi i S k/R) for the constant rotations of half-empty
// butterflies.
template<int R, int S, typename T>
__device__ __forceinline__ cplx<T> rotW(cplx<T> a, int k)
{
  if(k == 0) return a;
  if(4*k == R) return mulI<S>(a);
  if(8*k == R) {
    const T h=(T) FGB_SQRT1_2;
    return S > 0 ? mk((a.x-a.y)*h,(a.y+a.x)*h) : mk((a.x+a.y)*h,(a.y-a.x)*h);
  }
  if(8*k == 3*R) {
    const T h=(T) FGB_SQRT1_2;
    return S > 0 ? mk((-a.x-a.y)*h,(a.x-a.y)*h) : mk((a.y-a.x)*h,(-a.y-a.x)*h);
  }
  double c=1, s=0;
  if(R == 16) {
    c=k == 1 ? FGB_C161 : k == 3 ? FGB_S161 : k == 5 ? -FGB_S161 : -FGB_C161;
    s=k == 1 ? FGB_S161 : k == 3 ? FGB_C161 : k == 5 ? FGB_C161 : FGB_S161;
  } else if(R == 6) {
    c=k == 1 ? 0.5 : -0.5;
    s=FGB_SQRT3_2;
  }
  const T cc=(T) c, ss=(T) (S*s);
  return mk(fma(a.x,cc,-a.y*ss),fma(a.x,ss,a.y*cc));
}

// DFT_R of inputs whose second half is zero: the even outputs are DFT_{R/2}
// of the first half, the odd ones DFT_{R/2} of the first half rotated by
// W_R^k.
template<int R, int S, typename T>
__device__ __forceinline__ void halfDFT(cplx<T> *a)
{
  constexpr int H=R/2;
  cplx<T> e[H], o[H];
#pragma unroll
  for(int k=0; k < H; ++k) {
    e[k]=a[k];
    o[k]=rotW<R,S>(a[k],k);
  }
  if constexpr(H > 1) {
    Codelet<H,S,T>::run(e);
    Codelet<H,S,T>::run(o);
  }
#pragma unroll
  for(int k=0; k < H; ++k) {
    a[2*k]=e[k];
    a[2*k+1]=o[k];
  }
}

// Inputs r >= 1 times w_r, w_r at tw[k + (r-1) stride], then DFT_R; for NC
// columns with the twiddles loaded once.
template<typename T, int R, int NC>
__device__ __forceinline__ void inTwiddleDFT(cplx<T> (*a)[R],
                                             const typename TwT<T>::type *tw,
                                             unsigned k, unsigned stride)
{
  if constexpr(fusedTw<T,R>()) {
    double2 w[R];
#pragma unroll
    for(int r=1; r < R; ++r) w[r]=ldtw(tw+(k+(r-1)*stride));
#pragma unroll
    for(int c=0; c < NC; ++c) TwButterfly<R,1>::run(a[c],w);
  } else {
#pragma unroll
    for(int r=1; r < R; ++r) {
      const typename TwT<T>::type w=ldtw(tw+(k+(r-1)*stride));
#pragma unroll
      for(int c=0; c < NC; ++c) a[c][r]=twmul<1>(a[c][r],w);
    }
#pragma unroll
    for(int c=0; c < NC; ++c) Codelet<R,1,T>::run(a[c]);
  }
}

// A stage of radix R and span m on ld = 2^lt interleaved columns: butterfly
// i = b m + j (block b, position j) has its inputs at `step` elements from
// one another.  m is a multiple of 2^lg, or R m divides it (the pad unit is
// the product of the last radices), so the padded positions add up; with
// the additions left to the addressing modes, index arithmetic is a few
// instructions a butterfly instead of several an element.
struct StageMap {
  int m, lg, lt, sh, step, skip;
  float inv;
  __device__ __forceinline__ StageMap(int R, int m, int lg, int lt)
    : m(m), lg(lg), lt(lt), sh(-1), step(spl(m,lg) << lt), skip((R-1)*m),
      inv(0.0f) {
#ifdef __CUDA_ARCH__
    if((m & (m-1)) == 0) sh=__ffs(m)-1;
#endif
    if(sh < 0) inv=1.0f/(float) m;
  }
  __device__ __forceinline__ int block(int i) const {
    return sh >= 0 ? i >> sh : fdiv(i,inv);
  }
  // Offset of input 0 of butterfly i of block b, column cc.
  __device__ __forceinline__ int offset(int i, int b, int cc) const {
    return (spl(i+b*skip,lg) << lt)+cc;
  }
};

__device__ __forceinline__ int log2of(int ld)
{
#ifdef __CUDA_ARCH__
  return __ffs(ld)-1;
#else
  return 0;
#endif
}

// The column groups of a stage of `per` butterflies each, taken together so
// that short transforms fill a team's threads.
struct ColumnMap {
  int per;
  UDiv d;
  __device__ __forceinline__ explicit ColumnMap(int per) : per(per), d(per) {}
  __device__ __forceinline__ int operator()(int k) const {
    return k < per ? 0 : d(k);
  }
};

// Calls f(c, idx) for this thread's butterflies idx < per of the ncol column
// groups c: all of them in one loop, or (WIDE: the long FP32 transforms with
// radix 16, whose registers are short) one group after the other.
template<bool WIDE, class F>
__device__ __forceinline__ void forColumns(int ncol, int per, int t, int nt,
                                           const F& f)
{
  if constexpr(WIDE) {
#pragma unroll 1
    for(int c=0; c < ncol; ++c)
#pragma unroll 1
      for(int idx=t; idx < per; idx += nt) f(c,idx);
  } else {
    const ColumnMap cols(per);
#pragma unroll 1
    for(int k=t; k < ncol*per; k += nt) {
      const int c=cols(k);
      f(c,k-c*per);
    }
  }
}

// The first forward stage (one block, no twiddles): load(c, cc)(j) gives
// input j of interleaved column cc of group c (groups cs apart, `ncol` of
// them).  HALF: inputs j >= n/2 are zero.  (A thread takes one column
// through a stage at a time: two at once, sharing twiddles, need 128
// registers where three CTAs per SM at 85 serve better, 3D real FP32 rows
// of 512 points 481 against 508 us; FP64 measured the same either way.)
template<typename T, int R, bool HALF, bool WIDE, class Load>
__device__ __forceinline__ void fusedFirst(cplx<T> *x, int cs, int ncol,
                                           const FusedFFT& p, int lt, int t,
                                           int nt, const Load& load)
{
  const int m=p.n/R;
  const StageMap map(R,m,p.lg,lt);
  constexpr int NZ=HALF ? R/2 : R;
  forColumns<WIDE>(ncol,m << lt,t,nt,[&](int c, int idx) {
    const int j=idx >> lt, cc=idx & ((1 << lt)-1);
    cplx<T> a[R];
    const auto in=load(c,cc);
#pragma unroll
    for(int r=0; r < NZ; ++r) a[r]=in(j+r*m);
    cplx<T> *xq=x+c*cs+map.offset(j,0,cc);
#pragma unroll
    for(int r=0; r < NZ; ++r) a[r]=nrm(a[r]);
    if constexpr(HALF) halfDFT<R,1>(a);
    else Codelet<R,1,T>::run(a);
#pragma unroll
    for(int r=0; r < R; ++r) xq[r*map.step]=a[r];
  });
}

// A stage in place, of either direction: twiddles tw[(r-1) stride + b]
// (forward, b the block) or tw[(r-1) stride + j] (inverse, j the position in
// it).  OPT: tw may be NULL, no twiddles (runStages; a test before the
// twiddles keeps their loads behind those of the inputs, 94 against 83 us on
// 4096 FP32 pairs of 1024, so the fused form has none).
template<typename T, int R, bool WIDE, bool OPT=false>
__device__ __forceinline__ void fusedStage(cplx<T> *x, int cs, int ncol,
                                           const FusedFFT& p, int lt, int m,
                                           const typename TwT<T>::type *tw,
                                           int stride, bool inverse, int t,
                                           int nt)
{
  const StageMap map(R,m,p.lg,lt);
  forColumns<WIDE>(ncol,p.n/R << lt,t,nt,[&](int c, int idx) {
    const int i=idx >> lt, cc=idx & ((1 << lt)-1);
    const int b=map.block(i);
    cplx<T> *xq=x+c*cs+map.offset(i,b,cc);
    cplx<T> a[1][R];
#pragma unroll
    for(int r=0; r < R; ++r) a[0][r]=nrm(xq[r*map.step]);
    const int k=inverse ? i-b*m : b;
    if constexpr(!OPT) inTwiddleDFT<T,R,1>(a,tw,k,stride);
    else if constexpr(fusedTw<T,R>()) {
      if(tw) inTwiddleDFT<T,R,1>(a,tw,k,stride);
      else Codelet<R,1,T>::run(a[0]);
    } else {
      if(tw) {
#pragma unroll
        for(int r=1; r < R; ++r)
          a[0][r]=twmul<1>(a[0][r],ldtw(tw+(unsigned) (k+(r-1)*stride)));
      }
      Codelet<R,1,T>::run(a[0]);
    }
#pragma unroll
    for(int r=0; r < R; ++r) xq[r*map.step]=a[0][r];
  });
}

// The last inverse stage: store(c, cc)(j, v) takes output j, its parts in
// their own places again (HALF: only j < n/2, the others are not
// computed).
template<typename T, int R, bool HALF, bool WIDE, class Store>
__device__ __forceinline__ void fusedLast(const cplx<T> *x, int cs, int ncol,
                                          const FusedFFT& p, int lt, int t,
                                          int nt, const Store& store)
{
  const int m=p.n/R;
  const StageMap map(R,m,p.lg,lt);
  constexpr int NZ=HALF ? R/2 : R;
  const typename TwT<T>::type *tw=(const typename TwT<T>::type *) p.twj+(m-1);
  forColumns<WIDE>(ncol,m << lt,t,nt,[&](int c, int idx) {
    const int j=idx >> lt, cc=idx & ((1 << lt)-1);
    const cplx<T> *xq=x+c*cs+map.offset(j,0,cc);
    cplx<T> a[1][R];
#pragma unroll
    for(int r=0; r < R; ++r) a[0][r]=nrm(xq[r*map.step]);
    inTwiddleDFT<T,R,1>(a,tw,j,m);
    const auto out=store(c,cc);
#pragma unroll
    for(int r=0; r < NZ; ++r) out(j+r*m,swapXY(a[0][r]));
  });
}

// Whether the kernels of T hold radix R as an inner or first stage.  WIDE:
// the FP32 kernels with radix 16.
template<typename T, bool WIDE> __device__ constexpr bool fusedRadix(int R)
{
  return R <= 8 || (WIDE && R == 16);
}

#define FGB_FUSED_SWITCH(R,CALL) \
  switch(R) { \
    case 1: {constexpr int R_=1; CALL;} break; \
    case 2: {constexpr int R_=2; CALL;} break; \
    case 3: {constexpr int R_=3; CALL;} break; \
    case 4: {constexpr int R_=4; CALL;} break; \
    case 5: {constexpr int R_=5; CALL;} break; \
    case 6: {constexpr int R_=6; CALL;} break; \
    case 7: {constexpr int R_=7; CALL;} break; \
    case 8: {constexpr int R_=8; CALL;} break; \
    case 16: if constexpr(fusedRadix<T,WIDE>(16)) \
      {constexpr int R_=16; CALL;} break; \
    default: break; \
  }

template<typename T, bool WIDE, class Load>
__device__ __forceinline__ void runFusedFirst(cplx<T> *x, int cs, int ncol,
                                              const FusedFFT& p, int lt, int t,
                                              int nt, const Load& load)
{
  if(p.half) {
    switch(p.radix[0]) {
      case 2: fusedFirst<T,2,true,WIDE>(x,cs,ncol,p,lt,t,nt,load); break;
      case 4: fusedFirst<T,4,true,WIDE>(x,cs,ncol,p,lt,t,nt,load); break;
      case 6: fusedFirst<T,6,true,WIDE>(x,cs,ncol,p,lt,t,nt,load); break;
      case 8: fusedFirst<T,8,true,WIDE>(x,cs,ncol,p,lt,t,nt,load); break;
      case 16:
        if constexpr(fusedRadix<T,WIDE>(16))
          fusedFirst<T,16,true,WIDE>(x,cs,ncol,p,lt,t,nt,load);
        break;
      default: break;
    }
    return;
  }
  FGB_FUSED_SWITCH(p.radix[0],
                   (fusedFirst<T,R_,false,WIDE>(x,cs,ncol,p,lt,t,nt,load)))
}

template<typename T, bool WIDE, class Store>
__device__ __forceinline__ void runFusedLast(const cplx<T> *x, int cs,
                                             int ncol, const FusedFFT& p,
                                             int lt, int t, int nt,
                                             const Store& store)
{
  if(p.half) {
    switch(p.radix[0]) {
      case 2: fusedLast<T,2,true,WIDE>(x,cs,ncol,p,lt,t,nt,store); break;
      case 4: fusedLast<T,4,true,WIDE>(x,cs,ncol,p,lt,t,nt,store); break;
      case 6: fusedLast<T,6,true,WIDE>(x,cs,ncol,p,lt,t,nt,store); break;
      case 8: fusedLast<T,8,true,WIDE>(x,cs,ncol,p,lt,t,nt,store); break;
      case 16:
        if constexpr(fusedRadix<T,WIDE>(16))
          fusedLast<T,16,true,WIDE>(x,cs,ncol,p,lt,t,nt,store);
        break;
      default: break;
    }
    return;
  }
  FGB_FUSED_SWITCH(p.radix[0],
                   (fusedLast<T,R_,false,WIDE>(x,cs,ncol,p,lt,t,nt,store)))
}

// CTAs of 256 threads per SM the row kernels' registers leave room for.
template<typename T> __host__ __device__ constexpr int fusedBlocks()
{
  return std::is_same<T,double>::value ? 2 : 3;
}

// The middle stages, each after a team barrier: 1 .. nst-2 forward, nst-2 ..
// 1 inverse.  Returns the blocks of the last stage.
template<typename T, bool WIDE>
__device__ __forceinline__ int runFusedMiddle(cplx<T> *x, int cs, int ncol,
                                              const FusedFFT& p, int lt,
                                              bool inverse, int team, int t,
                                              int nt)
{
  typedef typename TwT<T>::type Tw;
  const int R0=p.radix[0];
  const Tw *twb=(const Tw *) p.twb, *twj=(const Tw *) p.twj;
  int nblk=R0, m=p.n/R0;
  if(inverse) m=p.radix[p.nst-1];
  for(int k=1; k < p.nst-1; ++k) {
    const int s=inverse ? p.nst-1-k : k;
    const int R=p.radix[s];
    if(!inverse) m /= R;
    const Tw *tw=inverse ? twj+(m-1) : twb+(nblk-R0);
    const int stride=inverse ? m : nblk;
    teamSync(team,nt);
    FGB_FUSED_SWITCH(R,(fusedStage<T,R_,WIDE>(x,cs,ncol,p,lt,m,tw,stride,
                                            inverse,t,nt)))
    if(inverse) m *= R;
    else nblk *= R;
  }
  return nblk;
}

// The staged form: the multiplier, the (un)packing of real data and the loads
// and stores of column tiles are loops of their own around the stages, and
// all stages of a radix, forward and inverse, share one piece of code.
//
// Float-float takes it but for outer axes of many columns (stagedColumns in
// engine.cu): one of its butterflies is up to 14 KB of instructions and its
// kernels are bound by fetching them.  With the last forward stage, the
// product and the first inverse stage fused, a Hermitian row kernel of 768 points stalled on instructions 3.8 times per issue
// against 0.9 here (89 against 72 us), and a 39 x 93 convolution took 43 us
// against 34.  Only complex rows keep their first and last stages fused (the
// half that padding leaves empty is not computed there): 4096 pairs of 1024
// points, 454 against 497 us.
//
// FP64 takes it for real outer axes and for those Hermitian rows that do not
// take the ping-pong transform (stagedReal and hermPingPong in engine.cu), FP32
// for small real outer launches, and complex rows as fusedRow says.
//
// The forward stages from `first` on for A columns at x (cs apart, each of
// 2^lt interleaved ones), mid(), the inverse stages down to `first` for B
// columns; A = 0: inverse only, B = 0: forward only.  Ends synchronised.
template<typename T, bool WIDE=false, class Mid>
__device__ __forceinline__ void runStages(cplx<T> *x, int cs, int A, int B,
                                          const FusedFFT& p, int lt,
                                          int first, int team, int t, int nt,
                                          const Mid& mid)
{
  typedef typename TwT<T>::type Tw;
  const int R0=p.radix[0], half=p.nst-first;
  const Tw *twb=(const Tw *) p.twb, *twj=(const Tw *) p.twj;
  int nblk=first ? R0 : 1, m=A == 0 ? 1 : p.n/(first ? R0 : 1);
#pragma unroll 1
  for(int q=A == 0 ? half : 0; q < (B == 0 ? half : 2*half); ++q) {
    const bool inverse=q >= half;
    if(q == half) {
      teamSync(team,nt);
      mid();
    }
    const int s=inverse ? p.nst-1-(q-half) : first+q;
    const int R=p.radix[s];
    if(!inverse) m /= R;
    const Tw *tw=inverse ? (m > 1 ? twj+(m-1) : NULL) :
      (s > 0 ? twb+(nblk-R0) : NULL);
    const int stride=inverse ? m : nblk, ncol=inverse ? B : A;
    teamSync(team,nt);
    FGB_FUSED_SWITCH(R,(fusedStage<T,R_,WIDE,true>(x,cs,ncol,p,lt,m,tw,stride,
                                                   inverse,t,nt)))
    if(inverse) m *= R;
    else nblk *= R;
  }
  teamSync(team,nt);
}

} // namespace fgb
