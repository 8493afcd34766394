// kernels.cu -- GB300 (sm_103a) kernels of the hybrid dealiased convolution.
// See kernels.cuh for the decomposition; reference routines are cited per
// kernel.  The innermost-axis (row) kernels live in rowkernels.cuh, templated
// on the multiplier; this file instantiates them for the built-in
// multipliers and holds the outer-axis, batched and copy kernels.
#include "rowkernels.cuh"

#include <algorithm>
#include <climits>
#include <type_traits>

namespace fgb {


// ---------------------------------------------------------------------------
// Offset of column col on the data side of an outer kernel (the caller's
// arrays): col itself for dense layouts, (col / cz) cs + col % cz for the
// strided layouts of fftPad(L, M, app, C, S) with S > C (convolve.h:515-536;
// Convolution2/3's Sx, Sy, convolve.h:1274, 1556).
template<typename T>
__device__ __forceinline__ long long dataCol(const OuterPlan<T>& P, int col)
{
  if(P.cz <= 0) return col;
  const int g=col/P.cz;
  return (long long) g*P.cs+(col-g*P.cz);
}

// The four-step twiddle W_NX^{col k} (col k < C m = NX).  FP32 multiplies two
// entries that stay in L1, W^{e mod 256} and W^{e - e mod 256}, in
// float-float (to 2^-44, far below the data's rounding): neighbouring
// columns' entries lie k apart in the full table, so reading it moved 32
// bytes from L2 for every 8 of data (512 uneven problems 576 us, 490 this
// way).  FP64, bound by its pipe, reads the table.
template<typename T>
__device__ __forceinline__ typename TwT<T>::type fourStep(const OuterPlan<T>& P,
                                                          long long e)
{
  if constexpr(std::is_same<T,float>::value) {
    const int i=(int) e;
    const float4 a=ldtw(P.twX+(i & 255)), b=ldtw(P.twC+(i >> 8));
    const cplx<ff> w=cmul(mk(ff(a.x,a.z),ff(a.y,a.w)),
                          mk(ff(b.x,b.z),ff(b.y,b.w)));
    return make_float4(w.x.hi,w.y.hi,w.x.lo,w.y.lo);
  } else return P.twX[e];
}

// ---------------------------------------------------------------------------
// Outer forward, complex data: residue block r of the padded transform along
// a strided axis for `tile` adjacent columns.
template<typename T>
__device__ __forceinline__ void outerFwdTile(const OuterPlan<T>& P, int ctile,
                                             int r, int z,
                                             unsigned char *smemRaw)
{
  const int tile=P.tile, m=P.m, N=P.N, c=P.cshift, L=P.L;
  cplx<T> *x=(cplx<T> *) smemRaw;
  cplx<T> *y=x+padded(m*tile);
  const int tid=threadIdx.x, nthr=blockDim.x;
  const int col0=ctile*tile;
  const int a=z % P.count;
  const long long batch=z/P.count;
  const cplx<T> *src=P.in[a]+batch*P.inBatch;
  cplx<T> *dst=P.out[a]+batch*P.outBatch;
  const typename TwT<T>::type *tw=P.twN;
  const UDiv dTile(tile);

  if(P.flat != FLAT_PAD) {
    // Long rows of the other kinds: every position n = t*C + col of the
    // flattened row holds the data index of its kind (FlatMode); loaded
    // and converted directly (conjugated mirror, real values).
    const T *srcR=(const T *) P.in[a]+batch*P.inBatch;
    const int sh=ioShift<T>(P.ioShift,a);
    for(int i=tid; i < m*tile; i += nthr) {
      int t=dTile(i), cc=i-t*tile;
      int col=col0+cc;
      cplx<T> v=mk((T) 0,(T) 0);
      if(col < P.C) {
        const long long n=(long long) t*P.inRow+col;
        if(P.flat == FLAT_CENTERED) {
          long long sx=n+P.flatC;
          if(sx >= P.NX) sx -= P.NX;
          if(sx < P.Ltot) v=loadIO(src+sx,P.io64 & 1,sh);
        } else if(P.flat == FLAT_HERMITIAN) {
          if(n < P.Ltot) {
            v=loadIO(src+n,P.io64 & 1,sh);
            if(n == 0) v.y=(T) 0;
          } else if(P.NX-n < P.Ltot) v=conjg(loadIO(src+(P.NX-n),P.io64 & 1,sh));
        } else if(n < P.Ltot) {
          v=mk(loadIOr(srcR+n,P.io64 & 1,sh),(T) 0);
        }
      }
      x[sp(i)]=v;
    }
    __syncthreads();
  } else if(L <= m) {
    // One term per output: asynchronous copies straight to each value's
    // transform slot, then the conversion and residue twiddle in place by
    // the same thread.
    for(int i=tid; i < m*tile; i += nthr) {
      int t=dTile(i), cc=i-t*tile;
      int col=col0+cc;
      int s=posmod(t+c,m);
      long long off=(long long) s*P.inRow+dataCol(P,col);
      if(s < L && col < P.C && off < P.Ltot) cpAsync(x+sp(i),src+off);
      else x[sp(i)]=mk((T) 0,(T) 0);
    }
    cpAsyncWait();
    if(r != 0 || (P.io64 & 1)) {
      for(int i=tid; i < m*tile; i += nthr) {
        int t=dTile(i), cc=i-t*tile;
        int col=col0+cc;
        int s=posmod(t+c,m);
        long long off=(long long) s*P.inRow+dataCol(P,col);
        if(s < L && col < P.C && off < P.Ltot) {
          if(P.io64 & 1) convertStaged(x,sp(i),ioShift<T>(P.ioShift,a));
          if(r != 0) x[sp(i)]=twmul<1>(x[sp(i)],tw[twExp(s,c,r,N)]);
        }
      }
    }
    __syncthreads();
  } else {
    // Stage the L x tile input block in y with asynchronous copies (many
    // loads in flight per thread instead of one dependent load per
    // output), then fold it into x with the residue twiddles.
    for(int i=tid; i < L*tile; i += nthr) {
      int s=dTile(i), cc=i-s*tile;
      int col=col0+cc;
      long long off=(long long) s*P.inRow+dataCol(P,col);
      if(col < P.C && off < P.Ltot) cpAsync(y+i,src+off);
      else y[i]=mk((T) 0,(T) 0);
    }
    cpAsyncWait();
    if(std::is_same<T,ff>::value && (P.io64 & 1)) {
      // The caller's FP64 values were staged as they are: convert them.
      for(int i=tid; i < L*tile; i += nthr) {
        int s=dTile(i), cc=i-s*tile;
        int col=col0+cc;
        long long off=(long long) s*P.inRow+dataCol(P,col);
        if(col < P.C && off < P.Ltot)
          convertStaged(y,i,ioShift<T>(P.ioShift,a));
      }
    }
    __syncthreads();
    for(int i=tid; i < m*tile; i += nthr) {
      int t=dTile(i), cc=i-t*tile;
      cplx<T> sum=mk((T) 0,(T) 0);
      int s0=posmod(t+c,m);
      // The twiddle exponent advances by m r mod N from term to term.
      int e=r != 0 ? twExp(s0,c,r,N) : 0;
      const int de=r != 0 ? twStep(m,r,N) : 0;
      for(int s=s0; s < L; s += m) {
        cplx<T> v=y[s*tile+cc];
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
  }

  cplx<T> *X=fftSmem<T,1>(x,y,P.fp,tile,tile,tid,nthr);
  for(int i=tid; i < m*tile; i += nthr) {
    int j=dTile(i), cc=i-j*tile;
    int col=col0+cc;
    if(col < P.C) {
      cplx<T> v=X[sp(i)];
      long long k=(long long) r*m+j;
      if(P.twX) v=twmul<1>(v,fourStep(P,col*k));
      dst[k*P.outRow+col]=v;
    }
  }
  __syncthreads();
}

template<typename T>
__global__ void __launch_bounds__(256)
outerFwdKernel(const OuterPlan<T> P)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  outerFwdTile<T>(P,blockIdx.x,blockIdx.y,blockIdx.z,smemRaw);
}

// Outer backward, complex data: all residues of a column tile, accumulated.
template<typename T>
__device__ __forceinline__ void outerBwdTile(const OuterPlan<T>& P, int ctile,
                                             int z, unsigned char *smemRaw)
{
  const int tile=P.tile, m=P.m, N=P.N, c=P.cshift, L=P.L;
  // One residue: the outputs come straight from the transform, with no
  // accumulator in shared memory.
  const bool direct=P.q == 1;
  cplx<T> *acc=(cplx<T> *) smemRaw;
  cplx<T> *x=direct ? acc : acc+L*tile;
  cplx<T> *y=x+padded(m*tile);
  const int tid=threadIdx.x, nthr=blockDim.x;
  const int col0=ctile*tile;
  const int b=z % P.count;
  const long long batch=z/P.count;
  const cplx<T> *src=P.in[b]+batch*P.inBatch;
  cplx<T> *dst=P.out[b]+batch*P.outBatch;
  const typename TwT<T>::type *tw=P.twN;
  const UDiv dTile(tile);

  if(!direct)
    for(int i=tid; i < L*tile; i += nthr) acc[i]=mk((T) 0,(T) 0);
  for(int r=0; r < P.q; ++r) {
    for(int i=tid; i < m*tile; i += nthr) {
      int j=dTile(i), cc=i-j*tile;
      int col=col0+cc;
      if(col < P.C) cpAsync(x+sp(i),src+((long long) r*m+j)*P.inRow+col);
      else x[sp(i)]=mk((T) 0,(T) 0);
    }
    cpAsyncWait();
    __syncthreads();
    if(P.twX) {
      for(int i=tid; i < m*tile; i += nthr) {
        int j=dTile(i), cc=i-j*tile;
        int col=col0+cc;
        if(col < P.C)
          x[sp(i)]=twmul<-1>(x[sp(i)],
                             fourStep(P,col*((long long) r*m+j)));
      }
      __syncthreads();
    }
    cplx<T> *X=fftSmem<T,-1>(x,y,P.fp,tile,tile,tid,nthr);
    if(direct && P.flat != FLAT_PAD) {
      // Long rows of the other kinds: the output of data index sx is the
      // flattened position n of its kind (FlatMode).
      T *dstR=(T *) P.out[b]+batch*P.outBatch;
      const int sh=ioShift<T>(P.ioShift,8+b);
      for(int i=tid; i < m*tile; i += nthr) {
        int t=dTile(i), cc=i-t*tile;
        int col=col0+cc;
        if(col >= P.C) continue;
        const long long n=(long long) t*P.outRow+col;
        const cplx<T> v=X[sp(i)]*P.scale;
        if(P.flat == FLAT_CENTERED) {
          long long sx=n+P.flatC;
          if(sx >= P.NX) sx -= P.NX;
          if(sx < P.Ltot) storeIO(dst+sx,v,P.io64 & 2,sh);
        } else if(n < P.Ltot) {
          if(P.flat == FLAT_REAL) storeIOr(dstR+n,v.x,P.io64 & 2,sh);
          else storeIO(dst+n,v,P.io64 & 2,sh);
        }
      }
      __syncthreads();
      return;
    }
    if(direct) {
      for(int i=tid; i < L*tile; i += nthr) {
        int s=dTile(i), cc=i-s*tile;
        int col=col0+cc;
        long long off=(long long) s*P.outRow+dataCol(P,col);
        if(col < P.C && off < P.Ltot)
          storeIO(dst+off,X[sp(posmod(s-c,m)*tile+cc)]*P.scale,P.io64 & 2,
                  ioShift<T>(P.ioShift,8+b));
      }
      __syncthreads();
      return;
    }
    for(int i=tid; i < L*tile; i += nthr) {
      int s=dTile(i), cc=i-s*tile;
      int t=posmod(s-c,m);
      cplx<T> v=X[sp(t*tile+cc)];
      if(r != 0) v=twmul<-1>(v,tw[twExp(s,c,r,N)]);
      acc[i]=accum(acc[i],v);
    }
    __syncthreads();
  }
  for(int i=tid; i < L*tile; i += nthr) {
    int s=dTile(i), cc=i-s*tile;
    int col=col0+cc;
    long long off=(long long) s*P.outRow+dataCol(P,col);
    if(col < P.C && off < P.Ltot)
      storeIO(dst+off,acc[i]*P.scale,P.io64 & 2,ioShift<T>(P.ioShift,8+b));
  }
  __syncthreads();
}

template<typename T>
__global__ void __launch_bounds__(256)
outerBwdKernel(const OuterPlan<T> P)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  outerBwdTile<T>(P,blockIdx.x,blockIdx.z,smemRaw);
}

// ---------------------------------------------------------------------------
// Fused outer kernels (fft_fused.cuh), for residue blocks at least as long as
// the data: the first forward stage reads the caller's columns and applies
// the residue twiddle, the last one writes the staging rows, in the
// digit-reversed order of the transform (the row kernels do not depend on
// row order and the backward undoes it).  The column tile's values cross
// shared memory once between stages and never before the first or after
// the last.
// The staged form (runStages): the tile's inputs into shared memory, and its
// outputs out of it.  in(cc, j) gives element j of column cc.
template<typename T, class In>
__device__ __forceinline__ void loadTile(cplx<T> *x, const FusedFFT& p,
                                           int lt, int tid, int nthr,
                                           const In& in)
{
#pragma unroll 4
  for(int idx=tid; idx < p.n << lt; idx += nthr) {
    const int j=idx >> lt, cc=idx & ((1 << lt)-1);
    x[(spl(j,p.lg) << lt)+cc]=in(cc,j);
  }
}

// FP64 bits read as a float-float value, converted in line (one place, whose
// loads the loop issues together).
template<typename T>
__device__ __forceinline__ cplx<T> fromBits(cplx<T> v, int) {return v;}
__device__ __forceinline__ cplx<ff> fromBits(cplx<ff> v, int sh)
{
  return mk(toFF(__hiloint2double(__float_as_int(v.x.lo),
                                  __float_as_int(v.x.hi)),sh),
            toFF(__hiloint2double(__float_as_int(v.y.lo),
                                  __float_as_int(v.y.hi)),sh));
}

template<typename T, class Store>
__device__ __forceinline__ void storeTile(const cplx<T> *x,
                                            const FusedFFT& p, int lt, int tid,
                                            int nthr, const Store& store)
{
#pragma unroll 2
  for(int idx=tid; idx < p.n << lt; idx += nthr) {
    const int j=idx >> lt, cc=idx & ((1 << lt)-1);
    store(0,cc)(j,swapXY(x[(spl(j,p.lg) << lt)+cc]));
  }
}

template<typename T, int R>
__device__ __forceinline__ void outerLastFwd(const OuterPlan<T>& P,
                                             const cplx<T> *x, cplx<T> *dst,
                                             int col0, int nblk, int tid,
                                             int nthr)
{
  typedef typename TwT<T>::type Tw;
  const FusedFFT& p=P.fz;
  const int lt=log2of(P.tile), total=nblk << lt;
  const Tw *tw=(const Tw *) p.twb+(nblk-p.radix[0]);
#pragma unroll 1
  for(int idx=tid; idx < total; idx += nthr) {
    const int b=idx >> lt, cc=idx & (P.tile-1), col=col0+cc;
    const cplx<T> *xq=x+(spl(b*R,p.lg) << lt)+cc;
    cplx<T> a[1][R];
#pragma unroll
    for(int r=0; r < R; ++r) a[0][r]=nrm(xq[r << lt]);
    inTwiddleDFT<T,R,1>(a,tw,b,nblk);
    if(col >= P.C) continue;
    if(P.twX) {
      // Position b R + r holds entry rev(b) + r nblk.
      const int k=P.fz.rev[b];
#pragma unroll
      for(int r=0; r < R; ++r)
        a[0][r]=twmul<1>(a[0][r],fourStep(P,(long long) col*(k+r*nblk)));
    }
    cplx<T> *d=dst+(long long) (b*R)*P.outRow+col;
#pragma unroll
    for(int r=0; r < R; ++r) d[r*P.outRow]=a[0][r];
  }
}

// Data entries of column col: all L, but for the flattened rows of the
// batched launch (twX), whose last one may be short.
template<typename T>
__device__ __forceinline__ int columnTop(const OuterPlan<T>& P, int col,
                                         long long row)
{
  if(col >= P.C) return 0;
  if(!P.twX) return P.L;
  return ((int) P.Ltot-col+(int) row-1)/(int) row;
}

// STAGED: the staged form (OuterPlan::staged), in kernels of its own.
template<typename T, bool WIDE, bool STAGED=false>
__device__ __forceinline__ void outerFwdFused(const OuterPlan<T>& P, int ctile,
                                              int r, int z,
                                              unsigned char *smemRaw)
{
  const int tile=P.tile, m=P.m, N=P.N, c=P.cshift, L=P.L;
  cplx<T> *x=(cplx<T> *) smemRaw;
  const int tid=threadIdx.x, nthr=blockDim.x;
  const int col0=ctile*tile;
  const int a=z % P.count;
  const long long batch=z/P.count;
  const cplx<T> *src=P.in[a]+batch*P.inBatch;
  cplx<T> *dst=P.out[a]+batch*P.outBatch+(long long) r*m*P.outRow;
  const int lt=log2of(tile);
  const int sh=ioShift<T>(P.ioShift,a);
  if constexpr(STAGED) {
    loadTile(x,P.fz,lt,tid,nthr,[&](int cc, int j) {
        int s=j+c;
        if(s >= m) s -= m;
        cplx<T> v=mk((T) 0,(T) 0);
        if(s < L && col0+cc < P.C) {
          v=src[s*P.inRow+dataCol(P,col0+cc)];
          if(P.io64 & 1) v=fromBits(v,sh);
          if(r != 0) v=twmul<1>(v,P.twN[twExp(s,c,r,N)]);
        }
        return v;
      });
    runStages<T,WIDE>(x,0,1,0,P.fz,lt,0,0,tid,nthr,[] {});
#pragma unroll 4
    for(int idx=tid; idx < m << lt; idx += nthr) {
      const int j=idx >> lt, cc=idx & (tile-1);
      if(col0+cc < P.C)
        dst[j*P.outRow+col0+cc]=x[(spl(j,P.fz.lg) << lt)+cc];
    }
  } else {
    const auto load=[&](int, int cc) {
      const int top=columnTop(P,col0+cc,P.inRow);
      const cplx<T> *f=src+dataCol(P,col0+cc);
      return [=,&P](int j) {
        int s=j+c;
        if(s >= m) s -= m;
        cplx<T> v=mk((T) 0,(T) 0);
        if(s < top) {
          v=loadIO(f+s*P.inRow,P.io64 & 1,sh);
          if(r != 0) v=twmul<1>(v,P.twN[twExp(s,c,r,N)]);
        }
        return v;
      };
    };
    runFusedFirst<T,WIDE>(x,0,1,P.fz,lt,tid,nthr,load);
    const int nblk=runFusedMiddle<T,WIDE>(x,0,1,P.fz,lt,false,0,tid,nthr);
    __syncthreads();
    FGB_FUSED_SWITCH(P.fz.radix[P.fz.nst-1],
                     (outerLastFwd<T,R_>(P,x,dst,col0,nblk,tid,nthr)))
  }
}

template<typename T>
__global__ void __launch_bounds__(256)
outerFwdFusedKernel(const OuterPlan<T> P)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  outerFwdFused<T,false>(P,blockIdx.x,blockIdx.y,blockIdx.z,smemRaw);
}

// The first inverse stage: staging rows into shared memory.
template<typename T, int R, bool CG>
__device__ __forceinline__ void outerFirstInv(const OuterPlan<T>& P,
                                              cplx<T> *x, const cplx<T> *src,
                                              int col0, int tid, int nthr)
{
  const FusedFFT& p=P.fz;
  const int lt=log2of(P.tile), total=p.n/R << lt;
#pragma unroll 1
  for(int idx=tid; idx < total; idx += nthr) {
    const int b=idx >> lt, cc=idx & (P.tile-1), col=col0+cc;
    const cplx<T> *s=src+(long long) (b*R)*P.inRow+col;
    cplx<T> a[R];
#pragma unroll
    for(int r=0; r < R; ++r)
      a[r]=col < P.C ? ldx<CG>(s+r*P.inRow) : mk((T) 0,(T) 0);
    if(P.twX && col < P.C) {
      const int k=P.fz.rev[b], nblk=p.n/R;
#pragma unroll
      for(int r=0; r < R; ++r)
        a[r]=twmul<-1>(a[r],fourStep(P,(long long) col*(k+r*nblk)));
    }
#pragma unroll
    for(int r=0; r < R; ++r) a[r]=nrm(swapXY(a[r]));
    Codelet<R,1,T>::run(a);
    cplx<T> *xq=x+(spl(b*R,p.lg) << lt)+cc;
#pragma unroll
    for(int r=0; r < R; ++r) xq[r << lt]=a[r];
  }
}

// All residues of a column tile; with several, a thread adds the outputs it
// computes into its own entries of an accumulator behind the tile.
template<typename T, bool WIDE, bool CG, bool STAGED=false>
__device__ __forceinline__ void outerBwdFused(const OuterPlan<T>& P, int ctile,
                                              int z, unsigned char *smemRaw)
{
  const int tile=P.tile, m=P.m, N=P.N, c=P.cshift, L=P.L, q=P.q;
  cplx<T> *x=(cplx<T> *) smemRaw;
  cplx<T> *acc=x+fusedSpan(P.fz.n,P.fz.lg)*tile;
  const int tid=threadIdx.x, nthr=blockDim.x;
  const int col0=ctile*tile;
  const int b=z % P.count;
  const long long batch=z/P.count;
  const cplx<T> *src=P.in[b]+batch*P.inBatch;
  cplx<T> *dst=P.out[b]+batch*P.outBatch;
  const int lt=log2of(tile);
  const int sh=ioShift<T>(P.ioShift,8+b);
  for(int r=0; r < q; ++r) {
    const cplx<T> *sr=src+(long long) r*m*P.inRow;
    const auto store=[&](int, int cc) {
      const int top=columnTop(P,col0+cc,P.outRow);
      cplx<T> *f=dst+dataCol(P,col0+cc);
      return [=,&P](int j, cplx<T> v) {
        int s=j+c;
        if(s >= m) s -= m;
        if(s >= top) return;
        if(q > 1) {
          if(r != 0) v=accum(acc[s*tile+cc],
                             twmul<-1>(v,P.twN[twExp(s,c,r,N)]));
          if(r < q-1) {
            acc[s*tile+cc]=v;
            return;
          }
        }
        storeIO(f+s*P.outRow,v*P.scale,P.io64 & 2,sh);
      };
    };
    if constexpr(STAGED) {
      loadTile(x,P.fz,lt,tid,nthr,[&](int cc, int j) {
          return col0+cc < P.C ? swapXY(sr[j*P.inRow+col0+cc]) :
            mk((T) 0,(T) 0);
        });
      runStages<T,WIDE>(x,0,0,1,P.fz,lt,0,0,tid,nthr,[] {});
      storeTile(x,P.fz,lt,tid,nthr,store);
    } else {
      FGB_FUSED_SWITCH(P.fz.radix[P.fz.nst-1],
                       (outerFirstInv<T,R_,CG>(P,x,sr,col0,tid,nthr)))
      runFusedMiddle<T,WIDE>(x,0,1,P.fz,lt,true,0,tid,nthr);
      __syncthreads();
      runFusedLast<T,WIDE>(x,0,1,P.fz,lt,tid,nthr,store);
    }
    if(r < q-1) __syncthreads();
  }
}

template<typename T>
__global__ void __launch_bounds__(256)
outerBwdFusedKernel(const OuterPlan<T> P)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  outerBwdFused<T,false,false>(P,blockIdx.x,blockIdx.z,smemRaw);
}

// FP32 plans with a radix-16 stage: their own instantiations, capped at 85
// registers a thread (the wider codelet needs more registers than the
// others may take).
template<typename T>
__global__ void __launch_bounds__(256,3)
outerFwdFusedKernel16(const OuterPlan<T> P)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  outerFwdFused<T,true>(P,blockIdx.x,blockIdx.y,blockIdx.z,smemRaw);
}

template<typename T>
__global__ void __launch_bounds__(256,3)
outerBwdFusedKernel16(const OuterPlan<T> P)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  outerBwdFused<T,true,false>(P,blockIdx.x,blockIdx.z,smemRaw);
}

// The staged form (FP32: with radix 16), for small launches (stagedColumns in
// engine.cu).  Kernels of their own: as a branch of the fused FP32 ones their
// code cost those 4 to 10 % (2D 1023 x 512 modes, forward 22.8 -> 24.2 us,
// backward 14.9 -> 16.7).
template<typename T>
__global__ void __launch_bounds__(256,3)
outerFwdStagedKernel(const OuterPlan<T> P)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  outerFwdFused<T,std::is_same<T,float>::value,true>(P,blockIdx.x,blockIdx.y,
                                                     blockIdx.z,smemRaw);
}

template<typename T>
__global__ void __launch_bounds__(256,3)
outerBwdStagedKernel(const OuterPlan<T> P)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  outerBwdFused<T,std::is_same<T,float>::value,false,true>(P,blockIdx.x,
                                                           blockIdx.z,smemRaw);
}

// ---------------------------------------------------------------------------
// Outer axis, real data (fftPadReal with explicit padding to even N), both
// directions in the fused form: z[t] = f[2t] + i f[2t+1] through a transform
// of length Nh = N/2, the N/2+1 modes in natural order on the other side.
// Unpacking pairs mode k with Nh-k; the last forward stage holds modes
// kappa + nblk t of block b (kappa = rev(b)), whose partners are all in the
// block of nblk - kappa, so one thread finishes both blocks of a pair
// (FusedFFT::pairs, blocks in order: b, its partner, kappa; the first entry
// holds blocks 0 and that of nblk/2, -1 if nblk is odd, which are their own
// partners).  The inverse packs in the same pairs as it loads.  That is the
// fused form, which FP32 takes for large launches; in FP64 and float-float,
// and in small FP32 launches, a pair's two butterflies one after the other
// leave most threads idle or waiting, and the staged form, one mode pair at a
// time, is faster (stagedReal in engine.cu).

// F[k] = e + W_N^k o and F[Nh-k] = conj(e - W_N^k o) from Z[k] and
// Z[Nh-k], e = (Z[k] + conj Z[Nh-k])/2, o = -i (Z[k] - conj Z[Nh-k])/2.
template<typename T>
__device__ __forceinline__ void realUnpack(cplx<T> zk, cplx<T> zm,
                                           typename TwT<T>::type w,
                                           cplx<T>& F, cplx<T>& Fc)
{
  const T half=(T) 0.5;
  const cplx<T> zb=conjg(zm);
  const cplx<T> e=(zk+zb)*half, dd=zk-zb;
  const cplx<T> o=mk(dd.y*half,-dd.x*half);
  if constexpr(std::is_same<T,double>::value) {
    F=fmaTw<1>(e,o,w);
    Fc=mk(fma((T) 2,e.x,-F.x),fma((T) -2,e.y,F.y));
  } else {
    const cplx<T> q=twmul<1>(o,w);
    F=e+q;
    Fc=conjg(e-q);
  }
}

// Y[k] = s + i d and Y[Nh-k] = conj(s - i d) from G[k] and G[Nh-k], s = G[k]
// + conj G[Nh-k], d = W_N^{-k} (G[k] - conj G[Nh-k]).
template<typename T>
__device__ __forceinline__ void realPack(cplx<T> gk, cplx<T> gm,
                                         typename TwT<T>::type w,
                                         cplx<T>& Y, cplx<T>& Yc)
{
  const cplx<T> gb=conjg(gm);
  const cplx<T> s=gk+gb;
  const cplx<T> d=twmul<-1>(gk-gb,w);
  Y=mk(s.x-d.y,s.y+d.x);
  Yc=mk(s.x+d.y,d.x-s.y);
}

template<typename T, int R>
__device__ __forceinline__ void realLastFwd(const OuterPlan<T>& P,
                                            const cplx<T> *x, cplx<T> *dst,
                                            int col0, int tid, int nthr)
{
  typedef typename TwT<T>::type Tw;
  const FusedFFT& p=P.fz;
  const int lt=log2of(P.tile), Nh=p.n, nblk=Nh/R, total=(nblk+1)/2 << lt;
  const Tw *tw=(const Tw *) p.twb+(nblk-p.radix[0]);
#pragma unroll 1
  for(int idx=tid; idx < total; idx += nthr) {
    const int i=idx >> lt, cc=idx & (P.tile-1), col=col0+cc;
    const int4 pr=__ldg(p.pairs+i);
    const int b=pr.x, b2=max(pr.y,0), kappa=pr.z;
    cplx<T> u[1][R], v[1][R];
    const cplx<T> *xq=x+(spl(b*R,p.lg) << lt)+cc;
    const cplx<T> *xr=x+(spl(b2*R,p.lg) << lt)+cc;
#pragma unroll
    for(int r=0; r < R; ++r) {
      u[0][r]=nrm(xq[r << lt]);
      v[0][r]=nrm(xr[r << lt]);
    }
    inTwiddleDFT<T,R,1>(u,tw,b,nblk);
    inTwiddleDFT<T,R,1>(v,tw,b2,nblk);
    if(col >= P.C) continue;
    cplx<T> *d=dst+col;
    const int top=P.kc > 0 ? P.kc : Nh+1;
    auto put=[&](int k, cplx<T> f) {
      if(k < top) d[(long long) k*P.outRow]=P.conj ? conjg(f) : f;
    };
    cplx<T> F, Fc;
    if(i != 0) {
#pragma unroll
      for(int r=0; r < R; ++r) {
        const int k=kappa+r*nblk;
        realUnpack(u[0][r],v[0][R-1-r],ldtw(P.twN+k),F,Fc);
        put(k,F);
        put(Nh-k,Fc);
      }
    } else {
#pragma unroll
      for(int r=0; r <= R/2; ++r) {
        realUnpack(u[0][r],u[0][(R-r)%R],ldtw(P.twN+r*nblk),F,Fc);
        put(r*nblk,F);
        if(2*r < R) put(Nh-r*nblk,Fc);
      }
      if(pr.y >= 0) {
#pragma unroll
        for(int r=0; r < (R+1)/2; ++r) {
          const int k=nblk/2+r*nblk;
          realUnpack(v[0][r],v[0][R-1-r],ldtw(P.twN+k),F,Fc);
          put(k,F);
          if(2*r < R-1) put(Nh-k,Fc);
        }
      }
    }
  }
}

template<typename T, bool WIDE, bool STAGED>
__device__ __forceinline__ void outerRealFwd(const OuterPlan<T>& P,
                                             unsigned char *smemRaw)
{
  const int tile=P.tile, L=P.L;
  cplx<T> *x=(cplx<T> *) smemRaw;
  const int tid=threadIdx.x, nthr=blockDim.x;
  const int col0=blockIdx.x*tile;
  const int a=blockIdx.z % P.count;
  const long long batch=blockIdx.z/P.count;
  const T *src=(const T *) P.in[a]+batch*P.inBatch;
  cplx<T> *dst=P.out[a]+batch*P.outBatch;
  const int lt=log2of(tile);
  const int sh=ioShift<T>(P.ioShift,a);
  if constexpr(STAGED) {
    loadTile(x,P.fz,lt,tid,nthr,[&](int cc, int j) {
        const int s=2*j, top=col0+cc < P.C ? L : 0;
        const T *f=src+dataCol(P,col0+cc);
        cplx<T> v=mk((T) 0,(T) 0);
        if(s < top) {
          v.x=f[s*P.inRow];
          if(s+1 < top) v.y=f[(s+1)*P.inRow];
          if(P.io64 & 1) v=fromBits(v,sh);
        }
        return v;
      });
    runStages<T,WIDE>(x,0,1,0,P.fz,lt,0,0,tid,nthr,[] {});
    const int Nh=P.N/2, top=P.kc > 0 ? P.kc : Nh+1;
#pragma unroll 2
    for(int idx=tid; idx < (Nh/2+1) << lt; idx += nthr) {
      const int k=idx >> lt, cc=idx & (tile-1), kk=Nh-k;
      if(col0+cc >= P.C) continue;
      cplx<T> *d=dst+col0+cc, F, Fc;
      const cplx<T> zk=x[(spl(P.fz.pos[k],P.fz.lg) << lt)+cc];
      const cplx<T> zm=x[(spl(P.fz.pos[k == 0 ? 0 : kk],P.fz.lg) << lt)+cc];
      realUnpack(zk,zm,ldtw(P.twN+k),F,Fc);
      if(k < top) d[k*P.outRow]=P.conj ? conjg(F) : F;
      if(kk != k && kk < top) d[kk*P.outRow]=P.conj ? conjg(Fc) : Fc;
    }
    return;
  }
  if constexpr(!STAGED) {
    const auto load=[&](int, int cc) {
      const int top=col0+cc < P.C ? L : 0;
      const T *f=src+dataCol(P,col0+cc);
      return [=,&P](int j) {
        const int s=2*j;
        cplx<T> v=mk((T) 0,(T) 0);
        if(s < top) v.x=loadIOr(f+s*P.inRow,P.io64 & 1,sh);
        if(s+1 < top) v.y=loadIOr(f+(s+1)*P.inRow,P.io64 & 1,sh);
        return v;
      };
    };
    runFusedFirst<T,WIDE>(x,0,1,P.fz,lt,tid,nthr,load);
    runFusedMiddle<T,WIDE>(x,0,1,P.fz,lt,false,0,tid,nthr);
    __syncthreads();
    FGB_FUSED_SWITCH(P.fz.radix[P.fz.nst-1],
                     (realLastFwd<T,R_>(P,x,dst,col0,tid,nthr)))
  }
}

template<typename T, int R>
__device__ __forceinline__ void realFirstInv(const OuterPlan<T>& P,
                                             cplx<T> *x, const cplx<T> *src,
                                             int col0, int tid, int nthr)
{
  const FusedFFT& p=P.fz;
  const int lt=log2of(P.tile), Nh=p.n, nblk=Nh/R, total=(nblk+1)/2 << lt;
  const int top=P.kc > 0 ? P.kc : Nh+1;
#pragma unroll 1
  for(int idx=tid; idx < total; idx += nthr) {
    const int i=idx >> lt, cc=idx & (P.tile-1), col=col0+cc;
    const int4 pr=__ldg(p.pairs+i);
    const int b=pr.x, b2=max(pr.y,0), kappa=pr.z;
    const int kappa2=i == 0 ? nblk/2 : nblk-kappa;
    auto get=[&](int k) {
      cplx<T> g=mk((T) 0,(T) 0);
      if(col < P.C && k < top) g=src[(long long) k*P.inRow+col];
      return P.conj ? conjg(g) : g;
    };
    cplx<T> g[R], h[R], u[R], v[R];
#pragma unroll
    for(int r=0; r < R; ++r) {
      g[r]=get(kappa+r*nblk);
      h[r]=get(kappa2+r*nblk);
    }
    if(i != 0) {
#pragma unroll
      for(int r=0; r < R; ++r)
        realPack(g[r],h[R-1-r],ldtw(P.twN+kappa+r*nblk),u[r],v[R-1-r]);
    } else {
      cplx<T> dummy, gN=get(Nh);
      g[0].y=gN.y=(T) 0;
      realPack(g[0],gN,ldtw(P.twN),u[0],dummy);
#pragma unroll
      for(int r=1; r <= R/2; ++r)
        realPack(g[r],g[R-r],ldtw(P.twN+r*nblk),u[r],
                 2*r == R ? dummy : u[R-r]);
#pragma unroll
      for(int r=0; r < (R+1)/2; ++r)
        realPack(h[r],h[R-1-r],ldtw(P.twN+nblk/2+r*nblk),v[r],
                 2*r == R-1 ? dummy : v[R-1-r]);
    }
#pragma unroll
    for(int r=0; r < R; ++r) {
      u[r]=nrm(swapXY(u[r]));
      v[r]=nrm(swapXY(v[r]));
    }
    Codelet<R,1,T>::run(u);
    Codelet<R,1,T>::run(v);
    cplx<T> *xq=x+(spl(b*R,p.lg) << lt)+cc;
    cplx<T> *xr=x+(spl(b2*R,p.lg) << lt)+cc;
#pragma unroll
    for(int r=0; r < R; ++r) xq[r << lt]=u[r];
    if(pr.y >= 0) {
#pragma unroll
      for(int r=0; r < R; ++r) xr[r << lt]=v[r];
    }
  }
}

template<typename T, bool WIDE, bool STAGED>
__device__ __forceinline__ void outerRealBwd(const OuterPlan<T>& P,
                                             unsigned char *smemRaw)
{
  const int tile=P.tile, L=P.L;
  cplx<T> *x=(cplx<T> *) smemRaw;
  const int tid=threadIdx.x, nthr=blockDim.x;
  const int col0=blockIdx.x*tile;
  const int b=blockIdx.z % P.count;
  const long long batch=blockIdx.z/P.count;
  const cplx<T> *src=P.in[b]+batch*P.inBatch;
  T *dst=(T *) P.out[b]+batch*P.outBatch;
  const int lt=log2of(tile);
  const int sh=ioShift<T>(P.ioShift,8+b);
  const auto store=[&](int, int cc) {
    const int top=col0+cc < P.C ? L : 0;
    T *f=dst+dataCol(P,col0+cc);
    return [=,&P](int j, cplx<T> v) {
      const int s=2*j;
      v=v*P.scale;
      if(s < top) storeIOr(f+s*P.outRow,v.x,P.io64 & 2,sh);
      if(s+1 < top) storeIOr(f+(s+1)*P.outRow,v.y,P.io64 & 2,sh);
    };
  };
  if constexpr(STAGED) {
    const int Nh=P.N/2, top=P.kc > 0 ? P.kc : Nh+1;
#pragma unroll 2
    for(int idx=tid; idx < (Nh/2+1) << lt; idx += nthr) {
      const int k=idx >> lt, cc=idx & (tile-1), kk=Nh-k;
      cplx<T> gk=mk((T) 0,(T) 0), gm=gk, Y, Yc;
      if(col0+cc < P.C) {
        const cplx<T> *g=src+col0+cc;
        if(k < top) gk=g[k*P.inRow];
        if(kk < top) gm=g[kk*P.inRow];
      }
      if(P.conj) {
        gk=conjg(gk);
        gm=conjg(gm);
      }
      if(k == 0) gk.y=gm.y=(T) 0;
      realPack(gk,gm,ldtw(P.twN+k),Y,Yc);
      x[(spl(P.fz.pos[k],P.fz.lg) << lt)+cc]=swapXY(Y);
      if(k != 0 && kk != k)
        x[(spl(P.fz.pos[kk],P.fz.lg) << lt)+cc]=swapXY(Yc);
    }
    runStages<T,WIDE>(x,0,0,1,P.fz,lt,0,0,tid,nthr,[] {});
    storeTile(x,P.fz,lt,tid,nthr,store);
    return;
  }
  if constexpr(!STAGED) {
    FGB_FUSED_SWITCH(P.fz.radix[P.fz.nst-1],
                     (realFirstInv<T,R_>(P,x,src,col0,tid,nthr)))
    runFusedMiddle<T,WIDE>(x,0,1,P.fz,lt,true,0,tid,nthr);
    __syncthreads();
    runFusedLast<T,WIDE>(x,0,1,P.fz,lt,tid,nthr,store);
  }
}

template<typename T, bool WIDE, bool STAGED>
__global__ void __launch_bounds__(256,2)
outerRealFwdKernel(const OuterPlan<T> P)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  outerRealFwd<T,WIDE,STAGED>(P,smemRaw);
}

template<typename T, bool WIDE, bool STAGED>
__global__ void __launch_bounds__(256,2)
outerRealBwdKernel(const OuterPlan<T> P)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  outerRealBwd<T,WIDE,STAGED>(P,smemRaw);
}

// ---------------------------------------------------------------------------
// Persistent batched kernel (see kernels.cuh).

template<typename T, template<typename> class Plan>
__device__ __forceinline__ void rebase(Plan<T>& plan, int count, bool relIn,
                                       bool relOut, void *const *inBase,
                                       void *const *outBase)
{
  for(int a=0; a < count; ++a) {
    if(relIn)
      plan.in[a]=(const cplx<T> *) ((char *) inBase[a]+(size_t) plan.in[a]);
    if(relOut)
      plan.out[a]=(cplx<T> *) ((char *) outBase[a]+(size_t) plan.out[a]);
  }
}

// Copy a task's plan from the problem table into shared memory (one copy per
// CTA, read by every thread through broadcast loads) and rebase its pointers
// there: a per-thread copy would live in local memory.
template<typename Plan>
__device__ __forceinline__ Plan& stagePlan(unsigned char *buf, const Plan& src)
{
  static_assert(sizeof(Plan) % sizeof(int) == 0, "plan size");
  int *d=(int *) buf;
  const int *s=(const int *) &src;
  for(int i=threadIdx.x; i < (int) (sizeof(Plan)/sizeof(int)); i += blockDim.x)
    d[i]=s[i];
  return *(Plan *) buf;
}

// CTAs per SM: three in FP32 (512 uneven problems 592 us, with two 722), two in
// FP64, whose registers three would spill (29 problems 215 against 246 us).
template<typename T> constexpr int batchBlocks()
{
  return std::is_same<T,float>::value ? 3 : 2;
}

template<typename T, int K>
__global__ void __launch_bounds__(256,batchBlocks<T>())
batchKernel(const BatchArgs<T> P)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  constexpr size_t planBytes=sizeof(RowPlan<T>) > sizeof(OuterPlan<T>) ?
    sizeof(RowPlan<T>) : sizeof(OuterPlan<T>);
  __shared__ __align__(16) unsigned char planBuf[planBytes];
  __shared__ int slot;
  __shared__ int gaveUp;
  for(;;) {
    if(threadIdx.x == 0) slot=atomicAdd(P.queue,1);
    __syncthreads();
    const int t=slot;
    __syncthreads();
    if(t >= P.ntasks) return;
    const BatchTask tk=P.tasks[t];
    const BatchProblem<T> *B=P.probs+tk.prob;
    if(tk.type == TASK_ROW || tk.type == TASK_COLBWD) {
      if(threadIdx.x == 0) {
        volatile int *d=P.done+2*tk.prob+(tk.type == TASK_ROW ? 0 : 1);
        const int target=tk.type == TASK_ROW ? B->nfwd : B->nrows;
        long long it=0;
        gaveUp=0;
        while(*d < target) {
          if(++it > P.spinLimit) {
            gaveUp=1;
            atomicExch(P.err,1);
            break;
          }
          __nanosleep(100);
        }
        __threadfence();
      }
      __syncthreads();
      if(gaveUp) continue;
    }
    const int rel=B->rel;
    if(tk.type == TASK_SMALL || tk.type == TASK_ROW) {
      RowPlan<T>& R=stagePlan(planBuf,B->row);
      __syncthreads();
      if(threadIdx.x == 0 && tk.type == TASK_SMALL)
        rebase(R,R.A,rel & 1,rel & 2,P.inBase,P.outBase);
      __syncthreads();
      const BuiltinMult<K> mul;
      if(R.direct) {
        // Fused rows, R.rpc of them one after another by teams.
        const int nt=blockDim.x/R.nteam;
        const int team=threadIdx.x/nt, th=threadIdx.x-team*nt;
        const int cs=fusedSpan(R.fz.n,R.fz.lg);
        cplx<T> *x=(cplx<T> *) smemRaw+team*R.A*cs;
        for(int rho=team; rho < R.rpc; rho += R.nteam)
          fusedRow<T,true,false>(R,mul,x,cs,(long long) tk.i*R.rpc+rho,team,
                                 th,nt);
        __syncthreads();
      } else rowConvRow<T,false,BuiltinMult<K>>(R,tk.i,smemRaw,mul);
    } else {
      const bool fwd=tk.type == TASK_COLFWD;
      OuterPlan<T>& O=stagePlan(planBuf,fwd ? B->fwd : B->bwd);
      __syncthreads();
      if(threadIdx.x == 0)
        rebase(O,O.count,fwd && (rel & 4),!fwd && (rel & 8),P.inBase,
               P.outBase);
      __syncthreads();
      if(fwd) outerFwdFused<T,false>(O,tk.i,0,tk.j,smemRaw);
      else outerBwdFused<T,false,true>(O,tk.i,tk.j,smemRaw);
      __syncthreads();
    }
    if(tk.type == TASK_COLFWD || tk.type == TASK_ROW) {
      __threadfence();
      __syncthreads();
      if(threadIdx.x == 0)
        atomicAdd(P.done+2*tk.prob+(tk.type == TASK_COLFWD ? 0 : 1),1);
    }
  }
}

template<typename T, int K>
static cudaError_t launchBatchK(const BatchArgs<T>& P, int grid, int threads,
                                size_t smem, cudaStream_t s)
{
  if(smem > 48*1024) {
    cudaError_t e=cudaFuncSetAttribute(batchKernel<T,K>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int) smem);
    if(e != cudaSuccess) return e;
  }
  batchKernel<T,K><<<grid,threads,smem,s>>>(P);
  return cudaGetLastError();
}

template<typename T>
cudaError_t launchBatch(const BatchArgs<T>& P, int grid, int threads,
                        size_t smem, cudaStream_t s)
{
  switch(multVariant(P.mult,P.A,P.B)) {
    case MULT_BINARY: return launchBatchK<T,MULT_BINARY>(P,grid,threads,smem,s);
    case MULT_REALBINARY:
      return launchBatchK<T,MULT_REALBINARY>(P,grid,threads,smem,s);
    default: return launchBatchK<T,MULT_GENERIC>(P,grid,threads,smem,s);
  }
}

template<typename T, int K>
static int batchBlocksK(int threads, size_t smem)
{
  if(smem > 48*1024)
    cudaFuncSetAttribute(batchKernel<T,K>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize,(int) smem);
  int n=0;
  if(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n,batchKernel<T,K>,threads,
                                                   smem) != cudaSuccess)
    return 1;
  return n > 0 ? n : 1;
}

template<typename T>
int batchBlocksPerSM(int threads, size_t smem, int mult, int A, int B)
{
  switch(multVariant(mult,A,B)) {
    case MULT_BINARY: return batchBlocksK<T,MULT_BINARY>(threads,smem);
    case MULT_REALBINARY: return batchBlocksK<T,MULT_REALBINARY>(threads,smem);
    default: return batchBlocksK<T,MULT_GENERIC>(threads,smem);
  }
}

// ---------------------------------------------------------------------------
// Launchers.

// Shared-memory bytes: FFT ping-pong buffers are padded (sp()); the forward
// outer kernel also stages its L x tile input block in the second buffer.
template<typename T> size_t rowSmem(int L, int m, int A, int B, int rpc)
{
  size_t nbuf=inplaceFFT<T>() ? 1 : 2;
  return sizeof(cplx<T>)*((size_t) (A+B)*rpc*L+
                          nbuf*(size_t) padded(m*A*rpc));
}
template<typename T> size_t outerFwdSmem(int L, int m, int tile)
{
  size_t pm=padded(m*tile);
  return sizeof(cplx<T>)*(pm+std::max(pm,(size_t) L*tile));
}
template<typename T> size_t outerBwdSmem(int L, int m, int tile, int q)
{
  size_t acc=q == 1 ? 0 : (size_t) L*tile;
  return sizeof(cplx<T>)*(acc+2*(size_t) padded(m*tile));
}
template<typename T> size_t outerRealSmem(int L, int Nh, int tile)
{
  return sizeof(cplx<T>)*2*(size_t) padded((Nh+1)*tile);
}

template<typename K>
static cudaError_t setSmem(K kernel, size_t bytes)
{
  if(bytes > 48*1024)
    return cudaFuncSetAttribute(kernel,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int) bytes);
  return cudaSuccess;
}

template<typename T>
cudaError_t launchRow(const RowPlan<T>& P, int threads, long long grid,
                      cudaStream_t s)
{
  switch(multVariant(P.mult,P.A,P.B)) {
    case MULT_BINARY:
      return launchRowWith(P,BuiltinMult<MULT_BINARY>(),threads,grid,s);
    case MULT_REALBINARY:
      return launchRowWith(P,BuiltinMult<MULT_REALBINARY>(),threads,grid,s);
    default:
      return launchRowWith(P,BuiltinMult<MULT_GENERIC>(),threads,grid,s);
  }
}

template<typename T>
cudaError_t launchHermRow(const HermRowPlan<T>& P, int threads,
                          long long grid, cudaStream_t s)
{
  switch(multVariant(P.mult,P.A,P.B)) {
    case MULT_REALBINARY:
      return launchHermRowWith(P,BuiltinMult<MULT_REALBINARY>(),threads,grid,
                               s);
    case MULT_REALJACOBIAN:
      return launchHermRowWith(P,BuiltinMult<MULT_REALJACOBIAN>(),threads,
                               grid,s);
    case MULT_REALJACADJ:
      return launchHermRowWith(P,BuiltinMult<MULT_REALJACADJ>(),threads,grid,
                               s);
    default:
      return launchHermRowWith(P,BuiltinMult<MULT_GENERIC>(),threads,grid,s);
  }
}

template<typename T>
cudaError_t launchOuterFwd(const OuterPlan<T>& P, int threads, cudaStream_t s)
{
  size_t sm=P.fused ? fusedOuterSmem<T>(P.L,P.fz.n,P.fz.lg,P.tile,1) :
    outerFwdSmem<T>(P.L,P.m,P.tile);
  dim3 grid((P.C+P.tile-1)/P.tile,P.q,P.nbatch*P.count);
  auto go=[&](auto kernel) {
    cudaError_t e=setSmem(kernel,sm);
    if(e != cudaSuccess) return e;
    kernel<<<grid,threads,sm,s>>>(P);
    return cudaGetLastError();
  };
  if(P.fused) {
    if constexpr(!std::is_same<T,double>::value)
      if(P.staged) return go(outerFwdStagedKernel<T>);
    if constexpr(std::is_same<T,float>::value)
      if(wideFused(P.fz)) return go(outerFwdFusedKernel16<T>);
    return go(outerFwdFusedKernel<T>);
  }
  return go(outerFwdKernel<T>);
}

template<typename T>
cudaError_t launchOuterBwd(const OuterPlan<T>& P, int threads, cudaStream_t s)
{
  size_t sm=P.fused ? fusedOuterSmem<T>(P.L,P.fz.n,P.fz.lg,P.tile,P.q) :
    outerBwdSmem<T>(P.L,P.m,P.tile,P.q);
  dim3 grid((P.C+P.tile-1)/P.tile,1,P.nbatch*P.count);
  auto go=[&](auto kernel) {
    cudaError_t e=setSmem(kernel,sm);
    if(e != cudaSuccess) return e;
    kernel<<<grid,threads,sm,s>>>(P);
    return cudaGetLastError();
  };
  if(P.fused) {
    if constexpr(!std::is_same<T,double>::value)
      if(P.staged) return go(outerBwdStagedKernel<T>);
    if constexpr(std::is_same<T,float>::value)
      if(wideFused(P.fz)) return go(outerBwdFusedKernel16<T>);
    return go(outerBwdFusedKernel<T>);
  }
  return go(outerBwdKernel<T>);
}

template<typename T>
static cudaError_t launchOuterReal(const OuterPlan<T>& P, bool fwd,
                                   int threads, cudaStream_t s)
{
  const size_t sm=fusedOuterSmem<T>(P.L,P.fz.n,P.fz.lg,P.tile,1);
  dim3 grid((P.C+P.tile-1)/P.tile,1,P.nbatch*P.count);
  auto go=[&](auto kernel) {
    cudaError_t e=setSmem(kernel,sm);
    if(e != cudaSuccess) return e;
    kernel<<<grid,threads,sm,s>>>(P);
    return cudaGetLastError();
  };
  if constexpr(std::is_same<T,float>::value)
    if(!P.staged) {
      if(wideFused(P.fz))
        return fwd ? go(outerRealFwdKernel<T,true,false>) :
          go(outerRealBwdKernel<T,true,false>);
      return fwd ? go(outerRealFwdKernel<T,false,false>) :
        go(outerRealBwdKernel<T,false,false>);
    }
  constexpr bool wide=std::is_same<T,float>::value;
  return fwd ? go(outerRealFwdKernel<T,wide,true>) :
    go(outerRealBwdKernel<T,wide,true>);
}

template<typename T>
cudaError_t launchOuterRealFwd(const OuterPlan<T>& P, int threads,
                               cudaStream_t s)
{
  return launchOuterReal(P,true,threads,s);
}

template<typename T>
cudaError_t launchOuterRealBwd(const OuterPlan<T>& P, int threads,
                               cudaStream_t s)
{
  return launchOuterReal(P,false,threads,s);
}

// build.py compiles this file once per precision (FGB_T) and kernel family
// (FGB_PART), in parallel.
#define FGB_ROWS 1
#define FGB_HERM 2
#define FGB_OUTER 3
#define FGB_BATCH 4
#define FGB_MISC 5
#define FGB_REAL_OUTER 6

#if FGB_PART == FGB_ROWS
template cudaError_t launchRow<FGB_T>(const RowPlan<FGB_T>&,int,long long,
                                      cudaStream_t);
template size_t rowSmem<FGB_T>(int,int,int,int,int);
#elif FGB_PART == FGB_HERM
template cudaError_t launchHermRow<FGB_T>(const HermRowPlan<FGB_T>&,int,
                                          long long,cudaStream_t);
#elif FGB_PART == FGB_OUTER
template cudaError_t launchOuterFwd<FGB_T>(const OuterPlan<FGB_T>&,int,
                                           cudaStream_t);
template cudaError_t launchOuterBwd<FGB_T>(const OuterPlan<FGB_T>&,int,
                                           cudaStream_t);
template size_t outerFwdSmem<FGB_T>(int,int,int);
template size_t outerBwdSmem<FGB_T>(int,int,int,int);
#elif FGB_PART == FGB_REAL_OUTER
template cudaError_t launchOuterRealFwd<FGB_T>(const OuterPlan<FGB_T>&,int,
                                               cudaStream_t);
template cudaError_t launchOuterRealBwd<FGB_T>(const OuterPlan<FGB_T>&,int,
                                               cudaStream_t);
template size_t outerRealSmem<FGB_T>(int,int,int);
#elif FGB_PART == FGB_BATCH
template cudaError_t launchBatch<FGB_T>(const BatchArgs<FGB_T>&,int,int,size_t,
                                        cudaStream_t);
template int batchBlocksPerSM<FGB_T>(int,size_t,int,int,int);
#else
// Bulk copy by the SMs (16-byte vectors, four in flight per thread): between
// page-locked host memory and the device it reads and writes whole lines
// over the host link.
__global__ void __launch_bounds__(256) bulkCopyKernel(CopyArgs P)
{
  const size_t n=P.bytes/16;
  const size_t stride=(size_t) gridDim.x*blockDim.x;
  for(int a=0; a < P.count; ++a) {
    const uint4 *src=(const uint4 *) P.src[a];
    uint4 *dst=(uint4 *) P.dst[a];
    size_t i=blockIdx.x*(size_t) blockDim.x+threadIdx.x;
    for(; i+3*stride < n; i += 4*stride) {
      uint4 v0=src[i], v1=src[i+stride], v2=src[i+2*stride],
        v3=src[i+3*stride];
      dst[i]=v0; dst[i+stride]=v1; dst[i+2*stride]=v2; dst[i+3*stride]=v3;
    }
    for(; i < n; i += stride) dst[i]=src[i];
  }
}

// Float-float range guard (kernels.cuh, FFScaleArgs).  Block b takes the
// largest biased exponent of chunk b % chunks of array b / chunks (integer
// work on the bit patterns, no FP64 pipe; infinities and NaNs ignored)
// into state[a]; the last block to finish (a wrapping counter in state[8])
// turns them into the scales and zeroes the accumulators.  A chunk is
// FGB_SCAN_CHUNK doubles, all of a thread's loads issued before any is
// used, so the whole scan is one round trip to HBM per wave.  Multipliers
// whose every output is one product of two inputs (or one input) take a
// scale per input, and the output scale is the sum (binary, correlation,
// the Jacobian adjoint).  Those whose outputs add products take one scale
// per factor group so that every term scales alike: the Jacobian
// u0 u3 - u1 u2 shares a scale between u0 and u1 and one between u2 and u3
// (the derivatives of psi and of omega), a dot product sum_k u_k u_{K+k}
// one per half.  A caller's functor gets no scaling.
#define FGB_SCAN_CHUNK 2048
__global__ void __launch_bounds__(256) ffScaleKernel(const FFScaleArgs P)
{
  __shared__ bool last;
  __shared__ unsigned wmax[8];
  const long long chunks=(P.n+FGB_SCAN_CHUNK-1)/FGB_SCAN_CHUNK;
  const int a=(int) (blockIdx.x/chunks);
  const long long c0=(blockIdx.x-a*chunks)*FGB_SCAN_CHUNK;
  const long long c1=min(c0+FGB_SCAN_CHUNK,P.n);
  const unsigned long long *src=P.in[a];
  unsigned m=0;
  auto take=[&](unsigned long long b) {
    const unsigned e=(unsigned) ((b >> 52) & 0x7ff);
    if(e != 0x7ff && e > m) m=e;
  };
  if(((size_t) src & 15) == 0) {
    // Pairs of doubles by 16-byte loads (four per thread); an odd last
    // double is read alone.
    const ulonglong2 *v=(const ulonglong2 *) src;
    const long long p0=c0/2, p1=c1/2;
    ulonglong2 b[FGB_SCAN_CHUNK/512];
#pragma unroll
    for(int u=0; u < FGB_SCAN_CHUNK/512; ++u) {
      const long long i=p0+threadIdx.x+u*256;
      b[u]=i < p1 ? __ldg(v+i) : make_ulonglong2(0,0);
    }
#pragma unroll
    for(int u=0; u < FGB_SCAN_CHUNK/512; ++u) {take(b[u].x); take(b[u].y);}
    if((c1 & 1) && threadIdx.x == 0) take(__ldg(src+c1-1));
  } else {
    unsigned long long b[FGB_SCAN_CHUNK/256];
#pragma unroll
    for(int u=0; u < FGB_SCAN_CHUNK/256; ++u) {
      const long long i=c0+threadIdx.x+u*256;
      b[u]=i < c1 ? __ldg(src+i) : 0ull;
    }
#pragma unroll
    for(int u=0; u < FGB_SCAN_CHUNK/256; ++u) take(b[u]);
  }
  // Block maximum (warp reduction, then across the warps): one atomic per
  // block reaches the shared accumulator of its array.
  m=__reduce_max_sync(0xffffffffu,m);
  if((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5]=m;
  __syncthreads();
  if(threadIdx.x < 32) {
    unsigned v=threadIdx.x < (blockDim.x+31)/32 ? wmax[threadIdx.x] : 0u;
    v=__reduce_max_sync(0xffffffffu,v);
    if(threadIdx.x == 0 && v) atomicMax((unsigned *) P.state+a,v);
  }
  __threadfence();
  __syncthreads();
  if(threadIdx.x == 0)
    last=atomicInc((unsigned *) P.state+8,gridDim.x-1) == gridDim.x-1;
  __syncthreads();
  if(!last || threadIdx.x != 0) return;
  __threadfence();
  int sh[FGB_MAXA];
  for(int a=0; a < P.count; ++a) {
    const unsigned m=atomicExch((unsigned *) P.state+a,0u);
    sh[a]=m ? (int) m-1023 : 0;
  }
  int in[FGB_MAXA], out[FGB_MAXA];
  const bool user=P.mult == MULT_USER;
  for(int a=0; a < P.count; ++a) in[a]=user ? 0 : sh[a];
  if(P.mult == MULT_REALJACOBIAN || P.mult == MULT_JACOBIAN) {
    in[0]=in[1]=max(sh[0],sh[1]);
    in[2]=in[3]=max(sh[2],sh[3]);
  } else if(P.mult == MULT_DOT || P.mult == MULT_REALDOT) {
    const int K=P.count/2;
    int t1=sh[0], t2=sh[K];
    for(int k=1; k < K; ++k) {
      t1=max(t1,sh[k]);
      t2=max(t2,sh[K+k]);
    }
    for(int k=0; k < K; ++k) {
      in[k]=t1;
      in[K+k]=t2;
    }
  }
  for(int b=0; b < P.B; ++b) out[b]=in[b];
  switch(P.mult) {
    case MULT_BINARY: case MULT_REALBINARY: case MULT_CORRELATION:
    case MULT_REALJACOBIAN: case MULT_JACOBIAN:
      out[0]=in[0]+in[P.mult == MULT_REALJACOBIAN ||
                     P.mult == MULT_JACOBIAN ? 3 : 1];
      break;
    case MULT_DOT: case MULT_REALDOT:
      out[0]=in[0]+in[P.count/2];
      break;
    case MULT_REALJACADJ:
      for(int b=0; b < 4; ++b) out[b]=in[4]+in[3-b];
      break;
    default:
      break;
  }
  for(int a=0; a < FGB_MAXA; ++a) {
    P.state[16+a]=a < P.count ? in[a] : 0;
    P.state[24+a]=a < P.B ? out[a] : 0;
  }
}

cudaError_t launchFFScale(const FFScaleArgs& P, cudaStream_t s)
{
  if(P.count < 1 || P.count > FGB_MAXA || P.n < 1) return cudaErrorInvalidValue;
  const long long blocks=(P.n+FGB_SCAN_CHUNK-1)/FGB_SCAN_CHUNK*P.count;
  if(blocks > INT_MAX) return cudaErrorInvalidValue;
  ffScaleKernel<<<(unsigned) blocks,256,0,s>>>(P);
  return cudaGetLastError();
}

// The origin shift of the fft0 transforms (fftw++.h:144-228, fftw::Shift):
// the real values of an nx x ny (x nz) array with (i + j) odd (2D: i odd)
// change sign, which moves the Fourier origin to (nx/2, 0) or
// (nx/2, ny/2, 0).
template<typename R>
__global__ void __launch_bounds__(256) originShiftKernel(R *f, long long nx,
                                                         long long ny,
                                                         long long nz)
{
  const long long n=nx*ny*nz;
  const long long stride=(long long) gridDim.x*blockDim.x;
  for(long long e=blockIdx.x*(long long) blockDim.x+threadIdx.x; e < n;
      e += stride) {
    const long long row=e/nz;        // i*ny + j
    const long long i=row/ny, j=row-i*ny;
    const long long parity=nz > 1 ? i+j : i;
    if(parity & 1) f[e]=-f[e];
  }
}

cudaError_t launchOriginShift(void *f, long long nx, long long ny,
                              long long nz, bool f64, cudaStream_t s)
{
  const long long n=nx*ny*nz;
  if(n <= 0) return cudaSuccess;
  const int grid=(int) std::min<long long>((n+255)/256,152*8);
  if(f64) originShiftKernel<double><<<grid,256,0,s>>>((double *) f,nx,ny,nz);
  else originShiftKernel<float><<<grid,256,0,s>>>((float *) f,nx,ny,nz);
  return cudaGetLastError();
}

cudaError_t launchBulkCopy(const CopyArgs& P, cudaStream_t s)
{
  if(P.bytes % 16) return cudaErrorInvalidValue;
  for(int a=0; a < P.count; ++a)
    if(((size_t) P.src[a] | (size_t) P.dst[a]) % 16)
      return cudaErrorInvalidValue;
  if(P.bytes == 0 || P.count == 0) return cudaSuccess;
  bulkCopyKernel<<<152*8,256,0,s>>>(P);
  return cudaGetLastError();
}
#endif

} // namespace fgb
