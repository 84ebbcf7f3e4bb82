// One batched 1-D transform pass along one axis of a column-major array.
//
// Data model.  A pass transforms Q independent "columns" of FFT length L.
// Column q is split as (qi, qo) = (q % I, q / I); element k of column q of a
// side (input or output) sits at  p[qi*si + qo*so + k*sk]  of that side.  One
// kernel therefore serves the contiguous axis (I = 1: a column is a whole
// pencil) and the strided axes (I = product of the faster dims: consecutive
// columns are adjacent in memory, so the strided loads coalesce).
//
// Work split.  A CTA owns C consecutive columns and runs P threads per column.
// With cfast the column index sits in the fastest thread bits (strided axes:
// a warp reads adjacent elements of one row of the tile); otherwise the
// butterfly index does (contiguous axis: a warp reads one pencil).
//
// Algorithm.  Stockham autosort FFT, stages s = 0..nst-1 with radix R_s and
// Ns = R_0*...*R_{s-1}.  Butterfly j of stage s reads k = j + r*(L/R_s),
// multiplies by w_{Ns*R}^{(j mod Ns)*r}, runs a radix-R_s codelet and writes
// k' = (j - j mod Ns)*R_s + j mod Ns + r*Ns.  The first stage reads straight
// from global memory and the last stage writes straight to global memory (both
// index patterns are unit-stride in j), so a pass costs one read and one write
// of HBM; the nst-1 intermediate exchanges go through shared memory.
//
// The inverse transform runs the forward kernel on conjugated data
// (IDFT(x) = conj(DFT(conj(x)))), with the 1/L scale folded into the store.
//
// axis_pass_static<T, LB, L, P, R...> serves plain complex sides; the other
// sides (real, r2r, Bluestein) and run-time radices run on the same stage
// body in any_pass.cuh.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>
#include "codelets.cuh"

namespace dfft {

constexpr int kMaxStages = 16;

// How a side of a pass maps FFT elements to memory.
enum IoKind : int {
  IO_CPLX = 0,       // complex elements
  IO_REAL_PAIR = 1,  // real pairs: z_m <-> (x_{2m}, x_{2m+1})
  IO_REAL = 2,       // load (x_k, 0) / store Re z_k
  IO_HERM_PAIR = 3,  // load only: even-length C2R pre-pass (real length 2n)
  IO_HERM_FULL = 4,  // load only: odd-length C2R, Hermitian mirror
  IO_TRUNC = 5,      // store only: complex, keep k <= n
  IO_R2R = 6,        // FFTW r2r kind `r2r` on real data of extent n
  IO_CPLX_TW = 7     // store only: complex times W_N^(j k), j = (b mod t_ia) / t_i (the twiddle
                     // between the two passes of a four-step axis of N points); w holds the
                     // split table of W_N, n the log2 of its split
};
// Split twiddle table of W_N with split S (a power of two up to kTwSplit):
// W_N^m - 1 for m < S, then for S m < N pairs of W_N^(S m) rounded and the
// rest of it (exact value minus the rounded one, rounded).
constexpr int kTwSplit = 1024;

// FFTW r2r kind numbers (fftw_r2r_kind).
enum : int { K_DHT = 2, K_REDFT00 = 3, K_REDFT01 = 4, K_REDFT10 = 5, K_REDFT11 = 6,
             K_RODFT00 = 7, K_RODFT01 = 8, K_RODFT10 = 9, K_RODFT11 = 10 };

struct IoAny {
  void* p;
  long long si, so, sk;
  int kind;          // IoKind
  int r2r;           // FFTW kind for IO_R2R
  int n;             // logical extent (see the kinds)
  const void* w;     // twiddle table for the kinds that need one
  // Bluestein wrapping (chirp-z) of any kind: element k < chirp_n is
  // multiplied by chirp[k] after loading / before storing, elements
  // k >= chirp_n load as zero and are not stored; mul[k] multiplies a load.
  const void* chirp;
  const void* mul;
  int chirp_n;
  // Two-level column split of the outer index (four-step input): with
  // o1 > 0 the column base is (qo mod o1) * so + (qo / o1) * so2.
  long long o1, so2;
  // Sub-axis of a four-step pair: the column at base b holds elements
  // j + t_m * k of the whole axis, j = (b mod t_ia) / t_i.  With t_m > 0 the
  // chirp and mul tables are indexed by j + t_m * k (Bluestein around a
  // four-step pair).
  long long t_i, t_ia;
  int t_m;
};

// Column base of side `io` for the outer column index qo.
__host__ __device__ __forceinline__ long long io_outer(const IoAny& io, long long qo) {
  return io.o1 > 0 ? (qo % io.o1) * io.so + (qo / io.o1) * io.so2 : qo * io.so;
}

struct PassDesc {
  int L;                    // transform length of this pass
  int nst;                  // number of Stockham stages (dynamic kernel only)
  int radix[kMaxStages];
  int ns[kMaxStages];
  int tws[kMaxStages];
  int P;                    // threads per column
  int C;                    // columns per CTA
  int ld;                   // shared-memory elements reserved per column
  int inverse;              // 1: conjugate on load and on store
  int cfast;                // thread -> (column, butterfly) mapping
  int epi;                  // 1: R2C half-length post-pass on the way out; kEpiChirp: Bluestein
  long long Q;              // number of columns
  long long I;              // column split q -> (q % I, q / I)
  double scale;             // multiplier applied at the store
  const void* tw;           // L entries exp(-2 pi i m / L)
  const void* tw2;          // epi 1: L+1 entries exp(-2 pi i m / (2L)); kEpiChirp: filter spectrum, L entries
  IoAny in, out;
};

constexpr int kEpiChirp = 2;  // PassDesc::epi of a one-launch Bluestein pass

// Bank-conflict swizzle for the shared-memory exchange: one pad element per
// 128 bytes of complex data.
template <typename V> __device__ __forceinline__ int swz(int k) {
  return sizeof(V) == 8 ? k + (k >> 4) : k + (k >> 3);
}

template <typename V> __device__ __forceinline__ V ldg_c(const V* p) { return __ldg(p); }

// W_N^m from its split table: lo = W_N^(m mod S) - 1, hi the pair of m / S.
// H (1 + lo) as H + (rest + H lo): |lo| <= 1/32, so only the last addition
// rounds at full size, as in a table of all N entries: at most 0.63 units of
// the last place, against 1.4 for the product of two rounded entries (relative
// error of a 2^18-point Float32 rfft 1.50e-7 and 1.53e-7, of 2^20 ComplexF32
// points 1.67e-7 and 1.69e-7; one fft of 2^20 points 14.1 us either way, of
// 2^18 11.4 against 10.4, of 45000 6.4 against 6.0).
template <typename V> __device__ __forceinline__ V split_twiddle(V lo, const V* hi) {
  V h, r;
  if constexpr (sizeof(V) == 8) {
    const float4 p = __ldg(reinterpret_cast<const float4*>(hi));
    h = mk<V>(p.x, p.y);
    r = mk<V>(p.z, p.w);
  } else {
    h = ldg_c(hi);
    r = ldg_c(hi + 1);
  }
  return cadd(h, cadd(r, cmul(h, lo)));
}

// Every pass kernel but mixed_pass (launched in the ordinary way) calls this
// before its first access to the arrays, from all threads: it waits until the kernels before it in the stream are
// complete and visible, then lets the next one be scheduled.  The passes of
// a transform are launched with programmatic stream serialization, so the
// next pass's launch and set-up overlap this one's tail instead of following
// it (a kernel launched without that attribute does not wait here).  Tables
// that never change may be read earlier; arrays another pass writes are read
// with plain loads, not through the read-only path, since that pass may still
// be running when this kernel starts.
__device__ __forceinline__ void pass_entry() {
  asm volatile("griddepcontrol.wait;\n griddepcontrol.launch_dependents;" ::: "memory");
}

// ---------------------------------------------------------------------------
// Element access for every side kind.  The r2r maps (FFTW kinds, all
// unnormalised) express each kind as one complex FFT:
//   kind      FFT length  input map                            output
//   REDFT10   N           v_k = x_{2k} | x_{2N-2k-1}            Y_k = 2 Re(e^{-i pi k/2N} V_k)
//   RODFT10   N           as REDFT10 on (-1)^n x_n              Y_{N-1-k} = that value
//   REDFT01   N, inverse  V_n = e^{i pi n/2N}(x_n - i x_{N-n})  y_{2m} | y_{2N-2m-1} = Re v_m
//   RODFT01   N, inverse  as REDFT01 on x reversed              times (-1)^k
//   REDFT11   2N          x_n e^{-i pi n/2N}, zero-padded       Y_k = 2 Re(e^{-i pi (2k+1)/4N} X_k)
//   RODFT11   2N          as REDFT11 on x reversed              times (-1)^k
//   REDFT00   2(N-1)      even extension                        Y_k = Re X_k
//   RODFT00   2(N+1)      odd extension [0, x, 0, -rev(x)]      Y_k = -Im X_{k+1}
//   DHT       N           x_n                                   Y_k = Re X_k - Im X_k
// ---------------------------------------------------------------------------

// One FFTW r2r kind's load map (element k of the FFT input, from real data
// of extent N at p[b + n*sk]) and store map (FFT output element k, scaled
// by s, into the real result); w is the kind's twiddle table.
template <typename T, int KIND>
__device__ __forceinline__ typename cvec<T>::type r2r_load(const T* p, long long b, long long sk, int N,
                                                         const typename cvec<T>::type* w, int k) {
  typedef typename cvec<T>::type V;
  const T z = (T)0;
  if constexpr (KIND == K_REDFT10 || KIND == K_RODFT10) {
    const int n = (2 * k < N) ? 2 * k : 2 * N - 2 * k - 1;
    T v = p[b + n * sk];
    if (KIND == K_RODFT10 && (n & 1)) v = -v;
    return mk<V>(v, z);
  } else if constexpr (KIND == K_REDFT01 || KIND == K_RODFT01) {
    const bool rev = (KIND == K_RODFT01);
    const T a = p[b + (rev ? N - 1 - k : k) * sk];
    const T c = (k == 0) ? z : p[b + (rev ? k - 1 : N - k) * sk];
    return cmul(ldg_c(w + k), mk<V>(a, -c));
  } else if constexpr (KIND == K_REDFT11 || KIND == K_RODFT11) {
    if (k >= N) return mk<V>(z, z);
    const T a = p[b + (KIND == K_RODFT11 ? N - 1 - k : k) * sk];
    const V t = ldg_c(w + k);
    return mk<V>(a * t.x, a * t.y);
  } else if constexpr (KIND == K_REDFT00) {
    const int n = (k < N) ? k : 2 * (N - 1) - k;
    return mk<V>(p[b + n * sk], z);
  } else if constexpr (KIND == K_RODFT00) {
    if (k == 0 || k == N + 1) return mk<V>(z, z);
    if (k <= N) return mk<V>(p[b + (k - 1) * sk], z);
    return mk<V>(-p[b + (2 * N + 1 - k) * sk], z);
  } else {  // K_DHT
    return mk<V>(p[b + k * sk], z);
  }
}

template <typename T, int KIND>
__device__ __forceinline__ void r2r_store(T* p, long long b, long long sk, int N, const typename cvec<T>::type* w,
                                          int k, typename cvec<T>::type v, T s) {
  typedef typename cvec<T>::type V;
  if constexpr (KIND == K_REDFT10 || KIND == K_RODFT10) {
    const V t = ldg_c(w + k);
    p[b + (KIND == K_RODFT10 ? N - 1 - k : k) * sk] = (T)2 * (v.x * t.x - v.y * t.y) * s;
  } else if constexpr (KIND == K_REDFT01 || KIND == K_RODFT01) {
    const int n = (2 * k < N) ? 2 * k : 2 * N - 2 * k - 1;
    T y = v.x * s;
    if (KIND == K_RODFT01 && (n & 1)) y = -y;
    p[b + n * sk] = y;
  } else if constexpr (KIND == K_REDFT11 || KIND == K_RODFT11) {
    if (k >= N) return;
    const V t = ldg_c(w + k);
    T y = (T)2 * (v.x * t.x - v.y * t.y) * s;
    if (KIND == K_RODFT11 && (k & 1)) y = -y;
    p[b + k * sk] = y;
  } else if constexpr (KIND == K_REDFT00) {
    if (k < N) p[b + k * sk] = v.x * s;
  } else if constexpr (KIND == K_RODFT00) {
    if (k >= 1 && k <= N) p[b + (k - 1) * sk] = -v.y * s;
  } else {  // K_DHT
    p[b + k * sk] = (v.x - v.y) * s;
  }
}

// ---------------------------------------------------------------------------
// Stage body.
// ---------------------------------------------------------------------------

// Shared-memory view of one column.  PadCol: column-major with one pad
// element per 128 bytes (direct-load kernels); StrideCol: the [k][c] layout a
// TMA tile box lands in (c fastest), conflict-free for the cfast mapping.
// Every view is addressed as (base, off): element base + off, where the
// stage passes its per-butterfly index as base and r * stride (a constant
// once the radix loop is unrolled) as off.  Views whose layout is a bitwise
// map use it to split the address into a per-butterfly part and a constant.
template <typename V> struct PadCol {
  V* p;
  __device__ __forceinline__ V ld(int b, int off) const { return p[swz<V>(b + off)]; }
  __device__ __forceinline__ void st(int b, int off, V v) const { p[swz<V>(b + off)] = v; }
};
template <typename V> struct StrideCol {
  V* p;
  int s;
  __device__ __forceinline__ V ld(int b, int off) const { return p[(b + off) * s]; }
  __device__ __forceinline__ void st(int b, int off, V v) const { p[(b + off) * s] = v; }
};
// StrideCol with a compile-time stride: every tile offset becomes an
// immediate of the shared-memory instruction instead of a live register.
template <typename V, int S> struct StrideColC {
  V* p;
  __device__ __forceinline__ V ld(int b, int off) const { return p[(b + off) * S]; }
  __device__ __forceinline__ void st(int b, int off, V v) const { p[(b + off) * S] = v; }
};

// Twiddle sources.  GlobalTw reads w_L^{jm*r*ts} from the L-entry table;
// StageTw reads a stage-major table laid out [stage][jm][r-1] (entry
// Ns - R_0 + jm*(R-1) + r-1 holds exp(-2 pi i jm r / (Ns R))), which the
// persistent kernels keep in shared memory: lanes with consecutive jm read
// consecutive (R-1)-strided entries, conflict-free.
template <typename V> struct GlobalTw {
  const V* p;
  __device__ __forceinline__ V w(int off, int jm, int r, int R, int ts) const {
    return ldg_c(p + jm * r * ts);
  }
};
template <typename V> struct StageTw {
  const V* p;
  __device__ __forceinline__ V w(int off, int jm, int r, int R, int ts) const {
    return p[off + jm * (R - 1) + r - 1];
  }
};
// The same table with the last stage's entries pre-multiplied by the
// inverse's 1/L as rounded to T (exact for power-of-two L): the last stage of an inverse
// then scales only its r = 0 inputs, and the DFT carries the scale to every
// output (linearity), instead of scaling every output.
template <typename V> struct StageTwScaledLast : StageTw<V> {};
template <class TW> struct scaled_last_tw { static constexpr bool value = false; };
template <typename V> struct scaled_last_tw<StageTwScaledLast<V>> { static constexpr bool value = true; };
// Twiddles computed in the kernel (no table in memory): exp(-2 pi i jm r ts / L)
// with the CUDA math library's sincospi in double precision.
template <typename V> struct ComputedTw {
  int L;
  __device__ __forceinline__ V w(int off, int jm, int r, int R, int ts) const {
    typedef typename scalar_of<V>::type S;
    const long long m = ((long long)jm * r * ts) % L;
    double sn, cs;
    sincospi(2.0 * (double)m / (double)L, &sn, &cs);
    return mk<V>((S)cs, (S)-sn);
  }
};

// The same stage-major table read from global memory through L1.
template <typename V> struct StageTwG {
  const V* p;
  __device__ __forceinline__ V w(int off, int jm, int r, int R, int ts) const {
    return ldg_c(p + off + jm * (R - 1) + r - 1);
  }
};

// Barrier between the stages: the whole CTA (BAR = 0) or named barrier 1
// over the BAR threads that run the stages (the other warps of the CTA do
// something else, e.g. feed the tile pipeline).
// The lanes of a warp may come to it apart: after a wait each lane polls for
// itself, a loop whose last round is not every lane's, stores behind a
// condition.  (bar.sync is the aligned form: a warp that reaches it in two
// parts hangs, and the compiler may well send the lanes of a loop's last
// round past it on a copy of their own, for instance where only they can meet
// the tid == 0 test that follows.)
template <int BAR> __device__ __forceinline__ void stage_sync() {
  if constexpr (BAR == 0) {
    __syncthreads();
  } else {
    __syncwarp();
    asm volatile("barrier.cta.sync 1, %0;" ::"n"(BAR) : "memory");
  }
}
// The aligned form, for code without a branch since the last stage_sync: the
// stages in which every thread has the same number of butterflies.
template <int BAR> __device__ __forceinline__ void stage_sync_converged() {
  if constexpr (BAR == 0) __syncthreads();
  else asm volatile("bar.sync 1, %0;" ::"n"(BAR) : "memory");
}

// BMAX: upper bound on butterflies per thread; in the static kernels it is
// exactly ceil((L/R)/P), in the dynamic kernel EMAX/R.
// SMEM_IO: 0 = the first stage reads and the last stage writes global
// memory; 1 = both go through shared memory (pipelined kernels); 2 = the
// first stage reads shared memory, the last stage writes whole pencils to
// global memory (unit stride); 3 = the same with the output's row stride.
// CIN/COUT: the shared-memory views the stage reads and writes (they differ
// when a stage moves a tile between a dense TMA buffer and a padded one).
// toff: offset of this stage in a StageTw table (Ns - R_0).
// CLAMP (static radices on a tile in shared memory): a thread past the last
// butterfly computes that one again and stores nothing.  Butterflies behind a
// condition, even one that always holds (t < P is not visible to the compiler
// when the mapping is chosen at run time), spilled in the kernels that loop
// over tiles: the 12 x 16 slab pass 300 bytes a thread, and 2^20 ComplexF32
// points 39 instead of 30 us through the pipelined pass.  The kernels that
// load and store memory directly hold fewer registers with the condition.
template <typename T, int R, int BMAX, int SMEM_IO, int BAR, int DIR, bool CLAMP, class CIN, class COUT, class TW>
__device__ __forceinline__ void stage_body(const PassDesc& d, int L, int P, int Ns, int ts, int toff,
                                           bool first, bool last, int t, const CIN& cin,
                                           const COUT& cout, const TW& tw, long long ib,
                                           long long ob, bool cv) {
  typedef typename cvec<T>::type V;
  const int Lr = L / R;
  // direction: at run time (DIR 0), or compiled in (1 forward: no
  // conjugation, unit scale; 2 inverse)
  const bool inv = DIR == 0 ? d.inverse != 0 : DIR == 2;
  // scale folded into the last stage's twiddles (inverse kernels whose
  // table says so): only the r = 0 inputs are scaled here
  const bool fold = scaled_last_tw<TW>::value && DIR == 2 && last && !first;
  const T scale = DIR == 1 || fold ? (T)1 : (T)d.scale;
  const bool to_global = SMEM_IO != 1 && last;
  const bool from_global = SMEM_IO == 0 && first;
  const bool exact = CLAMP && BMAX * P == Lr;
  V v[BMAX][R];
#pragma unroll
  for (int b = 0; b < BMAX; ++b) {
    const int j = CLAMP && !exact ? min(t + b * P, Lr - 1) : t + b * P;
    if (CLAMP || j < Lr) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int k = j + r * Lr;
        if (from_global) {
          V x;
          if (!cv) x = mk<V>((T)0, (T)0);
          else x = reinterpret_cast<const V*>(d.in.p)[ib + k * d.in.sk];
          if (inv) x.y = -x.y;
          v[b][r] = x;
        } else {
          V x = cin.ld(j, r * Lr);
          if (SMEM_IO != 0 && first && inv) x.y = -x.y;
          v[b][r] = x;
        }
      }
    }
  }
  if (!from_global) {
    if (exact) stage_sync_converged<BAR>();
    else stage_sync<BAR>();
  }
#pragma unroll
  for (int b = 0; b < BMAX; ++b) {
    const int j = CLAMP && !exact ? min(t + b * P, Lr - 1) : t + b * P;
    const bool mine = exact || t + b * P < Lr;
    if (CLAMP || j < Lr) {
      const int jm = j % Ns;
      if (!first) {
#pragma unroll
        for (int r = 1; r < R; ++r) v[b][r] = cmul(v[b][r], tw.w(toff, jm, r, R, ts));
        if (fold) v[b][0] = cscale(v[b][0], (T)d.scale);
      }
      Dft<R>::run(v[b]);
      const int o0 = (j - jm) * R + jm;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int k = o0 + r * Ns;
        if (to_global) {
          if (cv && mine) {
            V y = v[b][r];
            if (inv) y.y = -y.y;
            // SMEM_IO 2 (the fused slab pass) stores whole pencils: unit stride;
            // SMEM_IO 3 (the cp.async strided pass) rows d.out.sk apart
            reinterpret_cast<V*>(d.out.p)[ob + (SMEM_IO == 2 ? k : k * d.out.sk)] = cscale(y, scale);
          }
        } else if (SMEM_IO == 1 && last) {
          V y = v[b][r];
          if (inv) y.y = -y.y;
          if (mine) cout.st(o0, r * Ns, cscale(y, scale));
        } else {
          if (mine) cout.st(o0, r * Ns, v[b][r]);
        }
      }
    }
  }
  if (!to_global) {
    if (exact) stage_sync_converged<BAR>();
    else stage_sync<BAR>();
  }
}

// Shared prologue: thread -> (column, butterfly lane), column base offsets.
struct ColCtx {
  int c, t;
  bool cv;
  long long ib, ob;
};

__device__ __forceinline__ ColCtx col_ctx(const PassDesc& d, int P) {
  ColCtx x;
  const int tid = threadIdx.x;
  if (d.cfast) { x.c = tid % d.C; x.t = tid / d.C; }
  else { x.t = tid % P; x.c = tid / P; }
  const long long q = (long long)blockIdx.x * d.C + x.c;
  x.cv = q < d.Q;
  const long long qi = x.cv ? q % d.I : 0;
  const long long qo = x.cv ? q / d.I : 0;
  x.ib = qi * d.in.si + io_outer(d.in, qo);
  x.ob = qi * d.out.si + io_outer(d.out, qo);
  return x;
}

// ---------------------------------------------------------------------------
// Static-plan kernel.
// ---------------------------------------------------------------------------

// Compile-time stage sequence.  The first stage reads CFIRST, the last
// stage writes CLAST, every other access goes through CMID.
template <typename T, int L, int P, int SMEM_IO, int BAR, int DIR, int NS, int R0, int S, class CFIRST,
          class CMID, class CLAST, class TW, int R, int... Rest>
__device__ __forceinline__ void static_stages(const PassDesc& d, int t, const CFIRST& cf,
                                              const CMID& cm, const CLAST& cl, const TW& tw,
                                              long long ib, long long ob, bool cv) {
  constexpr int Lr = L / R;
  constexpr int BM = (Lr + P - 1) / P;
  constexpr int TS = L / (NS * R);
  constexpr bool FIRST = (S == 0);
  constexpr bool LAST = (sizeof...(Rest) == 0);
  constexpr int R0_ = FIRST ? R : R0;
  if constexpr (FIRST && LAST) {
    stage_body<T, R, BM, SMEM_IO, BAR, DIR, SMEM_IO != 0>(d, L, P, NS, TS, NS - R0_, true, true, t, cf, cl, tw, ib, ob, cv);
  } else if constexpr (FIRST) {
    stage_body<T, R, BM, SMEM_IO, BAR, DIR, SMEM_IO != 0>(d, L, P, NS, TS, NS - R0_, true, false, t, cf, cm, tw, ib, ob, cv);
  } else if constexpr (LAST) {
    stage_body<T, R, BM, SMEM_IO, BAR, DIR, SMEM_IO != 0>(d, L, P, NS, TS, NS - R0_, false, true, t, cm, cl, tw, ib, ob, cv);
  } else {
    stage_body<T, R, BM, SMEM_IO, BAR, DIR, SMEM_IO != 0>(d, L, P, NS, TS, NS - R0_, false, false, t, cm, cm, tw, ib, ob, cv);
  }
  if constexpr (sizeof...(Rest) > 0)
    static_stages<T, L, P, SMEM_IO, BAR, DIR, NS * R, R0_, S + 1, CFIRST, CMID, CLAST, TW, Rest...>(
        d, t, cf, cm, cl, tw, ib, ob, cv);
}

template <typename T, int LB, int L, int P, int... Rs>
__global__ void __launch_bounds__(LB) axis_pass_static(const PassDesc d) {
  typedef typename cvec<T>::type V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* sm = reinterpret_cast<V*>(smem_raw);
  const ColCtx x = col_ctx(d, P);
  pass_entry();
  const PadCol<V> col{sm + x.c * d.ld};
  const GlobalTw<V> tw{reinterpret_cast<const V*>(d.tw)};
  static_stages<T, L, P, 0, 0, 0, 1, 1, 0, PadCol<V>, PadCol<V>, PadCol<V>, GlobalTw<V>, Rs...>(
      d, x.t, col, col, col, tw, x.ib, x.ob, x.cv);
}

}  // namespace dfft
