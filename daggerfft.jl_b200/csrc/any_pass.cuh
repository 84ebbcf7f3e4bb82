// One-tile passes whose sides are not plain complex arrays: the real, r2r,
// truncated and four-step-twiddled sides (IoKind), and Bluestein's algorithm
// in one launch.
//
// A CTA brings its C columns into shared memory, runs the stages there and
// writes the columns back.  The two ends are loops over the tile with the
// side's kind decided once per column, outside the loop, in one out-of-line
// function per precision that every length shares.  (Applying the map to
// each radix input inside the unrolled stages instead repeats the whole kind
// switch once per element of the radix: the kernels were bound by
// instruction fetch, e.g. 50 us for one 512-point pass over 251 x 9800
// ComplexF32 columns whose 59 MB take 9 us of HBM time.)  The ends move
// several elements per thread at once, so their latency overlaps, and map
// lanes to consecutive elements of memory whatever the stages' own mapping
// of threads to butterflies is.
//
// Bluestein (chirp-z) of length N = d.in.chirp_n with FFT length L >= 2N-1
// (d.epi == kEpiChirp): load x_n chirp_n, zero-padded; FFT_L; times the
// filter spectrum d.tw2 and conjugated; FFT_L again; conjugated, times the
// chirp, to memory.  Both FFTs run on the tile in shared memory, so the
// transform costs one read and one write of the N-point columns instead of
// two passes through a scratch of L-point columns.
#pragma once
#include "axis_pass.cuh"

namespace dfft {

// The column of the tile a thread helps to move, and its elements of it, so
// that consecutive lanes touch consecutive memory of that side.  Columns
// side by side (cfast): elements nthreads / C apart.  Unit stride along the
// column (the contiguous axis, and the output of a four-step axis's first
// pass): the column's share of the threads, in order (fft + ifft of one column
// of 5003 ComplexF32 points: 405 us with one group of 32 lanes per column at
// work, 153 so; irfft of 29547 x 25 Float64 44 us, its columns taking turns,
// and 15).
struct TileLanes {
  int c, k, kstep;
};
__device__ __forceinline__ TileLanes tile_lanes(const PassDesc& d, const IoAny& io) {
  const int tid = threadIdx.x, share = blockDim.x / d.C;
  if (d.cfast && io.sk != 1) return TileLanes{tid % d.C, tid / d.C, share};
  return TileLanes{tid / share, tid % share, share};
}

// Elements in flight per thread.  (Eight execute twice the code for nothing
// where a thread has three or four: rfft of 200000 x 81 Float32 258 us, 223
// with four.)
constexpr int kAnyBatch = 4;

// Elements k, k + ks, ... < L of one column: get(k) from memory, times the
// chirp or filter where the side has one (zero beyond the chirp), conjugated
// for an inverse.  PLAIN: no chirp, no filter: their tests and 64-bit indexes
// per element are a good part of the instructions of a short column (columns
// of unit stride, rfft / irfft, us, general against plain: 27 x 200000 Float32
// 60 / 64 and 53 / 54, 81 x 200000 198 / 214 and 183 / 185, 105 x 50000
// Float64 62 / 75 and 58 / 58).
template <typename T, int N, bool PLAIN, class F>
__device__ __forceinline__ void column_in(const IoAny& io, bool inv, long long j, typename cvec<T>::type* col, int k,
                                          int ks, int L, const F& get) {
  typedef typename cvec<T>::type V;
  if constexpr (PLAIN) {
    for (; k < L; k += N * ks) {
      V v[N];
#pragma unroll
      for (int u = 0; u < N; ++u)
        if (k + u * ks < L) v[u] = get(k + u * ks);
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const int e = k + u * ks;
        if (e < L) col[swz<V>(e)] = inv ? cconj(v[u]) : v[u];
      }
    }
    return;
  }
  const V* ch = reinterpret_cast<const V*>(io.chirp);
  const V* mu = reinterpret_cast<const V*>(io.mul);
  const long long tm = io.t_m > 0 ? io.t_m : 1;
  for (; k < L; k += N * ks) {
    V v[N];
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const int e = k + u * ks;
      v[u] = mk<V>((T)0, (T)0);
      if (e < L && (!ch || j + tm * e < io.chirp_n)) v[u] = get(e);
    }
    if (ch || mu) {
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const int e = k + u * ks;
        const long long n = j + tm * e;
        if (e < L && (!ch || n < io.chirp_n)) v[u] = cmul(v[u], ldg_c((ch ? ch : mu) + n));
      }
    }
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const int e = k + u * ks;
      if (inv) v[u].y = -v[u].y;
      if (e < L) col[swz<V>(e)] = v[u];
    }
  }
}

// The way back: conjugation, chirp and factor(k), then put(k, value).  The
// table reads of a batch go out together.
struct NoFactor {};
template <typename T, int N, bool PLAIN, class G, class F>
__device__ __forceinline__ void column_out(const IoAny& io, bool inv, long long j, const typename cvec<T>::type* col,
                                           int k, int ks, int n, const G& factor, const F& put) {
  typedef typename cvec<T>::type V;
  if constexpr (PLAIN) {
    for (; k < n; k += N * ks) {
      V v[N];
#pragma unroll
      for (int u = 0; u < N; ++u) v[u] = col[swz<V>(k + u * ks < n ? k + u * ks : k)];
#pragma unroll
      for (int u = 0; u < N; ++u)
        if (k + u * ks < n) put(k + u * ks, inv ? cconj(v[u]) : v[u]);
    }
    return;
  }
  const V* ch = reinterpret_cast<const V*>(io.chirp);
  const long long tm = io.t_m > 0 ? io.t_m : 1;
  const long long last = io.chirp_n;
  for (; k < n; k += N * ks) {
    V v[N];
    bool ok[N];
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const int e = k + u * ks;
      ok[u] = e < n && (!ch || j + tm * e < last);
      v[u] = mk<V>((T)0, (T)0);
      if (ok[u]) v[u] = col[swz<V>(e)];
      if (inv) v[u].y = -v[u].y;
    }
    if (ch) {
#pragma unroll
      for (int u = 0; u < N; ++u)
        if (ok[u]) v[u] = cmul(v[u], ldg_c(ch + (j + tm * (k + u * ks))));
    }
    if constexpr (!std::is_same<G, NoFactor>::value) {
      V f[N];
#pragma unroll
      for (int u = 0; u < N; ++u) f[u] = factor(ok[u] ? k + u * ks : k);
#pragma unroll
      for (int u = 0; u < N; ++u) v[u] = cmul(v[u], f[u]);
    }
#pragma unroll
    for (int u = 0; u < N; ++u)
      if (ok[u]) put(k + u * ks, v[u]);
  }
}

// The r2r kinds read and write the whole axis: on a four-step sub-axis the
// column starts j rows before its base and its rows are t_i apart.
struct WholeAxis {
  long long b, s;
  int j, m;
  __device__ __forceinline__ int at(int k) const { return j + m * k; }
};
__device__ __forceinline__ WholeAxis whole_axis(const IoAny& io, long long b) {
  if (io.t_m <= 0) return WholeAxis{b, io.sk, 0, 1};
  const long long j = (b % io.t_ia) / io.t_i;
  return WholeAxis{b - j * io.t_i, io.t_i, (int)j, io.t_m};
}

// Do the real pairs of a column with unit stride sit on whole complex elements
// (one access per pair)?  An offset view of a larger real array is only
// aligned to its own type.
template <typename T> __device__ __forceinline__ bool whole_pairs(const T* first) {
  return (reinterpret_cast<uintptr_t>(first) & (2 * sizeof(T) - 1)) == 0;
}

// Base of column q on side io.
__device__ __forceinline__ long long column_base(const IoAny& io, long long I, long long q) {
  const long long qo = I == 1 ? q : q / I;
  return (I == 1 ? 0 : (q - qo * I) * io.si) + io_outer(io, qo);
}

template <typename V>
__device__ __forceinline__ V herm_pair(V A, V Bn, V wk, int k) {
  V B = cconj(Bn);
  if (k == 0) A.y = B.y = 0;
  return cadd(cadd(A, B), cmul_pi(cmul(wk, csub(A, B))));
}

template <typename T>
__device__ __noinline__ void tile_load(const PassDesc& d, typename cvec<T>::type* sm, int L) {
  typedef typename cvec<T>::type V;
  __builtin_assume(__isShared(sm));
  const IoAny& io = d.in;
  const TileLanes ln = tile_lanes(d, io);
  const bool inv = d.inverse != 0;
  const V* pc = reinterpret_cast<const V*>(io.p);
  const T* pr = reinterpret_cast<const T*>(io.p);
  const V* w = reinterpret_cast<const V*>(io.w);
  const long long sk = io.sk;
  const int io_n = io.n;
  const T z = (T)0;
  const int c = ln.c;
  const long long q = (long long)blockIdx.x * d.C + c;
  if (q >= d.Q) return;
  const long long b = column_base(io, d.I, q);
  // index along the whole axis of the column's element 0 (four-step sub-axes)
  const long long j = io.t_m > 0 ? (b % io.t_ia) / io.t_i : 0;
  V* col = sm + (size_t)c * d.ld;
  auto in = [&](auto get) { column_in<T, kAnyBatch, false>(io, inv, j, col, ln.k, ln.kstep, L, get); };
  if (sk == 1 && !io.chirp && !io.mul && io.t_m <= 0) {
    auto plain = [&](auto get) { column_in<T, kAnyBatch, true>(io, inv, 0, col, ln.k, ln.kstep, L, get); };
    const T* p = pr + b;
    const V* x = pc + b;
    if (io.kind == IO_REAL) return plain([=](int k) { return mk<V>(p[k], z); });
    if (io.kind == IO_REAL_PAIR && whole_pairs(p)) return plain([=](int k) { return reinterpret_cast<const V*>(p)[k]; });
    if (io.kind == IO_HERM_FULL)
      return plain([=](int k) {
        const int m = 2 * k <= io_n ? k : io_n - k;
        V v = x[m];
        if (k == 0) v.y = z;  // c2r ignores Im X_0
        return m == k ? v : cconj(v);
      });
    if (io.kind == IO_HERM_PAIR && w)
      return plain([=](int k) { return herm_pair(x[k], x[io_n - k], cconj(ldg_c(w + k)), k); });
  }
  switch (io.kind) {
    case IO_CPLX:
      in([=](int k) { return pc[b + k * sk]; });
      break;
    case IO_REAL_PAIR:
      if (sk == 1 && whole_pairs(pr + b)) in([=](int k) { return *reinterpret_cast<const V*>(pr + b + 2 * (long long)k); });
      else in([=](int k) { return mk<V>(pr[b + (2 * k) * sk], pr[b + (2 * k + 1) * sk]); });
      break;
    case IO_REAL:
      in([=](int k) { return mk<V>(pr[b + k * sk], z); });
      break;
    case IO_HERM_PAIR:
      // even-length C2R pre-pass: Z'_k = (A + B) + i conj(w^k) (A - B),
      // A = X_k, B = conj(X_{n-k}) (Im X_0 and Im X_n ignored); the inverse
      // FFT of Z' (length n) interleaves to 2n * x
      if (w) in([=](int k) { return herm_pair(pc[b + k * sk], pc[b + (io_n - k) * sk], cconj(ldg_c(w + k)), k); });
      else in([=](int k) {  // exp(+2 pi i k / (2n)), computed in the kernel
        double sn, cs;
        sincospi((double)k / (double)io_n, &sn, &cs);
        return herm_pair(pc[b + k * sk], pc[b + (io_n - k) * sk], mk<V>((T)cs, (T)sn), k);
      });
      break;
    case IO_HERM_FULL: {
      const WholeAxis a = whole_axis(io, b);
      in([=](int k) {
        const int kf = a.at(k), m = 2 * kf <= io_n ? kf : io_n - kf;
        V v = pc[a.b + m * a.s];
        if (kf == 0) v.y = z;  // c2r ignores Im X_0
        return m == kf ? v : cconj(v);
      });
      break;
    }
    default: {
      const WholeAxis a = whole_axis(io, b);
#define DFFT_R2R_IN(KIND) \
  case KIND: in([=](int k) { return r2r_load<T, KIND>(pr, a.b, a.s, io_n, w, a.at(k)); }); break;
      switch (io.r2r) {
        DFFT_R2R_IN(K_REDFT10) DFFT_R2R_IN(K_RODFT10) DFFT_R2R_IN(K_REDFT01) DFFT_R2R_IN(K_RODFT01)
        DFFT_R2R_IN(K_REDFT11) DFFT_R2R_IN(K_RODFT11) DFFT_R2R_IN(K_REDFT00) DFFT_R2R_IN(K_RODFT00)
        default: in([=](int k) { return r2r_load<T, K_DHT>(pr, a.b, a.s, io_n, w, a.at(k)); }); break;
      }
#undef DFFT_R2R_IN
    }
  }
}

template <typename T>
__device__ __noinline__ void tile_store(const PassDesc& d, const typename cvec<T>::type* sm, int L) {
  typedef typename cvec<T>::type V;
  __builtin_assume(__isShared(sm));
  const IoAny& io = d.out;
  const TileLanes ln = tile_lanes(d, io);
  const bool inv = d.inverse != 0 || d.epi == kEpiChirp;
  V* pc = reinterpret_cast<V*>(io.p);
  T* pr = reinterpret_cast<T*>(io.p);
  const V* w = reinterpret_cast<const V*>(io.w);
  const long long sk = io.sk;
  const T s = (T)d.scale;
  const int c = ln.c;
  const long long q = (long long)blockIdx.x * d.C + c;
  if (q >= d.Q) return;
  const long long b = column_base(io, d.I, q);
  const long long j = io.t_m > 0 ? (b % io.t_ia) / io.t_i : 0;
  const V* col = sm + (size_t)c * d.ld;
  auto out = [&](int n, auto put) { column_out<T, kAnyBatch, false>(io, inv, j, col, ln.k, ln.kstep, n, NoFactor{}, put); };
  if (d.epi == 1) {
    // R2C post-pass over the half-length spectrum Z (length M = L):
    // X_k = E_k + w^k O_k, E = (Z_k + conj Z_{M-k})/2, O = -i (Z_k - conj Z_{M-k})/2
    const V* w2 = reinterpret_cast<const V*>(d.tw2);
    for (int k = ln.k; k <= L; k += ln.kstep) {
      const V zk = col[swz<V>(k == L ? 0 : k)];
      const V zm = cconj(col[swz<V>(k == 0 ? 0 : L - k)]);
      const V e = cscale(cadd(zk, zm), (T)0.5);
      const V o = cscale(cmul_mi(csub(zk, zm)), (T)0.5);
      pc[b + k * sk] = cscale(cadd(e, cmul(ldg_c(w2 + k), o)), s);
    }
    return;
  }
  if (sk == 1 && !io.chirp && io.t_m <= 0) {
    auto plain = [&](int n, auto put) {
      column_out<T, kAnyBatch, true>(io, inv, 0, col, ln.k, ln.kstep, n, NoFactor{}, put);
    };
    T* p = pr + b;
    V* x = pc + b;
    if (io.kind == IO_REAL) return plain(L, [=](int k, V v) { p[k] = v.x * s; });
    if (io.kind == IO_REAL_PAIR && whole_pairs(p))
      return plain(L, [=](int k, V v) { reinterpret_cast<V*>(p)[k] = cscale(v, s); });
    if (io.kind == IO_TRUNC) return plain(io.n + 1, [=](int k, V v) { x[k] = cscale(v, s); });
  }
  switch (io.kind) {
    case IO_CPLX:
      out(L, [=](int k, V v) { pc[b + k * sk] = cscale(v, s); });
      break;
    case IO_TRUNC: {
      const long long tm = io.t_m > 0 ? io.t_m : 1;
      const int last = io.n;
      out(io.t_m > 0 ? L : last + 1, [=](int k, V v) {
        if (j + tm * k <= last) pc[b + k * sk] = cscale(v, s);
      });
      break;
    }
    case IO_CPLX_TW: {
      const unsigned jj = (unsigned)((b % io.t_ia) / io.t_i);
      const int sh = io.n;
      const V* hi = w + (1 << sh);
      const auto twiddle = [=](int k) {
        const unsigned m = jj * (unsigned)k;
        return split_twiddle(ldg_c(w + (m & ((1u << sh) - 1))), hi + 2 * (m >> sh));
      };
      column_out<T, kAnyBatch, false>(io, inv, j, col, ln.k, ln.kstep, L, twiddle, [=](int k, V v) { pc[b + k * sk] = cscale(v, s); });
      break;
    }
    case IO_REAL_PAIR:
      if (sk == 1 && whole_pairs(pr + b)) out(L, [=](int k, V v) { *reinterpret_cast<V*>(pr + b + 2 * (long long)k) = cscale(v, s); });
      else out(L, [=](int k, V v) {
        pr[b + (2 * k) * sk] = v.x * s;
        pr[b + (2 * k + 1) * sk] = v.y * s;
      });
      break;
    case IO_REAL:
      out(L, [=](int k, V v) { pr[b + k * sk] = v.x * s; });
      break;
    default: {
      const WholeAxis a = whole_axis(io, b);
      const int N = io.n;
#define DFFT_R2R_OUT(KIND) \
  case KIND: out(L, [=](int k, V v) { r2r_store<T, KIND>(pr, a.b, a.s, N, w, a.at(k), v, s); }); break;
      switch (io.r2r) {
        DFFT_R2R_OUT(K_REDFT10) DFFT_R2R_OUT(K_RODFT10) DFFT_R2R_OUT(K_REDFT01) DFFT_R2R_OUT(K_RODFT01)
        DFFT_R2R_OUT(K_REDFT11) DFFT_R2R_OUT(K_RODFT11) DFFT_R2R_OUT(K_REDFT00) DFFT_R2R_OUT(K_RODFT00)
        default: out(L, [=](int k, V v) { r2r_store<T, K_DHT>(pr, a.b, a.s, N, w, a.at(k), v, s); }); break;
      }
#undef DFFT_R2R_OUT
    }
  }
}

// Between the two FFTs of a one-launch Bluestein pass: the filter spectrum,
// and the conjugation that makes the second (forward) FFT an inverse one.
template <typename T>
__device__ __forceinline__ void tile_filter(const PassDesc& d, typename cvec<T>::type* col, int t, int P, int L) {
  typedef typename cvec<T>::type V;
  const V* f = reinterpret_cast<const V*>(d.tw2);
  for (int k = t; k < L; k += P) {
    V v = cmul(col[swz<V>(k)], ldg_c(f + k));
    v.y = -v.y;
    col[swz<V>(k)] = v;
  }
}

// Static radices.  The stages run forward on the tile (conjugation and scale
// belong to the two ends); thread -> (column, butterfly lane) as in
// axis_pass_static.  CHIRP: Bluestein.  (The second copy of the stages is
// spelled out: a loop over the two FFTs around one copy, entered once by the
// other sides, spilled 300 to 900 bytes a thread: 35 us for 1024 columns of
// 1024 ComplexF32 points.  One CTA per SM in the launch bounds: without it
// the double-precision kernels are held to 64 registers.)
template <typename T, int LB, bool CHIRP, int L, int P, int... Rs>
__global__ void __launch_bounds__(LB, 1) axis_pass_any(const __grid_constant__ PassDesc d) {
  typedef typename cvec<T>::type V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* sm = reinterpret_cast<V*>(smem_raw);
  const int tid = threadIdx.x;
  const int c = d.cfast ? tid % d.C : tid / P;
  const int t = d.cfast ? tid / d.C : tid % P;
  const PadCol<V> col{sm + (size_t)c * d.ld};
  const GlobalTw<V> tw{reinterpret_cast<const V*>(d.tw)};
  pass_entry();
  tile_load<T>(d, sm, L);
  __syncthreads();
  static_stages<T, L, P, 1, 0, 1, 1, 1, 0, PadCol<V>, PadCol<V>, PadCol<V>, GlobalTw<V>, Rs...>(d, t, col, col, col,
                                                                                             tw, 0, 0, true);
  if constexpr (CHIRP) {
    tile_filter<T>(d, col.p, t, P, L);
    __syncthreads();
    static_stages<T, L, P, 1, 0, 1, 1, 1, 0, PadCol<V>, PadCol<V>, PadCol<V>, GlobalTw<V>, Rs...>(d, t, col, col, col,
                                                                                               tw, 0, 0, true);
  }
  tile_store<T>(d, sm, L);
}

// Radices read at run time (lengths without a static plan).
template <typename T, int R, int EMAX, bool CTW>
__device__ __noinline__ void dyn_stage(const PassDesc& d, int s, int t, typename cvec<T>::type* col) {
  typedef typename cvec<T>::type V;
  __builtin_assume(__isShared(col));
  const PadCol<V> c{col};
  const int ns = d.ns[s], ts = d.tws[s];
  if constexpr (CTW) {
    const ComputedTw<V> g{d.L};
    stage_body<T, R, EMAX / R, 1, 0, 1, false>(d, d.L, d.P, ns, ts, 0, s == 0, s == d.nst - 1, t, c, c, g, 0, 0, true);
  } else {
    const GlobalTw<V> g{reinterpret_cast<const V*>(d.tw)};
    stage_body<T, R, EMAX / R, 1, 0, 1, false>(d, d.L, d.P, ns, ts, 0, s == 0, s == d.nst - 1, t, c, c, g, 0, 0, true);
  }
}

// CTW: twiddles computed in the kernel instead of read from d.tw (no table).
template <typename T, int EMAX, bool CTW = false>
__global__ void __launch_bounds__(1024) axis_pass_dynamic(const __grid_constant__ PassDesc d) {
  typedef typename cvec<T>::type V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* sm = reinterpret_cast<V*>(smem_raw);
  const int tid = threadIdx.x, P = d.P, L = d.L;
  const int c = d.cfast ? tid % d.C : tid / P;
  const int t = d.cfast ? tid / d.C : tid % P;
  V* col = sm + (size_t)c * d.ld;
  pass_entry();
  tile_load<T>(d, sm, L);
  __syncthreads();
  for (int half = 0;; ++half) {
    for (int s = 0; s < d.nst; ++s) {
      switch (d.radix[s]) {
        case 1: dyn_stage<T, 1, EMAX, CTW>(d, s, t, col); break;
        case 2: dyn_stage<T, 2, EMAX, CTW>(d, s, t, col); break;
        case 3: dyn_stage<T, 3, EMAX, CTW>(d, s, t, col); break;
        case 4: dyn_stage<T, 4, EMAX, CTW>(d, s, t, col); break;
        case 5: dyn_stage<T, 5, EMAX, CTW>(d, s, t, col); break;
        case 7: dyn_stage<T, 7, EMAX, CTW>(d, s, t, col); break;
        case 8: dyn_stage<T, 8, EMAX, CTW>(d, s, t, col); break;
        case 11: dyn_stage<T, 11, EMAX, CTW>(d, s, t, col); break;
        case 13: dyn_stage<T, 13, EMAX, CTW>(d, s, t, col); break;
        case 16: dyn_stage<T, 16, EMAX, CTW>(d, s, t, col); break;
        default: break;
      }
    }
    if (half || d.epi != kEpiChirp) break;
    tile_filter<T>(d, col, t, P, L);
    __syncthreads();
  }
  tile_store<T>(d, sm, L);
}

}  // namespace dfft
