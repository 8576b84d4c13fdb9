// Band-pruned 1-D transforms of the w planes along either grid axis, FP32 and
// FP64, any length 2^a 3^b 5^c whose transform fits in shared memory.
//
//   X[k] = sum_j x[j] exp(+-2 pi i j k / L), unnormalised (+: CUFFT_INVERSE)
//
// in place, for x[j] = 0 outside a window of `ni` inputs and only the window of
// `no` outputs wanted (both periodic): nothing else is read or written.  Before
// the inverse transform the data occupies the band of grid rows and columns that
// the visibilities reach, after it the image is kept; before the forward one
// the image is non-zero, after it the band is read.
//
// A CTA transforms NB neighbouring columns (rows) in place in shared memory by
// decimation-in-frequency passes of radix 2 to 16, one butterfly per thread at a
// time: the first pass loads from the grid, the last one stores to it at the
// digit-reversed index, taking its butterflies in output order so that neighbouring
// threads store neighbouring elements.
//
// Columns: what costs is the length of the contiguous pieces, NB elements of one
// grid row.  With ni <= L / 2 a column needs shared memory for L / 2 points
// only: the even and the odd outputs are two transforms of length n = L / 2,
//   X[2 k' + s] = sum_j (x[j] e^{+-2 pi i j s / L}) e^{+-2 pi i j k' / n},
// whose inputs do not overlap modulo n (H = 2).  Where the output window leaves
// the inputs alone (a band inside the middle half of the grid: the image's rows
// are the others), each has a CTA of its own; otherwise one CTA does both and the
// even outputs wait in a stash of shared memory until the inputs have been read
// a second time.
#include <utility>

#include "cg_band_shape.cuh"
#include "cg_launch.cuh"

namespace cg {
namespace {

using namespace band;

template <typename T>
struct FC;
template <>
struct FC<float> { using type = float2; };
template <>
struct FC<double> { using type = double2; };

template <typename C>
__device__ __forceinline__ C cadd(C a, C b) { return C{a.x + b.x, a.y + b.y}; }
template <typename C>
__device__ __forceinline__ C csub(C a, C b) { return C{a.x - b.x, a.y - b.y}; }
// a times b (inverse) or its conjugate (forward)
template <bool kInv, typename C>
__device__ __forceinline__ C cmul(C a, C b) {
  return kInv ? C{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x} : C{a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y};
}
// times +i (inverse) or -i (forward)
template <bool kInv, typename C>
__device__ __forceinline__ C mul_i(C a) { return kInv ? C{-a.y, a.x} : C{a.y, -a.x}; }
// times e^{+-2 pi i k / 16}
template <bool kInv, int K, typename C>
__device__ __forceinline__ C mul_w16(C a) {
  using T = decltype(a.x);
  constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173, c2 = 0.70710678118654752440;
  constexpr int k = K & 15;
  if constexpr (k == 0) return a;
  if constexpr (k == 4) return mul_i<kInv>(a);
  constexpr double cs[16] = {1, c1, c2, s1, 0, -s1, -c2, -c1, -1, -c1, -c2, -s1, 0, s1, c2, c1};
  constexpr double sn[16] = {0, s1, c2, c1, 1, c1, c2, s1, 0, -s1, -c2, -c1, -1, -c1, -c2, -s1};
  const T wr = (T)cs[k], wi = (T)(kInv ? sn[k] : -sn[k]);
  return C{a.x * wr - a.y * wi, a.x * wi + a.y * wr};
}

// cos and sin of 2 pi k / n for the constants of the composite radices
// (Taylor series on [-pi / 4, pi / 4] after folding; evaluated by the compiler)
struct CosSin {
  double c, s;
};
__host__ __device__ constexpr CosSin unit_root(int k, int n) {
  k = ((k % n) + n) % n;
  // octant: angle = 2 pi k / n = q pi / 2 + r, |r| <= pi / 4
  const int q = (8 * k + n) / (2 * n);
  const double r = 1.57079632679489661923 * ((4.0 * k) / n - q), r2 = r * r;
  double c = 0, s = 0;
  for (int i = 12; i >= 1; i--) {
    c = (1 + c) * -r2 / ((2 * i) * (2 * i - 1));
    s = (1 + s) * -r2 / ((2 * i) * (2 * i + 1));
  }
  c = 1 + c;
  s = r * (1 + s);
  return (q & 3) == 0 ? CosSin{c, s} : (q & 3) == 1 ? CosSin{-s, c} : (q & 3) == 2 ? CosSin{-c, -s} : CosSin{s, -c};
}

template <bool kInv, typename C>
__device__ __forceinline__ void dft2(C& a, C& b) {
  const C t = a;
  a = cadd(t, b);
  b = csub(t, b);
}
template <bool kInv, typename C>
__device__ __forceinline__ void dft4(C& a, C& b, C& c, C& d) {
  const C s0 = cadd(a, c), d0 = csub(a, c), s1 = cadd(b, d), d1 = mul_i<kInv>(csub(b, d));
  a = cadd(s0, s1);
  c = csub(s0, s1);
  b = cadd(d0, d1);
  d = csub(d0, d1);
}

// v[i + B j] *= e^{+-2 pi i i j / (A B)}, j the index of the first transform's output
template <int A, int B, bool kInv, int X, typename C>
__device__ __forceinline__ void twiddle_one(C* v) {
  using T = decltype(v[0].x);
  constexpr int i = X % B, j = X / B;
  if constexpr (4 * i * j == A * B) {
    v[X] = mul_i<kInv>(v[X]);
  } else if constexpr (2 * i * j == A * B) {
    v[X] = C{-v[X].x, -v[X].y};
  } else if constexpr (i > 0 && j > 0) {
    constexpr CosSin w = unit_root(i * j, A * B);
    const T wr = (T)w.c, wi = (T)(kInv ? w.s : -w.s);
    v[X] = C{v[X].x * wr - v[X].y * wi, v[X].x * wi + v[X].y * wr};
  }
}
template <int A, int B, bool kInv, typename C, int... X>
__device__ __forceinline__ void twiddle_all(C* v, std::integer_sequence<int, X...>) {
  (twiddle_one<A, B, kInv, X>(v), ...);
}

// in-register transform of R points, natural order in and out
template <int R, bool kInv, typename C>
__device__ __forceinline__ void dft(C* v) {
  using T = decltype(v[0].x);
  if constexpr (R == 2) {
    dft2<kInv>(v[0], v[1]);
  } else if constexpr (R == 3) {
    const T h = (T)0.86602540378443864676;
    const C s = cadd(v[1], v[2]), d = csub(v[1], v[2]);
    const C t = C{v[0].x - (T)0.5 * s.x, v[0].y - (T)0.5 * s.y};
    const C u = mul_i<kInv>(C{h * d.x, h * d.y});
    v[0] = cadd(v[0], s);
    v[1] = cadd(t, u);
    v[2] = csub(t, u);
  } else if constexpr (R == 4) {
    dft4<kInv>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 5) {
    const T c1 = (T)0.30901699437494742410, c2 = (T)-0.80901699437494742410;
    const T s1 = (T)0.95105651629515357212, s2 = (T)0.58778525229247312917;
    const C a1 = cadd(v[1], v[4]), b1 = csub(v[1], v[4]), a2 = cadd(v[2], v[3]), b2 = csub(v[2], v[3]);
    const C x0 = v[0];
    const C p = C{x0.x + c1 * a1.x + c2 * a2.x, x0.y + c1 * a1.y + c2 * a2.y};
    const C q = C{x0.x + c2 * a1.x + c1 * a2.x, x0.y + c2 * a1.y + c1 * a2.y};
    const C r = mul_i<kInv>(C{s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y});
    const C t = mul_i<kInv>(C{s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y});
    v[0] = cadd(x0, cadd(a1, a2));
    v[1] = cadd(p, r);
    v[4] = csub(p, r);
    v[2] = cadd(q, t);
    v[3] = csub(q, t);
  } else if constexpr (R == 8) {
    dft4<kInv>(v[0], v[2], v[4], v[6]);
    dft4<kInv>(v[1], v[3], v[5], v[7]);
    // even transform in v[0], v[2], v[4], v[6]; odd in v[1], v[3], v[5], v[7]
    const C o1 = mul_w16<kInv, 2>(v[3]), o2 = mul_w16<kInv, 4>(v[5]), o3 = mul_w16<kInv, 6>(v[7]);
    const C e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1); v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2); v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3); v[7] = csub(e3, o3);
  } else {
    // R = A B: transforms of A points at stride B, twiddles, transforms of B
    constexpr int A = R == 16 ? 4 : (R % 3 == 0 ? 3 : 2), B = R / A;
    static_assert(A * B == R && B <= 5, "radix");
    C u[A];
#pragma unroll
    for (int i = 0; i < B; i++) {
#pragma unroll
      for (int j = 0; j < A; j++) u[j] = v[i + B * j];
      dft<A, kInv>(u);
#pragma unroll
      for (int j = 0; j < A; j++) v[i + B * j] = u[j];
    }
    twiddle_all<A, B, kInv>(v, std::make_integer_sequence<int, R>());
    C w[R];
#pragma unroll
    for (int j = 0; j < A; j++) {
      dft<B, kInv>(v + B * j);
#pragma unroll
      for (int i = 0; i < B; i++) w[j + A * i] = v[B * j + i];
    }
#pragma unroll
    for (int i = 0; i < R; i++) v[i] = w[i];
  }
}

template <typename C>
struct Line {
  C* grid;      // first line's first element
  int lines;    // lines present (the last group may be short)
  int s;        // which of the H transforms
};

template <int R, bool kRows, bool kInv, typename C>
__device__ __forceinline__ void pass(const BandFft& a, const Line<C>& ln, C* __restrict__ sm,
                                     const C* __restrict__ tab, int i) {
  const BandPass& ps = a.pass[i];
  const bool first = i == 0, last = i == a.npass - 1;
  const int sub = ps.sub, step = ps.step;
#pragma unroll 1
  for (int b = threadIdx.x; b < ps.total; b += blockDim.x) {
    int c, bf;  // line, butterfly
    if constexpr (kRows) {
      c = div_by(b, ps.mnbf, ps.nbf);
      bf = b - c * ps.nbf;
    } else {
      c = b & (a.NB - 1);
      bf = b >> a.logNB;
    }
    C v[R];
    if (first) {
      // The inputs are taken from the window's start on, rounded down to the
      // butterfly's stride: v[t] is the input m0 + t (modulo R), a rotation that
      // the table's factors e^{+-2 pi i m m0 / R} undo.
      const C* src = ln.grid + (size_t)c * a.ls;
      const int ni = c < ln.lines ? a.ni : 0;
      int o = bf - a.delta;  // offset in the window
      if (o < 0) o += a.n;
      const int o1 = bf - a.delta + sub;
      int x = a.i0 + o1;
      if (x >= a.L) x -= a.L;
      const int x1 = x;
#pragma unroll
      for (int m = 0; m < R; m++) v[m] = C{0, 0};
      int x0 = a.i0 + o;
      if (x0 >= a.L) x0 -= a.L;
      if (o < ni) v[0] = src[(size_t)(unsigned)x0 * a.es];
#pragma unroll
      for (int m = 1; m < R; m++) {
        if (o1 + (m - 1) * sub < ni) v[m] = src[(size_t)(unsigned)x * a.es];
        x += sub;
        if (x >= a.L) x -= a.L;
      }
      if (ln.s == 1) {
        v[0] = cmul<kInv>(v[0], tab[x0]);
        x = x1;
#pragma unroll
        for (int m = 1; m < R; m++) {
          v[m] = cmul<kInv>(v[m], tab[x]);
          x += sub;
          if (x >= a.L) x -= a.L;
        }
      }
      dft<R, kInv>(v);
      const C* tp = tab + ps.tw + bf;
#pragma unroll
      for (int m = 1; m < R; m++) v[m] = cmul<kInv>(v[m], tp[m * sub]);
      C* sp = sm + c * a.cs + padded_at(a, bf) * a.js;
#pragma unroll
      for (int m = 0; m < R; m++) sp[m * step] = v[m];
    } else if (!last) {
      const int blkid = div_by(bf, ps.msub, sub), j = bf - blkid * sub;
      C* sp = sm + c * a.cs + padded_at(a, blkid * ps.blk + j) * a.js;
#pragma unroll
      for (int m = 0; m < R; m++) v[m] = sp[m * step];
      dft<R, kInv>(v);
      const C* tp = tab + ps.tw + j;
#pragma unroll
      for (int m = 1; m < R; m++) v[m] = cmul<kInv>(v[m], tp[m * sub]);
#pragma unroll
      for (int m = 0; m < R; m++) sp[m * step] = v[m];
    } else {
      // butterflies in output order: neighbours write neighbours
      const C* sp = sm + c * a.cs + padded_at(a, block_of(a, bf) * R) * a.js;
#pragma unroll
      for (int m = 0; m < R; m++) v[m] = sp[m * step];
      dft<R, kInv>(v);
      C* dst = ln.grid + (size_t)c * a.ls;
      int k = a.H == 2 ? 2 * bf + ln.s : bf, d = k - a.o0;
      if (d < 0) d += a.L;
      const int no = c < ln.lines ? a.no : 0, dk = a.H * ps.nbf;
      if (a.H == 2 && ln.s == 0 && !a.apart) {
        C* st = sm + a.stash + c;
#pragma unroll
        for (int m = 0; m < R; m++) {
          if (d < no) st[(d >> 1) << a.logNB] = v[m];
          d += dk;
          if (d >= a.L) d -= a.L;
        }
      } else {
#pragma unroll
        for (int m = 0; m < R; m++) {
          if (d < no) dst[(size_t)(unsigned)(k + m * dk) * a.es] = v[m];
          d += dk;
          if (d >= a.L) d -= a.L;
        }
      }
    }
  }
}

template <bool kRows, bool kInv, typename C>
__device__ __forceinline__ void pass_any(const BandFft& a, const Line<C>& ln, C* sm, const C* tab, int i) {
  switch (a.pass[i].R) {
    case 16: pass<16, kRows, kInv>(a, ln, sm, tab, i); break;
    case 15: pass<15, kRows, kInv>(a, ln, sm, tab, i); break;
    case 12: pass<12, kRows, kInv>(a, ln, sm, tab, i); break;
    case 10: pass<10, kRows, kInv>(a, ln, sm, tab, i); break;
    case 9: pass<9, kRows, kInv>(a, ln, sm, tab, i); break;
    case 8: pass<8, kRows, kInv>(a, ln, sm, tab, i); break;
    case 6: pass<6, kRows, kInv>(a, ln, sm, tab, i); break;
    case 5: pass<5, kRows, kInv>(a, ln, sm, tab, i); break;
    case 4: pass<4, kRows, kInv>(a, ln, sm, tab, i); break;
    case 3: pass<3, kRows, kInv>(a, ln, sm, tab, i); break;
    default: pass<2, kRows, kInv>(a, ln, sm, tab, i); break;
  }
}

template <typename T, bool kRows, bool kInv>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 1024 : 512, 1)
    k_band_fft(typename FC<T>::type* __restrict__ grid, const __grid_constant__ BandFft a,
               const typename FC<T>::type* __restrict__ tab) {
  using C = typename FC<T>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  C* sm = reinterpret_cast<C*>(smem);
  const int ga = (a.na + a.NB - 1) / a.NB;  // groups of the first range
  const int item = a.apart ? blockIdx.x >> 1 : blockIdx.x;
  const int p = item / a.groups, g = item - p * a.groups;
  const int l0 = g < ga ? a.c0a + g * a.NB : a.c0b + (g - ga) * a.NB;
  const int end = g < ga ? a.c0a + a.na : a.c0b + a.nb;
  Line<C> ln{grid + (size_t)p * a.plane + (size_t)l0 * a.ls, min(a.NB, end - l0), 0};
  for (int s = a.apart ? blockIdx.x & 1 : 0; s < a.H; s += a.apart ? 2 : 1) {
    ln.s = s;
    for (int i = 0; i < a.npass; i++) {
      pass_any<kRows, kInv>(a, ln, sm, tab, i);
      __syncthreads();
      if (i == 0 && s == 1 && !a.apart) {  // the inputs have been read for the last time: the even outputs leave the stash
        const int par = a.o0 & 1, half = (a.no - par + 1) / 2;
        const C* st = sm + a.stash;
        for (int u = threadIdx.x; u < half * a.NB; u += blockDim.x) {
          const int c = u & (a.NB - 1), pos = u >> a.logNB;
          int k = a.o0 + par + 2 * pos;
          if (k >= a.L) k -= a.L;
          if (c < ln.lines) ln.grid[(size_t)(unsigned)k * a.es + (size_t)c * a.ls] = st[u];
        }
      }
    }
  }
}

// Table of a shape: e^{2 pi i x / L}, x < L (the second transform's input
// factors), then each pass's twiddles, neighbouring butterflies next to each other.
template <typename C>
__global__ void k_band_table(const __grid_constant__ BandFft a, int len, C* __restrict__ tab) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= len) return;
  double arg = 2.0 * i / a.L;
  for (int q = 0; q < a.npass; q++) {
    const int e = i - a.pass[q].tw;
    if (e >= 0 && e < a.pass[q].blk) {
      const int m = e / a.pass[q].sub, j = e - m * a.pass[q].sub;
      // first pass: the rotation of its inputs too
      arg = 2.0 * ((int64_t)m * (j + (q == 0 ? a.m0 * a.pass[q].sub : 0)) % a.pass[q].blk) / a.pass[q].blk;
    }
  }
  double s, c;
  sincospi(arg, &s, &c);
  tab[i].x = c;
  tab[i].y = s;
}

BandFft band_args(const BandLines& b) {
  BandFft a{};
  a.L = b.L;
  a.i0 = b.i0; a.ni = b.ni; a.o0 = b.o0; a.no = b.no;
  a.c0a = b.c0a; a.na = b.na; a.c0b = b.c0b; a.nb = b.nb;
  return a;
}

}  // namespace

template <typename T>
bool band_fft_supported(const BandLines& b) {
  BandFft a = band_args(b);
  int threads;
  size_t smem;
  return band_shape(a, b.rows, 2 * sizeof(T), &threads, &smem);
}

template <typename T>
size_t band_table_len(const BandLines& b) {
  BandFft a = band_args(b);
  int threads;
  size_t smem;
  if (!band_shape(a, b.rows, 2 * sizeof(T), &threads, &smem)) return 0;
  return (size_t)a.pass[a.npass - 1].tw + a.pass[a.npass - 1].blk;
}

template <typename T>
int64_t band_table_key(const BandLines& b) {
  BandFft a = band_args(b);
  int threads;
  size_t smem;
  if (!band_shape(a, b.rows, 2 * sizeof(T), &threads, &smem)) return 0;
  return ((int64_t)a.L * 2 + (a.H - 1)) * 32 + a.m0 + 1;
}

template <typename T>
int make_band_table(const BandLines& b, void* d_tab, cudaStream_t st) {
  using C = typename FC<T>::type;
  BandFft a = band_args(b);
  int threads;
  size_t smem;
  if (!band_shape(a, b.rows, sizeof(C), &threads, &smem)) return CG_ERR_ARG;
  const int len = (int)band_table_len<T>(b);
  k_band_table<C><<<(len + 255) / 256, 256, 0, st>>>(a, len, (C*)d_tab);
  count_launches(1);
  CG_CUDA(cudaGetLastError());
  return CG_OK;
}

template <typename T>
int launch_band_fft(const BandLines& b, T* grid, int nf1, size_t plane, int nplanes, int sign, const void* d_tab,
                    cudaStream_t st) {
  using C = typename FC<T>::type;
  BandFft a = band_args(b);
  int threads;
  size_t smem;
  if (!band_shape(a, b.rows, sizeof(C), &threads, &smem)) return CG_ERR_ARG;
  a.es = b.rows ? 1 : nf1;
  a.ls = b.rows ? nf1 : 1;
  a.plane = (long long)plane;
  a.nplanes = nplanes;
  a.groups = (a.na + a.NB - 1) / a.NB + (a.nb + a.NB - 1) / a.NB;
  if (a.groups == 0 || nplanes == 0) return CG_OK;
  const int64_t ctas = (int64_t)a.groups * nplanes * (a.apart ? 2 : 1);
  if (ctas > 2147483647LL) return CG_ERR_SIZE;
  auto* kern = b.rows ? (sign > 0 ? k_band_fft<T, true, true> : k_band_fft<T, true, false>)
                      : (sign > 0 ? k_band_fft<T, false, true> : k_band_fft<T, false, false>);
  int per_sm = 0;
  CG_CUDA(kernel_occupancy((const void*)kern, threads, smem, &per_sm));
  if (per_sm < 1) return CG_ERR_ARG;
  kern<<<(int)ctas, threads, smem, st>>>((C*)grid, a, (const C*)d_tab);
  count_launches(1);
  CG_CUDA(cudaGetLastError());
  return CG_OK;
}

template bool band_fft_supported<float>(const BandLines&);
template bool band_fft_supported<double>(const BandLines&);
template size_t band_table_len<float>(const BandLines&);
template size_t band_table_len<double>(const BandLines&);
template int64_t band_table_key<float>(const BandLines&);
template int64_t band_table_key<double>(const BandLines&);
template int make_band_table<float>(const BandLines&, void*, cudaStream_t);
template int make_band_table<double>(const BandLines&, void*, cudaStream_t);
template int launch_band_fft<float>(const BandLines&, float*, int, size_t, int, int, const void*, cudaStream_t);
template int launch_band_fft<double>(const BandLines&, double*, int, size_t, int, int, const void*, cudaStream_t);

}  // namespace cg
