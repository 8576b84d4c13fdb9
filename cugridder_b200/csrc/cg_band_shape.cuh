// Shape of the band-pruned transforms (cg_fft_band.cu): radices, strides, padding, tables
// and launch size of a line length and its windows, and the index arithmetic that
// the kernel and its tests share.
#pragma once
#include <algorithm>

#include "cg_internal.cuh"

namespace cg {
namespace band {

constexpr int kMaxPass = 10;

// One pass: radix R splits blocks of `blk` positions; its butterfly takes the
// positions sub = blk / R apart.
struct BandPass {
  int R, sub, blk;
  int nbf, total;            // butterflies per line (n / R) and per CTA
  int step;                  // shared-memory stride of the butterfly
  int tw;                    // its twiddles in the table: e^{2 pi i m j / blk} at tw + m sub + j
  unsigned mr, msub, mnbf;   // reciprocals (see TileDiv) of R, sub and nbf
};

struct BandFft {
  int L, n, H;               // length, points per transform, transforms per line
  int npass;
  BandPass pass[kMaxPass];
  int Q, S1;                 // one element of padding per Q points and one per S1 (see band_shape)
  unsigned mq, ms1;
  int i0, ni, o0, no;        // input and output windows
  int m0, delta;             // i0 modulo n = m0 (n / R_0) + delta: see pass()
  int NB, logNB;             // lines per CTA
  int c0a, na, c0b, nb;      // lines [c0a, c0a + na) and [c0b, c0b + nb)
  int groups, nplanes;
  unsigned es;               // element stride (complex elements)
  long long ls;              // line stride
  long long plane;
  int cs, js;                // line and point stride in shared memory
  int apart;                 // H = 2 and the windows do not meet: the two transforms are CTAs of their own
  int stash;                 // offset of the stash in shared memory (complex elements); unused if apart
};

// n / d by d's reciprocal m (recip)
__host__ __device__ __forceinline__ int div_by(int n, unsigned m, int d) {
#ifdef __CUDA_ARCH__
  return d == 1 ? n : (int)__umulhi((unsigned)n, m);
#else
  return d == 1 ? n : (int)((unsigned long long)(unsigned)n * m >> 32);
#endif
}

constexpr int kPoints = 16;  // points per thread that a CTA is sized for

// Block of the last pass that holds the outputs k0 + m n / R: an output is
// k = m_1 + R_1 (m_2 + R_2 (...)), its position m_1 n / R_1 + m_2 n / (R_1 R_2) + ...
__host__ __device__ __forceinline__ int block_of(const BandFft& a, int k0) {
  int blk = 0;
  for (int i = 0; i < a.npass - 1; i++) {
    const int R = a.pass[i].R, q = div_by(k0, a.pass[i].mr, R);
    blk = blk * R + (k0 - q * R);
    k0 = q;
  }
  return blk;
}

// shared-memory index of a position: padded so that neighbouring butterflies of
// every pass, the last one's in output order included, lie on different banks
__host__ __device__ __forceinline__ int padded_at(const BandFft& a, int pos) {
  return pos + div_by(pos, a.mq, a.Q) + div_by(pos, a.ms1, a.S1);
}

// Radices of n: 16 as often as it divides, then the rest of the 2s joined to 3s
// and 5s (15, 12, 10, 9, 8, 6) so that few passes remain; 0 when n has another
// prime factor or fewer than two passes.
inline int factor(int n, int* radix) {
  int a = 0, b = 0, c = 0, np = 0;
  for (; n % 2 == 0; n /= 2) a++;
  for (; n % 3 == 0; n /= 3) b++;
  for (; n % 5 == 0; n /= 5) c++;
  if (n != 1) return 0;
  auto put = [&](int r) {
    if (np < kMaxPass) radix[np] = r;
    np++;
  };
  while (a >= 4 && a != 5) {
    put(16);
    a -= 4;
  }
  if (a == 5) {
    put(8);
    a = 2;
  }
  while (c > 0 && b > 0) { put(15); c--; b--; }
  while (c > 0 && a > 0) { put(10); c--; a--; }
  while (c > 0) { put(5); c--; }
  while (b >= 2 && a == 0) { put(9); b -= 2; }
  while (b > 0 && a >= 2) { put(12); b--; a -= 2; }
  while (b > 0 && a > 0) { put(6); b--; a--; }
  while (b >= 2) { put(9); b -= 2; }
  while (b > 0) { put(3); b--; }
  if (a > 0) put(1 << a);
  return np >= 2 && np <= kMaxPass ? np : 0;
}

inline unsigned recip(int d) { return 0xFFFFFFFFu / (unsigned)d + 1u; }

constexpr size_t kBandSmem = 226 * 1024;

// Fills a's shape for line length L, windows and element size; false where it
// does not fit.  rows: lines are grid rows.
inline bool band_shape(BandFft& a, bool rows, size_t esz, int* threads, size_t* smem) {
  const int L = a.L;
  // distance from one window's start to the other's, both ways round
  const int io = ((a.o0 - a.i0) % L + L) % L, oi = ((a.i0 - a.o0) % L + L) % L;
  const bool meet = io < a.ni || oi < a.no;
  const int most = esz == 8 ? 1024 * kPoints : 512 * kPoints;  // points of a CTA
  auto padded = [](int n) { return n + n / 8 + 18; };  // Q >= 8 for the lengths near the limit
  auto fits = [&](int H, int NB) {
    const size_t stash = H == 2 && meet ? (size_t)(a.no / 2 + 1) * NB : 0;
    return (int64_t)L / H * NB <= most && ((size_t)padded(L / H) * NB + stash) * esz <= kBandSmem;
  };
  // rows: from L = 8192 on, where half the length saves a pass and doubles the CTAs
  // of an SM (8192^2 x 14, both transforms 5.25 -> 4.25 ms; at 4096 0.85 -> 0.89)
  a.H = a.ni <= L / 2 && L % 2 == 0 && (!rows || (!meet && L >= 8192)) ? 2 : 1;
  a.apart = a.H == 2 && !meet;
  a.NB = 0;
  if (rows) {
    // rows: enough for 256 threads
    int NB = 1;
    while (NB < 16 && (int64_t)L / a.H * NB < 256 * kPoints && fits(a.H, 2 * NB)) NB *= 2;
    if (fits(a.H, NB)) a.NB = NB;
  } else {
    // 4 columns: a whole sector of 32 bytes a grid row in FP32, and CTAs small
    // enough that two or more share an SM up to L = 4096.  Measured with 2, 4
    // and 8: FP32 2048 x 2500 x 12 0.45, 0.43, 0.49 ms; 4096^2 x 12 1.72, 1.50,
    // 1.44; FP64 4096^2 x 20 4.12, 3.69, 3.69 (an earlier form of the kernel)
    for (int NB = 4; NB >= 1 && !a.NB; NB /= 2)
      if (fits(a.H, NB)) a.NB = NB;
  }
  if (!a.NB) return false;
  a.n = L / a.H;
  int radix[kMaxPass];
  a.npass = factor(a.n, radix);
  if (!a.npass) return false;
  a.logNB = 0;
  while ((1 << a.logNB) < a.NB) a.logNB++;
  // padding: one element per Q points, Q the product of the last radices up to
  // 8 or more, and one per point of the first pass's stride S1 (outputs that
  // follow one another lie S1 positions apart)
  a.Q = 1;
  for (int i = a.npass - 1; i > 0 && a.Q < 8; i--) a.Q *= radix[i];
  a.S1 = a.n / radix[0];
  a.mq = recip(a.Q);
  a.ms1 = recip(a.S1);
  const int pts = a.n + a.n / a.Q + radix[0] + 1;
  a.cs = rows ? pts : 1;
  a.js = rows ? 1 : a.NB;
  a.stash = pts * a.NB;
  a.m0 = a.i0 % a.n / a.S1;
  a.delta = a.i0 % a.n - a.m0 * a.S1;
  int tw = L;
  for (int i = 0, blk = a.n; i < a.npass; i++) {
    BandPass& p = a.pass[i];
    p.R = radix[i];
    p.blk = blk;
    p.sub = blk / p.R;
    p.nbf = a.n / p.R;
    p.total = p.nbf * a.NB;
    p.step = (p.sub + (p.sub >= a.Q ? p.sub / a.Q : 0) + (i == 0 ? 1 : 0)) * a.js;
    p.tw = tw;
    tw += blk;
    p.mr = recip(p.R);
    p.msub = recip(p.sub);
    p.mnbf = recip(p.nbf);
    blk = p.sub;
  }
  *threads = std::max(64, ((a.n * a.NB + kPoints - 1) / kPoints + 31) / 32 * 32);
  *smem = ((size_t)a.stash + (a.H == 2 && meet ? (size_t)(a.no / 2 + 1) * a.NB : 0)) * esz;
  return true;
}

}  // namespace band
}  // namespace cg
