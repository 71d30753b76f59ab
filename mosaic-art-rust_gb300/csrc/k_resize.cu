// k_resize.cu -- Lanczos3 resize of the material images into thumbnails.
//
// Reference: main.rs:710-738 resize_image, fast_image_resize 5.1.4 with its
// default ResizeOptions (a Lanczos3 convolution, no cropping) on U8x3 images;
// the GUI asks for Lanczos3 explicitly (gui/app_full.rs:1894-1898).  That
// crate's convolution resampler follows the published one of Pillow
// (ImagingResample), which this restates:
//   * per output coordinate o of a dimension in -> out: scale = in / out,
//     filterscale = max(scale, 1), support = 3 * filterscale, centre =
//     (o + 0.5) * scale; taps i in [int(centre - support + 0.5),
//     int(centre + support + 0.5)) clipped to [0, in), weight
//     lanczos3((i - centre + 0.5) / filterscale), lanczos3(x) = sinc(x)
//     sinc(x / 3) on [-3, 3), the weights divided by their sum, then rounded
//     (half away from zero) to 22-bit fixed point;
//   * a horizontal pass into an 8-bit intermediate, then a vertical pass;
//     each output channel is clip8((2^21 + sum of weight * sample) >> 22); a
//     dimension that keeps its size is copied.
// The weights are computed once per distinct source size on the host in FP64
// and uploaded; the passes are integer arithmetic, so the result is exact and
// the CPU oracle computes the same bytes.  Parity with fast_image_resize's own
// fixed-point choices is not pinned (the crate is not here to run).
//
// Two forms (choose_bands):
//  - resize_fused_kernel: both passes in one CTA per image or band of output rows,
//    the source and the 8-bit intermediate in shared
//    memory.  What bounds it is the multiply-adds: two passes of ~6 * scale taps
//    a sample, and at a byte a tap an extraction for each.  So bytes are kept
//    four to a word along the dimension the next pass sums over -- the source by
//    channel planes, the intermediate transposed -- and a weight is split into
//    three bytes, w = 2^16 p2 + 2^8 p1 + p0 (p2 signed): three dp4a do four taps
//    of a channel.  The sums are integers, so the split changes nothing.  A
//    thread makes four rows of a column, which share the weights it reads.
//  - resize_h_kernel, resize_v_kernel: the passes one after the other, a thread a
//    sample, the intermediate in global memory; also for images whose rows, weights
//    and intermediate do not fit in shared memory (kMaxFusedWords).
//
// Layout of a table for in -> out.  Two-kernel form: [out, kmax], then out (first
// tap, tap count) pairs, then out rows of kmax weights.  Fused form: [nw], then
// out (first word << 16 | words) of four taps, then out rows of (3 nw) | 1 words
// (odd: rows start in different banks), words p0, p1, p2 of each four taps.
#include <algorithm>
#include <cmath>
#include <map>
#include <vector>

#include "mg_internal.h"

namespace mg {

namespace {

constexpr int kResizeBits = 22;

double sinc(double x) {
  if (x == 0.0) return 1.0;
  x *= M_PI;
  return std::sin(x) / x;
}
double lanczos3(double x) { return (-3.0 <= x && x < 3.0) ? sinc(x) * sinc(x / 3.0) : 0.0; }

// The table of one dimension in -> out (out > 0, in > 0), two-kernel form.
std::vector<int32_t> build_table(int in, int out) {
  const double scale = (double)in / (double)out;
  const double filterscale = scale < 1.0 ? 1.0 : scale;
  const double support = 3.0 * filterscale;
  const int kmax = (int)std::ceil(support) * 2 + 1;
  std::vector<int32_t> t(2 + 2 * (size_t)out + (size_t)out * kmax, 0);
  t[0] = out;
  t[1] = kmax;
  std::vector<double> w(kmax);
  for (int o = 0; o < out; ++o) {
    const double centre = (o + 0.5) * scale;
    int lo = (int)(centre - support + 0.5);
    if (lo < 0) lo = 0;
    int hi = (int)(centre + support + 0.5);
    if (hi > in) hi = in;
    const int cnt = hi - lo;
    double sum = 0.0;
    for (int i = 0; i < cnt; ++i) {
      w[i] = lanczos3((i + lo - centre + 0.5) / filterscale);
      sum += w[i];
    }
    t[2 + 2 * (size_t)o] = lo;
    t[3 + 2 * (size_t)o] = cnt;
    int32_t* k = t.data() + 2 + 2 * (size_t)out + (size_t)o * kmax;
    for (int i = 0; i < cnt; ++i) {
      const double v = sum != 0.0 ? w[i] / sum : w[i];
      k[i] = (int32_t)(v < 0.0 ? -0.5 + v * (1 << kResizeBits) : 0.5 + v * (1 << kResizeBits));
    }
  }
  return t;
}

// The table of a copy: one tap of weight 1.
std::vector<int32_t> copy_table(int out) {
  std::vector<int32_t> o(2 + 3 * (size_t)out, 0);
  o[0] = out;
  o[1] = 1;
  for (int i = 0; i < out; ++i) {
    o[2 + 2 * (size_t)i] = i;
    o[3 + 2 * (size_t)i] = 1;
    o[2 + 2 * (size_t)out + i] = 1 << kResizeBits;
  }
  return o;
}

// The fused form of the table `o` of in -> out, appended to t; false when a weight
// does not split (its top byte is signed).
bool append_fused(int in, int out, const std::vector<int32_t>& o, std::vector<int32_t>& t) {
  const int kmax = o[1];
  const int32_t* bounds = o.data() + 2;
  const int32_t* coef = bounds + 2 * (size_t)out;
  int nw = 1;
  for (int i = 0; i < out; ++i) {
    const int lo = bounds[2 * i], cnt = bounds[2 * i + 1];
    nw = std::max(nw, (lo + std::max(cnt, 1) - 1) / 4 - lo / 4 + 1);
  }
  if (in > 4 * 65535 || nw > 65535) return false;
  const int pitch = (3 * nw) | 1;
  const size_t base = t.size();
  t.resize(base + 1 + out + (size_t)out * pitch, 0);
  t[base] = nw;
  for (int i = 0; i < out; ++i) {
    const int lo = bounds[2 * i], cnt = bounds[2 * i + 1], w0 = lo / 4;
    t[base + 1 + i] = (int32_t)((uint32_t)w0 << 16 | (uint32_t)((lo + std::max(cnt, 1) - 1) / 4 - w0 + 1));
    uint32_t* w = reinterpret_cast<uint32_t*>(t.data()) + base + 1 + out + (size_t)i * pitch;
    for (int j = 0; j < cnt; ++j) {
      const int32_t v = coef[(size_t)i * kmax + j];
      if (v >= 1 << 23 || v < -(1 << 23)) return false;
      const int at = lo - 4 * w0 + j, sh = 8 * (at & 3);
      uint32_t* q = w + 3 * (at >> 2);
      q[0] |= ((uint32_t)v & 255u) << sh;
      q[1] |= ((uint32_t)v >> 8 & 255u) << sh;
      q[2] |= ((uint32_t)v >> 16 & 255u) << sh;
    }
  }
  return true;
}

// ---- which form, and how many bands
// Neither form is the faster one everywhere: the fused one does a band by one CTA,
// which is slow where there are few images and each is scaled down far (one image of
// 1000 x 1000 to 16 x 12: 1290 us in two bands, 240 in two kernels), and a band reads
// 6 * scale source rows beside its own, which counts twice where the sources come over
// the CPU-GPU link (14 images of 1000 x 1000 to 64 x 48 there: 640 and 330 us); the
// other one does a tap a byte (400 of 500 x 500 to 16 x 12: 317 and 1430 us) and
// fetches bytes again and again from the link once its rows overflow the L1 caches.
// So both are estimated, the fused one for each number of bands.  The constants
// (microseconds) are fits to measured times of 739 sets of 1 to 2000 images of 40 to
// 1500 pixels a side, thumbnails of 8 to 200, in all forms; the choice is within 5%
// of the best form on the average, with the sources on the device and over the link.
struct ResizeShape {
  double n, w, h, tw, th;  // images, their mean size, the thumbnail's
  int sms;
};
constexpr int kFusedThreads = 256;
constexpr int kFusedPerSm = 3;          // CTAs of an SM the shared memory is planned for
constexpr int kFusedWords = 18 * 1024;  // ... in words; more only where one image needs it
constexpr int kMaxFusedWords = 50 * 1024;

double taps(double in, double out) { return in == out ? 1.0 : 6.0 * std::max(in / out, 1.0) + 1.0; }

double fused_us(const ResizeShape& s, int bands, bool link) {
  const double rows = std::ceil(s.th / bands);  // of output, by a CTA
  const double scale = std::max(s.h / s.th, 1.0), beside = bands == 1 ? 0 : bands == 2 ? 3 : 6;
  const double in_rows = std::min(s.h, rows * s.h / s.th + beside * scale);
  const double xw = s.w == s.tw ? 1.0 : std::floor(taps(s.w, s.tw) / 4) + 2, yw = s.h == s.th ? 1.0 : std::floor(taps(s.h, s.th) / 4) + 2;
  const double quads = std::min(std::ceil(s.h / 4), in_rows / 4 + 1);  // groups of four source rows
  const double fixed = s.tw * (3 * xw + 1) + rows * (3 * yw + 1) + 3 * s.tw * (quads + 1), group = 12 * (s.w / 4 + 1);
  const double at_once = std::max(1.0, std::min(quads, std::floor((kFusedWords - fixed) / group)));
  const double words = fixed + at_once * group;
  if (words > kMaxFusedWords) return 1e30;
  const double steps = std::ceil(quads / at_once);
  const double h_ops = std::ceil(quads / steps * s.tw / kFusedThreads) * steps * xw * 36;
  const double v_ops = std::ceil(rows * s.tw / kFusedThreads) * yw * 9;
  const double loads = in_rows * s.w / 4 / kFusedThreads;
  const double cta = link ? 0.00108 * h_ops + 0.0155 * v_ops + 0.869 * loads + 0.734 * steps
                          : 0.00106 * h_ops + 0.0162 * v_ops + 0.397 * loads + 0.535 * steps;
  const double turns = std::ceil(s.n * bands / s.sms);  // CTAs an SM, some of them at a time
  const int resident = (int)std::max(1.0, std::min({(double)kFusedPerSm, std::floor(227.0 * 1024 / (4 * words + 1024)), turns}));
  const double rate = resident == 1 ? 1.0 : resident == 2 ? 1.53 : 1.78;
  const double read = s.n * s.w * 3 * std::min(bands * s.h, s.h + (bands - 1) * 6 * scale);  // bytes
  return link ? 7.3 + cta * turns / rate + 3.04e-6 * read : 6.0 + cta * turns / rate;
}

double two_kernels_us(const ResizeShape& s, bool link) {
  const double tx = taps(s.w, s.tw), ty = taps(s.h, s.th);
  const double blocks = std::min(16.0, std::ceil(s.h * s.tw / 256));  // an image's
  auto pass = [](double chain, double all) { return std::pow(std::pow(chain, 4) + std::pow(all, 4), 0.25); };
  const double h_chain = std::ceil(s.h * s.tw / (256 * blocks)) * tx, h_all = 1e-6 * s.n * s.h * s.tw * tx;
  const double v_chain = std::ceil(s.th * s.tw / (256 * blocks)) * ty, v_all = 1e-6 * s.n * s.th * s.tw * ty;
  // KB of source rows that an SM's blocks are in at a time: what its L1 has to hold
  const double kb = std::min(8.0, s.n * blocks / s.sms) * std::max(1.0, 256 / s.tw) * 3 * s.w / 1024;
  const double mb = 1e-6 * s.n * s.w * s.h * 3;
  return link ? 11.3 + pass(0.104 * h_chain, 0.0) + pass(0.127 * v_chain, 1.17 * v_all) + 4.19 * mb * (1 + std::pow(kb / 57.2, 1.79))
              : 10.2 + pass(0.0904 * h_chain, 0.0347 * h_all) + pass(0.0790 * v_chain, 0.969 * v_all) + 0.812 * mb * std::pow(kb, 0.345);
}

// The bands of the fastest form by these, 0: two kernels.
int choose_bands(const ResizeShape& s, bool link) {
  int best = 0;
  double best_us = two_kernels_us(s, link);
  for (int b : {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48}) {
    if (b > std::max(1.0, s.th / 2)) break;
    const double us = fused_us(s, b, link);
    if (us < best_us) {
      best = b;
      best_us = us;
    }
  }
  return best;
}

// The band's rows of output.
__host__ __device__ inline int band_row(int b, int bands, int th) { return (int)((int64_t)b * th / bands); }

// Four taps of one channel: the three byte planes of the weights (the top one signed).
struct Sum3 {
  int32_t a = 0, b = 0, c = 0;
  __device__ __forceinline__ void add(uint32_t px, uint32_t w0, uint32_t w1, uint32_t w2) {
    a = (int32_t)__dp4a(px, w0, (uint32_t)a);
    b = (int32_t)__dp4a(px, w1, (uint32_t)b);
    asm("dp4a.u32.s32 %0, %1, %2, %0;" : "+r"(c) : "r"(px), "r"(w2));
  }
  __device__ __forceinline__ uint32_t value() const {  // modulo 2^32, as the one-word sum
    const int32_t v =
        (int32_t)((1u << (kResizeBits - 1)) + (uint32_t)a + ((uint32_t)b << 8) + ((uint32_t)c << 16)) >> kResizeBits;
    return (uint32_t)min(max(v, 0), 255);
  }
};

// Pixels 4 g .. 4 g + 3 of a row w wide (zeros beyond it), as a word per channel.
// Whole words where they lie inside the row's bytes, bytes elsewhere.
__device__ __forceinline__ void load_planar(const uint8_t* __restrict__ row, int w, int g, uint32_t& r, uint32_t& gr,
                                            uint32_t& b) {
  const uint8_t* p = row + 12 * g;
  uint32_t a0, a1, a2;  // the twelve bytes
  const uint32_t s = (uint32_t)(uintptr_t)p & 3u;
  if (4 * g + 4 <= w && s == 0) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p);
    a0 = __ldg(q);
    a1 = __ldg(q + 1);
    a2 = __ldg(q + 2);
  } else if (12 * g >= (int)s && 12 * g + 16 - (int)s <= 3 * w) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p - s);
    const uint32_t v0 = __ldg(q), v1 = __ldg(q + 1), v2 = __ldg(q + 2), v3 = __ldg(q + 3);
    a0 = __funnelshift_r(v0, v1, 8 * s);
    a1 = __funnelshift_r(v1, v2, 8 * s);
    a2 = __funnelshift_r(v2, v3, 8 * s);
  } else {
    a0 = a1 = a2 = 0u;
    const int n = min(12, 3 * w - 12 * g);
    for (int i = 0; i < n; ++i) {
      const uint32_t v = (uint32_t)p[i] << (8 * (i & 3));
      if (i < 4) a0 |= v;
      else if (i < 8) a1 |= v;
      else a2 |= v;
    }
  }
  // bytes R0 G0 B0 R1 | G1 B1 R2 G2 | B2 R3 G3 B3
  r = __byte_perm(__byte_perm(a0, a1, 0x0630), a2, 0x5210);
  gr = __byte_perm(__byte_perm(a0, a1, 0x0741), a2, 0x6210);
  b = __byte_perm(__byte_perm(a0, a1, 0x0052), a2, 0x7410);
}

// Image blockIdx.x, band blockIdx.y of its output rows.  Shared memory: the
// weights of the horizontal and of the band's vertical pass, source rows as
// [row][channel][word of four pixels], the intermediate as [channel][column]
// [word of four rows].
// Measured, GB300 (before: the two-kernel form), the materials stage: 5000
// materials of 128 x 128 to 32 x 32 1.16 -> 0.72 ms (the resize itself 0.25), 500
// to the default tile 0.134 -> 0.090.
__global__ void __launch_bounds__(kFusedThreads, kFusedPerSm)
    resize_fused_kernel(const uint8_t* __restrict__ base, const ResizeImage* __restrict__ imgs,
                        const int32_t* __restrict__ tabs, int tw, int th, int hw_words, int vw_words, int src_words,
                        int pi, uint8_t* __restrict__ out) {
  extern __shared__ __align__(16) uint32_t sm[];
  uint32_t* s_hw = sm;
  uint32_t* s_vw = s_hw + hw_words;
  uint32_t* s_src = s_vw + vw_words;
  uint32_t* s_int = s_src + src_words;
  const ResizeImage I = imgs[blockIdx.x];
  const int tid = threadIdx.x;
  const int o0 = band_row(blockIdx.y, gridDim.y, th), o1 = band_row(blockIdx.y + 1, gridDim.y, th);
  const int32_t* TH = tabs + I.htab;
  const int32_t* TV = tabs + I.vtab;
  const int hp = (3 * TH[0]) | 1, vp = (3 * TV[0]) | 1;
  for (int i = tid; i < tw * hp; i += kFusedThreads) s_hw[i] = (uint32_t)__ldg(TH + 1 + tw + i);
  for (int i = tid; i < (o1 - o0) * vp; i += kFusedThreads) s_vw[i] = (uint32_t)__ldg(TV + 1 + th + (size_t)o0 * vp + i);
  // rows of four that the band's taps lie in (first taps and last ones ascend)
  const uint32_t vlast = (uint32_t)TV[1 + o1 - 1];
  const int g0 = (int)((uint32_t)TV[1 + o0] >> 16), g1 = (int)(vlast >> 16) + (int)(vlast & 0xFFFFu);
  const int nwords = (I.w + 3) >> 2, pw = nwords | 1;
  const int dy = kFusedThreads / nwords, dg = kFusedThreads - dy * nwords;
  const int chunk = max(1, src_words / (12 * pw));  // groups of four rows at a time
  for (int c0 = g0; c0 < g1; c0 += chunk) {
    const int c1 = min(g1, c0 + chunk);
    const int rows = min(I.h, 4 * c1) - 4 * c0;  // (the last group's rows beyond the image: weights 0)
    __syncthreads();
    int y = tid / nwords, g = tid - y * nwords;
#pragma unroll 4
    for (int q = tid; q < rows * nwords; q += kFusedThreads) {
      uint32_t r, gr, b;
      load_planar(base + I.offset + (int64_t)(4 * c0 + y) * I.stride, I.w, g, r, gr, b);
      uint32_t* d = s_src + (3 * y) * pw + g;
      d[0] = r;
      d[pw] = gr;
      d[2 * pw] = b;
      g += dg;
      y += dy;
      if (g >= nwords) {
        g -= nwords;
        ++y;
      }
    }
    __syncthreads();
    for (int q = tid; q < (c1 - c0) * tw; q += kFusedThreads) {
      const int g = q / tw, x = q - g * tw;
      const uint32_t hb = (uint32_t)__ldg(TH + 1 + x);
      const uint32_t* w = s_hw + x * hp;
      const uint32_t* s = s_src + 12 * g * pw + (hb >> 16);
      Sum3 acc[4][3] = {};
      for (int n = (int)(hb & 0xFFFFu); n > 0; --n, w += 3, ++s) {
        const uint32_t w0 = w[0], w1 = w[1], w2 = w[2];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 3; ++c) acc[r][c].add(s[(3 * r + c) * pw], w0, w1, w2);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c)
        s_int[(c * tw + x) * pi + (c0 + g - g0)] = acc[0][c].value() | acc[1][c].value() << 8 |
                                                   acc[2][c].value() << 16 | acc[3][c].value() << 24;
    }
  }
  __syncthreads();
  uint8_t* dst = out + ((int64_t)blockIdx.x * th + o0) * tw * 3;
  for (int q = tid; q < (o1 - o0) * tw; q += kFusedThreads) {
    const int o = q / tw, x = q - o * tw;
    const uint32_t vb = (uint32_t)__ldg(TV + 1 + o0 + o);
    const uint32_t* w = s_vw + o * vp;
    const uint32_t* s = s_int + x * pi + ((int)(vb >> 16) - g0);
    Sum3 acc[3] = {};
    for (int n = (int)(vb & 0xFFFFu); n > 0; --n, w += 3, ++s)
#pragma unroll
      for (int c = 0; c < 3; ++c) acc[c].add(s[c * tw * pi], w[0], w[1], w[2]);
#pragma unroll
    for (int c = 0; c < 3; ++c) dst[3 * q + c] = (uint8_t)acc[c].value();
  }
}

__device__ __forceinline__ uint8_t clip8(int32_t v) {
  v >>= kResizeBits;
  return (uint8_t)(v < 0 ? 0 : (v > 255 ? 255 : v));
}

// Horizontal pass: image b's rows (sw wide) into its intermediate (tw wide),
// or a copy when the width is kept.
__global__ void __launch_bounds__(256) resize_h_kernel(const uint8_t* __restrict__ base, const ResizeImage* __restrict__ imgs,
                                                       const int32_t* __restrict__ tabs, int tw,
                                                       uint8_t* __restrict__ inter, int64_t inter_pitch) {
  const ResizeImage I = imgs[blockIdx.x];
  const uint8_t* src = base + I.offset;
  uint8_t* dst = inter + (int64_t)blockIdx.x * inter_pitch;
  const int total = I.h * tw;
  if (I.htab < 0) {  // same width
    for (int q = blockIdx.y * blockDim.x + threadIdx.x; q < total; q += gridDim.y * blockDim.x) {
      const int y = q / tw, x = q - y * tw;
      const uint8_t* s = src + (int64_t)y * I.stride + 3 * x;
      dst[3 * q] = s[0];
      dst[3 * q + 1] = s[1];
      dst[3 * q + 2] = s[2];
    }
    return;
  }
  const int32_t* T = tabs + I.htab;
  const int kmax = T[1];
  const int32_t* bounds = T + 2;
  const int32_t* coef = bounds + 2 * tw;
  for (int q = blockIdx.y * blockDim.x + threadIdx.x; q < total; q += gridDim.y * blockDim.x) {
    const int y = q / tw, x = q - y * tw;
    const int lo = bounds[2 * x], cnt = bounds[2 * x + 1];
    const uint8_t* s = src + (int64_t)y * I.stride + 3 * lo;
    const int32_t* k = coef + (int64_t)x * kmax;
    int32_t a0 = 1 << (kResizeBits - 1), a1 = a0, a2 = a0;
    for (int i = 0; i < cnt; ++i) {
      const int32_t w = __ldg(k + i);
      a0 += w * (int32_t)s[3 * i];
      a1 += w * (int32_t)s[3 * i + 1];
      a2 += w * (int32_t)s[3 * i + 2];
    }
    dst[3 * q] = clip8(a0);
    dst[3 * q + 1] = clip8(a1);
    dst[3 * q + 2] = clip8(a2);
  }
}

// Vertical pass: image b's intermediate (I.h rows of tw) into its thumbnail
// (th rows of tw), or a copy when the height is kept.
__global__ void __launch_bounds__(256) resize_v_kernel(const ResizeImage* __restrict__ imgs,
                                                       const int32_t* __restrict__ tabs, int tw, int th,
                                                       const uint8_t* __restrict__ inter, int64_t inter_pitch,
                                                       uint8_t* __restrict__ out) {
  const ResizeImage I = imgs[blockIdx.x];
  const uint8_t* src = inter + (int64_t)blockIdx.x * inter_pitch;
  uint8_t* dst = out + (int64_t)blockIdx.x * tw * th * 3;
  const int total = th * tw;
  const int pitch = 3 * tw;
  if (I.vtab < 0) {  // same height
    for (int q = blockIdx.y * blockDim.x + threadIdx.x; q < 3 * total; q += gridDim.y * blockDim.x) dst[q] = src[q];
    return;
  }
  const int32_t* T = tabs + I.vtab;
  const int kmax = T[1];
  const int32_t* bounds = T + 2;
  const int32_t* coef = bounds + 2 * th;
  for (int q = blockIdx.y * blockDim.x + threadIdx.x; q < total; q += gridDim.y * blockDim.x) {
    const int y = q / tw, x = q - y * tw;
    const int lo = bounds[2 * y], cnt = bounds[2 * y + 1];
    const uint8_t* s = src + (int64_t)lo * pitch + 3 * x;
    const int32_t* k = coef + (int64_t)y * kmax;
    int32_t a0 = 1 << (kResizeBits - 1), a1 = a0, a2 = a0;
    for (int i = 0; i < cnt; ++i) {
      const int32_t w = __ldg(k + i);
      const uint8_t* p = s + (int64_t)i * pitch;
      a0 += w * (int32_t)p[0];
      a1 += w * (int32_t)p[1];
      a2 += w * (int32_t)p[2];
    }
    dst[3 * q] = clip8(a0);
    dst[3 * q + 1] = clip8(a1);
    dst[3 * q + 2] = clip8(a2);
  }
}

}  // namespace

// The images' tables, in the fused form while `fused` holds (a table that has no
// such form clears it).  The weights themselves are computed once, into `weights`
// (by in and out), also where the fused form is given up: they are most of the
// host's time (4000 x 3000 to 400 x 300: 0.8 ms of a call of 2.6).
int ResizePlan::build_images(const Region* regions, ResizeWeights& weights, std::vector<int32_t>& t,
                             std::map<int, int>& wtab, std::map<int, int>& htab, std::vector<ResizeImage>& im) {
  max_h = 1;
  auto table = [&](std::map<int, int>& made, int in, int out) {
    if (!fused && in == out) return -1;
    auto it = made.find(in);
    if (it == made.end()) {
      it = made.emplace(in, (int)t.size()).first;
      std::vector<int32_t>& w = weights[{in, out}];
      if (w.empty()) w = in == out ? copy_table(out) : build_table(in, out);
      if (!fused) t.insert(t.end(), w.begin(), w.end());
      else if (!append_fused(in, out, w, t)) fused = false;
    }
    return it->second;
  };
  const bool was = fused;
  for (int i = 0; i < n && fused == was; ++i) {
    const Region& r = regions[i];
    if (r.w <= 0 || r.h <= 0) return fail(MG_ERR_ARG, "empty material image");
    const int ho = table(wtab, r.w, tw);
    const int vo = fused == was ? table(htab, r.h, th) : -1;
    im[i] = ResizeImage{r.offset, r.stride, r.w, r.h, ho, vo};
    max_h = std::max(max_h, r.h);
  }
  return MG_OK;
}

// Shared memory of the fused form in `bands` bands; false when it does not fit.
bool ResizePlan::plan_fused(const std::vector<int32_t>& t, const std::map<int, int>& wtab,
                            const std::map<int, int>& htab) {
  int64_t hw = 0, vw = 0, rows = 0, pw = 1;
  for (const auto& e : wtab) {
    hw = std::max(hw, (int64_t)tw * ((3 * t[e.second]) | 1));
    pw = std::max<int64_t>(pw, ((e.first + 3) / 4) | 1);
  }
  for (const auto& e : htab)
    for (int b = 0; b < bands; ++b) {
      const int o0 = band_row(b, bands, th), o1 = band_row(b + 1, bands, th);
      vw = std::max(vw, (int64_t)(o1 - o0) * ((3 * t[e.second]) | 1));
      const uint32_t first = (uint32_t)t[e.second + 1 + o0], last = (uint32_t)t[e.second + 1 + o1 - 1];
      rows = std::max<int64_t>(rows, (int64_t)(last >> 16) + (last & 0xFFFFu) - (first >> 16));
    }
  const int64_t pi = rows | 1, fixed = hw + vw + 3 * tw * pi, group = 12 * pw;
  if (fixed + group > kMaxFusedWords) return false;
  const int64_t groups = std::max<int64_t>(1, std::min(rows, (kFusedWords - fixed) / group));
  hw_words = (int)hw;
  vw_words = (int)vw;
  src_words = (int)(groups * group);
  inter_pitch = (int)pi;
  return true;
}

int ResizePlan::build(const Region* regions, int n_images, int tw_, int th_, bool over_link, cudaStream_t s) {
  if (n_images <= 0) {
    n = 0;
    return MG_OK;
  }
  if (tw_ <= 0 || th_ <= 0) return fail(MG_ERR_ARG, "thumbnail size must be positive");
  n = n_images;
  tw = tw_;
  th = th_;
  std::vector<int32_t> t;
  ResizeWeights weights;
  std::map<int, int> wtab, htab;  // source width / height -> table offset
  std::vector<ResizeImage> im((size_t)n);
  int dev = 0;
  ResizeShape shape{(double)n, 0.0, 0.0, (double)tw, (double)th, 0};
  MG_CUDA(cudaGetDevice(&dev));
  MG_CUDA(cudaDeviceGetAttribute(&shape.sms, cudaDevAttrMultiProcessorCount, dev));
  for (int i = 0; i < n; ++i) {
    shape.w += (double)regions[i].w / n;
    shape.h += (double)regions[i].h / n;
  }
  bands = choose_bands(shape, over_link);
  fused = bands > 0;
  MG_CHECK(build_images(regions, weights, t, wtab, htab, im));
  if (fused) fused = plan_fused(t, wtab, htab);
  if (!fused && bands > 0) {
    t.clear();
    wtab.clear();
    htab.clear();
    MG_CHECK(build_images(regions, weights, t, wtab, htab, im));
  }
  if (t.empty()) t.push_back(0);
  MG_CHECK(tabs.ensure(sizeof(int32_t) * t.size()));
  MG_CHECK(images.ensure(sizeof(ResizeImage) * im.size()));
  if (!fused) MG_CHECK(inter.ensure((size_t)n * max_h * tw * 3));
  MG_CUDA(cudaMemcpyAsync(tabs.p, t.data(), sizeof(int32_t) * t.size(), cudaMemcpyHostToDevice, s));
  // (from pageable memory: the sources are staged before the calls return)
  MG_CUDA(cudaMemcpyAsync(images.p, im.data(), sizeof(ResizeImage) * im.size(), cudaMemcpyHostToDevice, s));
  return MG_OK;
}

void ResizePlan::release() {
  tabs.release();
  images.release();
  inter.release();
  n = 0;
}

int launch_resize(const uint8_t* base, const ResizePlan& rp, uint8_t* out, cudaStream_t stream) {
  if (rp.n <= 0) return MG_OK;
  if (rp.fused) {
    const size_t bytes = 4 * ((size_t)rp.hw_words + rp.vw_words + rp.src_words + 3 * (size_t)rp.tw * rp.inter_pitch);
    if (bytes > 48 * 1024)
      MG_CUDA(cudaFuncSetAttribute(resize_fused_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kMaxFusedWords));
    resize_fused_kernel<<<dim3((unsigned)rp.n, (unsigned)rp.bands), kFusedThreads, bytes, stream>>>(
        base, rp.images.as<ResizeImage>(), rp.tabs.as<int32_t>(), rp.tw, rp.th, rp.hw_words, rp.vw_words, rp.src_words,
        rp.inter_pitch, out);
    g_launches += 1;
    MG_CUDA(cudaGetLastError());
    return MG_OK;
  }
  const int64_t pitch = (int64_t)rp.max_h * rp.tw * 3;
  const unsigned ys = (unsigned)std::min(16, std::max(1, (rp.max_h * rp.tw + 255) / 256));
  resize_h_kernel<<<dim3((unsigned)rp.n, ys), 256, 0, stream>>>(base, rp.images.as<ResizeImage>(), rp.tabs.as<int32_t>(),
                                                                 rp.tw, rp.inter.as<uint8_t>(), pitch);
  const unsigned yv = (unsigned)std::min(16, std::max(1, (rp.th * rp.tw + 255) / 256));
  resize_v_kernel<<<dim3((unsigned)rp.n, yv), 256, 0, stream>>>(rp.images.as<ResizeImage>(), rp.tabs.as<int32_t>(), rp.tw,
                                                                 rp.th, rp.inter.as<uint8_t>(), pitch, out);
  g_launches += 2;
  MG_CUDA(cudaGetLastError());
  return MG_OK;
}

}  // namespace mg
