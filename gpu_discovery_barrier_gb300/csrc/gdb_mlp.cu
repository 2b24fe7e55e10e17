// Schedule selector: loading the network, and its training on the GPU.
//
// Training is full-batch Adam over a masked squared loss.  One step is two
// kernels:
//   k_mlp_grad  a CTA takes tiles of up to 128 samples: forward and backward pass
//               into shared memory, then the tile's share of every gradient
//               entry from there (register tiles of 4 x 4 entries), kept in
//               FP64 registers from tile to tile;
//   k_mlp_step  one warp per gradient entry: the CTAs' sums in a fixed order
//               in FP64, then the Adam update of that parameter.
// Tiles, lanes and sums have a fixed order, so gradients are bit-identical
// from run to run.
#include <algorithm>
#include <cmath>
#include <vector>

#include "gdb_internal.h"
#include "gdb_selector.cuh"
#include "gdb_sweep.cuh"

using namespace gdbi;
using namespace gdb;

namespace {

// Gradient entries: W1, b1, W2, b2, W3, b3 (the blob minus shift/scale), then the loss.
constexpr int kGradEntries = kParams - kPW1;

__device__ __forceinline__ void mlp_thread(const float* p, const float* x, float* xn, float* h1,
                                           float* h2, float* y) {
  for (int i = 0; i < kFeat; ++i) xn[i] = __fmul_rn(__fsub_rn(x[i], p[kPShift + i]), p[kPScale + i]);
  for (int j = 0; j < kH1; ++j) {
    float h = p[kPB1 + j];
    for (int i = 0; i < kFeat; ++i) h = __fmaf_rn(xn[i], p[kPW1 + i * kH1 + j], h);
    h1[j] = fmaxf(h, 0.f);
  }
  for (int j = 0; j < kH2; ++j) {
    float h = p[kPB2 + j];
    for (int k = 0; k < kH1; ++k) h = __fmaf_rn(h1[k], p[kPW2 + k * kH2 + j], h);
    h2[j] = fmaxf(h, 0.f);
  }
  for (int j = 0; j < kOut; ++j) {
    float o = p[kPB3 + j];
    for (int k = 0; k < kH2; ++k) o = __fmaf_rn(h2[k], p[kPW3 + k * kOut + j], o);
    y[j] = o;
  }
}

__global__ void k_mlp_forward(const float* __restrict__ p, const float* __restrict__ X, uint32_t n,
                              float* __restrict__ Y) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  float x[kFeat], xn[kFeat], h1[kH1], h2[kH2], y[kOut];
  for (int i = 0; i < kFeat; ++i) x[i] = X[(size_t)s * kFeat + i];
  mlp_thread(p, x, xn, h1, h2, y);
  for (int j = 0; j < kOut; ++j) Y[(size_t)s * kOut + j] = y[j];
}

// Sum of the mask, in FP64 with a fixed order: one partial per CTA here,
// the CTAs' partials in order in mask_inverse.
constexpr int kMaskCtas = 64;
__global__ void k_mask_sum(const float* __restrict__ m, size_t count, double* __restrict__ part) {
  __shared__ double warp[8];
  double a = 0.0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x)
    a += (double)m[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if ((threadIdx.x & 31) == 0) warp[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) a += warp[w];
    part[blockIdx.x] = a;
  }
}

// Rows of a tile's activations in shared memory (kTile samples each): the
// normalised features, both hidden layers, their back-propagated errors,
// the output errors and the samples' losses.
constexpr int kTile = 128;
constexpr int kPitch = kTile + 4;  // rows 16-byte aligned, eight neighbouring rows on distinct banks
constexpr int kRXn = 0, kRH1 = kRXn + kFeat, kRH2 = kRH1 + kH1, kRDh1 = kRH2 + kH2, kRDh2 = kRDh1 + kH1,
              kRDy = kRDh2 + kH2, kRLoss = kRDy + kOut, kRows = kRLoss + 1;
constexpr int kMlpThreads = 256;
constexpr int kMlpSmem = (kRows * kPitch + ((kRows + 3) & ~3) + ((kParams + 3) & ~3)) * 4;
static_assert(kPW1 % 4 == 0 && kPW2 % 4 == 0, "weight rows are read as float4");

// Largest magnitude of a product or column value that a run of floats takes
// (2^32 values on 304 CTAs stay below 1e36), and the tiles of
// a run of products.
constexpr float kRunMax = 1e28f;
constexpr uint32_t kRunTiles = 8;

// Forward pass, errors and gradient sums of the CTA's tiles.  The gradient
// is the contraction of activation rows with error rows over the samples.
// It was one warp per entry with an FP64 FMA per (entry, sample) and both
// rows re-read from L2: 135,000 samples took 1.9 ms a step, bound by the
// FP64 pipe and the 1,694 x 2 row reads.  Here
//  * the rows stay in shared memory: a thread holds 4 x 4 entries and reads
//    eight 16-byte row pieces per four samples; tiles' rows interleave (t,
//    t + 8, ...), so a warp's eight distinct rows fall on distinct banks;
//  * FP64's place is taken by pairs of floats (Ogita, Rump, Oishi, "Accurate
//    sum and dot product", SIAM J. Sci. Comput. 26(6), 2005): p = a b and its
//    error fma(a, b, -p), hi + p and its error, both errors into lo.  Ten
//    FP32 operations per product, each exact but the adds into lo: measured
//    against 64 bits, a run of 64 products is within 2^-43 of the sum of
//    their magnitudes and one of 1,024 within 2^-39, whatever the rows' other
//    values are, and rounded to a float both are what FP64 sums give
//    (products below 2^-102 lose up to 2^-150 each).  Runs of kRunTiles tiles
//    go to FP64 sums in global memory.  The column sums (biases, loss) are
//    triples, beyond FP64's 53 bits.
//    Where a product or a value could bring a run near the floats' range, or
//    is not finite, the thread takes its tile in FP64 instead.
// 135,000 samples: 1.9 -> 0.17 ms a step, k_mlp_step included.
__global__ void __launch_bounds__(kMlpThreads, 2)
    k_mlp_grad(const float* __restrict__ p, const float* __restrict__ X, const float* __restrict__ T,
               const float* __restrict__ M, uint32_t n, uint32_t span, const float* __restrict__ inv_mask,
               double* __restrict__ part) {
  extern __shared__ float4 mlp_smem[];
  float* act = reinterpret_cast<float*>(mlp_smem);  // [kRows][kPitch]
  float* top = act + kRows * kPitch;                // [kRows] largest magnitude of a row
  float* sp = top + ((kRows + 3) & ~3);             // the parameters
  const int tid = threadIdx.x;
  const float inv_m = __ldg(inv_mask);
  for (int i = tid; i < kParams; i += kMlpThreads) sp[i] = __ldg(&p[i]);

  // phase 1 takes two samples and a quarter of each layer per thread
  const int quarter = (tid >> 6) * 8, sa = tid & 63, sb = sa + 64;

  // phase 2: 104 tiles of 4 x 4 entries, each over both halves of the
  // samples, on threads 0-207; the column sums (biases, loss) on the rest
  const bool tiled = tid < 208;
  int half, a0, as, d0, ds, out0, outw, ocol, nd = 4;
  if (tid < 128) {  // W2: h1 x dh2
    const int t = tid & 63;
    half = tid >> 6;
    a0 = kRH1 + (t >> 3), as = 8, d0 = kRDh2 + (t & 7), ds = 8;
    out0 = kPW2 + (t >> 3) * kH2 + (t & 7), outw = 8 * kH2, ocol = 8;
  } else if (tid < 176) {  // W1: xn x dh1
    const int t = (tid - 128) % 24;
    half = (tid - 128) / 24;
    a0 = kRXn + (t >> 3), as = 3, d0 = kRDh1 + (t & 7), ds = 8;
    out0 = kPW1 + (t >> 3) * kH1 + (t & 7), outw = 3 * kH1, ocol = 8;
  } else {  // W3: h2 x dy (three of the six columns; the last one is read twice)
    const int t = (tid - 176) & 15;
    half = ((tid - 176) >> 4) & 1;
    a0 = kRH2 + (t >> 1), as = 8, d0 = kRDy + (t & 1), ds = 2;
    out0 = kPW3 + (t >> 1) * kOut + (t & 1), outw = 8 * kOut, ocol = 2;
    nd = 3;
  }
  // error row of column j: its offset from row d0
  const int d3 = (nd - 1) * ds;
  auto drow = [&](int j) { return j < 3 ? j * ds : d3; };
  const int colr0 = tid - 208, colr1 = colr0 + 48;  // column sums: rows of dh1, dh2, dy, loss from kRDh1
  constexpr int kCols = kRows - kRDh1;
  // products: the run's pair of entry 4 i + j; columns: hi[k], lo[k], hi[2 + k]
  // are column k's triple
  float hi[16], lo[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) hi[i] = lo[i] = 0.f;
  // part[entry][slot]: two slots per CTA, one per half of the samples.  put
  // adds a sum to this thread's slot of an entry; `begun`: slots hold one
  const size_t slots = 2 * (size_t)gridDim.x;
  double* mine = part + 2 * blockIdx.x + (tiled ? half : 0);
  bool begun = false;
  auto put = [&](int entry, double x) {
    double* o = mine + (size_t)entry * slots;
    *o = begun ? *o + x : x;
  };
  auto entry = [&](int i, int j) { return out0 - kPW1 + i * outw + j * ocol; };
  // column c's entry: dh1, dh2 and dy are the biases; the loss is the last one
  auto column = [&](int c) {
    const int e = c < kH1 ? kPB1 + c : c < kH1 + kH2 ? kPB2 + c - kH1
                : c < kH1 + kH2 + kOut ? kPB3 + c - kH1 - kH2 : kParams;
    return e - kPW1;
  };
  auto end_run = [&] {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int e = 4 * i + j;
        if (j < nd) put(entry(i, j), (double)hi[e] + (double)lo[e]);
        hi[e] = lo[e] = 0.f;
      }
    begun = true;
  };
  uint32_t run = 0;

  const int halfspan = (int)span / 2;
  for (uint32_t tile = blockIdx.x; (size_t)tile * span < n; tile += gridDim.x) {
    const size_t base = (size_t)tile * span;
    const uint32_t have = n - base < (size_t)span ? (uint32_t)(n - base) : span;
    // targets and masks of thread tid < 128's sample, in flight early
    float tt[kOut], mm[kOut];
    if (tid < kTile) {
#pragma unroll
      for (int j = 0; j < kOut; ++j) {
        tt[j] = (uint32_t)tid < have ? __ldg(&T[(base + tid) * kOut + j]) : 0.f;
        mm[j] = (uint32_t)tid < have ? __ldg(&M[(base + tid) * kOut + j]) : 0.f;
      }
    }
    __syncthreads();  // the previous tile's rows (and the parameters) are done with (in place)
    for (int i = tid; i < kTile * kFeat; i += kMlpThreads) {
      const int s = i / kFeat, f = i - s * kFeat;
      act[(kRXn + f) * kPitch + s] =
          (uint32_t)s < have ? __fmul_rn(__fsub_rn(__ldg(&X[base * kFeat + i]), sp[kPShift + f]), sp[kPScale + f])
                             : 0.f;
    }
    __syncthreads();
    // one layer: outputs quarter .. quarter + 7 of both samples
    auto layer = [&](int rin, int nin, const float* w, const float* bias, int rout) {
      float ha[8], hb[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) ha[j] = hb[j] = bias[quarter + j];
#pragma unroll 4
      for (int i = 0; i < nin; ++i) {
        const float xa = act[(rin + i) * kPitch + sa], xb = act[(rin + i) * kPitch + sb];
        const float4 w0 = *reinterpret_cast<const float4*>(&w[i * 32 + quarter]);
        const float4 w1 = *reinterpret_cast<const float4*>(&w[i * 32 + quarter + 4]);
        const float wj[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          ha[j] = __fmaf_rn(xa, wj[j], ha[j]);
          hb[j] = __fmaf_rn(xb, wj[j], hb[j]);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        act[(rout + quarter + j) * kPitch + sa] = fmaxf(ha[j], 0.f);
        act[(rout + quarter + j) * kPitch + sb] = fmaxf(hb[j], 0.f);
      }
      __syncthreads();
    };
    layer(kRXn, kFeat, sp + kPW1, sp + kPB1, kRH1);
    layer(kRH1, kH1, sp + kPW2, sp + kPB2, kRH2);
    if (tid < kTile) {
      float y[kOut];
#pragma unroll
      for (int j = 0; j < kOut; ++j) y[j] = sp[kPB3 + j];
#pragma unroll 4
      for (int k = 0; k < kH2; ++k) {
        const float h = act[(kRH2 + k) * kPitch + tid];
#pragma unroll
        for (int j = 0; j < kOut; ++j) y[j] = __fmaf_rn(h, sp[kPW3 + k * kOut + j], y[j]);
      }
      float loss = 0.f;
#pragma unroll
      for (int j = 0; j < kOut; ++j) {
        const float e = y[j] - tt[j];
        act[(kRDy + j) * kPitch + tid] = mm[j] != 0.f ? 2.f * mm[j] * e * inv_m : 0.f;
        if (mm[j] != 0.f) loss = __fmaf_rn(mm[j] * e, e * inv_m, loss);
      }
      act[kRLoss * kPitch + tid] = loss;
    }
    __syncthreads();
    // dh2 = W3 . dy and dh1 = W2 . dh2, each masked by its ReLU
    {
      float da[kOut], db[kOut];
#pragma unroll
      for (int j = 0; j < kOut; ++j) {
        da[j] = act[(kRDy + j) * kPitch + sa];
        db[j] = act[(kRDy + j) * kPitch + sb];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = quarter + i;
        float a = 0.f, b = 0.f;
#pragma unroll
        for (int j = 0; j < kOut; ++j) {
          const float w = sp[kPW3 + k * kOut + j];
          a = __fmaf_rn(w, da[j], a);
          b = __fmaf_rn(w, db[j], b);
        }
        act[(kRDh2 + k) * kPitch + sa] = act[(kRH2 + k) * kPitch + sa] > 0.f ? a : 0.f;
        act[(kRDh2 + k) * kPitch + sb] = act[(kRH2 + k) * kPitch + sb] > 0.f ? b : 0.f;
      }
    }
    __syncthreads();
    {
      float a[8], b[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = b[i] = 0.f;
#pragma unroll 2
      for (int j = 0; j < kH2; j += 4) {
        float da[4], db[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          da[q] = act[(kRDh2 + j + q) * kPitch + sa];
          db[q] = act[(kRDh2 + j + q) * kPitch + sb];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 w = *reinterpret_cast<const float4*>(&sp[kPW2 + (quarter + i) * kH2 + j]);
          const float wq[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            a[i] = __fmaf_rn(wq[q], da[q], a[i]);
            b[i] = __fmaf_rn(wq[q], db[q], b[i]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = quarter + i;
        act[(kRDh1 + k) * kPitch + sa] = act[(kRH1 + k) * kPitch + sa] > 0.f ? a[i] : 0.f;
        act[(kRDh1 + k) * kPitch + sb] = act[(kRH1 + k) * kPitch + sb] > 0.f ? b[i] : 0.f;
      }
    }
    __syncthreads();
    for (int r = tid >> 5; r < kRows; r += kMlpThreads / 32) {
      const float4 v = *reinterpret_cast<const float4*>(&act[r * kPitch + 4 * (tid & 31)]);
      // magnitudes order as their bits do, NaN above infinity
      const uint32_t m = max(max(__float_as_uint(fabsf(v.x)), __float_as_uint(fabsf(v.y))),
                             max(__float_as_uint(fabsf(v.z)), __float_as_uint(fabsf(v.w))));
      const uint32_t w = __reduce_max_sync(0xffffffffu, m);
      if ((tid & 31) == 0) top[r] = __uint_as_float(w);
    }
    __syncthreads();
    if (tiled) {
      bool fits = true;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) fits = fits && top[a0 + i * as] * top[d0 + drow(j)] < kRunMax;
      const float* A = act + a0 * kPitch + halfspan * half;
      const float* D = act + d0 * kPitch + halfspan * half;
      if (fits) {
#pragma unroll 1
        for (int s = 0; s < halfspan; s += 4) {
          float av[4][4], dv[4][4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 x = *reinterpret_cast<const float4*>(A + i * as * kPitch + s);
            const float4 y = *reinterpret_cast<const float4*>(D + drow(i) * kPitch + s);
            av[i][0] = x.x, av[i][1] = x.y, av[i][2] = x.z, av[i][3] = x.w;
            dv[i][0] = y.x, dv[i][1] = y.y, dv[i][2] = y.z, dv[i][3] = y.w;
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const int e = 4 * i + j;
                const float t = __fmul_rn(av[i][q], dv[j][q]);
                float err;
                hi[e] = two_sum(hi[e], t, err);
                lo[e] = __fadd_rn(lo[e], __fadd_rn(err, __fmaf_rn(av[i][q], dv[j][q], -t)));
              }
        }
        if (++run == kRunTiles) {
          end_run();
          run = 0;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float *x = A + i * as * kPitch, *y = D + drow(j) * kPitch;
            double t = 0.0;
#pragma unroll 1
            for (int s = 0; s < halfspan && halfspan * half + s < (int)have; ++s) t += (double)x[s] * (double)y[s];
            if (j < nd) put(entry(i, j), t);
          }
        begun = true;
      }
    } else if (top[kRDh1 + colr0] < kRunMax && !(colr1 < kCols && !(top[kRDh1 + colr1] < kRunMax))) {
      const float* c0 = act + (kRDh1 + colr0) * kPitch;
      const float* c1 = act + (kRDh1 + (colr1 < kCols ? colr1 : colr0)) * kPitch;
#pragma unroll 4
      for (uint32_t s = 0; s < span; ++s)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          float e0, e1;
          hi[k] = two_sum(hi[k], k ? c1[s] : c0[s], e0);
          lo[k] = two_sum(lo[k], e0, e1);
          hi[2 + k] = __fadd_rn(hi[2 + k], e1);
        }
    } else {
#pragma unroll 1
      for (int k = 0; k < 2; ++k) {
        const int c = k ? colr1 : colr0;
        if (c >= kCols) break;
        const float* x = act + (kRDh1 + c) * kPitch;
        double t = 0.0;
        for (uint32_t s = 0; s < have; ++s) t += (double)x[s];
        put(column(c), t);
      }
      begun = true;
    }
  }
  if (tiled) {
    end_run();
  } else {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int c = k ? colr1 : colr0;
      if (c >= kCols) break;
      put(column(c), (double)hi[k] + ((double)lo[k] + (double)hi[2 + k]));
      mine[(size_t)column(c) * slots + 1] = 0.0;
    }
  }
}

// The CTAs' sums of one entry per warp, in a fixed order, then (m1 != null)
// the Adam update of its parameter.
__global__ void k_mlp_step(const double* __restrict__ part, int slots, float* __restrict__ grad,
                           double* __restrict__ loss, float* __restrict__ p, float* __restrict__ m1,
                           float* __restrict__ m2, float lr_t, float wd) {
  const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (e > kGradEntries) return;
  double acc = 0.0;
  for (int s = lane; s < slots; s += 32) acc += part[(size_t)e * slots + s];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane != 0) return;
  if (e == kGradEntries) {
    *loss = acc;
    return;
  }
  const int i = kPW1 + e;
  if (!m1) {
    grad[i] = (float)acc;
    return;
  }
  const bool weight = i < kPB1 || (i >= kPW2 && i < kPB2) || (i >= kPW3 && i < kPB3);
  float gi = (float)acc;
  if (weight) gi += wd * p[i];
  m1[i] = 0.9f * m1[i] + 0.1f * gi;
  m2[i] = 0.999f * m2[i] + 0.001f * gi * gi;
  p[i] -= lr_t * m1[i] / (sqrtf(m2[i]) + 1e-8f);
}

// Device buffers of one training / gradient call.
struct MlpBufs {
  float *p = nullptr, *x = nullptr, *t = nullptr, *m = nullptr, *g = nullptr, *m1 = nullptr, *m2 = nullptr,
        *inv_mask = nullptr;
  double *loss = nullptr, *part = nullptr;
  char* base = nullptr;
  int ctas = 0;
  uint32_t span = kTile;  // samples of a CTA's tile
};

// 1 / sum of the mask (0 for an empty one).
__global__ void k_mask_inverse(const double* __restrict__ part, float* __restrict__ inv) {
  double s = 0.0;
  for (int i = 0; i < kMaskCtas; ++i) s += part[i];
  *inv = s > 0 ? (float)(1.0 / s) : 0.f;
}

int mlp_upload(gdb_ctx* c, MlpBufs& b, const float* params, const float* x, const float* t,
               const float* m, uint32_t n, bool adam) {
  // two CTAs per SM hold the tiles; fewer tiles take a CTA each.  A step on
  // few samples lasts as long as one tile's products, so they go in tiles of
  // 16, 32 or 64 while these are no more than the SMs; more tiles cost more
  // sums (20 epochs and a forward, tiles of 16 / 32 / 64 / 128: 1,000 samples
  // 0.58 / 0.62 / 0.71 / 0.87 ms, 4,000 0.83 / 0.70 / 0.75 / 0.91, 6,000 0.95 /
  // 0.83 / 0.75 / 0.91, 10,000 1.16 / 1.00 / 0.89 / 0.92, 20,000 1.61 / 1.30 /
  // 1.20 / 1.19)
  b.span = 16;
  while (b.span < (uint32_t)kTile && (uint64_t)b.span * c->sm_count < n) b.span *= 2;
  b.ctas = (int)std::min<uint64_t>(2ull * c->sm_count, ((uint64_t)n + b.span - 1) / b.span);
  GDB_CUDA(c, cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, kMlpSmem));
  Bump bp;
  const size_t o_p = bp.take(kParams * 4), o_x = bp.take((size_t)n * kFeat * 4),
               o_t = bp.take((size_t)n * kOut * 4), o_m = bp.take((size_t)n * kOut * 4),
               o_g = bp.take(kParams * 4), o_m1 = bp.take(adam ? kParams * 4 : 0),
               o_m2 = bp.take(adam ? kParams * 4 : 0), o_l = bp.take(8), o_i = bp.take(4),
               o_s = bp.take((size_t)std::max((kGradEntries + 1) * 2 * b.ctas, kMaskCtas) * 8);
  GDB_CUDA(c, cudaMallocAsync((void**)&b.base, bp.off, c->stream));
  b.p = (float*)(b.base + o_p);
  b.x = (float*)(b.base + o_x);
  b.t = (float*)(b.base + o_t);
  b.m = (float*)(b.base + o_m);
  b.g = (float*)(b.base + o_g);
  b.m1 = adam ? (float*)(b.base + o_m1) : nullptr;
  b.m2 = adam ? (float*)(b.base + o_m2) : nullptr;
  b.loss = (double*)(b.base + o_l);
  b.inv_mask = (float*)(b.base + o_i);
  b.part = (double*)(b.base + o_s);
  GDB_CUDA(c, cudaMemcpyAsync(b.p, params, kParams * 4, cudaMemcpyHostToDevice, c->stream));
  GDB_CUDA(c, cudaMemcpyAsync(b.m, m, (size_t)n * kOut * 4, cudaMemcpyHostToDevice, c->stream));
  k_mask_sum<<<kMaskCtas, 256, 0, c->stream>>>(b.m, (size_t)n * kOut, b.part);
  k_mask_inverse<<<1, 1, 0, c->stream>>>(b.part, b.inv_mask);
  GDB_CUDA(c, cudaGetLastError());
  GDB_CUDA(c, cudaMemcpyAsync(b.x, x, (size_t)n * kFeat * 4, cudaMemcpyHostToDevice, c->stream));
  GDB_CUDA(c, cudaMemcpyAsync(b.t, t, (size_t)n * kOut * 4, cudaMemcpyHostToDevice, c->stream));
  GDB_CUDA(c, cudaMemsetAsync(b.g, 0, kParams * 4, c->stream));
  if (adam) {
    GDB_CUDA(c, cudaMemsetAsync(b.m1, 0, kParams * 4, c->stream));
    GDB_CUDA(c, cudaMemsetAsync(b.m2, 0, kParams * 4, c->stream));
  }
  return GDB_OK;
}

// Gradient and loss, then the Adam update where b has its moments.
int mlp_step(gdb_ctx* c, MlpBufs& b, uint32_t n, float lr_t, float wd) {
  k_mlp_grad<<<b.ctas, kMlpThreads, kMlpSmem, c->stream>>>(b.p, b.x, b.t, b.m, n, b.span, b.inv_mask,
                                                         b.part);
  k_mlp_step<<<(kGradEntries + 1 + 7) / 8, 256, 0, c->stream>>>(b.part, 2 * b.ctas, b.g, b.loss, b.p, b.m1,
                                                                b.m2, lr_t, wd);
  GDB_CUDA(c, cudaGetLastError());
  return GDB_OK;
}

}  // namespace

extern "C" {

int gdb_selector_set(gdb_ctx* c, const float* params) {
  if (!c) return GDB_ERR_INVALID;
  if (!params) {
    if (c->d_mlp) cudaFree(c->d_mlp);
    c->d_mlp = nullptr;
    c->h_mlp.clear();
    return GDB_OK;
  }
  for (int i = 0; i < kParams; ++i)
    if (!std::isfinite(params[i])) return set_error(c, GDB_ERR_INVALID, "selector parameters not finite");
  if (!c->d_mlp) GDB_CUDA(c, cudaMalloc((void**)&c->d_mlp, kParams * 4));
  GDB_CUDA(c, cudaMemcpy(c->d_mlp, params, kParams * 4, cudaMemcpyHostToDevice));
  c->h_mlp.assign(params, params + kParams);
  return GDB_OK;
}

int gdb_mlp_forward(gdb_ctx* c, const float* params, const float* x, uint32_t n, float* y) {
  if (!c || !params || !x || !y) return GDB_ERR_INVALID;
  if (n == 0) return GDB_OK;
  char* d = nullptr;
  const size_t bp = kParams * 4, bx = (size_t)n * kFeat * 4, by = (size_t)n * kOut * 4;
  GDB_CUDA(c, cudaMallocAsync((void**)&d, bp + bx + by, c->stream));
  cudaError_t e = cudaMemcpyAsync(d, params, bp, cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d + bp, x, bx, cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess) {
    k_mlp_forward<<<(n + 127) / 128, 128, 0, c->stream>>>((float*)d, (float*)(d + bp), n,
                                                          (float*)(d + bp + bx));
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(y, d + bp + bx, by, cudaMemcpyDeviceToHost, c->stream);
  cudaFreeAsync(d, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  return e == cudaSuccess ? GDB_OK : set_cuda_error(c, e, "mlp forward");
}

int gdb_mlp_loss_grad(gdb_ctx* c, const float* params, const float* x, const float* t, const float* m,
                      uint32_t n, float* grad, double* loss) {
  if (!c || !params || !x || !t || !m || !grad || n == 0) return GDB_ERR_INVALID;
  MlpBufs b;
  int rc = mlp_upload(c, b, params, x, t, m, n, false);
  if (rc == GDB_OK) rc = mlp_step(c, b, n, 0.f, 0.f);
  cudaError_t e = cudaSuccess;
  if (rc == GDB_OK) {
    e = cudaMemcpyAsync(grad, b.g, kParams * 4, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess && loss) e = cudaMemcpyAsync(loss, b.loss, 8, cudaMemcpyDeviceToHost, c->stream);
  }
  if (b.base) cudaFreeAsync(b.base, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (rc == GDB_OK && e != cudaSuccess) rc = set_cuda_error(c, e, "mlp gradient");
  return rc;
}

int gdb_mlp_train(gdb_ctx* c, float* params, const float* x, const float* t, const float* m, uint32_t n,
                  uint32_t epochs, float lr, float wd, double* loss) {
  if (!c || !params || !x || !t || !m || n == 0 || !(lr > 0.f)) return GDB_ERR_INVALID;
  MlpBufs b;
  int rc = mlp_upload(c, b, params, x, t, m, n, true);
  double b1t = 1.0, b2t = 1.0;
  for (uint32_t k = 0; rc == GDB_OK && k < epochs; ++k) {
    b1t *= 0.9;
    b2t *= 0.999;
    rc = mlp_step(c, b, n, (float)(lr * std::sqrt(1.0 - b2t) / (1.0 - b1t)), wd);
  }
  cudaError_t e = cudaSuccess;
  if (rc == GDB_OK) {
    e = cudaMemcpyAsync(params, b.p, kParams * 4, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess && loss) e = cudaMemcpyAsync(loss, b.loss, 8, cudaMemcpyDeviceToHost, c->stream);
  }
  if (b.base) cudaFreeAsync(b.base, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (rc == GDB_OK && e != cudaSuccess) rc = set_cuda_error(c, e, "mlp training");
  return rc;
}

int gdb_sssp_features(gdb_ctx* c, gdb_graph* g, uint32_t nsrc, float* x) {
  if (!graph_ok(c, g) || !x || nsrc == 0) return GDB_ERR_INVALID;
  gdbi::sssp_features(c, g, nsrc, x);
  return GDB_OK;
}

}  // extern "C"

void gdbi::sssp_features(gdb_ctx* c, const gdb_graph* g, uint32_t nsrc, float* x) {
  const double V = g->V, E = (double)g->E;
  const double nf = std::min<double>(nsrc, V);
  const double mf = nf * E / std::max(V, 1.0);
  // warps of the launch as the network was trained: the traversal kernels'
  // resident CTAs, capped by max_ctas (small_shape's cut is not in the traces)
  double ctas = (double)c->sm_count * std::max(gdbi::traversal_occupancy(c, c->opt.block_size), 1);
  if (c->opt.max_ctas > 0) ctas = std::min(ctas, (double)c->opt.max_ctas);
  const double warps = ctas * (c->opt.block_size / 32);
  bfs_features(x, (float)nf, (float)mf, (float)std::max(E - mf, 0.0), (float)V, (float)E,
               (float)std::max(V - nf, 0.0), 0, 2, (float)g->maxdeg, (float)warps);
}
