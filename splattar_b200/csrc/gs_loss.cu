// Fused L1 + D-SSIM loss and its analytic gradient
// (first_attempt/crates/gs-train/src/shaders/ssim.wgsl:41-143,
// first_attempt/crates/gs-train/src/ssim.rs:236-280).
//
// The reference runs 19 full-image passes (products, 8 separable blurs of
// two dispatches each, partials, combine) through ~17 image-sized buffers.
// Here two tiled kernels cover every view of a step:
//   k_ssim_moments: per 16×16 tile, stage x and y with a 5-pixel halo in
//     shared memory, blur the five moments (μx, μy, x², y², xy) of the three
//     channels separably, form SSIM and the three coefficient maps Cμ, Cx²,
//     Cxy per channel (ssim.wgsl:94-126), stored as four float2 planes and
//     one float plane, and accumulate the per-view loss sums.
//   k_ssim_grad: stage the nine coefficient planes with a halo, blur them
//     (the zero-padded symmetric window is self-adjoint) and combine with the
//     L1 term into dL/dx (ssim.wgsl:130-143).
// L = w_l1·mean|x−y| + w_ssim·mean(1−S) over pixels × rgb of each view.
#include <algorithm>

#include "gs_common.cuh"
#include "gs_kernels.h"

namespace gs {
namespace {

// Output tiles of 16×16 pixels, inputs staged with a 5-pixel halo (26×26).
// Separable 11-tap blurs run as sliding windows in registers: a horizontal
// pass where each thread owns one (row, channel or plane) and slides along x,
// then a vertical pass where each thread owns one (column, channel or plane)
// and slides along y, so every staged value is read from shared memory once
// per pass. Pairs of maps blur together in the packed two-wide FP32
// instructions of sm_100 (FFMA2/FADD2/FMUL2): (μx, μy) and (E[x²], E[y²]) per
// channel in the moments kernel, two coefficient planes at a time in the
// gradient kernel; each component rounds as the scalar operation would.
constexpr int T16 = 16, HALO = 5, EXT = T16 + 2 * HALO;  // 26
constexpr int TAPS = 2 * HALO + 1;                       // 11
// Staged rows use an odd pitch (read by lanes holding consecutive rows; for
// 8-byte elements the two 16-lane phases then hit distinct banks), horizontal
// results an odd row pitch, vertical results dense 16×16 planes.
constexpr int IN_PITCH = EXT + 1;                        // 27
constexpr int H_ROW = T16 + 1;                           // 17
constexpr int H_PLANE = EXT * H_ROW;                     // 442
constexpr int V_PLANE = T16 * T16;                       // 256

struct TileLoc {
  int v, x0, y0, W, H;
  long long pix_base;
};

template <int TS = T16>
__device__ __forceinline__ TileLoc locate(const SsimArgs& a, int t) {
  TileLoc L;
  int v = 0, base = 0;
  for (;;) {
    const ViewInfo* V = a.views + v;
    const int W = __ldg(&V->width), H = __ldg(&V->height);
    const int nt = ((W + TS - 1) / TS) * ((H + TS - 1) / TS);
    if (t < base + nt || v + 1 == a.n_views) {
      const int lt = t - base, tx = (W + TS - 1) / TS;
      L.v = v; L.W = W; L.H = H;
      L.x0 = (lt % tx) * TS; L.y0 = (lt / tx) * TS;
      L.pix_base = __ldg(&V->pix_base);
      return L;
    }
    base += nt;
    ++v;
  }
}

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }

// Asynchronous copy of B bytes (4, 8 or 16; both addresses B-aligned) from
// global to shared memory; when !valid nothing is read and the B bytes are
// zero-filled. Completion: cp.async.wait_all, then a barrier for other threads.
template <int B>
__device__ __forceinline__ void cp_async_zfill(void* smem, const void* gmem, bool valid) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(s), "l"(gmem), "n"(B), "r"(valid ? B : 0)
               : "memory");
}

// Slides an 11-tap window along `N_OUT` outputs: out[o] = Σ_d w[|d−5|]·in(o+d)
// (w[k] is the weight at offset ±k), for a scalar map.
template <int N_OUT, class In, class Out>
__device__ __forceinline__ void slide11(const float (&w)[6], In in, Out out) {
  float win[TAPS];
#pragma unroll
  for (int i = 0; i < TAPS - 1; ++i) win[i] = in(i);
#pragma unroll
  for (int o = 0; o < N_OUT; ++o) {
    win[TAPS - 1] = in(o + TAPS - 1);
    float acc = w[0] * win[HALO];
#pragma unroll
    for (int d = 0; d < HALO; ++d) acc += w[HALO - d] * (win[d] + win[TAPS - 1 - d]);
    out(o, acc);
#pragma unroll
    for (int i = 0; i < TAPS - 1; ++i) win[i] = win[i + 1];
  }
}

// The same for two maps at once (float2 windows, packed instructions).
template <int N_OUT, class In, class Out>
__device__ __forceinline__ void slide11x2(const float (&w)[6], In in, Out out) {
  float2 win[TAPS];
#pragma unroll
  for (int i = 0; i < TAPS - 1; ++i) win[i] = in(i);
#pragma unroll
  for (int o = 0; o < N_OUT; ++o) {
    win[TAPS - 1] = in(o + TAPS - 1);
    float2 acc = __fmul2_rn(f2(w[0]), win[HALO]);
#pragma unroll
    for (int d = 0; d < HALO; ++d) acc = __ffma2_rn(f2(w[HALO - d]), __fadd2_rn(win[d], win[TAPS - 1 - d]), acc);
    out(o, acc);
#pragma unroll
    for (int i = 0; i < TAPS - 1; ++i) win[i] = win[i + 1];
  }
}

// Moments → SSIM, its coefficient maps and the per-view loss sums.
// Eight blurred maps, seven of them packed pairs: per channel (μx, μy) and
// (E[x²], E[y²]), then (E[xy]_r, E[xy]_g), and E[xy]_b scalar. Eight maps
// give 208 horizontal row items and 256 vertical items (16 columns, two
// halves of 8 rows), so both passes occupy the block in a single round.
// Coefficient planes (scratch, coef_stride pixels each): float2 planes
// (Cμ_r, Cμ_g), (Cx²_r, Cx²_g), (Cxy_r, Cxy_g), (Cμ_b, Cx²_b) at
// coef + 2k·stride, and Cxy_b at coef + 8·stride.
constexpr int NM2 = 7;  // packed maps
__global__ void __launch_bounds__(256) k_ssim_moments(SsimArgs a) {
  __shared__ float2 s_in[3][EXT][IN_PITCH];     // (x, y) per channel, with halo
  __shared__ float2 s_h2[NM2][EXT * H_ROW];     // horizontal results of the packed maps [map][row][col]
  __shared__ float s_h1[EXT * H_ROW];           // horizontal E[xy]_b
  __shared__ double s_red[2][8];
  // Vertical results reuse s_in after the horizontal pass.
  float2* s_v2 = &s_in[0][0][0];                          // [map][16×16]
  float* s_v1 = reinterpret_cast<float*>(s_v2 + NM2 * V_PLANE);  // [16×16]
  static_assert(NM2 * V_PLANE * 2 + V_PLANE <= 3 * EXT * IN_PITCH * 2, "vertical results fit in s_in");
  const int tid = threadIdx.x;
  const TileLoc L = locate(a, blockIdx.x);
  for (int k = tid; k < EXT * EXT; k += 256) {
    const int ly = k / EXT, lx = k % EXT;
    const int gx = L.x0 + lx - HALO, gy = L.y0 + ly - HALO;
    float4 xv = make_float4(0, 0, 0, 0), yv = xv;
    if (gx >= 0 && gy >= 0 && gx < L.W && gy < L.H) {
      const long long p = L.pix_base + (long long)gy * L.W + gx;
      xv = a.img[p];
      yv = a.target[p];
    }
    s_in[0][ly][lx] = make_float2(xv.x, yv.x);
    s_in[1][ly][lx] = make_float2(xv.y, yv.y);
    s_in[2][ly][lx] = make_float2(xv.z, yv.z);
  }
  float w[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) w[k] = a.w[k];
  __syncthreads();
  // Horizontal: warp m blurs map m, lane r < EXT row r, so each warp runs one
  // of the four code paths (an item order that put two maps in a warp ran
  // both paths with half the lanes each).
  static_assert(NM2 + 1 == 8 && EXT <= 32, "one warp per map, one lane per staged row");
  if ((tid & 31) < EXT) {
    const int m = tid >> 5, r = tid & 31;
    if (m < 6) {
      const float2* XY = &s_in[m >> 1][r][0];
      float2* O = &s_h2[m][r * H_ROW];
      if (m & 1)
        slide11x2<T16>(w, [&](int i) { const float2 v = XY[i]; return __fmul2_rn(v, v); }, [&](int o, float2 v) { O[o] = v; });
      else
        slide11x2<T16>(w, [&](int i) { return XY[i]; }, [&](int o, float2 v) { O[o] = v; });
    } else if (m == 6) {
      const float2* R = &s_in[0][r][0];
      const float2* G = &s_in[1][r][0];
      float2* O = &s_h2[6][r * H_ROW];
      slide11x2<T16>(w, [&](int i) { const float2 u = R[i], v = G[i]; return make_float2(u.x * u.y, v.x * v.y); },
                     [&](int o, float2 v) { O[o] = v; });
    } else {
      const float2* B = &s_in[2][r][0];
      float* O = &s_h1[r * H_ROW];
      slide11<T16>(w, [&](int i) { const float2 v = B[i]; return v.x * v.y; }, [&](int o, float v) { O[o] = v; });
    }
  }
  // L1 of this thread's pixel, read before s_in is reused.
  const int ox = tid & 15, oy = tid >> 4;
  const int gx = L.x0 + ox, gy = L.y0 + oy;
  const bool inside = gx < L.W && gy < L.H;
  float l1 = 0.f;
#pragma unroll
  for (int ch = 0; ch < 3; ++ch) {
    const float2 v = s_in[ch][oy + HALO][ox + HALO];
    if (inside) l1 += fabsf(v.x - v.y);
  }
  __syncthreads();
  // Vertical: item = (map, column, half): rows 8h..8h+7 from input rows 8h..8h+17.
  {
    const int m = tid >> 5, c = tid & 15, h = (tid >> 4) & 1;
    if (m < NM2) {
      const float2* I = &s_h2[m][c + 8 * h * H_ROW];
      float2* O = s_v2 + m * V_PLANE + c + 8 * h * T16;
      slide11x2<8>(w, [&](int i) { return I[i * H_ROW]; }, [&](int o, float2 v) { O[o * T16] = v; });
    } else {
      const float* I = &s_h1[c + 8 * h * H_ROW];
      float* O = s_v1 + c + 8 * h * T16;
      slide11<8>(w, [&](int i) { return I[i * H_ROW]; }, [&](int o, float v) { O[o * T16] = v; });
    }
  }
  __syncthreads();
  float ss = 0.f;
  if (inside) {
    const long long pix = L.pix_base + (long long)gy * L.W + gx;
    const float inv_n3 = 1.0f / (3.0f * (float)L.W * (float)L.H);
    const float C1 = 1e-4f, C2 = 9e-4f;
    const float dw = -a.w_ssim * inv_n3;
    float cm[3], cx2[3], cxy[3];
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
      const int q = oy * T16 + ox;
      const float2 mu = s_v2[(ch * 2) * V_PLANE + q], b2 = s_v2[(ch * 2 + 1) * V_PLANE + q];
      const float bxy = ch == 0 ? s_v2[6 * V_PLANE + q].x : (ch == 1 ? s_v2[6 * V_PLANE + q].y : s_v1[q]);
      const float mu_x = mu.x, mu_y = mu.y;
      const float sx2 = b2.x - mu_x * mu_x, sy2 = b2.y - mu_y * mu_y, sxy = bxy - mu_x * mu_y;
      const float p = mu_x * mu_x + mu_y * mu_y + C1;
      const float qd = sx2 + sy2 + C2;
      // p >= C1 and qd ~>= C2: one approximate reciprocal each (about 1 ulp)
      // replaces the four IEEE divisions of the expressions.
      const float ip = __fdividef(1.0f, p), iq = __fdividef(1.0f, qd);
      const float l = (2.0f * mu_x * mu_y + C1) * ip;
      const float cs = (2.0f * sxy + C2) * iq;
      ss += l * cs;
      cm[ch] = (cs * (2.0f * mu_y - 2.0f * mu_x * l) * ip + l * (-2.0f * mu_y + 2.0f * mu_x * cs) * iq) * dw;
      cx2[ch] = (-l * cs * iq) * dw;
      cxy[ch] = (2.0f * l * iq) * dw;
    }
    float2* P2 = reinterpret_cast<float2*>(a.coef);
    const size_t st2 = a.coef_stride;  // float2 plane k starts at float offset 2k·stride
    P2[0 * st2 + pix] = make_float2(cm[0], cm[1]);
    P2[1 * st2 + pix] = make_float2(cx2[0], cx2[1]);
    P2[2 * st2 + pix] = make_float2(cxy[0], cxy[1]);
    P2[3 * st2 + pix] = make_float2(cm[2], cx2[2]);
    a.coef[8 * a.coef_stride + pix] = cxy[2];
  }
  // Per-view loss sums: warp, then block, then one double atomic each.
  double dl1 = warp_sum(l1), dss = warp_sum(ss);
  if ((tid & 31) == 0) { s_red[0][tid >> 5] = dl1; s_red[1][tid >> 5] = dss; }
  __syncthreads();
  if (tid == 0) {
    double t0 = 0, t1 = 0;
    for (int k = 0; k < 8; ++k) { t0 += s_red[0][k]; t1 += s_red[1][k]; }
    atomicAdd(a.loss_sums + 2 * L.v, t0);
    atomicAdd(a.loss_sums + 2 * L.v + 1, t1);
  }
}

// Blur of the nine coefficient maps (the zero-padded symmetric window is
// self-adjoint) combined with the L1 term into dL/dx: four float2 planes
// blurred as packed pairs and one scalar plane.
#ifndef GS_SSIM_GRAD_INPLACE
#define GS_SSIM_GRAD_INPLACE 1
#endif
__global__ void __launch_bounds__(256, GS_SSIM_GRAD_INPLACE ? 6 : 1) k_ssim_grad(SsimArgs a) {
  __shared__ float2 s_c2[4][EXT][IN_PITCH];
  __shared__ float s_c1[EXT][IN_PITCH];
  // In place, the horizontal pass writes each row's 16 results over the row's
  // first 16 staged values (a row belongs to one thread, and output o is
  // written after input o + 10 has been read), so the vertical results get a
  // buffer of their own and the block needs 34.5 KB of shared memory instead
  // of 41.2 KB: 6 resident blocks per SM instead of 5.
  constexpr bool INPL = GS_SSIM_GRAD_INPLACE;
  constexpr int HP = INPL ? IN_PITCH : H_ROW;  // row pitch of the horizontal results
  __shared__ float2 s_h2b[INPL ? 1 : 4][INPL ? 1 : EXT * H_ROW];
  __shared__ float s_h1b[INPL ? 1 : EXT * H_ROW];
  __shared__ float2 s_vb[INPL ? 4 * V_PLANE + V_PLANE / 2 : 1];
  auto s_h2 = [&](int m) -> float2* { return INPL ? &s_c2[m][0][0] : &s_h2b[INPL ? 0 : m][0]; };
  float* s_h1 = INPL ? &s_c1[0][0] : s_h1b;
  float2* s_v2 = INPL ? s_vb : &s_c2[0][0][0];                      // [4][16×16]
  float* s_v1 = reinterpret_cast<float*>(s_v2 + 4 * V_PLANE);        // [16×16]
  static_assert(4 * V_PLANE * 2 + V_PLANE <= 4 * EXT * IN_PITCH * 2, "vertical results fit in s_c2");
  const int tid = threadIdx.x;
  const TileLoc L = locate(a, blockIdx.x);
  // This thread's pixel of the image and target, loaded now so the loads are
  // in flight during the blurs.
  const int ox = tid & 15, oy = tid >> 4;
  const int gx = L.x0 + ox, gy = L.y0 + oy;
  const bool inside = gx < L.W && gy < L.H;
  const long long pix = inside ? L.pix_base + (long long)gy * L.W + gx : 0;
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
  if (inside) {
    x = a.img[pix];
    y = a.target[pix];
  }
  const float2* P2 = reinterpret_cast<const float2*>(a.coef);
  const size_t st2 = a.coef_stride;
  // Staged with asynchronous copies (global -> shared, no registers), so all
  // of a thread's loads are in flight at once; pixels outside the view are
  // zero-filled by the copy (source size 0).
  for (int k = tid; k < EXT * EXT; k += 256) {
    const int ly = k / EXT, lx = k % EXT;
    const int gx = L.x0 + lx - HALO, gy = L.y0 + ly - HALO;
    const bool in = gx >= 0 && gy >= 0 && gx < L.W && gy < L.H;
    const size_t p = in ? (size_t)(L.pix_base + (long long)gy * L.W + gx) : 0;
#pragma unroll
    for (int m = 0; m < 4; ++m) cp_async_zfill<8>(&s_c2[m][ly][lx], P2 + m * st2 + p, in);
    cp_async_zfill<4>(&s_c1[ly][lx], a.coef + 8 * a.coef_stride + p, in);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  float w[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) w[k] = a.w[k];
  __syncthreads();
  // Horizontal: warp m < 5 blurs plane m, lane r < EXT row r (one code path per warp).
  if (tid < 5 * 32 && (tid & 31) < EXT) {
    const int m = tid >> 5, r = tid & 31;
    if (m < 4) {
      const float2* X = &s_c2[m][r][0];
      float2* O = s_h2(m) + r * HP;
      slide11x2<T16>(w, [&](int i) { return X[i]; }, [&](int o, float2 v) { O[o] = v; });
    } else {
      const float* X = &s_c1[r][0];
      float* O = s_h1 + r * HP;
      slide11<T16>(w, [&](int i) { return X[i]; }, [&](int o, float v) { O[o] = v; });
    }
  }
  __syncthreads();
  // Vertical: item = (map, column, segment), segments of 6 rows starting at
  // rows 0, 5 and 10 (rows 5 and 10 are computed twice, identically).
  if (tid < 5 * T16 * 3) {
    const int m = tid / (3 * T16), rem = tid - m * 3 * T16, sg = rem / T16, c = rem - sg * T16;
    const int r0 = 5 * sg;
    if (m < 4) {
      const float2* I = s_h2(m) + c + r0 * HP;
      float2* O = s_v2 + m * V_PLANE + c + r0 * T16;
      slide11x2<6>(w, [&](int i) { return I[i * HP]; }, [&](int o, float2 v) { O[o * T16] = v; });
    } else {
      const float* I = s_h1 + c + r0 * HP;
      float* O = s_v1 + c + r0 * T16;
      slide11<6>(w, [&](int i) { return I[i * HP]; }, [&](int o, float v) { O[o * T16] = v; });
    }
  }
  __syncthreads();
  if (!inside) return;
  const float k1 = a.w_l1 / (3.0f * (float)L.W * (float)L.H);
  const int q = oy * T16 + ox;
  const float2 vm = s_v2[0 * V_PLANE + q], vx2 = s_v2[1 * V_PLANE + q], vxy = s_v2[2 * V_PLANE + q];
  const float2 vb = s_v2[3 * V_PLANE + q];
  const float vxy_b = s_v1[q];
  const float cmu[3] = {vm.x, vm.y, vb.x}, cx2[3] = {vx2.x, vx2.y, vb.y}, cxy[3] = {vxy.x, vxy.y, vxy_b};
  const float xs[3] = {x.x, x.y, x.z}, ys[3] = {y.x, y.y, y.z};
  float out[3];
#pragma unroll
  for (int ch = 0; ch < 3; ++ch) {
    const float diff = xs[ch] - ys[ch];
    const float sg = diff > 0.f ? 1.f : (diff < 0.f ? -1.f : 0.f);
    out[ch] = sg * k1 + cmu[ch] + 2.0f * xs[ch] * cx2[ch] + ys[ch] * cxy[ch];
  }
  a.dl_dcolor[pix] = make_float4(out[0], out[1], out[2], 0.f);
}

// ---- k_ssim_moments on 32×32 tiles, for images of many tiles (launch_ssim) ----
// A 16×16 tile reads 2.64 pixels and blurs 1.63 rows per output; a 32×32 tile
// 1.72 and 1.31. Planes and results are laid out alike. Bound by the latency
// of staging at two blocks (24 warps) per SM.
constexpr int T32 = 32, EXT32 = T32 + 2 * HALO;  // 42
constexpr int BIG_PITCH = EXT32 + 1;             // 43: odd, as IN_PITCH
constexpr int BIG_ROW = T32 + 1;                 // 33
constexpr int BM_THREADS = 384;                  // 3 channels × 4 row segments × 32 columns
constexpr size_t BM_SMEM = sizeof(float2) * (3 * EXT32 * BIG_PITCH + 6 * EXT32 * BIG_ROW);
// Two packed maps per channel: (μx, μy) and (E[x² + y²], E[xy]); SSIM needs
// the two variances as a sum only, so four maps do where five were blurred.
// x and y are shifted by one value per tile and channel (tile_shift; outside
// the image too), which leaves variances and covariances as they are and shrinks
// the squares that cancel in them; L1 is summed from the unshifted values. A
// vertical item slides both maps of its channel down 8 rows and forms that
// channel's coefficients from registers.
constexpr int BM_LOADS = (EXT32 * EXT32 + BM_THREADS - 1) / BM_THREADS;  // staged pixels per thread

// Mean of 8 × 4 sampled pixels of the tile, dark pixels and those like their
// diagonal neighbour counting most: SSIM is most sensitive to rounding where
// the variance is small beside C2, and a dark flat background must not be
// shifted by a bright or busy object in the same tile. The gradient's relative
// error against 64 bits, 16-pixel tiles unshifted, here, and with a fixed 0.5:
// smooth mid-tones 6.9e-6, 1.6e-6, 2.5e-6; values up to 0.05 2.4e-7, 2.4e-7,
// 7.3e-6; objects on black 2.8e-7, 3.2e-7, 2.9e-6 (1.7e-6 with the plain mean).
// Called by whole warps.
__device__ __forceinline__ float tile_shift(const SsimArgs& a, const TileLoc& L, int lane, int ch) {
  const int x0 = min(L.x0 + 2 + 4 * (lane & 7), L.W - 1), y0 = min(L.y0 + 4 + 8 * (lane >> 3), L.H - 1);
  const int x1 = min(x0 + 1, L.W - 1), y1 = min(y0 + 1, L.H - 1);
  const long long p = 4 * (L.pix_base + (long long)y0 * L.W + x0) + ch;
  const long long q = 4 * (L.pix_base + (long long)y1 * L.W + x1) + ch;
  const float* img = &a.img->x;
  const float* target = &a.target->x;
  const float x = img[p], y = target[p], dx = x - img[q], dy = y - target[q], m = 0.5f * (x + y);
  const float w = __fdividef(1.0f, (9e-4f + dx * dx + dy * dy) * (0.1f + m * m));
  const float s = __fdividef(warp_sum(w * m), warp_sum(w));
  return fabsf(s) < 1e15f ? s : 0.f;  // (no shift beside NaN and infinities)
}
__global__ void __launch_bounds__(BM_THREADS, 2) k_ssim_moments_big(SsimArgs a) {
  extern __shared__ __align__(16) unsigned char big_smem[];
  float2* s_in = reinterpret_cast<float2*>(big_smem);       // [ch][EXT32][BIG_PITCH]
  float2* s_h = s_in + 3 * EXT32 * BIG_PITCH;               // [ch·2 + map][EXT32][BIG_ROW]
  __shared__ double s_red[2][BM_THREADS / 32];
  __shared__ float s_shift[3];
  const int tid = threadIdx.x;
  const TileLoc L = locate<T32>(a, blockIdx.x);
  float l1 = 0.f, ss = 0.f, shift[3];
  if (tid < 3 * 32) {
    const float s = tile_shift(a, L, tid & 31, tid >> 5);
    if ((tid & 31) == 0) s_shift[tid >> 5] = s;
  }
  {
    float4 xv[BM_LOADS], yv[BM_LOADS];  // all in flight beside the samples
#pragma unroll
    for (int u = 0; u < BM_LOADS; ++u) {
      const int k = tid + u * BM_THREADS, ly = k / EXT32, lx = k - ly * EXT32;
      const int gx = L.x0 + lx - HALO, gy = L.y0 + ly - HALO;
      xv[u] = yv[u] = make_float4(0, 0, 0, 0);
      if (k < EXT32 * EXT32 && gx >= 0 && gy >= 0 && gx < L.W && gy < L.H) {
        const long long p = L.pix_base + (long long)gy * L.W + gx;
        xv[u] = a.img[p];
        yv[u] = a.target[p];
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k) shift[k] = s_shift[k];
#pragma unroll
    for (int u = 0; u < BM_LOADS; ++u) {
      const int k = tid + u * BM_THREADS, ly = k / EXT32, lx = k - ly * EXT32;
      if (k >= EXT32 * EXT32) break;
      const float4 x = xv[u], y = yv[u];
      if ((unsigned)(lx - HALO) < T32 && (unsigned)(ly - HALO) < T32)  // (outside the image both are zero)
        l1 += fabsf(x.x - y.x) + fabsf(x.y - y.y) + fabsf(x.z - y.z);
      float2* d = s_in + ly * BIG_PITCH + lx;
      d[0] = make_float2(x.x - shift[0], y.x - shift[0]);
      d[EXT32 * BIG_PITCH] = make_float2(x.y - shift[1], y.y - shift[1]);
      d[2 * EXT32 * BIG_PITCH] = make_float2(x.z - shift[2], y.z - shift[2]);
    }
  }
  float w[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) w[k] = a.w[k];
  __syncthreads();
  // Horizontal: item = (channel and map, 8-column segment, row), rows fastest.
  for (int it = tid; it < 6 * 4 * EXT32; it += BM_THREADS) {
    const int r = it % EXT32, q = it / EXT32, sg = q & 3, cm = q >> 2;
    const bool sq = cm & 1;
    const float2* I = s_in + ((cm >> 1) * EXT32 + r) * BIG_PITCH + 8 * sg;
    float2* O = s_h + (cm * EXT32 + r) * BIG_ROW + 8 * sg;
    slide11x2<8>(w, [&](int i) {
      const float2 v = I[i];
      return sq ? make_float2(fmaf(v.x, v.x, v.y * v.y), v.x * v.y) : v;
    }, [&](int o, float2 v) { O[o] = v; });
  }
  __syncthreads();
  // Vertical: item = (channel, 8-row segment, column).
  {
    const int c = tid & 31, sg = (tid >> 5) & 3, ch = tid >> 7;
    const int gx = L.x0 + c;
    const float2* M = s_h + (ch * 2 * EXT32 + 8 * sg) * BIG_ROW + c;
    const float2* S = M + EXT32 * BIG_ROW;
    const float inv_n3 = 1.0f / (3.0f * (float)L.W * (float)L.H);
    const float C1 = 1e-4f, C2 = 9e-4f;
    const float dw = -a.w_ssim * inv_n3, up = ch == 0 ? shift[0] : ch == 1 ? shift[1] : shift[2];
    // this channel's places: r and g are the halves of planes 0..2, b has
    // plane 3 (Cμ, Cx²) and the scalar plane (Cxy)
    const size_t st2 = 2 * a.coef_stride;
    const size_t at_m = ch < 2 ? ch : 3 * st2, at_x = ch < 2 ? st2 + ch : 3 * st2 + 1;
    const size_t at_xy = ch < 2 ? 2 * st2 + ch : 4 * st2;
    const int step = ch < 2 ? 2 : 1;
    float2 wm[TAPS], ws[TAPS];
#pragma unroll
    for (int i = 0; i < TAPS - 1; ++i) { wm[i] = M[i * BIG_ROW]; ws[i] = S[i * BIG_ROW]; }
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      wm[TAPS - 1] = M[(o + TAPS - 1) * BIG_ROW];
      ws[TAPS - 1] = S[(o + TAPS - 1) * BIG_ROW];
      float2 mu = __fmul2_rn(f2(w[0]), wm[HALO]), b = __fmul2_rn(f2(w[0]), ws[HALO]);
#pragma unroll
      for (int d = 0; d < HALO; ++d) {
        mu = __ffma2_rn(f2(w[HALO - d]), __fadd2_rn(wm[d], wm[TAPS - 1 - d]), mu);
        b = __ffma2_rn(f2(w[HALO - d]), __fadd2_rn(ws[d], ws[TAPS - 1 - d]), b);
      }
#pragma unroll
      for (int i = 0; i < TAPS - 1; ++i) { wm[i] = wm[i + 1]; ws[i] = ws[i + 1]; }
      const int gy = L.y0 + 8 * sg + o;
      if (gx < L.W && gy < L.H) {
        const float s2 = b.x - mu.x * mu.x - mu.y * mu.y, sxy = b.y - mu.x * mu.y;
        const float mu_x = mu.x + up, mu_y = mu.y + up;
        const float p = mu_x * mu_x + mu_y * mu_y + C1;
        const float qd = s2 + C2;
        const float ip = __fdividef(1.0f, p), iq = __fdividef(1.0f, qd);  // as in k_ssim_moments
        const float l = (2.0f * mu_x * mu_y + C1) * ip;
        const float cs = (2.0f * sxy + C2) * iq;
        ss += l * cs;
        const size_t pix = (size_t)(L.pix_base + (long long)gy * L.W + gx);
        float* P = a.coef + 2 * pix;
        P[at_m] = (cs * (2.0f * mu_y - 2.0f * mu_x * l) * ip + l * (-2.0f * mu_y + 2.0f * mu_x * cs) * iq) * dw;
        P[at_x] = (-l * cs * iq) * dw;
        a.coef[at_xy + step * pix] = (2.0f * l * iq) * dw;
      }
    }
  }
  const double dl1 = warp_sum(l1), dss = warp_sum(ss);
  if ((tid & 31) == 0) { s_red[0][tid >> 5] = dl1; s_red[1][tid >> 5] = dss; }
  __syncthreads();
  if (tid < 2) {
    double t = 0;
    for (int k = 0; k < BM_THREADS / 32; ++k) t += s_red[tid][k];
    atomicAdd(a.loss_sums + 2 * L.v + tid, t);
  }
}

// ---- normal-consistency loss (first_attempt/crates/gs-train/src/shaders/normal_loss.wgsl) ----
// Per pixel q with mean depth t̄ = depth_acc/α (0 below alpha_min): P(q) = t̄·ray(q),
// N_d = ±normalize((P(q+x) − P(q)) × (P(q+y) − P(q))) facing the camera,
// L = λ/(W·H) Σ α_q (1 − n̂_q·N_d) with α and the orientation sign detached.
// pass 1 writes dL/dnormal and the stencil coefficients dL/d(dPx), dL/d(dPy);
// pass 2 gathers the forward-difference adjoint into dL/d(depth_acc) = dl_dcolor.w.
__device__ __forceinline__ int view_of(const NormalArgs& a, uint64_t i) {
  int v = 0;
  while (v + 1 < a.n_views && (long long)i >= __ldg(&a.views[v + 1].pix_base)) ++v;
  return v;
}
__device__ __forceinline__ float3 ray_at(const ViewInfo* V, int x, int y) {
  const float cx = (float)__ldg(&V->width) * 0.5f, cy = (float)__ldg(&V->height) * 0.5f, f = __ldg(&V->focal);
  return make_float3(((float)x + 0.5f - cx) / f, -((float)y + 0.5f - cy) / f, -1.0f);
}
__device__ __forceinline__ float3 f3s(float3 a, float s) { return make_float3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float3 f3sub(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float f3dot(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 f3cross(float3 a, float3 b) {
  return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// The loss is summed per block and view before its double atomic: one atomic
// per pixel on a single address serialised the whole pass (VGA, every pixel
// covered: 279 us, now 8.2 us for 307,200 pixels, 96 B each).
__global__ void __launch_bounds__(256) k_normal_pass1(NormalArgs a) {
  __shared__ double s_red[8];
  for (int v = 0; v < a.n_views; ++v) {
    const ViewInfo* V = a.views + v;
    const int W = __ldg(&V->width), H = __ldg(&V->height);
    const uint64_t base = (uint64_t)__ldg(&V->pix_base), count = (uint64_t)W * (uint64_t)H;
    double part = 0.0;
    for (uint64_t li = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; li < count;
         li += (uint64_t)gridDim.x * blockDim.x) {
      const uint64_t i = base + li;
      float3 dn = make_float3(0.f, 0.f, 0.f), cx3 = dn, cy3 = dn;
      const int x = (int)(li % (uint64_t)W), y = (int)(li / (uint64_t)W);
      [&] {
        if (a.lambda == 0.f || x + 1 >= W || y + 1 >= H) return;
        const uint64_t ix = i + 1, iy = i + (uint64_t)W;
        const float aq = a.color[i].w, ax = a.color[ix].w, ay = a.color[iy].w;
        if (aq < a.alpha_min || ax < a.alpha_min || ay < a.alpha_min) return;
        const float3 p = f3s(ray_at(V, x, y), a.aux[i].y / aq);
        const float3 dpx = f3sub(f3s(ray_at(V, x + 1, y), a.aux[ix].y / ax), p);
        const float3 dpy = f3sub(f3s(ray_at(V, x, y + 1), a.aux[iy].y / ay), p);
        const float3 m = f3cross(dpx, dpy);
        const float len2 = f3dot(m, m);
        if (len2 < 1e-18f) return;
        const float len = sqrtf(len2);
        const float3 mhat = f3s(m, 1.0f / len);
        const float sign = f3dot(mhat, p) > 0.0f ? -1.0f : 1.0f;
        const float3 nd = f3s(mhat, sign);
        const float4 nv = a.normal[i];
        const float3 av = make_float3(nv.x, nv.y, nv.z);
        const float la2 = f3dot(av, av);
        if (la2 < 1e-18f) return;
        const float la = sqrtf(la2);
        const float3 nhat = f3s(av, 1.0f / la);
        const float lam = a.lambda / ((float)W * (float)H);
        part += (double)((1.0f - f3dot(nhat, nd)) * aq);
        const float3 dl_dnd = f3s(nhat, -lam * aq);
        const float3 dl_dnhat = f3s(nd, -lam * aq);
        dn = f3s(f3sub(dl_dnhat, f3s(nhat, f3dot(nhat, dl_dnhat))), 1.0f / la);
        const float3 dl_dm = f3s(f3sub(dl_dnd, f3s(mhat, f3dot(mhat, dl_dnd))), sign / len);
        cx3 = f3cross(dpy, dl_dm);
        cy3 = f3cross(dl_dm, dpx);
      }();
      float* cp = a.cp + i;
      a.dl_dnormal[i] = make_float4(dn.x, dn.y, dn.z, 0.f);
      cp[0 * a.stride] = cx3.x; cp[1 * a.stride] = cx3.y; cp[2 * a.stride] = cx3.z;
      cp[3 * a.stride] = cy3.x; cp[4 * a.stride] = cy3.y; cp[5 * a.stride] = cy3.z;
    }
    part = warp_sum(part);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int k = 0; k < 8; ++k) t += s_red[k];
      if (t != 0.0) atomicAdd(a.loss + v, t);
    }
    __syncthreads();  // s_red is written again for the next view
  }
}

__global__ void __launch_bounds__(256) k_normal_pass2(NormalArgs a) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.total_px;
       i += (uint64_t)gridDim.x * blockDim.x) {
    float4 c = a.dl_dcolor[i];
    c.w = 0.f;
    if (a.lambda != 0.f) {
      const int v = view_of(a, i);
      const ViewInfo* V = a.views + v;
      const int W = __ldg(&V->width);
      const uint64_t li = i - (uint64_t)__ldg(&V->pix_base);
      const int x = (int)(li % (uint64_t)W), y = (int)(li / (uint64_t)W);
      const float* cp = a.cp;
      // Adjoint of the forward differences: the centre gives −cpx −cpy, the
      // left neighbour's cpx and the upper neighbour's cpy give +.
      float3 acc = make_float3(-cp[0 * a.stride + i] - cp[3 * a.stride + i],
                               -cp[1 * a.stride + i] - cp[4 * a.stride + i],
                               -cp[2 * a.stride + i] - cp[5 * a.stride + i]);
      if (x > 0) {
        acc.x += cp[0 * a.stride + i - 1]; acc.y += cp[1 * a.stride + i - 1]; acc.z += cp[2 * a.stride + i - 1];
      }
      if (y > 0) {
        const uint64_t u = i - (uint64_t)W;
        acc.x += cp[3 * a.stride + u]; acc.y += cp[4 * a.stride + u]; acc.z += cp[5 * a.stride + u];
      }
      const float aq = a.color[i].w;
      if (aq >= a.alpha_min) c.w = f3dot(ray_at(V, x, y), acc) / aq;  // dL/d(depth_acc), α detached
    }
    a.dl_dcolor[i] = c;
  }
}

}  // namespace

int launch_normal_loss(const NormalArgs& a, cudaStream_t st) {
  if (a.total_px == 0) return 0;
  const int grid = (int)std::min<uint64_t>((a.total_px + 255) / 256, 148 * 16);
  k_normal_pass1<<<grid, 256, 0, st>>>(a);
  k_normal_pass2<<<grid, 256, 0, st>>>(a);
  return (int)cudaGetLastError();
}

int launch_ssim(const SsimArgs& a_in, cudaStream_t st) {
  if (a_in.total_tiles16 == 0) return 0;
  SsimArgs a = a_in;
  // Normalised 11-tap Gaussian, sigma 1.5 (ssim.wgsl:32-34 lists its f32 values).
  double g[6], s = 0;
  for (int k = 0; k <= 5; ++k) g[k] = exp(-(double)(k * k) / (2.0 * 1.5 * 1.5));
  s = g[0];
  for (int k = 1; k <= 5; ++k) s += 2 * g[k];
  for (int k = 0; k <= 5; ++k) a.w[k] = (float)(g[k] / s);
  // Moments on 32×32 tiles from five per SM on: 720p (920 tiles) 38.4 -> 36.7
  // us, 1080p 80.2 -> 75.2, 4K 300 -> 284 (of which the shift costs 1, 3 and 17
  // us; with its samples loaded beside the staged pixels instead of before them
  // 38.0, 79, 300); at 640x480 (300 tiles) they took 16.1 us against 15.1, at
  // 800x600 (475) 20.8 both ways. Only where they replace at least 3.5 small
  // tiles each: 33 pixels wide (3.0, 752 tiles) they took 28.4 us against 24.0,
  // 100 wide (3.5, 1000 tiles) 36.3 against 36.1. (The gradient
  // kernel gained nothing from them: 1080p 80.6 against 81.3 us, 4K 299 against
  // 293.)
  if (a.total_tiles32 >= 5 * 148 && 2 * a.total_tiles16 >= 7 * a.total_tiles32) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_ssim_moments_big, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BM_SMEM);
    if (e != cudaSuccess) return (int)e;
    k_ssim_moments_big<<<a.total_tiles32, BM_THREADS, BM_SMEM, st>>>(a);
  } else {
    k_ssim_moments<<<a.total_tiles16, 256, 0, st>>>(a);
  }
  k_ssim_grad<<<a.total_tiles16, 256, 0, st>>>(a);
  return (int)cudaGetLastError();
}

}  // namespace gs
