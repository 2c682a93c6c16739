// Kernels of the adjoint of L = sum_s sum M_s * D_s (included by kernels.cu
// inside namespace bimp_b200, after the forward kernels).
//
//   k_pyr_down_f        float pyramid level (pyrDown without uint8 rounding)
//   k_pyr_down_f_adj    its transpose
//   k_stencil_bwd       gather form of d L / d C over the stencil window from
//                       the ReLU states the forward stencil recorded (when
//                       fftW == dataW, window column dataW is the torus
//                       element (r+1, 0): its gradient is kept aside and
//                       added there by the tile backward)
//   k_gabor_tiles_bwd   per tile: the image spectrum X and, per orientation,
//                       z = e + i o, kept by the forward or recomputed as it
//                       computes them;
//                       a = dL/dC * z/|z|, A = FFT(a), alpha/rho dot products
//                       sum dG Re(conj(A) X), and the sum of A G in the
//                       frequency domain; one inverse transform per tile
//                       gives the window gradient, scattered to the level
#pragma once

__global__ void __launch_bounds__(256) k_pyr_down_f(const PyrJobF* __restrict__ jobs) {
  const PyrJobF j = jobs[blockIdx.z];
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= j.dw || y >= j.dh) return;
  const float w5[5] = {1.f, 4.f, 6.f, 4.f, 1.f};
  float acc = 0.f;
  if (x >= 1 && 2 * x + 2 < j.sw && y >= 1 && 2 * y + 2 < j.sh) {
    // inside: the five columns as two 8-byte loads and one (rows start
    // 128-byte aligned), no reflection
    const float* row = j.src + (size_t)(2 * y - 2) * j.sp + 2 * x - 2;
#pragma unroll
    for (int i = 0; i < 5; ++i, row += j.sp) {
      const float2 a = *reinterpret_cast<const float2*>(row), b = *reinterpret_cast<const float2*>(row + 2);
      const float v[5] = {a.x, a.y, b.x, b.y, row[4]};
      float h = 0.f;
#pragma unroll
      for (int k = 0; k < 5; ++k) h += w5[k] * v[k];
      acc += w5[i] * h;
    }
  } else {
    int cols[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) cols[k] = reflect101(2 * x + k - 2, j.sw);
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const float* row = j.src + (size_t)reflect101(2 * y + i - 2, j.sh) * j.sp;
      float h = 0.f;
#pragma unroll
      for (int k = 0; k < 5; ++k) h += w5[k] * row[cols[k]];
      acc += w5[i] * h;
    }
  }
  j.dst[(size_t)y * j.dp + x] = acc * (1.0f / 256.0f);
}

// The transpose of the reflected, decimated window along one axis of n source
// positions: weight w[k] with which source position p enters output Y0 + k (the
// outputs past the ends get weight 0).  Position p itself, and next to a border
// the window position -1, -2, n or n + 1 that reflects onto it, which lies in
// the window of the same three outputs.  Below 5 positions, where a window
// position can reflect twice, there are two outputs at most: their taps are
// reflected one by one.
__device__ __forceinline__ int pyr_adj_weights(int p, int n, float (&w)[3]) {
  auto f = [](int d) { return d == 0 ? 6.f : d == 1 || d == -1 ? 4.f : d == 2 || d == -2 ? 1.f : 0.f; };
  const int m = (n + 1) >> 1;
  if (n < 5) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      w[k] = 0.f;
      for (int i = -2; i <= 2; ++i)
        if (k < m && reflect101(2 * k + i, n) == p) w[k] += f(i);
    }
    return 0;
  }
  const int Y0 = (p - 1) >> 1;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int Y = Y0 + k;
    w[k] = f(p - 2 * Y);
    if (p >= 1 && p <= 2) w[k] += f(-p - 2 * Y);
    if (p >= n - 3 && p <= n - 2) w[k] += f(2 * n - 2 - p - 2 * Y);
    if (Y < 0 || Y >= m) w[k] = 0.f;
  }
  return Y0;
}

// g_src(r101(2y+i), r101(2x+j)) += w_i w_j / 256 * g_dst(y, x), gathered: a
// thread adds what reaches four adjacent pixels of the finer level, inside from
// 3 x 4 outputs (columns, then rows).  Scattering 25 atomics per output took
// 55 + 19 us for the two steps of 16 x 512 x 512 (six scales), this 24 + 13.
__global__ void __launch_bounds__(256) k_pyr_down_f_adj(const PyrJobF* __restrict__ jobs) {
  const PyrJobF j = jobs[blockIdx.z];
  const int x = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= j.sw || y >= j.sh) return;
  float* __restrict__ dst = j.dst + (size_t)y * j.dp + x;
  float wy[3];
  const int Y0 = pyr_adj_weights(y, j.sh, wy);
  if (x >= 4 && x + 8 < j.sw) {   // no border in x
    float4 d = *reinterpret_cast<const float4*>(dst);
    const float* src = j.src + (x >> 1) - 1;
    float v[4] = {0.f, 0.f, 0.f, 0.f};   // columns x/2 - 1 .. x/2 + 2
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      if (wy[i] == 0.f) continue;
      const float* row = src + (size_t)(Y0 + i) * j.sp;
      const float2 m = __ldg(reinterpret_cast<const float2*>(row + 1));   // x/2 is even
      const float c[4] = {__ldg(row), m.x, m.y, __ldg(row + 3)};
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = fmaf(wy[i], c[k], v[k]);
    }
    constexpr float s1 = 1.f / 256.f, s4 = 4.f / 256.f, s6 = 6.f / 256.f;
    d.x += s1 * (v[0] + v[2]) + s6 * v[1];
    d.y += s4 * (v[1] + v[2]);
    d.z += s1 * (v[1] + v[3]) + s6 * v[2];
    d.w += s4 * (v[2] + v[3]);
    *reinterpret_cast<float4*>(dst) = d;
    return;
  }
  for (int e = 0; e < 4 && x + e < j.sw; ++e) {
    float wx[3], acc = 0.f;
    const int X0 = pyr_adj_weights(x + e, j.sw, wx);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (wy[i] != 0.f && wx[k] != 0.f)
          acc = fmaf(wy[i] * wx[k], __ldg(j.src + (size_t)(Y0 + i) * j.sp + X0 + k), acc);
    dst[e] += acc * (1.0f / 256.0f);
  }
}

__device__ __forceinline__ void block_add_double(double v, double* dst) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  __shared__ double s_part[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) s_part[wid] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) s += s_part[k];
    atomicAdd(dst, s);
  }
}

// --- stencil backward ------------------------------------------------------
constexpr int kBwQW = kStX + 2 * kHalo;        // 48: source pixels +-8 around the block
constexpr int kStBwThreads = 256;

// Gather form of dL/dC_o(p) for a 32x32 block of window positions p
// (0 <= p <= (dataH, dataW)): every source pixel q whose stencils read p
// contributes its loss weight M(q) times the ReLU state the forward recorded
// at q (ScaleDev::bits).  Sources lie within +-8 of p.  The tangential and
// radial weights are constants here; their own gradients come from
// the forward stencil.
//
// A source's weight and states sit side by side in shared memory (one 8-byte
// load), and with a built-in offset set every address is an immediate off the
// pixel's and sources that several orientations share are loaded once (33
// instead of 80 loads a pixel; the run-time offsets cost 48 more): 238 -> 190 us
// for 16 x 512 x 512, 6 scales. What is left is those loads (80% of the L1 rate:
// two wavefronts each) and the selections (72% of the issue slots);
// multiply-adds under a predicate instead of selections: 210 us.
template <int PAT>
__device__ __forceinline__ void stencil_bwd_rows(const uint2* __restrict__ sQ, const int (*sOff)[6],
                                                 const ScaleDev* __restrict__ sd, int x0, int y0) {
  constexpr int sets[kNumOffsetSets][6][8] = BIMP_OFFSET_SETS;
  const int t = threadIdx.x, W = sd->dataW, H = sd->dataH, lx = t & 31, px = x0 + lx;
  const float wT = sd->wTan, wR = sd->wRad, gR = sd->radialGain * wR;
  const int wrapW = sd->wrapW, cPitch = sd->cPitch;
  const long long cStride = sd->cStride;
  float* __restrict__ gC = sd->gC;
#pragma unroll 1
  for (int ly = t >> 5; ly < kStY; ly += kStBwThreads / 32) {
    const int py = y0 + ly;
    if (py > H + 1 || px > W) continue;           // row H + 1: read by no stencil, gathers 0
    const uint2* q0 = sQ + (ly + kHalo) * kBwQW + lx + kHalo;   // p in source-pixel coordinates
    auto at = [&](int dy, int dx) { return q0[dy * kBwQW + dx]; };
    // the source's weight where its states have the bit
    auto weight = [](uint2 q, unsigned int bit) { return q.y & bit ? __uint_as_float(q.x) : 0.f; };
    const uint2 c = at(0, 0);
    const float m0 = __uint_as_float(c.x), mR = wR * m0;
    float g[kNumOri];
#pragma unroll
    for (int o = 0; o < kNumOri; ++o) {
      const int op = (o + kNumOri / 2) % kNumOri;
      auto off = [&](int k, int oo) {
        if constexpr (PAT > 0) return sets[PAT - 1][k][oo];
        else return sOff[oo][k];
      };
      const int o1 = off(0, o), o2 = off(1, o), i1 = off(2, o), i2 = off(3, o);
      const int ph1 = off(4, op), ph2 = off(5, op);
      const unsigned int bd = 1u << (4 * o), bt = 2u << (4 * o), br = 4u << (4 * o), br1 = 8u << (4 * o);
      const unsigned int pr = 4u << (4 * op), pr1 = 8u << (4 * op);
      // double-stopped: p is the centre of q = p, and a -1/2 tap of q = p +- 2 offset
      float v = weight(c, bd);
      v = fmaf(-0.5f, weight(at(2 * o1, -2 * o2), bd), v);
      v = fmaf(-0.5f, weight(at(-2 * o1, 2 * o2), bd), v);
      // tangential: p is read by q = p + i (as C(q - i)) and by q = p (centre)
      v = fmaf(-wT, weight(at(i1, i2), bt), v);
      v = fmaf(wT, weight(c, bt), v);
      // radial, o as the centre orientation (both terms when r1 > 0)
      v -= c.y & br ? mR * (c.y & br1 ? 2.f : 1.f) : 0.f;
      // radial, o as the perpendicular map of op: read at q + h (r1) and q - h (r)
      const uint2 q1 = at(-ph1, -ph2);
      v = fmaf(gR, q1.y & pr ? weight(q1, pr1) : 0.f, v);
      v = fmaf(gR, weight(at(ph1, ph2), pr), v);
      g[o] = v;
    }
    // fftW == dataW: window column dataW of row r is the torus element
    // (r + 1, 0); its gradient goes to gWrap[o][r], which the tile
    // backward adds at (r + 1, 0)
    const bool wrapped = wrapW && px == W;
    float* dst = gC + (size_t)py * cPitch + px;
#pragma unroll
    for (int o = 0; o < kNumOri; ++o) {
      if (wrapped && py <= H) sd->gWrap[o * (H + 1) + py] = g[o];
      dst[o * cStride] = wrapped ? 0.f : g[o];
    }
  }
}

__global__ void __launch_bounds__(kStBwThreads)
k_stencil_bwd(const ScaleDev* __restrict__ sds, const int2* __restrict__ work) {
  __shared__ uint2 sQ[kBwQW * kBwQW];   // per source pixel: loss weight, ReLU states (0 outside the map)
  __shared__ int sOff[kNumOri][6];
  const int2 item = work[blockIdx.x];
  const ScaleDev* __restrict__ sd = sds + item.x;
  const int W = sd->dataW, H = sd->dataH;
  const int nbx = (W + 1 + kStX - 1) / kStX;
  const int by = item.y / nbx, bx = item.y - by * nbx;
  const int x0 = bx * kStX, y0 = by * kStY;
  const int t = threadIdx.x;
  if (t < kNumOri) {
    sOff[t][0] = sd->es1[t]; sOff[t][1] = sd->es2[t];
    sOff[t][2] = sd->in1[t]; sOff[t][3] = sd->in2[t];
    sOff[t][4] = sd->ih1[t]; sOff[t][5] = sd->ih2[t];
  }
  const int dp = sd->dPitch;
  const float* __restrict__ M = sd->M;
  const unsigned int* __restrict__ bits = sd->bits;
#pragma unroll
  for (int i = 0; i < kBwQW * kBwQW / kStBwThreads; ++i) {
    const int idx = t + kStBwThreads * i;
    const int ly = idx / kBwQW, lx = idx - ly * kBwQW;
    const int gy = y0 - kHalo + ly, gx = x0 - kHalo + lx;
    const bool in = gy >= 0 && gy < H && gx >= 0 && gx < W;
    sQ[idx] = in ? make_uint2(__float_as_uint(__ldg(M + (size_t)gy * W + gx)), __ldg(bits + (size_t)gy * dp + gx))
                 : make_uint2(0u, 0u);
  }
  __syncthreads();
  if (sd->pattern == 1) stencil_bwd_rows<1>(sQ, sOff, sd, x0, y0);
  else if (sd->pattern == 2) stencil_bwd_rows<2>(sQ, sOff, sd, x0, y0);
  else stencil_bwd_rows<0>(sQ, sOff, sd, x0, y0);
}
static_assert(kBwQW * kBwQW % kStBwThreads == 0, "staging loop");

// --- tile backward -----------------------------------------------------------
// |e + i o| at or below kMagFloor counts as zero: no gradient flows through
// the magnitude there (the minimal-norm subgradient of |z| at 0).  Exactly
// flat image regions give |e + i o| = 0 up to rounding (the float taps'
// residual DC in FP64, FFT rounding of about 1e-6 of the map peak in FP32),
// where z / |z| is the direction of rounding noise.  The floor is an
// absolute value for images on the [0, 1] scale.
constexpr float kMagFloor = 3.0e-5f;
// Position of natural frequency k in the digit-permuted order of the 8x16
// transforms (the order of G and of the saved spectra).
__device__ __forceinline__ int perm128d(int k) { return 8 * (k & 15) + (k >> 4); }

// Persistent CTAs walk the work items, each a tile and a run of its
// orientations (one CTA per SM: 222 KiB of shared memory and all 512 TMEM
// columns).  The window gradient is linear in the per-orientation spectra,
// Re IFFT(sum_o A_o G_o), so the products are summed in the frequency domain
// (Hermitian half, Bh) and ONE inverse transform per item replaces one per
// orientation.  Per orientation a = dL/dC * z/|z| (0 where |z| <= kMagFloor or
// outside the valid outputs), A = FFT(a), the alpha/rho dot products
// sum dG Re(conj(A) X), and Bh += (A G + conj(A G)(-k))/2.  The
// per-orientation coefficients G(+-k), dGa, dGr come pre-gathered in the half
// layout (ScaleDev::bwA, bwB).
//
// KEPT: z = e + i o and the tile's image spectrum X (Hermitian half) are what
// the forward wrote (ScaleDev::Z, X), z in the order of these lanes: a block of
// four rows is eight coalesced 16-byte loads a lane, in L2 since the orientation
// before.  Otherwise, where the forward had no memory for them, X is
// recomputed per item from the float level (the forward's transform: full
// spectrum into TMEM, Hermitian half into this CTA's slot of `xscratch`) and z
// per orientation by the forward's inverse passes (G read from L2 instead of
// staged).  That costs 60 k + 30 k cycles per item + orientation against 40 k +
// 21 k here, which take 8 bytes more memory an output and orientation: 16
// images of 512 x 512 take 1640 us recomputed and 1130 kept, the forward 864 us
// instead of 791.
//
// The x-passes of both directions run on the same rows, so a warp takes
// blocks of four valid rows through all of them (inverse 8 and 16, magnitude,
// forward 16 and 8) with no CTA barrier, its dL/dC values loaded before the
// first; the y-passes meet at barriers of the four warps of a lane block.
constexpr int kBwRaw = kTile * RawWindow<true>::kPitch * 4;   // staged float window, over Bh
constexpr int kSmemBwBh = kBwRaw > kSmemXh ? kBwRaw : kSmemXh;
constexpr int kGaborBwdSmem = kSmemW + kSmemBwBh + kSmemTw + kSmemMaps + 32;
static_assert(kGaborBwdSmem <= 232448, "tile backward exceeds the 227 KB shared-memory limit");

// Prefetch into L2 of the block of dL/dC that one orientation's magnitude pass
// reads: rows [R0, R0 + rows), columns [x0, x1) of a map with row pitch `pitch`
// floats (rows start on 128-byte lines).  Four threads a row take its lines (at
// most five); addresses stay inside the map.
__device__ __forceinline__ void prefetch_block(const float* base, int pitch, int R0, int rows, int x0, int x1, int t) {
  static_assert(kTileThreads == 4 * kTile, "four threads a row");
  const int r = t >> 2, end = (x1 + 31) >> 5;   // 32 floats per line
  if (r >= rows) return;
  for (int l = (x0 >> 5) + (t & 3); l < end; l += 4)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(base + (size_t)(R0 + r) * pitch + 32 * l));
}

// Adds four consecutive floats (16-byte aligned).
__device__ __forceinline__ void red_add4(float* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// The coefficients and image spectrum of four entries of the accumulation.
struct BwEntries {
  float4 c4[4];   // G(k), G(-k), dGa(k), dGr(k)
  float2 c2[4];   // dGa(-k), dGr(-k)
  float2 X[4];    // (recomputed: from global memory)
};

template <bool KEPT>
__global__ void __launch_bounds__(kTileThreads, 1)
k_gabor_tiles_bwd(const ScaleDev* __restrict__ sds, const TileWork* __restrict__ work, int nwork,
                  float2* __restrict__ xscratch, double* __restrict__ gparams, unsigned int* __restrict__ fault_word) {
  extern __shared__ float4 smem4b[];
  char* base = reinterpret_cast<char*>(smem4b);
  float2* W = reinterpret_cast<float2*>(base);
  float2* Bh = reinterpret_cast<float2*>(base + kSmemW);
  float2* tw = reinterpret_cast<float2*>(base + kSmemW + kSmemBwBh);
  short* rmap = reinterpret_cast<short*>(base + kSmemW + kSmemBwBh + kSmemTw);
  short* cmap = rmap + kTile;
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + kSmemW + kSmemBwBh + kSmemTw + kSmemMaps);
  uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(bars + 2);
  const uint32_t barW = smem_u32(bars);
  float2* Nyq = Bh;                                 // forward transform only (Bh is cleared after it)
  float* rawBuf = reinterpret_cast<float*>(Bh);     // the staged window, before Bh and Nyq
  float2* Xs = KEPT ? nullptr : xscratch + (size_t)blockIdx.x * kSpecHalf;
  const int t = threadIdx.x;
  if (t < 8 * 17) {
    const int n1 = t / 17, k2 = t % 17;
    tw[t] = k2 < 16 ? c_w128[(n1 * k2) & 127] : make_float2(0.f, 0.f);
  }
  if (t == 0) {
    mbar_init(barW, kTileThreads / 32);
    fence_mbar_init();
  }
  if ((t >> 5) == 0) tmem_alloc_warp(smem_u32(tmemSlot));
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const uint32_t tlane = *tmemSlot + ((uint32_t)((t >> 5) & 3) << 21);
  const int h = t >> 7, pcol = PadLayout::col(t & 127);   // row group, this lane's column
  const int warp = t >> 5, quad = warp & 3, lane = t & 31;
  uint32_t phW = 0;
  bool fault = false;   // a wait of this thread expired: what follows is not valid
  double accA = 0.0, accR = 0.0;
  for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
    const TileWork item = work[w];
    const int oB = item.oBegin, oE = item.oEnd;
    if (oB >= oE) break;   // the empty slots of a padded plan follow a CTA's last item
    const ScaleDev* sd = sds + item.entry;
    const int kX = sd->kX, V = sd->V;
    const int ty = item.tile / sd->tilesX, tx = item.tile - ty * sd->tilesX;
    const int R0 = ty * V, C0 = tx * V;
    // rows and columns of the tile's valid outputs inside the map
    const int Vr = min(V, sd->cRows - R0), xHi = min(kX + V, sd->cCols - C0 + kX);
    const int cPitch = sd->cPitch;
    const float4* zTile = nullptr;   // KEPT: this lane's elements of orientation 0's first block
    size_t zOri = 0;                 // and from one orientation to the next
    if constexpr (KEPT) {
      const int cb = kept_column_blocks(*sd);
      zOri = (size_t)sd->tilesX * cb * (kKeptBlock / 2);
      zTile = reinterpret_cast<const float4*>(sd->Z + ((size_t)tx * cb + ty * kept_tile_blocks(V)) * kKeptBlock) + lane;
      Xs = sd->X + (size_t)item.tile * kSpecHalf;
    }
    // into L2, before orientation o's x-passes: its kept responses (the pairs
    // up to the last valid output) and its block of dL/dC
    auto prefetch_orientation = [&](int o) {
      if constexpr (KEPT) {
        if (t < (Vr + 3) >> 2) {
          const float4* z = zTile - lane + o * zOri + (size_t)t * (kKeptBlock / 2);
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(z), "r"(512 * ((xHi + 15) >> 4)) : "memory");
        }
      }
      prefetch_block(sd->gC + (size_t)o * sd->cStride, cPitch, R0, Vr, C0, C0 + xHi - kX, t);
    };
    __syncthreads();   // previous tile finished with every buffer
    if constexpr (!KEPT) raw_chunks_load<true>(sd, R0, C0, rawBuf, t);
    if (t < kTile) rmap[t] = (short)window_src(R0 - kX, t, sd->fftH, sd->dataH, kX);
    else if (t < 2 * kTile) cmap[t - kTile] = (short)window_src(C0 - kX, t - kTile, sd->fftW, sd->dataW, kX);
    prefetch_orientation(oB);
    if constexpr (!KEPT) {
      float* raw = rawBuf + ((C0 - kX) & 3);
      const WindowSpan<true> span(sd, C0);
      if (!span.all()) raw_window_copy<true>(sd, R0, C0, raw, span.iA, span.iB, t);
      cp_async_wait();
      __syncthreads();
      tile_forward_spectrum<true, true, PadLayout>(raw, W, Nyq, tw, tlane, Xs, t, [] {});
      tmem_fence_before();
      __syncthreads();   // the half spectrum in W / Bh is dead from here; X complete in TMEM and Xs
      tmem_fence_after();
    }
    if constexpr (KEPT) {
      // this thread's 16 entries of X for the accumulation, in its own lane of
      // the tensor memory (32 columns a warp): read from L2 with the
      // coefficients they were a quarter of that phase's traffic
#pragma unroll
      for (int r0 = 0; r0 < 16; r0 += 8) {
        float2 x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = __ldg(Xs + ((t >> 6) + 8 * (r0 + u)) * kXhCols + (t & 63));
        tmem_store8(tlane + 32 * (warp >> 2) + 2 * r0, x);
      }
      tmem_wait_st();
    }
    for (int j = t; j < kTile * kXhCols; j += kTileThreads) Bh[j] = make_float2(0.f, 0.f);
    // x-pass lanes keep column group n1 = t mod 8: bit n2 says whether output
    // x = n1 + 8 n2 is valid and inside the map; bit n2 + 16 it of yMask the
    // same of I2's row h + 4 it + 8 n2
    unsigned int xMask = 0, yMask = 0;
#pragma unroll
    for (int n2 = 0; n2 < 16; ++n2) {
      const int x = (t & 7) + 8 * n2, y = h + 8 * n2;
      xMask |= (x >= kX && x < xHi ? 1u : 0u) << n2;
      yMask |= (y >= kX && y < kX + Vr ? 1u : 0u) << n2 | (y + 4 >= kX && y + 4 < kX + Vr ? 0x10000u : 0u) << n2;
    }
    for (int o = oB; o < oE; ++o) {
      if constexpr (!KEPT) {
        // I1: y-dim pass B' with the spectrum product X * G_o (TMEM in, TMEM out)
        {
          // all of the thread's G under way before its first use
          const float4* Go = reinterpret_cast<const float4*>(sd->G + (size_t)o * kSpecFloats) + gpos(8 * h, t & 127) / 4;
          float4 g0[4], g1[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            g0[q] = __ldg(Go + 8 * q * kTile);
            g1[q] = __ldg(Go + (8 * q + 1) * kTile);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int k2 = h + 4 * q;
            float2 v[8];
            tmem_load8(tlane + 16 * k2, v);
            const float ga[8] = {g0[q].x, g0[q].y, g0[q].z, g0[q].w, g1[q].x, g1[q].y, g1[q].z, g1[q].w};
            float2 twr[8];
#pragma unroll
            for (int n1 = 1; n1 < 8; ++n1) twr[n1] = tw[n1 * 17 + k2];
#pragma unroll
            for (int k1 = 0; k1 < 8; ++k1) v[k1] = c_scale(v[k1], ga[k1]);
            dft8<true>(v);
#pragma unroll
            for (int n1 = 0; n1 < 8; ++n1)
              tmem_store1(tlane + kTmemY + 2 * (16 * n1 + k2), n1 ? c_mulc(v[n1], twr[n1]) : v[0]);
          }
        }
        tmem_wait_st();
        tmem_fence_before();
        named_barrier(1 + quad, kTileThreads / 4);   // the lane block's first y-pass is complete
        tmem_fence_after();
        if (o > oB) {   // every warp is done with the previous orientation's accumulation
          if (!mbar_wait(barW, phW)) fault = true;
          phW ^= 1u;
          __syncwarp();
        }
        // I2: y-dim pass A' -> natural y; rows outside the valid band are zero
        // (a is zero there, and the transform of a below reads every row)
#pragma unroll
        for (int it = 0; it < 2; ++it) {
          const int n1 = h + 4 * it;
          float2 v[16];
          tmem_load16(tlane + kTmemY + 32 * n1, v);
          dft16<true>(v);
#pragma unroll
          for (int n2 = 0; n2 < 16; ++n2) {
            W[widx(n1 + 8 * n2, pcol)] = (yMask >> (n2 + 16 * it)) & 1u ? v[n2] : make_float2(0.f, 0.f);
          }
        }
        tmem_fence_before();
        __syncthreads();
        tmem_fence_after();
      }
      if (o + 1 < oE) prefetch_orientation(o + 1);
      // KEPT: W is free when every warp is done with the previous
      // orientation's accumulation
      auto wait_w = [&] {
        if (KEPT && o > oB) {
          if (!mbar_wait(barW, phW)) fault = true;
          phW ^= 1u;
          __syncwarp();
        }
      };
      if (KEPT && 4 * warp >= Vr) wait_w();   // (a warp without rows)
      // The x-passes, four valid rows to a warp at a time: I3 (x-dim pass B');
      // I4 (pass A': z = e + i o at the row's outputs x = n1 + 8 n2),
      // a = dL/dC * z/|z| (|z| as the forward computed it) and the forward
      // pass A of a on the same 16 elements, in registers; pass B.
      {
        const int k2 = lane & 15, n1 = lane & 7;
        // dL/dC of output x = n1 + 8 n2 of the lane's row: src[8 n2]
        const float* __restrict__ src = sd->gC + o * sd->cStride + (long long)(R0 + 4 * warp + (lane >> 3)) * cPitch +
                                        (C0 - kX) + n1;
        // fftW == dataW: window element (r + 1, 0) also carries the gradient
        // of (r, dataW)
        const bool wrapped = sd->wrapW && C0 == 0 && n1 == (kX & 7);
#pragma unroll 1
        for (int r0 = 4 * warp; r0 < Vr; r0 += 4 * (kTileThreads / 32), src += 4 * (kTileThreads / 32) * cPitch) {
          const int r = r0 + (lane >> 3);
          float gcv[16];
#pragma unroll
          for (int n2 = 0; n2 < 16; ++n2) gcv[n2] = r < Vr && ((xMask >> n2) & 1u) ? __ldg(src + 8 * n2) : 0.f;
          if (wrapped && r < Vr && R0 + r >= 1) {
            const float add = __ldg(sd->gWrap + o * (sd->dataH + 1) + R0 + r - 1);
#pragma unroll
            for (int n2 = 0; n2 < 16; ++n2)
              if (n2 == (kX >> 3)) gcv[n2] += add;
          }
          float2 v[16];
          if constexpr (KEPT) {
            const float4* z = zTile + o * zOri + (size_t)(r0 >> 2) * (kKeptBlock / 2);
#pragma unroll
            for (int p = 0; p < 8; ++p) {
              const float4 zz = r < Vr && 16 * p + 15 >= kX && 16 * p < xHi ? __ldcs(z + 32 * p) : make_float4(0.f, 0.f, 0.f, 0.f);
              v[2 * p] = make_float2(zz.x, zz.y);
              v[2 * p + 1] = make_float2(zz.z, zz.w);
            }
            if (r0 == 4 * warp) wait_w();
          } else {
            {
              float2 twr[8];
#pragma unroll
              for (int m = 1; m < 8; ++m) twr[m] = tw[m * 17 + k2];
#pragma unroll 1
              for (int q = r0 + (lane >> 4); q < min(Vr, r0 + 4); q += 2) {
                float2* wr = W + widx(kX + q, 8 * k2);
                float2 v[8];
#pragma unroll
                for (int k1 = 0; k1 < 8; ++k1) v[k1] = wr[k1];
                dft8<true>(v);
#pragma unroll
                for (int m = 0; m < 8; ++m) wr[m] = m ? c_mulc(v[m], twr[m]) : v[0];
              }
            }
            __syncwarp();
          }
          if (r < Vr) {
            float2* wr = W + widx(kX + r, n1);
            if constexpr (!KEPT) {
#pragma unroll
              for (int m = 0; m < 16; ++m) v[m] = wr[9 * m];
              dft16<true>(v);
            }
#pragma unroll
            for (int n2 = 0; n2 < 16; ++n2) {
              // |z| as the forward computes it (s * rsqrt(s)); 1/|z| is the
              // same reciprocal square root, so a = gc z / |z| takes no
              // division; outside the valid outputs gc is 0
              const float sq = fmaf(v[n2].x, v[n2].x, v[n2].y * v[n2].y);
              float rs;
              asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(rs) : "f"(fmaxf(sq, 1e-30f)));
              const float sc = gcv[n2] * rs;
              v[n2] = ((xMask >> n2) & 1u) && sq * rs > kMagFloor ? make_float2(sc * v[n2].x, sc * v[n2].y)
                                                                  : make_float2(0.f, 0.f);
            }
            dft16<false>(v);
            // twiddles four at a time, read before the stores they scale
#pragma unroll
            for (int b = 0; b < 16; b += 4) {
              float2 twr[4];
#pragma unroll
              for (int m = 0; m < 4; ++m) twr[m] = tw[n1 * 17 + b + m];
#pragma unroll
              for (int m = 0; m < 4; ++m) wr[9 * (b + m)] = c_mul(v[b + m], twr[m]);
            }
          }
          __syncwarp();
#pragma unroll 1
          for (int q = r0 + (lane >> 4); q < min(Vr, r0 + 4); q += 2) {
            float2* wq = W + widx(kX + q, 8 * k2);
            float2 v[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) v[m] = wq[m];
            dft8<false>(v);
#pragma unroll
            for (int k1 = 0; k1 < 8; ++k1) wq[k1] = v[k1];
          }
        }
      }
      __syncthreads();
      // forward y-dim passes of a, each lane's column; between them through the
      // tensor memory as between I1 and I2 (through W they moved a third of the
      // 11 k cycles of shared-memory traffic an orientation: 16 x 512 x 512
      // 1165 -> 1130 us)
#pragma unroll
      for (int it = 0; it < 2; ++it) {
        const int n1 = h + 4 * it;
        float2* col = W + widx(n1, pcol);
        float2 v[16];
#pragma unroll
        for (int m = 0; m < 16; ++m) {
          // KEPT: the rows outside the valid band are left as they were
          const bool rowIn = !KEPT || ((yMask >> (m + 16 * it)) & 1u);
          v[m] = rowIn ? col[8 * m * kWPitch] : make_float2(0.f, 0.f);
        }
        dft16<false>(v);
#pragma unroll
        for (int k2 = 0; k2 < 16; ++k2) v[k2] = c_mul(v[k2], tw[n1 * 17 + k2]);
        tmem_store16(tlane + kTmemY + 32 * n1, v);
      }
      tmem_wait_st();
      tmem_fence_before();
      named_barrier(1 + quad, kTileThreads / 4);
      tmem_fence_after();
      // the first coefficients of the accumulation are under way during the last pass
      const float4* __restrict__ cA = sd->bwA + (size_t)o * kSpecHalf;
      const float2* __restrict__ cB = sd->bwB + (size_t)o * kSpecHalf;
      const int sl = t & 63, pr = t >> 6;
      auto fetch = [&](int r0, BwEntries& e) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = (pr + 8 * (r0 + u)) * kXhCols + sl;
          e.c4[u] = __ldg(cA + j);
          e.c2[u] = __ldg(cB + j);
          if constexpr (!KEPT) e.X[u] = Xs[j];   // written by this CTA for this item: a coherent load
        }
      };
      BwEntries next;
      fetch(0, next);
#pragma unroll
      for (int it = 0; it < 4; ++it) {
        float2* col = W + widx(8 * (h + 4 * it), pcol);
        float2 v[8];
        tmem_load8_strided(tlane + kTmemY + 2 * (h + 4 * it), v);
        dft8<false>(v);
#pragma unroll
        for (int k1 = 0; k1 < 8; ++k1) col[k1 * kWPitch] = v[k1];
      }
      tmem_fence_before();
      __syncthreads();
      tmem_fence_after();
      // Hermitian accumulation and the parameter dot products.  Entry j of
      // the half layout holds k = (ky, kx), kx in [0, 64]; its partner -k
      // covers the columns 65..127, so every frequency enters the dot
      // products once (columns 0 and 64 pair with themselves: their -k
      // coefficients are 0).  X is Hermitian, X(-k) = conj(X(k)).  Thread t
      // owns slot t mod 64 and the rows py = t / 64 + 8 r; four entries at a
      // time, the next four's loads issued before them.
      {
        float sa = 0.f, sr = 0.f;
        const int kx = half_group(sl) + 16 * (sl & 3);
        const float2* W1 = W + widx(pr, perm128d(kx));
        const float2* W2 = W + widx(0, perm128d((kTile - kx) & 127));
        float2 X8[8];
#pragma unroll
        for (int r0 = 0; r0 < 16; r0 += 4) {
          BwEntries e = next;
          if (r0 + 4 < 16) fetch(r0 + 4, next);
          if (KEPT && r0 % 8 == 0) tmem_load8(tlane + 32 * (warp >> 2) + 2 * r0, X8);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int py = pr + 8 * (r0 + u), j = py * kXhCols + sl;
            const int ky = 16 * (py & 7) + (py >> 3);
            const float2 A1 = W1[8 * (r0 + u) * kWPitch], A2 = W2[perm128d((kTile - ky) & 127) * kWPitch];
            const float2 bb = Bh[j], X = KEPT ? X8[(r0 & 4) + u] : e.X[u];
            Bh[j] = make_float2(fmaf(0.5f * e.c4[u].x, A1.x, fmaf(0.5f * e.c4[u].y, A2.x, bb.x)),
                                fmaf(0.5f * e.c4[u].x, A1.y, fmaf(-0.5f * e.c4[u].y, A2.y, bb.y)));
            const float re1 = A1.x * X.x + A1.y * X.y;   // Re(conj(A(k)) X(k))
            const float re2 = A2.x * X.x - A2.y * X.y;   // Re(conj(A(-k)) conj(X(k)))
            sa = fmaf(e.c4[u].z, re1, fmaf(e.c2[u].x, re2, sa));
            sr = fmaf(e.c4[u].w, re1, fmaf(e.c2[u].y, re2, sr));
          }
        }
        // slot 64 (kx = 64): one row for each of the first 128 threads
        if (t < kTile) {
          const int py = (t & 64) + 4 * half_group(sl) + (sl & 3), j = py * kXhCols + 64;
          const int ky = 16 * (py & 7) + (py >> 3), p = perm128d(64);
          const float4 c4 = __ldg(cA + j);
          const float2 c2 = __ldg(cB + j), X = Xs[j];
          const float2 A1 = W[widx(py, p)], A2 = W[widx(perm128d((kTile - ky) & 127), p)], bb = Bh[j];
          Bh[j] = make_float2(fmaf(0.5f * c4.x, A1.x, fmaf(0.5f * c4.y, A2.x, bb.x)),
                              fmaf(0.5f * c4.x, A1.y, fmaf(-0.5f * c4.y, A2.y, bb.y)));
          const float re1 = A1.x * X.x + A1.y * X.y, re2 = A2.x * X.x - A2.y * X.y;
          sa = fmaf(c4.z, re1, fmaf(c2.x, re2, sa));
          sr = fmaf(c4.w, re1, fmaf(c2.y, re2, sr));
        }
        accA += sa;
        accR += sr;
      }
      // this warp no longer reads W (the item's last orientation is ordered by
      // the barrier below)
      __syncwarp();
      if (lane == 0 && o + 1 < oE) mbar_arrive(barW);
    }
    __syncthreads();
    // one inverse transform of the Hermitian sum: Re -> window gradient,
    // scattered to the float level through the padded-torus index maps.
    // This lane's column of the full spectrum is read from the half Bh
    // without a branch (conj(Bh(-k)) for mirrored columns).
    {
      const HalfColumn hc(pcol);
      const float sign = hc.conj ? -1.f : 1.f;
#pragma unroll 1
      for (int it = 0; it < 4; ++it) {
        const int k2 = h + 4 * it;
        float2 v[8];
#pragma unroll
        for (int k1 = 0; k1 < 8; ++k1) {
          const int row = hc.conj ? (k2 > 0 ? 8 * (16 - k2) + (7 - k1) : (8 - k1) & 7) : 8 * k2 + k1;
          v[k1] = Bh[row * kXhCols + hc.slot];
          v[k1].y *= sign;
        }
        dft8<true>(v);
#pragma unroll
        for (int n1 = 0; n1 < 8; ++n1) W[widx(8 * k2 + n1, pcol)] = c_mulc(v[n1], tw[n1 * 17 + k2]);
      }
    }
    named_barrier(1 + quad, kTileThreads / 4);
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const int n1 = h + 4 * it;
      float2* col = W + widx(n1, pcol);
      float2 v[16];
#pragma unroll
      for (int k2 = 0; k2 < 16; ++k2) v[k2] = W[widx(8 * k2 + n1, pcol)];
      dft16<true>(v);
#pragma unroll
      for (int n2 = 0; n2 < 16; ++n2) col[8 * n2 * kWPitch] = v[n2];
    }
    __syncthreads();
    // x-passes: eight rows to a warp
    {
      float* __restrict__ gl = sd->gLvl;
      const int gp = sd->lvlPitchF, k2 = lane & 15, n1 = lane & 7;
      // window columns [iA, iB) are consecutive data columns; quads of them
      // start 16-byte aligned in the level `lead` columns before the window
      // (level rows start 16-byte aligned, their pitch is a multiple of 32)
      const int iA = min(max(kX - C0, 0), kTile), iB = max(iA, min(kTile, sd->dataW - (C0 - kX))), lead = (C0 - kX) & 3;
#pragma unroll 1
      for (int r0 = 8 * warp; r0 < 8 * warp + 8; r0 += 4) {
#pragma unroll 1
        for (int y = r0 + (lane >> 4); y < r0 + 4; y += 2) {
          float2* wr = W + widx(y, 8 * k2);
          float2 v[8];
#pragma unroll
          for (int k1 = 0; k1 < 8; ++k1) v[k1] = wr[k1];
          dft8<true>(v);
#pragma unroll
          for (int m = 0; m < 8; ++m) wr[m] = c_mulc(v[m], tw[m * 17 + k2]);
        }
        __syncwarp();
        const int y = r0 + (lane >> 3);
        const float2* wr = W + widx(y, n1);
        float2 v[16];
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = wr[9 * m];
        dft16<true>(v);
        // the row's values in natural order over its own (read) elements, from
        // float `lead` of it on, then four at a time into the level.  (Rows two
        // apart start 8 floats further on: their 4 x 8 stores hit all banks.)
        __syncwarp();
        {
          float* out = reinterpret_cast<float*>(W + widx(y, 0)) + 4 * (y & 2) + lead + n1;
#pragma unroll
          for (int n2 = 0; n2 < 16; ++n2) out[8 * n2] = kFloatLevelScale * v[n2].x;
        }
        __syncwarp();
#pragma unroll 1
        for (int i = 0; i < 5; ++i) {
          // step i: quads 0..31 of row r0 + i; last: quad 32 of the four rows
          const int yy = r0 + (i < 4 ? i : lane & 3), q = i < 4 ? lane : 32;
          if (i == 4 && (lane >= 4 || lead == 0)) break;
          const float* in = reinterpret_cast<const float*>(W + widx(yy, 0)) + 4 * (yy & 2);
          float4 g = reinterpret_cast<const float4*>(in)[q];
          const int x = 4 * q - lead;   // window column of g.x
          if (x < iA || x >= iB) g.x = 0.f;
          if (x + 1 < iA || x + 1 >= iB) g.y = 0.f;
          if (x + 2 < iA || x + 2 >= iB) g.z = 0.f;
          if (x + 3 < iA || x + 3 >= iB) g.w = 0.f;
          if (g.x != 0.f || g.y != 0.f || g.z != 0.f || g.w != 0.f)
            red_add4(gl + (size_t)rmap[yy] * gp + (C0 - kX + x), g);
        }
        // columns outside the data through the torus map, eight lanes to a
        // row: those of the padding fall on the row's first or last element and
        // are summed before they are added (one by one, up to 100 adds of a row
        // to one address, the tiles at the right edge took 70 k of 290 k cycles
        // longer than the others)
        if (iA > 0 || iB < kTile) {
          const float* in = reinterpret_cast<const float*>(W + widx(y, 0)) + 4 * (y & 2) + lead;
          float* row = gl + (size_t)rmap[y] * gp;
          const int last = sd->dataW - 1;
          float toFirst = 0.f, toLast = 0.f;
#pragma unroll 4
          for (int n2 = 0; n2 < 16; ++n2) {
            const int x = n1 + 8 * n2;
            const float g = x < iA || x >= iB ? in[x] : 0.f;
            const int c = cmap[x];
            if (c == last) toLast += g;
            else if (c == 0) toFirst += g;
            else if (g != 0.f) atomicAdd(row + c, g);
          }
#pragma unroll
          for (int d = 4; d > 0; d >>= 1) {
            toFirst += __shfl_xor_sync(0xffffffffu, toFirst, d);
            toLast += __shfl_xor_sync(0xffffffffu, toLast, d);
          }
          if (n1 == 0 && toFirst != 0.f) atomicAdd(row, toFirst);
          if (n1 == 1 && toLast != 0.f) atomicAdd(row + last, toLast);
        }
        __syncwarp();
      }
    }
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  if ((t >> 5) == 0) tmem_dealloc_warp(*tmemSlot);
  if (fault) atomicOr(fault_word, 4u);
  block_add_double(accA, gparams + 0);
  block_add_double(accR, gparams + 1);
}
