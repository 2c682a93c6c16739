// k_gabor_tiles: overlap-save 128x128 tile FFT Gabor filtering (included by
// kernels.cu).
//
// One CTA (512 threads, 16 warps) walks its work items, each a tile and a run
// of its orientations (all 8, or fewer where the plan splits a tile between
// CTAs, each of which then transforms the tile forward).  The tile's real input
// window is read from the pyramid level through the reference's padded-torus
// index map, transformed once (forward 2D FFT, Hermitian half), and the full
// spectrum is written to tensor memory (TMEM): lane l holds column
// PadLayout::col(l), 32-bit columns 2 py and 2 py + 1 the real and imaginary
// parts of row py, so that the spectrum product pass of every orientation
// fetches its 8 values with one tcgen05.ld and no Hermitian lookup.  For each
// orientation the spectrum is multiplied by that orientation's real Gabor
// spectrum G_o, inverse transformed as one complex FFT (e + i o) and reduced to
// |e + i o| on the valid outputs.  SAVE_Z also stores e + i o (the line/edge
// detector's even and odd responses).
//
// G_o (64 KB per orientation, L2-resident) comes by a TMA bulk copy
// (cp.async.bulk + mbarrier) issued when the previous one is consumed; it lands
// during the x-passes.  Before an item's first orientation the same buffer
// takes the item's byte window, fetched during the item before it.  The product
// pass writes its y-pass output to TMEM as well, where the second y-pass reads
// it back, so the product pass uses no work buffer, and one CTA barrier per
// orientation is enough: after the second y-pass, which turns columns into
// rows.  The x-passes run warp by warp; the warps of a lane block meet between
// the y-passes at a named barrier, and the work buffer is handed back by an
// mbarrier that each warp arrives at when its rows are done.
//
// What bounds it: FP32 issue and the latency around the passes (at 1080p 192 M
// warp instructions were 65% of the issue slots of 262.7 us; FP32 adds run at
// one a cycle and scheduler, paired f32x2 adds at half that, so they gain
// nothing).  1080p, 694 tiles: 262.7 -> 232.7 us; 3840 x 2160, 12 scales: 1072
// -> 859 us, by the padded layout and 16-byte G reads (247.4 us), the fused end
// of the forward transform and staged windows (241.2), x-passes without CTA
// barriers (238.0), balanced first y-passes (232.1) and, in larger batches of
// work, the plan's refitted costs.  Every mbarrier wait is bounded; on expiry
// the thread that saw it sets a bit of *fault_word, the kernel waits once more
// (bounded) for its copies and carries on, and the host reports the fault.
//
// Included inside namespace bimp_b200 by kernels.cu, after the helpers it uses
// (pad_src, pmod, c_w128).
#pragma once

// Work buffer: 128 rows x 128 complex.  Position p of row y sits at
// y * kWPitch + 9 (p / 8) + p mod 8 (one complex of padding per group of
// eight): an affine map, so that every pass addresses its elements as one
// register plus immediates.  In units of a complex (two banks), a half warp's
// 16 accesses fall into distinct residues mod 16 in every pass: 16 groups at
// one offset (9 k2), 8 positions of two adjacent rows (kWPitch = 8 mod 16),
// and the columns of 16 TMEM lanes (groups a and a + 8, see PadLayout::col).
// A rotate-and-xor swizzle without padding was conflict-free too, but cost a
// register or two integer operations per access: 262.7 against 253.9 us for
// the 1080p launch.
constexpr int kWPitch = 152;
constexpr int kSmemW = kTile * kWPitch * 8;
constexpr int kSmemXh = kTile * kXhCols * 8;             // Hermitian half spectrum (adjoint kernel)
constexpr int kSmemG = kSpecFloats * 4;                  // one orientation's Gabor spectrum
constexpr int kSmemTw = 8 * 17 * 8;                      // twiddles w128^(n1*k2) (1 for n1 k2 = 0: not applied)
constexpr int kSmemMaps = 2 * kTile * 2;                 // int16 row / column maps (adjoint kernel)
constexpr int kSmemNyq = kTile * 8;                      // column kx = 64 of the half spectrum
constexpr int kSmemBars = 2 * 8 + 16;                    // the G and work-buffer mbarriers, the TMEM base address
constexpr int kSmemQueue = 2 * (sizeof(TileWork) + sizeof(ScaleDev));   // work items and scale records, this and the next
constexpr int kGaborSmem = kSmemW + kSmemG + kSmemTw + kSmemNyq + kSmemBars + kSmemQueue;
static_assert(sizeof(TileWork) == 16 && sizeof(ScaleDev) % 16 == 0, "copied as 16-byte words");
static_assert(kGaborSmem <= 232448, "tile kernel exceeds the 227 KB shared-memory limit");

// Tensor memory, 128 lanes x 512 32-bit columns: the tile's full spectrum
// (columns [0, 256): lane p, columns 2 py, 2 py + 1 = X[py][p]) and the
// output of the first inverse y-pass (columns [256, 512): lane p, columns
// 256 + 2 (16 n1 + k2) + {0, 1} = row 8 k2 + n1 of column p).
constexpr uint32_t kTmemCols = 4 * kTile;
constexpr uint32_t kTmemY = 2 * kTile;

__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Whole warp: allocate kTmemCols columns, base address written to dst_smem.
__device__ __forceinline__ void tmem_alloc_warp(uint32_t dst_smem) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem),
               "n"(kTmemCols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_warp(uint32_t taddr) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "n"(kTmemCols) : "memory");
}
// Whole warp: each thread stores 8 complex (16 columns from taddr's column)
// into its own lane; completion is awaited with tmem_wait_st.
__device__ __forceinline__ void tmem_store8(uint32_t taddr, const float2 (&v)[8]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16};" ::"r"(taddr),
      "r"(__float_as_uint(v[0].x)), "r"(__float_as_uint(v[0].y)), "r"(__float_as_uint(v[1].x)),
      "r"(__float_as_uint(v[1].y)), "r"(__float_as_uint(v[2].x)), "r"(__float_as_uint(v[2].y)),
      "r"(__float_as_uint(v[3].x)), "r"(__float_as_uint(v[3].y)), "r"(__float_as_uint(v[4].x)),
      "r"(__float_as_uint(v[4].y)), "r"(__float_as_uint(v[5].x)), "r"(__float_as_uint(v[5].y)),
      "r"(__float_as_uint(v[6].x)), "r"(__float_as_uint(v[6].y)), "r"(__float_as_uint(v[7].x)),
      "r"(__float_as_uint(v[7].y)));
}
// The same for 16 complex (32 columns).
__device__ __forceinline__ void tmem_store16(uint32_t taddr, const float2 (&v)[16]) {
  uint32_t r[32];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    r[2 * i] = __float_as_uint(v[i].x);
    r[2 * i + 1] = __float_as_uint(v[i].y);
  }
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]));
}
// Whole warp: each thread stores one complex (2 columns) into its own lane;
// completion is awaited with tmem_wait_st.
__device__ __forceinline__ void tmem_store1(uint32_t taddr, float2 v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(taddr), "r"(__float_as_uint(v.x)),
               "r"(__float_as_uint(v.y)));
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Whole warp: each thread loads 16 complex (32 columns) from its own lane;
// the values are complete when the statement returns.
__device__ __forceinline__ void tmem_load16(uint32_t taddr, float2 (&v)[16]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}
// Whole warp: each thread loads 8 complex from its own lane; the values are
// complete when the statement returns.
__device__ __forceinline__ void tmem_load8(uint32_t taddr, float2 (&v)[8]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}

// Whole warp: each thread loads 8 complex, 32 columns apart, from its own lane.
__device__ __forceinline__ void tmem_load8_strided(uint32_t taddr, float2 (&v)[8]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%16];\n"
      "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%2, %3}, [%17];\n"
      "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%4, %5}, [%18];\n"
      "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%6, %7}, [%19];\n"
      "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%8, %9}, [%20];\n"
      "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%10, %11}, [%21];\n"
      "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%12, %13}, [%22];\n"
      "tcgen05.ld.sync.aligned.32x32b.x2.b32 {%14, %15}, [%23];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]),
        "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]), "=&r"(r[14]), "=&r"(r[15])
      : "r"(taddr), "r"(taddr + 32), "r"(taddr + 64), "r"(taddr + 96), "r"(taddr + 128), "r"(taddr + 160),
        "r"(taddr + 192), "r"(taddr + 224));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}

// |z| as s * rsqrt(max(s, 1e-30)), s = |z|^2 (hardware reciprocal square
// root, relative error a few 1e-7): exactly 0 for z = 0, and below 1e-15
// (where the max applies) the value stays below |z|.
__device__ __forceinline__ float cmag(float2 z) {
  const float s = fmaf(z.x, z.x, z.y * z.y);
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fmaxf(s, 1e-30f)));
  return s * r;
}

// Float levels hold X (a float image, X = u8/255 for the uint8 content);
// the uint8 path's value 255*u8/65536 is then (255*255/65536) * X.
constexpr float kFloatLevelScale = 65025.0f / 65536.0f;

__device__ __forceinline__ int widx(int y, int p) { return y * kWPitch + 9 * (p >> 3) + (p & 7); }

// Shared-memory layout of the work buffer and order of the spectrum columns
// over the TMEM lanes.  kHalf: first complex of the part behind the 64 packed
// rows, where the forward transform stages its window and keeps the half
// spectrum.
struct PadLayout {
  static constexpr int kHalf = 64 * kWPitch;
  static constexpr bool kFewRegs = false;
  static __device__ __forceinline__ int at(int y, int p) { return widx(y, p); }
  // lanes 16 j + i: columns of group j (i < 8) and of group j + 8
  static __device__ __forceinline__ int col(int lane) { return 8 * ((lane >> 4) + 8 * ((lane >> 3) & 1)) + (lane & 7); }
};
// The pipelined kernel's row buffers have no room for padding: positions
// rotate inside each group of eight, odd rows swap the halves of each 16.
struct RotLayout {
  static constexpr int kHalf = 64 * kTile;
  static constexpr bool kFewRegs = true;   // (its loop over the orientations keeps more of them)
  static __device__ __forceinline__ int at(int y, int p) { return y * kTile + (phys(p) ^ ((y & 1) << 3)); }
  static __device__ __forceinline__ int col(int lane) { return lane; }
};

// Slot of column kx = a + 16 b (0 <= a < 16, 0 <= b < 4) in the Hermitian
// half: the groups a are stored in the order 0, 4, 8, 12, 1, 5, ..., so that a
// half warp's 16 consecutive slots read work-buffer groups four apart
// (conflict-free), and so do the mirrored columns.
__device__ __forceinline__ int half_slot(int a, int b) { return 16 * (a & 3) + 4 * (a >> 2) + b; }
__device__ __forceinline__ int half_group(int slot) { return (slot >> 4) + 4 * ((slot >> 2) & 3); }

// Where column p (permuted order: kx = p / 8 + 16 (p mod 8)) of the full
// spectrum lives in the Hermitian half kx = 0..64; the other columns are
// conj(X(-k)) of column -kx.
struct HalfColumn {
  int slot;    // 0..63, or 64 for kx = 64
  bool conj;   // read from -kx
  __device__ __forceinline__ explicit HalfColumn(int p) {
    const int a = p >> 3, b = p & 7;
    conj = b > 4 || (b == 4 && a > 0);
    slot = b < 4 ? half_slot(a, b) : !conj ? 64 : a > 0 ? half_slot(16 - a, 7 - b) : half_slot(0, 8 - b);
  }
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void named_barrier(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// 1-D TMA bulk copy global -> shared, completion counted on `bar`.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// Bounded wait for phase `parity` of `bar`; false if it did not complete.
[[nodiscard]] __device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (int i = 0; i < (1 << 22); ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Position of spectrum row py, column p in a stored Gabor spectrum: columns in
// the TMEM lane order of PadLayout, rows in groups of four, so that a thread
// reads its eight rows of G as two conflict-free 16-byte loads.
__device__ __forceinline__ int gpos(int py, int lane) { return ((py >> 2) * kTile + lane) * 4 + (py & 3); }
__device__ __forceinline__ int glane(int p) { return 16 * ((p >> 3) & 7) + 8 * (p >> 6) + (p & 7); }

// Mean-removed value of a level pixel.  uint8: the reference's 255*u8/65536
// (convertTo, cuda_bimp.cu:481) minus 0.5, exactly, as (255*u8 -
// 32768)/65536: 12582912 + (255 u8 - 32768) as the bits of a float (1.5 * 2^23
// plus an integer of magnitude below 2^15 is exact), then x / 65536 exactly,
// without the conversion unit.  float: kFloatLevelScale * X - 0.5.
__device__ __forceinline__ float level_value(uint8_t u) {
  return fmaf(__int_as_float(0x4B400000 - 32768 + 255 * (int)u), 1.0f / 65536.0f, -192.0f);
}
__device__ __forceinline__ float level_value(float x) { return kFloatLevelScale * x - 0.5f; }

// A shared-memory read that is not kept in a register from an earlier one.
template <class T>
__device__ __forceinline__ T lds_now(const T* p) {
  return *reinterpret_cast<const volatile T*>(p);
}

// Asynchronous 16-byte copies global -> shared (this thread's, awaited with
// cp_async_wait).
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// --- forward transform -------------------------------------------------------
// The tile's 128 x 128 input window as staged in shared memory, one row per
// kPitch values (the pitch keeps a warp's 4 rows x 8 values in distinct banks).
template <bool FLT>
struct RawWindow {
  using T = uint8_t;
  static constexpr int kPitch = 160;   // 128 bytes behind a lead of up to 15
};
template <>
struct RawWindow<true> {
  using T = float;
  static constexpr int kPitch = 136;
};

// Level row / column of window index i (window origin o) through the padded
// torus.
__device__ __forceinline__ int window_src(int o, int i, int fft, int nData, int kHalf) {
  return pad_src(pmod(o + i, fft), nData, kHalf);
}

// The columns [iA, iB) of a window that are staged as 16-byte chunks: those
// whose chunk lies inside the data, or all of them.
template <bool FLT>
struct WindowSpan {
  static constexpr int kVals = 16 / sizeof(typename RawWindow<FLT>::T);   // values of a chunk
  int c0, iA, iB, end;   // end: chunks past it are not read
  __device__ __forceinline__ WindowSpan(const ScaleDev* sd, int C0) {
    c0 = C0 - sd->kX;
    const bool endInside = c0 + kTile <= sd->dataW;
    end = endInside ? c0 + kTile : sd->dataW & ~(kVals - 1);
    iA = min(max(-c0, 0), kTile);
    iB = endInside ? kTile : max(iA, end - c0);
  }
  __device__ __forceinline__ bool all() const { return iA == 0 && iB == kTile; }
};
// A window's data columns are staged as aligned 16-byte chunks (level rows
// start 16-byte aligned and their pitch is a multiple of 16 bytes),
// asynchronously: column i of row r goes to raw[r * kPitch + lead + i], lead =
// C0 - kX modulo the values of a chunk.  (A window that ends inside the data
// may read its last chunk past the data, inside the row's pitch.)
template <bool FLT>
__device__ __forceinline__ void raw_chunks_load(const ScaleDev* sd, int R0, int C0, typename RawWindow<FLT>::T* raw,
                                                int t) {
  using T = typename RawWindow<FLT>::T;
  constexpr int kVals = WindowSpan<FLT>::kVals, kChunks = kTile / kVals + 1;
  const WindowSpan<FLT> span(sd, C0);
  const int kX = sd->kX, r0 = R0 - kX;
  const T* lvl;
  int pitch;
  if constexpr (FLT) { lvl = sd->lvlF; pitch = sd->lvlPitchF; }
  else { lvl = sd->lvl; pitch = sd->lvlPitch; }
  // four threads a row
  const int r = t >> 2;
  const int row = r0 >= 0 && r0 + kTile <= sd->dataH ? r0 + r : window_src(r0, r, sd->fftH, sd->dataH, kX);
  const T* src = lvl + (size_t)row * pitch;
  raw += r * RawWindow<FLT>::kPitch;
#pragma unroll
  for (int c = t & 3; c < kChunks; c += 4) {
    const int x = (span.c0 & ~(kVals - 1)) + kVals * c;
    if (x >= 0 && x < span.end) cp_async16(raw + kVals * c, src + x);
  }
}
// The window's columns outside [iA, iB) (which no chunk writes), value by value
// through the padded-torus map: warp w stages rows w, w + 16, ..., lane l the columns l,
// l + 32, l + 64, l + 96 among them.  Bound by the latency of its loads: a group
// of columns at a time (most windows have one or two with columns outside), the
// loads of its eight rows in flight together.  All four groups of four rows at
// once took registers that the pipelined kernel spilled: 4 images of 512 x 512
// 139 us a detection with it and 134 so, 112 and 111 with k_gabor_tiles.
template <bool FLT>
__device__ __forceinline__ void raw_window_copy(const ScaleDev* sd, int R0, int C0, typename RawWindow<FLT>::T* raw,
                                                int iA, int iB, int t) {
  using T = typename RawWindow<FLT>::T;
  constexpr int P = RawWindow<FLT>::kPitch;
  const int lane = t & 31, w0 = t >> 5, kX = sd->kX;
  const T* lvl;
  int pitch;
  if constexpr (FLT) { lvl = sd->lvlF; pitch = sd->lvlPitchF; }
  else { lvl = sd->lvl; pitch = sd->lvlPitch; }
  const int myRow = window_src(R0 - kX, w0 + 16 * (lane & 7), sd->fftH, sd->dataH, kX);
#pragma unroll 1
  for (int k = 0; k < 4; ++k) {
    const int i = lane + 32 * k;
    const bool mine = i < iA || i >= iB;
    if (!__any_sync(0xffffffffu, mine)) continue;
    const int c = window_src(C0 - kX, i, sd->fftW, sd->dataW, kX);
    T v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = lvl[(size_t)__shfl_sync(0xffffffffu, myRow, r) * pitch + c];
    if (mine) {
#pragma unroll
      for (int r = 0; r < 8; ++r) raw[(w0 + 16 * r) * P + i] = v[r];
    }
  }
}

// Forward 2D FFT of the staged window `raw` (complete: a barrier after its
// staging; its memory is free when every thread has called windowRead): the
// full spectrum goes to TMEM, each thread writing the rows py = 8 k2 + k1, k2 =
// h + 4 q, of its lane's column (h = t / 128).  W: work buffer, of
// which the part behind the 64 packed rows (LY::kHalf; `raw` may lie there)
// later holds the half spectrum; Nyq its column kx = 64.  SAVE_X also writes the
// Hermitian half to global memory, Xs[py * kXhCols + slot], where Xs is given.
template <bool FLT, bool SAVE_X, class LY, class Hook>
__device__ __forceinline__ void tile_forward_spectrum(const typename RawWindow<FLT>::T* raw, float2* W, float2* Nyq,
                                                      const float2* tw, uint32_t tlane, float2* __restrict__ Xs, int t,
                                                      Hook windowRead) {
  float2* Xh = W + LY::kHalf;
  // F1: x-dim pass A on packed rows z[r] = in[r] + i in[r+64], r < 64.
  // Removing the mean keeps the butterflies' intermediate magnitudes, and so
  // their float rounding, small; the 0.5 offset goes back into the DC bin.
  {
    const int r = t >> 3, n1 = t & 7;
    const auto* in = raw + r * RawWindow<FLT>::kPitch + n1;
    float2 v[16];
#pragma unroll
    for (int m = 0; m < 16; ++m)
      v[m] = make_float2(level_value(in[8 * m]), level_value(in[64 * RawWindow<FLT>::kPitch + 8 * m]));
    dft16<false>(v);
    // twiddles into registers before the stores (loads of the table would
    // otherwise wait behind each store to the same shared memory)
    float2 twr[16];
#pragma unroll
    for (int k2 = 1; k2 < 16; ++k2) twr[k2] = tw[n1 * 17 + k2];
#pragma unroll
    for (int k2 = 0; k2 < 16; ++k2) W[LY::at(r, n1 + 8 * k2)] = k2 ? c_mul(v[k2], twr[k2]) : v[0];
  }
  __syncthreads();
  windowRead();
  // F2: x-dim pass B
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int j = t + it * kTileThreads;
    const int r = j >> 4, k2 = j & 15;
    float2 v[8];
#pragma unroll
    for (int n1 = 0; n1 < 8; ++n1) v[n1] = W[LY::at(r, 8 * k2 + n1)];
    dft8<false>(v);
#pragma unroll
    for (int k1 = 0; k1 < 8; ++k1) W[LY::at(r, 8 * k2 + k1)] = v[k1];
  }
  __syncthreads();
  // F3: y-dim pass A on the 65 half columns (kx = 0..64), reading the packed
  // rows and separating them on the way in: packed row r (< 64) holds
  // in[r] + i in[r + 64], so X[r][kx] = (Z[kx] + conj Z[-kx]) / 2 and
  // X[r + 64][kx] = (Z[kx] - conj Z[-kx]) / 2i.  One item per thread; the
  // eight items of kx = 64 are the second item of eight threads.
#pragma unroll 1
  for (int j = t; j < 8 * kXhCols; j += kTileThreads) {
    const bool nyq = j >= kTileThreads;
    const int n1 = nyq ? j - kTileThreads : j >> 6, s = j & 63;
    const int kx = nyq ? 64 : half_group(s) + 16 * (s & 3);
    const int nk = (128 - kx) & 127;
    const int pk = 8 * (kx & 15) + (kx >> 4), pn = 8 * (nk & 15) + (nk >> 4);
    float2 v[16];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const int r = n1 + 8 * m;
      const float2 Z = W[LY::at(r, pk)], Zn = W[LY::at(r, pn)];
      v[m] = make_float2(0.5f * (Z.x + Zn.x), 0.5f * (Z.y - Zn.y));
      v[m + 8] = make_float2(0.5f * (Z.y + Zn.y), 0.5f * (Zn.x - Z.x));
    }
    dft16<false>(v);
    float2* col = (nyq ? Nyq : Xh + s) + n1 * (nyq ? 1 : 64);
    const int st = nyq ? 8 : 8 * 64;
    float2 twr[16];
#pragma unroll
    for (int k2 = 1; k2 < 16; ++k2) twr[k2] = tw[n1 * 17 + k2];
#pragma unroll
    for (int k2 = 0; k2 < 16; ++k2) col[k2 * st] = k2 ? c_mul(v[k2], twr[k2]) : v[0];
  }
  __syncthreads();
  // F4: y-dim pass B and the store of the full spectrum.  Every thread
  // transforms what its lane's column needs; a mirrored column is the
  // conjugate of column -kx at row -ky, ky = 16 k1 + k2, that is of row block
  // 16 - k2 in reverse (block 0: output (8 - k1) mod 8).  Transforming a
  // column once and exchanging the mirrored half through shared memory took
  // another pass and a barrier (6.2 k cycles an item against 3.8 k).
  {
    const int p = LY::col(t & 127), h = t >> 7;
    const HalfColumn hc(p);
    const float sign = hc.conj ? -1.f : 1.f;
    const float2* src = hc.slot == 64 ? Nyq : Xh + hc.slot;
    const int st = hc.slot == 64 ? 1 : 64;
#pragma unroll(SAVE_X || LY::kFewRegs ? 1 : 4)
    for (int q = 0; q < 4; ++q) {
      const int k2 = h + 4 * q;
      const int kb = hc.conj ? (16 - k2) & 15 : k2;
      float2 v[8], x[8];
#pragma unroll
      for (int n1 = 0; n1 < 8; ++n1) v[n1] = src[(8 * kb + n1) * st];
      dft8<false>(v);
      if (p == 0 && k2 == 0) v[0].x += 0.5f * (float)(kTile * kTile);   // DC of the removed 0.5 offset
      if (k2 > 0) {
#pragma unroll
        for (int k1 = 0; k1 < 8; ++k1) x[k1] = hc.conj ? v[7 - k1] : v[k1];
      } else {
#pragma unroll
        for (int k1 = 0; k1 < 8; ++k1) x[k1] = hc.conj ? v[(8 - k1) & 7] : v[k1];
      }
#pragma unroll
      for (int k1 = 0; k1 < 8; ++k1) x[k1].y *= sign;
      tmem_store8(tlane + 16 * k2, x);
      if constexpr (SAVE_X) {
        if (Xs && !hc.conj) {
#pragma unroll
          for (int k1 = 0; k1 < 8; ++k1) Xs[(8 * k2 + k1) * kXhCols + hc.slot] = x[k1];
        }
      }
    }
    tmem_wait_st();
  }
}

template <bool FLT, bool SAVE_Z>
__global__ void __launch_bounds__(kTileThreads, 1)
k_gabor_tiles(const ScaleDev* __restrict__ sds, const TileWork* __restrict__ work, int nwork,
              unsigned int* __restrict__ fault_word) {
  extern __shared__ float4 smem4[];
  char* base = reinterpret_cast<char*>(smem4);
  float2* W = reinterpret_cast<float2*>(base);
  float* Gbuf = reinterpret_cast<float*>(base + kSmemW);
  float2* tw = reinterpret_cast<float2*>(base + kSmemW + kSmemG);
  float2* Nyq = reinterpret_cast<float2*>(base + kSmemW + kSmemG + kSmemTw);   // forward transform only
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + kSmemW + kSmemG + kSmemTw + kSmemNyq);
  uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(bars + 2);
  TileWork* qItem = reinterpret_cast<TileWork*>(bars + 4);
  ScaleDev* qScale = reinterpret_cast<ScaleDev*>(qItem + 2);
  uint8_t* rawG = reinterpret_cast<uint8_t*>(Gbuf);   // an inner tile's byte window, while no G is in it
  const uint32_t bar0 = smem_u32(&bars[0]), barW = bar0 + 8, gdst = smem_u32(Gbuf);
  const int t = threadIdx.x;

  if (t < 8 * 17) {
    const int n1 = t / 17, k2 = t % 17;
    tw[t] = k2 < 16 ? c_w128[(n1 * k2) & 127] : make_float2(0.f, 0.f);
  }
  if (t == 0) {
    mbar_init(bar0, 1);
    mbar_init(barW, kTileThreads / 32);
    fence_mbar_init();
  }
  if ((t >> 5) == 0) tmem_alloc_warp(smem_u32(tmemSlot));
  // This item's and the next one's work item and scale record live in shared
  // memory (slot = item index mod 2), fetched one item ahead: at an item's
  // start the dependent global loads work item -> record -> window cost 2.5 k
  // cycles and staging the window 1.2 k, of about 100 k an item.
  if ((t >> 5) == 0) {
    const int lane = t & 31;
    const TileWork first = work[blockIdx.x];
    if (lane < 2) qItem[lane] = (int)(blockIdx.x + lane * gridDim.x) < nwork ? work[blockIdx.x + lane * gridDim.x] : TileWork{0, 0, 0, 0};
    for (int i = lane; i < (int)(sizeof(ScaleDev) / 16); i += 32)
      reinterpret_cast<uint4*>(qScale)[i] = reinterpret_cast<const uint4*>(sds + first.entry)[i];
  }
  griddep_launch_dependents();
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  griddep_wait();   // the pyramid levels come from the previous kernel
  // this thread's lane (t mod 128) of the spectrum; (warp mod 4) * 32 is the
  // lane block the warp may access
  const uint32_t tlane = *tmemSlot + ((uint32_t)((t >> 5) & 3) << 21);

  uint32_t ph = 0;       // parity of the next fill of the G buffer (identical in every thread)
  uint32_t phW = 0;      // parity of the next release of W by the x-passes
  bool fault = false;
  const int h = t >> 7, pcol = PadLayout::col(t & 127);
  const int warp = t >> 5, quad = warp & 3;   // quad: the warp's lane block, and its scheduler

  if constexpr (!FLT) {
    const int tile = qItem[0].tile, ty = tile / qScale->tilesX, tx = tile - ty * qScale->tilesX;
    raw_chunks_load<false>(qScale, ty * qScale->V, tx * qScale->V, rawG, t);
  }

  for (int w = blockIdx.x, slot = 0; w < nwork; w += gridDim.x, slot ^= 1) {
    const TileWork item = qItem[slot];
    const int oB = item.oBegin, oE = item.oEnd;
    if (oB >= oE) break;   // the empty slots of a padded plan follow a CTA's last item
    const ScaleDev* sd = qScale + slot;
    const int kX = sd->kX, V = sd->V;
    const int ty = item.tile / sd->tilesX, tx = item.tile - ty * sd->tilesX;
    const int R0 = ty * V, C0 = tx * V;
    cp_async_wait();
    __syncthreads();   // previous tile finished with every buffer; a byte window's data columns are in the G buffer
    if ((t >> 5) == 1) {   // the next item's record, and the item after it (waited for before I1)
      const int lane = t & 31, w2 = w + 2 * (int)gridDim.x;
      for (int i = lane; i < (int)(sizeof(ScaleDev) / 16); i += 32)
        cp_async16(reinterpret_cast<uint4*>(qScale + (slot ^ 1)) + i,
                   reinterpret_cast<const uint4*>(sds + qItem[slot ^ 1].entry) + i);
      if (lane == 0) {
        if (w2 < nwork) cp_async16(qItem + slot, work + w2);
        else qItem[slot] = TileWork{0, 0, 0, 0};
      }
    }
    // orientation oB's spectrum lands during the forward transform: a byte
    // window leaves the G buffer with the first pass, a float window (64 KB)
    // is staged in the work buffer
    auto load_first = [&]() {
      if (t == 0) {
        fence_proxy_async();
        bulk_load(gdst, sd->G + (size_t)oB * kSpecFloats, kSmemG, bar0);
      }
    };
    if constexpr (FLT) {
      load_first();
      float* raw = reinterpret_cast<float*>(W + PadLayout::kHalf);
      raw_chunks_load<FLT>(sd, R0, C0, raw, t);
      raw += (C0 - kX) & 3;
      const WindowSpan<FLT> span(sd, C0);
      if (!span.all()) raw_window_copy<FLT>(sd, R0, C0, raw, span.iA, span.iB, t);
      cp_async_wait();
      __syncthreads();
      // the adjoint keeps the spectrum of every tile (orientation 0's item writes it)
      float2* Xk = SAVE_Z && oB == 0 ? sd->X + (size_t)item.tile * kSpecHalf : nullptr;
      tile_forward_spectrum<FLT, SAVE_Z, PadLayout>(raw, W, Nyq, tw, tlane, Xk, t, [] {});
    } else {
      uint8_t* raw = rawG + ((C0 - kX) & 15);
      const WindowSpan<FLT> span(sd, C0);
      if (!span.all()) {
        raw_window_copy<FLT>(sd, R0, C0, raw, span.iA, span.iB, t);
        __syncthreads();
      }
      tile_forward_spectrum<FLT, false, PadLayout>(raw, W, Nyq, tw, tlane, nullptr, t, load_first);
    }
    // the spectrum of a lane block is complete for its four warps; the next
    // item's record becomes visible with I2's barrier
    cp_async_wait();
    tmem_fence_before();
    named_barrier(1 + quad, kTileThreads / 4);
    tmem_fence_after();

    // tiles holding window column 0 or column dataW of a map with fftW == dataW
    const bool wrapTile = sd->wrapW != 0 && (C0 == 0 || C0 + V >= sd->cCols);
    // window positions x in [kX, xHi) are this tile's valid outputs; only
    // its first Vr valid rows lie inside the map, and the x-passes run on
    // those alone (a tile of the last tile row may hold only a few)
    const int xHi = min(kX + V, sd->cCols - C0 + kX);
    const int Vr = min(V, sd->cRows - R0);
    // I4's thread keeps column group n1 = t mod 8 for the whole tile: bit n2
    // of xMask says whether its output x = n1 + 8 n2 is in [kX, xHi)
    unsigned int xMask = 0;
#pragma unroll
    for (int n2 = 0; n2 < 16; ++n2) {
      const int x = (t & 7) + 8 * n2;
      xMask |= (x >= kX && x < xHi ? 1u : 0u) << n2;
    }
    // The x-passes give a warp every 16th block of four rows, so the first
    // (blocks mod 16) warps run one block more than the others.  A block takes
    // about as long as six of I1's 16 row groups, so in the I1 behind the
    // x-passes the m of a lane block's four warps that had the extra block
    // take fewer row groups (in twelfths: `few`) and the others more, and the
    // four reach I2 together.  1080p tile kernel: 238.0 us with four groups
    // each, 237.0 / 233.7 / 232.1 with a block counted as 2 / 4 / 6 groups;
    // 244.9 with the groups handed out by a shared-memory counter.
    const int extra = ((Vr + 3) >> 2) & 15;
    int m = 0, before = 0;   // of the lane block's warps with an extra block: all, and those before this one
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      m += quad + 4 * i < extra;
      before += i < h && quad + 4 * i < extra;
    }
    const int few = max(0, 48 - 18 * (4 - m)), many = m < 4 ? (192 - m * few) / (4 - m) : 0;
    const int begin12 = before * few + (h - before) * many + 6;
    const int k2Begin = begin12 / 12, k2End = (begin12 + (warp < extra ? few : many)) / 12;
    for (int o = oB; o < oE; ++o) {
      // I1: y-dim pass B' with the spectrum product Z = X * G on the rows
      // 8 k2 + k1 (the item's first I1 follows the forward transform: four
      // groups k2 a warp)
      if (!mbar_wait(bar0, ph)) fault = true;
      __syncwarp();   // the warp-collective TMEM stores below need a converged warp
      const int kB = o > oB ? k2Begin : 4 * h, kE = o > oB ? k2End : 4 * h + 4;
#pragma unroll 1
      for (int k2 = kB; k2 < kE; ++k2) {
        float2 v[8];
        tmem_load8(tlane + 16 * k2, v);
        const float4* Ga = reinterpret_cast<const float4*>(Gbuf) + gpos(8 * k2, t & 127) / 4;
        const float4 ga0 = Ga[0], ga1 = Ga[kTile];
        const float ga[8] = {ga0.x, ga0.y, ga0.z, ga0.w, ga1.x, ga1.y, ga1.z, ga1.w};
        // the group's twiddles, read before the TMEM stores
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
      ph ^= 1u;
      tmem_wait_st();
      tmem_fence_before();
      // a lane's first y-pass is complete when the four warps of its lane
      // block are done; W is free when every warp has finished the previous
      // orientation's x-passes, which they signal before their I1
      named_barrier(1 + quad, kTileThreads / 4);
      tmem_fence_after();
      if (o > oB) {
        if (!mbar_wait(barW, phW)) fault = true;
        phW ^= 1u;
        __syncwarp();
      }
      // I2: y-dim pass A' -> natural y (all 128 rows: storing only the
      // valid rows, under a predicate per store, measured 11% slower)
#pragma unroll
      for (int it = 0; it < 2; ++it) {
        const int n1 = h + 4 * it;
        float2 v[16];
        tmem_load16(tlane + kTmemY + 32 * n1, v);
        dft16<true>(v);
#pragma unroll
        for (int n2 = 0; n2 < 16; ++n2) W[widx(n1 + 8 * n2, pcol)] = v[n2];
      }
      tmem_fence_before();
      // W holds the y-transformed tile; the TMEM y-pass area is free and the
      // G buffer consumed
      __syncthreads();
      tmem_fence_after();
      if (o + 1 < oE) {
        if (t == 0) {   // orientation o + 1's spectrum lands during I3 and I4
          fence_proxy_async();
          bulk_load(gdst, sd->G + (size_t)(o + 1) * kSpecFloats, kSmemG, bar0);
        }
      } else if constexpr (!FLT) {   // the next item's window lands in the free G buffer
        const TileWork nx = qItem[slot ^ 1];
        const ScaleDev* nsd = qScale + (slot ^ 1);
        if (nx.oBegin < nx.oEnd) {
          const int ny = nx.tile / nsd->tilesX, nX = nx.tile - ny * nsd->tilesX;
          raw_chunks_load<false>(nsd, ny * nsd->V, nX * nsd->V, rawG, t);
        }
      }
      // The x-passes, four valid rows to a warp at a time: I3 (pass B', two
      // rows of 16 items a step), then I4 (pass A' -> natural x, the complex
      // magnitude of valid outputs; eight items a row) on the same rows, with
      // no CTA barrier between them.  Behind a barrier all four warps of a
      // scheduler loaded, then computed, then stored at the same time (65% of
      // cycles issued); warps that start a block, finish one or run the next
      // orientation's I1 at their own pace overlap these.  The map's
      // addresses are read from the record here (held across the
      // orientation's passes they cost registers the transforms need).
      {
        const int lane = t & 31, k2 = lane & 15, n1 = lane & 7;
        float2 twr[8];
#pragma unroll
        for (int m = 1; m < 8; ++m) twr[m] = tw[m * 17 + k2];
        const int cPitch = lds_now(&sd->cPitch);
        // output x = n1 + 8 n2 of the lane's row goes to dst[8 n2]
        float* __restrict__ dst = lds_now(&sd->C) + o * lds_now(&sd->cStride) +
                                  (long long)(R0 + 4 * warp + (lane >> 3)) * cPitch + (C0 - kX) + n1;
#pragma unroll 1
        for (int r0 = 4 * warp; r0 < Vr; r0 += 4 * (kTileThreads / 32), dst += 4 * (kTileThreads / 32) * cPitch) {
#pragma unroll 1
          for (int r = r0 + (lane >> 4); r < min(Vr, r0 + 4); r += 2) {
            float2* wr = W + widx(kX + r, 8 * k2);
            float2 v[8];
#pragma unroll
            for (int k1 = 0; k1 < 8; ++k1) v[k1] = wr[k1];
            dft8<true>(v);
#pragma unroll
            for (int m = 0; m < 8; ++m) wr[m] = m ? c_mulc(v[m], twr[m]) : v[0];
          }
          __syncwarp();
          const int r = r0 + (lane >> 3), gy = R0 + r;
          if (r < Vr) {
            const float2* wr = W + widx(kX + r, n1);
            float2 v[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m] = wr[9 * m];
            dft16<true>(v);
            if (!wrapTile) {
#pragma unroll
              for (int n2 = 0; n2 < 16; ++n2)
                if ((xMask >> n2) & 1u) dst[8 * n2] = cmag(v[n2]);
            } else {
              // fftW == dataW: the stencils read window column dataW of row r
              // at the flat address r*fftW + fftW, the torus element (r + 1, 0),
              // so that element also goes to (r, dataW); the window's own
              // (r, dataW) output is kept only on the last row
              const int cCols = lds_now(&sd->cCols), cRows = lds_now(&sd->cRows);
#pragma unroll
              for (int n2 = 0; n2 < 16; ++n2) {
                const int gx = C0 - kX + n1 + 8 * n2;
                if ((xMask >> n2) & 1u) {
                  const float m = cmag(v[n2]);
                  if (!(gx == cCols - 1 && gy < cRows - 1)) dst[8 * n2] = m;
                  if (gx == 0 && gy >= 1) dst[8 * n2 - cPitch + cCols - 1] = m;
                }
              }
            }
            if constexpr (SAVE_Z && FLT) {   // e + i o, as these lanes hold it
              const int bpt = kept_tile_blocks(V);
              float4* z = reinterpret_cast<float4*>(
                              lds_now(&sd->Z) + (((size_t)o * sd->tilesX + tx) * kept_column_blocks(*sd) + ty * bpt + (r0 >> 2)) * kKeptBlock) +
                          lane;
#pragma unroll
              for (int p = 0; p < 8; ++p)
                if (16 * p + 15 >= kX && 16 * p < xHi)
                  __stcs(z + 32 * p, make_float4(v[2 * p].x, v[2 * p].y, v[2 * p + 1].x, v[2 * p + 1].y));
            }
            if constexpr (SAVE_Z && !FLT) {   // e + i o, laid out as the magnitudes
              float2* __restrict__ z = sd->Z + (dst - sd->C);
              const int cCols = sd->cCols, cRows = sd->cRows;
#pragma unroll
              for (int n2 = 0; n2 < 16; ++n2) {
                const int gx = C0 - kX + n1 + 8 * n2;
                if ((xMask >> n2) & 1u) {
                  if (!(wrapTile && gx == cCols - 1 && gy < cRows - 1)) z[8 * n2] = v[n2];
                  if (wrapTile && gx == 0 && gy >= 1) z[8 * n2 - cPitch + cCols - 1] = v[n2];
                }
              }
            }
          }
        }
        // this warp no longer reads W (the item's last orientation is ordered
        // against the next item by its barrier)
        __syncwarp();
        if (lane == 0 && o + 1 < oE) mbar_arrive(barW);
      }
    }
  }
  if (fault) {
    // a wait expired: the thread that saw it records it (warps come to a wait
    // at different times: none speaks for another), then the copies still in
    // flight get a second bounded chance to land before the CTA releases its
    // memory
    atomicOr(fault_word, 1u);
    (void)mbar_wait(bar0, ph ^ 1);
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  if ((t >> 5) == 0) tmem_dealloc_warp(*tmemSlot);
}

// ---------------------------------------------------------------------------
// k_gabor_tiles_ws: the same tile computation with warp-specialised,
// pipelined orientations
// ---------------------------------------------------------------------------
// After the tile's forward transform (all 16 warps, as above), warps 0-7
// (group Y) run the spectrum product and the two inverse y-passes of each
// orientation (TMEM in, TMEM y-area, then the valid rows into a shared-memory
// row buffer), while warps 8-15 (group X) run the two inverse x-passes and
// the complex magnitude of the previous orientation from the other buffer.
// Two row buffers of kWsRows x 128 complex alternate between orientations;
// named barriers hand them over (full: Y -> X, empty: X -> Y), and each group
// orders its own passes with a 256-thread named barrier, so no CTA-wide
// barrier stands inside the orientation loop.  G_o is read from L2 (the
// second buffer takes the space it would be staged in), a thread's eight values
// as two 16-byte loads.  Needs V <= kWsRows.  64 mixed images, one CTA a tile:
// 7.47 ms a detection (8.69 with the values loaded one by one in the order of
// the stored spectrum and the window staged value by value; k_gabor_tiles
// 6.87).
constexpr int kWsRows = 104;                                  // largest V this kernel takes
constexpr int kWsBuf = kWsRows * kTile;                       // complex per row buffer
constexpr int kWsSmemW = 2 * kWsBuf * 8;                      // both row buffers (also the forward scratch)
constexpr int kWsSmem = kWsSmemW + kSmemTw + 16;              // + twiddles, TMEM base slot
static_assert(kWsSmem <= 232448, "warp-specialised tile kernel exceeds the 227 KB shared-memory limit");
// forward transform scratch inside the two buffers: packed rows 0..63, the
// Hermitian half at rows 64..127, the Nyquist slot column at row 192
static_assert(2 * kWsRows >= 193, "forward-transform scratch does not fit the row buffers");
constexpr int kWsGroup = kTileThreads / 2;   // threads per group
enum : int { kBarY = 1, kBarX = 2, kBarFull0 = 3, kBarEmpty0 = 5 };   // named barrier ids (0 is __syncthreads)

__device__ __forceinline__ void named_barrier_arrive(int id, int n) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

template <bool FLT>
__global__ void __launch_bounds__(kTileThreads, 1)
k_gabor_tiles_ws(const ScaleDev* __restrict__ sds, const TileWork* __restrict__ work, int nwork) {
  extern __shared__ float4 smem4[];
  char* base = reinterpret_cast<char*>(smem4);
  float2* Wb = reinterpret_cast<float2*>(base);
  float2* tw = reinterpret_cast<float2*>(base + kWsSmemW);
  uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(base + kWsSmemW + kSmemTw);
  float2* Nyq = Wb + 192 * kTile;    // forward transform only
  const int t = threadIdx.x;
  if (t < 8 * 17) {
    const int n1 = t / 17, k2 = t % 17;
    tw[t] = k2 < 16 ? c_w128[(n1 * k2) & 127] : make_float2(0.f, 0.f);
  }
  if ((t >> 5) == 0) tmem_alloc_warp(smem_u32(tmemSlot));
  griddep_launch_dependents();
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  griddep_wait();   // the pyramid levels come from the previous kernel
  const uint32_t tlane = *tmemSlot + ((uint32_t)((t >> 5) & 3) << 21);
  const int pI1 = t & 127;
  const bool groupY = t < kWsGroup;
  const int tg = t & (kWsGroup - 1);   // index within the group
  const int hY = tg >> 7;              // group Y: spectrum rows k2 = hY + 2 q

  for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
    const TileWork item = work[w];
    const int oB = item.oBegin, oE = item.oEnd, nO = oE - oB;
    if (nO <= 0) continue;   // empty slot of a padded plan
    const ScaleDev* sd = sds + item.entry;
    const int kX = sd->kX, V = sd->V;
    const int ty = item.tile / sd->tilesX, tx = item.tile - ty * sd->tilesX;
    const int R0 = ty * V, C0 = tx * V;
    __syncthreads();   // previous tile finished with every buffer
    auto* raw = reinterpret_cast<typename RawWindow<FLT>::T*>(Wb + RotLayout::kHalf);
    raw_chunks_load<FLT>(sd, R0, C0, raw, t);
    raw += (C0 - kX) & (WindowSpan<FLT>::kVals - 1);
    const WindowSpan<FLT> span(sd, C0);
    if (!span.all()) raw_window_copy<FLT>(sd, R0, C0, raw, span.iA, span.iB, t);
    cp_async_wait();
    __syncthreads();
    tile_forward_spectrum<FLT, false, RotLayout>(raw, Wb, Nyq, tw, tlane, nullptr, t, [] {});
    tmem_fence_before();
    __syncthreads();   // spectrum in TMEM; the forward scratch in the row buffers is dead
    tmem_fence_after();
    if (groupY) {
      for (int o = oB; o < oE; ++o) {
        const int b = (o - oB) & 1;
        float2* Wo = Wb + b * kWsBuf;
        const float4* __restrict__ Go = reinterpret_cast<const float4*>(sd->G + (size_t)o * kSpecFloats) + glane(pI1);
        // I1: y-dim pass B' with the spectrum product (TMEM in, TMEM y-area
        // out); each quarter's G values, two 16-byte loads, come one quarter
        // ahead
        float4 ga = __ldg(Go + 2 * hY * kTile), gb = __ldg(Go + (2 * hY + 1) * kTile);
#pragma unroll 1
        for (int q = 0; q < 8; ++q) {
          const int k2 = hY + 2 * q;
          float2 v[8];
          const int k2n = q < 7 ? k2 + 2 : k2;
          const float4 gan = __ldg(Go + 2 * k2n * kTile), gbn = __ldg(Go + (2 * k2n + 1) * kTile);
          tmem_load8(tlane + 16 * k2, v);
          float2 twr[8];
#pragma unroll
          for (int n1 = 1; n1 < 8; ++n1) twr[n1] = tw[n1 * 17 + k2];
          const float g[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
#pragma unroll
          for (int k1 = 0; k1 < 8; ++k1) v[k1] = c_scale(v[k1], g[k1]);
          dft8<true>(v);
#pragma unroll
          for (int n1 = 0; n1 < 8; ++n1)
            tmem_store1(tlane + kTmemY + 2 * (16 * n1 + k2), n1 ? c_mulc(v[n1], twr[n1]) : v[0]);
          ga = gan;
          gb = gbn;
        }
        tmem_wait_st();
        tmem_fence_before();
        named_barrier(kBarY, kWsGroup);   // the y-area holds orientation o's first y-pass
        tmem_fence_after();
        if (o - oB >= 2) named_barrier(kBarEmpty0 + b, kTileThreads);   // group X is done with orientation o - 2
        // I2: y-dim pass A' -> natural y; the valid rows into buffer b
#pragma unroll
        for (int it = 0; it < 4; ++it) {
          const int j = tg + it * kWsGroup;
          const int p = j & 127, n1 = j >> 7;
          float2 v[16];
          tmem_load16(tlane + kTmemY + 32 * n1, v);
          dft16<true>(v);
#pragma unroll
          for (int n2 = 0; n2 < 16; ++n2) {
            const int y = n1 + 8 * n2 - kX;
            if (y >= 0 && y < V) Wo[RotLayout::at(y, p)] = v[n2];
          }
        }
        tmem_fence_before();
        named_barrier_arrive(kBarFull0 + b, kTileThreads);   // buffer b holds orientation o
        named_barrier(kBarY, kWsGroup);                 // every thread is done reading the y-area
        tmem_fence_after();
      }
    } else {
      const int cRows = sd->cRows, cCols = sd->cCols, cPitch = sd->cPitch;
      const bool wrapTile = sd->wrapW != 0 && (C0 == 0 || C0 + V >= cCols);
      const int xHi = min(kX + V, cCols - C0 + kX);
      const int Vr = min(V, cRows - R0);   // valid rows inside the map
      // I4 keeps column group n1 = tg mod 8 for the whole tile
      unsigned int xMask = 0;
#pragma unroll
      for (int n2 = 0; n2 < 16; ++n2) {
        const int x = (tg & 7) + 8 * n2;
        xMask |= (x >= kX && x < xHi ? 1u : 0u) << n2;
      }
      float* __restrict__ C0p = sd->C;
      const long long cStride = sd->cStride;
      for (int o = oB; o < oE; ++o) {
        const int b = (o - oB) & 1;
        float2* Wo = Wb + b * kWsBuf;
        float* __restrict__ Cout = C0p + (size_t)o * cStride;
        named_barrier(kBarFull0 + b, kTileThreads);
        // I3: x-dim pass B' on the V rows of the buffer (a thread's k2 is
        // fixed: its twiddles are loaded once)
        {
          const int k2 = tg & 15;
          float2 twr[8];
#pragma unroll
          for (int n1 = 1; n1 < 8; ++n1) twr[n1] = tw[n1 * 17 + k2];
          for (int j = tg; j < Vr * 16; j += kWsGroup) {
            const int y = j >> 4;
            float2 v[8];
#pragma unroll
            for (int k1 = 0; k1 < 8; ++k1) v[k1] = Wo[RotLayout::at(y, 8 * k2 + k1)];
            dft8<true>(v);
#pragma unroll
            for (int n1 = 0; n1 < 8; ++n1) Wo[RotLayout::at(y, 8 * k2 + n1)] = n1 ? c_mulc(v[n1], twr[n1]) : v[0];
          }
        }
        named_barrier(kBarX, kWsGroup);
        // I4: x-dim pass A' -> natural x; complex magnitude of valid outputs
        for (int j = tg; j < Vr * 8; j += kWsGroup) {
          const int y = j >> 3, n1 = j & 7;
          float2 v[16];
#pragma unroll
          for (int k2 = 0; k2 < 16; ++k2) v[k2] = Wo[RotLayout::at(y, 8 * k2 + n1)];
          dft16<true>(v);
          const int gy = R0 + y;
          if (gy < cRows) {
            float* dst = Cout + (size_t)gy * cPitch;
            if (!wrapTile) {
              float* dstx = dst + (C0 - kX);
#pragma unroll
              for (int n2 = 0; n2 < 16; ++n2)
                if ((xMask >> n2) & 1u) dstx[n1 + 8 * n2] = cmag(v[n2]);
            } else {
              // fftW == dataW: window column dataW of row r is the torus
              // element (r + 1, 0) (see k_gabor_tiles)
#pragma unroll
              for (int n2 = 0; n2 < 16; ++n2) {
                const int x = n1 + 8 * n2;
                const int gx = C0 + x - kX;
                if (x >= kX && x < kX + V && gx < cCols) {
                  const float m = cmag(v[n2]);
                  if (!(gx == cCols - 1 && gy < cRows - 1)) dst[gx] = m;
                  if (gx == 0 && gy >= 1) Cout[(size_t)(gy - 1) * cPitch + cCols - 1] = m;
                }
              }
            }
          }
        }
        // buffer b may be refilled by orientation o + 2; the item's last two
        // orientations are ordered against the next tile by its barrier
        if (o - oB < nO - 2) named_barrier_arrive(kBarEmpty0 + b, kTileThreads);
      }
    }
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  if ((t >> 5) == 0) tmem_dealloc_warp(*tmemSlot);
}
