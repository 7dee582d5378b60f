// Learned artifact correction: a 2.5D residual CNN on reconstructed slices,
// with its own BF16 training and inference kernels.
//
// Network (8 conv layers, 3x3, zero padding, stride 1):
//   input  : 5 adjacent slices of a half-view reconstruction, u = mu / mu_w - 1,
//            NHWC BF16 with the 5 channels padded to 16
//   L1     : 16 -> 32, ReLU;   L2..L7: 32 -> 32, ReLU;   L8: 32 -> 16 (channel 0 used)
//   output : centre slice (FP32, not rounded) + mu_w * L8 channel 0
//
// Inside the network activations and gradients are stored by planes: [B][H][C / 8][Wp][8]
// BF16, a row of 16-byte pixel chunks per 8 channels with Wp = W + 2 chunks, a zero chunk
// before the image's first pixel and one after its last, so that a tile's halo row is at most
// 130 contiguous chunks wherever it lies (rows above and below the image come from a zero
// row). One untiled bulk copy brings such a row into shared memory, and an epilogue's stores
// are contiguous over the warp. (With NHWC activations the same rows were TMA boxes of 8
// channels x 130 pixels, 16 bytes at a time, and bounded the kernels.) Every epilogue writes
// its rows' two zero chunks too, and a row's last tile takes no more than the row has, so
// nothing depends on what a buffer held. (Rows padded to whole tiles would need no short
// tile, but up to eight times the memory for narrow images, twice for W = 129.)
//
// Buffers: inference alternates between two activations (layer k reads one and writes the
// other) and keeps the input: 80 channels per pixel instead of the 304 of all layers and
// gradients. A training step needs every layer's output; its gradients alternate between a
// buffer and the last layer's input, of which the gradient's first step is the last use (288
// channels per pixel). Both are kept from call to call.
//
// Convolutions run as implicit GEMMs on the 5th-generation tensor cores: one
// tile is 128 output pixels of one image row (M = 128, TMEM lanes) by COUT
// channels, K = 9 taps x CIN channels. The input rows lie in shared memory
// in the K-major no-swizzle layout (one plane of 16-byte pixel chunks per
// 8-channel group), so the A operand of horizontal tap dx is the same buffer
// seen 16 dx bytes further on: descriptor offsets replace an im2col copy.
//
// With N = COUT = 32 an MMA would spend its time reading A: 4 KB of shared
// memory (32 clocks) for 16 clocks of multiplication, nine times per input
// row. So the three vertical taps are stacked along N: input row r times the
// weights of dy = 2, 1, 0 adds to output rows r - 1, r, r + 1, whose
// accumulators are neighbouring column groups of a ring of kSlots in TMEM
// (N = 96: one MMA per horizontal tap and 16 channels, 6 instead of 18 per
// row, split in two where the three groups cross the ring's end). An output
// row's sums run over (dy, dx, channels) in the same order as nine separate
// taps', so the results are the same bits. 32 slices of 512 x 512, a 32 -> 32
// layer: 267 -> 189 us (its bytes at the copy rate: 165 us).
//
// The weights (B operand) stay in shared memory for the CTA's life.
// Persistent, warp-specialised CTAs: warp 0 issues the copies into a ring of
// input rows, warp 1 the MMAs, warps 2-5 read the finished accumulators and
// run the epilogue (bias + ReLU + BF16 store; gradient masking by the forward
// activation; fused residual + loss + output gradient), so loads, MMAs and
// stores of consecutive rows overlap. Every mbarrier wait is bounded and sets
// an error flag when it gives up. The backward data pass is the same kernel
// with the weights transposed and flipped. Weight gradients are a second
// tensor-core kernel that contracts over the pixels (wgrad_tc_kernel).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "hr_internal.h"

namespace {

constexpr int kTileM = 128;                  // output pixels per tile (one row segment)
constexpr int kHalo = kTileM + 2;            // halo pixels per row
constexpr int kBox = kHalo * 16;             // bytes of one halo row: 130 pixel chunks of 8 channels
constexpr int kPlane = 17 * 128;             // plane stride: one halo row, 128-byte aligned
// Four CTAs per SM (the most that TMEM holds with four accumulators each) with a short ring: the epilogue's
// latency per row, not the copies in flight, is what more CTAs hide (per 32 -> 32 layer of 32 slices of
// 512 x 512: two CTAs with rings of 6 232 us, three 202, four with rings of 4 201, of 3 189).
constexpr int kRing = 3;                     // halo ring: input rows in flight
constexpr int kConvCtas = 4;                 // CTAs per SM that registers must allow
constexpr int kThreads = 192;                // warp 0 TMA, warp 1 MMA, warps 2-5 epilogue
constexpr int kSlots = 4;                    // accumulators in flight: three being added to, one being read
// TMEM columns of a CTA. (More than it needs would be worse than a waste: the CTAs that registers and shared
// memory let onto an SM wait there for TMEM while other SMs are idle.)
constexpr int tmem_cols(int cout) { return kSlots * cout; }
constexpr uint32_t kWaitLimit = 1u << 22;    // try_wait rounds before a wait is declared hung
constexpr int kLayers = 8;
constexpr int kCin[kLayers] = {16, 32, 32, 32, 32, 32, 32, 32};
constexpr int kCout[kLayers] = {32, 32, 32, 32, 32, 32, 32, 16};

enum Epi { EPI_RELU = 0, EPI_MASK = 1, EPI_LOSS = 2, EPI_RESID = 3, EPI_RAW = 4 };

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// K-major, no-swizzle UMMA shared-memory descriptor: core matrices of 8 rows x
// 16 bytes (128 contiguous bytes); lbo = bytes between core matrices along K,
// sbo = bytes between 8-row groups along M/N; version 1, layout 0 (none).
__device__ __forceinline__ uint64_t desc_noswz(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
         (1ull << 46);
}

// BF16 x BF16 -> F32, both K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
}

__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

// Bounded wait on an mbarrier phase; gives up (returning false) when another
// role of the CTA has aborted, or after `limit` rounds (then records the
// error and aborts the CTA).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t phase, volatile int* abort_flag, int* err,
                                          uint32_t limit) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t i = 0; i < limit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(phase)
        : "memory");
    if (done) return true;
    if (*abort_flag) return false;
  }
  atomicExch(err, 1);
  *abort_flag = 1;
  return false;
}

// Bounded wait for a phase the thread itself started (issued TMA copies, or
// the completion of its own tensor-core operations), ignoring the abort flag:
// an aborting CTA still lets them finish before it frees TMEM and exits.
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t phase, int* err, uint32_t limit) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t i = 0; i < limit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(phase)
        : "memory");
    if (done) return;
  }
  atomicExch(err, 2);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// The convolution and weight-gradient kernels are launched as programmatic dependents: when the last CTA of the
// previous kernel has ended, this one's start, set up their barriers and take TMEM while that kernel's writes are
// still being flushed. No thread reads or writes global memory before this returns: the previous kernel is then
// complete and its writes visible. 64 slices of 512 x 512 in two chunks 3.06 -> 2.98 ms, slice by slice 11.9 ->
// 9.7, a training step of eight 2.00 -> 1.96. (With a trigger before a kernel's end, so that CTAs move in as
// others leave, the column strips of a row no longer run together: 3.10 and 2.03 ms.)
__device__ __forceinline__ void after_previous_kernel() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Untiled bulk copy of `bytes` (a multiple of 16; both addresses 16-byte aligned), reported to `bar`.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Chunks of a padded row, and the chunk offset of channel group c of image row (b, y) (G groups).
__host__ __device__ constexpr int padded_width(int W) { return W + 2; }
__device__ __forceinline__ size_t plane_row(int b, int H, int y, int G, int c, int Wp) {
  return (((size_t)b * H + y) * G + c) * Wp;
}

__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  uint32_t w;
  memcpy(&w, &h, sizeof w);
  return w;
}

template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float (&v)[N]);

template <>
__device__ __forceinline__ void tmem_ld<16>(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

template <>
__device__ __forceinline__ void tmem_ld<32>(uint32_t taddr, float (&v)[32]) {
  float a[16], b[16];
  tmem_ld<16>(taddr, a);
  tmem_ld<16>(taddr + 16, b);
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    v[i] = a[i];
    v[16 + i] = b[i];
  }
}

// Zeros into N accumulator columns of the warp's 32 lanes.
template <int N>
__device__ __forceinline__ void tmem_zero(uint32_t taddr) {
#pragma unroll
  for (int c = 0; c < N; c += 16)
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
        "%1};" ::"r"(taddr + c),
        "r"(0)
        : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

struct ConvArgs {
  const uint4* in;       // input planes, CIN / 8 groups
  const uint4* zero;     // kHalo zero chunks
  const uint16_t* wimg;  // B operand image [3*CIN/8][3*COUT][8] BF16
  const float* bias;     // [COUT] (EPI_RELU, EPI_LOSS, EPI_RESID)
  uint4* out;            // output planes, COUT / 8 groups (EPI_RELU, EPI_MASK); output gradient (EPI_LOSS)
  const uint4* mask;     // planes of the forward activation whose > 0 passes the gradient (EPI_MASK)
  // residual epilogues: element (b, y, x) of base/target/pred at b*sb + (y*W + x)*sp
  const float* base;
  const float* target;   // EPI_LOSS
  float* pred;           // EPI_RESID output (EPI_LOSS: optional); EPI_RAW: channel 0 itself, [B][H][W]
  long long sb, sp;
  float scale;           // mu_w: pred = base + scale * r
  float grad_scale;      // EPI_LOSS: d loss / d r = grad_scale * (pred - target) / scale
  float* loss;           // EPI_LOSS: accumulates sum ((pred - target) / scale)^2
  int B, H, W, Wp;
  int* err;
  int stall_row;         // test hook: the CTA's input row of this index is never loaded (-1: none)
  uint32_t wait_limit;   // polls before a pipeline wait gives up
};

// Epilogue of one output row segment: the thread's pixel (b, y, x) with its COUT accumulator values.
template <int COUT, int EPI>
__device__ __forceinline__ void conv_epilogue(const ConvArgs& a, const float (&v)[COUT], const float* bias_s, int b,
                                              int y, int x, int lane) {
  const bool valid = x < a.W;  // a tile's pixels beyond the image hold nothing
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const size_t row = plane_row(b, a.H, y, COUT / 8, 0, a.Wp);
  if constexpr (EPI != EPI_RESID && EPI != EPI_RAW) {  // the zero chunks before the first and after the last pixel
    if (x == 0) {
#pragma unroll
      for (int c = 0; c < COUT / 8; ++c) a.out[row + (size_t)c * a.Wp] = zero;
    }
    if (x == a.W - 1) {
#pragma unroll
      for (int c = 0; c < COUT / 8; ++c) a.out[row + (size_t)c * a.Wp + a.Wp - 1] = zero;
    }
  }
  if constexpr (EPI == EPI_RELU) {
    if (!valid) return;
    uint4* o = a.out + row + x + 1;
#pragma unroll
    for (int c = 0; c < COUT / 8; ++c) {
      const float4* bp = reinterpret_cast<const float4*>(bias_s) + 2 * c;
      const float4 b0 = bp[0], b1 = bp[1];
      const float bias[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
      float u[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) u[j] = fmaxf(v[8 * c + j] + bias[j], 0.0f);
      o[(size_t)c * a.Wp] = make_uint4(pack2(u[0], u[1]), pack2(u[2], u[3]), pack2(u[4], u[5]), pack2(u[6], u[7]));
    }
  } else if constexpr (EPI == EPI_MASK) {
    if (!valid) return;
    const uint4* m = a.mask + row + x + 1;
    uint4* o = a.out + row + x + 1;
#pragma unroll
    for (int c = 0; c < COUT / 8; ++c) {
      const uint4 mv = __ldg(m + (size_t)c * a.Wp);
      const uint32_t mw[4] = {mv.x, mv.y, mv.z, mv.w};
      float u[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        u[2 * j] = bf_lo(mw[j]) > 0.0f ? v[8 * c + 2 * j] : 0.0f;
        u[2 * j + 1] = bf_hi(mw[j]) > 0.0f ? v[8 * c + 2 * j + 1] : 0.0f;
      }
      o[(size_t)c * a.Wp] = make_uint4(pack2(u[0], u[1]), pack2(u[2], u[3]), pack2(u[4], u[5]), pack2(u[6], u[7]));
    }
  } else if constexpr (EPI == EPI_RAW) {
    if (valid) a.pred[((size_t)b * a.H + y) * a.W + x] = v[0] + bias_s[0];
  } else {
    const float r = v[0] + bias_s[0];
    float e2 = 0.0f;
    [[maybe_unused]] uint4 g0 = zero;
    if (valid) {
      const size_t off = (size_t)b * a.sb + ((size_t)y * a.W + x) * a.sp;
      const float pr = a.base[off] + a.scale * r;
      if constexpr (EPI == EPI_RESID) {
        a.pred[off] = pr;
      } else {
        if (a.pred) a.pred[off] = pr;
        const float e = (pr - a.target[off]) / a.scale;
        e2 = e * e;
        g0 = make_uint4(pack2(a.grad_scale * e, 0.0f), 0u, 0u, 0u);
      }
    }
    if constexpr (EPI == EPI_LOSS) {
#pragma unroll
      for (int c = 0; c < COUT / 8; ++c)
        if (valid) a.out[row + (size_t)c * a.Wp + x + 1] = c == 0 ? g0 : zero;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) e2 += __shfl_xor_sync(0xffffffffu, e2, o);
      if (lane == 0 && e2 != 0.0f) atomicAdd(a.loss, e2);
    }
  }
}

template <int CIN, int COUT, int EPI>
__global__ void __launch_bounds__(kThreads, kConvCtas) conv_tc_kernel(const __grid_constant__ ConvArgs a) {
  constexpr int G = CIN / 8;                 // 8-channel groups (copies per input row)
  constexpr int kRow = G * kPlane;           // bytes of one input row (130 pixels)
  constexpr int kWBytes = 9 * CIN * COUT * 2;
  constexpr int kKSteps = 3 * CIN / 16;      // per input row: horizontal taps x 16-channel steps
  static_assert(CIN % 16 == 0 && (COUT == 16 || COUT == 32), "unsupported channel counts");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  uint8_t* wsm = smem + kRing * kRow;  // weights
  uint64_t* full = reinterpret_cast<uint64_t*>(wsm + kWBytes);
  uint64_t* empty = full + kRing;
  uint64_t* tfull = empty + kRing;
  uint64_t* tempty = tfull + kSlots;
  uint64_t* mdone = tempty + kSlots;  // the MMA issuer's last commit (one spare slot keeps 16-byte alignment)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mdone + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* bias_s = reinterpret_cast<float*>(tmem_slot + 4);  // 16-byte aligned, COUT floats

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < kRing; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], 128);
    }
    mbar_init(mdone, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(tmem_cols(COUT)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  after_previous_kernel();
  for (int i = tid; i < kWBytes / 16; i += kThreads)
    reinterpret_cast<uint4*>(wsm)[i] = __ldg(reinterpret_cast<const uint4*>(a.wimg) + i);
  if (tid < COUT) bias_s[tid] = a.bias ? __ldg(a.bias + tid) : 0.0f;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const uint32_t smem_a = smem_u32(smem), w_a = smem_u32(wsm);

  // The B x H output rows are cut into equal shares of consecutive rows, one per group of nseg CTAs, and
  // each CTA of a group takes one 128-pixel column strip of the share: every CTA has the same work to
  // within a row (chunks of fixed length left five rounds of work for 4.1 rounds' worth at 8 images), and
  // a group's copies and stores fall into the same stretch of memory at about the same time (with every
  // CTA on a stretch of its own a 32 -> 32 layer of 32 slices of 512 x 512 took 248 us, so 202). A share
  // crosses from one image to the next in pieces; a piece of n output rows loads n + 2 input rows (zero
  // rows above and below the image).
  const int nseg = (a.W + kTileM - 1) / kTileM;
  const int seg = blockIdx.x % nseg, groups = gridDim.x / nseg, group = blockIdx.x / nseg;
  const long long rows = (long long)a.B * a.H;
  const long long r0 = rows * group / groups, r1 = rows * (group + 1) / groups;
  if (warp == 0) {
    // ---- producer: input rows of each piece into the ring, G halo rows each ------------------
    if (lane == 0) {
      // a row's last strip may be short: what lies behind its chunks in the ring feeds only accumulator rows
      // of pixels beyond the image, which the epilogue leaves out
      const uint32_t bytes = (uint32_t)(min(a.W - seg * kTileM, kTileM) + 2) * 16;
      int h = 0;  // input rows loaded by this CTA
      int last_h[kRing];
      for (int s = 0; s < kRing; ++s) last_h[s] = -1;
      bool ok = true;
      for (long long r = r0; r < r1 && ok;) {
        const int b = (int)(r / a.H);
        const int y0 = (int)(r - (long long)b * a.H), ny = (int)min((long long)(a.H - y0), r1 - r);
        r += ny;
        for (int j = 0; j < ny + 2; ++j, ++h) {
          const int s = h % kRing;
          if (h >= kRing && !mbar_wait(&empty[s], ((h / kRing) - 1) & 1, abort_flag, a.err, a.wait_limit)) {
            ok = false;
            break;
          }
          if (h == a.stall_row) continue;  // test hook: this row's slot is never filled
          last_h[s] = h;
          mbar_expect_tx(&full[s], G * bytes);
          const int y = y0 - 1 + j;
          const bool in = y >= 0 && y < a.H;
          const uint4* src = in ? a.in + plane_row(b, a.H, y, G, 0, a.Wp) + seg * kTileM : a.zero;
          for (int g = 0; g < G; ++g)
            bulk_load(smem_a + s * kRow + g * kPlane, src + (in ? (size_t)g * a.Wp : 0), bytes, &full[s]);
        }
      }
      // every issued copy lands before the CTA exits (after an abort nobody consumes them)
      for (int s = 0; s < kRing; ++s)
        if (last_h[s] >= 0) mbar_drain(&full[s], (last_h[s] / kRing) & 1, a.err, a.wait_limit);
    }
  } else if (warp == 1) {
    // ---- MMA issuer: input row i of a piece adds to its output rows i - 2, i - 1 and i -------
    if (lane == 0) {
      int h = 0, obase = 0;  // input rows consumed; output rows of the pieces before
      bool ok = true;
      for (long long r = r0; r < r1 && ok;) {
        const int ny = (int)min((long long)(a.H - (int)(r % a.H)), r1 - r);
        r += ny;
        for (int i = 0; i < ny + 2; ++i, ++h) {
          const int s = h % kRing;
          ok = mbar_wait(&full[s], (h / kRing) & 1, abort_flag, a.err, a.wait_limit);
          const int o = obase + i;  // the output row that starts here (if i < ny)
          if (ok && i < ny) ok = mbar_wait(&tempty[o % kSlots], (o / kSlots) & 1, abort_flag, a.err, a.wait_limit);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const int lo = max(i - 2, 0), hi = min(i, ny - 1);  // output rows of the piece
          const int first = (obase + lo) % kSlots, n = hi - lo + 1, m = min(n, kSlots - first);
          // the n column groups from row lo's on, in two where they cross the end of the ring; weights of
          // dy = i - lo downwards
          const uint32_t d0 = tmem + (uint32_t)first * COUT;
          const uint32_t bw = w_a + (uint32_t)(2 - (i - lo)) * (COUT * 16);
          const uint32_t id0 = idesc_bf16(m * COUT), id1 = idesc_bf16((n - m) * COUT);
#pragma unroll
          for (int k = 0; k < kKSteps; ++k) {
            const int dx = k / (CIN / 16), c0 = (k - dx * (CIN / 16)) * 16;
            const uint64_t ad = desc_noswz(smem_a + s * kRow + (c0 / 8) * kPlane + dx * 16, kPlane, 128);
            const uint32_t b = bw + (uint32_t)(dx * G + c0 / 8) * (3 * COUT * 16);
            umma(d0, ad, desc_noswz(b, 3 * COUT * 16, 128), id0, 1u);
            if (m < n) umma(tmem, ad, desc_noswz(b + (uint32_t)m * (COUT * 16), 3 * COUT * 16, 128), id1, 1u);
          }
          umma_commit(&empty[s]);                                    // the input row has been read
          if (i >= 2) umma_commit(&tfull[(obase + i - 2) % kSlots]);  // output row i - 2 is complete
        }
        obase += ny;
      }
      // every tensor-core operation issued above completes before TMEM is freed
      umma_commit(mdone);
      mbar_drain(mdone, 0, a.err, a.wait_limit);
    }
  } else {
    // ---- epilogue: warps 2-5, TMEM lane quarter warp % 4 --------------------------------------
    // Every accumulator is handed to the MMAs as zeros, so that one instruction may add to three.
    const int q = warp & 3;
    const uint32_t quarter = tmem + ((uint32_t)(q * 32) << 16);
    tmem_zero<COUT * kSlots>(quarter);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    for (int s = 0; s < kSlots; ++s) mbar_arrive(&tempty[s]);
    int it = 0;
    bool ok = true;
    for (long long r = r0; r < r1 && ok;) {
      const int b = (int)(r / a.H);
      const int y0 = (int)(r - (long long)b * a.H), ny = (int)min((long long)(a.H - y0), r1 - r);
      r += ny;
      for (int i = 0; i < ny; ++i, ++it) {
        const int acc = it % kSlots;
        const bool waited = mbar_wait(&tfull[acc], (it / kSlots) & 1, abort_flag, a.err, a.wait_limit);
        // the TMEM instructions below are warp-collective: the whole warp runs them or, where a lane saw an
        // abort that the others did not, none of it does
        if (!__all_sync(0xffffffffu, waited)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float v[COUT];
        tmem_ld<COUT>(quarter + acc * COUT, v);
        tmem_zero<COUT>(quarter + acc * COUT);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        mbar_arrive(&tempty[acc]);  // the registers hold the row: the accumulator may be reused
        conv_epilogue<COUT, EPI>(a, v, bias_s, b, y0 + i, seg * kTileM + q * 32 + lane, lane);
      }
    }
  }
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols(COUT)));
  }
}

// Weight gradients on the tensor cores: dW[co][tap][ci] += sum_p G[p][co] X[p + tap][ci],
// db[co] += sum_p G[p][co]. A contraction over pixels, so both operands are MN-major (a
// pixel's channels are contiguous). One tile is two output rows y, y + 1 of a 128-pixel
// column strip: the A operand is the four input rows y - 1 .. y + 2 (M = 128: row r, input
// channel ci), the B operand the two gradient rows (N = 2 COUT: row g, output channel), and
// for each horizontal tap dx the same buffer seen 16 dx bytes further on, so 3 x 8 MMAs
// (K = 16 pixels) give every D_dx[(r, ci)][(g, co)]; the combinations with 0 <= r - g <= 2
// are dW at dy = r - g, six of eight. Shared memory holds one plane of 16-byte pixel chunks
// per 8 channels (the no-swizzle layout: planes along M / N, groups of 8 pixels along K),
// filled by one bulk copy per row and group.
//
// Warp 9 issues the copies into a four-stage ring, warp 8 the MMAs; warps 0-7 sum each
// stage's gradient chunks for db, and every kWgGroup tiles add the finished accumulator (one
// of two in TMEM) to FP32 registers with rounding to nearest, so that the tensor core's own
// accumulation, which truncates, runs over 32 steps at most (left to run over a CTA's whole
// share it shrinks the gradients by 1.1e-5; over one, two or four tiles it cannot be told
// from the rounding of the FP32 sums). A warp reads its TMEM
// lane quarter (row r for 32 input channels) for one gradient row. At the end a CTA adds up what
// its warps hold of one gradient (two hold each weight's, eight each bias's) in shared memory
// and adds the sum to the result once: what is left of rounding are those additions, one
// after another, 2.5e-8 sqrt(CTAs / 3) of the sum (with an addition per warp the weights of 64
// CTAs' images were off by 1.4e-7 to 1.7e-7, now 1.2e-7, the biases of 148 CTAs' by 4e-7 to
// 9e-7, now below 4e-7; half the additions to memory, or an eighth, also take a training step
// of eight 512 x 512 from 1.91 to 1.75 ms).
// Every wait is bounded.
//
// The CUDA-core kernel this replaced (36 FP32 accumulators per thread, 13 shared-memory
// reads per 36 FMAs) took 1.40 ms per 32 -> 32 layer of 8 x 512 x 512, 11.0 of the 12.6 ms
// of a training step; this one 0.084 ms. Its MMAs would take 0.04 ms; the copies bound it:
// 0.147 ms with NHWC activations (16 bytes at a time), 0.114 by planes with one thread
// issuing a tile's 24 copies one after another, 0.104 with a lane to each (fewer MMAs,
// flushes or bias sums change nothing), 0.084 with one addition per CTA and weight to memory.
constexpr int kWgStages = 4;
constexpr int kWgGroup = 4;                          // tiles accumulated in TMEM before a flush
constexpr int kWgPlane = kHalo * 16;                 // bytes between planes
constexpr int kWgXPlanes = 16, kWgGPlanes = 8;       // M = 128, N <= 64
constexpr int kWgStage = (kWgXPlanes + kWgGPlanes) * kWgPlane;
constexpr int kWgWorkers = 8;                        // warps 0-7: bias sums and flushes
constexpr int kWgThreads = 32 * (kWgWorkers + 2);
constexpr int kWgTmemCols = 512;
constexpr size_t kWgSmem = (size_t)kWgStages * kWgStage + 256 + kWgWorkers * 32 * sizeof(float);
static_assert(3 * 32 * 3 * 32 * sizeof(float) <= (size_t)kWgStages * kWgStage, "the weights' sums reuse the ring");

template <int CIN, int COUT>
__global__ void __launch_bounds__(kWgThreads, 1) wgrad_tc_kernel(const uint4* __restrict__ X,
                                                                 const uint4* __restrict__ Gr,
                                                                 const uint4* __restrict__ zero, int B, int H, int W,
                                                                 float* __restrict__ dW, float* __restrict__ db,
                                                                 int* __restrict__ err) {
  constexpr int XC = CIN / 8, GC = COUT / 8;        // 16-byte chunks per pixel
  constexpr int kN = 2 * COUT;
  // BF16 x BF16 -> F32, both operands MN-major (bits 15 and 16), M = 128, N = kN
  constexpr uint32_t kIdesc = idesc_bf16(kN) | (1u << 15) | (1u << 16);
  extern __shared__ __align__(128) uint8_t wg_smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(wg_smem + kWgStages * kWgStage);
  uint64_t* empty = full + kWgStages;    // the MMAs have read the stage and the workers summed it
  uint64_t* tfull = empty + kWgStages;   // [2] accumulator complete
  uint64_t* tempty = tfull + 2;          // [2] accumulator read out
  uint64_t* mdone = tempty + 2;          // the MMA issuer's last commit
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mdone + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* bias_s = reinterpret_cast<float*>(wg_smem + kWgStages * kWgStage + 256);  // [kWgWorkers][COUT]
  float* sum_s = reinterpret_cast<float*>(wg_smem);  // [3 COUT][3 CIN], once the ring is done with
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int Wp = padded_width(W);
  const uint32_t nseg = (uint32_t)(W + kTileM - 1) / kTileM, npair = (uint32_t)(H + 1) / 2;
  // pixels of this CTA's tiles: where a row's last strip is short, all of a CTA's tiles are the same strip
  const int np = W % kTileM == 0 ? kTileM : min(W - (int)(blockIdx.x % nseg) * kTileM, kTileM);
  if constexpr (XC * 4 < kWgXPlanes) {  // planes no copy fills are read as rows of D that nobody uses
    for (int i = tid; i < kWgStages * kWgStage / 16; i += kWgThreads)
      reinterpret_cast<uint4*>(wg_smem)[i] = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  } else if (np < kTileM) {  // and pixels no copy fills stay zeros in both operands
    for (int i = warp; i < kWgStages * (kWgXPlanes + kWgGPlanes); i += kWgThreads / 32)
      for (int k = np + lane; k < kTileM + 2; k += 32)
        reinterpret_cast<uint4*>(wg_smem + (size_t)i * kWgPlane)[k] = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < kWgStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1 + kWgWorkers);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], kWgWorkers);
    }
    mbar_init(mdone, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kWgWorkers) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kWgTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  after_previous_kernel();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const uint32_t smem0 = smem_u32(wg_smem);

  const uint32_t tiles = (uint32_t)B * npair * nseg;                                 // < 2^31, checked at launch
  const int n = (int)((tiles - blockIdx.x + gridDim.x - 1) / gridDim.x);             // this CTA's (grid <= tiles)

  const int q = warp & 3, g = warp >> 2;  // workers: TMEM lane quarter and gradient row this warp flushes
  const int m = q * 32 + lane;            // row of D
  const int r = m / CIN, ci = m - r * CIN, dy = r - g;
  float acc[3][COUT];
#pragma unroll
  for (int dx = 0; dx < 3; ++dx)
#pragma unroll
    for (int c = 0; c < COUT; ++c) acc[dx][c] = 0.0f;
  if (warp < kWgWorkers) {
    // ---- bias sums and flushes -------------------------------------------------------------------
    float bacc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) bacc[k] = 0.0f;
    bool ok = true;
    // adds accumulator `grp` to the registers; uniform over the warp
    auto flush = [&](int grp) {
      const int b = grp & 1;
      const bool waited = lane != 0 || mbar_wait(&tfull[b], (uint32_t)(grp >> 1) & 1, abort_flag, err, kWaitLimit);
      if (!__all_sync(0xffffffffu, waited)) {
        ok = false;
        return;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int dx = 0; dx < 3; ++dx) {
        float v[COUT];
        tmem_ld<COUT>(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * 3 * kN + dx * kN + g * COUT), v);
#pragma unroll
        for (int c = 0; c < COUT; ++c) acc[dx][c] += v[c];
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[b]);
    };
    // a worker sums one channel group: group tid % GC, pixels tid / GC, + 256 / GC, ... of both gradient rows
    const int gc = tid % GC, gp = tid / GC;
    for (int j = 0; j < n && ok; ++j) {
      const int s = j % kWgStages;
      const bool waited =
          lane != 0 || mbar_wait(&full[s], (uint32_t)(j / kWgStages) & 1, abort_flag, err, kWaitLimit);
      if (!__all_sync(0xffffffffu, waited)) {
        ok = false;
        break;
      }
      const uint8_t* st = wg_smem + s * kWgStage + kWgXPlanes * kWgPlane;
#pragma unroll
      for (int row = 0; row < 2; ++row)
#pragma unroll
        for (int px = 0; px < kTileM; px += 32 * kWgWorkers / GC) {
          const uint4 w = *reinterpret_cast<const uint4*>(st + (row * GC + gc) * kWgPlane + (gp + px) * 16);
          const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            bacc[2 * c] += bf_lo(u[c]);
            bacc[2 * c + 1] += bf_hi(u[c]);
          }
        }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
      if (j >= kWgGroup && j % kWgGroup == 1) flush(j / kWgGroup - 1);
    }
    // groups not flushed in the loop: the last one, and the one before it when the last holds a single tile
    if (ok) {
      const int last = (n - 1) / kWgGroup;
      if (last >= 1 && (n - 1) % kWgGroup == 0) flush(last - 1);
      if (ok) flush(last);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
#pragma unroll
      for (int o = 16; o >= GC; o >>= 1) bacc[k] += __shfl_xor_sync(0xffffffffu, bacc[k], o);
      if (lane < GC) bias_s[warp * COUT + 8 * lane + k] = bacc[k];
    }
  } else if (warp == kWgWorkers) {
    // ---- MMA issuer -----------------------------------------------------------------------------
    if (lane == 0) {
      bool ok = true;
      for (int j = 0; j < n && ok; ++j) {
        const int s = j % kWgStages, grp = j / kWgGroup, b = grp & 1;
        const bool first = j % kWgGroup == 0;
        if (first && grp >= 2)
          ok = mbar_wait(&tempty[b], (uint32_t)((grp >> 1) - 1) & 1, abort_flag, err, kWaitLimit);
        if (ok) ok = mbar_wait(&full[s], (uint32_t)(j / kWgStages) & 1, abort_flag, err, kWaitLimit);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t xa = smem0 + s * kWgStage, ga = xa + kWgXPlanes * kWgPlane;
        // MN-major, no swizzle: 128 bytes between groups of 8 pixels (K), one plane between 8-channel groups;
        // an offset of 16 bytes is one unit of a descriptor's address
        const uint64_t ad = desc_noswz(xa, 128, kWgPlane), bd = desc_noswz(ga, 128, kWgPlane);
        const uint32_t acc = tmem + b * 3 * kN;
#pragma unroll
        for (int ks = 0; ks < kTileM / 16; ++ks)
#pragma unroll
          for (int dx = 0; dx < 3; ++dx)
            umma(acc + dx * kN, ad + (ks * 16 + dx), bd + ks * 16, kIdesc, first && ks == 0 ? 0u : 1u);
        umma_commit(&empty[s]);
        if (j % kWgGroup == kWgGroup - 1 || j == n - 1) umma_commit(&tfull[b]);
      }
      // every tensor-core operation issued above completes before TMEM is freed
      umma_commit(mdone);
      mbar_drain(mdone, 0, err, kWaitLimit);
    }
  } else {
    // ---- copies: halo rows of input rows y - 1 .. y + 2, tile rows of gradient rows y, y + 1, a lane to each --
    const bool xrow = lane < 4 * XC;                                   // lanes 0 .. 4 XC - 1: (input row, group)
    const int ln = xrow ? lane : lane - 4 * XC;                        // then (gradient row, group)
    const int row = xrow ? ln / XC : ln / GC, c = xrow ? ln % XC : ln % GC;
    const uint32_t dst = smem0 + (uint32_t)(xrow ? row * XC + c : kWgXPlanes + row * GC + c) * kWgPlane;
    int issued = 0;
    for (int i = 0; i < n; ++i) {
      const int s = i % kWgStages;
      const bool free = lane != 0 || i < kWgStages ||
                        mbar_wait(&empty[s], (uint32_t)(i / kWgStages - 1) & 1, abort_flag, err, kWaitLimit);
      if (!__all_sync(0xffffffffu, free)) break;
      const uint32_t t = blockIdx.x + (uint32_t)i * gridDim.x, by = t / nseg;
      const int x0 = (int)(t - by * nseg) * kTileM, b = (int)(by / npair), y = 2 * (int)(by - (uint32_t)b * npair);
      if (lane == 0) mbar_expect_tx(&full[s], (uint32_t)(4 * XC * (np + 2) + 2 * GC * np) * 16);
      __syncwarp();
      if (lane < 4 * XC + 2 * GC) {
        const int yy = xrow ? y + row - 1 : y + row;
        const uint4* src = zero;
        if (yy >= 0 && yy < H)
          src = xrow ? X + plane_row(b, H, yy, XC, c, Wp) + x0 : Gr + plane_row(b, H, yy, GC, c, Wp) + x0 + 1;
        bulk_load(dst + (uint32_t)s * kWgStage, src, (uint32_t)(xrow ? np + 2 : np) * 16, &full[s]);
      }
      issued = i + 1;
    }
    // every issued copy lands before the CTA exits (after an abort nobody consumes them)
    for (int i = issued > kWgStages ? issued - kWgStages : 0; i < issued; ++i)
      mbar_drain(&full[i % kWgStages], (uint32_t)(i / kWgStages) & 1, err, kWaitLimit);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();  // every copy has landed and every MMA has read its operands: the ring's memory is free
  if (warp == kWgWorkers) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kWgTmemCols));
  }
  // The CTA's sums (an aborted one has none): the second gradient row's warps hand theirs to the first's.
  const bool done = !*abort_flag, mine = warp < kWgWorkers && dy >= 0 && dy < 3;
  if (done && mine && g == 1) {
#pragma unroll
    for (int dx = 0; dx < 3; ++dx)
#pragma unroll
      for (int c = 0; c < COUT; ++c) sum_s[(dx * COUT + c) * 3 * CIN + dy * CIN + ci] = acc[dx][c];
  }
  __syncthreads();
  if (done && mine && g == 0) {
#pragma unroll
    for (int dx = 0; dx < 3; ++dx)
#pragma unroll
      for (int c = 0; c < COUT; ++c)
        atomicAdd(dW + ((size_t)c * 9 + 3 * dy + dx) * CIN + ci,
                  acc[dx][c] + sum_s[(dx * COUT + c) * 3 * CIN + dy * CIN + ci]);
  }
  if (done && tid >= 32 * kWgWorkers && tid < 32 * kWgWorkers + COUT) {  // the MMA warp: a channel's bias to a lane
    const int c = tid - 32 * kWgWorkers;
    float sum = 0.0f;
#pragma unroll
    for (int w = 0; w < kWgWorkers; ++w) sum += bias_s[w * COUT + c];
    atomicAdd(db + c, sum);
  }
}

// Master FP32 weights W[co][tap][ci] -> BF16 operand images:
//   forward  B[n = (2 - dy)*COUT + co][k = dx*CIN + ci]  at [(k/8)][n][k%8]  (tap = 3 dy + dx)
//   backward the same with channels exchanged and taps reversed: tap' = 8 - tap, n = (2 - dy')*CIN + ci,
//            k = dx'*COUT + co
__global__ void weight_images_kernel(const float* __restrict__ w, uint16_t* __restrict__ fwd,
                                     uint16_t* __restrict__ bwd, int CIN, int COUT) {
  const int n = 9 * CIN * COUT;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int ci = i % CIN, tap = (i / CIN) % 9, co = i / (9 * CIN);
    const uint16_t v = __bfloat16_as_ushort(__float2bfloat16_rn(w[i]));
    const int kf = tap % 3 * CIN + ci, nf = (2 - tap / 3) * COUT + co;
    fwd[((size_t)(kf / 8) * 3 * COUT + nf) * 8 + kf % 8] = v;
    if (bwd) {
      const int kb = (2 - tap % 3) * COUT + co, nb = tap / 3 * CIN + ci;  // dy' = 2 - dy, dx' = 2 - dx
      bwd[((size_t)(kb / 8) * 3 * CIN + nb) * 8 + kb % 8] = v;
    }
  }
}

// Adam (Kingma & Ba 2015) on the FP32 master parameters.
__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1,
                            float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// Input of the network from a volume [YN][XN][ZN] (z fastest): sample s is
// slice z = z0 + s, channels = slices z-2..z+2 (clamped to the volume), as
// u = mu / mu_w - 1 in BF16, padded to 16 channels.
__global__ void pack_input_kernel(uint16_t* __restrict__ out, const float* __restrict__ vol, int XN, int YN,
                                  int ZN, int z0, int nz, float inv_mu) {
  const long long total = (long long)nz * YN * XN;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long px = i % ((long long)YN * XN);
    const int s = (int)(i / ((long long)YN * XN));
    const int z = z0 + s;
    const float* col = vol + px * ZN;
    uint32_t w[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      float lo = 0.f, hi = 0.f;
      if (2 * c < 5) lo = col[min(max(z + 2 * c - 2, 0), ZN - 1)] * inv_mu - 1.0f;
      if (2 * c + 1 < 5) hi = col[min(max(z + 2 * c - 1, 0), ZN - 1)] * inv_mu - 1.0f;
      w[c] = pack2(lo, hi);
    }
    uint4* o = reinterpret_cast<uint4*>(out + i * 16);
    o[0] = make_uint4(w[0], w[1], w[2], w[3]);
    o[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// The same input as planes (two groups: 8 channels of which 5 are used, 8 of zeros) for the
// network itself. A CTA takes 32 padded pixels of one image row and 32 slices: it reads each
// pixel's 36 consecutive slices together (the volume's fastest axis) and writes rows of pixels. Images of more
// rows than a grid has are walked.
constexpr int kPackPx = 32, kPackZ = 32;
__global__ void __launch_bounds__(256) pack_planes_kernel(uint4* __restrict__ out, const float* __restrict__ vol, int XN,
                                                          int YN, int ZN, int z0, int nz, float inv_mu, int Wp) {
  __shared__ float t[kPackPx][kPackZ + 5];
  const int px0 = blockIdx.x * kPackPx, s0 = blockIdx.z * kPackZ;
  const int p = threadIdx.x & (kPackPx - 1), px = px0 + p, x = px - 1;
  for (int y = blockIdx.y; y < YN; y += gridDim.y) {
    for (int i = threadIdx.x; i < kPackPx * (kPackZ + 4); i += 256) {
      const int q = i / (kPackZ + 4), k = i - q * (kPackZ + 4);
      const int xq = px0 + q - 1, z = min(max(z0 + s0 + k - 2, 0), ZN - 1);
      if (xq >= 0 && xq < XN && s0 + k < nz + 4) t[q][k] = vol[((size_t)y * XN + xq) * ZN + z];
    }
    __syncthreads();
    for (int k = threadIdx.x / kPackPx; px < Wp && k < kPackZ && s0 + k < nz; k += 256 / kPackPx) {
      uint4 w = make_uint4(0u, 0u, 0u, 0u);
      if (x >= 0 && x < XN) {
        float u[5];
#pragma unroll
        for (int c = 0; c < 5; ++c) u[c] = t[p][k + c] * inv_mu - 1.0f;
        w = make_uint4(pack2(u[0], u[1]), pack2(u[2], u[3]), pack2(u[4], 0.0f), 0u);
      }
      const size_t o = plane_row(s0 + k, YN, y, 2, 0, Wp) + px;
      out[o] = w;
      out[o + Wp] = make_uint4(0u, 0u, 0u, 0u);
    }
    __syncthreads();  // before the next row's values
  }
}

// The residual epilogue of a whole volume: out = vol + scale r for slices [z0, z0 + nz), r by slices
// ([nz][YN][XN]), the volume with z fastest. A CTA turns 32 pixels x 32 slices through shared memory, so that
// both sides are read and written in runs. (From the convolution's epilogue, slice by slice, every 4-byte
// access of the volume was a sector of its own: that layer took 272 us per 32 slices of 512 x 512, now 119
// with this kernel's 37.)
__global__ void __launch_bounds__(256) add_residual_kernel(float* __restrict__ out, const float* __restrict__ vol,
                                                           const float* __restrict__ r, long long px, int ZN, int z0,
                                                           int nz, float scale) {
  __shared__ float t[32][33];
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const long long p0 = (long long)blockIdx.x * 32;
  const int s0 = blockIdx.y * 32;
  for (int k = row; k < 32; k += 8)
    if (s0 + k < nz && p0 + lane < px) t[k][lane] = r[(size_t)(s0 + k) * px + p0 + lane];
  __syncthreads();
  for (int p = row; p < 32; p += 8)
    if (s0 + lane < nz && p0 + p < px) {
      const size_t o = (size_t)(p0 + p) * ZN + z0 + s0 + lane;
      out[o] = vol[o] + scale * t[lane][p];
    }
}

// A caller's NHWC input [rows][W][16] as planes; ALIGN: the boundary it starts on, 16, 2 or 1 bytes.
template <int ALIGN>
__global__ void nhwc_to_planes_kernel(uint4* __restrict__ out, const uint16_t* __restrict__ in, long long rows, int W,
                                      int Wp) {
  const long long total = rows * Wp;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / Wp;
    const int px = (int)(i - r * Wp), x = px - 1;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint4 w = make_uint4(0u, 0u, 0u, 0u);
      if (x >= 0 && x < W) {
        const uint16_t* src = in + (r * W + x) * 16 + c * 8;
        auto at = [&](int k) -> uint32_t {
          if constexpr (ALIGN == 1) {
            const uint8_t* b = reinterpret_cast<const uint8_t*>(src) + 2 * k;
            return b[0] | (uint32_t)b[1] << 8;
          } else {
            return src[k];
          }
        };
        if constexpr (ALIGN == 16)
          w = __ldg(reinterpret_cast<const uint4*>(src));
        else
          w = make_uint4(at(0) | at(1) << 16, at(2) | at(3) << 16, at(4) | at(5) << 16, at(6) | at(7) << 16);
      }
      out[(r * 2 + c) * Wp + px] = w;
    }
  }
}

// Launches a kernel that calls after_previous_kernel.
template <class... P, class... A>
int launch_dependent(void (*kern)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  HR_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...));
  return HR_OK;
}

// Dynamic shared memory of a conv CTA: input-row ring + weights + barriers + alignment slack.
template <int CIN, int COUT>
constexpr size_t conv_smem() {
  return (size_t)kRing * (CIN / 8) * kPlane + 9 * CIN * COUT * 2 + 512 + COUT * 4 + 128;  // barriers fit in 512
}

template <int CIN, int COUT, int EPI>
int launch_conv(ConvArgs& a, cudaStream_t s) {
  const size_t smem = conv_smem<CIN, COUT>();
  HR_CUDA_TRY(cudaFuncSetAttribute(conv_tc_kernel<CIN, COUT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)smem));
  // the largest shared-memory carveout, so that several CTAs (input-row rings) fit on an SM
  HR_CUDA_TRY(cudaFuncSetAttribute(conv_tc_kernel<CIN, COUT, EPI>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   (int)cudaSharedmemCarveoutMaxShared));
  // resident CTAs per SM from the kernel's resources: shared memory (1 KiB reserved per CTA), TMEM
  // columns, registers and threads. CTAs never wait on one another, so a grid larger than what is
  // resident is only queued.
  cudaFuncAttributes fa;
  HR_CUDA_TRY(cudaFuncGetAttributes(&fa, conv_tc_kernel<CIN, COUT, EPI>));
  int dev = 0, smem_sm = 0;
  HR_CUDA_TRY(cudaGetDevice(&dev));
  HR_CUDA_TRY(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
  const int by_smem = smem_sm / (int)(smem + fa.sharedSizeBytes + 1024);
  const int by_tmem = 512 / tmem_cols(COUT);
  const int by_regs = 65536 / std::max(1, fa.numRegs * kThreads);
  const int per_sm = std::max(1, std::min({by_smem, by_tmem, by_regs, 2048 / kThreads}));
  const long long ctas = (long long)per_sm * hr::sm_count();
  // one share of the rows per group of CTAs that fit together, of at least 4 rows (each reloads 2 rows)
  const long long nseg = (a.W + kTileM - 1) / kTileM;
  const long long groups = std::min(((long long)a.B * a.H + 3) / 4, std::max(1LL, ctas / nseg));
  const long long grid = groups * nseg;
  if (grid <= 0) return HR_OK;
  return launch_dependent(conv_tc_kernel<CIN, COUT, EPI>, (unsigned)grid, kThreads, smem, s, a);
}

template <int CIN, int COUT>
int launch_wgrad(const uint4* X, const uint4* Gr, const uint4* zero, int B, int H, int W, float* dW, float* db,
                 int* err, cudaStream_t s) {
  const long long tiles = (long long)B * ((H + 1) / 2) * ((W + kTileM - 1) / kTileM);
  long long grid = std::min<long long>(tiles, hr::sm_count());
  if (grid <= 0) return HR_OK;
  const long long nseg = (W + kTileM - 1) / kTileM;
  if (W % kTileM) grid = std::max(grid / nseg, 1LL) * nseg;  // every CTA keeps one strip (tiles is such a multiple too)
  HR_REQUIRE(tiles < (1LL << 31), "conv weight gradients: %lld tiles exceed one launch", tiles);
  HR_CUDA_TRY(cudaFuncSetAttribute(wgrad_tc_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kWgSmem));
  return launch_dependent(wgrad_tc_kernel<CIN, COUT>, (unsigned)grid, kWgThreads, kWgSmem, s, X, Gr, zero, B, H, W,
                          dW, db, err);
}

}  // namespace

struct hr_cnn {
  // parameters: per layer W[co][tap][ci] then b[co], concatenated (FP32 master)
  size_t woff[kLayers], boff[kLayers], nparam = 0;
  float *d_p = nullptr, *d_g = nullptr, *d_m = nullptr, *d_v = nullptr;
  uint16_t *d_wf[kLayers] = {}, *d_wb[kLayers] = {};  // BF16 operand images (forward, backward)
  // activation planes for up to cap_pix padded pixels (B * H * padded_width(W)); those only training needs, [3]
  // to [7], d_gout and d_g1, for up to cap_train
  long long cap_pix = 0, cap_train = 0;
  uint4* d_act[kLayers] = {};  // [0]: input (16 ch), [k]: output of layer k (32 ch), k = 1..7; inference uses [1], [2]
  uint4* d_gout = nullptr;     // gradient at the last layer's output (16 ch)
  uint4* d_g1 = nullptr;       // gradients (32 ch), in turn with d_act[7]
  uint4* d_zero = nullptr;     // kHalo zero chunks: the rows above and below an image
  float* d_loss = nullptr;
  int* d_err = nullptr;
  long long step = 0;
  size_t bytes = 0;
  int stall_row = -1;               // test hook (hr_cnn_test_stall)
  uint32_t wait_limit = kWaitLimit;
};

namespace {

constexpr int kInferActs = 3;  // activations that inference uses too

void cnn_free_acts(hr_cnn* n, int l0, int l1) {
  for (int l = l0; l < l1; ++l) {
    cudaFree(n->d_act[l]);
    n->d_act[l] = nullptr;
  }
}

void cnn_free_infer(hr_cnn* n) {
  cnn_free_acts(n, 0, kInferActs);
  n->cap_pix = 0;
}

void cnn_free_train(hr_cnn* n) {
  cnn_free_acts(n, kInferActs, kLayers);
  cudaFree(n->d_gout);
  cudaFree(n->d_g1);
  n->d_gout = n->d_g1 = nullptr;
  n->cap_train = 0;
}

void cnn_destroy(hr_cnn* n) {
  if (!n) return;
  cnn_free_infer(n);
  cnn_free_train(n);
  cudaFree(n->d_p);
  cudaFree(n->d_g);
  cudaFree(n->d_m);
  cudaFree(n->d_v);
  for (int l = 0; l < kLayers; ++l) {
    cudaFree(n->d_wf[l]);
    cudaFree(n->d_wb[l]);
  }
  cudaFree(n->d_loss);
  cudaFree(n->d_err);
  cudaFree(n->d_zero);
  delete n;
}

// Buffers for `pix` padded pixels.
int ensure_infer(hr_cnn* n, long long pix) {
  if (pix <= n->cap_pix) return HR_OK;
  cnn_free_infer(n);
  for (int l = 0; l < kInferActs; ++l) HR_CUDA_TRY(cudaMalloc(&n->d_act[l], (size_t)pix * (l == 0 ? 16 : 32) * 2));
  n->cap_pix = pix;
  return HR_OK;
}

int ensure_train(hr_cnn* n, long long pix) {
  HR_TRY(ensure_infer(n, pix));
  if (pix <= n->cap_train) return HR_OK;
  cnn_free_train(n);
  for (int l = kInferActs; l < kLayers; ++l) HR_CUDA_TRY(cudaMalloc(&n->d_act[l], (size_t)pix * 32 * 2));
  HR_CUDA_TRY(cudaMalloc(&n->d_gout, (size_t)pix * 16 * 2));
  HR_CUDA_TRY(cudaMalloc(&n->d_g1, (size_t)pix * 32 * 2));
  n->cap_train = pix;
  return HR_OK;
}

int refresh_images(hr_cnn* n, cudaStream_t s) {
  for (int l = 0; l < kLayers; ++l) {
    weight_images_kernel<<<64, 256, 0, s>>>(n->d_p + n->woff[l], n->d_wf[l], n->d_wb[l], kCin[l], kCout[l]);
    HR_CUDA_TRY(cudaGetLastError());
  }
  return HR_OK;
}

// A caller's NHWC input into the planes d_act[0] (whose buffer is there).
int load_input(hr_cnn* n, const uint16_t* d_x, int B, int H, int W, cudaStream_t s) {
  const long long rows = (long long)B * H;
  const int Wp = padded_width(W);
  const long long blocks = std::min<long long>((rows * Wp + 255) / 256, 16LL * hr::sm_count());
  if (((uintptr_t)d_x & 15) == 0)
    nhwc_to_planes_kernel<16><<<(unsigned)blocks, 256, 0, s>>>(n->d_act[0], d_x, rows, W, Wp);
  else if (((uintptr_t)d_x & 1) == 0)
    nhwc_to_planes_kernel<2><<<(unsigned)blocks, 256, 0, s>>>(n->d_act[0], d_x, rows, W, Wp);
  else
    nhwc_to_planes_kernel<1><<<(unsigned)blocks, 256, 0, s>>>(n->d_act[0], d_x, rows, W, Wp);
  HR_CUDA_TRY(cudaGetLastError());
  return HR_OK;
}

ConvArgs base_args(const hr_cnn* n, int B, int H, int W) {
  ConvArgs a{};
  a.B = B;
  a.H = H;
  a.W = W;
  a.Wp = padded_width(W);
  a.zero = n->d_zero;
  a.err = n->d_err;
  a.stall_row = n->stall_row;
  a.wait_limit = n->wait_limit;
  return a;
}

// Where layer l's output (l = 1..7) is held: by inference in d_act[1] and d_act[2] in turn.
int act_index(int l, bool train) { return train || l == 0 ? l : 1 + (l - 1) % 2; }

// Layers 1..7 (ReLU) from d_act[0], into d_act[1..7] for training.
int forward_trunk(hr_cnn* n, int B, int H, int W, bool train, cudaStream_t s) {
  for (int l = 0; l < kLayers - 1; ++l) {
    ConvArgs a = base_args(n, B, H, W);
    a.in = n->d_act[act_index(l, train)];
    a.wimg = n->d_wf[l];
    a.bias = n->d_p + n->boff[l];
    a.out = n->d_act[act_index(l + 1, train)];
    if (l == 0)
      HR_TRY((launch_conv<16, 32, EPI_RELU>(a, s)));
    else
      HR_TRY((launch_conv<32, 32, EPI_RELU>(a, s)));
  }
  return HR_OK;
}

}  // namespace

extern "C" size_t hr_cnn_param_count(void) {
  size_t n = 0;
  for (int l = 0; l < kLayers; ++l) n += (size_t)9 * kCin[l] * kCout[l] + kCout[l];
  return n;
}

extern "C" int hr_cnn_create(hr_cnn** net, const float* h_params) {
  hr::clear_error();
  HR_REQUIRE(net != nullptr && h_params != nullptr, "hr_cnn_create: NULL argument");
  *net = nullptr;
  HR_TRY(hr::require_device());
  int dev = 0, major = 0;
  HR_CUDA_TRY(cudaGetDevice(&dev));
  HR_CUDA_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
  HR_REQUIRE(major == 10, "learned correction: needs an sm_100 device (found compute capability %d.x)", major);
  hr_cnn* n = new hr_cnn;
  size_t off = 0;
  for (int l = 0; l < kLayers; ++l) {
    n->woff[l] = off;
    off += (size_t)9 * kCin[l] * kCout[l];
    n->boff[l] = off;
    off += kCout[l];
  }
  n->nparam = off;
  cudaError_t e = cudaSuccess;
  for (float** p : {&n->d_p, &n->d_g, &n->d_m, &n->d_v})
    if (e == cudaSuccess) e = cudaMalloc(p, off * sizeof(float));
  for (int l = 0; l < kLayers && e == cudaSuccess; ++l) {
    e = cudaMalloc(&n->d_wf[l], (size_t)9 * kCin[l] * kCout[l] * 2);
    if (e == cudaSuccess) e = cudaMalloc(&n->d_wb[l], (size_t)9 * kCin[l] * kCout[l] * 2);
  }
  if (e == cudaSuccess) e = cudaMalloc(&n->d_loss, sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&n->d_err, sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&n->d_zero, kBox);
  if (e == cudaSuccess) e = cudaMemset(n->d_zero, 0, kBox);
  if (e == cudaSuccess) e = cudaMemcpy(n->d_p, h_params, off * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(n->d_m, 0, off * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(n->d_v, 0, off * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(n->d_err, 0, sizeof(int));
  int st = e == cudaSuccess ? HR_OK
                            : hr::fail(e == cudaErrorMemoryAllocation ? HR_ERR_OUT_OF_MEMORY : HR_ERR_CUDA,
                                       "hr_cnn_create: %s", cudaGetErrorString(e));
  if (st == HR_OK) st = refresh_images(n, nullptr);
  if (st == HR_OK && cudaStreamSynchronize(nullptr) != cudaSuccess)
    st = hr::fail(HR_ERR_CUDA, "hr_cnn_create: weight preparation failed");
  if (st != HR_OK) {
    cnn_destroy(n);
    return st;
  }
  *net = n;
  return HR_OK;
}

extern "C" int hr_cnn_get_params(const hr_cnn* n, float* h_params) {
  HR_REQUIRE(n != nullptr && h_params != nullptr, "hr_cnn_get_params: NULL argument");
  HR_CUDA_TRY(cudaMemcpy(h_params, n->d_p, n->nparam * sizeof(float), cudaMemcpyDeviceToHost));
  return HR_OK;
}

extern "C" int hr_cnn_get_grads(const hr_cnn* n, float* h_grads) {
  HR_REQUIRE(n != nullptr && h_grads != nullptr, "hr_cnn_get_grads: NULL argument");
  HR_CUDA_TRY(cudaMemcpy(h_grads, n->d_g, n->nparam * sizeof(float), cudaMemcpyDeviceToHost));
  return HR_OK;
}

// Forward + loss + backward (parameter gradients into the plan's gradient
// buffer); lr > 0 then applies one Adam step. d_x: network input NHWC16 BF16
// [B][H][W][16]; d_base/d_target: FP32 [B][H][W] centre slice and reference.
extern "C" int hr_cnn_train_step(hr_cnn* n, const uint16_t* d_x, const float* d_base, const float* d_target, int B,
                                 int H, int W, float mu_w, float lr, float* loss_out, void* stream) {
  HR_REQUIRE(n != nullptr && d_x != nullptr && d_base != nullptr && d_target != nullptr,
             "hr_cnn_train_step: NULL argument");
  HR_REQUIRE(B > 0 && H > 0 && W > 0 && mu_w > 0.0f, "hr_cnn_train_step: invalid sizes");
  HR_REQUIRE(((uintptr_t)d_x & 15) == 0, "hr_cnn_train_step: input must be 16-byte aligned");
  cudaStream_t s = hr::as_stream(stream);
  const long long pix = (long long)B * H * W;
  HR_TRY(ensure_train(n, (long long)B * H * padded_width(W)));
  HR_TRY(load_input(n, d_x, B, H, W, s));
  HR_CUDA_TRY(cudaMemsetAsync(n->d_loss, 0, sizeof(float), s));
  HR_CUDA_TRY(cudaMemsetAsync(n->d_g, 0, n->nparam * sizeof(float), s));
  HR_TRY(forward_trunk(n, B, H, W, true, s));
  // L8 with the fused residual, loss and output gradient (16 channels, channel 0 used)
  ConvArgs a = base_args(n, B, H, W);
  a.in = n->d_act[7];
  a.wimg = n->d_wf[7];
  a.bias = n->d_p + n->boff[7];
  a.out = n->d_gout;
  a.base = d_base;
  a.target = d_target;
  a.sb = (long long)H * W;
  a.sp = 1;
  a.scale = mu_w;
  a.grad_scale = 2.0f / (float)pix;
  a.loss = n->d_loss;
  HR_TRY((launch_conv<32, 16, EPI_LOSS>(a, s)));
  // backward: G_k (gradient at layer k's output) -> dW_k, and G_{k-1} masked by act_{k-1} > 0
  uint4* g = n->d_gout;
  uint4* gn = n->d_g1;
  for (int l = kLayers - 1; l >= 0; --l) {
    const int ci = kCin[l], co = kCout[l];
    float* dW = n->d_g + n->woff[l];
    float* db = n->d_g + n->boff[l];
    if (ci == 16)
      HR_TRY((launch_wgrad<16, 32>(n->d_act[l], g, n->d_zero, B, H, W, dW, db, n->d_err, s)));
    else if (co == 16)
      HR_TRY((launch_wgrad<32, 16>(n->d_act[l], g, n->d_zero, B, H, W, dW, db, n->d_err, s)));
    else
      HR_TRY((launch_wgrad<32, 32>(n->d_act[l], g, n->d_zero, B, H, W, dW, db, n->d_err, s)));
    if (l == 0) break;
    ConvArgs b = base_args(n, B, H, W);
    b.in = g;
    b.wimg = n->d_wb[l];
    b.out = gn;
    b.mask = n->d_act[l];
    if (co == 16)
      HR_TRY((launch_conv<16, 32, EPI_MASK>(b, s)));
    else
      HR_TRY((launch_conv<32, 32, EPI_MASK>(b, s)));
    g = gn;
    gn = g == n->d_g1 ? n->d_act[kLayers - 1] : n->d_g1;  // act_7 has served as mask and for dW_8
  }
  if (lr > 0.0f) {
    ++n->step;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - std::pow(b1, (float)n->step), c2 = 1.0f - std::pow(b2, (float)n->step);
    adam_kernel<<<128, 256, 0, s>>>(n->d_p, n->d_g, n->d_m, n->d_v, (int)n->nparam, lr, b1, b2, 1e-8f, c1, c2);
    HR_CUDA_TRY(cudaGetLastError());
    HR_TRY(refresh_images(n, s));
  }
  if (loss_out) {
    float l = 0.f;
    HR_CUDA_TRY(cudaMemcpyAsync(&l, n->d_loss, sizeof(float), cudaMemcpyDeviceToHost, s));
    HR_CUDA_TRY(cudaStreamSynchronize(s));
    *loss_out = l / (float)pix;
  }
  return HR_OK;
}

// Layers 1..8 from the input planes in d_act[0], with the residual epilogue.
static int forward_residual(hr_cnn* n, float* d_out, const float* d_base, long long sb, long long sp, int B, int H,
                            int W, float mu_w, cudaStream_t s) {
  HR_TRY(forward_trunk(n, B, H, W, false, s));
  ConvArgs a = base_args(n, B, H, W);
  a.in = n->d_act[act_index(7, false)];
  a.wimg = n->d_wf[7];
  a.bias = n->d_p + n->boff[7];
  a.base = d_base;
  a.pred = d_out;
  a.sb = sb;
  a.sp = sp;
  a.scale = mu_w;
  return launch_conv<32, 16, EPI_RESID>(a, s);
}

// Inference: out[b][y][x] = base + mu_w * net(x) for a batch of network inputs
// (the same layouts as hr_cnn_train_step; base and out may use any strides).
extern "C" int hr_cnn_forward(hr_cnn* n, float* d_out, const uint16_t* d_x, const float* d_base, long long sb,
                              long long sp, int B, int H, int W, float mu_w, void* stream) {
  HR_REQUIRE(n != nullptr && d_out != nullptr && d_x != nullptr && d_base != nullptr, "hr_cnn_forward: NULL argument");
  HR_REQUIRE(B > 0 && H > 0 && W > 0 && mu_w > 0.0f, "hr_cnn_forward: invalid sizes");
  cudaStream_t s = hr::as_stream(stream);
  HR_TRY(ensure_infer(n, (long long)B * H * padded_width(W)));
  HR_TRY(load_input(n, d_x, B, H, W, s));
  return forward_residual(n, d_out, d_base, sb, sp, B, H, W, mu_w, s);
}

// Corrects a whole reconstructed volume [YN][XN][ZN] (z fastest): every slice
// with its two neighbours on each side (clamped at the ends), chunk slices at
// a time. d_out must not alias d_vol.
extern "C" int hr_cnn_apply_volume(hr_cnn* n, float* d_out, const float* d_vol, int XN, int YN, int ZN, float mu_w,
                                   int chunk, void* stream) {
  HR_REQUIRE(n != nullptr && d_out != nullptr && d_vol != nullptr, "hr_cnn_apply_volume: NULL argument");
  HR_REQUIRE((const void*)d_out != (const void*)d_vol, "hr_cnn_apply_volume: in-place correction is not supported");
  HR_REQUIRE(XN > 0 && YN > 0 && ZN > 0 && chunk > 0 && mu_w > 0.0f, "hr_cnn_apply_volume: invalid sizes");
  cudaStream_t s = hr::as_stream(stream);
  const int Wp = padded_width(XN);
  constexpr int kGridMax = 65535;  // of a grid's y and z
  chunk = std::min(chunk, kGridMax * kPackZ);
  HR_TRY(ensure_infer(n, (long long)std::min(chunk, ZN) * YN * Wp));
  for (int z0 = 0; z0 < ZN; z0 += chunk) {
    const int nz = std::min(chunk, ZN - z0);
    const dim3 grid((Wp + kPackPx - 1) / kPackPx, std::min(YN, kGridMax), (nz + kPackZ - 1) / kPackZ);
    pack_planes_kernel<<<grid, 256, 0, s>>>(n->d_act[0], d_vol, XN, YN, ZN, z0, nz, 1.0f / mu_w, Wp);
    HR_CUDA_TRY(cudaGetLastError());
    HR_TRY(forward_trunk(n, nz, YN, XN, false, s));
    ConvArgs a = base_args(n, nz, YN, XN);
    a.in = n->d_act[act_index(7, false)];
    a.wimg = n->d_wf[7];
    a.bias = n->d_p + n->boff[7];
    a.pred = reinterpret_cast<float*>(n->d_act[act_index(6, false)]);  // the activation layer 8 does not read
    HR_TRY((launch_conv<32, 16, EPI_RAW>(a, s)));
    const long long px = (long long)XN * YN;
    const dim3 rgrid((unsigned)((px + 31) / 32), (nz + 31) / 32);
    add_residual_kernel<<<rgrid, 256, 0, s>>>(d_out, d_vol, a.pred, px, ZN, z0, nz, mu_w);
    HR_CUDA_TRY(cudaGetLastError());
  }
  return HR_OK;
}

// The network input for slices [z0, z0 + nz) of a volume (for training data).
extern "C" int hr_cnn_pack_input(uint16_t* d_x, const float* d_vol, int XN, int YN, int ZN, int z0, int nz, float mu_w,
                                 void* stream) {
  HR_REQUIRE(d_x != nullptr && d_vol != nullptr, "hr_cnn_pack_input: NULL argument");
  HR_REQUIRE(XN > 0 && YN > 0 && ZN > 0 && nz > 0 && z0 >= 0 && z0 + nz <= ZN && mu_w > 0.0f,
             "hr_cnn_pack_input: invalid sizes");
  pack_input_kernel<<<8 * hr::sm_count(), 256, 0, hr::as_stream(stream)>>>(d_x, d_vol, XN, YN, ZN, z0, nz,
                                                                          1.0f / mu_w);
  HR_CUDA_TRY(cudaGetLastError());
  return HR_OK;
}

extern "C" int hr_cnn_check(const hr_cnn* n) {
  HR_REQUIRE(n != nullptr, "hr_cnn_check: NULL network");
  int err = 0;
  HR_CUDA_TRY(cudaMemcpy(&err, n->d_err, sizeof(int), cudaMemcpyDeviceToHost));
  if (err) {
    HR_CUDA_TRY(cudaMemset(n->d_err, 0, sizeof(int)));
    return hr::fail(HR_ERR_CUDA, "learned correction: a tensor-core wait timed out (kernel aborted)");
  }
  return HR_OK;
}

extern "C" int hr_cnn_test_stall(hr_cnn* n, int row, unsigned int wait_polls) {
  HR_REQUIRE(n != nullptr, "hr_cnn_test_stall: NULL network");
  HR_REQUIRE(row < 0 || wait_polls > 0, "hr_cnn_test_stall: wait_polls must be positive");
  n->stall_row = row < 0 ? -1 : row;
  n->wait_limit = row < 0 ? kWaitLimit : (uint32_t)wait_polls;
  return HR_OK;
}

extern "C" void hr_cnn_destroy(hr_cnn* n) { cnn_destroy(n); }
