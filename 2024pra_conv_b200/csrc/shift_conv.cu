// Kernels and launch rules of the shift-reuse implicit GEMM (shift_conv.cuh).
#include <cuda_runtime.h>
#include "shift_conv.cuh"

namespace wino {

static __device__ uint32_t g_shift_err;

__global__ void __launch_bounds__(256) shift_weight_kernel(KernelParam p) {
  shift_weight_body<1>(p, static_cast<uint8_t*>(p.transform_filter));
}
__global__ void __launch_bounds__(256) shift_weight_pair_kernel(KernelParam p) {
  shift_weight_body<2>(p, static_cast<uint8_t*>(p.transform_filter));
}

// One CTA a unit (128 positions, up to 128 output channels).
__global__ void __launch_bounds__(sc::NTHREAD, 1) shift_conv_kernel(KernelParam p) {
  shift_conv_body<1>(p, static_cast<const uint8_t*>(p.transform_filter), &g_shift_err);
}

// A pair of CTAs a unit (256 positions, up to 256 output channels).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(sc::NTHREAD, 1) shift_conv_pair_kernel(KernelParam p) {
  shift_conv_body<2>(p, static_cast<const uint8_t*>(p.transform_filter), &g_shift_err);
}

}  // namespace wino

using namespace wino;

extern "C" {

void* wino_shift_kernel_ptr(int cg) { return cg == 2 ? (void*)shift_conv_pair_kernel : (void*)shift_conv_kernel; }
void* wino_shift_weight_kernel_ptr(int cg) {
  return cg == 2 ? (void*)shift_weight_pair_kernel : (void*)shift_weight_kernel;
}
size_t wino_shift_weight_bytes(const KernelParam* p, int cg) { return sc::weight_bytes(sc::make_plan(*p, cg), cg); }
unsigned wino_shift_weight_grid(const KernelParam* p, int cg) {
  return (unsigned)((wino_shift_weight_bytes(p, cg) / 16 + 255) / 256);
}
int wino_shift_threads() { return sc::NTHREAD; }
int wino_shift_smem_bytes() { return sc::SMEM_BYTES; }

// CTAs a unit for a problem (1 or 2), or 0 when the kernel does not take it:
// strides past 2, more than MAXTAP taps, a position tile whose pixels exceed
// the producers' items, fewer than two stages, or indices past 32 bits.
int wino_shift_cg(const KernelParam* p) {
  if (p->u > 2 || p->v > 2 || p->r * p->s > sc::MAXTAP) return 0;
  const sc::Plan g1 = sc::make_plan(*p, 1), g2 = sc::make_plan(*p, 2);
  if (g1.npos + 4096 >= (1LL << 31) || g1.GX >= (1 << 15) || g1.GY >= (1 << 15)) return 0;
  // element offsets of one unit: the images its rows touch, all channels
  const long long per = (long long)g1.GX * g1.GY;
  if (((long long)g1.rows / per + 3) * g1.C * g1.H * g1.W >= (1LL << 31)) return 0;
  const bool aligned = (p->h * p->w) % 4 == 0 && (reinterpret_cast<uintptr_t>(p->pin) & 7) == 0;
  const bool strided = p->u > 1 || p->v > 1;
  const int items = (!aligned ? sc::MAXITEM_ODD : strided ? sc::MAXITEM_STRIDED : sc::MAXITEM) * sc::NPROD;
  for (const sc::Plan* g : {&g1, &g2})
    if (2 * g->cps * g->qmax > items || g->nstage < 2 || g->rows > sc::MAXROWS) return 0;
  const long long w1 = (g1.units + sc::NSM - 1) / sc::NSM, w2 = (g2.units + sc::NSM / 2 - 1) / (sc::NSM / 2);
  const int n2 = g2.Kp < 256 ? (g2.Kp + 31) / 32 * 32 : 256;
  // a pair needs work for every pair of SMs
  if (g2.units < sc::NSM / 2) return 1;
  const long long t1 = w1 * sc::mma_cycles(1, g1.Kp < g1.NB ? g1.Kp : g1.NB), t2 = w2 * sc::mma_cycles(2, n2);
  return t2 <= t1 ? 2 : 1;
}

// The packed plan the kernels read from the argument's transform_pin.
unsigned long long wino_shift_pack(const KernelParam* p, int cg) { return sc::pack_plan(sc::make_plan(*p, cg)); }

unsigned wino_shift_grid(const KernelParam* p, int cg, int sms) {
  const sc::Plan g = sc::make_plan(*p, cg);
  const long long cap = sms / cg;
  return (unsigned)(cg * (g.units < cap ? g.units : cap));
}

int wino_shift_prepare() {
  // attributes are per function and device: set them once per device (a
  // repeated set from another thread is harmless)
  static int done[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  if (dev >= 0 && dev < 64 && done[dev]) return 0;
  for (const void* f : {(const void*)shift_conv_kernel, (const void*)shift_conv_pair_kernel}) {
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, sc::SMEM_BYTES) != cudaSuccess) return 1;
    // the warpgroups split exactly the registers the block launches with
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, f) != cudaSuccess || fa.numRegs != sc::REGS_LAUNCH) return 1;
  }
  if (dev >= 0 && dev < 64) done[dev] = 1;
  return 0;
}

// The plan's numbers (host tests): GX, GY, operand rows, blocks per stage,
// stages per unit, ring stages, stage bytes of input and weights, output
// channels per unit, units, planes, quads a tile may touch, quads an image.
void wino_shift_plan(const KernelParam* p, int cg, int* out) {
  const sc::Plan g = sc::make_plan(*p, cg);
  const int v[14] = {g.GX, g.GY, g.rows, g.cps, g.nst, g.nstage, g.stageA, g.stageB, g.NB, g.units, g.nu, g.nv,
                     g.qmax, g.qpi};
  for (int i = 0; i < 14; ++i) out[i] = v[i];
}

// Launches the kernel on a problem whose weight operand is at
// p->transform_filter and packed plan in p->transform_pin.
int wino_launch_shift(const KernelParam* p, int cg, int sms, cudaStream_t stream) {
  void* args[] = {const_cast<KernelParam*>(p)};
  return (int)cudaLaunchKernel(wino_shift_kernel_ptr(cg), dim3(wino_shift_grid(p, cg, sms)), dim3(sc::NTHREAD), args,
                               (size_t)sc::SMEM_BYTES, stream);
}

// Probe entry (tests): weights re-laid out into wprep when `weight` is given,
// then the conv.
int wino_conv2d_shift(const void* x, const void* weight, void* wprep, void* y, int n, int c, int h, int w, int k,
                      int r, int s, int u, int v, int pp, int q, int cg, void* stream) {
  KernelParam p{};
  p.pin = const_cast<void*>(x);
  p.pweight = const_cast<void*>(weight);
  p.pout = y;
  p.transform_filter = wprep;
  p.n = (short)n; p.c = (short)c; p.h = (short)h; p.w = (short)w; p.k = (short)k;
  p.r = (short)r; p.s = (short)s; p.u = (short)u; p.v = (short)v; p.p = (short)pp; p.q = (short)q;
  p.Oh = (short)((h - r + 2 * pp) / u + 1);
  p.Ow = (short)((w - s + 2 * q) / v + 1);
  if (wino_shift_cg(&p) == 0) return 2;
  if (cg == 0) cg = wino_shift_cg(&p);
  if (wino_shift_prepare() != 0) return 3;
  p.transform_pin = reinterpret_cast<void*>(wino_shift_pack(&p, cg));
  void* args[] = {&p};
  if (weight && cudaLaunchKernel(wino_shift_weight_kernel_ptr(cg), dim3(wino_shift_weight_grid(&p, cg)), dim3(256),
                                 args, 0, (cudaStream_t)stream) != cudaSuccess)
    return 3;
  if (!x) return 0;
  return wino_launch_shift(&p, cg, 148, (cudaStream_t)stream) == 0 ? 0 : 3;
}

uint32_t wino_shift_error_read_clear() {
  uint32_t v = 0, z = 0;
  cudaMemcpyFromSymbol(&v, g_shift_err, sizeof(v));
  cudaMemcpyToSymbol(g_shift_err, &z, sizeof(z));
  return v;
}

}  // extern "C"
