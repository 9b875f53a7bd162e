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

// The operand from a fused U cache (p.pweight).
template <int CG>
__global__ void __launch_bounds__(128) shift_weight_u_kernel(KernelParam p) {
  shift_weight_from_u<CG>(p, static_cast<const __half*>(p.pweight), static_cast<uint8_t*>(p.transform_filter),
                          blockIdx.x * 128 + threadIdx.x);
}
// ... of every layer of a table (grid y).
__global__ void __launch_bounds__(128) shift_weight_u_batch_kernel(const __grid_constant__ ShiftTable t) {
  const KernelParam& p = t.layer[blockIdx.y].p;
  shift_weight_from_u<2>(p, static_cast<const __half*>(p.pweight), static_cast<uint8_t*>(p.transform_filter),
                         blockIdx.x * 128 + threadIdx.x);
}

// One CTA a unit (128 positions, up to 128 output channels).
template <bool EDGES>
__global__ void __launch_bounds__(sc::NTHREAD, 1) shift_conv_kernel(KernelParam p) {
  shift_conv_body<1, sc::NOEPI>(sc::OneConv<sc::PLAIN, EDGES>{p}, sc::Epi{}, &g_shift_err);
}

// A pair of CTAs a unit (256 positions, up to 256 output channels).
template <bool EDGES>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(sc::NTHREAD, 1) shift_conv_pair_kernel(KernelParam p) {
  shift_conv_body<2, sc::NOEPI>(sc::OneConv<sc::PLAIN, EDGES>{p}, sc::Epi{}, &g_shift_err);
}

// The same for problems whose filter columns became channels.
__global__ void __launch_bounds__(sc::NTHREAD, 1) shift_conv_fold_kernel(KernelParam p) {
  shift_conv_body<1, sc::NOEPI>(sc::OneConv<sc::FOLDED>{p}, sc::Epi{}, &g_shift_err);
}
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(sc::NTHREAD, 1) shift_conv_fold_pair_kernel(KernelParam p) {
  shift_conv_body<2, sc::NOEPI>(sc::OneConv<sc::FOLDED>{p}, sc::Epi{}, &g_shift_err);
}

// The same with the fused epilogue.
template <int EPI, bool EDGES>
__global__ void __launch_bounds__(sc::NTHREAD, 1) shift_conv_epi_kernel(KernelParam p, sc::Epi e) {
  shift_conv_body<1, EPI>(sc::OneConv<sc::PLAIN, EDGES>{p}, e, &g_shift_err);
}
template <int EPI, bool EDGES>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(sc::NTHREAD, 1)
    shift_conv_epi_pair_kernel(KernelParam p, sc::Epi e) {
  shift_conv_body<2, EPI>(sc::OneConv<sc::PLAIN, EDGES>{p}, e, &g_shift_err);
}
template <int CG, bool EDGES>
static const void* epi_kernel(bool even) {
  if (CG == 2)
    return even ? (const void*)shift_conv_epi_pair_kernel<sc::EPI_PAIR, EDGES>
                : (const void*)shift_conv_epi_pair_kernel<sc::EPI_ODD, EDGES>;
  return even ? (const void*)shift_conv_epi_kernel<sc::EPI_PAIR, EDGES>
              : (const void*)shift_conv_epi_kernel<sc::EPI_ODD, EDGES>;
}

// A table of layers, passed by value: the roles read their layers' dims from
// the constant bank (from a table in memory every role kept them in registers
// and spilled).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(sc::NTHREAD, 1)
    shift_conv_batch_kernel(const __grid_constant__ ShiftTable t) {
  shift_conv_body<2, sc::NOEPI>(sc::ConvTable{t}, sc::Epi{}, &g_shift_err);
}

}  // namespace wino

using namespace wino;

extern "C" {

void* wino_shift_kernel_ptr(const KernelParam* p, int cg) {
  if (sc::folds(p->c, p->s)) return cg == 2 ? (void*)shift_conv_fold_pair_kernel : (void*)shift_conv_fold_kernel;
  if (sc::input_edges(*p)) return cg == 2 ? (void*)shift_conv_pair_kernel<true> : (void*)shift_conv_kernel<true>;
  return cg == 2 ? (void*)shift_conv_pair_kernel<false> : (void*)shift_conv_kernel<false>;
}
// Host tests: item_at_edge for an item of `ch` channels.
int wino_shift_item_at_edge(unsigned o, unsigned head, unsigned total, unsigned plane, int ch) {
  return sc::item_at_edge(o, head, total, sc::item_span(plane, ch)) ? 1 : 0;
}
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
  // byte offsets into input and output in 32 bits
  if ((long long)p->n * p->c * p->h * p->w >= (1LL << 31) || (long long)p->n * p->k * p->Oh * p->Ow >= (1LL << 31))
    return 0;
  const bool aligned = sc::input_aligned(p->h * p->w, p->pin);
  for (const sc::Plan* g : {&g1, &g2})
    if ((!g->fold && sc::stage_items(*g, aligned) > sc::MAXITEMS) || g->nstage < 2 || g->rows > sc::MAXROWS || g->nu > 2 ||
        (g->fold && g->nst > 1))
      return 0;
  const long long w1 = (g1.units + sc::NSM - 1) / sc::NSM, w2 = (g2.units + sc::NSM / 2 - 1) / (sc::NSM / 2);
  const int n2 = g2.Kp < 256 ? (g2.Kp + 31) / 32 * 32 : 256;
  // one wave of single CTAs beats pairs that leave SMs idle (3x3 N20 C128 28x28
  // K128 14.1 us alone, 15.5 in pairs); from the second wave on pairs win though
  // some idle (N64 C256 14x14 K256 31.2 / 24.7; N64 C256 28x28 K256 stride 2
  // 55.5 / 34.9; N128 C512 7x7 K512 52.3 / 36.1)
  if (g2.units < sc::NSM / 2 && w1 == 1) return 1;
  // narrow outputs: a pair's halved weights gain nothing there and the tiles of
  // one CTA balance better (3x3 N32 C64 56x56 K64 20.2 us alone, 22.6 in
  // pairs; 1x1 N32 C512 28x28 K128 16.3 / 20.6)
  if (g1.Kp <= (g1.taps == 1 ? 128 : 64)) return 1;
  const long long t1 = w1 * sc::mma_cycles(1, g1.Kp < g1.NB ? g1.Kp : g1.NB), t2 = w2 * sc::mma_cycles(2, n2);
  return t2 <= t1 ? 2 : 1;
}

// The packed plan the kernels read from the argument's transform_pin.
unsigned long long wino_shift_pack(const KernelParam* p, int cg) { return sc::pack_plan(sc::make_plan(*p, cg)); }

static unsigned units_grid(const sc::Plan& g, int cg, int sms) {
  const long long cap = sms / cg;
  return (unsigned)(cg * (g.units < cap ? g.units : cap));
}
unsigned wino_shift_grid(const KernelParam* p, int cg, int sms) { return units_grid(sc::make_plan(*p, cg), cg, sms); }

// Packed plan and both kernels' grids of a drop-in problem.
unsigned long long wino_shift_slots(const KernelParam* p, int cg, int sms, unsigned* grid, unsigned* weight_grid) {
  const sc::Plan g = sc::make_plan(*p, cg);
  *grid = units_grid(g, cg, sms);
  *weight_grid = (unsigned)((sc::weight_bytes(g, cg) / 16 + 255) / 256);
  return sc::pack_plan(g);
}

static int shift_prepare_context() {
  for (const void* f :
       {(const void*)shift_conv_kernel<false>, (const void*)shift_conv_kernel<true>,
        (const void*)shift_conv_pair_kernel<false>, (const void*)shift_conv_pair_kernel<true>,
        (const void*)shift_conv_fold_kernel, (const void*)shift_conv_fold_pair_kernel, epi_kernel<1, false>(true),
        epi_kernel<1, false>(false), epi_kernel<1, true>(true), epi_kernel<1, true>(false), epi_kernel<2, false>(true),
        epi_kernel<2, false>(false), epi_kernel<2, true>(true), epi_kernel<2, true>(false),
        (const void*)shift_conv_batch_kernel}) {
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, sc::SMEM_BYTES) != cudaSuccess) return 1;
  }
  return 0;
}
int wino_shift_prepare() {
  static OncePerContext once;
  return once.run(shift_prepare_context);
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

// Launch with programmatic stream serialization: the kernel may start while
// the one before it, which makes its weight operand, still runs (the operand
// is waited for in the kernel).
int wino_launch_dependent(const void* fn, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t stream) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelExC(&cfg, fn, args);
}

// Launches the kernel on a problem whose weight operand is at
// p->transform_filter and packed plan in p->transform_pin; the launch before
// it on the stream is the one that makes the operand.
int wino_launch_shift(const KernelParam* p, int cg, int sms, cudaStream_t stream) {
  void* args[] = {const_cast<KernelParam*>(p)};
  return wino_launch_dependent(wino_shift_kernel_ptr(p, cg), dim3(wino_shift_grid(p, cg, sms)), dim3(sc::NTHREAD), args,
                               (size_t)sc::SMEM_BYTES, stream);
}

// ---- convolutions on a fused U cache ------------------------------------
// Direct-conv FLOPs from which the fused entry points (conv, epilogue, batch)
// recover the filter from U and take this kernel.  Not where the kernels cross:
// in a graph, the conv takes 16.4 us on the fused Winograd kernel and 10.3 on this one at
// N1 C64 14x14 K64 (14 MFLOP), 30.8 and 14.4 at N2 C256 14x14 K256 (462); the
// epilogue 24 and 12, 37 and 16.  Below the line results are bit-identical to the fused
// kernel's configurations (wino_conv2d_fused_cfg), which tests hold at up to 265 MFLOP.
static constexpr double kFusedMinFlops = 512e6;

// CTAs a unit for a problem (dims and tensors set), or 0 when it stays with
// the fused kernel.
int wino_shift_fused_cg(const KernelParam* p) {
  if (p->c % 16 || p->k % 16 || 2.0 * p->n * p->k * p->h * p->w * p->c * 9 < kFusedMinFlops) return 0;
  return wino_shift_cg(p);
}
// Whether a batch's table can hold a problem that wino_shift_fused_cg takes
// (pairs): its producers own one item each, of words inside the input.
int wino_shift_in_table(const KernelParam* p) {
  return !sc::input_edges(*p) && sc::stage_items(sc::make_plan(*p, 2, sc::TABLE),
                                                 sc::input_aligned(p->h * p->w, p->pin)) <= sc::NPROD;
}

int wino_launch_shift_weight_u(const KernelParam* p, int cg, cudaStream_t stream) {
  const size_t items = wino_shift_weight_bytes(p, cg) / (9 * 16);
  void* args[] = {const_cast<KernelParam*>(p)};
  return (int)cudaLaunchKernel(cg == 2 ? (void*)shift_weight_u_kernel<2> : (void*)shift_weight_u_kernel<1>,
                               dim3((unsigned)((items + 127) / 128)), dim3(128), args, 0, stream);
}

// y = relu?(conv + bias + residual) on the U cache `u`; wop holds
// wino_shift_weight_bytes.
int wino_launch_shift_fused(const KernelParam* p0, const void* u, void* wop, int cg, const VariantArgs* va, int sms,
                            cudaStream_t stream) {
  if (wino_shift_prepare() != 0) return (int)cudaErrorInvalidValue;
  KernelParam p = *p0;
  p.pweight = const_cast<void*>(u);
  p.transform_filter = wop;
  p.transform_pin = reinterpret_cast<void*>(wino_shift_pack(&p, cg));
  const int rc = wino_launch_shift_weight_u(&p, cg, stream);
  if (rc != 0) return rc;
  if (!va || (!va->bias && !va->residual && !va->relu)) return wino_launch_shift(&p, cg, sms, stream);
  sc::Epi e{va->bias, static_cast<const __half*>(va->residual), va->relu};
  void* args[] = {&p, &e};
  const bool even = sc::store_pairs(p.Ow, p.pout, va->residual);
  const void* fn = sc::input_edges(p) ? (cg == 2 ? epi_kernel<2, true>(even) : epi_kernel<1, true>(even))
                                      : (cg == 2 ? epi_kernel<2, false>(even) : epi_kernel<1, false>(even));
  return wino_launch_dependent(fn, dim3(wino_shift_grid(&p, cg, sms)), dim3(sc::NTHREAD), args, (size_t)sc::SMEM_BYTES,
                               stream);
}

// Completes a table whose layers have dims, tensors, U cache (pweight) and
// operand buffer (transform_filter): plans, unit numbers, the common ring.
void wino_shift_table_finish(ShiftTable* t) {
  t->units = t->pitch = 0;
  for (int l = 0; l < t->nlayers; ++l) {
    ShiftLayer& d = t->layer[l];
    const sc::Plan g = sc::make_plan(d.p, 2, sc::TABLE);
    d.p.transform_pin = reinterpret_cast<void*>(sc::pack_plan(g));
    d.unit_begin = t->units;
    d.units = g.units;
    t->units += g.units;
    if (g.pitch > t->pitch) t->pitch = g.pitch;
  }
  const int fit = t->pitch > 0 ? sc::SMEM_STAGES / t->pitch : 0;
  t->nstage = fit < sc::MAXSTAGE ? fit : sc::MAXSTAGE;
}

// Cost of one unit of a layer in MMA cycles (to order a table by).
double wino_shift_unit_cost(const KernelParam* p) {
  const sc::Plan g = sc::make_plan(*p, 2);
  return (double)g.NKS * sc::mma_cycles(2, g.Kp < 256 ? (g.Kp + 31) / 32 * 32 : 256);
}

// The operands of a table's layers, then one launch over all of them.
int wino_launch_shift_batch(const ShiftTable* t, int sms, cudaStream_t stream) {
  size_t items = 0;
  for (int l = 0; l < t->nlayers; ++l) {
    const size_t i = wino_shift_weight_bytes(&t->layer[l].p, 2) / (9 * 16);
    if (i > items) items = i;
  }
  void* args[] = {const_cast<ShiftTable*>(t)};
  cudaError_t e = cudaLaunchKernel((void*)shift_weight_u_batch_kernel,
                                   dim3((unsigned)((items + 127) / 128), (unsigned)t->nlayers), dim3(128), args, 0,
                                   stream);
  if (e != cudaSuccess) return (int)e;
  const int pairs = sms / 2, grid = 2 * (t->units < pairs ? t->units : pairs);
  return wino_launch_dependent((void*)shift_conv_batch_kernel, dim3((unsigned)grid), dim3(sc::NTHREAD), args,
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
  if (weight) return wino_launch_shift(&p, cg, sc::NSM, (cudaStream_t)stream) == 0 ? 0 : 3;
  return cudaLaunchKernel(wino_shift_kernel_ptr(&p, cg), dim3(wino_shift_grid(&p, cg, sc::NSM)), dim3(sc::NTHREAD), args,
                          (size_t)sc::SMEM_BYTES, (cudaStream_t)stream) == cudaSuccess
             ? 0
             : 3;
}

uint32_t wino_shift_error_read_clear() {
  uint32_t v = 0, z = 0;
  cudaMemcpyFromSymbol(&v, g_shift_err, sizeof(v));
  cudaMemcpyToSymbol(g_shift_err, &z, sizeof(z));
  return v;
}

}  // extern "C"
