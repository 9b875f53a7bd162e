// Host side of the drop-in plugin ABI (include/conv2d.h) and of the
// extension C-ABI (include/winoconv.h).  Plain C++ (compiled by the host
// compiler, so the `_Float16` declarations of the reference-compatible
// headers compile); kernels are reached through their entry pointers.
//
// getParamsize / getkernelInfo replace the reference's src/conv2d.cpp:9-14 and
// :254-517.  The reference picks one of six hard-wired kernel quadruples by
// (n, c) and returns 0 for every input; here any shape inside the contract
// gets the same two real kernels (filter transform, fused conv) and anything
// else is rejected with an error code before a kernel is chosen.
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <cuda_runtime.h>

#include "conv2d.h"
#include "mykernelParamType.cuh"
#include "winoconv.h"
#include "wino_param.h"

// The kernel argument the device sees must be bit-for-bit the host struct.
static_assert(sizeof(mykernelParamType) == sizeof(wino::KernelParam), "param size");
#define WINO_SAME_OFFSET(f) \
  static_assert(offsetof(mykernelParamType, f) == offsetof(wino::KernelParam, f), #f)
WINO_SAME_OFFSET(pin);
WINO_SAME_OFFSET(pweight);
WINO_SAME_OFFSET(pout);
WINO_SAME_OFFSET(transform_pin);
WINO_SAME_OFFSET(transform_filter);
WINO_SAME_OFFSET(mid_result);
WINO_SAME_OFFSET(n);
WINO_SAME_OFFSET(c);
WINO_SAME_OFFSET(h);
WINO_SAME_OFFSET(w);
WINO_SAME_OFFSET(k);
WINO_SAME_OFFSET(r);
WINO_SAME_OFFSET(s);
WINO_SAME_OFFSET(u);
WINO_SAME_OFFSET(v);
WINO_SAME_OFFSET(p);
WINO_SAME_OFFSET(q);
WINO_SAME_OFFSET(Oh);
WINO_SAME_OFFSET(Ow);
#undef WINO_SAME_OFFSET
static_assert(sizeof(problem_t) == 96, "problem_t layout");
static_assert(sizeof(kernelInfo_t) == 160, "kernelInfo_t layout");

extern "C" {
void* wino_dropin_filter_kernel_ptr();
void* wino_fused_kernel_ptr();
void* wino_noop_kernel_ptr();
int wino_fused_prepare();
int wino_fused_smem_bytes();
int wino_fused_threads();
long long wino_fused_nblocks(int n, int h, int w, int k);
uint32_t wino_fused_error_read_clear();
void* wino_direct_kernel_ptr();
void wino_direct_grid(int n, int k, int oh, int ow, unsigned* gx, unsigned* gy);
int wino_launch_direct(const wino::KernelParam* p, cudaStream_t stream);
void* wino_xb_layout_kernel_ptr();
size_t wino_xb_bytes(int n, int c, int h, int w);
unsigned wino_xb_layout_grid(int n, int c, int h, int w);
long long wino_xb_items(int n, int c, int h, int w);
int wino_launch_xb_layout(const wino::KernelParam* p, cudaStream_t stream);
int wino_launch_xb_layout_beside(const wino::KernelParam* p, cudaStream_t stream);
int wino_launch_xb_layout_amax(const wino::KernelParam* p, cudaStream_t stream);
int wino_launch_xb_f8_scales(const unsigned* amax, float* sv, uint32_t* inv_sv2, int C,
                             cudaStream_t stream);
int wino_launch_filter_transform_f8(const void* weight, const float* sv, void* u8, float* su, int K,
                                    int C, cudaStream_t stream);
}
extern "C" {
int wino_fused_launch_variant(int variant, const wino::KernelParam* p, const wino::VariantArgs* va,
                              int cfg, unsigned grid, cudaStream_t stream);
size_t wino_unfused_v_bytes(int n, int c, int h, int w);
size_t wino_unfused_m_bytes(int n, int k, int h, int w);
int wino_unfused_prepare();
int wino_unfused_launch(const wino::KernelParam* p, int sms, cudaStream_t stream);
uint32_t wino_unfused_error_read_clear();
int wino_launch_filter_transform(const void* weight, void* ucache, void* ucache_lo, int K, int C,
                                 int bf16, int layout, cudaStream_t stream);
void* wino_dropin_filter_u2_kernel_ptr();
void* wino_twostage_gemm_kernel_ptr_for(int c);
void* wino_twostage_output_kernel_ptr();
void* wino_twostage_resv_kernel_ptr();
int wino_twostage_threads_for(int c);
int wino_twostage_smem_bytes_for(int c);
int wino_twostage_prepare();
size_t wino_twostage_m_bytes(int n, int h, int w, int k);
unsigned wino_twostage_gemm_grid(int n, int c, int h, int w, int k, int sms);
size_t wino_twostage_prepass_bytes(int n, int c, int h, int w);
long long wino_twostage_prepass_items(int n, int c, int h, int w);
void* wino_twostage_prepass_kernel_ptr_for(int c);
unsigned wino_twostage_prepass_grid(int n, int c, int h, int w);
int wino_launch_twostage_prepass(const wino::KernelParam* p, cudaStream_t stream);
int wino_twostage_prepass_smem_bytes(int c);
void wino_twostage_output_grid(int n, int h, int w, int k, int sms, unsigned* gx, unsigned* gy);
int wino_twostage_output_threads();
int wino_twostage_output_smem_bytes();
uint32_t wino_twostage_error_read_clear();
size_t wino_igemm_weight_bytes(int c, int k, int r, int s);
unsigned wino_igemm_weight_grid(int c, int k, int r, int s);
void* wino_igemm_weight_kernel_ptr();
void* wino_igemm_kernel_ptr(int k, int mode);
int wino_igemm_mode(const void* x, int k, int h, int w, int r, int s, int u, int v, int p, int q);
int wino_igemm_encode_map(void* map_host, const void* x, int n, int c, int hw);
size_t wino_igemm_operand_bytes(int c, int k, int r, int s);
size_t wino_igemm_map_offset(int c, int k, int r, int s);
int wino_igemm_threads();
int wino_igemm_smem_bytes();
unsigned wino_igemm_grid(int n, int k, int oh, int ow, int sms);
int wino_igemm_shape_ok(int n, int c, int h, int w, int k, int oh, int ow);
int wino_igemm_prepare();
uint32_t wino_igemm_error_read_clear();
int wino_shift_cg(const wino::KernelParam* p);
unsigned long long wino_shift_slots(const wino::KernelParam* p, int cg, int sms, unsigned* grid, unsigned* weight_grid);
size_t wino_shift_weight_bytes(const wino::KernelParam* p, int cg);
void* wino_shift_weight_kernel_ptr(int cg);
void* wino_shift_kernel_ptr(const wino::KernelParam* p, int cg);
int wino_shift_threads();
int wino_shift_smem_bytes();
int wino_shift_prepare();
uint32_t wino_shift_error_read_clear();
int wino_shift_fused_cg(const wino::KernelParam* p);
int wino_launch_dependent(const void* fn, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t stream);
int wino_launch_shift_fused(const wino::KernelParam* p0, const void* u, void* wop, int cg, const wino::VariantArgs* va,
                            int sms, cudaStream_t stream);
}

namespace {

constexpr int kMaxDim = 32767;  // dims are `short` in mykernelParamType
// implicit-GEMM pixel-operand producers (igemm_conv.cu)
constexpr int kIgemmModeFlat = 1, kIgemmModeTma = 2;

int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
    return 148;
  return n;
}

void set_slot(kernelInfo_t* ki, int slot, unsigned gx, unsigned gy, unsigned gz, unsigned tx,
              unsigned ty, unsigned tz, unsigned lds, void* fn) {
  unsigned* base = nullptr;
  void** ptr = nullptr;
  switch (slot) {
    case 1: base = &ki->blockx1; ptr = &ki->kernelPtr1; break;
    case 2: base = &ki->blockx2; ptr = &ki->kernelPtr2; break;
    case 3: base = &ki->blockx3; ptr = &ki->kernelPtr3; break;
    default: base = &ki->blockx4; ptr = &ki->kernelPtr4; break;
  }
  base[0] = gx; base[1] = gy; base[2] = gz;
  base[3] = tx; base[4] = ty; base[5] = tz;
  base[6] = lds;
  *ptr = fn;
}

wino::KernelParam make_param(const void* x, const void* w, void* y, void* vws, void* ucache,
                             void* mws, int n, int c, int h, int wd, int k) {
  wino::KernelParam p;
  p.pin = const_cast<void*>(x);
  p.pweight = const_cast<void*>(w);
  p.pout = y;
  p.transform_pin = vws;
  p.transform_filter = ucache;
  p.mid_result = mws;
  p.n = (short)n; p.c = (short)c; p.h = (short)h; p.w = (short)wd; p.k = (short)k;
  p.r = 3; p.s = 3; p.u = 1; p.v = 1; p.p = 1; p.q = 1;
  p.Oh = (short)h; p.Ow = (short)wd;
  return p;
}

// The pre-pass counts its items in 32 bits.
bool xb_items_ok(int n, int c, int h, int w) { return wino_xb_items(n, c, h, w) < (1LL << 31); }

// The two-stage producers address one (image, 16-channel) record block of
// their pre-pass records with 32-bit byte offsets: up to 4*ceil(h/2) + 2 rows
// of 64 * (ceil(w/2) + 1) bytes must stay below 2^31; the pre-pass counts its
// items and the GEMM its tiles in 32 bits.
bool twostage_ok(int n, int c, int h, int w) {
  const long long rows = 4LL * ((h + 1) / 2) + 2, row_bytes = 64LL * ((w + 1) / 2 + 1);
  const long long tiles = (long long)n * ((h + 1) / 2) * ((w + 1) / 2);
  return xb_items_ok(n, c, h, w) && wino_twostage_prepass_items(n, c, h, w) < (1LL << 31) &&
         rows * row_bytes < (1LL << 31) && tiles < (1LL << 30);
}

unsigned fused_grid(int n, int h, int w, int k) {
  const long long nb = wino_fused_nblocks(n, h, w, k);
  const long long sms = sm_count();
  return (unsigned)(nb < sms ? nb : sms);
}

}  // namespace

extern "C" int wino_check_shape(int n, int c, int h, int w, int k) {
  if (n < 1 || c < 1 || h < 1 || w < 1 || k < 1) return WINO_EINVAL;
  if (n > kMaxDim || c > kMaxDim || h > kMaxDim || w > kMaxDim || k > kMaxDim)
    return WINO_EUNSUPPORTED;
  if (c % 16 != 0 || k % 16 != 0) return WINO_EUNSUPPORTED;
  return WINO_OK;
}

extern "C" size_t wino_ucache_bytes(int k, int c, int variant) {
  const size_t elems = (size_t)16 * (size_t)k * (size_t)c;
  switch (variant) {
    case WINO_VAR_F8: return elems + (size_t)16 * k * sizeof(float);
    case WINO_VAR_F16_HILO: return 2 * elems * 2;
    default: return elems * 2;
  }
}

// --------------------------------------------------------- drop-in ABI ----
int getParamsize(problem_t* problem, int* paramSize) {
  (void)problem;
  if (!paramSize) return WINO_EINVAL;
  *paramSize = (int)sizeof(mykernelParamType);
  return WINO_OK;
}

// Validation shared by the drop-in and the direct-conv entry point: positive
// dims within the `short` fields, a filter no larger than the padded input.
int check_general(long long n, long long c, long long h, long long w, long long k, long long r,
                  long long s, long long u, long long v, long long p, long long q, int* oh, int* ow) {
  if (n < 1 || c < 1 || h < 1 || w < 1 || k < 1 || r < 1 || s < 1 || u < 1 || v < 1 || p < 0 || q < 0)
    return WINO_EINVAL;
  if (n > kMaxDim || c > kMaxDim || h > kMaxDim || w > kMaxDim || k > kMaxDim || r > kMaxDim ||
      s > kMaxDim || u > kMaxDim || v > kMaxDim || p > kMaxDim || q > kMaxDim)
    return WINO_EUNSUPPORTED;
  if (h + 2 * p < r || w + 2 * q < s) return WINO_EINVAL;
  const long long oh_ = (h - r + 2 * p) / u + 1, ow_ = (w - s + 2 * q) / v + 1;
  if (oh_ > kMaxDim || ow_ > kMaxDim) return WINO_EUNSUPPORTED;
  if (n * oh_ * ow_ / 64 >= (1LL << 31)) return WINO_EUNSUPPORTED;  // direct kernel's grid.x
  *oh = (int)oh_;
  *ow = (int)ow_;
  return WINO_OK;
}

// The shift-reuse implicit GEMM (shift_conv.cuh) for a drop-in problem: CTAs a
// unit and the workspace that holds its weight operand, or cg = 0.
struct ShiftPlan {
  int cg;
  void* wop;
};

// Direct-conv FLOPs from which the drop-in takes the shift kernel.  Not where
// the routes cross, which they do not: in a graph, N1 C16 16x16 K16 (1.2 MFLOP)
// takes 14.4 us on the two-stage route and 8.2 on the shift kernel, N2 C64 20x20
// K64 (59) 16.4 and 10.3, 3x3/2 N2 C128 14x14 K96 (22) 59 and 16, an RGB stem of
// one 112x112 image (59) 33 and 8.  Below the line results are bit-identical to
// wino_conv2d_twostage's, which tests hold at up to 36 MFLOP.
constexpr double kShiftMinFlops = 64e6;

// Two-stage route (input transform fused into full-width tap GEMMs, M in the
// caller's mid_result, output transform in slot 4): M fits the reference's
// mid_result size of 4*k*h*w*n fp16 elements (even H and W) and the pre-pass
// records fit transform_pin.
static bool two_stage_fits(const problem_t& pr) {
  return pr.transform_pin != nullptr && (reinterpret_cast<uintptr_t>(pr.transform_pin) & 15) == 0 &&
         pr.mid_result != nullptr && (reinterpret_cast<uintptr_t>(pr.mid_result) & 15) == 0 &&
         twostage_ok((int)pr.n, (int)pr.c, (int)pr.h, (int)pr.w) &&
         wino_twostage_prepass_bytes((int)pr.n, (int)pr.c, (int)pr.h, (int)pr.w) <=
             (size_t)4 * pr.h * pr.h * pr.n * pr.c * 2 &&
         wino_twostage_m_bytes((int)pr.n, (int)pr.h, (int)pr.w, (int)pr.k) <= (size_t)4 * pr.k * pr.h * pr.w * pr.n * 2;
}

// 3x3 / stride 1 / pad 1 with 16-channel multiples and a U-cache workspace.
static bool wino_contract(const problem_t& pr) {
  return pr.r == 3 && pr.s == 3 && pr.u == 1 && pr.v == 1 && pr.p == 1 && pr.q == 1 &&
         wino_check_shape((int)pr.n, (int)pr.c, (int)pr.h, (int)pr.w, (int)pr.k) == WINO_OK &&
         pr.transform_filter != nullptr;
}

// Problems that the shift route leaves the two-stage route's kernels in slots 3
// and 4, by which callers tell a problem that route fits; given no mid_result
// they have nothing to do.
static bool keeps_two_stage_slots(const problem_t& pr) {
  return wino_twostage_gemm_kernel_ptr_for((int)pr.c) == wino_twostage_resv_kernel_ptr() && wino_contract(pr) &&
         two_stage_fits(pr);
}

static ShiftPlan plan_shift(const problem_t& pr, int oh, int ow) {
  const ShiftPlan none{0, nullptr};
  if (!pr.transform_filter) return none;
  // strided filters of one or two taps stay with the gathering implicit GEMM,
  // which reads only the pixels it needs, where this kernel loads every one for
  // a few MMAs (1x1/2 N32 C256 56x56 K128 23 us against 29; 1x2/2 N60 C16
  // 137x137 K64 50 against 73; 2x1/2 N29 C256 67x67 K128 58 against 83).  From
  // three taps on it wins (3x1/2 N9 C256 42x42 K64 67 against 30)
  if (pr.r * pr.s <= 2 && (pr.u > 1 || pr.v > 1)) return none;
  if (2.0 * pr.n * pr.k * oh * ow * pr.c * pr.r * pr.s < kShiftMinFlops) return none;
  wino::KernelParam p{};
  p.pin = pr.in;
  p.n = (short)pr.n; p.c = (short)pr.c; p.h = (short)pr.h; p.w = (short)pr.w; p.k = (short)pr.k;
  p.r = (short)pr.r; p.s = (short)pr.s; p.u = (short)pr.u; p.v = (short)pr.v; p.p = (short)pr.p; p.q = (short)pr.q;
  p.Oh = (short)oh; p.Ow = (short)ow;
  int cg = wino_shift_cg(&p);
  if (cg == 0) return none;
  // weight operand: the caller's transform_filter (16*k*c fp16), else its
  // transform_pin (4*h*h*n*c fp16); reference src/main.cpp:36-38
  const size_t filter_bytes = (size_t)16 * pr.k * pr.c * 2, pin_bytes = (size_t)4 * pr.h * pr.h * pr.n * pr.c * 2;
  for (; cg >= 1; --cg) {
    const size_t need = wino_shift_weight_bytes(&p, cg);
    if (need <= filter_bytes && (reinterpret_cast<uintptr_t>(pr.transform_filter) & 15) == 0)
      return ShiftPlan{cg, pr.transform_filter};
    if (pr.transform_pin && need <= pin_bytes && (reinterpret_cast<uintptr_t>(pr.transform_pin) & 15) == 0)
      return ShiftPlan{cg, pr.transform_pin};
  }
  return none;
}

// Route of getkernelInfo for a validated problem (no CUDA calls).
static int plan_route(const problem_t& pr, ShiftPlan* shift) {
  const int oh = (int)((pr.h - pr.r + 2 * pr.p) / pr.u + 1), ow = (int)((pr.w - pr.s + 2 * pr.q) / pr.v + 1);
  *shift = plan_shift(pr, oh, ow);
  // (outside the contract it is the implicit-GEMM route with another kernel)
  if (shift->cg) return wino_contract(pr) ? WINO_ROUTE_SHIFT : WINO_ROUTE_IGEMM;
  // Winograd F(2x2,3x3) inside its contract; every other shape goes to the
  // implicit GEMM or the direct kernel.
  if (!wino_contract(pr)) {
    // Tensor-core implicit GEMM when its re-laid-out weights fit the
    // caller's transform_filter (16*k*c fp16, reference src/main.cpp:38).
    const bool igemm = pr.transform_filter != nullptr &&
                       (reinterpret_cast<uintptr_t>(pr.transform_filter) & 15) == 0 &&
                       wino_igemm_operand_bytes((int)pr.c, (int)pr.k, (int)pr.r, (int)pr.s) <=
                           (size_t)16 * pr.k * pr.c * 2 &&
                       wino_igemm_shape_ok((int)pr.n, (int)pr.c, (int)pr.h, (int)pr.w, (int)pr.k, oh, ow);
    return igemm ? WINO_ROUTE_IGEMM : WINO_ROUTE_DIRECT;
  }
  // The caller's transform_pin workspace holds 4*h*h*n*c fp16 elements
  // (reference src/main.cpp:36-38); when the channel-blocked input fits
  // there (and is 16-byte aligned) slot 2 writes it, otherwise the fused
  // kernel reads the NCHW input itself.
  const size_t pin_ws_bytes = (size_t)4 * pr.h * pr.h * pr.n * pr.c * 2;
  const bool use_xb = pr.transform_pin != nullptr &&
                      (reinterpret_cast<uintptr_t>(pr.transform_pin) & 15) == 0 &&
                      wino_xb_bytes((int)pr.n, (int)pr.c, (int)pr.h, (int)pr.w) <= pin_ws_bytes &&
                      xb_items_ok((int)pr.n, (int)pr.c, (int)pr.h, (int)pr.w);
  if (two_stage_fits(pr)) return WINO_ROUTE_TWOSTAGE;
  return use_xb ? WINO_ROUTE_FUSED_XB : WINO_ROUTE_FUSED;
}

int getkernelInfo(problem_t* problem, kernelInfo_t* kernelInfo, void* param) {
  if (!problem || !kernelInfo || !param) return WINO_EINVAL;
  const problem_t& pr = *problem;
  int oh = 0, ow = 0;
  const int st = check_general(pr.n, pr.c, pr.h, pr.w, pr.k, pr.r, pr.s, pr.u, pr.v, pr.p, pr.q, &oh, &ow);
  if (st != WINO_OK) return st;
  if (!pr.in || !pr.weight || !pr.out) return WINO_EINVAL;
  ShiftPlan shift{};
  int route = plan_route(pr, &shift);
  if (route == WINO_ROUTE_IGEMM && shift.cg == 0 && wino_igemm_prepare() != 0) route = WINO_ROUTE_DIRECT;
  const bool wino = route != WINO_ROUTE_DIRECT && route != WINO_ROUTE_IGEMM;

  mykernelParamType* a = static_cast<mykernelParamType*>(param);
  a->pin = pr.in;
  a->pweight = pr.weight;
  a->pout = pr.out;
  a->transform_filter = pr.transform_filter;
  a->mid_result = pr.mid_result;
  a->n = (short)pr.n; a->c = (short)pr.c; a->h = (short)pr.h; a->w = (short)pr.w;
  a->k = (short)pr.k; a->r = (short)pr.r; a->s = (short)pr.s; a->u = (short)pr.u;
  a->v = (short)pr.v; a->p = (short)pr.p; a->q = (short)pr.q;
  a->Oh = (short)oh; a->Ow = (short)ow;
  std::memset(kernelInfo, 0, sizeof(*kernelInfo));

  if (shift.cg != 0) {
    if (wino_shift_prepare() != 0) return WINO_ECUDA;
    a->transform_filter = static_cast<_Float16*>(shift.wop);
    a->mid_result = nullptr;
    wino::KernelParam* kp = static_cast<wino::KernelParam*>(param);
    // the packed plan travels in transform_pin, which the kernels need no
    // pointer in
    unsigned grid = 0, weight_grid = 0;
    kp->transform_pin =
        reinterpret_cast<void*>(wino_shift_slots(kp, shift.cg, sm_count(), &grid, &weight_grid));
    set_slot(kernelInfo, 1, weight_grid, 1, 1, 256, 1, 1, 0,
             wino_shift_weight_kernel_ptr(shift.cg));
    const bool keeps = keeps_two_stage_slots(pr);
    set_slot(kernelInfo, keeps ? 2 : 3, grid, 1, 1, (unsigned)wino_shift_threads(), 1, 1,
             (unsigned)wino_shift_smem_bytes(), wino_shift_kernel_ptr(kp, shift.cg));
    if (keeps) {
      set_slot(kernelInfo, 3, 1, 1, 1, (unsigned)wino_twostage_threads_for((int)pr.c), 1, 1, 0,
               wino_twostage_gemm_kernel_ptr_for((int)pr.c));
      set_slot(kernelInfo, 4, 1, 1, 1, (unsigned)wino_twostage_output_threads(), 1, 1, 0,
               wino_twostage_output_kernel_ptr());
    } else {
      set_slot(kernelInfo, 2, 1, 1, 1, 32, 1, 1, 0, wino_noop_kernel_ptr());
      set_slot(kernelInfo, 4, 1, 1, 1, 32, 1, 1, 0, wino_noop_kernel_ptr());
    }
    return WINO_OK;
  }
  if (route == WINO_ROUTE_IGEMM) {
    int mode = wino_igemm_mode(pr.in, (int)pr.k, (int)pr.h, (int)pr.w, (int)pr.r, (int)pr.s, (int)pr.u,
                               (int)pr.v, (int)pr.p, (int)pr.q);
    a->transform_pin = nullptr;
    if (mode == kIgemmModeTma) {
      // the input's tensor map goes to the (otherwise unused) transform_pin
      // workspace, 4*h*h*n*c fp16 >= 128 bytes, written once here
      alignas(64) unsigned char map[128];
      const bool ok = pr.transform_pin != nullptr && (reinterpret_cast<uintptr_t>(pr.transform_pin) & 127) == 0 &&
                      (size_t)4 * pr.h * pr.h * pr.n * pr.c * 2 >= sizeof(map) &&
                      wino_igemm_encode_map(map, pr.in, (int)pr.n, (int)pr.c, (int)(pr.h * pr.w)) == 0 &&
                      cudaMemcpy(pr.transform_pin, map, sizeof(map), cudaMemcpyHostToDevice) == cudaSuccess;
      if (ok) a->transform_pin = pr.transform_pin;
      else mode = kIgemmModeFlat;
    }
    set_slot(kernelInfo, 1, wino_igemm_weight_grid((int)pr.c, (int)pr.k, (int)pr.r, (int)pr.s), 1, 1, 256, 1,
             1, 0, wino_igemm_weight_kernel_ptr());
    set_slot(kernelInfo, 2, 1, 1, 1, 32, 1, 1, 0, wino_noop_kernel_ptr());
    set_slot(kernelInfo, 3, wino_igemm_grid((int)pr.n, (int)pr.k, oh, ow, sm_count()), 1, 1,
             (unsigned)wino_igemm_threads(), 1, 1, (unsigned)wino_igemm_smem_bytes(),
             wino_igemm_kernel_ptr((int)pr.k, mode));
    set_slot(kernelInfo, 4, 1, 1, 1, 32, 1, 1, 0, wino_noop_kernel_ptr());
    return WINO_OK;
  }
  if (!wino) {
    unsigned gx, gy;
    wino_direct_grid((int)pr.n, (int)pr.k, oh, ow, &gx, &gy);
    a->transform_pin = nullptr;
    set_slot(kernelInfo, 1, 1, 1, 1, 32, 1, 1, 0, wino_noop_kernel_ptr());
    set_slot(kernelInfo, 2, 1, 1, 1, 32, 1, 1, 0, wino_noop_kernel_ptr());
    set_slot(kernelInfo, 3, gx, gy, 1, 256, 1, 1, 0, wino_direct_kernel_ptr());
    set_slot(kernelInfo, 4, 1, 1, 1, 32, 1, 1, 0, wino_noop_kernel_ptr());
    return WINO_OK;
  }

  if (wino_fused_prepare() != 0) return WINO_ECUDA;
  if (route == WINO_ROUTE_TWOSTAGE && wino_twostage_prepare() != 0) route = WINO_ROUTE_FUSED_XB;
  const bool use_xb = route != WINO_ROUTE_FUSED;
  a->transform_pin = use_xb ? pr.transform_pin : nullptr;

  const long long kc = (long long)pr.k * pr.c;
  if (route == WINO_ROUTE_TWOSTAGE) {
    set_slot(kernelInfo, 1, (unsigned)((kc + 255) / 256), 1, 1, 256, 1, 1, 0,
             wino_dropin_filter_u2_kernel_ptr());
    const int c = (int)pr.c;
    set_slot(kernelInfo, 2, wino_twostage_prepass_grid((int)pr.n, c, (int)pr.h, (int)pr.w), 1, 1, 256, 1, 1,
             wino_twostage_prepass_smem_bytes(c), wino_twostage_prepass_kernel_ptr_for(c));
    set_slot(kernelInfo, 3, wino_twostage_gemm_grid((int)pr.n, c, (int)pr.h, (int)pr.w, (int)pr.k, sm_count()), 1,
             1, (unsigned)wino_twostage_threads_for(c), 1, 1, (unsigned)wino_twostage_smem_bytes_for(c),
             wino_twostage_gemm_kernel_ptr_for(c));
    unsigned ox, oy;
    wino_twostage_output_grid((int)pr.n, (int)pr.h, (int)pr.w, (int)pr.k, sm_count(), &ox, &oy);
    set_slot(kernelInfo, 4, ox, oy, 1, (unsigned)wino_twostage_output_threads(), 1, 1,
             (unsigned)wino_twostage_output_smem_bytes(),
             wino_twostage_output_kernel_ptr());
    return WINO_OK;
  }
  set_slot(kernelInfo, 1, (unsigned)((kc + 255) / 256), 1, 1, 256, 1, 1, 0,
           wino_dropin_filter_kernel_ptr());
  if (use_xb)
    set_slot(kernelInfo, 2, wino_xb_layout_grid((int)pr.n, (int)pr.c, (int)pr.h, (int)pr.w), 1, 1, 256, 1, 1, 0,
             wino_xb_layout_kernel_ptr());
  else
    set_slot(kernelInfo, 2, 1, 1, 1, 32, 1, 1, 0, wino_noop_kernel_ptr());
  set_slot(kernelInfo, 3, fused_grid((int)pr.n, (int)pr.h, (int)pr.w, (int)pr.k), 1, 1,
           (unsigned)wino_fused_threads(), 1, 1, (unsigned)wino_fused_smem_bytes(),
           wino_fused_kernel_ptr());
  set_slot(kernelInfo, 4, 1, 1, 1, 32, 1, 1, 0, wino_noop_kernel_ptr());
  return WINO_OK;
}

extern "C" int wino_dropin_route(const void* problem) {
  if (!problem) return -WINO_EINVAL;
  const problem_t& pr = *static_cast<const problem_t*>(problem);
  int oh = 0, ow = 0;
  const int st = check_general(pr.n, pr.c, pr.h, pr.w, pr.k, pr.r, pr.s, pr.u, pr.v, pr.p, pr.q, &oh, &ow);
  if (st != WINO_OK) return -st;
  if (!pr.in || !pr.weight || !pr.out) return -WINO_EINVAL;
  ShiftPlan shift{};
  return plan_route(pr, &shift);
}

extern "C" int wino_getParamsize(problem_t* problem, int* paramSize) {
  return getParamsize(problem, paramSize);
}
extern "C" int wino_getkernelInfo(problem_t* problem, kernelInfo_t* kernelInfo, void* param) {
  return getkernelInfo(problem, kernelInfo, param);
}

// ------------------------------------------------------- extension API ----
extern "C" int wino_filter_transform(const void* weight, void* ucache, int k, int c, void* stream) {
  if (!weight || !ucache) return WINO_EINVAL;
  const int st = wino_check_shape(1, c, 1, 1, k);
  if (st != WINO_OK) return st;
  return wino_launch_filter_transform(weight, ucache, nullptr, k, c, 0, 0, (cudaStream_t)stream) == 0
             ? WINO_OK
             : WINO_ECUDA;
}

extern "C" int wino_filter_transform_unfused(const void* weight, void* ucache2, int k, int c,
                                             void* stream) {
  if (!weight || !ucache2) return WINO_EINVAL;
  const int st = wino_check_shape(1, c, 1, 1, k);
  if (st != WINO_OK) return st;
  return wino_launch_filter_transform(weight, ucache2, nullptr, k, c, 0, 1, (cudaStream_t)stream) == 0
             ? WINO_OK
             : WINO_ECUDA;
}

extern "C" int wino_unfused_workspace_bytes(int n, int c, int h, int w, int k, size_t* v_bytes,
                                            size_t* m_bytes) {
  if (!v_bytes || !m_bytes) return WINO_EINVAL;
  const int st = wino_check_shape(n, c, h, w, k);
  if (st != WINO_OK) return st;
  *v_bytes = wino_unfused_v_bytes(n, c, h, w);
  *m_bytes = wino_unfused_m_bytes(n, k, h, w);
  return WINO_OK;
}

extern "C" int wino_conv2d_unfused(const void* x, const void* ucache2, void* y, void* v_ws,
                                   void* m_ws, int n, int c, int h, int w, int k, void* stream) {
  if (!x || !ucache2 || !y || !v_ws || !m_ws) return WINO_EINVAL;
  const int st = wino_check_shape(n, c, h, w, k);
  if (st != WINO_OK) return st;
  if (wino_unfused_prepare() != 0) return WINO_ECUDA;
  wino::KernelParam p = make_param(x, nullptr, y, v_ws, const_cast<void*>(ucache2), m_ws, n, c, h,
                                   w, k);
  return wino_unfused_launch(&p, sm_count(), (cudaStream_t)stream) == 0 ? WINO_OK : WINO_ECUDA;
}

extern "C" int wino_conv2d_fused(const void* x, const void* ucache, void* y, int n, int c, int h,
                                 int w, int k, void* stream) {
  if (!x || !ucache || !y) return WINO_EINVAL;
  const int st = wino_check_shape(n, c, h, w, k);
  if (st != WINO_OK) return st;
  if (wino_fused_prepare() != 0) return WINO_ECUDA;
  wino::KernelParam p = make_param(x, nullptr, y, nullptr, const_cast<void*>(ucache), nullptr, n, c,
                                   h, w, k);
  void* args[] = {&p};
  const cudaError_t e = cudaLaunchKernel(wino_fused_kernel_ptr(), dim3(fused_grid(n, h, w, k)),
                                         dim3(wino_fused_threads()), args,
                                         (size_t)wino_fused_smem_bytes(), (cudaStream_t)stream);
  return e == cudaSuccess ? WINO_OK : WINO_ECUDA;
}

// ------------------------------------------------------ two-stage path ----
// Workspace: the pre-pass output (the transformed tiles V2 when C <= 256,
// else the channel-blocked input XB) then M16, each 256-byte aligned.
extern "C" size_t wino_twostage_workspace_bytes(int n, int c, int h, int w, int k) {
  if (wino_check_shape(n, c, h, w, k) != WINO_OK || !twostage_ok(n, c, h, w)) return 0;
  const size_t xb = (wino_twostage_prepass_bytes(n, c, h, w) + 255) / 256 * 256;
  return xb + wino_twostage_m_bytes(n, h, w, k);
}

// One stage of the two-stage path (0: input pre-pass, 1: tap GEMM, 2: output
// transform) on the workspace layout of wino_conv2d_twostage, for callers
// that time or overlap the stages.
extern "C" int wino_twostage_stage(int stage, const void* x, const void* ucache2, void* workspace,
                                   void* y, int n, int c, int h, int w, int k, void* stream) {
  if (!x || !ucache2 || !y || !workspace || stage < 0 || stage > 2) return WINO_EINVAL;
  if ((reinterpret_cast<uintptr_t>(workspace) & 255) != 0) return WINO_EINVAL;
  const int st = wino_check_shape(n, c, h, w, k);
  if (st != WINO_OK) return st;
  if (!twostage_ok(n, c, h, w)) return WINO_EUNSUPPORTED;
  if (wino_twostage_prepare() != 0) return WINO_ECUDA;
  const size_t xb = (wino_twostage_prepass_bytes(n, c, h, w) + 255) / 256 * 256;
  wino::KernelParam p = make_param(x, nullptr, y, workspace, const_cast<void*>(ucache2),
                                   static_cast<uint8_t*>(workspace) + xb, n, c, h, w, k);
  const cudaStream_t s = (cudaStream_t)stream;
  void* args[] = {&p};
  if (stage == 0) return wino_launch_twostage_prepass(&p, s) == 0 ? WINO_OK : WINO_ECUDA;
  if (stage == 1)
    return cudaLaunchKernel(wino_twostage_gemm_kernel_ptr_for(c),
                            dim3(wino_twostage_gemm_grid(n, c, h, w, k, sm_count())),
                            dim3(wino_twostage_threads_for(c)), args,
                            (size_t)wino_twostage_smem_bytes_for(c), s) == cudaSuccess
               ? WINO_OK
               : WINO_ECUDA;
  unsigned ox, oy;
  wino_twostage_output_grid(n, h, w, k, sm_count(), &ox, &oy);
  return cudaLaunchKernel(wino_twostage_output_kernel_ptr(), dim3(ox, oy), dim3(wino_twostage_output_threads()), args,
                          (size_t)wino_twostage_output_smem_bytes(), s) ==
                 cudaSuccess
             ? WINO_OK
             : WINO_ECUDA;
}

extern "C" int wino_conv2d_twostage(const void* x, const void* ucache2, void* workspace, void* y,
                                    int n, int c, int h, int w, int k, void* stream) {
  for (int stage = 0; stage < 3; ++stage) {
    const int rc = wino_twostage_stage(stage, x, ucache2, workspace, y, n, c, h, w, k, stream);
    if (rc != WINO_OK) return rc;
  }
  return WINO_OK;
}

extern "C" size_t wino_fused_workspace_bytes(int n, int c, int h, int w) {
  if (wino_check_shape(n, c, h, w, 16) != WINO_OK) return 0;
  return wino_xb_bytes(n, c, h, w);
}

extern "C" int wino_input_layout(const void* x, void* workspace, int n, int c, int h, int w,
                                 void* stream) {
  if (!x || !workspace) return WINO_EINVAL;
  if ((reinterpret_cast<uintptr_t>(workspace) & 15) != 0) return WINO_EINVAL;
  const int st = wino_check_shape(n, c, h, w, 16);
  if (st != WINO_OK) return st;
  if (!xb_items_ok(n, c, h, w)) return WINO_EUNSUPPORTED;
  wino::KernelParam p = make_param(x, nullptr, nullptr, workspace, nullptr, nullptr, n, c, h, w, 16);
  return wino_launch_xb_layout(&p, (cudaStream_t)stream) == 0 ? WINO_OK : WINO_ECUDA;
}

// Workspace bytes of the fused entry points: the pre-pass records, and no less
// than the shift kernel's weight operand where that kernel serves the shape.
extern "C" size_t wino_fused_conv_workspace_bytes(int n, int c, int h, int w, int k) {
  if (wino_check_shape(n, c, h, w, k) != WINO_OK) return 0;
  const wino::KernelParam p = make_param(nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, n, c, h, w, k);
  const int cg = wino_shift_fused_cg(&p);
  const size_t xb = wino_xb_bytes(n, c, h, w), wop = cg ? wino_shift_weight_bytes(&p, cg) : 0;
  return xb > wop ? xb : wop;
}

// The fused conv by the shift-reuse implicit GEMM, the filter recovered from
// the U cache into the workspace: a WINO_* code, or -1 when the problem stays
// with the fused Winograd kernel (too small, or no room for the operand).
static int fused_shift(const void* x, const void* ucache, void* workspace, size_t workspace_bytes, void* y,
                       const wino::VariantArgs* va, int n, int c, int h, int w, int k, cudaStream_t s) {
  const wino::KernelParam p = make_param(x, nullptr, y, nullptr, nullptr, nullptr, n, c, h, w, k);
  const int cg = wino_shift_fused_cg(&p);
  if (cg == 0 || wino_shift_weight_bytes(&p, cg) > workspace_bytes) return -1;
  return wino_launch_shift_fused(&p, ucache, workspace, cg, va, sm_count(), s) == 0 ? WINO_OK : WINO_ECUDA;
}

extern "C" int wino_conv2d_fused_ws_sized(const void* x, const void* ucache, void* workspace, size_t workspace_bytes,
                                          void* y, int n, int c, int h, int w, int k, void* stream) {
  if (!x || !ucache || !y || !workspace) return WINO_EINVAL;
  if ((reinterpret_cast<uintptr_t>(workspace) & 15) != 0) return WINO_EINVAL;
  const int st = wino_check_shape(n, c, h, w, k);
  if (st != WINO_OK) return st;
  if (workspace_bytes < wino_xb_bytes(n, c, h, w)) return WINO_ESCRATCH;
  const int rc = fused_shift(x, ucache, workspace, workspace_bytes, y, nullptr, n, c, h, w, k, (cudaStream_t)stream);
  if (rc >= 0) return rc;
  if (!xb_items_ok(n, c, h, w)) return WINO_EUNSUPPORTED;
  if (wino_fused_prepare() != 0) return WINO_ECUDA;
  wino::KernelParam p = make_param(x, nullptr, y, workspace, const_cast<void*>(ucache), nullptr, n,
                                   c, h, w, k);
  if (wino_launch_xb_layout(&p, (cudaStream_t)stream) != 0) return WINO_ECUDA;
  void* args[] = {&p};
  return wino_launch_dependent(wino_fused_kernel_ptr(), dim3(fused_grid(n, h, w, k)), dim3(wino_fused_threads()), args,
                               (size_t)wino_fused_smem_bytes(), (cudaStream_t)stream) == 0
             ? WINO_OK
             : WINO_ECUDA;
}

extern "C" int wino_conv2d_fused_ws(const void* x, const void* ucache, void* workspace, void* y,
                                    int n, int c, int h, int w, int k, void* stream) {
  return wino_conv2d_fused_ws_sized(x, ucache, workspace, wino_fused_workspace_bytes(n, c, h, w), y, n, c, h, w, k,
                                    stream);
}

// ------------------------------------------------ precision variants ----
namespace {

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Workspace of wino_conv2d_variant: XB | U (| U_lo) (| su | amax | sv | inv_sv2).
struct VarLayout {
  size_t xb, u, ulo, su, amax, sv, inv, total;
};

VarLayout var_layout(int variant, int n, int c, int h, int w, int k) {
  VarLayout L{};
  size_t off = 0;
  L.xb = off; off += align256(wino_xb_bytes(n, c, h, w));
  L.u = off; off += align256(wino_ucache_bytes(k, c, variant == WINO_VAR_F8 ? WINO_VAR_F8 : WINO_VAR_F16));
  if (variant == WINO_VAR_F16_HILO) { L.ulo = off; off += align256((size_t)16 * k * c * 2); }
  if (variant == WINO_VAR_F8) {
    L.su = off; off += align256((size_t)16 * k * sizeof(float));
    L.amax = off; off += align256((size_t)c * sizeof(unsigned));
    L.sv = off; off += align256((size_t)c * sizeof(float));
    L.inv = off; off += align256((size_t)(c / 2) * sizeof(uint32_t));
  }
  L.total = off;
  return L;
}

int check_variant(int variant, int n, int c, int h, int w, int k) {
  if (variant < WINO_VAR_F16 || variant > WINO_VAR_F16_HILO) return WINO_EINVAL;
  const int st = wino_check_shape(n, c, h, w, k);
  if (st != WINO_OK) return st;
  if (variant == WINO_VAR_F8 && c % 32 != 0) return WINO_EUNSUPPORTED;
  if (!xb_items_ok(n, c, h, w)) return WINO_EUNSUPPORTED;
  return WINO_OK;
}

}  // namespace

extern "C" size_t wino_variant_workspace_bytes(int variant, int n, int c, int h, int w, int k) {
  if (check_variant(variant, n, c, h, w, k) != WINO_OK) return 0;
  return var_layout(variant, n, c, h, w, k).total;
}

extern "C" int wino_conv2d_variant(int variant, const void* x, const void* weight, void* y,
                                   void* workspace, int n, int c, int h, int w, int k, void* stream) {
  if (!x || !weight || !y || !workspace) return WINO_EINVAL;
  if ((reinterpret_cast<uintptr_t>(workspace) & 255) != 0) return WINO_EINVAL;
  const int st = check_variant(variant, n, c, h, w, k);
  if (st != WINO_OK) return st;
  const cudaStream_t s = (cudaStream_t)stream;
  const VarLayout L = var_layout(variant, n, c, h, w, k);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  wino::KernelParam p = make_param(x, nullptr, y, ws + L.xb, ws + L.u, nullptr, n, c, h, w, k);
  wino::VariantArgs va{nullptr, nullptr, nullptr};
  int rc = 0;
  switch (variant) {
    case WINO_VAR_F16:
      rc = wino_launch_filter_transform(weight, ws + L.u, nullptr, k, c, 0, 0, s);
      break;
    case WINO_VAR_BF16:
      rc = wino_launch_filter_transform(weight, ws + L.u, nullptr, k, c, 1, 0, s);
      break;
    case WINO_VAR_F16_HILO:
      rc = wino_launch_filter_transform(weight, ws + L.u, ws + L.ulo, k, c, 0, 0, s);
      va.u_lo = ws + L.ulo;
      break;
    default: {  // WINO_VAR_F8: input maxima first (pre-pass), then scales, then U8
      unsigned* amax = reinterpret_cast<unsigned*>(ws + L.amax);
      if (cudaMemsetAsync(amax, 0, (size_t)c * sizeof(unsigned), s) != cudaSuccess) return WINO_ECUDA;
      wino::KernelParam pl = p;
      pl.mid_result = amax;
      if (wino_launch_xb_layout_amax(&pl, s) != 0) return WINO_ECUDA;
      float* sv = reinterpret_cast<float*>(ws + L.sv);
      uint32_t* inv = reinterpret_cast<uint32_t*>(ws + L.inv);
      float* su = reinterpret_cast<float*>(ws + L.su);
      if (wino_launch_xb_f8_scales(amax, sv, inv, c, s) != 0) return WINO_ECUDA;
      rc = wino_launch_filter_transform_f8(weight, sv, ws + L.u, su, k, c, s);
      va.su = su;
      va.inv_sv2 = inv;
      break;
    }
  }
  if (rc != 0) return WINO_ECUDA;
  if (variant != WINO_VAR_F8 && wino_launch_xb_layout_beside(&p, s) != 0) return WINO_ECUDA;
  return wino_fused_launch_variant(variant, &p, &va, 0, fused_grid(n, h, w, k), s) == 0 ? WINO_OK
                                                                                         : WINO_ECUDA;
}

// Fused conv with the epilogue of the next ResNet step folded in:
// y = relu?(conv(x) + bias[k] + residual).
extern "C" int wino_conv2d_fused_epilogue(const void* x, const void* ucache, void* workspace, void* y,
                                          const float* bias, const void* residual, int relu, int n, int c,
                                          int h, int w, int k, void* stream) {
  return wino_conv2d_fused_epilogue_sized(x, ucache, workspace, wino_fused_workspace_bytes(n, c, h, w), y, bias, residual,
                                          relu, n, c, h, w, k, stream);
}

extern "C" int wino_conv2d_fused_epilogue_sized(const void* x, const void* ucache, void* workspace,
                                                size_t workspace_bytes, void* y, const float* bias,
                                                const void* residual, int relu, int n, int c, int h, int w, int k,
                                                void* stream) {
  if (!x || !ucache || !y || !workspace) return WINO_EINVAL;
  if ((reinterpret_cast<uintptr_t>(workspace) & 15) != 0) return WINO_EINVAL;
  if (residual && (reinterpret_cast<uintptr_t>(residual) & 3) != 0) return WINO_EINVAL;
  const int st = wino_check_shape(n, c, h, w, k);
  if (st != WINO_OK) return st;
  if (workspace_bytes < wino_xb_bytes(n, c, h, w)) return WINO_ESCRATCH;
  const cudaStream_t s = (cudaStream_t)stream;
  wino::VariantArgs va{};
  va.bias = bias;
  va.residual = residual;
  va.relu = relu ? 1 : 0;
  const int rc = fused_shift(x, ucache, workspace, workspace_bytes, y, &va, n, c, h, w, k, s);
  if (rc >= 0) return rc;
  if (!xb_items_ok(n, c, h, w)) return WINO_EUNSUPPORTED;
  wino::KernelParam p = make_param(x, nullptr, y, workspace, const_cast<void*>(ucache), nullptr, n, c, h,
                                   w, k);
  if (wino_launch_xb_layout(&p, s) != 0) return WINO_ECUDA;
  return wino_fused_launch_variant(WINO_VAR_F16, &p, &va, 0, fused_grid(n, h, w, k), s) == 0 ? WINO_OK
                                                                                          : WINO_ECUDA;
}

// Direct convolution of any filter size, stride and padding (the shapes the
// Winograd path does not take).
extern "C" int wino_conv2d_direct(const void* x, const void* weight, void* y, int n, int c, int h,
                                  int w, int k, int r, int s, int u, int v, int p, int q, void* stream) {
  if (!x || !weight || !y) return WINO_EINVAL;
  int oh = 0, ow = 0;
  const int st = check_general(n, c, h, w, k, r, s, u, v, p, q, &oh, &ow);
  if (st != WINO_OK) return st;
  wino::KernelParam pk = make_param(x, weight, y, nullptr, nullptr, nullptr, n, c, h, w, k);
  pk.r = (short)r; pk.s = (short)s; pk.u = (short)u; pk.v = (short)v; pk.p = (short)p; pk.q = (short)q;
  pk.Oh = (short)oh; pk.Ow = (short)ow;
  return wino_launch_direct(&pk, (cudaStream_t)stream) == 0 ? WINO_OK : WINO_ECUDA;
}

extern "C" int wino_igemm_weight_transform(const void* weight, void* wprep, int k, int c, int r, int s,
                                           void* stream) {
  if (!weight || !wprep) return WINO_EINVAL;
  if ((reinterpret_cast<uintptr_t>(wprep) & 15) != 0) return WINO_EINVAL;
  int oh = 0, ow = 0;
  const int st = check_general(1, c, r, s, k, r, s, 1, 1, 0, 0, &oh, &ow);
  if (st != WINO_OK) return st;
  wino::KernelParam pk = make_param(nullptr, weight, nullptr, nullptr, wprep, nullptr, 1, c, r, s, k);
  pk.r = (short)r; pk.s = (short)s;
  void* args[] = {&pk};
  return cudaLaunchKernel(wino_igemm_weight_kernel_ptr(), dim3(wino_igemm_weight_grid(c, k, r, s)), dim3(256),
                          args, 0, (cudaStream_t)stream) == cudaSuccess
             ? WINO_OK
             : WINO_ECUDA;
}

extern "C" int wino_conv2d_igemm(const void* x, const void* wprep, void* y, int n, int c, int h, int w, int k,
                                 int r, int s, int u, int v, int p, int q, void* stream) {
  if (!x || !wprep || !y) return WINO_EINVAL;
  if ((reinterpret_cast<uintptr_t>(wprep) & 15) != 0) return WINO_EINVAL;
  int oh = 0, ow = 0;
  const int st = check_general(n, c, h, w, k, r, s, u, v, p, q, &oh, &ow);
  if (st != WINO_OK) return st;
  if (!wino_igemm_shape_ok(n, c, h, w, k, oh, ow)) return WINO_EUNSUPPORTED;
  if (wino_igemm_prepare() != 0) return WINO_ECUDA;
  wino::KernelParam pk = make_param(x, nullptr, y, nullptr, const_cast<void*>(wprep), nullptr, n, c, h, w, k);
  pk.r = (short)r; pk.s = (short)s; pk.u = (short)u; pk.v = (short)v; pk.p = (short)p; pk.q = (short)q;
  pk.Oh = (short)oh; pk.Ow = (short)ow;
  int mode = wino_igemm_mode(x, k, h, w, r, s, u, v, p, q);
  if (mode == kIgemmModeTma) {
    // this call's tensor map goes to wprep's map slot, in stream order
    // (a pageable-source copy returns once the 128 bytes are staged)
    alignas(64) unsigned char map[128];
    void* slot = static_cast<uint8_t*>(const_cast<void*>(wprep)) + wino_igemm_map_offset(c, k, r, s);
    if ((reinterpret_cast<uintptr_t>(slot) & 63) == 0 && wino_igemm_encode_map(map, x, n, c, h * w) == 0 &&
        cudaMemcpyAsync(slot, map, sizeof(map), cudaMemcpyHostToDevice, (cudaStream_t)stream) == cudaSuccess)
      pk.transform_pin = slot;
    else
      mode = kIgemmModeFlat;
  }
  void* args[] = {&pk};
  return cudaLaunchKernel(wino_igemm_kernel_ptr(k, mode),
                          dim3(wino_igemm_grid(n, k, oh, ow, sm_count())),
                          dim3(wino_igemm_threads()), args, (size_t)wino_igemm_smem_bytes(),
                          (cudaStream_t)stream) == cudaSuccess
             ? WINO_OK
             : WINO_ECUDA;
}

// Launch the four slots of a filled kernelInfo_t in order on one stream, each
// with args[0] = param, exactly as the reference harness does
// (reference src/main.cpp:105-108, 121-124, hipExtLaunchKernel).
extern "C" int wino_launch_kernelinfo(const void* kiv, void* param, void* stream) {
  const kernelInfo_t* ki = static_cast<const kernelInfo_t*>(kiv);
  if (!ki || !param) return WINO_EINVAL;
  const unsigned* slots[4] = {&ki->blockx1, &ki->blockx2, &ki->blockx3, &ki->blockx4};
  void* const fns[4] = {ki->kernelPtr1, ki->kernelPtr2, ki->kernelPtr3, ki->kernelPtr4};
  // slots whose kernel has nothing to do are not launched: the empty kernel,
  // and the two-stage GEMM and output transform without an M
  const bool no_m = static_cast<const wino::KernelParam*>(param)->mid_result == nullptr;
  const bool shift = fns[0] == wino_shift_weight_kernel_ptr(1) || fns[0] == wino_shift_weight_kernel_ptr(2);
  for (int i = 0; i < 4; ++i) {
    if (fns[i] == wino_noop_kernel_ptr()) continue;
    if (no_m && (fns[i] == wino_twostage_resv_kernel_ptr() || fns[i] == wino_twostage_output_kernel_ptr())) continue;
    const unsigned* b = slots[i];
    const dim3 grid(b[0], b[1], b[2]), block(b[3], b[4], b[5]);
    // the shift kernel starts beside the weight kernel launched right before
    // it and waits for the weights itself; the fused route's pre-pass needs
    // nothing of its filter transform, and the fused kernel waits for both
    const bool xb = fns[1] == wino_xb_layout_kernel_ptr() && fns[0] == wino_dropin_filter_kernel_ptr();
    const bool dependent =
        (shift && (i == 1 || i == 2)) ||
        (xb && (i == 1 || (i == 2 && fns[2] == wino_fused_kernel_ptr())));
    const int e = dependent ? wino_launch_dependent(fns[i], grid, block, (void**)&param, (size_t)b[6], (cudaStream_t)stream)
                            : (int)cudaLaunchKernel(fns[i], grid, block, (void**)&param, (size_t)b[6],
                                                    (cudaStream_t)stream);
    if (e != (int)cudaSuccess) return WINO_ECUDA;
  }
  return WINO_OK;
}

// One drop-in call of the harness: getkernelInfo on a parameter block of its
// own, then the four slots.  WINO_* of getkernelInfo, or 256 more of the launch.
extern "C" int wino_dropin_conv2d(void* in, void* weight, void* out, void* transform_pin, void* transform_filter,
                                  void* mid_result, unsigned n, unsigned c, unsigned h, unsigned w, unsigned k,
                                  unsigned r, unsigned s, unsigned stride, unsigned pad, void* stream) {
  problem_t pr{};
  pr.in = static_cast<decltype(pr.in)>(in);
  pr.weight = static_cast<decltype(pr.weight)>(weight);
  pr.out = static_cast<decltype(pr.out)>(out);
  pr.transform_pin = static_cast<decltype(pr.transform_pin)>(transform_pin);
  pr.transform_filter = static_cast<decltype(pr.transform_filter)>(transform_filter);
  pr.mid_result = static_cast<decltype(pr.mid_result)>(mid_result);
  pr.n = n; pr.c = c; pr.h = h; pr.w = w; pr.k = k; pr.r = r; pr.s = s;
  pr.u = pr.v = stride;
  pr.p = pr.q = pad;
  kernelInfo_t ki;
  mykernelParamType param{};
  int rc = getkernelInfo(&pr, &ki, &param);
  if (rc != WINO_OK) return rc;
  rc = wino_launch_kernelinfo(&ki, &param, stream);
  return rc == WINO_OK ? WINO_OK : 256 + rc;
}

extern "C" int wino_error_read_clear(uint32_t* code) {
  if (!code) return WINO_EINVAL;
  const uint32_t a = wino_fused_error_read_clear();
  const uint32_t b = wino_unfused_error_read_clear();
  const uint32_t c = wino_twostage_error_read_clear();
  const uint32_t d = wino_igemm_error_read_clear();
  const uint32_t e = wino_shift_error_read_clear();
  *code = a ? a : (b ? b : (c ? c : (d ? d : e)));
  return WINO_OK;
}
