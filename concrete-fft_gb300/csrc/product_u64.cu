// product_u64.cu -- fused negacyclic u64 polynomial product on unordered::Plan.
//
// One CTA computes one product at a time (grid-stride over the batch): it
// reads N u64 coefficients and N/2 resident Fourier coefficients, writes N u64
// results, and keeps every intermediate in shared memory, so a product costs
// exactly 48 KiB of HBM traffic at N = 2048 (24 bytes per coefficient).
//
// Pipeline (the way the reference's caller uses unordered::Plan; the crate
// itself has no product code):
//   z_j = tau^j * (a_j + i a_{j+N/2}),  tau = exp(i pi / N),  a read as i64
//   Z = fwd(z)                      unordered forward, permuted order
//   P_k = Bhat_k * Z_k              Bhat = fwd of the twisted operand, resident
//   p = inv(P)                      unordered inverse, standard order
//   t_j = (conj(tau^j) / (N/2)) * p_j
//   c_j = floor(Re t_j + 1/2) mod 2^64,  c_{j+N/2} = floor(Im t_j + 1/2) mod 2^64
// Every complex product is the reference's FMA form (cmul); conversions are
// exact integer-pipe routines, so the result is bit-identical to the oracle's
// CPU restatement of the same pipeline.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "cfft_internal.h"
#include "runtime.h"
#include "c64_kernels.cuh"
#include "split_product.cuh"
#include "tune_cache.h"

using namespace cfft;

struct cfft_u64_product_plan {
  WorkspaceUser workspace;
  size_t N = 0, n = 0, base_n = 0;
  cfft_unordered_plan* fft = nullptr;  // the plan's transform, for the unfused entry points
  int base_algo = 0;
  LevelDesc lv{};
  DevLevels dlv{};
  double2 *d_w = nullptr, *d_winv = nullptr, *d_tw = nullptr, *d_itw = nullptr;
  int int_adds = kIntAddsAuto;  // cfft_u64_product_set_int_adds
  int cluster = 0;  // CTAs per product: 0 automatic, 1 one CTA, 2/4/8 a cluster of that size
  bool graph_workspace = false;  // captured calls may allocate where kernels without a workspace serve
};

namespace cfft {
// The product pipeline's elementwise steps as separate kernels (the unfused path).
__global__ void fold_twist_kernel(const uint64_t* __restrict__ a, double2* __restrict__ z, long total, int log2n,
                                  const double2* __restrict__ tw) {
  grid_dependency_wait();
  const long n = 1L << log2n;
  for (long g = (long)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (long)gridDim.x * blockDim.x) {
    const long p = g >> log2n, j = g & (n - 1);
    const uint64_t* ap = a + (p << (log2n + 1));
    const c64 v{i64_to_f64_rne((int64_t)ap[j]), i64_to_f64_rne((int64_t)ap[j + n])};
    st(z + g, cmul(ldg(tw + j), v));
  }
}
__global__ void pointwise_kernel(const double2* __restrict__ bhat, long bhat_stride, double2* __restrict__ z,
                                 long total, int log2n) {
  grid_dependency_wait();
  const long n = 1L << log2n;
  for (long g = (long)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (long)gridDim.x * blockDim.x) {
    const long p = g >> log2n, k = g & (n - 1);
    st(z + g, cmul(ldg(bhat + p * bhat_stride + k), ld(z + g)));
  }
}
// acc[g] = sum over t of bhat[g, t] * z[g, t] (terms back to back per group),
// the first product assigned and the others added in term order, as the fused
// sum kernels do.
__global__ void fourier_sum_kernel(const double2* __restrict__ bhat, const double2* __restrict__ z,
                                   double2* __restrict__ acc, int terms, long total, int log2n) {
  grid_dependency_wait();
  const long n = 1L << log2n;
  for (long g = (long)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (long)gridDim.x * blockDim.x) {
    const long grp = g >> log2n, k = g & (n - 1);
    const long base = ((grp * terms) << log2n) + k;
    c64 s = cmul(ldg(bhat + base), ld(z + base));
    for (int t = 1; t < terms; ++t) {
      const long o = base + ((long)t << log2n);
      s = cadd(s, cmul(ldg(bhat + o), ld(z + o)));
    }
    st(acc + g, s);
  }
}
// digits of the monomial X^degree mod (X^N + 1): one coefficient +-1 (X^N = -1)
__global__ void monomial_digits_kernel(int64_t* __restrict__ b, long N, unsigned long long degree) {
  grid_dependency_wait();
  const long pos = (long)(degree % (unsigned long long)N);
  const int64_t sign = ((degree / (unsigned long long)N) & 1) ? -1 : 1;
  for (long j = (long)blockIdx.x * blockDim.x + threadIdx.x; j < N; j += (long)gridDim.x * blockDim.x)
    b[j] = j == pos ? sign : 0;
}
__global__ void untwist_round_kernel(const double2* __restrict__ z, uint64_t* __restrict__ out, long total, int log2n,
                                     const double2* __restrict__ itw) {
  grid_dependency_wait();
  const long n = 1L << log2n;
  for (long g = (long)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (long)gridDim.x * blockDim.x) {
    const long p = g >> log2n, j = g & (n - 1);
    const c64 t = cmul(ldg(itw + j), ld(z + g));
    uint64_t* op = out + (p << (log2n + 1));
    op[j] = round_half_up_mod64(t.re);
    op[j + n] = round_half_up_mod64(t.im);
  }
}
}  // namespace cfft

namespace {

int ew_grid(long total) { return (int)std::max<long>(1, std::min<long>((total + 255) / 256, (long)sm_count() * 16)); }

void free_u64(cfft_u64_product_plan* p) {
  if (p->fft) cfft_unordered_plan_destroy(p->fft);
  if (p->d_w) cudaFree(p->d_w);
  if (p->d_winv) cudaFree(p->d_winv);
  if (p->d_tw) cudaFree(p->d_tw);
  if (p->d_itw) cudaFree(p->d_itw);
}

DevLevels dev_levels(const LevelDesc& l) {
  DevLevels d;
  std::memset(&d, 0, sizeof(d));
  d.nlevels = l.nlevels;
  for (int i = 0; i <= kMaxLevels; ++i) {
    d.log2n[i] = l.log2n[i];
    d.w_off[i] = l.w_off[i];
  }
  for (int i = 0; i < kMaxLevels; ++i) {
    d.log2r[i] = l.log2r[i];
    d.winv_off[i] = l.winv_off[i];
  }
  return d;
}

// One CTA per product (the block scheduler hands the next product to the
// first SM with room, which balances the SMs to within one product) up to a
// large count; beyond it a grid of the resident CTAs strides over the batch.
int grid_for(const void* kernel, int threads, size_t smem, long count) {
  if (count <= (1L << 20)) return (int)std::max<long>(1, count);
  return (int)((long)sm_count() * max_blocks_per_sm(kernel, threads, smem));
}

// Sums of products that no cluster holds (N > 65536) or too few to fill the SMs, unfused: fold and twist
// every term, the plan's forward transforms, the Fourier-domain sum per group,
// one inverse per group, untwist and round.  Groups run in chunks whose
// workspace (terms + 1 transforms per group) stays within what the pool keeps.
cfft_status product_sum_unfused(const cfft_u64_product_plan* plan, const uint64_t* a, const double* bhat,
                                size_t terms, uint64_t* out, size_t count, cudaStream_t s) {
  const size_t n = plan->n, per_group = (terms + 1) * n * sizeof(double2);
  const size_t chunk = std::min(count, std::max<size_t>(1, kWorkspaceKeep / per_group));
  void* ws = nullptr;
  if (plan->workspace.alloc((void**)&ws, chunk * per_group, s) != cudaSuccess)
    return fail(CFFT_ERR_OUT_OF_MEMORY, "product sum workspace");
  double2* z = (double2*)ws;
  double2* acc = z + chunk * terms * n;
  cfft_status st = CFFT_OK;
  for (size_t g0 = 0; g0 < count && st == CFFT_OK; g0 += chunk) {
    const size_t g = std::min(chunk, count - g0);
    st = cfft_u64_fold_twist(plan, a + g0 * terms * plan->N, (double*)z, g * terms, s);
    if (st == CFFT_OK) st = cfft_unordered_fwd(plan->fft, (double*)z, g * terms, s);
    if (st == CFFT_OK) {
      const long total = (long)(g * n);
      st = launch_dependent(fourier_sum_kernel, ew_grid(total), 256, 0, s, (const double2*)bhat + g0 * terms * n, z,
                            acc, (int)terms, total, ilog2(n)) == cudaSuccess
               ? CFFT_OK
               : fail(CFFT_ERR_CUDA, "fourier_sum_kernel launch");
    }
    if (st == CFFT_OK) st = cfft_unordered_inv(plan->fft, (double*)acc, g, s);
    if (st == CFFT_OK) st = cfft_u64_untwist_round(plan, (const double*)acc, out + g0 * plan->N, g, s);
  }
  cudaFreeAsync(ws, s);
  return st;
}

// Whether a launch of `ctas` one-CTA kernels of `points` points each has about one busy
// warp per SM sub-partition in a pass of the base, counting the CTAs that shared memory
// lets run at once (300 operands of 4096 points on Dit2, one per SM: 159 us on the integer
// pipes, 150).  A radix-16 pass of less than a warp of butterflies counts as such: what its
// idle lanes leave of an integer addition costs more than the FP64 one (1500 products of
// N = 256 on Dit16: 78.6 us, 66.8; of N = 1024, a full warp: 110 and 121).
bool few_warps(const cfft_u64_product_plan* plan, long ctas, size_t points) {
  if (plan->int_adds != kIntAddsAuto) return plan->int_adds == 0;
  const size_t radix = (size_t)algo_radix(plan->base_algo), pass = std::min<size_t>(kProdThreads, points / radix);
  if (radix == 16 && pass < 32) return true;
  const long per_sm = std::max<long>(1, (long)((size_t(227) << 10) / (2 * points * sizeof(double2))));
  return half_butterflies(std::min(ctas, (long)sm_count() * per_sm), pass);
}

cfft_status launch_product(const cfft_u64_product_plan* plan, const uint64_t* a, const double* bhat,
                           size_t bhat_stride, uint64_t* out, size_t count, cudaStream_t stream) {
  // N <= 128: 512 points per CTA iteration (one product of n = 32 would give a radix-4
  // pass 8 butterflies, a quarter warp: 122 vs 375 M products/s possible at N = 64)
  int log2p = 0;
  while ((plan->n << log2p) < 512 && plan->n <= 64) ++log2p;
  // likewise a radix whose pass over one product is less than a warp, while two CTAs per SM
  // remain (1500 products of N = 256: 74 us on Dif16, 67 on Dit16 with one per CTA)
  while ((plan->n << log2p) < 32 * (size_t)algo_radix(plan->base_algo) && (long)(count >> (log2p + 1)) >= 2L * sm_count())
    ++log2p;
  const void* fn = u64_product_kernel_ptr(
      plan->base_algo, few_warps(plan, ((long)count + (1L << log2p) - 1) >> log2p, plan->n << log2p));
  const size_t smem = 2 * (plan->n << log2p) * sizeof(double2);
  const int grid = grid_for(fn, kProdThreads, smem, ((long)count + (1L << log2p) - 1) >> log2p);
  DevLevels L = plan->dlv;
  long stride = (long)bhat_stride, cnt = (long)count;
  const double2* bh = (const double2*)bhat;
  void* args[] = {(void*)&a, (void*)&bh, &stride, (void*)&out, &cnt, &L, (void*)&plan->d_w, (void*)&plan->d_winv,
                  (void*)&plan->d_tw, (void*)&plan->d_itw, &log2p};
  return launch_kernel(fn, grid, kProdThreads, args, smem, stream);
}

// CTAs per product as a log2 (0: one CTA).  A product whose N/2-point
// transform exceeds one CTA's shared memory (N > 8192) always runs on a
// cluster, S = 2^ls with S <= level 0's radix, S <= 8 and n/S <= 4096 points
// per CTA (so N <= 65536); its default S gives each CTA 1024 points (the base
// size) where possible.  Smaller products use a cluster when the batch is too
// small to give every SM a product, or as the plan forces.
int product_split_log2(const cfft_u64_product_plan* p, size_t count, bool* ok) {
  *ok = true;
  const int log2n = ilog2(p->n);
  const int max_ls = p->lv.nlevels >= 1 ? std::min(3, p->lv.log2r[0]) : 0;
  const int min_ls = std::max(0, log2n - kSmemLog2Max);
  if (min_ls > max_ls) {
    *ok = false;
    return 0;
  }
  if (p->cluster >= 2) return std::max(min_ls, std::min(max_ls, ilog2((size_t)p->cluster)));
  if (min_ls > 0) return std::max(min_ls, std::min(max_ls, log2n - 10));
  if (p->cluster == 1 || max_ls == 0) return 0;
  // N = 8192: two CTAs of 2048 points (1.43 M products/s) beat one CTA of 4096,
  // which leaves one CTA per SM (1.12 M/s, 4864 products per launch)
  int ls = std::min(max_ls, std::max(0, log2n - kBlockLog2Auto));
  while (ls < max_ls && (count << ls) < (size_t)sm_count()) ++ls;
  return ls;
}

cfft_status launch_split_product(const cfft_u64_product_plan* plan, int ls, const uint64_t* a, const double* bhat,
                                 size_t bhat_stride, uint64_t* out, size_t count, cudaStream_t stream,
                                 const cfft_product_item* items = nullptr, int terms = 1) {
  const size_t part = plan->n >> ls;
  const bool big = part > 2048;  // 4096 points per CTA: one CTA per SM, 512 threads
  const size_t smem = 2 * (plan->n >> ls) * sizeof(double2);
  if ((count << ls) > 0x7fffffffUL) return fail(CFFT_ERR_INVALID_SIZE, "batch too large");
  DevLevels L = plan->dlv;
  long stride = (long)bhat_stride;
  const double2* bh = (const double2*)bhat;
  // 128 threads (several CTAs per SM) for parts up to 1024 points, 256 for 2048
  // (shared memory allows 3 CTAs per SM), 512 for 4096 (one CTA per SM)
  const int threads = part <= 1024 ? 128 : (part <= 2048 ? kSplitProdThreads : kSplitProdThreadsBig);
  const int grid = (int)(count << ls);
  const bool few =
      half_butterflies(grid, std::min<size_t>((size_t)threads, part / (size_t)algo_radix(plan->base_algo)));
  const void* fn = u64_product_split_ptr(plan->base_algo, ls, big, fp64_additions(plan->int_adds, few));
  void* args[] = {(void*)&a, (void*)&bh, &stride, (void*)&out, &terms, (void*)&items, &L, (void*)&plan->d_w,
                  (void*)&plan->d_winv, (void*)&plan->d_tw, (void*)&plan->d_itw};
  return launch_kernel_cluster(fn, grid, threads, 1 << ls, args, spread_smem(fn, grid, threads, 1 << ls, smem),
                               stream);
}

// CTAs per product as a log2 for plans without an outer level (n = base_n;
// u64_product_split0_kernel): S <= the base radix R and S <= 8, with at least
// 64 points per CTA.  `fast` also keeps at least 32 butterflies in each of a
// class's passes (64 for DIT, one thread per butterfly): with fewer, a lone
// product measured slower than on fewer CTAs (N = 2048, Dif8: 23.4 us on 8
// CTAs, 16.0 on 4; Dif16: 36.8 on 8, 25.0 on 2; Dit16 on 2: 45.9 against
// 39.8 for the five launches).  0 when the plan has levels or no S >= 2 fits.
int split0_log2(const cfft_u64_product_plan* p, bool fast = true) {
  if (p->lv.nlevels != 0) return 0;
  const int lr = p->base_algo / 2 + 1;
  const int log2n = ilog2(p->n);
  const int min_lb = !fast ? 0 : ((p->base_algo & 1) ? 6 : 5);
  int ls = std::min(3, lr);
  while (ls > 0 && (log2n - ls < 6 || log2n - ls - lr < min_lb)) --ls;
  return ls;
}

// Threads per CTA of the class-split product kernels (`ctas` CTAs of `part` points), and
// which instance.  DIF: two threads per butterfly of a pass (half butterflies) in small
// launches, DIT: one; at least a thread per two points for the elementwise steps (radix 16
// has few butterflies per pass).  Larger DIF launches take one thread per butterfly, and so
// does a part too large for two threads each.  Sums in one launch (kSum) always have a
// thread per two points, for their accumulators.
int split_product_threads(const cfft_u64_product_plan* plan, size_t part, long ctas, int phase, bool* few) {
  const int algo = plan->base_algo;
  const size_t radix = size_t(2) << (algo / 2);
  const size_t full = part / radix;
  const bool one = (algo & 1) || radix == 16 || phase == kSum, half = half_butterflies(ctas, full);
  *few = one || fp64_additions(plan->int_adds, half && 2 * full <= 256);
  const size_t want = one || half ? std::max(((algo & 1) ? 1 : 2) * full, part / 2) : full;
  return (int)std::min<size_t>(256, std::max<size_t>(32, want));
}

// phase kForward: `count` terms into ws; kInverse: `count` outputs of `terms` terms each
// from ws; kSum: `count` sums of `terms` terms without ws; kWhole: `count` products.
cfft_status launch_split0_product(const cfft_u64_product_plan* plan, int ls, const uint64_t* a, const double* bhat,
                                  size_t bhat_stride, uint64_t* out, size_t count, cudaStream_t stream,
                                  const cfft_product_item* items = nullptr, int phase = kWhole, int terms = 1,
                                  double2* ws = nullptr) {
  const int algo = plan->base_algo;
  const size_t part = plan->n >> ls;
  bool few = false;
  const int threads = split_product_threads(plan, part, (long)(count << ls), phase, &few);
  const void* fn = u64_product_split0_ptr(algo, ls, phase, few);
  if (!fn) return fail(CFFT_ERR_INVALID_SIZE, "no cluster product kernel for this base and cluster size");
  if ((count << ls) > 0x7fffffffUL) return fail(CFFT_ERR_INVALID_SIZE, "batch too large");
  const size_t smem = 3 * part * sizeof(double2);
  const int grid = (int)(count << ls);
  DevLevels L = plan->dlv;
  long stride = (long)bhat_stride;
  const double2* bh = (const double2*)bhat;
  void* args[] = {(void*)&a, (void*)&bh, &stride, (void*)&out, &terms, (void*)&items, &L, (void*)&plan->d_w,
                  (void*)&plan->d_winv, (void*)&plan->d_tw, (void*)&plan->d_itw, (void*)&ws};
  // a few products: every CTA on an SM of its own
  return launch_kernel_cluster(fn, grid, threads, 1 << ls, args, spread_smem(fn, grid, threads, 1 << ls, smem),
                               stream, phase == kForward || phase == kInverse);
}

// Launch shape of u64_product_split2_kernel with 2^ls1 classes: threads per CTA
// and shared memory (three buffers of the CTA's part of the base).
void split2_launch_shape(const cfft_u64_product_plan* p, int ls1, long ctas, int phase, int* threads, size_t* smem,
                         bool* few) {
  const size_t part = p->base_n >> ls1;
  *threads = split_product_threads(p, part, ctas, phase, few);
  *smem = 3 * part * sizeof(double2);
}

// The shape of u64_product_split2_kernel for a plan, as log2s: one outer level
// of radix R0 = 2^ls0 <= 8 over a DIF base of m points and S1 = 2^ls1 >= 2
// classes of the base, with S1 <= R, at least 64 points per CTA and at least 32
// butterflies in each of a class's passes (as split0_log2).  R0 * S1 is at most
// 16 where the `count` products' (or sums') 16-CTA clusters (a non-portable size)
// are resident at once with one CTA per SM; else at most 8.  Not for a radix-2 base under a radix-4 level: N = 4096
// on Dif2/512 measured slower than the five launches from 16 products (29.7
// against 24.9 us).  false when the plan has another shape.
bool split2_shape(const cfft_u64_product_plan* p, size_t count, int* ls0, int* ls1, int phase = kWhole,
                  bool allow16 = true) {
  if (p->lv.nlevels != 1 || (p->base_algo & 1) || p->lv.log2r[0] > 3) return false;
  const int lr = p->base_algo / 2 + 1;
  if (lr == 1 && p->lv.log2r[0] > 1) return false;
  const int log2m = ilog2(p->base_n);
  const int l0 = p->lv.log2r[0];
  for (int max_ls = allow16 && (count << 4) <= (size_t)sm_count() * (phase == kForward ? 2 : 1) ? 4 : 3; max_ls >= 3; --max_ls) {
    int l1 = std::min(max_ls - l0, lr);
    while (l1 > 0 && (log2m - l1 < 6 || log2m - l1 - lr < 5)) --l1;
    if (l1 < 1) return false;
    int threads = 0;
    size_t smem = 0;
    bool small = false;
    split2_launch_shape(p, l1, (long)(count << (l0 + l1)), phase, &threads, &smem, &small);
    const void* fn = u64_product_split2_ptr(p->base_algo, l0, l1, phase, small);
    if (!fn) continue;
    if (l0 + l1 > 3) {  // every product's 16-CTA cluster resident at once, one CTA per SM
      // the terms of a sum may take two rounds of clusters: two outputs of 4 terms, N = 16384
      const long rounds = phase == kForward ? 2 : 1;
      if ((long)count > rounds * spread_clusters(fn, threads, 16)) continue;
    }
    *ls0 = l0;
    *ls1 = l1;
    return true;
  }
  return false;
}

cfft_status launch_split2_product(const cfft_u64_product_plan* plan, int ls0, int ls1, const uint64_t* a,
                                  const double* bhat, size_t bhat_stride, uint64_t* out, size_t count,
                                  cudaStream_t stream, const cfft_product_item* items = nullptr, int phase = kWhole,
                                  int terms = 1, double2* ws = nullptr) {
  const int ls = ls0 + ls1;
  int threads = 0;
  size_t smem = 0;
  bool few = false;
  split2_launch_shape(plan, ls1, (long)(count << ls), phase, &threads, &smem, &few);
  const void* fn = u64_product_split2_ptr(plan->base_algo, ls0, ls1, phase, few);
  if (!fn) return fail(CFFT_ERR_INVALID_SIZE, "no one-level cluster product kernel for this shape");
  if ((count << ls) > 0x7fffffffUL) return fail(CFFT_ERR_INVALID_SIZE, "batch too large");
  const int grid = (int)(count << ls);
  DevLevels L = plan->dlv;
  long stride = (long)bhat_stride;
  const double2* bh = (const double2*)bhat;
  void* args[] = {(void*)&a, (void*)&bh, &stride, (void*)&out, &terms, (void*)&items, &L, (void*)&plan->d_w,
                  (void*)&plan->d_winv, (void*)&plan->d_tw, (void*)&plan->d_itw, (void*)&ws};
  return launch_kernel_cluster(fn, grid, threads, 1 << ls, args, spread_smem(fn, grid, threads, 1 << ls, smem),
                               stream, phase == kForward || phase == kInverse);
}

// Whether a call that has another route may take a workspace: not into a graph that the
// caller has not allowed it in (stream_capturing).
bool may_allocate(const cfft_u64_product_plan* plan, cudaStream_t s) {
  return plan->graph_workspace || !stream_capturing(s);
}

// Where the products of a call run.
struct ProductRoute {
  enum Kind {
    kSplit0,  // u64_product_split0_kernel on 2^ls0 CTAs each
    kSplit2,  // u64_product_split2_kernel on 2^ls0 slices x 2^ls1 classes
    kFive,    // five launches on a workspace
    kPlain    // u64_product_split_kernel on 2^ls0 CTAs each, or one CTA (ls0 = 0)
  } kind;
  int ls0 = 0, ls1 = 0;
  bool spare = false;  // of kFive: kPlain with ls0 serves as well
};
ProductRoute product_route(const cfft_u64_product_plan* plan, size_t count) {
  bool ok = true;
  const int ls = product_split_log2(plan, count, &ok);
  // The five-launch path on a workspace from the stream-ordered allocator: N > 65536
  // (no cluster holds it), and N >= 32768 at every batch, where it measured faster
  // than one cluster per product (Dif8/512, CUDA events: one product 30.5 vs 74.4 us
  // at 32768, 35.8 vs 142 at 65536; 38 products 134 vs 212 and 274 vs 423; large
  // batches 304 vs 280 k products/s at 32768, 129 vs 102 k at 65536)
  const bool many = (long)count >= (long)sm_count() / 2 && plan->cluster == 0;
  // A few products whose transform has no outer level (n = base_n): one cluster per
  // product on the base's residue classes (u64_product_split0_kernel), as does a plan
  // forced to a cluster size.  Device time per call at N = 2048, Dif4, 4
  // CTAs: 11.7 us for one product (one CTA: 32.2, the five launches: 13.7), 16.7 for
  // 38 (one CTA: 34.9, five launches: 19.4)
  if (plan->cluster >= 2 && split0_log2(plan, false) >= 1)
    return {ProductRoute::kSplit0, std::min(split0_log2(plan, false), ilog2((size_t)plan->cluster))};
  // Base radix >= 4: up to one product per SM (N = 2048, 152 products: 25.5 us on Dif4
  // clusters, 33.9 on one CTA each; Dif8 28.9 against 35.0); radix 2 lost there (Dif2,
  // N = 1024, 152 products: 24.9 against 20.5 us) and keeps the SMs/2 limit.
  const long split0_max = (plan->base_algo >= 2) ? (long)sm_count() : (long)sm_count() / 2 - 1;
  if (plan->cluster == 0 && plan->N >= 512 && (long)count <= split0_max && split0_log2(plan) >= 1)
    return {ProductRoute::kSplit0, split0_log2(plan)};
  // Likewise a plan with one outer level of radix 2, 4 or 8 over a DIF base: level 0's
  // slices times classes of the base (u64_product_split2_kernel).  One product, Dif4
  // on 1024 points: 13.7 us at N = 4096 (five launches 32.1), 20.9 at 8192 (34.2);
  // 38 products: 23.3 (33.5) and 44.7 (58.8)
  int ls0 = 0, ls1 = 0;
  if (plan->cluster == 0 && !many && split2_shape(plan, count, &ls0, &ls1))
    return {ProductRoute::kSplit2, ls0, ls1};
  // otherwise (no cluster kernel for the base) the five launches, whose transforms
  // split over 2-8 CTAs each
  const bool few_unsplit = ls == 0 && plan->cluster == 0 && plan->N >= 2048 && !many;
  // Fewer than SMs/4 products of N = 4096 or 8192 as well (one product: 34 vs 37 us at
  // 4096, 37 vs 39 us at 8192; from SMs/4 products of N = 8192 the cluster kernel is faster)
  const bool few_mid = plan->cluster == 0 && plan->N >= 4096 && plan->N <= 8192 &&
                       (long)count < (long)sm_count() / 4;
  // N = 4096 to 16384 from 4 products per SM (2 at 16384): whole transforms of 2048 points
  // run 3 CTAs per SM with the additions on the integer pipes, where the product kernels wait
  // for their clusters and, at N = 4096, for 128 threads per 2048 points.  2000 products,
  // kernel / five launches: N = 4096 on Dif4/1024 1.07, on Dif8/512 1.13; 8192 1.12 and 1.13;
  // 16384 1.12 and 1.16.  With fewer both are uneven (300 of N = 8192: 0.95 and 0.82).
  const long per_sm = (long)count / sm_count();
  const bool large = plan->cluster == 0 && plan->lv.nlevels > 0 && plan->N >= 4096 && plan->N <= 16384 &&
                     per_sm >= (plan->N == 16384 ? 2 : 4);
  if (!ok || (plan->N >= 32768 && plan->cluster == 0) || few_unsplit || few_mid || large)
    return {ProductRoute::kFive, ls, 0, ok && large};
  return {ProductRoute::kPlain, ls};
}

}  // namespace

// Products given as device items (all of the plan's N) on the largest cluster
// the plan allows, for latency: the serving loop's large products.
bool cfft::u64_product_splittable(const cfft_u64_product_plan* plan) {
  if (plan->lv.nlevels == 0) return split0_log2(plan) >= 1;
  const int max_ls = std::min(3, plan->lv.log2r[0]);
  const int min_ls = std::max(0, ilog2(plan->n) - kSmemLog2Max);
  return max_ls >= 1 && min_ls <= max_ls;
}

cfft_status cfft::u64_product_split_items(const cfft_u64_product_plan* plan, const cfft_product_item* items,
                                          size_t count, void* stream) {
  if (!u64_product_splittable(plan)) return fail(CFFT_ERR_INVALID_SIZE, "product size cannot be split over a cluster");
  if (count == 0) return CFFT_OK;
  if (plan->lv.nlevels == 0)
    return launch_split0_product(plan, split0_log2(plan), nullptr, nullptr, 0, nullptr, count, (cudaStream_t)stream,
                                 items);
  // At most 8 CTAs per product here: the serving loop and the work queue keep several
  // launches in flight, and a 16-CTA cluster waits for 16 free SMs of one GPC
  int ls0 = 0, ls1 = 0;
  if (split2_shape(plan, count, &ls0, &ls1, kWhole, false))
    return launch_split2_product(plan, ls0, ls1, nullptr, nullptr, 0, nullptr, count, (cudaStream_t)stream, items);
  const int max_ls = std::min(3, plan->lv.log2r[0]);
  return launch_split_product(plan, max_ls, nullptr, nullptr, 0, nullptr, count, (cudaStream_t)stream, items);
}

void cfft::u64_product_tables(const cfft_u64_product_plan* p, const void** w, const void** winv, const void** tw,
                              const void** itw) {
  *w = p->d_w;
  *winv = p->d_winv;
  *tw = p->d_tw;
  *itw = p->d_itw;
}

extern "C" {

cfft_status cfft_u64_fold_twist(const cfft_u64_product_plan* plan, const uint64_t* a, double* z, size_t count,
                                void* stream) {
  if (!plan || !a || !z) return fail(CFFT_ERR_INVALID_ARGUMENT, "null argument");
  if (count == 0) return CFFT_OK;
  const long total = (long)(count * plan->n);
  CFFT_CUDA_TRY(launch_dependent(fold_twist_kernel, ew_grid(total), 256, 0, (cudaStream_t)stream, a, (double2*)z,
                                 total, ilog2(plan->n), (const double2*)plan->d_tw));
  return CFFT_OK;
}

cfft_status cfft_c64_pointwise(const double* bhat, size_t bhat_stride, double* z, size_t n, size_t count,
                               void* stream) {
  if (!bhat || !z) return fail(CFFT_ERR_INVALID_ARGUMENT, "null argument");
  if (!is_pow2(n)) return fail(CFFT_ERR_INVALID_SIZE, "n must be a power of two");
  if (count == 0) return CFFT_OK;
  const long total = (long)(count * n);
  CFFT_CUDA_TRY(launch_dependent(pointwise_kernel, ew_grid(total), 256, 0, (cudaStream_t)stream, (const double2*)bhat,
                                 (long)bhat_stride, (double2*)z, total, ilog2(n)));
  return CFFT_OK;
}

cfft_status cfft_u64_untwist_round(const cfft_u64_product_plan* plan, const double* z, uint64_t* out, size_t count,
                                   void* stream) {
  if (!plan || !z || !out) return fail(CFFT_ERR_INVALID_ARGUMENT, "null argument");
  if (count == 0) return CFFT_OK;
  const long total = (long)(count * plan->n);
  CFFT_CUDA_TRY(launch_dependent(untwist_round_kernel, ew_grid(total), 256, 0, (cudaStream_t)stream,
                                 (const double2*)z, out, total, ilog2(plan->n), (const double2*)plan->d_itw));
  return CFFT_OK;
}

cfft_status cfft_u64_fourier_mul_monomial(const cfft_u64_product_plan* plan, unsigned long long degree, double* z,
                                          size_t count, void* stream) {
  if (!plan || !z) return fail(CFFT_ERR_INVALID_ARGUMENT, "null argument");
  if (count == 0) return CFFT_OK;
  cudaStream_t s = (cudaStream_t)stream;
  // the monomial's digits, its operand (the plan's own preparation), then the pointwise
  // product with every polynomial: the same bits as preparing X^degree and multiplying
  void* ws = nullptr;
  const size_t digit_bytes = plan->N * sizeof(int64_t);
  if (plan->workspace.alloc((void**)&ws, digit_bytes + plan->n * sizeof(double2), s) != cudaSuccess)
    return fail(CFFT_ERR_OUT_OF_MEMORY, "monomial workspace");
  int64_t* digits = (int64_t*)ws;
  double* mono = (double*)((char*)ws + digit_bytes);
  cfft_status st = launch_dependent(monomial_digits_kernel, ew_grid((long)plan->N), 256, 0, s, digits, (long)plan->N,
                                    degree) == cudaSuccess
                       ? CFFT_OK
                       : fail(CFFT_ERR_CUDA, "monomial digits launch");
  if (st == CFFT_OK) st = cfft_u64_prepare_operand(plan, digits, mono, 1, stream);
  if (st == CFFT_OK) st = cfft_c64_pointwise(mono, 0, z, plan->n, count, stream);
  cudaFreeAsync(ws, s);
  return st;
}

cfft_status cfft_u64_product_sum(const cfft_u64_product_plan* plan, const uint64_t* a, const double* bhat,
                                 size_t terms, uint64_t* out, size_t count, void* stream) {
  if (!plan || !a || !bhat || !out) return fail(CFFT_ERR_INVALID_ARGUMENT, "null argument");
  if (terms == 0 || terms > 0x7fffffff) return fail(CFFT_ERR_INVALID_ARGUMENT, "terms must be at least 1");
  if (count == 0) return CFFT_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const size_t all = count * terms;
  const bool few = plan->cluster == 0 && (long)count < (long)sm_count() / 2;
  const long fill = plan->n > (size_t(1) << kBlockLog2Auto) ? (long)sm_count() / 2 : 2L * sm_count();
  // outputs that do not fill the SMs
  const bool fewer = plan->cluster == 0 && (long)count < fill;
  const bool room = fewer && may_allocate(plan, s);
  // One term is a product where a product needs no workspace.  Else it takes the five
  // launches below, but on radix 16 a cluster for each output where there is one (one of
  // N = 8192 on Dit16/512: five launches 58 us, a cluster 50; on Dit16/1024 58 and 52, on
  // Dit4/1024 37 and 40, on Dit2/1024 43 and 49).
  bool on_cluster = false;
  if (terms == 1 && fewer) {
    const ProductRoute r = product_route(plan, count);
    if (r.kind != ProductRoute::kFive) return cfft_u64_product(plan, a, bhat, plan->n, out, count, stream);
    on_cluster = algo_radix(plan->base_algo) == 16 && r.ls0 > 0 && plan->N > (size_t(2) << kBlockLog2Auto);
  }
  // A few outputs of a plan on a DIF base without an outer level, or with one of radix 2,
  // 4 or 8 (the external product of a blind-rotation step): every term's forward on a
  // cluster of its own, then every output's sum and inverse on one, in two launches
  // around a small workspace of the terms' products.  Below SMs/2 outputs; more outputs
  // fill the SMs with one CTA or cluster each.
  const bool dif = !(plan->base_algo & 1);
  const int s0 = dif ? split0_log2(plan) : 0;
  if (few && room && dif && terms > 1 && all <= kWorkspaceSmall / (plan->n * sizeof(double2))) {
    int f0 = 0, f1 = 0, i0 = 0, i1 = 0;
    const bool level = split2_shape(plan, all, &f0, &f1, kForward) && split2_shape(plan, count, &i0, &i1, kInverse);
    void* ws = nullptr;
    if ((s0 >= 1 || level) && plan->workspace.alloc(&ws, all * plan->n * sizeof(double2), s) == cudaSuccess) {
      const int tr = (int)terms;
      cfft_status st =
          s0 >= 1 ? launch_split0_product(plan, s0, a, bhat, plan->n, nullptr, all, s, nullptr, kForward, 1, (double2*)ws)
                  : launch_split2_product(plan, f0, f1, a, bhat, plan->n, nullptr, all, s, nullptr, kForward, 1,
                                          (double2*)ws);
      if (st == CFFT_OK)
        st = s0 >= 1 ? launch_split0_product(plan, s0, nullptr, nullptr, 0, out, count, s, nullptr, kInverse, tr,
                                             (double2*)ws)
                     : launch_split2_product(plan, i0, i1, nullptr, nullptr, 0, out, count, s, nullptr, kInverse, tr,
                                             (double2*)ws);
      cudaFreeAsync(ws, s);
      return st;
    }
  }
  // Otherwise, while the outputs do not fill the SMs, five launches over all terms at once:
  // one CTA or cluster per output runs its terms one after the other (N = 2048 on Dit4: two
  // outputs of 8 terms 137 us, five launches 24; 75 of 6 108 and 44; 300 of 4, two CTAs per
  // SM, 106 and 93; N = 8192 on Dit8/1024: 40 of 3 101 and 90, 75 of 6 186 and 207).
  if (room && !on_cluster && all + count <= kWorkspaceSmall / (plan->n * sizeof(double2))) {
    const cfft_status st = product_sum_unfused(plan, a, bhat, terms, out, count, s);
    if (st != CFFT_ERR_OUT_OF_MEMORY) return st;
  }
  // Without a workspace, a few outputs on DIF bases run their terms one after another on
  // the cluster of each output.
  int l0 = 0, l1 = 0;
  if (few && dif && terms > 1 && s0 >= 1 && (plan->n >> s0) <= (size_t)kSplit0Acc * 256)
    return launch_split0_product(plan, s0, a, bhat, plan->n, out, count, s, nullptr, kSum, (int)terms);
  if (few && dif && terms > 1 && split2_shape(plan, count, &l0, &l1, kSum))
    return launch_split2_product(plan, l0, l1, a, bhat, plan->n, out, count, s, nullptr, kSum, (int)terms);
  if (plan->N > (size_t(2) << kBlockLog2Auto)) {  // one output per thread-block cluster (N = 8192: by default)
    bool ok = true;
    const int ls = product_split_log2(plan, count, &ok);
    // from N = 32768 the unfused sum, as the products take five launches there
    if (!ok || (plan->N >= 32768 && plan->cluster == 0))
      return product_sum_unfused(plan, a, bhat, terms, out, count, (cudaStream_t)stream);
    if (ls > 0)
      return launch_split_product(plan, ls, a, bhat, plan->n, out, count, (cudaStream_t)stream, nullptr,
                                  (int)terms);
  }
  const bool reg_acc = plan->n <= (size_t)(kSumRegAcc * kProdThreads);
  const void* fn = u64_product_sum_kernel_ptr(plan->base_algo, reg_acc, few_warps(plan, (long)count, plan->n));
  const size_t smem = (reg_acc ? 2 : 3) * plan->n * sizeof(double2);
  const int grid = grid_for(fn, kProdThreads, smem, (long)count);
  DevLevels L = plan->dlv;
  long cnt = (long)count;
  int tr = (int)terms;
  const double2* bh = (const double2*)bhat;
  void* args[] = {(void*)&a, (void*)&bh, &tr, (void*)&out, &cnt, &L, (void*)&plan->d_w, (void*)&plan->d_winv,
                  (void*)&plan->d_tw, (void*)&plan->d_itw};
  return launch_kernel(fn, grid, kProdThreads, args, smem, (cudaStream_t)stream);
}

cfft_unordered_plan* cfft_u64_product_fft(const cfft_u64_product_plan* plan) { return plan ? plan->fft : nullptr; }

cfft_status cfft_u64_product_set_cluster_size(cfft_u64_product_plan* plan, int ctas) {
  if (!plan || !(ctas == 0 || ctas == 1 || ctas == 2 || ctas == 4 || ctas == 8))
    return fail(CFFT_ERR_INVALID_ARGUMENT, "cluster size must be 0 (automatic), 1, 2, 4 or 8");
  plan->cluster = ctas;
  return CFFT_OK;
}

cfft_status cfft_u64_product_set_graph_workspace(cfft_u64_product_plan* plan, int on) {
  if (!plan || (on != 0 && on != 1)) return fail(CFFT_ERR_INVALID_ARGUMENT, "graph workspace must be 0 or 1");
  plan->graph_workspace = on == 1;
  return CFFT_OK;
}

cfft_status cfft_u64_product_set_int_adds(cfft_u64_product_plan* plan, int eighths) {
  if (!plan || eighths < 0 || eighths > 8) return fail(CFFT_ERR_INVALID_ARGUMENT, "eighths must be in 0..8");
  plan->int_adds = eighths;
  return CFFT_OK;
}
int cfft_u64_product_int_adds(const cfft_u64_product_plan* plan) {
  return plan ? int_adds_of(plan->int_adds) : -1;
}

cfft_status cfft_u64_product_plan_create(size_t N, cfft_algo base_algo, size_t base_n, cfft_u64_product_plan** out) {
  if (!out) return fail(CFFT_ERR_INVALID_ARGUMENT, "null output pointer");
  *out = nullptr;
  if (!is_pow2(N) || N < 64 || ilog2(N) > kUnorderedMaxLog2 + 1)
    return fail(CFFT_ERR_INVALID_SIZE, "u64 product: N must be a power of two in [64, 2^29]");
  const size_t n = N / 2;
  if (!is_pow2(base_n) || base_n > n || (base_n != n && base_n < 32) || ilog2(base_n) > 10)
    return fail(CFFT_ERR_INVALID_ARGUMENT, "u64 product: invalid base_n");
  if (base_algo < 0 || base_algo > 7) return fail(CFFT_ERR_INVALID_ARGUMENT, "unknown FftAlgo");
  cfft_status st = CFFT_OK;
  auto* p = new cfft_u64_product_plan();
  p->N = N;
  p->n = n;
  p->base_n = base_n;
  p->base_algo = base_algo;
  p->lv = make_levels(n, base_n);
  p->dlv = dev_levels(p->lv);
  std::vector<c64h> w(n + base_n), wi(n + base_n), tw(n), itw(n);
  unordered_twiddles(n, base_n, algo_radix(base_algo), w.data(), wi.data());
  product_twist_tables(N, tw.data(), itw.data());
  st = upload((const double2*)w.data(), n + base_n, &p->d_w);
  if (st == CFFT_OK) st = cfft_unordered_plan_create(n, base_algo, base_n, &p->fft);
  if (st == CFFT_OK) st = upload((const double2*)wi.data(), n + base_n, &p->d_winv);
  if (st == CFFT_OK) st = upload((const double2*)tw.data(), n, &p->d_tw);
  if (st == CFFT_OK) st = upload((const double2*)itw.data(), n, &p->d_itw);
  if (st != CFFT_OK) {
    free_u64(p);
    delete p;
    return st;
  }
  *out = p;
  return CFFT_OK;
}

void cfft_u64_product_plan_destroy(cfft_u64_product_plan* plan) {
  if (!plan) return;
  free_u64(plan);
  delete plan;
}

size_t cfft_u64_product_poly_size(const cfft_u64_product_plan* plan) { return plan ? plan->N : 0; }
void cfft_u64_product_algo(const cfft_u64_product_plan* plan, cfft_algo* base_algo, size_t* base_n) {
  if (!plan) return;
  if (base_algo) *base_algo = (cfft_algo)plan->base_algo;
  if (base_n) *base_n = plan->base_n;
}

cfft_status cfft_u64_prepare_operand(const cfft_u64_product_plan* plan, const int64_t* b, double* bhat, size_t count,
                                     void* stream) {
  if (!plan || !b || !bhat) return fail(CFFT_ERR_INVALID_ARGUMENT, "null argument");
  if (count == 0) return CFFT_OK;
  if (plan->N > (size_t(2) << kSmemLog2Max)) {  // unfused: fold and twist, then the plan's forward FFT
    cfft_status st = cfft_u64_fold_twist(plan, (const uint64_t*)b, bhat, count, stream);
    if (st != CFFT_OK) return st;
    return cfft_unordered_fwd(plan->fft, bhat, count, stream);
  }
  const size_t smem = 2 * plan->n * sizeof(double2);
  const void* fn = u64_prepare_kernel_ptr(plan->base_algo, few_warps(plan, (long)count, plan->n));
  const int grid = grid_for(fn, kProdThreads, smem, (long)count);
  DevLevels L = plan->dlv;
  long cnt = (long)count;
  double2* bh = (double2*)bhat;
  void* args[] = {(void*)&b, &bh, &cnt, &L, (void*)&plan->d_w, (void*)&plan->d_tw};
  return launch_kernel(fn, grid, kProdThreads, args, smem, (cudaStream_t)stream);
}

cfft_status cfft_u64_product(const cfft_u64_product_plan* plan, const uint64_t* a, const double* bhat,
                             size_t bhat_stride, uint64_t* out, size_t count, void* stream) {
  if (!plan || !a || !bhat || !out) return fail(CFFT_ERR_INVALID_ARGUMENT, "null argument");
  if (bhat_stride != 0 && bhat_stride != plan->n)
    return fail(CFFT_ERR_INVALID_ARGUMENT, "bhat_stride must be 0 or N/2");
  if (count == 0) return CFFT_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const ProductRoute r = product_route(plan, count);
  if (r.kind == ProductRoute::kSplit0)
    return launch_split0_product(plan, r.ls0, a, bhat, bhat_stride, out, count, s);
  if (r.kind == ProductRoute::kSplit2)
    return launch_split2_product(plan, r.ls0, r.ls1, a, bhat, bhat_stride, out, count, s);
  if (r.kind == ProductRoute::kFive && (!r.spare || may_allocate(plan, s))) {
    // in equal parts within what the pool keeps, or a small workspace where there is another route
    const size_t fit =
        std::max<size_t>(1, (r.spare ? kWorkspaceSmall : kWorkspaceKeep) / (plan->n * sizeof(double2)));
    const size_t parts = (count + fit - 1) / fit, part = (count + parts - 1) / parts;
    void* z = nullptr;
    const bool got = plan->workspace.alloc(&z, part * plan->n * sizeof(double2), s) == cudaSuccess;
    if (!got && !r.spare) return fail(CFFT_ERR_OUT_OF_MEMORY, "u64 product workspace");
    if (got) {
      cfft_status st = CFFT_OK;
      for (size_t c0 = 0; c0 < count && st == CFFT_OK; c0 += part) {
        const size_t c = std::min(part, count - c0);
        st = cfft_u64_fold_twist(plan, a + c0 * plan->N, (double*)z, c, stream);
        if (st == CFFT_OK) st = cfft_unordered_fwd(plan->fft, (double*)z, c, stream);
        if (st == CFFT_OK)
          st = cfft_c64_pointwise(bhat + 2 * c0 * bhat_stride, bhat_stride, (double*)z, plan->n, c, stream);
        if (st == CFFT_OK) st = cfft_unordered_inv(plan->fft, (double*)z, c, stream);
        if (st == CFFT_OK) st = cfft_u64_untwist_round(plan, (const double*)z, out + c0 * plan->N, c, stream);
      }
      cudaFreeAsync(z, s);
      return st;
    }
  }
  if (r.ls0 > 0) return launch_split_product(plan, r.ls0, a, bhat, bhat_stride, out, count, s);
  return launch_product(plan, a, bhat, bhat_stride, out, count, s);
}

// Method::Measure for the product: every (base_algo, base_n) the reference's
// unordered measurement considers for n = N/2 (src/unordered.rs:553-640: the
// ordered algorithms at n when n <= 256, else bases 512 and 1024), timed over
// a batch that fills every SM, on the route that such a batch takes: the
// fused kernel below N = 4096, the five launches from there.  The ranking is
// for full batches; smaller ones run other kernels, which are not timed.
// Several candidates come within noise of each other; among those within 2%
// of the fastest a DIF base is taken, whose few-product cluster kernels are
// the faster ones (one N = 4096 product: 12.8 us on Dif4/1024, 33 us on the
// five launches that DIT bases take).
cfft_status cfft_u64_product_plan_create_measure(size_t N, double seconds, cfft_u64_product_plan** out) {
  if (!out) return fail(CFFT_ERR_INVALID_ARGUMENT, "null output pointer");
  *out = nullptr;
  if (!is_pow2(N) || N < 64 || ilog2(N) > kUnorderedMaxLog2 + 1)
    return fail(CFFT_ERR_INVALID_SIZE, "u64 product: N must be a power of two in [64, 2^29]");
  const size_t n = N / 2;
  TuneVal tv;
  if (tune_lookup(2, N, &tv)) {  // measured before on this GPU model
    cfft_status st = cfft_u64_product_plan_create(N, (cfft_algo)tv.algo, tv.base_n, out);
    return st;
  }
  std::vector<size_t> bases;
  if (n <= 256) bases.push_back(n);
  else
    for (size_t b : {size_t(512), size_t(1024)})
      if (b <= n) bases.push_back(b);
  // eight products per SM up to N = 8192, the same number of CTAs for larger N,
  // within 2 GiB of operands, results and workspace (32 N bytes per product)
  const size_t per_sm = std::max<size_t>(1, 8 * 8192 / std::max<size_t>(N, 8192));
  const size_t count = std::max<size_t>(1, std::min((size_t)sm_count() * per_sm, (size_t(1) << 31) / (32 * N)));
  uint64_t *da = nullptr, *dout = nullptr;
  double* dbhat = nullptr;
  CFFT_CUDA_TRY(cudaMalloc(&da, count * N * sizeof(uint64_t)));
  CFFT_CUDA_TRY(cudaMalloc(&dout, count * N * sizeof(uint64_t)));
  CFFT_CUDA_TRY(cudaMalloc(&dbhat, count * n * sizeof(double2)));
  cudaStream_t s;
  CFFT_CUDA_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  // torus words and the spectra of 8-bit digits
  fill_timing_words(da, count * N, s);
  fill_timing_doubles(dbhat, 2 * count * n, 0x1p12, s);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  double best = 1e30;
  int best_algo = 0;
  size_t best_base = bases.front();
  struct Timed {
    int algo;
    size_t base;
    double ms;
  };
  std::vector<Timed> timed;
  cfft_status st = CFFT_OK;
  for (size_t base : bases) {
    for (int algo = 0; algo < 8 && st == CFFT_OK; ++algo) {
      cfft_u64_product_plan* p = nullptr;
      st = cfft_u64_product_plan_create(N, (cfft_algo)algo, base, &p);
      if (st != CFFT_OK) break;
      cfft_u64_product(p, da, dbhat, n, dout, count, s);  // warm-up
      int reps = 1;
      double per = 0;
      for (;;) {
        cudaEventRecord(e0, s);
        for (int r = 0; r < reps; ++r) cfft_u64_product(p, da, dbhat, n, dout, count, s);
        cudaEventRecord(e1, s);
        cudaEventSynchronize(e1);
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        per = ms / reps;
        if (ms * 1e-3 >= std::max(seconds, 1e-3) || reps >= 4096) break;
        reps *= 2;
      }
      if (per < best) {
        best = per;
        best_algo = algo;
        best_base = base;
      }
      timed.push_back(Timed{algo, base, per});
      cfft_u64_product_plan_destroy(p);
    }
  }
  if (best_algo & 1) {  // a DIT winner: the fastest DIF base within 2%, if any
    double dif_best = 1e30;
    for (const Timed& t : timed)
      if (!(t.algo & 1) && t.ms <= best * 1.02 && t.ms < dif_best) {
        dif_best = t.ms;
        best_algo = t.algo;
        best_base = t.base;
      }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaStreamDestroy(s);
  cudaFree(da);
  cudaFree(dout);
  cudaFree(dbhat);
  if (st != CFFT_OK) return st;
  st = cfft_u64_product_plan_create(N, (cfft_algo)best_algo, best_base, out);
  if (st != CFFT_OK) return st;
  tune_store(2, N, TuneVal{best_algo, best_base, kProdThreads, 1, 0});
  return CFFT_OK;
}

// Host-buffer products: the batch is cut into chunks that flow through three
// streams, so the host-to-device copy of one chunk, the kernel of the previous
// one and the device-to-host copy of the one before overlap (copy engines and
// SMs work at once).  Returns when every result is in host memory.
cfft_status cfft_u64_product_host(const cfft_u64_product_plan* plan, const uint64_t* a, const double* bhat,
                                  size_t bhat_stride, uint64_t* out, size_t count) {
  if (!plan || !a || !bhat || !out) return fail(CFFT_ERR_INVALID_ARGUMENT, "null argument");
  if (bhat_stride != 0 && bhat_stride != plan->n)
    return fail(CFFT_ERR_INVALID_ARGUMENT, "bhat_stride must be 0 or N/2");
  if (count == 0) return CFFT_OK;
  // About 24 chunks per call on 4 streams: the first copy in and the last
  // copy out, which nothing overlaps, are then 1/24 of the data each, and 4
  // chunks in flight keep kernels of several chunks resident at once.  When
  // `out` is page-locked the kernels store the results there themselves (no
  // copy out, no drain): 6.56 vs 6.40 M products/s at N = 2048, 8192 per call.
  // Measured schedules (M products/s, Dif4, 8192 per call, direct stores):
  // 24 chunks on 4 streams 6.58, on 6 6.53, on 8 6.48; 12 on 6 6.38, 48 on 6
  // 6.50; a first chunk of 76 or 152 products or a last one of 152: within
  // 0.03 of the equal chunks.  Device buffers alone: 6.88.
  // The operands still come in by copy: kernels reading them from host memory
  // wait on every product's first loads (6.60 M/s for one launch with both
  // sides in host memory, against 6.94 M/s on device buffers).
  const HostChunks hc = host_chunks();
  const int nslots = hc.slots;
  const size_t poly_bytes = plan->N * sizeof(uint64_t);
  // the schedule: an optional first and last chunk, the rest in `chunks` equal chunks of
  // at least two products per SM
  const size_t first_c = std::min(count, (size_t)hc.first);
  const size_t last_c = std::min(count - first_c, (size_t)hc.last);
  const size_t mid = count - first_c - last_c;
  const size_t min_chunk = (size_t)sm_count() * 2;
  const size_t chunk = mid ? std::min(mid, std::max(min_chunk, (mid + hc.chunks - 1) / hc.chunks)) : 0;
  const size_t cap = std::max(chunk, std::max(first_c, last_c));
  uint64_t* mapped_out = (uint64_t*)mapped_host_range(out, count * poly_bytes);
  PipeSlot slot[8];
  cfft_status st = host_pipeline(nslots, 2 * cap * poly_bytes, slot);
  if (st != CFFT_OK) return st;
  size_t i = 0;
  for (size_t first = 0; first < count; ++i) {
    const size_t c = first == 0 && first_c ? first_c
                     : (last_c && first + last_c >= count) ? count - first : std::min(chunk, count - first - last_c);
    const PipeSlot& sl = slot[i % nslots];
    uint64_t* da = (uint64_t*)sl.dev;
    uint64_t* dout = mapped_out ? mapped_out + first * plan->N : da + cap * plan->N;
    CFFT_CUDA_TRY(cudaMemcpyAsync(da, a + first * plan->N, c * poly_bytes, cudaMemcpyHostToDevice, sl.stream));
    const double* bh = bhat + (bhat_stride ? first * bhat_stride * 2 : 0);
    st = cfft_u64_product(plan, da, bh, bhat_stride, dout, c, sl.stream);
    if (st != CFFT_OK) return st;
    if (!mapped_out)
      CFFT_CUDA_TRY(cudaMemcpyAsync(out + first * plan->N, dout, c * poly_bytes, cudaMemcpyDeviceToHost, sl.stream));
    first += c;
  }
  for (int k = 0; k < nslots; ++k) CFFT_CUDA_TRY(cudaStreamSynchronize(slot[k].stream));
  return CFFT_OK;
}

}  // extern "C"
