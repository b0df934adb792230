// pac_vec_kernel.cuh -- the sm_100a kernels of the passes over 8-byte
// elements (pac_vec.cuh).
#pragma once

#include "pac_tma.cuh"
#include "pac_vec_list.h"

namespace pac {

// bytes [src, src + bytes) to this CTA's shared memory (16-byte aligned,
// bytes a multiple of 16); completion counted on bar
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// a one-warp CTA needs no CTA barrier
template <int NT>
__device__ __forceinline__ void vec_sync() {
  if constexpr (NT == 32) __syncwarp();
  else __syncthreads();
}
template <int NT>
__device__ __forceinline__ bool vec_all(bool ok) {
  if constexpr (NT == 32) return __all_sync(0xffffffffu, ok);
  else return __syncthreads_and(ok);
}

// one thread's registers and the CTA's barriers (VecPass::body)
template <class VP, class V, class Issue>
struct VecExec {
  CV<V> x[VP::TPT];
  typename VP::Mid m;
  long long next, ntiles;
  bool copies;
  Issue& issue;
  template <class F>
  __device__ __forceinline__ void each(F&& f) {
    f((int)threadIdx.x, x);
  }
  template <class F>
  __device__ __forceinline__ void each_mid(F&& f) {
    f((int)threadIdx.x, x, m);
  }
  __device__ __forceinline__ void sync() { vec_sync<VP::kThreads>(); }
  // every thread has read the buffer: its reads and writes precede the next
  // copy into it
  __device__ __forceinline__ void freed() {
    fence_proxy_async();
    sync();
    if (next >= ntiles) pdl_trigger();
    else if (threadIdx.x == 0 && copies) issue(next);
  }
};

// persistent CTAs over the tiles blockIdx.x, blockIdx.x + gridDim.x, ...
// issue(tile) starts the copies of a tile into the buffer (one thread).
template <class VP, class V, int TW4, class Issue>
__device__ __forceinline__ void vec_tiles(const PassDesc& d, CV<V>* B, uint64_t* bar,
                                          long long ntiles, Issue& issue) {
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_barrier_init();
  }
  using Real = typename VP::Real;
  Cx<Real>* tws = reinterpret_cast<Cx<Real>*>(B + VP::TILE);
  VP::tw_fill(d, threadIdx.x, tws);  // read after the first tile's barrier
  pdl_wait();
  __syncthreads();
  long long tile = blockIdx.x;
  if (threadIdx.x == 0 && tile < ntiles && !d.unaligned) issue(tile);
  uint32_t phase = 0;
  VecExec<VP, V, Issue> ex{{}, {}, tile, ntiles, !d.unaligned, issue};
  for (; tile < ntiles; tile += gridDim.x) {
    ex.next = tile + gridDim.x;
    bool ok = true;
    if (d.unaligned) {
      VP::copy_in(d, tile, threadIdx.x, B);
      vec_sync<VP::kThreads>();  // (a vote alone orders no memory accesses)
    } else {
      ok = mbar_wait_bounded(bar, phase, wait_limit_of(d));
    }
    if (!vec_all<VP::kThreads>(ok)) {
      // a wait gave up: report it, issue nothing more, keep the CTA (its
      // shared memory) alive until the copy in flight has landed
      if (threadIdx.x == 0) {
        report_timeout(d);
        mbar_wait_bounded(bar, phase);
      }
      break;
    }
    phase ^= 1;
    VP::template body<TW4>(d, tile, B, tws, ex);
  }
}

template <class V, int B2, int MODE, int SIGN, int LOGL, int LOGW, int NT, int MINB,
          int OFFS, int PORD>
__global__ void __launch_bounds__(NT, MINB) pac_vec_rows_kernel(const __grid_constant__ PassDesc d) {
  using VP = VecPass<V, B2, MODE, SIGN, LOGL, 0, LOGW, NT, 0, OFFS, PORD>;
  using Real = typename VP::Real;
  extern __shared__ unsigned char pac_smem_raw[];
  __shared__ __align__(8) uint64_t bar;
  CV<V>* B =
      reinterpret_cast<CV<V>*>(pac_smem_raw + ((128u - (smem_u32(pac_smem_raw) & 127u)) & 127u));
  V* D = reinterpret_cast<V*>(B);
  constexpr int WL = VP::W * VP::LPU;  // lines of a tile
  const long long ntiles = (d.nlines + WL - 1) / WL;
  auto issue = [&](long long tile) {
    const long long g0 = tile * WL;
    const long long n = d.nlines - g0 < WL ? d.nlines - g0 : WL;
    const uint32_t bytes = (uint32_t)(n << LOGL) * (uint32_t)sizeof(Real);
    mbar_arrive_expect_tx(&bar, 2 * bytes);
    if constexpr (OFFS) {  // line by line
      for (int l = 0; l < (int)n; ++l) {
        const long long o = VP::line_off(d, g0 + l);
        Real* dst = (Real*)D + (l << LOGL);
        bulk_load(dst, (const Real*)d.in_re + o, (uint32_t)sizeof(Real) << LOGL, &bar);
        bulk_load(dst + VP::LPU * VP::DIM, (const Real*)d.in_im + o, (uint32_t)sizeof(Real) << LOGL,
                  &bar);
      }
      return;
    }
    bulk_load(D, (const Real*)d.in_re + (g0 << LOGL), bytes, &bar);
    bulk_load(D + VP::DIM, (const Real*)d.in_im + (g0 << LOGL), bytes, &bar);
  };
  vec_tiles<VP, V, 0>(d, B, &bar, ntiles, issue);
}

// column tiles: a tensor map over the array as [O][L][S / LPU] 8-byte elements
template <class V, int B2, int MODE, int SIGN, int LOGL, int LOGW, int NT, int MINB, int TW4>
__global__ void __launch_bounds__(NT, MINB)
    pac_vec_cols_kernel(const __grid_constant__ PassDesc d, const __grid_constant__ CUtensorMap tre,
                        const __grid_constant__ CUtensorMap tim) {
  using VP = VecPass<V, B2, MODE, SIGN, LOGL, 1, LOGW, NT>;
  extern __shared__ unsigned char pac_smem_raw[];
  __shared__ __align__(8) uint64_t bar;
  CV<V>* B =
      reinterpret_cast<CV<V>*>(pac_smem_raw + ((128u - (smem_u32(pac_smem_raw) & 127u)) & 127u));
  V* D = reinterpret_cast<V*>(B);
  const long long ntiles = (d.nlines / VP::LPU) >> LOGW;
  auto issue = [&](long long tile) {
    int i0, o;
    VP::tile_coords(d, tile, i0, o);
    mbar_arrive_expect_tx(&bar, (uint32_t)(16 * VP::DIM));
    for (int k = 0; k < VP::L / VP::BOXR; ++k) {
      tma_load_3d(D + ((k * VP::BOXR) << LOGW), &tre, &bar, i0, k * VP::BOXR, o);
      tma_load_3d(D + VP::DIM + ((k * VP::BOXR) << LOGW), &tim, &bar, i0, k * VP::BOXR, o);
    }
  };
  vec_tiles<VP, V, TW4>(d, B, &bar, ntiles, issue);
}

// column tiles read straight from global memory: one tile a CTA
template <class VP, class V>
struct VecExecOnce {
  CV<V> x[VP::TPT];
  typename VP::Mid m;
  template <class F>
  __device__ __forceinline__ void each_mid(F&& f) {
    f((int)threadIdx.x, x, m);
  }
  template <class F>
  __device__ __forceinline__ void each(F&& f) {
    f((int)threadIdx.x, x);
  }
  __device__ __forceinline__ void sync() { vec_sync<VP::kThreads>(); }
  __device__ __forceinline__ void freed() { pdl_trigger(); }
};
template <class V, int B2, int MODE, int SIGN, int LOGL, int LOGW, int NT, int MINB, int TW4,
          int OFFS>
__global__ void __launch_bounds__(NT, MINB) pac_vec_direct_kernel(const __grid_constant__ PassDesc d) {
  using VP = VecPass<V, B2, MODE, SIGN, LOGL, 1, LOGW, NT, 1, OFFS>;
  using Real = typename VP::Real;
  extern __shared__ __align__(16) unsigned char pac_smem_raw[];
  CV<V>* B = reinterpret_cast<CV<V>*>(pac_smem_raw);
  VecExecOnce<VP, V> ex;
  pdl_wait();
  VP::template body<TW4>(d, blockIdx.x, B, (const Cx<Real>*)nullptr, ex);
}

template <class V, int B2, int MODE, int SIGN, int LOGL, int TW4, int OFFS>
__global__ void __launch_bounds__(256) pac_vec_small_kernel(const __grid_constant__ PassDesc d) {
  const long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  pdl_wait();
  if (u < d.nlines / VT<V>::LPU)
    VecSmall<V, B2, MODE, SIGN, LOGL, OFFS>::template run<TW4>(d, u, [] { pdl_trigger(); });
}

}  // namespace pac
