// Pipelined z-pass of the Born iteration for any z length n = A R up to 256
// (A <= R <= 31): forward z-FFT, Green's multiply G(k -/+ dk/4) / N, inverse
// z-FFT (FORWARD_SOLVER_CONVERGENT_BORN.m:606-615), the same transforms as
// born_z_body.
//
//   * persistent CTAs walk tiles of 16 or 32 adjacent columns of the flattened x-y
//     plane (so a plane wastes at most one partial tile: 152 columns in rows
//     of their own would fill 9.5 of 10 tiles);
//   * a tile (n rows of 128 or 256 bytes) arrives in shared memory while the CTA
//     computes the previous one from the other stage: through one tiled TMA
//     copy on an mbarrier where the planes are multiples of 16 bytes (px * py
//     even), else through 8-byte asynchronous copies of the threads;
//   * with z = R n1 + n2 and kz = k1 + A k2: step A, the A-point DFTs over n1
//     with twiddles; step B, per (column, k1) the R-point DFT, the Green's
//     multiply at kz and the inverse R-point DFT in registers; step C, the
//     inverse A-point DFTs to global memory.  Every step writes the rows it
//     read, so the landing stage is the only buffer.
//
// One kernel per R for A = 8 and one for the other A, which it dispatches once
// per tile (A is the same for the whole grid) to code with both factors known.
// z_split() takes A = 8 or the largest A <= 10: step B then has at most 160
// items (one round of the 160 threads), and the larger radix sits in registers
// between two transforms.
//
// What bounds it: the steps' instructions and the two barriers between them
// (153 points: issue slots 53 % busy, barrier the first of the stalls), not DRAM
// (16 bytes per element, 27 % of its rate).  The kernels of A != 8 spill at large odd R
// under their launch bounds: 212 bytes stored a thread at 17, 260 at 19, 372 at 23,
// 500 at 29, 596 at 31.  The correctly rounded reciprocal of the Green's function
// costs 8 % of a pass of 152 points (0.67 -> 0.73 ms, 49 illuminations) over the
// hardware's approximation with a refinement.
#include <type_traits>

#include "cols_any.cuh"

namespace odt {
namespace {

template <int R, bool kEight>
__global__ void __launch_bounds__(kThreads, min_ctas<R>())
    z_pass_kernel(const __grid_constant__ CUtensorMap map, const BornArgs a, const int jj,
                  const float2* __restrict__ twg, const int A_, const int use_tma, const int nxt, const int ntiles,
                  int* __restrict__ fault) {
#if defined(__CUDA_ARCH__)
  const int N = A_ * R;
  const int W = kEight ? 16 : tile_w(A_);
  const ZSmem L(N, W);
  extern __shared__ __align__(128) unsigned char sm[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm);
  float2* tw = reinterpret_cast<float2*>(sm + L.tw);
  float* kz = reinterpret_cast<float*>(sm + L.kz);
  float* gxy = reinterpret_cast<float*>(sm + L.gxy);
  float2* const s0 = reinterpret_cast<float2*>(sm + L.s0);
  float2* const s1 = reinterpret_cast<float2*>(sm + L.s1);
  const int tid = threadIdx.x;
  const int c = tid & (W - 1);
  const bool flip = a.acyclic && (jj & 1);
  if ((smem_addr(s0) & 127u) != 0u || (smem_addr(s1) & 127u) != 0u) {  // never issue a misaligned copy
    if (tid == 0) atomicCAS(fault, 0, kFaultAlign);
    return;
  }
  for (int i = tid; i < N; i += kThreads) {
    tw[i] = twg[i];
    kz[i] = a.kq2[2][flip ? (i == 0 ? 0 : N - i) : i];
  }
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_fence_init();
  }
  __syncthreads();
  int tile = blockIdx.x;
  if (tile >= ntiles) return;
  const int pxy = a.px * a.py;            // row stride of a column
  const uint32_t bytes = (uint32_t)(sizeof(float2) * N * W);
  // tile t -> (W columns from i0 = W (t mod nxt), batch entry t / nxt)
  auto issue = [&](int t, int stage) {
    float2* dst = stage ? s1 : s0;
    const int i0 = W * (t % nxt), b = t / nxt;
    if (use_tma) {
      if (tid == 0) {
        fence_proxy_async();
        mbar_arrive_expect_tx(&bar[stage], bytes);
        tma_tile(dst, &map, 2 * i0, b, &bar[stage]);
      }
    } else {
      const int col = min(i0 + c, pxy - 1);   // columns past the plane repeat the last one; not stored
      const float2* src = a.T + (long long)b * a.nvox + col;
      for (int r = tid / W; r < N; r += kThreads / W) copy8(dst + r * W + c, src + (long long)r * pxy);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
  };
  issue(tile, 0);
  uint32_t ph0 = 0, ph1 = 0;

  for (int it = 0; tile < ntiles; ++it, tile += gridDim.x) {
    const int s = it & 1;
    const int next = tile + gridDim.x;
    if (next < ntiles) issue(next, s ^ 1);
    const int i0 = W * (tile % nxt), b = tile / nxt;
    if (tid < W) {
      const int i = min(i0 + tid, pxy - 1);
      int y = i / a.px, kx = i - y * a.px;
      if (a.perm_xy) {   // position Rx k1 + k2 holds spectral index k1 + 8 k2
        const int rx = a.px >> 3, ry = a.py >> 3;
        kx = kx / rx + 8 * (kx % rx);
        y = y / ry + 8 * (y % ry);
      }
      const int ix = flip ? (kx == 0 ? 0 : a.px - kx) : kx;
      const int iy = flip ? (y == 0 ? 0 : a.py - y) : y;
      gxy[tid] = a.kq2[0][ix] + a.kq2[1][iy];
    }
    if (use_tma) {
      const bool ok = mbar_wait(&bar[s], s ? ph1 : ph0, a.wait_limit);
      if (__syncthreads_or(!ok)) {
        if (tid == 0) {  // give up; let the copies in flight land first
          atomicCAS(fault, 0, kFaultTimeout);
          mbar_wait(&bar[s], s ? ph1 : ph0);
          if (next < ntiles) mbar_wait(&bar[s ^ 1], s ? ph0 : ph1);
        }
        return;
      }
      if (s) ph1 ^= 1; else ph0 ^= 1;
    } else {
      if (next < ntiles) asm volatile("cp.async.wait_group 1;" ::: "memory");
      else asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
    }
    float2* const S = s ? s1 : s0;
    float2* const out = a.T + (long long)b * a.nvox + i0 + c;
    const bool live = i0 + c < pxy;

    auto steps = [&](auto Ac) {
      constexpr int A = decltype(Ac)::value;
      if constexpr (ZSplit<A * R>::kA == A && (A == 8) == kEight) {
        constexpr int kN = A * R;
        constexpr int kW = tile_w(A);
        // ---- A: A-point DFT over n1 at rows R n1 + n2, times W_N^(n2 k1)
        for (int n2 = tid / kW; n2 < R; n2 += kThreads / kW) {
          float2 v[A];
#pragma unroll
          for (int r = 0; r < A; ++r) v[r] = S[(R * r + n2) * kW + c];
          Butterfly<A, false>::run(v, tw, kN);
#pragma unroll
          for (int r = 1; r < A; ++r) v[r] = cmul(v[r], tw[r * n2]);
#pragma unroll
          for (int r = 0; r < A; ++r) S[(R * r + n2) * kW + c] = v[r];
        }
        __syncthreads();
        // ---- B: R-point DFT over n2 at rows R k1 + n2 (kz = k1 + A k2),
        //      Green's multiply, inverse R-point DFT, times conj W_N^(n2 k1)
        auto mid = [&](int k1) {
          float2 v[R];
#pragma unroll
          for (int r = 0; r < R; ++r) v[r] = S[(R * k1 + r) * kW + c];
          Butterfly<R, false>::run(v, tw, kN);
          const float qxy = gxy[c];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            float q = qxy + kz[k1 + A * r];
            q = a.g_scale * q - a.g_off;
            const float rden = __frcp_rn(q * q + a.eps * a.eps) * a.inv_n;
            v[r] = cmul(make_float2(q * rden, a.eps * rden), v[r]);  // (1 / (q - i eps)) / N
          }
          Butterfly<R, true>::run(v, tw, kN);
#pragma unroll
          for (int r = 1; r < R; ++r) v[r] = cmul(v[r], cconj(tw[r * k1]));
#pragma unroll
          for (int r = 0; r < R; ++r) S[(R * k1 + r) * kW + c] = v[r];
        };
        if constexpr (A <= kThreads / kW) {   // one round
          if (tid < A * kW) mid(tid / kW);
        } else {
          for (int k1 = tid / kW; k1 < A; k1 += kThreads / kW) mid(k1);
        }
        __syncthreads();
        // ---- C: inverse A-point DFT over k1 -> rows R n1 + n2 of T
        for (int n2 = tid / kW; n2 < R; n2 += kThreads / kW) {
          float2 v[A];
#pragma unroll
          for (int r = 0; r < A; ++r) v[r] = S[(R * r + n2) * kW + c];
          Butterfly<A, true>::run(v, tw, kN);
          if (live) {
#pragma unroll
            for (int r = 0; r < A; ++r) out[(long long)(R * r + n2) * pxy] = v[r];
          }
        }
      }
    };
    if constexpr (kEight) {
      steps(std::integral_constant<int, 8>{});
    } else switch (A_) {
#define ODT_Z_CASE(k) \
  case k: steps(std::integral_constant<int, k>{}); break;
      ODT_Z_CASE(2) ODT_Z_CASE(3) ODT_Z_CASE(4) ODT_Z_CASE(5) ODT_Z_CASE(6) ODT_Z_CASE(7)
      ODT_Z_CASE(9) ODT_Z_CASE(10) ODT_Z_CASE(11) ODT_Z_CASE(12) ODT_Z_CASE(13) ODT_Z_CASE(14) ODT_Z_CASE(15)
      ODT_Z_CASE(16)
#undef ODT_Z_CASE
      default: break;
    }
    // the next iteration's copy refills the stage just read
    __syncthreads();
  }
#endif
}

template <int R, bool kEight>
cudaError_t launch_one(const BornArgs& a, int jj, const DevFft& f, int* fault, cudaStream_t s) {
  const int W = tile_w(a.pz / R);
  const ZSmem L(a.pz, W);
  const void* fn = reinterpret_cast<const void*>(z_pass_kernel<R, kEight>);
  cudaError_t e = raise_smem_limit(fn, L.total);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0, per_sm = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, z_pass_kernel<R, kEight>, kThreads, L.total);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  CUtensorMap map{};
  // planes that are no multiple of 16 bytes cannot be mapped: 8-byte copies
  const int use_tma = (long long)a.px * a.py % 2 == 0;
  if (use_tma && !make_map(a.T, (long long)a.px * a.py, a.pz, a.nbatch, W, &map)) return cudaErrorInvalidValue;
  const int nxt = (a.px * a.py + W - 1) / W;
  const int ntiles = nxt * a.nbatch;
  const int cap = per_sm * nsm;
  z_pass_kernel<R, kEight><<<ntiles < cap ? ntiles : cap, kThreads, L.total, s>>>(map, a, jj, f.tw, a.pz / R, use_tma, nxt,
                                                                          ntiles, fault);
  return cudaGetLastError();
}
}  // namespace

// instantiated in one of the object files below
template <int R>
cudaError_t z_pass_launch(const BornArgs& a, int jj, const DevFft& f, int* fault, cudaStream_t s) {
  if constexpr (R >= 8)
    if (a.pz == 8 * R) return launch_one<R, true>(a, jj, f, fault, s);
  return launch_one<R, false>(a, jj, f, fault, s);
}
#define ODT_Z_LIST(X)                                                                                     \
  X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(17) X(18) X(19) X(20) \
  X(21) X(22) X(23) X(24) X(25) X(26) X(27) X(28) X(29) X(30) X(31)
#define ODT_Z_EXTERN(r) \
  extern template cudaError_t z_pass_launch<r>(const BornArgs&, int, const DevFft&, int*, cudaStream_t);
#define ODT_Z_HERE(r) \
  template cudaError_t z_pass_launch<r>(const BornArgs&, int, const DevFft&, int*, cudaStream_t);
ODT_Z_LIST(ODT_Z_EXTERN)
#if ODT_ZG == 0
ODT_Z_HERE(31) ODT_Z_HERE(20) ODT_Z_HERE(18) ODT_Z_HERE(9) ODT_Z_HERE(2)
#elif ODT_ZG == 1
ODT_Z_HERE(29) ODT_Z_HERE(22) ODT_Z_HERE(21) ODT_Z_HERE(12) ODT_Z_HERE(3)
#elif ODT_ZG == 2
ODT_Z_HERE(23) ODT_Z_HERE(24) ODT_Z_HERE(16) ODT_Z_HERE(14) ODT_Z_HERE(4)
#elif ODT_ZG == 3
ODT_Z_HERE(19) ODT_Z_HERE(26) ODT_Z_HERE(15) ODT_Z_HERE(11) ODT_Z_HERE(5)
#elif ODT_ZG == 4
ODT_Z_HERE(17) ODT_Z_HERE(25) ODT_Z_HERE(28) ODT_Z_HERE(8) ODT_Z_HERE(6)
#else
ODT_Z_HERE(13) ODT_Z_HERE(27) ODT_Z_HERE(30) ODT_Z_HERE(10) ODT_Z_HERE(7)
#endif

#if ODT_ZG == 0
bool z_pass_supported(const BornArgs& a, const DevFft& f) {
  if (f.plan.n != a.pz || a.pz > kMaxN || a.storage || !z_split(a.pz) || !encoder()) return false;
  const long long pxy = (long long)a.px * a.py;
  return pxy < (1 << 30) && (pxy + 15) / 16 * a.nbatch < (1LL << 31);
}

cudaError_t launch_z_pass(const BornArgs& a, int jj, const DevFft& fz, int* fault, cudaStream_t s) {
  const int A = z_split(a.pz);
  if (!A) return cudaErrorNotSupported;
  switch (a.pz / A) {
#define ODT_Z_CASE(r) \
  case r: return z_pass_launch<r>(a, jj, fz, fault, s);
    ODT_Z_LIST(ODT_Z_CASE)
#undef ODT_Z_CASE
    default: return cudaErrorNotSupported;
  }
}
#endif  // ODT_ZG == 0

}  // namespace odt
