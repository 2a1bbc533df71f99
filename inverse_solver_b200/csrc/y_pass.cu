// Pipelined y-FFTs of the Born loop, in place on T, for any y length n = A R up
// to 256 (cols_any.cuh) that the 8 R-point passes of cols_pipe.cu do not cover:
// persistent CTAs walk tiles of 16 (32) columns of one x-y plane, copied into
// shared memory while the previous tile is computed; with y = R n1 + n2 and
// ky = k1 + A k2, the A-point DFTs over n1 with twiddles in place, then per
// (column, k1) the R-point DFT over n2 straight to rows k1 + A k2 of T.  The
// inverse runs as the conjugate of the forward transform of the conjugate.
// What bounds it: instructions and the barrier between the two steps, as in
// z_pass.cu.  108 points, 125 x 69 planes, 6 illuminations: 0.025 against 0.045 ms
// of the generic tiles.
#include <type_traits>

#include "cols_any.cuh"

namespace odt {
namespace {

template <int R, bool kEight>
__global__ void __launch_bounds__(kThreads, min_ctas<R>())
    y_pass_kernel(const __grid_constant__ CUtensorMap map, float2* const T, const int cols, const float sgn,
                  const long long wait_limit, const float2* __restrict__ twg, const int A_, const int use_tma,
                  const int nxt, const int ntiles, int* __restrict__ fault) {
#if defined(__CUDA_ARCH__)
  const int N = A_ * R;
  const int W = kEight ? 16 : tile_w(A_);
  const ZSmem L(N, W);
  extern __shared__ __align__(128) unsigned char sm[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm);
  float2* tw = reinterpret_cast<float2*>(sm + L.tw);
  float2* const s0 = reinterpret_cast<float2*>(sm + L.s0);
  float2* const s1 = reinterpret_cast<float2*>(sm + L.s1);
  const int tid = threadIdx.x;
  const int c = tid & (W - 1);
  if ((smem_addr(s0) & 127u) != 0u || (smem_addr(s1) & 127u) != 0u) {  // never issue a misaligned copy
    if (tid == 0) atomicCAS(fault, 0, kFaultAlign);
    return;
  }
  for (int i = tid; i < N; i += kThreads) tw[i] = twg[i];
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_fence_init();
  }
  __syncthreads();
  int tile = blockIdx.x;
  if (tile >= ntiles) return;
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
      const int col = min(i0 + c, cols - 1);   // columns past the plane repeat the last one; not stored
      const float2* src = T + (long long)b * cols * N + col;
      for (int r = tid / W; r < N; r += kThreads / W) copy8(dst + r * W + c, src + (long long)r * cols);
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
    if (use_tma) {
      const bool ok = mbar_wait(&bar[s], s ? ph1 : ph0, wait_limit);
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
    float2* const out = T + (long long)b * cols * N + i0 + c;
    const bool live = i0 + c < cols;

    auto steps = [&](auto Ac) {
      constexpr int A = decltype(Ac)::value;
      if constexpr (ZSplit<A * R>::kA == A && (A == 8) == kEight) {
        constexpr int kN = A * R;
        constexpr int kW = tile_w(A);
        // ---- A: A-point DFT over n1 at rows R n1 + n2, times W_N^(n2 k1)
        for (int n2 = tid / kW; n2 < R; n2 += kThreads / kW) {
          float2 v[A];
#pragma unroll
          for (int r = 0; r < A; ++r) {
            v[r] = S[(R * r + n2) * kW + c];
            v[r].y *= sgn;
          }
          Butterfly<A, false>::run(v, tw, kN);
#pragma unroll
          for (int r = 1; r < A; ++r) v[r] = cmul(v[r], tw[r * n2]);
#pragma unroll
          for (int r = 0; r < A; ++r) S[(R * r + n2) * kW + c] = v[r];
        }
        __syncthreads();
        // ---- B: R-point DFT over n2 at rows R k1 + n2 -> rows k1 + A k2 of T
        auto mid = [&](int k1) {
          float2 v[R];
#pragma unroll
          for (int r = 0; r < R; ++r) v[r] = S[(R * k1 + r) * kW + c];
          Butterfly<R, false>::run(v, tw, kN);
          if (live) {
#pragma unroll
            for (int r = 0; r < R; ++r) out[(long long)(k1 + A * r) * cols] = make_float2(v[r].x, v[r].y * sgn);
          }
        };
        if constexpr (A <= kThreads / kW) {   // one round
          if (tid < A * kW) mid(tid / kW);
        } else {
          for (int k1 = tid / kW; k1 < A; k1 += kThreads / kW) mid(k1);
        }
      }
    };
    if constexpr (kEight) {
      steps(std::integral_constant<int, 8>{});
    } else switch (A_) {
#define ODT_Y_CASE(k) \
  case k: steps(std::integral_constant<int, k>{}); break;
      ODT_Y_CASE(2) ODT_Y_CASE(3) ODT_Y_CASE(4) ODT_Y_CASE(5) ODT_Y_CASE(6) ODT_Y_CASE(7)
      ODT_Y_CASE(9) ODT_Y_CASE(10) ODT_Y_CASE(11) ODT_Y_CASE(12) ODT_Y_CASE(13) ODT_Y_CASE(14) ODT_Y_CASE(15)
      ODT_Y_CASE(16)
#undef ODT_Y_CASE
      default: break;
    }
    // the next iteration's copy refills the stage just read
    __syncthreads();
  }
#endif
}

template <int R, bool kEight>
cudaError_t launch_one(const BornArgs& a, bool inverse, const DevFft& f, int* fault, cudaStream_t s) {
  const int W = tile_w(a.py / R);
  const ZSmem L(a.py, W);
  cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(y_pass_kernel<R, kEight>), L.total);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0, per_sm = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, y_pass_kernel<R, kEight>, kThreads, L.total);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  CUtensorMap map{};
  // rows that are no multiple of 16 bytes cannot be mapped: 8-byte copies
  const int use_tma = a.px % 2 == 0;
  const long long nb = (long long)a.pz * a.nbatch;
  if (use_tma && !make_map(a.T, a.px, a.py, nb, W, &map)) return cudaErrorInvalidValue;
  const int nxt = (a.px + W - 1) / W;
  const long long ntiles = nxt * nb, cap = (long long)per_sm * nsm;
  y_pass_kernel<R, kEight><<<(unsigned)(ntiles < cap ? ntiles : cap), kThreads, L.total, s>>>(
      map, a.T, a.px, inverse ? -1.f : 1.f, a.wait_limit, f.tw, a.py / R, use_tma, nxt, (int)ntiles, fault);
  return cudaGetLastError();
}
}  // namespace

// instantiated in one of the object files below
template <int R>
cudaError_t y_pass_launch(const BornArgs& a, bool inverse, const DevFft& f, int* fault, cudaStream_t s) {
  if constexpr (R >= 8)
    if (a.py == 8 * R) return launch_one<R, true>(a, inverse, f, fault, s);
  return launch_one<R, false>(a, inverse, f, fault, s);
}
#define ODT_Y_LIST(X)                                                                                     \
  X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(17) X(18) X(19) X(20) \
  X(21) X(22) X(23) X(24) X(25) X(26) X(27) X(28) X(29) X(30) X(31)
#define ODT_Y_EXTERN(r) \
  extern template cudaError_t y_pass_launch<r>(const BornArgs&, bool, const DevFft&, int*, cudaStream_t);
#define ODT_Y_HERE(r) \
  template cudaError_t y_pass_launch<r>(const BornArgs&, bool, const DevFft&, int*, cudaStream_t);
ODT_Y_LIST(ODT_Y_EXTERN)
#if ODT_YG == 0
ODT_Y_HERE(31) ODT_Y_HERE(20) ODT_Y_HERE(18) ODT_Y_HERE(9) ODT_Y_HERE(2)
#elif ODT_YG == 1
ODT_Y_HERE(29) ODT_Y_HERE(22) ODT_Y_HERE(21) ODT_Y_HERE(12) ODT_Y_HERE(3)
#elif ODT_YG == 2
ODT_Y_HERE(23) ODT_Y_HERE(24) ODT_Y_HERE(16) ODT_Y_HERE(14) ODT_Y_HERE(4)
#elif ODT_YG == 3
ODT_Y_HERE(19) ODT_Y_HERE(26) ODT_Y_HERE(15) ODT_Y_HERE(11) ODT_Y_HERE(5)
#elif ODT_YG == 4
ODT_Y_HERE(17) ODT_Y_HERE(25) ODT_Y_HERE(28) ODT_Y_HERE(8) ODT_Y_HERE(6)
#else
ODT_Y_HERE(13) ODT_Y_HERE(27) ODT_Y_HERE(30) ODT_Y_HERE(10) ODT_Y_HERE(7)
#endif

#if ODT_YG == 0
bool y_pass_supported(const BornArgs& a, const DevFft& f) {
  if (f.plan.n != a.py || a.py > kMaxN || a.storage || !z_split(a.py) || !encoder()) return false;
  return ((long long)a.px + 15) / 16 * a.pz * a.nbatch < (1LL << 31);
}

cudaError_t launch_y_pass(const BornArgs& a, bool inverse, const DevFft& fy, int* fault, cudaStream_t s) {
  const int A = z_split(a.py);
  if (!A) return cudaErrorNotSupported;
  switch (a.py / A) {
#define ODT_Y_CASE(r) \
  case r: return y_pass_launch<r>(a, inverse, fy, fault, s);
    ODT_Y_LIST(ODT_Y_CASE)
#undef ODT_Y_CASE
    default: return cudaErrorNotSupported;
  }
}
#endif  // ODT_YG == 0

}  // namespace odt
