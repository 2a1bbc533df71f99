// z-pass of dyadic (vector) solves for any z length n = A R up to 256
// (cols_any.cuh): forward z-FFT of the three field components, the dyadic
// Green's multiply Greenp (delta_ij - corr rads_i rads_j) / N
// (FORWARD_SOLVER_CONVERGENT_BORN.m:596-604) and inverse z-FFT, the transforms
// and the product of born_z_dyadic_kernel (vector.cu).
//
// A CTA takes 16 adjacent columns of all three components into shared memory
// (asynchronous copies, 34 KB at 88 points) and works in place: A-point DFTs
// over n1 with twiddles, R-point DFTs over n2 (z = R n1 + n2, kz = k1 + A k2),
// the product per (kz, column), and the same steps back.  Single stage: with
// several CTAs per SM one's copies overlap the others' steps.  What bounds it:
// the five barriers between the steps.  88^3 padded, 4 illuminations: 0.056 against
// 0.114 ms of the generic tiles (three transforms each way through two work
// tiles of 17 columns, 60 KB per CTA of 128 threads).
#include <type_traits>

#include "cols_any.cuh"

namespace odt {
namespace {

constexpr int kDW = 16;        // columns per tile
constexpr int kDThreads = 192;

struct DSmem {
  size_t tw, kz, rz, col, data, total;
  __host__ __device__ explicit DSmem(int n) {
    tw = 0;
    kz = a16(sizeof(float2) * n);
    rz = kz + a16(sizeof(float) * n);
    col = rz + a16(sizeof(float) * n);
    data = col + a16(3 * sizeof(float) * kDW);
    total = data + 3 * sizeof(float2) * n * kDW;
  }
};

template <int R>
__global__ void __launch_bounds__(kDThreads, R <= 16 ? 4 : R <= 23 ? 3 : 2)
    z_dyadic_kernel(const BornArgs a, const DyadArgs d, const int jj, const float2* __restrict__ twg, const int A_,
                    const int wide, const int nxt, const int ntiles) {
#if defined(__CUDA_ARCH__)
  const int N = A_ * R;
  const DSmem L(N);
  extern __shared__ __align__(16) unsigned char sm[];
  float2* tw = reinterpret_cast<float2*>(sm + L.tw);
  float* kz = reinterpret_cast<float*>(sm + L.kz);
  float* rz = reinterpret_cast<float*>(sm + L.rz);
  float* col = reinterpret_cast<float*>(sm + L.col);   // kq2 x + y, rads x, rads y per column
  float2* S = reinterpret_cast<float2*>(sm + L.data);  // [component][row][column]
  const int tid = threadIdx.x;
  const int c = tid & (kDW - 1);
  const bool flip = a.acyclic && (jj & 1);
  for (int i = tid; i < N; i += kDThreads) {
    const int iz = flip ? (i == 0 ? 0 : N - i) : i;
    tw[i] = twg[i];
    kz[i] = a.kq2[2][iz];
    rz[i] = d.rad[2][iz];
  }
  const int pxy = a.px * a.py;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int i0 = kDW * (tile % nxt), b = tile / nxt;
    const float2* const src = a.T + 3LL * b * a.nvox;
    if (wide) {   // even planes: 16-byte copies (a plane's last pair is whole)
      for (int i = tid; i < 3 * N * (kDW / 2); i += kDThreads) {
        const int h = i & (kDW / 2 - 1), q = i / (kDW / 2);
        const int comp = q / N, r = q - comp * N;
        const int cc = min(i0 + 2 * h, pxy - 2);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(S + q * kDW + 2 * h)),
                     "l"(src + comp * a.nvox + (long long)r * pxy + cc)
                     : "memory");
      }
    } else {
      const int cc = min(i0 + c, pxy - 1);   // columns past the plane repeat the last one; not stored
      for (int q = tid / kDW; q < 3 * N; q += kDThreads / kDW) {
        const int comp = q / N, r = q - comp * N;
        copy8(S + q * kDW + c, src + comp * a.nvox + (long long)r * pxy + cc);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (tid < kDW) {
      const int i = min(i0 + tid, pxy - 1);
      int y = i / a.px, kx = i - y * a.px;
      if (a.perm_xy) {   // position Rx k1 + k2 holds spectral index k1 + 8 k2
        const int rx = a.px >> 3, ry = a.py >> 3;
        kx = kx / rx + 8 * (kx % rx);
        y = y / ry + 8 * (y % ry);
      }
      const int ix = flip ? (kx == 0 ? 0 : a.px - kx) : kx;
      const int iy = flip ? (y == 0 ? 0 : a.py - y) : y;
      col[tid] = a.kq2[0][ix] + a.kq2[1][iy];
      col[kDW + tid] = d.rad[0][ix];
      col[2 * kDW + tid] = d.rad[1][iy];
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float2* const out = a.T + 3LL * b * a.nvox + i0 + c;
    const bool live = i0 + c < pxy;
    auto steps = [&](auto Ac) {
      constexpr int A = decltype(Ac)::value;
      if constexpr (ZSplit<A * R>::kA == A) {
        constexpr int kN = A * R;
        constexpr int kStep = kDThreads / kDW;
        // ---- A-point DFTs over n1 at rows R n1 + n2, times W_N^(n2 k1)
        for (int q = tid / kDW; q < 3 * R; q += kStep) {
          const int comp = q / R, n2 = q - comp * R;
          float2* const D = S + comp * (kN * kDW) + c;
          float2 v[A];
#pragma unroll
          for (int r = 0; r < A; ++r) v[r] = D[(R * r + n2) * kDW];
          Butterfly<A, false>::run(v, tw, kN);
#pragma unroll
          for (int r = 1; r < A; ++r) v[r] = cmul(v[r], tw[r * n2]);
#pragma unroll
          for (int r = 0; r < A; ++r) D[(R * r + n2) * kDW] = v[r];
        }
        __syncthreads();
        // ---- R-point DFTs over n2: row R k1 + k2 holds kz = k1 + A k2
        for (int q = tid / kDW; q < 3 * A; q += kStep) {
          float2* const D = S + q * (R * kDW) + c;   // comp kN + R k1 rows down
          float2 v[R];
#pragma unroll
          for (int r = 0; r < R; ++r) v[r] = D[r * kDW];
          Butterfly<R, false>::run(v, tw, kN);
#pragma unroll
          for (int r = 0; r < R; ++r) D[r * kDW] = v[r];
        }
        __syncthreads();
        // ---- Greenp (delta_ij - corr rads_i rads_j) / N
        for (int row = tid / kDW; row < kN; row += kStep) {
          const int k1 = row / R, iz = k1 + A * (row - R * k1);
          float q = col[c] + kz[iz];
          q = a.g_scale * q - a.g_off;
          const float rden = __frcp_rn(q * q + a.eps * a.eps);
          const float2 G = make_float2(q * rden, a.eps * rden);  // Greenp = 1 / (q - i eps)
          const float rd[3] = {col[kDW + c], col[2 * kDW + c], rz[iz]};
          float2* const D = S + row * kDW + c;
          float2 v[3];
#pragma unroll
          for (int j = 0; j < 3; ++j) v[j] = D[j * (kN * kDW)];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const float2 ci = cscale(d.absorb, rd[i]);  // corr * rads_i
            float2 acc = make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              float2 e = cscale(ci, -rd[j]);
              if (i == j) e.x += 1.f;
              const float2 t = cmul(cmul(G, e), v[j]);
              acc = j ? cadd(acc, t) : t;
            }
            D[i * (kN * kDW)] = cscale(acc, a.inv_n);
          }
        }
        __syncthreads();
        // ---- and back
        for (int q = tid / kDW; q < 3 * A; q += kStep) {
          const int k1 = q % A;
          float2* const D = S + q * (R * kDW) + c;
          float2 v[R];
#pragma unroll
          for (int r = 0; r < R; ++r) v[r] = D[r * kDW];
          Butterfly<R, true>::run(v, tw, kN);
#pragma unroll
          for (int r = 1; r < R; ++r) v[r] = cmul(v[r], cconj(tw[r * k1]));
#pragma unroll
          for (int r = 0; r < R; ++r) D[r * kDW] = v[r];
        }
        __syncthreads();
        for (int q = tid / kDW; q < 3 * R; q += kStep) {
          const int comp = q / R, n2 = q - comp * R;
          const float2* const D = S + comp * (kN * kDW) + c;
          float2 v[A];
#pragma unroll
          for (int r = 0; r < A; ++r) v[r] = D[(R * r + n2) * kDW];
          Butterfly<A, true>::run(v, tw, kN);
          if (live) {
#pragma unroll
            for (int r = 0; r < A; ++r) out[comp * a.nvox + (long long)(R * r + n2) * pxy] = v[r];
          }
        }
      }
    };
    switch (A_) {
#define ODT_D_CASE(k) \
  case k: steps(std::integral_constant<int, k>{}); break;
      ODT_D_CASE(2) ODT_D_CASE(3) ODT_D_CASE(4) ODT_D_CASE(5) ODT_D_CASE(6) ODT_D_CASE(7) ODT_D_CASE(8)
      ODT_D_CASE(9) ODT_D_CASE(10) ODT_D_CASE(11) ODT_D_CASE(12) ODT_D_CASE(13) ODT_D_CASE(14) ODT_D_CASE(15)
      ODT_D_CASE(16)
#undef ODT_D_CASE
      default: break;
    }
    __syncthreads();   // the next tile's copies overwrite the rows just read
  }
#endif
}

}  // namespace

// instantiated in one of the object files below
template <int R>
cudaError_t z_dyadic_launch(const BornArgs& a, const DyadArgs& d, int jj, const DevFft& f, cudaStream_t s) {
  const DSmem L(a.pz);
  cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(z_dyadic_kernel<R>), L.total);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0, per_sm = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, z_dyadic_kernel<R>, kDThreads, L.total);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  const int nxt = (a.px * a.py + kDW - 1) / kDW;
  const int ntiles = nxt * (a.nbatch / 3), cap = per_sm * nsm;
  z_dyadic_kernel<R><<<ntiles < cap ? ntiles : cap, kDThreads, L.total, s>>>(
      a, d, jj, f.tw, a.pz / R, (long long)a.px * a.py % 2 == 0, nxt, ntiles);
  return cudaGetLastError();
}

#define ODT_D_LIST(X)                                                                                     \
  X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(17) X(18) X(19) X(20) \
  X(21) X(22) X(23) X(24) X(25) X(26) X(27) X(28) X(29) X(30) X(31)
#define ODT_D_EXTERN(r) \
  extern template cudaError_t z_dyadic_launch<r>(const BornArgs&, const DyadArgs&, int, const DevFft&, cudaStream_t);
#define ODT_D_HERE(r) \
  template cudaError_t z_dyadic_launch<r>(const BornArgs&, const DyadArgs&, int, const DevFft&, cudaStream_t);
ODT_D_LIST(ODT_D_EXTERN)
#if ODT_DG == 0
ODT_D_HERE(31) ODT_D_HERE(20) ODT_D_HERE(18) ODT_D_HERE(9) ODT_D_HERE(2)
#elif ODT_DG == 1
ODT_D_HERE(29) ODT_D_HERE(22) ODT_D_HERE(21) ODT_D_HERE(12) ODT_D_HERE(3)
#elif ODT_DG == 2
ODT_D_HERE(23) ODT_D_HERE(24) ODT_D_HERE(16) ODT_D_HERE(14) ODT_D_HERE(4)
#elif ODT_DG == 3
ODT_D_HERE(19) ODT_D_HERE(26) ODT_D_HERE(15) ODT_D_HERE(11) ODT_D_HERE(5)
#elif ODT_DG == 4
ODT_D_HERE(17) ODT_D_HERE(25) ODT_D_HERE(28) ODT_D_HERE(8) ODT_D_HERE(6)
#else
ODT_D_HERE(13) ODT_D_HERE(27) ODT_D_HERE(30) ODT_D_HERE(10) ODT_D_HERE(7)
#endif

#if ODT_DG == 0
bool z_dyadic_supported(const BornArgs& a, const DevFft& f, int max_smem) {
  if (f.plan.n != a.pz || a.pz > kMaxN || a.storage || a.nbatch % 3 != 0 || !z_split(a.pz)) return false;
  const long long pxy = (long long)a.px * a.py;
  return pxy < (1 << 30) && DSmem(a.pz).total <= (size_t)max_smem && (pxy + 15) / 16 * a.nbatch < (1LL << 31);
}

cudaError_t launch_z_dyadic(const BornArgs& a, const DyadArgs& d, int jj, const DevFft& fz, cudaStream_t s) {
  const int A = z_split(a.pz);
  if (!A) return cudaErrorNotSupported;
  switch (a.pz / A) {
#define ODT_D_CASE(r) \
  case r: return z_dyadic_launch<r>(a, d, jj, fz, s);
    ODT_D_LIST(ODT_D_CASE)
#undef ODT_D_CASE
    default: return cudaErrorNotSupported;
  }
}
#endif  // ODT_DG == 0

}  // namespace odt
