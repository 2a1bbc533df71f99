// Transforms along an axis of length n = q p with a prime p > 31 (such as 127,
// 89, 202 = 2 * 101): with z = p n1 + n2 and
// k = k1 + q k2, q-point butterflies over n1 with twiddles, then per k1 the
// p-point DFT over n2 in the symmetric form
//   C_k = x_0 + sum_j s_j cos(2 pi j k / p),   S_k = sum_j d_j sin(2 pi j k / p),
//   X_k = C_k -/+ i S_k,   X_(p-k) = C_k +/- i S_k,
// s_j = x_j + x_(p-j), d_j = x_j - x_(p-j), j, k <= h = (p - 1) / 2: two real
// h x h matrices times the tile's columns, h^2 / p real multiply-adds per
// value and matrix.  A thread keeps 8 values of k for 2 pencils (64
// accumulators) and reads the next j's 16 coefficients (through L1, the same
// for a whole warp) and 4 inputs while this one's 64 multiply-adds run.  The
// z-pass runs both directions on one visit of the tile: a thread holds X_k and
// X_(p-k) and multiplies them by the Green's function on the way back to
// shared memory.
//
// What bounds it: issue latency at 16 warps per SM (128 registers); in the
// z-pass the FMA pipe is busy 55 % and the issue slots 57 %.  The coefficients
// in shared memory and a second landing stage (8 warps per SM) measured 0.38 ms,
// one stage with 4 pencils per thread 0.34 with half the speed for q > 1, pairs of k
// in the packed multiply-adds 0.40, against 0.34 ms for a 127-point axis of
// 16 x 127^3 as it stands.  One Bluestein kernel per axis and direction (two transforms of
// m >= 2 p - 1 points and two chirps through shared memory) took 0.58 ms, and
// the z-pass as two of those and a separate product 1.34 against 0.60 ms.
//
// Rounding of a sum of h FP32 products grows with p; Bluestein's hardly does.
// Measured per axis on random data against double precision: 0.9e-7 (p = 37),
// 1.3e-7 (89), 1.5e-7 (127) in one sum, but 1.6e-7 (151), 1.9e-7 (211), 2.1e-7
// (251); Bluestein's transforms 1.8e-7 to 2.5e-7 on the device, 1.5e-7 to 1.8e-7
// with ideal inner transforms.  Above p = 139 the sums therefore run in two
// halves: 1.2e-7 (151), 1.4e-7 (211), 1.55e-7 (251), for 3 to 14 % of the axis's time
// (20 M points, lines and columns: 151 points 0.280 -> 0.289 and 0.252 -> 0.287 ms, 251
// points 0.365 -> 0.387 and 0.324 -> 0.351) and 12 to 21 % of a z-pass's, which holds two
// such sums (36 x 40 x 149, 8 waves: 0.054 -> 0.060 ms, x 251: 0.116 -> 0.140).  FP32 throughout; tcgen05 has no FP32
// multiply, and its TF32 form would need the operands in three parts.
#include <cmath>
#include <type_traits>

#include "fft_core.cuh"
#include "prime_pass.cuh"
#include "tile_launch.cuh"
#include "tma.cuh"

namespace odt {
namespace {

constexpr int kKT = 8, kCT = 2;       // values of k, pencils per thread
constexpr int kMaxThreads = 256;
constexpr int kMaxQ = 13;
// largest prime whose rounding and speed were measured.  The work per value grows
// with p, but has not met Bluestein's there: y axis of a 36 x n x 36 grid of 8
// waves, Bluestein against direct, ms per launch: 0.063, 0.031 (n = 127), 0.079, 0.051
// (151), 0.131, 0.062 (211), 0.130, 0.071 (251, in one sum; 0.077 in two halves)
constexpr int kMaxP = 251;
constexpr int kSplitP = 139;          // above it the sums run in two halves

__host__ __device__ inline int pitch_of(int w, bool lines) { return lines ? w + 2 : w; }

size_t smem_of(const PrimePlan& f, int w) {   // lines: the larger pitch
  return align16(sizeof(float2) * f.n) + align16(sizeof(float) * f.n) + align16(sizeof(float) * w) +
         sizeof(float2) * (size_t)f.n * pitch_of(w, true);
}

int items_of(const PrimePlan& f, int w) { return f.kp / kKT * f.q * (w / kCT); }

struct AxisArgs {
  float2* x;
  long long n0, n2;       // columns: [n0, n, n2]; lines: n2 lines
  long long ntiles;
  int inv, sh;
  float scale;
};

// OP 0: one transform; 1: forward, Green's multiply, inverse (columns)
// (HALVES: the sums over j in two parts, see kSplitP)
template <bool LINES, int OP, bool HALVES>
__global__ void __launch_bounds__(kMaxThreads, 2) prime_kernel(const AxisArgs g, const PrimePlan f, const BornArgs a,
                                                            const int jj) {
  extern __shared__ __align__(16) unsigned char sm[];
  const int n = f.n, q = f.q, p = f.p, h = f.h, kp = f.kp, W = f.w;
  const int pitch = pitch_of(W, LINES);
  const float* tc = f.tab;
  const float* ts = tc + (size_t)h * kp;
  float2* tw = reinterpret_cast<float2*>(sm);
  float* kz = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(tw) + align16(sizeof(float2) * n));
  float* gxy = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(kz) + align16(sizeof(float) * n));
  float2* D = reinterpret_cast<float2*>(reinterpret_cast<unsigned char*>(gxy) + align16(sizeof(float) * W));
  const int tid = threadIdx.x, nthr = blockDim.x;
  const bool flip = OP == 1 && a.acyclic && (jj & 1);
  for (int i = tid; i < n; i += nthr) {
    tw[i] = f.tw[i];
    if (OP == 1) kz[i] = a.kq2[2][flip ? (i == 0 ? 0 : n - i) : i];
  }
  // this thread's products: pencils c0 and c0 + W/2 (adjacent threads read and
  // write adjacent pencils) of sub-block blk, k0 .. k0+7
  const int ncg = W / kCT;
  const int c0 = tid % ncg, blk = tid / ncg % q, k0 = kKT * (tid / ncg / q);
  const bool active = k0 < kp;
  const long long ntx = LINES ? 1 : (g.n0 + W - 1) / W;
  const long long rs = LINES ? 1 : g.n0, cst = LINES ? n : 1;   // strides of rows and pencils

  // (r, c) of this thread's items, r < rows: the index that is contiguous in
  // global memory runs fastest over the threads (a multiple of W of them)
  auto first = [&](int rows, int& r, int& c) {
    if (LINES) {
      c = tid / rows;
      r = tid - c * rows;
    } else {
      r = tid / W;
      c = tid - r * W;
    }
  };
  auto advance = [&](int rows, int& r, int& c) {
    if (LINES) {
      for (r += nthr; r >= rows; r -= rows) ++c;
    } else {
      r += nthr / W;
    }
  };
  auto more = [&](int rows, int r, int c) { return LINES ? c < W : r < rows; };
  auto pos = [&](int row) {   // centred transforms gather and scatter shifted rows
    const int r = row + g.sh;
    return (long long)(r >= n ? r - n : r);
  };
  // tile t: live pencils, address of its first element
  auto locate = [&](long long t, int& np, long long& i0) {
    const long long o = LINES ? 0 : t / ntx;
    i0 = LINES ? t * W : (t - o * ntx) * W;
    np = (int)min((long long)W, (LINES ? g.n2 : g.n0) - i0);
    return g.x + (LINES ? i0 * n : o * g.n0 * n + i0);
  };
  // asynchronous copy of tile t into a stage; dead pencils become zeros
  auto fetch = [&](long long t, float2* dst) {
    int np, r, c;
    long long i0;
    const float2* src = locate(t, np, i0);
    for (first(n, r, c); more(n, r, c); advance(n, r, c)) {
      const int live = c < np ? 8 : 0;
      const float2* from = live ? src + pos(r) * rs + c * cst : src;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                       (unsigned)__cvta_generic_to_shared(dst + r * pitch + c)),
                   "l"(from), "r"(live)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (long long t = blockIdx.x; t < g.ntiles; t += gridDim.x) {
    int np;
    long long i0;
    float2* const base = locate(t, np, i0);
    if (OP == 1 && tid < W) {
      const int i = (int)min(i0 + tid, g.n0 - 1);
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
    fetch(t, D);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // ---- q-point butterflies over n1 with twiddles, in place
    if (q > 1) {
      auto qsteps = [&](auto qc) {
        constexpr int Q = decltype(qc)::value;
        for (int i = tid; i < p * W; i += nthr) {
          const int n2 = i / W, c = i - n2 * W;
          float2 v[Q];
#pragma unroll
          for (int r = 0; r < Q; ++r) v[r] = D[(p * r + n2) * pitch + c];
          if (OP == 0 && g.inv) Butterfly<Q, true>::run(v, tw, n);
          else Butterfly<Q, false>::run(v, tw, n);
#pragma unroll
          for (int r = 0; r < Q; ++r) {
            float2 w = tw[r * n2];
            if (OP == 0 && g.inv) w.y = -w.y;
            D[(p * r + n2) * pitch + c] = r ? cmul(v[r], w) : v[r];
          }
        }
      };
      switch (q) {
#define ODT_Q(k) \
  case k: qsteps(std::integral_constant<int, k>{}); break;
        ODT_Q(2) ODT_Q(3) ODT_Q(4) ODT_Q(5) ODT_Q(6) ODT_Q(7) ODT_Q(8) ODT_Q(9) ODT_Q(10) ODT_Q(11) ODT_Q(12)
        ODT_Q(13)
#undef ODT_Q
        default: break;
      }
      __syncthreads();
    }

    // ---- the p-point DFTs: C = x_0 + cos . s, S = sin . d
    float2 C[kKT][kCT], S[kKT][kCT];
    const float2* const Db = D + p * blk * pitch + c0;
    auto product = [&] {
      if (!active) return;
#pragma unroll
      for (int c = 0; c < kCT; ++c) {
        const float2 x0 = Db[c * ncg];
#pragma unroll
        for (int k = 0; k < kKT; ++k) {
          C[k][c] = x0;
          S[k][c] = make_float2(0.f, 0.f);
        }
      }
      const float* pc = tc + k0;
      const float* ps = ts + k0;
      const float2* pu = Db + pitch;
      const float2* pv = Db + (p - 1) * pitch;
      // operands of the next j are read while this one's products run (past the
      // last j: rows and table entries that exist but are not used)
      float4 cc[2], ss[2];
      float2 x[kCT], y[kCT];
      auto read = [&] {
        cc[0] = __ldg(reinterpret_cast<const float4*>(pc));
        cc[1] = __ldg(reinterpret_cast<const float4*>(pc + 4));
        ss[0] = __ldg(reinterpret_cast<const float4*>(ps));
        ss[1] = __ldg(reinterpret_cast<const float4*>(ps + 4));
#pragma unroll
        for (int c = 0; c < kCT; ++c) {
          x[c] = pu[c * ncg];
          y[c] = pv[c * ncg];
        }
        pc += kp;
        ps += kp;
        pu += pitch;
        pv -= pitch;
      };
      read();
      auto sum = [&](int n) {
#pragma unroll 2
        for (int j = 0; j < n; ++j) {
          const float ck[kKT] = {cc[0].x, cc[0].y, cc[0].z, cc[0].w, cc[1].x, cc[1].y, cc[1].z, cc[1].w};
          const float sk[kKT] = {ss[0].x, ss[0].y, ss[0].z, ss[0].w, ss[1].x, ss[1].y, ss[1].z, ss[1].w};
          float2 u[kCT], v[kCT];
#pragma unroll
          for (int c = 0; c < kCT; ++c) {
            u[c] = cadd(x[c], y[c]);
            v[c] = csub(x[c], y[c]);
          }
          read();
#pragma unroll
          for (int k = 0; k < kKT; ++k)
#pragma unroll
            for (int c = 0; c < kCT; ++c) {
              C[k][c] = cfma_real(ck[k], u[c], C[k][c]);
              S[k][c] = cfma_real(sk[k], v[c], S[k][c]);
            }
        }
      };
      if constexpr (!HALVES) {
        sum(h);
      } else {
        // the first half's sums wait in local memory (64 stores and loads a
        // thread; volatile, or the compiler keeps both halves in registers and
        // spills inside the loop)
        volatile float part[4 * kKT * kCT];
        sum(h / 2);
#pragma unroll
        for (int k = 0; k < kKT; ++k)
#pragma unroll
          for (int c = 0; c < kCT; ++c) {
            const int i = 4 * (k * kCT + c);
            part[i] = C[k][c].x;
            part[i + 1] = C[k][c].y;
            part[i + 2] = S[k][c].x;
            part[i + 3] = S[k][c].y;
            C[k][c] = S[k][c] = make_float2(0.f, 0.f);
          }
        sum(h - h / 2);
#pragma unroll
        for (int k = 0; k < kKT; ++k)
#pragma unroll
          for (int c = 0; c < kCT; ++c) {
            const int i = 4 * (k * kCT + c);
            C[k][c] = make_float2(C[k][c].x + part[i], C[k][c].y + part[i + 1]);
            S[k][c] = make_float2(S[k][c].x + part[i + 2], S[k][c].y + part[i + 3]);
          }
      }
    };
    // X_k (m = 0) or X_(p-k) (m = 1) of the products
    auto value = [&](int k, int c, bool m, bool inv) {
      return m != inv ? addrot<true>(C[k][c], S[k][c]) : subrot<true>(C[k][c], S[k][c]);
    };
    product();
    bool inv = OP == 0 && g.inv;
    if constexpr (OP == 1) {
      __syncthreads();
      if (active) {
        auto green = [&](int c, int k2, float2 v) {
          const float qq = a.g_scale * (gxy[c] + kz[blk + q * k2]) - a.g_off;
          const float rden = __frcp_rn(qq * qq + a.eps * a.eps) * a.inv_n;
          return cmul(make_float2(qq * rden, a.eps * rden), v);
        };
#pragma unroll
        for (int k = 0; k < kKT; ++k) {
          if (k0 + k > h) continue;
#pragma unroll
          for (int c = 0; c < kCT; ++c) {
            const float2 u = green(c0 + c * ncg, k0 + k, value(k, c, false, false));
            float2* d = D + p * blk * pitch + c0 + c * ncg;
            if (k0 + k == 0) {
              d[0] = u;
            } else {
              d[(k0 + k) * pitch] = u;
              d[(p - k0 - k) * pitch] = green(c0 + c * ncg, p - k0 - k, value(k, c, true, false));
            }
          }
        }
      }
      __syncthreads();
      product();
      inv = true;
    }
    auto store = [&](int row, int c, float2 v) {
      if (c < np) base[pos(row) * rs + c * cst] = g.scale == 1.f ? v : cscale(v, g.scale);
    };
    // ---- results: with one transform value k2 of sub-block k1 is row
    // k1 + q k2; after the z-pass's inverse it is the sum over k2 at n2, whose
    // q values over k1 the last butterflies combine into rows p n1 + n2
    if (OP == 0 || q == 1) {
      if (active) {
#pragma unroll
        for (int k = 0; k < kKT; ++k) {
          if (k0 + k > h) continue;
#pragma unroll
          for (int c = 0; c < kCT; ++c) {
            store(blk + q * (k0 + k), c0 + c * ncg, value(k, c, false, inv));
            if (k0 + k > 0) store(blk + q * (p - k0 - k), c0 + c * ncg, value(k, c, true, inv));
          }
        }
      }
    } else {
      __syncthreads();
      if (active) {
#pragma unroll
        for (int k = 0; k < kKT; ++k) {
          const int n2 = k0 + k;
          if (n2 > h) continue;
#pragma unroll
          for (int c = 0; c < kCT; ++c) {
            float2* d = D + p * blk * pitch + c0 + c * ncg;
            d[n2 * pitch] = cmul(value(k, c, false, true), cconj(tw[n2 * blk]));
            if (n2 > 0) d[(p - n2) * pitch] = cmul(value(k, c, true, true), cconj(tw[(p - n2) * blk]));
          }
        }
      }
      __syncthreads();
      auto qback = [&](auto qc) {
        constexpr int Q = decltype(qc)::value;
        int n2, c;
        for (first(p, n2, c); more(p, n2, c); advance(p, n2, c)) {
          float2 v[Q];
#pragma unroll
          for (int r = 0; r < Q; ++r) v[r] = D[(p * r + n2) * pitch + c];
          Butterfly<Q, true>::run(v, tw, n);
#pragma unroll
          for (int r = 0; r < Q; ++r) store(p * r + n2, c, v[r]);
        }
      };
      switch (q) {
#define ODT_Q(k) \
  case k: qback(std::integral_constant<int, k>{}); break;
        ODT_Q(2) ODT_Q(3) ODT_Q(4) ODT_Q(5) ODT_Q(6) ODT_Q(7) ODT_Q(8) ODT_Q(9) ODT_Q(10) ODT_Q(11) ODT_Q(12)
        ODT_Q(13)
#undef ODT_Q
        default: break;
      }
    }
    __syncthreads();   // D's readers, before the next tile's copy
  }
}

template <bool LINES, int OP, bool HALVES>
cudaError_t launch_sums(const AxisArgs& g, const PrimePlan& f, const BornArgs& a, int jj, cudaStream_t s) {
  const size_t sm = smem_of(f, f.w);
  const int unit = f.w > 32 ? f.w : 32;
  const int nthr = (items_of(f, f.w) + unit - 1) / unit * unit;
  cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(prime_kernel<LINES, OP, HALVES>), sm);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0, per_sm = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, prime_kernel<LINES, OP, HALVES>, nthr, sm);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  const long long cap = (long long)per_sm * nsm;
  prime_kernel<LINES, OP, HALVES><<<(unsigned)(g.ntiles < cap ? g.ntiles : cap), nthr, sm, s>>>(g, f, a, jj);
  return cudaGetLastError();
}

template <bool LINES, int OP>
cudaError_t launch(const AxisArgs& g, const PrimePlan& f, const BornArgs& a, int jj, cudaStream_t s) {
  return f.p > kSplitP ? launch_sums<LINES, OP, true>(g, f, a, jj, s) : launch_sums<LINES, OP, false>(g, f, a, jj, s);
}

}  // namespace

PrimePlan prime_plan(int n, size_t max_smem) {
  PrimePlan f;
  int p = 1, r = n;
  for (int d = 2; d <= r; ++d)
    while (r % d == 0) {
      p = d;
      r /= d;
    }
  if (n < 37 || p <= 31 || p > kMaxP || n / p > kMaxQ) return PrimePlan{};
  f.n = n;
  f.p = p;
  f.q = n / p;
  f.h = (p - 1) / 2;
  f.kp = kKT * ((f.h + kKT) / kKT);
  // the widest tile whose products fit the threads, with room for four CTAs
  // per SM if there is one, else fewer
  for (const size_t room : {max_smem / 4 - 1024, max_smem / 2 - 1024, max_smem})
    for (int w : {64, 32, 16})
      if (items_of(f, w) <= kMaxThreads && smem_of(f, w) <= room) {
        f.w = w;
        return f;
      }
  return PrimePlan{};
}

void prime_table(const PrimePlan& f, float* tab) {
  for (int j = 1; j <= f.h; ++j)
    for (int k = 0; k < f.kp; ++k) {
      const double t = 6.283185307179586476925286766559 * (double)((long long)j * k % f.p) / (double)f.p;
      tab[(size_t)(j - 1) * f.kp + k] = k <= f.h ? (float)std::cos(t) : 0.f;
      tab[(size_t)(f.h + j - 1) * f.kp + k] = k <= f.h ? (float)std::sin(t) : 0.f;
    }
}

cudaError_t launch_prime_axis(float2* x, int n0, long long n2, bool inv, int sh, float scale, const PrimePlan& f,
                              cudaStream_t s) {
  if (!f.q || n0 < 1 || n2 < 1) return cudaErrorInvalidValue;
  AxisArgs g{x, n0, n2, 0, inv ? 1 : 0, sh, scale};
  if (n0 == 1) {
    g.ntiles = (n2 + f.w - 1) / f.w;
    return launch<true, 0>(g, f, BornArgs{}, 0, s);
  }
  g.ntiles = ((long long)n0 + f.w - 1) / f.w * n2;
  return launch<false, 0>(g, f, BornArgs{}, 0, s);
}

cudaError_t launch_prime_z(const BornArgs& a, int jj, const PrimePlan& f, cudaStream_t s) {
  if (f.n != a.pz || !f.q || a.storage) return cudaErrorInvalidValue;
  AxisArgs g{a.T, (long long)a.px * a.py, a.nbatch, 0, 0, 0, 1.f};
  g.ntiles = (g.n0 + f.w - 1) / f.w * g.n2;
  return launch<false, 1>(g, f, a, jj, s);
}

}  // namespace odt
