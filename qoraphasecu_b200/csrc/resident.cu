// Resident iteration kernel for square 2D problems of side N = 64, 128, 256.
//
// One start lives in a cluster of C CTAs; CTA `rank` owns rows
// [rank R, rank R + R) of the start and as many columns (R = N / C). For a
// whole chunk of iterations it keeps
//   in registers      the iterate's rows, their support bits, the amplitudes of
//                     its columns and (where the budget allows) its twiddles;
//   in shared memory  cs and ws, its columns and its rows as they arrive: N x Q
//                     complex64 (element of the line first, Q >= R a padded
//                     pitch), and the lines' exchange rows,
// so an iteration reads nothing from HBM or L2. It is the same sequence as
// the streamed passes (src/cuda/cuda_solver.cu:395-399 and kernels.cu:96-168
// of the reference): rows transformed along x are stored to their columns'
// owners through distributed shared memory; after a cluster barrier each CTA
// transforms its columns, applies the modulus projection and the Fourier-
// error sum, transforms back and stores the columns to their rows' owners;
// after a second barrier it transforms its rows back along x (= P_M x),
// applies the update x <- S ? P : a x + b P and transforms the new iterate
// forward. The chunk starts from x and ends by writing x and w = FFT_x(x) to
// HBM, which keeps the invariant of the streamed passes: shrinkwrap, detwin
// and results work on the HBM copies between chunks.
//
// Bound: the serial chain of an iteration (two transforms, the projection and
// two barriers each way round), not bandwidth: few starts leave most SMs idle,
// so a launch takes the largest cluster at which all of its starts are
// resident at once, one CTA per SM (resident_cluster). Both phases store to
// remote memory and load from their own, so no load waits for another SM; the
// threads of a line store to neighbouring slots (scattered 8-byte stores took
// 12.7 us an iteration at 256 x 256 in clusters of 16). A line's threads share
// a warp in both phases, so the Stockham exchanges need warp barriers only,
// and the error sum is a warp reduction with one atomic.
//
// Measured, an iteration of all starts (before: 1, 2 and 8 CTAs a start with
// everything in shared memory and the amplitude read from L2 in every
// iteration): 64 x 64, 8 starts 5.0 -> 2.1 us; 128 x 128, 4 starts 12.9 -> 3.8;
// 256 x 256, 4 starts 15.2 -> 7.7 (streamed passes: 7.4, 7.4 and 8.2 us).
//
// No thread waits on anything but hardware barriers that every thread of the
// cluster reaches the same number of times (the loop count is uniform), and
// no CTA touches another CTA's shared memory before the first or after the
// last cluster barrier.

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <map>
#include <mutex>
#include <stdexcept>
#include <type_traits>
#include <utility>
#include <vector>

#include "bulk_copy.cuh"
#include "cluster_share.hpp"
#include "line_fft.cuh"
#include "projection.cuh"
#include "reduce.cuh"
#include "resident.cuh"

namespace qpb {

namespace {

template <int N, int C_>
struct Resident {
  using G = Geometry<N>;
  static constexpr int C = C_;
  static constexpr int E = G::E;
  static constexpr int T = G::T;
  static constexpr int R = N / C;  // rows and columns per CTA
  static constexpr int NT = R * T;
  static constexpr int P = G::PITCH;
  // Pitch of cs and ws: a half-warp reads T elements (Q apart) of 16 / T
  // neighbouring lines, on different banks for Q odd (T = 16) or 2 mod 16 (T = 8).
  static constexpr int Q = T == 16 ? (R | 1) : R + ((2 - R) % 16 + 16) % 16;
  static constexpr int kBytes = (2 * N * Q + R * P) * 8;
  // 256-point lines in CTAs of 512 threads leave 128 registers a thread, which
  // hold the iterate and the amplitudes but not the twiddles too.
  static constexpr bool kTwiddlesHeld = N < 256 || NT <= 256;
  static_assert(G::STAGES == 2 && G::R0 == E, "one butterfly a thread in the first stage");
  static_assert(NT % 32 == 0 && NT <= 1024 && 32 % T == 0, "whole lines per warp, whole warps");
  static_assert(kBytes + 512 <= 227 * 1024, "shared memory");
};

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// Every thread of every CTA of the cluster arrives; shared-memory writes
// before it (local and remote) are visible to every thread after it.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile(
      "barrier.cluster.arrive.release.aligned;\n\t"
      "barrier.cluster.wait.acquire.aligned;" ::
          : "memory");
}

// Address in CTA `rank`'s shared memory of the same offset as `local`.
__device__ __forceinline__ unsigned cluster_map(unsigned local, unsigned rank) {
  unsigned remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  return remote;
}

__device__ __forceinline__ void store_cluster(unsigned addr, float2 v) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y)
               : "memory");
}

template <int C>
__device__ __forceinline__ void group_barrier() {
  if constexpr (C > 1) {
    __syncwarp();  // the cluster barrier is one of whole warps
    cluster_barrier();
  } else {
    __syncthreads();
  }
}

// The two-stage transform of line_fft.cuh on a line whose threads share a
// warp, with the second stage's twiddles of thread t in registers (HELD) or
// read from the table. `row` is the line's alone and free again when it returns.
template <int N, bool HELD>
struct Line {
  using G = Geometry<N>;
  static constexpr int Q = G::E / G::R1;  // second-stage butterflies of a thread
  static constexpr int kHeld = HELD ? Q * (G::R1 - 1) : 1;
  float2 held[kHeld];
  const float2* table;

  __device__ __forceinline__ void init(const float2* tw, int t) {
    table = tw;
    if constexpr (HELD) {
#pragma unroll
      for (int q = 0; q < Q; ++q) {
#pragma unroll
        for (int r = 1; r < G::R1; ++r) {
          held[q * (G::R1 - 1) + r - 1] = __ldg(tw + (r - 1) * G::R0 + t + G::T * q);
        }
      }
    }
  }

  template <bool INV>
  __device__ __forceinline__ void transform(float2 (&v)[G::E], int t, float2* row) const {
    butterfly<G::R0, INV>(v);
#pragma unroll
    for (int r = 0; r < G::R0; ++r) row[swz(t * G::R0 + r)] = v[r];
    __syncwarp();
#pragma unroll
    for (int m = 0; m < G::E; ++m) v[m] = row[swz(t + G::T * m)];
    __syncwarp();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      float2 u[G::R1];
      u[0] = v[q];
#pragma unroll
      for (int r = 1; r < G::R1; ++r) {
        float2 w;
        if constexpr (HELD) {
          w = held[q * (G::R1 - 1) + r - 1];
        } else {
          w = __ldg(table + (r - 1) * G::R0 + t + G::T * q);
        }
        u[r] = INV ? cmulc(v[q + r * Q], w) : cmul(v[q + r * Q], w);
      }
      butterfly<G::R1, INV>(u);
#pragma unroll
      for (int r = 0; r < G::R1; ++r) v[q + r * Q] = u[r];
    }
  }
};

template <int N, int C, class AmpT>
__global__ void __launch_bounds__(Resident<N, C>::NT, 1) resident_kernel(const ResidentParams p) {
  using K = Resident<N, C>;
  constexpr int E = K::E, T = K::T, R = K::R, P = K::P, Q = K::Q;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* ws = reinterpret_cast<float2*>(smem_raw);
  float2* cs = ws + N * Q;

  const int tid = threadIdx.x;
  const int rank = C > 1 ? static_cast<int>(cluster_rank()) : 0;
  const int start = blockIdx.x / C;
  // Line l and thread t of it, in both phases: row l of this CTA's rows and
  // column l of its columns.
  const int l = tid / T, t = tid % T;
  const int line = rank * R + l;  // row or column of the start
  float2* exchange = cs + N * Q + l * P;
  const long long at = static_cast<long long>(start) * N * N + static_cast<long long>(line) * N + t;

  Line<N, K::kTwiddlesHeld> lines;
  lines.init(p.twiddle, t);
  const Ctrl* ctrl = p.ctrl;
  const float ca = ctrl->a, cb = ctrl->b;
  const int row0 = ctrl->counters[p.group];
  const int capacity = ctrl->capacity;
  double* errs = ctrl->errs + static_cast<long long>(row0) * p.starts_total + p.start0 + start;

  float2 x[E];
  unsigned outside = 0;  // bit m: element t + T m of the row lies outside the support
  float a[E];
  {
    const AmpT* __restrict__ amp =
        static_cast<const AmpT*>(p.amp) +
        (p.amp_stride
             ? static_cast<long long>((p.start0 + start) / p.starts_per_problem) * p.amp_stride
             : 0);
#pragma unroll
    for (int m = 0; m < E; ++m) {
      x[m] = p.x[at + T * m];
      outside |= (p.support[at + T * m] == 0 ? 1u : 0u) << m;
      a[m] = to_float(amp[(t + T * m) * N + line]);
    }
  }
  float2 v[E];
#pragma unroll
  for (int m = 0; m < E; ++m) v[m] = x[m];
  lines.template transform<false>(v, t, exchange);

  const unsigned ws_addr = smem_addr(ws), cs_addr = smem_addr(cs);
  // Element t + T m of this thread's line, to line t + T m of the other
  // buffer (of its owner), as its element `line`.
  auto send = [&](float2* local, unsigned addr) {
#pragma unroll
    for (int m = 0; m < E; ++m) {
      const int i = t + T * m;
      if constexpr (C > 1) {
        store_cluster(cluster_map(addr, i / R) + static_cast<unsigned>(line * Q + i % R) * 8u, v[m]);
      } else {
        local[line * Q + i] = v[m];
      }
    }
  };
  if constexpr (C > 1) cluster_barrier();  // every CTA of the cluster has started

  const float scale = p.scale;
  for (int it = 0; it < p.iterations; ++it) {
    send(cs, cs_addr);
    group_barrier<C>();  // every column is complete
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = cs[(t + T * m) * Q + l];
    lines.template transform<false>(v, t, exchange);
    float acc = 0.0f;
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = pointwise_projection<Mode::kMod>(v[m], a[m], scale, acc);
    lines.template transform<true>(v, t, exchange);
    send(ws, ws_addr);
    const double total = warp_sum_double(static_cast<double>(acc));
    if ((tid & 31) == 0 && row0 + it < capacity) {
      atomicAdd(errs + static_cast<long long>(it) * p.starts_total, total);
    }
    group_barrier<C>();  // every row is complete
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = ws[(t + T * m) * Q + l];
    lines.template transform<true>(v, t, exchange);
#pragma unroll
    for (int m = 0; m < E; ++m) {
      if (outside >> m & 1u) v[m] = relaxed(ca, x[m], cb, v[m]);
      x[m] = v[m];
    }
    lines.template transform<false>(v, t, exchange);
  }

#pragma unroll
  for (int m = 0; m < E; ++m) {
    p.x[at + T * m] = x[m];
    p.w[at + T * m] = v[m];
  }
}

__global__ void advance_counter_kernel(Ctrl* ctrl, int group, int count) {
  ctrl->counters[group] += count;
}

// f(std::integral_constant<int, C>{}) for the cluster size `cluster` of side N.
template <int N, class F>
void with_cluster(int cluster, F&& f) {
  auto is = [&](auto c) {
    if (cluster != c) return false;
    f(c);
    return true;
  };
  bool done = false;
  if constexpr (N == 64) {
    done = is(std::integral_constant<int, 1>{}) || is(std::integral_constant<int, 2>{}) ||
           is(std::integral_constant<int, 4>{}) || is(std::integral_constant<int, 8>{});
  } else if constexpr (N == 128) {
    done = is(std::integral_constant<int, 2>{}) || is(std::integral_constant<int, 4>{}) ||
           is(std::integral_constant<int, 8>{}) || is(std::integral_constant<int, 16>{});
  } else {
    done = is(std::integral_constant<int, 8>{}) || is(std::integral_constant<int, 16>{});
  }
  if (!done) throw std::logic_error("resident kernel: unsupported cluster size");
}

// f(std::integral_constant<int, N>{}) for a supported side.
template <class F>
void with_side(int side, F&& f) {
  switch (side) {
    case 64: return f(std::integral_constant<int, 64>{});
    case 128: return f(std::integral_constant<int, 128>{});
    case 256: return f(std::integral_constant<int, 256>{});
    default: throw std::logic_error("resident kernel: unsupported side");
  }
}

template <int N, int C>
cudaLaunchConfig_t launch_config(int starts, cudaLaunchAttribute* attr, cudaStream_t stream) {
  using K = Resident<N, C>;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(starts * C));
  cfg.blockDim = dim3(K::NT);
  cfg.dynamicSmemBytes = K::kBytes;
  cfg.stream = stream;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = C;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

template <int N, int C, class AmpT>
void launch_typed(const ResidentParams& p, int starts, cudaStream_t stream) {
  cudaLaunchAttribute attr{};
  const cudaLaunchConfig_t cfg = launch_config<N, C>(starts, &attr, stream);
  QPB_CHECK(cudaLaunchKernelEx(&cfg, resident_kernel<N, C, AmpT>, p));
  count_launches(1);
}

template <int N, int C, class AmpT>
void allow() {
  QPB_CHECK(cudaFuncSetAttribute(resident_kernel<N, C, AmpT>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 Resident<N, C>::kBytes));
  QPB_CHECK(cudaFuncSetAttribute(resident_kernel<N, C, AmpT>,
                                 cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared));
  if constexpr (C > 8) {
    QPB_CHECK(cudaFuncSetAttribute(resident_kernel<N, C, AmpT>,
                                   cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  }
}

// Clusters of each size that the current device runs at once, the attributes
// set on the way; once per device and side.
const std::map<int, int>& cluster_room(int side) {
  static std::mutex mutex;
  static std::map<std::pair<int, int>, std::map<int, int>> rooms;
  int device = 0;
  QPB_CHECK(cudaGetDevice(&device));
  std::lock_guard<std::mutex> lock(mutex);
  auto [it, fresh] = rooms.try_emplace({device, side});
  if (fresh) {
    try {
      with_side(side, [&](auto n) {
        for (const ClusterSize& s : cluster_sizes(n)) {
          const int size = s.ctas;
          with_cluster<n>(size, [&](auto c) {
            allow<n, c, float>();
            allow<n, c, __half>();
            allow<n, c, __nv_bfloat16>();
            cudaLaunchAttribute attr{};
            const cudaLaunchConfig_t cfg = launch_config<n, c>(64, &attr, nullptr);
            int clusters = 0;
            QPB_CHECK(cudaOccupancyMaxActiveClusters(&clusters, resident_kernel<n, c, float>, &cfg));
            it->second[size] = clusters;
          });
        }
      });
    } catch (...) {
      rooms.erase(it);
      throw;
    }
  }
  return it->second;
}

}  // namespace

int resident_max_clusters(int side, int cluster) { return cluster_room(side).at(cluster); }

int resident_smallest_cluster(int side) { return cluster_sizes(side).front().ctas; }

bool resident_supports(int ndim, int d1, int d2) {
  return ndim == 2 && d1 == d2 && (d1 == 64 || d1 == 128 || d1 == 256);
}

int resident_cluster(int side, int starts) {
  int device = 0, sms = 0;
  QPB_CHECK(cudaGetDevice(&device));
  QPB_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  int best = 0;
  for (const auto& [size, room] : cluster_room(side)) {
    if (best == 0 || (starts <= room && starts * size <= sms)) best = size;
  }
  return best;
}

void launch_resident(const ResidentParams& p, int side, int starts, cudaStream_t stream) {
  if (p.iterations < 1) return;
  with_side(side, [&](auto n) {
    with_cluster<n>(p.cluster, [&](auto c) {
      switch (p.amp_storage) {
        case AmpStorage::kF32:
          return launch_typed<n, c, float>(p, starts, stream);
        case AmpStorage::kF16:
          return launch_typed<n, c, __half>(p, starts, stream);
        case AmpStorage::kBF16:
          return launch_typed<n, c, __nv_bfloat16>(p, starts, stream);
      }
    });
  });
  advance_counter_kernel<<<1, 1, 0, stream>>>(p.ctrl, p.group, p.iterations);
  QPB_CHECK(cudaGetLastError());
  count_launches(1);
}

}  // namespace qpb
