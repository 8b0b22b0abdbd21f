// Groups of boundary-band sweeps as one thread-block-cluster launch.
//
// A V-cycle smooths each level with boundary_smoothing sweeps over the nodes of
// the Dirichlet band before and after the full sweeps (24 colour passes for
// three sweeps).  A pass updates only 10 to 1500 nodes and depends on the pass
// before it, so as separate launches each costs its launch and its dependent
// loads: 2.3 us (coarse levels, FP32) to 7.4 us (level 0, one thread per node
// in FP64) whatever the band's size.  Here the CTAs of one cluster (BG_CTAS)
// own the band's nodes for the whole group: the iterate of the owned nodes and
// of their band neighbours (the halo), the right-hand sides, inverse diagonal
// blocks and stencil rows (level 0: cell stiffnesses) stay in shared memory.
// An updated node is written to the halos of the CTAs that read it through
// distributed shared memory, and a pass ends with a cluster barrier.  (Reading
// neighbours from their owners instead took 8 us a pass at 56 nodes a CTA.)
// Nodes outside the band do not change during a group: their share of a row is
// subtracted from the right-hand side once, at the start.
// Measured per V-cycle (three sweeps, four groups a level): 867 nodes in the
// reference rounding 858 -> 292 us for the whole cycle (16^3 box), two levels of
// 1260 and 645 nodes in FP32 629 -> 349 us (97 x 25 x 49 bridge).  A pass is
// bound by its chain: the cluster barrier behind remote stores (about 800 cycles
// of an otherwise empty pass), the shared loads, FMAs and shuffles.  With more
// nodes a CTA works through several rounds a pass, and the separate launches,
// which spread over the whole GPU, are faster: band_slots() is the line, and the
// tables of a CTA's share must fit its shared memory.
#pragma once
#include "kernels.cuh"

namespace sgs {

constexpr int BG_CTAS = 16, BG_THREADS = 512;
constexpr uint32_t BG_OUTSIDE = 0xffffffffu;
constexpr int BG_NONE = INT32_MIN;  // unused slot

// Slots a CTA (nodes it owns) up to which a level's groups run as one cluster.
// V-cycles of boxes with the level's passes launched one by one / as a cluster (us):
//   level 0, FP64           572 538 / 483,   620 542 / 506,   720 566 / 585
//   level 0, ref. rounding  572 589 / 554,   620 585 / 574,   720 614 / 656
//   level 0, FP32           515 370 / 355,   559 371 / 368,   608 392 / 407
//   stencil level, FP32     140 658 / 623,   155 651 / 637,   176 713 / 727
//   stencil level, FP64     101 749 / 735;   from about 105 on the rows do not fit
template <typename T>
constexpr int band_slots(int level) { return level > 0 ? 160 : sizeof(T) == 4 ? 560 : 640; }

// The band's nodes in ascending order are cut into BG_CTAS equal parts (the
// block order is a space-filling curve, so a part is compact); a CTA's nodes of
// colour c are the first own[c] of the slots from off[c] on.
struct BandPlan {
  int slots = 0;  // owned, per CTA
  int halo = 0;   // read from other CTAs, the largest CTA's
  int off[8];
  int16_t own[BG_CTAS][8];
};

__device__ __forceinline__ uint32_t cluster_address(const void* p, uint32_t rank) {
  uint32_t a = uint32_t(__cvta_generic_to_shared(p)), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// (the forms without .aligned: a warp may arrive here diverged)
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// write a slot of another CTA's shared memory
__device__ __forceinline__ void cluster_store(uint32_t a, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t a, double4 v) {
  asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a + 16), "d"(v.z) : "memory");
}

// global index of g's neighbour at offset (q / 9, q / 3 % 3, q % 3) - 1, or -1
__device__ __forceinline__ int neighbour27(const int* __restrict__ nbr, int g, int q) {
  const int x = ((g >> 5) & 3) + q / 9 - 1, y = ((g >> 3) & 3) + q / 3 % 3 - 1, z = (g & 7) + q % 3 - 1;
  const int b = __ldg(nbr + long(g >> 7) * 27 + (x < 0 ? 0 : (x > 3 ? 2 : 1)) * 9 + (y < 0 ? 0 : (y > 3 ? 2 : 1)) * 3 +
                      (z < 0 ? 0 : (z > 7 ? 2 : 1)));
  return b < 0 ? -1 : (b << 7) + ((x & 3) << 5) + ((y & 3) << 3) + (z & 7);
}

// map [level nodes]: owner << 16 | slot of the nodes of the node table [CTA][slot]
__global__ void band_map_kernel(int n, int slots, const int* __restrict__ node, uint32_t* __restrict__ map) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && node[i] != BG_NONE) map[node[i]] = uint32_t(i / slots) << 16 | uint32_t(i % slots);
}

// [CTA][slot][27]: owner << 16 | slot of the neighbours in the band, BG_OUTSIDE elsewhere
__global__ void band_codes_kernel(int n, const int* __restrict__ node, const int* __restrict__ nbr,
                                  const uint32_t* __restrict__ map, uint32_t* __restrict__ code) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * 27) return;
  const int g = node[t / 27], q = t % 27;
  uint32_t c = BG_OUTSIDE;
  if (g != BG_NONE) {
    const int i = neighbour27(nbr, g, q);
    if (i >= 0) c = map[i];
  }
  code[t] = c;
}

// need[r][i] = 1 where CTA r reads the entry i = owner * slots + slot of another CTA
__global__ void band_need_kernel(int n, int slots, const uint32_t* __restrict__ code, uint8_t* __restrict__ need) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * 27) return;
  const uint32_t c = code[t];
  const int r = t / 27 / slots;
  if (c != BG_OUTSIDE && int(c >> 16) != r) need[long(r) * n + int(c >> 16) * slots + int(c & 0xffffu)] = 1;
}

// One CTA of 256 threads per cluster rank r numbers r's halo in entry order:
// push[i][r] = the local slot of entry i in CTA r (slots + number), BG_NOWHERE
// where r does not read it; hnode[r][number] = its node; count[r].
constexpr int BG_NOWHERE = 0xffff;
__global__ void band_halo_kernel(int n, int slots, const uint8_t* __restrict__ need, const int* __restrict__ node,
                                 uint16_t* __restrict__ push, int* __restrict__ hnode, int* __restrict__ count) {
  __shared__ int warp_sum[8];
  const int r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int base = 0;
  for (int i0 = 0; i0 < n; i0 += 256) {
    const int i = i0 + int(threadIdx.x);
    const bool on = i < n && need[long(r) * n + i];
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (lane == 0) warp_sum[warp] = __popc(m);
    __syncthreads();
    int at = base + __popc(m & ((1u << lane) - 1));
    for (int w = 0; w < 8; ++w) {
      if (w < warp) at += warp_sum[w];
      base += warp_sum[w];
    }
    if (i < n) push[long(i) * BG_CTAS + r] = uint16_t(on ? slots + at : BG_NOWHERE);
    if (on) hnode[long(r) * n + at] = node[i];
    __syncthreads();
  }
  if (threadIdx.x == 0) count[r] = base;
}

// [CTA][slot][27]: local slots of the neighbours, BG_NOWHERE outside the band
__global__ void band_local_kernel(int n, int slots, const uint32_t* __restrict__ code, const uint16_t* __restrict__ push,
                                  uint16_t* __restrict__ local) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * 27) return;
  const uint32_t c = code[t];
  const int r = t / 27 / slots, o = int(c >> 16), s = int(c & 0xffffu);
  local[t] = uint16_t(c == BG_OUTSIDE ? BG_NOWHERE : o == r ? s : push[(o * slots + s) * BG_CTAS + r]);
}

// shared memory of one CTA in bytes: records of the owned nodes, the halo and a
// zero; per owned node `vals` values, 27 neighbours, 16 destinations, flags
template <typename T>
constexpr size_t band_smem(const BandPlan& p, int vals) {
  return (size_t(p.slots) + p.halo + 1) * 4 * sizeof(T) +
         size_t(p.slots) * (vals * sizeof(T) + 16 * sizeof(uint16_t) + sizeof(uint32_t) + 27 * sizeof(uint16_t));
}
template <typename T>
constexpr size_t band0_smem(const BandPlan& p) { return band_smem<T>(p, 8 + 9); }
template <typename T>
constexpr size_t bandc_smem(const BandPlan& p) { return band_smem<T>(p, 243 + 9); }

// Level 0, eight threads per node as in gs0_cell_kernel (thread I the cell of
// which the node is corner I).  PACKED: the iterate is u4 (u, E), else the
// planes of u.  What bounds a pass is its chain: 8 loads from the CTA's own
// copies, 24 dependent FMAs, three rounds of shuffles, the 3x3 update, the remote
// stores into the halos, the cluster barrier (16 SMs at 0.39 instructions a cycle
// and scheduler, long-scoreboard and barrier stalls: 256^3 shell, FP32).
template <typename T, bool PACKED>
__global__ void __launch_bounds__(BG_THREADS, 1) band0_group_kernel(
    BandPlan p, const int* __restrict__ node, const uint16_t* __restrict__ local, const uint16_t* __restrict__ push,
    const int* __restrict__ hnode, const int* __restrict__ hcount, const int* __restrict__ nbr, typename Pack4<T>::type* u4,
    T* u, const T* __restrict__ E, const T* __restrict__ b, const uint32_t* __restrict__ flags, int N, T dx,
    const KcReg<T> K, int sweeps, int forward, int round) {
  using V = typename Pack4<T>::type;
  extern __shared__ __align__(32) unsigned char band_mem[];
  const int S = p.slots;
  const int zero = S + p.halo;                             // slot that stays zero
  V* su = reinterpret_cast<V*>(band_mem);                  // [S + halo + 1]
  T* sE = reinterpret_cast<T*>(su + zero + 1);             // [S][8] E of the node's cells
  T* sb = sE + 8 * S;                                      // [S][3]
  T* sd = sb + 3 * S;                                      // [S][6]
  uint32_t* sp = reinterpret_cast<uint32_t*>(sd + 6 * S);  // [S][8] destinations, two ranks each
  uint32_t* sf = sp + 8 * S;                               // [S] flags
  uint16_t* sn = reinterpret_cast<uint16_t*>(sf + S);      // [S][27] neighbours' slots
  const int rank = int(cluster_rank());
  __shared__ int s_own[8], s_off[8];  // this CTA's nodes of each colour
  if (threadIdx.x < 8) {
    s_own[threadIdx.x] = p.own[rank][threadIdx.x];
    s_off[threadIdx.x] = p.off[threadIdx.x];
  }
  __syncthreads();
  const int I = threadIdx.x & 7, first = threadIdx.x >> 3;
  constexpr int STEP = BG_THREADS / 8;
  const int Ix = I >> 2, Iy = (I >> 1) & 1, Iz = I & 1;
  const T s0 = Ix ? T(-1) : T(1), s1 = Iy ? T(-1) : T(1), s2 = Iz ? T(-1) : T(1);
  const uint32_t to0 = cluster_address(su, 2 * I), to1 = cluster_address(su, 2 * I + 1);
  auto send = [&](uint32_t two, const V& v) {
    const uint32_t d0 = two & 0xffffu, d1 = two >> 16;
    if (d0 != BG_NOWHERE) cluster_store(to0 + d0 * uint32_t(sizeof(V)), v);
    if (d1 != BG_NOWHERE) cluster_store(to1 + d1 * uint32_t(sizeof(V)), v);
  };
  // index in the 3x3x3 neighbourhood of corner I ^ Jp of this thread's cell
  auto corner = [&](int Jp) {
    const int a = (Jp >> 2) ? 2 - 2 * Ix : 1, c = ((Jp >> 1) & 1) ? 2 - 2 * Iy : 1, d = (Jp & 1) ? 2 - 2 * Iz : 1;
    return a * 9 + c * 3 + d;
  };
  // constant data: addresses, cell stiffnesses, inverse diagonal blocks
  if (threadIdx.x == 0) su[zero] = Pack4<T>::make(T(0), T(0), T(0), T(0));
  // (a warp's four nodes go through each loop together: a missing one computes
  // on zeros and writes nothing)
  const int lead = first & ~3;
  for (int w = lead; w < S; w += STEP) {
    const int s = w + (first & 3);
    const int g = s < S ? node[rank * S + s] : BG_NONE;
    const bool on = g != BG_NONE;
    T Ec = 0;
    if (on) {
      for (int q = I; q < 27; q += 8) {
        const int n = local[(rank * S + s) * 27 + q];
        sn[s * 27 + q] = uint16_t(n == BG_NOWHERE ? zero : n);
      }
      sp[s * 8 + I] = reinterpret_cast<const uint32_t*>(push)[(rank * S + s) * 8 + I];
      const int i = neighbour27(nbr, g, (1 - Ix) * 9 + (1 - Iy) * 3 + 1 - Iz);
      Ec = i < 0 ? T(0) : E[i];
      sE[s * 8 + I] = Ec;
    }
    __syncwarp();
    T red[6] = {Ec * K(0, 0, 0, 0), Ec * K(0, 0, 1, 1), Ec * K(0, 0, 2, 2),
                Ec * (s0 * s1) * K(0, 0, 0, 1), Ec * (s0 * s2) * K(0, 0, 0, 2), Ec * (s1 * s2) * K(0, 0, 1, 2)};
#pragma unroll
    for (int o = 4; o; o >>= 1)
#pragma unroll
      for (int q = 0; q < 6; ++q) red[q] += __shfl_xor_sync(0xffffffffu, red[q], o);
    if (on && I == 0) {
      const uint32_t fl = flags[g];
      sf[s] = fl;
      T a[6];
      diagonal_inverse<T>(red[0] * dx, red[1] * dx, red[2] * dx, red[3] * dx, red[4] * dx, red[5] * dx, fl, a);
#pragma unroll
      for (int q = 0; q < 6; ++q) sd[s * 6 + q] = a[q];
    }
  }
  pdl_wait();
  // the iterate, and the right-hand side less the share of the nodes outside the band
  for (int w = lead; w < S; w += STEP) {
    const int s = w + (first & 3);
    const int g = s < S ? node[rank * S + s] : BG_NONE;
    const bool on = g != BG_NONE;
    const T Ec = on ? sE[s * 8 + I] : T(0);
    T gv[3] = {0, 0, 0};
#pragma unroll
    for (int Jp = 0; Jp < 8; ++Jp) {
      const int q = corner(Jp);
      T w0 = 0, w1 = 0, w2 = 0;
      if (on && sn[s * 27 + q] == zero) {
        const int i = neighbour27(nbr, g, q);
        if (i >= 0) {
          if (PACKED) {
            const V v = u4[packed_index(i)];
            w0 = s0 * v.x, w1 = s1 * v.y, w2 = s2 * v.z;
          } else {
            w0 = s0 * u[i], w1 = s1 * u[i + N], w2 = s2 * u[i + 2 * N];
          }
        }
      }
#pragma unroll
      for (int r = 0; r < 3; ++r)
        gv[r] = fma(K(0, Jp, r, 0), w0, fma(K(0, Jp, r, 1), w1, fma(K(0, Jp, r, 2), w2, gv[r])));
    }
    T red[3] = {Ec * s0 * gv[0], Ec * s1 * gv[1], Ec * s2 * gv[2]};
    __syncwarp();
#pragma unroll
    for (int o = 4; o; o >>= 1)
#pragma unroll
      for (int q = 0; q < 3; ++q) red[q] += __shfl_xor_sync(0xffffffffu, red[q], o);
    if (on && I == 0) {
      if (PACKED) su[s] = u4[packed_index(g)];
      else su[s] = Pack4<T>::make(u[g], u[g + N], u[g + 2 * N], T(0));
#pragma unroll
      for (int q = 0; q < 3; ++q) sb[s * 3 + q] = b[g + q * N] - red[q] * dx;
    }
  }
  for (int h = threadIdx.x; h < hcount[rank]; h += BG_THREADS) {
    const int g = hnode[rank * S * BG_CTAS + h];
    if (PACKED) su[S + h] = u4[packed_index(g)];
    else su[S + h] = Pack4<T>::make(u[g], u[g + N], u[g + 2 * N], T(0));
  }
  __syncthreads();  // a pass reads tables that other warps of the CTA filled before its barrier completes
  cluster_arrive();
  for (int sw = 0; sw < sweeps; ++sw) {
    for (int kk = 0; kk < 8; ++kk) {
      const int c = forward ? kk : 7 - kk;
      const int own = s_own[c], off = s_off[c];
      // addresses and stiffness of the first node, read before the barrier completes
      int w = lead;
      int at[8];
      T Ec = 0, rb[3], a[6];
      uint32_t fl = 0, two = 0;
      auto fetch = [&]() {
        const int s = off + min(w + (first & 3), own - 1);
#pragma unroll
        for (int Jp = 0; Jp < 8; ++Jp) at[Jp] = sn[s * 27 + corner(Jp)];
        Ec = sE[s * 8 + I];
#pragma unroll
        for (int q = 0; q < 3; ++q) rb[q] = sb[s * 3 + q];
#pragma unroll
        for (int q = 0; q < 6; ++q) a[q] = sd[s * 6 + q];
        fl = sf[s];
        two = sp[s * 8 + I];
      };
      if (w < own) fetch();
      cluster_wait();
      while (w < own) {
        const int k = w + (first & 3), s = off + min(k, own - 1);
        T gv[3] = {0, 0, 0}, uc[4] = {0, 0, 0, 0};
#pragma unroll
        for (int Jp = 0; Jp < 8; ++Jp) {
          const V v = su[at[Jp]];
          if (Jp == 0) uc[0] = v.x, uc[1] = v.y, uc[2] = v.z, uc[3] = v.w;  // the node itself
          const T w0 = s0 * v.x, w1 = s1 * v.y, w2 = s2 * v.z;
#pragma unroll
          for (int r = 0; r < 3; ++r)
            gv[r] = fma(K(0, Jp, r, 0), w0, fma(K(0, Jp, r, 1), w1, fma(K(0, Jp, r, 2), w2, gv[r])));
        }
        T red[3] = {Ec * s0 * gv[0], Ec * s1 * gv[1], Ec * s2 * gv[2]};
#pragma unroll
        for (int o = 4; o; o >>= 1)
#pragma unroll
          for (int q = 0; q < 3; ++q) red[q] += __shfl_xor_sync(0xffffffffu, red[q], o);
        if (k < own) {  // every thread of the node has the sums: thread 0 keeps the node, each sends it to two CTAs
          const T r0 = rb[0] - red[0] * dx, r1 = rb[1] - red[1] * dx, r2 = rb[2] - red[2] * dx;
          V v;
          v.x = (fl & DIR_X) ? T(0) : uc[0] + r0 * a[0] + r1 * a[3] + r2 * a[4];
          v.y = (fl & DIR_Y) ? T(0) : uc[1] + r0 * a[3] + r1 * a[1] + r2 * a[5];
          v.z = (fl & DIR_Z) ? T(0) : uc[2] + r0 * a[4] + r1 * a[5] + r2 * a[2];
          v.w = uc[3];
          if (I == 0) su[s] = v;
          send(two, v);
        }
        w += STEP;
        if (w < own) fetch();
      }
      cluster_arrive();
    }
    if (round) {  // Cast_To_Float after a sweep
      cluster_wait();
      for (int t = threadIdx.x; t < 8 * S; t += BG_THREADS) {
        const int s = t >> 3;  // t & 7 == I
        if (node[rank * S + s] == BG_NONE) continue;
        V v = su[s];
        v.x = T(round_to_float(v.x)), v.y = T(round_to_float(v.y)), v.z = T(round_to_float(v.z));
        if (I == 0) su[s] = v;
        send(sp[s * 8 + I], v);
      }
      cluster_arrive();
    }
  }
  cluster_wait();  // every CTA has read what it needs of the others
  for (int s = threadIdx.x; s < S; s += BG_THREADS) {
    const int g = node[rank * S + s];
    if (g == BG_NONE) continue;
    const V v = su[s];
    if (PACKED) {
      u4[packed_index(g)] = v;
    } else {
      u[g] = v.x;
      u[g + N] = v.y;
      u[g + 2 * N] = v.z;
    }
  }
}

// Levels with stencils: one warp per node, lane q < 27 the spoke q (as in
// stencil_op_kernel), the rows in shared memory.  Colours in the order of
// Solver::sweep.
template <typename T>
__global__ void __launch_bounds__(BG_THREADS, 1) bandc_group_kernel(
    BandPlan p, const int* __restrict__ node, const uint16_t* __restrict__ local, const uint16_t* __restrict__ push,
    const int* __restrict__ hnode, const int* __restrict__ hcount, const int* __restrict__ nbr,
    const T* __restrict__ A, T* u, const T* __restrict__ b, const uint32_t* __restrict__ flags, long N, int sweeps,
    int forward, int round) {
  using V = typename Pack4<T>::type;
  extern __shared__ __align__(32) unsigned char band_mem[];
  const int S = p.slots;
  const int zero = S + p.halo;
  V* su = reinterpret_cast<V*>(band_mem);
  T* sA = reinterpret_cast<T*>(su + zero + 1);  // [S][243]
  T* sb = sA + 243 * S;
  T* sd = sb + 3 * S;
  uint32_t* sp = reinterpret_cast<uint32_t*>(sd + 6 * S);
  uint32_t* sf = sp + 8 * S;
  uint16_t* sn = reinterpret_cast<uint16_t*>(sf + S);
  const int rank = int(cluster_rank());
  __shared__ int s_own[8], s_off[8];  // this CTA's nodes of each colour
  if (threadIdx.x < 8) {
    s_own[threadIdx.x] = p.own[rank][threadIdx.x];
    s_off[threadIdx.x] = p.off[threadIdx.x];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int WARPS = BG_THREADS / 32;
  const int I = threadIdx.x & 7;  // lanes 0..7 send to two CTAs each
  const uint32_t to0 = cluster_address(su, 2 * I), to1 = cluster_address(su, 2 * I + 1);
  auto send = [&](uint32_t two, const V& v) {
    const uint32_t d0 = two & 0xffffu, d1 = two >> 16;
    if (d0 != BG_NOWHERE) cluster_store(to0 + d0 * uint32_t(sizeof(V)), v);
    if (d1 != BG_NOWHERE) cluster_store(to1 + d1 * uint32_t(sizeof(V)), v);
  };
  if (threadIdx.x == 0) su[zero] = Pack4<T>::make(T(0), T(0), T(0), T(0));
  for (int s = warp; s < S; s += WARPS) {
    const int g = node[rank * S + s];
    if (g == BG_NONE) continue;
    const T* row = A + long(g) * 243;
    for (int k = lane; k < 243; k += 32) sA[s * 243 + k] = row[k];
    if (lane < 27) {
      const int n = local[(rank * S + s) * 27 + lane];
      sn[s * 27 + lane] = uint16_t(n == BG_NOWHERE ? zero : n);
    }
    if (lane < 8) sp[s * 8 + lane] = reinterpret_cast<const uint32_t*>(push)[(rank * S + s) * 8 + lane];
    if (lane == 27) {
      const uint32_t fl = flags[g];
      const T* m = row + 13 * 9;
      T a[6];
      diagonal_inverse<T>(m[0], m[4], m[8], m[1], m[2], m[5], fl, a);
      sf[s] = fl;
#pragma unroll
      for (int q = 0; q < 6; ++q) sd[s * 6 + q] = a[q];
    }
  }
  pdl_wait();
  for (int s = warp; s < S; s += WARPS) {
    const int g = node[rank * S + s];
    if (g == BG_NONE) continue;
    T f0 = 0, f1 = 0, f2 = 0;
    if (lane < 27 && sn[s * 27 + lane] == zero) {
      const int i = neighbour27(nbr, g, lane);
      if (i >= 0) {
        const T* a = A + long(g) * 243 + lane * 9;
        const T ux = u[i], uy = u[i + N], uz = u[i + 2 * N];
        f0 = a[0] * ux + a[1] * uy + a[2] * uz;
        f1 = a[3] * ux + a[4] * uy + a[5] * uz;
        f2 = a[6] * ux + a[7] * uy + a[8] * uz;
      }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      f0 += __shfl_xor_sync(0xffffffffu, f0, o);
      f1 += __shfl_xor_sync(0xffffffffu, f1, o);
      f2 += __shfl_xor_sync(0xffffffffu, f2, o);
    }
    if (lane == 0) {
      su[s] = Pack4<T>::make(u[g], u[g + N], u[g + 2 * N], T(0));
      sb[s * 3] = b[g] - f0;
      sb[s * 3 + 1] = b[g + N] - f1;
      sb[s * 3 + 2] = b[g + 2 * N] - f2;
    }
  }
  for (int h = threadIdx.x; h < hcount[rank]; h += BG_THREADS) {
    const int g = hnode[rank * S * BG_CTAS + h];
    su[S + h] = Pack4<T>::make(u[g], u[g + N], u[g + 2 * N], T(0));
  }
  __syncthreads();
  cluster_arrive();
  const unsigned order = forward ? 0x02376451u : 0x15467320u;  // colour of pass kk in bits 4kk..
  for (int sw = 0; sw < sweeps; ++sw) {
    for (int kk = 0; kk < 8; ++kk) {
      const int c = int(order >> (4 * kk)) & 7;
      const int own = s_own[c], off = s_off[c];
      int k = warp;
      int at = zero;
      T a[9], rb[3], d[6];
      uint32_t fl = 0, two = 0;
      auto fetch = [&]() {
        const int s = off + k;
        if (lane < 27) at = sn[s * 27 + lane];
#pragma unroll
        for (int q = 0; q < 3; ++q) rb[q] = sb[s * 3 + q];
#pragma unroll
        for (int q = 0; q < 6; ++q) d[q] = sd[s * 6 + q];
        fl = sf[s];
        two = sp[s * 8 + I];
#pragma unroll
        for (int q = 0; q < 9; ++q) a[q] = lane < 27 ? sA[s * 243 + lane * 9 + q] : T(0);
      };
      if (k < own) fetch();
      cluster_wait();
      while (k < own) {
        const int s = off + k;
        const V n = su[at];
        V v = su[s];
        T f0 = a[0] * n.x + a[1] * n.y + a[2] * n.z;
        T f1 = a[3] * n.x + a[4] * n.y + a[5] * n.z;
        T f2 = a[6] * n.x + a[7] * n.y + a[8] * n.z;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
          f0 += __shfl_xor_sync(0xffffffffu, f0, o);
          f1 += __shfl_xor_sync(0xffffffffu, f1, o);
          f2 += __shfl_xor_sync(0xffffffffu, f2, o);
        }
        if (lane < 8) {
          const T r0 = rb[0] - f0, r1 = rb[1] - f1, r2 = rb[2] - f2;
          v.x = (fl & DIR_X) ? T(0) : v.x + (d[0] * r0 + d[3] * r1 + d[4] * r2);
          v.y = (fl & DIR_Y) ? T(0) : v.y + (d[3] * r0 + d[1] * r1 + d[5] * r2);
          v.z = (fl & DIR_Z) ? T(0) : v.z + (d[4] * r0 + d[5] * r1 + d[2] * r2);
          if (lane == 0) su[s] = v;
          send(two, v);
        }
        __syncwarp();
        k += WARPS;
        if (k < own) fetch();
      }
      cluster_arrive();
    }
    if (round) {
      cluster_wait();
      for (int t = threadIdx.x; t < 8 * S; t += BG_THREADS) {
        const int s = t >> 3;  // t & 7 == I
        if (node[rank * S + s] == BG_NONE) continue;
        V v = su[s];
        v.x = T(round_to_float(v.x)), v.y = T(round_to_float(v.y)), v.z = T(round_to_float(v.z));
        if (I == 0) su[s] = v;
        send(sp[s * 8 + I], v);
      }
      cluster_arrive();
    }
  }
  cluster_wait();
  for (int s = threadIdx.x; s < S; s += BG_THREADS) {
    const int g = node[rank * S + s];
    if (g == BG_NONE) continue;
    const V v = su[s];
    u[g] = v.x;
    u[g + N] = v.y;
    u[g + 2 * N] = v.z;
  }
}

}  // namespace sgs
