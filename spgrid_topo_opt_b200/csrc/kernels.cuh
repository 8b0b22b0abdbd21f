// CUDA kernels of the narrow-band SPGrid elasticity MGPCG (sm_100a).
//
// Layout: a level holds nb active blocks of 4x4x8 nodes in SPGrid page order;
// node slot e = x*32 + y*8 + z inside a block, global node index b*128 + e.
// A 3-vector field is stored as three planes of N = nb*128 values ([3][N]).
// Level 0 carries the per-cell stiffness scale E (cell = its min-corner node,
// 0 = empty); the element matrix of a cell is E * (mu0*K_mu + lambda0*K_la).
// Coarse levels carry 27-point Galerkin stencils node-major, [N][243], entry
// ((i*3+j)*3+k)*9 + v*3 + w = row (node, v), column (node + (i,j,k) - 1, w).
#pragma once
#include <cstdint>

namespace sgs {

constexpr uint32_t ACTIVE_NODE = 0x10, DIR_X = 0x20, DIR_Y = 0x40, DIR_Z = 0x80, BOUNDARY_NODE = 0x1000;

// Combined element matrix Kc[I][J][v][w] = mu0*K_mu + lambda0*K_la.  It and its
// ten values below are launch arguments: sessions of several materials share the
// device.
template <typename T>
struct ElementMatrix {
  T v[8 * 8 * 9];
};

__device__ __forceinline__ double round_to_float(double v) { return double(float(v)); }

// The element matrix in exact integers, 72 K_mu and 72 K_la of the Q1 hex on the
// unit cube (node a = 4x + 2y + z), from the 1D integrals of the linear shape
// functions times 6 (mass {2, 1}, derivative-mass {-3, 3}, stiffness {6, -6});
// the same formulas as element_tables() in solver.cu.  Up to sign the 576
// entries take 10 values (m, l), so Kc = (mu0 m + lambda0 l) / 72 is 10 numbers,
// which the level-0 kernels keep in registers (KcReg).
__host__ __device__ constexpr int q1_g(int a, int b, int i, int j) {
  int v = 1;
  for (int ax = 0; ax < 3; ++ax) {
    const int pa = (a >> (2 - ax)) & 1, pb = (b >> (2 - ax)) & 1;
    const bool da = ax == i, db = ax == j;
    v *= (da && db) ? (pa == pb ? 6 : -6) : da ? (pa ? 3 : -3) : db ? (pb ? 3 : -3) : (pa == pb ? 2 : 1);
  }
  return v;
}
__host__ __device__ constexpr int q1_mu72(int a, int b, int i, int j) {
  return (q1_g(a, b, j, i) + (i == j ? q1_g(a, b, 0, 0) + q1_g(a, b, 1, 1) + q1_g(a, b, 2, 2) : 0)) / 3;
}
__host__ __device__ constexpr int q1_la72(int a, int b, int i, int j) { return q1_g(a, b, i, j) / 3; }
// class of a sign-normalised pair (m > 0, or m = 0 and l >= 0); -1 if it is none of the 10
__host__ __device__ constexpr int q1_class(int m, int l) {
  return (m == 3 && l == -3) ? 0 : (m == 3 && l == 3) ? 1 : (m == 4 && l == -2) ? 2 : (m == 4 && l == 4) ? 3
       : (m == 6 && l == -6) ? 4 : (m == 6 && l == 6) ? 5 : (m == 8 && l == 2) ? 6 : (m == 8 && l == 8) ? 7
       : (m == 10 && l == 4) ? 8 : (m == 32 && l == 8) ? 9 : -1;
}
constexpr int Q1_CLASS_M[10] = {3, 3, 4, 4, 6, 6, 8, 8, 10, 32}, Q1_CLASS_L[10] = {-3, 3, -2, 4, -6, 6, 2, 8, 4, 8};

// (mu0 m_c + lambda0 l_c) / 72 per class, in single precision rounded like the entries of Kc
template <typename T>
struct KcReg {
  T v[10];
  // Kc[I][J][r][s]; with constant arguments this folds to one register (and a sign)
  __device__ __forceinline__ T operator()(int I, int J, int r, int s) const {
    const int m = q1_mu72(I, J, r, s), l = q1_la72(I, J, r, s);
    const bool neg = m < 0 || (m == 0 && l < 0);
    const T k = v[q1_class(neg ? -m : m, neg ? -l : l)];
    return neg ? -k : k;
  }
};

// The level-0 operator at large sizes streams from HBM, whose latency its
// resident warps do not cover: a CTA asks for the data of the one that will
// follow it on the chip (about one wave of CTAs ahead) to be brought into L2
// (1024^3, without it / with it: FP32 residual 1039 / 885 us, FP64 matvec 1824 /
// 1801 us).  The Gauss-Seidel passes, whose gathers
// keep more lines in flight, lost by it (1476 -> 1686 us a sweep), as by prefetches of their
// later gathers into L1 (1453 -> 1574 us).
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
constexpr int WAVE_SMS = 148;

// the packed node record of level 0: (u_x, u_y, u_z, E)
template <typename T>
struct Pack4;
template <>
struct Pack4<float> {
  using type = float4;
  static __device__ __forceinline__ float4 make(float a, float b, float c, float d) { return make_float4(a, b, c, d); }
};
template <>
struct Pack4<double> {
  using type = double4;
  static __device__ __forceinline__ double4 make(double a, double b, double c, double d) {
    return make_double4(a, b, c, d);
  }
};

// Slots of the packed level-0 iterate: colour-major inside a block (the 16 nodes
// of each coordinate-parity colour contiguous), so that a colour pass's gather
// of one neighbour offset reads whole 128-byte lines (FP32: 8 nodes a line, two
// lines a block) instead of every other record of eight lines.  The terms of
// the three axes add up.
__host__ __device__ __forceinline__ constexpr int packed_x(int x) { return (x & 1) << 6 | (x & 2) << 2; }
__host__ __device__ __forceinline__ constexpr int packed_y(int y) { return (y & 1) << 5 | (y & 2) << 1; }
__host__ __device__ __forceinline__ constexpr int packed_z(int z) { return (z & 1) << 4 | (z & 7) >> 1; }
// index in the packed iterate of node g (block * 128 + x * 32 + y * 8 + z)
template <typename I>
__host__ __device__ __forceinline__ constexpr I packed_index(I g) {
  const int e = int(g & 127);
  return (g & ~I(127)) | I(packed_x(e >> 5) | packed_y(e >> 3 & 3) | packed_z(e & 7));
}

// Inverse of a node's symmetric 3x3 diagonal block {00, 11, 22, 01, 02, 12}, the
// rows of Dirichlet components replaced by the identity and then dropped.  In
// FP32 the block is scaled by a power of two first (exact): its determinant,
// the cube of a stiffness, underflows on coarse levels and for soft material.
template <typename T>
__device__ __forceinline__ void diagonal_inverse(T d0, T d1, T d2, T d3, T d4, T d5, uint32_t fl, T* a) {
  const bool fx = fl & DIR_X, fy = fl & DIR_Y, fz = fl & DIR_Z;
  T s = 1;
  if (sizeof(T) == 4) {
    s = T(__int_as_float(0x7f000000 - (__float_as_int(float(d0 + d1 + d2)) & 0x7f800000)));
    d0 *= s, d1 *= s, d2 *= s, d3 *= s, d4 *= s, d5 *= s;
  }
  if (fx) { d0 = 1; d3 = 0; d4 = 0; }
  if (fy) { d1 = 1; d3 = 0; d5 = 0; }
  if (fz) { d2 = 1; d4 = 0; d5 = 0; }
  const T m11 = d1 * d2 - d5 * d5, m12 = d5 * d4 - d2 * d3, m13 = d3 * d5 - d4 * d1;
  const T m22 = d2 * d0 - d4 * d4, m23 = d4 * d3 - d0 * d5, m33 = d0 * d1 - d3 * d3;
  const T inv = T(1) / (d0 * m11 + d3 * m12 + d4 * m13) * s;
  a[0] = fx ? T(0) : m11 * inv;
  a[1] = fy ? T(0) : m22 * inv;
  a[2] = fz ? T(0) : m33 * inv;
  a[3] = fx || fy ? T(0) : m12 * inv;
  a[4] = fx || fz ? T(0) : m13 * inv;
  a[5] = fy || fz ? T(0) : m23 * inv;
}

// Programmatic dependent launch: kernels of the solve are launched so that they
// may start while their predecessor drains.  Each waits here until the
// predecessor has completed and its writes are visible, then lets its own
// successor be scheduled; code before the wait (a prologue) reads only data
// that no kernel of the solve writes (lists, neighbour tables, flags, E,
// stencils), since the predecessor may still be running.
__device__ __forceinline__ void pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---------------------------------------------------------------------------
// Level-0 matrix-free operator (solver/CPU_Kernels/SPGrid_Linear_Elasticity.h:96-344):
// OP_KU: out = dx*K*u, OP_RES: out = b - dx*K*u, OP_KUP: dx*K*u with Project
// and the CTA's partial u.(Ku) (the PCG matvec).
//
// The trilinear element is evaluated in the basis of the monomials xi^p, p in
// {0,1}^3, of its reference cube [-1,1]^3, where the energy almost decouples:
// of the 24 x 24 entries of the element matrix 33 remain (diagonal, the volume
// terms lambda tr, the shear pairs).  Corner values go to modes and modal
// forces back to corners by sums and differences along one axis after the
// other; edges and faces share them.  One thread marches a column of cells
// along x: it reads a node plane's four corners once for the cells on both
// sides, and hands its corner forces to the nodes through shared memory, plane
// by plane.  About 160 operations a cell, against 576 FMAs a node and 24 shared
// loads a node and cell in the nodal form.
// Two blocks per CTA of 96 threads (2 x 45 columns of cells, the block's 4 x 8
// and one layer below): 90 of 96 lanes work where one block would leave 19 of
// 64 idle.  Cells without material (E = 0) skip the modal part.
// PACKED: the iterate is the record u4 = (u, E) with the neighbour table nbrz
// (a zero pad block for missing blocks), else the planes of u, E and nbr (-1).
// Bound by L1 and by latency: the LSU data pipe is 81% busy in the FP32 residual,
// 72% in FP64, 64% in the FP64 matvec (256^3 shell), and the stalls are the
// plane loads (long scoreboard): a CTA's five steps are a chain of loads, about
// 15 dependent operations and a barrier each.  Registers allow 5 CTAs an SM in
// FP64, 9 in FP32, with 64 to 120 and 40 to 84 bytes spilled (1024^3 matvec and
// residual 1801 and 885 us; 4 / 8 CTAs, without spills in FP64: 1786 and 867; 6 / 10,
// 412 to 588 and 120 to 156 bytes: 2413 and 963).  At 1024^3 (340713 blocks), nodal
// form -> this: FP64 matvec 2240 -> 1801 us, FP32 residual 1348 -> 885 us; 48^3
// 14.3 -> 8.3 us and 11.9 -> 8.6 us.  (The operands of the node phase are
// requested at the step's start: 2010 and 962 us when loaded where used.)
// ---------------------------------------------------------------------------
enum { OP_KU = 0, OP_RES = 1, OP_KUP = 2 };

constexpr int MODAL_THREADS = 96, MODAL_BLOCKS = 2;

// dx/16 times the Lame parameters and their modal combinations
template <typename T>
struct ModalCoef {
  T m, l, A, L, M, B;  // mu, lambda, (3 mu + lambda)/3, lambda/3, mu/3, (4 mu + lambda)/9
  void set(double mu, double la, double dx) {
    const double mm = mu * dx / 16, ll = la * dx / 16;
    m = T(mm), l = T(ll), A = T((3 * mm + ll) / 3), L = T(ll / 3), M = T(mm / 3), B = T((4 * mm + ll) / 9);
  }
};

template <typename T, int OP, bool PACKED>
__global__ void __launch_bounds__(MODAL_THREADS, sizeof(T) == 8 ? 5 : 9) level0_modal_kernel(
    int nblocks, const int* __restrict__ nbr, const T* __restrict__ E, const T* __restrict__ u,
    const typename Pack4<T>::type* __restrict__ u4, const T* __restrict__ b, T* __restrict__ out, long N,
    ModalCoef<T> K, const uint32_t* __restrict__ flags, double* __restrict__ part) {
  __shared__ T sx[2][12][MODAL_THREADS];
  const int t = threadIdx.x;
  const int b0 = blockIdx.x * MODAL_BLOCKS;
  // this thread's column of cells, min corners at (cy, cz) - 1 of block b0 + blk:
  // 40 columns with cz > 0 a block, then the 5 with cz = 0 of each
  const int rest = t - 80;
  const int blk = t < 80 ? t / 40 : rest / 5, cy = t < 80 ? t % 40 / 8 : rest % 5, cz = t < 80 ? t % 8 + 1 : 0;
  const bool on = t < 90 && b0 + blk < nblocks;
  // first records of the column's four corners in the blocks behind, at and ahead of it in x
  int at[3][4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int y = cy - 1 + (k >> 1), z = cz - 1 + (k & 1);
    const int nb = (y < 0 ? 0 : (y > 3 ? 2 : 1)) * 3 + (z < 0 ? 0 : (z > 7 ? 2 : 1));
    const int yz = PACKED ? packed_y(y & 3) + packed_z(z & 7) : ((y & 3) << 3) + (z & 7);
#pragma unroll
    for (int g = 0; g < 3; ++g) {
      const int j = on ? __ldg(nbr + long(b0 + blk) * 27 + g * 9 + nb) : -1;
      at[g][k] = j < 0 ? -1 : (j << 7) + yz;
    }
  }
  {
    constexpr int PER = 128 / int(sizeof(T));                  // values per line
    constexpr int UL = (PACKED ? 4 : 3) * 128 / PER, EL = PACKED ? 0 : 128 / PER, BL = OP == OP_RES ? 3 * 128 / PER : 0;
    const int ahead = b0 + MODAL_BLOCKS * WAVE_SMS * (sizeof(T) == 8 ? 5 : 9);
    for (int l = t; l < MODAL_BLOCKS * (UL + EL + BL); l += MODAL_THREADS) {
      const int k = l / (UL + EL + BL), j = l % (UL + EL + BL);
      if (ahead + k >= nblocks) continue;
      const long first = long(ahead + k) * 128;
      if (j < UL) prefetch_l2(PACKED ? reinterpret_cast<const T*>(u4 + first) + j * PER
                                     : u + first + (j / (128 / PER)) * N + (j % (128 / PER)) * PER);
      else if (j < UL + EL) prefetch_l2(E + first + (j - UL) * PER);
      else prefetch_l2(b + first + ((j - UL - EL) / (128 / PER)) * N + ((j - UL - EL) % (128 / PER)) * PER);
    }
  }
  pdl_wait();
  // a node plane's four corners (plane 0 and 5: one node beyond the block), and
  // the stiffness of the cell ahead of it
  T R[4][3], eR = 0;
  auto fetch = [&](int plane, const int (&a)[4]) {
    const int ox = PACKED ? packed_x((plane + 3) & 3) : ((plane + 3) & 3) << 5;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      R[k][0] = R[k][1] = R[k][2] = T(0);
      if (k == 0) eR = T(0);
      if (a[k] < 0) continue;
      const int i = a[k] + ox;
      if (PACKED) {
        const auto r = u4[i];
        R[k][0] = r.x, R[k][1] = r.y, R[k][2] = r.z;
        if (k == 0) eR = r.w;
      } else {
        R[k][0] = u[i], R[k][1] = u[i + N], R[k][2] = u[i + 2 * N];
        if (k == 0) eR = E[i];
      }
    }
  };
  // its modes 1, z, y, yz
  auto face = [&](T (&m)[4][3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const T s0 = R[0][c] + R[1][c], s1 = R[2][c] + R[3][c], d0 = R[1][c] - R[0][c], d1 = R[3][c] - R[2][c];
      m[0][c] = s0 + s1;
      m[1][c] = d0 + d1;
      m[2][c] = s1 - s0;
      m[3][c] = d1 - d0;
    }
  };
  T P[4][3], H[4][3];  // the last plane's modes; the modal forces on it from the cell behind
  fetch(0, at[0]);
  face(P);
  T e = eR;
  fetch(1, at[1]);
#pragma unroll
  for (int k = 0; k < 4; ++k) H[k][0] = H[k][1] = H[k][2] = T(0);
  double dot = 0;
#pragma unroll
  for (int x = 0; x < 5; ++x) {  // cell x - 1, between node planes x - 1 and x of the block (x and x + 1 here)
    // what the nodes of the finished plane need besides the forces, requested early
    const int nc = t >> 5;  // warp c sums component c of the plane's 32 nodes
    T extra[MODAL_BLOCKS];
    uint32_t fl[MODAL_BLOCKS];
#pragma unroll
    for (int k = 0; k < MODAL_BLOCKS; ++k) {
      extra[k] = T(0);
      fl[k] = 0;
      if (x == 0 || OP == OP_KU || b0 + k >= nblocks) continue;
      const long node = long(b0 + k) * 128 + (x - 1) * 32 + (t & 31);
      extra[k] = OP == OP_RES ? b[node + nc * N] : u[node + nc * N];
      if (OP == OP_KUP) fl[k] = flags[node];
    }
    T Q[4][3];
    face(Q);
    const T e_next = eR;
    // the next plane's loads are in flight while this cell is computed
    if (x < 3) fetch(x + 2, at[1]);
    else if (x == 3) fetch(5, at[2]);
    if (e != T(0)) {
      T D[4][3], S1[3], S2[3], S3[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        S1[c] = P[1][c] + Q[1][c];
        S2[c] = P[2][c] + Q[2][c];
        S3[c] = P[3][c] + Q[3][c];
#pragma unroll
        for (int k = 0; k < 4; ++k) D[k][c] = Q[k][c] - P[k][c];
      }
      const T m = e * K.m, l = e * K.l, A = e * K.A, L = e * K.L, M = e * K.M, B = e * K.B;
      T G0[3], G1[3], G2[3], F1[3], F2[3], F3[3];  // forces of D[0..2], S1..S3
      const T lt = l * (D[0][0] + S2[1] + S1[2]), m2 = m + m;
      G0[0] = fma(m2, D[0][0], lt);
      F2[1] = fma(m2, S2[1], lt);
      F1[2] = fma(m2, S1[2], lt);
      G0[1] = F2[0] = m * (D[0][1] + S2[0]);
      G0[2] = F1[0] = m * (D[0][2] + S1[0]);
      F2[2] = F1[1] = m * (S2[2] + S1[1]);
      G1[0] = fma(A, D[1][0], L * S3[1]);
      F3[1] = fma(A, S3[1], L * D[1][0]);
      G1[2] = fma(A, D[1][2], L * D[2][1]);
      G2[1] = fma(A, D[2][1], L * D[1][2]);
      G2[0] = fma(A, D[2][0], L * S3[2]);
      F3[2] = fma(A, S3[2], L * D[2][0]);
      const T q = D[1][1] + S3[0] + D[2][2];
      G1[1] = M * (D[1][1] + q);
      F3[0] = M * (S3[0] + q);
      G2[2] = M * (D[2][2] + q);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const T G3 = B * D[3][c];
        H[0][c] -= G0[c];
        H[1][c] += F1[c] - G1[c];
        H[2][c] += F2[c] - G2[c];
        H[3][c] += F3[c] - G3;
        P[0][c] = G0[c];  // the next plane's share, kept in P while H is handed out
        P[1][c] = F1[c] + G1[c];
        P[2][c] = F2[c] + G2[c];
        P[3][c] = F3[c] + G3;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) P[k][0] = P[k][1] = P[k][2] = T(0);
    }
    if (x > 0) {  // plane x - 1 of the block is complete: corner forces to the nodes
      T(*ex)[MODAL_THREADS] = sx[x & 1];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const T e0 = H[0][c] - H[1][c], e1 = H[0][c] + H[1][c], o0 = H[2][c] - H[3][c], o1 = H[2][c] + H[3][c];
        ex[c][t] = e0 - o0;
        ex[3 + c][t] = e1 - o1;
        ex[6 + c][t] = e0 + o0;
        ex[9 + c][t] = e1 + o1;
      }
      __syncthreads();
      const int c = nc, y = (t >> 3) & 3, z = t & 7;
#pragma unroll
      for (int k = 0; k < MODAL_BLOCKS; ++k) {
        if (b0 + k >= nblocks) continue;
        const int q = k * 40 + (y + 1) * 8 + z;  // the column whose min corner is the node, and its neighbour in z
        const int qz = z > 0 ? q - 1 : 80 + k * 5 + y + 1;
        T f = (ex[c][q] + ex[3 + c][qz]) + (ex[6 + c][q - 8] + ex[9 + c][z > 0 ? q - 9 : qz - 1]);
        const long node = long(b0 + k) * 128 + (x - 1) * 32 + (t & 31), g = node + c * N;
        if (OP == OP_RES) {
          f = extra[k] - f;
        } else if (OP == OP_KUP) {
          if (fl[k] & (DIR_X << c)) f = 0;
          dot += double(extra[k]) * double(f);
        }
        out[g] = f;
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        H[k][c] = P[k][c];
        P[k][c] = Q[k][c];
      }
    e = e_next;
  }
  if (OP == OP_KUP) {
#pragma unroll
    for (int o = 16; o; o >>= 1) dot += __shfl_down_sync(0xffffffffu, dot, o);
    __shared__ double sd[3];
    if ((t & 31) == 0) sd[t >> 5] = dot;
    __syncthreads();
    if (t == 0) part[blockIdx.x] = (sd[0] + sd[1]) + sd[2];
  }
}

// ---------------------------------------------------------------------------
// Level-0 Gauss-Seidel colour pass over a compact list of the colour's nodes
// (solver/CPU_Kernels/SPGrid_Gauss_Seidel.h:876-1180), one node per thread.
// The residual is accumulated cell by cell, g_I = sum_J Kc[I][J] u_J over the
// node's 8 cells and f = sum_I E_I g_I, visiting the 27 neighbours one x-plane
// (9 nodes) at a time; a cell is folded into f after its last plane.  Same-
// colour nodes share no cell, so a pass updates u in place.  List entries
// ~node (negative) name nodes the pass does not update: only their Dirichlet
// components are cleared.  MINB bounds the registers (resident CTAs per SM):
// the pass is latency-bound, so occupancy is worth a few spilled registers.
// ---------------------------------------------------------------------------

// Addressing of the 3x3x3 neighbourhood of a level-0 node: per axis, the terms
// of the neighbour-block selector (into the block's 27-entry nbr row) and of the
// slot inside that block, for the offsets -1, 0, +1.
struct Nbhd {
  const int* nb;
  int sx[3], sy[3], sz[3], lx[3], ly[3], lz[3];
  __device__ __forceinline__ void init(const int* __restrict__ nbr, int g) {
    const int bi = g >> 7, e = g & 127;
    const int x = e >> 5, y = (e >> 3) & 3, z = e & 7;
    nb = nbr + long(bi) * 27;
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      const int xx = x + o - 1, yy = y + o - 1, zz = z + o - 1;
      sx[o] = (xx < 0 ? 0 : (xx > 3 ? 2 : 1)) * 9;
      sy[o] = (yy < 0 ? 0 : (yy > 3 ? 2 : 1)) * 3;
      sz[o] = zz < 0 ? 0 : (zz > 7 ? 2 : 1);
      lx[o] = (xx & 3) << 5;
      ly[o] = (yy & 3) << 3;
      lz[o] = zz & 7;
    }
  }
  // global index of the neighbour at offset (ix-1, iy-1, iz-1), -1 if its block is not active
  __device__ __forceinline__ int at(int ix, int iy, int iz) const {
    const int b = __ldg(nb + sx[ix] + sy[iy] + sz[iz]);
    return b < 0 ? -1 : (b << 7) + lx[ix] + ly[iy] + lz[iz];
  }
};

template <typename T, int MINB>
__global__ void __launch_bounds__(128, MINB) gs0_list_kernel(const int* __restrict__ list, int n,
                                                             const int* __restrict__ nbr, const T* __restrict__ E,
                                                             T* u, const T* __restrict__ b,
                                                             const uint32_t* __restrict__ flags, int N, T dx,
                                                             const __grid_constant__ ElementMatrix<T> K) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) {
    pdl_wait();
    return;
  }
  // prologue: list, flags, neighbour table and E do not change during a solve
  const int raw = list[t];
  const int g = raw >= 0 ? raw : ~raw;
  const uint32_t fl = flags[g];
  const bool fx = fl & DIR_X, fy = fl & DIR_Y, fz = fl & DIR_Z;
  Nbhd nh;
  nh.init(nbr, g);
  T Ec[8];
#pragma unroll
  for (int I = 0; I < 8; ++I) {  // the cell of corner I (min corner = node - I) sits at offset -I
    const int i = nh.at(1 - (I >> 2), 1 - ((I >> 1) & 1), 1 - (I & 1));
    Ec[I] = (raw < 0 || i < 0) ? T(0) : E[i];
  }
  pdl_wait();
  if (raw < 0) {
    if (fx) u[g] = T(0);
    if (fy) u[g + N] = T(0);
    if (fz) u[g + 2 * N] = T(0);
    return;
  }
  T gc[8][3], uc[3];
  T f[3] = {0, 0, 0}, dg[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int I = 0; I < 8; ++I) gc[I][0] = gc[I][1] = gc[I][2] = T(0);
#pragma unroll
  for (int px = 0; px < 3; ++px) {
    T up[9][3];
#pragma unroll
    for (int p = 0; p < 9; ++p) {
      const int iy = p / 3, iz = p % 3;
      const int i = (px == 1 && p == 4) ? g : nh.at(px, iy, iz);
      up[p][0] = i < 0 ? T(0) : u[i];
      up[p][1] = i < 0 ? T(0) : u[i + N];
      up[p][2] = i < 0 ? T(0) : u[i + 2 * N];
    }
    if (px == 1) {
      uc[0] = up[4][0];
      uc[1] = up[4][1];
      uc[2] = up[4][2];
    }
#pragma unroll
    for (int I = 0; I < 8; ++I) {
      const int Ix = I >> 2, Iy = (I >> 1) & 1, Iz = I & 1;
      const int Jx = px - 1 + Ix;
      if (Jx < 0 || Jx > 1) continue;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int Jy = q >> 1, Jz = q & 1;
        const int p = (Jy - Iy + 1) * 3 + (Jz - Iz + 1);
        const int k = (I * 8 + Jx * 4 + Jy * 2 + Jz) * 9;
#pragma unroll
        for (int v = 0; v < 3; ++v)
#pragma unroll
          for (int w = 0; w < 3; ++w) gc[I][v] = fma(K.v[k + v * 3 + w], up[p][w], gc[I][v]);
      }
      if (Jx == 1) {  // last plane of this cell
#pragma unroll
        for (int v = 0; v < 3; ++v) f[v] = fma(Ec[I], gc[I][v], f[v]);
        const int kd = (I * 8 + I) * 9;
        dg[0] = fma(K.v[kd + 0], Ec[I], dg[0]);
        dg[1] = fma(K.v[kd + 4], Ec[I], dg[1]);
        dg[2] = fma(K.v[kd + 8], Ec[I], dg[2]);
        dg[3] = fma(K.v[kd + 1], Ec[I], dg[3]);
        dg[4] = fma(K.v[kd + 2], Ec[I], dg[4]);
        dg[5] = fma(K.v[kd + 5], Ec[I], dg[5]);
      }
    }
  }
  // u += D^{-1} (b - K u), Dirichlet rows replaced by the identity
  const T r0 = b[g] - f[0] * dx, r1 = b[g + N] - f[1] * dx, r2 = b[g + 2 * N] - f[2] * dx;
  T a[6];
  diagonal_inverse<T>(dg[0] * dx, dg[1] * dx, dg[2] * dx, dg[3] * dx, dg[4] * dx, dg[5] * dx, fl, a);
  const T a0 = a[0], a1 = a[1], a2 = a[2], a3 = a[3], a4 = a[4], a5 = a[5];
  T v0 = uc[0] + r0 * a0 + r1 * a3 + r2 * a4;
  T v1 = uc[1] + r0 * a3 + r1 * a1 + r2 * a5;
  T v2 = uc[2] + r0 * a4 + r1 * a5 + r2 * a2;
  if (fx) v0 = 0;
  if (fy) v1 = 0;
  if (fz) v2 = 0;
  u[g] = v0;
  u[g + N] = v1;
  u[g + 2 * N] = v2;
}

// ---------------------------------------------------------------------------
// Packed level 0 of the V-cycle (mixed and FP64 modes).  The iterate of level 0
// is one record per node, (u_x, u_y, u_z, E of the node's cell): the 27-point
// gathers of the smoother and the plane loads of the residual then read a
// node's displacement and its cell's stiffness scale in one access (16 B in
// FP32, 32 B in FP64), the same bytes as three planes of u plus the E plane.
// ---------------------------------------------------------------------------

// u4 = (0, 0, 0, E): the zero start of the V-cycle's level-0 correction
template <typename T>
__global__ void reset_u4_kernel(typename Pack4<T>::type* __restrict__ u4, const T* __restrict__ E, long N) {
  pdl_wait();
  const long i = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < N) u4[packed_index(i)] = Pack4<T>::make(T(0), T(0), T(0), E[i]);
}

// gs0_list_kernel on the packed iterate (one record gather per neighbour; the
// cells' E come with the nodes at offsets -I).  nbrz names the zero pad block
// (index nb) for missing neighbours, so the gathers need no test.  A node's
// neighbourhood lies in at most eight blocks (a block is even, so a node next to
// a face has one face per axis): their indices are loaded once, and each gather
// selects one by the axes it crosses a face on.  Bound by the latency of the
// gathers: at 256^3 (FP32) the long-scoreboard stalls lead at 42% of the warps
// resident, with the LSU data pipe 40% and DRAM 45% busy.  Every colour streams
// the iterate once: at 1024^3 8 x 0.70 GB, about 6.9 GB of DRAM traffic in 1411 us
// a sweep (FP32).  FP64 at 512^3 893 -> 664 us a sweep by the layout, 48^3 47 -> 34 us.
template <typename T, int MINB>
__global__ void __launch_bounds__(128, MINB) gs0_list4_kernel(const int* __restrict__ list, int n,
                                                              const int* __restrict__ nbrz,
                                                              typename Pack4<T>::type* u4, const T* __restrict__ b,
                                                              const uint32_t* __restrict__ flags, int N, T dx,
                                                              const KcReg<T> K) {
  using V = typename Pack4<T>::type;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) {
    pdl_wait();
    return;
  }
  const int raw = list[t];
  const int g = raw >= 0 ? raw : ~raw;
  const uint32_t fl = flags[g];
  const bool fx = fl & DIR_X, fy = fl & DIR_Y, fz = fl & DIR_Z;
  const int x = (g >> 5) & 3, y = (g >> 3) & 3, z = g & 7;
  // per axis the face the node lies next to: -1, +1 or 0
  const int ax = x == 0 ? -1 : (x == 3 ? 1 : 0), ay = y == 0 ? -1 : (y == 3 ? 1 : 0), az = z == 0 ? -1 : (z == 7 ? 1 : 0);
  int blk[2][2][2];  // first records of the blocks across the faces
  {
    const int* nb = nbrz + long(g >> 7) * 27 + 13;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      blk[i >> 2][i >> 1 & 1][i & 1] = __ldg(nb + ((i >> 2) ? ax * 9 : 0) + ((i >> 1 & 1) ? ay * 3 : 0) + ((i & 1) ? az : 0)) << 7;
  }
  const int gx[3] = {packed_x((x + 3) & 3), packed_x(x), packed_x((x + 1) & 3)};
  const int gy[3] = {packed_y((y + 3) & 3), packed_y(y), packed_y((y + 1) & 3)};
  const int gz[3] = {packed_z((z + 7) & 7), packed_z(z), packed_z((z + 1) & 7)};
  const int own = blk[0][0][0] + gx[1] + gy[1] + gz[1];
  pdl_wait();
  if (raw < 0) {
    V v = u4[own];
    if (fx) v.x = T(0);
    if (fy) v.y = T(0);
    if (fz) v.z = T(0);
    u4[own] = v;
    return;
  }
  T gc[8][3], Ec[8], uc[3];
  T f[3] = {0, 0, 0}, dg[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int I = 0; I < 8; ++I) gc[I][0] = gc[I][1] = gc[I][2] = T(0);
#pragma unroll
  for (int px = 0; px < 3; ++px) {
    T up[9][3];
    const bool cx = px != 1 && ax == px - 1;  // this plane lies across the x face
#pragma unroll
    for (int p = 0; p < 9; ++p) {
      const int iy = p / 3, iz = p % 3;
      const bool cy = iy != 1 && ay == iy - 1, cz = iz != 1 && az == iz - 1;
      const int b00 = cx ? blk[1][0][0] : blk[0][0][0], b01 = cx ? blk[1][0][1] : blk[0][0][1];
      const int b10 = cx ? blk[1][1][0] : blk[0][1][0], b11 = cx ? blk[1][1][1] : blk[0][1][1];
      const int base = cy ? (cz ? b11 : b10) : (cz ? b01 : b00);
      const V v = u4[base + gx[px] + gy[iy] + gz[iz]];
      up[p][0] = v.x;
      up[p][1] = v.y;
      up[p][2] = v.z;
      if (px <= 1 && iy <= 1 && iz <= 1) Ec[(1 - px) * 4 + (1 - iy) * 2 + (1 - iz)] = v.w;
    }
    if (px == 1) {
      uc[0] = up[4][0];
      uc[1] = up[4][1];
      uc[2] = up[4][2];
    }
#pragma unroll
    for (int I = 0; I < 8; ++I) {
      const int Ix = I >> 2, Iy = (I >> 1) & 1, Iz = I & 1;
      const int Jx = px - 1 + Ix;
      if (Jx < 0 || Jx > 1) continue;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int Jy = q >> 1, Jz = q & 1;
        const int p = (Jy - Iy + 1) * 3 + (Jz - Iz + 1);
        const int J = Jx * 4 + Jy * 2 + Jz;
#pragma unroll
        for (int v = 0; v < 3; ++v)
#pragma unroll
          for (int w = 0; w < 3; ++w) gc[I][v] = fma(K(I, J, v, w), up[p][w], gc[I][v]);
      }
      if (Jx == 1) {
#pragma unroll
        for (int v = 0; v < 3; ++v) f[v] = fma(Ec[I], gc[I][v], f[v]);
        dg[0] = fma(K(I, I, 0, 0), Ec[I], dg[0]);
        dg[1] = fma(K(I, I, 1, 1), Ec[I], dg[1]);
        dg[2] = fma(K(I, I, 2, 2), Ec[I], dg[2]);
        dg[3] = fma(K(I, I, 0, 1), Ec[I], dg[3]);
        dg[4] = fma(K(I, I, 0, 2), Ec[I], dg[4]);
        dg[5] = fma(K(I, I, 1, 2), Ec[I], dg[5]);
      }
    }
  }
  const T r0 = b[g] - f[0] * dx, r1 = b[g + N] - f[1] * dx, r2 = b[g + 2 * N] - f[2] * dx;
  T a[6];
  diagonal_inverse<T>(dg[0] * dx, dg[1] * dx, dg[2] * dx, dg[3] * dx, dg[4] * dx, dg[5] * dx, fl, a);
  const T a0 = a[0], a1 = a[1], a2 = a[2], a3 = a[3], a4 = a[4], a5 = a[5];
  T v0 = uc[0] + r0 * a0 + r1 * a3 + r2 * a4;
  T v1 = uc[1] + r0 * a3 + r1 * a1 + r2 * a5;
  T v2 = uc[2] + r0 * a4 + r1 * a5 + r2 * a2;
  if (fx) v0 = 0;
  if (fy) v1 = 0;
  if (fz) v2 = 0;
  u4[own] = Pack4<T>::make(v0, v1, v2, Ec[0]);  // corner I = 0: the node's own cell
}

// The colour pass for few nodes (a boundary band, a small level: up to
// GS_CELL_NODES of them): such a pass is bound by one thread's chain of dependent loads
// and its 600 FMAs, so eight threads share a node, thread I taking the cell of
// which the node is corner I.
// The Q1 element is symmetric under reflections, K(I, J) = S K(0, I^J) S with S
// = diag(-1 on the axes where I has its bit) (checked on the host at set-up);
// looping over J' = I^J keeps the coefficients K(0, J') compile-time register
// selections while the corner J a thread reads varies with I.  Per thread: 8
// gathers and 72 FMA; the cells' E g and diagonal blocks are summed over the
// eight threads with shuffles and thread 0 updates the node.  Same products as
// gs0_list4_kernel, summed in another order.  PACKED: on u4 with nbrz, else on
// the planes of u with E and nbr (-1 for missing blocks).
// The line is where a sweep takes as long either way (us a sweep of eight passes;
// box with that many nodes a pass, eight threads / one thread a node):
//   FP32 packed  14706 31.2 / 35.5, 20796 37.0 / 37.7, 32757 50.4 / 41.3
//   FP64 packed   2460 29.7 / 34.2,  3048 30.4 / 28.6,  4492 32.0 / 28.6
//   FP64 planes  34328 74.4 / 87.8, 44738 88.8 / 86.2, 57066 107.4 / 93.4
// (FP32 planes: the unit sweep of a mixed session only, with the line of FP64.)
template <typename T, bool PACKED>
constexpr int GS_CELL_NODES = !PACKED ? 40960 : sizeof(T) == 4 ? 20480 : 2560;
template <typename T, bool PACKED>
__global__ void __launch_bounds__(128) gs0_cell_kernel(const int* __restrict__ list, int n,
                                                       const int* __restrict__ nbr,
                                                       typename Pack4<T>::type* u4, T* u, const T* __restrict__ E,
                                                       const T* __restrict__ b,
                                                       const uint32_t* __restrict__ flags, int N, T dx,
                                                       const KcReg<T> K) {
  using V = typename Pack4<T>::type;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = t >> 3, I = t & 7;  // groups of 8 threads never straddle a warp
  if (k >= n) {
    pdl_wait();
    return;
  }
  const int raw = list[k];
  const int g = raw >= 0 ? raw : ~raw;
  const uint32_t fl = flags[g];
  const bool fx = fl & DIR_X, fy = fl & DIR_Y, fz = fl & DIR_Z;
  // per axis: block selector and slot for offset 0 and for the offset 1 - 2 I_a
  // towards the cell's other corners
  const int bi = g >> 7, e = g & 127;
  const int x = e >> 5, y = (e >> 3) & 3, z = e & 7;
  const int Ix = I >> 2, Iy = (I >> 1) & 1, Iz = I & 1;
  const int x1 = x + 1 - 2 * Ix, y1 = y + 1 - 2 * Iy, z1 = z + 1 - 2 * Iz;
  const int sx[2] = {9, (x1 < 0 ? 0 : (x1 > 3 ? 2 : 1)) * 9}, sy[2] = {3, (y1 < 0 ? 0 : (y1 > 3 ? 2 : 1)) * 3};
  const int sz[2] = {1, z1 < 0 ? 0 : (z1 > 7 ? 2 : 1)};
  const int lx[2] = {PACKED ? packed_x(x) : x << 5, PACKED ? packed_x(x1 & 3) : (x1 & 3) << 5};
  const int ly[2] = {PACKED ? packed_y(y) : y << 3, PACKED ? packed_y(y1 & 3) : (y1 & 3) << 3};
  const int lz[2] = {PACKED ? packed_z(z) : z, PACKED ? packed_z(z1 & 7) : z1 & 7};
  const int* nb = nbr + long(bi) * 27;
  int idx[8];
#pragma unroll
  for (int Jp = 0; Jp < 8; ++Jp) {
    const int a = Jp >> 2, c = (Jp >> 1) & 1, d = Jp & 1;
    const int k27 = __ldg(nb + sx[a] + sy[c] + sz[d]);
    idx[Jp] = !PACKED && k27 < 0 ? -1 : (k27 << 7) + lx[a] + ly[c] + lz[d];
  }
  T Ec = 0;  // the cell's min corner carries its E: J = 0, so J' = I
  if (!PACKED) {
    int at = idx[0];
#pragma unroll
    for (int Jp = 1; Jp < 8; ++Jp)
      if (Jp == I) at = idx[Jp];
    Ec = (raw < 0 || at < 0) ? T(0) : E[at];
  }
  pdl_wait();
  if (raw < 0) {
    if (I == 0) {
      if (PACKED) {
        V v = u4[idx[0]];
        if (fx) v.x = T(0);
        if (fy) v.y = T(0);
        if (fz) v.z = T(0);
        u4[idx[0]] = v;
      } else {
        if (fx) u[g] = T(0);
        if (fy) u[g + N] = T(0);
        if (fz) u[g + 2 * N] = T(0);
      }
    }
    return;
  }
  if (sizeof(T) == 4 && I == 0) {  // the right-hand side, read after the shuffles, into L1 now
    asm volatile("prefetch.global.L1 [%0];" ::"l"(b + g));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(b + g + N));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(b + g + 2 * N));
  }
  const T s0 = Ix ? T(-1) : T(1), s1 = Iy ? T(-1) : T(1), s2 = Iz ? T(-1) : T(1);
  T gv[3] = {0, 0, 0}, uc[3] = {0, 0, 0};
#pragma unroll
  for (int Jp = 0; Jp < 8; ++Jp) {
    V v = Pack4<T>::make(T(0), T(0), T(0), T(0));
    if (PACKED) {
      v = u4[idx[Jp]];
    } else if (idx[Jp] >= 0) {
      v.x = u[idx[Jp]];
      v.y = u[idx[Jp] + N];
      v.z = u[idx[Jp] + 2 * N];
    }
    if (Jp == 0) {  // J = I: the node itself
      uc[0] = v.x;
      uc[1] = v.y;
      uc[2] = v.z;
    }
    if (PACKED && Jp == I) Ec = v.w;
    const T w0 = s0 * v.x, w1 = s1 * v.y, w2 = s2 * v.z;
#pragma unroll
    for (int r = 0; r < 3; ++r)
      gv[r] = fma(K(0, Jp, r, 0), w0, fma(K(0, Jp, r, 1), w1, fma(K(0, Jp, r, 2), w2, gv[r])));
  }
  // this cell's share of the node's row and of its diagonal block
  T red[9] = {Ec * s0 * gv[0], Ec * s1 * gv[1], Ec * s2 * gv[2],
              Ec * K(0, 0, 0, 0), Ec * K(0, 0, 1, 1), Ec * K(0, 0, 2, 2),
              Ec * (s0 * s1) * K(0, 0, 0, 1), Ec * (s0 * s2) * K(0, 0, 0, 2), Ec * (s1 * s2) * K(0, 0, 1, 2)};
  // the eight threads of a node take the same branches: shuffle within the group only
  const unsigned group = 0xffu << (threadIdx.x & 24);
#pragma unroll
  for (int o = 4; o; o >>= 1)
#pragma unroll
    for (int q = 0; q < 9; ++q) red[q] += __shfl_xor_sync(group, red[q], o);
  if (I != 0) return;
  const T r0 = b[g] - red[0] * dx, r1 = b[g + N] - red[1] * dx, r2 = b[g + 2 * N] - red[2] * dx;
  T a[6];
  diagonal_inverse<T>(red[3] * dx, red[4] * dx, red[5] * dx, red[6] * dx, red[7] * dx, red[8] * dx, fl, a);
  const T a0 = a[0], a1 = a[1], a2 = a[2], a3 = a[3], a4 = a[4], a5 = a[5];
  T v0 = uc[0] + r0 * a0 + r1 * a3 + r2 * a4;
  T v1 = uc[1] + r0 * a3 + r1 * a1 + r2 * a5;
  T v2 = uc[2] + r0 * a4 + r1 * a5 + r2 * a2;
  if (fx) v0 = 0;
  if (fy) v1 = 0;
  if (fz) v2 = 0;
  if (PACKED) {
    u4[idx[0]] = Pack4<T>::make(v0, v1, v2, Ec);  // thread 0: the node's own cell
  } else {
    u[g] = v0;
    u[g + N] = v1;
    u[g + 2 * N] = v2;
  }
}

// ---------------------------------------------------------------------------
// Coarse-level stencil operators (solver/MG/SPGrid_Stencil_Multiply.h:15-280)
// ---------------------------------------------------------------------------
struct GridView {
  const int* bgrid;  // dense block grid -> active block index or -1
  int gx, gy, gz;
  __device__ __forceinline__ long node(int x, int y, int z) const {
    if (x < 0 || y < 0 || z < 0) return -1;
    const int bx = x >> 2, by = y >> 2, bz = z >> 3;
    if (bx >= gx || by >= gy || bz >= gz) return -1;
    const int b = bgrid[(long(bx) * gy + by) * gz + bz];
    return b < 0 ? -1 : long(b) * 128 + ((x & 3) << 5) + ((y & 3) << 3) + (z & 7);
  }
};

enum { SOP_MUL = 0, SOP_RES = 1, SOP_GS = 2 };

// One warp per node: lane q < 27 multiplies the 3x3 block of spoke q with the
// neighbour's u, the warp sums the three components.  Stencils are node-major,
// A[node*243 + q*9 + v*3 + w]: lane q reads its nine entries, and the warp's
// reads together cover one contiguous row (972 bytes in FP32), which L1
// fetches once.  The neighbour's block comes from the level's 27-entry
// neighbour table (one load that needs only the block index, issued with the
// flags load), and the row is loaded whether or not the neighbour exists, so
// no load waits for another; a missing neighbour's spoke is skipped.  GS
// updates the nodes of a list: the active nodes of one colour, or the active
// boundary-band nodes of one colour (no node has a neighbour of its own
// colour, so the order inside a pass does not change the result).
// Results on Dirichlet components are zeroed (Project).  The reference
// projects the whole level after every colour; here only updated nodes are
// projected, which is the same because the V-cycle keeps u zero on Dirichlet
// components (cleared levels, projected transfers and updates).
template <typename T, int OP>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 8 : 5) stencil_op_kernel(const int* __restrict__ list, int count,
                                                         const int* __restrict__ nbr,
                                                         const T* __restrict__ A, const uint32_t* __restrict__ flags,
                                                         const T* u, T* out_u, const T* __restrict__ b,
                                                         T* __restrict__ out, long N, int round_out) {
  const long w = (long(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;  // one warp per node
  const int lane = threadIdx.x & 31;
  // GS: node list[w] of the `count` listed; MUL / RES: node w of the first `count` blocks
  if (w >= (OP == SOP_GS ? long(count) : long(count) * 128)) {
    pdl_wait();
    return;
  }
  const long gidx = OP == SOP_GS ? long(list[w]) : w;
  const int bi = int(gidx >> 7), e = int(gidx & 127);
  // prologue: flags, neighbour table and stencil row do not change during a solve
  // neighbour (X, Y, Z) of the node in block coordinates, -1..4 x -1..4 x -1..8
  const int X = (e >> 5) + lane / 9 - 1, Y = ((e >> 3) & 3) + (lane / 3) % 3 - 1, Z = (e & 7) + lane % 3 - 1;
  const uint32_t fl = flags[gidx];
  const int nbk = lane < 27 ? nbr[long(bi) * 27 + (X < 0 ? 0 : (X > 3 ? 2 : 1)) * 9 + (Y < 0 ? 0 : (Y > 3 ? 2 : 1)) * 3 +
                                  (Z < 0 ? 0 : (Z > 7 ? 2 : 1))]
                            : -1;
  // an inactive node's row is zero (the operator build writes only the rows of
  // active nodes into zeroed storage): its result needs no neighbour
  if (OP != SOP_GS && !(fl & ACTIVE_NODE)) {
    pdl_wait();
    if (lane < 3) {
      const T r = OP == SOP_RES ? b[gidx + lane * N] : T(0);
      out[gidx + lane * N] = (fl & (DIR_X << lane)) ? T(0) : (round_out ? T(round_to_float(r)) : r);
    }
    return;
  }
  T a[9];
  if (lane < 27) {
    const T* ap = A + gidx * 243 + lane * 9;
#pragma unroll
    for (int k = 0; k < 9; ++k) a[k] = ap[k];
  } else {
#pragma unroll
    for (int k = 0; k < 9; ++k) a[k] = T(0);
  }
  const long n = nbk < 0 ? -1 : long(nbk) * 128 + ((X & 3) << 5) + ((Y & 3) << 3) + (Z & 7);
  T inv[6] = {0, 0, 0, 0, 0, 0};  // off the pass's chain: before the wait
  if (OP == SOP_GS && lane == 0) {
    const T* c = A + gidx * 243 + 13 * 9;
    diagonal_inverse<T>(c[0], c[4], c[8], c[1], c[2], c[5], fl, inv);
  }
  pdl_wait();
  // lane 0 reads its right-hand side (and in GS its own u) after the warp's
  // reduction; prefetched here, after the wait, those loads find them in L1
  if (OP != SOP_MUL && lane == 0) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(b + gidx));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(b + gidx + N));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(b + gidx + 2 * N));
    if (OP == SOP_GS) {
      asm volatile("prefetch.global.L1 [%0];" ::"l"(u + gidx));
      asm volatile("prefetch.global.L1 [%0];" ::"l"(u + gidx + N));
      asm volatile("prefetch.global.L1 [%0];" ::"l"(u + gidx + 2 * N));
    }
  }
  T f0 = 0, f1 = 0, f2 = 0;
  if (n >= 0) {
    const T ux = u[n], uy = u[n + N], uz = u[n + 2 * N];
    f0 = a[0] * ux + a[1] * uy + a[2] * uz;
    f1 = a[3] * ux + a[4] * uy + a[5] * uz;
    f2 = a[6] * ux + a[7] * uy + a[8] * uz;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    f0 += __shfl_down_sync(0xffffffffu, f0, o);
    f1 += __shfl_down_sync(0xffffffffu, f1, o);
    f2 += __shfl_down_sync(0xffffffffu, f2, o);
  }
  if (lane != 0) return;
  if (OP == SOP_MUL) {
    out[gidx] = (fl & DIR_X) ? T(0) : f0;
    out[gidx + N] = (fl & DIR_Y) ? T(0) : f1;
    out[gidx + 2 * N] = (fl & DIR_Z) ? T(0) : f2;
    return;
  }
  const T r0 = b[gidx] - f0, r1 = b[gidx + N] - f1, r2 = b[gidx + 2 * N] - f2;
  if (OP == SOP_RES) {
    T o0 = (fl & DIR_X) ? T(0) : r0, o1 = (fl & DIR_Y) ? T(0) : r1, o2 = (fl & DIR_Z) ? T(0) : r2;
    if (round_out) { o0 = T(round_to_float(o0)); o1 = T(round_to_float(o1)); o2 = T(round_to_float(o2)); }
    out[gidx] = o0;
    out[gidx + N] = o1;
    out[gidx + 2 * N] = o2;
    return;
  }
  const bool fx = fl & DIR_X, fy = fl & DIR_Y, fz = fl & DIR_Z;
  T u0 = u[gidx] + (inv[0] * r0 + inv[3] * r1 + inv[4] * r2);
  T u1 = u[gidx + N] + (inv[3] * r0 + inv[1] * r1 + inv[5] * r2);
  T u2 = u[gidx + 2 * N] + (inv[4] * r0 + inv[5] * r1 + inv[2] * r2);
  if (fx) u0 = 0;
  if (fy) u1 = 0;
  if (fz) u2 = 0;
  out_u[gidx] = u0;
  out_u[gidx + N] = u1;
  out_u[gidx + 2 * N] = u2;
}

// ---------------------------------------------------------------------------
// Transfers (solver/MG/Restriction.h:52-88, solver/MG/Prolongation.h:151-193)
// ---------------------------------------------------------------------------
// coarse(c) = sum_{d in {-1,0,1}^3} w(d) fine(2c - (4,4,8) + d), w = prod (1/2,1,1/2);
// Dirichlet components zeroed afterwards.  One CTA per coarse block (launched
// with nb CTAs of 128 threads, thread = node): the 9x9x17 fine nodes the block
// reads are staged in shared memory once (the 27 fine blocks they lie in are
// looked up once), then every node sums its 27 in the reference's order; a
// missing fine node reads 0, which adds nothing.
template <typename T>
__global__ void __launch_bounds__(128) restrict_kernel(int nb, const int* __restrict__ coords,
                                                       const uint32_t* __restrict__ cflags, GridView fine,
                                                       const T* __restrict__ fin, long Nf, T* __restrict__ cout,
                                                       long Nc, T* __restrict__ zero) {
  constexpr int RX = 9, RY = 9, RZ = 17, RN = RX * RY * RZ;
  __shared__ T sf[3][RN];
  __shared__ int sblk[27];
  const int bi = blockIdx.x, e = threadIdx.x;
  if (bi >= nb) return;
  const int CX = coords[3 * bi], CY = coords[3 * bi + 1], CZ = coords[3 * bi + 2];
  const int x0 = 2 * CX - 5, y0 = 2 * CY - 5, z0 = 2 * CZ - 9;  // fine region origin
  const int bx0 = x0 >> 2, by0 = y0 >> 2, bz0 = z0 >> 3;
  if (e < 27) {  // block indices are fixed during a solve: looked up before the wait
    const int bx = bx0 + e / 9, by = by0 + (e / 3) % 3, bz = bz0 + e % 3;
    const long n = fine.node(bx * 4, by * 4, bz * 8);
    sblk[e] = n < 0 ? -1 : int(n >> 7);
  }
  pdl_wait();
  __syncthreads();
#pragma unroll 4
  for (int h = e; h < RN; h += 128) {  // (four nodes of a thread in flight: the loop is bound by their latency)
    const int fx = x0 + h / (RY * RZ), fy = y0 + (h / RZ) % RY, fz = z0 + h % RZ;
    const int b = sblk[((fx >> 2) - bx0) * 9 + ((fy >> 2) - by0) * 3 + ((fz >> 3) - bz0)];
    T a = 0, c = 0, d = 0;
    if (b >= 0) {
      const long n = long(b) * 128 + ((fx & 3) << 5) + ((fy & 3) << 3) + (fz & 7);
      a = fin[n];
      c = fin[n + Nf];
      d = fin[n + 2 * Nf];
    }
    sf[0][h] = a;
    sf[1][h] = c;
    sf[2][h] = d;
  }
  __syncthreads();
  const int lx = e >> 5, ly = (e >> 3) & 3, lz = e & 7;
  T v0 = 0, v1 = 0, v2 = 0;
  for (int q = 0; q < 27; ++q) {
    const int i = q / 9, j = (q / 3) % 3, k = q % 3;
    const int h = (2 * lx + i) * (RY * RZ) + (2 * ly + j) * RZ + (2 * lz + k);
    const T w = T((i == 1 ? 1.0 : 0.5) * (j == 1 ? 1.0 : 0.5) * (k == 1 ? 1.0 : 0.5));
    v0 += w * sf[0][h];
    v1 += w * sf[1][h];
    v2 += w * sf[2][h];
  }
  const long t = long(bi) * 128 + e;
  const uint32_t fl = cflags[t];
  cout[t] = (fl & DIR_X) ? T(0) : v0;
  cout[t + Nc] = (fl & DIR_Y) ? T(0) : v1;
  cout[t + 2 * Nc] = (fl & DIR_Z) ? T(0) : v2;
  if (zero) zero[t] = zero[t + Nc] = zero[t + 2 * Nc] = T(0);  // the coarse iterate starts from zero
}

// The 3x3x5 coarse nodes that the 4x4x8 fine nodes of a fine block interpolate
// from ((f + (4,4,8)) >> 1 + {0,1}^3), staged in shared memory by one CTA per
// fine block (128 threads, thread = node); missing coarse nodes read 0.
template <typename T>
__device__ __forceinline__ void stage_coarse_patch(T (*sc)[45], int FX, int FY, int FZ, GridView coarse,
                                                   const T* __restrict__ cin, long Nc) {
  const int e = threadIdx.x;
  if (e < 45) {
    const long n = coarse.node(FX / 2 + 2 + e / 15, FY / 2 + 2 + (e / 5) % 3, FZ / 2 + 4 + e % 5);
    sc[0][e] = n < 0 ? T(0) : cin[n];
    sc[1][e] = n < 0 ? T(0) : cin[n + Nc];
    sc[2][e] = n < 0 ? T(0) : cin[n + 2 * Nc];
  }
  __syncthreads();
}

// fine(f) += sum of trilinear weights * coarse(((f + (4,4,8)) >> 1) + {0,1}^3); then
// Project (Dirichlet), optional float rounding, Project_Null_Space (inactive nodes),
// as Run_VCycle does after Prolongate (solver/MG/Multigrid_Hierarchy.h:600-603).
template <typename T>
__global__ void __launch_bounds__(128) prolongate_kernel(int nb, const int* __restrict__ coords,
                                                         const uint32_t* __restrict__ fflags, GridView coarse,
                                                         const T* __restrict__ cin, long Nc, T* __restrict__ fu,
                                                         long Nf, int round_out, int onto_zero) {
  __shared__ T sc[3][45];
  const int bi = blockIdx.x, e = threadIdx.x;
  if (bi >= nb) return;
  const int FX = coords[3 * bi], FY = coords[3 * bi + 1], FZ = coords[3 * bi + 2];
  pdl_wait();
  stage_coarse_patch<T>(sc, FX, FY, FZ, coarse, cin, Nc);
  const int lx = e >> 5, ly = (e >> 3) & 3, lz = e & 7;
  const long t = long(bi) * 128 + e;
  T v0 = 0, v1 = 0, v2 = 0;
  if (!onto_zero) v0 = fu[t], v1 = fu[t + Nf], v2 = fu[t + 2 * Nf];  // else fu is zero and only written
  for (int q = 0; q < 8; ++q) {
    const int ii = q >> 2, jj = (q >> 1) & 1, kk = q & 1;
    const double wx = (lx & 1) ? 0.5 : (ii ? 0.0 : 1.0);
    const double wy = (ly & 1) ? 0.5 : (jj ? 0.0 : 1.0);
    const double wz = (lz & 1) ? 0.5 : (kk ? 0.0 : 1.0);
    const T w = T(wx * wy * wz);
    if (!(w > T(0))) continue;
    const int h = ((lx >> 1) + ii) * 15 + ((ly >> 1) + jj) * 5 + (lz >> 1) + kk;
    v0 += w * sc[0][h];
    v1 += w * sc[1][h];
    v2 += w * sc[2][h];
  }
  const uint32_t fl = fflags[t];
  if (fl & DIR_X) v0 = 0;
  if (fl & DIR_Y) v1 = 0;
  if (fl & DIR_Z) v2 = 0;
  if (round_out) { v0 = T(round_to_float(v0)); v1 = T(round_to_float(v1)); v2 = T(round_to_float(v2)); }
  if (!(fl & ACTIVE_NODE)) v0 = v1 = v2 = 0;
  fu[t] = v0;
  fu[t + Nf] = v1;
  fu[t + 2 * Nf] = v2;
}

// prolongate_kernel into the packed level-0 iterate (E in .w is kept).  Only
// active nodes are read and written: the V-cycle starts from u = 0 and no
// kernel before this one writes an inactive node's displacement, so those
// slots already hold the zeros that the projection would write.
template <typename T>
__global__ void __launch_bounds__(128) prolongate4_kernel(int nb, const int* __restrict__ coords,
                                                          const uint32_t* __restrict__ fflags, GridView coarse,
                                                          const T* __restrict__ cin, long Nc,
                                                          typename Pack4<T>::type* __restrict__ fu4) {
  __shared__ T sc[3][45];
  const int bi = blockIdx.x, e = threadIdx.x;
  if (bi >= nb) return;
  const int FX = coords[3 * bi], FY = coords[3 * bi + 1], FZ = coords[3 * bi + 2];
  const long t = long(bi) * 128 + e;
  const uint32_t fl = fflags[t];
  pdl_wait();
  stage_coarse_patch<T>(sc, FX, FY, FZ, coarse, cin, Nc);
  if (!(fl & ACTIVE_NODE)) return;
  const int lx = e >> 5, ly = (e >> 3) & 3, lz = e & 7;
  const long at = packed_index(t);
  auto v = fu4[at];
  for (int q = 0; q < 8; ++q) {
    const int ii = q >> 2, jj = (q >> 1) & 1, kk = q & 1;
    const double wx = (lx & 1) ? 0.5 : (ii ? 0.0 : 1.0);
    const double wy = (ly & 1) ? 0.5 : (jj ? 0.0 : 1.0);
    const double wz = (lz & 1) ? 0.5 : (kk ? 0.0 : 1.0);
    const T w = T(wx * wy * wz);
    if (!(w > T(0))) continue;
    const int h = ((lx >> 1) + ii) * 15 + ((ly >> 1) + jj) * 5 + (lz >> 1) + kk;
    v.x += w * sc[0][h];
    v.y += w * sc[1][h];
    v.z += w * sc[2][h];
  }
  if (fl & DIR_X) v.x = 0;
  if (fl & DIR_Y) v.y = 0;
  if (fl & DIR_Z) v.z = 0;
  fu4[at] = v;
}

// ---------------------------------------------------------------------------
// Elementwise helpers
// ---------------------------------------------------------------------------
template <typename T>
__global__ void round_float_kernel(T* p, long n) {
  pdl_wait();
  long t = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t < n) p[t] = T(round_to_float(p[t]));
}

template <typename T>
__global__ void zero_list_kernel(T* p, const int* __restrict__ idx, int n) {
  pdl_wait();
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) p[idx[t]] = T(0);
}

// zero the three components of nodes without ACTIVE_NODE (Project_Null_Space.h:223-232)
template <typename T>
__global__ void project_null_kernel(T* p, const uint32_t* __restrict__ flags, long N) {
  pdl_wait();
  long t = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t < N && !(flags[t] & ACTIVE_NODE)) p[t] = p[t + N] = p[t + 2 * N] = T(0);
}

template <typename TD, typename TS>
__global__ void convert_kernel(TD* __restrict__ d, const TS* __restrict__ s, long n) {
  pdl_wait();
  long t = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t < n) d[t] = TD(s[t]);
}

}  // namespace sgs
