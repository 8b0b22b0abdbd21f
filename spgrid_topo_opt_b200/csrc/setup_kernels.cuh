// Set-up kernels: Galerkin coarse operators, Dirichlet deletion, dense bottom
// operator and its inverse.
#pragma once
#include "kernels.cuh"

namespace sgs {

// ---------------------------------------------------------------------------
// Galerkin operator of a coarse level at `depth` (solver/MG/Galerkin_Coarsen.h:40-100).
// The reference prolongates a unit vector cell by cell down to the finest level,
// applies the finest element matrices and restricts back.  The same quantity is
// assembled here in two steps.  For a coarse cell C and a finest cell p inside
// it, table[p][a][b][v][w] = sum_ij W_p[i][a] W_p[j][b] Kc[i][j][v][w] (W_p: the
// trilinear weights of C's corners at p's nodes), so the 24x24 cell matrix is
//     K_C[(a,v),(b,w)] = sum_p E_p * table[p][a][b][v][w],
// one row of a GEMM [cells x 8^depth] x [8^depth x 576].  Each active coarse
// node then sums the row blocks of its corner from its 8 incident cells.
// ---------------------------------------------------------------------------

// table[p][(a*8+b)*9 + v*3 + w], one thread per (p, a, b)
__global__ void galerkin_table_kernel(int depth, const __grid_constant__ ElementMatrix<double> K, double* __restrict__ table) {
  const long t = long(blockIdx.x) * blockDim.x + threadIdx.x;
  const int side = 1 << depth;
  const long npos = long(side) * side * side;
  if (t >= npos * 64) return;
  const long p = t >> 6;
  const int a = int(t >> 3) & 7, b = int(t) & 7;
  const int pc[3] = {int(p / (long(side) * side)), int((p / side) % side), int(p % side)};
  double Wa[8], Wb[8];
  for (int i = 0; i < 8; ++i) {
    double wa = 1, wb = 1;
    for (int ax = 0; ax < 3; ++ax) {
      const double tpos = double(pc[ax] + ((i >> (2 - ax)) & 1)) / side;
      wa *= ((a >> (2 - ax)) & 1) ? tpos : 1 - tpos;
      wb *= ((b >> (2 - ax)) & 1) ? tpos : 1 - tpos;
    }
    Wa[i] = wa;
    Wb[i] = wb;
  }
  double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int i = 0; i < 8; ++i) {
    if (Wa[i] == 0) continue;
    for (int j = 0; j < 8; ++j) {
      const double w = Wa[i] * Wb[j];
      if (w == 0) continue;
      for (int m = 0; m < 9; ++m) acc[m] += w * K.v[(i * 8 + j) * 9 + m];
    }
  }
  double* out = table + p * 576 + (a * 8 + b) * 9;
  for (int m = 0; m < 9; ++m) out[m] = acc[m];
}

// Cell matrices: C[cell][576] = sum_p E(origin_cell + p) * table[p][576], 64x64
// output tiles, the E operand gathered from the finest level on the fly.
constexpr int GT = 64;
__global__ void __launch_bounds__(256) galerkin_cell_kernel(int ncells, const int* __restrict__ origin, int depth,
                                                           GridView g0, const double* __restrict__ E0,
                                                           const double* __restrict__ table, double* __restrict__ C) {
  extern __shared__ double gsm[];
  double* sA = gsm;            // [64 cells][65]
  double* sB = gsm + GT * 65;  // [64 p][65]
  const int col0 = blockIdx.x * GT;
  const int cell0 = blockIdx.y * GT;
  const int side = 1 << depth;
  const long npos = long(side) * side * side;
  const int t = threadIdx.x, ty = t / 16, tx = t % 16;
  double acc[4][4] = {};
  for (long p0 = 0; p0 < npos; p0 += GT) {
    for (int i = t; i < GT * GT; i += 256) {
      const int r = i / GT, k = i % GT;
      const int cell = cell0 + r;
      const long p = p0 + k;
      double ev = 0;
      if (cell < ncells && p < npos) {
        const int px = int(p / (long(side) * side)), py = int((p / side) % side), pz = int(p % side);
        const long n = g0.node(origin[3 * cell] + px, origin[3 * cell + 1] + py, origin[3 * cell + 2] + pz);
        if (n >= 0) ev = E0[n];
      }
      sA[r * 65 + k] = ev;
    }
    __syncthreads();
    for (int i = t; i < GT * GT; i += 256) {
      const int k = i / GT, c = i % GT;
      const long p = p0 + k;
      sB[k * 65 + c] = p < npos ? table[p * 576 + col0 + c] : 0.0;
    }
    __syncthreads();
    for (int k = 0; k < GT; ++k) {
      double av[4], bv[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) av[r] = sA[(ty + 16 * r) * 65 + k];
#pragma unroll
      for (int s = 0; s < 4; ++s) bv[s] = sB[k * 65 + tx + 16 * s];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int s = 0; s < 4; ++s) acc[r][s] += av[r] * bv[s];
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int cell = cell0 + ty + 16 * r;
    if (cell >= ncells) continue;
#pragma unroll
    for (int s = 0; s < 4; ++s) C[long(cell) * 576 + col0 + tx + 16 * s] = acc[r][s];
  }
}

// Cell matrices of the next coarser level from this level's: a coarse cell
// covers 2x2x2 cells of the finer level (child d at finer cell 2c - (4,4,8) + d),
// and the trilinear basis of its corners restricted to a child is the child's
// basis times w_d[i][a], the weight of coarse corner a at child corner i (a
// product of 0, 1/2, 1 per axis, exact).  So
//     K_C[(a,v),(b,w)] = sum_d sum_ij w_d[i][a] w_d[j][b] K_d[(i,v),(j,w)],
// which equals the sum over the finest cells of galerkin_cell_kernel up to
// rounding, at 8 children instead of 8^depth positions per coarse cell.  One
// CTA of 576 threads per coarse cell, one output entry per thread, children in
// fixed order.
__global__ void __launch_bounds__(576) galerkin_coarsen_kernel(const int* __restrict__ ccoord, GridView gf,
                                                              const int* __restrict__ fine_cell_of_slot,
                                                              const double* __restrict__ Cf, double* __restrict__ Cc) {
  __shared__ double sK[8][576];
  __shared__ double sw[8][64];  // sw[d][i * 8 + a]
  __shared__ int child[8];
  const int cell = blockIdx.x, t = threadIdx.x;
  if (t < 8) {
    const int fx = 2 * ccoord[3 * cell] - 4 + ((t >> 2) & 1), fy = 2 * ccoord[3 * cell + 1] - 4 + ((t >> 1) & 1),
              fz = 2 * ccoord[3 * cell + 2] - 8 + (t & 1);
    const long n = gf.node(fx, fy, fz);
    child[t] = n >= 0 ? fine_cell_of_slot[n] : -1;
  }
  if (t < 512) {
    const int d = t >> 6, i = (t >> 3) & 7, a = t & 7;
    double w = 1;
    for (int ax = 0; ax < 3; ++ax) {
      const int sh = 2 - ax;
      const double pos = 0.5 * double(((d >> sh) & 1) + ((i >> sh) & 1));  // child corner in the coarse cell
      w *= ((a >> sh) & 1) ? pos : 1 - pos;
    }
    sw[d][i * 8 + a] = w;
  }
  __syncthreads();
  for (int d = 0; d < 8; ++d) sK[d][t] = child[d] >= 0 ? Cf[long(child[d]) * 576 + t] : 0.0;
  __syncthreads();
  const int a = t / 72, b = (t / 9) & 7, m = t % 9;
  double acc = 0;
  for (int d = 0; d < 8; ++d) {
    if (child[d] < 0) continue;
    for (int i = 0; i < 8; ++i) {
      const double wa = sw[d][i * 8 + a];
      if (wa == 0) continue;
      for (int j = 0; j < 8; ++j) {
        const double wab = wa * sw[d][j * 8 + b];
        if (wab != 0) acc = __fma_rn(wab, sK[d][(i * 8 + j) * 9 + m], acc);
      }
    }
  }
  Cc[long(cell) * 576 + t] = acc;
}

// Node stencils from the cell matrices: entry (q, v, w) sums the (corner, neighbour)
// blocks of the incident cells in a fixed order; spoke q is active when any of
// those blocks has a non-zero entry (Galerkin_Coarsen.h:79-93).  One CTA per node.
__global__ void __launch_bounds__(256) galerkin_assemble_kernel(const int* __restrict__ coords,
                                                               const uint32_t* __restrict__ flags,
                                                               const int* __restrict__ cell_of_slot, GridView g,
                                                               const double* __restrict__ C, double* __restrict__ A,
                                                               uint32_t* __restrict__ spokes, double dx) {
  __shared__ int scell[8];
  const long gidx = blockIdx.x;
  if (!(flags[gidx] & ACTIVE_NODE)) return;
  const int bi = int(gidx >> 7), e = int(gidx & 127);
  const int x = coords[3 * bi] + (e >> 5), y = coords[3 * bi + 1] + ((e >> 3) & 3), z = coords[3 * bi + 2] + (e & 7);
  const int t = threadIdx.x;
  if (t < 8) {
    const long n = g.node(x + (t >> 2) - 1, y + ((t >> 1) & 1) - 1, z + (t & 1) - 1);
    scell[t] = n >= 0 ? cell_of_slot[n] : -1;
  }
  __syncthreads();
  if (t < 243) {
    const int q = t / 9, vw = t % 9;
    const int qi = q / 9, qj = (q / 3) % 3, qk = q % 3;
    double s = 0;
    for (int c = 0; c < 8; ++c) {
      const int bx = qi - (c >> 2), by = qj - ((c >> 1) & 1), bz = qk - (c & 1);
      if (bx < 0 || bx > 1 || by < 0 || by > 1 || bz < 0 || bz > 1 || scell[c] < 0) continue;
      s += C[long(scell[c]) * 576 + ((7 - c) * 8 + ((bx << 2) | (by << 1) | bz)) * 9 + vw];
    }
    A[gidx * 243 + t] = s * dx;
  }
  if (t < 32) {
    bool nz = false;
    if (t < 27) {
      const int qi = t / 9, qj = (t / 3) % 3, qk = t % 3;
      for (int c = 0; c < 8; ++c) {
        const int bx = qi - (c >> 2), by = qj - ((c >> 1) & 1), bz = qk - (c & 1);
        if (bx < 0 || bx > 1 || by < 0 || by > 1 || bz < 0 || bz > 1 || scell[c] < 0) continue;
        const double* blk = C + long(scell[c]) * 576 + ((7 - c) * 8 + ((bx << 2) | (by << 1) | bz)) * 9;
        for (int k = 0; k < 9; ++k) nz |= blk[k] != 0.0;
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, nz);
    if (t == 0) spokes[gidx] = m & 0x07ffffffu;
  }
}

// Delete_Dirichlet_Equations (solver/MG/Delete_Dirichlet_Equations.h:24-50)
__global__ void delete_dirichlet_kernel(int nb, const int* __restrict__ coords, const uint32_t* __restrict__ flags,
                                        const uint32_t* __restrict__ spokes, GridView g, double* __restrict__ A, long N) {
  const long gidx = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (gidx >= long(nb) * 128) return;
  const uint32_t fl = flags[gidx];
  if (!(fl & ACTIVE_NODE)) return;
  const uint32_t sp = spokes[gidx];
  const int bi = int(gidx >> 7), e = int(gidx & 127);
  const int x = coords[3 * bi] + (e >> 5), y = coords[3 * bi + 1] + ((e >> 3) & 3), z = coords[3 * bi + 2] + (e & 7);
  for (int q = 0; q < 27; ++q) {
    if (!(sp & (1u << q))) continue;
    const long n = g.node(x + q / 9 - 1, y + (q / 3) % 3 - 1, z + q % 3 - 1);
    const uint32_t nf = n >= 0 ? flags[n] : 0u;
    for (int v = 0; v < 3; ++v)
      for (int w = 0; w < 3; ++w) {
        double* a = A + gidx * 243 + q * 9 + v * 3 + w;
        if (fl & (DIR_X << v)) *a = (v == w && q == 13) ? 1.0 : 0.0;
        else if ((nf & ACTIVE_NODE) && (nf & (DIR_X << w))) *a = 0.0;
      }
  }
}

// Dense bottom operator over the DOF nodes (nodes with an active spoke), the way
// Build_CSR_Matrix forms PARDISO's upper triangle (solver/MG/Elasticity_Matrix.cpp:98-161):
// entry (r,c), r <= c, comes from row r's stencil; Dirichlet rows/columns become identity.
// node_pos: first unknown of a node of the level, -1 without unknowns.
__global__ void bottom_assemble_kernel(int ndof_nodes, const int* __restrict__ dof_node, const int* __restrict__ node_pos,
                                       const int* __restrict__ coords, const uint32_t* __restrict__ flags,
                                       const uint32_t* __restrict__ spokes, GridView g, const double* __restrict__ A,
                                       long N, double* __restrict__ M, long ld) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ndof_nodes) return;
  const long gidx = dof_node[i];
  const uint32_t fl = flags[gidx], sp = spokes[gidx];
  const bool fact = fl & ACTIVE_NODE;
  const int bi = int(gidx >> 7), e = int(gidx & 127);
  const int x = coords[3 * bi] + (e >> 5), y = coords[3 * bi + 1] + ((e >> 3) & 3), z = coords[3 * bi + 2] + (e & 7);
  for (int q = 0; q < 27; ++q) {
    if (!(sp & (1u << q))) continue;
    const long n = g.node(x + q / 9 - 1, y + (q / 3) % 3 - 1, z + q % 3 - 1);
    if (n < 0) continue;
    const int j = node_pos[n];
    if (j < 0) continue;
    const uint32_t nf = flags[n];
    for (int v = 0; v < 3; ++v)
      for (int w = 0; w < 3; ++w) {
        const long r = node_pos[gidx] + v, c = j + w;
        if (r > c) continue;
        double val = A[gidx * 243 + q * 9 + v * 3 + w];
        const bool dr = fact && (fl & (DIR_X << v));
        const bool dc = (nf & ACTIVE_NODE) && (nf & (DIR_X << w));
        if (dr || dc) val = (r == c) ? 1.0 : 0.0;
        M[r * ld + c] = val;
        M[c * ld + r] = val;
      }
  }
}

__global__ void identity_pad_kernel(double* M, long ld, const int* __restrict__ row, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) M[long(row[i]) * ld + row[i]] = 1.0;
}

// ---------------------------------------------------------------------------
// Inverse of the bottom matrix: symmetric blocked Gauss-Jordan with 128-wide
// pivots.  The matrix is SPD, and after pivots 0..K-1 tile (I, J) equals the
// transpose of tile (J, I), negated when exactly one of I, J has been pivoted.
// So only the lower tiles (I >= J) are updated; the panels a step needs are
// gathered from them:
//   row panel  R_J = A_KJ  (J < K), A_JK^T (J > K)
//   col panel  C_I = A_IK  (I > K), -A_KI^T (I < K)
// then T = P^-1 R, lower tiles A_IJ -= C_I T_J, A_IK = -C_I P^-1 (I > K),
// A_KJ = T_J (J < K), A_KK = P^-1.  After the last pivot the lower tiles hold
// the lower half of M^-1 and are mirrored.  I and J run over the tiles that row
// K has reached (BottomOrder): with the unknowns in nested-dissection order and
// separators eliminated among themselves, the steps of the 14739-unknown bottom
// of a 64^3 box take a thirtieth of the tile products of a full elimination.
// FP64 GEMM tiles of 128 x 128.  Measured (assembly, inverse and copies): 14739
// unknowns 170 -> 22 ms, 20064 409 -> 30 ms, 9006 45 -> 13 ms, 4287 10 -> 6 ms.
// Bound by the chain of a step (gather 6 us, row product 30, cross update 30,
// beside it the next pivot 62): its products run on few SMs (5 to 28 of the 148
// in the steps captured at 9006 unknowns).
// ---------------------------------------------------------------------------
constexpr int SGJ = 128, SGJ_K = 16;

// P = (128 x 128 SPD tile M)^-1 by one CTA of 256 threads, Gauss-Jordan with
// the tile in registers: thread (ti, tj) holds rows ti + 16 r, columns tj + 16 s.
// A step publishes the pivot's row and column in shared memory (two buffers, one
// barrier a step).  Bound by the step's chain (barrier, shared loads, the
// division, 64 FMAs a thread).
__global__ void __launch_bounds__(256, 1) sgj_pivot_kernel(const double* __restrict__ M, long ld, double* __restrict__ P,
                                                           int* bad) {
  __shared__ double col[2][SGJ], row[2][SGJ];
  const int ti = threadIdx.x >> 4, tj = threadIdx.x & 15;
  double a[8][8];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int s = 0; s < 8; ++s) a[r][s] = M[long(ti + 16 * r) * ld + tj + 16 * s];
#pragma unroll
  for (int kb = 0; kb < 8; ++kb) {
    for (int kt = 0; kt < 16; ++kt) {
      const int p = kt & 1;
      if (tj == kt)
#pragma unroll
        for (int r = 0; r < 8; ++r) col[p][ti + 16 * r] = a[r][kb];
      if (ti == kt)
#pragma unroll
        for (int s = 0; s < 8; ++s) row[p][tj + 16 * s] = a[kb][s];
      __syncthreads();
      const double piv = col[p][16 * kb + kt], ip = 1.0 / piv;
      if (threadIdx.x == 0 && !(piv > 0)) *bad = 1;
      double rr[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) rr[s] = row[p][tj + 16 * s] * ip;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const double c = col[p][ti + 16 * r];
#pragma unroll
        for (int s = 0; s < 8; ++s) a[r][s] -= c * rr[s];
        if (tj == kt) a[r][kb] = -c * ip;
      }
      if (ti == kt) {
#pragma unroll
        for (int s = 0; s < 8; ++s) a[kb][s] = rr[s];
        if (tj == kt) a[kb][kb] = ip;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int s = 0; s < 8; ++s) P[(ti + 16 * r) * SGJ + tj + 16 * s] = a[r][s];
}

// panels of step K for the listed tiles J: R [128][ld] and Cp [ld][128]; one CTA
// (32 x 8 threads) per tile and 32 x 32 part, transposed through shared memory
__global__ void __launch_bounds__(256) sgj_gather_kernel(const double* __restrict__ M, long ld, int K,
                                                         const int* __restrict__ list, double* __restrict__ R,
                                                         double* __restrict__ Cp) {
  __shared__ double t[32][33];
  const int J = list[blockIdx.x], pr = int(blockIdx.y >> 2) * 32, pc = int(blockIdx.y & 3) * 32;
  const bool pivoted = J < K;  // source tile: (K, J) below the diagonal order, else (J, K)
  const double* src = pivoted ? M + long(K) * SGJ * ld + long(J) * SGJ : M + long(J) * SGJ * ld + long(K) * SGJ;
  const int x = threadIdx.x, y = threadIdx.y;
  for (int i = y; i < 32; i += 8) {
    const double v = src[long(pr + i) * ld + pc + x];
    t[i][x] = v;
    if (pivoted) R[long(pr + i) * ld + long(J) * SGJ + pc + x] = v;
    else Cp[(long(J) * SGJ + pr + i) * SGJ + pc + x] = v;
  }
  __syncthreads();
  for (int i = y; i < 32; i += 8) {
    const double v = t[x][i];
    if (pivoted) Cp[(long(J) * SGJ + pc + i) * SGJ + pr + x] = -v;
    else R[long(pc + i) * ld + long(J) * SGJ + pr + x] = v;
  }
}

// A_KJ = T_J for the first n listed tiles (J < K), A_KK = P (last CTA row)
__global__ void sgj_store_kernel(double* __restrict__ M, long ld, int K, const int* __restrict__ list, int n,
                                 const double* __restrict__ T, const double* __restrict__ P) {
  const int r = blockIdx.y, c = threadIdx.x;  // grid (n + 1, 128), 128 threads
  double* out = M + (long(K) * SGJ + r) * ld;
  if (int(blockIdx.x) < n) {
    const long at = long(list[blockIdx.x]) * SGJ + c;
    out[at] = T[long(r) * ld + at];
  } else {
    out[long(K) * SGJ + c] = P[r * SGJ + c];
  }
}

// One FP64 tensor-core MMA (m16n8k8): D = A B + D on a 16 x 8 tile.  With
// g = lane / 4 and t = lane % 4, a lane holds A[g][t], A[g+8][t], A[g][t+4],
// A[g+8][t+4]; B[t][g], B[t+4][g]; D[g][2t], D[g][2t+1], D[g+8][2t], D[g+8][2t+1].
__device__ __forceinline__ void dmma_16x8x8(double (&d)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// C(tile) = alpha * A(tile rows, 0:k) * B(0:k, tile cols) + beta * C(tile) on
// 128 x 128 tiles: sixteen warps of 32 x 32 (four per SM sub-partition, to hide
// the MMA latency), k staged through shared memory in chunks of 16, FP64 MMAs.
// Tiles of the list (ascending): SGJ_ROW (0, list[blockIdx.x]); SGJ_COL
// (list[blockIdx.x], 0); SGJ_LOWER the pairs I >= J (blockIdx.x), leaving out
// row and column `skip` (none if < 0); SGJ_CROSS the lower tiles of row and
// column `skip`.
constexpr int SGJ_THREADS = 512;          // sixteen warps of 32 x 32 per 128 x 128 tile
constexpr int SGJ_AS = 20, SGJ_BS = 132;  // padded strides (4 mod 16 doubles): conflict-free fragment loads
constexpr int SGJ_STAGE = SGJ * SGJ_AS + SGJ_K * SGJ_BS;  // doubles per pipeline stage
constexpr size_t SGJ_SMEM = 2 * SGJ_STAGE * sizeof(double);
enum { SGJ_ROW = 0, SGJ_COL = 1, SGJ_LOWER = 2, SGJ_CROSS = 3 };

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = unsigned(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_prior() { asm volatile("cp.async.wait_group 1;\n" ::); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::); }

// k staged through two shared-memory stages filled by cp.async: the copy of
// chunk c + 1 runs while chunk c is multiplied.
__global__ void __launch_bounds__(SGJ_THREADS, 1) sgj_gemm_kernel(int k, const double* __restrict__ A, long lda,
                                                          const double* __restrict__ B, long ldb, double* C, long ldc,
                                                          double alpha, double beta, int mode, int skip,
                                                          const int* __restrict__ list) {
  extern __shared__ __align__(16) double sg[];
  long I, J;
  if (mode == SGJ_LOWER) {
    const long t = blockIdx.x;
    long i = long((sqrt(8.0 * double(t) + 1.0) - 1.0) * 0.5);
    while ((i + 1) * (i + 2) / 2 <= t) ++i;
    while (i * (i + 1) / 2 > t) --i;
    I = list[i];
    J = list[t - i * (i + 1) / 2];
    if (I == skip || J == skip) return;
  } else if (mode == SGJ_CROSS) {
    const long b = list[blockIdx.x];
    I = b <= skip ? skip : b;
    J = b <= skip ? b : skip;
  } else {
    I = mode == SGJ_COL ? list[blockIdx.x] : 0;
    J = mode == SGJ_ROW ? list[blockIdx.x] : 0;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wr = (warp >> 2) * 32, wc = (warp & 3) * 32;  // the warp's 32 x 32 sub-tile
  if (beta != 0) {  // the epilogue reads this C tile: bring it into L2 while the products run
    const double* quarter_row = C + (I * SGJ + (tid >> 2)) * ldc + J * SGJ + (tid & 3) * 32;
#pragma unroll
    for (int q = 0; q < 2; ++q) asm volatile("prefetch.global.L2 [%0];" ::"l"(quarter_row + 16 * q));
  }
  const int fr = lane >> 2, fc = lane & 3;
  const double* Ab = A + I * SGJ * lda;
  const double* Bb = B + J * SGJ;
  const int ar = tid >> 2, ak = (tid & 3) * 4;    // A chunk: row, first k
  const int bk = tid >> 5, bc = (tid & 31) * 4;   // B chunk: k, first column
  auto stage = [&](int k0, int st) {
    double* As = sg + st * SGJ_STAGE;
    double* Bs = As + SGJ * SGJ_AS;
    const double* a = Ab + long(ar) * lda + k0 + ak;
    const double* b = Bb + long(k0 + bk) * ldb + bc;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      cp_async16(&As[ar * SGJ_AS + ak + 2 * q], a + 2 * q);
      cp_async16(&Bs[bk * SGJ_BS + bc + 2 * q], b + 2 * q);
    }
    cp_async_commit();
  };
  double acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0;
  const int nchunks = k / SGJ_K;
  stage(0, 0);
  for (int c = 0; c < nchunks; ++c) {
    if (c + 1 < nchunks) {
      stage((c + 1) * SGJ_K, (c + 1) & 1);
      cp_async_wait_prior();
    } else {
      cp_async_wait_all();
    }
    __syncthreads();
    const double* As = sg + (c & 1) * SGJ_STAGE;
    const double* Bs = As + SGJ * SGJ_AS;
#pragma unroll
    for (int k8 = 0; k8 < SGJ_K; k8 += 8) {
      double a[2][4], b[4][2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const double* r = As + (wr + 16 * i + fr) * SGJ_AS + k8 + fc;
        a[i][0] = r[0];
        a[i][1] = r[8 * SGJ_AS];
        a[i][2] = r[4];
        a[i][3] = r[8 * SGJ_AS + 4];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        b[j][0] = Bs[(k8 + fc) * SGJ_BS + wc + 8 * j + fr];
        b[j][1] = Bs[(k8 + fc + 4) * SGJ_BS + wc + 8 * j + fr];
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma_16x8x8(acc[i][j], a[i], b[j]);
    }
    __syncthreads();  // the stage is refilled two chunks later
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int hr = 0; hr < 2; ++hr) {
      double* row = C + (I * SGJ + wr + 16 * i + 8 * hr + fr) * ldc + J * SGJ + wc + 2 * fc;
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          double* p = row + 8 * j + h;
          *p = (beta != 0 ? beta * *p : 0.0) + alpha * acc[i][j][2 * hr + h];
        }
    }
}

// mirror the lower triangle into the upper one
__global__ void sgj_mirror_kernel(double* M, long ld) {
  __shared__ double tile[32][33];
  const int bx = blockIdx.x, by = blockIdx.y;  // source tile (row by, col bx), by > bx
  if (by <= bx) {
    if (by < bx) return;
    // diagonal 32x32 tile: copy lower to upper in place
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
      const int j = threadIdx.x;
      if (j > i) M[(long(by) * 32 + i) * ld + long(bx) * 32 + j] = M[(long(bx) * 32 + j) * ld + long(by) * 32 + i];
    }
    return;
  }
  for (int i = threadIdx.y; i < 32; i += blockDim.y)
    tile[i][threadIdx.x] = M[(long(by) * 32 + i) * ld + long(bx) * 32 + threadIdx.x];
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y)
    M[(long(bx) * 32 + i) * ld + long(by) * 32 + threadIdx.x] = tile[threadIdx.x][i];
}

// ---------------------------------------------------------------------------
// Bottom solve (Exact_Solve, solver/MG/Multigrid_Hierarchy.h:346-372): nodes of
// the level take b, DOF nodes then get the exact solution x = M^-1 b.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void bottom_gather_kernel(const int* __restrict__ node_pos, const T* __restrict__ b, long N,
                                     double* __restrict__ xb, T* __restrict__ u) {
  pdl_wait();
  const long n = long(blockIdx.x) * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const int p = node_pos[n];
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    if (p >= 0) xb[p + v] = double(b[n + v * N]);
    else u[n + v * N] = b[n + v * N];  // nodes without unknowns keep b
  }
}

// One phase of the bottom's application (BottomOrder), one warp per row over the
// row tile's column ranges, FP64 sums (TM float: the FP32 copy of the matrix that
// the mixed V-cycle applies).  Row r is entry out[r] of the level's field u (-1:
// padding).  PHASE 0: y = M x over the leaves' columns (plus x on the separators);
// SINGLE: straight to u.  PHASE 1: xs = M y on the separators.  PHASE 2: u = y +
// M xs on the leaves.  Every entry is read once per application, and the loads are in
// flight for most of it: bound by their latency (9006 unknowns, FP32 copy, from DRAM:
// 41 + 10 + 11 us for the phases, DRAM 36% busy in the first).
template <typename TM>
struct MatrixVec;
template <>
struct MatrixVec<double> {
  static constexpr int W = 2;
  static __device__ __forceinline__ double dot(const double* m, const double* v, double s) {
    const double2 a = __ldcs(reinterpret_cast<const double2*>(m)), w = *reinterpret_cast<const double2*>(v);
    return fma(a.y, w.y, fma(a.x, w.x, s));
  }
};
template <>
struct MatrixVec<float> {
  static constexpr int W = 4;
  static __device__ __forceinline__ double dot(const float* m, const double* v, double s) {
    const float4 a = __ldcs(reinterpret_cast<const float4*>(m));
    const double2 w0 = reinterpret_cast<const double2*>(v)[0], w1 = reinterpret_cast<const double2*>(v)[1];
    return fma(double(a.w), w1.y, fma(double(a.z), w1.x, fma(double(a.y), w0.y, fma(double(a.x), w0.x, s))));
  }
};
constexpr int APPLY_ROWS = 8;  // rows per CTA of 256 threads
template <typename TM, typename T, int PHASE, bool SINGLE>
__global__ void __launch_bounds__(256) bottom_apply_kernel(const TM* __restrict__ M, long ld,
                                                           const int* __restrict__ tiles, const int* __restrict__ first,
                                                           const int* __restrict__ ranges, const double* __restrict__ x,
                                                           double* y, double* xs, const int* __restrict__ out,
                                                           const int* __restrict__ separator, T* __restrict__ u) {
  constexpr int PER = SGJ / APPLY_ROWS;
  const int k = blockIdx.x / PER, lane = threadIdx.x & 31;
  const long row = long(tiles[k]) * SGJ + (blockIdx.x % PER) * APPLY_ROWS + (threadIdx.x >> 5);
  const int r0 = first[k], r1 = first[k + 1], to = out[row];
  pdl_wait();
  if (to < 0) return;
  const TM* m = M + row * ld;
  const double* v = PHASE == 0 ? x : (PHASE == 1 ? y : xs);
  constexpr int W = MatrixVec<TM>::W, STEP = 32 * W;
  double s0 = 0, s1 = 0;
  for (int r = r0; r < r1; ++r) {
    int c = ranges[2 * r] + lane * W;
    const int end = ranges[2 * r + 1];  // ranges are multiples of the tile, 128 columns
    for (; c + STEP < end; c += 2 * STEP) {
      s0 = MatrixVec<TM>::dot(m + c, v + c, s0);
      s1 = MatrixVec<TM>::dot(m + c + STEP, v + c + STEP, s1);
    }
    if (c < end) s0 = MatrixVec<TM>::dot(m + c, v + c, s0);
  }
  double s = s0 + s1;
  for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane != 0) return;
  if (PHASE == 0) {
    if (SINGLE) u[to] = T(s);
    else y[row] = separator[tiles[k]] ? x[row] + s : s;
  } else if (PHASE == 1) {
    xs[row] = s;
    u[to] = T(s);
  } else {
    u[to] = T(y[row] + s);
  }
}

}  // namespace sgs
