// New values of H_loc for a new effective potential, on the device.
//
// The reference rebuilds H_loc on the host every SCF iteration
// (ProjectHamiltonianSparse::Create_Hloc, dft/ProjectHamiltonianSparse.cc:
// 330-575, called from main.cc:965-972): for row I = (xI, yI, zI) and column
// J = (xJ, yJ, zJ)
//   H[I,J] = 0.5 (DX MY MZ + MX DY MZ + MX MY DZ)[I,J]
//          + sum_abc G_abc PX_a[xI,xJ] PY_b[yI,yJ] PZ_c[zI,zJ]
// with V_eff = sum_abc G_abc u_a(x) v_b(y) w_c(z) its Tucker decomposition
// (main.cc:951-955) and PX_a[i,j] = int psi_i u_a psi_j.
//
// Here the sparsity pattern is the one fixed when the operator was created,
// and the values are recomputed in place: the Tucker sum is factorised
// through (x-pair, y-pair) intermediates
//   T1[b][xp][c]     = sum_a PX_a[xp] G_abc                  (one FP64 GEMM)
//   T2[yp][xp][c]    = sum_b PY_b[yp] T1[b][xp][c]           (one FP64 GEMM)
//   H_pot[I,J]       = sum_c PZ_c[zp] T2[yp][xp][c]
// and each new value is written straight into every device format through
// the position maps recorded when the formats were packed.
//
// The last sum, r_c FMAs per entry, was FP64 work on the CUDA cores (64 atoms,
// r_c = 72: 15 ms of FP64 pipe, 24.6 ms measured).  It is a matrix product too,
// of the (y, x) index pairs by the z pairs, of which the pattern needs a band:
// the (y, x) pair's entries reach |z_J - z_I| <= w.  With the z pairs ordered by
// |dz| a pair needs a prefix of them, and with the (y, x) pairs sorted by w, tiles
// of 128 of them share a prefix: one ragged FP64 GEMM on the tensor cores (a few
// GB of values at most at a time, in slabs of y), from which the entries are
// gathered.  64 atoms: 24.6 -> 12.1 ms in all, 5.9 of
// them the gather and the scattered writes into the formats.  The per-entry sum stays where it
// is faster (entry_seconds), for operators that the plan does not fit and where
// the tensor cores are off.

#include <algorithm>
#include <cmath>
#include <vector>

#include "ttg_internal.cuh"

namespace ttg {
namespace {

struct UpdateArgs {
  const int64_t* row_ptr;
  const int* col;
  const int* rg_pos;
  const int* tile_base;
  const uint8_t* tile_slot;
  int rx, ry, rz;
  int bw[3];                  // half-bandwidths of the pair tables
  const double* kin;          // DX DY DZ MX MY MZ, each r_d x r_d row-major
  const double* T2;           // [yp][xp][c]
  const double* PZp;          // [zp][c]
  int rc;                     // Tucker rank of the potential along z
  const double* G;            // values of the slab's (y, x) pairs by z pairs, or null
  const int* where;           // offset of a (y, x) pair's values
  const int* zq;              // position of a z pair
  int y0;                     // first y of the slab
  int64_t nxp;
  double* v64;
  float2* vdf;
  float* v32;
  __nv_bfloat16* v16;
  float* t32;
  __nv_bfloat16* t16;
  const int64_t* rg_gptr;     // slot offset of each row group
  const int* umma_pos;        // slot of the entry within its 128-row tile
  const int* umma_row;        // tile * 128 + lane of each row
  const int64_t* umma_tptr;   // slot offset of each tile (multiples of 16)
  __nv_bfloat16* u16;         // the tiles' BF16 plane
  __half* h16;                // and their two FP16 planes (2048 elements apart)
  const float* rscale;        // inverse scale of each tile row's FP16 planes
  float* rmax;                // largest new |value| of each tile row
  int64_t n;
};

__device__ __forceinline__ int pair_index(int i, int j, int bw) {
  const int d = j - i;
  return (d < -bw || d > bw) ? -1 : i * (2 * bw + 1) + d + bw;
}

// A block updates eight rows, neighbours in x (one row group where rx is a
// multiple of 8), a warp each; blocks run through z first, whose rows gather
// neighbouring values of the same (y, x) pairs.
// An entry's value is at the end of a chain of loads (column, the pair's
// offset, value), and the kernel is bound by their latency (FP64 pipe 30 %, L2
// 25 %, HBM 2.7 TB/s at 28^3 functions).  So the chain runs ahead: while an entry
// is computed and stored, the value of the lane's next one, the offset of the
// one after and the column of the third are on their way.  64 atoms: 9.1 ms
// without it, now 5.9.
__global__ void __launch_bounds__(256) k_update_values(const UpdateArgs a) {
  const int lane = threadIdx.x & 31;
  const int nxg = (a.rx + 7) >> 3;
  const int zI = blockIdx.x % a.rz, yx = blockIdx.x / a.rz;
  const int yI = a.y0 + yx / nxg, xI = (yx % nxg) * 8 + (threadIdx.x >> 5);
  if (xI >= a.rx) return;
  const int64_t row = xI + (int64_t)a.rx * (yI + (int64_t)a.ry * zI);
  const int rx = a.rx, ry = a.ry, rz = a.rz;
  const double* DX = a.kin + xI * rx;
  const double* DY = a.kin + rx * rx + yI * ry;
  const double* DZ = a.kin + rx * rx + ry * ry + zI * rz;
  const int64_t mass = (int64_t)rx * rx + (int64_t)ry * ry + (int64_t)rz * rz;
  const double* MX = DX + mass;
  const double* MY = DY + mass;
  const double* MZ = DZ + mass;
  const int ur = a.u16 ? __ldg(a.umma_row + row) : 0;
  const int64_t chunk0 = a.u16 ? __ldg(a.umma_tptr + (ur >> 7)) / 16 : 0;
  const float up = a.u16 ? 1.f / a.rscale[ur] : 1.f;       // a power of two
  const int64_t rg0 = __ldg(a.rg_gptr + (row >> 3)) * 8 + (row & 7);
  const int64_t e1 = __ldg(a.row_ptr + row + 1);
  float hmax = 0.f;
  auto column = [&](int64_t e) { return e < e1 ? __ldg(a.col + e) : -1; };
  // offset of column J's value in G (0 where there is none)
  auto offset = [&](int J, int& zq) {
    if (J < 0 || !a.G) return zq = 0;
    const int yx = J / rx, xJ = J - yx * rx, zJ = yx / ry, yJ = yx - zJ * ry;
    zq = __ldg(a.zq + pair_index(zI, zJ, a.bw[2]));
    return __ldg(a.where + (int64_t)pair_index(yI, yJ, a.bw[1]) * a.nxp + pair_index(xI, xJ, a.bw[0]));
  };
  int64_t e = __ldg(a.row_ptr + row) + lane;
  int J0 = column(e), J1 = column(e + 32), J2 = column(e + 64);
  int z0, z1;
  int o0 = offset(J0, z0), o1 = offset(J1, z1);
  double g0 = J0 >= 0 && a.G ? __ldg(a.G + o0 + z0) : 0.0;
  for (; e < e1; e += 32) {
    const double g1 = J1 >= 0 && a.G ? __ldg(a.G + o1 + z1) : 0.0;
    int z2;
    const int o2 = offset(J2, z2), J3 = column(e + 96), J = J0;
    const int rg = __ldg(a.rg_pos + e), sl = a.u16 ? __ldg(a.umma_pos + e) : 0;
    const int base = a.t16 ? __ldg(a.tile_base + e) : 0, j = a.t16 ? __ldg(a.tile_slot + e) : 0;
    const int yxJ = J / rx, xJ = J - yxJ * rx, zJ = yxJ / ry, yJ = yxJ - zJ * ry;
    const double dx = __ldg(DX + xJ), mx = __ldg(MX + xJ);
    const double dy = __ldg(DY + yJ), my = __ldg(MY + yJ);
    const double dz = __ldg(DZ + zJ), mz = __ldg(MZ + zJ);
    double val = 0.5 * (dx * my * mz + mx * dy * mz + mx * my * dz);
    if (a.G) {
      val += g0;
    } else {
      const int xp = pair_index(xI, xJ, a.bw[0]);
      const int yp = pair_index(yI, yJ, a.bw[1]);
      const int zp = pair_index(zI, zJ, a.bw[2]);
      if (xp >= 0 && yp >= 0 && zp >= 0) {
        const double* t2 = a.T2 + ((int64_t)yp * a.nxp + xp) * a.rc;
        const double* pz = a.PZp + (int64_t)zp * a.rc;
        // four independent partial sums: the FP64 FMA chain of one sum would
        // otherwise serialise the rc terms of every entry
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        int c = 0;
        for (; c + 3 < a.rc; c += 4) {
          s0 = fma(pz[c], t2[c], s0);
          s1 = fma(pz[c + 1], t2[c + 1], s1);
          s2 = fma(pz[c + 2], t2[c + 2], s2);
          s3 = fma(pz[c + 3], t2[c + 3], s3);
        }
        for (; c < a.rc; ++c) s0 = fma(pz[c], t2[c], s0);
        val += (s0 + s1) + (s2 + s3);
      }
    }
    J0 = J1;
    J1 = J2;
    J2 = J3;
    o1 = o2;
    z1 = z2;
    g0 = g1;
    // value index in the row groups: (group slot offset + slot) * 8 + row in group
    const int64_t p = rg0 + (int64_t)rg * 8;
    a.v64[p] = val;
    const float h = __double2float_rn(val);
    if (a.vdf) a.vdf[p] = make_float2(h, __double2float_rn(val - (double)h));
    if (a.v32) a.v32[p] = h;
    if (a.v16) a.v16[p] = __double2bfloat16(val);
    if (a.t16) {
      // fragment order of spmm_tc.cu: TF32 lane 4g+(j%4), element j/4;
      // BF16 lane 4g+((j%8)/2), element (j%2) + 2*(j/8)
      if (a.t32) a.t32[(int64_t)(base + (j & 3)) * 4 + (j >> 2)] = h;
      a.t16[(int64_t)(base + ((j & 7) >> 1)) * 4 + (j & 1) + 2 * (j >> 3)] = __double2bfloat16(val);
    }
    if (a.u16) {
      // the BF16 value and two FP16 terms of the scaled one, as the tile
      // builder has them: chunk (tile's first + slot / 16), canonical K-major
      // position of (lane, slot % 16) within the chunk's 128 x 16 plane
      const int m = ur & 127;
      const int64_t chunk = chunk0 + (sl >> 4);
      const int s16 = sl & 15;
      const int at = (m >> 3) * 128 + (s16 >> 3) * 64 + (m & 7) * 8 + (s16 & 7);
      a.u16[chunk * 2048 + at] = __float2bfloat16_rn(h);
      const float v = h * up;
      const __half v0 = __float2half_rn(v);
      __half* u = a.h16 + chunk * 4096 + at;
      u[0] = v0;
      u[2048] = __float2half_rn(v - __half2float(v0));
      if (fabsf(h) <= 3.402823466e38f) hmax = fmaxf(hmax, fabsf(h));
    }
  }
  if (a.u16) {
    for (int o = 16; o > 0; o >>= 1) hmax = fmaxf(hmax, __shfl_xor_sync(0xffffffffu, hmax, o));
    if (lane == 0) a.rmax[ur] = hmax;
  }
}

}  // namespace
}  // namespace ttg

using namespace ttg;

namespace ttg {
namespace {

// pair tables PXp[xp][a] = PX_a[i][j], xp = i (2b + 1) + (j - i) + b, from
// the (rk x r x r) row-major matrices on the device
__global__ void k_pair_table(const double* __restrict__ pm, int r, int rk, int b,
                             double* __restrict__ out) {
  const int64_t np = (int64_t)r * (2 * b + 1);
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < np * rk;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = e / rk;
    const int a = (int)(e - p * rk);
    const int i = (int)(p / (2 * b + 1));
    const int j = i + (int)(p - (int64_t)i * (2 * b + 1)) - b;
    out[e] = (j >= 0 && j < r) ? pm[((int64_t)a * r + i) * r + j] : 0.0;
  }
}

// largest |dz| of the entries of each (y, x) pair (-1: none)
__global__ void __launch_bounds__(256) k_pair_width(const UpdateArgs a, int* __restrict__ width) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= a.n) return;
  const int xI = (int)(row % a.rx), yI = (int)((row / a.rx) % a.ry);
  const int zI = (int)(row / ((int64_t)a.rx * a.ry));
  for (int64_t e = a.row_ptr[row] + lane; e < a.row_ptr[row + 1]; e += 32) {
    const int J = a.col[e];
    const int xp = pair_index(xI, J % a.rx, a.bw[0]);
    const int yp = pair_index(yI, (J / a.rx) % a.ry, a.bw[1]);
    int* w = width + (int64_t)yp * a.nxp + xp;
    const int dz = abs(J / (a.rx * a.ry) - zI);
    if (*w < dz) atomicMax(w, dz);
  }
}

// From this many flops on T1 and T2 go to the tensor cores: their eight launches
// cost 40 us more than the CUDA-core GEMM's two.  Update of 40 x 40 x 1
// functions, both ways: rank 6 (3.4e7 flops) 132 against 158 us on the tensor
// cores, rank 16 (2.4e8) 224 against 200; of 14^3, rank 32 (1.3e8) 612 against 623.
constexpr double kTensorFlops = 1.5e8;

// Seconds of the last sum on the CUDA cores and on the tensor cores (ragged
// product of `pairs` rows, launches, scales and digits of the rows), fitted to
// 80 updates of 125 to 13,824 functions, ranks 1 to 72, flat and long bases
// among them.  14^3 functions, by entry against ragged: rank 1 203 and 234 us,
// rank 6 249 and 239, rank 32 612 and 301; 60 x 60 x 3 (a million pairs), rank 6
// 416 and 737.
double entry_seconds(int64_t nnz, int rc) { return 2.0 * nnz * rc / 0.7e12 + 0.2e-6 * rc; }
double ragged_seconds(int64_t pairs, int64_t nq, int rc) {
  const double tiles = (double)pairs / 128.0 * (double)((nq + 63) / 64) * 0.6;
  return 35e-6 + pairs * (1.5e-10 + (rc + 15) / 16 * 16 * 32 / 6e12) +
         tiles / 152.0 * ((rc + 127) / 128 + 2) * 0.4e-6;
}

// The tests' small operators take the tensor cores where this is set.
bool tensor_forced() { return getenv("TTG_UPDATE_SLAB_VALUES") != nullptr; }

// Most values of a slab (8 bytes each); TTG_UPDATE_SLAB_VALUES sets another limit.
int64_t slab_values() {
  const char* e = getenv("TTG_UPDATE_SLAB_VALUES");
  return e ? std::max<int64_t>(atoll(e), 1) : (int64_t)1 << 28;
}

ttg_status upload_vec(cudaStream_t st, DevBuf& b, const void* p, size_t bytes) {
  TTG_TRY(b.alloc(std::max<size_t>(bytes, 16)));
  TTG_CUDA_TRY(cudaMemcpyAsync(b.p, p, bytes, cudaMemcpyHostToDevice, st));
  return TTG_OK;
}

// The slabs, pair lists and tiles of the pattern (see UpdatePlan); no slabs if
// the pairs of one y exceed a slab.
ttg_status make_plan(ttg_op* op, const UpdateArgs& a, int64_t nxp, int64_t nyp, int rc) {
  Pattern& P = op->pattern;
  UpdatePlan& L = P.plan;
  cudaStream_t st = op->stream;
  const int ry = P.r[1], rz = P.r[2], by = 2 * P.bw[1] + 1, bz = P.bw[2];
  L = UpdatePlan();
  std::vector<int> width(nxp * nyp);
  {
    DevBuf wd;
    TTG_TRY(wd.alloc(width.size() * 4));
    TTG_CUDA_TRY(cudaMemsetAsync(wd.p, 0xff, width.size() * 4, st));
    k_pair_width<<<(unsigned)((op->n + 7) / 8), 256, 0, st>>>(a, wd.as<int>()); TTG_COUNT();
    TTG_LAUNCHED(op);
    TTG_CUDA_TRY(cudaMemcpyAsync(width.data(), wd.p, width.size() * 4, cudaMemcpyDeviceToHost, st));
    TTG_CUDA_TRY(cudaStreamSynchronize(st));
  }
  // z pairs in the order of |dz|
  std::vector<int> zlist, zq((size_t)rz * (2 * bz + 1), -1), cols(bz + 1);
  for (int d = 0; d <= bz; ++d) {
    for (int sgn = 0; sgn < (d ? 2 : 1); ++sgn) {
      const int dz = sgn ? d : -d;
      for (int i = std::max(0, -dz); i < rz - std::max(0, dz); ++i) {
        const int zp = i * (2 * bz + 1) + dz + bz;
        zq[zp] = (int)zlist.size();
        zlist.push_back(zp);
      }
    }
    cols[d] = ((int)zlist.size() + 1) / 2 * 2;
  }
  L.nq = (int)zlist.size();
  const int64_t max_rows = L.max_rows = ozgemm_ragged_rows(rc, L.nq), max_values = slab_values();
  std::vector<int> pairs, where(nxp * nyp, -1), first, ld;
  std::vector<int64_t> base;
  for (int y0 = 0; y0 < ry;) {
    // rows of y until a slab is full
    int64_t cnt = 0, vals = 0;
    int y1 = y0;
    for (; y1 < ry; ++y1) {
      int64_t c = 0, v = 0;
      for (int64_t i = (int64_t)y1 * by * nxp; i < (int64_t)(y1 + 1) * by * nxp; ++i)
        if (width[i] >= 0) {
          ++c;
          v += cols[width[i]];
        }
      v += 128 * (int64_t)cols[bz];          // a tile's columns are its widest pair's
      if (cnt + c > max_rows || vals + v > max_values) break;
      cnt += c;
      vals += v;
    }
    if (y1 == y0) {                          // no plan for these
      L.slabs.clear();
      L.made = true;
      return TTG_OK;
    }
    std::vector<std::vector<int>> by_width(bz + 1);
    for (int64_t i = (int64_t)y0 * by * nxp; i < (int64_t)y1 * by * nxp; ++i)
      if (width[i] >= 0) by_width[width[i]].push_back((int)i);
    UpdatePlan::Slab s{y0, y1, (int)pairs.size(), 0, (int)ld.size(), 0};
    int64_t off = 0;
    for (int w = bz; w >= 0; --w)
      for (int i : by_width[w]) {
        if (s.pairs % 128 == 0) {            // a new tile, as wide as its first pair
          first.push_back(s.items);
          base.push_back(off);
          ld.push_back(cols[w]);
          s.items += (cols[w] + 63) / 64;
          off += 128 * (int64_t)cols[w];
        }
        where[i] = (int)(base.back() + (int64_t)(s.pairs++ % 128) * ld.back());
        pairs.push_back(i);
      }
    first.push_back(s.items);
    L.out_max = std::max(L.out_max, off);
    L.slabs.push_back(s);
    y0 = y1;
  }
  TTG_TRY(upload_vec(st, L.pairs, pairs.data(), pairs.size() * 4));
  TTG_TRY(upload_vec(st, L.where, where.data(), where.size() * 4));
  TTG_TRY(upload_vec(st, L.first, first.data(), first.size() * 4));
  TTG_TRY(upload_vec(st, L.base, base.data(), base.size() * 8));
  TTG_TRY(upload_vec(st, L.ld, ld.data(), ld.size() * 4));
  TTG_TRY(upload_vec(st, L.zq, zq.data(), zq.size() * 4));
  TTG_TRY(upload_vec(st, L.zlist, zlist.data(), zlist.size() * 4));
  TTG_CUDA_TRY(cudaStreamSynchronize(st));      // the vectors go out of scope
  L.made = true;
  return TTG_OK;
}

struct UpdateLayout {
  int ra, rb, rc;
  int64_t nxp, nyp, nzp, off_x, off_y, off_z, off_g, off_t1, off_t2, total;
};

ttg_status update_layout(ttg_op* op, const int32_t* pot_ranks, UpdateLayout& L) {
  Pattern& P = op->pattern;
  L.ra = pot_ranks[0];
  L.rb = pot_ranks[1];
  L.rc = pot_ranks[2];
  if (L.ra <= 0 || L.rb <= 0 || L.rc <= 0) return TTG_BAD_ARG;
  L.nxp = (int64_t)P.r[0] * (2 * P.bw[0] + 1);
  L.nyp = (int64_t)P.r[1] * (2 * P.bw[1] + 1);
  L.nzp = (int64_t)P.r[2] * (2 * P.bw[2] + 1);
  const int64_t ncore = (int64_t)L.ra * L.rb * L.rc;
  L.off_x = 0;
  L.off_y = L.off_x + L.nxp * L.ra;
  L.off_z = L.off_y + L.nyp * L.rb;
  L.off_g = L.off_z + L.nzp * L.rc;
  L.off_t1 = L.off_g + ncore;
  L.off_t2 = L.off_t1 + L.nxp * L.rb * L.rc;
  L.total = L.off_t2 + L.nyp * L.nxp * L.rc;
  if ((int64_t)P.work.bytes < L.total * 8) TTG_TRY(P.work.alloc(L.total * 8));
  return TTG_OK;
}

// T1, T2 and the per-entry update, from the pair tables and the core in work
ttg_status update_from_tables(ttg_op* op, const UpdateLayout& L) {
  Pattern& P = op->pattern;
  const int rx = P.r[0], ry = P.r[1], rz = P.r[2];
  const int ra = L.ra, rb = L.rb, rc = L.rc;
  const int bw[3] = {P.bw[0], P.bw[1], P.bw[2]};
  const int64_t nxp = L.nxp, nyp = L.nyp;
  const int64_t off_x = L.off_x, off_y = L.off_y, off_z = L.off_z, off_g = L.off_g,
                off_t1 = L.off_t1, off_t2 = L.off_t2;
  double* w = P.work.as<double>();
  cudaStream_t st = op->stream;
  // T1[b][xp][c] = sum_a PXp[xp][a] G[a + ra (b + rb c)], then
  // T2[yp][(xp, c)] = sum_b PYp[yp][b] T1[b][(xp, c)]: FP64 GEMMs on the tensor
  // cores with the long dimension, (b, c) and (xp, c), as their rows; the
  // double-FP32 GEMM on the CUDA cores where they are small or those are off.
  // 64-atom system, potential ranks 72: 18.2 -> 2.2 ms for both.
  const int64_t xc = nxp * rc;
  const OzOperand g1{w + off_g, (int64_t)rb * rc, ra, ra, 1}, p1{w + off_x, nxp, ra, ra, 1};
  const OzOperand g2{w + off_t1, xc, rb, 1, xc}, p2{w + off_y, nyp, rb, rb, 1};
  ttg_status s = TTG_OOM;
  const double flops = 2.0 * xc * rb * ra + 2.0 * nyp * xc * rb;
  if ((flops >= kTensorFlops || tensor_forced()) && ozgemm_supported(g1, p1) &&
      ozgemm_supported(g2, p2)) {
    s = ozgemm(op, g1, p1, w + off_t1, OzLayout{xc, rc, rb, 1}, false);
    if (s == TTG_OK) s = ozgemm(op, g2, p2, w + off_t2, OzLayout{1, xc}, false);
  }
  if (s == TTG_OOM) {
    TTG_TRY(dgemm(st, (int)nxp, rc, ra, rb, DOp{w + off_x, ra, 1, 0},
                  DOp{w + off_g, 1, (int64_t)ra * rb, ra}, w + off_t1, rc, 1, xc, P.work2));
    s = dgemm(st, (int)nyp, (int)xc, rb, 1, DOp{w + off_y, rb, 1, 0},
              DOp{w + off_t1, xc, 1, 0}, w + off_t2, xc, 1, 0, P.work2);
  }
  if (s != TTG_OK) return s;
  UpdateArgs a{};
  a.row_ptr = P.row_ptr.as<int64_t>();
  a.col = P.col.as<int>();
  a.rg_pos = P.rg_pos.as<int>();
  a.tile_base = P.tile_base.as<int>();
  a.tile_slot = P.tile_slot.as<uint8_t>();
  a.rx = rx;
  a.ry = ry;
  a.rz = rz;
  for (int d = 0; d < 3; ++d) a.bw[d] = bw[d];
  a.kin = P.kin.as<double>();
  a.T2 = w + off_t2;
  a.PZp = w + off_z;
  a.rc = rc;
  a.nxp = nxp;
  a.v64 = op->rg.v64.as<double>();
  a.vdf = op->rg.vdf.as<float2>();
  a.v32 = op->rg.v32.as<float>();
  a.v16 = op->rg.v16.as<__nv_bfloat16>();
  a.t32 = op->tiles.v32.as<float>();
  a.t16 = op->tiles.n_tiles > 0 && P.tile_base.p ? op->tiles.v16.as<__nv_bfloat16>() : nullptr;
  a.rg_gptr = op->rg.gptr.as<int64_t>();
  a.umma_pos = P.umma_pos.as<int>();
  a.umma_row = P.umma_row.as<int>();
  a.umma_tptr = op->umma.tptr.as<int64_t>();
  a.u16 = op->umma.n_tiles > 0 && P.umma_pos.p ? op->umma.hpl.as<__nv_bfloat16>() : nullptr;
  a.h16 = reinterpret_cast<__half*>(op->umma.fp16);
  a.rscale = op->umma.rscale.as<float>();
  a.rmax = op->umma.rmax.as<float>();
  a.n = op->n;
  op->ozrows.cut = false;
  if (op->nnz_h == 0) return TTG_OK;           // no entry to update
  const int nxg = (rx + 7) / 8;
  UpdatePlan& plan = P.plan;
  int64_t nq = rz;                             // z pairs
  for (int d = 1; d <= bw[2]; ++d) nq += 2 * std::max(0, rz - d);
  const bool oz = (ragged_seconds(nxp * nyp, nq, rc) < entry_seconds(op->nnz_h, rc) || tensor_forced()) &&
                  ozgemm_supported(g1, p1);
  // the plan's slabs hold for the rank it was made for and smaller ones; a rank
  // without a plan says nothing about smaller ones
  const int64_t max_rows = ozgemm_ragged_rows(rc, plan.nq);
  int64_t most = 0;                            // pairs of a slab
  for (const UpdatePlan::Slab& sl : plan.slabs) most = std::max<int64_t>(most, sl.pairs);
  if (most > max_rows || (plan.slabs.empty() && max_rows > plan.max_rows)) plan.made = false;
  if (oz && !plan.made) {
    const ttg_status ps = make_plan(op, a, nxp, nyp, rc);
    if (ps == TTG_OOM) plan = UpdatePlan();    // this time without one
    else if (ps != TTG_OK) return ps;
    most = 0;
    for (const UpdatePlan::Slab& sl : plan.slabs) most = std::max<int64_t>(most, sl.pairs);
  }
  // all workspaces before the first new value: H is then updated as a whole
  bool ragged = oz && !plan.slabs.empty();
  if (ragged && P.values.bytes < (size_t)plan.out_max * 8 && P.values.alloc(plan.out_max * 8) != TTG_OK)
    ragged = false;
  if (ragged && ozgemm_reserve(op, most, plan.nq, rc) != TTG_OK) ragged = false;
  if (ragged) {
    a.G = P.values.as<double>();
    a.where = plan.where.as<int>();
    a.zq = plan.zq.as<int>();
    OzOperand pz{w + off_z, plan.nq, rc, rc, 1};
    pz.idx = plan.zlist.as<int>();
    for (size_t i = 0; i < plan.slabs.size(); ++i) {
      const UpdatePlan::Slab& sl = plan.slabs[i];
      if (sl.pairs == 0) continue;
      a.y0 = sl.y0;
      OzOperand t2{w + off_t2, sl.pairs, rc, rc, 1};
      t2.idx = plan.pairs.as<int>() + sl.pair0;
      const OzRagged R{plan.first.as<int>() + sl.tile0 + i, plan.base.as<int64_t>() + sl.tile0,
                       plan.ld.as<int>() + sl.tile0, sl.items};
      TTG_TRY(ozgemm(op, t2, pz, P.values.as<double>(), OzLayout{0, 1}, false, false, nullptr, &R));
      k_update_values<<<(unsigned)((int64_t)(sl.y1 - sl.y0) * nxg * rz), 256, 0, st>>>(a); TTG_COUNT();
      TTG_LAUNCHED(op);
    }
  }
  if (!ragged) {
    a.G = nullptr;
    a.y0 = 0;
    k_update_values<<<(unsigned)((int64_t)ry * nxg * rz), 256, 0, st>>>(a); TTG_COUNT();
    TTG_LAUNCHED(op);
  }
  return a.u16 ? launch_umma_rescale(op) : TTG_OK;
}

}  // namespace
}  // namespace ttg


extern "C" {

ttg_status ttg_op_set_kinetic(ttg_op* op, const double* dx, const double* dy, const double* dz,
                              const double* mx, const double* my, const double* mz) {
  if (!op || !op->keep_pattern || !dx || !dy || !dz || !mx || !my || !mz) return TTG_BAD_ARG;
  Pattern& P = op->pattern;
  const int rx = P.r[0], ry = P.r[1], rz = P.r[2];
  const size_t cnt = 2 * ((size_t)rx * rx + (size_t)ry * ry + (size_t)rz * rz);
  if (!P.kin.p) TTG_TRY(P.kin.alloc(cnt * 8));
  std::vector<double> h;
  h.reserve(cnt);
  h.insert(h.end(), dx, dx + rx * rx);
  h.insert(h.end(), dy, dy + ry * ry);
  h.insert(h.end(), dz, dz + rz * rz);
  h.insert(h.end(), mx, mx + rx * rx);
  h.insert(h.end(), my, my + ry * ry);
  h.insert(h.end(), mz, mz + rz * rz);
  TTG_CUDA_TRY(cudaMemcpyAsync(P.kin.p, h.data(), cnt * 8, cudaMemcpyHostToDevice, op->stream));
  TTG_CUDA_TRY(cudaStreamSynchronize(op->stream));
  P.kinetic_set = true;
  return TTG_OK;
}

ttg_status ttg_op_update_potential(ttg_op* op, const int32_t* pot_ranks, const double* G,
                                   const double* px, const double* py, const double* pz) {
  if (!op || !op->keep_pattern || !op->pattern.kinetic_set || !pot_ranks || !G || !px || !py ||
      !pz)
    return TTG_BAD_ARG;
  Pattern& P = op->pattern;
  UpdateLayout L;
  TTG_TRY(update_layout(op, pot_ranks, L));
  // pair tables PXp[xp][a] = PX_a[i][j] (host: O(pairs * rank))
  auto pairs = [](const double* pm, int r, int rk, int b, std::vector<double>& out) {
    const int64_t np = (int64_t)r * (2 * b + 1);
    out.assign(np * rk, 0.0);
    for (int i = 0; i < r; ++i)
      for (int d = -b; d <= b; ++d) {
        const int j = i + d;
        if (j < 0 || j >= r) continue;
        const int64_t p = (int64_t)i * (2 * b + 1) + d + b;
        for (int a = 0; a < rk; ++a) out[p * rk + a] = pm[((int64_t)a * r + i) * r + j];
      }
  };
  std::vector<double> hx, hy, hz;
  pairs(px, P.r[0], L.ra, P.bw[0], hx);
  pairs(py, P.r[1], L.rb, P.bw[1], hy);
  pairs(pz, P.r[2], L.rc, P.bw[2], hz);
  double* w = P.work.as<double>();
  cudaStream_t st = op->stream;
  const int64_t ncore = (int64_t)L.ra * L.rb * L.rc;
  TTG_CUDA_TRY(cudaMemcpyAsync(w + L.off_x, hx.data(), hx.size() * 8, cudaMemcpyHostToDevice, st));
  TTG_CUDA_TRY(cudaMemcpyAsync(w + L.off_y, hy.data(), hy.size() * 8, cudaMemcpyHostToDevice, st));
  TTG_CUDA_TRY(cudaMemcpyAsync(w + L.off_z, hz.data(), hz.size() * 8, cudaMemcpyHostToDevice, st));
  TTG_CUDA_TRY(cudaMemcpyAsync(w + L.off_g, G, ncore * 8, cudaMemcpyHostToDevice, st));
  TTG_TRY(update_from_tables(op, L));
  return ozgemm_error(op);
}

ttg_status ttg_op_update_potential_device(ttg_op* op, const int32_t* pot_ranks,
                                          const double* g_dev, const double* px_dev,
                                          const double* py_dev, const double* pz_dev) {
  if (!op || !op->keep_pattern || !op->pattern.kinetic_set || !pot_ranks || !g_dev || !px_dev ||
      !py_dev || !pz_dev)
    return TTG_BAD_ARG;
  Pattern& P = op->pattern;
  UpdateLayout L;
  TTG_TRY(update_layout(op, pot_ranks, L));
  double* w = P.work.as<double>();
  cudaStream_t st = op->stream;
  const double* pm[3] = {px_dev, py_dev, pz_dev};
  const int rk[3] = {L.ra, L.rb, L.rc};
  const int64_t off[3] = {L.off_x, L.off_y, L.off_z};
  const int64_t np[3] = {L.nxp, L.nyp, L.nzp};
  for (int d = 0; d < 3; ++d) {
    const int64_t n = np[d] * rk[d];
    const int blocks = (int)std::min<int64_t>((n + 255) / 256, 152 * 8);
    k_pair_table<<<std::max(blocks, 1), 256, 0, st>>>(pm[d], P.r[d], rk[d], P.bw[d], w + off[d]); TTG_COUNT();
    TTG_LAUNCHED(op);
  }
  TTG_CUDA_TRY(cudaMemcpyAsync(w + L.off_g, g_dev, (size_t)L.ra * L.rb * L.rc * 8,
                               cudaMemcpyDeviceToDevice, st));
  return update_from_tables(op, L);
}

}  // extern "C"
