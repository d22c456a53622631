// surf.cuh — surface reconstruction of a particle set on the GPU: the reference's
// SRTool.dual_contouring (SPH/surf_recon/srtool.py:1264-1304).
//
// Pipeline (one launch sequence per call, all on the caller's stream):
//   1. particles binned by voxel (counting sort, id order inside a voxel)
//      — update_particles, srtool.py:1192-1195
//   2. isotropic poly6 splat onto the 27 vertices around each particle's voxel
//      — generate_fluid_field, srtool.py:1238-1251
//   3. anisotropic kernel per particle: weighted mean x_bar and covariance C over the
//      particles within 2 * smooth_radius, eigen-decomposition, G = (1/r_s) U S^-1 U^T
//      — pre_process_data, srtool.py:1006-1095 (particle 0 is skipped, as there)
//   4. anisotropic splat of the reference's kernel onto every vertex of every voxel in
//      the smoothing range, once per adjacent voxel (the multiplicity is computed, not
//      looped) — generate_smooth_fluid_field_impl, srtool.py:1135-1157
//   5. one value-weighted Gaussian smoothing pass with the standard deviation of the
//      negative vertex values — smooth_sdf, srtool.py:1425-1484
//   6. dual contouring: a QEF point per crossing cube (vertex ids by a scan in cube
//      order), then two triangles per crossing x/y/z edge of each cube's first corner
//      — dual_contouring_impl / dual_contouring_polygen, srtool.py:1531-1763
//   7. optional vertex normals — process_normal, srtool.py:1383-1410
//
// Layout: the vertex grid is dense, x fastest; blocks of NN_SR_BLOCK^3 vertices carry
// an "active" flag that emulates the reference's sparse fields (a block becomes active
// when any of its vertices is written; the smoothing and contouring visit every vertex
// of the active blocks and read 0 elsewhere). Splats accumulate in 64-bit fixed point
// (2^-32 units) with integer atomics, so the field is the same bits on every run
// whatever the order of the atomics.
//
// Restatement choices where the reference is undefined or nondeterministic: the QEF
// uses every crossing edge (the reference's 4x4 matrix overflows past 4 edges) through
// the normal equations with the reference's 0.1 clamp on the singular values;
// vertices and triangles are numbered in cube order.
#pragma once
#include "ns.cuh"

#define SR_FIX 4294967296.0  // fixed-point units per field unit
#define SR_PI 3.14159265358979323846

struct SrGrid {
  int nx, ny, nz, bx, by, bz;
  float ox, oy, oz, vs;        // f32, as the reference's get_voxel_index computes
  double dox, doy, doz, dvs;   // the same values in double
  __device__ __forceinline__ int64_t idx(int x, int y, int z) const {
    return x + (int64_t)nx * (y + (int64_t)ny * z);
  }
  __device__ __forceinline__ bool in(int x, int y, int z) const {
    return x >= 0 && y >= 0 && z >= 0 && x < nx && y < ny && z < nz;
  }
  __device__ __forceinline__ int64_t bidx(int x, int y, int z) const {
    return x / NN_SR_BLOCK + (int64_t)bx * (y / NN_SR_BLOCK + (int64_t)by * (z / NN_SR_BLOCK));
  }
  // get_voxel_index (srtool.py:799-803): f32, int() truncates toward zero
  __device__ __forceinline__ void voxel_of(float px, float py, float pz, int& x, int& y, int& z) const {
    x = (int)((px - ox) / vs);
    y = (int)((py - oy) / vs);
    z = (int)((pz - oz) / vs);
  }
};

struct SrResult { uint32_t nv, ni; int32_t status, pad; double sd; };  // what the host reads back

struct SrDev {
  SrGrid g;
  int n;
  const float* pos;         // [n,3]
  int32_t* status;
  uint32_t* vcount;         // [cells+1] voxel counts, then starts
  uint32_t* vkey;           // [n]
  uint32_t* vrank;          // [n]
  int32_t* vsrc;            // [n] particles in voxel order
  float4* spos;             // [n] their positions, in the same order
  unsigned long long* fix;  // [cells] fixed-point field
  float* splat;             // [cells] field after the splats
  float* field;             // [cells] field after smoothing
  float* tmp;               // [cells]
  uint8_t* active;          // [blocks]
  float* G;                 // [n,9]
  float* xbar;              // [n,3]
  double* stats;            // sum, count, var, sd
  int32_t* scan_n;          // [2]: last index of the next scan
  SrResult* result;
  uint32_t* vflag;          // [cells+1] crossing-cube flags, then vertex ids
  uint32_t* tcount;         // [cells+1] index counts, then offsets
  uint32_t* cube_of;        // [max_v] cube (linear index) of each vertex id
  float* vert;              // [max_v,3]
  int32_t* tri;             // [max_i]
  float* nrm;               // [max_v,3]
  const float* vel;         // [n,3] particle velocities, or null (no velocity recording)
  unsigned long long* vfix; // [3][cells] fixed-point vertex velocities
  float* mvel;              // [max_v,3] mesh-vertex velocities
  int32_t max_v, max_i;
  float iso, sr, volume, acoeff;
  float q1_thr, q05_thr;     // largest f32 whose rounded square root is <= 1, <= 0.5
  float rr_thr;              // smallest f32 whose rounded square root is >= 2 smooth_radius
  int range, off, smooth_cells, record_normals;
};

// corner w of cube (x, y, z) is vertex (x, y, z) + off (srtool.py:775-783)
__constant__ int8_t c_sr_off[8][3] = {{0, 1, 0}, {1, 1, 0}, {1, 0, 0}, {0, 0, 0},
                                      {0, 1, 1}, {1, 1, 1}, {1, 0, 1}, {0, 0, 1}};
// corners of edge w (srtool.py:931-942)
__constant__ int8_t c_sr_edge[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                                        {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};

// The dense passes walk the vertices by rows of one block: a warp takes the 32 x-neighbours
// (x, y, z) of a block's row, so coordinates cost three 32-bit divisions per warp instead of
// three 64-bit ones per vertex, and the block's activity (`act`) is uniform in the warp.
#define FOR_SR_ROWS(s, x, y, z, c, act)                                                                  \
  for (uint32_t _w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5,                                       \
                _bx = (uint32_t)(s).g.bx, _rows = _bx * (uint32_t)(s).g.ny * (uint32_t)(s).g.nz;         \
       _w < _rows; _w += (gridDim.x * blockDim.x) >> 5)                                                  \
    for (int x = (int)(_w % _bx) * NN_SR_BLOCK + (int)(threadIdx.x & 31), _r = (int)(_w / _bx),          \
             y = _r % (s).g.ny, z = _r / (s).g.ny, _once = 1;                                            \
         _once; _once = 0)                                                                               \
      if (const int64_t c = (s).g.idx(x, y, z); x < (s).g.nx)                                            \
        for (bool act = (s).active[(s).g.bidx(x, y, z)]; _once; _once = 0)
static_assert(NN_SR_BLOCK == 32, "a warp covers a block's row");

// Where particle (or vertex) i starts in an array of 3 words each; in int, the 9 words of G would
// end at 238 million particles.
__device__ __forceinline__ size_t at3(int i) { return 3 * (size_t)i; }

__device__ __forceinline__ void sr_fail(const SrDev& s, int code) { atomicCAS(s.status, 0, code); }

__device__ __forceinline__ void sr_add(const SrDev& s, int64_t c, double val) {
  if (!isfinite(val)) { sr_fail(s, NN_ERR_NAN); return; }
  val = fmin(fmax(val, -1e8), 1e8);
  atomicAdd(&s.fix[c], (unsigned long long)(long long)llrint(val * SR_FIX));
}

// ---- 1. voxel binning --------------------------------------------------------------
__global__ void k_sr_keys(SrDev s, int32_t cells) {
  if (blockIdx.x == 0 && threadIdx.x == 0) s.scan_n[2] = cells;
  GRID_STRIDE(i, s.n) {
    int x, y, z;
    s.g.voxel_of(s.pos[at3(i)], s.pos[at3(i) + 1], s.pos[at3(i) + 2], x, y, z);
    if (!s.g.in(x, y, z)) { sr_fail(s, NN_ERR_INVALID_ARG); s.vkey[i] = 0xffffffffu; continue; }
    const uint32_t k = (uint32_t)s.g.idx(x, y, z);
    s.vkey[i] = k;
    s.vrank[i] = atomicAdd(&s.vcount[k], 1u);
    if (s.vrank[i] >= NN_SR_MAX_PER_VOXEL) sr_fail(s, NN_ERR_CAPACITY);
  }
}
__global__ void k_sr_scatter(SrDev s) {
  GRID_STRIDE(i, s.n) {
    const uint32_t k = s.vkey[i];
    if (k != 0xffffffffu) s.vsrc[s.vcount[k] + s.vrank[i]] = i;
  }
}
// id order inside a voxel (at most a few particles)
__global__ void k_sr_voxel_sort(SrDev s, int64_t cells) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < cells; c += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t b = s.vcount[c], e = s.vcount[c + 1];
    for (uint32_t i = b + 1; i < e; ++i) {
      const int v = s.vsrc[i];
      uint32_t j = i;
      while (j > b && s.vsrc[j - 1] > v) { s.vsrc[j] = s.vsrc[j - 1]; --j; }
      s.vsrc[j] = v;
    }
  }
}

// Positions in voxel order; only the first vcount[cells] entries of vsrc are filled
// (particles outside the grid are not binned, and the call then fails).
__global__ void k_sr_sorted_pos(SrDev s, int64_t cells) {
  const int nb = (int)min((int64_t)s.vcount[cells], (int64_t)s.n);
  GRID_STRIDE(k, nb) {
    const int i = s.vsrc[k];
    if (i < 0 || i >= s.n) continue;
    s.spos[k] = make_float4(s.pos[at3(i)], s.pos[at3(i) + 1], s.pos[at3(i) + 2], 0.f);
  }
}

// ---- 2. isotropic splat (generate_fluid_field) --------------------------------------
__global__ void k_sr_iso(SrDev s) {
  GRID_STRIDE(i, s.n) {
    const float px = s.pos[at3(i)], py = s.pos[at3(i) + 1], pz = s.pos[at3(i) + 2];
    int cx, cy, cz;
    s.g.voxel_of(px, py, pz, cx, cy, cz);
    if (!s.g.in(cx, cy, cz)) continue;
    const float h = s.sr, h2 = h * h;
    const float h9 = h2 * h2 * h2 * h2 * h;
    for (int dz = -1; dz <= 1; ++dz)
      for (int dy = -1; dy <= 1; ++dy)
        for (int dx = -1; dx <= 1; ++dx) {
          const int x = cx + dx, y = cy + dy, z = cz + dz;
          if (x < 0 || y < 0 || z < 0) continue;
          if (!s.g.in(x, y, z)) { sr_fail(s, NN_ERR_CAPACITY); continue; }
          const float rx = px - (x * s.g.vs + s.g.ox), ry = py - (y * s.g.vs + s.g.oy), rz = pz - (z * s.g.vs + s.g.oz);
          const float r2 = rx * rx + ry * ry + rz * rz;
          float w = 0.f;  // poly6_weight, srtool.py:1212-1227
          if (sqrtf(r2) <= h) {
            const float t = h2 - r2;
            w = s.acoeff * (t * t * t) / h9;
          }
          s.active[s.g.bidx(x, y, z)] = 1;
          sr_add(s, s.g.idx(x, y, z), (double)(s.volume * w));
        }
  }
}

// ---- 3. anisotropic kernels (pre_process_data) ---------------------------------------
// symmetric 3x3 eigen-decomposition (cyclic Jacobi, double), descending eigenvalues,
// eigenvectors as the columns of V
__device__ void sr_sym_eig(const double S0[3][3], double lam[3], double V[3][3]) {
  double S[3][3], W[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) S[i][j] = S0[i][j];
  for (int sweep = 0; sweep < 16; ++sweep) {
    const double off = S[0][1] * S[0][1] + S[0][2] * S[0][2] + S[1][2] * S[1][2];
    const double dg = S[0][0] * S[0][0] + S[1][1] * S[1][1] + S[2][2] * S[2][2];
    if (off == 0.0 || off <= 1e-30 * dg) break;
#pragma unroll
    for (int pq = 0; pq < 3; ++pq) {
      const int p = pq == 2 ? 1 : 0, q = pq == 0 ? 1 : 2;
      if (S[p][q] == 0.0) continue;
      const double th = (S[q][q] - S[p][p]) / (2.0 * S[p][q]);
      const double t = (th >= 0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
      const double c = 1.0 / sqrt(t * t + 1.0), sn = t * c;
#pragma unroll
      for (int k = 0; k < 3; ++k) { const double a = S[k][p], b = S[k][q]; S[k][p] = c * a - sn * b; S[k][q] = sn * a + c * b; }
#pragma unroll
      for (int k = 0; k < 3; ++k) { const double a = S[p][k], b = S[q][k]; S[p][k] = c * a - sn * b; S[q][k] = sn * a + c * b; }
#pragma unroll
      for (int k = 0; k < 3; ++k) { const double a = W[k][p], b = W[k][q]; W[k][p] = c * a - sn * b; W[k][q] = sn * a + c * b; }
    }
  }
  const double d[3] = {S[0][0], S[1][1], S[2][2]};
  int o0 = 0, o1 = 1, o2 = 2;  // sort descending
  if (d[o1] > d[o0]) { int t = o0; o0 = o1; o1 = t; }
  if (d[o2] > d[o1]) { int t = o1; o1 = o2; o2 = t; }
  if (d[o1] > d[o0]) { int t = o0; o0 = o1; o1 = t; }
  const int o[3] = {o0, o1, o2};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    lam[c] = d[o[c]];
#pragma unroll
    for (int r = 0; r < 3; ++r) V[r][c] = W[r][o[c]];
  }
}

// Visits the particles within the smoothing range of voxel (cx, cy, cz) whose voxel
// can hold a point closer than `reach`, row by row (the voxels of one (y, z) row are
// one contiguous stretch of the voxel-sorted arrays, whose index k is passed to f);
// lane `lane` of `lanes` takes every lanes-th row.
// The particles of the voxel rows (x-runs) of the range around voxel (cx, cy, cz)
// whose y-z slab comes within `reach` of p, visited by a whole warp. Only about one
// row in four of the range crosses a particle lattice at half the voxel density, so
// lanes owning rows would mostly idle: each lane takes one row of a group of 32, a
// warp scan of the row counts lays their particles end to end, and lane l handles
// particles l, l + 32, ... of the group, finding its row by a search over the scan.
// f(k) gets the voxel-sorted index of each particle; `valid` lanes only.
template <typename F>
__device__ __forceinline__ void sr_range_particles(const SrDev& s, int cx, int cy, int cz, float px, float py,
                                                   float pz, float reach, int lane, F f) {
  const SrGrid& g = s.g;
  const unsigned full = 0xffffffffu;
  const int lo = -s.off, hi = s.range - 1 - s.off;
  const float r2 = reach * reach;
  const int x0 = max(cx + lo, 0), x1 = min(cx + hi, g.nx - 1);
  if (x0 > x1) return;  // warp-uniform
  const int nrows = s.range * s.range;
  for (int r0 = 0; r0 < nrows; r0 += 32) {
    const int r = r0 + lane;
    uint32_t b = 0, cnt = 0;
    if (r < nrows) {
      const int z = cz + lo + r / s.range, y = cy + lo + r % s.range;
      if (z >= 0 && z < g.nz && y >= 0 && y < g.ny) {
        const float zc = fmaxf(fmaxf(g.oz + z * g.vs - pz, pz - (g.oz + (z + 1) * g.vs)), 0.f);
        const float yc = fmaxf(fmaxf(g.oy + y * g.vs - py, py - (g.oy + (y + 1) * g.vs)), 0.f);
        if (yc * yc + zc * zc <= r2) {
          b = s.vcount[g.idx(x0, y, z)];
          cnt = s.vcount[g.idx(x1, y, z) + 1] - b;
        }
      }
    }
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(full, incl, o);
      if (lane >= o) incl += v;
    }
    const uint32_t total = __shfl_sync(full, incl, 31);
    for (uint32_t base = 0; base < total; base += 32) {
      const uint32_t t = base + lane;
      int l = 0;  // the first row lane whose inclusive count exceeds t
#pragma unroll
      for (int step = 16; step >= 1; step >>= 1)
        if (__shfl_sync(full, incl, l + step - 1) <= t) l += step;
      const uint32_t bl = __shfl_sync(full, b, l), il = __shfl_sync(full, incl, l), cl = __shfl_sync(full, cnt, l);
      if (t < total) f(bl + (t - (il - cl)));
    }
  }
}

// A block takes 8 * ppw particles: its warps gather the moments of ppw particles each
// (lanes split the particles of the range, the sums are reduced with shuffles), then one
// thread per particle does the rest, the FP64 eigen-decomposition above all. On lane 0 of
// the particle's warp that tail was a third of the kernel's issue slots with one lane of 32
// active (20.9 threads per instruction). ppw grows to SR_PRE_PPW with the particles, so
// that a small set still spreads over the chip (sr_pre_ppw).
#define SR_PRE_PPW 8
#define SR_PRE_WARPS 8
struct SrMoments { double tw, m1[3], m2[6]; int nnb; };

__device__ __forceinline__ void sr_aniso_kernel_of(const SrDev& s, int i, const SrMoments& a) {
  const float px = s.pos[at3(i)], py = s.pos[at3(i) + 1], pz = s.pos[at3(i) + 2];
  const double tw = a.tw;
  const double *m1 = a.m1, *m2 = a.m2;
  double db[3] = {0.0, 0.0, 0.0}, C[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  if (tw != 0.0) {
    db[0] = m1[0] / tw; db[1] = m1[1] / tw; db[2] = m1[2] / tw;
    C[0][0] = m2[0] / tw - db[0] * db[0]; C[1][1] = m2[1] / tw - db[1] * db[1]; C[2][2] = m2[2] / tw - db[2] * db[2];
    C[0][1] = C[1][0] = m2[3] / tw - db[0] * db[1];
    C[0][2] = C[2][0] = m2[4] / tw - db[0] * db[2];
    C[1][2] = C[2][1] = m2[5] / tw - db[1] * db[2];
  }
  const double xw[3] = {tw != 0.0 ? px + db[0] : 0.0, tw != 0.0 ? py + db[1] : 0.0, tw != 0.0 ? pz + db[2] : 0.0};
  const double lam_ = 0.9;  // akLambda
  s.xbar[at3(i)] = (float)((1 - lam_) * px + lam_ * xw[0]);
  s.xbar[at3(i) + 1] = (float)((1 - lam_) * py + lam_ * xw[1]);
  s.xbar[at3(i) + 2] = (float)((1 - lam_) * pz + lam_ * xw[2]);
  double lam[3], V[3][3];
  sr_sym_eig(C, lam, V);
  double sg[3] = {lam[0], lam[1], lam[2]};
  if (a.nnb > 25) {  // Nvep, kr = 4, ks = 1400 (srtool.py:910-914, 1072-1079)
    sg[1] = fmax(sg[1], sg[0] / 4.0);
    sg[2] = fmax(sg[2], sg[0] / 4.0);
    sg[0] *= 1400.0; sg[1] *= 1400.0; sg[2] *= 1400.0;
  } else {
    sg[0] = sg[1] = sg[2] = 0.5;  // kn
  }
#pragma unroll
  for (int a_ = 0; a_ < 3; ++a_)
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const double m = V[a_][0] * V[b][0] / sg[0] + V[a_][1] * V[b][1] / sg[1] + V[a_][2] * V[b][2] / sg[2];
      s.G[3 * at3(i) + 3 * a_ + b] = (float)(tw != 0.0 ? m / (double)s.sr : (a_ == b ? 1.0 : 0.0));
    }
}

__global__ void __launch_bounds__(SR_PRE_WARPS * 32) k_sr_aniso_pre(SrDev s, int ppw) {
  __shared__ SrMoments mom[SR_PRE_WARPS * SR_PRE_PPW];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int per = SR_PRE_WARPS * ppw, base = blockIdx.x * per;
  for (int k = w; k < per && base + k < s.n; k += SR_PRE_WARPS) {
    const int i = base + k;
    if (i == 0) continue;  // the reference's loop starts at 1 (srtool.py:1013)
    const float px = s.pos[at3(i)], py = s.pos[at3(i) + 1], pz = s.pos[at3(i) + 2];
    int cx, cy, cz;
    s.g.voxel_of(px, py, pz, cx, cy, cz);
    const float rr = 2.f * s.sr;  // isoweight radius
    // one pass over the neighbourhood: weights, and the first and second moments of
    // the offsets d_j = x_j - x_i, from which x_w = x_i + <d> and
    // C = sum w (x_j - x_w)(x_j - x_w)^T / sum w = <d d^T> - <d><d>^T (srtool.py:1021-1061)
    double tw = 0.0, m1[3] = {0.0, 0.0, 0.0}, m2[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    int nnb = 0;
    // a margin of one voxel on the pruning distance keeps every pair with w > 0
    sr_range_particles(s, cx, cy, cz, px, py, pz, rr + s.g.vs, lane, [&](uint32_t q_) {
      const float4 pj = s.spos[q_];
      const float dx = __fsub_rn(px, pj.x), dy = __fsub_rn(py, pj.y), dz = __fsub_rn(pz, pj.z);
      const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
      // |x_i - x_j| in f32 (unfused, as any f32 evaluation of it) < 2 r_s, decided on
      // the square: rn(sqrt(d2)) < rr exactly when d2 < rr_thr
      if (d2 < s.rr_thr) {
        const float dn = __fsqrt_rn(d2);
        const float q = dn / rr;
        const double w_ = 1.0 - (double)(q * q * q);  // isoweight, srtool.py:993-999
        const double d[3] = {(double)pj.x - px, (double)pj.y - py, (double)pj.z - pz};
        tw += w_;
        m1[0] += w_ * d[0]; m1[1] += w_ * d[1]; m1[2] += w_ * d[2];
        if (w_ > 0) {
          ++nnb;
          m2[0] += w_ * d[0] * d[0]; m2[1] += w_ * d[1] * d[1]; m2[2] += w_ * d[2] * d[2];
          m2[3] += w_ * d[0] * d[1]; m2[4] += w_ * d[0] * d[2]; m2[5] += w_ * d[1] * d[2];
        }
      }
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      tw += __shfl_xor_sync(0xffffffffu, tw, o);
#pragma unroll
      for (int q = 0; q < 3; ++q) m1[q] += __shfl_xor_sync(0xffffffffu, m1[q], o);
#pragma unroll
      for (int q = 0; q < 6; ++q) m2[q] += __shfl_xor_sync(0xffffffffu, m2[q], o);
      nnb += __shfl_xor_sync(0xffffffffu, nnb, o);
    }
    if (lane == 0) {
      SrMoments& a = mom[k];
      a.tw = tw;
#pragma unroll
      for (int q = 0; q < 3; ++q) a.m1[q] = m1[q];
#pragma unroll
      for (int q = 0; q < 6; ++q) a.m2[q] = m2[q];
      a.nnb = nnb;
    }
  }
  __syncthreads();
  const int k = (int)threadIdx.x;
  if (k < per && base + k < s.n) {
    if (base + k != 0) {
      sr_aniso_kernel_of(s, base + k, mom[k]);
    } else {
      for (int q = 0; q < 9; ++q) s.G[q] = 0.f;
      for (int q = 0; q < 3; ++q) s.xbar[q] = 0.f;
    }
  }
}
// Particles per warp of the pre-pass: one until every SM has two blocks' worth.
static int sr_pre_ppw(int n, int sms) { return std::min(std::max(n / (SR_PRE_WARPS * 2 * sms), 1), SR_PRE_PPW); }

// ---- 4. anisotropic splat (generate_smooth_fluid_field_impl) -------------------------
// One warp per particle; each lane owns (x, y) columns of the kernel's support box and
// walks z two vertices at a time in packed f32x2 arithmetic. Bound by instruction issue:
// 2.2 G kernel evaluations per call on the 125,000-particle drop, about half of them
// inside the support. What depends on z alone (the z terms of G d and the multiplicity
// scale) is the same for all columns: the warp's lanes compute it once per particle into
// shared memory, in chunks of SR_ZC planes. Where the particle's largest contribution is
// known to fit, the fixed-point conversion is the 32-bit one (the 64-bit conversion issues
// at a quarter of its rate) and needs no range checks. Every value rounds as the scalar
// expressions of the kernel do (packed squares as fma(q, q, +0), see ns.cuh), so the field
// has the same bits as one vertex at a time: the drop's splat 4.8 -> 2.85 ms.
#define SR_ZC 32
#define SR_SPLAT_WARPS 8
// c times the scale m (2^32 x multiplicity) in fixed point, over the whole f32 range
__device__ __forceinline__ void sr_splat_add(const SrDev& s, unsigned long long* out, float c, float m) {
  if (!isfinite(c)) { sr_fail(s, NN_ERR_NAN); return; }
  atomicAdd(out, (unsigned long long)__float2ll_rn(fminf(fmaxf(c, -1e8f), 1e8f) * m));
}
__device__ __forceinline__ uint64_t pack_x2(float a, float b) {
  return (uint64_t)__float_as_uint(a) | ((uint64_t)__float_as_uint(b) << 32);
}
__device__ __forceinline__ float lo_x2(uint64_t a) { return __uint_as_float((uint32_t)a); }
__device__ __forceinline__ float hi_x2(uint64_t a) { return __uint_as_float((uint32_t)(a >> 32)); }
__device__ __forceinline__ uint64_t mul_rn_x2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma_rn_x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// 1 / sqrt(x) of a normal x, finite for x below the normal range: MUFU alone, without the
// rescaling of subnormal arguments that rsqrtf adds (x * this is then below 2^-62, where the
// kernel rounds to its value at 0)
__device__ __forceinline__ float rsqrt_min(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fmaxf(x, 1.17549435e-38f)));
  return r;
}
__global__ void __launch_bounds__(SR_SPLAT_WARPS * 32) k_sr_aniso_splat(SrDev s, int parts) {
  // per pair of planes: the z terms G[.][2] d2 and the scale (2^32 x multiplicity, times the
  // volume where the conversion is the narrow one)
  __shared__ __align__(16) float zt_all[SR_SPLAT_WARPS][4 * SR_ZC];
  float* zt = zt_all[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < s.n * parts; k += warps) {
    const int i = k / parts, part = k % parts;
    const SrGrid& g = s.g;
    int cx, cy, cz;
    g.voxel_of(s.pos[at3(i)], s.pos[at3(i) + 1], s.pos[at3(i) + 2], cx, cy, cz);
    // voxels [c - off, c - off + range - 1]; their vertices one further
    const int lo[3] = {cx - s.off, cy - s.off, cz - s.off};
    const int hi[3] = {lo[0] + s.range - 1, lo[1] + s.range - 1, lo[2] + s.range - 1};
    if (hi[0] + 1 >= g.nx || hi[1] + 1 >= g.ny || hi[2] + 1 >= g.nz) {
      if (lane == 0) sr_fail(s, NN_ERR_CAPACITY);
      continue;
    }
    const int v0[3] = {max(lo[0], 0), max(lo[1], 0), max(lo[2], 0)};
    const int v1[3] = {hi[0] + 1, hi[1] + 1, hi[2] + 1};
    if (v1[0] < 0 || v1[1] < 0 || v1[2] < 0) continue;
    {  // every vertex of the box is written (+= 0 included): activate its blocks
      const int b0 = v0[0] / NN_SR_BLOCK, b1 = v1[0] / NN_SR_BLOCK, c0 = v0[1] / NN_SR_BLOCK,
                c1 = v1[1] / NN_SR_BLOCK, e0 = v0[2] / NN_SR_BLOCK, e1 = v1[2] / NN_SR_BLOCK;
      const int nbx = b1 - b0 + 1, nby = c1 - c0 + 1, nb = nbx * nby * (e1 - e0 + 1);
      for (int t = lane; t < nb; t += 32) {
        const int bx = b0 + t % nbx, by = c0 + (t / nbx) % nby, bz = e0 + t / (nbx * nby);
        s.active[bx + (int64_t)g.bx * (by + (int64_t)g.by * bz)] = 1;
      }
    }
    float Gm[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) Gm[k] = s.G[3 * at3(i) + k];
    const double det = (double)Gm[0] * ((double)Gm[4] * Gm[8] - (double)Gm[5] * Gm[7]) -
                       (double)Gm[1] * ((double)Gm[3] * Gm[8] - (double)Gm[5] * Gm[6]) +
                       (double)Gm[2] * ((double)Gm[3] * Gm[7] - (double)Gm[4] * Gm[6]);
    if (det == 0.0) continue;  // G = 0 (particle 0): the kernel is 0 everywhere
    // support |G d| <= 1 is an ellipsoid; its bounding half-widths are the row norms of G^-1
    double Gi[3][3];
    Gi[0][0] = ((double)Gm[4] * Gm[8] - (double)Gm[5] * Gm[7]) / det;
    Gi[0][1] = ((double)Gm[2] * Gm[7] - (double)Gm[1] * Gm[8]) / det;
    Gi[0][2] = ((double)Gm[1] * Gm[5] - (double)Gm[2] * Gm[4]) / det;
    Gi[1][0] = ((double)Gm[5] * Gm[6] - (double)Gm[3] * Gm[8]) / det;
    Gi[1][1] = ((double)Gm[0] * Gm[8] - (double)Gm[2] * Gm[6]) / det;
    Gi[1][2] = ((double)Gm[2] * Gm[3] - (double)Gm[0] * Gm[5]) / det;
    Gi[2][0] = ((double)Gm[3] * Gm[7] - (double)Gm[4] * Gm[6]) / det;
    Gi[2][1] = ((double)Gm[1] * Gm[6] - (double)Gm[0] * Gm[7]) / det;
    Gi[2][2] = ((double)Gm[0] * Gm[4] - (double)Gm[1] * Gm[3]) / det;
    const float xb[3] = {s.xbar[at3(i)], s.xbar[at3(i) + 1], s.xbar[at3(i) + 2]};
    const double org[3] = {g.dox, g.doy, g.doz};
    int w0[3], w1[3];
    bool empty = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double hw = sqrt(Gi[a][0] * Gi[a][0] + Gi[a][1] * Gi[a][1] + Gi[a][2] * Gi[a][2]);
      const double lo_v = (xb[a] - hw - org[a]) / g.dvs, hi_v = (xb[a] + hw - org[a]) / g.dvs;
      w0[a] = max(v0[a], (int)fmax(floor(lo_v) - 1.0, -1e9));
      w1[a] = min(v1[a], (int)fmin(ceil(hi_v) + 1.0, 1e9));
      empty |= w0[a] > w1[a];
    }
    if (empty) continue;
    const float k1 = (float)(48.0 / SR_PI * det), k2 = (float)(16.0 / SR_PI * det);
    // the largest |contribution| over the support, q in (0, 1]: 1 + |k1| (q^2 - q^3) up to
    // q = 0.5 and |k2| / 8 beyond; times the multiplicity 8 it must stay below 2^31 units
    const float top = s.volume * (2.f + 0.125f * fabsf(k1) + 0.125f * fabsf(k2));
    const bool narrow = top < 0.06f;  // 8 * 0.06 * 2^32 < 2^31; false for NaN
    const uint64_t nk1 = pack_x2(-k1, -k1), k2x2 = pack_x2(k2, k2), one = pack_x2(1.f, 1.f),
                   minus = pack_x2(-1.f, -1.f);
    // the x and y terms of G d are per column and the sums keep the order
    // ((G0 d0 + G1 d1) + G2 d2)
    const int nxw = w1[0] - w0[0] + 1, ncol = nxw * (w1[1] - w0[1] + 1);
    const int64_t plane = (int64_t)g.nx * g.ny;
    for (int zc = w0[2]; zc <= w1[2]; zc += SR_ZC) {
      const int nz = min(SR_ZC, w1[2] - zc + 1);
      __syncwarp();
      {
        const int z = zc + lane;
        const float d2 = __fsub_rn(xb[2], __fadd_rn(__fmul_rn((float)z, g.vs), g.oz));
        const int mz = (z - 1 >= lo[2] && z - 1 <= hi[2]) + (z >= lo[2] && z <= hi[2]);
        float* e = zt + (lane >> 1) * 8 + (lane & 1);
        // the plane past an odd chunk is NaN, which no test lets into the support
        e[0] = lane < nz ? __fmul_rn(Gm[2], d2) : __uint_as_float(0x7fffffffu);
        e[2] = __fmul_rn(Gm[5], d2);
        e[4] = __fmul_rn(Gm[8], d2);
        e[6] = narrow ? s.volume * (4294967296.f * (float)mz) : 4294967296.f * (float)mz;
      }
      __syncwarp();
      for (int col = lane + 32 * part; col < ncol; col += 32 * parts) {
        const int x = w0[0] + col % nxw, y = w0[1] + col / nxw;
        const int mxy = ((x - 1 >= lo[0] && x - 1 <= hi[0]) + (x >= lo[0] && x <= hi[0])) *
                        ((y - 1 >= lo[1] && y - 1 <= hi[1]) + (y >= lo[1] && y <= hi[1]));
        if (mxy == 0) continue;
        const float d0 = __fsub_rn(xb[0], __fadd_rn(__fmul_rn((float)x, g.vs), g.ox));
        const float d1 = __fsub_rn(xb[1], __fadd_rn(__fmul_rn((float)y, g.vs), g.oy));
        const float a0 = __fadd_rn(__fmul_rn(Gm[0], d0), __fmul_rn(Gm[1], d1));
        const float a1 = __fadd_rn(__fmul_rn(Gm[3], d0), __fmul_rn(Gm[4], d1));
        const float a2 = __fadd_rn(__fmul_rn(Gm[6], d0), __fmul_rn(Gm[7], d1));
        const uint64_t a0x2 = pack_x2(a0, a0), a1x2 = pack_x2(a1, a1), a2x2 = pack_x2(a2, a2),
                       mx2 = pack_x2((float)mxy, (float)mxy);
        unsigned long long* out = s.fix + g.idx(x, y, zc);
        // f(value pair, scale pair, in a, in b) per pair of planes inside the support
        auto walk = [&](auto put) {
          for (int t = 0; t < nz; t += 2, out += 2 * plane) {
            const ulonglong2 ta = *reinterpret_cast<const ulonglong2*>(zt + 4 * t);
            const ulonglong2 tb = *reinterpret_cast<const ulonglong2*>(zt + 4 * t + 4);
            // q = |G (x_bar - vertex)| in f32 with unfused operations: the kernel as written
            // jumps at q = 0.5, so q must round the same way in every f32 evaluation
            const uint64_t q0 = add_rn_x2(a0x2, ta.x), q1 = add_rn_x2(a1x2, ta.y), q2 = add_rn_x2(a2x2, tb.x);
            const uint64_t qs = add_rn_x2(add_rn_x2(sq_rn_x2(q0), sq_rn_x2(q1)), sq_rn_x2(q2));
            const float qa = lo_x2(qs), qb = hi_x2(qs);
            // outside the support: rn(sqrt(q2s)) > 1 exactly when q2s > q1_thr
            const bool ina = qa <= s.q1_thr && qa > 0.f, inb = qb <= s.q1_thr && qb > 0.f;
            if (!(ina || inb)) continue;
            // the branch of cubic_spline_kernel (srtool.py:1114-1124) is decided exactly
            // (rn(sqrt(q2s)) <= 0.5 exactly when q2s <= q05_thr); its value, continuous
            // within a branch, takes q from the hardware reciprocal square root:
            //   k1 (q^3 - q^2) + 1 as fma(-k1, fma(q^2, -q, q^2), 1), and k2 (1 - q)^3
            const uint64_t q = mul_rn_x2(qs, pack_x2(rsqrt_min(qa), rsqrt_min(qb)));
            const uint64_t qq = mul_rn_x2(q, q), nq = mul_rn_x2(q, minus);
            const uint64_t inner = fma_rn_x2(nk1, fma_rn_x2(qq, nq, qq), one);
            const uint64_t u = add_rn_x2(one, nq);
            const uint64_t outer = mul_rn_x2(mul_rn_x2(mul_rn_x2(k2x2, u), u), u);
            // vertex (x, y, z) belongs to the voxels x - 1 and x of the box, per axis; the
            // multiplicity is 1, 2, 4 or 8, a power of two, so scaling by it is exact
            put(pack_x2(qa <= s.q05_thr ? lo_x2(inner) : lo_x2(outer), qb <= s.q05_thr ? hi_x2(inner) : hi_x2(outer)),
                mul_rn_x2(mx2, tb.y), ina, inb);
          }
        };
        if (narrow) {
          walk([&](uint64_t res, uint64_t m, bool ina, bool inb) {
            const uint64_t f = mul_rn_x2(res, m);
            if (ina) atomicAdd(out, (unsigned long long)(long long)__float2int_rn(lo_x2(f)));
            if (inb) atomicAdd(out + plane, (unsigned long long)(long long)__float2int_rn(hi_x2(f)));
          });
        } else {
          walk([&](uint64_t res, uint64_t m, bool ina, bool inb) {
            if (ina) sr_splat_add(s, out, s.volume * lo_x2(res), lo_x2(m));
            if (inb) sr_splat_add(s, out + plane, s.volume * hi_x2(res), hi_x2(m));
          });
        }
      }
    }
  }
}

// Velocity splat (generate_smooth_fluid_field_with_velocity_impl, srtool.py:1159-1190):
// every vertex of every voxel in the smoothing range, once per adjacent voxel, gets
// v_i * poly6(x_i - vertex, r_s) * voxel_size^3. One warp per particle; lanes own
// (x, y) columns of the poly6 support's box and walk z.
__global__ void k_sr_vel_splat(SrDev s) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const float h = s.sr, h2 = h * h, h9 = h2 * h2 * h2 * h2 * h;
  const float coeff = s.g.vs * s.g.vs * s.g.vs;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < s.n; i += warps) {
    const SrGrid& g = s.g;
    const float px = s.pos[at3(i)], py = s.pos[at3(i) + 1], pz = s.pos[at3(i) + 2];
    int cx, cy, cz;
    g.voxel_of(px, py, pz, cx, cy, cz);
    const int lo[3] = {cx - s.off, cy - s.off, cz - s.off};
    const int hi[3] = {lo[0] + s.range - 1, lo[1] + s.range - 1, lo[2] + s.range - 1};
    if (hi[0] + 1 >= g.nx || hi[1] + 1 >= g.ny || hi[2] + 1 >= g.nz) continue;  // flagged by the field splat
    const float p[3] = {px, py, pz};
    const float org[3] = {g.ox, g.oy, g.oz};
    int w0[3], w1[3];
    bool empty = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {  // the poly6 support |x_i - vertex| <= r_s, one vertex of margin
      w0[a] = max(max(lo[a], 0), (int)floorf((p[a] - h - org[a]) / g.vs) - 1);
      w1[a] = min(hi[a] + 1, (int)ceilf((p[a] + h - org[a]) / g.vs) + 1);
      empty |= w0[a] > w1[a];
    }
    if (empty) continue;
    const float v[3] = {s.vel[at3(i)], s.vel[at3(i) + 1], s.vel[at3(i) + 2]};
    const int nxw = w1[0] - w0[0] + 1, ncol = nxw * (w1[1] - w0[1] + 1);
    const int64_t plane = (int64_t)g.nx * g.ny, cells = plane * g.nz;
    for (int col = lane; col < ncol; col += 32) {
      const int x = w0[0] + col % nxw, y = w0[1] + col / nxw;
      const int mxy = ((x - 1 >= lo[0] && x - 1 <= hi[0]) + (x >= lo[0] && x <= hi[0])) *
                      ((y - 1 >= lo[1] && y - 1 <= hi[1]) + (y >= lo[1] && y <= hi[1]));
      if (mxy == 0) continue;
      const float rx = px - (x * g.vs + g.ox), ry = py - (y * g.vs + g.oy);
      const int64_t base = g.idx(x, y, 0);
      for (int z = w0[2]; z <= w1[2]; ++z) {
        const float rz = pz - (z * g.vs + g.oz);
        const float r2 = rx * rx + ry * ry + rz * rz;
        if (!(sqrtf(r2) <= h)) continue;  // poly6_weight, srtool.py:1212-1227
        const float t = h2 - r2;
        const float w = s.acoeff * (t * t * t) / h9 * coeff;
        const int m = mxy * ((z - 1 >= lo[2] && z - 1 <= hi[2]) + (z >= lo[2] && z <= hi[2]));
        if (m == 0) continue;
        const int64_t c = base + z * plane;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float cv = v[k] * w;
          if (!isfinite(cv)) { sr_fail(s, NN_ERR_NAN); continue; }
          const long long u = __float2ll_rn(fminf(fmaxf(cv, -1e8f), 1e8f) * (4294967296.f * (float)m));
          atomicAdd(&s.vfix[k * cells + c], (unsigned long long)u);
        }
      }
    }
  }
}

// process_velocity (srtool.py:1351-1381): trilinear blend of the 8 vertex velocities
// around each mesh vertex
__global__ void k_sr_mesh_velocity(SrDev s, int nv) {
  const int64_t plane = (int64_t)s.g.nx * s.g.ny, cells = plane * s.g.nz;
  GRID_STRIDE(i, min(nv, s.max_v)) {
    const double p[3] = {s.vert[at3(i)], s.vert[at3(i) + 1], s.vert[at3(i) + 2]};
    int x0, y0, z0;
    s.g.voxel_of((float)p[0], (float)p[1], (float)p[2], x0, y0, z0);
    const double xd = (p[0] - (x0 * s.g.dvs + s.g.dox)) / s.g.dvs, yd = (p[1] - (y0 * s.g.dvs + s.g.doy)) / s.g.dvs,
                 zd = (p[2] - (z0 * s.g.dvs + s.g.doz)) / s.g.dvs;
    double acc[3] = {0.0, 0.0, 0.0};
    for (int a = 0; a < 2; ++a)
      for (int b = 0; b < 2; ++b)
        for (int e = 0; e < 2; ++e) {
          const int x = x0 + a, y = y0 + b, z = z0 + e;
          if (!s.g.in(x, y, z)) continue;
          const double wgt = (a ? xd : 1 - xd) * (b ? yd : 1 - yd) * (e ? zd : 1 - zd);
          const int64_t c = s.g.idx(x, y, z);
          for (int k = 0; k < 3; ++k) acc[k] += wgt * ((double)(long long)s.vfix[k * cells + c] / SR_FIX);
        }
    for (int k = 0; k < 3; ++k) s.mvel[at3(i) + k] = (float)acc[k];
  }
}

// Sum of two values over the block into dst[0] and dst[1]: one atomic each per block (one
// per warp, on the same two addresses, took 49 us on a 3 M vertex grid).
__device__ __forceinline__ void sr_block_add(double a, double b, double* dst, bool second) {
  __shared__ double sh[2][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (lane == 0) { sh[0][w] = a; sh[1][w] = b; }
  __syncthreads();
  if (threadIdx.x == 0) {
    a = b = 0.0;
    for (int k = 0; k < nw; ++k) { a += sh[0][k]; b += sh[1][k]; }
    if (a != 0.0) atomicAdd(&dst[0], a);
    if (second && b != 0.0) atomicAdd(&dst[1], b);
  }
}

// The splat field in floats, and the first pass of the smoothing's statistics over it (the
// sum and count of its negative values; only active blocks hold any).
__global__ void k_sr_fix_to_field(SrDev s, int32_t cells) {
  if (blockIdx.x == 0 && threadIdx.x == 0) s.scan_n[2] = cells;
  double a = 0.0, b = 0.0;
  FOR_CELLS(c, cells) {
    const float v = (float)((double)(long long)s.fix[c] / SR_FIX);
    s.splat[c] = v;
    s.field[c] = v;
    if (v < 0.f) { a += v; b += 1.0; }
  }
  sr_block_add(a, b, &s.stats[0], true);
}

// ---- 5. smoothing (smooth_sdf) --------------------------------------------------------
// A field's value at a vertex, 0 outside the grid. Vertices of inactive blocks hold 0: no
// splat reaches them and the smoothing writes 0 there.
__device__ __forceinline__ float sr_get(const SrDev& s, const float* f, int x, int y, int z) {
  return s.g.in(x, y, z) ? f[s.g.idx(x, y, z)] : 0.f;
}

// density_field_stats (srtool.py:1436-1456): pass 0 sums the negative values of the
// active vertices and counts them, pass 1 their squared deviations from the mean
__global__ void k_sr_stats(SrDev s, int pass) {
  double a = 0.0, b = 0.0;
  const double mean = pass ? s.stats[0] / s.stats[1] : 0.0;
  FOR_SR_ROWS(s, x, y, z, c, act) {
    if (!act) continue;
    const float v = s.field[c];
    if (v < 0.f) {
      if (pass == 0) { a += v; b += 1.0; }
      else { const double d = v - mean; a += d * d; }
    }
  }
  sr_block_add(a, b, &s.stats[pass ? 2 : 0], pass == 0);
}
__global__ void k_sr_sd(SrDev s) {
  // 0/0 = NaN without negative values, as in the reference (the smoothing then
  // produces NaN and the contouring finds no crossing)
  if (threadIdx.x == 0) s.stats[3] = sqrt(s.stats[2] / s.stats[1]);
}

// Equal values, above all the zeros around the splats, take the weight of a zero difference,
// computed once; the others the exponential and the division.
template <int RT>
__global__ void k_sr_smooth(SrDev s) {
  const float sd = (float)s.stats[3];
  const float inv2s2 = 1.f / (2.f * sd * sd);
  const float norm = powf(2.f * (float)SR_PI * sd * sd, 1.5f);
  auto gauss = [&](float diff) { return expf(-diff * diff * inv2s2) / norm; };  // gaussian_blur, srtool.py:1432-1434
  const float g0 = gauss(0.f);
  const int R = RT ? RT : s.smooth_cells;
  const int64_t sy = s.g.nx, sz = (int64_t)s.g.nx * s.g.ny;
  FOR_SR_ROWS(s, x, y, z, c, act) {
    if (!act) { s.tmp[c] = 0.f; continue; }
    const float v0 = s.field[c];
    float avg = 0.f, wsum = 0.f;
    const bool inside = x >= R && y >= R && z >= R && x + R < s.g.nx && y + R < s.g.ny && z + R < s.g.nz;
    for (int dz = -R; dz <= R; ++dz)
      for (int dy = -R; dy <= R; ++dy)
#pragma unroll
        for (int dx = -R; dx <= R; ++dx) {
          float vv;
          if (inside) {
            vv = s.field[c + dx + dy * sy + dz * sz];
          } else {
            const int a = x + dx, b = y + dy, e = z + dz;
            if (a < 0 || b < 0 || e < 0) continue;
            vv = sr_get(s, s.field, a, b, e);
          }
          const float diff = fabsf(v0 - vv);
          const float gw = diff == 0.f ? g0 : gauss(diff);
          avg += gw * vv;
          wsum += gw;
        }
    if (wsum != 0.f) avg /= wsum;
    s.tmp[c] = avg;
  }
}

// ---- 6. dual contouring ---------------------------------------------------------------
__device__ __forceinline__ int sr_cube_mask(const SrDev& s, int x, int y, int z) {
  int ci = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w)
    if (sr_get(s, s.field, x + c_sr_off[w][0], y + c_sr_off[w][1], z + c_sr_off[w][2]) < s.iso) ci |= 1 << w;
  return ci;
}
__device__ __forceinline__ bool sr_edge_cross(int ci, int w) {
  return ((ci >> c_sr_edge[w][0]) ^ (ci >> c_sr_edge[w][1])) & 1;
}

__global__ void k_sr_dc_flag(SrDev s, int32_t cells) {
  if (blockIdx.x == 0 && threadIdx.x == 0) s.vflag[cells] = 0u;
  FOR_SR_ROWS(s, x, y, z, c, act) {
    uint32_t f = 0u;
    if (act) {
      const int ci = sr_cube_mask(s, x, y, z);
      f = (ci != 0 && ci != 255) ? 1u : 0u;
    }
    s.vflag[c] = f;
  }
}

// calc_vertex_normal (srtool.py:1306-1321), normalised
__device__ void sr_vertex_normal(const SrDev& s, int x, int y, int z, double n[3]) {
  const float* f = s.field;
  n[0] = (x == 0) ? -(double)sr_get(s, f, x + 1, y, z) : (double)sr_get(s, f, x - 1, y, z) - sr_get(s, f, x + 1, y, z);
  n[1] = (y == 0) ? -(double)sr_get(s, f, x, y + 1, z) : (double)sr_get(s, f, x, y - 1, z) - sr_get(s, f, x, y + 1, z);
  n[2] = (z == 0) ? -(double)sr_get(s, f, x, y, z + 1) : (double)sr_get(s, f, x, y, z - 1) - sr_get(s, f, x, y, z + 1);
  const double l = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
  if (l != 0.0) { n[0] /= l; n[1] /= l; n[2] /= l; }
}
// process_normal_at (srtool.py:1335-1349)
__device__ void sr_normal_at(const SrDev& s, const double p[3], double n[3]) {
  int x0, y0, z0;
  s.g.voxel_of((float)p[0], (float)p[1], (float)p[2], x0, y0, z0);
  const double xd = (p[0] - (x0 * s.g.dvs + s.g.dox)) / s.g.dvs, yd = (p[1] - (y0 * s.g.dvs + s.g.doy)) / s.g.dvs,
               zd = (p[2] - (z0 * s.g.dvs + s.g.doz)) / s.g.dvs;
  double acc[3] = {0.0, 0.0, 0.0};
  for (int a = 0; a < 2; ++a)
    for (int b = 0; b < 2; ++b)
      for (int e = 0; e < 2; ++e) {
        double c[3];
        sr_vertex_normal(s, x0 + a, y0 + b, z0 + e, c);
        const double wgt = (a ? xd : 1 - xd) * (b ? yd : 1 - yd) * (e ? zd : 1 - zd);
        acc[0] += wgt * c[0]; acc[1] += wgt * c[1]; acc[2] += wgt * c[2];
      }
  const double l = sqrt(acc[0] * acc[0] + acc[1] * acc[1] + acc[2] * acc[2]);
  if (l != 0.0) { n[0] = acc[0] / l; n[1] = acc[1] / l; n[2] = acc[2] / l; }
  else n[0] = n[1] = n[2] = 0.0;
}

// The crossing cubes in vertex-id order, so that the QEF kernel runs on dense work.
__global__ void k_sr_dc_list(SrDev s, int32_t cells) {
  FOR_CELLS(c, cells) {
    const uint32_t id = s.vflag[c];
    if (s.vflag[c + 1] != id && (int64_t)id < s.max_v) s.cube_of[id] = c;
  }
}

// One point per crossing cube: the mass point of the edge crossings plus the clamped
// QEF solution, kept only if it stays in its cube (srtool.py:1536-1596).
//
// Bound by the FP64 chain per cube, above all the field normals at its 4 to 12 crossings
// (8 vertex normals each). SR_QEF_LANES lanes share a cube: lane l takes the crossings
// l, l + 4, l + 8 of its edge order, and all of them fold the crossings' terms in that
// order by shuffles, so the sums are the one-thread sums. 52 -> 25 us on 5,400 cubes,
// 90 -> 94 us on 61,000 (the eigen-decomposition is every lane's).
#define SR_QEF_LANES 4
__global__ void __launch_bounds__(128) k_sr_dc_point(SrDev s, int64_t cells) {
  constexpr int L = SR_QEF_LANES, SLOTS = 12 / L;
  const unsigned full = 0xffffffffu;
  const int nv = (int)min((int64_t)s.vflag[cells], (int64_t)s.max_v);
  const int l = (int)threadIdx.x & (L - 1), g0 = (int)threadIdx.x & 31 & ~(L - 1);
  // the warp's first cube decides, so that all its lanes reach the shuffles
  for (int first = (int)(blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) / L; first < nv;
       first += (int)(gridDim.x * blockDim.x) / L) {
    const int id = min(first + (int)(threadIdx.x & 31) / L, nv - 1);
    const int c = (int)s.cube_of[id];
    const int x = c % s.g.nx, y = (c / s.g.nx) % s.g.ny, z = c / (s.g.nx * s.g.ny);
    const int ci = sr_cube_mask(s, x, y, z);
    uint32_t em = 0u;
#pragma unroll
    for (int w = 0; w < 12; ++w) em |= (uint32_t)sr_edge_cross(ci, w) << w;
    const int cnt = __popc(em);
    double P[SLOTS][3], N[SLOTS][3], bb[SLOTS];
    for (int k = 0; k < l; ++k) em &= em - 1u;  // to this lane's first crossing
#pragma unroll
    for (int q = 0; q < SLOTS; ++q) {
      if (q * L + l < cnt) {
        const int w = __ffs(em) - 1;
#pragma unroll
        for (int k = 0; k < L; ++k) em &= em - 1u;
        const int a = c_sr_edge[w][0], b = c_sr_edge[w][1];
        const int ax = x + c_sr_off[a][0], ay = y + c_sr_off[a][1], az = z + c_sr_off[a][2];
        const int bx = x + c_sr_off[b][0], by = y + c_sr_off[b][1], bz = z + c_sr_off[b][2];
        const double v1 = sr_get(s, s.field, ax, ay, az), v2 = sr_get(s, s.field, bx, by, bz);
        const double delta = v2 - v1;
        const double t = fabs(delta) < 1e-5 ? 0.5 : ((double)s.iso - v1) / delta;  // vertex_interpolate
        const double p1[3] = {ax * s.g.dvs + s.g.dox, ay * s.g.dvs + s.g.doy, az * s.g.dvs + s.g.doz};
        const double p2[3] = {bx * s.g.dvs + s.g.dox, by * s.g.dvs + s.g.doy, bz * s.g.dvs + s.g.doz};
#pragma unroll
        for (int k = 0; k < 3; ++k) P[q][k] = p1[k] + t * (p2[k] - p1[k]);
      } else {
        P[q][0] = P[q][1] = P[q][2] = 0.0;
      }
    }
    double mean[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int r = 0; r < 12; ++r)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double v = __shfl_sync(full, P[r / L][k], g0 + r % L);
        if (r < cnt) mean[k] += v;
      }
#pragma unroll
    for (int k = 0; k < 3; ++k) mean[k] /= cnt;
#pragma unroll
    for (int q = 0; q < SLOTS; ++q) {
      N[q][0] = N[q][1] = N[q][2] = bb[q] = 0.0;
      if (q * L + l < cnt) {
        sr_normal_at(s, P[q], N[q]);
        bb[q] = N[q][0] * (P[q][0] - mean[0]) + N[q][1] * (P[q][1] - mean[1]) + N[q][2] * (P[q][2] - mean[2]);
      }
    }
    double NtN[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, Ntb[3] = {0, 0, 0};
#pragma unroll
    for (int r = 0; r < 12; ++r) {
      double n[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) n[k] = __shfl_sync(full, N[r / L][k], g0 + r % L);
      const double b = __shfl_sync(full, bb[r / L], g0 + r % L);
      if (r < cnt)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          Ntb[i] += n[i] * b;
#pragma unroll
          for (int k = 0; k < 3; ++k) NtN[i][k] += n[i] * n[k];
        }
    }
    double lam[3], V[3][3], res[3] = {0.0, 0.0, 0.0};
    sr_sym_eig(NtN, lam, V);
    for (int i = 0; i < 3; ++i) {
      const double sv = sqrt(fmax(lam[i], 0.0));
      if (!(sv > 0.0)) continue;
      const double f = (V[0][i] * Ntb[0] + V[1][i] * Ntb[1] + V[2][i] * Ntb[2]) / (sv * fmax(sv, 0.1));
      for (int k = 0; k < 3; ++k) res[k] += f * V[k][i];
    }
    int qx, qy, qz;
    s.g.voxel_of((float)(res[0] + mean[0]), (float)(res[1] + mean[1]), (float)(res[2] + mean[2]), qx, qy, qz);
    const bool keep = qx == x && qy == y && qz == z;
    if (l != 0 || id != first + (int)(threadIdx.x & 31) / L) continue;
    for (int k = 0; k < 3; ++k) s.vert[3 * (int64_t)id + k] = (float)(keep ? res[k] + mean[k] : mean[k]);
  }
}

// get_edge_adjacent_cubes (srtool.py:1612-1705) for edges 2 (x), 3 (y), 11 (z) of corner 3
__device__ __forceinline__ void sr_edge_cubes(int w, int d[4][3]) {
  const int t2[4][3] = {{0, 0, 0}, {0, 0, -1}, {0, -1, -1}, {0, -1, 0}};
  const int t3[4][3] = {{0, 0, 0}, {0, 0, -1}, {-1, 0, -1}, {-1, 0, 0}};
  const int t11[4][3] = {{0, 0, 0}, {0, -1, 0}, {-1, -1, 0}, {-1, 0, 0}};
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int k = 0; k < 3; ++k) d[i][k] = w == 2 ? t2[i][k] : w == 3 ? t3[i][k] : t11[i][k];
}
// the vertex id of cube (x, y, z), or -1
__device__ __forceinline__ int64_t sr_vid(const SrDev& s, int x, int y, int z) {
  if (!s.g.in(x, y, z)) return -1;
  const int64_t c = s.g.idx(x, y, z);
  return s.vflag[c + 1] != s.vflag[c] ? (int64_t)s.vflag[c] : -1;
}

// The cubes around edge w (2, 3 or 11) of cube (x, y, z), as vertex ids; false where
// the edge has no crossing or a cube no vertex.
__device__ __forceinline__ bool sr_quad(const SrDev& s, int x, int y, int z, int ci, int w, int64_t id[4]) {
  if (!sr_edge_cross(ci, w)) return false;
  int d[4][3];
  sr_edge_cubes(w, d);
  bool ok = true;
  for (int q = 0; q < 4; ++q) {
    id[q] = sr_vid(s, x + d[q][0], y + d[q][1], z + d[q][2]);
    ok = ok && id[q] >= 0;
  }
  return ok;
}

// pass 0 counts the indices each crossing cube emits (into tcount, by vertex id, which
// follows the cube order), pass 1 writes them at the scanned offsets
__global__ void k_sr_tris(SrDev s, int64_t cells, int pass) {
  const int nv = (int)min((int64_t)s.vflag[cells], (int64_t)s.max_v);
  if (!pass && blockIdx.x == 0 && threadIdx.x == 0) { s.tcount[nv] = 0u; s.scan_n[2] = nv; }
  GRID_STRIDE(v, nv) {
    const int c = (int)s.cube_of[v];
    const int x = c % s.g.nx, y = (c / s.g.nx) % s.g.ny, z = c / (s.g.nx * s.g.ny);
    uint32_t cnt = 0;
    const int ci = sr_cube_mask(s, x, y, z);
    int64_t o = pass ? (int64_t)s.tcount[v] : 0;
    for (int k = 0; k < 3; ++k) {
      const int w = k == 0 ? 2 : k == 1 ? 3 : 11;
      int64_t id[4];
      if (!sr_quad(s, x, y, z, ci, w, id)) continue;
      cnt += 6;
      if (pass) {
        if (o + 6 > s.max_i) { sr_fail(s, NN_ERR_CAPACITY); continue; }
        const bool cond0 = (ci >> c_sr_edge[w][0]) & 1;
        const bool flip = cond0 != (w == 11);
        const int64_t t[6] = {id[2], id[1], id[0], id[3], id[2], id[0]};
        const int64_t tf[6] = {id[0], id[1], id[2], id[0], id[2], id[3]};
        for (int q = 0; q < 6; ++q) s.tri[o + q] = (int32_t)(flip ? tf[q] : t[q]);
        o += 6;
      }
    }
    if (!pass) s.tcount[v] = cnt;
  }
}

// All the indices of a mesh whose vertices overflow, for the error message: k_sr_tris has walked
// the cubes of the first max_v vertices only. result->ni is zero.
__global__ void k_sr_tris_total(SrDev s, int32_t cells) {
  uint32_t cnt = 0;
  FOR_CELLS(c, cells) {
    if (s.vflag[c + 1] == s.vflag[c]) continue;
    const int x = (int)c % s.g.nx, y = ((int)c / s.g.nx) % s.g.ny, z = (int)c / (s.g.nx * s.g.ny);
    const int ci = sr_cube_mask(s, x, y, z);
    int64_t id[4];
    for (int k = 0; k < 3; ++k) cnt += sr_quad(s, x, y, z, ci, k == 0 ? 2 : k == 1 ? 3 : 11, id) ? 6u : 0u;
  }
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(&s.result->ni, cnt);
}

// What the host reads back, in one copy.
__global__ void k_sr_result(SrDev s, int64_t cells, int marching_cubes) {
  const uint32_t nv = s.vflag[cells];
  *s.result = SrResult{nv, s.tcount[marching_cubes ? cells : min((int64_t)nv, (int64_t)s.max_v)], *s.status, 0,
                       s.stats[3]};
}

// ---- 6b. marching cubes (marching_cube_impl, srtool.py:1765-1800) ----------------------
// The reference's 256-case triangle table is not reproduced. This build's table is
// computed at compile time from the corner states of each case ("in": value <
// isolevel): faces list their corners counter-clockwise seen from outside; on a face,
// every run of in-corners gets one segment from the edge where the walk leaves the run
// to the edge where it entered it (in-corners stay separate on ambiguous faces, which
// depends on the face alone, so neighbouring cubes agree and the surface is closed);
// the segments chain into loops over the crossing edges; loops are taken in order of
// their smallest edge id, start there, and are fanned as (l0, l[k+1], l[k]).
#define SR_MC_MAXT 5
struct SrMcTable {
  uint16_t edges[256];               // crossing edges of each case
  uint8_t ntri[256];
  int8_t tri[256][SR_MC_MAXT][3];    // edge ids
  bool overflow;                     // a case needs more than SR_MC_MAXT triangles
};

constexpr int sr_mc_edge_of(const int8_t (&e)[12][2], int c0, int c1) {
  for (int w = 0; w < 12; ++w)
    if ((e[w][0] == c0 && e[w][1] == c1) || (e[w][0] == c1 && e[w][1] == c0)) return w;
  return -1;
}

constexpr SrMcTable sr_make_mc_table() {
  // the same corner offsets and edges as c_sr_off and c_sr_edge (srtool.py:775-783, 931-942)
  const int8_t off[8][3] = {{0, 1, 0}, {1, 1, 0}, {1, 0, 0}, {0, 0, 0}, {0, 1, 1}, {1, 1, 1}, {1, 0, 1}, {0, 0, 1}};
  const int8_t edge[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6}, {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};
  SrMcTable t{};
  for (int ci = 0; ci < 256; ++ci) {
    int next[12] = {-1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1};
    for (int a = 0; a < 3; ++a)
      for (int side = 0; side < 2; ++side) {
        const int u = (a + 1) % 3, v = (a + 2) % 3;
        int uv[4][2] = {{0, 0}, {1, 0}, {1, 1}, {0, 1}};  // counter-clockwise around +e_a
        if (side == 0) { uv[1][0] = 0; uv[1][1] = 1; uv[3][0] = 1; uv[3][1] = 0; }
        int q[4] = {0, 0, 0, 0};
        for (int k = 0; k < 4; ++k)
          for (int c = 0; c < 8; ++c)
            if (off[c][a] == side && off[c][u] == uv[k][0] && off[c][v] == uv[k][1]) q[k] = c;
        bool in[4] = {false, false, false, false};
        for (int k = 0; k < 4; ++k) in[k] = (ci >> q[k]) & 1;
        for (int k = 0; k < 4; ++k) {
          if (!in[k] || in[(k + 1) % 4]) continue;  // the walk leaves a run of in-corners at q[k]
          int j = k;
          while (in[(j + 3) % 4]) j = (j + 3) % 4;  // the run starts at q[j]
          next[sr_mc_edge_of(edge, q[k], q[(k + 1) % 4])] = sr_mc_edge_of(edge, q[(j + 3) % 4], q[j]);
        }
      }
    bool seen[12] = {false, false, false, false, false, false, false, false, false, false, false, false};
    int nt = 0;
    for (int e = 0; e < 12; ++e) {
      if (next[e] < 0) continue;
      t.edges[ci] = (uint16_t)(t.edges[ci] | (1u << e));
      if (seen[e]) continue;
      int loop[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
      int m = 0;
      for (int f = e; !seen[f]; f = next[f]) {
        seen[f] = true;
        loop[m++] = f;
      }
      for (int k = 1; k + 1 < m; ++k) {
        if (nt == SR_MC_MAXT) { t.overflow = true; break; }
        t.tri[ci][nt][0] = (int8_t)loop[0];
        t.tri[ci][nt][1] = (int8_t)loop[k + 1];
        t.tri[ci][nt][2] = (int8_t)loop[k];
        ++nt;
      }
    }
    t.ntri[ci] = (uint8_t)nt;
  }
  return t;
}
static_assert(!sr_make_mc_table().overflow, "a marching-cubes case needs more than SR_MC_MAXT triangles");
__constant__ SrMcTable c_sr_mc = sr_make_mc_table();

// pass 0: vertices (crossing edges) and indices per cube into vflag / tcount;
// pass 1: both written at the scanned offsets, in edge order within a cube
__global__ void k_sr_mc(SrDev s, int32_t cells, int pass) {
  if (!pass && blockIdx.x == 0 && threadIdx.x == 0) s.vflag[cells] = s.tcount[cells] = 0u;
  FOR_SR_ROWS(s, x, y, z, c, act) {
    (void)act;
    if (pass == 1 && s.vflag[c + 1] == s.vflag[c]) continue;
    // a cube with a crossing has a nonzero corner, which lies in an active block: the
    // reference's visit of the cubes around the active vertices reaches every such cube
    const int ci = sr_cube_mask(s, x, y, z);
    const uint32_t em = c_sr_mc.edges[ci];
    if (pass == 0) {
      s.vflag[c] = __popc(em);
      s.tcount[c] = 3u * c_sr_mc.ntri[ci];
      continue;
    }
    const int64_t vb = s.vflag[c], tb = s.tcount[c];
    const int nt = c_sr_mc.ntri[ci];
    if (vb + __popc(em) > s.max_v || tb + 3 * nt > s.max_i) { sr_fail(s, NN_ERR_CAPACITY); continue; }
    for (int w = 0; w < 12; ++w) {
      if (!((em >> w) & 1u)) continue;
      const int a = c_sr_edge[w][0], b = c_sr_edge[w][1];
      const int ax = x + c_sr_off[a][0], ay = y + c_sr_off[a][1], az = z + c_sr_off[a][2];
      const int bx = x + c_sr_off[b][0], by = y + c_sr_off[b][1], bz = z + c_sr_off[b][2];
      const double v1 = sr_get(s, s.field, ax, ay, az), v2 = sr_get(s, s.field, bx, by, bz);
      const double delta = v2 - v1;
      const double t = fabs(delta) < 1e-5 ? 0.5 : ((double)s.iso - v1) / delta;  // vertex_interpolate
      const double p1[3] = {ax * s.g.dvs + s.g.dox, ay * s.g.dvs + s.g.doy, az * s.g.dvs + s.g.doz};
      const double p2[3] = {bx * s.g.dvs + s.g.dox, by * s.g.dvs + s.g.doy, bz * s.g.dvs + s.g.doz};
      const int64_t v = vb + __popc(em & ((1u << w) - 1u));
      for (int k = 0; k < 3; ++k) s.vert[3 * v + k] = (float)(p1[k] + t * (p2[k] - p1[k]));
    }
    for (int q = 0; q < nt; ++q)
      for (int k = 0; k < 3; ++k) {
        const int w = c_sr_mc.tri[ci][q][k];
        s.tri[tb + 3 * q + k] = (int32_t)(vb + __popc(em & ((1u << w) - 1u)));
      }
  }
}

// ---- 7. vertex normals (process_normal) ----------------------------------------------
__global__ void k_sr_normals(SrDev s, int nv) {
  GRID_STRIDE(i, min(nv, s.max_v)) {
    const double p[3] = {s.vert[at3(i)], s.vert[at3(i) + 1], s.vert[at3(i) + 2]};
    double n[3];
    sr_normal_at(s, p, n);
    s.nrm[at3(i)] = (float)n[0]; s.nrm[at3(i) + 1] = (float)n[1]; s.nrm[at3(i) + 2] = (float)n[2];
  }
}

// ---- host side: context and C ABI -------------------------------------------------------
struct nn_sr_ctx {
  int dev_id = 0;
  int sms = 148;
  int32_t max_particles = 0, max_v = 0, max_i = 0;
  int64_t max_cells = 0, blocks = 0;
  int32_t* d_n = nullptr;  // scan sizes ([2] = last index of the current scan, set on the device)
  int32_t* status = nullptr;  // behind the four stats
  uint32_t *vcount = nullptr, *vkey = nullptr, *vrank = nullptr, *vflag = nullptr, *tcount = nullptr,
           *tile_sums = nullptr, *cube_of = nullptr;
  int32_t *vsrc = nullptr, *tri = nullptr;
  float4* spos = nullptr;
  unsigned long long* vfix = nullptr;  // [3][cells], with NN_SR_VELOCITY only
  float* mvel = nullptr;
  unsigned long long* fix = nullptr;
  float *splat = nullptr, *fa = nullptr, *fb = nullptr, *G = nullptr, *xbar = nullptr, *vert = nullptr, *nrm = nullptr;
  uint8_t* active = nullptr;
  double* stats = nullptr;
  SrResult *result = nullptr, *h_result = nullptr;  // h_result: pinned
  // last call
  SrDev last{};
  int64_t cells = 0;
  int32_t nv = 0, ni = 0, n = 0;
  double sd = 0.0;
  bool have = false;
  std::string err;
};

static int sr_fail_host(nn_sr_ctx* c, int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  if (c) c->err = buf;
  return code;
}
#define SRCK(call)                                                                                         \
  do {                                                                                                     \
    cudaError_t _e = (call);                                                                               \
    if (_e != cudaSuccess) return sr_fail_host(c, NN_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(_e));   \
  } while (0)

static void sr_free(nn_sr_ctx* c) {
  if (c->h_result) cudaFreeHost(c->h_result);
  void* bufs[] = {c->d_n, c->result, c->vcount, c->vkey, c->vrank, c->vflag, c->tcount, c->tile_sums, c->vsrc,
                  c->tri, c->fix, c->splat, c->fa, c->fb, c->G, c->xbar, c->vert, c->nrm, c->active, c->stats,
                  c->cube_of, c->spos, c->vfix, c->mvel};
  for (void* b : bufs) cudaFree(b);
}

// An exclusive scan in place with the neighbour search's scan kernels, of a[0 .. d_n[2]],
// at most len entries.
static int sr_scan(nn_sr_ctx* c, uint32_t* a, int64_t len, cudaStream_t st) {
  Dev d{};
  d.d_n = c->d_n;
  d.cell_count = a;
  d.tile_sums = c->tile_sums;
  const int tiles = (int)((len + SCAN_TILE - 1) / SCAN_TILE);
  k_scan_tiles<<<std::max(1, std::min(tiles, c->sms * 2)), SCAN_THREADS, 0, st>>>(d);
  k_scan_apply<<<std::max(1, std::min(tiles, c->sms * 2)), SCAN_THREADS, 0, st>>>(d);
  SRCK(cudaGetLastError());
  return NN_OK;
}

extern "C" {

// Vertices of a grid stay this far below 2^31 - 1 (indices are int32; the scans need no margin).
#define NN_SR_CELL_MARGIN 4096

int nn_sr_create(int32_t max_particles, int64_t max_cells, int32_t max_vertices, int32_t max_indices,
                 int32_t options, nn_sr_ctx** out) {
  if (!out) return NN_ERR_INVALID_ARG;
  *out = nullptr;
  if (max_particles <= 0 || max_cells <= 0 || max_cells >= (int64_t)INT32_MAX - NN_SR_CELL_MARGIN || max_vertices <= 0 ||
      max_indices <= 0 || (options & ~NN_SR_VELOCITY))
    return NN_ERR_INVALID_ARG;
  nn_sr_ctx* c = new nn_sr_ctx();
  cudaGetDevice(&c->dev_id);
  cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, c->dev_id);
  c->max_particles = max_particles;
  c->max_cells = max_cells;
  c->max_v = max_vertices;
  c->max_i = max_indices;
  const size_t N = (size_t)max_particles, CL = (size_t)max_cells + 1;
  const size_t blocks = (size_t)max_cells / 512 + 4096;  // block flags: checked against each grid's shape
  const size_t tiles = CL / SCAN_TILE + 2;
  cudaError_t e = cudaSuccess;
  auto al = [&](auto** p, size_t cnt) {
    if (e == cudaSuccess) e = cudaMalloc((void**)p, cnt * sizeof(**p));
  };
  al(&c->d_n, 4); al(&c->stats, 5); al(&c->result, 1);
  if (e == cudaSuccess) e = cudaMallocHost((void**)&c->h_result, sizeof(SrResult));
  c->status = reinterpret_cast<int32_t*>(c->stats + 4);
  al(&c->vcount, CL); al(&c->vflag, CL); al(&c->tcount, CL); al(&c->tile_sums, tiles);
  al(&c->vkey, N); al(&c->vrank, N); al(&c->vsrc, N); al(&c->spos, N); al(&c->G, 9 * N); al(&c->xbar, 3 * N);
  al(&c->fix, CL); al(&c->splat, CL); al(&c->fa, CL); al(&c->fb, CL); al(&c->active, blocks);
  al(&c->vert, 3 * (size_t)max_vertices); al(&c->nrm, 3 * (size_t)max_vertices); al(&c->tri, (size_t)max_indices);
  al(&c->cube_of, (size_t)max_vertices); al(&c->mvel, 3 * (size_t)max_vertices);
  if (options & NN_SR_VELOCITY) al(&c->vfix, 3 * CL);
  if (e != cudaSuccess) {
    sr_free(c);
    delete c;
    return NN_ERR_OOM;
  }
  c->blocks = (int64_t)blocks;
  *out = c;
  return NN_OK;
}

int nn_sr_destroy(nn_sr_ctx* c) {
  if (!c) return NN_ERR_INVALID_ARG;
  sr_free(c);
  delete c;
  return NN_OK;
}

const char* nn_sr_last_error(const nn_sr_ctx* c) { return c ? c->err.c_str() : "null context"; }

// The shared pipeline of SRTool.dual_contouring (srtool.py:1264-1304): binning, splats,
// smoothing, then dual contouring or marching cubes, normals and velocities.
static int sr_run(nn_sr_ctx* c, const nn_sr_params* p, const float* pos, const float* vel, int32_t n, void* stream,
                  bool marching_cubes) {
  if (!c) return NN_ERR_INVALID_ARG;
  const char* fn = marching_cubes ? "nn_sr_marching_cubes" : "nn_sr_dual_contouring";
  c->have = false;
  if (!p || p->size != (int32_t)sizeof(nn_sr_params) || (!pos && n > 0) || n < 0)
    return sr_fail_host(c, NN_ERR_INVALID_ARG, "%s: invalid argument", fn);
  if (n > c->max_particles)
    return sr_fail_host(c, NN_ERR_CAPACITY, "%d particles exceed the context's %d", n, c->max_particles);
  if (vel && !c->vfix)
    return sr_fail_host(c, NN_ERR_STATE, "velocities given to a context created without NN_SR_VELOCITY");
  if (!(p->voxel_size > 0) || !(p->smooth_radius > 0) || !(p->particle_radius > 0) || p->dims[0] <= 0 ||
      p->dims[1] <= 0 || p->dims[2] <= 0 || p->smooth_iterations < 0 || p->smooth_cells < 0)
    return sr_fail_host(c, NN_ERR_INVALID_ARG, "%s: bad parameters", fn);
  const int64_t cells = (int64_t)p->dims[0] * p->dims[1] * p->dims[2];
  const int bx = (p->dims[0] + NN_SR_BLOCK - 1) / NN_SR_BLOCK, by = (p->dims[1] + NN_SR_BLOCK - 1) / NN_SR_BLOCK,
            bz = (p->dims[2] + NN_SR_BLOCK - 1) / NN_SR_BLOCK;
  const int64_t blocks = (int64_t)bx * by * bz;
  if (cells > c->max_cells || blocks > c->blocks)
    return sr_fail_host(c, NN_ERR_CAPACITY, "grid of %lld vertices exceeds the context's %lld", (long long)cells,
                        (long long)c->max_cells);
  cudaStream_t st = (cudaStream_t)stream;
  SrDev s{};
  s.g.nx = p->dims[0]; s.g.ny = p->dims[1]; s.g.nz = p->dims[2];
  s.g.bx = bx; s.g.by = by; s.g.bz = bz;
  s.g.ox = (float)p->origin[0]; s.g.oy = (float)p->origin[1]; s.g.oz = (float)p->origin[2];
  s.g.vs = (float)p->voxel_size;
  s.g.dox = s.g.ox; s.g.doy = s.g.oy; s.g.doz = s.g.oz; s.g.dvs = s.g.vs;
  s.n = n; s.pos = pos; s.status = c->status;
  s.vcount = c->vcount; s.vkey = c->vkey; s.vrank = c->vrank; s.vsrc = c->vsrc; s.spos = c->spos;
  s.fix = c->fix; s.splat = c->splat; s.field = c->fa; s.tmp = c->fb; s.active = c->active;
  s.G = c->G; s.xbar = c->xbar; s.stats = c->stats; s.scan_n = c->d_n; s.result = c->result; s.vflag = c->vflag; s.tcount = c->tcount;
  s.vert = c->vert; s.tri = c->tri; s.nrm = c->nrm; s.max_v = c->max_v; s.max_i = c->max_i;
  s.cube_of = c->cube_of;
  s.vel = vel; s.vfix = c->vfix; s.mvel = c->mvel;
  s.iso = (float)p->isolevel;
  s.sr = (float)p->smooth_radius;
  const double r = p->particle_radius;
  s.volume = (float)(r * r * r * SR_PI * 4.0 / 3.0);  // srtool.py:920
  s.acoeff = (float)(315.0 / (64.0 * SR_PI));        // srtool.py:921
  s.range = (int)std::ceil(4.0 * (double)s.sr / (double)s.g.vs) + 1;  // srtool.py:1137
  s.off = s.range / 2;
  s.smooth_cells = p->smooth_cells;
  {  // the pre-pass's in-range test rn(sqrt(r2)) < 2 r_s  <=>  r2 < rr_thr
    const float rr = 2.f * s.sr;
    float t = rr * rr;
    while (std::sqrt(t) >= rr) t = std::nextafter(t, 0.f);
    while (std::sqrt(t) < rr) t = std::nextafter(t, INFINITY);
    s.rr_thr = t;
  }
  {  // exact branch tests without the square root: rn(sqrt(t)) <= 1 (0.5)  <=>  t <= q1_thr (q05_thr)
    float t = 1.f;
    while (std::sqrt(std::nextafter(t, INFINITY)) <= 1.f) t = std::nextafter(t, INFINITY);
    while (std::sqrt(t) > 1.f) t = std::nextafter(t, 0.f);
    s.q1_thr = t;
    t = 0.25f;
    while (std::sqrt(std::nextafter(t, INFINITY)) <= 0.5f) t = std::nextafter(t, INFINITY);
    while (std::sqrt(t) > 0.5f) t = std::nextafter(t, 0.f);
    s.q05_thr = t;
  }
  s.record_normals = p->record_normals;
  const int B = 256;
  const int grid_n = std::max(1, std::min((n + B - 1) / B, c->sms * 8));
  const int grid_c = (int)std::max<int64_t>(1, std::min<int64_t>((cells + B - 1) / B, (int64_t)c->sms * 16));
  const int grid_r = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)bx * s.g.ny * s.g.nz * 32 + B - 1) / B,
                                                                 (int64_t)c->sms * 16));  // rows, a warp each
  SRCK(cudaMemsetAsync(c->stats, 0, 5 * sizeof(double), st));  // and the status
  SRCK(cudaMemsetAsync(c->vcount, 0, (cells + 1) * sizeof(uint32_t), st));
  SRCK(cudaMemsetAsync(c->fix, 0, cells * sizeof(unsigned long long), st));
  if (vel) SRCK(cudaMemsetAsync(c->vfix, 0, 3 * cells * sizeof(unsigned long long), st));
  SRCK(cudaMemsetAsync(c->active, 0, blocks, st));
  if (!p->use_smooth_field) {  // else the pre-pass writes every particle's
    SRCK(cudaMemsetAsync(c->G, 0, 9 * (size_t)std::max(n, 1) * sizeof(float), st));
    SRCK(cudaMemsetAsync(c->xbar, 0, 3 * (size_t)std::max(n, 1) * sizeof(float), st));
  }
  if (n > 0) {
    // 1. binning
    k_sr_keys<<<grid_n, B, 0, st>>>(s, (int32_t)cells);
    RC(sr_scan(c, c->vcount, cells + 1, st));
    k_sr_scatter<<<grid_n, B, 0, st>>>(s);
    k_sr_voxel_sort<<<grid_c, B, 0, st>>>(s, cells);
    k_sr_sorted_pos<<<grid_n, B, 0, st>>>(s, cells);
    // 2. isotropic splat
    k_sr_iso<<<grid_n, B, 0, st>>>(s);
    if (p->use_smooth_field) {
      // 3-4. anisotropic kernels and splat (one warp per particle each)
      const int grid_w = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)n * 32 + B - 1) / B, c->sms * 16));
      const int ppw = sr_pre_ppw(n, c->sms), per = SR_PRE_WARPS * ppw;
      k_sr_aniso_pre<<<(n + per - 1) / per, SR_PRE_WARPS * 32, 0, st>>>(s, ppw);
      // several warps share a particle's columns in a small set, whose warps (one chain of
      // 20 column rounds each) would leave most of an SM's 24 slots empty: 71 -> 53 us on
      // 1,791 particles (2 warps 58, 8 58)
      const int parts = std::min(std::max((48 * c->sms + n / 2) / n, 1), 8);
      const int grid_s = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)n * parts * 32 + B - 1) / B, c->sms * 16));
      k_sr_aniso_splat<<<grid_s, B, 0, st>>>(s, parts);
      if (vel) k_sr_vel_splat<<<grid_w, B, 0, st>>>(s);
    }
  }
  k_sr_fix_to_field<<<grid_c, B, 0, st>>>(s, (int32_t)cells);
  // 5. smoothing (the first iteration's pass 0 ran with the conversion)
  for (int it = 0; it < p->smooth_iterations; ++it) {
    if (it > 0) {
      SRCK(cudaMemsetAsync(c->stats, 0, 4 * sizeof(double), st));
      k_sr_stats<<<grid_r, B, 0, st>>>(s, 0);
    }
    k_sr_stats<<<grid_r, B, 0, st>>>(s, 1);
    k_sr_sd<<<1, 32, 0, st>>>(s);
    if (p->smooth_cells == 1) k_sr_smooth<1><<<grid_r, B, 0, st>>>(s);
    else k_sr_smooth<0><<<grid_r, B, 0, st>>>(s);
    std::swap(s.field, s.tmp);
  }
  if (marching_cubes) {
    // 6b. marching cubes: count, scan, write
    k_sr_mc<<<grid_r, B, 0, st>>>(s, (int32_t)cells, 0);
    RC(sr_scan(c, c->vflag, cells + 1, st));
    RC(sr_scan(c, c->tcount, cells + 1, st));
    k_sr_mc<<<grid_r, B, 0, st>>>(s, (int32_t)cells, 1);
  } else {
    // 6. dual contouring
    const int64_t most = std::min<int64_t>(cells, s.max_v);  // vertices
    const int grid_v = (int)std::max<int64_t>(1, std::min<int64_t>((most + 127) / 128, (int64_t)c->sms * 16));
    k_sr_dc_flag<<<grid_r, B, 0, st>>>(s, (int32_t)cells);
    RC(sr_scan(c, c->vflag, cells + 1, st));
    k_sr_dc_list<<<grid_c, B, 0, st>>>(s, (int32_t)cells);
    k_sr_dc_point<<<grid_v, 128, 0, st>>>(s, cells);
    k_sr_tris<<<grid_v, 128, 0, st>>>(s, cells, 0);
    RC(sr_scan(c, c->tcount, most + 1, st));
    k_sr_tris<<<grid_v, 128, 0, st>>>(s, cells, 1);
  }
  k_sr_result<<<1, 1, 0, st>>>(s, cells, marching_cubes ? 1 : 0);
  SRCK(cudaGetLastError());
  SRCK(cudaMemcpyAsync(c->h_result, c->result, sizeof(SrResult), cudaMemcpyDeviceToHost, st));
  SRCK(cudaStreamSynchronize(st));
  if (!marching_cubes && c->h_result->nv > (uint32_t)c->max_v) {
    SRCK(cudaMemsetAsync(&c->result->ni, 0, sizeof(uint32_t), st));
    k_sr_tris_total<<<grid_c, B, 0, st>>>(s, (int32_t)cells);
    SRCK(cudaGetLastError());
    SRCK(cudaMemcpyAsync(c->h_result, c->result, sizeof(SrResult), cudaMemcpyDeviceToHost, st));
    SRCK(cudaStreamSynchronize(st));
  }
  int32_t status = c->h_result->status;
  c->nv = (int32_t)c->h_result->nv;
  c->ni = (int32_t)c->h_result->ni;
  c->sd = c->h_result->sd;
  if (status == 0 && (c->nv > c->max_v || c->ni > c->max_i)) status = NN_ERR_CAPACITY;
  if (status != 0) {
    if (status == NN_ERR_INVALID_ARG) return sr_fail_host(c, status, "a particle lies outside the grid");
    if (status == NN_ERR_NAN) return sr_fail_host(c, status, "non-finite splat contribution");
    return sr_fail_host(c, status, "grid, voxel list or mesh capacity exceeded (%d vertices, %d indices)", c->nv,
                        c->ni);
  }
  if (p->record_normals && c->nv > 0) {
    k_sr_normals<<<std::max(1, std::min((c->nv + B - 1) / B, c->sms * 8)), B, 0, st>>>(s, c->nv);
    SRCK(cudaGetLastError());
  }
  if (vel && c->nv > 0) {  // process_velocity (srtool.py:1298-1300); a zero field without the smooth splat
    k_sr_mesh_velocity<<<std::max(1, std::min((c->nv + B - 1) / B, c->sms * 8)), B, 0, st>>>(s, c->nv);
    SRCK(cudaGetLastError());
  }
  c->last = s;
  c->cells = cells;
  c->n = n;
  c->have = true;
  return NN_OK;
}

int nn_sr_dual_contouring(nn_sr_ctx* c, const nn_sr_params* p, const float* pos, const float* vel, int32_t n,
                          void* stream) {
  return sr_run(c, p, pos, vel, n, stream, false);
}

int nn_sr_marching_cubes(nn_sr_ctx* c, const nn_sr_params* p, const float* pos, const float* vel, int32_t n,
                         void* stream) {
  return sr_run(c, p, pos, vel, n, stream, true);
}

int nn_sr_get_mesh(nn_sr_ctx* c, int32_t* num_vertices, int32_t* num_indices, float* vertices, int32_t* indices,
                   float* normals, float* velocities, void* stream) {
  if (!c) return NN_ERR_INVALID_ARG;
  if (!c->have) return sr_fail_host(c, NN_ERR_STATE, "no mesh: run nn_sr_dual_contouring or nn_sr_marching_cubes first");
  cudaStream_t st = (cudaStream_t)stream;
  if (num_vertices) *num_vertices = c->nv;
  if (num_indices) *num_indices = c->ni;
  if (vertices && c->nv)
    SRCK(cudaMemcpyAsync(vertices, c->vert, 3 * (size_t)c->nv * sizeof(float), cudaMemcpyDeviceToDevice, st));
  if (indices && c->ni)
    SRCK(cudaMemcpyAsync(indices, c->tri, (size_t)c->ni * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
  if (normals && c->nv) {
    if (!c->last.record_normals) return sr_fail_host(c, NN_ERR_STATE, "normals were not recorded");
    SRCK(cudaMemcpyAsync(normals, c->nrm, 3 * (size_t)c->nv * sizeof(float), cudaMemcpyDeviceToDevice, st));
  }
  if (velocities && c->nv) {
    if (!c->last.vel) return sr_fail_host(c, NN_ERR_STATE, "velocities were not recorded");
    SRCK(cudaMemcpyAsync(velocities, c->mvel, 3 * (size_t)c->nv * sizeof(float), cudaMemcpyDeviceToDevice, st));
  }
  return NN_OK;
}

int nn_sr_get_stage(nn_sr_ctx* c, int32_t stage, float* field, uint8_t* active_blocks, float* G, float* xbar,
                    double* sd, void* stream) {
  if (!c) return NN_ERR_INVALID_ARG;
  if (!c->have) return sr_fail_host(c, NN_ERR_STATE, "no result: run nn_sr_dual_contouring first");
  if (stage != 0 && stage != 1) return sr_fail_host(c, NN_ERR_INVALID_ARG, "stage must be 0 or 1");
  cudaStream_t st = (cudaStream_t)stream;
  const SrDev& s = c->last;
  const int64_t blocks = (int64_t)s.g.bx * s.g.by * s.g.bz;
  if (field)
    SRCK(cudaMemcpyAsync(field, stage == 0 ? c->splat : s.field, c->cells * sizeof(float), cudaMemcpyDeviceToDevice, st));
  if (active_blocks) SRCK(cudaMemcpyAsync(active_blocks, c->active, blocks, cudaMemcpyDeviceToDevice, st));
  if (G && c->n) SRCK(cudaMemcpyAsync(G, c->G, 9 * (size_t)c->n * sizeof(float), cudaMemcpyDeviceToDevice, st));
  if (xbar && c->n)
    SRCK(cudaMemcpyAsync(xbar, c->xbar, 3 * (size_t)c->n * sizeof(float), cudaMemcpyDeviceToDevice, st));
  if (sd) *sd = c->sd;
  return NN_OK;
}

}  // extern "C"
