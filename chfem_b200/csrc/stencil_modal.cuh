// stencil_modal.cuh -- thermal / elastic 3D operator passes in the modes of the voxel element.
//
// The 8 nodal values of a voxel, written in the products of sums and differences along the
// three axes (the Hadamard basis of the trilinear element: û = H u, mode (a, b, c) the
// coefficient of y^a x^b z^c), almost diagonalise the element matrix of an isotropic material:
// of the 24 x 24 entries of M = H K H^T / 64 an elastic voxel keeps 21 diagonal entries and 12
// couplings, all functions of its Lame pair, and a thermal voxel 7 diagonal entries, all
// multiples of its conductivity.  So a voxel costs 8 additions per component and plane to
// transform, 21 to 54 to combine two planes, and as many back, and reads two material constants
// -- against 243 multiply-adds and 243 coefficients per elastic node in the form assembled by
// neighbour (stencil_asm.cuh), whose coefficient loads bound it.  f = K u = H^T M û is the same
// operator as the reference's 64 row blocks per node (chfem/src/femhmg/cudapcg/kernels/
// matrix_free.cu:191-323 thermal, :410-459 elastic) up to the order of summation; the rigid
// modes drop out exactly instead of cancelling.
//
// Orientation: x runs along +columns, y against the rows, z against the layers (the element
// matrices of femhmg_elastic_3D.c:37-120), so differences along rows and layers are taken from
// the smaller index to the larger one.
//
// B200 design: a CTA owns a 32 x 8 column of nodes and marches through a run of layers.  Thread p
// owns node p of the haloed plane (34 x 10) and the voxels of which it is the smallest corner: per
// layer it forms the node's input from loads issued a layer earlier, passes it on through shared
// memory, reads the other 3 corners, keeps the plane's modes in registers for the next layer,
// applies M, and writes the lower plane's 4 corner forces to shared memory; the upper plane's
// share stays in registers until the next layer completes it.  The finished rows are summed and
// stored word by word in storage order (ND interleaved components), each warp one contiguous run.
// One barrier per layer: in interval l the CTA stages and reads plane l, and stores the rows of
// layer l - 2.  Modes, outputs and finishers are those of k_te_apply (stencil_te.cuh) and, for a
// block of right-hand sides, k_blk_apply (stencil_block.cuh).
//
// What bounds it: instruction issue and the latency of a layer's chain, not memory (DRAM 15 to
// 45 %).  Registers decide the CTAs per SM: with the 4 forces and 4 modes per component of two
// planes live, FP64 elastic and FP32 pairs take 168 at one CTA per SM; capped at 80 for two they
// spill to local memory, which the 95 KB of shared memory leaves little L1 for (0.120 against
// 0.091 ms; a form that staged word by word at two CTAs per SM 0.176).
// Measured on one B200, PCG pass, against the pass it replaced: elastic 128^3 FP64 0.091 ms
// (0.216 assembled by neighbour), six FP32 cases 0.250 ms (0.337); thermal 256^3 FP64 0.195 ms
// (0.308 voxel by voxel with coefficients from a table), FP32 0.165 (0.181).
#pragma once
#include <type_traits>
#include "common.cuh"
#include "stencil_te.cuh"

namespace chfem {

// ---- table: inverse Jacobi diagonal by material counts, then the materials' constants -----
// count index n1 + 9 n2 + 81 n3 (n_m: voxels of material m among the node's 8); the materials'
// pairs (lambda, mu) / 16 (elastic) or (k / 16, -) (thermal) follow.
constexpr int MD_NCOUNT = 729;
constexpr int MD_MAT = MD_NCOUNT + 1;
constexpr int MD_WORDS = MD_MAT + 8;

__device__ __forceinline__ int md_count_index(unsigned key, bool two) {
  const unsigned lo = key & 0x5555u;
  if (two) return __popc(lo);  // materials 0 and 1 only
  const unsigned hi = (key >> 1) & 0x5555u;
  const int n3 = __popc(lo & hi);
  return (__popc(lo) - n3) + 9 * (__popc(hi) - n3) + 81 * n3;
}
// material of the voxel whose smallest corner is the node: the voxel in which it is local node 3
__device__ __forceinline__ unsigned md_material(unsigned key) { return (key >> 6) & 3u; }

// ---- one field value, or a pair of right-hand sides in one packed FP32 operand -------------
__device__ __forceinline__ double md_add(double a, double b) { return a + b; }
__device__ __forceinline__ double md_sub(double a, double b) { return a - b; }
__device__ __forceinline__ double md_mul(double s, double a) { return s * a; }
__device__ __forceinline__ double md_fma(double s, double a, double c) { return fma(s, a, c); }
__device__ __forceinline__ double md_neg(double a) { return -a; }
__device__ __forceinline__ float md_add(float a, float b) { return a + b; }
__device__ __forceinline__ float md_sub(float a, float b) { return a - b; }
__device__ __forceinline__ float md_mul(float s, float a) { return s * a; }
__device__ __forceinline__ float md_fma(float s, float a, float c) { return fmaf(s, a, c); }
__device__ __forceinline__ float md_neg(float a) { return -a; }
__device__ __forceinline__ float2 md_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 md_sub(float2 a, float2 b) { return __ffma2_rn(make_float2(-1.f, -1.f), b, a); }
__device__ __forceinline__ float2 md_mul(float s, float2 a) { return __fmul2_rn(make_float2(s, s), a); }
__device__ __forceinline__ float2 md_fma(float s, float2 a, float2 c) { return __ffma2_rn(make_float2(s, s), a, c); }
__device__ __forceinline__ float2 md_neg(float2 a) { return make_float2(-a.x, -a.y); }

template <typename V>
struct MdV {
  using T = V;
  static constexpr int W = 1;
};
template <>
struct MdV<float2> {
  using T = float;
  static constexpr int W = 2;
};
// element at a 32-bit byte offset from a (warp-uniform) base; n: the stride between right-hand sides
template <typename P>
__device__ __forceinline__ P* md_at(P* base, unsigned byte) {
  return reinterpret_cast<P*>(reinterpret_cast<uintptr_t>(base) + byte);
}
template <typename V>
__device__ __forceinline__ V md_ld(const typename MdV<V>::T* base, unsigned byte, long n) {
  if constexpr (MdV<V>::W == 2) return make_float2(*md_at(base, byte), *md_at(base + n, byte));
  else return *md_at(base, byte);
}
template <typename V>
__device__ __forceinline__ void md_st(typename MdV<V>::T* base, unsigned byte, long n, V v) {
  if constexpr (MdV<V>::W == 2) { *md_at(base, byte) = v.x; *md_at(base + n, byte) = v.y; }
  else *md_at(base, byte) = v;
}

// ---- the voxel ---------------------------------------------------------------------------
// In-plane modes of one component: 0 sum, 1 row difference, 2 column difference, 3 both.
template <typename V>
__device__ __forceinline__ void md_plane(V v00, V v10, V v01, V v11, V (&m)[4]) {  // v[row][column]
  const V p0 = md_add(v00, v10), m0 = md_sub(v00, v10), p1 = md_add(v01, v11), m1 = md_sub(v01, v11);
  m[0] = md_add(p0, p1);
  m[1] = md_add(m0, m1);
  m[2] = md_sub(p1, p0);
  m[3] = md_sub(m1, m0);
}
// transpose: nodal forces of a plane from its modes
template <typename V>
__device__ __forceinline__ void md_plane_t(const V (&m)[4], V& f00, V& f10, V& f01, V& f11) {
  const V t0 = md_add(m[0], m[1]), t1 = md_sub(m[0], m[1]), u0 = md_add(m[2], m[3]), u1 = md_sub(m[2], m[3]);
  f00 = md_sub(t0, u0);
  f10 = md_sub(t1, u1);
  f01 = md_add(t0, u0);
  f11 = md_add(t1, u1);
}

// Layer sums s and differences d (lower minus upper plane) of the in-plane modes; the sum of
// mode 0 is rigid and not formed.
template <typename V>
__device__ __forceinline__ void md_layers(const V (&o)[4], const V (&n)[4], V (&s)[4], V (&d)[4]) {
  d[0] = md_sub(o[0], n[0]);
#pragma unroll
  for (int m = 1; m < 4; m++) { s[m] = md_add(o[m], n[m]); d[m] = md_sub(o[m], n[m]); }
}
// Forces of a voxel's modes: on entry c holds the lower plane's forces from the voxel below; on
// exit a = the lower plane's complete forces and c the upper plane's.  lam, mu: the material's
// constants / 16 (thermal: lam = k / 16).
template <int ND, typename V, typename T>
__device__ __forceinline__ void md_voxel(const V (&s)[ND][4], const V (&d)[ND][4], T lam, T mu, V (&c)[ND][4], V (&a)[ND][4]) {
  auto fin = [&](int i, int m, V fs, V fd) {  // forces of the layer-sum and layer-difference modes
    a[i][m] = md_add(c[i][m], md_add(fs, fd));
    c[i][m] = md_sub(fs, fd);
  };
  auto fin0 = [&](int i, V fd) {
    a[i][0] = md_add(c[i][0], fd);
    c[i][0] = md_neg(fd);
  };
  if constexpr (ND == 1) {
    const T k1 = lam, k2 = lam * T(2.0 / 3.0), k3 = lam * T(1.0 / 3.0);
    fin0(0, md_mul(k1, d[0][0]));
    fin(0, 1, md_mul(k1, s[0][1]), md_mul(k2, d[0][1]));
    fin(0, 2, md_mul(k1, s[0][2]), md_mul(k2, d[0][2]));
    fin(0, 3, md_mul(k2, s[0][3]), md_mul(k3, d[0][3]));
  } else {
    // components 0 x (columns), 1 y (rows), 2 z (layers); modes 1 y, 2 x, 3 xy; d: times z
    const T mu2 = mu + mu, mu3 = mu * T(1.0 / 3.0), b1 = lam * T(1.0 / 3.0), b0 = b1 + mu, t9 = fma(T(4), mu, lam) * T(1.0 / 9.0);
    // shear pairs x010 y100, x001 z100, y001 z010: equal forces
    const V gxy = md_mul(mu, md_add(s[0][1], s[1][2]));
    const V gxz = md_mul(mu, md_add(d[0][0], s[2][2]));
    const V gyz = md_mul(mu, md_add(d[1][0], s[2][1]));
    fin0(0, gxz);
    fin0(1, gyz);
    // twist x011 y101 z110
    const V ws = md_mul(mu3, md_add(md_add(d[0][1], d[1][2]), s[2][3]));
    fin(0, 1, gxy, md_fma(mu3, d[0][1], ws));
    fin(1, 2, gxy, md_fma(mu3, d[1][2], ws));
    // normal strains x100, y010, z001
    const V tr = md_mul(lam, md_add(md_add(s[0][2], s[1][1]), d[2][0]));
    fin0(2, md_fma(mu2, d[2][0], tr));
    // pairs x101 y011, x110 z011, y110 z101; x111 y111 z111
    fin(0, 2, md_fma(mu2, s[0][2], tr), md_fma(b0, d[0][2], md_mul(b1, d[1][1])));
    fin(1, 1, md_fma(mu2, s[1][1], tr), md_fma(b0, d[1][1], md_mul(b1, d[0][2])));
    fin(0, 3, md_fma(b0, s[0][3], md_mul(b1, d[2][1])), md_mul(t9, d[0][3]));
    fin(2, 1, gyz, md_fma(b0, d[2][1], md_mul(b1, s[0][3])));
    fin(1, 3, md_fma(b0, s[1][3], md_mul(b1, d[2][2])), md_mul(t9, d[1][3]));
    fin(2, 2, gxz, md_fma(b0, d[2][2], md_mul(b1, s[1][3])));
    fin(2, 3, md_fma(mu3, s[2][3], ws), md_mul(t9, d[2][3]));
  }
}

// ---- the pass ------------------------------------------------------------------------------
template <int ND, typename T>
struct MdArgs {
  TeArgs<ND, T> te;  // the pass's fields; a block: those of its first right-hand side
  const T* tab;      // MD_WORDS
  long n;            // unknowns per right-hand side (the stride between them)
  int nr;            // right-hand sides (1: a single pass)
};

constexpr int MD_TC = 8;                       // columns of a tile
constexpr int MD_PR = TE_TR + 2;               // nodes of a haloed column
constexpr int MD_PP = MD_PR * (MD_TC + 2);     // nodes of a haloed plane: one thread each
constexpr int MD_NT = (MD_PP + 31) / 32 * 32;
constexpr int MD_TAB = (MD_WORDS + 3) / 4 * 4;
template <int ND>
struct MdGeom {
  static constexpr int CP = MD_PR * ND;           // words of a haloed column
  static constexpr int PPW = CP * (MD_TC + 2);    // words of a haloed plane
  static constexpr int CW = CP * (MD_TC + 1);     // words of one corner's forces
};
template <int ND, typename V>
inline size_t md_smem_bytes() {
  using G = MdGeom<ND>;
  return (size_t)MD_TAB * sizeof(typename MdV<V>::T) + ((size_t)4 * G::PPW + (size_t)8 * G::CW) * sizeof(V);
}

// How the work line of a pass -- (column tile, layer) units -- is cut for P CTAs: one run each
// where that costs fewer layers (a run restages 3), else equal slices of the line (TeWork).
struct MdWork {
  int R, C, L, tiles_r, tiles;
  int nc;  // one run per CTA: chunks of layers per tile; 0: slices
  int P, bid;
  __device__ MdWork(int R_, int C_, int L_, int P_, int bid_) : R(R_), C(C_), L(L_), nc(0), P(P_), bid(bid_) {
    tiles_r = (R + TE_TR - 1) / TE_TR;
    tiles = tiles_r * ((C + MD_TC - 1) / MD_TC);
    const int per = P / tiles;
    if (per >= 1) {
      const int n = min(L, per);
      if ((float)((L + n - 1) / n + 3) <= (float)tiles * (float)L / (float)P + 6.f) nc = n;
    }
  }
  __device__ TeWork slices() const {
    TeWork w(R, C, L, MD_TC);
    w.share(P);
    return w;
  }
  __device__ long begin() const { return nc ? 0 : (long)bid * ((long)tiles * L) / P; }
  __device__ long end() const { return nc ? (bid < nc * tiles ? 1 : 0) : ((long)bid + 1) * ((long)tiles * L) / P; }
  __device__ void run(long w, long w_end, int& r0, int& c0, int& l0, int& l1) const {
    if (!nc) { slices().run(w, w_end, r0, c0, l0, l1); return; }
    const int c = bid / tiles, t = bid - c * tiles;
    const int q = L / nc, rem = L - q * nc;  // the first rem chunks hold one layer more
    l0 = c * q + min(c, rem);
    l1 = l0 + q + (c < rem ? 1 : 0);
    r0 = (t % tiles_r) * TE_TR;
    c0 = (t / tiles_r) * MD_TC;
  }
  __device__ long step(int l0, int l1) const { return nc ? 1 : l1 - l0; }
};

// BLK: a block of ma.nr right-hand sides, W of them per CTA; the CTAs are dealt in equal shares
// to the groups of W with a right-hand side that still iterates.  DENS: a scalar density field
// (a.sdf, a.invd).
// Thread p stages node p of the haloed plane and owns the voxel whose smallest corner it is;
// warp w < 8 stores the tile's column w, 32 words at a time.
template <int ND, typename V, int MODE, int MINB, bool BLK, bool DENS>
__global__ void __launch_bounds__(MD_NT, MINB) k_modal_apply(MdArgs<ND, typename MdV<V>::T> ma) {
  using T = typename MdV<V>::T;
  using G = MdGeom<ND>;
  constexpr int W = MdV<V>::W, NT = MD_NT, CP = G::CP, PPW = G::PPW, CW = G::CW;
  constexpr bool TWO_IN = (MODE == TE_PCG || MODE == TE_DIRDOT || MODE == TE_MR);
  constexpr unsigned ES = sizeof(T), XS = 8 / ES;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double sred[NT / 32];
  const auto& a = ma.te;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const bool pre = a.cfg.precond != 0, two = a.nmat <= 2;
  T* sTab = reinterpret_cast<T*>(smem_raw);
  auto table = [&]() {  // filled while the scalar records are on their way
    const int counts = two ? 9 : MD_NCOUNT;  // the entries that the keys' counts can index, then the materials
    for (int i = tid; i < counts + 8; i += NT) {
      const int j = i < counts ? i : MD_MAT + i - counts;
      sTab[j] = (pre || j >= MD_MAT) ? ma.tab[j] : T(1);
    }
  };
  // the group of right-hand sides and this CTA's share of its work line
  int k0 = 0, P = gridDim.x, bid = blockIdx.x;
  bool idle = false;
  [[maybe_unused]] unsigned live = 1u;  // BLK: right-hand sides that still iterate
  if constexpr (BLK) {
    live = 0u;
    for (int k = 0; k < ma.nr; k++) live |= a.sc[k].done ? 0u : 1u << k;
    table();
    if (!live) return;
    int ng = 0;
    for (int g = 0; g < ma.nr / W; g++) ng += (live >> (g * W)) & ((1u << W) - 1u) ? 1 : 0;
    P = gridDim.x / ng;
    int ga = blockIdx.x / P;
    bid = blockIdx.x - ga * P;
    idle = ga >= ng;
    for (int g = 0; g < ma.nr / W; g++)
      if ((live >> (g * W)) & ((1u << W) - 1u)) { if (ga == 0) k0 = g * W; ga--; }
  } else {
    const int done = a.skip_if_done ? a.sc->done : 0;
    table();
    if (done) return;
  }
  V* sP = reinterpret_cast<V*>(sTab + MD_TAB);  // [4][PPW] formed input
  V* sC = sP + 4 * PPW;                         // [2][4][CW] corner forces
  const DevScalars* sc0 = a.sc + (BLK ? k0 : 0);
  V beta{}, alpha{};
  if constexpr (MODE == TE_PCG || MODE == TE_DIRDOT) {
    if constexpr (W == 2) beta = make_float2((float)sc0[0].beta, (float)sc0[1].beta);
    else beta = T(sc0->beta);
  }
  if constexpr (MODE == TE_MR) alpha = mr_steps(a.finish) ? T(sc0->alpha) : T(0);
  const double alpha64 = (MODE == TE_UPD) ? sc0->alpha : 0.0;
  const int R = a.R, C = a.C, L = a.L;
  const size_t RC = (size_t)R * C, RCL = RC * L;
  const long n = ma.n;
  const size_t kofs = BLK ? (size_t)k0 * n : 0;
  const T* const in0 = a.in0 + kofs;
  const T* const in1 = TWO_IN ? a.in1 + kofs : nullptr;
  T* const vout = MODE != TE_PLAIN ? a.vout + kofs : nullptr;
  T* const yout = MODE != TE_DIRDOT && MODE != TE_UPD ? a.y + kofs : nullptr;

  double acc[W], acc_rz = 0.0, mr = 0.0, md = 0.0, mx = 0.0;
#pragma unroll
  for (int u = 0; u < W; u++) acc[u] = 0.0;
  const int vr = tid % MD_PR, vc = tid / MD_PR;  // this thread's node of the plane
  const bool point = tid < MD_PP, voxel = vr < MD_PR - 1 && vc < MD_TC + 1;
  unsigned poff = 0, koff = 0;     // byte offsets in a layer: the thread's node (vectors, keys)
  unsigned ooff = 0, act = 0;      // output word lane of the warp's column; bit k: word 32 k + lane is stored
  [[maybe_unused]] bool mine = false;  // TE_MR: the node is one of the tile's own
  V g0[ND], g1[TWO_IN ? ND : 1];   // loads of the next plane
  unsigned gk = 0;

  auto load = [&](size_t lofs) {  // lofs: first node of the layer
    if (!point) return;
    const T* b0 = in0 + lofs * ND;
#pragma unroll
    for (int i = 0; i < ND; i++) g0[i] = md_ld<V>(b0, poff + i * ES, n);
    gk = *md_at(a.keys + lofs, koff);
    if constexpr (TWO_IN) {
      const T* b1 = in1 + lofs * ND;
#pragma unroll
      for (int i = 0; i < ND; i++) g1[i] = md_ld<V>(b1, poff + i * ES, n);
    }
  };

  V mo[ND][4], fc[ND][4];
  const MdWork wk(R, C, L, P, bid);
  __syncthreads();
  const long w_end = idle ? 0 : wk.end();
  for (long wu = idle ? 0 : wk.begin(); wu < w_end;) {
    int l0, l1, r0, c0;
    wk.run(wu, w_end, r0, c0, l0, l1);
    {
      const unsigned node = point ? (unsigned)(wrap(r0 + vr - 1, R) + wrap(c0 + vc - 1, C) * R) : 0u;
      poff = node * (ND * ES);
      koff = node * 2u;
      mine = point && vr >= 1 && vr <= TE_TR && r0 + vr - 1 < R && vc >= 1 && vc <= MD_TC && c0 + vc - 1 < C;
      act = 0;
      if (w < MD_TC && c0 + w < C) {
        ooff = ((unsigned)((c0 + w) * R + r0) * ND + lane) * ES;
#pragma unroll
        for (int k = 0; k < ND; k++) act |= r0 * ND + 32 * k + lane < R * ND ? 1u << k : 0u;
      }
    }
    __syncthreads();  // the previous run's reads of the planes are done
    // first nodes of layers l - 2, l - 1, l, l + 1
    size_t om2 = 0, om1 = 0, o0 = (size_t)(l0 > 0 ? l0 - 1 : L - 1) * RC, op1 = (size_t)l0 * RC;
    unsigned vmat = 0;
    [[maybe_unused]] T vscl = T(1);
    load(o0);
    for (int l = l0 - 1; l <= l1 + 1; l++) {
      V v[ND];
      unsigned vnext = 0;
      [[maybe_unused]] T vsnext = T(1);
      if (l <= l1) {  // plane l, loaded during the previous interval, formed into its ring slot
        T inv = T(1);
        if constexpr (TWO_IN && !DENS) inv = sTab[md_count_index(gk, two)];
        vnext = md_material(gk);
#pragma unroll
        for (int i = 0; i < ND; i++) {
          v[i] = g0[i];
          if constexpr (TWO_IN) {
            if constexpr (DENS) inv = pre && point ? T(*md_at(a.invd + o0 * ND, (poff + i * ES) * XS)) : T(1);
            if constexpr (MODE == TE_MR) {
              const V rn = md_fma(-alpha, g1[i], v[i]);
              v[i] = md_mul(inv, rn);
              if (mine && l >= l0 && l < l1) {
                *md_at(vout + o0 * ND, poff + i * ES) = rn;
                const T dv = *md_at(a.d + o0 * ND, poff + i * ES);
                double* xp = md_at(a.x + o0 * ND, (poff + i * ES) * XS);
                const double xn = fma((double)alpha, (double)dv, *xp);
                *xp = xn;
                acc_rz += (double)rn * (double)v[i];
                mr = fmax(mr, fabs((double)rn));
                md = fmax(md, fabs((double)dv));
                mx = fmax(mx, fabs(xn));
              }
            } else if constexpr (W == 2) {
              v[i] = __ffma2_rn(beta, g1[i], md_mul(inv, v[i]));
            } else {
              v[i] = fma(beta, g1[i], v[i] * inv);
            }
          }
          if (point) sP[(l & 3) * PPW + tid * ND + i] = v[i];
        }
        if constexpr (DENS) {
          if (point) vsnext = T(a.sdf_min + a.sdf_rng * (double)*md_at(a.sdf + o0, koff) * (1.0 / 65535.0));
        }
        if (l < l1) load(op1);
      }
      __syncthreads();
      if (l <= l1 && voxel) {
        const V* pl = sP + (l & 3) * PPW + tid * ND;
        if (l >= l0) {
          const T* mat = sTab + MD_MAT + 2 * vmat;
          T lam = mat[0], mu = mat[1];
          if constexpr (DENS) { lam *= vscl; mu *= vscl; }
          V ms[ND][4], mdif[ND][4], fa[ND][4];
#pragma unroll
          for (int i = 0; i < ND; i++) {
            V nm[4];
            md_plane<V>(v[i], pl[ND + i], pl[CP + i], pl[CP + ND + i], nm);
            md_layers<V>(mo[i], nm, ms[i], mdif[i]);
#pragma unroll
            for (int m = 0; m < 4; m++) mo[i][m] = nm[m];
          }
          md_voxel<ND, V, T>(ms, mdif, lam, mu, fc, fa);
          if (l > l0) {
            V* f = sC + (l & 1) * 4 * CW + tid * ND;
#pragma unroll
            for (int i = 0; i < ND; i++) {
              V f00, f10, f01, f11;
              md_plane_t<V>(fa[i], f00, f10, f01, f11);
              f[i] = f00;
              f[CW + i] = f10;
              f[2 * CW + i] = f01;
              f[3 * CW + i] = f11;
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < ND; i++) {
            md_plane<V>(v[i], pl[ND + i], pl[CP + i], pl[CP + ND + i], mo[i]);
#pragma unroll
            for (int m = 0; m < 4; m++) fc[i][m] = V{};
          }
        }
      }
      vmat = vnext;
      vscl = vsnext;
      if (l - 2 >= l0 && act) {  // rows of layer l - 2: the 4 voxel columns' forces
        const V* f = sC + ((l - 1) & 1) * 4 * CW + w * CP + lane;
        const V* pv = sP + ((l - 2) & 3) * PPW + (w + 1) * CP + ND + lane;
#pragma unroll
        for (int k = 0; k < ND; k++) {
          if (!((act >> k) & 1u)) continue;
          const unsigned ob = ooff + 32 * k * ES;
          const V q = md_add(md_add(f[CP + ND + 32 * k], f[CW + CP + 32 * k]), md_add(f[2 * CW + ND + 32 * k], f[3 * CW + 32 * k]));
          const V vv = pv[32 * k];
          if constexpr (MODE != TE_DIRDOT && MODE != TE_UPD) md_st<V>(yout + om2 * ND, ob, n, q);
          if constexpr (MODE == TE_PCG || MODE == TE_DIRDOT) md_st<V>(vout + om2 * ND, ob, n, vv);
          if constexpr (MODE == TE_UPD) {
            T inv = T(1);
            if (pre) {
              if constexpr (DENS) inv = T(*md_at(a.invd + om2 * ND, ob * XS));
              else inv = sTab[md_count_index(*md_at(a.keys + om2, ob / (ES * ND) * 2u), two)];
            }
            T* rp = md_at(vout + om2 * ND, ob);
            const T rn = fma(-T(alpha64), q, *rp);
            *rp = rn;
            double* xp = md_at(a.x + om2 * ND, ob * XS);
            const double xn = fma(alpha64, (double)vv, *xp);
            *xp = xn;
            acc_rz += (double)rn * (double)(rn * inv);
            mr = fmax(mr, fabs((double)rn));
            md = fmax(md, fabs((double)vv));
            mx = fmax(mx, fabs(xn));
          }
          if constexpr (W == 2) {
            acc[0] += (double)vv.x * (double)q.x;
            acc[1] += (double)vv.y * (double)q.y;
          } else {
            acc[0] += (double)vv * (double)q;
          }
        }
      }
      om2 = om1; om1 = o0; o0 = op1;
      op1 += RC;
      if (op1 >= RCL) op1 = 0;
    }
    wu += wk.step(l0, l1);
  }
  if constexpr (BLK) {
    // partial sums of this CTA's right-hand sides; the last CTA sums each live right-hand side
    // over its group's CTAs in order
    __shared__ unsigned s_last;
#pragma unroll
    for (int u = 0; u < W; u++) {
      const double t = block_sum<NT>(acc[u], sred);
      if (tid == 0 && !idle) a.rc.part[(k0 + u) * a.rc.nblocks + bid] = t;
    }
    if (tid == 0) {
      __threadfence();
      s_last = atomicAdd(a.rc.ticket, 1u) == (unsigned)a.rc.nblocks - 1u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int k = 0; k < ma.nr; k++) {
      if (!((live >> k) & 1u)) continue;
      double t = 0.0;
      for (int b = tid; b < P; b += NT) t += __ldcg(a.rc.part + k * a.rc.nblocks + b);
      t = block_sum<NT>(t, sred);
      if (tid == 0) { a.sc[k].red[0] = t; a.sc[k].alpha = a.sc[k].delta / t; }
    }
    if (tid == 0) *a.rc.ticket = 0u;
  } else {
    if (a.finish == FIN_NONE) return;
    if constexpr (MODE == TE_UPD) {
      const double vals[4] = {acc_rz, mr, md, mx};
      const bool ismax[4] = {false, true, true, true};
      double out[4];
      if (grid_reduce<NT, 4>(vals, ismax, a.rc, bid, out, sred) && tid == 0) {
        for (int k = 0; k < 4; k++) a.sc->red[k] = out[k];
        const SolveCfg cfg{a.cfg.tol, a.cfg.maxit, a.cfg.norm, a.cfg.precond, a.cfg.nhmg};
        pcg_finish(PW_PCG, out, a.sc, cfg);
      }
    } else if constexpr (MODE == TE_MR) {
      const double vals[5] = {acc[0], acc_rz, mr, md, mx};
      const bool ismax[5] = {false, false, true, true, true};
      double out[5];
      if (grid_reduce<NT, 5>(vals, ismax, a.rc, bid, out, sred) && tid == 0) {
        for (int k = 0; k < 5; k++) a.sc->red[k] = out[k];
        mr_finish(a.finish, out, a.sc, a.cfg);
      }
    } else {
      const double vals[1] = {acc[0]};
      const bool ismax[1] = {false};
      double out[1];
      if (grid_reduce<NT, 1>(vals, ismax, a.rc, bid, out, sred) && tid == 0) {
        a.sc->red[0] = out[0];
        if (a.finish == FIN_ALPHA) a.sc->alpha = a.sc->delta / out[0];
      }
    }
  }
}

}  // namespace chfem
