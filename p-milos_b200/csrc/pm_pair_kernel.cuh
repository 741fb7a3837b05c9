// pm_pair_kernel.cuh -- the FP32 inversion kernel of normal Zeeman triplets on grids
// of up to 32 wavelengths: a warp inverts two pixels at a time.  Streamed like the
// one-pixel kernel of pm_stream_kernel.cuh (ticket queue, job ring), and per pixel
// the arithmetic and its order are that kernel's.  Everything here has internal
// linkage.
//
// What bounds this path is instruction issue, and the issue rate is bound by the
// instruction cache: straight-line code, 16 warps at different places, runs at 0.96
// instructions per cycle and scheduler up to 32 KB, at 0.87 at 36 KB, 0.6 at 40-48 KB
// and 0.38 from 80 KB on.  So the LM loop is written for few instructions and little
// code: the response functions, the correlation and the factorisation are rolled
// loops, the sums of the normal equations go through shared memory, and branches that
// the warp takes as one are marked so (uniform).
#pragma once
#include "pm_stream_kernel.cuh"

namespace {

static_assert(kRow == kLaneStatePad, "the response functions overwrite the synthesis states row by row");

// Per block: the PSF taps, centred and reversed, so that the window of a group of
// inputs is read with aligned 16-byte broadcast loads; the shared stray-light
// profile; 1 / sigma^2; the parameters' bounds.
struct alignas(16) PairBlock {
  // rv[0][u] = G[31 - u + half] (0 outside [0, nl)): the tap of input m and output k
  // is rv[0][31 - m + k]; rv[1][u] = rv[0][u + 1], for aligned pairs at odd offsets
  float rv[2][2 * NL + 4];
  float taps[NL];          // G[j], zero for j >= nl
  float sl[4 * NL];        // [4][nl] (PM_SLIGHT_SHARED)
  float isig[2];           // of a sample, of a ghost sample
  float pad_[2];
  double lo[11], hi[11];
};

// A warp's buffers.  tr: response functions [profile][lambda] (transpose buffer,
// and scratch of the solvers and of the reductions); ls: the synthesis state that
// the response functions are formed from, per lane; xs: padded Stokes rows of the
// synthesis correlation.  The response functions overwrite the states (every lane
// has its own in registers by then); the macroturbulence kernel is formed in xs, so
// that its instances share the rows too (16 warps per SM fit where 12 did: 16,384
// pixels, 11 parameters: 7.63 -> 7.12 ms).
struct alignas(16) RowsSmem {
  static constexpr bool kSharedRows = true;
  union {
    float tr[NL * kRow];
    float ls[NL][kLaneStatePad];
  };
  float xs[4][XSR];
  int xs_dirty;  // xs holds macroturbulence data: restore its zero padding before psf_rows
  int grid_cur;  // the grid whose padding xs has
  int pad_[2];
};

// Bounds of check for the parameters it only clamps (the field's sign and the
// angles are folded first).
__constant__ double kModelMin[11] = {1, 0, -20, 0.0001, 0.0001, 0, 0, 0.0001, 0.0001, 0, 0};
__constant__ double kModelMax[11] = {2500, 5000, 20, 0.6, 10, 180, 180, 2, 2, 4, 1};

// The stray-light profile a pixel mixes in: the block's copy of the shared one,
// the pixel's own row of a per-pixel cube, or none.
__device__ __forceinline__ const float* pair_slight(const PmParams& P, const PairBlock& bs, const float* cube,
                                                    size_t base) {
  if (P.slight_mode == PM_SLIGHT_SHARED) return bs.sl;
  if (P.slight_mode == PM_SLIGHT_PER_PIXEL && cube) return cube + base;
  return nullptr;
}

__device__ __forceinline__ void pair_block(const PmParams& P, PairBlock& bs) {
  for (int e = threadIdx.x; e < 2 * (2 * NL + 4); e += blockDim.x) {
    const int odd = e / (2 * NL + 4), u = e % (2 * NL + 4);
    const int j = 31 - (u + odd) + P.half;
    bs.rv[odd][u] = (j >= 0 && j < P.nl) ? P.taps_f[j] : 0.0f;
  }
  if (threadIdx.x < NL) bs.taps[threadIdx.x] = P.taps_f[threadIdx.x];
  if (threadIdx.x < 2) bs.isig[threadIdx.x] = float(1.0 / (threadIdx.x ? kGhostSigma : P.noise));
  if (threadIdx.x < 11) {
    bs.lo[threadIdx.x] = kModelMin[threadIdx.x];
    bs.hi[threadIdx.x] = kModelMax[threadIdx.x];
  }
  if (P.slight_mode == PM_SLIGHT_SHARED)
    for (int e = threadIdx.x; e < 4 * NL; e += blockDim.x) bs.sl[e] = e < 4 * P.nl ? P.sl_f[e] : 0.0f;
}

// The per-model terms (model_terms) from the sines and cosines of the inclination (s0, c0) and of twice
// the azimuth (s1, c1).
__device__ __forceinline__ void terms_from(const PmParams& P, const double* m, float s0, float c0, float s1, float c1,
                                           ModelTerms<float>& T) {
  T.E0 = m[0] * P.fo;
  T.B0 = m[7];
  T.B1 = -(m[8] * P.mu);
  T.ALF = m[10];
  T.alf = float(m[10]);
  T.oma = float(1.0 - m[10]);
  T.A = float(m[4]);
  T.sin_gm = s0;
  T.cosi = c0;
  T.sina = s1;
  T.cosa = c1;
  T.sinis = T.sin_gm * T.sin_gm;
  T.cosis = T.cosi * T.cosi;
  T.cosis_2 = (1.0f + T.cosis) / 2.0f;
  const float CCr = float(kPi / 180.0), CC2 = CCr * 2.0f;
  T.sinda = T.cosa * CC2;
  T.cosda = -T.sina * CC2;
  T.sindi = T.cosi * T.sin_gm * CC2;
  T.cosdi = -T.sin_gm * CCr;
  T.sinis_cosa = T.sinis * T.cosa;
  T.sinis_sina = T.sinis * T.sina;
  const float LD = float(m[3]), E0 = float(T.E0), l0 = float(P.lambda0);
  T.E0_2 = E0 / 2.0f;
  T.cosi_E0_2 = T.E0_2 * T.cosi;
  T.invLD = __frcp_rn(LD);
  T.invE0 = __frcp_rn(E0);
  T.ulos = (float(m[2]) * l0) * T.invLD * float(1.0 / kVLight);
  const float parcial = (l0 * l0) * T.invLD * float(kZeeman);
#pragma unroll
  for (int g = 0; g < 3; ++g) {
    T.zs[g] = parcial * float(P.nu[g][0]);
    T.zsB[g] = T.zs[g] * float(m[1]);
  }
  T.auxCte = (-l0) * T.invLD * float(1.0 / kVLight);
  T.sc = E0 * T.sinis_cosa / 2.0f;
  T.ss = E0 * T.sinis_sina / 2.0f;
  T.cosi_2_E0 = E0 * T.cosi / 2.0f;
}

// voigt<float> with its roundings spelled out (which product of a sum of two is
// rounded on its own is the compiler's choice there, and depends on the code
// around it): the same bits wherever it is inlined.
__device__ __forceinline__ void pair_voigt(float a, float v, float& h, float& f) {
  float nr = fmaf(float(kP[6]), a, float(kP[5]));
  float ni = float(kP[6]) * -v;
#pragma unroll
  for (int j = 4; j >= 0; --j) {
    const float tr = __fadd_rn(fmaf(nr, a, __fmul_rn(ni, v)), float(kP[j]));
    ni = fmaf(ni, a, -__fmul_rn(nr, v));
    nr = tr;
  }
  float dr = __fadd_rn(a, float(kQ[6]));
  float di = -v;
  {
    const float tr = __fadd_rn(fmaf(-v, v, __fmul_rn(dr, a)), float(kQ[5]));
    di = fmaf(-v, a, -__fmul_rn(dr, v));
    dr = tr;
  }
#pragma unroll
  for (int j = 4; j >= 0; --j) {
    const float tr = __fadd_rn(fmaf(dr, a, __fmul_rn(di, v)), float(kQ[j]));
    di = fmaf(di, a, -__fmul_rn(dr, v));
    dr = tr;
  }
  // Smith's division
  const bool c = fabsf(dr) >= fabsf(di);
  const float big = c ? dr : di, small = c ? di : dr;
  const float x1 = c ? nr : ni, x2 = c ? ni : nr;
  const float r = __fdividef(small, big);
  const float inv = __frcp_rn(fmaf(small, r, big));
  h = __fmul_rn(fmaf(x2, r, x1), inv);
  const float w = fmaf(-x1, r, x2);
  f = __fmul_rn(c ? w : -w, inv) * 0.5f;
}

// synth_lane of a triplet: the three groups go through one copy of the Voigt
// function's code (unrolled: 7.2 KB with what follows).  ls: this lane's LaneState.
__device__ __forceinline__ void pair_synth(const PmParams& P, const ModelTerms<float>& T, double dl, float* ls,
                                           float (&S)[4]) {
  LaneState<float> s;
  const float u = float(dl) * T.invLD - T.ulos;
#pragma unroll 1
  for (int g = 0; g < 3; ++g) {
    const float uu = u - (g == 0 ? T.zsB[0] : g == 1 ? T.zsB[1] : T.zsB[2]);
    float H, F;
    pair_voigt(T.A, uu, H, F);
    const float we = float(P.we[g][0]);
    ls[g] = we * H;
    ls[3 + g] = we * F * 2.0f;
    ls[6 + g] = uu;
    ls[9 + g] = H;
    ls[12 + g] = F;
  }
  static_assert(offsetof(LaneState<float>, shi) == 12 && offsetof(LaneState<float>, parcial1) == 60, "LaneState layout");
  copy16(s, *reinterpret_cast<const LaneState<float>*>(ls));
  propagate<float>(T, s, S);
  copy16(*reinterpret_cast<LaneState<float>*>(ls), s);
}

// psf_rows in a loop over the taps, eight at a time (unrolled with the taps as
// constant operands: 2.5 KB of code more for 30 instructions less); the outputs go
// where the inputs were.
template <typename SM>
__device__ __forceinline__ void pair_psf(const PmParams& P, const PairBlock& bs, SM& sm, int lane, bool valid,
                                         float S[4]) {
  const float i0 = __shfl_sync(kFull, S[0], 0), in = __shfl_sync(kFull, S[0], P.nl - 1);
  const float ic = (i0 > in) ? i0 : in;
  const int off = NL + (P.half & 3);  // data at xs[s][off + i]; off - half is a multiple of 4
#pragma unroll
  for (int s = 0; s < 4; ++s) sm.xs[s][off + lane] = valid ? (s == 0 ? ic - S[0] : S[s]) : 0.0f;
  __syncwarp();
  const int st = lane >> 3, c = lane & 7;
  const float4* w0 = reinterpret_cast<const float4*>(&sm.xs[st][off + 4 * c - P.half]);
  float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  float4 cur = w0[0];
#pragma unroll 2
  for (int q = 0; q < NL / 4; ++q) {
    const float4 nxt = w0[q + 1];
    const float4 g4 = reinterpret_cast<const float4*>(bs.taps)[q];
    const float w[8] = {cur.x, cur.y, cur.z, cur.w, nxt.x, nxt.y, nxt.z, nxt.w};
    const float g[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) acc[kk] = fmaf(g[j], w[kk + j], acc[kk]);
    cur = nxt;
  }
  __syncwarp();  // every window is read
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) sm.xs[st][off + 4 * c + kk] = (st == 0) ? ic - acc[kk] : acc[kk];
  __syncwarp();
#pragma unroll
  for (int s = 0; s < 4; ++s) S[s] = valid ? sm.xs[s][off + lane] : 0.0f;
  __syncwarp();
}

// Response functions at this thread's wavelength (me_der.c:85-312), profile p
// stored at col[p * kRow]: p = r*4 + s for rows r = 0..6 (eta0, B, vlos, dopp,
// a, gamma, azimuth) and r = 7 holding RF row 8 (S1).  Row 7 of the reference
// (S0: I = 1, Q = U = V = 0) is not convolved and is added in registers later.
// The seven rows go through one copy of the code (unrolled: 12.5 KB).  What lanes
// beyond the grid store is not read.
__device__ __forceinline__ void rf_rows(const PmParams& P, const ModelTerms<float>& T, const LaneState<float>& st,
                                        float* col) {
  float dHu[3], dFu[3], uun[3];  // of each group: dH/du and dF/du times the strength, du/d(Doppler width)
#pragma unroll
  for (int g = 0; g < 3; ++g) {
    const float we = float(P.we[g][0]);
    const float uu = st.uu[g], H = st.H[g], F = st.F[g];
    dHu[g] = ((4.0f * T.A * F) - (2.0f * uu * H)) * we;
    dFu[g] = (float(kRsqrtPi) - T.A * H - 2.0f * uu * F) * we;
    uun[g] = -uu * T.invLD;
  }
  const float E0_2 = T.E0_2;
  const float dtaux = float(T.B1) / (st.dt * st.dt);
  const float etai = st.etai, etai_2 = st.etai_2, etaq = st.etaq, etau = st.etau, etav = st.etav;
  const float rhoq = st.rhoq, rhou = st.rhou, rhov = st.rhov;
  const float etai_gp3 = etai * st.gp3;
  const float a2 = 2.0f * etai;
  const float ext1 = a2 * etaq + etav * rhou - etau * rhov;
  const float ext2 = a2 * etau + etaq * rhov - etav * rhoq;
  const float ext3 = a2 * etav + etau * rhoq - etaq * rhou;
  const float ext4 = a2 * st.gp1;
#pragma unroll 1
  for (int il = 0; il < 7; ++il) {
    float de, dq, du, dv, rq, ru, rv;
    if (il == 0) {
      const float invE0 = T.invE0;
      de = st.etain * invE0; dq = st.etaq * invE0; du = st.etau * invE0; dv = st.etav * invE0;
      rq = st.rhoq * invE0; ru = st.rhou * invE0; rv = st.rhov * invE0;
    } else if (il < 5) {
      // B, vlos, Doppler width: dH/du and dF/du times du/dp; the damping: -2 dF/du and dH/du / 2
      float dfi[3], dshi[3];
#pragma unroll
      for (int g = 0; g < 3; ++g) {
        const float c = il == 1 ? -T.zs[g] : il == 2 ? T.auxCte : uun[g];
        dfi[g] = il == 4 ? -2.0f * dFu[g] : dHu[g] * c;
        dshi[g] = il == 4 ? dHu[g] / 2.0f : dFu[g] * c;
      }
      const float dfisum = dfi[1] + dfi[2];
      const float aux = dfi[0] - dfisum / 2.0f;
      de = dfi[0] * (T.sinis * E0_2) + dfisum * (T.cosis_2 * E0_2);
      dq = aux * T.sc;
      du = aux * T.ss;
      dv = (dfi[2] - dfi[1]) * T.cosi_2_E0;
      const float auxr = dshi[0] - (dshi[1] + dshi[2]) / 2.0f;
      rq = auxr * T.sc;
      ru = auxr * T.ss;
      rv = (dshi[2] - dshi[1]) * T.cosi_2_E0;
    } else if (il == 5) {
      const float cosdi_E0_2 = E0_2 * T.cosdi;
      de = st.fi[0] * (T.sindi * E0_2) + st.parcial1 * (T.cosi * T.cosdi * E0_2);
      dq = st.parcial2 * (T.sindi * T.cosa);
      du = st.parcial2 * (T.sindi * T.sina);
      dv = (st.fi[2] - st.fi[1]) * cosdi_E0_2;
      rq = st.parcial3 * (T.sindi * T.cosa);
      ru = st.parcial3 * (T.sindi * T.sina);
      rv = (st.shi[2] - st.shi[1]) * cosdi_E0_2;
    } else {
      de = 0; dv = 0; rv = 0;
      dq = st.parcial2 * (T.sinis * T.cosda);
      du = st.parcial2 * (T.sinis * T.sinda);
      rq = st.parcial3 * (T.sinis * T.cosda);
      ru = st.parcial3 * (T.sinis * T.sinda);
    }
    const float dgp1 = 2.0f * (etai * de - etaq * dq - etau * du - etav * dv + rhoq * rq + rhou * ru + rhov * rv);
    const float dgp2 = rhoq * dq + etaq * rq + rhou * du + etau * ru + rhov * dv + etav * rv;
    const float d_dt = ext4 * de + etai_2 * dgp1 - 2.0f * st.gp2 * dgp2;
    const float dgp3 = 2.0f * (etai * de + rhoq * rq + rhou * ru + rhov * rv);
    float dI = -(((de * st.gp3 + etai * dgp3) * st.dt - d_dt * etai_gp3) * dtaux);
    const float dgp4 = de * ext1 + etai_2 * dq + etai * (rhou * dv + etav * ru - rhov * du - etau * rv);
    const float dQ = ((dgp4 + rq * st.gp2 + rhoq * dgp2) * st.dt - d_dt * st.g4) * dtaux;
    const float dgp5 = de * ext2 + etai_2 * du + etai * (rhov * dq + etaq * rv - rhoq * dv - etav * rq);
    const float dU = ((dgp5 + ru * st.gp2 + rhou * dgp2) * st.dt - d_dt * st.g5) * dtaux;
    const float dgp6 = de * ext3 + etai_2 * dv + etai * (rhoq * du + etau * rq - rhou * dq - etaq * ru);
    float dV = ((dgp6 + rv * st.gp2 + rhov * dgp2) * st.dt - d_dt * st.g6) * dtaux;
    if (il == 6) { dI = 0; dV = 0; }  // me_der.c:309-312
    float* c = col + (il * 4) * kRow;
    c[0] = dI;
    c[kRow] = dQ;
    c[2 * kRow] = dU;
    c[3 * kRow] = dV;
  }
  // S1 (me_der.c:281-298)
  const float dti_s1 = -(st.dti * float(P.mu));
  col[(7 * 4 + 0) * kRow] = -dti_s1 * etai_gp3;
  col[(7 * 4 + 1) * kRow] = dti_s1 * st.g4;
  col[(7 * 4 + 2) * kRow] = dti_s1 * st.g5;
  col[(7 * 4 + 3) * kRow] = dti_s1 * st.g6;
}

// PSF correlation of the 32 response-function profiles, one profile per lane
// (me_der.c:471-496): out[k] = sum_m x[m] G[m - k + nl/2].  A loop over the inputs
// m, four at a time: one load of the inputs from the lane's own row, and their taps
// as one window of 35 consecutive entries of a reversed tap row, which is there twice,
// once shifted by an entry, so that the pairs at odd offsets are aligned too: 18
// broadcast vector loads for 128 products (the second row: 8.57 -> 8.41 ms for 65,536
// pixels of the form of then; shared memory is the busiest pipe of this kernel).  Every
// output adds its products in the order of m.  The last group's inputs beyond the
// grid are zero.  Stokes-I rows correlate Ic - x with Ic = max of the row's end
// points; the other rows run the same code with sign 1 and Ic = 0.
template <typename SM>
__device__ __forceinline__ void pair_correlate(const PmParams& P, const PairBlock& bs, SM& sm, int lane) {
  __syncwarp();
  float* row = sm.tr + lane * kRow;
  const bool isI = (lane & 3) == 0;
  const float e0 = row[0], en = row[P.nl - 1];
  const float ic = isI ? ((e0 > en) ? e0 : en) : 0.0f;
  const float sgn = isI ? -1.0f : 1.0f;
  const int groups = (P.nl + 3) / 4;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (P.nl + i < groups * 4) row[P.nl + i] = ic;  // a zero input
  // the products in pairs, one packed FMA (sm_100 f32x2) per two outputs; each half
  // of a pair rounds exactly as a scalar fma would
  float2 acc[NL / 2];
#pragma unroll
  for (int k = 0; k < NL / 2; ++k) acc[k] = make_float2(0.0f, 0.0f);
#pragma unroll 1
  for (int q = 0; q < groups; ++q) {
    const float4 r4 = *reinterpret_cast<const float4*>(row + 4 * q);
    const float xb[4] = {fmaf(sgn, r4.x, ic), fmaf(sgn, r4.y, ic), fmaf(sgn, r4.z, ic), fmaf(sgn, r4.w, ic)};
    // the taps of inputs 4q .. 4q + 3; input 4q + i and output k: t[3 - i + k]
    const float4* t0 = reinterpret_cast<const float4*>(bs.rv[0] + (NL - 4 - 4 * q));
    const float4* t1 = reinterpret_cast<const float4*>(bs.rv[1] + (NL - 4 - 4 * q));
    float4 e0 = t0[0], o0 = t1[0];
#pragma unroll
    for (int k = 0; k < NL; k += 4) {
      const float4 e1 = t0[k / 4 + 1], o1 = t1[k / 4 + 1];
      float2 lo = acc[k / 2], hi = acc[k / 2 + 1];
      lo = __ffma2_rn(make_float2(xb[0], xb[0]), make_float2(o0.z, o0.w), lo);
      hi = __ffma2_rn(make_float2(xb[0], xb[0]), make_float2(o1.x, o1.y), hi);
      lo = __ffma2_rn(make_float2(xb[1], xb[1]), make_float2(e0.z, e0.w), lo);
      hi = __ffma2_rn(make_float2(xb[1], xb[1]), make_float2(e1.x, e1.y), hi);
      lo = __ffma2_rn(make_float2(xb[2], xb[2]), make_float2(o0.x, o0.y), lo);
      hi = __ffma2_rn(make_float2(xb[2], xb[2]), make_float2(o0.z, o0.w), hi);
      acc[k / 2] = __ffma2_rn(make_float2(xb[3], xb[3]), make_float2(e0.x, e0.y), lo);
      acc[k / 2 + 1] = __ffma2_rn(make_float2(xb[3], xb[3]), make_float2(e0.z, e0.w), hi);
      e0 = e1;
      o0 = o1;
    }
  }
#pragma unroll
  for (int k = 0; k < NL; k += 4)
    *reinterpret_cast<float4*>(row + k) =
        make_float4(fmaf(sgn, acc[k / 2].x, ic), fmaf(sgn, acc[k / 2].y, ic), fmaf(sgn, acc[k / 2 + 1].x, ic),
                    fmaf(sgn, acc[k / 2 + 1].y, ic));
  __syncwarp();
}

// Entries E.. of the packed normal equations (upper triangle of alpha by rows, then
// beta) plus one Stokes profile's terms: d its response functions at this lane's
// wavelength, c its weight, r its weighted residual.  Columns b and b + 1 of a row
// go through packed f32x2 products, each half rounded as the scalar form.
template <int KT, int E>
__device__ __forceinline__ void ne_add(float (&acc)[KT * (KT + 1) / 2 + KT], const float (&d)[KT], float c, float r) {
  if constexpr (E < KT * (KT + 1) / 2 + KT) {
    constexpr int a = ne_row(E, KT), b = ne_col(E, KT);
    if constexpr (b % 2 == 0 && b + 1 < KT) {
      const float2 db = make_float2(d[b], d[b + 1]);
      float2 v = make_float2(acc[E], acc[E + 1]);
      if constexpr (a < KT) v = __ffma2_rn(__fmul2_rn(make_float2(d[a], d[a]), db), make_float2(c, c), v);
      else v = __ffma2_rn(make_float2(r, r), db, v);
      acc[E] = v.x;
      acc[E + 1] = v.y;
      ne_add<KT, E + 2>(acc, d, c, r);
    } else {
      if constexpr (a < KT) acc[E] = fmaf(d[a] * d[b], c, acc[E]);
      else acc[E] = fmaf(r, d[b], acc[E]);
      ne_add<KT, E + 1>(acc, d, c, r);
    }
  }
}

// Normal equations (covarm2): alpha = sum w_s/sigma^2 d_a d_b (upper triangle), beta
// = sum w_s (S - O)/sigma^2 d_b, packed in FP64 into ab.  One copy of the products'
// code for the four Stokes profiles, whose response functions (after correlation,
// filling factor and FijaACeroDerivadasNoNecesarias) are read from tr as they are
// used; then the sums over the warp, 32 entries at a time transposed through tr: 56
// instructions per 32 entries, where a reduction by shuffles takes 124 (the order
// of the additions is its).
template <int KT, typename SM>
__device__ __forceinline__ void pair_normal_eq(const PmParams& P, SM& sm, double* ab, int lane, bool valid, float alf,
                                               const float S[4], const float Sff[4], const float O[4],
                                               const float isig[4], const float* sl, const float (&dmac)[4]) {
  constexpr int NE = KT * (KT + 1) / 2 + KT;
  float cw[4], rw[4], sf[4], dm[4], acc[NE];
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    cw[s] = float(P.w[s]) * isig[s];
    rw[s] = float(P.w[s]) * (S[s] - O[s]) * isig[s];
    sf[s] = Sff[s];
    dm[s] = dmac[s];
  }
#pragma unroll
  for (int e = 0; e < NE; ++e) acc[e] = 0.0f;
  const float* col = sm.tr + lane;
#pragma unroll 1
  for (int s = 0; s < 4; ++s) {
    float d[KT];
#pragma unroll
    for (int r = 0; r < KT; ++r) {
      float v;
      if (r < 7) v = col[r * 4 * kRow];
      else if (r == 7) v = s == 0 ? 1.0f : 0.0f;  // S0 (me_der.c:301-306)
      else if (r == 8) v = col[7 * 4 * kRow];
      else v = r == 9 && P.mac_row == 9 ? dm[0] : 0.0f;  // zero while v_mac <= 1e-4
      d[r] = valid ? v : 0.0f;
    }
    if (KT >= 10 && P.slight_mode != PM_SLIGHT_NONE) {
      // me_der.c:499-525: every RF scaled by alpha; the filling-factor row is
      // S_mag - S_stray, built from the spectrum the caller passes (Sff)
      const float slv = sl[s * P.nl + (valid ? lane : 0)];
#pragma unroll
      for (int r = 0; r < KT; ++r) {
        d[r] = d[r] * alf;
        if (r >= 9 && r == P.ff_row) d[r] = valid ? sf[0] - slv : 0.0f;
      }
    }
    if (P.any_zero_row) {
#pragma unroll
      for (int r = 0; r < KT; ++r)
        if (P.zero_row[r]) d[r] = 0.0f;
    }
    ne_add<KT, 0>(acc, d, cw[0], rw[0]);
    col += kRow;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      cw[q] = cw[q + 1];
      rw[q] = rw[q + 1];
      if (KT >= 10) {
        sf[q] = sf[q + 1];
        dm[q] = dm[q + 1];
      }
    }
  }
#pragma unroll
  for (int c = 0; c < NE; c += 32) {
    __syncwarp();  // tr is read no more
#pragma unroll
    for (int e = c; e < NE && e < c + 32; ++e) sm.tr[(e - c) * kRow + lane] = acc[e];
    __syncwarp();
    const float v = ne_row_sum(sm.tr, lane);
    if (c + lane < NE) ab[c + lane] = double(v);
  }
}

// The response functions of the last synthesis in tr (rows 0..31: profile, columns:
// wavelength), after the PSF or macroturbulence convolution; dmac: the v_mac row at
// this lane's wavelength.  mt, mac: the terms and v_mac of the model.  MAC: compiled
// with the macroturbulence branch (the grid has a v_mac row; NTERMS >= 10).
template <bool MAC, typename SM>
__device__ __forceinline__ void pair_response(const PmParams& P, const PairBlock& bs, SM& sm,
                                              const ModelTerms<float>& mt, int lane, bool valid, double mac, double dl,
                                              float (&dmac)[4]) {
  const bool mac_on = MAC && uniform(mac > kMacMin);
  if (mac_on) mac_prepare<float, true>(P, sm, mac, dl, lane, valid);
  {
    ModelTerms<float> T;
    copy16(T, mt);
    LaneState<float> st;
    copy16(st, *reinterpret_cast<const LaneState<float>*>(sm.ls[lane]));
    __syncwarp();  // the profiles overwrite the lanes' states
    rf_rows(P, T, st, sm.tr + lane);
  }
  if (mac_on) {
    mac_rf_circular<float, kRow>(P, sm, lane);
    const float* xf = &sm.xs[0][0];
    mac_circular4<float>(P, xf, xf + kMacD, lane, dmac);
  } else if (P.has_psf) {
    pair_correlate(P, bs, sm, lane);
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------
// A warp inverts two pixels at a time.  What is parallel over wavelengths (the
// synthesis with chi^2, the response functions, the normal equations) takes all
// lanes, one pixel after the other; what is serial or parallel over the 9-11
// parameters (the damped solve, the trial model and its per-model terms, the LM
// bookkeeping) runs once for both, half a warp for each.  A pixel's state lives in
// shared memory between the parts (PixelSlot).
// ---------------------------------------------------------------------------
template <int KT>
struct alignas(16) PixelSlot {
  static constexpr int NA = KT * (KT + 1) / 2, NE = NA + KT;
  ModelTerms<float> mt;                // of the trial model
  double ab[NE];                   // packed alpha (upper triangle by rows) and beta of the model
  double model[11], trial[11], delta[11];
  double chi, ochi, chi0, flambda, factor;
  float S[4][NL];                      // the last synthesis
  const PmJob* job;                // this slot's pixel: its job, ...
  unsigned long long pix;          // ... index in the job, ...
  unsigned long long job_t0, job_n;  // ... the job's first ticket and pixel count
  const float* obs;
  const float* sl;
  const double* lam;
  int nfree, status, iter, accepted, fallbacks;
  int accept, stop, first, grid;
  long long job_k;
};

template <int KT>
struct alignas(16) PairSmem : RowsSmem {
  PixelSlot<KT> px[2];
};

// FP64 Cholesky solve of the damped normal equations, one slot per half warp:
// lane i of the half owns row i.  Right-looking; one reciprocal square root per
// pivot (no divisions), formed while the column before it is still being applied.
// The columns go through one loop body (the rows shift by a column each time, what
// lies beyond the triangle is never used): unrolled, its code was 11.5 KB, a third
// of what the instruction cache holds.  A column of L goes through shared memory:
// four vector loads where shuffles took sixteen, which bound the loop.  The back
// solve reads the factor from there, in every lane.  Exactly-zero rows (fixed
// parameters) get a zero step, as the pseudo-inverse gives them.  False on a pivot
// <= 1e-12 (the caller then uses the eigen solver for this step).
template <int KT>
struct CholeskyScratch {  // per half, in doubles
  static constexpr int ROW = (KT + 2) & ~1;  // column j: L[j + 1 + m][j] at j * ROW + m, the last entry unused
  static constexpr int SIZE = KT * ROW + 2 * KT;
};

template <int KT>
__device__ __forceinline__ bool solve_cholesky_half(const double* ab, double* lt, int i16, double flambda,
                                                    double (&delta)[KT]) {
  constexpr int NA = KT * (KT + 1) / 2, ROW = CholeskyScratch<KT>::ROW;
  const int i = i16 < KT ? i16 : KT - 1;
  double* Y = lt + KT * ROW;  // the forward solution
  double* Rv = Y + KT;        // 1 / pivot
  double a[KT + 1];           // row i from column j, left of the diagonal
#pragma unroll
  for (int k = 0; k < KT; ++k) a[k] = ab[k * KT - (k * (k - 1)) / 2 - k + i];
  a[KT] = 0.0;
  const double diag = ab[i * KT - (i * (i - 1)) / 2];
  double dg = diag * (1.0 + flambda);
  const unsigned zr = __ballot_sync(kFull, i16 < KT && diag == 0.0) >> (threadIdx.x & 16);
  double b = (zr >> i) & 1u ? 0.0 : ab[NA + i];
  bool ok = true;
  auto pivot = [&](int j) {  // 1 / sqrt of pivot j (j == KT: not used)
    const double piv = __shfl_sync(kFull, dg, j, 16);
    const bool skip = ((zr >> j) & 1u) || j == KT;
    ok = ok && (skip || (piv > 1e-12 && piv < 1e300));
    const double rs = rsqrt(skip ? 1.0 : piv);
    return skip ? 0.0 : rs;
  };
  double r = pivot(0);
#pragma unroll 1
  for (int j = 0; j < KT; ++j) {
    const double l = a[0] * r;  // L[i][j] for i > j
    const double y = __shfl_sync(kFull, b, j, 16) * r;
    // selections and stores without branches: the lanes past the last row repeat it,
    // and y and r are the same in the half
    const double bn = fma(-l, y, b), dn = fma(-l, l, dg);
    b = i > j ? bn : b;
    dg = i > j ? dn : dg;
    lt[j * ROW + (i > j ? i - j - 1 : KT)] = l;
    Y[j] = y;
    Rv[j] = r;
    __syncwarp();
    const double2* col = reinterpret_cast<const double2*>(lt + j * ROW);
    r = pivot(j + 1);
#pragma unroll
    for (int k = 0; k < KT; k += 2) {
      const double2 lk = col[k / 2];
      a[k] = fma(-l, lk.x, a[k + 1]);
      if (k + 1 < KT) a[k + 1] = fma(-l, lk.y, a[k + 2 <= KT ? k + 2 : KT]);
    }
  }
  __syncwarp();
#pragma unroll
  for (int j = KT - 1; j >= 0; --j) {
    double s = Y[j];
#pragma unroll
    for (int k = j + 1; k < KT; ++k) s = fma(-lt[j * ROW + k - j - 1], delta[k], s);
    delta[j] = s * Rv[j];
  }
  return ok;
}

// Entry e of the full symmetric alpha (K x K) followed by beta: its place in the
// packed vector.
template <int KT>
__device__ __forceinline__ int ne_packed(int e) {
  if (e >= KT * KT) return KT * (KT + 1) / 2 + (e - KT * KT);
  int a = e / KT, b = e % KT;
  if (a > b) { int t = a; a = b; b = t; }
  return a * KT - (a * (a - 1)) / 2 + (b - a);
}

// The damped solve of slot px by eigen-decomposition, the whole warp.
template <int KT, typename SM>
__device__ __forceinline__ void solve_eigen_slot(SM& sm, PixelSlot<KT>& px, int lane) {
  SolveSmem& sv = *reinterpret_cast<SolveSmem*>(&sm.xs[0][0]);
  for (int e = lane; e < KT * KT + KT; e += 32) sv.ab[e] = px.ab[ne_packed<KT>(e)];
  __syncwarp();
  solve_eigen<KT>(sv, reinterpret_cast<double*>(sm.tr), lane, px.flambda);
  if (lane < KT) px.delta[lane] = sv.delta[lane];
  __syncwarp();
  xs_restore<float>(sm, lane);
}

// Half a warp per slot: the damped solve and the trial model (every pass but a
// pixel's first), then the per-model terms.  on: the half's slot holds a pixel.
template <int KT, typename SM>
__device__ __forceinline__ void pair_step(const PmParams& P, const PairBlock& bs, SM& sm, int lane, bool on) {
  const int half = lane >> 4, i16 = lane & 15;
  PixelSlot<KT>& px = sm.px[half];
  const bool go = on && !px.first;
  if (uniform(go)) {
    bool ok = false;
    if (uniform(go && P.solver == PM_SOLVE_CHOLESKY)) {
      double delta[KT];
      double* lt = reinterpret_cast<double*>(sm.tr) + half * CholeskyScratch<KT>::SIZE;
      ok = solve_cholesky_half<KT>(px.ab, lt, i16, px.flambda, delta) && P.solver == PM_SOLVE_CHOLESKY;
      if (i16 == 0) {
#pragma unroll
        for (int j = 0; j < KT; ++j) px.delta[j] = delta[j];
      }
      __syncwarp();
    }
    const unsigned bad = __ballot_sync(kFull, go && !ok && i16 == 0);
    if (bad) {
      if (go && !ok && i16 == 0 && P.solver == PM_SOLVE_CHOLESKY) ++px.fallbacks;
#pragma unroll 1
      for (int s = 0; s < 2; ++s)
        if ((bad >> (16 * s)) & 1u) solve_eigen_slot<KT>(sm, sm.px[s], lane);
    }
    // AplicaDelta (milosUtils.c:47-115) and check (:118-196), a parameter per lane:
    // p <- p - delta for free parameters, with the step on B clamped to +-300 G and
    // on gamma, azimuth to +-30 deg; then the bounds
    const int i = i16 < 11 ? i16 : 0;
    const double old = px.trial[i];
    // NTERMS 10: the tenth step is v_mac's or alpha's, whichever is inverted
    double d = px.delta[KT == 10 && i == 10 ? 9 : i];
    const double lim = i == 1 ? 300.0 : (i == 5 || i == 6) ? 30.0 : HUGE_VAL;
    d = d < -lim ? -lim : (d > lim ? lim : d);
    const double stepped = px.model[i] - d;
    double v = ((P.fix_mask >> i) & 1) && (i < 9 || KT > 9) ? stepped : old;
    const bool flip = __shfl_sync(kFull, v < 0 ? 1 : 0, 1, 16);  // B changes sign: so does cos(gamma)
    if (i == 5) {
      if (flip) v = 180.0 - v;
      if (v < 0) v = -v;
      if (v > 180) v = 360.0 - v;
    } else if (i == 6) {
      if (v < 0) v = 180 + v;
      if (v > 180) v = v - 180.0;
    } else {
      if (i == 1 && flip) v = -v;
      if (i != 1 && v < bs.lo[i]) v = bs.lo[i];
      if (v > bs.hi[i]) v = bs.hi[i];
    }
    if (go && i16 < 11) px.trial[i] = v;
    __syncwarp();
  }
  ModelTerms<float> T;
  {
    // lane 0 of the half evaluates the inclination, lane 1 the azimuth
    const float CC = float(kPi / 180.0);
    const float ang = (lane & 1) ? 2.0f * (float(px.trial[6]) * CC) : float(px.trial[5]) * CC;
    float s, c;
    sincosf(ang, &s, &c);
    terms_from(P, px.trial, __shfl_sync(kFull, s, 0, 16), __shfl_sync(kFull, c, 0, 16), __shfl_sync(kFull, s, 1, 16),
               __shfl_sync(kFull, c, 1, 16), T);
  }
  if (i16 == 0) copy16(px.mt, T);
  __syncwarp();
}

// One pass of the LM loop for one slot: the trial model's synthesis and chi^2, and
// when it is accepted its response functions and normal equations.  MAC: compiled
// with the macroturbulence branch (grids with a v_mac row).  PIXGRID: the pixel has
// its own wavelengths.
template <int KT, bool MAC, bool PIXGRID, typename SM>
__device__ __forceinline__ void pair_pass(const PmParams& P, const PairBlock& bs, SM& sm, PixelSlot<KT>& px,
                                          int lane, double dl) {
  const bool valid = lane < P.nl;
  const float* sl = px.sl;
  const bool first = px.first != 0;
  const double mac = MAC ? px.trial[9] : 0.0;
  // the profiles may have been written by a copy engine while the kernel runs:
  // they are read from L2, in every pass (they are in use again before a copy kept
  // in registers or shared memory would pay)
  float O[4];
  float S[4], Su[4], isig[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) O[s] = valid ? __ldcg(px.obs + s * P.nl + lane) : 0.0f;
  if constexpr (PIXGRID) dl = valid ? __ldcg(px.lam + lane) - P.lambda0 : 0.0;
  {
    ModelTerms<float> T;
    copy16(T, px.mt);
    pair_synth(P, T, dl, sm.ls[lane], S);
    convolve_and_mix<float, MAC, (KT >= 10)>(P, sm, T, mac, sl, lane, valid, dl, S, Su,
                                             [&] { pair_psf(P, bs, sm, lane, valid, S); });
  }
#pragma unroll
  for (int s = 0; s < 4; ++s) isig[s] = bs.isig[valid && O[s] <= -1.0f ? 1 : 0];
  const double chi = chisq<float>(P, S, O, isig, valid, double(px.nfree));
  const bool accept = first || chi - px.ochi < 0.;
#pragma unroll
  for (int s = 0; s < 4; ++s) px.S[s][lane] = S[s];
  if (lane == 0) {
    px.chi = chi;
    px.accept = accept ? 1 : 0;
  }
  if (uniform(accept)) {
    // the filling-factor row is built from the unmixed synthesis on the first
    // call of me_der and from the mixed one after a step (milosUtils.c:537 vs :587)
    float Sff[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) Sff[s] = first ? Su[s] : S[s];
    float dmac[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    pair_response<MAC>(P, bs, sm, px.mt, lane, valid, mac, dl, dmac);
    pair_normal_eq<KT>(P, sm, px.ab, lane, valid, px.mt.alf, S, Sff, O, isig, sl, dmac);
  }
  __syncwarp();
}

// The LM loop's bookkeeping after a pass (lm_mils, milosUtils.c:540-630), half a
// warp per slot: stopping and acceptance, the damping, the iteration count.  True
// when the half's pixel is finished.
template <int KT, typename SM>
__device__ __forceinline__ bool pair_update(const PmParams& P, SM& sm, int lane, bool on) {
  const int i16 = lane & 15;
  PixelSlot<KT>& px = sm.px[lane >> 4];
  bool finished = false;
  const double chi = px.chi, ochi = px.ochi, factor = px.factor;
  const bool accept = px.accept != 0, first = px.first != 0;
  bool stop = px.stop != 0;
  int status = px.status, iter = px.iter;
  double flambda = px.flambda;
  __syncwarp();
  if (on) {
    if (!first) {
      if ((fabs((ochi - chi) * 100 / chi) < P.toplim) || (chi < 0.0001)) {
        stop = true;
        status = PM_PIX_CONVERGED;
      }
      if (accept) flambda = flambda / (5.0 * factor);
      else flambda = flambda * 10.0 * factor;
      if ((flambda > 1e+7) || (flambda < 1e-25)) {
        if (!stop) status = PM_PIX_LAMBDA;
        stop = true;
      }
      ++iter;
      finished = !(iter < P.miter && !stop);  // lm_mils' do-while: at least one step
    }
    if (accept && i16 < 11) px.model[i16] = px.trial[i16];
    if (i16 == 0) {
      if (accept) {
        px.ochi = chi;
        if (first) px.chi0 = chi;
        else ++px.accepted;
      }
      if (!first && P.logclambda) px.factor = double(log10f(float(chi)) / log10f(float(px.chi0)));
      px.flambda = flambda;
      px.stop = stop;
      px.status = status;
      px.iter = iter;
      px.first = 0;
    }
  }
  __syncwarp();
  return finished;
}

// A pixel's start (invert_pixel up to its loop): its profiles, ghosts and starting
// model -- the classical estimates (milos.c:958-983) of the pre-pass kernel when
// the whole cube was on the device before the launch, else computed here.
template <int KT, bool PIXGRID>
__device__ __forceinline__ void pair_begin(const PmParams& P, const PairBlock& bs, PixelSlot<KT>& px, int lane) {
  const bool valid = lane < P.nl;
  const PmJob* jp = px.job;
  const size_t p = px.pix;
  const size_t base = p * 4 * P.nl;
  const float* obs = ld_ptr(&jp->spectro) + base;
  const double* model_in = ld_ptr(&jp->model_in);
  const float* sl = pair_slight(P, bs, P.slight_mode == PM_SLIGHT_PER_PIXEL ? ld_ptr(&jp->slight) : nullptr, base);
  const double* lam = PIXGRID ? ld_ptr(&jp->lambda) + p * P.nl : nullptr;
  float O[4];
  int ghosts = 0;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    O[s] = valid ? __ldcg(obs + s * P.nl + lane) : 0.0f;
    ghosts += __popc(__ballot_sync(kFull, valid && O[s] <= -1.0f));
  }
  double mine = 0;
  if (uniform(model_in != nullptr)) {
    if (lane < 11) mine = __ldcg(model_in + p * 11 + lane);
  } else {
    double g[11];
#pragma unroll
    for (int i = 0; i < 11; ++i) g[i] = P.guess[i];
    double dl;
    if constexpr (PIXGRID) dl = valid ? __ldcg(lam + lane) - P.lambda0 : 0.0;
    else dl = P.dl[valid ? lane : 0];
    if (P.classical) classical(P, O, lane, valid, dl, g);
    mine = g[0];
#pragma unroll
    for (int i = 1; i < 11; ++i)
      if (lane == i) mine = g[i];
  }
  if (lane < 11) {
    px.model[lane] = mine;
    px.trial[lane] = mine;
  }
#pragma unroll
  for (int s = 0; s < 4; ++s) px.S[s][lane] = 0;  // the result when nfree == 0
  if (lane == 0) {
    const int nfree = P.nfree_base - ghosts;
    px.obs = obs;
    px.sl = sl;
    px.lam = lam;
    px.nfree = nfree;
    px.status = nfree == 0 ? PM_PIX_NFREE : PM_PIX_MAXITER;
    px.iter = nfree == 0 ? -1 : 0;
    px.accepted = px.fallbacks = 0;
    px.ochi = px.chi0 = px.chi = 0;
    px.flambda = P.ilambda;
    px.factor = 1.0;
    px.stop = 0;
    px.first = 1;
  }
  __syncwarp();
}

// A pixel's end: the finite check, its results, its job's counter and, when it was
// the job's last pixel, the job's host flag (the server's completion signal).
template <int KT>
__device__ __forceinline__ void pair_end(const PmParams& P, PixelSlot<KT>& px, int lane, unsigned long long* ctr) {
  const PmJob* jp = px.job;
  const size_t p = px.pix;
  if (lane < 11) ld_ptr(&jp->models)[p * 11 + lane] = px.model[lane];
  if (lane == 0) {
    bool finite = isfinite(px.ochi);
#pragma unroll 1
    for (int i = 0; i < 11; ++i) finite = finite && isfinite(px.model[i]);
    const int status = px.nfree != 0 && !finite ? PM_PIX_NONFINITE : px.status;
    ld_ptr(&jp->chisq)[p] = float(px.ochi);
    ld_ptr(&jp->iters)[p] = px.iter;
    int* st = ld_ptr(&jp->status);
    if (st) st[p] = status;
    atomicAdd(&ctr[PMC_ITERS], (unsigned long long)(px.iter > 0 ? px.iter : 0));
    atomicAdd(&ctr[PMC_ACCEPTED], (unsigned long long)px.accepted);
    if (px.fallbacks) atomicAdd(&ctr[PMC_FALLBACK], (unsigned long long)px.fallbacks);
  }
  float* spectra = ld_ptr(&jp->spectra);
  if (spectra && lane < P.nl) {
#pragma unroll
    for (int s = 0; s < 4; ++s) spectra[p * 4 * P.nl + s * P.nl + lane] = float(px.S[s][lane]);
  }
  unsigned long long* done = ld_ptr(&jp->done);
  if (uniform(done != nullptr)) {
    __threadfence();  // every lane: its part of this pixel's results before the count
    __syncwarp();
    if (lane == 0) {
      int* flag = ld_ptr(&jp->host_flag);
      const unsigned long long np = __ldcg(reinterpret_cast<const unsigned long long*>(&jp->npix));
      if (atomicAdd(done, 1ull) + 1 == np && flag) {
        __threadfence_system();
        *reinterpret_cast<volatile int*>(flag) = 1;
      }
    }
  }
  __syncwarp();
}

// The warps of a block work for themselves: nothing in the loop waits for another
// warp.  A slot without a pixel draws its next ticket (one atomicAdd, at most one
// a round, so that the warps of a launch share a small call's pixels evenly) and
// owns it: the pixel starts once the ticket is published.  While the other slot
// holds a pixel the warp goes on with it; with nothing to do it sleeps between
// looks at the queue, up to the wait limit after the last publication it saw (then
// PMQ_ERR_WAIT: its own tickets may be far ahead of a slow producer's), and ends once
// the queue is closed and its tickets are beyond the final count.  MULTI: the launch
// serves up to PMK_MAX_GRIDS grids (a server's), each pixel on its own.
template <int KT, bool MULTI, bool MAC, bool PIXGRID>
__global__ void __launch_bounds__(128, 4) invert_pair_kernel(
    const __grid_constant__ GridParams<MULTI ? PMK_MAX_GRIDS : 1> GS, const PmStreamIO sio) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NG = MULTI ? PMK_MAX_GRIDS : 1;
  using SM = PairSmem<KT>;
  const int lane = threadIdx.x & 31, warp = __shfl_sync(kFull, int(threadIdx.x >> 5), 0);
  const int half = lane >> 4;
  PairBlock* bs = reinterpret_cast<PairBlock*>(smem_raw);
  SM& sm = reinterpret_cast<SM*>(smem_raw + NG * sizeof(PairBlock))[warp];
#pragma unroll 1
  for (int g = 0; g < NG && g < GS.ngrids; ++g) pair_block(GS.g[g], bs[g]);
  for (int e = lane; e < int(sizeof(SM) / 4); e += 32) reinterpret_cast<unsigned*>(&sm)[e] = 0;
  __syncthreads();
  if (lane < 11) sm.px[0].trial[lane] = sm.px[1].trial[lane] = 1.0;  // an empty slot's terms: ordinary values
  if (lane == 0) {
    sm.grid_cur = -1;
    sm.px[0].job_k = sm.px[1].job_k = sio.first_job;
  }
  __syncwarp();
  double dl = 0.0;                  // this lane's wavelength offset on the grid in use
  // bit per slot; when every pixel has a warp of its own, the second slot stays empty
  unsigned active = 0, drained = sio.published && sio.published <= (long long)gridDim.x * (blockDim.x >> 5) ? 2u : 0u;
  long long held = -1;              // lanes 0 and 16: the slot's drawn ticket that is not published yet
  unsigned long long avail = (unsigned long long)sio.published;  // tickets published, as last seen
  long long since = -1;
  unsigned sleep_ns = 32, age = 0;
  while (true) {
    if ((active | drained) != 3u) {
      const bool want = (lane & 15) == 0 && !(((active | drained) >> half) & 1u);
      const unsigned draw = __ballot_sync(kFull, want && held < 0);
      if (draw && lane == __ffs(draw) - 1) held = (long long)atomicAdd(&sio.q->next, 1ull);
      const bool waiting = want && held >= 0;
      bool closed = sio.published != 0;
      if (!closed && __ballot_sync(kFull, waiting && (unsigned long long)held >= avail) && (active == 0 || ++age >= 4)) {
        age = 0;
        closed = ld_acquire(&sio.q->closed) != 0;  // written after the last publication
        const unsigned long long seen = ld_acquire(&sio.q->avail);
        if (uniform(seen != avail)) since = -1;
        avail = seen;
      }
      bool start = false, end = false;
      if (waiting && (unsigned long long)held < avail) {
        // the job of the ticket: usually the slot's previous one, else at or after
        // it (jobs are appended in ticket order)
        PixelSlot<KT>& px = sm.px[half];
        const unsigned long long t = (unsigned long long)held;
        held = -1;
        start = px.job && t >= px.job_t0 && t < px.job_t0 + px.job_n;
        long long k = px.job_k;
        for (int guard = 0; !start && guard <= sio.jobs_cap; ++guard, ++k) {
          const PmJob* c = sio.jobs + (k % sio.jobs_cap);
          const unsigned long long c0 = __ldcg(&c->t0);
          const unsigned long long cn = __ldcg(reinterpret_cast<const unsigned long long*>(&c->npix));
          if (t >= c0 && t < c0 + cn) {
            px.job = c;
            px.job_t0 = c0;
            px.job_n = cn;
            px.job_k = k;
            start = true;
          }
        }
        if (start) {
          px.pix = t - px.job_t0;
          px.grid = MULTI ? __ldcg(&px.job->grid) : 0;
        } else {
          atomicExch(&sio.q->err, (unsigned long long)PMQ_ERR_JOB);
          end = true;
        }
      } else if (waiting && closed) {
        end = true;  // the held ticket will never be published
      }
      const unsigned started = __ballot_sync(kFull, start), ended = __ballot_sync(kFull, end);
      drained |= (ended & 1u) | ((ended >> 15) & 2u);
      __syncwarp();
#pragma unroll 1
      for (int s = 0; s < 2; ++s) {
        if (!((started >> (16 * s)) & 1u)) continue;
        PixelSlot<KT>& px = sm.px[s];
        const int gi = MULTI ? __shfl_sync(kFull, px.grid, 0) : 0;
        pair_begin<KT, PIXGRID>(GS.g[gi], bs[gi], px, lane);
        if (uniform(px.nfree == 0)) pair_end<KT>(GS.g[gi], px, lane, sio.q->ctr);
        else active |= 1u << s;
      }
      if (active == 0) {
        if (drained == 3u) break;
        if (started) {
          since = -1;
          sleep_ns = 32;
          continue;
        }
        const long long now = global_ns();
        if (since < 0) since = now;
        if (uniform(now - since > sio.wait_limit_ns)) {
          if (lane == 0) atomicExch(&sio.q->err, (unsigned long long)PMQ_ERR_WAIT);
          break;
        }
        if (!draw) {
          __nanosleep(sleep_ns);
          sleep_ns = sleep_ns < 2048 ? 2 * sleep_ns : 2048;
        }
        continue;
      }
      since = -1;
      sleep_ns = 32;
    }
    const bool on = (active >> half) & 1u;
    const int gh = MULTI ? sm.px[half].grid : 0;  // the half's grid
    const PmParams& Ph = GS.g[gh];
    pair_step<KT>(Ph, bs[gh], sm, lane, on);
#pragma unroll 1
    for (int s = 0; s < 2; ++s) {
      if (!((active >> s) & 1u)) continue;
      PixelSlot<KT>& px = sm.px[s];
      const int gi = MULTI ? __shfl_sync(kFull, px.grid, 0) : 0;
      const PmParams& P = GS.g[gi];
      if (uniform(gi != sm.grid_cur)) {  // the padded rows' offset depends on the grid
        for (int e = lane; e < 4 * XSR; e += 32) (&sm.xs[0][0])[e] = 0.0f;
        dl = P.dl[lane < P.nl ? lane : 0];
        __syncwarp();
        if (lane == 0) {
          sm.grid_cur = gi;
          sm.xs_dirty = 0;
        }
        __syncwarp();
      }
      pair_pass<KT, MAC, PIXGRID>(P, bs[gi], sm, px, lane, dl);
    }
    const bool finished = pair_update<KT>(Ph, sm, lane, on);
    const unsigned fin = __ballot_sync(kFull, finished && (lane & 15) == 0);
    if (fin) {
#pragma unroll 1
      for (int s = 0; s < 2; ++s) {
        if (!((fin >> (16 * s)) & 1u)) continue;
        const int gi = MULTI ? __shfl_sync(kFull, sm.px[s].grid, 0) : 0;
        pair_end<KT>(GS.g[gi], sm.px[s], lane, sio.q->ctr);
        active &= ~(1u << s);
      }
    }
  }
}

// 16 warps per SM (128 registers).  20 (96 registers, spills) hide more latency and gain
// up to 1% on large calls of nine parameters, but lose elsewhere: 65,536 pixels 7.80 ms
// with 16, 7.78 with 20; 2,800 pixels 787, 851 us; 65,025 pixels of 15 wavelengths 6.73,
// 7.00 ms; nine served scans of 10,000 pixels 13.9, 14.5 ms; 11 parameters, 16,384
// pixels 7.16, 8.08 ms.
template <int KT, bool MULTI, bool MAC, bool PIXGRID = false>
int launch_invert_pair(const PmGridSet& GS, const PmStreamIO& sio, cudaStream_t st, int num_sms, size_t* smem_out,
                       int wpb, int reserve) {
  if (wpb > 4) wpb = 4;
  const int threads = 32 * wpb;
  constexpr int NG = MULTI ? PMK_MAX_GRIDS : 1;
  using SM = PairSmem<KT>;
  static_assert(sizeof(PairBlock) % 16 == 0 && sizeof(PixelSlot<KT>) % 16 == 0 && sizeof(SM) % 16 == 0 &&
                    sizeof(SolveSmem) <= 4 * XSR * sizeof(float) &&
                    eigen_scratch_doubles<KT>() * sizeof(double) <= NL * kRow * sizeof(float) &&
                    2 * CholeskyScratch<KT>::SIZE * sizeof(double) <= NL * kRow * sizeof(float) &&
                    CholeskyScratch<KT>::SIZE % 2 == 0,
                "pair shared-memory layout");
  const size_t smem = NG * sizeof(PairBlock) + sizeof(SM) * wpb;
  if (smem_out) *smem_out = smem;
  auto kern = invert_pair_kernel<KT, MULTI, MAC, PIXGRID>;
  GridParams<NG> gp;  // copied into the launch
  gp.ngrids = GS.ngrids < NG ? GS.ngrids : NG;
  for (int g = 0; g < gp.ngrids; ++g) gp.g[g] = GS.g[g];
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess) return snprintf(pmk_g_err, sizeof pmk_g_err, "%s", cudaGetErrorString(e)), PM_EIO;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  if (e != cudaSuccess || per_sm < 1) return snprintf(pmk_g_err, sizeof pmk_g_err, "occupancy: %s", cudaGetErrorString(e)), PM_EIO;
  int blocks = per_sm * num_sms - reserve > 1 ? per_sm * num_sms - reserve : 1;
  // a call of few pixels: one per warp, and no warps that would only draw tickets
  // beyond the last (without the limit: 100 pixels from host arrays 509 us, with it 428;
  // 592 on the device 564, 407; 1,800 on the device 666, 630; one lm_mils call the same)
  if (sio.max_pixels > 0 && blocks > (sio.max_pixels + wpb - 1) / wpb) blocks = (sio.max_pixels + wpb - 1) / wpb;
  kern<<<unsigned(blocks), threads, smem, st>>>(gp, sio);
  e = cudaGetLastError();
  if (e != cudaSuccess) return snprintf(pmk_g_err, sizeof pmk_g_err, "pair launch: %s", cudaGetErrorString(e)), PM_EIO;
  return PM_OK;
}

}  // namespace
