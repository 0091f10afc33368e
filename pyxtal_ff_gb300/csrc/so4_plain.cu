// so4_plain.cu -- the "plain" path: B, dB/dr per (i, j) pair and the per-pair
// virial rdxdr, as pyxtal_ff/descriptors/SO4.py:1409-1548 (derivative + stress
// branch of get_bispectrum_components) returns them through calculate()
// (SO4.py:190-199).  Four kernels:
//   k_plain_u  U_tot (:1480-1505), one CTA per centre;
//   k_plain_z  every Z block the components read (compute_zi, :1020-1068), 32 centres
//              across the lanes of a warp;
//   k_plain_b  B (compute_bi, :1071-1111), the same way;
//   k_plain_d64, k_plain_d32  per image t = dB/dr (compute_dbidrj, :1113-1227), one CTA per
//              centre, and per pair dxdr[p] = sum t (j != i), dxdr[(i,i)] = -sum over the
//              other pairs, rdxdr[p] = (R_i (x) dxdr[p] + sum r (x) t) / vol -- algebraically
//              the reference's -bstress/vol (:1458-1468).
//
// U is carried in the scaled form V = U / F of so4_rowchain.cuh and Z as Z' = F Z, so that
// sum conj(U) Z = sum conj(V) Z' and the recursion is V_l[ma] = conj(a) V_{l-1}[ma] -
// conj(b) V_{l-1}[ma-1].
//
// The gradient of U.  Row mb of level l is the polynomial p(t)^(l-mb) q(t)^mb with
// (p, q) = M (t1, t2), M = [[a*, -b*], [b, a]] in SU(2).  A step dr moves M by M X with
// X = M^+ dM = [[i alpha, beta + i gamma], [-beta + i gamma, -i alpha]], three real numbers,
// and so
//   dV[m] = i alpha (l-2m) V[m] + beta ((l-m+1) V[m-1] - (m+1) V[m+1])
//         + i gamma ((l-m+1) V[m-1] + (m+1) V[m+1]).
// Contracted with a row of Z' the shifts move over to Z':  Re sum conj(dV) Z' =
// alpha P1 + beta P2 + gamma P3,  P_g = Re sum conj(V) W_g,
//   W0 = Z',  W1 = -i (l-2m) Z'[m],  W2 = (l-m) Z'[m+1] - m Z'[m-1],
//   W3 = -i ((l-m) Z'[m+1] + m Z'[m-1])
// (P0 is the term of the cutoff's derivative).  No dU is ever formed: an image costs its rows
// of V (8 multiply-adds per entry; three derivative recursions take 48 more).  Every block
// has roles in one component only, so its factor (2, 2 (l+1)/(l1+1), ...) goes into Z'.
//
// Measured on a GB300 (one pass with the neighbour list; before: one CTA per centre for
// everything, dU by recursion, every lane of a warp computing the image's set-up): FP64, 32,000
// Si atoms, 0.93 M images, lmax 4: 142.3 -> 25.7 ms (k_plain_d64 13.8, k_plain_z 7.9, k_plain_u
// 3.3); FP32, 16,232 atoms in 256 structures, lmax 3: 2.92 -> 1.04 ms.  k_plain_z is bound by the
// FP64 pipe (95 % busy), k_plain_u too (91 %); k_plain_d64 by latency at twelve warps per SM: of
// a CTA's 263,000 cycles the digit products take 115,000 (integer and shared-memory work around
// the matrix instructions), V 48,000, the rows 46,000 (FP64), the set-up beside the rounding of
// Z' 25,000.
#include <cstdio>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include <cuda_fp16.h>

#include "so4_atom.cuh"

namespace {

// a complex value, aligned so that it moves as one 8- or 16-byte word
template <typename T>
struct __align__(2 * sizeof(T)) pc {
    T re, im;
};

template <typename T>
struct PlainArgs {
    so4_params prm;
    int a0, natoms;  // centres a0 .. natoms - 1
    int n_u, n_half, n_z, n_b, n_unit;
    T rc, psi_fac;  // rcut and rfac0 pi / rcut
    int cw;  // k_plain_d64: 2^cw bounds the weights in W, times 4
    const so4_geom *geom;
    const int *astruct;
    const double *pos, *w_nb, *w_site, *img_r;
    const int32_t *img_ptr, *img_j, *pair_ptr, *pair_img, *nsite;
    const int4 *unit, *vent, *lam, *blk;
    const int2 *hfull;
    const T *ca, *cb;
    const double *fac;
    const int *sent, *bblk, *zent, *wk, *kord;
    const int4 *wpos;
    const float4 *wfac;
    SmallTables st;
    int want_stress;
    T *x, *dxdr, *rdxdr;
    // scratch of this pass, centre c = a - a0 in tile c / 32, lane c % 32:
    pc<T> *ut;       // U_tot, full rows: [tile][n_u][32]
    pc<T> *zt;       // Z': [tile][32 / ZQ][n_z][ZQ]
    float2 *uh;      // FP32: V_tot, half layout [centre][n_half]
    longlong2 *zi;   // k_plain_d64 without room for them in shared memory: integers [centre][n_z]
};

// ---------------------------------------------------------------- U_tot
// FP64: V of 16 images at a time (40 KB at lmax 4), V[entry][image], the images of entry e
// permuted so that the four entries x eight images of a matrix fragment (k_plain_d64) lie in
// different banks.
constexpr int VI = 16;
__device__ __forceinline__ int v_at(int e, int img) { return e * VI + (img ^ ((e & 3) << 1)); }

// -x or x by the sign bit: a negation is an FP64 instruction otherwise
__device__ __forceinline__ double flip(double x, int neg) {
    return __hiloint2double(__double2hiint(x) ^ (neg << 31), __double2loint(x));
}

// V of n <= 16 images (Cayley-Klein parameters ck[4][32], from image c0 on), all levels.  Lanes
// take (entry, image) pairs of a level, image fastest: the FP64 pipe (1/64 of the FP32 rate)
// is what counts, and this leaves no lane idle.
template <int NT>
__device__ __forceinline__ void plain_rows(const SmallTables &st, const int4 *__restrict__ vent, const double *ck,
                                           int c0, int n, pc<double> *V) {
    const int tid = threadIdx.x;
    const unsigned inv = (1u << 20) / (unsigned)n + 1u;  // t / n for t < 2^16
    if (tid < n) V[v_at(0, tid)] = {1.0, 0.0};
    for (int l = 1; l <= st.twol; ++l) {
        __syncthreads();
        const int cnt = (l / 2 + 1) * (l + 1) * n, hb = st.h_block[l];
        for (int t = tid; t < cnt; t += NT) {
            const int e = (int)(((unsigned)t * inv) >> 20), img = t - e * n;
            const int4 en = __ldg(vent + hb + e);
            const double ar = ck[c0 + img], ai = ck[32 + c0 + img], br = ck[64 + c0 + img], bi = ck[96 + c0 + img];
            double re = 0.0, im = 0.0;
            if (en.y >= 0) {
                const pc<double> p = V[v_at(en.y, img)];
                const double pr = flip(p.re, en.z >> 2), pi = flip(p.im, (en.z >> 2) ^ (en.z & 1));
                re = fma(bi, pi, -br * pr);
                im = fma(-bi, pr, -br * pi);
            }
            if (en.x >= 0) {
                const pc<double> p = V[v_at(en.x, img)];
                const double pr = flip(p.re, (en.z >> 1) & 1), pi = flip(p.im, ((en.z >> 1) ^ en.z) & 1);
                re = fma(ar, pr, fma(-ai, pi, re));
                im = fma(ar, pi, fma(ai, pr, im));
            }
            V[v_at(hb + e, img)] = {re, im};
        }
    }
    __syncthreads();
}

// conj(a) and conj(b) of an image (SO4.py:879-884): {cos psi, g z, g y, g x}, with g = sin psi / r, as
// one rounded quotient (ir = 1 / r and a correction by its remainder), returned.  The rounding of
// these four numbers, l times over at level l, is the largest error of U and dB/dr next to that of
// psi: with sin psi (z (1 / r)) dB/dr was up to 1.2 times as far off (FP64, lmax 6, against 64-bit
// mantissas: 2.24e-15 instead of 1.87e-15 in the 2-norm).  FP32 takes the quotient's remainder into
// the products as well.
template <typename T>
__device__ __forceinline__ T cayley_klein(T sn, T cs, T x, T y, T z, T r, T ir, T (&ck)[4]) {
    const T q = sn * ir, lo = fma(-q, r, sn) * ir, g = q + lo;
    ck[0] = cs;
    ck[1] = sizeof(T) == 8 ? g * z : fma(q, z, lo * z);
    ck[2] = sizeof(T) == 8 ? g * y : fma(q, y, lo * y);
    ck[3] = sizeof(T) == 8 ? g * x : fma(q, x, lo * x);
    return g;
}

constexpr int UT = 256;  // threads of k_plain_u

__global__ void __launch_bounds__(UT) k_plain_u(PlainArgs<double> A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SmallTables st;
    __shared__ double ck[4 * 32], wsf[32];
    const int tid = threadIdx.x;
    if (tid == 0) st = A.st;
    const int nh = A.n_half, c = blockIdx.x, a = A.a0 + c;
    pc<double> *V = (pc<double> *)smem_raw;
    const int m0 = A.img_ptr[a], m1 = A.img_ptr[a + 1];
    // sum over images of w_j f_c V, thread = half entry (at most two each: n_half <= 434)
    double ar[2] = {0.0, 0.0}, ai[2] = {0.0, 0.0};
    __syncthreads();
    for (int base = m0; base < m1; base += 32) {
        const int n = min(32, m1 - base);
        if (tid < 32) {  // Cayley-Klein parameters and weights, lane = image
            double x = 1.0, y = 0.0, z = 0.0, w = 0.0;
            if (tid < n) {
                const int m = base + tid;
                x = A.img_r[3 * m];
                y = A.img_r[3 * m + 1];
                z = A.img_r[3 * m + 2];
                const double r = sqrt(x * x + y * y + z * z);
                if (r < 1e-8) {  // SO4.py:1441 skips r < 1e-8
                    x = 1.0;
                    y = z = 0.0;
                } else {
                    double sf, dsf;
                    cutoff_fn<double>(A.prm.cutoff_id, r, A.rc, sf, dsf);
                    w = A.w_nb[A.img_j[m]] * sf;
                }
            }
            const double r = sqrt(x * x + y * y + z * z);
            double sn, cs, k[4];
            sincos(A.psi_fac * r, &sn, &cs);
            cayley_klein<double>(sn, cs, x, y, z, r, 1.0 / r, k);
#pragma unroll
            for (int i = 0; i < 4; ++i) ck[32 * i + tid] = k[i];
            wsf[tid] = w;
        }
        __syncthreads();
        const int part = n > VI ? (n + 1) / 2 : n;  // the images in one or two near-equal parts
        for (int c0 = 0; c0 < n; c0 += part) {
            const int nc = min(part, n - c0);
            plain_rows<UT>(st, A.vent, ck, c0, nc, V);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int e = tid + q * UT;
                if (e < nh) {
                    double pr[2] = {0.0, 0.0}, pi[2] = {0.0, 0.0};  // even and odd images of this part
#pragma unroll 2
                    for (int i = 0; i < nc; ++i) {
                        const pc<double> v = V[v_at(e, i)];
                        pr[i & 1] = fma(wsf[c0 + i], v.re, pr[i & 1]);
                        pi[i & 1] = fma(wsf[c0 + i], v.im, pi[i & 1]);
                    }
                    ar[q] += pr[0] + pr[1];
                    ai[q] += pi[0] + pi[1];
                }
            }
            __syncthreads();
        }
    }
    // the self term f_c(0) w_site on the diagonal (where F = 1), u_norm, then the full rows
    double f0, df0;
    cutoff_fn<double>(A.prm.cutoff_id, 0.0, A.rc, f0, df0);
    const double selfw = f0 * A.w_site[a];
    pc<double> *ut = A.ut + (size_t)(c >> 5) * A.n_u * 32 + (c & 31);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int e = tid + q * UT;
        if (e < nh) {
            const int w = __ldg(&A.vent[e].w);
            const double un = st.unorm[(w >> 8) & 0xff];
            pc<double> v = {(ar[q] + ((w & 2) ? selfw : 0.0)) * un, ai[q] * un};
            const int2 m = __ldg(A.hfull + e);
            ut[(size_t)m.x * 32] = v;
            if (m.y >= 0) {
                v.im = -v.im;
                if (m.y & (1 << 14)) v = {-v.re, -v.im};
                ut[(size_t)(m.y & 0x3fff) * 32] = v;
            }
        }
    }
}

// FP32: the tiles of 32 centres from the row-chain kernel's sums, which are V already (U divided by F
// here took two more roundings: x at lmax 4 2.84e-7 off instead of 2.5e-7); a CTA per tile, lane =
// centre within a warp.
__global__ void __launch_bounds__(256) k_plain_tile(PlainArgs<float> A) {
    __shared__ float2 s[32 * 33];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, c0 = blockIdx.x * 32, nh = A.n_half;
    const int live = min(32, A.natoms - A.a0 - c0);
    pc<float> *ut = A.ut + (size_t)blockIdx.x * A.n_u * 32 + lane;
    for (int e0 = 0; e0 < nh; e0 += 32) {  // transpose 32 entries x 32 centres
        __syncthreads();
        for (int c = wid; c < live; c += 8)
            if (e0 + lane < nh) s[lane * 33 + c] = A.uh[(size_t)(c0 + c) * nh + e0 + lane];
        __syncthreads();
        for (int i = wid; i < 32 && e0 + i < nh; i += 8) {
            const float2 u = lane < live ? s[i * 33 + lane] : make_float2(0.f, 0.f);
            pc<float> v = {u.x, u.y};
            const int2 m = __ldg(A.hfull + e0 + i);
            ut[(size_t)m.x * 32] = v;
            if (m.y >= 0) {
                v.im = -v.im;
                if (m.y & (1 << 14)) v = {-v.re, -v.im};
                ut[(size_t)(m.y & 0x3fff) * 32] = v;
            }
        }
    }
}

// FP32: V of up to 32 images, lane = image, V[entry][P]; a warp takes a row of the level, the
// previous row's entry ma - 1 stays in registers, so an entry is one shared load, eight
// multiply-adds and one store.
// Pitch of an entry: at 40, four consecutive entries x eight images fill the banks twice, evenly;
// 33 where that does not fit (twol 11 and 12).
__host__ __device__ inline int vp32(int nh) { return nh > 320 ? 33 : 40; }
template <int NT>
__device__ __forceinline__ void plain_rows32(const SmallTables &st, const float *ck, pc<float> *V, int P) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const float ar = ck[lane], ai = ck[32 + lane], br = ck[64 + lane], bi = ck[96 + lane];
    if (wid == 0) V[lane] = {1.f, 0.f};
    for (int l = 1; l <= st.twol; ++l) {
        __syncthreads();
        const int L = l - 1;
        for (int mb = wid; 2 * mb <= l; mb += NT / 32) {
            pc<float> *out = V + (size_t)(st.h_block[l] + mb * (l + 1)) * P + lane;
            // row mb of level L, or its mirror (-1)^(mb + c) conj of row L - mb read backwards
            const bool mir = 2 * mb > L;
            const pc<float> *in = V + (size_t)(st.h_block[L] + (mir ? (L - mb) * l + L : mb * l)) * P + lane;
            const int step = mir ? -P : P;
            float sg = (mir && (mb & 1)) ? -1.f : 1.f;
            float pr = 0.f, pi = 0.f;
            for (int ma = 0; ma <= l; ++ma) {
                float cr = 0.f, ci = 0.f;
                if (ma < l) {
                    const pc<float> v = in[ma * step];
                    cr = sg * v.re;
                    ci = mir ? -sg * v.im : v.im;
                    if (mir) sg = -sg;
                }
                float re = fmaf(ar, cr, -(ai * ci)), im = fmaf(ar, ci, ai * cr);
                re = fmaf(-br, pr, fmaf(bi, pi, re));
                im = fmaf(-br, pi, fmaf(-bi, pr, im));
                out[ma * P] = {re, im};
                pr = cr;
                pi = ci;
            }
        }
    }
    __syncthreads();
}

// ---------------------------------------------------------------- Z' and B
// Z' of centre c of the pass: its elements stand ZQ apart, those of ZQ centres side by side, a
// sector of 32 bytes.  k_plain_z stores a centre per lane, the derivative kernels gather one
// centre's elements.  8,000 atoms, k_plain_z + k_plain_d at ZQ = 32 / a sector / 1: FP32 lmax 3
// 405 / 391 / 414 us, lmax 4 1,248 / 1,081 / 1,178; FP64 lmax 3 2,193 / 2,214 / 2,216, lmax 4
// 5,590 / 5,490 / 5,477.
template <typename T>
constexpr int ZQ = 32 / sizeof(pc<T>);
template <typename T>
__device__ __forceinline__ pc<T> *plain_zt(const PlainArgs<T> &A, int c) {
    return A.zt + (size_t)(c / ZQ<T>) * ZQ<T> * A.n_z + c % ZQ<T>;
}

// One Z unit (so4_tables.cu) of 32 centres, lane = centre, for N levels: the products
// V_l1 V_l2 are formed once for all of them.
template <typename T, int N>
__device__ __forceinline__ void plain_z_unit(const int4 q0, const int4 q1, const int4 q2, const T *__restrict__ cat,
                                             const T *__restrict__ cbt, const pc<T> *__restrict__ U, pc<T> *Z) {
    const int u1 = q0.x & 0xffff, u2 = (int)((unsigned)q0.x >> 16), na = q0.y & 0xff, nb = (q0.y >> 8) & 0xff;
    const int r1 = q1.x & 0xffff, r2 = (int)((unsigned)q1.x >> 16), pitch = q1.y;
    T zr[N], zi[N];
#pragma unroll
    for (int j = 0; j < N; ++j) zr[j] = zi[j] = T(0);
    const T *cb = cbt + q0.w;
    for (int ib = 0; ib < nb; ++ib, cb += pitch) {
        T tr[N], ti[N];
#pragma unroll
        for (int j = 0; j < N; ++j) tr[j] = ti[j] = T(0);
        const pc<T> *p1 = U + (size_t)(u1 + ib * r1) * 32, *p2 = U + (size_t)(u2 - ib * r2) * 32;
        const T *ca = cat + q0.z;
#pragma unroll 2
        for (int ia = 0; ia < na; ++ia, ca += pitch) {
            const pc<T> a = p1[ia * 32], b = p2[-ia * 32];
            const T pr = fma(a.re, b.re, -(a.im * b.im)), pi = fma(a.re, b.im, a.im * b.re);
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const T c = __ldg(ca + j);
                tr[j] = fma(c, pr, tr[j]);
                ti[j] = fma(c, pi, ti[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const T c = __ldg(cb + j);
            zr[j] = fma(c, tr[j], zr[j]);
            zi[j] = fma(c, ti[j], zi[j]);
        }
    }
    const int out[PZ_G] = {q1.z, q1.w, q2.x, q2.y};
#pragma unroll
    for (int j = 0; j < N; ++j) Z[(size_t)out[j] * ZQ<T>] = {zr[j], zi[j]};
}

constexpr int ZT = 256;  // threads of k_plain_z

// CTA (tile, part): the units wid + 8 part, + 8 parts, .. (most expensive first) of 32 centres.
template <typename T>
__global__ void __launch_bounds__(ZT) k_plain_z(PlainArgs<T> A) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const pc<T> *U = A.ut + (size_t)blockIdx.x * A.n_u * 32 + lane;
    pc<T> *Z = plain_zt(A, blockIdx.x * 32 + lane);
    for (int u = wid + (ZT / 32) * blockIdx.y; u < A.n_unit; u += (ZT / 32) * gridDim.y) {
        const int4 q0 = __ldg(A.unit + 3 * u), q1 = __ldg(A.unit + 3 * u + 1), q2 = __ldg(A.unit + 3 * u + 2);
        switch (q0.y >> 16) {
            case 4: plain_z_unit<T, 4>(q0, q1, q2, A.ca, A.cb, U, Z); break;
            case 3: plain_z_unit<T, 3>(q0, q1, q2, A.ca, A.cb, U, Z); break;
            case 2: plain_z_unit<T, 2>(q0, q1, q2, A.ca, A.cb, U, Z); break;
            default: plain_z_unit<T, 1>(q0, q1, q2, A.ca, A.cb, U, Z); break;
        }
    }
}

// B_k = 2 Re sum' conj(U_l) Z (an even level's section ends at the middle-row centre, weight
// 1/2), a warp per (32 centres, component), lane = centre.
template <typename T>
__global__ void __launch_bounds__(256) k_plain_b(PlainArgs<T> A) {
    const int lane = threadIdx.x & 31, k = blockIdx.y * 8 + (int)(threadIdx.x >> 5);
    const int a = A.a0 + blockIdx.x * 32 + lane;
    if (k >= A.n_b) return;
    const int4 b = __ldg(A.blk + __ldg(A.bblk + k));
    const int lam = b.w, cnt = b.z;
    const pc<T> *u = A.ut + ((size_t)blockIdx.x * A.n_u + A.st.u_block[lam]) * 32 + lane;
    const pc<T> *z = plain_zt(A, blockIdx.x * 32 + lane) + (size_t)b.y * ZQ<T>;
    // four sums side by side: half the rounding of one of up to 49 terms (x at lmax 6 5.6e-16
    // instead of 6.0e-16 off)
    T s4[4] = {T(0), T(0), T(0), T(0)};
    const int full = (lam & 1) ? cnt : cnt - 1;
    for (int e = 0; e < full; e += 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (e + i < full) {
                const pc<T> p = u[(size_t)(e + i) * 32], q = z[(size_t)(e + i) * ZQ<T>];
                s4[i] = fma(p.re, q.re, fma(p.im, q.im, s4[i]));
            }
    }
    T s = (s4[0] + s4[1]) + (s4[2] + s4[3]);
    if (full < cnt) {
        const pc<T> p = u[(size_t)full * 32], q = z[(size_t)full * ZQ<T>];
        s += T(0.5) * (p.re * q.re + p.im * q.im);
    }
    if (a < A.natoms) A.x[(size_t)a * A.n_b + k] = T(2) * s;
}

// 1 / v in FP64, rounded to FP32: two Newton steps from FP32's quotient instead of an FP64 division
// (some thirty instructions of a pipe with 1/64 of the FP32 rate, in the one warp that the CTA waits
// for).  The first leaves 2^-46, the second FP64's own rounding.
__device__ __forceinline__ float inv32(double v) {
    const float f = (float)v;
    if (!(f > 1e-37f && f < 1e37f)) return (float)(1.0 / v);
    double y = (double)(1.f / f);
    y = fma(fma(-v, y, 1.0), y, y);
    y = fma(fma(-v, y, 1.0), y, y);
    return (float)y;
}

// ---------------------------------------------------------------- dB/dr
// What the images of one pass need (warp 0, lane = image base + lane of n): conj(a), conj(b),
// the 3 x 4 matrix q that takes (P0..P3) to t = dB/dr, and rv = (R_i + r) / vol (r / vol for an
// image of the centre itself).  j is the image's neighbour (-1 past n).
// With n the unit vector, M = cos psi + i sin psi m . sigma, m = (-n_x, -n_y, n_z), and
// X_c = i v_c . sigma, v_c = (gamma, beta, alpha):
//   v_c = (psi' - sin cos / r) n_c m + (sin cos / r) D e_c + (sin^2 / r) m x D e_c,
// D = diag(-1, -1, 1), psi' = dpsi/dr.
template <typename T>
__device__ __forceinline__ void plain_image(const PlainArgs<T> &A, int a, int m, bool in, T inv_vol, int j, T (&ck)[4],
                                            T (&q)[12], T (&rv)[3]) {
    T x = T(1), y = T(0), z = T(0), w = T(0);
    if (in) {
        x = (T)A.img_r[3 * m];
        y = (T)A.img_r[3 * m + 1];
        z = (T)A.img_r[3 * m + 2];
    }
    T r = sqrt(x * x + y * y + z * z);
    const bool live = in && !(r < T(1e-8));  // SO4.py:1441
    if (live) w = (T)A.w_nb[j];
    if (!live) {
        x = r = T(1);
        y = z = T(0);
    }
    T sf, dsf, sn, cs;
    cutoff_fn<T>(A.prm.cutoff_id, r, A.rc, sf, dsf);
    // psi as the U_tot kernels round it: its error moves U and dU/dr alike, and most of it cancels (with
    // what it lost put back in here alone FP32 dB/dr at lmax 6 was 1.4e-6 off instead of 1.1e-6)
    if (sizeof(T) == 8) {
        double s_, c_;
        sincos((double)(A.psi_fac * r), &s_, &c_);
        sn = (T)s_;
        cs = (T)c_;
    } else {
        float s_, c_;
        sincosf((float)(A.psi_fac * r), &s_, &c_);
        sn = (T)s_;
        cs = (T)c_;
    }
    const T ir = T(1) / r;
    auto unit = [&](T v) {  // v / r, rounded once
        const T q = v * ir;
        return fma(fma(-q, r, v), ir, q);
    };
    const T n[3] = {unit(x), unit(y), unit(z)};
    const T sr = cayley_klein<T>(sn, cs, x, y, z, r, ir, ck);
    const T ws = w * sf, wd = w * dsf;
    const T u = ws * (sr * cs), v = ws * (sr * sn), p = fma(ws, A.psi_fac, -u);
    const T md[3] = {-n[0], -n[1], n[2]};  // m
    const T vm[3] = {v * md[0], v * md[1], v * md[2]};
    const T cross[3][3] = {{T(0), -vm[2], vm[1]}, {vm[2], T(0), -vm[0]}, {vm[1], -vm[0], T(0)}};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const T pk = p * n[k];
        q[4 * k] = wd * n[k];
#pragma unroll
        for (int c = 0; c < 3; ++c) {  // alpha, beta, gamma = components 2, 1, 0 of v
            T t = fma(pk, md[c], cross[k][c]);
            if (c == k) t += (k < 2) ? -u : u;
            q[4 * k + 3 - c] = t;
        }
        const T ri = (k == 0) ? x : (k == 1 ? y : z);
        rv[k] = (j == a ? ri : (T)A.pos[3 * a + k] + ri) * inv_vol;
    }
}

// Runs of images of one pair among a pass's images, cut into parts of `part` images: pid per
// image, run[h] the runs' first images (and the end), cont[h] whether part h's first run goes
// on with a pair begun before it.  Warp 0; npair counts the distinct neighbours so far.
struct PlainRuns {
    int run[2][33], nrun[2], cont[2], pid[32];
};
__device__ __forceinline__ void plain_runs(PlainRuns &R, int n, int part, int j, bool fresh, int a, int p0,
                                           bool self_img, int &npair) {
    const int lane = threadIdx.x & 31;
    const unsigned fm = __ballot_sync(0xffffffffu, fresh), upto = 0xffffffffu >> (31 - lane);
    // the pairs are the distinct neighbours in order, with (i, i) among them also without images
    if (lane < n) R.pid[lane] = p0 + npair + __popc(fm & upto) - 1 + ((j > a && !self_img) ? 1 : 0);
    npair += __popc(fm);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int lo = h * part, hi = min(n, lo + part);
        const bool first = lane >= lo && lane < hi && (fresh || lane == lo);
        const unsigned sm = __ballot_sync(0xffffffffu, first);
        if (first) R.run[h][__popc(sm & upto) - 1] = lane;
        if (lane == 0) {
            R.nrun[h] = __popc(sm);
            R.run[h][__popc(sm)] = hi;
            R.cont[h] = lo < n && !((fm >> lo) & 1);
        }
    }
}

// The (i, i) row of component k from the other pairs' sum d; rdxdr's row holds the images of
// the centre itself (self_img) already.
template <typename T>
__device__ __forceinline__ void plain_self_row(const PlainArgs<T> &A, int a, int ns, int k, T inv_vol, const T (&d)[3],
                                               bool self_img) {
    T *dx = A.dxdr + ((size_t)ns * A.n_b + k) * 3;
#pragma unroll
    for (int q = 0; q < 3; ++q) dx[q] = d[q];
    if (A.want_stress) {
        T *rd = A.rdxdr + ((size_t)ns * A.n_b + k) * 9;
#pragma unroll
        for (int aa = 0; aa < 3; ++aa)
#pragma unroll
            for (int q = 0; q < 3; ++q)
                rd[3 * aa + q] = fma((T)A.pos[3 * a + aa] * inv_vol, d[q], self_img ? rd[3 * aa + q] : T(0));
    }
}

// FP64.  The products P_g of a level are one matrix product [W: (block, g)] [V: images] per
// centre, 17,768 multiply-adds per image at lmax 4 (60 % of the path's FP64 work, and FP64
// runs at 1/64 of the FP32 rate here).  It runs on the tensor cores on integers cut into
// signed 8-bit digits (the error-free splitting of Ozaki, Ogita, Oishi and Rump, Numer.
// Algorithms 59, 95 (2012)): V is rounded once to 61 bits relative to its bound and Z' to 55
// or more relative to the component's largest entry, W formed from Z' in integers, the digits are
// exact in FP16, and the sums of the digit products p + q = s < ND stay below 2^24, exact in
// the FP32 accumulators.  Each component's P_g is summed over its blocks as integers (any
// order gives the same bits, so warps add with shared-memory atomics) and converted once.
// Both integers are scaled entry by entry with the power of two next to F: with one per row the
// rounding grew with the range of F within a row (dB/dr at lmax 6 was 5.8e-15 off).  In an
// emulation with 64-bit mantissas, stage by stage, this rounding alone puts dB/dr 2e-17 off; what is
// left are the image's psi and Cayley-Klein parameters, 1.5e-15 at lmax 4 and 2.0e-15 at lmax 6.
constexpr int DT = 192;    // threads: two CTAs per SM with 168 registers each
constexpr int ND = 8;      // digits
constexpr int VB = 61, ZB = 62;  // bits of V and W
constexpr int VS = 1;  // |V| 2^exponent <= 2: |U| <= 1, and both powers of two are within sqrt(2)
// The integer of P counts units of 2^66 of the product of V's and W's integers.  By the norms of
// U's rows a block's |V| sum to 2^60 x 25.3 at most (twol 12), and |W| <= 2^62.5: a component's
// three blocks stay below 2^62.8.
constexpr int PSH = 66;
constexpr int EMIN = -900;  // smallest exponent a component is scaled by
constexpr int KBAD = 1 << 20;  // the exponent of a component with Inf or NaN in its Z'

__device__ __forceinline__ void mma_f16(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The digits of re and im as FP16 pairs, most significant first: with 128 added to every byte,
// byte b is the digit b - 128, and 0x6400 | b is 1024 + b.  Bytes of re and im are interleaved
// first, so that one permutation makes a pair's two halves.
__device__ __forceinline__ unsigned digit_pair(unsigned w, int hi) {
    const unsigned t = __byte_perm(w, 0x64646464u, hi ? 0x4342 : 0x4140);
    const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&t), __floats2half2_rn(1152.f, 1152.f));
    return *reinterpret_cast<const unsigned *>(&h);
}
__device__ __forceinline__ void digits(unsigned long long re, unsigned long long im, unsigned (&d)[ND]) {
    re += 0x8080808080808080ULL;
    im += 0x8080808080808080ULL;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const unsigned wr = (unsigned)(h ? re : re >> 32), wi = (unsigned)(h ? im : im >> 32);
        const unsigned top = __byte_perm(wr, wi, 0x7362), low = __byte_perm(wr, wi, 0x5140);
        d[4 * h] = digit_pair(top, 1);
        d[4 * h + 1] = digit_pair(top, 0);
        d[4 * h + 2] = digit_pair(low, 1);
        d[4 * h + 3] = digit_pair(low, 0);
    }
}
// acc + x c for a small unsigned c, modulo 2^64
__device__ __forceinline__ unsigned long long mad64(unsigned long long acc, unsigned long long x, unsigned c) {
    acc += (unsigned long long)(unsigned)x * c;
    return acc + ((unsigned long long)((unsigned)(x >> 32) * c) << 32);
}
// sum_s acc_s 2^(46 - 8 s), its last terms rounded: acc_s are integers of at most 2^24 (the
// first two far smaller, their leading digits being below 2^6)
__device__ __forceinline__ long long combine(const float (&acc)[ND][4], int c) {
    int a[ND];
#pragma unroll
    for (int s = 0; s < ND; ++s) a[s] = __float2int_rn(acc[s][c]);
    long long v = (long long)(a[0] * 256 + a[1]) << 38;
    v += (long long)a[2] * (1 << 30);
    v += (long long)a[3] * (1 << 22);
    v += (long long)a[4] * (1 << 14);
    v += (long long)a[5] * (1 << 6);
    return v + ((a[6] + ((a[7] + 128) >> 8) + 2) >> 2);
}
// x 2^e by exponent arithmetic (no FP64 instruction), x and x 2^e normal; zero (and anything
// denormal) becomes a value below 2^(e - 1000)
__device__ __forceinline__ double mul2(double x, int e) {
    return __hiloint2double(__double2hiint(x) + (e << 20), __double2loint(x));
}

struct D64Smem {
    int cb;  // pitch of a row of C: n_b rounded up to odd
    size_t z, c, par, c00, kex, total;
    __host__ __device__ D64Smem(int nh, int nz, int nB, bool zs) {
        cb = nB | 1;
        z = sizeof(pc<double>) * (size_t)nh * VI;
        c = z + (zs ? sizeof(longlong2) * (size_t)nz : 0);
        // C: low and high words [4][VI][cb]; afterwards the slots' sums of the (i, i) row
        const size_t nc = 4 * VI * (size_t)cb;
        par = c + ((8 * (nc > 3 * DT ? nc : 3 * DT) + 15) & ~(size_t)15);
        c00 = par + sizeof(double) * 32 * 19;
        kex = c00 + sizeof(long long) * (size_t)nB;
        total = (kex + sizeof(int) * (size_t)nB + 15) & ~(size_t)15;
    }
};

// ZS: the integers of Z' in shared memory, else in this centre's global slot (read through L1).
template <bool ZS>
__global__ void __launch_bounds__(DT, 2) k_plain_d64(PlainArgs<double> A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SmallTables st;
    __shared__ int4 lamt[SO4_LDIM_MAX];
    __shared__ PlainRuns R;
    __shared__ int s_unit;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) st = A.st;
    if (tid <= A.st.twol) lamt[tid] = __ldg(A.lam + tid);
    const int nh = A.n_half, nz = A.n_z, nB = A.n_b, c = blockIdx.x, a = A.a0 + c;
    const D64Smem L(nh, nz, nB, ZS);
    const int CB = L.cb;
    pc<double> *V = (pc<double> *)smem_raw;
    longlong2 *Vi = (longlong2 *)V;
    const pc<double> *Zt = plain_zt(A, c);
    longlong2 *Zi = ZS ? (longlong2 *)(smem_raw + L.z) : A.zi + (size_t)c * nz;
    unsigned *Cl = (unsigned *)(smem_raw + L.c);
    int *Ch = (int *)Cl + 4 * VI * CB;
    double *par = (double *)(smem_raw + L.par);
    long long *c00 = (long long *)(smem_raw + L.c00);  // level-0 part of P_0, the same for every image
    int *kex = (int *)(smem_raw + L.kex);              // exponent of each component
    for (int q = tid; q < nB; q += DT) {
        c00[q] = 0;
        kex[q] = EMIN;
    }
    __syncthreads();

    const int m0 = A.img_ptr[a], m1 = A.img_ptr[a + 1], p0 = A.pair_ptr[a], ns = A.nsite[a];
    const bool self_img = A.pair_img[ns] < A.pair_img[ns + 1];
    int npair = 0;
    // warp 0: the set-up of up to 32 images, and how they fall into pairs
    auto setup = [&](int base, int n, int part) {
        const int m = base + lane;
        const int j = lane < n ? A.img_j[m] : -1;
        const bool fresh = lane < n && (m == m0 || A.img_j[m - 1] != j);
        double ck[4], q[12], rv[3];
        plain_image<double>(A, a, m, lane < n, 1.0 / A.geom[A.astruct[a]].vol, j, ck, q, rv);
#pragma unroll
        for (int i = 0; i < 4; ++i) par[32 * i + lane] = ck[i];
#pragma unroll
        for (int i = 0; i < 12; ++i) par[128 + 32 * i + lane] = q[i];
#pragma unroll
        for (int i = 0; i < 3; ++i) par[512 + 32 * i + lane] = rv[i];
        plain_runs(R, n, part, j, fresh, a, p0, self_img, npair);
    };
    // ---- Z' as integers relative to each component's largest entry: the values into their
    // slots and the components' exponents (warps 1.., while warp 0 sets up the first images),
    // then the integers in place
    if (wid == 0) {
        const int n = min(32, m1 - m0);
        setup(m0, n, n > VI ? (n + 1) / 2 : n);
    } else {
        constexpr int NQ = DT - 32, RQ = 7;
        for (int q0 = 0; q0 < nz; q0 += RQ * NQ) {
            pc<double> v[RQ];
            int ze[RQ];
#pragma unroll
            for (int r = 0; r < RQ; ++r) {
                const int q = q0 + r * NQ + tid - 32;
                ze[r] = q < nz ? __ldg(A.zent + q) : -1;
                if (q < nz) v[r] = Zt[(size_t)q * ZQ<double>];
            }
#pragma unroll
            for (int r = 0; r < RQ; ++r) {
                int ex = EMIN, k = -1;
                if (ze[r] >= 0) {
                    const int b = ze[r] & 0xffff;
                    ((pc<double> *)Zi)[q0 + r * NQ + tid - 32] = v[r];
                    k = __ldg(&A.blk[b].x);
                    const int hf = __double2hiint(__ldg(A.fac + b));
                    const unsigned top = max((unsigned)__double2hiint(v[r].re) & 0x7fffffffu,
                                             (unsigned)__double2hiint(v[r].im) & 0x7fffffffu);
                    // f v 2^-row < 2^ex: the exponents, and one less where the leading 11 bits of
                    // the mantissas, rounded up, multiply to less than 2; Inf and NaN far above
                    const unsigned mant = (((top >> 10) & 0x3ff) + 0x401) * (((hf >> 10) & 0x3ff) + 0x401);
                    ex = top >= 0x7ff00000u
                             ? KBAD
                             : (int)(top >> 20) + (hf >> 20) - 2044 - ((ze[r] >> 16) - 64) - (mant < (1u << 21) ? 1 : 0);
                }
                const unsigned peers = __match_any_sync(0xffffffffu, k);
                const int big = __reduce_max_sync(peers, ex);
                if (k >= 0 && lane == __ffs(peers) - 1) atomicMax(kex + k, big);
            }
        }
    }
    __syncthreads();
    const int bz = ZB - A.cw;
    // P = integer x 2^(psh + kex), for g = 0 2^-cw and else 2^-2 less (W is Z' x 2^cw, and x 4)
    const int psh = PSH - (VB - VS) - bz;
    for (int q0 = tid; q0 < nz; q0 += 4 * DT) {
        pc<double> v[4];
        int4 bk[4];
        int ex[4], row[4];
        double f[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int q = q0 + r * DT;
            if (q >= nz) break;
            const int ze = __ldg(A.zent + q), b = ze & 0xffff;
            v[r] = ((const pc<double> *)Zi)[q];
            bk[r] = __ldg(A.blk + b);
            f[r] = __ldg(A.fac + b);
            row[r] = (ze >> 16) - 64;
            ex[r] = kex[bk[r].x];
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int q = q0 + r * DT;
            if (q >= nz) break;
            const double s = ex[r] >= KBAD ? 0.0 : mul2(f[r], bz - ex[r] - row[r]);
            longlong2 z;
            z.x = __double2ll_rn(v[r].re * s);
            z.y = __double2ll_rn(v[r].im * s);
            Zi[q] = z;
            if (bk[r].w == 0 && ex[r] < KBAD) c00[bk[r].x] = __double2ll_rn(v[r].re * mul2(f[r], A.cw - psh - ex[r] - 1));
        }
    }

    const int nslot = DT / nB, slot = tid / nB, k = tid - slot * nB;
    double dsum[3] = {0.0, 0.0, 0.0};
    // the (i, i) row takes the centre's own images as they come
    if (self_img && A.want_stress)
        for (int q = tid; q < 9 * nB; q += DT) A.rdxdr[(size_t)ns * nB * 9 + q] = 0.0;
    // units of four blocks of one level (16 rows: block, g), largest level first
    int nunit = 0;
    __syncthreads();
    for (int lam = 1; lam <= st.twol; ++lam) nunit += (lamt[lam].z + 3) / 4;
    const int g4 = (lane >> 2) & 3;

    for (int base = m0; base < m1; base += 32) {
        const int n = min(32, m1 - base), part = n > VI ? (n + 1) / 2 : n;
        if (base != m0) {
            if (wid == 0) setup(base, n, part);
            __syncthreads();
        }
        for (int h = 0; h * part < n; ++h) {
            const int c0 = h * part, nc = min(part, n - c0);
            plain_rows<DT>(st, A.vent, par, c0, nc, V);
            // V to integers (the half weight of a middle row's centre with it), zeros up to the
            // column tiles' ends
            const int sh = nc > 8 ? 4 : 3;
            for (int t = tid; t < nh << sh; t += DT) {
                const int e = t >> sh, i = t & ((1 << sh) - 1), at = v_at(e, i);
                const int w = __ldg(&A.vent[e].w), ex = VB - VS + (w >> 16) - 64 - (w & 1);
                longlong2 z = {0, 0};
                if (i < nc) {
                    const pc<double> v = V[at];
                    z.x = __double2ll_rn(mul2(v.re, ex));
                    z.y = __double2ll_rn(mul2(v.im, ex));
                }
                Vi[at] = z;
            }
            for (int q = tid; q < 8 * VI * CB; q += DT) Cl[q] = 0;
            if (tid == 0) s_unit = 0;
            __syncthreads();
            // ---- P_g of every block
            for (;;) {
                int u = 0;
                if (lane == 0) u = atomicAdd(&s_unit, 1);
                u = __shfl_sync(0xffffffffu, u, 0);
                if (u >= nunit) break;
                int lam = st.twol;
                while (u >= (lamt[lam].z + 3) / 4) u -= (lamt[lam--].z + 3) / 4;
                const int4 lt = lamt[lam];
                const int E = lt.x, nb = lt.z, hb = st.h_block[lam];
                const int *sent = A.sent + lt.w;
                const int bl[2] = {4 * u + (lane >> 4), 4 * u + (lane >> 4) + 2};
                int4 bk[2];
#pragma unroll
                for (int r = 0; r < 2; ++r) bk[r] = __ldg(A.blk + lt.y + min(bl[r], nb - 1));
                float acc[2][ND][4];
#pragma unroll
                for (int ct = 0; ct < 2; ++ct)
#pragma unroll
                    for (int s = 0; s < ND; ++s)
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc[ct][s][i] = 0.f;
                for (int e0 = 0; e0 < E; e0 += 8) {
                    unsigned da[ND][4];
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        const int e = e0 + 4 * hf + (lane & 3), ec = min(e, E - 1);
                        const int se = __ldg(sent + ec), ma = se & 0xff;
                        const bool ctr = (se >> 8) & 1;
                        // W = p X -+ m Y: X = Y = Z'[m] (g = 0: p = 2^cw, m = 0; g = 1), else
                        // X = Z'[m+1], Y = Z'[m-1] (at the centre X is the mirror -conj(Y)), on
                        // their own scales; a neighbour past a row's end has weight 0, the clamps
                        // keep it in the block
                        const int sx = g4 >= 2 ? (se >> 16) & 15 : 2, sy = g4 >= 2 ? (se >> 20) & 15 : 2;
                        unsigned wp = g4 == 0 ? 1u << A.cw : (unsigned)(lam - ma) << sx;
                        unsigned wm = g4 == 0 ? 0u : (unsigned)ma << sy;
                        if (e >= E) wp = wm = 0;
                        const int iy = g4 >= 2 ? max(ec - 1, 0) : ec;
                        const int ix = g4 >= 2 ? (ctr ? iy : min(ec + 1, E - 1)) : ec;
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            longlong2 x = Zi[bk[r].y + ix], y = Zi[bk[r].y + iy];
                            if (g4 >= 2 && ctr) x.x = -x.x;
                            if (g4 != 3) {
                                y.x = -y.x;
                                y.y = -y.y;
                            }
                            const unsigned long long wr = mad64(mad64(0, x.x, wp), y.x, wm);
                            const unsigned long long wi = mad64(mad64(0, x.y, wp), y.y, wm);
                            unsigned dw[ND];
                            digits((g4 & 1) ? wi : wr, (g4 & 1) ? 0ULL - wr : wi, dw);  // -i W for g = 1, 3
#pragma unroll
                            for (int p = 0; p < ND; ++p) da[p][2 * hf + r] = dw[p];
                        }
                    }
#pragma unroll
                    for (int ct = 0; ct < 2; ++ct) {
                        if (ct == 1 && nc <= 8) continue;
                        unsigned db[2][ND];
#pragma unroll
                        for (int hf = 0; hf < 2; ++hf) {
                            const int ec = min(e0 + 4 * hf + (lane & 3), E - 1);
                            const longlong2 v = Vi[v_at(hb + ec, 8 * ct + (lane >> 2))];
                            digits(v.x, v.y, db[hf]);
                        }
#pragma unroll
                        for (int p = 0; p < ND; ++p)
#pragma unroll
                            for (int q = 0; q < ND - p; ++q) mma_f16(acc[ct][p + q], da[p], db[0][q], db[1][q]);
                    }
                    // 128 real terms at most before a digit sum could pass 2^24
                    const bool flush = (e0 & 63) == 56, last = e0 + 8 >= E;
                    if (flush || last) {
#pragma unroll
                        for (int ct = 0; ct < 2; ++ct) {
                            if (ct == 1 && nc <= 8) continue;
#pragma unroll
                            for (int r = 0; r < 2; ++r) {
                                if (bl[r] >= nb) continue;
                                const int at = (g4 * VI + 8 * ct + 2 * (lane & 3)) * CB + bk[r].x;
#pragma unroll
                                for (int i = 0; i < 2; ++i) {
                                    const long long v = combine(acc[ct], 2 * r + i);
                                    const unsigned lo = (unsigned)v, old = atomicAdd(Cl + at + i * CB, lo);
                                    atomicAdd(Ch + at + i * CB, (int)(v >> 32) + (old + lo < lo ? 1 : 0));
                                }
                            }
#pragma unroll
                            for (int s = 0; s < ND; ++s)
#pragma unroll
                                for (int i = 0; i < 4; ++i) acc[ct][s][i] = 0.f;
                        }
                    }
                }
            }
            __syncthreads();
            // ---- rows: thread = (slot, component), slots over the pairs of these images
            if (slot < nslot) {
                const int kx = kex[k], ek = kx + psh;
                const bool bad = kx >= KBAD;
                const long long z0 = c00[k];
                for (int rr = slot; rr < R.nrun[h]; rr += nslot) {
                    double D[3], E[9];
                    const int i0 = R.run[h][rr], i1 = R.run[h][rr + 1];
                    auto image = [&](int i, bool first) {
                        double p[4], t[3];
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            const int at = (g * VI + i - c0) * CB + k;
                            const long long v = ((long long)Ch[at] << 32) + Cl[at] + (g == 0 ? z0 : 0);
                            p[g] = bad ? NAN : (v == 0 ? 0.0 : mul2((double)v, g == 0 ? ek - A.cw : ek - 2));
                        }
#pragma unroll
                        for (int q = 0; q < 3; ++q) {
                            const double *o = par + 128 + 128 * q + i;
                            t[q] = fma(o[0], p[0], fma(o[32], p[1], fma(o[64], p[2], o[96] * p[3])));
                            D[q] = first ? t[q] : D[q] + t[q];
                        }
                        if (A.want_stress) {
#pragma unroll
                            for (int aa = 0; aa < 3; ++aa) {
                                const double rv = par[512 + 32 * aa + i];
#pragma unroll
                                for (int q = 0; q < 3; ++q)
                                    E[3 * aa + q] = first ? rv * t[q] : fma(rv, t[q], E[3 * aa + q]);
                            }
                        }
                    };
                    image(i0, true);
                    for (int i = i0 + 1; i < i1; ++i) image(i, false);
                    const int p = R.pid[i0];
                    if (p == ns) {
                        if (A.want_stress) {
                            double *rd = A.rdxdr + ((size_t)ns * nB + k) * 9;
#pragma unroll
                            for (int q = 0; q < 9; ++q) rd[q] += E[q];
                        }
                        continue;
                    }
                    const bool add = rr == 0 && R.cont[h];
                    double *dx = A.dxdr + ((size_t)p * nB + k) * 3;
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        dsum[q] += D[q];
                        dx[q] = add ? dx[q] + D[q] : D[q];
                    }
                    if (A.want_stress) {
                        double *rd = A.rdxdr + ((size_t)p * nB + k) * 9;
#pragma unroll
                        for (int q = 0; q < 9; ++q) rd[q] = add ? rd[q] + E[q] : E[q];
                    }
                }
            }
            __syncthreads();
        }
    }
    // ---- the (i, i) row: minus the sum of the others
    const double inv_vol = 1.0 / A.geom[A.astruct[a]].vol;
    double *Ds = (double *)Cl;
    if (slot < nslot)
        for (int q = 0; q < 3; ++q) Ds[(slot * nB + k) * 3 + q] = dsum[q];
    __syncthreads();
    for (int kk = tid; kk < nB; kk += DT) {
        double d[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            double s = 0.0;
            for (int w = 0; w < nslot; ++w) s += Ds[(w * nB + kk) * 3 + q];
            d[q] = -s;
        }
        plain_self_row<double>(A, a, ns, kk, inv_vol, d, self_img);
    }
}

// FP32.  The threads form W of a batch of components' entries in shared memory; then a warp
// takes a component, its four groups of eight lanes every fourth entry and four images a lane:
// six shared loads for 4 entries x 32 images (with an entry at a time and an image per lane it
// was three loads of as many wavefronts for 1 x 32), and the groups' sums are exchanged so that
// every lane ends with one image's P and forms its t.
constexpr int ST = 256;     // threads
constexpr int WCAP = 1024;  // entries of a batch: whole components, at least one

// Batches of positions in the longest-first order of components: batch b holds [k[b], k[b + 1])
struct PlainBatches {
    int n, k[24];
};

struct D32Smem {
    int cb, wcap;  // pitch of a row of t: n_b rounded up to odd; entries of the W buffer
    size_t t, w, vrow, par, total;
    __host__ __device__ D32Smem(int nh, int nz, int nB, int emax) {
        cb = nB | 1;
        wcap = nz < WCAP ? nz : (3 * emax > WCAP ? 3 * emax : WCAP);
        // V, and over it the warps' row buffers (9 floats per component) or partial (i, i) sums
        const size_t v = sizeof(pc<float>) * (size_t)nh * vp32(nh), s = sizeof(float) * 9 * (size_t)nB * (ST / 32);
        w = ((v > s ? v : s) + 15) & ~(size_t)15;
        vrow = w + sizeof(float) * 8 * (size_t)wcap;
        t = vrow + sizeof(int) * (size_t)wcap;
        par = t + sizeof(float) * 3 * 32 * (size_t)cb;
        total = (par + sizeof(float) * 32 * 19 + 15) & ~(size_t)15;
    }
};

// KS: components per lane in the row phase, 32 KS >= n_b
template <int KS>
__global__ void __launch_bounds__(ST, KS == 1 ? 3 : 2) k_plain_d32(PlainArgs<float> A, int emax, PlainBatches Bt) {
    const int P = vp32(A.n_half);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SmallTables st;
    __shared__ PlainRuns R;
    __shared__ int s_comp;
    __shared__ float inv_s;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) st = A.st;
    const int nB = A.n_b, c = blockIdx.x, a = A.a0 + c;
    const D32Smem L(A.n_half, A.n_z, nB, emax);
    const int CB = L.cb;
    pc<float> *V = (pc<float> *)smem_raw;
    float4 *W = (float4 *)(smem_raw + L.w);
    int *vrow = (int *)(smem_raw + L.vrow);
    float *t3 = (float *)(smem_raw + L.t), *par = (float *)(smem_raw + L.par);
    const pc<float> *Zt = plain_zt(A, c);
    const int m0 = A.img_ptr[a], m1 = A.img_ptr[a + 1], p0 = A.pair_ptr[a], ns = A.nsite[a];
    const bool self_img = A.pair_img[ns] < A.pair_img[ns + 1];
    // the (i, i) row takes the centre's own images as they come
    if (self_img && A.want_stress)
        for (int q = tid; q < 9 * nB; q += ST) A.rdxdr[(size_t)ns * nB * 9 + q] = 0.f;
    float dsum[KS][3];
#pragma unroll
    for (int s = 0; s < KS; ++s) dsum[s][0] = dsum[s][1] = dsum[s][2] = 0.f;
    int npair = 0;
    // W of a batch's components, by threads t0.. of nt
    auto form = [&](int b, int t0, int nt) {
        const int w0 = __ldg(A.wk + Bt.k[b]), w1 = __ldg(A.wk + Bt.k[b + 1]);
#pragma unroll 4
        for (int e = w0 + t0; e < w1; e += nt) {
            const int4 ps = __ldg(A.wpos + e);
            const float4 f = __ldg(A.wfac + e);
            const pc<float> z = Zt[(size_t)ps.x * ZQ<float>], zq = Zt[(size_t)ps.z * ZQ<float>];
            pc<float> zn = Zt[(size_t)ps.y * ZQ<float>];
            if (ps.w & 1) zn.re = -zn.re;  // the mirror -conj(Z'[m-1]) past a middle row's centre
            const float yr = f.w * zq.re, yi = f.w * zq.im;
            // (re of W0..W3), (im of W0..W3)
            W[2 * (e - w0)] = make_float4(f.x * z.re, f.y * z.im, fmaf(f.z, zn.re, -yr), fmaf(f.z, zn.im, yi));
            W[2 * (e - w0) + 1] = make_float4(f.x * z.im, -f.y * z.re, fmaf(f.z, zn.im, -yi), -fmaf(f.z, zn.re, yr));
            vrow[e - w0] = (ps.w >> 1) * P;
        }
    };
    float s_inv = 0.f;  // 1 / volume: warp 0's, the others read inv_s
    auto setup = [&](int base, int n) {  // warp 0
        const int m = base + lane;
        const int j = lane < n ? A.img_j[m] : -1;
        const bool fresh = lane < n && (m == m0 || A.img_j[m - 1] != j);
        float ck[4], q[12], rv[3];
        plain_image<float>(A, a, m, lane < n, s_inv, j, ck, q, rv);
#pragma unroll
        for (int i = 0; i < 4; ++i) par[32 * i + lane] = ck[i];
#pragma unroll
        for (int i = 0; i < 12; ++i) par[128 + 32 * i + lane] = q[i];
#pragma unroll
        for (int i = 0; i < 3; ++i) par[512 + 32 * i + lane] = rv[i];
        plain_runs(R, n, 32, j, fresh, a, p0, self_img, npair);
    };
    // the first images' set-up (warp 0) beside the first batch's W (the others)
    if (wid == 0) {
        s_inv = inv32(A.geom[A.astruct[a]].vol);
        if (lane == 0) inv_s = s_inv;
        setup(m0, min(32, m1 - m0));
    }
    else form(0, tid - 32, ST - 32);
    int have = 0;  // the batch the buffer holds
    const int sub = lane >> 3, il = lane & 7;
    __syncthreads();

    for (int base = m0; base < m1; base += 32) {
        const int n = min(32, m1 - base);
        if (base != m0) {
            if (wid == 0) setup(base, n);
            __syncthreads();
        }
        plain_rows32<ST>(st, par, V, P);
        float qm[12];  // of this lane's image, il + 8 sub = lane after the exchange below
        const int img = 8 * sub + il;
#pragma unroll
        for (int i = 0; i < 12; ++i) qm[i] = par[128 + 32 * i + img];
        // ---- t of every component, a batch of components at a time
        for (int b = 0; b < Bt.n; ++b) {
            if (have != b) {
                form(b, tid, ST);
                have = b;
            }
            const int w0 = __ldg(A.wk + Bt.k[b]), k1 = Bt.k[b + 1];
            if (tid == 0) s_comp = Bt.k[b];
            __syncthreads();
            for (;;) {
                int pos = 0;
                if (lane == 0) pos = atomicAdd(&s_comp, 1);
                pos = __shfl_sync(0xffffffffu, pos, 0);
                if (pos >= k1) break;
                const int e1 = __ldg(A.wk + pos + 1) - w0, kk = __ldg(A.kord + pos);
                float2 p01[4], p23[4];  // (P0, P1), (P2, P3) of images il + 8 i
#pragma unroll
                for (int i = 0; i < 4; ++i) p01[i] = p23[i] = make_float2(0.f, 0.f);
#pragma unroll 2
                for (int e = __ldg(A.wk + pos) - w0 + sub; e < e1; e += 4) {
                    const float4 wr = W[2 * e], wi = W[2 * e + 1];
                    const pc<float> *v = V + vrow[e] + il;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const pc<float> u = v[8 * i];
                        const float2 ur = make_float2(u.re, u.re), ui = make_float2(u.im, u.im);
                        p01[i] = __ffma2_rn(ur, make_float2(wr.x, wr.y), p01[i]);
                        p23[i] = __ffma2_rn(ur, make_float2(wr.z, wr.w), p23[i]);
                        p01[i] = __ffma2_rn(ui, make_float2(wi.x, wi.y), p01[i]);
                        p23[i] = __ffma2_rn(ui, make_float2(wi.z, wi.w), p23[i]);
                    }
                }
                // add the four groups' sums, each group keeping the images 8 sub ..
                float2 a01[2], a23[2];
                const bool up = sub & 2, odd = sub & 1;
                auto swap2 = [](float2 keep, float2 give, int d) {
                    keep.x += __shfl_xor_sync(0xffffffffu, give.x, d);
                    keep.y += __shfl_xor_sync(0xffffffffu, give.y, d);
                    return keep;
                };
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    a01[i] = swap2(up ? p01[2 + i] : p01[i], up ? p01[i] : p01[2 + i], 16);
                    a23[i] = swap2(up ? p23[2 + i] : p23[i], up ? p23[i] : p23[2 + i], 16);
                }
                const float2 s01 = swap2(odd ? a01[1] : a01[0], odd ? a01[0] : a01[1], 8);
                const float2 s23 = swap2(odd ? a23[1] : a23[0], odd ? a23[0] : a23[1], 8);
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    t3[(q * 32 + img) * CB + kk] = fmaf(
                        qm[4 * q], s01.x, fmaf(qm[4 * q + 1], s01.y, fmaf(qm[4 * q + 2], s23.x, qm[4 * q + 3] * s23.y)));
            }
            __syncthreads();
        }
        // ---- rows: a warp per pair, lane = component; whole lines through the warp's buffer
        float *buf = (float *)smem_raw + (size_t)9 * nB * wid;
        for (int rr = wid; rr < R.nrun[0]; rr += ST / 32) {
            const int i0 = R.run[0][rr], i1 = R.run[0][rr + 1], p = R.pid[i0];
            const bool own = p == ns, add = rr == 0 && R.cont[0];
            float *dx = A.dxdr + (size_t)p * nB * 3, *rd = A.want_stress ? A.rdxdr + (size_t)p * nB * 9 : nullptr;
            float D[KS][3];
#pragma unroll
            for (int s = 0; s < KS; ++s) {
                const int k = lane + 32 * s;
                if (k >= nB) break;
                float E[9];
                auto image = [&](int i, bool first) {
                    float t[3];
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        t[q] = t3[(q * 32 + i) * CB + k];
                        D[s][q] = first ? t[q] : D[s][q] + t[q];
                    }
                    if (!rd) return;
#pragma unroll
                    for (int aa = 0; aa < 3; ++aa) {
                        const float rv = par[512 + 32 * aa + i];
#pragma unroll
                        for (int q = 0; q < 3; ++q) E[3 * aa + q] = first ? rv * t[q] : fmaf(rv, t[q], E[3 * aa + q]);
                    }
                };
                image(i0, true);
                for (int i = i0 + 1; i < i1; ++i) image(i, false);
                if (rd)
#pragma unroll
                    for (int q = 0; q < 9; ++q) buf[9 * k + q] = E[q];
                if (!own)
#pragma unroll
                    for (int q = 0; q < 3; ++q) dsum[s][q] += D[s][q];
            }
            if (rd) {
                __syncwarp();
                for (int q = lane; q < 9 * nB; q += 32) rd[q] = (add || own) ? rd[q] + buf[q] : buf[q];
                __syncwarp();
            }
            if (own) continue;
#pragma unroll
            for (int s = 0; s < KS; ++s) {
                const int k = lane + 32 * s;
                if (k < nB)
                    for (int q = 0; q < 3; ++q) buf[3 * k + q] = D[s][q];
            }
            __syncwarp();
            for (int q = lane; q < 3 * nB; q += 32) dx[q] = add ? dx[q] + buf[q] : buf[q];
            __syncwarp();
        }
        __syncthreads();
    }
    // ---- the (i, i) row: minus the sum of the others
    const float inv_vol = inv_s;
    float *Ds = (float *)smem_raw;
#pragma unroll
    for (int s = 0; s < KS; ++s) {
        const int k = lane + 32 * s;
        if (k < nB)
            for (int q = 0; q < 3; ++q) Ds[(wid * nB + k) * 3 + q] = dsum[s][q];
    }
    __syncthreads();
    for (int k = tid; k < nB; k += ST) {
        float d[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            float s = 0.f;
            for (int w = 0; w < ST / 32; ++w) s += Ds[(w * nB + k) * 3 + q];
            d[q] = -s;
        }
        plain_self_row<float>(A, a, ns, k, inv_vol, d, self_img);
    }
}

// ---------------------------------------------------------------- launch
constexpr size_t ONE_CTA = 226 * 1024, TWO_CTAS = 112 * 1024;  // dynamic shared memory per CTA

// Whether k_plain_d64 keeps the integers of Z' in shared memory: unless that costs the second
// CTA of an SM, or they do not fit at all.
bool d64_zs(const so4_tables *t) {
    const size_t with = D64Smem(t->n_half, t->n_pz, t->n_b, true).total;
    const size_t without = D64Smem(t->n_half, t->n_pz, t->n_b, false).total;
    return with <= TWO_CTAS || (without > TWO_CTAS && with <= ONE_CTA);
}

// Scratch per 32 centres, and the centres of one pass: all of them, or what fits in PLAIN_BYTES.
constexpr size_t PLAIN_BYTES = (size_t)768 << 20;

template <typename T>
size_t plain_tile_bytes(const so4_tables *t) {
    size_t b = sizeof(pc<T>) * 32 * ((size_t)t->n_u + t->n_pz);
    if (sizeof(T) == 8 && !d64_zs(t)) b += sizeof(longlong2) * 32 * (size_t)t->n_pz;
    if (sizeof(T) == 4) b += sizeof(float2) * 32 * (size_t)t->n_half;
    return b;
}
// centres of a pass in that many bytes (0: not one tile)
template <typename T>
int plain_pass(const so4_tables *t, int natoms, size_t bytes) {
    // equal passes of whole tiles
    const size_t most = std::min(bytes, PLAIN_BYTES) / plain_tile_bytes<T>(t), tiles = ((size_t)natoms + 31) / 32;
    if (most == 0) return 0;
    const size_t np = std::max<size_t>(1, (tiles + most - 1) / most);
    return (int)std::min<size_t>((size_t)natoms, 32 * ((tiles + np - 1) / np));
}
template <typename T>
size_t plain_scratch(const so4_tables *t, int natoms) {
    return plain_tile_bytes<T>(t) * (size_t)((plain_pass<T>(t, natoms, PLAIN_BYTES) + 31) / 32);
}

// Scratch of the call's own, in the stream's order, for a caller who gave none.
struct OwnScratch {
    void *p = nullptr;
    cudaStream_t st;
    explicit OwnScratch(cudaStream_t s) : st(s) {}
    ~OwnScratch() {
        if (p) cudaFreeAsync(p, st);
    }
    int take(size_t bytes) {
        if (cudaMallocAsync(&p, bytes, st) == cudaSuccess) return SO4_OK;
        p = nullptr;
        cudaGetLastError();
        return SO4_ERR_WORKSPACE;
    }
};

template <typename T>
int run_plain(const so4_tables *t, const so4_params *p, const so4_geom *geom, const int *astruct, int natoms,
              const double *pos, const double *w_nb, const double *w_site, const int32_t *img_ptr,
              const int32_t *img_j, const double *img_r, const int32_t *pair_ptr, const int32_t *pair_img,
              const int32_t *nsite, int want_deriv, int want_stress, void *x, void *dxdr, void *rdxdr,
              void *work, size_t work_bytes, cudaStream_t st) {
    if (natoms == 0) return SO4_OK;
    PlainArgs<T> A;
    A.prm = *p;
    A.n_u = t->n_u;
    A.n_half = t->n_half;
    A.n_z = t->n_pz;
    A.n_b = t->n_b;
    A.n_unit = t->n_pz_unit;
    A.geom = geom;
    A.astruct = astruct;
    A.pos = pos;
    A.w_nb = w_nb;
    A.w_site = w_site;
    A.img_r = img_r;
    A.img_ptr = img_ptr;
    A.img_j = img_j;
    A.pair_ptr = pair_ptr;
    A.pair_img = pair_img;
    A.nsite = nsite;
    A.unit = t->d_pz_unit;
    A.vent = t->d_p_vent;
    A.lam = t->d_p_lam;
    A.blk = t->d_p_blk;
    A.kord = t->d_p_kord;
    A.hfull = t->d_hfull;
    A.ca = (const T *)(sizeof(T) == 8 ? (const void *)t->d_pz_ca : (const void *)t->d_pz_ca32);
    A.cb = (const T *)(sizeof(T) == 8 ? (const void *)t->d_pz_cb : (const void *)t->d_pz_cb32);
    A.fac = t->d_p_fac;
    A.sent = t->d_p_sent;
    A.bblk = t->d_p_bblk;
    A.zent = t->d_p_zent;
    A.wk = t->d_p_wk;
    A.wpos = t->d_p_wpos;
    A.wfac = t->d_p_wfac;
    A.rc = (T)p->rcut;
    A.psi_fac = (T)(p->rfac0 * SO4_PI / p->rcut);
    fill_small_tables(t, A.st);
    A.want_stress = want_stress;
    A.x = (T *)x;
    A.dxdr = (T *)dxdr;
    A.rdxdr = (T *)rdxdr;
    A.cw = t->p_cw;
    // As many centres a pass as the caller's scratch holds; without a tile's worth the call takes
    // its own (but for FP64 at twol 12, which always asked for scratch).  The tiles start where 16-byte
    // words can be read, whatever the caller's alignment.
    OwnScratch own(st);
    const size_t skip = SO4_WS_HEADER + (size_t)(-(uintptr_t)work & 31);
    char *base = work ? (char *)work + skip : nullptr;
    int pass = plain_pass<T>(t, natoms, work && work_bytes > skip ? work_bytes - skip : 0);
    if (pass == 0) {
        if (sizeof(T) == 8 && t->twol == 12) return SO4_ERR_WORKSPACE;
        const int rc = own.take(plain_scratch<T>(t, natoms));
        if (rc) return rc;
        base = (char *)own.p;
        pass = plain_pass<T>(t, natoms, PLAIN_BYTES);
    }
    const size_t tiles = (size_t)(pass + 31) / 32;
    A.ut = (pc<T> *)base;
    A.zt = A.ut + tiles * 32 * t->n_u;
    A.zi = (longlong2 *)(A.zt + tiles * 32 * t->n_pz);
    A.uh = (float2 *)A.zi;
    int rc = SO4_OK;
    for (int a0 = 0; a0 < natoms; a0 += pass) {
        const int n = std::min(pass, natoms - a0), nt = (n + 31) / 32;
        A.a0 = a0;
        A.natoms = a0 + n;
        if constexpr (sizeof(T) == 8) {
            const size_t smu = sizeof(pc<double>) * (size_t)t->n_half * VI;
            if ((rc = so4_set_smem((const void *)k_plain_u, smu))) return rc;
            k_plain_u<<<n, UT, smu, st>>>(A);
        } else {
            rc = so4_utot32_as(t, p, t->d_hmap_v, n, w_nb, w_site + a0, img_ptr + a0, img_j, img_r, (float *)A.uh, st);
            if (rc) return rc;
            k_plain_tile<<<nt, 256, 0, st>>>(A);
        }
        // A tile's Z units are spread over up to n_unit / 16 CTAs while the grid has fewer than eight
        // CTAs per SM: 64 centres (two tiles) at lmax 3 would otherwise run on two SMs.
        const int parts = std::max(1, std::min((A.n_unit + 15) / 16, 1216 / nt));
        k_plain_z<T><<<dim3(nt, parts), ZT, 0, st>>>(A);
        k_plain_b<T><<<dim3(nt, (t->n_b + 7) / 8), 256, 0, st>>>(A);
        so4_count_launch(3);
        if (!want_deriv) continue;
        if constexpr (sizeof(T) == 8) {
            const bool zs = d64_zs(t);
            const size_t sm = D64Smem(t->n_half, t->n_pz, t->n_b, zs).total;
            auto kern = zs ? k_plain_d64<true> : k_plain_d64<false>;
            if ((rc = so4_set_smem((const void *)kern, sm))) return rc;
            kern<<<n, DT, sm, st>>>(A);
        } else {
            const int emax = section_count(t->twol);
            const size_t sm = D32Smem(t->n_half, t->n_pz, t->n_b, emax).total;
            const int wcap = D32Smem(t->n_half, t->n_pz, t->n_b, emax).wcap;
            PlainBatches bt;
            bt.n = 0;
            bt.k[0] = 0;
            while (bt.k[bt.n] < t->n_b) {  // every component has at most 3 emax <= wcap entries
                int k = bt.k[bt.n] + 1;
                while (k < t->n_b && t->p_wk[k + 1] - t->p_wk[bt.k[bt.n]] <= wcap) ++k;
                if (bt.n + 1 >= 23) return SO4_ERR_UNSUPPORTED;
                bt.k[++bt.n] = k;
            }
            auto kern = t->n_b <= 32 ? k_plain_d32<1> : (t->n_b <= 64 ? k_plain_d32<2> : (t->n_b <= 96 ? k_plain_d32<3> : k_plain_d32<5>));
            if ((rc = so4_set_smem((const void *)kern, sm))) return rc;
            kern<<<n, ST, sm, st>>>(A, emax, bt);
        }
        so4_count_launch();
    }
    return cudaGetLastError() == cudaSuccess ? SO4_OK : SO4_ERR_CUDA;
}

}  // namespace

extern "C" size_t so4_plain_workspace_size(const so4_tables *t, int natoms) {
    if (!t || natoms < 0) return SO4_WS_HEADER;
    // U_tot and Z of one pass of centres, the larger of the two precisions
    return SO4_WS_HEADER + std::max(plain_scratch<double>(t, natoms), plain_scratch<float>(t, natoms));
}

extern "C" int so4_plain(const so4_tables *t, const so4_params *p, int precision, const so4_geom *d_geom,
                         const int *d_astruct, int natoms, const double *d_pos, const double *d_w_nb,
                         const double *d_w_site, const int32_t *d_img_ptr, const int32_t *d_img_j,
                         const double *d_img_r, const int32_t *d_pair_ptr, const int32_t *d_pair_img,
                         const int32_t *d_nsite, int want_deriv, int want_stress, void *d_x, void *d_dxdr,
                         void *d_rdxdr, void *d_work, size_t work_bytes, void *stream) {
    if (!t || !p || natoms < 0 || !d_x) return SO4_ERR_ARG;
    if (p->twol != t->twol) return SO4_ERR_ARG;
    if (p->cutoff_id < 1 || p->cutoff_id > 7) return SO4_ERR_UNSUPPORTED;
    if (!(p->rcut > 0.0) || !(p->rfac0 > 0.0)) return SO4_ERR_ARG;
    if (want_deriv && !d_dxdr) return SO4_ERR_ARG;
    if (want_deriv && want_stress && !d_rdxdr) return SO4_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if (precision == 0)
        return run_plain<double>(t, p, d_geom, d_astruct, natoms, d_pos, d_w_nb, d_w_site, d_img_ptr, d_img_j, d_img_r,
                                 d_pair_ptr, d_pair_img, d_nsite, want_deriv, want_deriv && want_stress, d_x, d_dxdr,
                                 d_rdxdr, d_work, work_bytes, st);
    if (precision == 1)
        return run_plain<float>(t, p, d_geom, d_astruct, natoms, d_pos, d_w_nb, d_w_site, d_img_ptr, d_img_j, d_img_r,
                                d_pair_ptr, d_pair_img, d_nsite, want_deriv, want_deriv && want_stress, d_x, d_dxdr,
                                d_rdxdr, d_work, work_bytes, st);
    return SO4_ERR_ARG;
}

// ---------------------------------------------------------------------------
// Per-atom stress rows.  The reference's caller turns the per-pair rdxdr of
// calculate() into one row per centre (pyxtal_ff/utilities/__init__.py:226-233):
//   out[m, k, :] = sum over the pairs (m, j) of rdxdr[p, k, a, b], (a, b) in the Voigt
//   order (0,0) (1,1) (2,2) (0,1) (0,2) (1,2),
// with a Python loop over atoms.  Pairs are grouped by centre here (pair_ptr), so
// one thread per (m, k, component) sums its centre's pairs in pair order.
namespace {
template <typename T>
__global__ void k_rdxdr_atom(const T *__restrict__ rdxdr, const int32_t *__restrict__ pair_ptr, int natoms, int nB,
                             T *__restrict__ out) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t total = (int64_t)natoms * nB * 6;
    if (idx >= total) return;
    const int v = (int)(idx % 6);
    const int64_t mk = idx / 6;
    const int k = (int)(mk % nB);
    const int m = (int)(mk / nB);
    const int comp = (v < 3) ? 4 * v : ((v == 3) ? 1 : ((v == 4) ? 2 : 5));  // row-major a * 3 + b
    T s = T(0);
    const int p1 = __ldg(pair_ptr + m + 1);
    for (int p = __ldg(pair_ptr + m); p < p1; ++p) s += __ldg(rdxdr + ((size_t)p * nB + k) * 9 + comp);
    out[idx] = s;
}
}  // namespace

extern "C" int so4_rdxdr_atom(int precision, const void *d_rdxdr, const int32_t *d_pair_ptr, int natoms, int nB,
                              void *d_out, void *stream) {
    if (natoms < 0 || nB <= 0 || (natoms > 0 && (!d_rdxdr || !d_pair_ptr || !d_out))) return SO4_ERR_ARG;
    if (precision != 0 && precision != 1) return SO4_ERR_ARG;
    if (natoms == 0) return SO4_OK;
    const int64_t total = (int64_t)natoms * nB * 6;
    const unsigned grid = (unsigned)((total + 255) / 256);
    cudaStream_t st = (cudaStream_t)stream;
    if (precision == 0)
        k_rdxdr_atom<double><<<grid, 256, 0, st>>>((const double *)d_rdxdr, d_pair_ptr, natoms, nB, (double *)d_out);
    else
        k_rdxdr_atom<float><<<grid, 256, 0, st>>>((const float *)d_rdxdr, d_pair_ptr, natoms, nB, (float *)d_out);
    so4_count_launch();
    return cudaGetLastError() == cudaSuccess ? SO4_OK : SO4_ERR_CUDA;
}
