// The operator in the element's Legendre modes: device side.
//
// On a uniform quadratic B-spline grid the 81 x 81 matrix of an isotropic (or orthotropic) element
// is dense in the B-spline basis but has only 78 + 144 entries in the tensor-product Legendre basis
// of the element: with the modes 1, eta/2, (eta^2 - 1/12)/2 per direction (eta the distance from the
// element's centre) the 1-D mass and stiffness matrices are diagonal and the mixed ones d(phi_1)/dx phi_0 and
// d(phi_2)/dx phi_1 only, so the diagonal blocks are diagonal and two components couple where one
// index falls by one and the other rises by one.  The modes of three control values u0, u1, u2 are
//     d0 = a (u0 - u1), d2 = b (u2 - u1):  mean u1 + (d0 + d2)/6, slope d2 - d0, curvature d0 + d2,
// with a = b = 1 except a = 2 on the first and b = 2 on the last element of an open knot vector
// (there N_0 = 2 B_0 and N_1 = B_1 - B_0 in terms of the translated B-splines B).  Every mode but the
// mean of means is formed from differences of control values, so its rounding error scales with
// the variation over the element, not with |u|; the mean of means is never needed (K maps it to 0).
//
// An element so costs about 1,400 operations instead of 2 x 81^2 = 13,122.
#pragma once

#include <type_traits>

#include "icc_device.cuh"
#include "icc_tc.cuh"
#include "icc_vec.cuh"

namespace icc {

// Entries of the uniform element matrix in the modes.  Mode (i, j, k) of component c is i + 3 j + 9 k.
// off[p][q][n][k], pair p = (x,y), (x,z), (y,z) of components (A, B), which are also directions:
//   q = 0: row A with index i >= 1 along A, j <= 1 along B, to column B with (i - 1, j + 1); n = 2 (i - 1) + j
//   q = 1: row A with i <= 1, j >= 1, to column B with (i + 1, j - 1); n = 2 i + (j - 1)
// k is the index along the third direction, the same in both; the matrix is symmetric.
template <class T>
struct ModalK {
    T diag[3][27];
    T off[3][2][4][3];
};

// One system (an operator and the vectors of its solve) as the kernels of this path see it.
template <class T>
struct ModalSys {
    int nx, ny, nz, cx, cy, cz, nsc;
    Tiles t;
    T a[3], b[3];                // end factors of the first and last element per direction
    const T *scale;              // s_e
    const uint8_t *mask;
    int mask_mode;
    T *patch;                    // tile partial sums [tile][3][tz + 2][ty + 2][tx + 2]
    const T *x;                  // input of a plain apply
    // PCG: direction of iteration i in p[i & 1] (the next one is formed while it is read)
    const T *inv;
    T *r, *z, *p[2], *xs, *ap;   // z = D^-1 r
    int p_zero;                  // directions are kept zero on fixed DOFs
    int dot;                     // the apply forms p'Ap and the step length (no sparse term)
    Sparse<T> sp;
    double *part_a, *part_v;     // partial sums of its CTAs: [ncta] p'Ap, [2][ncta] r'r and r'z
    unsigned long long *bar;     // barrier counter
    PcgState *st;
    int ncta;                    // CTAs of the solve
};

constexpr int kModalRing = 5;   // planes staged: one arriving, one in use, three back for p'Ap

// Parity class of mode (i, j, .) of component c under reflection in x and y: modes of different
// classes do not couple, so a thread works through the four classes one after the other.
__host__ __device__ constexpr int modal_class(int c, int m) {
    return ((m % 3 & 1) ^ (c == 0 ? 1 : 0)) + 2 * ((m / 3 & 1) ^ (c == 1 ? 1 : 0));
}
// modes of a class, and the place of mode m of component c among them
__host__ __device__ constexpr int modal_count(int k4) { return k4 == 0 ? 8 : (k4 == 3 ? 5 : 7); }
__host__ __device__ constexpr int modal_place(int c, int m) {
    int n = 0;
    for (int d = 0; d < 3; ++d)
        for (int l = 0; l < 9; ++l)
            if (d * 9 + l < c * 9 + m && modal_class(d, l) == modal_class(c, m)) ++n;
    return n;
}
// A column's state along z, kept in tensor memory class by class (registers do not hold it): per mode
// two running sums, the middle plane's value and the difference to the plane before, and the
// deviation of the class's (0, 0) mode.  In 32-bit columns:
__host__ __device__ constexpr int modal_eq(int k4, int w) { return (2 * modal_count(k4) + (k4 < 3 ? 1 : 0)) * w; }
__host__ __device__ constexpr int modal_eqc(int k4, int w) { return (modal_eq(k4, w) + 1) & ~1; }
__host__ __device__ constexpr int modal_cols(int k4, int w) { return 2 * modal_count(k4) * w + modal_eqc(k4, w); }
__host__ __device__ constexpr int modal_col0(int k4, int w) {
    int n = 0;
    for (int k = 0; k < k4; ++k) n += modal_cols(k, w);
    return n;
}

// Row (c; m, k) of the element matrix times the modes C.
template <class T>
__device__ __forceinline__ T modal_row(const ModalK<T> &K, const T (&C)[3][27], int c, int m, int k) {
    if (m == 0 && k == 0) return T(0);
    const int idx[3] = {m % 3, m / 3, k}, pw[3] = {1, 3, 9}, n = m + 9 * k;
    T a = K.diag[c][n] * C[c][n];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (d == c) continue;
        const int A = c < d ? c : d, B = c < d ? d : c, pr = A + B - 1;
        const int ia = idx[A], ib = idx[B], kt = idx[3 - A - B];
        // partner with A index - 1, B index + 1
        if (ia >= 1 && ib <= 1)
            a += (c == A ? K.off[pr][0][2 * (ia - 1) + ib][kt] : K.off[pr][1][2 * (ia - 1) + ib][kt]) * C[d][n - pw[A] + pw[B]];
        // partner with A index + 1, B index - 1
        if (ia <= 1 && ib >= 1)
            a += (c == A ? K.off[pr][1][2 * ia + ib - 1][kt] : K.off[pr][0][2 * ia + ib - 1][kt]) * C[d][n + pw[A] - pw[B]];
    }
    return a;
}

// A march uses NT threads, one per column: at most as many as tensor memory holds columns' states.  Fewer take
// fewer clocks a step, which decides where a grid gives an SM only a few steps.
template <class T>
struct ModalMarch {
    static constexpr int words = sizeof(T) / 4;
    static constexpr int cols = modal_col0(4, words);       // 222 (FP64), 114 (FP32) of the 512 columns
    static constexpr int max_nt = 128 * (512 / cols);       // 256 (FP64), 512 (FP32)
};
__host__ __device__ constexpr int march_slots(int nt) { return nt >= 256 ? 4 : 5; }   // control values a thread stages per plane

// Shared memory of a march in values: staged planes, the row exchange (27 values per column, two steps),
// arriving values.
__host__ __device__ inline int march_smem(int nt, int ltx, bool pcg) {
    return kModalRing * (3 * ((nt >> ltx) + 2) * ((1 << ltx) + 2) + 1) + 2 * 27 * nt + (pcg ? 2 : 1) * march_slots(nt) * nt;
}

// value i of an array of 32-bit words
template <class T>
__device__ __forceinline__ T word_get(const uint32_t *w, int i) {
    if constexpr (sizeof(T) == 8) return __hiloint2double((int)w[2 * i + 1], (int)w[2 * i]);
    else return __uint_as_float(w[i]);
}
template <class T>
__device__ __forceinline__ void word_set(uint32_t *w, int i, T v) {
    if constexpr (sizeof(T) == 8) {
        w[2 * i] = (uint32_t)__double2loint(v);
        w[2 * i + 1] = (uint32_t)__double2hiint(v);
    } else {
        w[i] = __float_as_uint(v);
    }
}

__device__ __forceinline__ void cp_value(float *dst, const float *src) { tc::cp_async4(dst, src); }
__device__ __forceinline__ void cp_value(double *dst, const double *src) { tc::cp_async8(dst, src); }

template <int NT, bool WHOLE>
__device__ __forceinline__ void march_sync() {
    if constexpr (WHOLE) __syncthreads();
    else tc::named_sync(1, NT);
}

// y = K x on one tile, tx x ty columns of elements, tz long in z, by the first NT threads of a CTA: thread tid
// marches along column (tid % tx, tid / tx).  Per plane of control points: the column's nine control values per
// component become modes along x and y; per element: modes along z, the sparse product, and the
// transposed z step into running sums of the three planes.  A finished plane goes back to control
// values along y (neighbouring columns summed through shared memory) and x (through shuffles), and
// the tile's sums are written as its patch; the node-side pass adds the patches that share a control
// point.  With PCG the input is formed on the fly, p = z + beta p_old, written to p_new where the
// tile owns the control point, and this thread's part of p'Ap is returned.  No atomics: bitwise
// reproducible.  sm: march_smem values; tm: the warp's tensor memory.
//
// A column per thread shares the z direction's transforms along the march and leaves x and y to two cheap
// exchanges.  It is bound by the issue of few warps: 1.8 (FP64) and 2.8 (FP32) instructions per clock
// and SM of 4, as tensor memory holds the state of 256 and 512 columns (in registers it spills).  Measured at
// 128x64x64, whole FP64 apply: dense DMMA contraction 375 us, this 65 us; two or four threads per column 77
// to 94 us.  FP32 at 256x128x128: tensor-core contraction 635 us, this 333 us.  DRAM traffic is the input and
// the scale once (19.5 and 10.6 MB at 128x64x64).
template <class T, int NT, bool PCG, bool WHOLE>
__device__ __forceinline__ double modal_march(const ModalK<T> &K, const ModalSys<T> &S, int tile, T *sm, uint32_t tm, T beta,
                                              const T *p_old, T *p_new) {
    constexpr int kS = march_slots(NT), kW = ModalMarch<T>::words;
    const int tid = threadIdx.x;
    const int ltx = S.t.ltx, TX = 1 << ltx, TY = S.t.ty, TZ = S.t.tz;
    const int bx = tile % S.t.ntx, by = (tile / S.t.ntx) % S.t.nty, bz = tile / (S.t.ntx * S.t.nty);
    const int x0 = bx << ltx, y0 = by * TY, z0 = bz * TZ;
    const int lx = tid & (TX - 1), ly = tid >> ltx;
    const int pitch = TX + 2, rows = (NT >> ltx) + 2;
    const int cstr = rows * pitch, plane = 3 * cstr;
    T *ring = sm, *F = sm + kModalRing * (plane + 1), *raw = F + 2 * 27 * NT + tid;
    const int nez = min(TZ, S.nz - z0), np = nez + 2;
    const bool valid = ly < TY && x0 + lx < S.nx && y0 + ly < S.ny;
    const T ax = x0 + lx == 0 ? S.a[0] : T(1), bxf = x0 + lx == S.nx - 1 ? S.b[0] : T(1);
    const T ay = y0 + ly == 0 ? S.a[1] : T(1), byf = y0 + ly == S.ny - 1 ? S.b[1] : T(1);
    const T sixth = T(1.0 / 6.0);
    const int cxy = S.cx * S.cy;

    // this thread's share of a plane: control values i = tid + s NT of the (TY + 2) x (TX + 2) x 3.  No
    // branches, so the loads of a plane are all in flight at once: a slot outside the grid reads
    // the tile's first value and stages 0, a slot beyond the plane stages into a spare value
    int goff[kS], soff[kS];
    unsigned in = 0u, own = 0u;   // bit s: inside the grid / this tile writes the new direction there
    {
        const int w = TX + 2, pl = w * (TY + 2);
#pragma unroll
        for (int s = 0; s < kS; ++s) {
            const int i = tid + s * NT;
            goff[s] = (z0 * S.cy + y0) * S.cx + x0;
            soff[s] = plane;
            if (i < 3 * pl) {
                const int c = i / pl, q = i - c * pl, py = q / w, px = q - py * w;
                soff[s] = c * cstr + py * pitch + px;
                if (x0 + px < S.cx && y0 + py < S.cy) {
                    goff[s] = c * S.nsc + (z0 * S.cy + y0 + py) * S.cx + x0 + px;
                    in |= 1u << s;
                    if ((px < TX || bx == S.t.ntx - 1) && (py < TY || by == S.t.nty - 1)) own |= 1u << s;
                }
            }
        }
    }
    const bool masked = S.mask_mode != ICC_MASK_NONE;
    unsigned mk[kS];
    double dot = 0.0;
    // plane j's values on their way to this thread's slots (z = D^-1 r and p_old, or x)
    auto fetch = [&](int j) {
#pragma unroll
        for (int s = 0; s < kS; ++s) {
            const int g = goff[s] + j * cxy;
            if constexpr (PCG) {
                cp_value(raw + s * NT, S.z + g);
                cp_value(raw + (kS + s) * NT, p_old + g);
            } else {
                cp_value(raw + s * NT, S.x + g);
            }
        }
        tc::cp_async_commit();
        if (masked) {
#pragma unroll
            for (int s = 0; s < kS; ++s) mk[s] = S.mask[goff[s] + j * cxy];
        } else {
#pragma unroll
            for (int s = 0; s < kS; ++s) mk[s] = 1u;
        }
    };
    auto stage = [&](int j) {
        T *dst = ring + (j % kModalRing) * (plane + 1);
        const bool zown = j < TZ || bz == S.t.ntz - 1;
        tc::cp_async_wait<0>();
#pragma unroll
        for (int s = 0; s < kS; ++s) {
            T v = raw[s * NT];
            if constexpr (PCG) {
                v += beta * raw[(kS + s) * NT];
                if (zown && (own >> s & 1u)) {
                    p_new[goff[s] + j * cxy] = (S.p_zero && !mk[s]) ? T(0) : v;
                    if (S.mask_mode == ICC_MASK_IDENTITY && !mk[s]) dot += double(v) * double(v);
                }
            }
            dst[soff[s]] = (mk[s] && (in >> s & 1u)) ? v : T(0);
        }
    };

    const int ebase = (valid ? x0 + lx + S.nx * (y0 + ly) : 0) + S.nx * S.ny * z0, estr = S.nx * S.ny;
    T *const pb = S.patch + (size_t)tile * (size_t)S.t.vol;
    const int prow = TX + 2, pplane = prow * (TY + 2), pcomp = pplane * (TZ + 2);

    // one row of control values of plane jo from the row sums G of its x modes
    auto emit = [&](const T (&G)[9], int jo, int py, bool on) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const T w0 = G[c * 3], w1 = G[c * 3 + 1], w2 = G[c * 3 + 2];
            const T g = w2 + sixth * w0;
            const T h0 = ax * (g - w1), h2 = bxf * (g + w1), h1 = w0 - h0 - h2;
            T up = __shfl_up_sync(0xffffffffu, h2, 1, TX);
            const T u = h1 + (lx >= 1 ? up : T(0));
            up = __shfl_up_sync(0xffffffffu, u, 1, TX);
            const T v = h0 + (lx >= 1 ? up : T(0));
            if (on) {
                T *o = pb + c * pcomp + jo * pplane + py * prow + lx;
                o[0] = v;
                if (lx == TX - 1) {
                    o[1] = u;
                    o[2] = h2;
                }
                if constexpr (PCG) {
                    const T *q = ring + (jo % kModalRing) * (plane + 1) + c * cstr + py * pitch + lx;
                    dot += double(q[0]) * double(v);
                    if (lx == TX - 1) dot += double(q[1]) * double(u) + double(q[2]) * double(h2);
                }
            }
        }
    };

    fetch(0);
    stage(0);
    march_sync<NT, WHOLE>();
    T s_next = T(0);
#pragma unroll 1
    for (int j = 0; j < np + 3; ++j) {
        if (j + 1 < np) fetch(j + 1);
        const T se = valid ? s_next : T(0);
        if (j >= 1 && j - 1 < nez) s_next = S.scale[ebase + (j - 1) * estr];
        // ---- finish plane j - 3: sum the columns along y, back to control values along x
        if (j >= 3) {
            const int jo = j - 3;
            const T *Fp = F + ((j - 1) & 1) * 27 * NT;
            T G[9];
            const T *Fa = Fp + 9 * NT + (ly >= 1 ? tid - TX : tid), *Fb = Fp + 18 * NT + (ly >= 2 ? tid - 2 * TX : tid);
#pragma unroll
            for (int m = 0; m < 9; ++m) {
                const T u = Fa[m * NT], v = Fb[m * NT];
                G[m] = Fp[m * NT + tid] + (ly >= 1 ? u : T(0)) + (ly >= 2 ? v : T(0));
            }
            emit(G, jo, ly, ly < TY);
            if (((tid & ~31) >> ltx) < 2) {   // warps that hold the first two rows also finish rows TY, TY + 1
                const T *Fc = Fp + (ly == 0 ? 9 : 18) * NT + (TY - 1) * TX + lx, *Fd = Fp + 18 * NT + max(TY - 2, 0) * TX + lx;
#pragma unroll
                for (int m = 0; m < 9; ++m) {
                    const T u = Fc[m * NT], v = Fd[m * NT];
                    G[m] = u + (ly == 0 && TY >= 2 ? v : T(0));
                }
                emit(G, jo, TY + ly, ly < 2);
            }
        }
        if (j < np + 2) {
            // finished modes of plane j - 2, at the places their row sums take (a thread's own until the barrier)
            T *Fn = F + (j & 1) * 27 * NT + tid;
            auto put = [&](int c, int m, T v) { Fn[(m / 3 * 9 + c * 3 + m % 3) * NT] = v; };
            if (j < np) {
                // ---- modes along x and y of plane j
                const T *q0 = ring + (j % kModalRing) * (plane + 1) + ly * pitch + lx;
                T qn[3][9], dn[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    T r[3], c1[3], s2[3];
#pragma unroll
                    for (int l = 0; l < 3; ++l) {
                        const T *q = q0 + c * cstr + l * pitch;
                        r[l] = q[1];
                        const T d0 = ax * (q[0] - q[1]), d2 = q[2] - q[1];
                        c1[l] = bxf * d2 - d0;
                        s2[l] = bxf * d2 + d0;
                    }
                    {
                        const T d0 = ay * (c1[0] - c1[1]), d2 = c1[2] - c1[1];
                        qn[c][4] = byf * d2 - d0;
                        qn[c][7] = byf * d2 + d0;
                        qn[c][1] = c1[1] + sixth * qn[c][7];
                    }
                    const T e0 = s2[0] - s2[1], e2 = s2[2] - s2[1];
                    {
                        const T d0 = ay * e0;
                        qn[c][5] = byf * e2 - d0;
                        qn[c][8] = byf * e2 + d0;
                        qn[c][2] = s2[1] + sixth * qn[c][8];
                    }
                    {
                        const T d0 = ay * ((r[0] - r[1]) + sixth * e0), d2 = (r[2] - r[1]) + sixth * e2;
                        qn[c][3] = byf * d2 - d0;
                        qn[c][6] = byf * d2 + d0;
                    }
                    qn[c][0] = r[1];
                    dn[c] = s2[1] + qn[c][6];
                }
                const int e = j - 2;   // the element whose last plane this is
                const T az = z0 + e == 0 ? S.a[2] : T(1), bzf = z0 + e == S.nz - 1 ? S.b[2] : T(1);
                const T sa = se * az, sb = se * bzf;
                auto one_class = [&](auto kc) {
                    constexpr int k4 = decltype(kc)::value, cnt = modal_count(k4);
                    const uint32_t tp = tm + modal_col0(k4, kW), tq = tp + 2 * cnt * kW;
                    // ---- state: value on the middle plane and difference to the plane before; (0, 0) as a
                    // control value plus a deviation (in sixths)
                    uint32_t eq[modal_eqc(k4, kW)], pp[2 * cnt * kW];
                    eq[modal_eqc(k4, kW) - 1] = 0u;
                    tc::tm_load<modal_eqc(k4, kW)>(tq, eq);
                    tc::tm_arrive<modal_eqc(k4, kW)>(eq);
                    // ---- modes along z
                    T C[3][27];
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int m = 0; m < 9; ++m) {
                            if (modal_class(c, m) != k4) continue;
                            const int n = modal_place(c, m);
                            const T q1 = word_get<T>(eq, 2 * n), e1 = word_get<T>(eq, 2 * n + 1);
                            T en = qn[c][m] - q1;
                            if (m == 0) en += sixth * (dn[c] - word_get<T>(eq, 2 * cnt));
                            const T d0 = az * e1;   // minus the difference to the first plane
                            C[c][m + 9] = bzf * en + d0;
                            C[c][m + 18] = bzf * en - d0;
                            C[c][m] = m == 0 ? T(0) : q1 + sixth * C[c][m + 18];
                            word_set<T>(eq, 2 * n, qn[c][m]);
                            word_set<T>(eq, 2 * n + 1, en);
                            if (m == 0) word_set<T>(eq, 2 * cnt, dn[c]);
                        }
                    tc::tm_store<modal_eqc(k4, kW)>(tq, eq);
                    if (e < 0) return;   // the first two planes only fill the state
                    if (e > 0) {
                        tc::tm_load<2 * cnt * kW>(tp, pp);
                    } else {
#pragma unroll
                        for (int i = 0; i < 2 * cnt * kW; ++i) pp[i] = 0u;
                    }
                    // ---- the element matrix in the modes, and the transposed z step
                    bool first = true;
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int m = 0; m < 9; ++m) {
                            if (modal_class(c, m) != k4) continue;
                            T w[3];
#pragma unroll
                            for (int k = 0; k < 3; ++k) w[k] = modal_row(K, C, c, m, k);
                            if (first) tc::tm_arrive<2 * cnt * kW>(pp);
                            first = false;
                            const int n = modal_place(c, m);
                            const T g = m == 0 ? w[2] : w[2] + sixth * w[0];
                            const T a = g - w[1], b = g + w[1];
                            const T mid = m == 0 ? -az * a - bzf * b : w[0] - az * a - bzf * b;
                            put(c, m, word_get<T>(pp, 2 * n) + sa * a);
                            word_set<T>(pp, 2 * n, word_get<T>(pp, 2 * n + 1) + se * mid);
                            word_set<T>(pp, 2 * n + 1, sb * b);
                        }
                    tc::tm_store<2 * cnt * kW>(tp, pp);
                };
                one_class(std::integral_constant<int, 0>());
                one_class(std::integral_constant<int, 1>());
                one_class(std::integral_constant<int, 2>());
                one_class(std::integral_constant<int, 3>());
                tc::tmem_wait_st();
            } else {
                // ---- the last two planes take no further element
                auto drain = [&](auto kc) {
                    constexpr int k4 = decltype(kc)::value, cnt = modal_count(k4);
                    const uint32_t tp = tm + modal_col0(k4, kW);
                    uint32_t pp[2 * cnt * kW];
                    tc::tm_load<2 * cnt * kW>(tp, pp);
                    tc::tm_arrive<2 * cnt * kW>(pp);
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int m = 0; m < 9; ++m) {
                            if (modal_class(c, m) != k4) continue;
                            const int n = modal_place(c, m);
                            put(c, m, word_get<T>(pp, 2 * n));
                            word_set<T>(pp, 2 * n, word_get<T>(pp, 2 * n + 1));
                        }
                    tc::tm_store<2 * cnt * kW>(tp, pp);
                };
                drain(std::integral_constant<int, 0>());
                drain(std::integral_constant<int, 1>());
                drain(std::integral_constant<int, 2>());
                drain(std::integral_constant<int, 3>());
                tc::tmem_wait_st();
            }
            if (j >= 2) {
                // ---- transposed y step of plane j - 2; rows ly + 1 and ly + 2 through shared memory
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        const T w0 = Fn[(c * 3 + i) * NT], w1 = Fn[(9 + c * 3 + i) * NT], w2 = Fn[(18 + c * 3 + i) * NT];
                        const T g = w2 + sixth * w0;
                        const T a = ay * (g - w1), b = byf * (g + w1);
                        Fn[(c * 3 + i) * NT] = a;
                        Fn[(9 + c * 3 + i) * NT] = w0 - a - b;
                        Fn[(18 + c * 3 + i) * NT] = b;
                    }
            }
        }
        if (j + 1 < np) stage(j + 1);
        march_sync<NT, WHOLE>();
    }
    return dot;
}

// ---- a cube of 4 x 4 x 4 elements --------------------------------------------------------------------
//
// The same product on a small tile, all its elements at once: 256 threads, four per element (one a parity
// class), go through the directions one after the other in shared memory, six barriers in all.  A
// march's steps follow one another, about 2 us each however few columns there are; on grids that give
// an SM only a few cubes this is sooner, on large ones its small tiles (3.4
// partial sums per control point) and its traffic through shared memory cost more than the march.
// Bound by the latency of its phases where it is used.  Measured at 24x16x12, whole FP64 apply: dense DMMA
// contraction 13.0 us, this 6.4 us; a PCG iteration on cubes 12.6 us, on marches 22 us.
constexpr int kCube = 4, kCubeP = kCube + 2, kCubeThreads = 256;
constexpr int kCubeU = 3 * kCubeP * kCubeP * kCubeP;                    // control values [c][z][y][x]
constexpr int kCubeX = 9 * kCubeP * kCubeP * kCube;                     // x modes [v][c][z][y][ex]; row sums [c][i][z][y][ex]
constexpr int kCubeY = 30 * kCubeP * kCube * kCube;                     // x, y modes [m][c][z][ey][ex]; plane sums [m][z][ey][ex]
constexpr int kCubeW = 81 * kCube * kCube * kCube;                      // the elements' planes [k][m][e]
constexpr int kCubeSmem = kCubeU + kCubeX + kCubeY + kCubeW;            // values

template <bool WHOLE>
__device__ __forceinline__ void cube_sync(int bar) {
    if constexpr (WHOLE) __syncthreads();
    else tc::named_sync(bar, kCubeThreads);
}

template <class T, int K4>
__device__ __forceinline__ void cube_class(const ModalK<T> &K, const T *Y, T *W, int e, T se, T az, T bz) {
    constexpr int kZ = kCube * kCube, kM = 3 * kCubeP * kZ;   // strides of Y: plane, mode
    const T sixth = T(1.0 / 6.0);
    T C[3][27];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int m = 0; m < 9; ++m) {
            if (modal_class(c, m) != K4) continue;
            const T *q = Y + m * kM + c * (kCubeP * kZ) + e;
            const T q1 = q[kZ];
            T e0 = q[0] - q1, e2 = q[2 * kZ] - q1;
            if (m == 0) {   // a control value plus a deviation (in sixths)
                const T *d = Y + 9 * kM + c * (kCubeP * kZ) + e;
                e0 += sixth * (d[0] - d[kZ]);
                e2 += sixth * (d[2 * kZ] - d[kZ]);
            }
            const T d0 = az * e0;
            C[c][m + 9] = bz * e2 - d0;
            C[c][m + 18] = bz * e2 + d0;
            C[c][m] = m == 0 ? T(0) : q1 + sixth * C[c][m + 18];
        }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int m = 0; m < 9; ++m) {
            if (modal_class(c, m) != K4) continue;
            T w[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) w[k] = modal_row(K, C, c, m, k);
            const T g = m == 0 ? w[2] : w[2] + sixth * w[0];
            const T a = az * (g - w[1]), b = bz * (g + w[1]);
            T *o = W + (m / 3 * 9 + c * 3 + m % 3) * 64 + e;
            o[0] = se * a;
            o[27 * 64] = se * ((m == 0 ? T(0) : w[0]) - a - b);
            o[54 * 64] = se * b;
        }
}

// tid in [0, 256); the other arguments as modal_march's.  sm: kCubeSmem values.
template <class T, bool PCG, bool WHOLE>
__device__ __forceinline__ double modal_cube(const ModalK<T> &K, const ModalSys<T> &S, int tile, int tid, int bar, T *sm, T beta,
                                             const T *p_old, T *p_new) {
    T *const U = sm, *const X = U + kCubeU, *const Y = X + kCubeX, *const W = Y + kCubeY;
    constexpr int P = kCubeP, E = kCube;
    const int r = tile / S.t.dntx, bx = tile - r * S.t.ntx, bz = r / S.t.dnty, by = r - bz * S.t.nty;
    const int x0 = bx * E, y0 = by * E, z0 = bz * E;
    const T sixth = T(1.0 / 6.0);
    const bool masked = S.mask_mode != ICC_MASK_NONE;
    double dot = 0.0;
    // this thread's element and its scale, asked for before the first barrier
    const int e = tid & 63, k4 = __shfl_sync(0xffffffffu, tid >> 6, 0);
    const int ex = e & 3, ey = e >> 2 & 3, ez = e >> 4;
    const bool valid = x0 + ex < S.nx && y0 + ey < S.ny && z0 + ez < S.nz;
    const T se = valid ? S.scale[(x0 + ex) + S.nx * ((y0 + ey) + S.ny * (z0 + ez))] : T(0);
    // ---- control values
    {
        constexpr int kS = (kCubeU + kCubeThreads - 1) / kCubeThreads;
        T v[kS], v2[kS];
        int g[kS];
        unsigned char mk[kS];
        bool in[kS];
#pragma unroll
        for (int s = 0; s < kS; ++s) {
            const int i = tid + s * kCubeThreads, c = i / (P * P * P), q = i - c * (P * P * P), pz = q / (P * P), py = q / P % P, px = q % P;
            in[s] = i < kCubeU && x0 + px < S.cx && y0 + py < S.cy && z0 + pz < S.cz;
            g[s] = in[s] ? c * S.nsc + ((z0 + pz) * S.cy + y0 + py) * S.cx + x0 + px : 0;
            // past the L1: other CTAs of a running solve wrote them
            if constexpr (PCG) {
                v[s] = __ldcg(S.z + g[s]);
                v2[s] = __ldcg(p_old + g[s]);
            } else {
                v[s] = __ldcg(S.x + g[s]);
            }
            mk[s] = masked ? S.mask[g[s]] : (unsigned char)1;
        }
#pragma unroll
        for (int s = 0; s < kS; ++s) {
            const int i = tid + s * kCubeThreads;
            if (i >= kCubeU) break;
            T u = v[s];
            if constexpr (PCG) {
                u += beta * v2[s];
                const int q = i % (P * P * P), pz = q / (P * P), py = q / P % P, px = q % P;
                if (in[s] && (px < E || bx == S.t.ntx - 1) && (py < E || by == S.t.nty - 1) && (pz < E || bz == S.t.ntz - 1)) {
                    p_new[g[s]] = (S.p_zero && !mk[s]) ? T(0) : u;
                    if (S.mask_mode == ICC_MASK_IDENTITY && !mk[s]) dot += double(u) * double(u);
                }
            }
            U[i] = in[s] && mk[s] ? u : T(0);
        }
    }
    cube_sync<WHOLE>(bar);
    // ---- modes along x: items (c, z, y, ex)
    for (int i = tid; i < 3 * P * P * E; i += kCubeThreads) {
        const int x = i & 3, row = i >> 2;
        const T *u = U + row * P + x;
        const T ax = x0 + x == 0 ? S.a[0] : T(1), bxf = x0 + x == S.nx - 1 ? S.b[0] : T(1);
        const T rr = u[1], d0 = ax * (u[0] - rr), d2 = u[2] - rr;
        X[i] = rr;
        X[3 * P * P * E + i] = bxf * d2 - d0;
        X[6 * P * P * E + i] = bxf * d2 + d0;
    }
    cube_sync<WHOLE>(bar);
    // ---- modes along y: items (c, z, ey, ex)
    for (int i = tid; i < 3 * P * E * E; i += kCubeThreads) {
        const int x = i & 3, y = i >> 2 & 3, cz = i >> 4;
        const T ay = y0 + y == 0 ? S.a[1] : T(1), byf = y0 + y == S.ny - 1 ? S.b[1] : T(1);
        const T *q = X + (cz * P + y) * E + x;
        constexpr int V = 3 * P * P * E, M = 3 * P * E * E;
        T rr[3], c1[3], s2[3];
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            rr[l] = q[l * E];
            c1[l] = q[V + l * E];
            s2[l] = q[2 * V + l * E];
        }
        T *o = Y + i;
        {
            const T d0 = ay * (c1[0] - c1[1]), d2 = c1[2] - c1[1], s = byf * d2 + d0;
            o[4 * M] = byf * d2 - d0;
            o[7 * M] = s;
            o[1 * M] = c1[1] + sixth * s;
        }
        const T e0 = s2[0] - s2[1], e2 = s2[2] - s2[1];
        {
            const T d0 = ay * e0, s = byf * e2 + d0;
            o[5 * M] = byf * e2 - d0;
            o[8 * M] = s;
            o[2 * M] = s2[1] + sixth * s;
        }
        {
            const T d0 = ay * ((rr[0] - rr[1]) + sixth * e0), d2 = (rr[2] - rr[1]) + sixth * e2, s = byf * d2 + d0;
            o[3 * M] = byf * d2 - d0;
            o[6 * M] = s;
            o[0] = rr[1];
            o[9 * M] = s2[1] + s;
        }
    }
    cube_sync<WHOLE>(bar);
    // ---- elements: modes along z, the sparse product, the transposed z step
    {
        const T az = z0 + ez == 0 ? S.a[2] : T(1), bzf = z0 + ez == S.nz - 1 ? S.b[2] : T(1);
        if (k4 == 0) cube_class<T, 0>(K, Y, W, e, se, az, bzf);
        else if (k4 == 1) cube_class<T, 1>(K, Y, W, e, se, az, bzf);
        else if (k4 == 2) cube_class<T, 2>(K, Y, W, e, se, az, bzf);
        else cube_class<T, 3>(K, Y, W, e, se, az, bzf);
    }
    cube_sync<WHOLE>(bar);
    // ---- sums along z: items (m, z, ey, ex), in place of Y
    {
        constexpr int N = 27 * P * E * E, kN = (N + kCubeThreads - 1) / kCubeThreads;
        T s[kN];
#pragma unroll
        for (int u = 0; u < kN; ++u) {
            const int i = tid + u * kCubeThreads, m = i / (P * E * E), q = i - m * (P * E * E), pz = q >> 4, yx = q & 15;
            s[u] = T(0);
            if (i < N)
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    if (pz - k >= 0 && pz - k < E) s[u] += W[(k * 27 + m) * 64 + (pz - k) * 16 + yx];
        }
#pragma unroll
        for (int u = 0; u < kN; ++u)
            if (tid + u * kCubeThreads < N) Y[tid + u * kCubeThreads] = s[u];
    }
    cube_sync<WHOLE>(bar);
    // ---- transposed y step and sums along y: items (c, i, z, y, ex), in place of X
    {
        constexpr int N = 9 * P * P * E, kN = (N + kCubeThreads - 1) / kCubeThreads;
        T s[kN];
#pragma unroll
        for (int u = 0; u < kN; ++u) {
            const int i = min(tid + u * kCubeThreads, N - 1), x = i & 3, row = i >> 2, py = row % P, cz = row / P, n = cz / P,
                      pz = cz - n * P;
            s[u] = T(0);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int y = py - k;
                if (y < 0 || y >= E) continue;
                const T ay = y0 + y == 0 ? S.a[1] : T(1), byf = y0 + y == S.ny - 1 ? S.b[1] : T(1);
                const T *q = Y + (n * P + pz) * (E * E) + y * E + x;
                const T w0 = q[0], w1 = q[9 * P * E * E], w2 = q[18 * P * E * E], g = w2 + sixth * w0;
                const T a = ay * (g - w1), b = byf * (g + w1);
                s[u] += k == 0 ? a : (k == 1 ? w0 - a - b : b);
            }
        }
#pragma unroll
        for (int u = 0; u < kN; ++u)
            if (tid + u * kCubeThreads < N) X[tid + u * kCubeThreads] = s[u];
    }
    cube_sync<WHOLE>(bar);
    // ---- transposed x step and sums along x, to the patch: items (c, z, y, x)
    T *const pb = S.patch + (size_t)tile * (size_t)S.t.vol;
#pragma unroll
    for (int u = 0; u < (kCubeU + kCubeThreads - 1) / kCubeThreads; ++u) {
        const int i = tid + u * kCubeThreads;
        if (i >= kCubeU) break;
        const int px = i % P, row = i / P, c = row / (P * P), zy = row - c * (P * P);
        T s = T(0);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int x = px - k;
            if (x < 0 || x >= E) continue;
            const T ax = x0 + x == 0 ? S.a[0] : T(1), bxf = x0 + x == S.nx - 1 ? S.b[0] : T(1);
            const T *q = X + (c * 3 * (P * P) + zy) * E + x;
            const T w0 = q[0], w1 = q[P * P * E], w2 = q[2 * P * P * E], g = w2 + sixth * w0;
            const T a = ax * (g - w1), b = bxf * (g + w1);
            s += k == 0 ? a : (k == 1 ? w0 - a - b : b);
        }
        pb[i] = s;
        if constexpr (PCG) dot += double(U[i]) * double(s);
    }
    cube_sync<WHOLE>(bar);
    return dot;
}

// ---- kernels ----------------------------------------------------------------------------------------

// Tensor memory for a CTA's march: this warp's lanes and columns.
template <class T>
__device__ __forceinline__ uint32_t modal_tmem(uint32_t *base, int cols) {
    if (threadIdx.x < 32) {
        tc::tmem_alloc(base, cols);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // the same for the warp, as its TMEM addresses are
    return *base + ((uint32_t)(warp & 3) << 21) + (uint32_t)((warp >> 2) * ModalMarch<T>::cols);
}

// A plain apply, a tile per CTA.
template <class T, int NT>
__global__ void __launch_bounds__(NT, NT <= 128 ? 2 : 1)
modal_march_kernel(const __grid_constant__ ModalK<T> K, const __grid_constant__ ModalSys<T> S) {
    constexpr int kCols = NT <= 128 ? 256 : 512;
    extern __shared__ __align__(16) unsigned char modal_raw[];
    __shared__ uint32_t tmem_base;
    const uint32_t tm = modal_tmem<T>(&tmem_base, kCols);
    modal_march<T, NT, false, true>(K, S, blockIdx.x, reinterpret_cast<T *>(modal_raw), tm, T(0), nullptr, nullptr);
    if (threadIdx.x < 32) tc::tmem_dealloc(tmem_base, kCols);
}
template <class T>
__global__ void __launch_bounds__(kCubeThreads, 2)
modal_cube_kernel(const __grid_constant__ ModalK<T> K, const __grid_constant__ ModalSys<T> S) {
    extern __shared__ __align__(16) unsigned char modal_raw[];
    modal_cube<T, false, true>(K, S, blockIdx.x, threadIdx.x, 0, reinterpret_cast<T *>(modal_raw), T(0), nullptr, nullptr);
}

// ---- the PCG loop ---------------------------------------------------------------------------------

// Barrier of a system's CTAs (cooperative launch: all are resident): passed when the counter has reached
// `target` arrivals.  Bounded by `limit` polls, false on time-out (err = 2).
__device__ __forceinline__ bool modal_barrier(unsigned long long *ctr, unsigned long long target, int *err, long long limit) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        // release: the CTA's writes before the barrier above; acquire: the other CTAs'
        asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(ctr) : "memory");
        int ok = 0;
        for (long long i = 0; i < limit; ++i) {
            unsigned long long v;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(ctr) : "memory");
            if (v >= target) {
                ok = 1;
                break;
            }
        }
        if (!ok) atomicExch(err, 2);
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Sums of part[k G .. (k + 1) G), the same in every CTA that forms them; valid in the first warp.  Loads are issued
// together: one trip to the L2, not one after the other.
template <int N>
__device__ __forceinline__ void modal_total(const double *part, int G, double (&v)[N]) {
    if (threadIdx.x >= 32) return;
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = 0.0;
    for (int i0 = threadIdx.x; i0 < G; i0 += 160) {
        double t[N][5];
#pragma unroll
        for (int k = 0; k < N; ++k)
#pragma unroll
            for (int u = 0; u < 5; ++u) t[k][u] = i0 + 32 * u < G ? __ldcg(part + k * G + i0 + 32 * u) : 0.0;
#pragma unroll
        for (int k = 0; k < N; ++k)
#pragma unroll
            for (int u = 0; u < 5; ++u) v[k] += t[k][u];
    }
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = warp_sum(v[k]);
}

// Sums over the CTA's threads, valid in thread 0.
template <int N, int CT>
__device__ __forceinline__ void modal_block(double (&v)[N]) {
    __shared__ double ws[N][CT / 32];
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = warp_sum(v[k]);
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int k = 0; k < N; ++k) ws[k][threadIdx.x >> 5] = v[k];
    __syncthreads();
    if (threadIdx.x < 32)
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] = warp_sum(threadIdx.x < CT / 32 ? ws[k][threadIdx.x] : 0.0);
}

// A control point's tile partials: the last tile that holds it, and which of the tiles before it do too.
struct ModalNode {
    long long at;       // its first component in that tile's patch
    int lo;             // bits 0-2: also the tile before along x, y, z
};
template <class T>
__device__ __forceinline__ ModalNode modal_locate(const ModalSys<T> &S, int n) {
    const Tiles &t = S.t;
    const int row = n / t.dcx, ix = n - row * S.cx, iz = row / t.dcy, iy = row - iz * S.cy;
    const TileAt tx = tile_at(ix, t.dx, t.tx, t.ntx), ty = tile_at(iy, t.dy, t.ty, t.nty), tz = tile_at(iz, t.dz, t.tz, t.ntz);
    ModalNode m;
    m.at = (long long)(tx.b + t.ntx * (ty.b + t.nty * tz.b)) * t.vol + (tz.l * (t.ty + 2) + ty.l) * (t.tx + 2) + tx.l;
    m.lo = (tx.two ? 1 : 0) | (ty.two ? 2 : 0) | (tz.two ? 4 : 0);
    return m;
}
// The partials of the tiles before along y and z added to sv, in a fixed order (read past the L1: other CTAs wrote
// them); the one before along x comes with the main one.
template <class T>
__device__ __forceinline__ void modal_others(const ModalSys<T> &S, const ModalNode &m, T (&sv)[3]) {
    const Tiles &t = S.t;
    const int w = t.tx + 2, plane = w * (t.ty + 2), comp = plane * (t.tz + 2);
    // from a control point's place in a tile to its place in the tile before
    const long long back[3] = {(long long)t.tx - t.vol, (long long)t.ty * w - (long long)t.ntx * t.vol,
                               (long long)t.tz * plane - (long long)t.ntx * t.nty * t.vol};
    T o[6][3];
#pragma unroll
    for (int k = 2; k < 8; ++k) {
        const bool on = (k & ~m.lo) == 0;
        const T *q = S.patch + m.at + (k & 1 ? back[0] : 0) + (k & 2 ? back[1] : 0) + (k & 4 ? back[2] : 0);
#pragma unroll
        for (int c = 0; c < 3; ++c) o[k - 2][c] = on ? __ldcg(q + c * comp) : T(0);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k)
#pragma unroll
        for (int c = 0; c < 3; ++c) sv[c] += o[k][c];
}

// `iters` PCG iterations (rust/src/solver.rs:38-71).  Per iteration: the apply with the new direction and
// p'Ap; barrier; the step length, then per control point Ap = the sum of the tile partials (never stored),
// x += alpha p, r -= alpha Ap and the exact r'r, r'z; barrier; stopping test and beta.  Every CTA forms the
// scalars from the same partial sums in the same order.  An operator with a sparse term stores Ap between the
// two (one barrier more: p'Ap needs the whole direction).  The loop ends when the state says so.
//
// One launch for many iterations instead of four (FP64) or two (FP32) per iteration, because at 24x16x12 an
// iteration is a chain of latencies (FP64, 24,000 clocks: the apply 10,100, the vector step 2,400, two sums over a CTA,
// two barriers and two totals of the CTAs' partials the rest) and the launches between them came on top: FP64 46 ->
// 12.6 us, FP32 27 -> 12.4 us an iteration.  At 128x64x64 the march bounds it: FP64 156,000 of 215,000 clocks, FP32
// 101,000 of 137,000 (447 -> 105 us and 97 -> 70 us).  The march
// has one CTA per SM: its state fills the SM's tensor memory and its exchange most of the shared memory.
//
// NT: columns of a march; kCubeOne or kCubePair for cubes, one or two at a time a CTA.  A system of no more cubes than
// SMs takes CTAs of one, of which an SM holds two, so that such systems on several streams (a batch of FP64
// solves, threads of the host) run beside one another: 16 FP64 designs of 24x12x12 to 32x16x16 in one call 80.8 -> 37.5
// ms, a mixed solve of 24x16x12 with eight threads at it 3.43 -> 2.02 ms, by itself 8.2 as before.  Three FP32 CTAs
// an SM spill (296 B; 16.0 us an iteration at 24x16x12 instead of 12.4).
constexpr int kCubeOne = 1, kCubePair = 2;
template <class T, int NT>
__host__ __device__ constexpr int modal_threads() { return NT <= kCubePair ? NT * kCubeThreads : ModalMarch<T>::max_nt; }

template <class T, int NT>
__global__ void __launch_bounds__((modal_threads<T, NT>()), NT == kCubeOne ? 2 : 1)
modal_pcg_kernel(const __grid_constant__ ModalK<T> K, const __grid_constant__ ModalSys<T> S, int iters, int *err, long long limit) {
    constexpr bool CUBE = NT <= kCubePair;
    constexpr int CT = modal_threads<T, NT>(), kGroups = CUBE ? CT / kCubeThreads : 1;
    extern __shared__ __align__(16) unsigned char modal_raw[];
    __shared__ uint32_t tmem_base;
    __shared__ PcgState st;
    const int tid = threadIdx.x;
    const int G = S.ncta, bid = (int)blockIdx.x;
    if (tid == 0) st = *S.st;
    __syncthreads();
    if (st.status != 0) return;   // the same for all CTAs of the system
    uint32_t tm = 0;
    if constexpr (!CUBE) tm = modal_tmem<T>(&tmem_base, 512);
    unsigned long long bars = (unsigned long long)st.bars;   // barriers this solve has passed
    T *const sm = reinterpret_cast<T *>(modal_raw);
    const bool masked = S.mask_mode != ICC_MASK_NONE;
    const int comp = S.t.vol / 3, stride = G * CT;
    for (int it = 0; it < iters; ++it) {
        const int par = int(st.iter & 1);
        const T *p_old = S.p[par];
        T *p = S.p[par ^ 1];
        double d[1] = {0.0};
        // tiles go to the CTAs first, then to a CTA's groups of threads
        if constexpr (CUBE) {
            const int group = tid / kCubeThreads;
            for (int tile = group * G + bid; tile < S.t.n; tile += G * kGroups)
                d[0] += modal_cube<T, true, kGroups == 1>(K, S, tile, tid & (kCubeThreads - 1), 1 + group, sm + group * kCubeSmem,
                                                          T(st.beta), p_old, p);
        } else {
            if (tid < NT)
                for (int tile = bid; tile < S.t.n; tile += G)
                    d[0] += modal_march<T, NT, true, NT == CT>(K, S, tile, sm, tm, T(st.beta), p_old, p);
        }
        if (S.dot) {
            modal_block<1, CT>(d);
            if (tid == 0) S.part_a[bid] = d[0];
        }
        if (!modal_barrier(S.bar, ++bars * G, err, limit)) break;
        if (!S.dot) {
            d[0] = 0.0;
            for (int n = bid * CT + tid; n < S.nsc; n += stride) {
                const ModalNode m = modal_locate(S, n);
                T sv[3];
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    sv[c] = __ldcg(S.patch + m.at + c * comp) + (m.lo & 1 ? __ldcg(S.patch + m.at + c * comp + S.t.tx - S.t.vol) : T(0));
                if (m.lo >> 1) modal_others(S, m, sv);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int i = c * S.nsc + n;
                    const T pi = __ldcg(p + i);
                    T a = sv[c] + sparse_row_cg(S.sp, i, p, S.mask, S.mask_mode);
                    if (masked && !S.mask[i]) a = S.mask_mode == ICC_MASK_ZERO ? T(0) : pi;
                    S.ap[i] = a;
                    d[0] += double(pi) * double(a);
                }
            }
            modal_block<1, CT>(d);
            if (tid == 0) S.part_a[bid] = d[0];
            if (!modal_barrier(S.bar, ++bars * G, err, limit)) break;
        }
        modal_total(S.part_a, G, d);
        if (tid == 0) pcg_alpha_step(&st, d[0]);
        __syncthreads();
        if (st.status != 0) break;
        const T alpha = T(st.alpha);
        double v[2] = {0.0, 0.0};
        // kU control points at a time, their loads issued together: a CTA per SM has few threads to hide a
        // trip to the L2 behind
        constexpr int kU = sizeof(T) == 8 ? (CUBE ? 1 : 3) : 2;
        for (int n0 = bid * CT + tid; n0 < S.nsc; n0 += kU * stride) {
            ModalNode m[kU];
            T sv[kU][3], sx[kU][3], pv[kU][3], xv[kU][3], rv[kU][3], iv[kU][3];
            bool on[kU][3];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int n = n0 + u * stride < S.nsc ? n0 + u * stride : n0;
                if (S.dot) m[u] = modal_locate(S, n);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int i = c * S.nsc + n;
                    sv[u][c] = S.dot ? __ldcg(S.patch + m[u].at + c * comp) : S.ap[i];   // Ap: this thread's own
                    sx[u][c] = S.dot && (m[u].lo & 1) ? __ldcg(S.patch + m[u].at + c * comp + S.t.tx - S.t.vol) : T(0);
                    pv[u][c] = __ldcg(p + i);
                    xv[u][c] = S.xs[i];
                    rv[u][c] = S.r[i];
                    iv[u][c] = S.inv[i];
                    on[u][c] = !masked || S.mask[i] != 0;
                }
            }
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int n = n0 + u * stride;
                if (n >= S.nsc) break;
                if (S.dot) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) sv[u][c] += sx[u][c];
                    if (m[u].lo >> 1) modal_others(S, m[u], sv[u]);
#pragma unroll
                    for (int c = 0; c < 3; ++c)
                        if (!on[u][c]) sv[u][c] = S.mask_mode == ICC_MASK_ZERO ? T(0) : pv[u][c];
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int i = c * S.nsc + n;
                    S.xs[i] = xv[u][c] + alpha * pv[u][c];
                    const T ri = rv[u][c] - alpha * sv[u][c], zi = iv[u][c] * ri;
                    S.r[i] = ri;
                    S.z[i] = zi;
                    v[0] += double(ri) * double(ri);
                    v[1] += double(ri) * double(zi);
                }
            }
        }
        modal_block<2, CT>(v);
        if (tid == 0) {
            S.part_v[bid] = v[0];
            S.part_v[G + bid] = v[1];
        }
        if (!modal_barrier(S.bar, ++bars * G, err, limit)) break;
        modal_total(S.part_v, G, v);
        if (tid < 32) {   // the two quotients side by side
            const double q = tid == 0 ? sqrt(v[0]) / st.norm_b : v[1] / st.rz_old, beta = __shfl_sync(0xffffffffu, q, 1);
            if (tid == 0) pcg_beta_step(&st, q, v[1], beta);
        }
        __syncthreads();
        if (st.status != 0) break;
    }
    if (bid == 0 && tid == 0) {
        st.bars = (long long)bars;
        if (*(volatile int *)err) st.status = kStatNan;   // a wait ran out: ends the launches queued behind this one too
        *S.st = st;
    }
    __syncthreads();
    if constexpr (!CUBE) {
        if (tid < 32) tc::tmem_dealloc(tmem_base, 512);
    }
}

// Host side (icc_modal.cu): the entries in the kernel's type, the grid part of a system's entry, the launches.
template <class T>
ModalK<T> modal_entries(const ModalHost &m);
template <class T>
ModalSys<T> modal_sys(const Op &op, const ModalTile &t);
template <class T>
[[nodiscard]] cudaError_t launch_modal_apply(cudaStream_t s, const ModalHost &m, const ModalSys<T> &S, const ModalTile &t);
// `iters` iterations of a system on S.ncta CTAs, in the form of `t`.
template <class T>
[[nodiscard]] cudaError_t launch_modal_pcg(cudaStream_t s, const ModalHost &m, const ModalSys<T> &S, const ModalTile &t, int iters,
                                           int *err, long long limit);

}  // namespace icc
