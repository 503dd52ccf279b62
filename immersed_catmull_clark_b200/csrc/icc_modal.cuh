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
// An element so costs about 700 operations instead of 81^2 = 6,561 multiply-adds.
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
    T kfac;                      // the system's element matrix = kfac * the launch's
    const T *scale;              // s_e
    const uint8_t *mask;
    int mask_mode;
    T *patch;                    // tile partial sums [tile][3][tz + 2][ty + 2][tx + 2]
    const T *x;                  // input of a plain apply
    // PCG: direction of iteration i in p[i & 1] (the next one is formed while it is read)
    const T *inv;
    T *r, *p[2], *xs, *ap;
    int p_zero;                  // directions are kept zero on fixed DOFs
    int dot;                     // the apply forms p'Ap and the step length (no sparse term)
    Sparse<T> sp;
    double *part_a, *part_v;     // partial sums: [tiles] of the apply, [2][ncta] of the vector step
    unsigned *counter;           // last-CTA counters: [0] apply, [1] vector step
    PcgState *st;
    int cta0, ncta;              // CTAs of the vector step that serve it
};

// Shared-memory row pitch of the staged control-point planes: lanes of different rows of a warp must
// fall into different banks.
template <class T>
__host__ __device__ __forceinline__ int modal_pitch(int ltx) {
    if (ltx >= 5) return (1 << ltx) + 2;
    if (sizeof(T) == 8) return ltx == 4 ? 18 : (ltx == 3 ? 24 : 20);
    return ltx == 4 ? 48 : (ltx == 3 ? 40 : 36);
}

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

template <class T, int NT>
struct ModalCfg {
    static constexpr int slots = NT >= 256 ? 4 : (NT == 128 ? 5 : 6);   // control values a thread stages per plane
    static constexpr int words = sizeof(T) / 4;
    static constexpr int cols = modal_col0(4, words);                    // 222 (FP64), 114 (FP32)
    static constexpr int need = cols * ((NT + 127) / 128);
    static constexpr int alloc = need <= 128 ? 128 : (need <= 256 ? 256 : 512);
    static constexpr int per_sm = NT >= 256 ? 1 : 512 / alloc;           // CTAs an SM can hold
};

// Shared memory: staged planes, the row exchange (27 values per column, two steps), arriving values.
template <class T>
size_t modal_smem(int nt, int ltx, int slots, bool pcg) {
    const size_t ring = (size_t)kModalRing * (3 * ((nt >> ltx) + 2) * modal_pitch<T>(ltx) + 1);
    return (ring + (size_t)2 * 27 * nt + (size_t)(pcg ? 3 : 1) * slots * nt) * sizeof(T);
}

__device__ __forceinline__ void cp_value(float *dst, const float *src) { tc::cp_async4(dst, src); }
__device__ __forceinline__ void cp_value(double *dst, const double *src) { tc::cp_async8(dst, src); }

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

// y = K x, tile by tile: a tile is tx x ty columns of elements, tz long in z; thread t marches along
// column (t % tx, t / tx).  Per plane of control points: the column's nine control values per
// component become modes along x and y; per element: modes along z, the sparse product, and the
// transposed z step into running sums of the three planes.  A finished plane goes back to control
// values along y (neighbouring columns summed through shared memory) and x (through shuffles),
// and the tile's sums are written as its patch; the node-side pass adds the patches that share a
// control point.  With PCG the input is formed on the fly, p = D^-1 r + beta p_old, and p'Ap and the
// step length come out of the same launch.  No atomics on data: results are bitwise reproducible.
template <class T, int NT, bool PCG, bool MANY>
__global__ void __launch_bounds__(NT, (ModalCfg<T, NT>::per_sm))
modal_apply_kernel(const __grid_constant__ ModalK<T> K, const __grid_constant__ ModalSys<T> one,
                   const ModalSys<T> *__restrict__ many, const int2 *__restrict__ list) {
    constexpr int kS = ModalCfg<T, NT>::slots, kW = ModalCfg<T, NT>::words;
    extern __shared__ __align__(16) unsigned char modal_raw[];
    T *sm = reinterpret_cast<T *>(modal_raw);

    // one system by value (its entry stays in the constant bank), or one of a table (staged in shared memory)
    __shared__ __align__(16) unsigned char s_sys[MANY ? sizeof(ModalSys<T>) : 16];
    int tile = blockIdx.x;
    if constexpr (MANY) {
        const int2 l = list[blockIdx.x];
        tile = l.y;
        const int *src = reinterpret_cast<const int *>(many + l.x);
        for (int i = threadIdx.x; i < (int)(sizeof(ModalSys<T>) / 4); i += NT) reinterpret_cast<int *>(s_sys)[i] = src[i];
        __syncthreads();
    }
    const ModalSys<T> &S = MANY ? *reinterpret_cast<const ModalSys<T> *>(s_sys) : one;
    T beta = T(0);
    const T *p_old = nullptr;
    T *p_new = nullptr;
    if (S.st && S.st->status != 0) return;   // the solve has stopped
    if constexpr (PCG) {
        beta = T(S.st->beta);
        const int par = int(S.st->iter & 1);
        p_old = S.p[par];
        p_new = S.p[par ^ 1];
    }
    const int tid = threadIdx.x;
    const int ltx = S.t.ltx, TX = 1 << ltx, TY = S.t.ty, TZ = S.t.tz;
    const int bx = tile % S.t.ntx, by = (tile / S.t.ntx) % S.t.nty, bz = tile / (S.t.ntx * S.t.nty);
    const int x0 = bx << ltx, y0 = by * TY, z0 = bz * TZ;
    const int lx = tid & (TX - 1), ly = tid >> ltx;
    const int pitch = modal_pitch<T>(ltx), rows = (NT >> ltx) + 2;
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
    // plane j's values on their way to this thread's slots (r, D^-1 and p_old, or x)
    auto fetch = [&](int j) {
#pragma unroll
        for (int s = 0; s < kS; ++s) {
            const int g = goff[s] + j * cxy;
            if constexpr (PCG) {
                cp_value(raw + s * NT, S.r + g);
                cp_value(raw + (kS + s) * NT, S.inv + g);
                cp_value(raw + (2 * kS + s) * NT, p_old + g);
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
                v = raw[(kS + s) * NT] * v + beta * raw[(2 * kS + s) * NT];
                if (zown && (own >> s & 1u)) {
                    p_new[goff[s] + j * cxy] = (S.p_zero && !mk[s]) ? T(0) : v;
                    if (S.mask_mode == ICC_MASK_IDENTITY && !mk[s]) dot += double(v) * double(v);
                }
            }
            dst[soff[s]] = (mk[s] && (in >> s & 1u)) ? v : T(0);
        }
    };

    // tensor memory: this thread's lane of the warp's quadrant, columns by groups of four warps
    __shared__ uint32_t tmem_base;
    if (tid < 32) {
        tc::tmem_alloc(&tmem_base, ModalCfg<T, NT>::alloc);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // the same for the warp, as its TMEM addresses are
    const uint32_t tm = tmem_base + ((uint32_t)(warp & 3) << 21) + (uint32_t)((warp >> 2) * ModalCfg<T, NT>::cols);
    {
        uint32_t z[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) z[i] = 0u;
#pragma unroll
        for (int i = 0; i + 16 <= ModalCfg<T, NT>::cols; i += 16) tc::tm_st<16>(tm + i, z);
        tc::tm_store<ModalCfg<T, NT>::cols % 16>(tm + ModalCfg<T, NT>::cols / 16 * 16, z);
        tc::tmem_wait_st();
    }

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
    __syncthreads();
    T s_next = T(0);
#pragma unroll 1
    for (int j = 0; j < np + 3; ++j) {
        if (j + 1 < np) fetch(j + 1);
        const T se = valid ? S.kfac * s_next : T(0);
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
                    tc::tm_load<2 * cnt * kW>(tp, pp);
                    // ---- the element matrix in the modes, and the transposed z step
                    bool first = true;
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int m = 0; m < 9; ++m) {
                            if (modal_class(c, m) != k4) continue;
                            T w[3];
#pragma unroll
                            for (int k = 0; k < 3; ++k) {
                                const int idx[3] = {m % 3, m / 3, k};
                                if (m == 0 && k == 0) {
                                    w[k] = T(0);
                                    continue;
                                }
                                T a = K.diag[c][m + 9 * k] * C[c][m + 9 * k];
#pragma unroll
                                for (int d = 0; d < 3; ++d) {
                                    if (d == c) continue;
                                    const int A = c < d ? c : d, B = c < d ? d : c, pr = A + B - 1, th = 3 - A - B;
                                    const int ia = idx[A], ib = idx[B], kt = idx[th];
                                    const int pw[3] = {1, 3, 9};
                                    // partner with A index - 1, B index + 1
                                    if (ia >= 1 && ib <= 1) {
                                        const int n2 = m + 9 * k - pw[A] + pw[B];
                                        a += (c == A ? K.off[pr][0][2 * (ia - 1) + ib][kt]
                                                     : K.off[pr][1][2 * (ia - 1) + ib][kt]) * C[d][n2];
                                    }
                                    // partner with A index + 1, B index - 1
                                    if (ia <= 1 && ib >= 1) {
                                        const int n2 = m + 9 * k + pw[A] - pw[B];
                                        a += (c == A ? K.off[pr][1][2 * ia + ib - 1][kt]
                                                     : K.off[pr][0][2 * ia + ib - 1][kt]) * C[d][n2];
                                    }
                                }
                                w[k] = a;
                            }
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
        __syncthreads();
    }
    if (tid < 32) tc::tmem_dealloc(tmem_base, ModalCfg<T, NT>::alloc);
    if constexpr (PCG) {
        if (!S.dot) return;
        dot = block_sum(dot);
        if (tid == 0) S.part_a[tile] = dot;
        if (last_block(S.counter, (unsigned)S.t.n)) {
            double s2 = 0.0;
            for (int i = tid; i < S.t.n; i += NT) s2 += __ldcg(S.part_a + i);
            s2 = block_sum(s2);
            if (tid == 0) pcg_alpha_step(S.st, s2);
        }
    }
}

// Host side (icc_modal.cu): the entries in the kernel's type, the grid part of a system's entry, the launch.
template <class T>
ModalK<T> modal_entries(const ModalHost &m);
template <class T>
ModalSys<T> modal_sys(const Op &op, const ModalTile &t);
template <class T>
cudaError_t launch_modal_apply(cudaStream_t s, const ModalK<T> &K, const ModalSys<T> &one, const ModalSys<T> *many,
                               const int2 *list, int ntiles, int nt, int ltx, bool pcg);

}  // namespace icc
