// Host side of the operator in Legendre modes (icc_modal.cuh): the test whether a handle's element
// matrices have that form, the choice of the tile, and the launches.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "icc_device.cuh"
#include "icc_vec.cuh"
#include "icc_modal.cuh"

namespace icc {

// ---- set-up ---------------------------------------------------------------------------------------

namespace {

// M <- (Az (x) Ay (x) Ax per component) M for 3 x 3 matrices (row-major): rows of M (81 x 81) combined one
// direction after the other
void rows_by(const double *Ax, const double *Ay, const double *Az, double *M) {
    const double *A[3] = {Ax, Ay, Az};
    const int st[3] = {1, 3, 9};
    const double unit[9] = {1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0};
    for (int d = 0; d < 3; ++d) {
        if (std::equal(unit, unit + 9, A[d])) continue;
        for (int i = 0; i < 81; ++i) {
            if ((i % 27) / st[d] % 3 != 0) continue;
            double *r0 = M + i * 81, *r1 = r0 + st[d] * 81, *r2 = r1 + st[d] * 81;
            const double *a = A[d];
            for (int j = 0; j < 81; ++j) {
                const double u = r0[j], v = r1[j], w = r2[j];
                r0[j] = a[0] * u + a[1] * v + a[2] * w;
                r1[j] = a[3] * u + a[4] * v + a[5] * w;
                r2[j] = a[6] * u + a[7] * v + a[8] * w;
            }
        }
    }
}

// out = L K L' with L = Az (x) Ay (x) Ax per component (81 x 81, row-major)
void congruence(const double *Ax, const double *Ay, const double *Az, const double *K, double *out) {
    double t[81 * 81];
    std::memcpy(t, K, sizeof(t));
    rows_by(Ax, Ay, Az, t);
    for (int i = 0; i < 81; ++i)
        for (int j = 0; j < 81; ++j) out[j * 81 + i] = t[i * 81 + j];
    rows_by(Ax, Ay, Az, out);
    for (int i = 0; i < 81; ++i)
        for (int j = 0; j < i; ++j) std::swap(out[i * 81 + j], out[j * 81 + i]);
}

}  // namespace

// The element's B-splines in terms of the translated ones, N = R B: R of an element whose end factors
// are a (first control value) and b (last): N_0 = a B_0, N_2 = b B_2, N_1 = B_1 + (1 - a) B_0 + (1 - b) B_2.
static void end_matrix(double a, double b, double r[9]) {
    const double m[9] = {a, 0.0, 0.0, 1.0 - a, 1.0, 1.0 - b, 0.0, 0.0, b};
    std::memcpy(r, m, sizeof(m));
}

bool modal_setup(const Op &op, ModalHost &m) {
    m.ok = false;
    const Geom &g = op.g;
    const int n[3] = {g.nx, g.ny, g.nz};
    if (op.ndof >= (1LL << 31) || op.nel >= (1LL << 31)) return false;   // 32-bit indices in the kernels
    // end factors of every 1-D type, from its basis values at the three Gauss points
    const double xg[3] = {-std::sqrt(0.6), 0.0, std::sqrt(0.6)};
    double bu[9];
    for (int q = 0; q < 3; ++q) {
        const double t = 0.5 * (xg[q] + 1.0);
        bu[q] = 0.5 * (1.0 - t) * (1.0 - t);
        bu[3 + q] = 0.5 + t - t * t;
        bu[6 + q] = 0.5 * t * t;
    }
    for (int d = 0; d < 3; ++d) {
        if ((int)op.host_type1d[d].size() != n[d] || op.host_basis1d[d].empty()) return false;
        m.a[d] = m.b[d] = 1.0;
        for (int e = 0; e < n[d]; ++e) {
            const auto &v = op.host_basis1d[d][(size_t)op.host_type1d[d][(size_t)e]];
            const double a = std::round(v[1] / bu[1]), b = std::round(v[7] / bu[7]);
            double r[9];
            end_matrix(a, b, r);
            for (int i = 0; i < 3; ++i)
                for (int q = 0; q < 3; ++q) {
                    const double w = r[3 * i] * bu[q] + r[3 * i + 1] * bu[3 + q] + r[3 * i + 2] * bu[6 + q];
                    if (!(std::fabs(w - v[(size_t)(3 * i + q)]) <= 1e-12)) return false;
                }
            if ((a != 1.0 && e != 0) || (b != 1.0 && e != n[d] - 1)) return false;
            if (e == 0) m.a[d] = a;
            if (e == n[d] - 1) m.b[d] = b;
        }
    }
    // the (element type, position class) pairs that occur; class 0 interior, 1 first, 2 last, 3 both
    std::vector<uint8_t> seen((size_t)op.ntypes * 64, 0);
    std::vector<long long> count((size_t)op.ntypes, 0);
    auto cls = [&](int d, int e) { return (e == 0 ? 1 : 0) | (e == n[d] - 1 ? 2 : 0); };
    for (int ez = 0, e = 0; ez < g.nz; ++ez)
        for (int ey = 0; ey < g.ny; ++ey) {
            const int cyz = 4 * cls(1, ey) + 16 * cls(2, ez);
            for (int ex = 0; ex < g.nx; ++ex, ++e) {
                const int t = op.host_type_id[(size_t)e];
                seen[(size_t)t * 64 + cls(0, ex) + cyz] = 1;
                count[(size_t)t]++;
            }
        }
    auto matrix_of = [&](int c, double R[3][9], bool inverse) {
        for (int d = 0; d < 3; ++d) {
            const int k = c >> (2 * d) & 3;
            const double a = k & 1 ? m.a[d] : 1.0, b = k & 2 ? m.b[d] : 1.0;
            if (!inverse) {
                end_matrix(a, b, R[d]);
            } else {
                const double w[9] = {1.0 / a, 0.0, 0.0, (a - 1.0) / a, 1.0, (b - 1.0) / b, 0.0, 0.0, 1.0 / b};
                std::memcpy(R[d], w, sizeof(w));
            }
        }
    };
    // the uniform matrix from the most frequent type, then its modes
    int mt = 0;
    for (int t = 1; t < op.ntypes; ++t)
        if (count[(size_t)t] > count[(size_t)mt]) mt = t;
    int mc = 0;
    while (!seen[(size_t)mt * 64 + mc]) ++mc;
    std::vector<double> ku(81 * 81), kl(81 * 81), kp(81 * 81, 0.0), kt(81 * 81);
    double R[3][9];
    matrix_of(mc, R, true);
    congruence(R[0], R[1], R[2], op.host_ktypes.data() + (size_t)mt * 81 * 81, ku.data());
    // rows: control values (u0, u1, u2) of the modes mean, slope, curvature
    const double sh[9] = {1.0, 1.0, 1.0, -0.5, 0.0, 0.5, 1.0 / 3.0, -1.0 / 6.0, 1.0 / 3.0};
    const double shinv_t[9] = {1.0 / 6.0, -1.0, 1.0, 2.0 / 3.0, 0.0, -2.0, 1.0 / 6.0, 1.0, 1.0};   // T', modes = T u
    congruence(sh, sh, sh, ku.data(), kl.data());
    const int pw[3] = {1, 3, 9};
    for (int c = 0; c < 3; ++c)
        for (int i = 0; i < 27; ++i) {
            const int r = c * 27 + i;
            m.diag[c][i] = i ? kl[(size_t)r * 81 + r] : 0.0;
            kp[(size_t)r * 81 + r] = m.diag[c][i];
        }
    std::memset(m.off, 0, sizeof(m.off));
    for (int A = 0; A < 3; ++A)
        for (int B = A + 1; B < 3; ++B)
            for (int i = 0; i < 27; ++i) {
                const int ia = i / pw[A] % 3, ib = i / pw[B] % 3, k = i / pw[3 - A - B] % 3, p = A + B - 1;
                for (int q = 0; q < 2; ++q) {
                    const bool on = q == 0 ? (ia >= 1 && ib <= 1) : (ia <= 1 && ib >= 1);
                    if (!on) continue;
                    const int r = A * 27 + i, s = B * 27 + (q == 0 ? i - pw[A] + pw[B] : i + pw[A] - pw[B]);
                    const double v = 0.5 * (kl[(size_t)r * 81 + s] + kl[(size_t)s * 81 + r]);
                    m.off[p][q][q == 0 ? 2 * (ia - 1) + ib : 2 * ia + ib - 1][k] = v;
                    kp[(size_t)r * 81 + s] = kp[(size_t)s * 81 + r] = v;
                }
            }
    // Every matrix that occurs must be the one of these entries, seen through its element's basis: in every column
    // (the response to one control value) to a quarter of the 1e-12 to which the apply follows the matrices given.
    // The knots i/n round, so a handle's own matrices are about 1e-16 n away: 1.5e-14 at n = 128, 2e-13 at 2,000;
    // longer grids may take the dense kernels.
    congruence(shinv_t, shinv_t, shinv_t, kp.data(), ku.data());
    constexpr double tol = 2.5e-13;
    for (int t = 0; t < op.ntypes; ++t)
        for (int c = 0; c < 64; ++c) {
            if (!seen[(size_t)t * 64 + c]) continue;
            matrix_of(c, R, false);
            congruence(R[0], R[1], R[2], ku.data(), kt.data());
            const double *K = op.host_ktypes.data() + (size_t)t * 81 * 81;
            double kmax = 0.0;   // the squares below must neither overflow nor vanish
            for (int i = 0; i < 81 * 81; ++i) kmax = std::fabs(K[i]) > kmax ? std::fabs(K[i]) : kmax;
            const double unit = kmax > 0.0 ? 1.0 / kmax : 1.0;
            double dev[81] = {}, norm[81] = {};
            for (int i = 0; i < 81; ++i)
                for (int j = 0; j < 81; ++j) {
                    const double k = K[i * 81 + j] * unit, d = kt[(size_t)i * 81 + j] * unit - k;
                    dev[j] += d * d;
                    norm[j] += k * k;
                }
            for (int j = 0; j < 81; ++j)
                if (!(dev[j] <= tol * tol * norm[j])) return false;
        }
    m.kunif = ku;
    m.ok = true;
    return true;
}

// ---- the tile ------------------------------------------------------------------------------------

// Cubes or a march, and its tile, by a model of the kernel in clocks (all measured with the kernels alone on the
// chip): a cube takes its share of an SM's pipes or its own latency, a march its steps (of elements and
// of planes alone) in rounds of one per SM; fewer columns make shorter steps.  Measured, us an iteration of
// solves forced to cubes / marches of 128 / 256 / 512 columns: FP32 12.4 / 21.1 / 23.0 at 24x16x12, 24.0 / 24.9 /
// 23.9 at 53x31x27, 148.9 / 114.8 / 77.8 / 69.8 at 128x64x64; FP64 12.6 / 22.3 / 26.1, 27.3 / 27.0 / 27.2 and
// 214 / 148 / 105 there.
template <class T>
static void modal_plan(const Geom &g, int sms, ModalTile &best) {
    const bool f64 = sizeof(T) == 8;
    const Tiles cubes = make_tiles(g.nx, g.ny, g.nz, kCube, kCube, kCube);
    double cost = std::fmax(f64 ? 7500.0 : 6700.0, (double)cubes.n / sms * (f64 ? 7000.0 : 4800.0));
    best.nt = 0;
    best.t = cubes;
    best.clocks = cost;
    // clocks of an element step and of a plane-only step by columns
    struct Step { int nt; double el, pl; };
    const Step f64_steps[] = {{128, 5400.0, 2400.0}, {256, 7000.0, 3100.0}};
    const Step f32_steps[] = {{128, 4850.0, 2150.0}, {256, 5800.0, 2500.0}, {512, 9200.0, 4100.0}};
    const Step *st = f64 ? f64_steps : f32_steps;
    for (int q = 0; q < (f64 ? 2 : 3); ++q) {
        for (int ltx = 5; ltx >= 4; --ltx) {
            const int tx = 1 << ltx, rows = st[q].nt >> ltx;
            if (tx == 32 && tx >= 2 * g.nx) continue;
            for (int nty = (g.ny + rows - 1) / rows, k = 0; k < 3; ++k, ++nty) {
                const int ty = (g.ny + nty - 1) / nty;
                if (ty < 2 && g.ny > 1) break;
                for (int ntz = 1; ntz <= g.nz; ++ntz) {
                    const int tz = (g.nz + ntz - 1) / ntz;
                    if (tz < 2 && g.nz > 1) break;
                    const double n = (double)((g.nx + tx - 1) / tx) * ((g.ny + ty - 1) / ty) * ((g.nz + tz - 1) / tz);
                    if (n > 1e9) break;
                    const double c = std::ceil(n / sms) * (tz * st[q].el + 5 * st[q].pl);
                    if (c < cost) {
                        cost = best.clocks = c;
                        best.nt = st[q].nt;
                        best.t = make_tiles(g.nx, g.ny, g.nz, tx, ty, tz);
                    }
                }
            }
        }
    }
}

// Of a plain apply (a CTA a tile) and of a solve (tiles dealt to a CTA per SM).
template <class T>
ModalTile modal_tile(const Geom &g, int num_sms) {
    ModalTile t;
    modal_plan<T>(g, num_sms, t);
    return t;
}
template ModalTile modal_tile<double>(const Geom &g, int num_sms);
template ModalTile modal_tile<float>(const Geom &g, int num_sms);

// CTAs of a solve of one system: no more than it has tiles or control points for.
int modal_ctas(const Geom &g, const ModalTile &t, int num_sms) {
    return std::min(num_sms, std::max(t.t.n, (int)((g.nsc + 511) / 512)));
}

// A launch takes every SM, so work on other streams waits until it ends: about 8 ms of an FP64 solve and 16 of a
// mixed one, by a model of an iteration's time (measured, us: FP64 12.6 at 24x16x12, 27 at 53x31x27, 105 at 128x64x64,
// 161 at 96^3; FP32 12.4, 24, 70, 102; the sparse term by its bytes).  The cuts cost nothing that shows (152.9 ms FP64 and
// 126.6 mixed at 128x64x64 with and without; mixed ones of 8 ms 0.15%).  The host looks after up to 16 launches of an
// FP64 solve, which stops once and whose queued launches then return at once, and after each one of a mixed solve,
// which leaves it for a replacement every 75 iterations or so.
ModalRun modal_run(const Op &op, bool f64, int check_every) {
    const double us = 12.5 + (f64 ? 1.8e-4 : 1.1e-4) * (double)op.nel + 5e-6 * (double)op.sp_nnz;
    const double want = 8.0 * check_every;
    ModalRun r;
    r.iters = (int)std::fmax(1.0, std::fmin(std::fmin(want, 1e6), std::floor((f64 ? 8000.0 : 16000.0) / us)));
    r.launches = (int)std::fmin(std::ceil(want / r.iters), f64 ? 16.0 : 1.0);
    return r;
}

// ---- launches -------------------------------------------------------------------------------------

template <class T>
ModalK<T> modal_entries(const ModalHost &m) {
    ModalK<T> k;
    for (int c = 0; c < 3; ++c)
        for (int i = 0; i < 27; ++i) k.diag[c][i] = T(m.diag[c][i]);
    for (int p = 0; p < 3; ++p)
        for (int q = 0; q < 2; ++q)
            for (int n = 0; n < 4; ++n)
                for (int l = 0; l < 3; ++l) k.off[p][q][n][l] = T(m.off[p][q][n][l]);
    return k;
}

constexpr int kMaxDynSmem = 224 * 1024;   // beside the kernels' static 1.7 KB

template <class T, int NT>
static cudaError_t launch_march(cudaStream_t s, const ModalK<T> &K, const ModalSys<T> &S, const ModalTile &t) {
    const cudaError_t e = cudaFuncSetAttribute(modal_march_kernel<T, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
    if (e != cudaSuccess) return e;
    modal_march_kernel<T, NT><<<t.t.n, NT, march_smem(NT, t.t.ltx, false) * sizeof(T), s>>>(K, S);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_modal_apply(cudaStream_t s, const ModalHost &m, const ModalSys<T> &S, const ModalTile &t) {
    const ModalK<T> K = modal_entries<T>(m);
    if (t.nt == 0) {
        const cudaError_t e = cudaFuncSetAttribute(modal_cube_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
        if (e != cudaSuccess) return e;
        modal_cube_kernel<T><<<t.t.n, kCubeThreads, kCubeSmem * sizeof(T), s>>>(K, S);
        return cudaGetLastError();
    }
    if (t.nt == 128) return launch_march<T, 128>(s, K, S, t);
    if (t.nt == 256) return launch_march<T, 256>(s, K, S, t);
    if constexpr (sizeof(T) == 4) return launch_march<T, 512>(s, K, S, t);
    return cudaErrorInvalidValue;
}
template cudaError_t launch_modal_apply<double>(cudaStream_t, const ModalHost &, const ModalSys<double> &, const ModalTile &);
template cudaError_t launch_modal_apply<float>(cudaStream_t, const ModalHost &, const ModalSys<float> &, const ModalTile &);

// Every CTA of a march takes more than half of an SM's shared memory, so two of these kernels (two solves on
// two streams) never share an SM: tensor memory is then always there for a resident CTA, and no CTA waits
// for it while others wait for that CTA at a barrier.  Cubes use no tensor memory.
template <class T, int NT>
static cudaError_t launch_pcg(cudaStream_t s, const ModalHost &m, const ModalSys<T> &S, const ModalTile &t, int iters, int *err,
                              long long limit) {
    constexpr bool cube = NT <= kCubePair;
    const size_t smem = (size_t)(cube ? NT * kCubeSmem : march_smem(NT, t.t.ltx, true)) * sizeof(T);
    cudaError_t e = cudaFuncSetAttribute(modal_pcg_kernel<T, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)S.ncta);
    cfg.blockDim = dim3(modal_threads<T, NT>());
    cfg.dynamicSmemBytes = cube ? smem : std::max(smem, (size_t)120 * 1024);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;   // the barriers need every CTA resident
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, modal_pcg_kernel<T, NT>, modal_entries<T>(m), S, iters, err, limit);
}

template <class T>
cudaError_t launch_modal_pcg(cudaStream_t s, const ModalHost &m, const ModalSys<T> &S, const ModalTile &t, int iters, int *err,
                             long long limit) {
    if (t.nt == 0)
        return t.t.n <= S.ncta ? launch_pcg<T, kCubeOne>(s, m, S, t, iters, err, limit) : launch_pcg<T, kCubePair>(s, m, S, t, iters, err, limit);
    if (t.nt == 128) return launch_pcg<T, 128>(s, m, S, t, iters, err, limit);
    if (t.nt == 256) return launch_pcg<T, 256>(s, m, S, t, iters, err, limit);
    if constexpr (sizeof(T) == 4) return launch_pcg<T, 512>(s, m, S, t, iters, err, limit);
    return cudaErrorInvalidValue;
}
template cudaError_t launch_modal_pcg<double>(cudaStream_t, const ModalHost &, const ModalSys<double> &, const ModalTile &, int,
                                              int *, long long);
template cudaError_t launch_modal_pcg<float>(cudaStream_t, const ModalHost &, const ModalSys<float> &, const ModalTile &, int,
                                             int *, long long);

// The grid part of a system's entry.
template <class T>
ModalSys<T> modal_sys(const Op &op, const ModalTile &t) {
    ModalSys<T> S;
    std::memset((void *)&S, 0, sizeof(S));
    const Geom &g = op.g;
    S.nx = g.nx; S.ny = g.ny; S.nz = g.nz;
    S.cx = g.cx; S.cy = g.cy; S.cz = g.cz;
    S.nsc = (int)g.nsc;
    S.t = t.t;
    for (int d = 0; d < 3; ++d) {
        S.a[d] = T(op.modal.a[d]);
        S.b[d] = T(op.modal.b[d]);
    }
    S.mask = op.d_mask;
    S.mask_mode = op.mask_mode;
    return S;
}
template ModalSys<double> modal_sys<double>(const Op &op, const ModalTile &t);
template ModalSys<float> modal_sys<float>(const Op &op, const ModalTile &t);

}  // namespace icc
