// Bandwidth kernels between the packed doubles and full (v,o,v,o) arrays (FP64).
//
// For a fixed occupied pair i <= j the packed element of (ai, bj) is T_ij[a, b], contiguous along a
// (ai never exceeds bj for i < j), and everything the full forms need of it lies in the same pair:
// S_aibj = T[a, b], S_ajbi = T[b, a], and the mirrored block (bj, ai) is the transpose.  A block of
// threads therefore takes one occupied pair and a 32 x 32 tile of (a, b) with its mirror tile: each
// packed element is read once, each full element written (or read) once, all along a.
#include <algorithm>
#include <type_traits>

#include "amp_forms.cuh"

namespace ccsd {

namespace {

constexpr int TILE = 32, ROWS = 8;
// 48 warps of sym_pack on an SM: 0.35 ms at o=32, v=320 where its natural 78 registers (24 warps) take 0.51 ms
constexpr int MIN_BLOCKS = 6;

// (M, m) with M >= m from M(M+1)/2 + m
__device__ __forceinline__ void untri32(unsigned idx, int &M, int &m) {
    int r = (int)((sqrt(8.0 * (double)idx + 1.0) - 1.0) * 0.5);
    while ((unsigned)r * (unsigned)(r + 1) / 2 > idx) r--;
    while ((unsigned)(r + 1) * (unsigned)(r + 2) / 2 <= idx) r++;
    M = r;
    m = (int)(idx - (unsigned)r * (unsigned)(r + 1) / 2);
}

__device__ __forceinline__ int64_t packed_at(int64_t x, int64_t y) {
    const int64_t M = x > y ? x : y, m = x > y ? y : x;
    return M * (M + 1) / 2 + m;
}

__device__ __forceinline__ void put(double *p, double v, int acc) { *p = acc ? *p + v : v; }

// Bound by HBM: n_t2 read, 2 (o v)^2 written.  At o=32, v=320 it takes 0.41 ms (5.1 TB/s) where the
// element-wise square-up and the two exchange passes that formed u took 1.19 ms.
__global__ void __launch_bounds__(TILE * ROWS)
square_forms_kernel(const double *__restrict__ packed, int no, int nv, int64_t nvec, double c1, double c2,
                    double *__restrict__ S, double *__restrict__ U, int acc_s, int acc_u) {
    __shared__ double t1[TILE][TILE + 1], t2[TILE][TILE + 1];   // T[a0 + x, b0 + r], T[b0 + x, a0 + r] at [r][x]
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int64_t nov = (int64_t)no * nv, nt2 = nov * (nov + 1) / 2;
    const int64_t npair = (int64_t)no * (no + 1) / 2;
    int at, bt, i, j;
    untri32(blockIdx.x, bt, at);
    const int a0 = TILE * at, b0 = TILE * bt;
    const bool mirror = at != bt;
    for (int64_t w = blockIdx.y; w < npair * nvec; w += gridDim.y) {
        const int64_t n = w / npair, vec = nov * nov * n;
        untri32((unsigned)(w - n * npair), j, i);
        const double *p = packed + nt2 * n;
        for (int r = ty; r < TILE; r += ROWS) {
            if (a0 + tx < nv && b0 + r < nv) t1[r][tx] = p[packed_at(a0 + tx + (int64_t)nv * i, b0 + r + (int64_t)nv * j)];
            if (mirror && b0 + tx < nv && a0 + r < nv)
                t2[r][tx] = p[packed_at(b0 + tx + (int64_t)nv * i, a0 + r + (int64_t)nv * j)];
        }
        __syncthreads();
        double(*m2)[TILE + 1] = mirror ? t2 : t1;
        for (int r = ty; r < TILE; r += ROWS) {
#pragma unroll
            for (int side = 0; side < 2; side++) {
                if (side && !mirror) break;
                const int x = (side ? b0 : a0) + tx, y = (side ? a0 : b0) + r;
                if (x >= nv || y >= nv) continue;
                const double d = side ? m2[r][tx] : t1[r][tx];       // T[x, y]
                const double e = side ? t1[tx][r] : m2[tx][r];       // T[y, x]
                const int64_t ij = vec + x + (int64_t)nv * i + nov * (y + (int64_t)nv * j);
                const int64_t ji = vec + x + (int64_t)nv * j + nov * (y + (int64_t)nv * i);
                if (S) put(S + ij, d, acc_s);
                if (U) put(U + ij, c1 * d + c2 * e, acc_u);
                if (i != j) {
                    if (S) put(S + ji, e, acc_s);
                    if (U) put(U + ji, c1 * e + c2 * d, acc_u);
                }
            }
        }
        __syncthreads();
    }
}

// Bound by HBM: F and X read once, n_t2 written.  At o=32, v=320 0.35 ms (5.9 TB/s); adding the two
// forms of X to F in passes of their own and packing the sum took 1.26 ms.
template <bool HAS_F, bool HAS_X, bool ACC>
__global__ void __launch_bounds__(TILE * ROWS, MIN_BLOCKS)
sym_pack_kernel(const double *__restrict__ F, const double *__restrict__ X, int no, int nv, int64_t nvec, double c1,
                double c2, double *__restrict__ packed) {
    constexpr int N = TILE / ROWS;
    __shared__ double s1[TILE][TILE + 1], s2[TILE][TILE + 1];   // Z_ji of the tile and of its mirror
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int64_t nov = (int64_t)no * nv, nt2 = nov * (nov + 1) / 2;
    const int64_t npair = (int64_t)no * (no + 1) / 2;
    int at, bt, i, j;
    untri32(blockIdx.x, bt, at);
    const int a0 = TILE * at, b0 = TILE * bt;
    const bool mirror = at != bt;
    for (int64_t w = blockIdx.y; w < npair * nvec; w += gridDim.y) {
        const int64_t n = w / npair, vec = nov * nov * n;
        untri32((unsigned)(w - n * npair), j, i);
        double *p = packed + nt2 * n;
        double z[2][N];     // Z_ij of the two tiles
        double old[2][N];   // what the results are added to, loaded before any store
#pragma unroll
        for (int side = 0; side < 2; side++) {
            if (side && !mirror) break;
#pragma unroll
            for (int k = 0; k < N; k++) {
                const int r = ty + ROWS * k;
                const int x = (side ? b0 : a0) + tx, y = (side ? a0 : b0) + r;
                double zij = 0.0, zji = 0.0;
                if (x < nv && y < nv) {
                    if (ACC) {
                        const int64_t M = y + (int64_t)nv * j;   // i == j: the other triangle is not stored
                        old[side][k] = i == j && x > y ? 0.0 : p[M * (M + 1) / 2 + x + (int64_t)nv * i];
                    }
                    const int64_t ij = vec + x + (int64_t)nv * i + nov * (y + (int64_t)nv * j);
                    const int64_t ji = vec + x + (int64_t)nv * j + nov * (y + (int64_t)nv * i);
                    if (HAS_F) {
                        zij = F[ij];
                        zji = F[ji];
                    }
                    if (HAS_X) {
                        const double xij = X[ij], xji = X[ji];
                        zij += c1 * xij + c2 * xji;
                        zji += c1 * xji + c2 * xij;
                    }
                }
                z[side][k] = zij;
                if (side) s2[r][tx] = zji;
                else s1[r][tx] = zji;
            }
        }
        __syncthreads();
        double(*m2)[TILE + 1] = mirror ? s2 : s1;
#pragma unroll
        for (int side = 0; side < 2; side++) {
            if (side && (!mirror || i == j)) break;   // i == j: the mirror tile is the other triangle
#pragma unroll
            for (int k = 0; k < N; k++) {
                const int r = ty + ROWS * k;
                const int x = (side ? b0 : a0) + tx, y = (side ? a0 : b0) + r;
                if (x >= nv || y >= nv || (i == j && x > y)) continue;
                double v = z[side][k] + (side ? s1[tx][r] : m2[tx][r]);
                if (i == j && x == y) v *= 0.5;
                const int64_t M = y + (int64_t)nv * j;
                p[M * (M + 1) / 2 + x + (int64_t)nv * i] = ACC ? old[side][k] + v : v;
            }
        }
        __syncthreads();
    }
}

struct TpmOut {
    double *p, *m;                 // FP64 columns
    __nv_bfloat16 *bp, *bm;        // or bf16 planes
    int64_t ldp, ldm, plane_p, plane_m;
    int np;
    int64_t rows_p, rows_m;        // rows of a plane; those beyond the vectors' pairs are cleared
};

__device__ __forceinline__ void put_planes(double x, int np, int64_t plane, __nv_bfloat16 *out) {
    for (int q = 0; q < np; q++) {
        const __nv_bfloat16 h = __double2bfloat16(x);
        out[q * plane] = h;
        x -= (double)__bfloat162float(h);
    }
}

// The padding of one form's planes: K positions beyond the k pairs cd and rows beyond the used ones (ld is a
// multiple of 8), shared out over the whole grid.  As up to four 2-D memsets before the kernel a residual at o=13,
// v=107 took 1.081 ms, so 1.067; from o=16, v=128 on it makes no difference.
__device__ __forceinline__ void clear_pads(__nv_bfloat16 *t, int np, int64_t rows, int64_t used, int64_t ld, int64_t k) {
    const int64_t id = ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * (TILE * ROWS) + threadIdx.y * TILE + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * gridDim.y * (TILE * ROWS);
    const int pad = (int)(ld - k);
    for (int64_t x = id; x < (int64_t)np * used * pad; x += step) {
        const int64_t row = x / pad, q = row / used;   // plane q
        t[(q * rows + row - q * used) * ld + k + (x - row * pad)] = __float2bfloat16(0.0f);
    }
    const int64_t tail = (rows - used) * ld / 8;
    for (int64_t x = id; x < np * tail; x += step) {
        const int64_t q = x / tail;
        reinterpret_cast<uint4 *>(t + (q * rows + used) * ld)[x - q * tail] = make_uint4(0, 0, 0, 0);
    }
}

// An occupied pair i >= j and a 32 x 32 tile of (c, d), c >= d: t_cidj lies along d in its packed row
// (c, i), t_cjdi along c in row (d, i), turned in shared memory; both forms are stored along d.  Bound by
// HBM: n_t2 read, the forms written; each thread of the element-wise version found its four indices by two
// square roots and read two elements whose neighbours lay a packed row apart.  bf16 planes at o=32, v=320
// 0.34 ms (1.9 TB/s; 0.38 with the padding), 0.54 without MIN_BLOCKS.
template <bool PLANES>
__global__ void __launch_bounds__(TILE * ROWS, MIN_BLOCKS)
tpm_forms_kernel(const double *__restrict__ packed, int no, int nv, int64_t nvec, TpmOut o) {
    __shared__ double s[TILE][TILE + 1];   // t_cjdi of (c0 + x, d0 + r) at [r][x]
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int64_t nov = (int64_t)no * nv, nt2 = nov * (nov + 1) / 2;
    const int64_t nop = (int64_t)no * (no + 1) / 2, nom = (int64_t)no * (no - 1) / 2;
    if (PLANES) {
        clear_pads(o.bp, o.np, o.rows_p, nvec * nop, o.ldp, (int64_t)nv * (nv + 1) / 2);
        clear_pads(o.bm, o.np, o.rows_m, nvec * nom, o.ldm, (int64_t)nv * (nv - 1) / 2);
    }
    int ct, dt, i, j;
    untri32(blockIdx.x, ct, dt);
    const int c0 = TILE * ct, d0 = TILE * dt;
    for (int64_t w = blockIdx.y; w < nop * nvec; w += gridDim.y) {
        const int64_t n = w / nop;
        untri32((unsigned)(w - n * nop), i, j);
        const double *p = packed + nt2 * n;
        double x[TILE / ROWS];
#pragma unroll
        for (int k = 0; k < TILE / ROWS; k++) {
            const int r = ty + ROWS * k;
            if (c0 + tx < nv && d0 + r < nv) s[r][tx] = p[packed_at(d0 + r + (int64_t)nv * i, c0 + tx + (int64_t)nv * j)];
            x[k] = c0 + r < nv && d0 + tx <= c0 + r ? p[packed_at(c0 + r + (int64_t)nv * i, d0 + tx + (int64_t)nv * j)] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < TILE / ROWS; k++) {
            const int c = c0 + ty + ROWS * k, d = d0 + tx;
            if (c >= nv || d > c) continue;
            const double y = s[tx][ty + ROWS * k];
            const double f = (c == d ? 0.5 : 1.0) * (i == j ? 0.5 : 1.0);
            const int64_t at = w * o.ldp + (int64_t)c * (c + 1) / 2 + d;
            if (PLANES) put_planes(f * (x[k] + y), o.np, o.plane_p, o.bp + at);
            else o.p[at] = f * (x[k] + y);
            if (i > j && c > d) {
                const int64_t am = (n * nom + (int64_t)i * (i - 1) / 2 + j) * o.ldm + (int64_t)c * (c - 1) / 2 + d;
                if (PLANES) put_planes(x[k] - y, o.np, o.plane_m, o.bm + am);
                else o.m[am] = x[k] - y;
            }
        }
        __syncthreads();
    }
}

// An occupied pair i >= j and a 32 x 32 tile of (a, b), a >= b: w+- are read along b, Omega_aibj is added
// to along b in its packed row (a, i), Omega_ajbi along a in row (b, i) through shared memory.  Bound by
// HBM: w+- read, n_t2 read and written.  The element-wise version ran along ij, so that neighbouring threads
// updated packed rows far apart: 1.37 ms at o=32, v=320; so 0.34 (3.7 TB/s), 0.54
// without MIN_BLOCKS.
__global__ void __launch_bounds__(TILE * ROWS, MIN_BLOCKS)
add_omega_pm_kernel(double *__restrict__ om2, const double *__restrict__ wp, const double *__restrict__ wm, int no, int nv,
                    int64_t nvec, int a0, int a1, int64_t ldwp, int64_t ldwm) {
    __shared__ double s[TILE][TILE + 1];   // the Omega_ajbi share of (a, b) at [a][b]
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int64_t nov = (int64_t)no * nv, nt2 = nov * (nov + 1) / 2;
    const int64_t nop = (int64_t)no * (no + 1) / 2, nom = (int64_t)no * (no - 1) / 2;
    const int at0 = a0 / TILE, nbt = (a1 - 1) / TILE + 1;
    const int at = at0 + (int)blockIdx.x / nbt, bt = (int)blockIdx.x % nbt;
    if (bt > at) return;
    const int64_t row0 = (int64_t)a0 * (a0 + 1) / 2, row0m = (int64_t)a0 * (a0 - 1) / 2;
    for (int64_t w = blockIdx.y; w < nop * nvec; w += gridDim.y) {
        const int64_t n = w / nop;
        int i, j;
        untri32((unsigned)(w - n * nop), i, j);
        const int64_t cm = n * nom + (int64_t)i * (i - 1) / 2 + j;
        double *om = om2 + nt2 * n;
        double v[TILE / ROWS], old[TILE / ROWS];
#pragma unroll
        for (int k = 0; k < TILE / ROWS; k++) {
            const int a = TILE * at + ty + ROWS * k, b = TILE * bt + tx;
            double x1 = 0.0, x2 = 0.0;
            old[k] = 0.0;
            if (a >= a0 && a < a1 && b <= a) {
                const int64_t M = a + (int64_t)nv * i;
                old[k] = om[M * (M + 1) / 2 + b + (int64_t)nv * j];
                const double p = wp[(int64_t)a * (a + 1) / 2 + b - row0 + ldwp * w] * (a == b ? 0.5 : 1.0);
                if (i == j || a == b) {
                    x1 = p + p;   // both shares fall on one element
                } else {
                    const double m = wm[(int64_t)a * (a - 1) / 2 + b - row0m + ldwm * cm];
                    x1 = p + m;
                    x2 = p - m;
                }
            }
            v[k] = x1;
            s[ty + ROWS * k][tx] = x2;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < TILE / ROWS; k++) {
            const int a = TILE * at + ty + ROWS * k, b = TILE * bt + tx;
            if (a >= a0 && a < a1 && b <= a) {
                const int64_t M = a + (int64_t)nv * i;
                om[M * (M + 1) / 2 + b + (int64_t)nv * j] = old[k] + v[k];
            }
        }
        if (i != j) {
            double e[TILE / ROWS];
#pragma unroll
            for (int k = 0; k < TILE / ROWS; k++) {
                const int b = TILE * bt + ty + ROWS * k, a = TILE * at + tx;
                const int64_t M = b + (int64_t)nv * i;
                e[k] = a >= a0 && a < a1 && b < a ? om[M * (M + 1) / 2 + a + (int64_t)nv * j] : 0.0;
            }
#pragma unroll
            for (int k = 0; k < TILE / ROWS; k++) {
                const int b = TILE * bt + ty + ROWS * k, a = TILE * at + tx;
                const int64_t M = b + (int64_t)nv * i;
                if (a >= a0 && a < a1 && b < a) om[M * (M + 1) / 2 + a + (int64_t)nv * j] = e[k] + s[tx][ty + ROWS * k];
            }
        }
        __syncthreads();
    }
}

dim3 pair_grid(int64_t no, int64_t nv, int64_t nvec) {
    const int64_t nt = (nv + TILE - 1) / TILE;
    return dim3((unsigned)(nt * (nt + 1) / 2), (unsigned)std::min<int64_t>(no * (no + 1) / 2 * nvec, 65535));
}

}  // namespace

void square_forms(Exec &ex, const double *p, int64_t no, int64_t nv, int64_t nvec, double c1, double c2, double *S,
                  double *U, bool acc_s, bool acc_u) {
    square_forms_kernel<<<pair_grid(no, nv, nvec), dim3(TILE, ROWS), 0, ex.stream>>>(p, (int)no, (int)nv, nvec, c1, c2, S,
                                                                                    U, acc_s, acc_u);
    ex.launches++;
    CU_CHECK(cudaGetLastError());
}

void sym_pack(Exec &ex, const double *F, const double *X, int64_t no, int64_t nv, int64_t nvec, double c1, double c2,
              double *p, bool accumulate) {
    auto run = [&](auto f, auto x, auto acc) {
        sym_pack_kernel<decltype(f)::value, decltype(x)::value, decltype(acc)::value>
            <<<pair_grid(no, nv, nvec), dim3(TILE, ROWS), 0, ex.stream>>>(F, X, (int)no, (int)nv, nvec, c1, c2, p);
    };
    const std::true_type yes;
    const std::false_type none;
    auto pick = [&](auto f, auto x) { accumulate ? run(f, x, yes) : run(f, x, none); };
    if (F && X) pick(yes, yes);
    else if (F) pick(yes, none);
    else pick(none, yes);
    ex.launches++;
    CU_CHECK(cudaGetLastError());
}

void build_tpm(Exec &ex, const double *t2, int64_t no, int64_t nv, int64_t nvec, double *tp, int64_t ldp, double *tm,
               int64_t ldm) {
    const TpmOut o{tp, tm, nullptr, nullptr, ldp, ldm, 0, 0, 0, 0, 0};
    tpm_forms_kernel<false><<<pair_grid(no, nv, nvec), dim3(TILE, ROWS), 0, ex.stream>>>(t2, (int)no, (int)nv, nvec, o);
    ex.launches++;
    CU_CHECK(cudaGetLastError());
}

void build_tpm_planes(Exec &ex, const double *t2, int64_t no, int64_t nv, int64_t nvec, int np, __nv_bfloat16 *tp,
                      int64_t rows_p, int64_t ldp, __nv_bfloat16 *tm, int64_t rows_m, int64_t ldm) {
    const TpmOut o{nullptr, nullptr, tp, tm, ldp, ldm, rows_p * ldp, rows_m * ldm, np, rows_p, rows_m};
    tpm_forms_kernel<true><<<pair_grid(no, nv, nvec), dim3(TILE, ROWS), 0, ex.stream>>>(t2, (int)no, (int)nv, nvec, o);
    ex.launches++;
    CU_CHECK(cudaGetLastError());
}

void add_omega_pm(Exec &ex, double *om2, const double *wp, const double *wm, int64_t no, int64_t nv, int64_t nvec,
                  int64_t a0, int64_t a1, int64_t ldwp, int64_t ldwm) {
    if (a1 <= a0) return;
    const int64_t nbt = (a1 - 1) / TILE + 1, nat = nbt - a0 / TILE;
    const dim3 g((unsigned)(nat * nbt), (unsigned)std::min<int64_t>(no * (no + 1) / 2 * nvec, 65535));
    add_omega_pm_kernel<<<g, dim3(TILE, ROWS), 0, ex.stream>>>(om2, wp, wm, (int)no, (int)nv, nvec, (int)a0, (int)a1,
                                                              ldwp, ldwm);
    ex.launches++;
    CU_CHECK(cudaGetLastError());
}

}  // namespace ccsd
