// Tensor primitives: strided permutations (smem-tiled when the fastest index changes),
// GEMM-backed contractions, packed-doubles conversions and deterministic reductions.
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "autotune.cuh"
#include "mixed_gemm.cuh"
#include "ozaki_gemm.cuh"
#include "tensor_ops.cuh"

namespace ccsd {

namespace {

constexpr int MAXD = 6;

struct PermArgs {
    int nd;
    int64_t n[MAXD];
    int64_t si[MAXD];
    int64_t so[MAXD];
};

// Index arithmetic in I: 32-bit divisions wherever the count of rows, tiles or elements allows, a third of the
// 64-bit chain's time, which is what bounds these kernels on small tensors.
template <class I>
__device__ __forceinline__ void locate(const PermArgs &a, int first, I r, int64_t &oi, int64_t &oo) {
#pragma unroll
    for (int d = 0; d < MAXD; d++) {
        if (d >= first && d < a.nd) {
            const I n = (I)a.n[d], q = r / n, i = r - q * n;
            r = q;
            oi += (int64_t)i * a.si[d];
            oo += (int64_t)i * a.so[d];
        }
    }
}

// One output element per thread; dims are ordered by output stride (dim 0 fastest).
template <class I>
__global__ void permute_simple_kernel(PermArgs a, int64_t total, double alpha, const double *__restrict__ in,
                                      double beta, double *__restrict__ out) {
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        int64_t oi = 0, oo = 0;
        locate<I>(a, 0, (I)idx, oi, oo);
        double v = alpha * in[oi];
        if (beta != 0.0) v += beta * out[oo];
        out[oo] = v;
    }
}

// Rows of the output-fastest dim (dim 0, at least 16 long): a warp takes a row or a segment of a long one, so the
// division chain that locates it in the other dims runs once per row instead of once per element, and both sides
// stream along dim 0 (this kernel serves permutations whose input-fastest dim is dim 0 as well, or whose other
// dims are too short for the tiled transpose).  Bound by HBM or, for rows of a few hundred, by loads in flight:
// four per lane.
template <class I>
__global__ void __launch_bounds__(256) permute_rows_kernel(PermArgs a, int64_t nwork, int nseg, int seg, double alpha,
                                                           const double *__restrict__ in, double beta,
                                                           double *__restrict__ out) {
    const int64_t n0 = a.n[0], si0 = a.si[0], so0 = a.so[0];
    for (int64_t w = (int64_t)blockIdx.x * 8 + threadIdx.y; w < nwork; w += (int64_t)gridDim.x * 8) {
        I row = (I)w;
        int64_t lo = 0, oi = 0, oo = 0;
        if (nseg > 1) {
            const I q = row / (I)nseg;
            lo = (int64_t)(row - q * (I)nseg) * seg;
            row = q;
        }
        locate<I>(a, 1, row, oi, oo);
        const int64_t end = nseg > 1 ? min(n0, lo + seg) : n0;
        const double *src = in + oi;
        double *dst = out + oo;
        for (int64_t i0 = lo + threadIdx.x; i0 < end; i0 += 128) {
            double v[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int64_t i = i0 + 32 * k;
                v[k] = i < end ? alpha * src[i * si0] : 0.0;
            }
            if (beta != 0.0) {
                double old[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int64_t i = i0 + 32 * k;
                    old[k] = i < end ? dst[i * so0] : 0.0;
                }
#pragma unroll
                for (int k = 0; k < 4; k++) v[k] += beta * old[k];
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int64_t i = i0 + 32 * k;
                if (i < end) dst[i * so0] = v[k];
            }
        }
    }
}

// 32x32 tile over (p = input-fastest dim, q = output-fastest dim); the remaining dims
// are flattened into the z loop.  Dims 2.. of `a` are the batch dims.
template <class I>
__global__ void __launch_bounds__(256) permute_tiled_kernel(PermArgs a, int64_t nbatch, double alpha,
                                                            const double *__restrict__ in, double beta,
                                                            double *__restrict__ out) {
    __shared__ double tile[32][33];
    const int64_t np = a.n[0], nq = a.n[1];
    const int64_t p0 = (int64_t)blockIdx.x * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int64_t b = blockIdx.z; b < nbatch; b += gridDim.z) {
        int64_t bi = 0, bo = 0;
        locate<I>(a, 2, (I)b, bi, bo);
        for (int64_t q0 = (int64_t)blockIdx.y * 32; q0 < nq; q0 += (int64_t)gridDim.y * 32) {
            double v[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int64_t p = p0 + tx, q = q0 + ty + 8 * k;
                v[k] = p < np && q < nq ? in[bi + p * a.si[0] + q * a.si[1]] : 0.0;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) tile[ty + 8 * k][tx] = v[k];
            __syncthreads();
            const int64_t q = q0 + tx;
            double *dst = out + bo + q * a.so[1];
            if (beta != 0.0) {
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int64_t p = p0 + ty + 8 * k;
                    v[k] = p < np && q < nq ? beta * dst[p * a.so[0]] : 0.0;
                }
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int64_t p = p0 + ty + 8 * k;
                const double x = alpha * tile[tx][ty + 8 * k];
                if (p < np && q < nq) dst[p * a.so[0]] = beta != 0.0 ? x + v[k] : x;
            }
            __syncthreads();
        }
    }
}

int grid_for(int64_t total, int block) {
    int64_t g = (total + block - 1) / block;
    return (int)std::min<int64_t>(std::max<int64_t>(g, 1), 148 * 32);
}

}  // namespace

namespace {
// CCSD_GPU_TRACE=2: every permutation on stderr, tagged with the contraction that asked for it
thread_local const char *g_perm_tag = nullptr;
int trace_level() {
    static const int level = [] {
        const char *e = std::getenv("CCSD_GPU_TRACE");
        return e ? std::atoi(e) : 0;
    }();
    return level;
}
// CCSD_GPU_TRACE=3 adds the host time spent inside each contraction call: a call that blocks (an
// allocation that grows the pool, a synchronising library call) shows up as a long one
struct PermTag {
    const char *prev;
    std::chrono::steady_clock::time_point t0;
    explicit PermTag(const char *t) : prev(g_perm_tag), t0(std::chrono::steady_clock::now()) { g_perm_tag = t; }
    ~PermTag() {
        if (trace_level() >= 3)
            std::fprintf(stderr, "ccsd_gpu   [%s] host %.3f ms\n", g_perm_tag,
                         std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count());
        g_perm_tag = prev;
    }
};
}  // namespace

void permute_add(Exec &ex, double alpha, const TV &in, double beta, const TV &out) {
    REQUIRE(in.nd == out.nd, CCSD_GPU_EINVAL, "permute_add: rank mismatch");
    if (trace_level() >= 2) {
        std::string d;
        for (int k = 0; k < in.nd; k++)
            d += " " + std::to_string(in.n[k]) + ":" + std::to_string(in.s[k]) + "->" + std::to_string(out.s[k]);
        std::fprintf(stderr, "ccsd_gpu permute [%s] %.1f MB beta %g dims%s\n", g_perm_tag ? g_perm_tag : "direct",
                     8e-6 * (double)in.size(), beta, d.c_str());
    }
    // drop unit dims
    std::vector<int> dims;
    for (int d = 0; d < in.nd; d++) {
        REQUIRE(in.n[d] == out.n[d], CCSD_GPU_EINVAL, "permute_add: extent mismatch");
        if (in.n[d] > 1) dims.push_back(d);
    }
    int64_t total = in.size();
    if (total == 0) return;
    PermArgs a{};
    if (dims.empty()) dims.push_back(0);
    // order by output stride, neighbours that are one run on both sides taken as one dim (the long runs that
    // leaves fill the tiles below: 1.6 GB of six [a,j,b,k] with j of 24 moved in front of a 1.39 ms in tiles
    // of 32 x 24, 0.85 ms so)
    std::sort(dims.begin(), dims.end(), [&](int x, int y) { return out.s[x] < out.s[y]; });
    for (int d : dims) {
        const int k = a.nd;
        if (k > 0 && in.s[d] == a.si[k - 1] * a.n[k - 1] && out.s[d] == a.so[k - 1] * a.n[k - 1]) {
            a.n[k - 1] *= in.n[d];
            continue;
        }
        a.n[k] = in.n[d];
        a.si[k] = in.s[d];
        a.so[k] = out.s[d];
        a.nd++;
    }
    int p = 0;   // the input-fastest dim; the output-fastest is 0
    for (int d = 1; d < a.nd; d++)
        if (a.si[d] < a.si[p]) p = d;
    const bool small = total < (1ll << 31);
    if (p != 0 && a.n[p] >= 8 && a.n[0] >= 8) {
        // (p, 0, the others)
        const int64_t n = a.n[p], si = a.si[p], so = a.so[p];
        for (int d = p; d > 0; d--) {
            a.n[d] = a.n[d - 1];
            a.si[d] = a.si[d - 1];
            a.so[d] = a.so[d - 1];
        }
        a.n[0] = n;
        a.si[0] = si;
        a.so[0] = so;
        const int64_t nb = total / (a.n[0] * a.n[1]);
        const dim3 grid((unsigned)((a.n[0] + 31) / 32), (unsigned)std::min<int64_t>((a.n[1] + 31) / 32, 65535),
                        (unsigned)std::min<int64_t>(nb, 65535));
        auto kernel = nb < (1ll << 31) ? permute_tiled_kernel<uint32_t> : permute_tiled_kernel<int64_t>;
        kernel<<<grid, dim3(32, 8), 0, ex.stream>>>(a, nb, alpha, in.p, beta, out.p);
    } else if (a.n[0] >= 16) {
        // segments of 128 to 1024, short enough for 48 warps an SM
        const int64_t per_warp = (total / (148 * 48) + 127) / 128 * 128;
        const int seg = (int)std::min<int64_t>(1024, std::max<int64_t>(128, per_warp));
        const int nseg = (int)((a.n[0] + seg - 1) / seg);
        const int64_t nwork = total / a.n[0] * nseg;
        const int blocks = (int)std::min<int64_t>((nwork + 7) / 8, 148 * 64);
        auto kernel = nwork < (1ll << 31) ? permute_rows_kernel<uint32_t> : permute_rows_kernel<int64_t>;
        kernel<<<blocks, dim3(32, 8), 0, ex.stream>>>(a, nwork, nseg, seg, alpha, in.p, beta, out.p);
    } else {
        auto kernel = small ? permute_simple_kernel<uint32_t> : permute_simple_kernel<int64_t>;
        kernel<<<grid_for(total, 256), 256, 0, ex.stream>>>(a, total, alpha, in.p, beta, out.p);
    }
    ex.launches++;
    CU_CHECK(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// GEMM dispatch
// ---------------------------------------------------------------------------

namespace {

// Route of an m x n x k product: tensor cores (mixed, with `splits` K splits; -1 = the fixed rule's
// count) or the FP64 engines.  known = false: the product is to be timed first (autotune on, a shape
// not seen before); `key` then names it.
struct Route {
    bool known = true, mixed = false;
    int splits = -1;
    std::string key;
};

// fixed rule: the tensor-core tile is 128 x 256 x 64, so skinny products stay on the FP64 pipe
Route fixed_route(const Exec &ex, int64_t m, int64_t n, int64_t k, double fl, bool allow_mixed) {
    Route r;
    const bool tc_ok = allow_mixed && ex.prec == Prec::MIXED && k >= 16;
    r.mixed = tc_ok && fl >= ex.mixed_min_flops && (ex.mixed_min_flops <= 1 || (m >= 64 && n >= 64 && k >= 64));
    return r;
}

// products big enough to be worth timing on the tensor cores
bool worth_timing(int64_t m, int64_t n, int64_t k, double fl) { return k >= 16 && fl >= 5e7 && m >= 16 && n >= 16; }

Route lookup_route(Exec &ex, bool transA, bool transB, int64_t m, int64_t n, int64_t k, double fl, bool allow_mixed) {
    Route r;
    const bool tc_ok = allow_mixed && ex.prec == Prec::MIXED && k >= 16;
    if (tc_ok && ex.autotune) {
        // measured route (0 = DGEMM, s >= 1 = tensor cores with s K-splits)
        if (!worth_timing(m, n, k, fl)) {
            r.splits = 0;
            return r;
        }
        r.key = tune_key('g', m, n, k, transA, transB, ex);
        const int route = tune_lookup(r.key);
        if (route < 0) {
            r.known = false;
            return r;
        }
        r.mixed = route > 0;
        r.splits = route;
        return r;
    }
    return fixed_route(ex, m, n, k, fl, allow_mixed);
}

}  // namespace

bool gemm_takes_digits(const Exec &ex, int64_t m, int64_t n, int64_t k, double fl) {
    return ex.fp64_digits > 0 && fl >= ex.fp64_digits_min_flops &&
           (ex.fp64_digits_min_flops <= 1 || (m >= 256 && n >= 256 && k >= 512));
}

namespace {

// The route of a product that lookup_route does not know yet: every candidate timed on these operands
// (the fixed rule when that cannot be done now: another thread is timing, or the stream is captured).
Route measure_route(Exec &ex, const Route &unknown, bool transA, bool transB, int64_t m, int64_t n, int64_t k, double alpha,
                    const double *A, int64_t lda, const double *B, int64_t ldb, double fl, bool allow_mixed) {
    std::vector<int> routes;
    if (fl <= 4e11) routes.push_back(0);   // larger products never favour FP64
    for (int sp : tc_split_candidates(m, n, k, ex.planes)) routes.push_back(sp);
    DBuf scratch = dalloc(m * n, ex.stream);
    const int route = tune_measure(ex, unknown.key, routes, [&](int r) {
        if (r == 0) {
            const double zero = 0.0;
            BLAS_CHECK(cublasDgemm_64(ex.blas, transA ? CUBLAS_OP_T : CUBLAS_OP_N, transB ? CUBLAS_OP_T : CUBLAS_OP_N, m,
                                      n, k, &alpha, A, lda, B, ldb, &zero, scratch.d(), m));
        } else {
            mixed_gemm(ex, transA, transB, m, n, k, alpha, A, lda, B, ldb, 0.0, scratch.d(), m, r);
        }
    });
    if (route < 0) return fixed_route(ex, m, n, k, fl, allow_mixed);
    Route rt;
    rt.mixed = route > 0;
    rt.splits = route;
    return rt;
}

void run_gemm(Exec &ex, const Route &rt, bool transA, bool transB, int64_t m, int64_t n, int64_t k, double alpha,
              const double *A, int64_t lda, const double *B, int64_t ldb, double beta, double *C, int64_t ldc) {
    const double fl = 2.0 * double(m) * double(n) * double(k);
    if (trace_level() >= 2)
        std::fprintf(stderr, "ccsd_gpu gemm [%s] %s m %lld n %lld k %lld  %.3g flop  splits %d\n",
                     g_perm_tag ? g_perm_tag : "direct", rt.mixed ? "bf16x3" : "fp64", (long long)m, (long long)n,
                     (long long)k, fl, rt.splits);
    if (rt.mixed) {
        mixed_gemm(ex, transA, transB, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, rt.splits);
        return;
    }
    if (gemm_takes_digits(ex, m, n, k, fl)) {
        ozaki_gemm(ex, transA, transB, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, ex.fp64_digits);
        return;
    }
    BLAS_CHECK(cublasDgemm_64(ex.blas, transA ? CUBLAS_OP_T : CUBLAS_OP_N, transB ? CUBLAS_OP_T : CUBLAS_OP_N, m,
                              n, k, &alpha, A, lda, B, ldb, &beta, C, ldc));
}

}  // namespace

bool gemm_may_take_tensor_cores(const Exec &ex, int64_t m, int64_t n, int64_t k) {
    const double fl = 2.0 * double(m) * double(n) * double(k);
    if (ex.prec == Prec::MIXED && ex.autotune) return worth_timing(m, n, k, fl);
    return fixed_route(ex, m, n, k, fl, true).mixed;
}

void gemm(Exec &ex, bool transA, bool transB, int64_t m, int64_t n, int64_t k, double alpha, const double *A,
          int64_t lda, const double *B, int64_t ldb, double beta, double *C, int64_t ldc, bool allow_mixed) {
    if (m == 0 || n == 0) return;
    const double fl = 2.0 * double(m) * double(n) * double(k);
    ex.flops += fl;
    Route rt = lookup_route(ex, transA, transB, m, n, k, fl, allow_mixed);
    if (!rt.known) rt = measure_route(ex, rt, transA, transB, m, n, k, alpha, A, lda, B, ldb, fl, allow_mixed);
    run_gemm(ex, rt, transA, transB, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
}

void gemm_batched_f64(Exec &ex, bool transA, bool transB, int64_t m, int64_t n, int64_t k, double alpha,
                      const double *A, int64_t lda, int64_t strideA, const double *B, int64_t ldb, int64_t strideB,
                      double beta, double *C, int64_t ldc, int64_t strideC, int64_t batch) {
    if (m == 0 || n == 0 || batch == 0) return;
    ex.flops += 2.0 * double(m) * double(n) * double(k) * double(batch);
    BLAS_CHECK(cublasDgemmStridedBatched_64(ex.blas, transA ? CUBLAS_OP_T : CUBLAS_OP_N,
                                            transB ? CUBLAS_OP_T : CUBLAS_OP_N, m, n, k, &alpha, A, lda, strideA, B,
                                            ldb, strideB, &beta, C, ldc, strideC, batch));
}

// ---------------------------------------------------------------------------
// contract()
// ---------------------------------------------------------------------------

namespace {

// What a contraction keeps per label and the short lists it sorts them into live on the stack: a small
// system makes some forty contractions of a few microseconds per residual, and a map and a dozen heap
// vectors per contraction took as long as their launches.
struct LabelInfo {
    int64_t n = 1;
    int dA = -1, dB = -1, dC = -1;
    bool used = false;
};

struct LabelTable {
    LabelInfo t[128];
    LabelInfo &operator[](char c) {
        LabelInfo &l = t[(unsigned char)c & 127];
        l.used = true;
        return l;
    }
    const LabelInfo &at(char c) const { return t[(unsigned char)c & 127]; }
};

template <class T>
struct Short {   // at most 12 labels or dims (two operands of six)
    T v[12];
    int n = 0;
    void push_back(T x) { v[n++] = x; }
    T *begin() { return v; }
    T *end() { return v + n; }
    const T *begin() const { return v; }
    const T *end() const { return v + n; }
    bool empty() const { return n == 0; }
    T operator[](int i) const { return v[i]; }
};
using Labels = Short<char>;
using Dims = Short<int>;

// Is `v` (dims given by `order1` then `order2`) a column-major matrix [group1][group2]?
// Returns the leading dimension in *ld.
bool groupable(const TV &v, const Dims &g1, const Dims &g2, int64_t *ld) {
    int64_t expect = 1;
    for (int d : g1) {
        if (v.n[d] == 1) continue;
        if (v.s[d] != expect) return false;
        expect *= v.n[d];
    }
    int64_t lead = -1, exp2 = -1;
    for (int d : g2) {
        if (v.n[d] == 1) continue;
        if (lead < 0) {
            lead = v.s[d];
            if (lead < expect) return false;
            exp2 = lead * v.n[d];
        } else {
            if (v.s[d] != exp2) return false;
            exp2 *= v.n[d];
        }
    }
    *ld = lead < 0 ? std::max<int64_t>(expect, 1) : lead;
    return true;
}

Labels natural_order(const TV &v, const Labels &labels, const LabelTable &info,
                                int which) {
    Labels out = labels;
    auto stride = [&](char c) {
        const LabelInfo &l = info.at(c);
        return v.s[which == 0 ? l.dA : which == 1 ? l.dB : l.dC];
    };
    for (int i = 1; i < out.n; i++)   // insertion sort: stable, a handful of labels
        for (int j = i; j > 0 && stride(out.v[j]) < stride(out.v[j - 1]); j--) std::swap(out.v[j], out.v[j - 1]);
    return out;
}

Dims dims_of(const Labels &labels, const LabelTable &info, int which) {
    Dims d;
    for (char c : labels) {
        const LabelInfo &li = info.at(c);
        d.push_back(which == 0 ? li.dA : which == 1 ? li.dB : li.dC);
    }
    return d;
}

int64_t prod(const Labels &labels, const LabelTable &info) {
    int64_t p = 1;
    for (char c : labels) p *= info.at(c).n;
    return p;
}

// Contiguous copy of v with dims reordered as [g1 labels][g2 labels].
TV make_contiguous(Exec &ex, const TV &v, const Dims &g1, const Dims &g2, DBuf &buf) {
    buf = dalloc(v.size(), ex.stream);
    TV dst;
    dst.p = buf.d();
    dst.nd = v.nd;
    int64_t st = 1;
    for (int k = 0; k < v.nd; k++) dst.n[k] = v.n[k];
    for (int d : g1) {
        dst.s[d] = st;
        st *= v.n[d];
    }
    for (int d : g2) {
        dst.s[d] = st;
        st *= v.n[d];
    }
    permute_add(ex, 1.0, v, 0.0, dst);
    return dst;
}

// v as a GEMM operand gather: rows over the dims `rows`, K over the dims `ks` (each in the order
// given, first fastest; unit dims dropped).  False when a group spans more than four dims.
bool gather_view(const TV &v, const Dims &rows, const Dims &ks, SplitView *out) {
    SplitView g{};
    g.p = v.p;
    for (int d : rows) {
        if (v.n[d] == 1) continue;
        if (g.nr == 4) return false;
        g.rn[g.nr] = v.n[d];
        g.rs[g.nr++] = v.s[d];
    }
    for (int d : ks) {
        if (v.n[d] == 1) continue;
        if (g.nk == 4) return false;
        g.kn[g.nk] = v.n[d];
        g.ks[g.nk++] = v.s[d];
    }
    if (g.nr == 0) g.rn[g.nr++] = 1;   // a single row (stride unused)
    if (g.nk == 0) g.kn[g.nk++] = 1;
    *out = g;
    return true;
}

// C as the output of a GEMM with rows over the dims `rows` and columns over `cols` (first fastest)
bool out_view(const TV &C, const Dims &rows, const Dims &cols, OutView *out) {
    OutView v{};
    v.p = C.p;
    // neighbouring dims that are one run of memory become one (a matrix then is one by one)
    auto add = [&](int d, int &n, int *ext, long long *str) {
        if (C.n[d] == 1) return true;
        if (n > 0 && C.s[d] == str[n - 1] * ext[n - 1]) {
            ext[n - 1] *= (int)C.n[d];
            return true;
        }
        if (n == 4) return false;
        ext[n] = (int)C.n[d];
        str[n++] = C.s[d];
        return true;
    };
    for (int d : rows)
        if (!add(d, v.nr, v.rn, v.rs)) return false;
    for (int d : cols)
        if (!add(d, v.nc, v.cn, v.cs)) return false;
    if (v.nr == 0) v.rn[v.nr++] = 1;
    if (v.nc == 0) v.cn[v.nc++] = 1;
    *out = v;
    return true;
}

// A small product of strided tensors in one launch: C = alpha sum_k A B + beta C for any order of the indices.
// Such a product is bound by its launches: with cuBLAS an operand's copy, the product, the sum of its K
// slices and the output's scatter are up to five of some 3 us each.  The offsets of the K positions in A and B
// stand in shared memory; G threads sum one element, 1 for a short K (the warp then runs along the output), else
// 32 or 256 along K.  An H2O iteration in cc-pVDZ (n_o = 5, n_v = 19) 542 us without, 461 with it; at
// n_o = 9, n_v = 71 few products are this small and nothing changes.
struct SmallDims {
    int nd;
    int n[4];
    long long s0[4], s1[4];   // strides in the two tensors that have these dims
    __device__ __forceinline__ void locate(int x, long long &o0, long long &o1) const {
        o0 = o1 = 0;
#pragma unroll
        for (int d = 0; d < 4; d++) {
            if (d < nd) {
                const int q = x / n[d], i = x - q * n[d];
                x = q;
                o0 += i * s0[d];
                o1 += i * s1[d];
            }
        }
    }
};

struct SmallProduct {
    SmallDims m, n, k;   // in (A, C), (B, C) and (A, B)
    int M, N, K;
    const double *A, *B;
    double *C;
    double alpha, beta;
};

constexpr int SMALL_K = 1024;            // K positions per table
// The line: products of up to 2^18 flops alone leave the H2O iteration at 493 us instead of 456; up to 2^23
// would give it 447 but the residual at n_o = 9, n_v = 71 1054 us instead of 987, cuBLAS being faster there.
constexpr double SMALL_FLOPS = 1 << 20;

template <int G>
__global__ void __launch_bounds__(256) small_product_kernel(SmallProduct p) {
    __shared__ long long ka[SMALL_K], kb[SMALL_K];
    __shared__ double part[8];
    const int lane = threadIdx.x % G, o = blockIdx.x * (256 / G) + threadIdx.x / G;
    const bool live = o < p.M * p.N;
    long long oa = 0, ob = 0, ocm = 0, ocn = 0;
    if (live) {
        p.m.locate(o % p.M, oa, ocm);
        p.n.locate(o / p.M, ob, ocn);
    }
    const double *A = p.A + oa, *B = p.B + ob;
    double acc = 0.0;
    for (int k0 = 0; k0 < p.K; k0 += SMALL_K) {
        const int nk = min(SMALL_K, p.K - k0);
        __syncthreads();
        for (int i = threadIdx.x; i < nk; i += 256) p.k.locate(k0 + i, ka[i], kb[i]);
        __syncthreads();
        if (live) {
#pragma unroll 4
            for (int i = lane; i < nk; i += G) acc += A[ka[i]] * B[kb[i]];
        }
    }
    if (G > 1)
        for (int h = 16; h > 0; h >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, h);
    if (G > 32) {
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0)
            for (int w = 1; w < 8; w++) acc += part[w];
    }
    if (live && lane == 0) {
        double *c = p.C + ocm + ocn;
        *c = p.beta != 0.0 ? p.alpha * acc + p.beta * *c : p.alpha * acc;
    }
}

// the dims of labels v with their strides in x (dims d0) and y (dims d1), runs in both taken as one
bool small_dims(const TV &x, const Dims &d0, const TV &y, const Dims &d1, SmallDims *out) {
    SmallDims v{};
    for (int i = 0; i < d0.n; i++) {
        const int64_t n = x.n[d0[i]], s0 = x.s[d0[i]], s1 = y.s[d1[i]];
        if (n == 1) continue;
        if (v.nd > 0 && s0 == v.s0[v.nd - 1] * v.n[v.nd - 1] && s1 == v.s1[v.nd - 1] * v.n[v.nd - 1]) {
            v.n[v.nd - 1] *= (int)n;
            continue;
        }
        if (v.nd == 4) return false;
        v.n[v.nd] = (int)n;
        v.s0[v.nd] = s0;
        v.s1[v.nd++] = s1;
    }
    *out = v;
    return true;
}

void run_small(Exec &ex, const SmallProduct &p) {
    const int outs = p.M * p.N;
    if (p.K <= 64) small_product_kernel<1><<<(outs + 255) / 256, 256, 0, ex.stream>>>(p);
    else if (p.K < 1024 || outs > 1024) small_product_kernel<32><<<(outs + 7) / 8, 256, 0, ex.stream>>>(p);
    else small_product_kernel<256><<<outs, 256, 0, ex.stream>>>(p);
    ex.launches++;
    CU_CHECK(cudaGetLastError());
}

// bytes that the reordering copies of a product move (each read and written once; an output that is
// scattered also reads its old values)
double copy_bytes(const TV &A, bool packA, const TV &B, bool packB, const TV &C, bool scatter) {
    return 16.0 * ((packA ? (double)A.size() : 0.0) + (packB ? (double)B.size() : 0.0)) +
           (scatter ? 24.0 * (double)C.size() : 0.0);
}

// A contraction as a strided batch of GEMMs: one or two output labels of one operand are taken out (z the
// batch, w a loop on the host; -1: none), what is left of A, B and C are matrices as they lie.
struct BatchPlan {
    bool swap = false;            // C' is N x M: the operands change places
    bool tA = false, tB = false;
    int64_t m = 0, n = 0, k = 0, lda = 0, ldb = 0, ldc = 0;
    int64_t nz = 1, zA = 0, zB = 0, zC = 0;   // batch count and strides
    int64_t nw = 1, wA = 0, wB = 0, wC = 0;   // loop count and strides
    bool copyA = false, copyB = false;        // an operand still needs its copy (the one without z, w)
    Dims a1, a2, b1, b2;          // its dims as (first group, second group)
};

// The plan that spares the most copying of those whose launches cost less than that: a copy of 16 MB takes
// about as long as two launches.  False when none beats `base` bytes.
bool find_batch(const TV &A, const TV &B, const TV &C, const LabelTable &info, const Labels &K,
                const Labels &oM, const Labels &oN, double base, BatchPlan *best) {
    bool found = false;
    double best_gain = 0.0;
    // a product bound by its flops gains little from the copies it is spared and loses more when the batch
    // falls on a narrower DGEMM tile (2048^3 with a batch of 16: 1.02 ms, 0.55 ms with both copies)
    const double fl = 2.0 * (double)prod(oM, info) * (double)prod(oN, info) * (double)prod(K, info);
    if (fl / 35e12 > 3.0 * base / 4e12) return false;
    auto without = [](const Labels &v, char z, char w) {
        Labels o;
        for (char c : v)
            if (c != z && c != w) o.push_back(c);
        return o;
    };
    Labels outs = oM;
    for (char c : oN) outs.push_back(c);
    auto try_plan = [&](char z, char w) {
        BatchPlan p;
        const auto M = without(oM, z, w), N = without(oN, z, w);
        const LabelInfo &iz = info.at(z);
        p.nz = iz.n;
        p.zA = iz.dA >= 0 ? A.s[iz.dA] : 0;
        p.zB = iz.dB >= 0 ? B.s[iz.dB] : 0;
        p.zC = C.s[iz.dC];
        if (w) {
            const LabelInfo &iw = info.at(w);
            p.nw = iw.n;
            p.wA = iw.dA >= 0 ? A.s[iw.dA] : 0;
            p.wB = iw.dB >= 0 ? B.s[iw.dB] : 0;
            p.wC = C.s[iw.dC];
            if (p.wA == p.zA * p.nz && p.wB == p.zB * p.nz && p.wC == p.zC * p.nz) {   // one longer batch
                p.nz *= p.nw;
                p.nw = 1;
                p.wA = p.wB = p.wC = 0;
            }
        }
        const auto cM = dims_of(M, info, 2), cN = dims_of(N, info, 2);
        if (groupable(C, cM, cN, &p.ldc)) p.swap = false;
        else if (groupable(C, cN, cM, &p.ldc)) p.swap = true;
        else return;
        p.m = prod(M, info);
        p.n = prod(N, info);
        p.k = prod(K, info);
        // the output tiles of what is left must stay full (cuBLAS runs a batch of thin products, or one of
        // gemv shape, several times slower than one product over copies)
        if ((p.m < 64 && p.m < prod(oM, info)) || (p.n < 64 && p.n < prod(oN, info)) || p.m == 1 || p.n == 1) return;
        // a strided batch runs without K splits: a long K needs enough 64 x 64 output tiles for the SMs
        if (p.k > 4096 && ((p.m + 63) / 64) * ((p.n + 63) / 64) * p.nz < 148) return;
        const bool freeA = p.zA == 0 && p.wA == 0, freeB = p.zB == 0 && p.wB == 0;
        for (int which = 0; which < 2; which++) {   // the K order of A, then of B
            BatchPlan q = p;
            const auto oK = natural_order(which == 0 ? A : B, K, info, which);
            const auto aK = dims_of(oK, info, 0), aM = dims_of(M, info, 0), bK = dims_of(oK, info, 1), bN = dims_of(N, info, 1);
            if (groupable(A, aM, aK, &q.lda)) q.tA = false;
            else if (groupable(A, aK, aM, &q.lda)) q.tA = true;
            else if (freeA) {
                q.copyA = q.tA = true;
                q.lda = q.k;
                q.a1 = aK;
                q.a2 = aM;
            } else continue;
            if (groupable(B, bK, bN, &q.ldb)) q.tB = false;
            else if (groupable(B, bN, bK, &q.ldb)) q.tB = true;
            else if (freeB) {
                q.copyB = true;
                q.tB = false;
                q.ldb = q.k;
                q.b1 = bK;
                q.b2 = bN;
            } else continue;
            const double gain = base - copy_bytes(A, q.copyA, B, q.copyB, C, false);
            // of equal plans the one with the larger products
            if (gain < best_gain || (gain == best_gain && found && q.m * q.n <= best->m * best->n)) continue;
            if (gain <= 0.0 || (double)(q.nw - 1) * 16e6 > gain) continue;
            best_gain = gain;
            *best = q;
            found = true;
        }
    };
    for (char z : outs) {
        const LabelInfo &iz = info.at(z);
        if (iz.n < 2) continue;
        try_plan(z, 0);
        for (char w : outs) {
            const LabelInfo &iw = info.at(w);
            if (w == z || iw.n < 2 || (iw.dA >= 0) != (iz.dA >= 0)) continue;
            try_plan(z, w);
        }
    }
    return found;
}

void run_batch(Exec &ex, const BatchPlan &p, const TV &A, const TV &B, const TV &C, double alpha, double beta) {
    DBuf bufA, bufB;
    const TV Au = p.copyA ? make_contiguous(ex, A, p.a1, p.a2, bufA) : A;
    const TV Bu = p.copyB ? make_contiguous(ex, B, p.b1, p.b2, bufB) : B;
    if (trace_level() >= 2)
        std::fprintf(stderr, "ccsd_gpu gemm [%s] fp64 batch %lld x %lld m %lld n %lld k %lld%s%s%s\n",
                     g_perm_tag ? g_perm_tag : "direct", (long long)p.nw, (long long)p.nz, (long long)p.m, (long long)p.n,
                     (long long)p.k, p.swap ? " swap" : "", p.copyA ? " copyA" : "", p.copyB ? " copyB" : "");
    for (int64_t w = 0; w < p.nw; w++) {
        const double *a = Au.p + w * p.wA, *b = Bu.p + w * p.wB;
        double *c = C.p + w * p.wC;
        if (p.swap)
            gemm_batched_f64(ex, !p.tB, !p.tA, p.n, p.m, p.k, alpha, b, p.ldb, p.zB, a, p.lda, p.zA, beta, c, p.ldc, p.zC,
                             p.nz);
        else
            gemm_batched_f64(ex, p.tA, p.tB, p.m, p.n, p.k, alpha, a, p.lda, p.zA, b, p.ldb, p.zB, beta, c, p.ldc, p.zC,
                             p.nz);
    }
}

}  // namespace

void contract(Exec &ex, const char *spec, double alpha, const TV &A, const TV &B, double beta, const TV &C) {
    PermTag tag(spec);
    const char *comma = std::strchr(spec, ','), *arrow = std::strstr(spec, "->");
    REQUIRE(comma && arrow && comma < arrow, CCSD_GPU_EINVAL, "contract: bad spec");
    const char *la = spec, *lb = comma + 1, *lc = arrow + 2;
    REQUIRE(comma - la == A.nd && arrow - lb == B.nd && (int)std::strlen(lc) == C.nd, CCSD_GPU_EINVAL,
            std::string("contract: rank mismatch in ") + spec);
    LabelTable info;
    for (int d = 0; d < A.nd; d++) {
        info[la[d]].dA = d;
        info[la[d]].n = A.n[d];
    }
    for (int d = 0; d < B.nd; d++) {
        auto &li = info[lb[d]];
        if (li.dA >= 0 && li.n != B.n[d]) throw Error(CCSD_GPU_EINVAL, std::string("contract: extent mismatch in ") + spec);
        li.dB = d;
        li.n = B.n[d];
    }
    for (int d = 0; d < C.nd; d++) {
        auto &li = info[lc[d]];
        REQUIRE(li.dA >= 0 || li.dB >= 0, CCSD_GPU_EINVAL, std::string("contract: free output label in ") + spec);
        REQUIRE(li.n == C.n[d], CCSD_GPU_EINVAL, std::string("contract: output extent mismatch in ") + spec);
        li.dC = d;
    }
    Labels K, M, N;
    for (int c = 0; c < 128; c++) {
        const LabelInfo &li = info.t[c];
        if (!li.used) continue;
        int cnt = (li.dA >= 0) + (li.dB >= 0) + (li.dC >= 0);
        REQUIRE(cnt == 2, CCSD_GPU_EINVAL, std::string("contract: label must appear exactly twice in ") + spec);
        if (li.dA >= 0 && li.dB >= 0) K.push_back((char)c);
        else if (li.dA >= 0) M.push_back((char)c);
        else N.push_back((char)c);
    }
    const int64_t mK = prod(K, info), mM = prod(M, info), mN = prod(N, info);
    if (mM == 0 || mN == 0) return;

    // label orders: M/N from C where possible, K from A
    Labels oM = natural_order(C, M, info, 2), oN = natural_order(C, N, info, 2);
    Labels oK = natural_order(A, K, info, 0);
    {
        Labels bK = natural_order(B, K, info, 1);
        int64_t ld;
        // prefer B's K order when B is the bigger operand and already groupable with it
        if (B.size() > A.size() && (groupable(B, dims_of(bK, info, 1), dims_of(oN, info, 1), &ld) ||
                                    groupable(B, dims_of(oN, info, 1), dims_of(bK, info, 1), &ld)))
            oK = bK;
    }
    DBuf bufA, bufB, bufC;
    TV Au = A, Bu = B;
    bool tA, tB;
    int64_t lda, ldb, ldc;
    // an operand whose indices are not two contiguous groups is reordered into a copy, unless the
    // product goes to the tensor cores, whose operand split gathers it from its own layout
    bool packA = false, packB = false;
    const auto aK = dims_of(oK, info, 0), aM = dims_of(oM, info, 0);
    const auto bK = dims_of(oK, info, 1), bN = dims_of(oN, info, 1);
    if (groupable(A, aM, aK, &lda)) tA = false;
    else if (groupable(A, aK, aM, &lda)) tA = true;
    else {
        packA = true;
        tA = true;
        lda = std::max<int64_t>(mK, 1);
    }
    if (groupable(B, bK, bN, &ldb)) tB = false;
    else if (groupable(B, bN, bK, &ldb)) tB = true;
    else {
        packB = true;
        tB = false;
        ldb = std::max<int64_t>(mK, 1);
    }
    auto cM = dims_of(oM, info, 2), cN = dims_of(oN, info, 2);
    const int cmode = groupable(C, cM, cN, &ldc) ? 0 : groupable(C, cN, cM, &ldc) ? 1 : 2;
    // C = beta C + the column-major mM x mN product in bufC
    auto scatter_C = [&]() {
        TV t;
        t.p = bufC.d();
        t.nd = C.nd;
        int64_t st = 1;
        for (int k = 0; k < C.nd; k++) t.n[k] = C.n[k];
        for (int d : cM) {
            t.s[d] = st;
            st *= C.n[d];
        }
        for (int d : cN) {
            t.s[d] = st;
            st *= C.n[d];
        }
        permute_add(ex, 1.0, t, beta, C);
    };
    const double fl = 2.0 * double(mM) * double(mN) * double(mK);
    // the operands change places when C lies the other way round; a scattered C takes the group that holds
    // its unit stride as the rows, so that the epilogue writes along it
    const bool swap = cmode == 1 || (cmode == 2 && !cM.empty() && !cN.empty() && C.s[cN[0]] < C.s[cM[0]]);
    Route rt = swap ? lookup_route(ex, !tB, !tA, mN, mM, mK, fl, true)
                    : lookup_route(ex, tA, tB, mM, mN, mK, fl, true);
    // a product whose operands or output are not matrices as they lie: the tensor-core GEMM gathers and
    // scatters them itself; for cuBLAS a strided batch of GEMMs over an output index (the trial index, or
    // one that sits between the others) may spare the copies
    const bool strided = packA || packB || cmode == 2;
    auto copies = [&]() {
        if (packA && Au.p == A.p) Au = make_contiguous(ex, A, aK, aM, bufA);
        if (packB && Bu.p == B.p) Bu = make_contiguous(ex, B, bK, bN, bufB);
    };
    if (!rt.known) {
        // timed on the operands as matrices, then dispatched like every later product of this shape
        copies();
        rt = swap ? measure_route(ex, rt, !tB, !tA, mN, mM, mK, alpha, Bu.p, ldb, Au.p, lda, fl, true)
                        : measure_route(ex, rt, tA, tB, mM, mN, mK, alpha, Au.p, lda, Bu.p, ldb, fl, true);
    }
    // a small product that cuBLAS needs several launches for: copies, or K slices and their sum (rows: the group
    // of C's unit stride)
    SmallProduct sp{};
    if ((strided || (mK >= 512 && mM * mN <= 1024)) && !rt.mixed && fl <= SMALL_FLOPS && mK > 0 && !gemm_takes_digits(ex, mM, mN, mK, fl)) {
        const bool flip = !cM.empty() && !cN.empty() && C.s[cN[0]] < C.s[cM[0]];
        if (flip ? small_dims(B, bN, C, cN, &sp.m) && small_dims(A, aM, C, cM, &sp.n) && small_dims(B, bK, A, aK, &sp.k)
                 : small_dims(A, aM, C, cM, &sp.m) && small_dims(B, bN, C, cN, &sp.n) && small_dims(A, aK, B, bK, &sp.k)) {
            sp.M = (int)(flip ? mN : mM);
            sp.N = (int)(flip ? mM : mN);
            sp.K = (int)mK;
            sp.A = flip ? B.p : A.p;
            sp.B = flip ? A.p : B.p;
            sp.C = C.p;
            sp.alpha = alpha;
            sp.beta = beta;
            ex.flops += fl;
            if (trace_level() >= 2)
                std::fprintf(stderr, "ccsd_gpu gemm [%s] fp64 small m %lld n %lld k %lld\n", spec, (long long)mM,
                             (long long)mN, (long long)mK);
            run_small(ex, sp);
            return;
        }
    }
    SplitView va, vb;
    OutView vc;
    if (strided && rt.mixed && gather_view(A, aM, aK, &va) && gather_view(B, bN, bK, &vb) &&
        out_view(C, swap ? cN : cM, swap ? cM : cN, &vc)) {
        ex.flops += fl;
        if (trace_level() >= 2)
            std::fprintf(stderr, "ccsd_gpu gemm [%s] bf16x3 strided m %lld n %lld k %lld  %.3g flop  splits %d\n", spec,
                         (long long)mM, (long long)mN, (long long)mK, fl, rt.splits);
        if (swap) mixed_gemm_views(ex, vb, va, mN, mM, mK, alpha, beta, vc, rt.splits);
        else mixed_gemm_views(ex, va, vb, mM, mN, mK, alpha, beta, vc, rt.splits);
        return;
    }
    BatchPlan bp;
    if (strided && !rt.mixed && !gemm_takes_digits(ex, mM, mN, mK, fl) &&
        find_batch(A, B, C, info, K, oM, oN, copy_bytes(A, packA, B, packB, C, cmode == 2), &bp)) {
        run_batch(ex, bp, A, B, C, alpha, beta);
        return;
    }
    copies();
    ex.flops += fl;
    if (cmode == 0) {
        run_gemm(ex, rt, tA, tB, mM, mN, mK, alpha, Au.p, lda, Bu.p, ldb, beta, C.p, ldc);
    } else if (cmode == 1) {
        run_gemm(ex, rt, !tB, !tA, mN, mM, mK, alpha, Bu.p, ldb, Au.p, lda, beta, C.p, ldc);
    } else {
        bufC = dalloc(mM * mN, ex.stream);
        run_gemm(ex, rt, tA, tB, mM, mN, mK, alpha, Au.p, lda, Bu.p, ldb, 0.0, bufC.d(), mM);
        scatter_C();
    }
}

// ---------------------------------------------------------------------------
// reductions
// ---------------------------------------------------------------------------

namespace {
constexpr int RBLOCKS = 592;   // 4 x 148 SMs
constexpr int RTHREADS = 256;

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

__device__ double block_sum(double v) {
    __shared__ double sh[32];
    v = warp_sum(v);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (w == 0) {
        r = lane < (blockDim.x + 31) / 32 ? sh[lane] : 0.0;
        r = warp_sum(r);
    }
    __syncthreads();
    return r;
}

struct PtrList {
    const double *p[16];
};

__global__ void multi_dot_partial(const double *__restrict__ x, PtrList ys, int nys, int64_t n,
                                  double *__restrict__ partial) {
    for (int k = 0; k < nys; k++) {
        const double *y = ys.p[k];
        double acc = 0.0;
        for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
            acc += x[i] * y[i];
        acc = block_sum(acc);
        if (threadIdx.x == 0) partial[k * gridDim.x + blockIdx.x] = acc;
    }
}

__global__ void finish_partial(const double *__restrict__ partial, int nblocks, int nys, double *__restrict__ out) {
    int k = blockIdx.x;
    double acc = 0.0;
    for (int i = threadIdx.x; i < nblocks; i += blockDim.x) acc += partial[k * nblocks + i];
    acc = block_sum(acc);
    if (threadIdx.x == 0) out[k] = acc;
}

__global__ void fill_kernel(double *p, int64_t n, double v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = v;
}

__global__ void axpby_kernel(int64_t n, double a, const double *__restrict__ x, double b, double *__restrict__ y) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = a * x[i] + (b == 0.0 ? 0.0 : b * y[i]);
}
}  // namespace

void multi_dot(Exec &ex, const double *x, const double *const *ys, int nys, int64_t n, double *d_results) {
    if (nys == 0) return;
    REQUIRE(nys <= 16, CCSD_GPU_EINVAL, "multi_dot: at most 16 vectors");
    PtrList pl{};
    for (int k = 0; k < nys; k++) pl.p[k] = ys[k];
    DBuf part = dalloc((int64_t)RBLOCKS * nys, ex.stream);
    multi_dot_partial<<<RBLOCKS, RTHREADS, 0, ex.stream>>>(x, pl, nys, n, part.d());
    finish_partial<<<nys, RTHREADS, 0, ex.stream>>>(part.d(), RBLOCKS, nys, d_results);
    ex.launches += 2;
    CU_CHECK(cudaGetLastError());
}

void dot(Exec &ex, const double *x, const double *y, int64_t n, double *d_result) {
    const double *ys[1] = {y};
    multi_dot(ex, x, ys, 1, n, d_result);
}

void fill(Exec &ex, double *p, int64_t n, double value) {
    if (n == 0) return;
    fill_kernel<<<grid_for(n, 256), 256, 0, ex.stream>>>(p, n, value);
    ex.launches++;
    CU_CHECK(cudaGetLastError());
}

void axpby(Exec &ex, int64_t n, double alpha, const double *x, double beta, double *y) {
    if (n == 0) return;
    axpby_kernel<<<grid_for(n, 256), 256, 0, ex.stream>>>(n, alpha, x, beta, y);
    ex.launches++;
    CU_CHECK(cudaGetLastError());
}

}  // namespace ccsd
