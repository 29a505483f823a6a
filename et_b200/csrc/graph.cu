// Recorded tensor computation with forward- and reverse-mode derivative passes.
#include <algorithm>

#include "amp_forms.cuh"
#include "graph.cuh"
#include "tensor_ops.cuh"

namespace ccsd {

namespace {

constexpr char BATCH = '#';   // label of the trailing trial index of tangents / adjoints

#define GRID_STRIDE(i, total) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (total); i += (int64_t)gridDim.x * blockDim.x)

inline int grid_for(int64_t total, int block) {
    int64_t g = (total + block - 1) / block;
    return (int)std::max<int64_t>(1, std::min<int64_t>(g, 148 * 64));
}

// out[J, n] += sum_k a[J, k, k, n]  /  adjoint: a[J, k, k, n] += out[J, n]
__global__ void trace_batch_kernel(const double *__restrict__ a, double *__restrict__ out, int64_t nJ, int64_t no,
                                   int64_t nbatch, int adjoint) {
    GRID_STRIDE(idx, nJ * nbatch) {
        int64_t J = idx % nJ, n = idx / nJ;
        if (!adjoint) {
            double s = 0.0;
            for (int64_t k = 0; k < no; k++) s += a[n * nJ * no * no + J + nJ * (k + no * k)];
            out[idx] += s;
        } else {
            double v = a[idx];   // here a is the adjoint of out (nJ x nbatch)
            for (int64_t k = 0; k < no; k++) out[n * nJ * no * no + J + nJ * (k + no * k)] += v;
        }
    }
}

std::string with_batch(const std::string &labels) { return labels + BATCH; }

// An op recorded as FP64 (the first-order terms of the mixed residual) runs in FP64 arithmetic; in a
// mixed-precision evaluation its large products go to the int8 digit GEMM (ex.mixed_fp64_digits
// digits, FP64-accurate) rather than DGEMM, unless the caller already chose the FP64 arithmetic.
struct Fp64Scope {
    Exec &ex;
    Prec prec;
    int digits;
    Fp64Scope(Exec &e, bool on) : ex(e), prec(e.prec), digits(e.fp64_digits) {
        if (!on) return;
        if (prec == Prec::MIXED && ex.fp64_digits == 0) ex.fp64_digits = ex.mixed_fp64_digits;
        ex.prec = Prec::FP64;
    }
    ~Fp64Scope() {
        ex.prec = prec;
        ex.fp64_digits = digits;
    }
    Fp64Scope(const Fp64Scope &) = delete;
    Fp64Scope &operator=(const Fp64Scope &) = delete;
};

}  // namespace

int Graph::input(const std::string &name, std::vector<int64_t> dims, const double *p) {
    GNode n;
    n.name = name;
    n.dims = std::move(dims);
    for (int64_t d : n.dims) n.size *= d;
    n.v = const_cast<double *>(p);
    nodes_.push_back(std::move(n));
    return (int)nodes_.size() - 1;
}

int Graph::zeros(const std::string &name, std::vector<int64_t> dims) {
    GNode n;
    n.name = name;
    n.dims = std::move(dims);
    for (int64_t d : n.dims) n.size *= d;
    n.own = dalloc(n.size, ex_.stream);
    n.v = n.own.d();
    n.zero = true;
    nodes_.push_back(std::move(n));
    return (int)nodes_.size() - 1;
}

void Graph::materialize(int i) {
    GNode &n = nodes_[i];
    if (!n.zero) return;
    fill(ex_, n.v, n.size, 0.0);
    n.zero = false;
}

int Graph::alias(int node) { return node; }

TV Graph::view(int i) const {
    const GNode &n = nodes_[i];
    TV v;
    v.p = n.v;
    v.nd = (int)n.dims.size();
    int64_t st = 1;
    for (int k = 0; k < v.nd; k++) {
        v.n[k] = n.dims[k];
        v.s[k] = st;
        st *= n.dims[k];
    }
    return v;
}

double *Graph::derivative(int i, int nvec, bool adj) {
    GNode &n = nodes_[i];
    DBuf &buf = adj ? n.adj : n.tan;
    if (!buf) {
        buf = dalloc(n.size * nvec, ex_.stream);
        (adj ? n.adj_zero : n.tan_zero) = true;
    }
    return buf.d();
}

double *Graph::tangent(int i, int nvec) {
    double *p = derivative(i, nvec, false);
    if (nodes_[i].tan_zero) fill(ex_, p, nodes_[i].size * nvec, 0.0);
    nodes_[i].tan_zero = false;
    return p;
}

double *Graph::adjoint(int i, int nvec) {
    double *p = derivative(i, nvec, true);
    if (nodes_[i].adj_zero) fill(ex_, p, nodes_[i].size * nvec, 0.0);
    nodes_[i].adj_zero = false;
    return p;
}

TV Graph::tview(int i, int nvec, bool adj) {
    TV v = view(i);
    v.p = adj ? adjoint(i, nvec) : tangent(i, nvec);
    v.n[v.nd] = nvec;
    v.s[v.nd] = nodes_[i].size;
    v.nd++;
    return v;
}

TV Graph::twrite(int i, int nvec, bool adj, double *beta) {
    derivative(i, nvec, adj);
    bool &zero = adj ? nodes_[i].adj_zero : nodes_[i].tan_zero;
    *beta = zero ? 0.0 : 1.0;
    zero = false;
    return tview(i, nvec, adj);
}

void Graph::run_forward(const GOp &op) {
    Fp64Scope fp64(ex_, op.fp64);
    // inputs never written read as zero; an output never written is overwritten (beta = 0) by the
    // ops that write every element of it, and zero-filled first for the others
    if (op.a >= 0) materialize(op.a);
    if (op.b >= 0) materialize(op.b);
    if (op.kind == OpKind::Custom)
        for (int i : custom_ins_[op.custom]) materialize(i);
    const auto first_write = [&](int i) {
        const bool zero = nodes_[i].zero;
        nodes_[i].zero = false;
        return zero;
    };
    const bool overwrites = op.kind != OpKind::Trace && op.kind != OpKind::Custom;
    if (!overwrites) materialize(op.out);
    const bool fresh = first_write(op.out);
    const double beta = fresh ? 0.0 : 1.0;
    switch (op.kind) {
    case OpKind::Contract:
        ccsd::contract(ex_, op.spec.c_str(), op.alpha, view(op.a), view(op.b), beta, view(op.out));
        break;
    case OpKind::Permute: {
        std::string s = op.spec;
        size_t ar = s.find("->");
        std::string lin = s.substr(0, ar), lout = s.substr(ar + 2);
        TV in = view(op.a), out = view(op.out), pin;
        pin.p = in.p;
        pin.nd = out.nd;
        for (int k = 0; k < out.nd; k++) {
            size_t pos = lin.find(lout[k]);
            REQUIRE(pos != std::string::npos, CCSD_GPU_EINVAL, "permute: bad spec " + s);
            pin.n[k] = in.n[pos];
            pin.s[k] = in.s[pos];
        }
        permute_add(ex_, op.alpha, pin, beta, out);
        break;
    }
    case OpKind::SquareForms: {
        const bool fresh_u = first_write(op.out2);
        ccsd::square_forms(ex_, nodes_[op.a].v, no, nv, 1, op.c1, op.c2, nodes_[op.out].v, nodes_[op.out2].v, !fresh,
                           !fresh_u);
        break;
    }
    case OpKind::SymPack:
        ccsd::sym_pack(ex_, nodes_[op.a].v, nodes_[op.b].v, no, nv, 1, op.c1, op.c2, nodes_[op.out].v, !fresh);
        break;
    case OpKind::Trace: {
        const GNode &a = nodes_[op.a];
        trace_batch_kernel<<<grid_for(a.dims[0], 128), 128, 0, ex_.stream>>>(a.v, nodes_[op.out].v, a.dims[0],
                                                                              a.dims[1], 1, 0);
        ex_.launches++;
        break;
    }
    case OpKind::Custom:
        customs_[op.custom].forward();
        break;
    }
    CU_CHECK(cudaGetLastError());
}

void Graph::contract(int out, const char *spec, double alpha, int a, int b, bool fp64) {
    GOp op;
    op.kind = OpKind::Contract;
    op.out = out;
    op.a = a;
    op.b = b;
    op.alpha = alpha;
    op.spec = spec;
    op.fp64 = fp64;
    record(std::move(op));
}

void Graph::contract_sym(int out, const char *spec, double alpha, int a, bool fp64) {
    GOp op;
    op.kind = OpKind::Contract;
    op.out = out;
    op.a = op.b = a;
    op.alpha = alpha;
    op.spec = spec;
    op.fp64 = fp64;
    op.sym = true;
    record(std::move(op));
}

void Graph::contract_given(int out, const char *spec, double alpha, int a, int b,
                           const std::function<void()> &forward) {
    GOp op;
    op.kind = OpKind::Contract;
    op.out = out;
    op.a = a;
    op.b = b;
    op.alpha = alpha;
    op.spec = spec;
    materialize(out);
    forward();
    nodes_[a].last_use = nodes_[b].last_use = (int)ops_.size();
    ops_.push_back(std::move(op));
}

void Graph::record(GOp op) {
    run_forward(op);
    for (int i : {op.a, op.b})
        if (i >= 0) nodes_[i].last_use = (int)ops_.size();
    ops_.push_back(std::move(op));
}

void Graph::permute(int out, const char *spec, double alpha, int a) {
    GOp op;
    op.kind = OpKind::Permute;
    op.out = out;
    op.a = a;
    op.alpha = alpha;
    op.spec = spec;
    record(std::move(op));
}

void Graph::square_forms(int t, int u, int a, double c1, double c2) {
    GOp op;
    op.kind = OpKind::SquareForms;
    op.out = t;
    op.out2 = u;
    op.a = a;
    op.c1 = c1;
    op.c2 = c2;
    record(std::move(op));
}

void Graph::sym_pack(int out, int a, int x, double c1, double c2) {
    GOp op;
    op.kind = OpKind::SymPack;
    op.out = out;
    op.a = a;
    op.b = x;
    op.c1 = c1;
    op.c2 = c2;
    record(std::move(op));
}

void Graph::trace(int out, int a) {
    GOp op;
    op.kind = OpKind::Trace;
    op.out = out;
    op.a = a;
    record(std::move(op));
}

int Graph::custom(CustomOp c, int out, std::vector<int> ins) {
    customs_.push_back(std::move(c));
    custom_ins_.push_back(ins);
    GOp op;
    op.kind = OpKind::Custom;
    op.out = out;
    op.custom = (int)customs_.size() - 1;
    run_forward(op);
    for (int i : ins) nodes_[i].last_use = (int)ops_.size();
    ops_.push_back(op);
    return op.custom;
}

void Graph::mark_active(const std::vector<int> &inputs) {
    for (auto &n : nodes_) n.active = false;
    for (int i : inputs) nodes_[i].active = true;
    for (const GOp &op : ops_) {
        bool act = false;
        if (op.kind == OpKind::Custom) {
            for (int i : custom_ins_[op.custom]) act = act || nodes_[i].active;
        } else {
            act = nodes_[op.a].active || (op.b >= 0 && nodes_[op.b].active);
        }
        if (act) nodes_[op.out].active = true;
        if (act && op.out2 >= 0) nodes_[op.out2].active = true;
    }
}

void Graph::clear_derivatives() {
    for (auto &n : nodes_) {
        n.tan.release();
        n.adj.release();
        n.tan_zero = n.adj_zero = false;
    }
}

void Graph::copy_columns(double *dst, int64_t ldd, const double *src, int64_t lds, int64_t size, int nvec) {
    if (size == 0) return;
    const size_t eb = sizeof(double);
    if (nvec == 1 || (ldd == size && lds == size))
        CU_CHECK(cudaMemcpyAsync(dst, src, eb * size * nvec, cudaMemcpyDeviceToDevice, ex_.stream));
    else if (eb * (size_t)std::max(ldd, lds) < ((size_t)1 << 31))   // the pitch of a 2-D copy is limited
        CU_CHECK(cudaMemcpy2DAsync(dst, eb * ldd, src, eb * lds, eb * size, nvec, cudaMemcpyDeviceToDevice, ex_.stream));
    else
        for (int k = 0; k < nvec; k++) copy_columns(dst + k * ldd, ldd, src + k * lds, lds, size, 1);
}

void Graph::store_result(int i, int nvec, bool adj, const Out &out) {
    const GNode &n = nodes_[i];
    const DBuf &buf = adj ? n.adj : n.tan;
    if (n.active && buf && !(adj ? n.adj_zero : n.tan_zero))
        copy_columns(out.p, out.ld, buf.d(), n.size, n.size, nvec);
    else
        for (int k = 0; k < nvec; k++) fill(ex_, out.p + k * out.ld, n.size, 0.0);
}

void Graph::jvp(const std::vector<int> &inputs, const std::vector<In> &seeds, int nvec, const std::vector<int> &outputs,
                const std::vector<Out> &results, const std::function<void()> &seeded) {
    clear_derivatives();
    mark_active(inputs);
    for (size_t k = 0; k < inputs.size(); k++) {
        double *t = derivative(inputs[k], nvec, false);
        nodes_[inputs[k]].tan_zero = false;
        copy_columns(t, nodes_[inputs[k]].size, seeds[k].p, seeds[k].ld, nodes_[inputs[k]].size, nvec);
    }
    seeded();
    // the tangents that the outputs depend on: an op feeding only others is skipped
    std::vector<char> needed(nodes_.size(), 0);
    for (int i : outputs) needed[i] = 1;
    for (int oi = (int)ops_.size() - 1; oi >= 0; --oi) {
        const GOp &op = ops_[oi];
        if (!needed[op.out] && !(op.out2 >= 0 && needed[op.out2])) continue;
        if (op.kind == OpKind::Custom) {
            for (int i : customs_[op.custom].tangent_reads) needed[i] = 1;
        } else {
            for (int i : {op.a, op.b})
                if (i >= 0) needed[i] = 1;
        }
    }
    double beta = 1.0;
    for (const GOp &op : ops_) {
        if (!nodes_[op.out].active || !(needed[op.out] || (op.out2 >= 0 && needed[op.out2]))) continue;
        Fp64Scope fp64(ex_, op.fp64);
        switch (op.kind) {
        case OpKind::Contract: {
            std::string s = op.spec;
            size_t comma = s.find(','), ar = s.find("->");
            std::string la = s.substr(0, comma), lb = s.substr(comma + 1, ar - comma - 1), lc = s.substr(ar + 2);
            if (nodes_[op.a].active && !op.sym) {
                std::string sp = with_batch(la) + "," + lb + "->" + with_batch(lc);
                const TV in = tview(op.a, nvec, false), out = twrite(op.out, nvec, false, &beta);
                ccsd::contract(ex_, sp.c_str(), op.alpha, in, view(op.b), beta, out);
            }
            if (nodes_[op.b].active) {
                std::string sp = la + "," + with_batch(lb) + "->" + with_batch(lc);
                const TV in = tview(op.b, nvec, false), out = twrite(op.out, nvec, false, &beta);
                ccsd::contract(ex_, sp.c_str(), op.sym ? 2.0 * op.alpha : op.alpha, view(op.a), in, beta, out);
            }
            break;
        }
        case OpKind::Permute: {
            if (!nodes_[op.a].active) break;
            size_t ar = op.spec.find("->");
            std::string lin = op.spec.substr(0, ar) + BATCH, lout = op.spec.substr(ar + 2) + BATCH;
            TV in = tview(op.a, nvec, false), out = twrite(op.out, nvec, false, &beta), pin;
            pin.p = in.p;
            pin.nd = out.nd;
            for (int k = 0; k < out.nd; k++) {
                size_t pos = lin.find(lout[k]);
                pin.n[k] = in.n[pos];
                pin.s[k] = in.s[pos];
            }
            permute_add(ex_, op.alpha, pin, beta, out);
            break;
        }
        case OpKind::SquareForms: {
            double beta_u = 1.0;
            const TV t = twrite(op.out, nvec, false, &beta), u = twrite(op.out2, nvec, false, &beta_u);
            ccsd::square_forms(ex_, tangent(op.a, nvec), no, nv, nvec, op.c1, op.c2, t.p, u.p, beta != 0.0, beta_u != 0.0);
            break;
        }
        case OpKind::SymPack: {
            const double *fa = nodes_[op.a].active ? tangent(op.a, nvec) : nullptr;
            const double *xa = nodes_[op.b].active ? tangent(op.b, nvec) : nullptr;
            const TV out = twrite(op.out, nvec, false, &beta);
            ccsd::sym_pack(ex_, fa, xa, no, nv, nvec, op.c1, op.c2, out.p, beta != 0.0);
            break;
        }
        case OpKind::Trace: {
            if (!nodes_[op.a].active) break;
            const GNode &a = nodes_[op.a];
            trace_batch_kernel<<<grid_for(a.dims[0] * nvec, 128), 128, 0, ex_.stream>>>(
                tangent(op.a, nvec), tangent(op.out, nvec), a.dims[0], a.dims[1], nvec, 0);
            ex_.launches++;
            break;
        }
        case OpKind::Custom:
            customs_[op.custom].tangent(nvec);
            break;
        }
        CU_CHECK(cudaGetLastError());
    }
    for (size_t k = 0; k < outputs.size(); k++) store_result(outputs[k], nvec, false, results[k]);
}

void Graph::vjp(const std::vector<int> &outputs, const std::vector<In> &seeds, int nvec, const std::vector<int> &inputs,
                const std::vector<Out> &results) {
    clear_derivatives();
    mark_active(inputs);
    for (size_t k = 0; k < outputs.size(); k++) {
        double beta;
        const TV a = twrite(outputs[k], nvec, true, &beta);
        copy_columns(a.p, nodes_[outputs[k]].size, seeds[k].p, seeds[k].ld, nodes_[outputs[k]].size, nvec);
    }
    double beta = 1.0;
    for (int oi = (int)ops_.size() - 1; oi >= 0; --oi) {
        const GOp &op = ops_[oi];
        if (!nodes_[op.out].active) continue;
        if (!has_adjoint(op.out) && !(op.out2 >= 0 && has_adjoint(op.out2))) continue;
        Fp64Scope fp64(ex_, op.fp64);
        switch (op.kind) {
        case OpKind::Contract: {
            std::string s = op.spec;
            size_t comma = s.find(','), ar = s.find("->");
            std::string la = s.substr(0, comma), lb = s.substr(comma + 1, ar - comma - 1), lc = s.substr(ar + 2);
            const TV cbar = tview(op.out, nvec, true);
            if (nodes_[op.a].active && !op.sym) {
                std::string sp = with_batch(lc) + "," + lb + "->" + with_batch(la);
                const TV out = twrite(op.a, nvec, true, &beta);
                ccsd::contract(ex_, sp.c_str(), op.alpha, cbar, view(op.b), beta, out);
            }
            if (nodes_[op.b].active) {
                std::string sp = la + "," + with_batch(lc) + "->" + with_batch(lb);
                const TV out = twrite(op.b, nvec, true, &beta);
                ccsd::contract(ex_, sp.c_str(), op.sym ? 2.0 * op.alpha : op.alpha, view(op.a), cbar, beta, out);
            }
            break;
        }
        case OpKind::Permute: {
            if (!nodes_[op.a].active) break;
            // a_bar[lin] += alpha * out_bar[lout]
            size_t ar = op.spec.find("->");
            std::string lin = op.spec.substr(0, ar) + BATCH, lout = op.spec.substr(ar + 2) + BATCH;
            TV obar = tview(op.out, nvec, true), abar = twrite(op.a, nvec, true, &beta), pin;
            pin.p = obar.p;
            pin.nd = abar.nd;
            for (int k = 0; k < abar.nd; k++) {
                size_t pos = lout.find(lin[k]);
                pin.n[k] = obar.n[pos];
                pin.s[k] = obar.s[pos];
            }
            permute_add(ex_, op.alpha, pin, beta, abar);
            break;
        }
        case OpKind::SquareForms: {
            // p enters S_aibj and S_bjai (its diagonal once) and both through the exchanged form: the
            // transpose is the symmetrised packing of the two adjoints
            const double *sa = has_adjoint(op.out) ? adjoint(op.out, nvec) : nullptr;
            const double *ua = has_adjoint(op.out2) ? adjoint(op.out2, nvec) : nullptr;
            const TV out = twrite(op.a, nvec, true, &beta);
            ccsd::sym_pack(ex_, sa, ua, no, nv, nvec, op.c1, op.c2, out.p, beta != 0.0);
            break;
        }
        case OpKind::SymPack: {
            // d packed[(M, m)] / d z[x, y] = 1 for {x, y} = {M, m} (the diagonal's 1/2 meets two
            // equal entries): the adjoint is the full symmetric square-up of the packed adjoint
            double *fa = nullptr, *xa = nullptr, beta_x = 1.0;
            if (nodes_[op.a].active) fa = twrite(op.a, nvec, true, &beta).p;
            if (nodes_[op.b].active) xa = twrite(op.b, nvec, true, &beta_x).p;
            ccsd::square_forms(ex_, adjoint(op.out, nvec), no, nv, nvec, op.c1, op.c2, fa, xa, beta != 0.0, beta_x != 0.0);
            break;
        }
        case OpKind::Trace: {
            if (!nodes_[op.a].active) break;
            const GNode &a = nodes_[op.a];
            trace_batch_kernel<<<grid_for(a.dims[0] * nvec, 128), 128, 0, ex_.stream>>>(
                adjoint(op.out, nvec), adjoint(op.a, nvec), a.dims[0], a.dims[1], nvec, 1);
            ex_.launches++;
            break;
        }
        case OpKind::Custom:
            customs_[op.custom].adjoint(nvec);
            break;
        }
        CU_CHECK(cudaGetLastError());
    }
    for (size_t k = 0; k < inputs.size(); k++) store_result(inputs[k], nvec, true, results[k]);
}

}  // namespace ccsd
