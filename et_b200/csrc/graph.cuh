// A recorded computation over device tensors with forward (JVP) and reverse (VJP) derivative
// passes.  The CCSD residual is written once against this interface: the plain residual runs
// the recorded ops eagerly; the Jacobian transformation replays them with tangents (one extra
// trailing index over the trial vectors), the transpose transformation and the adjoints into the
// Cholesky vectors and h run them backwards.
#pragma once

#include <functional>
#include <string>
#include <vector>

#include "common.cuh"

namespace ccsd {

struct GNode {
    std::string name;
    std::vector<int64_t> dims;   // column-major, contiguous
    int64_t size = 1;
    double *v = nullptr;         // primal value
    DBuf own;                    // storage when the graph owns the primal
    DBuf tan, adj;               // [size x nvec]
    // allocated and not written yet: reads as zero, and the first op writing it overwrites (clearing every
    // derivative first took 2.1 of 130 ms for six trials at o=24, v=240, and the first addition read it again)
    bool tan_zero = false, adj_zero = false;
    bool active = false;         // depends on a differentiated input
    bool zero = false;           // allocated by zeros() and not written yet: reads as zero, and the
                                 // first op writing it overwrites instead of accumulating
    int last_use = -1;           // index of the last op reading this node
};

enum class OpKind { Contract, Permute, SquareForms, SymPack, Trace, Custom };

// A custom op supplies its own forward / tangent / adjoint callbacks.
struct CustomOp {
    std::function<void()> forward;
    std::function<void(int nvec)> tangent;   // reads input tangents, accumulates out tangent
    std::function<void(int nvec)> adjoint;   // reads out adjoint, accumulates input adjoints
    std::vector<int> tangent_reads;          // the nodes whose tangents `tangent` reads
};

struct GOp {
    OpKind kind;
    int out = -1, a = -1, b = -1;
    int out2 = -1;               // SquareForms: the exchanged form
    double alpha = 1.0;
    double c1 = 0.0, c2 = 0.0;   // SquareForms, SymPack: weights of a form and of its exchange
    std::string spec;            // contract: "la,lb->lc"; permute: "lin->lout"
    bool fp64 = false;           // force FP64 (first-order terms)
    // contract of a node with itself whose output is only read as out + out^T: one of the two equal halves of
    // its derivative, 7 of 128 ms for six trials at o=24, v=240
    bool sym = false;
    int custom = -1;
};

class Graph {
  public:
    explicit Graph(Exec &ex) : ex_(ex) {}
    Graph(const Graph &) = delete;
    Graph &operator=(const Graph &) = delete;

    // node creation
    int input(const std::string &name, std::vector<int64_t> dims, const double *p);
    int zeros(const std::string &name, std::vector<int64_t> dims);
    int alias(int node);   // same value (e.g. an unchanged block)

    // out += alpha * einsum(spec, a, b)
    void contract(int out, const char *spec, double alpha, int a, int b, bool fp64 = false);
    // out += alpha * einsum(spec, a, a), symmetric under exchange of the two factors' indices, where every
    // reader of out takes its symmetric part (sym_pack): the two terms of its derivative count the same
    void contract_sym(int out, const char *spec, double alpha, int a, bool fp64 = false);
    // the same product when its value is at hand: `forward` adds it to out, the derivative passes contract
    void contract_given(int out, const char *spec, double alpha, int a, int b, const std::function<void()> &forward);
    // out += alpha * permute(a), spec "ajbi->aibj" (labels name the dims of a / out)
    void permute(int out, const char *spec, double alpha, int a);
    // t (full (v,o,v,o)) += squareup(a packed), u += c1 t_aibj + c2 t_ajbi
    void square_forms(int t, int u, int a, double c1, double c2);
    // out(packed) += pack with the diagonal halved of z + z^T, z = a + c1 x_aibj + c2 x_ajbi (a, x full)
    void sym_pack(int out, int a, int x, double c1, double c2);
    // out[J] += sum_k a[J, k, k]
    void trace(int out, int a);
    // custom op over existing nodes
    int custom(CustomOp op, int out, std::vector<int> ins);

    GNode &node(int i) {
        materialize(i);
        return nodes_[i];
    }
    const double *value(int i) {
        materialize(i);
        return nodes_[i].v;
    }
    int64_t no = 0, nv = 0;        // for square_forms / sym_pack

    // derivative passes; the seeds and results of a node are nvec device columns of its size, ld elements
    // apart.  Each pass starts from zero tangents / adjoints, so a recording can serve several passes.
    // `seeded` (jvp) runs once the seeds stand in the tangents.
    // Strided, so that the singles and doubles of a block of vectors go in and out as they lie: splitting and
    // joining them were two more passes, 0.8 of 101.7 ms for six trials at o=24, v=240.
    struct In {
        const double *p;
        int64_t ld;
    };
    struct Out {
        double *p;
        int64_t ld;
    };
    void mark_active(const std::vector<int> &inputs);
    void clear_derivatives();
    void jvp(const std::vector<int> &inputs, const std::vector<In> &seeds, int nvec, const std::vector<int> &outputs,
             const std::vector<Out> &results, const std::function<void()> &seeded);
    void vjp(const std::vector<int> &outputs, const std::vector<In> &seeds, int nvec, const std::vector<int> &inputs,
             const std::vector<Out> &results);
    // helpers for custom ops
    double *tangent(int i, int nvec);   // allocated on first use; zero where nothing has been written
    double *adjoint(int i, int nvec);
    bool has_adjoint(int i) const { return (bool)nodes_[i].adj && !nodes_[i].adj_zero; }
    Exec &exec() { return ex_; }

  private:
    Exec &ex_;
    std::vector<GNode> nodes_;
    std::vector<GOp> ops_;
    std::vector<CustomOp> customs_;
    std::vector<std::vector<int>> custom_ins_;
    void run_forward(const GOp &op);
    TV view(int node) const;
    // fills a node that zeros() allocated and nothing has written yet
    void materialize(int node);
    // the node's tangents / adjoints as a view over (node dims, trial)
    TV tview(int node, int nvec, bool adjoint);
    // the same for an op that writes every element: *beta is 0 when nothing has been written yet (the op
    // then overwrites), else 1
    TV twrite(int node, int nvec, bool adjoint, double *beta);
    double *derivative(int node, int nvec, bool adjoint);   // allocated, contents undefined while zero
    void record(GOp op);
    // nvec columns of `size` elements between strided arrays; results that nothing reached are zero
    void copy_columns(double *dst, int64_t ldd, const double *src, int64_t lds, int64_t size, int nvec);
    void store_result(int node, int nvec, bool adjoint, const Out &out);
};

}  // namespace ccsd
