// The CCSD residual Omega(t) recorded on a Graph, and the Jacobian transformations derived from
// it: rho = A c = (dOmega/dt) D c (forward mode) and sigma = b^T A = D (dOmega/dt)^T b (reverse
// mode), D = 2 on the packed doubles diagonal (jacobian_ccsd.F90:74-176).  Every term restates
// the routine of the eT file cited beside it.
#include <cstdio>
#include <cstdlib>
#include <memory>

#include "amp_forms.cuh"
#include "ccsd.cuh"
#include "ccsd_kernels.cuh"
#include "graph.cuh"
#include "mixed_gemm.cuh"
#include "tensor_ops.cuh"

namespace ccsd {

// ---------------------------------------------------------------------------
// Omega on the graph
// ---------------------------------------------------------------------------
OmegaNodes Context::record_omega(Graph &g, bool const_ovov, bool const_t1) {
    OmegaNodes n{};
    g.no = no;
    g.nv = nv;
    const std::vector<int64_t> V4 = {nv, no, nv, no};
    n.t1 = g.input("t1", {nv, no}, t.d());
    n.t2 = g.input("t2", {nt2}, t.d() + nt1);
    n.L_oo = g.input("L_oo", {nJ, no, no}, L_oo.d());
    n.L_ov = g.input("L_ov", {nJ, no, nv}, L_ov.d());
    n.L_vo = g.input("L_vo", {nJ, nv, no}, L_vo.d());
    n.L_vv = g.input("L_vv", {nJ, nv, nv}, L_vv.d());
    n.h_oo = g.input("h_oo", {no, no}, hb_oo.d());
    n.h_ov = g.input("h_ov", {no, nv}, hb_ov.d());
    n.h_vo = g.input("h_vo", {nv, no}, hb_vo.d());
    n.h_vv = g.input("h_vv", {nv, nv}, hb_vv.d());
    const int t1 = n.t1;

    int Lt_ov, Lt_oo, Lt_vo, Lt_vv, F_oo, F_ov, F_vo, F_vv;
    if (const_t1) {
        // the context transformed the blocks and built the Fock matrix at this t1 (refresh())
        Lt_oo = g.input("Lt_oo", {nJ, no, no}, this->Lt_oo.d());
        Lt_ov = g.input("Lt_ov", {nJ, no, nv}, this->Lt_ov.d());
        Lt_vo = g.input("Lt_vo", {nJ, nv, no}, this->Lt_vo.d());
        Lt_vv = g.input("Lt_vv", {nJ, nv, nv}, this->Lt_vv.d());
        F_oo = g.input("F_oo", {no, no}, fb_oo.d());
        F_ov = g.input("F_ov", {no, nv}, fb_ov.d());
        F_vo = g.input("F_vo", {nv, no}, fb_vo.d());
        F_vv = g.input("F_vv", {nv, nv}, fb_vv.d());
        n.Lt_vv = Lt_vv;
    } else {
        // construct_t1_cholesky (src/wavefunctions/ccs/t1_ccs.F90:208-499); the ov block is unchanged
        auto t1_timer = std::make_unique<TermTimer>(ex, "T1 transform cholesky");
        Lt_ov = g.alias(n.L_ov);
        Lt_oo = g.zeros("Lt_oo", {nJ, no, no});
        g.permute(Lt_oo, "Jij->Jij", 1.0, n.L_oo);
        g.contract(Lt_oo, "Jia,aj->Jij", 1.0, n.L_ov, t1, true);
        Lt_vo = g.zeros("Lt_vo", {nJ, nv, no});
        g.permute(Lt_vo, "Jai->Jai", 1.0, n.L_vo);
        g.contract(Lt_vo, "Jab,bi->Jai", 1.0, n.L_vv, t1, true);
        g.contract(Lt_vo, "aj,Jji->Jai", -1.0, t1, Lt_oo, true);
        Lt_vv = g.zeros("Lt_vv", {nJ, nv, nv});
        g.permute(Lt_vv, "Jab->Jab", 1.0, n.L_vv);
        g.contract(Lt_vv, "aj,Jjb->Jab", -1.0, t1, n.L_ov, true);
        n.Lt_vv = Lt_vv;
        t1_timer.reset();

        // T1 Fock matrix in blocks (fock_ccs.F90:242-1107): h~ = (1 - t1) h (1 + t1) then
        // F_pq = h~_pq + 2 sum_J L~_pq X_J - sum_Jk L~_pk L~_kq, X_J = sum_k L~_kk
        auto fock_timer = std::make_unique<TermTimer>(ex, "Fock matrix construction (T1 basis)");
        F_oo = g.zeros("F_oo", {no, no});
        F_ov = g.zeros("F_ov", {no, nv});
        F_vo = g.zeros("F_vo", {nv, no});
        F_vv = g.zeros("F_vv", {nv, nv});
        g.permute(F_oo, "ij->ij", 1.0, n.h_oo);
        g.contract(F_oo, "ia,aj->ij", 1.0, n.h_ov, t1, true);          // h~_oo = h_oo + h_ov t1
        g.permute(F_ov, "ia->ia", 1.0, n.h_ov);                          // h~_ov = h_ov
        g.permute(F_vv, "ab->ab", 1.0, n.h_vv);
        g.contract(F_vv, "ai,ib->ab", -1.0, t1, n.h_ov, true);          // h~_vv = h_vv - t1 h_ov
        const int Woo = g.zeros("W_oo", {no, no});
        g.permute(Woo, "ij->ij", 1.0, n.h_oo);
        g.contract(Woo, "ia,aj->ij", 1.0, n.h_ov, t1, true);
        g.permute(F_vo, "ai->ai", 1.0, n.h_vo);
        g.contract(F_vo, "ab,bi->ai", 1.0, n.h_vv, t1, true);
        g.contract(F_vo, "aj,ji->ai", -1.0, t1, Woo, true);             // h~_vo = h_vo + h_vv t1 - t1 W_oo
        const int X = g.zeros("X_J", {nJ});
        g.trace(X, Lt_oo);
        g.contract(F_oo, "Jpq,J->pq", 2.0, Lt_oo, X, true);
        g.contract(F_ov, "Jpq,J->pq", 2.0, Lt_ov, X, true);
        g.contract(F_vo, "Jpq,J->pq", 2.0, Lt_vo, X, true);
        // 2 sum_J L~_vv X_J through L~_vv = L_vv - t1 L_ov, so that no derivative of L~_vv is formed
        g.contract(F_vv, "Jpq,J->pq", 2.0, n.L_vv, X, true);
        const int V = g.zeros("V_jb", {no, nv});
        g.contract(V, "Jjb,J->jb", 1.0, n.L_ov, X, true);
        g.contract(F_vv, "aj,jb->ab", -2.0, t1, V, true);
        g.contract(F_oo, "Jpk,Jkq->pq", -1.0, Lt_oo, Lt_oo, true);
        g.contract(F_ov, "Jpk,Jkq->pq", -1.0, Lt_oo, Lt_ov, true);
        g.contract(F_vo, "Jpk,Jkq->pq", -1.0, Lt_vo, Lt_oo, true);
        g.contract(F_vv, "Jpk,Jkq->pq", -1.0, Lt_vo, Lt_ov, true);
        fock_timer.reset();
    }

    // construct_omega_ccsd (src/wavefunctions/ccsd/omega_ccsd.F90:39-110)
    const int om1 = g.zeros("omega1", {nv, no});
    g.permute(om1, "ai->ai", 1.0, F_vo);                            // omega_ccs_a1 (omega_ccs.F90:62)
    const int tf = g.zeros("t_aibj", V4);
    const int u = g.zeros("u_aibj", V4);                             // construct_u_aibj (omega_ccsd.F90:881)
    {
        TermTimer tt(ex, "Construct u_aibj");
        g.square_forms(tf, u, n.t2, 2.0, -1.0);                      // squareup (reordering.F90:4174), 2 t_aibj - t_ajbi
    }
    {
        // omega_doubles_a1 (src/wavefunctions/doubles/omega_doubles.F90:36-138)
        TermTimer tt(ex, "omega doubles a1");
        const int XJ = g.zeros("X_Jbi", {nJ, nv, no});
        g.contract(XJ, "Jcj,cjbi->Jbi", 1.0, n.L_vo, u);
        if (const_t1) {
            g.contract(om1, "Jab,Jbi->ai", 1.0, Lt_vv, XJ);
        } else {
            g.contract(om1, "Jab,Jbi->ai", 1.0, n.L_vv, XJ);
            const int W = g.zeros("W_ji", {no, no});
            g.contract(W, "Jjb,Jbi->ji", 1.0, n.L_ov, XJ);
            g.contract(om1, "aj,ji->ai", -1.0, t1, W);
        }
    }
    {
        // omega_doubles_b1 (:141-204)
        TermTimer tt(ex, "omega doubles b1");
        const int gkbji = g.zeros("g_kbji", {no, nv, no, no});
        g.contract(gkbji, "Jkb,Jji->kbji", 1.0, Lt_ov, Lt_oo);
        g.contract(om1, "ajbk,kbji->ai", -1.0, u, gkbji);
    }
    {
        // omega_doubles_c1 (:207-258)
        TermTimer tt(ex, "omega doubles c1");
        g.contract(om1, "bjai,jb->ai", 1.0, u, F_ov, true);
    }

    // g_ldkc, shared below (FP64 cache unless the adjoint into L_ov is wanted)
    int G4;
    if (const_ovov) {
        G4 = g.input("g_ovov", {no, nv, no, nv}, g_ovov_const());
    } else {
        G4 = g.zeros("g_ovov", {no, nv, no, nv});
        g.contract(G4, "Jia,Jjb->iajb", 1.0, Lt_ov, Lt_ov);
    }
    // its forms in the pair layout of the amplitudes: H = g_lckd - 1/2 g_kcld and the exchanged g_kcld, both
    // as [c, l, d, k], so that the products with t and u below are matrix products as they lie.  H, g_kcld, t, u
    // and the exchanged t are symmetric in their two pairs: each product names the pair that it sums first, so
    // that its operands run along the summed index in memory
    int H, GX;
    if (const_ovov) {
        g_pairs_const();
        H = g.input("H_cldk", V4, hov.d());
        GX = g.input("gx_cldk", V4, gex.d());
    } else {
        H = g.zeros("H_cldk", V4);
        GX = g.zeros("gx_cldk", V4);
        g.permute(GX, "kcld->cldk", 1.0, G4);
        g.permute(H, "lckd->cldk", 1.0, G4);
        g.permute(H, "cldk->cldk", -0.5, GX);
    }
    // omega_ccsd_e2 (omega_ccsd.F90:712-878); Fock parts in FP64
    const int om = g.zeros("omega_aibj", V4), x = g.zeros("x_c2", V4);
    {
        TermTimer tt(ex, "omega ccsd e2");
        const int Xbc = g.zeros("X_bc", {nv, nv}), Ykj = g.zeros("Y_kj", {no, no});
        // sum_kdl u_bkdl g_ldkc = 2 sum t_bkdl H_kcld, sum_dlc g_kdlc u_djcl = 2 sum H_lckd t_cldj
        g.contract(Xbc, ex.prec == Prec::FP64 ? "bkdl,ckdl->bc" : "dlbk,dlck->bc", -2.0, tf, H);
        g.contract(Ykj, "cldk,cldj->kj", 2.0, H, tf);
        // the Fock blocks join X and Y, so each side is one FP64 product with t (the Fock parts are
        // first-order terms)
        g.permute(Xbc, "bc->bc", 1.0, F_vv);
        g.permute(Ykj, "kj->kj", 1.0, F_oo);
        g.contract(om, "bc,cjai->bjai", 1.0, Xbc, tf, true);
        g.contract(om, "aibk,kj->aibj", -1.0, tf, Ykj, true);
    }
    auto yq = std::make_shared<LadderY>();
    // om collects the terms that eT symmetrises (symmetric_sum, reordering.F90:416), x the C2 term whose
    // third and exchanged two thirds join them: the doubles residual is pack(z + z^T), z = om + x_aibj/3
    // + 2 x_ajbi/3, with the diagonal halved, formed in one pass at the end.  Terms
    // that are symmetric already enter with weight 1/2.
    // omega_ccsd_b2 (omega_ccsd.F90:483-583); g_aibj in FP64
    {
        TermTimer tt(ex, "omega ccsd b2");
        g.contract_sym(om, "Jai,Jbj->aibj", 0.5, Lt_vo, true);
        const int X4 = g.zeros("X_klij", {no, no, no, no});
        g.contract(X4, "Jki,Jlj->klij", 1.0, Lt_oo, Lt_oo);
        if (const_ovov && plain_ladder()) {
            // Q_kilj of the ladder's t1 part is this term
            *yq = ladder_y_plain(g.value(tf));
            g.contract_given(X4, "kcld,cidj->klij", 1.0, G4, tf, [&]() {
                TV q = tv(yq->Q.d(), {no, no, no, no});   // [k, i, l, j] read as [k, l, i, j]
                std::swap(q.s[1], q.s[2]);
                permute_add(ex, 1.0, q, 1.0, tv(g.node(X4).v, {no, no, no, no}));
            });
        } else {
            g.contract(X4, "kcld,cidj->klij", 1.0, G4, tf);
        }
        g.contract(om, "akbl,klij->aibj", 0.5, tf, X4);
    }
    // omega_ccsd_c2_d2 (omega_ccsd.F90:586-709) in contraction form
    {
        TermTimer tt(ex, "omega ccsd c2 and d2");
        const int C = g.zeros("C_term", V4), D = g.zeros("D_term", V4);
        if (const_t1) {
            g.contract(C, "Jac,Jkj->ckaj", 1.0, Lt_vv, Lt_oo);
        } else {
            // g_ackj through L~_vv = L_vv - t1 L_ov: a derivative in t1 costs a product over n_o instead of
            // one over N_J with an n_v^2 N_J tangent of L~_vv
            g.contract(C, "Jac,Jkj->ckaj", 1.0, n.L_vv, Lt_oo);
            const int G = g.zeros("g_lckj", {no, nv, no, no});
            g.contract(G, "Jlc,Jkj->lckj", 1.0, n.L_ov, Lt_oo);
            g.contract(C, "al,lckj->ckaj", -1.0, t1, G);
        }
        g.permute(D, "ckaj->ckaj", -1.0, C);
        g.contract(D, "Jai,Jkc->ckai", 2.0, Lt_vo, Lt_ov);
        if (ex.prec == Prec::FP64) {
            // t_djak as [d, k, a, j], shared by both of its products (the tensor-core GEMM gathers it itself)
            const int tx = g.zeros("tx_dkaj", V4);
            g.permute(tx, "djak->dkaj", 1.0, tf);
            g.contract(C, "dkcl,dkaj->claj", -0.5, GX, tx);
            g.contract(x, "ckai,ckbj->aibj", -1.5, tx, C);
        } else {
            g.contract(C, "dkcl,djak->claj", -0.5, GX, tf);
            g.contract(x, "ciak,ckbj->aibj", -1.5, tf, C);
        }
        g.contract(D, "dkcl,dkaj->claj", 1.0, H, u);
        g.contract(om, "ckai,ckbj->aibj", 0.5, u, D);
    }
    // omega_ccsd_a2 (omega_ccsd.F90:113-480) as custom ops: its t1 part joins om, its t2 part the packed residual
    record_ladder_t1(g, om, Lt_vv, t1, n.L_vv, tf, yq);
    const int om2 = g.zeros("omega2", {nt2});
    g.sym_pack(om2, om, x, 1.0 / 3.0, 2.0 / 3.0);   // symmetric_sum + scale_diagonal(1/2) + packin
    record_ladder(g, om2, Lt_vv, n.t2);
    n.om1 = om1;
    n.om2 = om2;
    return n;
}

// Y[k,i,b,j] = sum_cd g_kcbd t_cidj with g_kcbd = sum_J L_kc L~_bd (batched over b; in mixed
// precision the residual and the derivatives take Y from the resident ovvv planes instead)
void Context::ladder_y(const double *Lvv, const double *tfull, double *Y) {
    cudaStream_t s = ex.stream;
    const int64_t nb = std::max<int64_t>(1, std::min<int64_t>(nv, (int64_t)(2.0e9 / (8.0 * no * nv * nv))));
    DBuf gblk = dalloc(no * nv * nb * nv, s);
    for (int64_t b0 = 0; b0 < nv; b0 += nb) {
        const int64_t b1 = std::min(nv, b0 + nb), len = b1 - b0;
        TV Lb = tv(Lvv + nJ * b0, {nJ, len, nv});
        Lb.s[1] = nJ;
        Lb.s[2] = nJ * nv;
        TV gb = tv(gblk.d(), {no, nv, len, nv});
        contract(ex, "Jkc,Jbd->kcbd", 1.0, tv(L_ov.d(), {nJ, no, nv}), Lb, 0.0, gb);
        TV Yb = tv(Y + no * no * b0, {no, no, len, no});
        Yb.s[1] = no;
        Yb.s[2] = no * no;
        Yb.s[3] = no * no * nv;
        contract(ex, "kcbd,cidj->kibj", 1.0, gb, tv(tfull, {nv, no, nv, no}), 0.0, Yb);
    }
}

// The part of the A2 ladder that depends on t1, as terms A_aibj of om (which is packed as A + A^T): in
// the residual the corrections that turn integrals of the untransformed vectors into T1-transformed
// ones (nothing when the integrals are formed from transformed vectors); in the derivative passes the
// t1 derivative through Y.
void Context::record_ladder_t1(Graph &g, int om, int Lvv, int t1, int L_vv_in, int tf, std::shared_ptr<LadderY> yq) {
    auto Ycache = std::make_shared<DBuf>();
    auto getY = [this, &g, Lvv, t1, tf, yq, Ycache]() -> const double * {
        if (!*Ycache) {
            *Ycache = dalloc(no * no * nv * no, ex.stream);
            ladder_y_t1(g.value(t1), g.value(Lvv), g.value(tf), *yq, Ycache->d());
        }
        return Ycache->d();
    };
    CustomOp op;
    op.forward = [this, &g, om, t1, tf, yq]() {
        TermTimer tt(ex, "omega ccsd a2");
        if (!plain_ladder()) return;
        if (!yq->Y) *yq = ladder_y_plain(g.value(tf));
        ladder_t1_corrections(g.value(t1), *yq, g.node(om).v);
    };
    op.tangent_reads = {t1};
    op.tangent = [this, &g, om, Lvv, t1, getY](int nvec) {
        REQUIRE(!g.node(Lvv).active || g.node(t1).active, CCSD_GPU_EINVAL,
                "ladder tangent: L_vv directions are not supported");
        if (!g.node(t1).active) return;
        // d L~_ac = -sum_k c_ak L_kc: A_aibj = -sum_k c_ak Y_kibj
        double *out = g.tangent(om, nvec);
        const double *Y = getY(), *c1 = g.tangent(t1, nvec);
        for (int n = 0; n < nvec; n++)
            contract(ex, "ak,kibj->aibj", -1.0, tv(c1 + n * nt1, {nv, no}), tv(Y, {no, no, nv, no}), 1.0,
                     tv(out + n * nov * nov, {nv, no, nv, no}));
    };
    op.adjoint = [this, &g, om, Lvv, t1, tf, L_vv_in, getY](int nvec) {
        // adjoint into the Cholesky vectors requested: dense route through L~_vv (its adjoint also
        // reaches t1 through the recorded T1 transformation); otherwise the rank-n_o route via Y.  The
        // adjoint of om is the symmetric square-up S of the packed residual's adjoint.
        const bool dense = g.node(L_vv_in).active;
        if (!g.node(t1).active && !dense) return;
        const double *S = g.adjoint(om, nvec);
        for (int n = 0; n < nvec; n++) {
            const TV B = tv(S + n * nov * nov, {nv, no, nv, no});
            if (!dense) {
                // t1bar_ak -= sum_ibj S_aibj Y_kibj
                contract(ex, "aibj,kibj->ak", -1.0, B, tv(getY(), {no, no, nv, no}), 1.0,
                         tv(g.adjoint(t1, nvec) + n * nt1, {nv, no}));
            } else {
                // Lbar_J,ac += sum_bd L_J,bd Z_acbd, Z_acbd = sum_ij S_aibj t_cidj
                REQUIRE((double)nv * nv * nv * nv * 8.0 < 24e9, CCSD_GPU_EINVAL,
                        "ladder adjoint into L_vv needs v^4 doubles of scratch; system too large");
                DBuf Z = dalloc(nv * nv * nv * nv, ex.stream);
                contract(ex, "aibj,cidj->acbd", 1.0, B, tv(g.value(tf), {nv, no, nv, no}), 0.0,
                         tv(Z.d(), {nv, nv, nv, nv}));
                contract(ex, "Jbd,acbd->Jac", 1.0, tv(g.value(Lvv), {nJ, nv, nv}), tv(Z.d(), {nv, nv, nv, nv}), 1.0,
                         tv(g.adjoint(Lvv, nvec) + n * nJ * nv * nv, {nJ, nv, nv}));
            }
        }
    };
    g.custom(std::move(op), om, {Lvv, t1, tf});
}

// sum_cd g_acbd t_cidj into the packed residual: in the residual with integrals of the untransformed
// vectors where they are kept, in the derivative passes with the T1-transformed ones
void Context::record_ladder(Graph &g, int om2, int Lvv, int t2) {
    auto LTcache = std::make_shared<DBuf>();
    auto getLT = [this, &g, Lvv, LTcache]() -> const double * {
        if (!*LTcache) {
            *LTcache = dalloc(nJ * nv * nv, ex.stream);
            TV src = tv(g.value(Lvv), {nJ, nv, nv});
            TV dst = tv(LTcache->d(), {nJ, nv, nv});
            dst.s[1] = nJ * nv;
            dst.s[2] = nJ;
            permute_add(ex, 1.0, src, 0.0, dst);
        }
        return LTcache->d();
    };
    CustomOp op;
    op.forward = [this, &g, om2, Lvv, t2]() {
        TermTimer tt(ex, "omega ccsd a2");
        if (ex.prec == Prec::MIXED)
            ladder_tc(L_vv.d(), g.value(t2), g.node(om2).v, 1, true);
        else if (f64_resident())
            ladder_f64(g.value(t2), g.node(om2).v);
        else
            ladder(g.value(Lvv), g.value(t2), g.node(om2).v);
    };
    op.tangent_reads = {t2};
    op.tangent = [this, &g, om2, Lvv, t2](int nvec) {
        if (g.node(t2).active) ladder(g.value(Lvv), g.tangent(t2, nvec), g.tangent(om2, nvec), nvec);
    };
    op.adjoint = [this, &g, om2, t2, getLT](int nvec) {
        // the transpose of the packed ladder is the same ladder with L~_vv transposed
        if (g.node(t2).active) ladder(getLT(), g.adjoint(om2, nvec), g.adjoint(t2, nvec), nvec);
    };
    g.custom(std::move(op), om2, {Lvv, t2});
}

void Context::omega_eager(double *om_out) {
    Graph g(ex);
    OmegaNodes n = record_omega(g, true, t1_current);
    CU_CHECK(cudaMemcpyAsync(om_out, g.value(n.om1), sizeof(double) * nt1, cudaMemcpyDeviceToDevice, ex.stream));
    CU_CHECK(cudaMemcpyAsync(om_out + nt1, g.value(n.om2), sizeof(double) * nt2, cudaMemcpyDeviceToDevice, ex.stream));
}

void Context::prepare_residual_caches() {
    g_pairs_const();
    if (ex.prec == Prec::MIXED) {
        if (ladder_pairs_resident()) ladder_pairs(L_vv.d(), true);
        if (ovvv_resident()) ovvv_pairs();
    } else if (f64_resident()) {
        f64_integrals();
        const YqRoute yq = yq_route();
        if (yq.y_digits) f64_ovvv_planes(ex.fp64_digits, yq.joined ? no * nmo : nov);
        const int digits = f64_ladder_digits();
        if (digits) f64_ladder_planes(digits);
    }
}

Context::ResidualGraph::Key Context::graph_key() const {
    return {l_version, cache_epoch, ex.k_chunk, ex.planes, ex.fp64_digits, ex.fp64_digits_min_flops,
            digit_arena.as<void>()};
}

// Records the residual on ex.stream into G.  A capture that fails (a call that cannot be captured)
// leaves G empty and turns graphs off for this context; the caller then evaluates eagerly.
void Context::capture_residual(ResidualGraph &G, double *om_out) {
    G.reset();
    graphs_captured = true;
    const double flops0 = ex.flops;
    const int64_t launches0 = ex.launches;
    cudaGraph_t graph = nullptr;
    std::string why;
    CU_CHECK(cudaStreamBeginCapture(ex.stream, cudaStreamCaptureModeThreadLocal));
    ex.capturing = true;
    try {
        omega_eager(om_out);
    } catch (const std::exception &e) {
        why = e.what();
    }
    ex.capturing = false;
    cudaError_t rc = cudaStreamEndCapture(ex.stream, &graph);
    if (why.empty() && rc == cudaSuccess && graph) {
        rc = cudaGraphInstantiate(&G.exec, graph, 0);
        if (rc != cudaSuccess) G.exec = nullptr;
    }
    if (graph) cudaGraphDestroy(graph);
    if (!G.exec) {
        if (why.empty()) why = cudaGetErrorString(rc);
        cudaGetLastError();
        use_graphs = false;
        if (std::getenv("CCSD_GPU_TRACE"))
            std::fprintf(stderr, "ccsd_gpu residual graph capture failed (%s); evaluating eagerly\n", why.c_str());
    }
    G.flops = ex.flops - flops0;
    G.launches = ex.launches - launches0;
    ex.flops = flops0;
    ex.launches = launches0;
    G.key = graph_key();
}

void Context::omega(double *om_out) {
    REQUIRE(have_t, CCSD_GPU_ESTATE, "amplitudes not set");
    if (!t1_current) refresh();   // the residual reads the context's T1-transformed blocks
    TermTimer tt(ex, "Construct CCSD Omega");
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CU_CHECK(cudaStreamIsCapturing(ex.stream, &cap));
    const bool graphs = use_graphs && !(ex.prof && ex.prof->on) && cap == cudaStreamCaptureStatusNone;
    if (!graphs) {
        omega_eager(om_out);
    } else {
        prepare_residual_caches();
        ResidualGraph &G = rgraph[ex.prec == Prec::MIXED ? 1 : 0];
        if (!G.warm || !G.key.same_digits(graph_key())) {
            omega_eager(om_out);
            G.reset();
            G.key = graph_key();
            G.warm = true;
        } else {
            // the graph writes a buffer of its own, so callers may pass any output
            if (!om_stage) om_stage = dalloc(namp, ex.stream);
            if (!(G.exec && G.key == graph_key())) capture_residual(G, om_stage.d());
            if (G.exec) {
                CU_CHECK(cudaGraphLaunch(G.exec, ex.stream));
                CU_CHECK(cudaMemcpyAsync(om_out, om_stage.d(), sizeof(double) * namp, cudaMemcpyDeviceToDevice,
                                         ex.stream));
                ex.flops += G.flops;
                ex.launches += G.launches;
                graph_replays++;
            } else {
                omega_eager(om_out);
            }
        }
    }
    check_gemm();
}

void Context::check_gemm() {
    const int code = gemm_error(ex, true);
    REQUIRE(code == 0, CCSD_GPU_ETIMEOUT,
            "tensor-core GEMM barrier wait timed out (code " + std::to_string(code) + ")");
}

// prepare_for_jacobian (jacobian_ccsd.F90:46-71) / prepare_for_jacobian_transpose
// (jacobian_transpose_ccsd.F90:44-126): eT computes and stores the t-dependent intermediates of its
// hand-written terms once per Davidson run; here the whole residual is recorded once at the current
// amplitudes, so every later transformation runs only its derivative pass over the stored values.
void Context::prepare_jacobian() {
    REQUIRE(have_t, CCSD_GPU_ESTATE, "amplitudes not set");
    drop_jacobian();
    auto p = std::make_unique<PreparedJacobian>();
    p->g = std::make_unique<Graph>(ex);
    p->n = record_omega(*p->g);
    p->prec = ex.prec;
    p->planes = ex.planes;
    p->k_chunk = ex.k_chunk;
    p->l_version = l_version;
    p->id = ++prep_counter;
    CU_CHECK(cudaStreamSynchronize(ex.stream));
    check_gemm();
    prep = std::move(p);
}

void Context::drop_jacobian() {
    if (!prep) return;
    prep.reset();
    if (mbuf_kind == 2) mbuf_reuse = -1;
}

Graph &Context::transform_graph(std::unique_ptr<Graph> &local, OmegaNodes &n) {
    if (prep && prep->prec == ex.prec && prep->planes == ex.planes && prep->k_chunk == ex.k_chunk &&
        prep->l_version == l_version) {
        n = prep->n;
        pairs_reuse_id = prep->id;
        return *prep->g;
    }
    local = std::make_unique<Graph>(ex);
    n = record_omega(*local);
    return *local;
}

namespace {
// a prepared transformation's ladder integrals stay reusable only while it runs
struct ReuseScope {
    int64_t &id;
    ~ReuseScope() { id = -1; }
};
}  // namespace

// rho_k = A c_k for n_vec device columns [t1 | packed t2]
void Context::jacobian(int64_t nvec, const double *c, double *rho) {
    REQUIRE(have_t, CCSD_GPU_ESTATE, "amplitudes not set");
    TermTimer tt(ex, "Jacobian CCSD transformation");
    ReuseScope scope{pairs_reuse_id};
    std::unique_ptr<Graph> local;
    OmegaNodes n;
    Graph &g = transform_graph(local, n);
    // the diagonal factor D = 2 goes on the copy of c that the tangents start from
    g.jvp({n.t1, n.t2}, {{c, namp}, {c + nt1, namp}}, (int)nvec, {n.om1, n.om2}, {{rho, namp}, {rho + nt1, namp}},
          [&] { scale_doubles_diag(ex, g.tangent(n.t2, (int)nvec), nov, nvec, nt2, 2.0); });
    g.clear_derivatives();
    CU_CHECK(cudaStreamSynchronize(ex.stream));
    check_gemm();
}

// sigma_k = b_k^T A = D (dOmega/dt)^T b_k
void Context::jacobian_transpose(int64_t nvec, const double *b, double *sigma) {
    REQUIRE(have_t, CCSD_GPU_ESTATE, "amplitudes not set");
    TermTimer tt(ex, "Jacobian transpose CCSD");
    ReuseScope scope{pairs_reuse_id};
    std::unique_ptr<Graph> local;
    OmegaNodes n;
    Graph &g = transform_graph(local, n);
    g.vjp({n.om1, n.om2}, {{b, namp}, {b + nt1, namp}}, (int)nvec, {n.t1, n.t2}, {{sigma, namp}, {sigma + nt1, namp}});
    scale_doubles_diag(ex, sigma + nt1, nov, nvec, namp, 2.0);
    g.clear_derivatives();
    CU_CHECK(cudaStreamSynchronize(ex.stream));
    check_gemm();
}

// b^T dOmega/d(t, L, h): amplitude part without the D scaling, plus the adjoints into the MO
// Cholesky blocks (J, p, q) and the MO one-electron Hamiltonian (n_mo x n_mo, column-major)
void Context::adjoint(const double *b, double *dt, double *dL, double *dh) {
    REQUIRE(have_t, CCSD_GPU_ESTATE, "amplitudes not set");
    Graph g(ex);
    OmegaNodes n = record_omega(g, dL == nullptr);
    std::vector<int> ins = {n.t1, n.t2};
    std::vector<DBuf> outs;
    DBuf dt_own;
    if (!dt) {
        dt_own = dalloc(namp, ex.stream);
        dt = dt_own.d();
    }
    const bool wantL = dL != nullptr, wanth = dh != nullptr;
    if (wantL)
        for (int node : {n.L_oo, n.L_ov, n.L_vo, n.L_vv}) {
            ins.push_back(node);
            outs.push_back(dalloc(g.node(node).size, ex.stream));
        }
    if (wanth)
        for (int node : {n.h_oo, n.h_ov, n.h_vo, n.h_vv}) {
            ins.push_back(node);
            outs.push_back(dalloc(g.node(node).size, ex.stream));
        }
    std::vector<Graph::Out> res = {{dt, namp}, {dt + nt1, namp}};
    for (auto &o : outs) res.push_back({o.d(), 0});
    g.vjp({n.om1, n.om2}, {{b, namp}, {b + nt1, namp}}, 1, ins, res);
    size_t k = 0;
    auto scatter = [&](double *full, int64_t ld, int64_t p0, int64_t q0, int64_t np, int64_t nq, const double *blk,
                       int64_t inner) {
        // full[(inner) x (p0+p) x (q0+q)] <- blk[inner x p x q]
        TV src = tv(blk, {inner, np, nq});
        TV dst;
        dst.p = full + inner * (p0 + ld * q0);
        dst.nd = 3;
        dst.n[0] = inner;
        dst.n[1] = np;
        dst.n[2] = nq;
        dst.s[0] = 1;
        dst.s[1] = inner;
        dst.s[2] = inner * ld;
        permute_add(ex, 1.0, src, 0.0, dst);
    };
    if (wantL) {
        scatter(dL, nmo, 0, 0, no, no, outs[k++].d(), nJ);
        scatter(dL, nmo, 0, no, no, nv, outs[k++].d(), nJ);
        scatter(dL, nmo, no, 0, nv, no, outs[k++].d(), nJ);
        scatter(dL, nmo, no, no, nv, nv, outs[k++].d(), nJ);
    }
    if (wanth) {
        scatter(dh, nmo, 0, 0, no, no, outs[k++].d(), 1);
        scatter(dh, nmo, 0, no, no, nv, outs[k++].d(), 1);
        scatter(dh, nmo, no, 0, nv, no, outs[k++].d(), 1);
        scatter(dh, nmo, no, no, nv, nv, outs[k++].d(), 1);
    }
    CU_CHECK(cudaGetLastError());
    CU_CHECK(cudaStreamSynchronize(ex.stream));
    check_gemm();
}

}  // namespace ccsd
