// Sweep operators of the composed ("state") form of the apply.
//
// A level call of the multi-split recursion sweeps x += B (f - A x), where B is
// the level's split factorisation: with A^ = the level matrix without its
// dropped links, B = Gt P with P = (I + L)^{-1} on the eliminated (E) and
// coarse (C) rows and the identity on the diagonal (D) rows, and
//   Gt [w_E; y_C; r_D] = [G (w_E, y_C); y_C; dval r_D],   y_C = coarse solve of w_C.
// Written in the variables s = [w_E; y_C; r_D] instead of x, a sweep is
//   v = P (f - A Gt s) = v0 - [s_E; 0; s_D] - K s,   v0 = P f,
//   K = P (A - A^) Gt + S on the C x C block,
// S being the Schur complement (the next level's matrix): P A^ Gt is the
// identity on E and D and S on C, exactly, so only the DROPPED links and the
// diagonal compensation (the rows of A - A^) enter K. One sparse product per
// sweep replaces phase 1, phase 2 and the correction, and nothing cancels that
// the separate steps would have had to cancel.
//
// The levels are chained: level l's P carries level l+1's on its coarse rows
// and Gt carries level l+1's on its coarse columns, so that phase 1 and phase
// 2 of every inner call disappear into the rows of the operator above it. What
// remains per sweep of a level is the call of the level below and one product.
//
// The uh_cheb recursion has the same shape: its Chebyshev steps run on the next
// level's system. There A^ holds the kept links divided by beta, so A - beta A^
// takes the place of A - A^ (again only dropped links and the diagonal):
//   v = v0 - beta [s_E; 0; s_D] - K s,   K = P (A - beta A^) Gt + beta S,
// and a step is the three-term combination of v with the last two states.
#pragma once

#include "setup.cuh"

namespace mlp {

// An operator with its rows stored by length class: rows of more than 32, 17
// to 32, 9 to 16, 5 to 8 and at most 4 entries (classes 1 to 5), taken by 32,
// 8, 4, 2 and 1 lanes, so that a lane holds four entries in registers (all of
// them issued together, ahead of the dependent-launch wait) and no row is a
// chain of dependent loads. Class 0 holds the rows with a dense part (a warp
// each). Rows keep their order inside a class.
constexpr int ROW_CLASSES = 6;
struct ClassedRows {
    DCSR m;                                // the rows, in class order
    DBuf<uint32_t> row;                    // stored position -> row
    uint32_t first[ROW_CLASSES + 1] = {};  // first stored position of each class
    DBuf<double> D;                        // class 0: dense part, dn entries a row
    uint32_t dn = 0;
};

struct StateOps {
    uint32_t m = 0;         // systems 1..m have a K
    bool absorbed = false;  // system m's sweeps need no coarse call: its coarse operator is part
                            // of K (absorbed whole, or as the dense part of K's class 0)
    bool whole = false;     // absorbed in G as well (FP64): the state's C entries stay w_C to the end
    ClassedRows P;          // rows [0, R0): [w_E0; v0 of system 1] = P f
    ClassedRows G;          // rows [0, R0), columns [0, R0): x = G [w_E0; state of system 1]
    std::vector<ClassedRows> K;  // K[j - 1]: the N_j rows of system j, in its frame
    DBuf<double> coarse;    // uh_cheb: the tabulated Chebyshev solve of system m + 1
    DBuf<uint32_t> Pcol, Grow;  // P's columns and G's rows in natural order
};

// Builds the operators of systems 1..m of H (levels 1..m must not be direct and
// must hold their dropped-link values). C (cn x cn, row-major, FP64) is the
// dense operator of level m + 1, or null. Up to ABSORB_WHOLE rows it becomes
// part of K_m and G as any other factor; not in an FP32 hierarchy, whose coarse
// solve keeps FP64 entries and sums (one launch more a call of system m:
// 60x220x20 iid, 4 coarse rows, 24.5 us an application in place of 23). Larger,
// K_m's rows with coarse columns (nd of them) take their product with it as a
// dense part, K_C C, where that is at most ABSORB_DENSE bytes and ABSORB_DENSE_N
// columns: a sweep then reads nd x cn entries but needs no coarse launch (without
// a system, m = 0, G's rows do). Past it the sweeps call the coarse operator.
// An application's launches in a graph, FP64, us (fields layered, or iid where
// said so; other levels tabulated than by default in the lines marked *):
//   cn                              whole   dense part   separate
//    4  60x220x20 iid                12.5      14.4
//   18  60x220x85 iid                18.5      18.5
//   31  59x211x37, c = 0.1 *         1250      1430
//   58  30x40x20, c = 0.1 *           230       285          422
//   76  60x110x40, c = 0.3 *          259       319          445
//  138  60x220x85, c = 0.3            521       503          657
//  204  60x220x20                     100        78          101
//  422  60x220x85 (nd = 2,292)        262       129          154
// so a whole absorption pays up to somewhere near 100 rows (32 keeps well inside
// it: its fill grows with nd), a dense part wherever it fits the registers.
// Returns null when a row of an operator
// holds more than STATE_ROW_MAX entries. fp32: the sparse values are stored in
// FP32, rounded once from their FP64 products.
constexpr uint32_t STATE_ROW_MAX = 1024;
constexpr uint32_t ABSORB_WHOLE = 32;
constexpr size_t ABSORB_DENSE = 12u << 20;
constexpr uint32_t ABSORB_DENSE_N = 512;  // columns of a dense part (a lane holds 16 in registers)
std::unique_ptr<StateOps> build_state(const Hierarchy& H, uint32_t m, const double* C, uint32_t cn, bool fp32,
                                      cudaStream_t s);

// Tabulates a Chebyshev solve of a system of n unknowns with the dense operator
// B of its preconditioner: `steps` iterations of Prec::solve (cheb_solve.cc:
// 49-100) on the matrix As, spectral bounds lmin, lmax. The result is n x n.
void tabulate_cheb(const DCSR& As, const double* B, uint32_t n, uint32_t steps, double lmin, double lmax,
                   DBuf<double>& out, cudaStream_t s);

}  // namespace mlp
