// Construction of the composed sweep operators (state.cuh): a handful of
// row-wise sparse products over the level operators of the set-up.
#include <memory>

#include "solve.cuh"
#include "state.cuh"

namespace mlp {

namespace {

// One row-wise sparse product out(q) = sum_t coef_t * right row_t (+ extra row).
// The four kinds of row share the accumulation below.
enum ProdMode : int {
    PM_G,  // Gt of a level: rows E (G with its coarse columns expanded), C, D
    PM_P,  // P of a level: rows E, C (the next level's P on the coarse rows of P1)
    PM_Q,  // (A - A^) Gt
    PM_K,  // P Q, plus the coarse block on the C rows
};

// A CSR operand; padded ones keep their rows at start[q], len[q] entries long.
struct Rows {
    const uint32_t* start = nullptr;  // row q begins at start[q]
    const uint32_t* len = nullptr;    // null: row q ends at start[q + 1]
    const uint32_t* col = nullptr;
    const double* val = nullptr;
    __device__ __forceinline__ uint32_t b(uint32_t q) const { return start[q]; }
    __device__ __forceinline__ uint32_t e(uint32_t q) const { return len ? start[q] + len[q] : start[q + 1]; }
};

struct Prod {
    int mode;
    uint32_t M, R, N;      // the level's E rows, E + C rows, all rows
    uint32_t M2, R2;       // of the next system (PM_P, PM_K)
    uint32_t rows;         // rows to compute
    Rows left, right, extra;
    const double* dval;                // PM_G: the level's D rows (null: not computed)
    const uint32_t *phi, *iphi;        // PM_Q: frame -> natural row, natural -> frame column
    const double* C;                   // dense coarse operator, cn x cn (PM_G, absorbed PM_K)
    uint32_t cn;
    bool chained;                      // the next level has operators of its own
    double theta, theta2;              // beta of this level and of the next system
};

// Visits the terms of row q. one(col, v) is a single entry, row(rows, k, shift,
// coef) all entries of row k of an operand, dense(k, shift, coef) row k of C;
// every lane of the group makes the same calls.
template <class One, class Row, class Dense>
__device__ __forceinline__ void prod_terms(const Prod& g, uint32_t q, One one, Row row, Dense dense) {
    if (g.mode == PM_G) {
        if (q < g.M) {
            for (uint32_t j = g.left.b(q), e = g.left.e(q); j < e; j++) {
                const uint32_t c = g.left.col[j];
                const double v = g.left.val[j];
                if (c < g.M) one(c, v);
                else if (g.C) dense(c - g.M, g.M, v);
                else if (g.chained) row(g.right, c - g.M, g.M, v);
                else one(c, v);
            }
        } else if (q < g.R) {
            if (g.C) dense(q - g.M, g.M, 1.0);
            else if (g.chained) row(g.right, q - g.M, g.M, 1.0);
            else one(q, 1.0);
        } else {
            one(q, g.dval[q - g.R]);
        }
    } else if (g.mode == PM_P) {
        // left: the next level's P; right: this level's P1
        if (q >= g.M && g.chained && q - g.M < g.R2) {
            for (uint32_t j = g.left.b(q - g.M), e = g.left.e(q - g.M); j < e; j++)
                row(g.right, g.M + g.left.col[j], 0, g.left.val[j]);
        } else {
            row(g.right, q, 0, 1.0);
        }
    } else if (g.mode == PM_Q) {
        const uint32_t i = g.phi[q];
        for (uint32_t j = g.left.b(i), e = g.left.e(i); j < e; j++) {
            const double v = g.left.val[j];
            if (v != 0) row(g.right, g.iphi[g.left.col[j]], 0, v);
        }
    } else {
        if (q < g.R) {
            for (uint32_t j = g.left.b(q), e = g.left.e(q); j < e; j++) row(g.right, g.left.col[j], 0, g.left.val[j]);
        } else {
            row(g.right, q, 0, 1.0);
        }
        if (q >= g.M && q < g.R) {
            const uint32_t i = q - g.M;
            if (g.C) {
                for (uint32_t j = g.extra.b(i), e = g.extra.e(i); j < e; j++)
                    dense(g.extra.col[j], g.M, g.theta * g.extra.val[j]);
            } else {
                row(g.extra, i, g.M, g.theta);
                if (g.chained && (i < g.M2 || i >= g.R2)) one(q, g.theta * g.theta2);
            }
        }
    }
}

// Upper bound of every row's length (its number of products), and their sum
// in 64 bits: the 32-bit row offsets are used only when it fits.
__global__ void __launch_bounds__(256) k_prod_bound(Prod g, uint32_t* __restrict__ ub, unsigned long long* sum) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t n = 0;
    if (q < g.rows) {
        prod_terms(
            g, q, [&](uint32_t, double) { n++; },
            [&](const Rows& r, uint32_t k, uint32_t, double) { n += r.e(k) - r.b(k); },
            [&](uint32_t, uint32_t, double) { n += g.cn; });
        ub[q] = n;
    }
    unsigned long long t = n;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0 && t) atomicAdd(sum, t);
}

// Computes rows with W lanes each and a hash table of CAP entries per row in
// shared memory. The terms of a row are added one after another (the lanes
// share a term's entries, whose columns differ), so every value is summed in
// a fixed order, and the row leaves sorted by column: the operator does not
// depend on the schedule. Rows that do not fit go to the list `over` (first
// pass, W = 8 and CAP = 64: 99 % of the rows at 60x220x85; the second pass
// takes the list with a warp and a 1,024-entry table a row) or, past that,
// raise flags bit 0.
template <int W, int CAP, int THREADS>
__global__ void __launch_bounds__(THREADS) k_prod_rows(Prod g, const uint32_t* __restrict__ base,
                                                       uint32_t* __restrict__ ocol, double* __restrict__ oval,
                                                       uint32_t* __restrict__ olen, uint32_t* over, uint32_t* nover,
                                                       int second, int* flags) {
    constexpr int GROUPS = THREADS / W;
    __shared__ double s_val[GROUPS][CAP];
    __shared__ uint32_t s_key[GROUPS][CAP];
    __shared__ uint16_t s_list[GROUPS][CAP];
    constexpr uint32_t EMPTY = 0xffffffffu;
    const int grp = threadIdx.x / W, lane = threadIdx.x % W;
    const uint32_t mask = W == 32 ? 0xffffffffu : ((1u << (W & 31)) - 1u) << ((threadIdx.x & 31) / W * W);
    double* val = s_val[grp];
    uint32_t* key = s_key[grp];
    uint16_t* list = s_list[grp];
    const uint32_t total = second ? *nover : g.rows;
    for (uint32_t t = blockIdx.x * GROUPS + grp; t < total; t += gridDim.x * GROUPS) {
        const uint32_t q = second ? over[t] : t;
        for (int i = lane; i < CAP; i += W) {
            key[i] = EMPTY;
            val[i] = 0;
        }
        __syncwarp(mask);
        bool full = false;
        auto add = [&](uint32_t c, double v) {
            if (full) return;  // the row is lost already
            uint32_t h = (c * 2654435761u) >> 16;
            for (int p = 0; p < CAP; p++) {
                const uint32_t slot = (h + p) & (CAP - 1);
                const uint32_t k = atomicCAS(&key[slot], EMPTY, c);
                if (k == EMPTY || k == c) {
                    val[slot] += v;
                    return;
                }
            }
            full = true;
        };
        prod_terms(
            g, q,
            [&](uint32_t c, double v) {
                if (lane == 0) add(c, v);
                __syncwarp(mask);
            },
            [&](const Rows& r, uint32_t k, uint32_t shift, double v) {
                for (uint32_t j = r.b(k) + lane, e = r.e(k); j < e; j += W) add(r.col[j] + shift, v * r.val[j]);
                __syncwarp(mask);
            },
            [&](uint32_t k, uint32_t shift, double v) {
                for (uint32_t j = lane; j < g.cn; j += W) add(j + shift, v * g.C[(size_t)k * g.cn + j]);
                __syncwarp(mask);
            });
        if (__any_sync(mask, full)) {
            if (lane == 0) {
                olen[q] = 0;
                if (second) atomicOr(flags, 1);
                else over[atomicAdd(nover, 1u)] = q;
            }
            __syncwarp(mask);
            continue;
        }
        // the occupied slots, then each entry's rank by column
        uint32_t n = 0;
        for (int i = lane; i < CAP; i += W) {
            const bool occ = key[i] != EMPTY;
            const uint32_t b = __ballot_sync(mask, occ) & mask;
            if (occ) list[n + __popc(b & ((1u << (threadIdx.x & 31)) - 1u))] = (uint16_t)i;
            n += __popc(b);
        }
        __syncwarp(mask);
        const uint32_t o = base[q];
        for (uint32_t i = lane; i < n; i += W) {
            const uint32_t c = key[list[i]];
            uint32_t rank = 0;
            for (uint32_t u = 0; u < n; u++) rank += key[list[u]] < c;
            ocol[o + rank] = c;
            oval[o + rank] = val[list[i]];
        }
        if (lane == 0) olen[q] = n;
        __syncwarp(mask);
    }
}

// Length class of every row (ClassedRows); len2: the row without its columns in
// [c0, c1), whose rows are class 0.
__global__ void k_row_class(uint32_t n, Rows in, uint32_t c0, uint32_t c1, uint8_t* __restrict__ cls,
                            uint32_t* __restrict__ len2) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    uint32_t l = in.e(q) - in.b(q);
    bool dense = false;
    if (c1 > c0) {
        uint32_t k = 0;
        for (uint32_t j = in.b(q), e = in.e(q); j < e; j++) k += in.col[j] >= c0 && in.col[j] < c1;
        dense = k != 0;
        l -= k;
    }
    len2[q] = l;
    cls[q] = dense ? 0 : l > 32 ? 1 : l > 16 ? 2 : l > 8 ? 3 : l > 4 ? 4 : 5;
}
__global__ void k_len_by_row(uint32_t n, const uint32_t* __restrict__ row, const uint32_t* __restrict__ len,
                             uint32_t* __restrict__ out) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n) out[p] = len[row[p]];
}

// Copies padded rows, without their columns in [c0, c1), to their places in
// class order, eight lanes a row (columns are sorted, so the others keep
// their order).
template <class V>
__global__ void k_prod_compact(uint32_t rows, Rows in, uint32_t c0, uint32_t c1, const uint32_t* __restrict__ row,
                               const uint32_t* __restrict__ ia, uint32_t* __restrict__ ja, V* __restrict__ a) {
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t p = gid / 8, lane = gid % 8;
    if (p >= rows) return;
    const uint32_t q = row[p], o = ia[p], b = in.b(q), n = in.e(q) - b;
    const uint32_t cut = n - (ia[p + 1] - o);  // columns left out
    for (uint32_t t = lane; t < n; t += 8) {
        const uint32_t c = in.col[b + t];
        if (c1 > c0 && c >= c0 && c < c1) continue;
        const uint32_t u = o + t - (c1 > c0 && c >= c1 ? cut : 0);
        ja[u] = c;
        a[u] = (V)in.val[b + t];
    }
}

// Dense part of the class-0 rows: row i of D = sum over the row's columns c in
// [c0, c0 + cn) of value * row c - c0 of C.
__global__ void k_dense_part(uint32_t nd, const uint32_t* __restrict__ row, Rows in, uint32_t c0, uint32_t cn,
                             const double* __restrict__ C, double* __restrict__ D) {
    const uint32_t i = blockIdx.x;
    if (i >= nd) return;
    const uint32_t q = row[i], b = in.b(q), e = in.e(q);
    for (uint32_t t = threadIdx.x; t < cn; t += blockDim.x) {
        double s = 0;
        for (uint32_t j = b; j < e; j++) {
            const uint32_t c = in.col[j];
            if (c >= c0 && c < c0 + cn) s += in.val[j] * C[(size_t)(c - c0) * cn + t];
        }
        D[(size_t)i * cn + t] = s;
    }
}

// A product in padded form (scratch of the build): row q has room for its
// number of products from base[q] on and holds len[q] entries.
struct Padded {
    Tmp<uint32_t> base, len, col;
    Tmp<double> val;
    Rows view() const { return Rows{base.p, len.p, col.p, val.p}; }
};

Rows csr(const DCSR& m) { return Rows{m.ia.p, nullptr, m.ja.p, m.a.p}; }

struct Builder {
    cudaStream_t s;
    bool fp32;
    static constexpr size_t ROUND_MAX = 4;
    Tmp<int> flags;
    Tmp<unsigned long long> sums;
    Builder(cudaStream_t stream, bool single) : s(stream), fp32(single), flags(1), sums(ROUND_MAX) {
        flags.zero(s);
        sums.zero(s);
    }
    // entries of one product's scratch: 2 GB of columns and values
    static constexpr uint64_t MAX_PRODUCTS = ((uint64_t)1 << 31) / 12;

    // A round of products: measure() each, then one run() for all of them.
    std::vector<std::pair<Prod, Padded*>> due;
    void measure(const Prod& g, Padded& out) {
        unsigned long long* sum = sums.p + due.size();
        due.emplace_back(g, &out);
        out.base.alloc((size_t)g.rows + 1);
        out.len.alloc((size_t)g.rows + 1);
        k_prod_bound<<<grid_for(g.rows, 256), 256, 0, s>>>(g, out.len.p, sum);
        CK_LAUNCH();
        exclusive_scan_u32_async(out.len.p, out.base.p, g.rows, s);
    }
    // Computes them; one host synchronisation, for the sizes. False when one is
    // too large.
    bool run() {
        unsigned long long h[ROUND_MAX];
        CK(cudaMemcpyAsync(h, sums.p, due.size() * sizeof(h[0]), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        sums.zero(s);
        for (size_t i = 0; i < due.size(); i++) {
            if (h[i] > MAX_PRODUCTS) return false;
            due[i].second->col.alloc(h[i] + 1);
            due[i].second->val.alloc(h[i] + 1);
            compute(due[i].first, *due[i].second);
        }
        due.clear();
        return true;
    }
    void compute(const Prod& g, Padded& out) {
        Tmp<uint32_t> over(g.rows + 1), nover(1);
        nover.zero(s);
        constexpr int W1 = 8, T1 = 256, W2 = 32, T2 = 64;
        k_prod_rows<W1, 64, T1><<<grid_for((size_t)g.rows * W1, T1), T1, 0, s>>>(
            g, out.base.p, out.col.p, out.val.p, out.len.p, over.p, nover.p, 0, flags.p);
        CK_LAUNCH();
        k_prod_rows<W2, STATE_ROW_MAX, T2><<<(unsigned)num_sms() * 6, T2, 0, s>>>(
            g, out.base.p, out.col.p, out.val.p, out.len.p, over.p, nover.p, 1, flags.p);
        CK_LAUNCH();
    }

    // A product on its way into length classes (FP32 values: rounded once).
    // Columns [c0, c0 + cn) leave the rows for the dense part.
    struct Sorting {
        Rows in;
        uint32_t rows;
        ClassedRows* out;
        uint32_t c0 = 0, cn = 0;
        Tmp<uint8_t> cls;
        Tmp<uint32_t> len2, len;
        uint32_t* info = nullptr;  // device: the classes' first positions, the entries
    };
    static constexpr int INFO = ROW_CLASSES + 2;
    void sort(Sorting& t) {
        const uint32_t n = t.rows;
        t.cls.alloc(n + 1);
        t.len2.alloc((size_t)n + 1);
        t.len.alloc((size_t)n + 1);
        t.out->row.alloc((size_t)n + 1);
        t.out->m.ia.alloc((size_t)n + 1);
        k_row_class<<<grid_for(n, 256), 256, 0, s>>>(n, t.in, t.c0, t.c0 + t.cn, t.cls.p, t.len2.p);
        CK_LAUNCH();
        stable_partition_async(n, t.cls.p, ROW_CLASSES, t.out->row.p, t.info, s);
        k_len_by_row<<<grid_for(n, 256), 256, 0, s>>>(n, t.out->row.p, t.len2.p, t.len.p);
        CK_LAUNCH();
        exclusive_scan_u32_async(t.len.p, t.out->m.ia.p, n, s);
        CK(cudaMemcpyAsync(t.info + INFO - 1, t.out->m.ia.p + n, 4, cudaMemcpyDeviceToDevice, s));
    }
    // The sorted products' sizes and the flags (one host synchronisation).
    int sizes(std::vector<Sorting>& ts, const Tmp<uint32_t>& info) {
        std::vector<uint32_t> h(ts.size() * INFO);
        int fl = 0;
        CK(cudaMemcpyAsync(h.data(), info.p, 4 * h.size(), cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(&fl, flags.p, 4, cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        for (size_t i = 0; i < ts.size(); i++) {
            std::copy_n(h.data() + i * INFO, ROW_CLASSES + 1, ts[i].out->first);
            ts[i].out->m.nnz = h[i * INFO + INFO - 1];
        }
        return fl;
    }
    void store(const Sorting& t, const double* C) {
        ClassedRows& out = *t.out;
        DCSR& m = out.m;
        const uint32_t n = t.rows, c1 = t.c0 + t.cn;
        m.nrow = m.ncol = n;
        const size_t nz = m.nnz ? m.nnz : 1;
        m.ja.alloc(nz);
        if (fp32) m.a32.alloc(nz);
        else m.a.alloc(nz);
        if (n && m.nnz) {
            const unsigned g = grid_for((size_t)n * 8, 256);
            if (fp32) k_prod_compact<float><<<g, 256, 0, s>>>(n, t.in, t.c0, c1, out.row.p, m.ia.p, m.ja.p, m.a32.p);
            else k_prod_compact<double><<<g, 256, 0, s>>>(n, t.in, t.c0, c1, out.row.p, m.ia.p, m.ja.p, m.a.p);
            CK_LAUNCH();
        }
        out.dn = t.cn;
        const uint32_t nd = out.first[1];
        if (t.cn) {
            out.D.alloc((size_t)(nd ? nd : 1) * t.cn);
            if (nd) {
                k_dense_part<<<nd, 256, 0, s>>>(nd, out.row.p, t.in, t.c0, t.cn, C, out.D.p);
                CK_LAUNCH();
            }
        }
    }
};

}  // namespace

std::unique_ptr<StateOps> build_state(const Hierarchy& H, uint32_t m, const double* C, uint32_t cn, bool fp32,
                                      cudaStream_t s) {
    auto S = std::unique_ptr<StateOps>(new StateOps());
    S->m = m;
    S->whole = C && cn <= ABSORB_WHOLE && !fp32;
    S->absorbed = S->whole;
    S->K.resize(m);
    Builder B(s, fp32);
    // From the deepest level up. A product needs its operands' sizes, so the
    // host waits for every one's before it can be stored; the rounds below take
    // P and G of level l with Q of level l + 1 and K of level l + 2, m + 3
    // waits in place of one per product.
    std::vector<Padded> P(m + 1), G(m + 1), Q(m + 1), K(m + 1);
    auto prod = [&](uint32_t l) {
        const Level& L = *H.lv[l];
        Prod g{};
        g.M = L.M;
        g.R = L.N - L.Md;
        g.N = L.N;
        g.chained = l < m;
        if (g.chained) {
            const Level& Ln = *H.lv[l + 1];
            g.M2 = Ln.M;
            g.R2 = Ln.N - Ln.Md;
            g.theta2 = H.kind == PREC_CHEB ? Ln.beta : 1.0;
        }
        g.theta = H.kind == PREC_CHEB ? L.beta : 1.0;
        g.C = !g.chained && S->whole ? C : nullptr;
        g.cn = cn;
        g.dval = L.dval.p;
        g.phi = L.phi.p;
        g.iphi = L.iphi.p;
        return g;
    };
    auto p_rows = [&](uint32_t l) { return l < m ? P[l].view() : csr(H.lv[l]->P1); };  // the last one's are P1's
    auto prod_p = [&](uint32_t l) {
        Prod g = prod(l);
        g.mode = PM_P;
        g.rows = g.R;
        g.left = p_rows(l + 1);
        g.right = csr(H.lv[l]->P1);
        return g;
    };
    auto prod_g = [&](uint32_t l) {
        Prod g = prod(l);
        g.mode = PM_G;
        g.rows = l ? g.N : g.R;  // level 0's D rows are applied by the first launch
        g.left = csr(H.lv[l]->G);
        if (g.chained) g.right = G[l + 1].view();
        return g;
    };
    auto prod_q = [&](uint32_t l) {
        const Level& L = *H.lv[l];
        Prod g = prod(l);
        g.mode = PM_Q;
        g.rows = g.N;
        g.left = Rows{L.A.ia.p, nullptr, L.A.ja.p, L.dropped.p};
        g.right = G[l].view();
        return g;
    };
    auto prod_k = [&](uint32_t l) {
        Prod g = prod(l);
        g.mode = PM_K;
        g.rows = g.N;
        g.left = p_rows(l);
        g.right = Q[l].view();
        // the coarse block: the next level's matrix, or its system's operator
        if (g.chained) g.extra = K[l + 1].view();
        else if (H.lv[l]->n) g.extra = csr(H.lv[l + 1]->Af);
        return g;
    };
    const int top = (int)m;
    for (int l = top; l >= -1; l--) {
        if (l >= 0 && l < top) B.measure(prod_p(l), P[l]);
        if (l >= 0) B.measure(prod_g(l), G[l]);
        if (l + 1 > 0 && l + 1 <= top) B.measure(prod_q(l + 1), Q[l + 1]);
        if (l + 2 > 0 && l + 2 <= top) B.measure(prod_k(l + 2), K[l + 2]);
        if (!B.due.empty() && !B.run()) return nullptr;
    }
    // into length classes
    const uint32_t R0 = H.lv[0]->N - H.lv[0]->Md;
    std::vector<Builder::Sorting> sort(m + 2);
    Tmp<uint32_t> info(sort.size() * Builder::INFO);
    for (uint32_t j = 0; j < m + 2; j++) {
        Builder::Sorting& t = sort[j];
        t.in = j == 0 ? p_rows(0) : j == 1 ? G[0].view() : K[j - 1].view();
        t.rows = j < 2 ? R0 : H.lv[j - 1]->N;
        t.out = j == 0 ? &S->P : j == 1 ? &S->G : &S->K[j - 2];
        if (j == m + 1 && C && !S->whole && cn <= ABSORB_DENSE_N) {  // K_m, or G where there is no system
            t.c0 = H.lv[m]->M;
            t.cn = cn;
        }
        t.info = info.p + (size_t)j * Builder::INFO;
        B.sort(t);
    }
    int fl = B.sizes(sort, info);
    Builder::Sorting& last = sort[m + 1];
    if (last.cn && (size_t)last.out->first[1] * cn * sizeof(double) > ABSORB_DENSE) {
        last.cn = 0;
        B.sort(last);
        fl |= B.sizes(sort, info);
    }
    if (fl) return nullptr;
    for (Builder::Sorting& t : sort) B.store(t, C);
    if (last.cn) S->absorbed = true;
    trace("composed sweep operators");
    return S;
}

// T = I - As Y, a block per row of As.
__global__ void k_dense_residual(uint32_t n, const uint32_t* __restrict__ ia, const uint32_t* __restrict__ ja,
                                 const double* __restrict__ a, const double* __restrict__ Y, double* __restrict__ T) {
    const uint32_t i = blockIdx.x;
    for (uint32_t c = threadIdx.x; c < n; c += blockDim.x) {
        double s = i == c ? 1.0 : 0.0;
        for (uint32_t j = ia[i]; j < ia[i + 1]; j++) s -= a[j] * Y[(size_t)ja[j] * n + c];
        T[(size_t)i * n + c] = s;
    }
}
__global__ void k_dense_scale(size_t n, const double* __restrict__ B, double a, double* __restrict__ Y) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) Y[i] = a * B[i];
}
// Out = al B T + c1 Y1 + c0 Y0 (Y0 may be null, or Out): 64 x 64 of Out a block
// of 256 threads, 4 x 4 a thread, through slabs of 16 columns of B. A contraction
// of 1,073^3 in FP64, kept in FP64 on the FP64 units (three of them: about a millisecond of the set-up).
constexpr int DG_T = 64, DG_K = 16;
__global__ void __launch_bounds__(256) k_dense_gemm(uint32_t n, const double* __restrict__ B,
                                                    const double* __restrict__ T, double al, const double* Y1, double c1,
                                                    const double* Y0, double c0, double* Out) {
    __shared__ double sb[DG_K][DG_T + 1], st[DG_K][DG_T];
    const uint32_t i0 = blockIdx.y * DG_T, j0 = blockIdx.x * DG_T;
    const uint32_t tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    double acc[4][4] = {};
    for (uint32_t k0 = 0; k0 < n; k0 += DG_K) {
        for (uint32_t t = threadIdx.x; t < DG_K * DG_T; t += 256) {
            const uint32_t bi = t / DG_K, bk = t % DG_K, tk = t / DG_T, tj = t % DG_T;
            sb[bk][bi] = i0 + bi < n && k0 + bk < n ? B[(size_t)(i0 + bi) * n + k0 + bk] : 0.0;
            st[tk][tj] = k0 + tk < n && j0 + tj < n ? T[(size_t)(k0 + tk) * n + j0 + tj] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < DG_K; k++) {
            double x[4], y[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                x[u] = sb[k][ty + 16 * u];
                y[u] = st[k][tx + 16 * u];
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int v = 0; v < 4; v++) acc[u][v] = fma(x[u], y[v], acc[u][v]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) {
            const uint32_t i = i0 + ty + 16 * u, j = j0 + tx + 16 * v;
            if (i >= n || j >= n) continue;
            const size_t at = (size_t)i * n + j;
            double r = al * acc[u][v] + c1 * Y1[at];
            if (Y0) r += c0 * Y0[at];
            Out[at] = r;
        }
}

void tabulate_cheb(const DCSR& As, const double* B, uint32_t n, uint32_t steps, double lmin, double lmax,
                   DBuf<double>& out, cudaStream_t s) {
    const size_t nn = (size_t)n * n;
    const double eta = (lmax + lmin) / (lmax - lmin), a1 = 2 / (lmax + lmin);
    const dim3 grid((n + DG_T - 1) / DG_T, (n + DG_T - 1) / DG_T);
    Tmp<double> t(nn), y(nn);
    out.alloc(nn);
    // the iterates alternate between out and y, the last one in out
    double *cur = steps & 1 ? out.p : y.p, *other = steps & 1 ? y.p : out.p;
    k_dense_scale<<<grid_for(nn, 256), 256, 0, s>>>(nn, B, a1, cur);
    CK_LAUNCH();
    for (uint32_t i = 2; i <= steps; i++) {
        const double al = 4 / (lmax - lmin) * cheb_poly(eta, i - 1) / cheb_poly(eta, i);
        const double be = cheb_poly(eta, i - 2) / cheb_poly(eta, i);
        k_dense_residual<<<n, 256, 0, s>>>(n, As.ia.p, As.ja.p, As.a.p, cur, t.p);
        CK_LAUNCH();
        // x2 = u1 + al B (F - As u1) + be (u1 - u0); u0 = 0 in step 2
        k_dense_gemm<<<grid, 256, 0, s>>>(n, B, t.p, al, cur, 1 + be, i > 2 ? other : nullptr, -be, other);
        CK_LAUNCH();
        std::swap(cur, other);
    }
}

}  // namespace mlp
