// qmb_expval.cu -- zero-temperature expectation values <psi|A|psi> in a
// symmetry-adapted sector, for operators that are sums of products of Sz, S+
// and S-.  This is the computation of ComputeStaticExpValZeroT
// (exact_diagonalization/HeisenbergGenericXXZ_AbelianSymms_CUDA.cu:421-601,
// exact_diagonalization/HeisenbergHamAbelianSymms_CUDA.cu:448-617) and of its
// kernel ExpecValArbOperatorAbelianIrrepProjHeisenbergZeroT
// (exact_diagonalization/utils.cu:442-550) with its thrust reduction.
//
// Method.  psi lies in a one-dimensional irrep of the sector's group, so
// <psi|A|psi> = <psi|U_e^-1 A U_e|psi> for every element e, and A can be
// replaced by its group average Abar = (1/n_ext) sum_e U_e^-1 A U_e (site
// maps, and Sz -> -Sz, S+ <-> S- for the spin-inversion elements).  Abar
// commutes with the group, so its matrix on the symmetric basis follows from
// its action on the representatives alone: the rule of the Hamiltonian
// (gen_row_range).  One pass over the rows then gives
//     s = sum_r conj(psi_r) (Abar psi)_r,
// and with operator tables in the Hamiltonian's convention (each term the
// daggered operator sequence with a conjugated scalar, as BuildOperatorVecs
// writes it) the expectation value is conj(s) / <psi|psi>.
//
// The reference applies the operator to every member of every orbit (|G|
// applications per term and row) and finds the target orbit through a table
// over the whole Sz sector.  Here each row applies averaged terms to its
// representative only, and a term is evaluated once however many operators hold
// it: <psi|T|psi> is the same for all images of T under the group (up to the
// sign of an odd number of Sz under inversion), so the terms of all operators
// are sorted into classes, one value per class is computed on the device, and an
// operator is the sum of its scalars times its classes' values.  The structure
// factor at all 24 momenta of a 24-site chain with the 24 correlators has 13,848
// terms in 13 classes.  Terms that change Sz are dropped (zero expectation in a
// fixed-Sz sector).
//
// Products of Sz are signs: a class's value is a sum over its distinct images m
// of Q(m) = sum_r |psi_r|^2 (-1)^popc(m & down_r), and k_ev_diag computes all Q
// in one launch.  Other classes go through the Hamiltonian's row rule, their
// averaged terms back to back in shared memory, in segments that are reduced
// separately: one per class that several operators hold, and one per operator for
// the classes that it alone holds (gen_terms).
#include <algorithm>
#include <chrono>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <unordered_map>
#include <vector>

#include "qmb_ham.cuh"
#include "qmb_b200.h"

namespace qmb {
namespace {

constexpr int kEvBlock = 256;
constexpr size_t kEvSmemCap = 200 * 1024;  // dynamic shared memory per block
constexpr int64_t kEvSlab = (int64_t)1 << 23;     // rows of one pass of the sign sums
constexpr int64_t kEvSlabMin = (int64_t)1 << 16;  // the fewest, where memory is short

using cplx = std::complex<double>;

// A product of operators: up to 8 words code << 8 | site in application order.
struct TermKey {
    uint64_t a = 0, b = 0;
    int n = 0;
    bool operator==(const TermKey& o) const { return a == o.a && b == o.b && n == o.n; }
};
struct TermKeyHash {
    size_t operator()(const TermKey& k) const {
        uint64_t h = k.a * 0x9E3779B97F4A7C15ull ^ (k.b + 0x632BE59BD9B4E019ull + (uint64_t)k.n) * 0xC2B2AE3D27D4EB4Full;
        return (size_t)(h ^ (h >> 29));
    }
};
TermKey make_key(const uint16_t* w, int n) {
    TermKey k;
    k.n = n;
    for (int i = 0; i < n; ++i) (i < 4 ? k.a : k.b) |= (uint64_t)w[i] << (16 * (i & 3));
    return k;
}
void key_words(const TermKey& k, uint16_t* w) {
    for (int i = 0; i < k.n; ++i) w[i] = (uint16_t)((i < 4 ? k.a : k.b) >> (16 * (i & 3)));
}

// The classes of the operators' terms.
struct Classes {
    const qmb_sector_s* s;
    int n = 0;                                  // classes
    // products of Sz, by the XOR of their sites (a site taken twice is 1/4, no sign)
    std::unordered_map<uint64_t, int> of_mask;
    std::vector<int> pair_class;                // [L][L] classes of masks of one or two sites, -1: not seen
    std::vector<uint64_t> masks;                // images of all diagonal classes
    std::vector<double> mask_w;                 // elements reaching them (weight = that / G)
    std::vector<int> mask_class;
    // other terms
    struct At {
        int cls;
        double sign;
    };
    std::unordered_map<TermKey, At, TermKeyHash> of_key;
    std::vector<TermKey> gen_key;               // averaged terms, class by class
    std::vector<double> gen_w;                  // signed elements reaching them (weight = that / n_ext)
    std::unordered_map<int, std::pair<size_t, size_t>> gen_range;  // class -> its terms

    explicit Classes(const qmb_sector_s* sec) : s(sec), pair_class(sec->L * sec->L, -1) {}

    // Class of a product of Sz, or -1 where the average vanishes.
    int diag_class(uint64_t m) {
        const auto it = of_mask.find(m);
        if (it != of_mask.end()) return it->second;
        const bool zero = s->flip && (__builtin_popcountll(m) & 1);  // inversion takes it to its negative
        const int c = zero ? -1 : n++;
        const size_t first = masks.size();
        for (int g = 0; g < s->G; ++g) {
            const uint32_t* p = s->perm.data() + (size_t)g * s->L;
            uint64_t y = 0;
            for (uint64_t b = m; b; b &= b - 1) y |= 1ull << p[__builtin_ctzll(b)];
            if (of_mask.emplace(y, c).second) {
                if (zero) continue;
                masks.push_back(y);
                mask_w.push_back(1.0);
                mask_class.push_back(c);
            } else if (!zero) {
                for (size_t k = first; k < masks.size(); ++k)
                    if (masks[k] == y) mask_w[k] += 1.0;
            }
        }
        of_mask.emplace(m, c);  // (among its images already when the group has the identity)
        return c;
    }

    // Class of a term with S+ and S-, and the sign of its value.
    At gen_class_of(const uint16_t* w, int nw, int n_z) {
        uint16_t img[kMaxCol];
        auto image = [&](int e) {
            const uint32_t* p = s->perm.data() + (size_t)(e % s->G) * s->L;
            const bool z = e >= s->G;
            for (int j = 0; j < nw; ++j) {
                int c = w[j] >> 8;
                if (z && c != QMB_OP_SZ) c = c == QMB_OP_SP ? QMB_OP_SM : QMB_OP_SP;
                img[j] = (uint16_t)(c << 8 | (int)p[w[j] & 0xff]);
            }
            // factors on distinct sites commute: order them by site
            bool distinct = true;
            for (int a = 0; a < nw && distinct; ++a)
                for (int b = a + 1; b < nw; ++b)
                    if ((img[a] & 0xff) == (img[b] & 0xff)) {
                        distinct = false;
                        break;
                    }
            if (distinct)
                std::sort(img, img + nw, [](uint16_t x, uint16_t y) { return (x & 0xff) < (y & 0xff); });
            return make_key(img, nw);
        };
        // (element 0 may be any element: look the term itself up in image order)
        const TermKey k0 = image(0);
        const auto it = of_key.find(k0);
        if (it != of_key.end()) return it->second;
        const int c = n++;
        const size_t first = gen_key.size();
        for (int e = 0; e < s->n_ext; ++e) {
            const TermKey k = image(e);
            const double sign = (e >= s->G && (n_z & 1)) ? -1.0 : 1.0;
            if (of_key.emplace(k, At{c, sign}).second) {
                gen_key.push_back(k);
                gen_w.push_back(sign);
            } else {
                for (size_t q = first; q < gen_key.size(); ++q)
                    if (gen_key[q] == k) gen_w[q] += sign;
            }
        }
        gen_range.emplace(c, std::make_pair(first, gen_key.size()));
        return of_key.find(k0)->second;
    }
};

// An averaged term of the general kernel and the value that its sum goes to.
struct GenTerm {
    int target;  // a class, or cls.n + operator
    size_t key;
    cplx sc;
};

// What the general kernel evaluates: a class that one operator alone holds goes, with
// the operator's scalar, into the one sum of that operator, so that a row's data are
// read once for all of them; a class that several operators hold is a sum of its
// own, evaluated once.  Without a group (184,756 rows) the 80 classes of a J1-J2
// Hamiltonian take 0.30 ms, as sums of their own 0.40; eight operators of 300 distinct
// four-site terms 7.9 against 12.1.
std::vector<GenTerm> gen_terms(const Classes& cls, const std::vector<std::vector<std::pair<int, cplx>>>& terms) {
    std::vector<GenTerm> out;
    if (cls.gen_key.empty()) return out;
    std::vector<int> users(cls.n, 0);
    for (const auto& op : terms)
        for (const auto& t : op) ++users[t.first];
    out.reserve(cls.gen_key.size());
    auto add = [&](int target, int c, cplx s) {
        const auto& r = cls.gen_range.at(c);
        for (size_t i = r.first; i < r.second; ++i)
            if (cls.gen_w[i] != 0.0) out.push_back(GenTerm{target, i, s * (cls.gen_w[i] / cls.s->n_ext)});
    };
    for (size_t k = 0; k < terms.size(); ++k)
        for (const auto& t : terms[k])
            if (users[t.first] == 1 && cls.gen_range.count(t.first)) add(cls.n + (int)k, t.first, t.second);
    for (int c = 0; c < cls.n; ++c)
        if (users[c] > 1 && cls.gen_range.count(c)) add(c, c, 1.0);
    return out;
}

// Adds the terms of one operator: (class, scalar) pairs, one per class.
void sort_terms(const qmb_terms& A, Classes& cls, std::vector<int>& last_op, std::vector<size_t>& last_at, int op,
                std::vector<std::pair<int, cplx>>& out) {
    QMB_REQUIRE(A.n_terms >= 0, QMB_ERR_INVALID, "expval: n_terms must be >= 0");
    if (A.n_terms == 0) return;
    QMB_REQUIRE(A.n_ops && A.op_code && A.op_site && A.scalar, QMB_ERR_INVALID,
                "expval: null table");
    QMB_REQUIRE(A.n_col >= 1 && A.n_col <= kMaxCol, QMB_ERR_INVALID, "expval: n_col must be in 1..8");
    const int L = cls.s->L;
    auto add = [&](int c, cplx v) {
        if (c < 0) return;
        if ((int)last_op.size() < cls.n) {
            last_op.resize(2 * cls.n + 16, -1);
            last_at.resize(last_op.size(), 0);
        }
        if (last_op[c] != op) {
            last_op[c] = op;
            last_at[c] = out.size();
            out.emplace_back(c, v);
        } else {
            out[last_at[c]].second += v;
        }
    };
    for (int i = 0; i < A.n_terms; ++i) {
        const int no = A.n_ops[i];
        QMB_REQUIRE(no >= 0 && no <= A.n_col, QMB_ERR_INVALID, "expval: n_ops out of range");
        const cplx sc(A.scalar[2 * i], A.scalar[2 * i + 1]);
        QMB_REQUIRE(std::isfinite(sc.real()) && std::isfinite(sc.imag()), QMB_ERR_INVALID,
                    "expval: non-finite scalar");
        const int *code = A.op_code + (size_t)i * A.n_col, *site = A.op_site + (size_t)i * A.n_col;
        uint16_t w[kMaxCol];
        int nb = 0, n_p = 0, n_m = 0, n_z = 0;
        uint64_t m = 0;
        double f = 1.0;
        for (int j = 0; j < no; ++j) {
            const int c = code[j], q = site[j];
            QMB_REQUIRE(c == QMB_OP_SZ || c == QMB_OP_SP || c == QMB_OP_SM || c == QMB_OP_I,
                        QMB_ERR_INVALID, "expval: operator codes must be Sz, Sp, Sm or I");
            QMB_REQUIRE(q >= 0 && q < L, QMB_ERR_INVALID, "expval: site out of range");
            if (c == QMB_OP_I) continue;
            n_p += c == QMB_OP_SP;
            n_m += c == QMB_OP_SM;
            if (c == QMB_OP_SZ) {
                ++n_z;
                m ^= 1ull << q;
                f *= 0.5;
            }
            w[nb++] = (uint16_t)(c << 8 | q);
        }
        if (n_p != n_m || sc == 0.0) continue;  // leaves the Sz sector, or zero
        if (n_p == 0) {
            if (nb == 2 && m) {  // two sites, the common product: no hash lookup
                int& pc = cls.pair_class[(w[0] & 0xff) * L + (w[1] & 0xff)];
                if (pc == -1) pc = cls.diag_class(m) + 1 ? cls.diag_class(m) : -2;
                add(pc, sc * f);
            } else {
                add(cls.diag_class(m), sc * f);
            }
        } else {
            const Classes::At at = cls.gen_class_of(w, nb, n_z);
            add(at.cls, sc * at.sign);
        }
    }
}

bool trace_on() {
    static int v = -1;
    if (v < 0) {
        const char* e = std::getenv("QMB_TRACE");
        v = (e && *e && *e != '0') ? 1 : 0;
    }
    return v == 1;
}

__device__ __forceinline__ double2 block_sum2(double x, double y, double2* red) {
    for (int o = 16; o; o >>= 1) {
        x += __shfl_down_sync(0xffffffffu, x, o);
        y += __shfl_down_sync(0xffffffffu, y, o);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = make_double2(x, y);
    __syncthreads();
    double2 t = make_double2(0.0, 0.0);
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
            t.x += red[i].x;
            t.y += red[i].y;
        }
    return t;
}

// Rows r0 .. r0 + n - 1 for the sign sums: down_r, the string's down spins, and
// |psi_r|^2, with the block partials of <psi|psi> added to npart.
template <class V>
__global__ void __launch_bounds__(kEvBlock) k_ev_rows(RowGen rg, int64_t r0, int64_t n, const V* __restrict__ psi,
                                                      uint64_t* __restrict__ down64, uint32_t* __restrict__ down32,
                                                      double* __restrict__ p2, double* __restrict__ npart) {
    extern __shared__ __align__(16) unsigned char smem_er[];
    __shared__ double2 red[kEvBlock / 32];
    const GroupSmem gs = load_group(rg.g, smem_er);
    double nn = 0.0;
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
        const double p = Sc<V>::abs2(psi[r0 + r]);
        nn += p;
        if (p2) {
            const uint64_t d = ~apply_elem(rg.g, gs, 0, rg.rt.reps[rg.orbit_of_row[r0 + r]]);
            p2[r] = p;
            if (down32) down32[r] = (uint32_t)d;
            else down64[r] = d;
        }
    }
    const double2 t = block_sum2(nn, 0.0, red);
    if (threadIdx.x == 0) npart[blockIdx.x] += t.x;
}

// part[chunk][m] = sum over the chunk's rows of p2_r (-1)^popc(mask_m & down_r).
// A warp takes 8 masks over one chunk of rows, lanes over rows, so that a row's
// 12 bytes serve 8 masks from registers: an AND, a population count, a sign flip
// (the parity moved to the sign bit) and an FP64 addition each.  13 classes of a
// 24-site chain are 300 masks over 112,720 rows: all values with their copies take
// 75 us (640 us for one kernel over the 7,764 averaged terms of the operators).
// The population counts bound it (16 a cycle and SM).
constexpr int kEvMasks = 8;
template <class U>
__global__ void __launch_bounds__(kEvBlock) k_ev_diag(int64_t n, const U* __restrict__ down,
                                                      const double* __restrict__ p2, const U* __restrict__ mask,
                                                      int n_mask, int n_groups, int n_chunks, int64_t chunk,
                                                      double* __restrict__ part) {
    const int lane = threadIdx.x & 31;
    const int item = blockIdx.x * (kEvBlock / 32) + (threadIdx.x >> 5);
    if (item >= n_groups * n_chunks) return;
    const int g = item % n_groups, c = item / n_groups, m0 = g * kEvMasks;
    U mk[kEvMasks];
    double acc[kEvMasks];
#pragma unroll
    for (int k = 0; k < kEvMasks; ++k) {
        mk[k] = m0 + k < n_mask ? mask[m0 + k] : (U)0;
        acc[k] = 0.0;
    }
    const int64_t r1 = min(n, (c + 1) * chunk);
#pragma unroll 2
    for (int64_t r = c * chunk + lane; r < r1; r += 32) {
        const U d = down[r];
        const double p = p2[r];
        const int hi = __double2hiint(p), lo = __double2loint(p);
#pragma unroll
        for (int k = 0; k < kEvMasks; ++k) {
            const int par = sizeof(U) == 8 ? __popcll((unsigned long long)(mk[k] & d)) : __popc((unsigned)(mk[k] & d));
            acc[k] += __hiloint2double(hi ^ (int)((unsigned)par << 31), lo);
        }
    }
#pragma unroll
    for (int k = 0; k < kEvMasks; ++k) {
        for (int o = 16; o; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
        if (lane == 0 && m0 + k < n_mask) part[(int64_t)c * n_mask + m0 + k] = acc[k];
    }
}

// q[m] += the chunks' part[chunk][m] by a warp a mask, the rounding of each addition
// carried along (Neumaier 1974 within a lane, Knuth's two-sum between lanes).  (One
// mask over 705,432 rows has 2,756 chunks: with one thread adding them up the call
// took 211 us, 83 this way.)
__global__ void __launch_bounds__(kEvBlock) k_ev_diag_sum(const double* __restrict__ part, int n_mask, int n_chunks,
                                                          double* __restrict__ q) {
    const int lane = threadIdx.x & 31, m = blockIdx.x * (kEvBlock / 32) + (threadIdx.x >> 5);
    if (m >= n_mask) return;
    double t = lane == 0 ? q[m] : 0.0, low = 0.0;
#pragma unroll 4
    for (int c = lane; c < n_chunks; c += 32) {
        const double v = part[(int64_t)c * n_mask + m], s = __dadd_rn(t, v);
        low += fabs(t) >= fabs(v) ? __dadd_rn(__dadd_rn(t, -s), v) : __dadd_rn(__dadd_rn(v, -s), t);
        t = s;
    }
    for (int o = 16; o; o >>= 1) {
        const double v = __shfl_xor_sync(0xffffffffu, t, o), s = __dadd_rn(t, v), b = __dadd_rn(s, -t);
        low = __dadd_rn(low, __shfl_xor_sync(0xffffffffu, low, o));
        low += __dadd_rn(__dadd_rn(t, -__dadd_rn(s, -b)), __dadd_rn(v, -b));
        t = s;
    }
    if (lane == 0) q[m] = t + low;
}

// One launch over the other terms: every block strides over the rows for each
// segment sg and writes its partial sum of conj(psi_r) (Abar_sg psi)_r to
// part[sg][block].  Segment sg holds terms seg[sg].x .. seg[sg].y - 1.
template <class V>
__global__ void __launch_bounds__(kEvBlock) k_expval(RowGen rg, int64_t n, const V* __restrict__ psi, int n_seg,
                                                     const int2* __restrict__ seg, double2* __restrict__ part) {
    extern __shared__ __align__(16) unsigned char smem_ev[];
    __shared__ double2 red[kEvBlock / 32];
    const size_t gb = align16(group_smem_bytes(rg.g));
    const GroupSmem gs = load_group(rg.g, smem_ev);
    const TermsSmem ts = load_terms(rg.terms, smem_ev + gb);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int sg = 0; sg < n_seg; ++sg) {
        const int2 sd = seg[sg];
        double ax = 0.0, ay = 0.0;
        for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += stride) {
            const int64_t o = rg.orbit_of_row[r];
            const uint64_t src = apply_elem(rg.g, gs, 0, rg.rt.reps[o]);
            // complex row sum even for a real psi: characters may be complex
            const double2 pr = Sc<V>::to2(psi[r]);
            double2 y = make_double2(0.0, 0.0);
            const double2 d = gen_row_range(rg, gs, ts, sd.x, sd.y, src, rg.norms[o], [&](int64_t ot, double2 v) {
                const double2 x = Sc<V>::to2(__ldg(psi + rg.row_of_orbit[ot]));
                y.x += v.x * x.x - v.y * x.y;
                y.y += v.x * x.y + v.y * x.x;
            });
            y.x += d.x * pr.x - d.y * pr.y;
            y.y += d.x * pr.y + d.y * pr.x;
            ax += pr.x * y.x + pr.y * y.y;  // conj(pr) * y
            ay += pr.x * y.y - pr.y * y.x;
        }
        const double2 t = block_sum2(ax, ay, red);
        if (threadIdx.x == 0) part[(size_t)sg * gridDim.x + blockIdx.x] = t;
    }
}

// Fixed-order sum of the block partials of every segment (one block each).
__global__ void __launch_bounds__(kEvBlock) k_expval_sum(const double2* __restrict__ part, int n_blocks,
                                                         double2* __restrict__ seg_out) {
    __shared__ double2 red[kEvBlock / 32];
    const double2* p = part + (size_t)blockIdx.x * n_blocks;
    double x = 0.0, y = 0.0;
    for (int i = threadIdx.x; i < n_blocks; i += blockDim.x) {
        x += p[i].x;
        y += p[i].y;
    }
    const double2 t = block_sum2(x, y, red);
    if (threadIdx.x == 0) seg_out[blockIdx.x] = t;
}

// The values of the classes, val[c] = sum_r conj(psi_r) (Tbar_c psi)_r, behind them
// the operators' own sums of general terms (gen_terms), and <psi|psi>.
template <class V>
void class_values(qmb_ham_s* h, const V* psi, const Classes& cls, const std::vector<GenTerm>& gen, int n_ops,
                  std::vector<cplx>& val, double* norm2) {
    RowGen rg = h->row_gen();
    const size_t gbytes = align16(group_smem_bytes(rg.g));
    int sms = 148, max_smem = 0;
    QMB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device));
    QMB_CUDA_TRY(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device));
    const size_t smem_cap = std::min(kEvSmemCap, (size_t)max_smem);
    QMB_REQUIRE(gbytes + 64 < smem_cap, QMB_ERR_INVALID, "expval: group tables leave no shared memory");
    val.assign(cls.n + n_ops, cplx(0.0, 0.0));
    const int64_t n = h->n;
    size_t off = 0;
    auto place = [&](size_t bytes) {
        const size_t o = off;
        off = align16(off + bytes);
        return o;
    };

    // products of Sz, and the norm
    {
        const int nm = (int)cls.masks.size(), groups = (nm + kEvMasks - 1) / kEvMasks;
        const bool small = cls.s->L <= 32;
        // rows in slabs, which bounds the scratch (12 or 16 bytes a row; smaller ones
        // where the memory is short); about 48 warps an SM, chunks of at least 256 rows
        int64_t slab = std::min<int64_t>(n, nm ? kEvSlab : n), chunk = 0;
        int chunks = 0, nblk = 0;
        const size_t us = small ? 4 : 8;
        size_t o_mask, o_q, o_norm, o_p, o_down, o_part;
        DevBuf<unsigned char> blk;
        for (;;) {
            const int64_t want = groups ? std::max<int64_t>(1, (int64_t)sms * 48 / groups) : 1;
            chunks = (int)std::min<int64_t>(want, (slab + 255) / 256);
            chunk = ((slab + chunks - 1) / chunks + 31) / 32 * 32;
            nblk = (int)std::min<int64_t>((slab + kEvBlock - 1) / kEvBlock, (int64_t)sms * 4);
            off = 0;
            o_mask = place(us * nm);
            o_q = place(sizeof(double) * nm);
            o_norm = place(sizeof(double) * nblk);
            o_p = place(nm ? sizeof(double) * slab : 0);
            o_down = place(nm ? us * slab : 0);
            o_part = place(sizeof(double) * (size_t)nm * chunks);
            try {
                blk.alloc(off);
                break;
            } catch (const Error& e) {
                if (e.code != QMB_ERR_NOMEM || slab <= kEvSlabMin) throw;
                (void)cudaGetLastError();
                slab = std::max(kEvSlabMin, slab / 2);
            }
        }
        unsigned char* b = blk.p;
        double* q = reinterpret_cast<double*>(b + o_q);
        double* npart = reinterpret_cast<double*>(b + o_norm);
        double* p2 = nm ? reinterpret_cast<double*>(b + o_p) : nullptr;
        uint32_t* d32 = small ? reinterpret_cast<uint32_t*>(b + o_down) : nullptr;
        uint64_t* d64 = reinterpret_cast<uint64_t*>(b + o_down);
        double* part = reinterpret_cast<double*>(b + o_part);
        std::vector<uint32_t> m32;
        const void* hm = cls.masks.data();
        if (small) {
            m32.assign(cls.masks.begin(), cls.masks.end());
            hm = m32.data();
        }
        if (nm) QMB_CUDA_TRY(cudaMemcpyAsync(b + o_mask, hm, us * nm, cudaMemcpyHostToDevice, 0));
        QMB_CUDA_TRY(cudaMemsetAsync(b + o_q, 0, o_norm + sizeof(double) * nblk - o_q, 0));
        set_group_smem_attr((const void*)k_ev_rows<V>, gbytes);
        for (int64_t r0 = 0; r0 < n; r0 += slab) {
            const int64_t rows = std::min(slab, n - r0);
            k_ev_rows<V><<<nblk, kEvBlock, gbytes>>>(rg, r0, rows, psi, d64, d32, p2, npart);
            check_launch("k_ev_rows");
            if (!nm) continue;
            const int grid = (groups * chunks + kEvBlock / 32 - 1) / (kEvBlock / 32);
            if (small)
                k_ev_diag<uint32_t><<<grid, kEvBlock>>>(rows, d32, p2, reinterpret_cast<const uint32_t*>(b + o_mask), nm,
                                                        groups, chunks, chunk, part);
            else
                k_ev_diag<uint64_t><<<grid, kEvBlock>>>(rows, d64, p2, reinterpret_cast<const uint64_t*>(b + o_mask), nm,
                                                        groups, chunks, chunk, part);
            check_launch("k_ev_diag");
            k_ev_diag_sum<<<(nm + kEvBlock / 32 - 1) / (kEvBlock / 32), kEvBlock>>>(part, nm, chunks, q);
            check_launch("k_ev_diag_sum");
        }
        std::vector<unsigned char> res(o_norm + sizeof(double) * nblk - o_q);
        QMB_CUDA_TRY(cudaMemcpy(res.data(), b + o_q, res.size(), cudaMemcpyDeviceToHost));
        blk.mark_idle();
        const double* hq = reinterpret_cast<const double*>(res.data());
        const double* hn = reinterpret_cast<const double*>(res.data() + (o_norm - o_q));
        std::vector<long double> sum(cls.n, 0.0L);
        for (int k = 0; k < nm; ++k) sum[cls.mask_class[k]] += (long double)cls.mask_w[k] * hq[k];
        for (int c = 0; c < cls.n; ++c) val[c] = (double)(sum[c] / cls.s->G);
        long double nn = 0.0L;
        for (int k = 0; k < nblk; ++k) nn += hn[k];
        *norm2 = (double)nn;
    }

    // the other terms, as many as fit in shared memory at a time
    const size_t n_gen = gen.size();
    if (!n_gen) return;
    DevBuf<int> err(1);
    err.zero();
    rg.err = err.p;
    for (size_t pos = 0; pos < n_gen;) {
        std::vector<int2> seg;
        std::vector<int> seg_target, nops;
        std::vector<double2> sc;
        int n_col = 1;
        size_t end = pos;
        for (; end < n_gen; ++end) {
            const size_t ng = end - pos + 1;
            const TermKey& key = cls.gen_key[gen[end].key];
            const int c = std::max(n_col, key.n);
            if (gbytes + ((20 + 2 * (size_t)c) * ng + 15) / 16 * 16 > smem_cap || ng > (size_t)kMaxTerms) break;
            n_col = c;
            if (seg.empty() || seg_target.back() != gen[end].target) {
                seg.push_back(make_int2((int)ng - 1, (int)ng - 1));
                seg_target.push_back(gen[end].target);
            }
            seg.back().y += 1;
            nops.push_back(key.n);
            sc.push_back(make_double2(gen[end].sc.real(), gen[end].sc.imag()));
        }
        QMB_REQUIRE(end > pos, QMB_ERR_INVALID, "expval: a term does not fit");
        const int ng = (int)(end - pos), n_seg = (int)seg.size();
        std::vector<uint16_t> opw((size_t)ng * n_col, 0);
        for (int i = 0; i < ng; ++i) key_words(cls.gen_key[gen[pos + i].key], opw.data() + (size_t)i * n_col);
        rg.terms.n_terms = ng;
        rg.terms.n_col = n_col;
        const size_t smem = gbytes + terms_smem_bytes(rg.terms);
        set_group_smem_attr((const void*)k_expval<V>, smem);
        int per_sm = 0;
        QMB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_expval<V>, kEvBlock, smem));
        const int grid = (int)std::max<int64_t>(
            1, std::min<int64_t>((n + kEvBlock - 1) / kEvBlock, (int64_t)sms * std::max(1, per_sm)));
        off = 0;
        const size_t o_nops = place(sizeof(int) * ng), o_ops = place(sizeof(uint16_t) * opw.size()),
                     o_sc = place(sizeof(double2) * ng), o_seg = place(sizeof(int2) * n_seg);
        const size_t in_bytes = off;
        const size_t o_res = place(sizeof(double2) * n_seg), o_part = place(sizeof(double2) * (size_t)n_seg * grid);
        std::vector<unsigned char> stage(in_bytes);
        std::memcpy(stage.data() + o_nops, nops.data(), sizeof(int) * ng);
        std::memcpy(stage.data() + o_ops, opw.data(), sizeof(uint16_t) * opw.size());
        std::memcpy(stage.data() + o_sc, sc.data(), sizeof(double2) * ng);
        std::memcpy(stage.data() + o_seg, seg.data(), sizeof(int2) * n_seg);
        DevBuf<unsigned char> blk(off);
        QMB_CUDA_TRY(cudaMemcpy(blk.p, stage.data(), in_bytes, cudaMemcpyHostToDevice));
        unsigned char* b = blk.p;
        rg.terms.n_ops = reinterpret_cast<const int*>(b + o_nops);
        rg.terms.ops = reinterpret_cast<const uint16_t*>(b + o_ops);
        rg.terms.scalar = reinterpret_cast<const double2*>(b + o_sc);
        double2* res_d = reinterpret_cast<double2*>(b + o_res);
        double2* part = reinterpret_cast<double2*>(b + o_part);
        k_expval<V><<<grid, kEvBlock, smem>>>(rg, n, psi, n_seg, reinterpret_cast<const int2*>(b + o_seg), part);
        check_launch("k_expval");
        k_expval_sum<<<n_seg, kEvBlock>>>(part, grid, res_d);
        check_launch("k_expval_sum");
        std::vector<double2> res(n_seg);
        QMB_CUDA_TRY(cudaMemcpy(res.data(), res_d, sizeof(double2) * n_seg, cudaMemcpyDeviceToHost));
        blk.mark_idle();
        for (int i = 0; i < n_seg; ++i) val[seg_target[i]] += cplx(res[i].x, res[i].y);
        pos = end;
    }
    int herr = 0;
    QMB_CUDA_TRY(cudaMemcpy(&herr, err.p, sizeof(int), cudaMemcpyDeviceToHost));
    err.mark_idle();
    QMB_REQUIRE(herr == 0, QMB_ERR_INVALID, "expval: a term left the sector's representative table");
}

}  // namespace
}  // namespace qmb

using namespace qmb;

extern "C" qmb_status qmb_expval(qmb_ham h, int n_ops, const qmb_terms* ops, const void* psi_dev,
                                 double* out) {
    return guarded([&] {
        QMB_REQUIRE(h && out && (ops || n_ops == 0), QMB_ERR_INVALID, "null argument");
        QMB_REQUIRE(n_ops >= 0, QMB_ERR_INVALID, "n_ops must be >= 0");
        QMB_REQUIRE(h->sector && h->sector->has_irrep, QMB_ERR_INVALID, "handle has no sector irrep");
        QMB_REQUIRE(h->irrep_gen == h->sector->irrep_gen, QMB_ERR_INVALID,
                    "the sector's irrep changed since the handle was built");
        const void* psi = psi_dev;
        if (!psi) {
            QMB_REQUIRE(h->psi.p && h->psi_n == h->n, QMB_ERR_INVALID,
                        "no ground state kept (run qmb_lanczos with want_vector, or qmb_set_ground_state)");
            psi = h->psi.p;
        }
        if (n_ops == 0) return;
        DeviceGuard dg(h->device);
        const auto t0 = std::chrono::steady_clock::now();
        Classes cls(h->sector);
        std::vector<std::vector<std::pair<int, cplx>>> terms(n_ops);
        std::vector<int> last_op;
        std::vector<size_t> last_at;
        for (int k = 0; k < n_ops; ++k) sort_terms(ops[k], cls, last_op, last_at, k, terms[k]);
        const auto t1 = std::chrono::steady_clock::now();
        std::vector<cplx> val;
        double norm2 = 0.0;
        const std::vector<GenTerm> gen = gen_terms(cls, terms);
        if (h->cplx) class_values<double2>(h, (const double2*)psi, cls, gen, n_ops, val, &norm2);
        else class_values<double>(h, (const double*)psi, cls, gen, n_ops, val, &norm2);
        QMB_REQUIRE(norm2 > 0.0, QMB_ERR_INVALID, "expval: psi is zero");
        for (int k = 0; k < n_ops; ++k) {
            // (operators such as S(q) cancel among their classes)
            std::complex<long double> sum(val[cls.n + k]);
            for (const auto& t : terms[k])
                sum += std::complex<long double>(t.second) * std::complex<long double>(val[t.first]);
            out[2 * k] = (double)(sum.real() / norm2);  // conj(s) / <psi|psi>
            out[2 * k + 1] = (double)(-sum.imag() / norm2);
        }
        if (trace_on()) {
            size_t nt = 0;
            for (int k = 0; k < n_ops; ++k) nt += (size_t)ops[k].n_terms;
            const auto t2 = std::chrono::steady_clock::now();
            std::fprintf(stderr, "[qmb expval] %d operators, %zu terms in %d classes: sorting %.3f ms, values %.3f ms\n",
                         n_ops, nt, cls.n, std::chrono::duration<double, std::milli>(t1 - t0).count(),
                         std::chrono::duration<double, std::milli>(t2 - t1).count());
        }
    });
}
