// The FP64 per-cell passes of designs without few distinct rows: bread /
// per-cluster score sums (src/variance.cpp:22-47, :207-217; PassSandwich of
// passes.cuh) above eight columns, and from three where the size gives blocks
// enough (cell64_pays), and MOM moments above eight (src/mom_overdispersion.cpp:
// 34-45; PassMOM, mom_cells_kernel below).
//
// Bread, per gene and cell: eta = off + x . beta, mu = exp(eta), the weight; then
// sum_c w_gc x_ci x_cj for every i <= j: a contraction of the weights (genes x
// cells) with the products z (cells x p (p + 1) / 2).  Both run on the FP64
// matrix instruction (mma.m8n8k4): eta of 8 genes x 8 cells, and 16 genes x 8
// products per warp and step, so an operand element is fetched once per 8 or 16
// multiply-adds instead of once per two.
//
// Block = 32 genes x one run of cells, 256 threads, chunks of 32 cells: the
// chunk's design rows by cp.async one chunk ahead, the genes' nonzero counts
// scattered into a 32 x 32 tile (eight lanes per gene, their entries loaded one
// chunk ahead), eta by warps (8 genes x 16 cells each), the weights through
// shared memory, then each warp adds its share of the (16 genes, 8 products)
// units with the accumulators in registers (136 products: 5 units a warp; 528:
// 17).  The products are formed at the fetch (two reads and one multiply for two
// instructions).  Row strides are 4 mod 16 doubles, so the 4 x 4 doubles that
// half a warp fetches lie in different banks.
//
// The accumulators hold the sums of kCRun chunks (64 cells), which are then added
// to the thread's totals in shared memory: one sum over a whole run of 1,024
// cells rounds two to ten times as much as short sums of sums do.  Against 80-bit
// sums, rms of the diagonal scale, 16 genes: p = 9, 2,000 cells 3.5e-16 with one
// sum, 0.8e-16 so (the shared-memory engine: 0.8e-16); p = 16, 20,000 cells
// 1.1e-16, 0.6e-16 (0.8e-16); p = 4, 1,500 cells 9.8e-16, 1.1e-16 (the register
// engine: 1.2e-16).  It costs 500 genes x 20,000 cells 298 -> 306 us at p = 16,
// 574 -> 588 at p = 24, 929 -> 990 at p = 32.  Two chunks: the error of a run of r
// cells in s is about u sqrt((r / 3) (r / s) + (s / r) / 3), least at r = 64 to 80
// for s = 1,024; up to three units (p <= 12) the shared memory takes a second
// level, four runs to a total, as short as the register engine's sums.
//
// Up to nine units a thread keeps to 128 registers for two blocks per SM.  At p =
// 18..22 it then spills about 88 bytes; with one block and no spill, 4,000 x
// 50,000, p = 18 takes 5.5 ms instead of 4.8.
//
// Bound by the FP64 tensor pipe and the latency around it: at 4,000 x 20,000, p =
// 16 (two blocks of 122 registers per SM) that pipe is 49 % busy, 65 % with 40
// clusters, issue slots 45 %, and warps wait for it, for shared memory and at the
// two barriers of a chunk.  The engine it replaces kept one output per thread and
// read two shared doubles per multiply-add.  Measured, 8,500 genes x 30,000 cells,
// p = 16: bread 42.5 -> 4.9 ms, MOM 19.0 -> 1.6 ms.
#include "internal.h"
#include "tc_common.cuh"

#include <algorithm>

namespace devil {

namespace {

constexpr int kCG = 32;   // genes per block
constexpr int kCC = 32;   // cells per chunk
constexpr int kCNT = 256;
constexpr int kCW = kCG + 4;  // weight row stride (4 mod 16)
constexpr int kCY = kCC + 1;  // count row stride
constexpr int kCRun = 2;      // chunks whose sums the accumulators hold (see above)
constexpr int kCRuns = 4;     // runs in a total where there are two levels of them

// smallest stride >= xs that is 4 mod 16
__host__ __device__ constexpr int c64_stride(int xs) { return xs + ((20 - xs % 16) % 16); }

// tiles of 8 products (and of 8 score sums), and the units of a warp
__host__ __device__ constexpr int c64_tiles(int P, bool vec) { return (P * (P + 1) / 2 + 7) / 8 + (vec ? (P + 7) / 8 : 0); }
__host__ __device__ constexpr int c64_units(int P, bool vec) { return (c64_tiles(P, vec) + 3) / 4; }
// levels of totals: one per run, and up to three units a second one per kCRuns runs
__host__ __device__ constexpr int c64_totals(int units) { return units <= 3 ? 2 : 1; }

template <bool VEC>
constexpr size_t c64_smem(int P, int xs) {
    return (size_t)(2 * kCC + kCG) * c64_stride(xs) * sizeof(double) +
           (VEC ? 2 : 1) * (size_t)kCC * kCW * sizeof(double) +
           (size_t)c64_totals(c64_units(P, VEC)) * c64_units(P, VEC) * 4 * kCNT * sizeof(double) +
           (size_t)2 * kCG * kCY * sizeof(float);
}

// C (8 x 8) += A (8 x 4, row) B (4 x 8, column): lane l holds A[l / 4][l % 4],
// B[l % 4][l / 4] and C[l / 4][2 (l % 4) + {0, 1}]
DEV void mma_f64(double& c0, double& c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

// UN: units of (16 genes, 8 outputs) a warp holds at most; VEC: the score sums
// too (clusters)
template <int UN, bool VEC, class VT>
__global__ void __launch_bounds__(kCNT, UN <= 9 ? 2 : 1) cell64_kernel(PassGeom geo, const double* beta,
                                                                       const double* theta, int P) {
    if (geo.reset_next && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *geo.reset_next = 0;
    const int nact = *geo.n_act;
    const int tile = blockIdx.y, seg = blockIdx.x;
    if (tile * kCG >= nact) return;
    const int xs = geo.xs, RS = c64_stride(xs);
    extern __shared__ __align__(16) double c64sm[];
    double* xsm = c64sm;                      // [2][kCC][RS] design rows
    double* bsm = xsm + 2 * kCC * RS;         // [kCG][RS] coefficients
    double* wsm = bsm + kCG * RS;             // [VEC ? 2 : 1][kCC][kCW] weights
    constexpr int TL = c64_totals(UN);
    const int TS = c64_units(P, VEC) * 4 * kCNT;
    double* tot = wsm + (VEC ? 2 : 1) * kCC * kCW;            // [TL][units][4][kCNT] sums of the runs before
    float* ysm = reinterpret_cast<float*>(tot + TL * TS);     // [2][kCG][kCY]
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, r4 = lane >> 2, k4 = lane & 3;
    const int NE = P * (P + 1) / 2;

    auto gene_at = [&](int r) {  // (beyond the list: its tile's first gene again, not written)
        int slot = tile * kCG + r;
        if (slot >= nact) slot = tile * kCG;
        return __ldg(geo.act + slot);
    };
    for (int i = t; i < kCG * xs; i += kCNT) {
        const int r = i / xs, k = i - r * xs;
        bsm[r * RS + k] = k < P ? __ldg(beta + (int64_t)gene_at(r) * P + k) : 0.0;
    }
    for (int i = t; i < 2 * kCG * kCY; i += kCNT) ysm[i] = 0.f;

    const int nfs = geo.nbound - 1;
    const int b0 = (int)(((int64_t)seg * nfs) / geo.nseg);
    const int b1 = (int)(((int64_t)(seg + 1) * nfs) / geo.nseg);
    const int c0 = __ldg(geo.bound + b0), c1 = __ldg(geo.bound + b1);
    const int nchunk = (c1 - c0 + kCC - 1) / kCC;

    // the nonzeros: lanes 8 s .. 8 s + 7 of a warp hold up to 32 entries of gene
    // 4 warp + s, from its first one at or after the chunk
    const VT* __restrict__ val = static_cast<const VT*>(geo.val);
    const int yr = 4 * warp + (lane >> 3), yl = lane & 7;
    int64_t cur, cend;
    {
        const int64_t* sp = geo.segptr + (int64_t)gene_at(yr) * geo.nbound;
        cur = __ldg(sp + b0);
        cend = __ldg(sp + b1);
    }
    int ec[4];
    float ev[4];
    auto load_entries = [&]() {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int64_t e = cur + yl + 8 * q;
            ec[q] = e < cend ? __ldg(geo.col + e) : INT32_MAX;
            ev[q] = e < cend ? load_val(val, e) : 0.f;
        }
    };
    // this chunk's entries into the tile; the cursor moves past them
    auto scatter = [&](int cb, float* ys) {
        int took = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool in = ec[q] < cb + kCC;  // (entries are ascending, none lies before cb)
            if (in) ys[yr * kCY + ec[q] - cb] = ev[q];
            took += __popc(__ballot_sync(0xffffffffu, in) >> (lane & 24) & 0xffu);
        }
        cur += took;
    };
    // the chunk's design rows (zeros past the run's end)
    auto fetch = [&](int cb, int s) {
        const int per = xs / 2;
        for (int i = t; i < kCC * per; i += kCNT) {
            const int c = i / per, q = i - c * per;
            const bool in = cb + c < c1;
            cp_async_zfill(xsm + (s * kCC + c) * RS + 2 * q, geo.Xd + (int64_t)(in ? cb + c : c0) * xs + 2 * q,
                           in ? 16u : 0u);
        }
    };

    // eta tile of this warp: genes 8 mt + r4, cells 8 (ct + h) + 2 k4 + {0, 1}, h = 0, 1
    const int mt = warp & 3, ct = (warp >> 2) * 2;
    const double th = __ldg(theta + gene_at(8 * mt + r4));
    double offn[4];
    auto load_off = [&](int cb) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = cb + 8 * (ct + h) + 2 * k4 + e;
                offn[2 * h + e] = c < c1 ? __ldg(geo.offd + c) : 0.0;
            }
    };

    // the warp's units u = warp + 8 i: genes 16 (u % 2) .., outputs 8 (u / 2) ..
    const int NTo = (NE + 7) / 8, NT = NTo + (VEC ? (P + 7) / 8 : 0);
    double acc[UN][2][2];
    int pair[UN];
#pragma unroll
    for (int i = 0; i < UN; ++i) {
        acc[i][0][0] = acc[i][0][1] = acc[i][1][0] = acc[i][1][1] = 0.0;
        const int nt = (warp + 8 * i) >> 1;
        int n = 8 * nt + r4;
        if (nt >= NTo) {
            n -= 8 * NTo;
            pair[i] = n < P ? n : 0;
        } else {
            if (n >= NE) n = 0;
            int j = 0;
            while ((j + 1) * (j + 2) / 2 <= n) ++j;
            pair[i] = (n - j * (j + 1) / 2) | j << 16;
        }
    }

    // run r's sums into the totals (each thread its own place)
    auto add_run = [&](int r) {
        const bool fresh = TL == 2 ? r % kCRuns == 0 : r == 0;
#pragma unroll
        for (int i = 0; i < UN; ++i) {
            if ((warp + 8 * i) >> 1 >= NT) break;
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    double& o = tot[(4 * i + 2 * m + q) * kCNT + t];
                    const double v = fresh ? acc[i][m][q] : o + acc[i][m][q];
                    acc[i][m][q] = 0.0;
                    o = v;
                    if (TL == 2 && r % kCRuns == kCRuns - 1) (&o)[TS] = r < kCRuns ? v : (&o)[TS] + v;
                }
        }
    };

    if (nchunk > 0) {
        fetch(c0, 0);
        load_entries();
        load_off(c0);
    }
    cp_async_commit();
    __syncthreads();  // the zeroed tiles, the coefficients
    for (int k = 0; k < nchunk; ++k) {
        const int cb = c0 + k * kCC, s = k & 1;
        float* ys = ysm + s * kCG * kCY;
        if (k > 0 && k % kCRun == 0) add_run(k / kCRun - 1);
        scatter(cb, ys);
        load_entries();  // the next chunk's
        cp_async_wait<0>();
        __syncthreads();  // rows and counts of chunk k; the warps are done with chunk k - 1
        if (k + 1 < nchunk) fetch(cb + kCC, s ^ 1);
        cp_async_commit();
        {
            // the other tile, read in chunk k - 1, for chunk k + 1
            float* yo = ysm + (s ^ 1) * kCG * kCY + yr * kCY;
#pragma unroll
            for (int q = 0; q < 4; ++q) yo[yl + 8 * q] = 0.f;
            __syncwarp();  // (the same warp scatters into it next)
        }
        const double* xr = xsm + s * kCC * RS;
        double e[2][2] = {{offn[0], offn[1]}, {offn[2], offn[3]}};
        load_off(cb + kCC);
        for (int kk = 0; kk < xs; kk += 4) {
            const double a = bsm[(8 * mt + r4) * RS + kk + k4];
#pragma unroll
            for (int h = 0; h < 2; ++h) mma_f64(e[h][0], e[h][1], a, xr[(8 * (ct + h) + r4) * RS + kk + k4]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int c = 8 * (ct + h) + 2 * k4 + q;
                const bool in = cb + c < c1;
                const double mu = exp(e[h][q]);
                const double y = ys[(8 * mt + r4) * kCY + c];
                const double r = rcp_nr(fma(th, mu, 1.0));
                double w = mu * r * r;
                if (y != 0.0) w = fma(y * th, w, w);
                wsm[c * kCW + 8 * mt + r4] = in ? w : 0.0;
                if constexpr (VEC) wsm[(kCC + c) * kCW + 8 * mt + r4] = in ? (y - mu) * r : 0.0;
            }
        {
            __syncthreads();  // the weights
            const int mh = warp & 1;
#pragma unroll 2
            for (int kk = 0; kk < kCC; kk += 4) {
                const double* wr = wsm + (kk + k4) * kCW + 16 * mh + r4;
                const double a0 = wr[0], a1 = wr[8];
                double v0 = 0.0, v1 = 0.0;
                if constexpr (VEC) {
                    v0 = wr[kCC * kCW];
                    v1 = wr[kCC * kCW + 8];
                }
                const double* row = xr + (kk + k4) * RS;
#pragma unroll
                for (int i = 0; i < UN; ++i) {
                    const int nt = (warp + 8 * i) >> 1;
                    if (nt >= NT) break;
                    const double xi = row[pair[i] & 0xffff];
                    if (VEC && nt >= NTo) {
                        mma_f64(acc[i][0][0], acc[i][0][1], v0, xi);
                        mma_f64(acc[i][1][0], acc[i][1][1], v1, xi);
                    } else {
                        const double z = xi * row[pair[i] >> 16];
                        mma_f64(acc[i][0][0], acc[i][0][1], a0, z);
                        mma_f64(acc[i][1][0], acc[i][1][1], a1, z);
                    }
                }
            }
        }
    }
    cp_async_wait<0>();
    const int runs = nchunk > 0 ? (nchunk - 1) / kCRun + 1 : 1;
    add_run(runs - 1);
    {
        const int NA = NE + P;
        // the totals: the second level, and runs that did not fill one
        const bool low = TL == 1 || runs % kCRuns != 0, high = TL == 2 && runs >= kCRuns;
#pragma unroll
        for (int i = 0; i < UN; ++i) {
            const int nt = (warp + 8 * i) >> 1;
            if (nt >= NT) break;
            const bool vec = nt >= NTo;
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const int slot = tile * kCG + 16 * (warp & 1) + 8 * m + r4;
                if (slot >= nact) continue;
                double* o = static_cast<double*>(geo.partW) + ((int64_t)seg * geo.slot_stride + slot) * NA;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int n = 8 * (vec ? nt - NTo : nt) + 2 * k4 + q;
                    const double* v = tot + (4 * i + 2 * m + q) * kCNT + t;
                    if (n < (vec ? P : NE)) o[(vec ? NE : 0) + n] = (high ? v[TS] : 0.0) + (low ? v[0] : 0.0);
                }
            }
        }
    }
}

// MOM moments, with each gene's sums in cell order (one chain of additions per
// run of cells): the MLE search starts from this estimate and resolves its last
// bracket at rounding level, so another order would move the theta of some
// genes by 1e-7.  Block = 32 GPT genes x one run of cells, chunks of 32 cells:
// lane = GPT genes with their coefficients in registers, warp = four of the
// chunk's cells, whose design rows all lanes read at once; the per-cell terms go
// to shared memory and a thread per (gene, moment) adds them up while the other
// warps and the SM's other block evaluate.  Bound by the FP64 pipe (p
// multiply-adds, exp and five more operations a gene-cell); GPT = 2 halves the
// shared reads and fits the registers up to p = 16.  The engine it replaces took
// four barriers for 32 cells of eight genes.
template <int XS, int GPT, class VT>
__global__ void __launch_bounds__(kCNT, XS <= 16 ? 2 : 1) mom_cells_kernel(PassGeom geo, const double* beta, int P) {
    constexpr int NG = 32 * GPT;
    if (geo.reset_next && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *geo.reset_next = 0;
    const int nact = *geo.n_act;
    const int tile = blockIdx.y, seg = blockIdx.x;
    if (tile * NG >= nact) return;
    extern __shared__ __align__(16) double c64sm[];
    double* xsm = c64sm;                                      // [2][kCC][XS] design rows
    double* vsm = xsm + 2 * kCC * XS;                         // [2][NG][kCY] terms of the two moments
    float* ysm = reinterpret_cast<float*>(vsm + 2 * NG * kCY);  // [2][NG][kCY]
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    auto gene_at = [&](int r) {
        int slot = tile * NG + r;
        if (slot >= nact) slot = tile * NG;
        return __ldg(geo.act + slot);
    };
    double b[GPT][XS];
#pragma unroll
    for (int j = 0; j < GPT; ++j) {
        const double* bg = beta + (int64_t)gene_at(lane + 32 * j) * P;
#pragma unroll
        for (int i = 0; i < XS; ++i) b[j][i] = i < P ? __ldg(bg + i) : 0.0;
    }
    for (int i = t; i < 2 * NG * kCY; i += kCNT) ysm[i] = 0.f;
    const int nfs = geo.nbound - 1;
    const int b0 = (int)(((int64_t)seg * nfs) / geo.nseg);
    const int b1 = (int)(((int64_t)(seg + 1) * nfs) / geo.nseg);
    const int c0 = __ldg(geo.bound + b0), c1 = __ldg(geo.bound + b1);
    const int nchunk = (c1 - c0 + kCC - 1) / kCC;
    // the nonzeros: eight lanes per gene, GPT genes each (see cell64_kernel)
    const VT* __restrict__ val = static_cast<const VT*>(geo.val);
    const int yr = 4 * warp + (lane >> 3), yl = lane & 7;
    int64_t cur[GPT], cend[GPT];
    int ec[GPT][4];
    float ev[GPT][4];
#pragma unroll
    for (int j = 0; j < GPT; ++j) {
        const int64_t* sp = geo.segptr + (int64_t)gene_at(yr + 32 * j) * geo.nbound;
        cur[j] = __ldg(sp + b0);
        cend[j] = __ldg(sp + b1);
    }
    auto load_entries = [&]() {
#pragma unroll
        for (int j = 0; j < GPT; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int64_t e = cur[j] + yl + 8 * q;
                ec[j][q] = e < cend[j] ? __ldg(geo.col + e) : INT32_MAX;
                ev[j][q] = e < cend[j] ? load_val(val, e) : 0.f;
            }
    };
    auto scatter = [&](int cb, float* ys) {
#pragma unroll
        for (int j = 0; j < GPT; ++j) {
            int took = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool in = ec[j][q] < cb + kCC;
                if (in) ys[(yr + 32 * j) * kCY + ec[j][q] - cb] = ev[j][q];
                took += __popc(__ballot_sync(0xffffffffu, in) >> (lane & 24) & 0xffu);
            }
            cur[j] += took;
        }
    };
    auto fetch = [&](int cb, int s) {
        for (int i = t; i < kCC * XS / 2; i += kCNT) {
            const int c = i / (XS / 2), q = i - c * (XS / 2);
            const bool in = cb + c < c1;
            cp_async_zfill(xsm + (s * kCC + c) * XS + 2 * q, geo.Xd + (int64_t)(in ? cb + c : c0) * XS + 2 * q,
                           in ? 16u : 0u);
        }
    };
    double offn[4];
    auto load_off = [&](int cb) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int c = cb + 4 * warp + q;
            offn[q] = c < c1 ? __ldg(geo.offd + c) : 0.0;
        }
    };
    double sum = 0.0;  // threads t < 2 NG: moment t / NG of gene t % NG
    if (nchunk > 0) {
        fetch(c0, 0);
        load_entries();
        load_off(c0);
    }
    cp_async_commit();
    __syncthreads();
    for (int k = 0; k < nchunk; ++k) {
        const int cb = c0 + k * kCC, s = k & 1, nc = min(kCC, c1 - cb);
        float* ys = ysm + s * NG * kCY;
        scatter(cb, ys);
        load_entries();
        cp_async_wait<0>();
        __syncthreads();  // rows and counts of chunk k; the sums of chunk k - 1 are done
        if (k + 1 < nchunk) fetch(cb + kCC, s ^ 1);
        cp_async_commit();
#pragma unroll
        for (int j = 0; j < GPT; ++j) {
            float* yo = ysm + (s ^ 1) * NG * kCY + (yr + 32 * j) * kCY;
#pragma unroll
            for (int q = 0; q < 4; ++q) yo[yl + 8 * q] = 0.f;
        }
        __syncwarp();
        const double off[4] = {offn[0], offn[1], offn[2], offn[3]};
        load_off(cb + kCC);
        const double2* xr = reinterpret_cast<const double2*>(xsm + (s * kCC + 4 * warp) * XS);
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // two cells at a time
            double e[2][GPT];
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int j = 0; j < GPT; ++j) e[q][j] = off[2 * h + q];
#pragma unroll
            for (int i = 0; i < XS / 2; ++i)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const double2 x = xr[(2 * h + q) * (XS / 2) + i];
#pragma unroll
                    for (int j = 0; j < GPT; ++j) e[q][j] = fma(x.x, b[j][2 * i], e[q][j]);
#pragma unroll
                    for (int j = 0; j < GPT; ++j) e[q][j] = fma(x.y, b[j][2 * i + 1], e[q][j]);  // (pads: 0 x 0)
                }
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int j = 0; j < GPT; ++j) {
                    const int c = 4 * warp + 2 * h + q, r = lane + 32 * j;
                    const float y = ys[r * kCY + c];
                    RecAcc<0, 2, double, double> rec;
                    rec.zero();
                    const double mu = exp(e[q][j]);
                    PassMOM::dense<double>(PassMOM::Gene{0}, mu, rec);
                    if (y != 0.f) PassMOM::sparse<double>(PassMOM::Gene{0}, mu, y, rec);
                    vsm[r * kCY + c] = rec.s[0];
                    vsm[(NG + r) * kCY + c] = rec.s[1];
                }
        }
        __syncthreads();  // the chunk's terms
        if (t < 2 * NG) {
            const double* v = vsm + t * kCY;
            if (nc == kCC) {
#pragma unroll
                for (int c = 0; c < kCC; ++c) sum += v[c];
            } else {
                for (int c = 0; c < nc; ++c) sum += v[c];
            }
        }
    }
    cp_async_wait<0>();
    if (t < 2 * NG) {
        const int slot = tile * NG + t % NG;
        if (slot < nact) geo.partS[((int64_t)seg * geo.slot_stride + slot) * 2 + t / NG] = sum;
    }
}

template <int XS, int GPT>
cudaError_t run_mom(const PassLaunch& L, int max_slots) {
    constexpr int NG = 32 * GPT;
    constexpr size_t smem = (size_t)(2 * kCC * XS + 2 * NG * kCY) * sizeof(double) + (size_t)2 * NG * kCY * sizeof(float);
    auto go = [&](auto kern) -> cudaError_t {
        cudaError_t e = raise_dyn_smem(kern, smem);
        if (e != cudaSuccess) return e;
        kern<<<dim3(L.nseg, (max_slots + NG - 1) / NG), kCNT, smem, L.stream>>>(L.geo, L.prm.beta_d, L.P);
        return cudaGetLastError();
    };
    return L.val_u16 ? go(mom_cells_kernel<XS, GPT, uint16_t>) : go(mom_cells_kernel<XS, GPT, float>);
}

template <int UN, bool VEC>
cudaError_t run(const PassLaunch& L) {
    const size_t smem = c64_smem<VEC>(L.P, L.xs_pad);
    auto go = [&](auto kern) -> cudaError_t {
        cudaError_t e = raise_dyn_smem(kern, smem);
        if (e != cudaSuccess) return e;
        if (L.occ_out) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(L.occ_out, kern, kCNT, smem);
        kern<<<dim3(L.nseg, L.ntiles), kCNT, smem, L.stream>>>(L.geo, L.prm.beta_d, L.prm.theta, L.P);
        return cudaGetLastError();
    };
    return L.val_u16 ? go(cell64_kernel<UN, VEC, uint16_t>) : go(cell64_kernel<UN, VEC, float>);
}

template <bool VEC>
cudaError_t run_bread(const PassLaunch& L) {
    const int units = c64_units(L.P, VEC);
    if (units <= 3) return run<3, VEC>(L);
    if (units <= 5) return run<5, VEC>(L);
    if (units <= 9) return run<9, VEC>(L);
    if (units <= 13) return run<13, VEC>(L);
    return run<18, VEC>(L);
}

}  // namespace

int cell64_tile_genes() { return kCG; }
// (row strides of 4, 8, 12, .. doubles)
bool cell64_supported(PassKind k, int P, int xs) { return k == PASS_SANDWICH && P >= 3 && P <= 32 && xs % 4 == 0; }
cudaError_t launch_cell64_pass(const PassLaunch& L) {
    if (!cell64_supported(L.kind, L.P, L.xs_pad)) return cudaErrorInvalidValue;
    return L.vec ? run_bread<true>(L) : run_bread<false>(L);
}

bool mom_cells_supported(int P, int xs) { return P > 8 && P <= 32 && xs == ((P + 3) & ~3); }
cudaError_t launch_mom_cells(const PassLaunch& L, int max_slots) {
    if (max_slots <= 0) return cudaSuccess;
    switch (L.xs_pad) {
        case 12: return run_mom<12, 2>(L, max_slots);
        case 16: return run_mom<16, 2>(L, max_slots);
        case 20: return run_mom<20, 1>(L, max_slots);
        case 24: return run_mom<24, 1>(L, max_slots);
        case 28: return run_mom<28, 1>(L, max_slots);
        case 32: return run_mom<32, 1>(L, max_slots);
    }
    return cudaErrorInvalidValue;
}

}  // namespace devil
