// IRLS and dispersion (MLE) passes with the per-gene p x p contractions on
// the tensor cores (sm_100a tcgen05, kind::tf32) for designs of p = 5..32
// columns that do not collapse to a few distinct rows (continuous
// covariates).  The IRLS form is described here; the MLE form (the Cox-Reid
// matrices) is described at tcw_pass_kernel.
//
// beta_fit (src/beta.cpp:35-42) needs per gene g and IRLS step
//     H_g = sum_c hw_gc z_c,   z_c = the products x_ci x_cj (i <= j),
//     s_g = sum_c sw_gc x_c,
// with r = 1/(mu + k), hw = r (1 + y / k), sw = (mu - y) r (PassIRLS in
// passes.cuh: the dense terms of every cell plus the nonzero corrections).
// Over a tile of 128 genes and a chunk of 32 cells the Hessian part is the
// product
//     D[128 genes x NBLK products] += HW[128 x 32 cells] Z[NBLK x 32 cells]^T
// with NE = p (p + 1) / 2 products split over gridDim.z blocks of at most
// 176 columns (p = 32: three blocks of 176).  The counts enter the weights
// directly: the pass reads a dense image of the counts (gene rows of
// npad cells, uint16 or float), so no separate nonzero pass is needed.
//
// Per chunk the CUDA cores compute eta = off + x beta (FP32, packed FMAs; the
// images hold a quad's cells in the order 0, 2, 1, 3, so that every pair that a
// packed instruction takes is one register pair as loaded),
// mu (ex2), r (rcp), the weights, and the chunk's products z = x_i x_j;
// HW and Z enter as split TF32 pairs (v = hi + lo) and the MMA sums
//     HW_hi Z_hi + HW_lo Z_hi + HW_hi Z_lo
// (3 x TF32: about 2^-21 relative per term, the hi x lo terms of both
// operands kept; lo x lo, ~2^-22, dropped).  The score, which fixes the
// solution, stays on the CUDA cores in FP32 (block z = 0).
//
// Accumulation: D accumulates a run of 8 chunks (256 cells) in tensor
// memory; the run is then added in FP32 on the CUDA cores into a running
// total (tensor-memory columns T.., T = 128 or 256, tcgen05.ld / add /
// tcgen05.st), so no tensor-core accumulation spans more than 256 terms.
// A block allocates 2 T columns: two blocks of a small product count
// (T = 128) can share an SM's 512 columns.
//
// Pipeline: cp.async brings the chunk's design rows (transposed: feature
// rows of 32 cells), offsets and count rows two chunks ahead (ring of 3);
// the operand stages (HW_hi, HW_lo, Z_hi, Z_lo) are double-buffered and a
// stage is rewritten only after the MMAs that read it have completed
// (mbarrier, bounded wait).  A run is added to the total after the next
// chunk's CUDA-core work, so that work overlaps the run's last MMAs.  On a
// bounded wait's expiry the block records an error, skips its output,
// drains its MMAs (bounded) and frees its tensor memory.
#include "internal.h"
#include "tc_common.cuh"

#include <algorithm>

namespace devil {

namespace {

constexpr int kWM = 128;                  // genes per tile: MMA M, tensor-memory lanes
constexpr int kWKC = 32;                  // cells per chunk (4 K-steps of 8 TF32)
constexpr int kWNT = 384;                 // threads per block: 256 of the weights, 128 of the products
constexpr int kWW = 256;
constexpr int kWNmax = 176;               // product columns per block at most
constexpr int kWRun = 8;                  // chunks per tensor-memory run (256 cells)
constexpr int kWA = kWM * kWKC * 4;       // one of HW_hi, HW_lo: 16 KB
constexpr int kWRing = 3;                 // input ring depth

constexpr int op_bytes(int nblk) { return 2 * kWA + 2 * nblk * kWKC * 4; }
template <class VT, int GTn>
constexpr int in_bytes(int XS) { return XS * kWKC * 4 + kWKC * 4 + GTn * kWKC * (int)sizeof(VT); }
constexpr int kMleG = 32;                             // genes per tile of the MLE pass
constexpr int kPsiBytes = kMleG * 2 * kPsiTab * 8;    // their psi tables
template <class VT, bool MLE>
constexpr int tcw_smem(int XS, int nblk) {
    return 2 * op_bytes(nblk) + kWRing * in_bytes<VT, MLE ? kMleG : kWM>(XS) + (MLE ? kPsiBytes : 0);
}

static_assert(tcw_smem<float, false>(32, kWNmax) <= 227 * 1024, "stages fit the shared memory of one block");
static_assert(tcw_smem<float, true>(32, kWNmax) <= 227 * 1024, "stages fit the shared memory of one block");

// pairs of FP32 values in one 64-bit register pair
DEV uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
DEV void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
// a + b * c, both halves (two correctly rounded FMAs)
DEV uint64_t fma2(uint64_t b, uint64_t c, uint64_t a) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(c), "l"(a));
    return r;
}
DEV uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a quad's four values of one feature: cells (0, 2) and (1, 3) as pairs (the
// order the images are written in, tcw_quad_pos)
DEV void ld_quad(const void* p, uint64_t& c02, uint64_t& c13) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    c02 = v.x;
    c13 = v.y;
}

// counts of cells 4q..4q+3 of gene row gr in a count stage of R rows
template <int R>
DEV void load_counts(const uint16_t* ys, int q, int gr, float* y) {
    // piece (gene, 8 cells) at ((q >> 1) * R + gene) * 16; this quad is its half q & 1
    const uint2 h = *reinterpret_cast<const uint2*>(
        reinterpret_cast<const unsigned char*>(ys) + (((q >> 1) * R + gr) * 16 + (q & 1) * 8));
    y[0] = (float)(h.x & 0xFFFFu);
    y[1] = (float)(h.x >> 16);
    y[2] = (float)(h.y & 0xFFFFu);
    y[3] = (float)(h.y >> 16);
}
template <int R>
DEV void load_counts(const float* ys, int q, int gr, float* y) {
    const float4 v = *reinterpret_cast<const float4*>(
        reinterpret_cast<const unsigned char*>(ys) + (q * R + gr) * 16);
    y[0] = v.x;
    y[1] = v.y;
    y[2] = v.z;
    y[3] = v.w;
}

// add the run (columns [c0, c1) of this warp's 32 lanes) into the total
// at column offset tot
DEV void tcw_drain(uint32_t tmem, uint32_t lanes, uint32_t tot, int c0, int c1, bool first) {
    for (int c = c0; c < c1; c += 8) {
        float v[8];
        tc_ld8(tmem + lanes + (uint32_t)c, v);
        if (!first) {
            float t[8];
            tc_ld8(tmem + lanes + tot + (uint32_t)c, t);
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] += t[u];
        }
        tc_st8(tmem + lanes + tot + (uint32_t)c, v);
    }
    tc_wait_st();
}

DEV void store_split(unsigned char* sA, int row, int q, const float* v) {
    float hi[4], lo[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) tf32_split(v[c], hi[c], lo[c]);
    *reinterpret_cast<float4*>(sA + stage_off(row, q, kWM)) = make_float4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<float4*>(sA + kWA + stage_off(row, q, kWM)) = make_float4(lo[0], lo[1], lo[2], lo[3]);
}

// Threads 0..255 (the weights) form the weights of a chunk and the score;
// threads 256..383 (the products) bring the inputs and the products (from the
// image by bulk copies; formed here when the image does not fit the memory), add
// finished runs into the total and issue the MMAs, so that the two halves of the
// work overlap and one barrier per chunk is left.
// The IRLS pass (MLE = false): 128 genes per tile, A row = gene, weight
// r (1 + y / k); weight thread = (gene row tid % 128, cells of quads 4 h .. 4 h
// + 3 with h = tid / 128), the score in registers; up to 16 features a quad's
// values stay in registers from eta to the score (one shared read each: 16-byte
// reads that all lanes share take the register file's write bandwidth).
// The dispersion pass (MLE = true; PassMLE in passes.cuh,
// src/overdispersion.cpp:95-242): 32 genes per tile, A rows 32 b + gene
// carry the Cox-Reid weights w, -w^2, 2 w^3 (b = 0, 1, 2; rows 96..127
// zero); thread = (gene tid % 32, quad tid / 32); the two FP32 scalar sums
// and, at the gene's nonzeros, the four FP64 sums with per-gene psi tables,
// all in block z = 0.
template <int XS, class VT, bool MLE>
__global__ void __launch_bounds__(kWNT, 1) tcw_pass_kernel(PassGeom geo, PassParamsAny prm, TcwGeom tw) {
    constexpr int GTn = MLE ? kMleG : kWM;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[2];   // MMAs of the stage's chunk done
    __shared__ __align__(8) uint64_t zbars[2];  // the stage's products in place (zimg)
    __shared__ uint32_t tslot;
    __shared__ int abort_flag;
    __shared__ int16_t ptab[kWNmax];  // product row -> i | j << 8 (-1: padding)
    __shared__ double psia[MLE ? kMleG : 1];

    grid_trigger();
    if (geo.reset_next && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.x == 0)
        *geo.reset_next = 0;
    const int nact = *geo.n_act;
    const int tile = blockIdx.y;
    if (tile * GTn >= nact) return;
    const int seg = blockIdx.x;
    const int zb = blockIdx.z;
    const int nblk = tw.nblk;
    const uint32_t tot = nblk <= 128 ? 128u : 256u;  // column of the running total
    const uint32_t ncols = 2 * tot;                  // columns allocated
    const int tid = threadIdx.x, warp = tid >> 5;
    const int gi = tid & (GTn - 1);  // this thread's gene within the tile
    const bool wt = tid < kWW;       // a weight thread
    const int pt = tid - kWW;        // product thread
    const int hh = (tid >> 7) & 1;   // IRLS: half of the chunk's cells (and of the last run's columns)
    const bool extra = zb == 0;      // block z = 0 adds the score / scalar sums

    int slot = tile * GTn + gi;
    const bool valid_slot = slot < nact;
    if (!valid_slot) slot = tile * GTn;  // duplicate a valid gene; not written
    const int g = __ldg(geo.act + slot);
    uint64_t bt[XS];  // the coefficient, twice
    if (wt) {
#pragma unroll
        for (int i = 0; i < XS; ++i) {
            const float b = i < tw.P ? __ldg(prm.beta + (int64_t)g * tw.P + i) * kLog2e : 0.f;
            bt[i] = pack2(b, b);
        }
    }
    float kk = 0.f, rk = 0.f, thf = 0.f;
    double theta = 0.0, aa = 0.0;
    if constexpr (MLE) {
        theta = exp(prm.log_theta[g]);
        aa = 1.0 / theta;
        thf = (float)theta;
    } else {
        kk = __ldg(prm.k + g);
        rk = 1.f / kk;
    }

    for (int r = tid; r < nblk; r += kWNT) {
        const int gp = zb * nblk + r;
        int16_t v = -1;
        if (gp < tw.NE) {
            int j = 0;
            while ((j + 1) * (j + 2) / 2 <= gp) ++j;
            const int i = gp - j * (j + 1) / 2;
            v = (int16_t)(i | (j << 8));
        }
        ptab[r] = v;
    }

    // this block's cells: fine segments [b0, b1) (multiples of 32 cells up
    // to n; the last chunk reads the padding of the images past n)
    const int nfs = geo.nbound - 1;
    const int b0 = (int)(((int64_t)seg * nfs) / geo.nseg);
    const int b1 = (int)(((int64_t)(seg + 1) * nfs) / geo.nseg);
    const int64_t k0 = __ldg(geo.bound + b0) / kWKC;
    const int64_t k1 = (__ldg(geo.bound + b1) + kWKC - 1) / kWKC;
    const int nchunk = (int)(k1 - k0);

    const int OPB = op_bytes(nblk);
    constexpr int INB = in_bytes<VT, GTn>(XS);
    auto op = [&](int s) { return smem + s * OPB; };
    auto in_slot = [&](int s) { return smem + 2 * OPB + s * INB; };
    const VT* __restrict__ yrow = static_cast<const VT*>(tw.ydense) + (int64_t)g * tw.ld;

    // MLE: the tile's psi tables (scratch in the first operand stage), then
    // the zero rows 96..127 of both A stages
    PsiTable tab{nullptr, nullptr, 0.0, 0.0};
    if constexpr (MLE) {
        double* psitab = reinterpret_cast<double*>(smem + 2 * OPB + kWRing * INB);
        if (tid < kMleG) psia[tid] = aa;
        __syncthreads();
        build_psi_tables(kMleG, psia, psitab, reinterpret_cast<double*>(smem));
        tab.d1 = psitab + (gi * 2 + 0) * kPsiTab;
        tab.d2 = psitab + (gi * 2 + 1) * kPsiTab;
        if (extra) {
            tab.pa = digamma_d(aa);
            tab.ta = trigamma_d(aa);
        }
        for (int t = tid; t < 2 * 2 * 32 * 8; t += kWNT) {
            const int s = t >> 9, hl = (t >> 8) & 1, row = 96 + ((t >> 3) & 31), q = t & 7;
            *reinterpret_cast<float4*>(op(s) + hl * kWA + stage_off(row, q, kWM)) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }

    auto fetch = [&](int kc) {  // (product threads)
        unsigned char* ib = in_slot(kc % kWRing);
        const int64_t cs = (k0 + kc) * kWKC;
        for (int idx = pt; idx < XS * 8 + 8; idx += kWNT - kWW) {
            if (idx < XS * 8) {
                const int i = idx >> 3, q = idx & 7;
                cp_async<16>(ib + stage_off(i, q, XS), tw.xt + (int64_t)i * tw.npad + cs + 4 * q);
            } else {
                const int q = idx - XS * 8;
                cp_async<16>(ib + XS * kWKC * 4 + 16 * q, tw.offp + cs + 4 * q);
            }
        }
        unsigned char* yb = ib + XS * kWKC * 4 + kWKC * 4;
        constexpr int CPP = 16 / (int)sizeof(VT);  // cells per piece
        constexpr int NPG = kWKC / CPP;            // pieces per gene row
        // gene gi; IRLS: its whole row, MLE: every fourth piece from pt / 32
#pragma unroll
        for (int u = 0; u < (MLE ? NPG / 4 : NPG); ++u) {
            const int p = MLE ? (pt >> 5) + 4 * u : u;
            cp_async<16>(yb + (p * GTn + gi) * 16, yrow + cs + p * CPP);
        }
    };

    if (!wt) {
        if (nchunk > 0) fetch(0);
        cp_async_commit();
        if (nchunk > 1) fetch(1);
        cp_async_commit();
        cp_async_wait<1>();  // chunk 0 has landed
    }

    if (tid == 0) {
        abort_flag = 0;
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        mbar_init(&zbars[0], 1);
        mbar_init(&zbars[1], 1);
        mbar_fence_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tslot)),
                     "r"(ncols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tslot;
    const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
    const int dc0 = hh * (nblk / 2), dc1 = dc0 + nblk / 2;  // this warp's drained columns
    const uint32_t idesc = tf32_idesc(kWM, nblk);

    // IRLS score: cells (0, 1) and (2, 3) of each quad; MLE: the FP32 and
    // FP64 scalar sums
    uint64_t vab[MLE ? 1 : XS];
    float fs[2] = {0.f, 0.f};
    double sc[4] = {0.0, 0.0, 0.0, 0.0};
    if constexpr (!MLE) {
#pragma unroll
        for (int i = 0; i < XS; ++i) vab[i] = 0;
    }

    // the chunk's products of this block from the image: one bulk copy
    const uint32_t zbytes = (uint32_t)(2 * nblk * kWKC * 4);
    const unsigned char* zsrc =
        tw.zimg ? reinterpret_cast<const unsigned char*>(tw.zimg) + ((int64_t)zb * (tw.npad / kWKC) + k0) * zbytes
                : nullptr;
    bool zlost = false;  // (thread kWW) a bulk copy did not arrive in time

    int issued = 0;   // chunks whose MMAs were committed (uniform; after zlost not the last one's)
    int drained = 0;  // runs added into the total (uniform)
    for (int k = 0; k < nchunk; ++k) {
        const int st = k & 1;
        bool ok = !zlost;
        // chunk k - 2's MMAs have completed: operand stage st is free.  (Chunk
        // k's inputs: the last barrier.)
        if (k >= 2) ok = mbar_wait_bounded(&bars[st], (uint32_t)(((k - 2) >> 1) & 1)) && ok;
        const unsigned char* ib = in_slot(k % kWRing);
        unsigned char* sA = op(st);
        if (wt && ok) {
            const float4* o4 = reinterpret_cast<const float4*>(ib + XS * kWKC * 4);
            const VT* ys = reinterpret_cast<const VT*>(ib + XS * kWKC * 4 + kWKC * 4);
            // the weights of this thread's gene at its cells
#pragma unroll(XS <= 16 ? 2 : 1)
            for (int qi = 0; qi < (MLE ? 1 : 4); ++qi) {
                const int q = MLE ? warp : 4 * hh + qi;
                const float4 o = o4[q];  // cells 0, 2, 1, 3
                uint64_t e02 = pack2(o.x * kLog2e, o.y * kLog2e), e13 = pack2(o.z * kLog2e, o.w * kLog2e);
                constexpr bool KEEP = !MLE && XS <= 16;
                uint64_t xa[KEEP ? XS : 1], xb[KEEP ? XS : 1];
#pragma unroll
                for (int i = 0; i < XS; ++i) {
                    uint64_t a, b;
                    ld_quad(ib + stage_off(i, q, XS), a, b);
                    e02 = fma2(bt[i], a, e02);
                    e13 = fma2(bt[i], b, e13);
                    if constexpr (KEEP) {
                        xa[i] = a;
                        xb[i] = b;
                    }
                }
                float y[4];
                load_counts<GTn>(ys, q, gi, y);
                float e[4];
                unpack2(e02, e[0], e[2]);
                unpack2(e13, e[1], e[3]);
                if constexpr (MLE) {
                    float w1[4], w2[4], w3[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float mu = ex2_approx(e[c]);
                        const float xx = mu * thf;
                        const float r = rcp_r(1.f + xx);
                        const float w = mu * r;
                        w1[c] = w;
                        w2[c] = -w * w;
                        w3[c] = 2.f * w * w * w;
                        if (extra) {
                            fs[0] += nb_ll_term<float>(xx, r);
                            fs[1] += w * xx * r;
                            if (y[c] > 0.f) {
                                const double m = mu, yy = y[c];
                                const double den = 1.0 + m * theta;
                                double rr = (double)rcp_approx((float)den);
                                rr = rr + rr * (1.0 - den * rr);
                                sc[0] += yy * theta * rr;
                                sc[1] += yy * rr * rr;
                                double d1, d2;
                                psi_diffs_tab(yy, aa, tab, d1, d2);
                                sc[2] += d1;
                                sc[3] += d2;
                            }
                        }
                    }
                    store_split(sA, gi, q, w1);
                    store_split(sA, 32 + gi, q, w2);
                    store_split(sA, 64 + gi, q, w3);
                } else {
                    float hw[4], sw[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float mu = ex2_approx(e[c]);
                        const float r = rcp_approx(mu + kk);
                        const float yr = y[c] * r;
                        hw[c] = fmaf(yr, rk, r);    // r + y r / k
                        sw[c] = fmaf(mu, r, -yr);   // (mu - y) r
                    }
                    store_split(sA, gi, q, hw);
                    if (extra) {
                        const uint64_t s02 = pack2(sw[0], sw[2]), s13 = pack2(sw[1], sw[3]);
#pragma unroll
                        for (int i = 0; i < XS; ++i) {
                            uint64_t a, b;
                            if constexpr (KEEP) {
                                a = xa[i];
                                b = xb[i];
                            } else {
                                ld_quad(ib + stage_off(i, q, XS), a, b);
                            }
                            vab[i] = fma2(s02, a, vab[i]);
                            vab[i] = fma2(s13, b, vab[i]);
                        }
                    }
                }
            }
        } else if (!wt) {
            if (tid == kWW && zsrc && ok) {
                mbar_arrive_expect_tx(&zbars[st], zbytes);
                bulk_g2s(sA + 2 * kWA, zsrc + (int64_t)k * zbytes, zbytes, &zbars[st]);
            }
            if (k + 2 < nchunk) fetch(k + 2);  // (its slot was read in chunk k - 1)
            cp_async_commit();
            // without the image: the chunk's products of this block, split
            if (ok && !zsrc) {
                unsigned char* sB = sA + 2 * kWA;
                int row = pt, q = 0;
                while (row >= nblk) {
                    row -= nblk;
                    ++q;
                }
                for (; q < 8;) {
                    const int pr = ptab[row];
                    float4 hz = make_float4(0.f, 0.f, 0.f, 0.f), lz = hz;
                    if (pr >= 0) {
                        uint64_t ia, ic, ja, jc;
                        ld_quad(ib + stage_off(pr & 0xFF, q, XS), ia, ic);
                        ld_quad(ib + stage_off(pr >> 8, q, XS), ja, jc);
                        float z0, z1, z2, z3;
                        unpack2(mul2(ia, ja), z0, z2);
                        unpack2(mul2(ic, jc), z1, z3);
                        tf32_split(z0, hz.x, lz.x);
                        tf32_split(z1, hz.y, lz.y);
                        tf32_split(z2, hz.z, lz.z);
                        tf32_split(z3, hz.w, lz.w);
                    }
                    *reinterpret_cast<float4*>(sB + stage_off(row, q, nblk)) = hz;
                    *reinterpret_cast<float4*>(sB + nblk * kWKC * 4 + stage_off(row, q, nblk)) = lz;
                    row += kWNT - kWW;
                    while (row >= nblk) {
                        row -= nblk;
                        ++q;
                    }
                }
            }
            // chunk k - 1 closed a run: add it into the total once its MMAs
            // have completed (the work above overlapped them)
            if (k > 0 && k % kWRun == 0) {
                bool okd = mbar_wait_bounded(&bars[(k - 1) & 1], (uint32_t)(((k - 1) >> 1) & 1));
                okd = __all_sync(0xffffffffu, okd);
                if (okd) {
                    tc_fence_after();
                    tcw_drain(tmem, lanes, tot, 0, nblk, drained == 0);
                } else {
                    ok = false;
                }
            }
            cp_async_wait<1>();  // chunk k + 1 has landed
        }
        if (k > 0 && k % kWRun == 0) ++drained;
        fence_async_smem();
        tc_fence_before();
        // operands of chunk k and inputs of chunk k + 1 are in place; every
        // thread learns of a wait that gave up
        if (__syncthreads_or(!ok)) {
            if (tid == 0) abort_flag = 1;
            break;
        }
        if (tid == kWW && zsrc && !mbar_wait_bounded(&zbars[st], (uint32_t)((k >> 1) & 1))) zlost = true;
        if (tid == kWW && !zlost) {
            tc_fence_after();
            const uint32_t a_hi = smem_u32(sA), a_lo = a_hi + kWA;
            const uint32_t b_hi = a_hi + 2 * kWA, b_lo = b_hi + (uint32_t)(nblk * kWKC * 4);
#pragma unroll
            for (int s = 0; s < kWKC / 8; ++s) {
                const uint32_t acc = (k % kWRun != 0 || s > 0) ? 1u : 0u;
                const uint64_t ah = umma_desc(a_hi + s * 2 * kWM * 16, kWM * 16, 128);
                const uint64_t al = umma_desc(a_lo + s * 2 * kWM * 16, kWM * 16, 128);
                const uint64_t bh = umma_desc(b_hi + s * 2 * nblk * 16, nblk * 16, 128);
                const uint64_t bl = umma_desc(b_lo + s * 2 * nblk * 16, nblk * 16, 128);
                tc_mma_n(tmem, ah, bh, acc, idesc);
                tc_mma_n(tmem, al, bh, 1u, idesc);
                tc_mma_n(tmem, ah, bl, 1u, idesc);
            }
            tc_commit(&bars[st]);
        }
        issued = k + 1;
    }
    cp_async_wait<0>();
    // No copy may be in flight when the stages are used again or the block ends,
    // and no MMA when the tensor memory is freed, on the error path too.  Thread
    // kWW waits for the bulk copy that it has not seen land: the one that it lost,
    // or, when the loop was left, that of the chunk it was left at (not issued if
    // this thread's wait had given up: then this one runs out too).
    if (tid == kWW && tw.zimg && (zlost || issued < nchunk)) {
        const int z = zlost ? issued - 1 : issued;
        mbar_wait_bounded(&zbars[z & 1], (uint32_t)((z >> 1) & 1));
        atomicExch(&abort_flag, 1);
    }
    // the last commit completes after every MMA (after zlost there is none for the
    // last chunk: thread kWW waits for the one before, the others' wait runs out)
    const int last = issued - 1 - (zlost ? 1 : 0);
    if (last >= 0 && !mbar_wait_bounded(&bars[last & 1], (uint32_t)((last >> 1) & 1))) atomicExch(&abort_flag, 1);
    tc_fence_after();
    __syncthreads();  // abort_flag is final from here on
    const bool good = !abort_flag;
    if (wt && good && issued > 0) tcw_drain(tmem, lanes, tot, dc0, dc1, drained == 0);  // the last run
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    // the Hessian-like columns of this warp's lanes: IRLS rows = genes;
    // MLE rows 32 b + gene (b = warp % 4 < 3)
    if (wt) {
        const int b = MLE ? (warp & 3) : 0;
        const int lg = MLE ? (tid & 31) : gi;  // gene of this thread's tensor-memory lane
        const bool write = good && tile * GTn + lg < nact && (!MLE || b < 3);
        float* out = static_cast<float*>(geo.partW) + ((int64_t)seg * geo.slot_stride + tile * GTn + lg) * tw.NA +
                     b * tw.NE;
        for (int c = dc0; c < dc1; c += 8) {
            float v[8];
            if (issued > 0) {
                tc_ld8(tmem + lanes + tot + (uint32_t)c, v);
            } else {
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = 0.f;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int gp = zb * nblk + c + u;
                if (write && c + u < nblk && gp < tw.NE) out[gp] = v[u];
            }
        }
    }
    if (extra) {
        const bool write = good && valid_slot;
        float* out = static_cast<float*>(geo.partW) + ((int64_t)seg * geo.slot_stride + tile * GTn + gi) * tw.NA;
        if constexpr (MLE) {
            // the 8 quads' sums of each gene, added in quad order
            float* fred = reinterpret_cast<float*>(smem);                  // [8][32][2]
            double* dred = reinterpret_cast<double*>(smem + 8 * 32 * 2 * 4);  // [8][32][4]
            if (wt) {
                fred[(warp * 32 + gi) * 2 + 0] = fs[0];
                fred[(warp * 32 + gi) * 2 + 1] = fs[1];
#pragma unroll
                for (int j = 0; j < 4; ++j) dred[(warp * 32 + gi) * 4 + j] = sc[j];
            }
            __syncthreads();
            if (warp == 0 && write) {
                float f0 = 0.f, f1 = 0.f;
                double d[4] = {0.0, 0.0, 0.0, 0.0};
                for (int w = 0; w < 8; ++w) {
                    f0 += fred[(w * 32 + gi) * 2 + 0];
                    f1 += fred[(w * 32 + gi) * 2 + 1];
#pragma unroll
                    for (int j = 0; j < 4; ++j) d[j] += dred[(w * 32 + gi) * 4 + j];
                }
                out[3 * tw.NE + 0] = f0;
                out[3 * tw.NE + 1] = f1;
                double* os = geo.partS + ((int64_t)seg * geo.slot_stride + tile * GTn + gi) * 4;
#pragma unroll
                for (int j = 0; j < 4; ++j) os[j] = d[j];
            }
        } else {
            // the two halves of the cells: half 1 hands its sums to half 0
            // through the (idle) first operand stage
            float* red = reinterpret_cast<float*>(smem);  // [128 genes][XS]
            float v[XS];
#pragma unroll
            for (int i = 0; i < XS; ++i) {
                float a, b;
                unpack2(vab[i], a, b);
                v[i] = a + b;
            }
            if (wt && hh == 1) {
#pragma unroll
                for (int i = 0; i < XS; ++i) red[gi * XS + i] = v[i];
            }
            __syncthreads();
            if (wt && hh == 0 && write) {
#pragma unroll
                for (int i = 0; i < XS; ++i)
                    if (i < tw.P) out[tw.NE + i] = v[i] + red[gi * XS + i];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols)
                     : "memory");
    if (abort_flag && tid == 0) atomicExch(geo.err, 1);
}

template <int XS, class VT, bool MLE>
cudaError_t run_tcw(const PassLaunch& L, const TcwGeom& tw) {
    auto k = tcw_pass_kernel<XS, VT, MLE>;
    const int smem = tcw_smem<VT, MLE>(XS, tw.nblk);
    cudaError_t e = raise_dyn_smem(k, smem);
    if (e != cudaSuccess) return e;
    if (L.occ_out) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(L.occ_out, k, kWNT, smem);
    dim3 grid(L.nseg, L.ntiles, tcw_blocks(L.P));
    k<<<grid, kWNT, smem, L.stream>>>(L.geo, L.prm, tw);
    return cudaGetLastError();
}

template <class VT, bool MLE>
cudaError_t run_tcw_xs(const PassLaunch& L, const TcwGeom& tw) {
    switch (L.xs_pad) {
        case 8: return run_tcw<8, VT, MLE>(L, tw);
        case 12: return run_tcw<12, VT, MLE>(L, tw);
        case 16: return run_tcw<16, VT, MLE>(L, tw);
        case 20: return run_tcw<20, VT, MLE>(L, tw);
        case 24: return run_tcw<24, VT, MLE>(L, tw);
        case 28: return run_tcw<28, VT, MLE>(L, tw);
        case 32: return run_tcw<32, VT, MLE>(L, tw);
    }
    return cudaErrorInvalidValue;
}

// count rows of the dense image: one warp per gene
template <class VT>
__global__ void tcw_dense_kernel(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                                 const VT* __restrict__ val, int64_t G, int64_t ld, VT* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    for (int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < G;
         g += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        VT* row = out + g * ld;
        for (int64_t e = rowptr[g] + lane; e < rowptr[g + 1]; e += 32) row[col[e]] = val[e];
    }
}

// The products of every chunk and block z as the MMA reads them: [z][chunk][hi,
// lo][quad][row][4 cells], split as the kernel splits them.  Made once per fit:
// forming them per tile cost the 128 product threads more instructions a chunk
// than the weights cost the other 256 (8,500 genes x 30,000 cells, p = 16, first
// IRLS pass: 1,479 us with the products formed in the kernel, 1,033 with the
// image; first MLE pass 4,712 and 3,641).
__global__ void tcw_zimg_kernel(const float* __restrict__ xt, int64_t npad, int NE, int nblk, int nz, float* z) {
    const int64_t nch = npad / kWKC, total = (int64_t)nz * nch * nblk * 8;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int row = (int)(t % nblk);
        const int64_t u = t / nblk;
        const int q = (int)(u % 8);
        const int64_t v = u / 8;  // z * nch + chunk
        const int gp = (int)(v / nch) * nblk + row;
        float4 hz = make_float4(0.f, 0.f, 0.f, 0.f), lz = hz;
        if (gp < NE) {
            int j = (int)((sqrtf(8.f * (float)gp + 1.f) - 1.f) * 0.5f);
            while (j * (j + 1) / 2 > gp) --j;
            while ((j + 1) * (j + 2) / 2 <= gp) ++j;
            const int i = gp - j * (j + 1) / 2;
            const int64_t c = (v % nch) * kWKC + 4 * q;
            const float4 a = __ldg(reinterpret_cast<const float4*>(xt + (int64_t)i * npad + c));
            const float4 b = __ldg(reinterpret_cast<const float4*>(xt + (int64_t)j * npad + c));
            tf32_split(a.x * b.x, hz.x, lz.x);  // (xt holds cells 0, 2, 1, 3)
            tf32_split(a.z * b.z, hz.y, lz.y);
            tf32_split(a.y * b.y, hz.z, lz.z);
            tf32_split(a.w * b.w, hz.w, lz.w);
        }
        unsigned char* o = reinterpret_cast<unsigned char*>(z) + v * (2 * nblk * kWKC * 4);
        *reinterpret_cast<float4*>(o + stage_off(row, q, nblk)) = hz;
        *reinterpret_cast<float4*>(o + nblk * kWKC * 4 + stage_off(row, q, nblk)) = lz;
    }
}

// place of cell c in its quad: 0, 2, 1, 3 (the pairs of ld_quad)
DEV int64_t tcw_quad_pos(int64_t c) { return (c & ~(int64_t)3) | ((c & 1) << 1) | ((c >> 1) & 1); }

// feature rows of the design (zero past n and past p) and the offsets, the cells
// of a quad in the order of tcw_quad_pos:
// -1e30 past n, so that mu = 0 there and the padding cells of the last
// chunk add nothing to any sum (the products and the score vanish with
// x = 0 as well, the dispersion pass's scalar sums only with mu = 0)
__global__ void tcw_xt_kernel(const float* __restrict__ Xrm, int xs, int64_t n, int64_t npad,
                              const float* __restrict__ off, float* __restrict__ xt, float* __restrict__ offp) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < (int64_t)(xs + 1) * npad;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(t / npad);
        const int64_t c = t - (int64_t)i * npad;
        const int64_t at = tcw_quad_pos(c);
        if (i < xs) xt[(int64_t)i * npad + at] = c < n ? Xrm[c * xs + i] : 0.f;
        else offp[at] = c < n ? off[c] : -1e30f;
    }
}

__global__ void irls_rescue_kernel(const int32_t* iters_in, int64_t G, int limit, double beta_limit,
                                   const double* __restrict__ beta0, int P, double* beta, float* beta_f,
                                   int32_t* iters, int32_t* status, int32_t* act, int32_t* cnt, int32_t* flag) {
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < G; g += (int64_t)gridDim.x * blockDim.x) {
        double bmax = 0.0;
        for (int i = 0; i < P; ++i) bmax = fmax(bmax, fabs(beta[g * P + i]));
        const bool slow = iters_in[g] > limit || !(bmax <= beta_limit);
        flag[g] = slow ? 1 : 0;
        if (!slow) continue;
        act[atomicAdd(cnt, 1)] = (int32_t)g;
        for (int i = 0; i < P; ++i) {
            const double b = beta0[g * P + i];
            beta[g * P + i] = b;
            beta_f[g * P + i] = (float)b;
        }
        iters[g] = 0;
        status[g] = 0;
    }
}

__global__ void mask_i32_kernel(const int32_t* v, const int32_t* flag, int64_t G, int32_t* out) {
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < G; g += (int64_t)gridDim.x * blockDim.x)
        out[g] = flag[g] ? v[g] : 0;
}

}  // namespace

cudaError_t launch_irls_rescue_select(const int32_t* iters_in, int64_t G, int limit, double beta_limit,
                                      const double* beta0, int P, double* beta, float* beta_f, int32_t* iters,
                                      int32_t* status, int32_t* act, int32_t* cnt, int32_t* flag, cudaStream_t st) {
    if (G == 0) return cudaSuccess;
    irls_rescue_kernel<<<(unsigned)std::min<int64_t>((G + 255) / 256, 1024), 256, 0, st>>>(
        iters_in, G, limit, beta_limit, beta0, P, beta, beta_f, iters, status, act, cnt, flag);
    return cudaGetLastError();
}

cudaError_t launch_mask_i32(const int32_t* v, const int32_t* flag, int64_t G, int32_t* out, cudaStream_t st) {
    if (G == 0) return cudaSuccess;
    mask_i32_kernel<<<(unsigned)std::min<int64_t>((G + 255) / 256, 1024), 256, 0, st>>>(v, flag, G, out);
    return cudaGetLastError();
}

int tcw_blocks(int P) {
    const int ne = P * (P + 1) / 2;
    return (ne + kWNmax - 1) / kWNmax;
}
int tcw_nblk(int P) {
    const int ne = P * (P + 1) / 2, nb = tcw_blocks(P);
    return ((ne + nb - 1) / nb + 15) / 16 * 16;
}
int64_t tcw_npad(int64_t n) { return (n + kWKC - 1) / kWKC * kWKC; }
bool tcw_supported(int P, int xs) { return P >= 5 && P <= 32 && xs >= 8 && xs <= 32 && xs % 4 == 0; }

cudaError_t launch_tcw_prepare(const int64_t* rowptr, const int32_t* col, const void* val, int val_u16,
                               int64_t G, int64_t n, const float* Xrm, int xs, const float* off,
                               const TcwGeom& tw, cudaStream_t st) {
    const size_t esz = val_u16 ? 2 : 4;
    cudaError_t e = cudaMemsetAsync(const_cast<void*>(tw.ydense), 0, (size_t)G * tw.ld * esz, st);
    if (e != cudaSuccess) return e;
    if (G > 0) {
        const unsigned blocks = (unsigned)std::min<int64_t>((G * 32 + 255) / 256, 148 * 32);
        if (val_u16)
            tcw_dense_kernel<uint16_t><<<blocks, 256, 0, st>>>(rowptr, col, static_cast<const uint16_t*>(val), G,
                                                              tw.ld, static_cast<uint16_t*>(const_cast<void*>(tw.ydense)));
        else
            tcw_dense_kernel<float><<<blocks, 256, 0, st>>>(rowptr, col, static_cast<const float*>(val), G, tw.ld,
                                                           static_cast<float*>(const_cast<void*>(tw.ydense)));
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    const int64_t tot = (int64_t)(xs + 1) * tw.npad;
    tcw_xt_kernel<<<(unsigned)std::min<int64_t>((tot + 255) / 256, 148 * 16), 256, 0, st>>>(
        Xrm, xs, n, tw.npad, off, const_cast<float*>(tw.xt), const_cast<float*>(tw.offp));
    if (tw.zimg)
        tcw_zimg_kernel<<<148 * 16, 256, 0, st>>>(tw.xt, tw.npad, tw.NE, tw.nblk, tcw_blocks(tw.P),
                                                  const_cast<float*>(tw.zimg));
    return cudaGetLastError();
}
size_t tcw_zimg_bytes(int P, int64_t n) {
    return (size_t)tcw_blocks(P) * (size_t)(tcw_npad(n) / kWKC) * (size_t)(2 * tcw_nblk(P) * kWKC * 4);
}

int tcw_tile_genes(PassKind k) { return k == PASS_MLE ? kMleG : kWM; }

// L.GT = tcw_tile_genes(L.kind) genes per tile; grid (L.nseg, L.ntiles, tcw_blocks(P))
cudaError_t launch_tcw_pass(const PassLaunch& L, const TcwGeom& tw) {
    if ((L.kind != PASS_IRLS && L.kind != PASS_MLE) || L.GT != tcw_tile_genes(L.kind) ||
        !tcw_supported(L.P, L.xs_pad))
        return cudaErrorInvalidValue;
    TcwGeom t = tw;
    t.NA = pass_na(L.kind, L.P);
    if (L.occ_out) t.nblk = tcw_nblk(L.P);
    else if (tw.nblk != tcw_nblk(L.P) || tw.NE != L.P * (L.P + 1) / 2 || tw.P != L.P)
        return cudaErrorInvalidValue;
    if (L.kind == PASS_MLE)
        return L.val_u16 ? run_tcw_xs<uint16_t, true>(L, t) : run_tcw_xs<float, true>(L, t);
    return L.val_u16 ? run_tcw_xs<uint16_t, false>(L, t) : run_tcw_xs<float, false>(L, t);
}

}  // namespace devil
