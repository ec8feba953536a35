// FP64 Schur update on the 5th-generation tensor cores (sm_100a) by splitting
// the operands into 8-bit integer digits.
//
//     C(rows, cols) -= (L D)(rows, K) * L(cols, K)'        (LMMY18, lmmy18.f:5-192)
//
// With M = L |D|^(1/2) the update is C -= sum_k sign(d_k) M_ik M_jk.  Row i of M
// is brought to fixed point with one exponent E_i for the whole of K:
// X = M 2^(55-E_i) rounded to an integer |X| <= 127 * 2^48, which is seven
// balanced base-256 digits (each in [-128, 127]).  The products of digits p
// and q are exact integers, their sums over K are exact in 32 bits for K <=
// kI8MaxK, and the sums of one level s = p + q share a TMEM accumulator: levels
// 0..7, i.e. 34 of the 49 digit products (the splitting of Ozaki, Ogita, Oishi
// and Rump, "Error-free transformations of matrix multiplication by using fast
// routines of matrix multiplication", 2012, with integer digits).
// What is lost, per term of the sum unless said otherwise:
//   operands  each rounded by up to 2^-56 2^E: 2^-56 (2^E_i |M_jk| + 2^E_j |M_ik|), at most
//             2^-55 2^(E_i+E_j); the leading part
//   levels    8 .. 12, left out: at most 2^-61.6 2^(E_i+E_j), typically 2^-64 (with levels 0 .. 6
//             alone, 28 products, at most 2^-53.4, typically 2^-56, and the factor's error against
//             an 80-bit factorisation came out up to 13 % larger than k_gemm's)
//   sum       rounded once to FP64; before that its levels 6 and 7 to 2^-59 2^(E_i+E_j)
// where the FP64 multiply-adds of k_gemm round every partial sum, by up to 2^-53 of its size.
// The measure is the rows' scales and not a term's own size: an entry 2^-20 of its row's
// largest keeps 35 bits, and two rows whose large entries lie in different columns have
// a sum that is less accurate than k_gemm's relative to itself, though not to
// |M_i| |M_j|, by which the update of the diagonal is rounded.  Measured: one update's
// errors (root mean square) are 1/7, 1/15 and 1/26 of k_gemm's at K = 128, 512 and 1600, for
// rows whose entries span six decades 1/3, 1/5 and 1/9; solutions against ones refined with
// 80-bit residuals (16^3 to 48^3, shifted and not, 60 right-hand sides) 0.93 of those with
// k_gemm alone (geometric mean).
//
// Two kernels per update:
//   k_split_i8  forms the digits of a panel: slabs of 128-column blocks,
//               [k block][digit][row][128 bytes], and the row scales 2^(E_i-31);
//               a second slab with the signs of D where a pivot is negative;
//   k_gemm_i8   CTAs over the lower 128x64 tiles: a TMA warp streams, per block
//               of 128 columns, the seven 64x128 digit tiles of the columns (double
//               buffered) and the seven 128x128 digit tiles of the rows (one buffer per
//               digit), one thread issues tcgen05.mma kind::i8 - digit p of the rows
//               against the digits 0 .. 7-p of the columns (N up to 256 an
//               instruction), which land in the levels p .. 7 - and sixteen epilogue
//               warps put the levels of an entry together in 64-bit integers,
//               scale them and subtract from the FP64 front.
// Every mbarrier wait is bounded like those of k_gemm_tc.
#pragma once

namespace i8 {
using namespace tc;                           // mbarrier, TMA, TMEM helpers

constexpr int kM = kI8TileM, kN = kI8TileN, kK = kI8BK;      // 128 x 64 tile, 128-byte K blocks
constexpr int kDig = kI8Digits;               // digits of an entry
constexpr int kLev = 8;                       // levels p + q = 0 .. 7: 8 x 64 TMEM columns
constexpr int kABytes = kM * kK;              // 16 KB
constexpr int kBBytes = kN * kK;              // 8 KB, seven of them contiguous
constexpr size_t kSmemI8 = 1024 + (size_t)kDig * (2 * kBBytes + kABytes);
constexpr int kEpiWarps = 16;                 // four per TMEM quadrant, 16 columns each
constexpr int kEpiCols = kN / (kEpiWarps / 4);
constexpr int kThreadsI8 = 32 * (2 + kEpiWarps);
// D s32, A and B signed 8-bit, both K-major, M = 128; N is added per instruction
constexpr uint32_t kIdescI8 = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kM >> 4) << 24);
// N = n column digits
__device__ __forceinline__ constexpr uint32_t idesc(int n) { return kIdescI8 | ((uint32_t)(n * kN >> 3) << 17); }

__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

// 32 lanes x 4 consecutive 32-bit columns, without the wait
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, int (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}

// Lower tiles of an nr x nct grid of 128 x 64 tiles: row tile it has the
// column tiles 0 .. min(nct, 2 it + 2) - 1.  Taken in groups of kI8Group column
// tiles, row by row inside a group, so that the CTAs running together share
// operand slabs in L2.
constexpr int kI8Group = 16;
__device__ __forceinline__ void tile_of_i8(int64_t u, int nct, int nr, int& it, int& jt) {
    for (int g0 = 0;; g0 += kI8Group) {
        const int w = min(kI8Group, nct - g0), t0 = g0 >> 1, T = nr - t0, h = w >> 1;
        const int64_t tri = (int64_t)h * (h + 1);               // rows t0 .. t0 + h - 1: 2, 4, ..., 2h tiles
        const int64_t cnt = T <= h ? (int64_t)T * (T + 1) : tri + (int64_t)(T - h) * w;
        if (u < cnt || g0 + w >= nct) {
            if (u < tri) {
                int t = (int)((sqrtf(4.0f * (float)u + 1.0f) - 1.0f) * 0.5f);
                while ((t + 1) * (t + 2) <= u) ++t;
                while (t * (t + 1) > u) --t;
                it = t0 + t;
                jt = g0 + (int)(u - t * (t + 1));
            } else {
                it = t0 + h + (int)((u - tri) / w);
                jt = g0 + (int)((u - tri) % w);
            }
            return;
        }
        u -= cnt;
    }
}

__device__ __forceinline__ int k_blocks_i8(const Job& jb) { return (jb.k_hi - jb.k_lo + kK - 1) / kK; }

// What the split leaves in a job's flag: 0, 1 with a negative pivot, or that the
// front's update is left out.  k_gemm_i8 goes by this alone: PV::sn_bad may change
// while the columns beyond the next super-panel run beside the same front's panel
// chain, and the roles of a CTA, each on its own way through the tiles, have to
// agree on the ones that are skipped.  A front that fails after its split
// gets the rest of that update, which nobody reads.
constexpr double kOffI8 = -1.0;
__device__ __forceinline__ bool off_i8(const Job& jb, const double* scales) { return scales[jb.aux_job] < 0.0; }

// 2^e for -1022 <= e <= 1023
__device__ __forceinline__ double pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }

}  // namespace i8

// Digits of 32 rows of a job's panel, all of its K, by 256 threads (lane =
// row, a warp per column quad).  The first pass over K finds each row's
// largest |M|, the second (from L2) writes the digits, 128 columns at a
// time, through shared memory so that both sides are coalesced.
// P.sqd holds sign(d) sqrt|d| and its rounding error, so that M carries more
// than 53 bits into the rounding to X.
__global__ void __launch_bounds__(256) k_split_i8(const Job* jobs, int64_t njobs, const int32_t* tmap, PV P, uint8_t* slab,
                                                  double* scales) {
    using namespace i8;
    __shared__ uint32_t dig[kDig][32][kK / 4 + 1];
    __shared__ uint32_t red[8][32];
    if (P.st->any_fail) return;
    const int64_t task = blockIdx.x;
    const Job& jb = job_of(jobs, njobs, tmap, task);
    const int js = jb.node;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rb = (int)(task - jb.task0);
    if (P.sn_bad[js] || node_off(P, js)) {
        if (rb == 0 && tid == 0) scales[jb.aux_job] = kOffI8;
        return;
    }
    const int K = jb.k_hi - jb.k_lo, nkb = k_blocks_i8(jb);
    const int64_t np = jb.np, ld = P.buf_ld[js];
    const int r = jb.c0 + rb * 32 + lane;
    const bool in = r < jb.r_end;
    const double* src = P.arena + P.buf_off[js] + (int64_t)jb.k_lo * ld + (in ? r : jb.c0);
    const double2* sq = reinterpret_cast<const double2*>(P.sqd) + P.fst[js] + jb.k_lo;
    // pass 1: the high words of |M| order like the values (a NaN or Inf comes last)
    uint32_t top = 0;
    int neg = 0;
#pragma unroll 8
    for (int k = warp; k < K; k += 8) {
        const double s = __ldg(&sq[k].x);
        const double m = __ldcg(src + (int64_t)k * ld) * s;
        top = max(top, (uint32_t)__double2hiint(m) & 0x7fffffffu);
        neg |= s < 0.0;
    }
    red[warp][lane] = top;
    neg = __syncthreads_or(neg);
#pragma unroll
    for (int w = 0; w < 8; ++w) top = max(top, red[w][lane]);
    const bool bad = top >= 0x7ff00000u;
    // |M| <= 127/128 2^E: the biased exponent - 1022, one more where the mantissa is 63/64 or above
    int E = (int)(top >> 20) - 1022 + ((top & 0xfffffu) >= 0xfc000u ? 1 : 0);
    E = max(E, -900);
    if (warp == 0) {
        if (rb == 0 && lane == 0) scales[jb.aux_job] = neg ? 1.0 : 0.0;
        scales[jb.aux + rb * 32 + lane] = in ? (bad ? __longlong_as_double(0x7ff8000000000000ll) : pow2(E - 31)) : 0.0;
    }
    const double scale = (in && !bad) ? pow2(55 - E) : 0.0;
    for (int kb = 0; kb < nkb; ++kb) {
        double l[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            const int k = kb * kK + 4 * (warp + 8 * (u >> 2)) + (u & 3);
            l[u] = (in && k < K) ? __ldcg(src + (int64_t)k * ld) : 0.0;
        }
        long long x[16];
        uint32_t flip = 0;
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            const int k = kb * kK + 4 * (warp + 8 * (u >> 2)) + (u & 3);
            double2 s = make_double2(0.0, 0.0);
            if (k < K) s = __ldg(sq + k);
            if (s.x < 0.0) flip |= 1u << u;
            const double a = l[u] * scale;                       // exact: a power of two
            const double as = fabs(s.x);
            const double p = __dmul_rn(a, as);
            const double t = fma(a, as, -p) + a * copysign(1.0, s.x) * s.y;   // M's part below p's rounding
            const long long xi = bad ? 0 : __double2ll_rn(p);
            x[u] = bad ? 0 : xi + __double2ll_rn((p - __ll2double_rn(xi)) + t);
        }
        for (int side = 0; side < (neg ? 2 : 1); ++side) {
            // balanced digits: the bytes of x + 0x80..80, each minus 128 (its top bit flipped)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                unsigned long long y[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const long long xv = (side && (flip >> (4 * v + c) & 1u)) ? -x[4 * v + c] : x[4 * v + c];
                    y[c] = ((unsigned long long)xv + 0x0080808080808080ull) ^ 0x0080808080808080ull;
                }
#pragma unroll
                for (int d = 0; d < kDig; ++d) {
                    const int sh = 8 * (kDig - 1 - d);           // digit 0 is the leading one
                    uint32_t word = 0;
#pragma unroll
                    for (int c = 0; c < 4; ++c) word |= ((uint32_t)(y[c] >> sh) & 0xffu) << (8 * c);
                    dig[d][lane][warp + 8 * v] = word;
                }
            }
            __syncthreads();
            uint8_t* out = slab + (jb.slab + ((int64_t)side * nkb + kb) * kDig * np + rb * 32) * kK;
#pragma unroll
            for (int q = 0; q < kDig; ++q) {                     // 32 rows x 128 bytes per digit
                const int rr = tid >> 3, c4 = 4 * (tid & 7);
                const uint32_t* w = &dig[q][rr][c4];
                *reinterpret_cast<uint4*>(out + ((int64_t)q * np + rr) * kK + 4 * c4) =
                    make_uint4(w[0], w[1], w[2], w[3]);
            }
            __syncthreads();
        }
    }
}

// map_a: boxes of 128 x 128 bytes, map_b: boxes of 64 x 128 bytes, over one slab arena.
__global__ void __launch_bounds__(i8::kThreadsI8, 1)
    k_gemm_i8(const Job* jobs, int64_t njobs, const int32_t* tmap, int64_t ntasks, PV P, const double* scales,
              const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b) {
    using namespace i8;
    extern __shared__ uint8_t i8_raw[];
    __shared__ uint64_t bars[2 * kDig + 4 + 3];
    __shared__ double scol[2][kN];                     // column scales of a tile and the next
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    if (P.st->any_fail) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = (smem_u32(i8_raw) + 1023u) & ~1023u;
    const uint32_t sb = base, sa = base + 2u * kDig * kBBytes;
    const uint32_t afull = smem_u32(&bars[0]), aempty = smem_u32(&bars[kDig]);
    const uint32_t bfull = smem_u32(&bars[2 * kDig]), bempty = bfull + 16;
    const uint32_t accf = bfull + 32, acce = accf + 8, drain = accf + 16;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kDig; ++s) {
            mbar_init(afull + 8 * s, 1);
            mbar_init(aempty + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(bfull + 8 * b, 1);
            mbar_init(bempty + 8 * b, 1);
        }
        mbar_init(accf, 1);
        mbar_init(acce, kEpiWarps);
        mbar_init(drain, 1);                              // MMA drain before the TMEM is freed
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_slot;

    if (warp == 0 && lane == 0) {
        // ---- TMA producer
        uint32_t issued = 0;                              // 8 K block + digit, of the last row load, + 1
        uint32_t g = 0;                                   // K blocks so far
        bool stop = false;
        for (int64_t task = blockIdx.x; task < ntasks && !stop && !*(volatile int*)&failed; task += gridDim.x) {
            const Job& jb = job_of(jobs, njobs, tmap, task);
            if (off_i8(jb, scales)) continue;
            int it, jt;
            tile_of_i8(task - jb.task0, (jb.c_end - jb.c0 + kN - 1) / kN, (jb.r_end - jb.c0 + kM - 1) / kM, it, jt);
            const int nkb = k_blocks_i8(jb), np = jb.np;
            const int wofs = scales[jb.aux_job] != 0.0 ? nkb * kDig * np : 0;   // signed row slab
            int ya = (int)jb.slab + wofs + it * kM, yb = (int)jb.slab + jt * kN;
            for (int kb = 0; kb < nkb && !stop; ++kb, ++g) {
                const uint32_t b = g & 1u, bf = bfull + 8 * b;
                if (g >= 2 && !mbar_wait(bempty + 8 * b, ((g >> 1) - 1) & 1u, P.wait_ns)) {
                    stop = true;
                    break;
                }
                if (!(P.tc_drop && blockIdx.x == 0 && g == 0)) {          // watchdog test: never loaded
                    mbar_expect_tx(bf, kDig * kBBytes);
                    const uint32_t dst = sb + b * (uint32_t)(kDig * kBBytes);
#pragma unroll
                    for (int d = 0; d < kDig; ++d, yb += np) tma_load_2d(dst + d * kBBytes, &map_b, bf, 0, yb);
                } else {
                    yb += kDig * np;
                }
#pragma unroll
                for (int d = 0; d < kDig; ++d, ya += np) {
                    if (g >= 1 && !stop && !mbar_wait(aempty + 8 * d, (g - 1) & 1u, P.wait_ns)) stop = true;
                    if (!stop) {
                        mbar_expect_tx(afull + 8 * d, kABytes);
                        tma_load_2d(sa + d * kABytes, &map_a, afull + 8 * d, 0, ya);
                        issued = 8 * g + d + 1;
                    }
                }
            }
        }
        if (stop) failed = 1;
        // drain: what was issued must have landed before exit (the last use of
        // each buffer; an earlier one has been consumed)
        for (int d = 0; d < kDig; ++d)
            if (issued > (uint32_t)d) {
                const uint32_t last = (issued - 1 - d) >> 3;            // last K block whose digit d was issued
                mbar_wait(afull + 8 * d, last & 1u, P.wait_ns);
            }
        if (issued) {
            const uint32_t last = (issued - 1) >> 3;
            mbar_wait(bfull + 8 * (last & 1u), (last >> 1) & 1u, P.wait_ns);
            if (last) mbar_wait(bfull + 8 * ((last - 1) & 1u), ((last - 1) >> 1) & 1u, P.wait_ns);
        }
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer
        uint32_t g = 0, tile = 0;
        bool stop = false;
        const uint64_t ad0 = sw128_desc(sa), bd0 = sw128_desc(sb);
        for (int64_t task = blockIdx.x; task < ntasks && !stop; task += gridDim.x) {
            const Job& jb = job_of(jobs, njobs, tmap, task);
            if (off_i8(jb, scales)) continue;
            const int nkb = k_blocks_i8(jb);
            if (tile >= 1 && !mbar_wait(acce, (tile - 1) & 1u, P.wait_ns)) {
                stop = true;
                break;
            }
            fence_after_sync();
            for (int kb = 0; kb < nkb && !stop; ++kb, ++g) {
                const uint32_t b = g & 1u;
                if (!mbar_wait(bfull + 8 * b, (g >> 1) & 1u, P.wait_ns) || *(volatile int*)&failed) {
                    stop = true;
                    break;
                }
                const uint64_t bd = bd0 + (uint64_t)(b * (kDig * kBBytes >> 4));
                const uint32_t first = kb ? 1u : 0u;
                // straight-line code: every descriptor is a constant away from the
                // base ones, so that one thread issues faster than the MMAs run
#pragma unroll
                for (int p = 0; p < kDig; ++p) {
                    if (!stop && !mbar_wait(afull + 8 * p, g & 1u, P.wait_ns)) stop = true;
                    if (!stop) {
                        fence_after_sync();
                        // digits q = 0 .. min(6, 7 - p) of the columns, levels p + q: four
                        // digits in the first instruction, the rest in the second
                        const int cnt = kDig < kLev - p ? kDig : kLev - p, n0 = cnt < 4 ? cnt : 4, n1 = cnt - n0;
                        const uint64_t ad = ad0 + (uint64_t)(p * kABytes >> 4);
                        constexpr uint64_t bq = (uint64_t)(kBBytes >> 4);
#pragma unroll
                        for (int kk = 0; kk < kK / 32; ++kk) {
                            const uint64_t adv = (uint64_t)(kk * 32) >> 4;
                            const uint32_t add = (p | kk) ? 1u : first;       // digit 0 opens the levels 0 .. 6
                            mma_i8(tmem + (uint32_t)(kN * p), ad + adv, bd + adv, idesc(n0), add);
                            if (p == 1 && kk == 0) {                          // and digit 1 the last level
                                mma_i8(tmem + (uint32_t)(kN * 5), ad + adv, bd + adv + 4 * bq, idesc(2), 1u);
                                mma_i8(tmem + (uint32_t)(kN * 7), ad + adv, bd + adv + 6 * bq, idesc(1), first);
                            } else if (n1 > 0) {
                                mma_i8(tmem + (uint32_t)(kN * (p + 4)), ad + adv, bd + adv + 4 * bq, idesc(n1), add);
                            }
                        }
                        mma_commit(aempty + 8 * p);
                    }
                }
                mma_commit(bempty + 8 * b);
            }
            if (stop) break;
            mma_commit(accf);
            ++tile;
        }
        if (stop) failed = 1;
        mma_commit(drain);
        if (!mbar_wait(drain, 0u, P.wait_ns)) failed = 1;
    } else if (warp >= 2) {
        // ---- epilogue: TMEM lanes 32 (warp % 4) .. + 31, kEpiCols of the 64 columns each.
        // The front's entries and the column scales are loaded before the wait for
        // the products, so that a tile's TMEM is free again after the reads and
        // the arithmetic alone (8192-row block, split included: K = 512 0.61 -> 0.46 ms,
        // K = 2048 1.60 -> 1.53 ms).
        const int q = warp & 3, h = (warp - 2) >> 2;
        const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(kEpiCols * h);
        uint32_t tile = 0;
        for (int64_t task = blockIdx.x; task < ntasks; task += gridDim.x) {
            const Job& jb = job_of(jobs, njobs, tmap, task);
            const int js = jb.node;
            if (off_i8(jb, scales)) continue;
            int it, jt;
            tile_of_i8(task - jb.task0, (jb.c_end - jb.c0 + kN - 1) / kN, (jb.r_end - jb.c0 + kM - 1) / kM, it, jt);
            const int row = it * kM + 32 * q + lane, col0 = jt * kN + kEpiCols * h;
            const int r = jb.c0 + row, c0 = jb.c0 + col0;
            // columns of this thread's row that belong to the lower triangle of the block
            const int ncol = r < jb.r_end ? min(kEpiCols, min(jb.c_end - c0, r - c0 + 1)) : 0;
            const int64_t ld = P.buf_ld[js];
            const double* sc = scales + jb.aux;
            double* dst = P.arena + P.buf_off[js] + r + (int64_t)c0 * ld;
            double cv[kEpiCols];
#pragma unroll
            for (int t = 0; t < kEpiCols; ++t) cv[t] = t < ncol ? __ldcg(dst + (int64_t)t * ld) : 0.0;
            const double si = sc[row];
            // (the four quadrants' warps write the same values; a warp is never
            // two tiles ahead of another)
            double* sj = &scol[tile & 1u][kEpiCols * h];
            if (lane < kEpiCols) sj[lane] = 16.0 * sc[col0 + lane];
            __syncwarp();
            if (!mbar_wait(accf, tile & 1u, P.wait_ns) || *(volatile int*)&failed) {
                failed = 1;
                break;
            }
            ++tile;
            fence_after_sync();
#pragma unroll
            for (int c4 = 0; c4 < kEpiCols; c4 += 4) {
                int lv[kLev][4];
#pragma unroll
                for (int s = 0; s < kLev; ++s) tmem_ld4(lane_base + (uint32_t)(kN * s + c4), lv[s]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    // sum of level s times 256^(6-s): the leading three levels (47 bits) and, with
                    // levels 6 and 7 rounded to 16, the others (51 bits) as exact doubles
                    const long long magic = 0x4338000000000000ll;        // 1.5 2^52
                    const long long hi = (long long)lv[0][t] * 65536 + ((long long)lv[1][t] * 256 + (magic + lv[2][t]));
                    const long long lo = (long long)lv[3][t] * (1 << 20) +
                                         ((long long)lv[4][t] * (1 << 12) +
                                          ((long long)lv[5][t] * (1 << 4) +
                                           (magic + ((lv[6][t] + ((lv[7][t] + 128) >> 8) + 8) >> 4))));
                    const double v = fma(__longlong_as_double(hi) - 6755399441055744.0, 268435456.0,
                                         __longlong_as_double(lo) - 6755399441055744.0);
                    cv[c4 + t] -= (v * si) * sj[c4 + t];
                }
            }
            fence_before_sync();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acce) : "memory");
#pragma unroll
            for (int t = 0; t < kEpiCols; ++t)
                if (t < ncol) dst[(int64_t)t * ld] = cv[t];
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && failed) atomicExch(&P.st->tc_timeout, 1);
    if (warp == 1) {
        fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}
