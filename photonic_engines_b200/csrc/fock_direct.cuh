// Steps of few columns without plan or schedules: shared by the warp-per-stream and CTA forms and the cofactor step.
#pragma once

namespace pe {

constexpr int DIRECT_MAX = 8;  // CTA form: steps of at most this many columns sum over the chosen rows themselves

// One warp: the chosen rows [i0, i1) of the stream's instance into rows [i0, i1) of B, the first COLS columns of
// the chain at once: the direct steps after them read their blocks from shared memory.
template <int COLS, class SM>
static __device__ __forceinline__ void load_rows(SM& sm, const double2* __restrict__ A, int64_t rs, int64_t cs, int i0,
                                                 int i1, int nk) {
    const int lane = threadIdx.x & 31, j = lane & (COLS - 1);
    for (int i = i0 + lane / COLS; i < i1; i += 32 / COLS)
        if (j < nk) sm.B[i][j] = A[(int64_t)sm.rows[i] * rs + (int64_t)sm.cols[j] * cs];
}

// One warp: cofactors of a step of K <= 2 KH columns, FP64: Glynn's sum over the 2^(K1 - 1) sign vectors of the K1 chosen
// rows as they are (repeated rows are not collapsed), two threads per sign vector and 16 sign vectors
// at a time.  No multiplicities, plan or schedules: chains this short are bound by the
// instructions and latencies of that set-up, not by the sum (FP64 pipe 11 % busy with it).  256 circuits of at most 12
// photons, 1 000 shots each: 3.14 -> 1.75 ms; n = 6, m = 12, 10 000 chains: 100 -> 48 us.  In the CTA form one warp
// does it: 7 000 cycles of plan, schedules and sweep per step become about 1 500.  The sum over the lanes is halved: every
// exchange carries half of the values still held.
template <int KH, class WS>
__device__ __forceinline__ void cofactors_direct_kh(WS& sm, int K) {
    static_assert(KH <= 5, "the reduction over the lanes knows halves of one or two columns and odd KH");
    const int lid = threadIdx.x & 31, h = lid & 1, c0 = h * KH, K1 = K - 1;
    const int N = 1 << (K1 - 1);
    double ar[KH], ai[KH];
#pragma unroll
    for (int j = 0; j < KH; ++j) { ar[j] = 0.0; ai[j] = 0.0; }
    // sign vector t: bits 0-3 the lane's, the bits above walk a Gray code over the rounds (one row flips per round)
    const int tl = lid >> 1;
    double sr[KH], si[KH];
#pragma unroll
    for (int j = 0; j < KH; ++j) {
        const double2 b = sm.B[0][c0 + j];
        sr[j] = b.x;
        si[j] = b.y;
    }
    for (int i = 1; i < K1; ++i) {
        const double d = (i <= 4 && ((tl >> (i - 1)) & 1)) ? -1.0 : 1.0;
#pragma unroll
        for (int j = 0; j < KH; ++j) {
            const double2 b = sm.B[i][c0 + j];
            sr[j] = fma(d, b.x, sr[j]);
            si[j] = fma(d, b.y, si[j]);
        }
    }
#pragma unroll
    for (int j = 0; j < KH; ++j)                           // columns past K count as 1 (their B may be unset)
        if (c0 + j >= K) { sr[j] = 1.0; si[j] = 0.0; }
    double w = tl >= N ? 0.0 : ((__popc(tl) & 1) ? -1.0 : 1.0);
    term<KH, 2, double, double2>(sr, si, ar, ai, nullptr, 0.0, w, h, 0xffffffffu);
    for (int r = 1; r < (N >> 4); ++r) {
        const int q = __ffs(r) - 1;
        const double f = (((r ^ (r >> 1)) >> q) & 1) ? -2.0 : 2.0;
#pragma unroll
        for (int j = 0; j < KH; ++j) {
            const double2 b = sm.B[5 + q][c0 + j];
            const bool pad = c0 + j >= K;
            sr[j] = pad ? 1.0 : fma(f, b.x, sr[j]);
            si[j] = pad ? 0.0 : fma(f, b.y, si[j]);
        }
        w = -w;
        term<KH, 2, double, double2>(sr, si, ar, ai, nullptr, 0.0, w, h, 0xffffffffu);
    }
    // lanes with bit 4 clear keep the real parts, the others the imaginary ones; then (KH 2, 4) half of the columns
    const bool im = (lid & 16) != 0;
    double v[KH];
#pragma unroll
    for (int j = 0; j < KH; ++j) {
        const double give = im ? ar[j] : ai[j];
        v[j] = (im ? ai[j] : ar[j]) + __shfl_xor_sync(0xffffffffu, give, 16);
    }
    const double scale = __longlong_as_double((long long)(1023 - (K1 - 1)) << 52);      // 2^-(K1 - 1)
    double* P = reinterpret_cast<double*>(&sm.P[0]);
    if constexpr (KH % 2 == 0) {
        constexpr int KQ = KH / 2;
        const int up = (lid >> 3) & 1;
        double x[KQ];
#pragma unroll
        for (int j = 0; j < KQ; ++j) {
            const double give = up ? v[j] : v[KQ + j];
            x[j] = (up ? v[KQ + j] : v[j]) + __shfl_xor_sync(0xffffffffu, give, 8);
        }
        double y;
        int col = c0 + up * KQ;
        if constexpr (KQ == 2) {
            const int up2 = (lid >> 2) & 1;
            const double give = up2 ? x[0] : x[1];
            y = (up2 ? x[1] : x[0]) + __shfl_xor_sync(0xffffffffu, give, 4);
            col += up2;
        } else {
            y = x[0] + __shfl_xor_sync(0xffffffffu, x[0], 4);
        }
        y += __shfl_xor_sync(0xffffffffu, y, 2);
        if (!(lid & 2) && (KQ == 2 || !(lid & 4))) P[2 * col + (im ? 1 : 0)] = y * scale;
    } else {
#pragma unroll
        for (int j = 0; j < KH; ++j) {
#pragma unroll
            for (int o = 8; o > 1; o >>= 1) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
            if (!(lid & 14)) P[2 * (c0 + j) + (im ? 1 : 0)] = v[j] * scale;
        }
    }
    __syncwarp();
}

template <int KMAX, class WS>
__device__ __forceinline__ void cofactors_direct(WS& sm, int K) {             // K <= KMAX
    if (K <= 4) { cofactors_direct_kh<2>(sm, K); return; }
    if (K <= 6) { cofactors_direct_kh<3>(sm, K); return; }
    if constexpr (KMAX <= 8) {
        cofactors_direct_kh<4>(sm, K);
    } else {
        static_assert(KMAX <= 10, "five columns per thread at most");
        if (K <= 8) cofactors_direct_kh<4>(sm, K);
        else cofactors_direct_kh<5>(sm, K);
    }
}

// One stream's slice of shared memory for direct steps of a warp.
struct DirectSmem {
    double2 P[DIRECT_MAX];
    double2 B[DIRECT_MAX][DIRECT_MAX];
    int rows[DIRECT_MAX];
    int cols[DIRECT_MAX];
};

}  // namespace pe
