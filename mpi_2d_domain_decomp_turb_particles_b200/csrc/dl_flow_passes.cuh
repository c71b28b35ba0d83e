// The passes of the flow step along z, y and x for the grids dl_fft.cuh transforms
// (included by dl_flow.cu inside its namespace, after Grid).
//
// The spectral state is dealiased to the sphere k^2 <= nek (nek + 1) (shell int(|k| + 1/2) <=
// nek = int(n/2 - 3/2)), so only the columns (kx, ky) inside its circle are transformed along
// z and along y only the kx <= nek: 0.79 of the spectral plane, and 0.52 of the box for the
// state itself.  One step moves, in units of one spectral component (16 n^2 n/2 bytes):
//   k_ypass (+)      read 6 x 0.79, write 6     curl u and u, ky -> y
//   k_xpass          read 6, write 3 (+ u, + the droplet field)   kx -> x, u x omega, x -> kx
//   k_ypass (-)      read 3, write 3 x 0.79     N, y -> ky
//   k_zforward       read and write 3 x 0.79    N, z -> kz
//   k_update_sphere  read 9 x 0.52, write 6 x 0.52
//   k_zinverse       read 3 x 0.52, write 6 x 0.79   the next step's u^ and curl u^, kz -> z
// Work arrays: W[6][y][z][n/2], curl u (0..2) and u (3..5) transformed along z (N in 0..2 between
// the y pass and the update); P[6][z][y][n/2], transformed along z and y (in place in W the y
// passes would save P and take 8 % longer).
// Columns kx = n/2 and everything outside the circle are neither written nor read.
// Rows are read and written 8 kx at a time (128 bytes): the load/store unit takes a wavefront
// per 128-byte line, and narrower tiles double them.  That, and the few threads that three
// components in shared memory leave per SM, is why the forward transform, update and inverse
// transform along z are three kernels: as one (13.3 components moved instead of 18.8, 4 kx x 3
// components per block) they took 0.65 ms at 256^3 and 6.9 ms at 512^3.

__host__ __device__ __forceinline__ int sphere_lim(int nek) { return nek * (nek + 1); }
__device__ __forceinline__ int wave(int i, int n) { return i <= n / 2 ? i : i - n; }

// padded slot of a line element: R0-strided stage writes of neighbouring threads fall into
// different 16-byte banks
template <class P>
__device__ __forceinline__ int slot_at(int i) { return i + i / P::R0; }
template <class P>
__host__ __device__ constexpr int slot_len() { return P::N + P::N / P::R0; }

// modes per y plane of W: n * n/2 and WPAD more, so that the y lines of a grid 2^a do not step
// by a power of two bytes (2^19 at 256^3), which would map them onto few L2 sets
constexpr int WPAD = 8;
template <int N>
__host__ __device__ constexpr int64_t w_plane() { return (int64_t)N * (N / 2) + WPAD; }

// ---- y ------------------------------------------------------------------------------------
// 8 kx (one 128-byte row) x all y of one field and z plane per block.  Bound by DRAM: 0.24 ms for
// six fields at 256^3 (1.44 GB, 6.0 TB/s), 0.12 for three; the library's strided passes ran at 5.9
// TB/s over the whole spectrum
template <int N, int SIGN>
__global__ void __launch_bounds__(8 * dlfft::Wide<N>::T) k_ypass(double2 *__restrict__ W, double2 *__restrict__ planes,
                                                                  int nek, const double2 *__restrict__ tw)
{
    using P = dlfft::Wide<N>;
    constexpr int H = N / 2, L = P::S - 1, E = dlfft::elems<P>();
    extern __shared__ double2 sm[];
    const int xi = threadIdx.x & 7, t = threadIdx.x >> 3;
    const int x = blockIdx.x * 8 + xi, z = blockIdx.y, f = blockIdx.z;
    double2 *w = W + (int64_t)f * N * w_plane<N>() + z * H + x, *p = planes + ((int64_t)f * N + z) * N * H + x;
    const int lim = sphere_lim(nek) - x * x;   // ky^2 <= lim inside the circle
    double2 v[E];
    dlfft::each<P, 0>(t, [&](int i, int m) {
        const int y = dlfft::in_at<P, 0>(t, i, m), ky = wave(y, N);
        double2 a = make_double2(0.0, 0.0);
        if (SIGN > 0) {
            if (ky * ky <= lim) a = w[y * w_plane<N>()];
        } else if (x <= nek) a = p[y * H];
        v[i * dlfft::Stage<P, 0>::R + m] = a;
    });
    dlfft::line<P, SIGN>(t, v, sm, [xi](int i) { return slot_at<P>(i) * 8 + xi; }, tw, dlfft::BlockSync());
    dlfft::each<P, L>(t, [&](int i, int m) {
        const int y = dlfft::out_at<P, L>(t, i, m), ky = wave(y, N);
        const double2 a = v[i * dlfft::Stage<P, L>::R + m];
        if (SIGN > 0) {
            if (x <= nek) p[y * H] = a;
        } else if (ky * ky <= lim) w[y * w_plane<N>()] = a;
    });
}

// ---- x ------------------------------------------------------------------------------------
template <int N> using XPlan = dlfft::Narrow<N>;
struct XArgs {
    double2 *P;          // [6][z][y][n/2]
    int nek;
    double *vel;         // [3][n^3]
    void *fp;            // droplet field (padded), or null
    int64_t fpy, fpz, fpc;
    double *diss;        // DISSIP result [n^3]
    double nu2;          // 2 nu
    const double2 *tw;
};
constexpr int X_STEP = 0, X_EMIT32 = 1, X_EMIT64 = 2, X_DISS = 3;

// pairs of rows per block
template <int N>
__host__ __device__ constexpr int x_units() { return N <= 64 ? (N == 32 ? 8 : 4) : 64 / XPlan<N>::T; }
template <int N>
__host__ __device__ constexpr int x_threads() { return 3 * XPlan<N>::T * x_units<N>(); }
// blocks per SM that the registers are cut for: 80 a thread at 8 elements (168 at the 12 of 96)
template <int N>
__host__ __device__ constexpr int x_blocks() { return dlfft::elems<XPlan<N>>() > 8 ? 2 : 4; }
template <int N>
__host__ __device__ constexpr int x_smem() { return x_units<N>() * 6 * slot_len<XPlan<N>>() * 16; }

template <typename F>
__device__ __forceinline__ void emit_value(F *row, int x, int n, double u)
{
    row[x + DL_PAD_LO] = (F)u;
    const int xi = pad_image(x, n);
    if (xi >= 0) row[xi] = (F)u;
}

// Two rows (y, y + 1) of one z plane per group of 3 T threads.  The half spectra A, B of two
// real lines go through one complex transform of A + i B: thread group p takes component p of
// both rows, for the velocity, for the vorticity and for N, 4.5 transforms per row.  Both
// lines of a pair round at the larger one's magnitude, so they are of one component (the
// transforms along z and y have rounded its rows alike): beside another component a small one
// would lose their ratio, and one that is zero would not stay so (and the components (0, 1) of a
// row took 0.49 ms at 256^3).
// Bound by the load/store unit and the latency of its phases: 31 16-byte accesses of the SM per
// element and thread group with three stages (0.34 ms at 256^3), 1.6 GB of DRAM (0.25 ms); 0.47 ms,
// where the library's x transforms and the cross-product kernel took 0.78.
template <int N, int MODE>
__global__ void __launch_bounds__(x_threads<N>(), x_blocks<N>()) k_xpass(XArgs A)
{
    using P = XPlan<N>;
    constexpr int H = N / 2, T = P::T, L = P::S - 1, E = dlfft::elems<P>();
    constexpr int SL = slot_len<P>(), RI = dlfft::Stage<P, 0>::R, RO = dlfft::Stage<P, L>::R;
    extern __shared__ double2 sm[];
    const int unit = threadIdx.x / (3 * T), p = (threadIdx.x / T) % 3, t = threadIdx.x % T;
    const int y0 = (blockIdx.x * x_units<N>() + unit) * 2, z = blockIdx.y;
    const dlfft::LineSync<T> sync{unit * 3 + p};
    double2 *reg = sm + unit * 6 * SL;   // lines of the velocity (0..2) and the vorticity (3..5)
    constexpr int64_t fstride = (int64_t)N * N * H;
    double2 *rows = A.P + ((int64_t)z * N + y0) * H;
    const auto at = [](int i) { return slot_at<P>(i); };
    double2 v[E];
#pragma unroll 1
    for (int r = 0; r < 2; r++) {
        const double2 *a = rows + (p + 3 - 3 * r) * fstride, *b = a + H;
        dlfft::each<P, 0>(t, [&](int i, int m) {
            const int k = dlfft::in_at<P, 0>(t, i, m);
            const int kk = k <= H ? k : N - k;
            double2 q = make_double2(0.0, 0.0);
            if (kk <= A.nek) {
                const double2 c = a[kk], d = b[kk];
                if (k == 0) q = make_double2(c.x, d.x);
                else if (k < H) q = make_double2(c.x - d.y, c.y + d.x);
                else q = make_double2(c.x + d.y, d.x - c.y);
            }
            v[i * RI + m] = q;
        });
        double2 *mine = reg + (r * 3 + p) * SL;
        dlfft::line<P, 1>(t, v, mine, at, A.tw, sync);
        sync();
        dlfft::each<P, L>(t, [&](int i, int m) { mine[at(dlfft::out_at<P, L>(t, i, m))] = v[i * RO + m]; });
        if (MODE != X_DISS && r == 0) {
            double *ua = A.vel + (((int64_t)p * N + z) * N + y0) * N, *ub = ua + N;
            dlfft::each<P, L>(t, [&](int i, int m) {
                const int x = dlfft::out_at<P, L>(t, i, m);
                ua[x] = v[i * RO + m].x;
                ub[x] = v[i * RO + m].y;
            });
            if (MODE == X_EMIT32 || MODE == X_EMIT64) {
                using F = typename std::conditional<MODE == X_EMIT32, float, double>::type;
                const int Z[2] = {z + DL_PAD_LO, pad_image(z, N)};
#pragma unroll 1
                for (int q = 0; q < 8; q++) {   // both lines and their periodic images in y and z
                    const int y = y0 + (q & 1);
                    const int Yq = q & 2 ? pad_image(y, N) : y + DL_PAD_LO, Zq = q & 4 ? Z[1] : Z[0];
                    if (Yq < 0 || Zq < 0) continue;
                    F *row = static_cast<F *>(A.fp) + p * A.fpc + A.fpz * Zq + A.fpy * Yq;
                    dlfft::each<P, L>(t, [&](int i, int m) {
                        emit_value(row, dlfft::out_at<P, L>(t, i, m), N, q & 1 ? v[i * RO + m].y : v[i * RO + m].x);
                    });
                }
            }
        }
    }
    __syncthreads();
    if (MODE == X_DISS) {
        // lines 3..5 hold the off-diagonal strain e12, e23, e31, lines 0..2 the diagonal; the
        // reference's order (partlib.f90:4007-4080)
        double *e = A.diss + ((int64_t)z * N + y0) * N;
        for (int x = p * T + t; x < N; x += 3 * T) {
            double2 s[6];
            for (int c = 0; c < 6; c++) s[c] = reg[(c < 3 ? 3 + c : c - 3) * SL + at(x)];
            double ea = 0.0, eb = 0.0;
            for (int c = 0; c < 6; c++) {
                ea = c < 3 ? ea + 2.0 * s[c].x * s[c].x : ea + s[c].x * s[c].x;
                eb = c < 3 ? eb + 2.0 * s[c].y * s[c].y : eb + s[c].y * s[c].y;
            }
            e[x] = A.nu2 * ea;
            e[N + x] = A.nu2 * eb;
        }
        return;
    }
    // N = u x omega (turb.f90:634-637)
    const double2 *u1 = reg + (p + 1) % 3 * SL, *u2 = reg + (p + 2) % 3 * SL, *w1 = u1 + 3 * SL, *w2 = u2 + 3 * SL;
    dlfft::each<P, 0>(t, [&](int i, int m) {
        const int x = at(dlfft::in_at<P, 0>(t, i, m));
        const double2 a = u1[x], b = u2[x], c = w1[x], d = w2[x];
        v[i * RI + m] = make_double2(a.x * d.x - b.x * c.x, a.y * d.y - b.y * c.y);
    });
    __syncthreads();
    double2 *mine = reg + p * SL;
    dlfft::line<P, -1>(t, v, mine, at, A.tw, sync);
    sync();
    dlfft::each<P, L>(t, [&](int i, int m) { mine[at(dlfft::out_at<P, L>(t, i, m))] = v[i * RO + m]; });
    sync();
    double2 *oa = rows + p * fstride, *ob = oa + H;
    for (int k = t; k <= A.nek; k += T) {
        const double2 a = mine[at(k)], b = mine[at(k ? N - k : 0)];
        oa[k] = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
        ob[k] = make_double2(0.5 * (a.y + b.y), 0.5 * (b.x - a.x));
    }
}

// ---- z ------------------------------------------------------------------------------------
struct ZArgs {
    double2 *W;
    double2 *u, *nold;      // [3][y][z][px]
    double2 *box;           // u^ of the forcing's modes before k_low: [3][75]
    int n, px, nek;
    double nu, dt, inv_n3;
    const double *afor;     // stochastic forcing a1r..a3r (3 x 5 x 5 x 6) or null
    int det;                // deterministic forcing of shells 1, 2 to the energies f1, f2
    double f1, f2;
    const double2 *tw;
};

// N_0..2 along z, in place: 8 kx x all z of one component and ky per block.  0.104 ms at 256^3, 0.63 GB
// at 6.1 TB/s
template <int N>
__global__ void __launch_bounds__(8 * dlfft::Wide<N>::T) k_zforward(ZArgs A)
{
    using P = dlfft::Wide<N>;
    constexpr int H = N / 2, L = P::S - 1, E = dlfft::elems<P>();
    extern __shared__ double2 sm[];
    const int xi = threadIdx.x & 7, t = threadIdx.x >> 3;
    const int x0 = blockIdx.x * 8, x = x0 + xi, ky = wave(blockIdx.y, N), lim = sphere_lim(A.nek);
    if (x0 * x0 + ky * ky > lim) return;
    const bool in = x * x + ky * ky <= lim;
    double2 *w = A.W + ((int64_t)blockIdx.z * N + blockIdx.y) * w_plane<N>() + x;
    double2 v[E];
    dlfft::each<P, 0>(t, [&](int i, int m) {
        v[i * dlfft::Stage<P, 0>::R + m] = in ? w[dlfft::in_at<P, 0>(t, i, m) * H] : make_double2(0.0, 0.0);
    });
    dlfft::line<P, -1>(t, v, sm, [xi](int i) { return slot_at<P>(i) * 8 + xi; }, A.tw, dlfft::BlockSync());
    if (!in) return;
    dlfft::each<P, L>(t, [&](int i, int m) {
        w[dlfft::out_at<P, L>(t, i, m) * H] = v[i * dlfft::Stage<P, L>::R + m];
    });
}

constexpr int Z_STATE = 0, Z_STRAIN = 1;
// The state's six fields along z into W: field 3 + c is u^_c, field c its curl (Z_STATE); or
// the strain e12, e23, e31 (0..2) and e11, e22, e33 (Z_STRAIN, DISSIP).  Six blocks side by side
// read the same three components (out of L2); 0.194 ms at 256^3, 0.85 GB at 4.4 TB/s
template <int N, int MODE>
__global__ void __launch_bounds__(8 * dlfft::Wide<N>::T) k_zinverse(ZArgs A)
{
    using P = dlfft::Wide<N>;
    constexpr int H = N / 2, L = P::S - 1, E = dlfft::elems<P>();
    extern __shared__ double2 sm[];
    const int xi = threadIdx.x & 7, t = threadIdx.x >> 3;
    const int x0 = blockIdx.x * 8, x = x0 + xi, y = blockIdx.z, ky = wave(y, N), lim = sphere_lim(A.nek);
    if (x0 * x0 + ky * ky > lim) return;
    const int f = blockIdx.y, g = f % 3, rho = x * x + ky * ky;
    const int a = (g + 1) % 3, b = MODE == Z_STRAIN ? g : (g + 2) % 3;
    const double kx = (double)x, kyd = (double)ky;
    const double2 *u = A.u + (int64_t)y * N * A.px + x;
    const int64_t uc = (int64_t)N * N * A.px;
    double2 v[E];
    if (f >= 3) {
        const double2 *ug = u + g * uc;
        dlfft::each<P, 0>(t, [&](int i, int m) {
            const int z = dlfft::in_at<P, 0>(t, i, m), kz = wave(z, N);
            double2 q = make_double2(0.0, 0.0);
            if (rho + kz * kz <= lim) q = ug[z * A.px];
            if (MODE == Z_STRAIN) {   // i k_g u_g
                const double kg = g == 0 ? kx : (g == 1 ? kyd : (double)kz);
                q = make_double2(-(kg * q.y), kg * q.x);
            }
            v[i * dlfft::Stage<P, 0>::R + m] = q;
        });
    } else {
        const double2 *ua = u + a * uc, *ub = u + b * uc;
        dlfft::each<P, 0>(t, [&](int i, int m) {
            const int z = dlfft::in_at<P, 0>(t, i, m), kz = wave(z, N);
            double2 p = make_double2(0.0, 0.0), q = p;
            if (rho + kz * kz <= lim) {
                p = ua[z * A.px];
                q = ub[z * A.px];
            }
            const double ka = a == 0 ? kx : (a == 1 ? kyd : (double)kz);
            const double kb = b == 0 ? kx : (b == 1 ? kyd : (double)kz);
            // strain (i k_a u_b + i k_b u_a) / 2 with b = g; curl i (k_a u_b - k_b u_a)
            v[i * dlfft::Stage<P, 0>::R + m] =
                MODE == Z_STRAIN ? make_double2(0.5 * (-(ka * q.y) - kb * p.y), 0.5 * (ka * q.x + kb * p.x))
                                 : make_double2(-(ka * q.y - kb * p.y), ka * q.x - kb * p.x);
        });
    }
    dlfft::line<P, 1>(t, v, sm, [xi](int i) { return slot_at<P>(i) * 8 + xi; }, A.tw, dlfft::BlockSync());
    if (rho > lim) return;
    double2 *o = A.W + ((int64_t)f * N + y) * w_plane<N>() + x;
    dlfft::each<P, L>(t, [&](int i, int m) {
        o[dlfft::out_at<P, L>(t, i, m) * H] = v[i * dlfft::Stage<P, L>::R + m];
    });
}

// The update inside the sphere (turb.f90:648-676): Crank-Nicolson + AB2, stochastic forcing,
// projection, N_old <- N.  Outside, the state and N_old are zero and stay so.  0.20 ms at 256^3, 1.05 GB at
// 5.2 TB/s; k_update over the whole spectrum, with the transform inputs written, 0.45 ms
__global__ void __launch_bounds__(256) k_update_sphere(ZArgs A)
{
    const int h = A.n / 2;
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x, zy = i / h;
    const int x = i - zy * h, y = zy / A.n, z = zy - y * A.n;
    if (y >= A.n) return;
    const int ky = wave(y, A.n), kz = wave(z, A.n), k2i = x * x + ky * ky + kz * kz;
    if (k2i > sphere_lim(A.nek)) return;
    const int64_t s = ((int64_t)y * A.n + z) * A.px + x, sc = (int64_t)A.n * A.n * A.px;
    const int64_t wy = (int64_t)A.n * h + WPAD, q = y * wy + (int64_t)z * h + x, wc = A.n * wy;
    // all nine loads first: the compiler cannot move them over the stores
    double2 nh[3], no[3], uu[3], v[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        nh[c] = A.W[c * wc + q];
        no[c] = A.nold[c * sc + s];
        uu[c] = A.u[c * sc + s];
    }
    const double kk[3] = {(double)x, (double)ky, (double)kz};
    const double k2 = k2_of(kk[0], kk[1], kk[2]), dth = 0.5 * A.dt, dtr = 1.5 * A.dt, lin = 1.0 - A.nu * dth * k2;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const double2 nn = make_double2(nh[c].x * A.inv_n3, nh[c].y * A.inv_n3);
        v[c].x = uu[c].x * lin + dtr * nn.x - dth * no[c].x;
        v[c].y = uu[c].y * lin + dtr * nn.y - dth * no[c].y;
        A.nold[c * sc + s] = nn;
    }
    const bool box = x <= 2 && ky >= -2 && ky <= 2 && kz >= -2 && kz <= 2;
    if (A.afor && box) {
        // modes kx <= 2, |ky|, |kz| <= 2 (flowlib.f90:522-560), indices 0..4 <-> 0, 1, 2, -2, -1
        for (int c = 0; c < 3; c++) {
            const double *a = A.afor + ((c * 5 + (kz >= 0 ? kz : kz + 5)) * 5 + (ky >= 0 ? ky : ky + 5)) * 6 + 2 * x;
            v[c].x = v[c].x + A.dt * a[0];
            v[c].y = v[c].y + A.dt * a[1];
        }
    }
    const double ik2 = 1.0 / k2, iden = 1.0 / (1.0 + A.nu * dth * k2);
    const double tr = (kk[0] * v[0].x + kk[1] * v[1].x + kk[2] * v[2].x) * ik2;
    const double ti = (kk[0] * v[0].y + kk[1] * v[1].y + kk[2] * v[2].y) * ik2;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const double2 w = make_double2((v[c].x - kk[c] * tr) * iden, (v[c].y - kk[c] * ti) * iden);
        A.u[c * sc + s] = w;
        if (A.det && box) A.box[c * 75 + ((kz + 2) * 5 + ky + 2) * 3 + x] = w;
    }
}

// What couples modes: shells 1 and 2 rescaled to the energies f1, f2 (supforDET,
// flowlib.f90:195-229; from the copies in box, since the modes are rescaled in place), zero
// mean and the conjugate symmetry of kx = 0 (symmetrize, 233-334).  One thread per (ky, kz); a few
// round trips to memory (9 us at 256^3, 5 at 64^3; the serial forcing kernel alone took 26)
__global__ void __launch_bounds__(128) k_low(ZArgs A)
{
    __shared__ double e[75];
    const int n = A.n, i = blockIdx.x * blockDim.x + threadIdx.x, y = i / n, z = i - y * n;
    const int ky = wave(y, n), kz = wave(z, n);
    const bool row = y < n, box = row && ky >= -2 && ky <= 2 && kz >= -2 && kz <= 2;
    double scale[3] = {1.0, 1.0, 1.0};
    if (A.det && __syncthreads_or(box)) {
        for (int q = threadIdx.x; q < 75; q += blockDim.x) {
            double s = 0.0;
            for (int c = 0; c < 3; c++) {
                const double2 w = A.box[c * 75 + q];
                s += w.x * w.x + w.y * w.y;
            }
            e[q] = q % 3 == 0 ? 0.5 * s : s;   // kx = 0 modes count half
        }
        __syncthreads();
        double es[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int q = 0; q < 75; q++) {   // shell 1: k^2 = 1, 2; shell 2: k^2 = 3..6
            const int qx = q % 3, qy = (q / 3) % 5 - 2, qz = q / 15 - 2, k2 = qx * qx + qy * qy + qz * qz;
            if (k2 >= 1 && k2 <= 2) es[1] += e[q];
            if (k2 >= 3 && k2 <= 6) es[2] += e[q];
        }
        scale[1] = sqrt(A.f1 / es[1]);
        scale[2] = sqrt(A.f2 / es[2]);
    }
    if (!row || ky * ky + kz * kz > sphere_lim(A.nek)) return;
    const int64_t sc = (int64_t)n * n * A.px, m = (int64_t)i * A.px;
    // the thread of the lower index of each conjugate pair averages both; all loads first
    const int64_t mp = ((int64_t)((n - y) % n) * n + (n - z) % n) * A.px;
    const int k2 = ky * ky + kz * kz;
    const bool scaled = A.det && box, pair = mp >= m;
    double2 v[3][3], b[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        if (pair) {
            v[c][0] = A.u[c * sc + m];
            b[c] = A.u[c * sc + mp];
        }
        if (scaled) {
            v[c][1] = A.u[c * sc + m + 1];
            v[c][2] = A.u[c * sc + m + 2];
        }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
        if (scaled)
            for (int x = 1; x <= 2; x++) {
                const int q2 = x * x + k2;   // shells 1, 2: k^2 = 1, 2 and 3..6
                if (q2 > 6) continue;
                const double f = q2 <= 2 ? scale[1] : scale[2];
                A.u[c * sc + m + x] = make_double2(v[c][x].x * f, v[c][x].y * f);
            }
        if (!pair) continue;
        double2 a = v[c][0], p = b[c];
        if (scaled && k2 >= 1 && k2 <= 6) {
            const double f = k2 <= 2 ? scale[1] : scale[2];
            a = make_double2(a.x * f, a.y * f);
            p = make_double2(p.x * f, p.y * f);
        }
        a = make_double2(0.5 * (a.x + p.x), 0.5 * (a.y - p.y));
        if (i == 0) a = make_double2(0.0, 0.0);
        A.u[c * sc + m] = a;
        A.u[c * sc + mp] = make_double2(a.x, -a.y);
    }
}
