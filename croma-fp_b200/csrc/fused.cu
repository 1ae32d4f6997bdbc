// fused.cu -- the on-chip FP64 evolve: the segment matrices of a tracer
// chunk are built and factored by one kernel, and a second kernel runs every
// sub-step of every segment with the spectrum held in registers.
//
// Per chunk of tracers (sized to the workspace budget) and species:
//   0. seg_pre_kernel, one thread per (segment, tracer): the segment's
//      interpolated background and the scalars of its coefficients, once for
//      both species.
//   1. factor_kernel, persistent: the loss / diffusion terms, Chang-Cooper faces
//      and rows of every (tracer, segment[, on/off set]) (losses / Dpp / CC
//      assembly of src/fp_shared_core.c:729-842, 1241-1317, 2358-2431 and
//      src/Chang_Cooper.c:22-184), 16 rows a lane, and the Thomas pivots d_i =
//      b_i - a_i c_{i-1}/d_{i-1} as ratios of continuants, combined across the
//      lanes by a scan of 2x2 matrices.  It stores 1/d, a/d and c/d per row.
//      Nothing here depends on the evolving spectra (the eta cap aside, which
//      then runs the chunk one segment at a time), so every segment of the
//      snapshot is factored by one launch with full occupancy.
//   2. steps_packed_kernel (runs of 64 tracers and more): 16 rows a lane, the
//      constants of a segment in registers and tensor memory; below that
//      steps_kernel, one warp per tracer: for each segment it loads the
//      factored rows (and the segment's source), and runs each sub-step as
//      the two first-order linear recurrences of fp_thomas_solve_ws
//      (src/fp_shared_core.c:226-257), each an affine warp scan: a local pass
//      per lane, five shuffle levels, a second local pass (substep); at 512
//      bins radix-4 scans of three shuffle levels with the back pass run
//      while the forward scan is in flight (substep4).  The proton kernel
//      records the spectrum at each segment start for the secondaries.
//   3. secondary_kernel: the electron source of every segment from those
//      proton spectra (prepare_secondary_sources_cell_major,
//      src/fp_shared_core.c:1591-1672), a tiled [segments*tracers x nb] .
//      [nb x nb] product on the FP64 tensor cores, between the proton and
//      the electron steps.
//
// Divisions by grid quantities use reciprocals tabulated on the host; the
// results agree with the reference's divisions to an ulp per operation.
// Spectra are cell-major [tracer][nb] so that a warp's rows are contiguous.
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "croma_bits.cuh"
#include "croma_segment.cuh"

namespace croma {

namespace {

constexpr int kR = NB / 32;          // rows per lane
// Row pitch of the swizzled arrays of the PCR sub-step: lane-blocked reads (m =
// R lane + r) and those at a stride then touch distinct bank pairs.
constexpr int kPitch = 32 + 16 / kR;
constexpr int kSw = kPitch * kR;     // swizzled row-array length
constexpr unsigned kFull = 0xffffffffu;
// Packed layout (factor and packed steps kernels): 16 rows a lane at every bin
// count, so 8, 16 or 32 lanes hold a system and a warp 4, 2 or 1 of them.
constexpr int kPkRows = 16;
constexpr int kPkLanes = NB / kPkRows;
constexpr int kPkTracers = 32 / kPkLanes;
constexpr int kFacDoubles = 3 * NB;  // 1/d, a/d, c/d of one system
// Per-segment scalars of one (segment slot, tracer): what the factor kernels
// of both species need of the schedule's segment and of the background
// interpolated to it, computed once by seg_pre_kernel.  Kernels copy it to shared
// memory 16 bytes at a time, which its members alone (8 bytes) do not align it for.
struct alignas(16) SegPre {
    double n_gas, kbt, inv_kbt, log_n, adiab, synch_coeff, coulomb_coeff;
    double dt, dt_over_tloss_pref, dtT_e, alpha, dpp_inv;
    int flags;               // bit 0 active, 1 windowed, 2 interpolated, 3 "on" Dpp filled
    int sl, el, steps;       // Dpp window within the segment, sub-steps
};
enum { kPreActive = 1, kPreWindowed = 2, kPreInterp = 4, kPreFill = 8 };

struct FusedParams {
    SnapArgs a;              // spectra and sources cell-major [tracer][nb]
    GridTables gt;
    ModelParams mp;
    int g0, g1;              // segment slots of this launch
    int t0, nt;              // tracer chunk [t0, t0 + nt)
    int sets;                // factor sets per segment: 1 (on) or 2 (on, off)
    // One caller-defined segment shared by every tracer (run_tracer_pipeline):
    // when set, ex replaces the per-tracer schedule.
    int explicit_seg;
    SegInfo ex;
    // IC rows: shared row (stride 0) or per tracer, momentum-major
    // [nb][ntracer] (stride = ntracer)
    int ic_stride;
    const double *eta_scale; // [ntracer] Dpp eta-cap scale of slot g0, or null (no cap)
    int pack;                // systems a warp of the factor kernel takes together, 1 .. kPkTracers
    double *fac;             // [2 species][g1 - g0][sets][nt][3][nb]
    SegPre *pre;             // [g1 - g0][nt]
    double *np_seg;          // [g1 - g0][nt][nb] proton spectra at segment starts, or null
    double *inje;            // [g1 - g0][nt][nb] electron source per segment, or null
    const int *np_min_qe;    // [nb]
    // solver calibration (the autotuner): when cal_spec is set, the steps
    // kernel reads and writes the spectra rows of tracer tl at cal_spec + tl nb
    // instead of the resident ones and stops after cal_steps sub-steps
    double *cal_spec;
    int cal_steps;
    const int *order;        // [nt] the packed steps kernel's tracer order within the chunk, or null (as they are)
};

__device__ __forceinline__ SegInfo segment_of(const FusedParams &P, int t, int slot)
{
    return P.explicit_seg ? P.ex : seg_info(P.a.sched, t, slot, P.a.dt_snap);
}

__device__ __forceinline__ double *fac_ptr(const FusedParams &P, int S, int gi, int set, int tl)
{
    return P.fac + ((((size_t)S * (P.g1 - P.g0) + gi) * P.sets + set) * P.nt + tl) * kFacDoubles;
}

// Which factor sets a segment needs: 0 = Dpp on, 1 = off (windowed segments).
// The window is clamped to the segment's sub-steps as the steps kernel runs it.
__device__ __forceinline__ bool needs_set(const SegInfo &g, int set)
{
    if (!g.windowed) return set == 0;
    const int sl = min(max(g.sl, 0), g.steps), el = min(max(g.el, sl), g.steps);
    return (set == 0) ? el > sl : (sl > 0 || el < g.steps);
}

__device__ __forceinline__ int swz(int m) { return (m % kR) * kPitch + m / kR; }
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ double sup(double v, int d) { return __shfl_up_sync(kFull, v, d); }
__device__ __forceinline__ double sdn(double v, int d) { return __shfl_down_sync(kFull, v, d); }
// 32-byte accesses of four consecutive doubles (sm_100 256-bit vector
// loads and stores).  The lanes of a warp own 128-byte row blocks, so a
// 16-byte access per lane would touch 32 sectors and use half of each (a
// scalar access a quarter); 32 bytes per lane use every sector fully.  The
// asm is volatile, so that loads and stores keep their order.
// ld4_cg / st4_cg: L2 only (rows and sources); ld4 / st4: the default caching.
__device__ __forceinline__ void ld4_cg(const double *p, double *v)
{
    asm volatile("ld.global.cg.v4.f64 {%0,%1,%2,%3}, [%4];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}
__device__ __forceinline__ void ld4(const double *p, double *v)
{
    asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p) : "memory");
}
__device__ __forceinline__ void st4(double *p, const double *v)
{
    asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3])
                 : "memory");
}
// st4 bypassing L1 (rows written for another kernel).
__device__ __forceinline__ void st4_cg(double *p, const double *v)
{
    asm volatile("st.global.cg.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3])
                 : "memory");
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool valid)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = valid ? 16 : 0;   // 0 source bytes: the 16 destination bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// coulomb_kernel_fast with its erf / exp branch out of line: the proton
// terms otherwise inline four copies of it, and the factor kernel's code
// outgrows the instruction cache.  Same arithmetic.
__device__ __noinline__ double coulomb_slow(double x)
{
    return 0.5 * sqrt(kPi) * erf(sqrt(x)) - sqrt(x) * exp_tab(-x);
}
__device__ __forceinline__ double coulomb_one(double x)
{
    return (x > 40.0) ? 0.5 * sqrt(kPi) : coulomb_slow(x);
}

// The scalars of one segment's coefficients (seg_pre_kernel).
struct SegTerms {
    double n_gas, kbt, inv_kbt, log_n, adiab;
    double synch_coeff, coulomb_coeff;
    double dt, dt_over_tloss_pref;   // protons: dt / T = sig_eff * dt_over_tloss_pref
    double dtT_e;                    // electrons: dt / 1e100
    double alpha;
    int interp;
};

__device__ __forceinline__ SegTerms seg_terms(const Bg &bg, int dis, const SegInfo &g)
{
    SegTerms T;
    T.n_gas = bg.n_gas;
    T.kbt = bg.kbt;
    T.inv_kbt = 1.0 / bg.kbt;
    T.log_n = log(bg.n_gas);
    T.adiab = 1.0 / 3.0 * (dis ? 0.0 : bg.divv);
    const double b_ratio = bg.b_field * 1.0e+6 / 3.2;
    T.synch_coeff = 4.8e-4 * b_ratio * b_ratio * 9.11e-28 * 3.0e+10 * 3.1536e+16;
    T.coulomb_coeff = 3.05e-29 * bg.n_gas * kC * kGyr / (kMe * kGeV);
    T.dt = g.dt;
    T.dt_over_tloss_pref = g.dt / (1.0 / (0.5 * kC * bg.n_gas) / kGyr);
    T.dtT_e = g.dt / 1.0e+100;
    T.alpha = g.alpha;
    T.interp = g.nseg > 1;
    return T;
}

// Power-of-two factor that brings the larger of |x|, |y| into [1, 2) (1 where
// that is zero, subnormal or not finite).
__device__ __forceinline__ double pow2_norm(double x, double y)
{
    const int ex = max(__double2hiint(x) & 0x7fffffff, __double2hiint(y) & 0x7fffffff) >> 20;
    return (ex <= 0 || ex >= 2046) ? 1.0 : __hiloint2double((2046 - ex) << 20, 0);
}

// The last two continuants before a lane's rows, from every lane's matrix of its
// rows' recurrence (an exclusive scan over the LANES lanes of a system).
template <int LANES>
__device__ __forceinline__ void continuant_scan(double t00, double t01, double t10, double t11, int gl, double &th,
                                                double &thp)
{
    auto up = [](double v, int d) { return __shfl_up_sync(kFull, v, d, LANES); };
#pragma unroll
    for (int off = 1; off < LANES; off <<= 1) {
        const double u00 = up(t00, off), u01 = up(t01, off), u10 = up(t10, off), u11 = up(t11, off);
        if (gl >= off) {
            const double n00 = fma(t00, u00, t01 * u10), n01 = fma(t00, u01, t01 * u11);
            const double n10 = fma(t10, u00, t11 * u10), n11 = fma(t10, u01, t11 * u11);
            t00 = n00; t01 = n01; t10 = n10; t11 = n11;
        }
    }
    th = up(t00, 1);
    thp = up(t10, 1);
    if (gl == 0) {
        th = 1.0;
        thp = 0.0;
    }
}

// Thomas pivots of the rows a, b, c of a system, in place: Bd <- 1/d, A <- a/d,
// Cc <- c/d, with d_i = b_i - a_i c_{i-1} / d_{i-1} (fp_thomas_solve_ws,
// src/fp_shared_core.c:226-257); R rows a lane, LANES lanes a system, gl the
// lane's place among them.  The pivots are ratios of continuants, d_i = theta_i
// / theta_{i-1} with theta_i = b_i theta_{i-1} - e_i theta_{i-2}, e_i = a_i
// c_{i-1}: each lane forms the 2x2 matrix of its rows' recurrence (rescaled by
// exact powers of two to a largest entry in [1, 2); the scan's products stay
// below 2^63), a scan over the lanes gives it its incoming pair, and it runs the
// recurrence on its rows from there.  One FMA a row is all that is serial: the
// reciprocals theta_{i-1} / theta_i are independent of each other, where the
// pivot recurrence itself waits for one reciprocal a row (66 cycles against 8).
// A row's rounding errors are those of d = b - e / d, since only the ratio of
// the last two continuants enters it, as one rounded quotient: the product with a
// rounded reciprocal doubled the spectra's error growth over 500 sub-steps (mean
// 2-norm error against 80 bits, 21 runs of 64 tracers: 1.08 of the former
// recurrence's, 1.00 with the quotient; no change in time but 1 % of the per-step
// path's, 4466 -> 4515 us at 256 bins, 4,096 tracers).
template <int R, int LANES>
__device__ __forceinline__ unsigned pivot_rows(double A[R], double Bd[R], double Cc[R], int gl)
{
    auto up = [](double v, int d) { return __shfl_up_sync(kFull, v, d, LANES); };
    unsigned err = 0;
    double c_in = up(Cc[R - 1], 1);   // c of the row before this lane's first
    c_in = gl > 0 ? c_in : 0.0;
    double t00 = 1.0, t01 = 0.0, t10 = 0.0, t11 = 1.0;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const double e = A[r] * (r > 0 ? Cc[r - 1] : c_in);
        const double n00 = fma(Bd[r], t00, -(e * t10));
        const double n01 = fma(Bd[r], t01, -(e * t11));
        t10 = t00;
        t11 = t01;
        t00 = n00;
        t01 = n01;
        if ((r & 3) == 3) {   // d < 2^255 cannot leave the range in four rows
            const double sc = pow2_norm(t00, t01);
            t00 *= sc; t01 *= sc; t10 *= sc; t11 *= sc;
        }
    }
    double th, thp;
    continuant_scan<LANES>(t00, t01, t10, t11, gl, th, thp);
    double cprev = c_in;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const double n = fma(Bd[r], th, -(A[r] * cprev * thp));
        if (continuant_singular(n, th)) err = kErrSingular;
        const double inv = quot_nr(th, n);
        cprev = Cc[r];
        Bd[r] = inv;
        A[r] *= inv;
        Cc[r] *= inv;
        thp = th;
        th = n;
        if ((r & 3) == 3 && r < R - 1) {
            const double sc = pow2_norm(th, thp);
            th *= sc;
            thp *= sc;
        }
    }
    return err;
}

// Sixteen (eight) 32-bit TMEM columns of the warp's lanes.  The loads are
// asynchronous: the registers are valid after tmem_wait, which names them so
// that no use is scheduled before it (tmem_after8: a further load that the same
// wait covers).
struct Tmem16 {
    unsigned r[16];
    __device__ __forceinline__ double d(int i) const { return __hiloint2double((int)r[2 * i + 1], (int)r[2 * i]); }
};
__device__ __forceinline__ void tmem_ld16(unsigned t, Tmem16 &u)
{
    unsigned *r = u.r;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(t));
}
__device__ __forceinline__ void tmem_ld8(unsigned t, unsigned *r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(t));
}
__device__ __forceinline__ void tmem_wait(Tmem16 &u)
{
    unsigned *r = u.r;
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]));
}
__device__ __forceinline__ void tmem_after8(unsigned *r)
{
    asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]));
}
__device__ __forceinline__ void tmem_wait8(unsigned *r)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]));
}
__device__ __forceinline__ void tmem_st8(unsigned t, const unsigned *r)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(t), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

__device__ __forceinline__ void pk_set(unsigned *r, int i, double v)
{
    r[2 * i] = (unsigned)__double2loint(v);
    r[2 * i + 1] = (unsigned)__double2hiint(v);
}
__device__ __forceinline__ double pk_get(const unsigned *r, int i) { return __hiloint2double((int)r[2 * i + 1], (int)r[2 * i]); }

// TMEM columns of a block, its base address through shared memory; one warp of
// the block calls each.  The allocation waits until the SM has the columns,
// which the blocks that hold them give back when they end.
template <int COLUMNS>
__device__ __forceinline__ void tmem_alloc(unsigned *base)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(base)),
                 "n"(COLUMNS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
template <int COLUMNS>
__device__ __forceinline__ void tmem_free(unsigned base)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "n"(COLUMNS));
}
__device__ __forceinline__ void tmem_st2(unsigned t, double v)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};" ::"r"(t), "r"(__double2loint(v)),
                 "r"(__double2hiint(v))
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------------------
// Factor kernel, persistent: a block stages the species' grid tables once, in
// the packed layout (lane gl holds rows 16 gl .. 16 gl + 15 of its system; the
// systems of a warp are neighbouring segments and sets of one tracer), and its
// warps take units of kPkTracers systems in turn, the next unit's scalars
// copied to shared memory meanwhile.
//
// It is bound by the latency of its FP64 instructions, exponentials and
// reciprocals.  So their number is kept down: what depends on the grid alone
// is tabulated -- with the diffusion coefficient kappa g(p), g = p^2 exp(-1/p)
// (protons: times exp(-E/E_max)) and kappa the segment's 1 / (4 t_acc) times
// the eta cap's scale, or the "off" form g = p^2, kappa = 1 / (4e5), a face
// needs 2 g / p, dx / (g_j + g_j+1) and (g_j + g_j+1) / (2 dx) -- and each face
// is evaluated once: the row above takes it from the lane's registers or its
// neighbour's.  And the rows wait in tensor memory between the face loop, which
// also runs the continuants' recurrence, and the second pass (pivot_rows'
// arithmetic): 128 registers, 16 warps per SM.  The face loop is unrolled by four
// rows only, so that it stays in the instruction cache.  Rows with a vanishing
// diffusion coefficient (kappa g <= 1e-200) have their own forms
// (Chang_Cooper.c:66-184); a warp with a system that could meet them takes a copy
// of the face loop that knows them: snapshots of 4,096 tracers on a grid from p =
// 10^-3.2 (both species) 0.80 ms at 128 bins and 1.60 at 256, on the ordinary grid
// 0.77 and 1.57; those systems' rows one by one, each row's terms formed three
// times, 2.51 and 6.63, a warp per system before the packed layout 1.71 and 2.24.
// The copy costs the other calls 0.3 to 0.7 %.
//
// Measured, before (a warp per system at every bin count, coefficients staged
// in shared memory, a reciprocal a row in the serial chain of the pivots) and
// now, protons and electrons: 512 bins, 131,072 tracers x 16 segments 20.6 and
// 16.7 -> 11.0 and 8.8 ms; 256 bins, 65,536 tracers 3.82 and 3.18 -> 2.83 and
// 2.18 ms; 128 bins, 131,072 tracers (electrons) 3.53 -> 2.18 ms; 64 tracers 61
// -> 10 us.  12 warps with the rows in registers 12.5 and 11.2 ms at 512 bins,
// the face loop unrolled whole 12.4 and 9.9.  FP64 pipe 46 and 42 % (512 bins,
// 4,096 tracers).
// Tables are pairs of doubles, read 16 bytes at a time:
enum { FT_X01,      // electrons: p^2, 1/beta^2;  protons: 1/beta^2, that / (2 m_p (gamma - 1))
       FT_X2P,      // electrons: log p / beta^2, p;  protons: sig_eff, p
       FT_X34,      // electrons: IC row at z_curr, its change to z_next;  protons: gamma m_p - m_p of two bins, grid order
       FT_GR,       // filled Dpp form: 2 g / p, dx / (g_j + g_j+1)
       FT_FK,       //                  (g_j + g_j+1) / (2 dx), 1 / dp
       FT_OFF,      // the same two of the off form
       kFacTabs = FT_OFF + 2 };
constexpr int kFacWarps = 8;
constexpr int kFacBlocks = 2;      // blocks per SM
constexpr int kFacColumns = 256;   // TMEM: two warps a lane quarter, 96 of 128 columns each
// Protons: the Coulomb kernel of a warp's systems, lane-strided (so that the
// bins that need its erf and exp are whole warps), read back packed: row r of
// lane gl at r * kCoulPitch + gl, an odd pitch for distinct banks.
constexpr int kCoulPitch = kPkLanes + 1;
constexpr int kCoulSys = kPkRows * kCoulPitch;
constexpr int kCoulWarp = kPkTracers * kCoulSys;

// Chang-Cooper weights of a face (face_weights, croma_phys.cuh) with one
// exponential exp(-|w| / 2) for both branches and one quotient; agrees with it to
// a few ulp.
__device__ __forceinline__ void face_weights_half(double w, double &wp, double &wm)
{
    const double aw = fabs(w);
    const bool series = aw < 0.1;
    // exp(-700) squared is 0, as exp(-1400) is (a NaN comes through aw below)
    const double E = exp_tab_normal(aw < 1400.0 ? -0.5 * aw : -700.0);
    const double e2 = E * E, w2 = w * w;
    const double dser = fma(w2, fma(w2, 1.0 / 1920.0, 1.0 / 24.0), 1.0);
    const double q = quot_nr(series ? 1.0 : aw, series ? E * dser : fma(-E, E, 1.0));
    const double s = q * e2;
    wp = (w >= 0.0) ? q : s;
    wm = (w >= 0.0) ? s : q;
}

// ROWS: stores the raw rows a, b, c for the per-step path, which factors them
// again on every sub-step; else the factored 1/d, a/d, c/d.
template <int S, bool ROWS>
__global__ void __launch_bounds__(kFacWarps * 32, kFacBlocks) factor_kernel(const __grid_constant__ FusedParams P)
{
    constexpr int R = kPkRows, G = kPkLanes;
    extern __shared__ double4 smem_raw[];
    double2 *tab = reinterpret_cast<double2 *>(smem_raw);
    __shared__ double g_warp[2][kFacWarps];        // least g of the filled and the off form, per warp's share
    __shared__ SegPre pre_next[2][kFacWarps * kPkTracers];   // scalars of the warp's systems, one unit ahead
    static_assert(sizeof(SegPre) == 7 * 16 && alignof(SegPre) >= 16 && G >= 7,
                  "a group's lanes copy its SegPre 16 bytes each");
    __shared__ unsigned tmem_base;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, gl = lane & (G - 1);
    if (w == 0) tmem_alloc<kFacColumns>(&tmem_base);
    const SnapArgs &a = P.a;
    const SpeciesTables &st = P.gt.s[S];
    auto g_of = [&](int form, int i) {
        return form ? st.p2[i] : (S == 0 ? st.p2[i] * st.expE[i] * st.exp_cut[i] : st.p2[i] * st.exp_cut[i]);
    };
    double g_min[2] = {1.0e+308, 1.0e+308};
    for (int i = threadIdx.x; i < NB; i += blockDim.x) {
        const int at = (i % R) * G + i / R;
        if (S == 0) {
            tab[FT_X01 * NB + at] = make_double2(P.gt.cp_inv_betap2[i], P.gt.cp_inv_betap2[i] * P.gt.cp_inv2mpkin[i]);
            tab[FT_X2P * NB + at] = make_double2(P.gt.sig_eff[i], st.p[i]);
            reinterpret_cast<double *>(tab + FT_X34 * NB)[i] = P.gt.cp_Ep[i];
        } else {
            const double r0 = P.ic_stride == 0 ? a.ic_curr[i] : 0.0;
            tab[FT_X01 * NB + at] = make_double2(st.p2[i], P.gt.ce_inv_beta2[i]);
            tab[FT_X2P * NB + at] = make_double2(P.gt.ce_logp[i] * P.gt.ce_inv_beta2[i], st.p[i]);
            tab[FT_X34 * NB + at] = make_double2(r0, P.ic_stride == 0 ? a.ic_next[i] - r0 : 0.0);
        }
#pragma unroll
        for (int form = 0; form < 2; form++) {
            const double g = g_of(form, i);
            const bool face = i < NB - 1;   // the last bin has no face above: weights of a zero flux
            const double gs = face ? g + g_of(form, i + 1) : 0.0;
            tab[(FT_GR + 2 * form) * NB + at] = make_double2(st.two_over_p[i] * g, face ? st.dxf[i] / gs : 0.0);
            tab[(FT_FK + 2 * form) * NB + at] = make_double2(face ? 0.5 * gs * st.inv_dxr[i] : 0.0, st.inv_dx[i]);
            g_min[form] = fmin(g_min[form], g);
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        g_min[0] = fmin(g_min[0], __shfl_xor_sync(kFull, g_min[0], off));
        g_min[1] = fmin(g_min[1], __shfl_xor_sync(kFull, g_min[1], off));
    }
    if (lane == 0) {
        g_warp[0][w] = g_min[0];
        g_warp[1][w] = g_min[1];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kFacWarps; k++) {
        g_min[0] = fmin(g_min[0], g_warp[0][k]);
        g_min[1] = fmin(g_min[1], g_warp[1][k]);
    }
    // rows a, b, c of chunk k (four rows) of the warp's lanes: 8 columns each
    const unsigned tm = tmem_base + ((unsigned)((w & 3) * 32) << 16) + (w >> 2) * 128;
    // A unit: P.pack segments of one tracer and one set, or, with fewer segments
    // than that, those of several tracers; unit numbers run over the tracers
    // first, so that segments beyond a tracer's last fall evenly on the warps, and
    // over the sets last: most windowed segments need one of the two, and a warp
    // whose systems all need none of its set leaves at once (28 to 25 us a slot at
    // 10,000 windowed tracers).
    const int nslot = P.g1 - P.g0, segs = min(nslot, P.pack), tracers = P.pack / segs;
    const int nq = (P.nt + tracers - 1) / tracers, nblk = (nslot + segs - 1) / segs;
    const int units = nblk * nq * P.sets, stride = gridDim.x * kFacWarps;
    const int sub = (lane / G) / segs, off = (lane / G) - sub * segs;   // the group's place in the unit
    double *coul = reinterpret_cast<double *>(tab + kFacTabs * NB) + w * kCoulWarp;
    const double2 *row = tab + gl;                // table k, row r of the lane: row[k * NB + r * G]
    const int group = w * kPkTracers + lane / G;
    auto locate = [&](int unit, int &tl, int &gi, int &set) {
        const int b = unit / nq;
        set = b / nblk;
        gi = (b - set * nblk) * segs + off;
        tl = (unit - b * nq) * tracers + sub;
        return unit < units && sub < tracers && tl < P.nt && gi < nslot;
    };
    auto fetch = [&](int unit, int buf) {         // the unit's scalars, 16 bytes a lane
        int tl, gi, set;
        if (locate(unit, tl, gi, set) && gl < 7)
            cp_async16(reinterpret_cast<char *>(&pre_next[buf][group]) + 16 * gl,
                       reinterpret_cast<const char *>(P.pre + (size_t)gi * P.nt + tl) + 16 * gl, true);
    };
    int buf = 1;
    fetch(blockIdx.x * kFacWarps + w, 0);
#pragma unroll 1
    for (int unit = blockIdx.x * kFacWarps + w; unit < units; unit += stride) {
        int tl, gi, set;
        const bool here = locate(unit, tl, gi, set);
        if (!here) tl = gi = set = 0;
        buf ^= 1;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        fetch(unit + stride, buf ^ 1);
        const int t = P.t0 + tl;
        const SegPre &pre = pre_next[buf][group];
        const int flags = here ? pre.flags : 0;
        SegInfo si{};
        si.windowed = (flags & kPreWindowed) ? 1 : 0;
        si.sl = pre.sl;
        si.el = pre.el;
        si.steps = pre.steps;
        bool on = (flags & kPreActive) && needs_set(si, set);
        if (on && needs_set(si, 1) && P.sets < 2) {   // checked on the host; never write past the sets
            if (gl == 0) atomicOr(a.err, kErrBadInput);
            on = false;
        }
        const unsigned firsts = __ballot_sync(kFull, on && gl == 0);   // first lanes of the systems in use
        if (!firsts) continue;
        const bool fill = set == 0 && (flags & kPreFill);
        const double scale = (set == 0 && P.mp.dpp_model != kDppOff && P.eta_scale) ? P.eta_scale[t] : 1.0;
        const double kappa = fill ? pre.dpp_inv * scale : (1.0 / (4.0 * 1.0e+5)) * scale;
        const double inv_kappa = 1.0 / kappa;
        const double alpha = (flags & kPreInterp) ? pre.alpha : 0.0;
        const double g_lo = g_min[fill ? 0 : 1];
        const bool general = on && !(g_lo > 1.0e-290 && kappa * g_lo > 1.0e-200 && isfinite(kappa) && isfinite(inv_kappa));
        const double dt = pre.dt, adiab = pre.adiab;
        double *out = fac_ptr(P, S, gi, set, tl);
        unsigned err = 0;
        // per-bin scalars of B
        double s0, s1, s2;
        if (S == 0) {
            s0 = kGyr * kC / (kMp * kGeV) * 3.5e-29 * pre.n_gas;
            s1 = pre.kbt;
            s2 = pre.dt_over_tloss_pref;
            // the Coulomb kernels of the warp's systems
#pragma unroll 1
            for (unsigned m = firsts; m; m &= m - 1) {
                const int l0 = __ffs(m) - 1;
                const double ik = __shfl_sync(kFull, pre.inv_kbt, l0);
                double *to = coul + l0 / G * kCoulSys;
#pragma unroll 2
                for (int j = lane; j < NB; j += 32) {
                    const double xp = reinterpret_cast<const double *>(tab + FT_X34 * NB)[j] * ik;
                    const double sum = coulomb_one(xp * (kMe / kMp)) + coulomb_one(xp) * (kMe / kMp);
                    to[(j % R) * kCoulPitch + j / R] = sum;
                }
            }
            __syncwarp();
        } else {
            s0 = pre.synch_coeff;
            s1 = pre.coulomb_coeff * (1.0 - pre.log_n * (1.0 / 74.8));
            s2 = pre.coulomb_coeff * (1.0 / 74.8);
            if (P.ic_stride) {   // the tracers' own IC rows
#pragma unroll 1
                for (unsigned m = firsts; m; m &= m - 1) {
                    const int l0 = __ffs(m) - 1, ts = __shfl_sync(kFull, t, l0);
                    const double as = __shfl_sync(kFull, alpha, l0);
                    double *to = coul + l0 / G * kCoulSys;
#pragma unroll 4
                    for (int j = lane; j < NB; j += 32) {
                        const size_t at = (size_t)j * P.ic_stride + ts;
                        const double c = a.ic_curr[at], n = a.ic_next[at];
                        to[(j % R) * kCoulPitch + j / R] = lerp(c, n, as);
                    }
                }
                __syncwarp();
            }
        }
        const double2 *form = row + (fill ? 0 : 2 * NB);
        const double *cs = coul + (lane / G) * kCoulSys + gl;
        const double al = alpha <= 0.0 ? 0.0 : (alpha >= 1.0 ? 1.0 : alpha);
        auto B_of = [&](int r, double g2p) {
            const double2 x01 = row[FT_X01 * NB + r * G], x2p = row[FT_X2P * NB + r * G];
            double B;
            if (S == 0) {
                const double ct = fma(-s1, x01.y, x01.x);
                B = s0 * cs[r * kCoulPitch] * (ct < 0.0 ? 0.0 : ct);
            } else {
                double ric;
                if (P.ic_stride == 0) {
                    const double2 x34 = row[FT_X34 * NB + r * G];
                    ric = fma(al, x34.y, x34.x);
                } else {
                    ric = cs[r * kCoulPitch];
                }
                B = fma(s0, x01.x, ric);
                B = fma(s1, x01.y, B);
                B = fma(s2, x2p.x, B);
            }
            B = fma(adiab, x2p.y, B);
            return fma(-kappa, g2p, B);
        };
        // Rows from the faces above them (cc_build_*, Chang_Cooper.c:66-184), into
        // TMEM, and the matrix of the continuants' recurrence over rows 1 .. 15.
        // A lane's first row waits for its neighbour's last face.  FLOOR: with the
        // forms of rows whose diffusion coefficient vanishes (Chang_Cooper.c:66-184:
        // no flux through the face above, upwind differences of B in the row); a
        // system whose rows are all above the floor gets the same bits from both,
        // the roundings being written out.
        double t00 = 1.0, t01 = 0.0, t10 = 0.0, t11 = 1.0;
        double a0, b0, e1;
        auto face_rows = [&](auto floor) {
            constexpr bool FLOOR = decltype(floor)::value;
            double2 gr = form[FT_GR * NB];
            double Bc = B_of(0, gr.x), Pl = 0.0, Ml = 0.0, cl = 0.0;   // flux times weights of the face below; c of the row below
            const double B_up = __shfl_down_sync(kFull, Bc, 1, G);
            double Bl = 0.0;               // B of the row below
            bool live0 = true;
            auto dpp_of = [&](int r, double g2p) { return 0.5 * (kappa * g2p) * row[FT_X2P * NB + r * G].y; };
            if (FLOOR) Bl = __shfl_up_sync(kFull, B_of(R - 1, form[FT_GR * NB + (R - 1) * G].x), 1, G);
#pragma unroll 1
            for (int kk = 0; kk < R / 4; kk++) {
                unsigned ua[8], ub[8], uc[8];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int r = 4 * kk + i;
                    const double rf = gr.y, g2p = gr.x;
                    double Bn = B_up;
                    if (r < R - 1) {
                        gr = form[FT_GR * NB + (r + 1) * G];
                        Bn = B_of(r + 1, gr.x);
                    }
                    const double2 fk = form[FT_FK * NB + r * G];
                    double wp, wm;
                    face_weights_half((Bc + Bn) * (rf * inv_kappa), wp, wm);
                    bool live = true;
                    double Dpp = 0.0;
                    if (FLOOR) {
                        Dpp = dpp_of(r, g2p);
                        live = !general || fabs(Dpp) > 1.0e-200;
                        wp = live ? wp : 0.0;
                        wm = live ? wm : 0.0;
                    }
                    const double F = kappa * fk.x;
                    const double Pu = F * wp, Mu = F * wm;
                    const double k = dt * fk.y;
                    double ar = k * Ml, br = fma(k, __dadd_rn(Pl, Mu), 1.0), cr = k * Pu;
                    if (FLOOR && !live) {
                        const bool first = gl == 0 && r == 0, last = gl == G - 1 && r == R - 1;
                        const double Bs = 0.5 * (Bc + Bl);
                        ar = 0.0;
                        br = first ? 1.0 : fma(k, Bs, 1.0);
                        cr = last ? 0.0 : k * (0.5 * (Bc + Bn));
                        if (last) {
                            const double Dl = dpp_of(R - 2, form[FT_GR * NB + (R - 2) * G].x);
                            if (fabs(Dl) > 1.0e-200) ar = -face_delta((Bl + Bc) / (Dl + Dpp) * (st.p[NB - 1] - st.p[NB - 2])) * Bs * k;
                        }
                    }
                    br = S == 0 ? fma(row[FT_X2P * NB + r * G].x, s2, br) : br + pre.dtT_e;
                    pk_set(ua, i, ar);
                    pk_set(ub, i, br);
                    pk_set(uc, i, cr);
                    if (r == 0) {
                        b0 = br;
                        live0 = live;
                    } else {
                        const double e = ar * cl;
                        const double n00 = fma(br, t00, -(e * t10)), n01 = fma(br, t01, -(e * t11));
                        t10 = t00;
                        t11 = t01;
                        t00 = n00;
                        t01 = n01;
                        if (i == 3) {   // d < 2^255 cannot leave the range in four rows
                            const double sc = pow2_norm(t00, t01);
                            t00 *= sc; t01 *= sc; t10 *= sc; t11 *= sc;
                        }
                        if (r == R - 1 && gl == G - 1 && on && live && isnan(ar)) err |= kErrCcNan;
                    }
                    if (FLOOR) Bl = Bc;
                    cl = cr;
                    Bc = Bn;
                    Pl = Pu;
                    Ml = Mu;
                }
                tmem_st8(tm + kk * 24, ua);
                tmem_st8(tm + kk * 24 + 8, ub);
                tmem_st8(tm + kk * 24 + 16, uc);
            }
            Pl = __shfl_up_sync(kFull, Pl, 1, G);
            Ml = __shfl_up_sync(kFull, Ml, 1, G);
            const double k0 = dt * form[FT_FK * NB].y;
            a0 = gl > 0 && live0 ? k0 * Ml : 0.0;
            b0 = gl > 0 && live0 ? fma(k0, Pl, b0) : b0;
            tmem_wait_st();   // chunk 0 is there before two of its columns are written again
            tmem_st2(tm, a0);
            tmem_st2(tm + 8, b0);
            e1 = __shfl_up_sync(kFull, cl, 1, G);   // c of the row below the lane's first
        };
        if (__builtin_expect(__any_sync(kFull, general), 0)) face_rows(std::true_type{});
        else face_rows(std::false_type{});
        const double c_in = gl > 0 ? e1 : 0.0;
        tmem_wait_st();
        if (ROWS) {
#pragma unroll
            for (int kk = 0; kk < R / 4; kk++) {
                unsigned u[3][8];
#pragma unroll
                for (int k = 0; k < 3; k++) tmem_ld8(tm + kk * 24 + 8 * k, u[k]);
                tmem_wait8(u[0]);
                tmem_after8(u[1]);
                tmem_after8(u[2]);
                if (on) {
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        const double v[4] = {pk_get(u[k], 0), pk_get(u[k], 1), pk_get(u[k], 2), pk_get(u[k], 3)};
                        st4_cg(out + k * NB + gl * R + 4 * kk, v);
                    }
                }
                __syncwarp();
            }
        } else {
            // the first row's matrix, the scan, then pivot_rows' second pass
            {
                const double e = a0 * c_in;
                const double n00 = fma(t00, b0, t01), n10 = fma(t10, b0, t11);
                t01 = -(t00 * e);
                t11 = -(t10 * e);
                t00 = n00;
                t10 = n10;
                const double sc = pow2_norm(t00, t01);
                t00 *= sc; t01 *= sc; t10 *= sc; t11 *= sc;
            }
            unsigned u[3][8];
#pragma unroll
            for (int k = 0; k < 3; k++) tmem_ld8(tm + 8 * k, u[k]);
            double th, thp, cp = c_in;
            continuant_scan<G>(t00, t01, t10, t11, gl, th, thp);
            bool bad = false;
#pragma unroll
            for (int kk = 0; kk < R / 4; kk++) {
                tmem_wait8(u[0]);
                tmem_after8(u[1]);
                tmem_after8(u[2]);
                double vi[4], vh[4], vq[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    vh[i] = pk_get(u[0], i);
                    vi[i] = pk_get(u[1], i);
                    vq[i] = pk_get(u[2], i);
                }
                if (kk < R / 4 - 1) {
#pragma unroll
                    for (int k = 0; k < 3; k++) tmem_ld8(tm + (kk + 1) * 24 + 8 * k, u[k]);
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const double n = fma(vi[i], th, -(vh[i] * cp * thp));
                    bad |= continuant_singular(n, th);
                    vi[i] = quot_nr(th, n);
                    cp = vq[i];
                    vh[i] *= vi[i];
                    vq[i] *= vi[i];
                    thp = th;
                    th = n;
                }
                if (kk < R / 4 - 1) {
                    const double sc = pow2_norm(th, thp);
                    th *= sc;
                    thp *= sc;
                }
                if (on) {
                    st4_cg(out + gl * R + 4 * kk, vi);
                    st4_cg(out + NB + gl * R + 4 * kk, vh);
                    st4_cg(out + 2 * NB + gl * R + 4 * kk, vq);
                }
                __syncwarp();
            }
            if (on && bad) err |= kErrSingular;
        }
        if (err) atomicOr(a.err, err);
        __syncwarp();
    }
    __syncthreads();
    if (w == 0) tmem_free<kFacColumns>(tmem_base);
}

// The factored rows of one segment as a lane holds them for its sub-steps,
// with the warp-scan multipliers.  hk[lv] / qk[lv] are zero on the lanes a
// scan level does not combine, and lane 0's a/d of row 0 and lane 31's c/d of
// the last row are zero, so the scans need no lane predicates.
template <bool SRC>
struct Coef {
    double inv[kR];      // 1 / d_i
    double h[kR];        // a_i / d_i      (forward recurrence)
    double q[kR];        // c_i / d_i      (back substitution)
    double sd[SRC ? kR : 1];  // dt * source_i / d_i
    double hk[5], qk[5];
    // products of h over the lower and upper half of the lane's rows, and of
    // q likewise: the local passes run as two half-length chains
    double hlo, hhi, qlo, qhi;
};

// The lane's rows of three arrays at in[0..3nb) (64 contiguous bytes each).
__device__ __forceinline__ void load_rows(const double *in, int lane, double X[kR], double Y[kR], double Z[kR])
{
    const int row0 = lane * kR;
#pragma unroll
    for (int r = 0; r < kR; r += 4) {
        ld4_cg(in + row0 + r, X + r);
        ld4_cg(in + NB + row0 + r, Y + r);
        ld4_cg(in + 2 * NB + row0 + r, Z + r);
    }
}

template <bool SRC>
__device__ __forceinline__ void scan_multipliers(Coef<SRC> &F, int lane);

// The rest of Coef once inv, h, q hold the lane's factored rows: the source
// term and the scan multipliers.
template <bool SRC>
__device__ __forceinline__ void finish_coef(Coef<SRC> &F, const double *src, double dt, int lane)
{
    const int row0 = lane * kR;
    if (lane == 0) F.h[0] = 0.0;
    if (lane == 31) F.q[kR - 1] = 0.0;
    if (SRC) {
#pragma unroll
        for (int r = 0; r < kR; r += 4) {
            double v[4];
            ld4_cg(src + row0 + r, v);
#pragma unroll
            for (int i = 0; i < 4; i++) F.sd[r + i] = (dt * v[i]) * F.inv[r + i];
        }
    }
    scan_multipliers<SRC>(F, lane);
}

// The half-chain products (hlo, hhi, qlo, qhi) and the warp-scan
// multipliers (hk, qk) of the lane's h and q rows.
template <bool SRC>
__device__ __forceinline__ void scan_multipliers(Coef<SRC> &F, int lane)
{
    double hlo = 1.0, hhi = 1.0, qlo = 1.0, qhi = 1.0;
#pragma unroll
    for (int r = 0; r < kR / 2; r++) {
        hlo *= F.h[r];
        qlo *= F.q[r];
        hhi *= F.h[r + kR / 2];
        qhi *= F.q[r + kR / 2];
    }
    F.hlo = hlo;
    F.hhi = hhi;
    F.qlo = qlo;
    F.qhi = qhi;
    double H = hlo * hhi, Q = qlo * qhi;
#pragma unroll
    for (int lv = 0; lv < 5; lv++) {
        const int off = 1 << lv;
        F.hk[lv] = (lane >= off) ? H : 0.0;
        F.qk[lv] = (lane + off < 32) ? Q : 0.0;
        const double Hu = sup(H, off), Qd = sdn(Q, off);
        if (lane >= off) H *= Hu;
        if (lane + off < 32) Q *= Qd;
    }
}

template <bool SRC>
__device__ __forceinline__ void load_coef(Coef<SRC> &F, const double *fac, const double *src, double dt,
                                          int lane)
{
    load_rows(fac, lane, F.inv, F.h, F.q);
    finish_coef<SRC>(F, src, dt, lane);
}

// One implicit sub-step: N <- M^{-1} (N + dt src) with the factored M.
// A shuffle from a lane outside the warp returns the caller's own (finite)
// value, which the zero multipliers discard exactly.  Each local pass runs
// as two independent half-length chains joined by one multiply-add, and the
// second pass seeds its upper (lower) half from the scanned carry directly,
// so no dependent chain is longer than half the lane's rows plus one.
template <bool SRC>
__device__ __forceinline__ void substep(const Coef<SRC> &F, double N[kR])
{
    constexpr int H2 = kR / 2;
    // forward: z_i = y_i + h_i z_{i-1}, y = N / d + dt src / d
    double alo = 0.0, ahi = 0.0;
#pragma unroll
    for (int r = 0; r < H2; r++) {
        N[r] = SRC ? fma(N[r], F.inv[r], F.sd[r]) : N[r] * F.inv[r];
        N[r + H2] = SRC ? fma(N[r + H2], F.inv[r + H2], F.sd[r + H2]) : N[r + H2] * F.inv[r + H2];
        alo = fma(F.h[r], alo, N[r]);
        ahi = fma(F.h[r + H2], ahi, N[r + H2]);
    }
    double acc = fma(F.hhi, alo, ahi);
#pragma unroll
    for (int lv = 0; lv < 5; lv++) acc = fma(F.hk[lv], sup(acc, 1 << lv), acc);
    const double cin = sup(acc, 1);
    double plo = cin, phi = fma(F.hlo, cin, alo);
#pragma unroll
    for (int r = 0; r < H2; r++) {
        plo = fma(F.h[r], plo, N[r]);
        phi = fma(F.h[r + H2], phi, N[r + H2]);
        N[r] = plo;
        N[r + H2] = phi;
    }
    // back substitution: x_i = z_i + q_i x_{i+1}
    alo = 0.0;
    ahi = 0.0;
#pragma unroll
    for (int r = H2 - 1; r >= 0; r--) {
        alo = fma(F.q[r], alo, N[r]);
        ahi = fma(F.q[r + H2], ahi, N[r + H2]);
    }
    acc = fma(F.qlo, ahi, alo);
#pragma unroll
    for (int lv = 0; lv < 5; lv++) acc = fma(F.qk[lv], sdn(acc, 1 << lv), acc);
    const double cout = sdn(acc, 1);
    phi = cout;
    plo = fma(F.qhi, cout, ahi);
#pragma unroll
    for (int r = H2 - 1; r >= 0; r--) {
        phi = fma(F.q[r + H2], phi, N[r + H2]);
        plo = fma(F.q[r], plo, N[r]);
        N[r + H2] = phi;
        N[r] = plo;
    }
}

// The steps kernel's registers bound its occupancy: warps are spread over
// the SM's four sub-partitions, each with a quarter of the register file, so
// at 512 bins (16 rows a lane) 8 warps per SM allow 255 registers a thread
// and 12 allow 168, at 256 bins 16 allow 128 and 20 allow 102.  The
// kSolveScanShared variant keeps the per-segment constants that a sub-step
// only reads -- dt src / d of each row and the ten scan multipliers -- in the
// warp's slice of shared memory ([r][lane] and [level][lane], one
// conflict-free 8-byte read each per sub-step) instead of registers, for the
// larger warp count.  The kSolveScanRhs variant also moves 1 / d of each
// row there, as (1 / d, dt src / d) pairs ([r][lane], one conflict-free
// 16-byte read per row and sub-step): the lane then holds only N, h and q
// (about 100 registers at 512 bins), for 16 warps per SM at 512 bins and 24
// at 256 with one warp per block (12 and 20 with two).
constexpr int kCoefSmemDoubles = NB + 10 * 32;       // per warp: dt src / d, hk, qk
constexpr int kRhsSmemDoubles = 2 * NB + 10 * 32;    // per warp: (1 / d, dt src / d), hk, qk

// substep() with the per-segment constants of the warp's shared-memory slice
// wsm.  RHS false (kSolveScanShared): dt src / d at wsm[r * 32 + lane] (SRC),
// the scan multipliers at wsm[NB + lv * 32 + lane] (hk) and
// wsm[NB + (5 + lv) * 32 + lane] (qk).  RHS true (kSolveScanRhs): the pair
// (1 / d, dt src / d) of row r at double2 index r * 32 + lane, hk and qk
// after the 2 NB doubles of pairs.  Same arithmetic as substep().
template <bool SRC, bool RHS>
__device__ __forceinline__ void substep_sm(const Coef<SRC> &F, const double *wsm, int lane, double N[kR])
{
    constexpr int H2 = kR / 2;
    const double *sm = wsm + lane;
    const double2 *rhs = reinterpret_cast<const double2 *>(wsm) + lane;
    const double *hk = sm + (RHS ? 2 * NB : NB), *qk = hk + 5 * 32;
    double alo = 0.0, ahi = 0.0;
#pragma unroll
    for (int r = 0; r < H2; r++) {
        if (RHS) {
            const double2 u = rhs[r * 32], v = rhs[(r + H2) * 32];
            N[r] = SRC ? fma(N[r], u.x, u.y) : N[r] * u.x;
            N[r + H2] = SRC ? fma(N[r + H2], v.x, v.y) : N[r + H2] * v.x;
        } else {
            N[r] = SRC ? fma(N[r], F.inv[r], sm[r * 32]) : N[r] * F.inv[r];
            N[r + H2] = SRC ? fma(N[r + H2], F.inv[r + H2], sm[(r + H2) * 32]) : N[r + H2] * F.inv[r + H2];
        }
        alo = fma(F.h[r], alo, N[r]);
        ahi = fma(F.h[r + H2], ahi, N[r + H2]);
    }
    double acc = fma(F.hhi, alo, ahi);
#pragma unroll
    for (int lv = 0; lv < 5; lv++) acc = fma(hk[lv * 32], sup(acc, 1 << lv), acc);
    const double cin = sup(acc, 1);
    double plo = cin, phi = fma(F.hlo, cin, alo);
#pragma unroll
    for (int r = 0; r < H2; r++) {
        plo = fma(F.h[r], plo, N[r]);
        phi = fma(F.h[r + H2], phi, N[r + H2]);
        N[r] = plo;
        N[r + H2] = phi;
    }
    alo = 0.0;
    ahi = 0.0;
#pragma unroll
    for (int r = H2 - 1; r >= 0; r--) {
        alo = fma(F.q[r], alo, N[r]);
        ahi = fma(F.q[r + H2], ahi, N[r + H2]);
    }
    acc = fma(F.qlo, ahi, alo);
#pragma unroll
    for (int lv = 0; lv < 5; lv++) acc = fma(qk[lv * 32], sdn(acc, 1 << lv), acc);
    const double cout = sdn(acc, 1);
    phi = cout;
    plo = fma(F.qhi, cout, ahi);
#pragma unroll
    for (int r = H2 - 1; r >= 0; r--) {
        phi = fma(F.q[r + H2], phi, N[r + H2]);
        plo = fma(F.q[r], plo, N[r]);
        N[r + H2] = phi;
        N[r] = plo;
    }
}

// kSolveScanRhs's coefficient load: the (1 / d, dt src / d) pairs of the
// lane's rows go from the factored rows (and the source) straight to the
// warp's slice, h and q into registers, and the scan multipliers, formed as
// load_coef forms them, into the slice after the pairs.
template <bool SRC>
__device__ __forceinline__ void load_coef_rhs(Coef<SRC> &F, const double *fac, const double *src, double dt,
                                              int lane, double *wsm)
{
    const int row0 = lane * kR;
    double2 *rhs = reinterpret_cast<double2 *>(wsm) + lane;
    __syncwarp();   // the previous run's reads of the slice are done
#pragma unroll
    for (int r = 0; r < kR; r += 4) {
        double vi[4], vs[4] = {0.0, 0.0, 0.0, 0.0};
        ld4_cg(fac + row0 + r, vi);
        if (SRC) ld4_cg(src + row0 + r, vs);
#pragma unroll
        for (int i = 0; i < 4; i++) rhs[(r + i) * 32] = make_double2(vi[i], SRC ? (dt * vs[i]) * vi[i] : 0.0);
    }
#pragma unroll
    for (int r = 0; r < kR; r += 4) {
        ld4_cg(fac + NB + row0 + r, F.h + r);
        ld4_cg(fac + 2 * NB + row0 + r, F.q + r);
    }
    if (lane == 0) F.h[0] = 0.0;
    if (lane == 31) F.q[kR - 1] = 0.0;
    scan_multipliers<SRC>(F, lane);
    double *hk = wsm + 2 * NB + lane;
#pragma unroll
    for (int lv = 0; lv < 5; lv++) {
        hk[lv * 32] = F.hk[lv];
        hk[(5 + lv) * 32] = F.qk[lv];
    }
    __syncwarp();
}

// ---------------------------------------------------------------------------
// Short-chain sub-step (kSolveScan4).  substep() runs, per sub-step, the
// forward recurrence (local pass, 5-level warp scan, carry shuffle, second
// local pass) and then the back substitution the same way, one after the
// other: two scans of six dependent shuffles each plus four dependent local
// passes.  This form shortens that chain in two ways.
//
// * Radix-4 warp scans: the carry into lane i is gathered from the
//   aggregates of lanes i-1..i-4 (four shuffles issued together), then from
//   those partial carries at lanes i-4, i-8, i-12, then at i-16: three
//   dependent shuffle levels instead of six, exclusive directly.
// * The back substitution's local pass runs on the forward pass's raw
//   (zero-carry) values while the forward scan is in flight.  Both
//   recurrences are linear, so the true back aggregate of the lane is the raw
//   one plus per-segment constants times the forward carry; the forward
//   carry then reaches the rows as z = raw + (product of h) carry, a chain of
//   multiplies that runs while the back scan is in flight.
//
// The sums are the same as substep()'s, regrouped (results agree to
// rounding, not bit for bit).
struct Scan4 {
    double fw[3];    // forward level 1: weights of the aggregates of lanes i-2, i-3, i-4 (i-1: 1)
    double fp[4];    // forward levels 2, 3: products of H over lanes i-4..i-1, i-8.., i-12.., i-16..
    double bw[3];    // the same for the back substitution (lanes i+2, i+3, i+4)
    double bp[4];
    double kh;       // back aggregate of the upper half's carry response to z at its first row - 1
    double qk, kc;   // qlo kh, and the full back aggregate's response to the forward carry
};

// Forward exclusive scan: the carry into this lane (z at the last row of the
// lane below), from each lane's zero-carry aggregate a.  Weights outside the
// warp are zero, so the shuffles need no lane predicates (a shuffle from
// outside the warp returns the caller's own finite value).
__device__ __forceinline__ double scan4_up(double a, const double fw[3], const double fp[4], int lane)
{
    const double s1 = sup(a, 1), s2 = sup(a, 2), s3 = sup(a, 3), s4 = sup(a, 4);
    const double S = fma(fw[0], s2, lane >= 1 ? s1 : 0.0) + fma(fw[2], s4, fw[1] * s3);
    const double t4 = sup(S, 4), t8 = sup(S, 8), t12 = sup(S, 12);
    const double E = fma(fp[0], t4, S) + fma(fp[2], t12, fp[1] * t8);
    return fma(fp[3], sup(E, 16), E);
}

// Back exclusive scan: the carry into this lane from above (x at the first
// row of the lane above).
__device__ __forceinline__ double scan4_down(double a, const double bw[3], const double bp[4], int lane)
{
    const double s1 = sdn(a, 1), s2 = sdn(a, 2), s3 = sdn(a, 3), s4 = sdn(a, 4);
    const double S = fma(bw[0], s2, lane <= 30 ? s1 : 0.0) + fma(bw[2], s4, bw[1] * s3);
    const double t4 = sdn(S, 4), t8 = sdn(S, 8), t12 = sdn(S, 12);
    const double E = fma(bp[0], t4, S) + fma(bp[2], t12, bp[1] * t8);
    return fma(bp[3], sdn(E, 16), E);
}

// The Scan4 constants of the lane's coefficients (after load_coef).
template <bool SRC>
__device__ __forceinline__ void make_scan4(const Coef<SRC> &F, Scan4 &R, int lane)
{
    const double H = F.hlo * F.hhi, Q = F.qlo * F.qhi;   // products over the lane's rows
    {
        const double h1 = sup(H, 1), h2 = sup(H, 2), h3 = sup(H, 3), h4 = sup(H, 4);
        const double w3 = h1 * h2, w4 = w3 * h3, p4 = w4 * h4;
        const double p8 = p4 * sup(p4, 4);
        const double p12 = p8 * sup(p4, 8);
        const double p16 = p8 * sup(p8, 8);
        R.fw[0] = lane >= 2 ? h1 : 0.0;
        R.fw[1] = lane >= 3 ? w3 : 0.0;
        R.fw[2] = lane >= 4 ? w4 : 0.0;
        R.fp[0] = lane >= 4 ? p4 : 0.0;
        R.fp[1] = lane >= 8 ? p8 : 0.0;
        R.fp[2] = lane >= 12 ? p12 : 0.0;
        R.fp[3] = lane >= 16 ? p16 : 0.0;
    }
    {
        const double q1 = sdn(Q, 1), q2 = sdn(Q, 2), q3 = sdn(Q, 3), q4 = sdn(Q, 4);
        const double w3 = q1 * q2, w4 = w3 * q3, p4 = w4 * q4;
        const double p8 = p4 * sdn(p4, 4);
        const double p12 = p8 * sdn(p4, 8);
        const double p16 = p8 * sdn(p8, 8);
        R.bw[0] = lane <= 29 ? q1 : 0.0;
        R.bw[1] = lane <= 28 ? w3 : 0.0;
        R.bw[2] = lane <= 27 ? w4 : 0.0;
        R.bp[0] = lane <= 27 ? p4 : 0.0;
        R.bp[1] = lane <= 23 ? p8 : 0.0;
        R.bp[2] = lane <= 19 ? p12 : 0.0;
        R.bp[3] = lane <= 15 ? p16 : 0.0;
    }
    // the back aggregate of each half applied to the half's forward carry
    // response (the running products of h from the half's first row)
    constexpr int H2 = kR / 2;
    double clo[H2], chi[H2];
    double c0 = 1.0, c1 = 1.0;
#pragma unroll
    for (int r = 0; r < H2; r++) {
        c0 *= F.h[r];
        c1 *= F.h[r + H2];
        clo[r] = c0;
        chi[r] = c1;
    }
    double kl = 0.0, kh = 0.0;
#pragma unroll
    for (int r = H2 - 1; r >= 0; r--) {
        kl = fma(F.q[r], kl, clo[r]);
        kh = fma(F.q[r + H2], kh, chi[r]);
    }
    R.kh = kh;
    R.qk = F.qlo * kh;
    R.kc = fma(R.qk, F.hlo, kl);
}

template <bool SRC>
__device__ __forceinline__ void substep4(const Coef<SRC> &F, const Scan4 &R, int lane, double N[kR])
{
    constexpr int H2 = kR / 2;
    // forward, zero carry into each half: N <- the raw chain values
    double alo = 0.0, ahi = 0.0;
#pragma unroll
    for (int r = 0; r < H2; r++) {
        const double ylo = SRC ? fma(N[r], F.inv[r], F.sd[r]) : N[r] * F.inv[r];
        const double yhi = SRC ? fma(N[r + H2], F.inv[r + H2], F.sd[r + H2]) : N[r + H2] * F.inv[r + H2];
        alo = fma(F.h[r], alo, ylo);
        ahi = fma(F.h[r + H2], ahi, yhi);
        N[r] = alo;
        N[r + H2] = ahi;
    }
    const double af = fma(F.hhi, alo, ahi);
    // back aggregates of the raw values, independent of the forward scan
    double blo = 0.0, bhi = 0.0;
#pragma unroll
    for (int r = H2 - 1; r >= 0; r--) {
        blo = fma(F.q[r], blo, N[r]);
        bhi = fma(F.q[r + H2], bhi, N[r + H2]);
    }
    const double bpre = fma(R.qk, alo, fma(F.qlo, bhi, blo));
    const double cin = scan4_up(af, R.fw, R.fp, lane);
    const double zh = fma(F.hlo, cin, alo);          // z at the lower half's last row
    const double cout = scan4_down(fma(R.kc, cin, bpre), R.bw, R.bp, lane);
    const double bhi_t = fma(R.kh, zh, bhi);         // the upper half's true back aggregate
    // the forward carry's response: z = raw + (running product of h) carry
    double d = cin, e = zh;
#pragma unroll
    for (int r = 0; r < H2; r++) {
        d *= F.h[r];
        e *= F.h[r + H2];
        N[r] += d;
        N[r + H2] += e;
    }
    // back substitution: x_i = z_i + q_i x_{i+1}
    double phi = cout, plo = fma(F.qhi, cout, bhi_t);
#pragma unroll
    for (int r = H2 - 1; r >= 0; r--) {
        phi = fma(F.q[r + H2], phi, N[r + H2]);
        plo = fma(F.q[r], plo, N[r]);
        N[r + H2] = phi;
        N[r] = plo;
    }
}

// ---------------------------------------------------------------------------
// FP32-refined sub-step (the "precision" form of the chosen path): the solve
// of each sub-step in FP32 followed by one iterative-refinement sweep whose
// residual is formed in FP64, the result kept in FP64.
//
//   y   = N / d + dt src / d                       FP64 (the scaled right-hand side)
//   x0  = M^-1 y                                   FP32, the same two recurrences
//   rho = y - (u - h u_{-1}),  u = x0 - q x0_{+1}  FP64: r / d - M x0 / d with M = L U,
//                                                  L = (d, -a), U = (1, -c/d) the
//                                                  FP64 factors of the segment
//   e   = M^-1 rho                                 FP32
//   N   = x0 + e                                   FP64
//
// The FP32 solves see y scaled by a per-segment power of two s (exact), so
// that the largest |y| of the tracer is near 1 and the spectra, which span
// more decades than FP32 does, keep their dominant bins in range; rho is
// scaled by s 2^20.  The factored rows stay FP64 (the residual needs them);
// the multipliers of the FP32 recurrences are their FP32 roundings.
struct Coef32 {
    float h[kR], q[kR];
    float hk[5], qk[5];
    float hlo, hhi, qlo, qhi;
};

__device__ __forceinline__ float supf(float v, int d) { return __shfl_up_sync(kFull, v, d); }
__device__ __forceinline__ float sdnf(float v, int d) { return __shfl_down_sync(kFull, v, d); }

template <bool SRC>
__device__ __forceinline__ void make_coef32(const Coef<SRC> &F, Coef32 &G, int lane)
{
#pragma unroll
    for (int r = 0; r < kR; r++) {
        G.h[r] = (float)F.h[r];
        G.q[r] = (float)F.q[r];
    }
    float hlo = 1.0f, hhi = 1.0f, qlo = 1.0f, qhi = 1.0f;
#pragma unroll
    for (int r = 0; r < kR / 2; r++) {
        hlo *= G.h[r];
        qlo *= G.q[r];
        hhi *= G.h[r + kR / 2];
        qhi *= G.q[r + kR / 2];
    }
    G.hlo = hlo;
    G.hhi = hhi;
    G.qlo = qlo;
    G.qhi = qhi;
    float H = hlo * hhi, Q = qlo * qhi;
#pragma unroll
    for (int lv = 0; lv < 5; lv++) {
        const int off = 1 << lv;
        G.hk[lv] = (lane >= off) ? H : 0.0f;
        G.qk[lv] = (lane + off < 32) ? Q : 0.0f;
        const float Hu = supf(H, off), Qd = sdnf(Q, off);
        if (lane >= off) H *= Hu;
        if (lane + off < 32) Q *= Qd;
    }
}

// x <- M^-1 x in FP32, x holding the scaled right-hand side (substep's two
// recurrences without the 1/d and source step).
__device__ __forceinline__ void solve32(const Coef32 &G, float x[kR])
{
    constexpr int H2 = kR / 2;
    float alo = 0.0f, ahi = 0.0f;
#pragma unroll
    for (int r = 0; r < H2; r++) {
        alo = fmaf(G.h[r], alo, x[r]);
        ahi = fmaf(G.h[r + H2], ahi, x[r + H2]);
    }
    float acc = fmaf(G.hhi, alo, ahi);
#pragma unroll
    for (int lv = 0; lv < 5; lv++) acc = fmaf(G.hk[lv], supf(acc, 1 << lv), acc);
    const float cin = supf(acc, 1);
    float plo = cin, phi = fmaf(G.hlo, cin, alo);
#pragma unroll
    for (int r = 0; r < H2; r++) {
        plo = fmaf(G.h[r], plo, x[r]);
        phi = fmaf(G.h[r + H2], phi, x[r + H2]);
        x[r] = plo;
        x[r + H2] = phi;
    }
    alo = 0.0f;
    ahi = 0.0f;
#pragma unroll
    for (int r = H2 - 1; r >= 0; r--) {
        alo = fmaf(G.q[r], alo, x[r]);
        ahi = fmaf(G.q[r + H2], ahi, x[r + H2]);
    }
    acc = fmaf(G.qlo, ahi, alo);
#pragma unroll
    for (int lv = 0; lv < 5; lv++) acc = fmaf(G.qk[lv], sdnf(acc, 1 << lv), acc);
    const float cout = sdnf(acc, 1);
    phi = cout;
    plo = fmaf(G.qhi, cout, ahi);
#pragma unroll
    for (int r = H2 - 1; r >= 0; r--) {
        phi = fmaf(G.q[r + H2], phi, x[r + H2]);
        plo = fmaf(G.q[r], plo, x[r]);
        x[r + H2] = phi;
        x[r] = plo;
    }
}

// Power-of-two scale that brings the tracer's largest scaled right-hand side
// |N / d + dt src / d| near 1 (1 for an all-zero spectrum).
template <bool SRC>
__device__ __forceinline__ double refine_scale(const Coef<SRC> &F, const double N[kR])
{
    double m = 0.0;
#pragma unroll
    for (int r = 0; r < kR; r++) m = fmax(m, fabs(N[r] * F.inv[r]) + (SRC ? fabs(F.sd[r]) : 0.0));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_xor_sync(kFull, m, off));
    if (!(m > 0.0) || !isfinite(m)) return 1.0;
    int e = ilogb(m);
    e = max(-1000, min(1000, e));
    return ldexp(1.0, -e);
}

template <bool SRC>
__device__ __forceinline__ void substep_refined(const Coef<SRC> &F, const Coef32 &G, double N[kR], double s)
{
    const double inv_s = 1.0 / s, s2 = s * 1048576.0, inv_s2 = inv_s * (1.0 / 1048576.0);
    float x[kR], e[kR];
#pragma unroll
    for (int r = 0; r < kR; r++) {
        const double y = SRC ? fma(N[r], F.inv[r], F.sd[r]) : N[r] * F.inv[r];
        x[r] = (float)(y * s);
    }
    solve32(G, x);
    // u_r = x0_r - q_r x0_{r+1}; the row after the lane's last is the next
    // lane's first (the last lane's last q is zero, so its own value is harmless)
    const double xnext = sdn((double)x[0] * inv_s, 1);
    const double ulast = (double)x[kR - 1] * inv_s - F.q[kR - 1] * xnext;
    double uprev = sup(ulast, 1);   // lane 0: h of row 0 is zero
#pragma unroll
    for (int r = 0; r < kR; r++) {
        const double x0 = (double)x[r] * inv_s;
        const double x1 = (r < kR - 1) ? (double)x[r + 1] * inv_s : xnext;
        const double u = x0 - F.q[r] * x1;
        const double y = SRC ? fma(N[r], F.inv[r], F.sd[r]) : N[r] * F.inv[r];
        const double rho = (y - u) + F.h[r] * uprev;
        e[r] = (float)(rho * s2);
        uprev = u;
    }
    solve32(G, e);
#pragma unroll
    for (int r = 0; r < kR; r++) N[r] = (double)x[r] * inv_s + (double)e[r] * inv_s2;
}

// ---------------------------------------------------------------------------
// Warp PCR sub-step: parallel cyclic reduction of the tridiagonal system
// b_i x_i - a_i x_{i-1} - c_i x_{i+1} = N_i + dt src_i, the algorithm of the
// reference's solve_cc_pcr_kernel (src/fp_cuda_solver.cu:144-206) with one
// warp per system instead of one thread block: each lane keeps its R rows in
// registers, and at stride s every row combines with rows i - s and i + s
// read back from the warp's slice of shared memory (swizzled rows, so both
// partners of a lane's row r sit in distinct banks):
//   alpha = a_i / b_{i-s},  gamma = c_i / b_{i+s},
//   b <- b - alpha c_{i-s} - gamma a_{i+s},  a <- alpha a_{i-s},
//   c <- gamma c_{i+s},  d <- d + alpha d_{i-s} + gamma d_{i+s},
// log2(nb) levels, then x_i = d_i / b_i.  The rows a, b, c are rebuilt from
// the segment's factored rows (d = 1/inv, a = h d, c = q d,
// b = d + a q_{i-1}).  It does O(nb log nb) work and data movement per
// sub-step against the scan's O(nb); the autotuner times both.
struct PcrSmem {
    double a[kSw], b[kSw], c[kSw], d[kSw];
};

template <bool SRC>
__device__ __forceinline__ void pcr_rows_from_factored(Coef<SRC> &F, double cc[kR], int lane)
{
    // in place: inv -> b, h -> a, sd -> dt src; c into cc (q is read as the
    // previous row's multiplier, so it stays)
    const double q_in = sup(F.q[kR - 1], 1);   // q of the row before this lane's first
#pragma unroll
    for (int r = 0; r < kR; r++) {
        const double dd = 1.0 / F.inv[r];
        const double qprev = (r > 0) ? F.q[r - 1] : (lane > 0 ? q_in : 0.0);
        const double aa = F.h[r] * dd;
        cc[r] = F.q[r] * dd;
        F.inv[r] = dd + aa * qprev;
        if (SRC) F.sd[r] = F.sd[r] * dd;
        F.h[r] = aa;
    }
}

template <bool SRC>
__device__ __forceinline__ void substep_pcr(const Coef<SRC> &F, const double cc[kR], double N[kR], PcrSmem &sm,
                                            int lane)
{
    double a[kR], b[kR], c[kR];
#pragma unroll
    for (int r = 0; r < kR; r++) {
        a[r] = F.h[r];
        b[r] = F.inv[r];
        c[r] = cc[r];
        N[r] = SRC ? N[r] + F.sd[r] : N[r];
    }
#pragma unroll 1
    for (int st = 1; st < NB; st <<= 1) {
        __syncwarp();
#pragma unroll
        for (int r = 0; r < kR; r++) {
            const int o = r * kPitch + lane;
            sm.a[o] = a[r];
            sm.b[o] = b[r];
            sm.c[o] = c[r];
            sm.d[o] = N[r];
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < kR; r++) {
            const int m = lane * kR + r;
            double na = 0.0, nb = b[r], nc = 0.0, nd = N[r];
            if (m - st >= 0) {
                const int o = swz(m - st);
                const double al = a[r] / sm.b[o];
                na = al * sm.a[o];
                nb -= al * sm.c[o];
                nd += al * sm.d[o];
            }
            if (m + st < NB) {
                const int o = swz(m + st);
                const double ga = c[r] / sm.b[o];
                nc = ga * sm.c[o];
                nb -= ga * sm.a[o];
                nd += ga * sm.d[o];
            }
            a[r] = na;
            b[r] = nb;
            c[r] = nc;
            N[r] = nd;
        }
    }
#pragma unroll
    for (int r = 0; r < kR; r++) N[r] = N[r] / b[r];
}

// Sub-step solvers of the steps kernel: the FP64 warp-scan Thomas (its
// per-segment constants in registers, or in shared memory to leave registers
// for more warps), the short-chain FP64 form (radix-4 scans, back pass
// overlapping the forward scan), the warp scan with FP32 solves refined by
// an FP64 residual, and warp PCR.
enum { kSolveScan = 0, kSolveRefined = 1, kSolvePcr = 2, kSolveScanShared = 3, kSolveScanRhs = 4,
       kSolveScan4 = 5, kSolvePacked = 6 };

// Steps kernel: warp w of block b runs every segment [g0, g1) of tracer
// t0 + b * WPB + w for species S with sub-step solver SOLVER.
template <int S, bool SRC, int SOLVER, int WPB>
__global__ void __launch_bounds__(WPB * 32,
                                  (SOLVER == kSolveScanShared ? (NB <= 256 ? 20 : 12)
                                   : SOLVER == kSolveScanRhs  ? (WPB == 1 ? (NB <= 256 ? 24 : 16) : (NB <= 256 ? 20 : 12))
                                                              : (NB <= 256 ? 16 : 8)) / WPB)
    steps_kernel(FusedParams P)
{
    extern __shared__ double4 steps_smem[];
    constexpr bool kSm = SOLVER == kSolveScanShared;
    constexpr bool kRhs = SOLVER == kSolveScanRhs;
    const int w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int tl = blockIdx.x * WPB + w;
    if (tl >= P.nt) return;
    const int t = P.t0 + tl;
    const SnapArgs &a = P.a;
    const int row0 = lane * kR;
    double *Nrow = (P.cal_spec ? P.cal_spec + (size_t)tl * NB : (S == 0 ? a.crp : a.cre) + (size_t)t * NB) + row0;
    double N[kR];
#pragma unroll
    for (int r = 0; r < kR; r += 4) ld4(Nrow + r, N + r);
    const double *qsrc = (S == 0) ? a.qpi : a.qepri;
    Coef<SRC> F;
    Coef32 G;
    Scan4 R4;
    double cc[SOLVER == kSolvePcr ? kR : 1];
    PcrSmem *pcr_sm = reinterpret_cast<PcrSmem *>(steps_smem) + w;
    double *coef_sm = reinterpret_cast<double *>(steps_smem) + (size_t)w * (kRhs ? kRhsSmemDoubles : kCoefSmemDoubles);
    double scale = 1.0;
    int budget = P.cal_steps > 0 ? P.cal_steps : 0x7fffffff;
    const int nslot = P.g1 - P.g0;
#pragma unroll 1
    for (int gi = 0; gi < nslot && budget > 0; gi++) {
        const SegPre *__restrict__ pre = P.pre + (size_t)gi * P.nt + tl;
        const int flags = pre->flags;
        if (!(flags & kPreActive)) continue;
        SegInfo g{};
        g.windowed = (flags & kPreWindowed) ? 1 : 0;
        g.sl = pre->sl;
        g.el = pre->el;
        g.steps = pre->steps;
        g.dt = pre->dt;
        // the next segment's rows (Dpp-on set) and source into L2 while this
        // segment's sub-steps run: its loads then wait on L2, not on DRAM
        if (gi + 1 < nslot) {
            const double *nf = fac_ptr(P, S, gi + 1, 0, tl) + row0;
            if (lane < 2)   // and the next segment's scalars this loop reads (dt .. steps of its SegPre)
                prefetch_l2(reinterpret_cast<const char *>(P.pre + (size_t)(gi + 1) * P.nt + tl) +
                            (lane ? offsetof(SegPre, steps) : offsetof(SegPre, dt)));
            prefetch_l2(nf);
            prefetch_l2(nf + NB);
            prefetch_l2(nf + 2 * NB);
            if (SRC && S == 1 && P.inje) prefetch_l2(P.inje + ((size_t)(gi + 1) * P.nt + tl) * NB + row0);
        }
        if (S == 0 && P.np_seg && !P.cal_spec) {
            double *o = P.np_seg + ((size_t)gi * P.nt + tl) * NB + row0;
#pragma unroll
            for (int r = 0; r < kR; r += 4) st4_cg(o + r, N + r);
        }
        const double *src = nullptr;
        if (SRC) {
            src = (S == 1 && P.inje) ? P.inje + ((size_t)gi * P.nt + tl) * NB
                                     : qsrc + (size_t)t * NB;
        }
        // runs of sub-steps with one coefficient set: Dpp off before the
        // window, on inside it, off after it (all on when not windowed)
        const int sl = g.windowed ? min(max(g.sl, 0), g.steps) : 0;
        const int el = g.windowed ? min(max(g.el, sl), g.steps) : g.steps;
        int cur = -1;
#pragma unroll 1
        for (int k = 0; k < 3; k++) {
            const int want = (k == 1) ? 0 : 1;
            int run_n = (k == 0) ? sl : (k == 1 ? el - sl : g.steps - el);
            if (run_n <= 0) continue;
            if (want >= P.sets) {   // no off set in the workspace: report, leave N as it was
                if (lane == 0) atomicOr(a.err, kErrBadInput);
                return;
            }
            run_n = min(run_n, budget);
            budget -= run_n;
            if (want != cur) {
                if (kRhs) load_coef_rhs<SRC>(F, fac_ptr(P, S, gi, want, tl), src, g.dt, lane, coef_sm);
                else load_coef<SRC>(F, fac_ptr(P, S, gi, want, tl), src, g.dt, lane);
                if (SOLVER == kSolveRefined) make_coef32<SRC>(F, G, lane);
                if (SOLVER == kSolveScan4) make_scan4<SRC>(F, R4, lane);
                if (SOLVER == kSolvePcr) pcr_rows_from_factored<SRC>(F, cc, lane);
                if (kSm) {
                    __syncwarp();   // the previous run's reads of the slice are done
                    if (SRC) {
#pragma unroll
                        for (int r = 0; r < kR; r++) coef_sm[r * 32 + lane] = F.sd[r];
                    }
#pragma unroll
                    for (int lv = 0; lv < 5; lv++) {
                        coef_sm[NB + lv * 32 + lane] = F.hk[lv];
                        coef_sm[NB + (5 + lv) * 32 + lane] = F.qk[lv];
                    }
                    __syncwarp();
                }
                cur = want;
            }
            if (SOLVER == kSolveRefined) {
                scale = refine_scale<SRC>(F, N);
#pragma unroll 1
                for (int istep = 0; istep < run_n; istep++) substep_refined<SRC>(F, G, N, scale);
            } else if (SOLVER == kSolvePcr) {
#pragma unroll 1
                for (int istep = 0; istep < run_n; istep++) substep_pcr<SRC>(F, cc, N, *pcr_sm, lane);
            } else if (kSm) {
#pragma unroll 2
                for (int istep = 0; istep < run_n; istep++) substep_sm<SRC, false>(F, coef_sm, lane, N);
            } else if (kRhs) {
#pragma unroll 1
                for (int istep = 0; istep < run_n; istep++) substep_sm<SRC, true>(F, coef_sm, lane, N);
            } else if (SOLVER == kSolveScan4) {
#pragma unroll 2   // two sub-steps per trip, as for substep (no spills at 254 registers)
                for (int istep = 0; istep < run_n; istep++) substep4<SRC>(F, R4, lane, N);
            } else {
                // two sub-steps per trip: the carried spectrum keeps its
                // registers across the loop (fewer copies per sub-step)
#pragma unroll 2
                for (int istep = 0; istep < run_n; istep++) substep<SRC>(F, N);
            }
            if (budget <= 0) break;
        }
    }
#pragma unroll
    for (int r = 0; r < kR; r += 4) st4(Nrow + r, N + r);
}

// ---------------------------------------------------------------------------
// Packed steps kernel: 16 rows a lane at every bin count, so NB / 16 lanes (8,
// 16 or 32) run a tracer and a warp runs 4, 2 or 1 of them.
//
// What bounds a sub-step (measured on B200): a DFMA with three different
// register operands takes 3 cycles of a scheduler, one that shares an operand
// with the instruction before it 2.2, a DMUL or DADD 2; a dependent FP64
// instruction waits 8; a 64-bit shuffle takes 25 and two cycles of the whole
// SM.  A warp per tracer at 128 bins (4 rows a lane) spends more on its twelve
// shuffles than on its arithmetic, and at 512 bins (16 rows) eight warps per
// SM wait on their own chains.  So:
//
// * 16 rows a lane at 128 and 256 bins too: the scans of a sub-step serve
//   four (two) tracers.
// * The solve in block form.  Each lane solves its 16 rows with zero carries
//   (forward chain, back chain); the solution is that plus the rows'
//   responses to the two carries, x_r = raw_r + g_r cin + e_r cout, with
//     c_r = h_0 .. h_r,  e_r = q_r .. q_15,  g_15 = c_15, g_r = c_r + q_r g_r+1
//   constants of the segment.  cin is the exclusive scan of the forward
//   chains' ends over the tracer's lanes, cout that of the back chains' ends
//   plus g_0 cin.  The responses are independent rows sharing an operand.
// * Both scans run under a chain.  While cout is still being scanned the next
//   sub-step's forward chain runs on x without cout; its response to cout,
//   E_r = e_r / d_r + h_r E_r-1, is added to the rows afterwards, during the
//   forward scan and the back chain.
// * The constants g, 1/d, E and dt src/d sit in tensor memory (96 or 128 of
//   the 128 columns that a block of four warps holds) and are read a few rows
//   ahead: tcgen05.ld is there after ~17 cycles, and the shared memory's
//   bandwidth would not do.  N, h and q stay in registers.  That fits 168 of
//   them: 12 warps per SM instead of 8.
// * The next segment's rows come into shared memory by cp.async during the
//   present one: all warps of an SM keep step, and would ask for 190 KB at once.
//
// All terms are nonnegative (an M-matrix, nonnegative spectra), so nothing
// cancels.  A row is rounded five times a sub-step where the two-pass form rounds
// three times: after 500 sub-steps the mean 2-norm error against 80 bits is 1.04
// of that form's with the same factors (3e-15; the largest element's, 1e-12 at
// the spectra's far ends, is the coefficients' and the same).
//
// Measured, whole kernel with its segment switches, before (a warp per tracer)
// and now: 131,072 tracers x 500 sub-steps of 128 bins 8.20 -> 4.42 ms, of 512
// bins 24.6 -> 20.8 ms (with a source 25.4 -> 21.0), 65,536 of 256 bins 6.24 ->
// 5.2 ms; 30,011 with 11 to 500 sub-steps 0.60 -> 0.25 ms; 64 tracers 152 ->
// 130 us.  FP64 pipe 49 % at 512 bins and 4,096 tracers, stalls per issue:
// dependent FP64 1.9, shuffles and tensor memory 0.7 to 1.2.
constexpr int kPkWarps = 4;               // one per TMEM lane quarter
constexpr int kPkColumns = 128;           // TMEM columns of a block: 3 blocks per SM hold 384 of 512

__device__ __forceinline__ double pk_up(double v, int d) { return __shfl_up_sync(kFull, v, d, kPkLanes); }
__device__ __forceinline__ double pk_down(double v, int d) { return __shfl_down_sync(kFull, v, d, kPkLanes); }

// TMEM columns of the four rows of chunk k: their (g, 1/d) pairs, their E,
// their dt src/d.
__device__ __forceinline__ unsigned pk_fwd(unsigned tm, int k) { return tm + k * 16; }
__device__ __forceinline__ unsigned pk_resp(unsigned tm, int k) { return tm + 64 + k * 8; }
__device__ __forceinline__ unsigned pk_src(unsigned tm, int k) { return tm + 96 + k * 8; }

// The walk of each lane's tracer through its runs of sub-steps, kept in
// shared memory (each lane its own copy): it is touched once a run, and in
// registers it would push the sub-step's constants out of theirs.
constexpr int kPkThreads = kPkWarps * 32;
struct PkWalk {
    int tl[kPkThreads];      // tracer within the chunk
    int gi[kPkThreads];      // segment
    int run[kPkThreads];     // run within the segment: before, inside, after the Dpp window
    int rem[kPkThreads];     // sub-steps left in the run; < 0: no run left
    int sl[kPkThreads], el[kPkThreads], steps[kPkThreads];
    int pgi[kPkThreads], pset[kPkThreads];   // segment and set whose rows the row buffer holds
    double dt[kPkThreads];
};
// The next segment's scalars of each group (the last 16 bytes of its SegPre, and dt).
struct PkNext {
    int4 meta[kPkWarps * kPkTracers];   // flags, sl, el, steps
    double dt[kPkWarps * kPkTracers];
};
static_assert(offsetof(SegPre, flags) % 16 == 0 && offsetof(SegPre, steps) == offsetof(SegPre, flags) + 12 &&
                  sizeof(SegPre) % 16 == 0 && offsetof(SegPre, dt) % 8 == 0,
              "the packed steps kernel copies flags .. steps as 16 bytes");

// Row buffer of a warp: the arrays 1/d, a/d, c/d (and the source) of its
// groups' next run, 512 doubles each, filled by cp.async while the present
// run's sub-steps go on.  Without it all warps of an SM, which keep step, ask
// for their rows at once at each segment: 190 KB an SM, 12 % of the kernel's
// time at 512 bins.  Copies are contiguous across the lanes; 16-byte piece c
// of a group's array (owner lane c / 8) sits at c ^ (owner & 7), so that the
// lanes' reads of their own 128 bytes meet no bank twice.
__device__ __forceinline__ int pk_piece(int c) { return c ^ ((c >> 3) & 7); }

template <int S, bool SRC>
__device__ __forceinline__ void pk_fetch(const FusedParams &P, double *buf, int gi, int set, int tl, int gl)
{
    const double *f = fac_ptr(P, S, gi, set, tl);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int c = i * kPkLanes + gl;
#pragma unroll
        for (int k = 0; k < 3; k++) cp_async16(buf + k * 512 + 2 * pk_piece(c), f + k * NB + 2 * c, true);
    }
    if (SRC) {
        const double *src = (S == 1 && P.inje) ? P.inje + ((size_t)gi * P.nt + tl) * NB
                                               : (S == 0 ? P.a.qpi : P.a.qepri) + (size_t)(P.t0 + tl) * NB;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int c = i * kPkLanes + gl;
            cp_async16(buf + 3 * 512 + 2 * pk_piece(c), src + 2 * c, true);
        }
    }
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// the lane's 16 rows of array k
__device__ __forceinline__ void pk_read(const double *buf, int k, int gl, double v[kPkRows])
{
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const double2 x = *reinterpret_cast<const double2 *>(buf + k * 512 + 2 * pk_piece(gl * 8 + j));
        v[2 * j] = x.x;
        v[2 * j + 1] = x.y;
    }
}

// Species S of the chunk's tracers, every segment [g0, g1).  Tracers come in
// the chunk's order (P.order: by falling sub-step count, so that the tracers
// of a warp and of a block end together); each group of kPkLanes lanes walks
// its own tracer's runs of sub-steps (the segments, split by the Dpp window)
// and the warp advances all its groups by the smallest remaining run.  When
// any group starts a run, all load their constants again (the others' are
// what they were).  A group without work holds the identity (1/d = 1, the
// rest 0), which leaves finite rows as they are.
template <int S, bool SRC>
__global__ void __launch_bounds__(kPkThreads, 3) steps_packed_kernel(FusedParams P)
{
    constexpr int R = kPkRows;
    extern __shared__ double4 steps_smem[];
    __shared__ unsigned tmem_base;
    __shared__ PkWalk walk_smem;
    __shared__ PkNext next;
    volatile PkWalk &walk = walk_smem;
    const int me = threadIdx.x, w = me >> 5, gl = me & (kPkLanes - 1);
    if (w == 0) {
        tmem_alloc<kPkColumns>(&tmem_base);
    }
    __syncthreads();
    const unsigned tm = tmem_base + ((unsigned)(w * 32) << 16);   // the warp's lane quarter
    double N[R], h[R], q[R];
    double cin = 0.0, b = 0.0;   // the forward carry, the back chain's end
    {
        const int pos = (blockIdx.x * kPkWarps + w) * kPkTracers + (me & 31) / kPkLanes;
        const bool mine = pos < P.nt;
        const int tl = mine ? (P.order ? P.order[pos] : pos) : -1;
        walk.tl[me] = tl;
        walk.gi[me] = -1;
        walk.run[me] = 2;
        walk.rem[me] = mine ? 0 : -1;
        walk.pgi[me] = -1;
        const double *row = (S == 0 ? P.a.crp : P.a.cre) + (size_t)(P.t0 + max(tl, 0)) * NB + gl * R;
#pragma unroll
        for (int r = 0; r < R; r++) N[r] = 0.0;
        if (mine) {
#pragma unroll
            for (int r = 0; r < R; r += 4) ld4(row + r, N + r);
        }
    }
#pragma unroll 1
    for (;;) {
        const int group = me / kPkLanes;
        double *buf = reinterpret_cast<double *>(steps_smem) + (size_t)w * (SRC ? 4 : 3) * 512 +
                      (group % kPkTracers) * NB;
        bool load = walk.rem[me] >= 0;   // the group has work
        int want = 0;                    // its coefficient set
        cp_async_wait_all();             // the rows and scalars fetched for the next run
        __syncwarp();
        {
            const int tl = max(walk.tl[me], 0), nslot = P.g1 - P.g0;
            int k = walk.run[me];
            if (walk.rem[me] == 0) {     // the next run of a group that has none
                int gi = walk.gi[me], rem = 0, sl = walk.sl[me], el = walk.el[me], steps = walk.steps[me];
#pragma unroll 1
                while (rem <= 0) {
                    if (k < 2) {
                        k++;
                    } else {
                        if (++gi >= nslot) {
                            rem = -1;
                            break;
                        }
                        int4 mt;
                        if (gi > 0) {
                            mt = next.meta[group];
                            walk.dt[me] = next.dt[group];
                        } else {
                            const SegPre *__restrict__ pre = P.pre + tl;
                            mt = make_int4(pre->flags, pre->sl, pre->el, pre->steps);
                            walk.dt[me] = pre->dt;
                        }
                        if (!(mt.x & kPreActive)) {   // a tracer's active segments come first
                            rem = -1;
                            break;
                        }
                        steps = mt.w;
                        sl = (mt.x & kPreWindowed) ? min(max(mt.y, 0), steps) : 0;
                        el = (mt.x & kPreWindowed) ? min(max(mt.z, sl), steps) : steps;
                        k = 0;
                        if (S == 0 && P.np_seg) {
                            double *o = P.np_seg + ((size_t)gi * P.nt + tl) * NB + gl * R;
#pragma unroll
                            for (int r = 0; r < R; r += 4) st4_cg(o + r, N + r);
                        }
                    }
                    rem = (k == 0) ? sl : (k == 1 ? el - sl : steps - el);
                }
                if (rem > 0 && k != 1 && P.sets < 2) {   // no off set in the workspace: report, leave N as it was
                    if (gl == 0) atomicOr(P.a.err, kErrBadInput);
                    rem = -1;
                }
                load = rem > 0;
                walk.gi[me] = gi;
                walk.run[me] = k;
                walk.rem[me] = rem;
                walk.sl[me] = sl;
                walk.el[me] = el;
                walk.steps[me] = steps;
            }
            want = (k == 1) ? 0 : 1;
        }
        __syncwarp();
        if (!__any_sync(kFull, load)) break;
        const bool miss = load && (walk.pgi[me] != walk.gi[me] || walk.pset[me] != want);
        if (__any_sync(kFull, miss)) {
            if (miss) pk_fetch<S, SRC>(P, buf, walk.gi[me], want, walk.tl[me], gl);
            cp_async_wait_all();
            __syncwarp();
        }
        // the constants of the run: h and q to registers, g, E, 1/d and the
        // source to TMEM, the scan multipliers
        double hk[5], qk[5];
        {
            double iv[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                iv[r] = 1.0;
                h[r] = q[r] = 0.0;
            }
            if (load) {
                pk_read(buf, 0, gl, iv);
                if (SRC) pk_read(buf, 3, gl, h);
            }
            if (SRC) {
                const double dt = walk.dt[me];
                __syncwarp();
#pragma unroll
                for (int kk = 0; kk < R / 4; kk++) {
                    unsigned u[8];
#pragma unroll
                    for (int i = 0; i < 4; i++) pk_set(u, i, load ? (dt * h[4 * kk + i]) * iv[4 * kk + i] : 0.0);
                    tmem_st8(pk_src(tm, kk), u);
                }
            }
            if (load) {
                pk_read(buf, 1, gl, h);
                pk_read(buf, 2, gl, q);
                if (gl == 0) h[0] = 0.0;
                if (gl == kPkLanes - 1) q[R - 1] = 0.0;
            }
            __syncwarp();   // the buffer is read
            if (load) {
                // the rows of the next run (another set of this segment, or
                // the next one's first run, taken to be of the set this one
                // ends with) and the scalars of the next segment
                const int gi = walk.gi[me], k = walk.run[me], tl = walk.tl[me];
                const int sl = walk.sl[me], el = walk.el[me], steps = walk.steps[me];
                int pgi = gi, pset = 0;
                if (k == 0 && el > sl) pset = 0;
                else if (k < 2 && steps > el) pset = 1;
                else {
                    pgi = gi + 1;
                    pset = (steps > el || el == sl) ? 1 : 0;
                }
                if (pgi < P.g1 - P.g0 && pset < P.sets) pk_fetch<S, SRC>(P, buf, pgi, pset, tl, gl);
                else pgi = -1;
                walk.pgi[me] = pgi;
                walk.pset[me] = pset;
                if (gl == 0 && gi + 1 < P.g1 - P.g0) {
                    const SegPre *pre = P.pre + (size_t)(gi + 1) * P.nt + tl;
                    cp_async16(&next.meta[group], &pre->flags, true);
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                                     (unsigned)__cvta_generic_to_shared(&next.dt[group])),
                                 "l"(&pre->dt)
                                 : "memory");
                }
            }
            // e, then E = 1/d e + h E_r-1 (upwards)
            double v[R], H = 1.0, Q = 1.0;
#pragma unroll
            for (int r = R - 1; r >= 0; r--) {
                Q *= q[r];
                v[r] = iv[r] * Q;
            }
            __syncwarp();
#pragma unroll
            for (int kk = 0; kk < R / 4; kk++) {
                unsigned u[8];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int r = 4 * kk + i;
                    if (r > 0) v[r] = fma(h[r], v[r - 1], v[r]);
                    pk_set(u, i, v[r]);
                }
                tmem_st8(pk_resp(tm, kk), u);
            }
            // c, then g = c + q g_r+1 (downwards)
#pragma unroll
            for (int r = 0; r < R; r++) {
                H *= h[r];
                v[r] = H;
            }
#pragma unroll
            for (int r2 = R / 2 - 1; r2 >= 0; r2--) {
                unsigned u[8];
#pragma unroll
                for (int i = 1; i >= 0; i--) {
                    const int r = 2 * r2 + i;
                    if (r < R - 1) v[r] = fma(q[r], v[r + 1], v[r]);
                    pk_set(u, 2 * i, v[r]);
                    pk_set(u, 2 * i + 1, iv[r]);
                }
                tmem_st8(pk_fwd(tm, r2 / 2) + 8 * (r2 & 1), u);
            }
            tmem_wait_st();
#pragma unroll
            for (int lv = 0; (1 << lv) < kPkLanes; lv++) {
                const int off = 1 << lv;
                hk[lv] = gl >= off ? H : 0.0;
                qk[lv] = gl + off < kPkLanes ? Q : 0.0;
                const double Hu = pk_up(H, off), Qd = pk_down(Q, off);
                H *= gl >= off ? Hu : 1.0;
                Q *= gl + off < kPkLanes ? Qd : 1.0;
            }
        }
        int m = load ? walk.rem[me] : 0x7fffffff;
#pragma unroll
        for (int off = 16; off >= kPkLanes; off >>= 1) m = min(m, __shfl_xor_sync(kFull, m, off));
        __syncwarp();
        // m sub-steps of every group.  At the group's ends the shuffles return
        // the lane's own value, whose responses are zero (h of the first row,
        // q of the last).
        constexpr int kLevels = kPkLanes == 8 ? 3 : (kPkLanes == 16 ? 4 : 5);
        double cout = 0.0;
        Tmem16 U;            // (g, 1/d) of four rows
        unsigned V[8];       // dt src/d of four rows
        unsigned W[2][8];    // E of four rows
        tmem_ld16(pk_fwd(tm, 0), U);
        if (SRC) tmem_ld8(pk_src(tm, 0), V);
#pragma unroll 1
        for (int go = m; go > 0; go--) {
            // forward chain of the rows without cout, under the back scan
            double s = 0.0;
#pragma unroll
            for (int kk = 0; kk < R / 4; kk++) {
                tmem_wait(U);
                if (SRC) tmem_after8(V);
                if (kk == 0) b = fma(U.d(0), cin, b);   // the back chain's end and its response to cin, g_0
                const double t = kk < kLevels ? pk_down(b, 1 << kk) : 0.0;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int r = 4 * kk + i;
                    N[r] = fma(U.d(2 * i), cin, N[r]);
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int r = 4 * kk + i;
                    N[r] = SRC ? fma(N[r], U.d(2 * i + 1), pk_get(V, i)) : N[r] * U.d(2 * i + 1);
                }
                if (kk < R / 4 - 1) {
                    tmem_ld16(pk_fwd(tm, kk + 1), U);
                    if (SRC) tmem_ld8(pk_src(tm, kk + 1), V);
                } else {
                    tmem_ld8(pk_resp(tm, 3), W[1]);
                    tmem_ld8(pk_resp(tm, 2), W[0]);
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int r = 4 * kk + i;
                    s = fma(h[r], s, N[r]);
                    N[r] = s;
                }
                if (kk < kLevels) b = fma(qk[kk], t, b);
            }
            if (kLevels > 4) b = fma(qk[4], pk_down(b, 16), b);
            cout = pk_down(b, 1);
            // the rows' responses to cout and the back chain, under the forward scan
            tmem_wait8(W[1]);
            tmem_after8(W[0]);
            s = fma(pk_get(W[1], 3), cout, s);
            b = 0.0;
#pragma unroll
            for (int kk = R / 4 - 1; kk >= 0; kk--) {
                unsigned *E = W[kk & 1];
                if (kk < R / 4 - 2) tmem_wait8(E);
                const double t = R / 4 - 1 - kk < kLevels ? pk_up(s, 1 << (R / 4 - 1 - kk)) : 0.0;
#pragma unroll
                for (int i = 3; i >= 0; i--) {
                    const int r = 4 * kk + i;
                    N[r] = fma(pk_get(E, i), cout, N[r]);
                }
                if (kk >= 2) {
                    tmem_ld8(pk_resp(tm, kk - 2), W[kk & 1]);
                } else if (kk == 0) {
                    tmem_ld16(pk_fwd(tm, 0), U);
                    if (SRC) tmem_ld8(pk_src(tm, 0), V);
                }
#pragma unroll
                for (int i = 3; i >= 0; i--) {
                    const int r = 4 * kk + i;
                    b = fma(q[r], b, N[r]);
                    N[r] = b;
                }
                if (R / 4 - 1 - kk < kLevels) s = fma(hk[R / 4 - 1 - kk], t, s);
            }
            if (kLevels > 4) s = fma(hk[4], pk_up(s, 16), s);
            cin = pk_up(s, 1);
        }
        tmem_wait(U);
        if (SRC) tmem_after8(V);
        // where the run ends, the last sub-step's responses: x = raw + g cin +
        // e cout; the other groups go on from their raw rows, so that no
        // result depends on which tracers share a warp
        const int left = load ? walk.rem[me] - m : 0;
        const bool done = kPkTracers == 1 || left == 0;
        double bb = fma(U.d(0), cin, b);
#pragma unroll
        for (int lv = 0; lv < kLevels; lv++) bb = fma(qk[lv], pk_down(bb, 1 << lv), bb);
        cout = pk_down(bb, 1);
#pragma unroll
        for (int r = R - 1; r >= 0; r--) {
            cout *= q[r];   // e_r cout
            N[r] = done ? N[r] + cout : N[r];
        }
#pragma unroll
        for (int kk = 0; kk < R / 4; kk++) {
            tmem_ld16(pk_fwd(tm, kk), U);
            tmem_wait(U);
#pragma unroll
            for (int i = 0; i < 4; i++) N[4 * kk + i] = done ? fma(U.d(2 * i), cin, N[4 * kk + i]) : N[4 * kk + i];
        }
        cin = done ? 0.0 : cin;
        b = done ? 0.0 : b;
        if (load) walk.rem[me] = left;
    }
    if (walk.tl[me] >= 0) {
        double *row = (S == 0 ? P.a.crp : P.a.cre) + (size_t)(P.t0 + walk.tl[me]) * NB + gl * R;
#pragma unroll
        for (int r = 0; r < R; r += 4) st4(row + r, N + r);
    }
    __syncthreads();
    if (w == 0) tmem_free<kPkColumns>(tmem_base);
}

template <int S, bool SRC>
cudaError_t launch_packed(cudaStream_t st, const FusedParams &P)
{
    constexpr size_t smem = (size_t)kPkWarps * (SRC ? 4 : 3) * 512 * sizeof(double);
    static OncePerDevice once;
    const cudaError_t attr = allow_smem(once, steps_packed_kernel<S, SRC>, smem);
    if (attr != cudaSuccess) return attr;
    const int per = kPkWarps * kPkTracers;
    steps_packed_kernel<S, SRC><<<(P.nt + per - 1) / per, kPkThreads, smem, st>>>(P);
    return cudaGetLastError();
}

// Order of the chunk's tracers for the packed steps kernel: by falling
// sub-step count, in bins a sixteenth of an octave wide (exact below 32), the
// order within a bin left open -- no tracer's result depends on which tracers
// share its warp, only the time does.  One block up to kOrderOneBlock tracers;
// beyond, the counts (order_count_kernel) and then the places, each block
// reserving its range of a bin with one atomic.
constexpr int kOrderBins = 288;
constexpr int kOrderOneBlock = 4096;
constexpr int kOrderThreads = 1024;

__device__ __forceinline__ int order_bin(int nsub)   // 0 = most sub-steps
{
    int b = nsub;
    if (nsub >= 32) {
        const int e = 31 - __clz(nsub);   // >= 5; nsub <= 1e6 gives e <= 19
        b = 32 + (min(e, 19) - 5) * 16 + ((nsub >> (e - 4)) & 15);
    }
    return kOrderBins - 1 - max(0, min(b, kOrderBins - 1));
}

// exclusive prefix of the bins in place (all threads call it)
__device__ __forceinline__ void order_prefix(unsigned *bins)
{
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned carry = 0;
        for (int b0 = 0; b0 < kOrderBins; b0 += 32) {
            const unsigned v = bins[b0 + threadIdx.x];
            unsigned s = v;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const unsigned o = __shfl_up_sync(kFull, s, off);
                if ((int)threadIdx.x >= off) s += o;
            }
            bins[b0 + threadIdx.x] = carry + s - v;
            carry += __shfl_sync(kFull, s, 31);
        }
    }
    __syncthreads();
}

// one atomic per bin and warp: most tracers of a run have the same count
__device__ __forceinline__ unsigned order_take(unsigned *bins, int b, bool on)
{
    const unsigned peers = __match_any_sync(kFull, on ? b : -1);
    const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
    unsigned base = 0;
    if (on && lane == leader) base = atomicAdd(bins + b, (unsigned)__popc(peers));
    base = __shfl_sync(kFull, base, leader);
    return base + __popc(peers & ((1u << lane) - 1u));
}

__global__ void __launch_bounds__(kOrderThreads) order_one_kernel(int nt, const int *nsub, int *order)
{
    __shared__ unsigned bins[kOrderBins];
    for (int b = threadIdx.x; b < kOrderBins; b += blockDim.x) bins[b] = 0;
    __syncthreads();
    const int top = (nt + 31) & ~31;
    for (int i = threadIdx.x; i < top; i += blockDim.x) order_take(bins, i < nt ? order_bin(nsub[i]) : 0, i < nt);
    order_prefix(bins);
    for (int i = threadIdx.x; i < top; i += blockDim.x) {
        const unsigned p = order_take(bins, i < nt ? order_bin(nsub[i]) : 0, i < nt);
        if (i < nt) order[p] = i;
    }
}

// counts of the bins in bins[0 .. kOrderBins), zeroed before the launch
__global__ void __launch_bounds__(kOrderThreads) order_count_kernel(int nt, const int *nsub, unsigned *bins)
{
    __shared__ unsigned mine[kOrderBins];
    for (int b = threadIdx.x; b < kOrderBins; b += blockDim.x) mine[b] = 0;
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    order_take(mine, i < nt ? order_bin(nsub[i]) : 0, i < nt);
    __syncthreads();
    for (int b = threadIdx.x; b < kOrderBins; b += blockDim.x)
        if (mine[b]) atomicAdd(bins + b, mine[b]);
}

// bins: the counts, then kOrderBins cursors (zeroed before the count)
__global__ void __launch_bounds__(kOrderThreads) order_place_kernel(int nt, const int *nsub, unsigned *bins, int *order)
{
    __shared__ unsigned first[kOrderBins], mine[kOrderBins];
    for (int b = threadIdx.x; b < kOrderBins; b += blockDim.x) {
        first[b] = bins[b];
        mine[b] = 0;
    }
    order_prefix(first);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = i < nt ? order_bin(nsub[i]) : 0;
    const unsigned at = order_take(mine, b, i < nt);
    __syncthreads();
    for (int c = threadIdx.x; c < kOrderBins; c += blockDim.x)
        if (mine[c]) first[c] += atomicAdd(bins + kOrderBins + c, mine[c]);
    __syncthreads();
    if (i < nt) order[first[b] + at] = i;
}

cudaError_t launch_order(cudaStream_t st, int nt, const int *nsub, unsigned *bins, int *order)
{
    if (nt <= kOrderOneBlock) {
        order_one_kernel<<<1, kOrderThreads, 0, st>>>(nt, nsub, order);
        return cudaGetLastError();
    }
    const cudaError_t e = cudaMemsetAsync(bins, 0, 2 * kOrderBins * sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    const int blocks = (nt + kOrderThreads - 1) / kOrderThreads;
    order_count_kernel<<<blocks, kOrderThreads, 0, st>>>(nt, nsub, bins);
    order_place_kernel<<<blocks, kOrderThreads, 0, st>>>(nt, nsub, bins, order);
    return cudaGetLastError();
}

// Per-step kernel (the plain path): a block of one warp advances a tracer
// through the sub-steps of segment slot g0 with the reference's per-step data
// contract -- every sub-step reads the rows a, b, c of its on/off set from
// memory, solves M N' = N + dt src with the pivots recomputed
// (tracer_fp_cpu_evolve, src/tracer_fp_cpu.c:149-190; fp_thomas_solve_ws,
// src/fp_shared_core.c:226-257) and writes N back.
// The rows come through shared memory, copied across the lanes in 16-byte
// pieces while the sub-step before is solved; lane l's pieces sit where the
// lanes' reads of their own rows meet no bank twice.  The scans' shuffles (some
// 40 of 64 bits a sub-step) and their latency bound it.  Before (each lane
// loading its rows, half a cache line apart, as the sub-step began; the source
// and all scan multipliers in registers) and now, both species, 512 bins 58.1 ->
// 41.0 ms a snapshot of 16,384 tracers and 3.06 -> 2.98 ms of 64, 256 bins 19.8
// -> 18.3 and 2.28 -> 2.09, 128 bins 11.3 -> 11.0 and 1.91 -> 1.62.  Sixteen
// rows a lane and two or four systems a warp, with half the shuffles, took 22.0
// and 11.5 ms at 256 and 128 bins: too few warps for the longer chains.
constexpr int kPlainBlocks = NB <= 128 ? 24 : (NB <= 256 ? 20 : 12);   // per SM
__device__ __forceinline__ int plain_piece(int c) { return c ^ ((c >> 3) & (kR / 2 - 1)); }
__device__ __forceinline__ void plain_read(const double *buf, int lane, double v[kR])
{
#pragma unroll
    for (int j = 0; j < kR / 2; j++) {
        const double2 x = *reinterpret_cast<const double2 *>(buf + 2 * plain_piece(lane * (kR / 2) + j));
        v[2 * j] = x.x;
        v[2 * j + 1] = x.y;
    }
}
template <int S, bool SRC>
__global__ void __launch_bounds__(32, kPlainBlocks) plain_steps_kernel(const __grid_constant__ FusedParams P)
{
    constexpr int R = kR, H2 = R / 2;
    __shared__ __align__(16) double buf[(SRC ? 4 : 3) * NB];   // a, b, c, the source
    const int lane = threadIdx.x, tl = blockIdx.x, t = P.t0 + tl;
    const SegPre *__restrict__ pre = P.pre + tl;
    const int flags = pre->flags;
    if (!(flags & kPreActive)) return;
    const bool windowed = flags & kPreWindowed;
    const int steps = pre->steps, sl = windowed ? pre->sl : 0, el = windowed ? pre->el : steps;
    const double dt = pre->dt;
    double *Nrow = (S == 0 ? P.a.crp : P.a.cre) + (size_t)t * NB + lane * R;
    auto fetch = [&](int istep) {   // the rows of a sub-step's set
        const int set = istep >= sl && istep < el ? 0 : 1;
        if (set >= P.sets) return false;   // no off set in the workspace
        const double *f = fac_ptr(P, S, 0, set, tl);
#pragma unroll
        for (int i = 0; i < R / 2; i++) {
            const int c = i * 32 + lane;
#pragma unroll
            for (int k = 0; k < 3; k++) cp_async16(buf + k * NB + 2 * plain_piece(c), f + k * NB + 2 * c, true);
        }
        return true;
    };
    if (SRC) {
        const double *src = (S == 1 && P.inje) ? P.inje + (size_t)tl * NB : (S == 0 ? P.a.qpi : P.a.qepri) + (size_t)t * NB;
#pragma unroll
        for (int i = 0; i < R / 2; i++) {
            const int c = i * 32 + lane;
            cp_async16(buf + 3 * NB + 2 * plain_piece(c), src + 2 * c, true);
        }
    }
    bool there = steps > 0 && fetch(0);
    double N[R];
#pragma unroll
    for (int r = 0; r < R; r += 4) ld4(Nrow + r, N + r);
#pragma unroll 1
    for (int istep = 0; istep < steps; istep++) {
        if (!there) {   // report, leave N as it is
            if (lane == 0) atomicOr(P.a.err, kErrBadInput);
            break;
        }
        double A[R], B[R], C[R];
        cp_async_wait_all();
        __syncwarp();
        plain_read(buf, lane, A);
        plain_read(buf + NB, lane, B);
        plain_read(buf + 2 * NB, lane, C);
        __syncwarp();   // the buffer is read
        there = istep + 1 < steps && fetch(istep + 1);
        const unsigned err = pivot_rows<R, 32>(A, B, C, lane);
        if (__any_sync(kFull, err != 0)) {
            if (lane == 0) atomicOr(P.a.err, kErrSingular);
            break;
        }
        if (lane == 0) A[0] = 0.0;
        if (lane == 31) C[R - 1] = 0.0;
        // y = (N + dt src) / d
        if (SRC) {
            double v[R];
            plain_read(buf + 3 * NB, lane, v);
#pragma unroll
            for (int r = 0; r < R; r++) N[r] = fma(N[r], B[r], (dt * v[r]) * B[r]);
        } else {
#pragma unroll
            for (int r = 0; r < R; r++) N[r] *= B[r];
        }
        // forward: z_i = y_i + h_i z_{i-1}, two half-length chains a lane
        double alo = 0.0, ahi = 0.0, hlo = 1.0, hhi = 1.0;
#pragma unroll
        for (int r = 0; r < H2; r++) {
            alo = fma(A[r], alo, N[r]);
            ahi = fma(A[r + H2], ahi, N[r + H2]);
            hlo *= A[r];
            hhi *= A[r + H2];
        }
        double acc = fma(hhi, alo, ahi), m = hlo * hhi;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const double u = sup(acc, off), mu = sup(m, off);
            if (lane >= off) {
                acc = fma(m, u, acc);
                m *= mu;
            }
        }
        double cin = sup(acc, 1);
        cin = lane > 0 ? cin : 0.0;
        double plo = cin, phi = fma(hlo, cin, alo);
#pragma unroll
        for (int r = 0; r < H2; r++) {
            plo = fma(A[r], plo, N[r]);
            phi = fma(A[r + H2], phi, N[r + H2]);
            N[r] = plo;
            N[r + H2] = phi;
        }
        // back substitution: x_i = z_i + q_i x_{i+1}
        alo = ahi = 0.0;
        double qlo = 1.0, qhi = 1.0;
#pragma unroll
        for (int r = H2 - 1; r >= 0; r--) {
            alo = fma(C[r], alo, N[r]);
            ahi = fma(C[r + H2], ahi, N[r + H2]);
            qlo *= C[r];
            qhi *= C[r + H2];
        }
        acc = fma(qlo, ahi, alo);
        m = qlo * qhi;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const double d = sdn(acc, off), md = sdn(m, off);
            if (lane + off < 32) {
                acc = fma(m, d, acc);
                m *= md;
            }
        }
        double cout = sdn(acc, 1);
        cout = lane < 31 ? cout : 0.0;
        phi = cout;
        plo = fma(qhi, cout, ahi);
#pragma unroll
        for (int r = H2 - 1; r >= 0; r--) {
            phi = fma(C[r + H2], phi, N[r + H2]);
            plo = fma(C[r], plo, N[r]);
            N[r + H2] = phi;
            N[r] = plo;
        }
#pragma unroll
        for (int r = 0; r < R; r += 4) st4(Nrow + r, N + r);
    }
    cp_async_wait_all();   // rows asked for before a singular system's end
}

// The per-segment scalars of every (slot, tracer) of the chunk, one thread
// each: the schedule's segment (tracer_fp_batch.c segment split), the
// background interpolated to it, the loss coefficients and the "on" Dpp form
// (prepare_momentumdiff_cell_major, src/fp_shared_core.c:1241-1317) -- the
// same arithmetic the factor kernels would repeat per species and set.
__global__ void __launch_bounds__(256) seg_pre_kernel(FusedParams P)
{
    const SnapArgs &a = P.a;
    const long long total = (long long)(P.g1 - P.g0) * P.nt;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int gi = (int)(i / P.nt);
        const int tl = (int)(i - (long long)gi * P.nt);
        const int t = P.t0 + tl;
        SegPre o{};
        const SegInfo g = segment_of(P, t, P.g0 + gi);
        if (!g.active) {   // nothing reads more of it than its flags; 112 strided bytes a
                           // thread bound this kernel (43 to 27 us, most of 16 slots inactive)
            *reinterpret_cast<int4 *>(&P.pre[i].flags) = make_int4(0, 0, 0, 0);
            continue;
        }
        {
            const Bg bg = load_bg(a, t, g);
            const int dis = a.dis ? a.dis[t] : 0;
            const SegTerms T = seg_terms(bg, dis, g);
            const DppForm on = dpp_form(P.mp, P.mp.dpp_model, bg, segment_tacc(P.mp, a, g));
            o.n_gas = T.n_gas;
            o.kbt = T.kbt;
            o.inv_kbt = T.inv_kbt;
            o.log_n = T.log_n;
            o.adiab = T.adiab;
            o.synch_coeff = T.synch_coeff;
            o.coulomb_coeff = T.coulomb_coeff;
            o.dt = T.dt;
            o.dt_over_tloss_pref = T.dt_over_tloss_pref;
            o.dtT_e = T.dtT_e;
            o.alpha = T.alpha;
            o.dpp_inv = on.inv;
            o.flags = kPreActive | (g.windowed ? kPreWindowed : 0) | (T.interp ? kPreInterp : 0) |
                      (on.fill ? kPreFill : 0);
            o.sl = g.sl;
            o.el = g.el;
            o.steps = g.steps;
        }
        P.pre[i] = o;
    }
}

// Dpp eta-cap scale of every tracer of the chunk with a segment in slot g0,
// from the spectra at the start of the segment (prepare_momentumdiff_cell_major,
// src/fp_shared_core.c:1032-1081, runs before either species evolves), one
// warp per tracer.  The energy sum is split over the lanes and combined by a
// shuffle tree, so it agrees with the reference's sequential sum to rounding.
__global__ void __launch_bounds__(128) eta_scale_kernel(FusedParams P, double *eta)
{
    const int lane = threadIdx.x & 31;
    const int tl = blockIdx.x * 4 + (threadIdx.x >> 5);
    const SnapArgs &a = P.a;
    if (tl >= P.nt) return;
    const int t = P.t0 + tl;
    const SegInfo g = segment_of(P, t, P.g0);
    if (!g.active) return;
    const Bg bg = load_bg(a, t, g);
    const double tacc_direct = segment_tacc(P.mp, a, g);
    const double mass = a.mass ? a.mass[t] : 0.0;
    const double *crp = a.crp + (size_t)t * NB, *cre = a.cre + (size_t)t * NB;
    double ecr = 0.0;
    for (int j = 2 + lane; j < NB - 2; j += 32) {
        const double ekp = P.gt.s[0].E[j] - kMp, vp = crp[j];
        if (ekp > 0.0 && isfinite(vp)) ecr += ekp * kGeV * vp * P.gt.s[0].dp[j];
        const double eke = P.gt.s[1].E[j] - kMe, ve = cre[j];
        if (eke > 0.0 && isfinite(ve)) ecr += eke * kGeV * ve * P.gt.s[1].dp[j];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ecr += __shfl_xor_sync(kFull, ecr, off);
    if (lane == 0) eta[t] = eta_cap_scale_from_ecr(P.mp, bg, mass, tacc_direct, ecr);
}

// Secondary source of every segment of the chunk, cell-major:
// inje[m][je] = Gyr n_gas(t, segment) sum_{jp} N_p[m][jp] fqe[jp][je] + qepri[t][je]
// over the rows m = gi * nt + tl of np_seg -- a [rows x nb] . [nb x nb] FP64
// GEMM on the FP64 tensor cores (mma.sync m8n8k4 .f64: one instruction is
// 256 multiply-adds).  A 128 x 64 output tile per 256-thread block, each warp
// a 32 x 32 tile of 4 x 4 MMA fragments; k-tiles of 16 double-buffered in
// shared memory by cp.async.  The proton index starts at the first k-tile
// holding a nonzero weight for the block's columns; fqe is zero below
// np_min_qe[je] (prepare_secondary_kernel_flat, src/fp_shared_core.c:1453-1506),
// so the rounded-down start adds exact zeros only.
constexpr int kGM = 128, kGN = 64, kGK = 16;
// Row pitches chosen so that the fragment reads of a half warp (rows gid or
// tig, 4 x 4 lanes) land on 16 distinct bank pairs: 20 and 68 doubles.
constexpr int kGPitchA = kGK + 4;    // sA[m][k], 20 doubles per row
constexpr int kGPitchB = kGN + 4;    // sB[k][n], 68 doubles per row

struct GemmSmem {
    double A[2][kGM][kGPitchA];
    double B[2][kGK][kGPitchB];
};

__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

__global__ void __launch_bounds__(256, 2) secondary_kernel(FusedParams P)
{
    extern __shared__ double4 smem_raw[];
    GemmSmem &sm = *reinterpret_cast<GemmSmem *>(smem_raw);
    const SnapArgs &a = P.a;
    const int nrows = (P.g1 - P.g0) * P.nt;   // < 2^31, checked on the host
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;   // warp tile origin in the block tile
    const int gid = lane >> 2, tig = lane & 3;                // MMA fragment coordinates
    // column tile fastest, so the NB / kGN blocks of one row tile run together
    // and read their A tile from L2
    const int n0 = (int)(blockIdx.x % (NB / kGN)) * kGN;
    const int m0 = (int)(blockIdx.x / (NB / kGN)) * kGM;
    int jstart = NB;
    for (int i = 0; i < kGN; i++) jstart = min(jstart, P.np_min_qe[n0 + i]);
    jstart = max(jstart, P.gt.fqe_jp0);
    const int kbeg = (jstart / kGK) * kGK;

    // loader roles: A rows (4 chunks of 16 B per thread), B rows (2 chunks)
    auto load_tile = [&](int buf, int k0) {
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int q = tid + 256 * c;          // 0..1023: row q / 8, chunk q % 8
            const int r = q >> 3, ch = q & 7;
            const int m = m0 + r;
            const bool ok = m < nrows;
            const double *src = P.np_seg + (size_t)(ok ? m : 0) * NB + k0 + ch * 2;
            cp_async16(&sm.A[buf][r][ch * 2], src, ok);
        }
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const int q = tid + 256 * c;          // 0..511: row q / 32, chunk q % 32
            const int r = q >> 5, ch = q & 31;
            const double *src = P.gt.fqe + (size_t)(k0 + r) * NB + n0 + ch * 2;
            cp_async16(&sm.B[buf][r][ch * 2], src, true);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };

    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.0;

    if (kbeg < NB) load_tile(0, kbeg);
    int buf = 0;
#pragma unroll 1
    for (int k0 = kbeg; k0 < NB; k0 += kGK) {
        const bool more = k0 + kGK < NB;
        if (more) {
            load_tile(buf ^ 1, k0 + kGK);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kGK; kk += 4) {
            double af[4], bf[4];
#pragma unroll
            for (int i = 0; i < 4; i++) af[i] = sm.A[buf][wm + 8 * i + gid][kk + tig];
#pragma unroll
            for (int j = 0; j < 4; j++) bf[j] = sm.B[buf][kk + tig][wn + 8 * j + gid];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) dmma(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
        }
        __syncthreads();
        buf ^= 1;
    }

    // epilogue: fragment (i, j) holds C[wm + 8i + gid][wn + 8j + 2 tig + {0, 1}]
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int m = m0 + wm + 8 * i + gid;
        if (m >= nrows) continue;
        const int gi = m / P.nt, tl = m - gi * P.nt;
        const int t = P.t0 + tl;
        const SegPre *__restrict__ pre = P.pre + (size_t)gi * P.nt + tl;
        if (!(pre->flags & kPreActive)) continue;
        const double ng = pre->n_gas;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int je = n0 + wn + 8 * j + 2 * tig;
            double q0 = 0.0, q1 = 0.0;
            if (a.qepri) {
                q0 = a.qepri[(size_t)t * NB + je];
                q1 = a.qepri[(size_t)t * NB + je + 1];
            }
            *reinterpret_cast<double2 *>(P.inje + (size_t)m * NB + je) =
                make_double2(acc[i][j][0] * kGyr * ng + q0, acc[i][j][1] * kGyr * ng + q1);
        }
    }
}

cudaError_t launch_secondary(Context &ctx, const FusedParams &P)
{
    constexpr size_t smem = sizeof(GemmSmem);
    static OncePerDevice once;
    const cudaError_t attr = allow_smem(once, secondary_kernel, smem);
    if (attr != cudaSuccess) return attr;
    const long long rows = (long long)(P.g1 - P.g0) * P.nt;
    if (rows > 0x7fffffffLL) return cudaErrorInvalidValue;
    const long long blocks = (rows + kGM - 1) / kGM * (NB / kGN);
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    secondary_kernel<<<(unsigned)blocks, 256, smem, ctx.stream>>>(P);
    return cudaGetLastError();
}

template <int S, bool ROWS>
cudaError_t launch_factor(Context &ctx, FusedParams &P)
{
    constexpr size_t tables = (size_t)kFacTabs * NB * sizeof(double2), rows = (size_t)kFacWarps * kCoulWarp * sizeof(double);
    static_assert(2 * (tables + rows + 8192) <= 227 * 1024, "two blocks per SM");
    const size_t smem = tables + (S == 0 || P.ic_stride ? rows : 0);
    static OncePerDevice once;
    const cudaError_t attr = allow_smem(once, factor_kernel<S, ROWS>, tables + rows);
    if (attr != cudaSuccess) return attr;
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const long long systems = (long long)P.nt * (P.g1 - P.g0) * P.sets;
    if (systems > 0x7fff0000LL) return cudaErrorInvalidValue;
    // the occupancy query counts one block per SM for any kernel that allocates
    // TMEM; kFacBlocks of these fit by registers, columns and shared memory
    const long long full = (long long)nsm * kFacBlocks;
    // A warp takes several systems together only where there are more than warps:
    // a launch below that lasts as long as one unit, whose Coulomb terms and IC rows
    // are formed system by system.  Bucket calls of 64 tracers, protons and electrons:
    // 128 bins 15.0 and 17.6 us, now 10.2 and 10.4; 256 bins 15.1 and 18.7, 11.4 and
    // 12.4 (512 bins: one system a warp either way).
    const long long pack = (systems + full * kFacWarps - 1) / (full * kFacWarps);
    P.pack = pack < 1 ? 1 : (pack > kPkTracers ? kPkTracers : (int)pack);
    long long blocks = (systems + kFacWarps * P.pack - 1) / (kFacWarps * P.pack);
    if (blocks > full) blocks = full;
    if (blocks < 1) return cudaSuccess;
    factor_kernel<S, ROWS><<<(unsigned)blocks, kFacWarps * 32, smem, ctx.stream>>>(P);
    return cudaGetLastError();
}

// One steps-kernel variant: solver and warps per block (1, 2 or 4), on the
// first `tracers` tracers of the chunk (all when <= 0).
template <int S, bool SRC, int SOLVER, int WPB>
cudaError_t launch_steps_variant(cudaStream_t st, const FusedParams &P, int tracers)
{
    const int n = tracers > 0 ? min(tracers, P.nt) : P.nt;
    const int blocks = (n + WPB - 1) / WPB;
    const size_t smem = SOLVER == kSolvePcr ? WPB * sizeof(PcrSmem)
                      : SOLVER == kSolveScanShared ? (size_t)WPB * kCoefSmemDoubles * sizeof(double)
                      : SOLVER == kSolveScanRhs    ? (size_t)WPB * kRhsSmemDoubles * sizeof(double)
                                                   : 0;
    if (smem > 48 * 1024) {
        static OncePerDevice once;
        const cudaError_t attr = allow_smem(once, steps_kernel<S, SRC, SOLVER, WPB>, smem);
        if (attr != cudaSuccess) return attr;
    }
    steps_kernel<S, SRC, SOLVER, WPB><<<blocks, WPB * 32, smem, st>>>(P);
    return cudaGetLastError();
}

// Variants the autotuner chooses between: (solver, warps per block).
constexpr int kStepVariants = CROMA_B200_STEPS_VARIANTS;
constexpr int kPackedVariant = kStepVariants;   // the packed kernel: by rule (packed_rule), never tuned
constexpr int kVariantSolver[kStepVariants + 1] = {kSolveScan, kSolveScan, kSolveScanShared, kSolveScanShared,
                                                   kSolvePcr, kSolveScanRhs, kSolveScanRhs, kSolveScan4,
                                                   kSolveScan4, kSolvePacked};
constexpr int kVariantWpb[kStepVariants + 1] = {1, 2, 1, 2, 1, 1, 2, 1, 2, kPkWarps * kPkTracers};

// Arithmetic families: variants of one family compute bit-identical results
// (the same operations in the same order; only where the constants live and
// how many warps share a block differ), so the tuner's timing-based choice
// within a family never changes a result.  0: the scan; 1: the short-chain
// scan; 2: PCR.
constexpr int kVariantFamily[kStepVariants] = {0, 0, 0, 0, 2, 0, 0, 1, 1};

// The family the tuner times: PCR when CROMA_CUDA_TRIDIAG=pcr, else the
// short-chain scan at 512 bins and more (measured faster there: its shorter
// shuffle chain outweighs its extra instructions at 8 warps per SM) and the
// scan below (where the short-chain form spills at the larger warp count).
int tune_family(int env) { return env == 2 ? 2 : (NB >= 512 ? 1 : 0); }

template <int S, bool SRC>
cudaError_t launch_variant(cudaStream_t st, const FusedParams &P, int v, int tracers)
{
    switch (v) {
    case 1: return launch_steps_variant<S, SRC, kSolveScan, 2>(st, P, tracers);
    case 2: return launch_steps_variant<S, SRC, kSolveScanShared, 1>(st, P, tracers);
    case 3: return launch_steps_variant<S, SRC, kSolveScanShared, 2>(st, P, tracers);
    case 4: return launch_steps_variant<S, SRC, kSolvePcr, 1>(st, P, tracers);
    case 5: return launch_steps_variant<S, SRC, kSolveScanRhs, 1>(st, P, tracers);
    case 6: return launch_steps_variant<S, SRC, kSolveScanRhs, 2>(st, P, tracers);
    case 7: return launch_steps_variant<S, SRC, kSolveScan4, 1>(st, P, tracers);
    case 8: return launch_steps_variant<S, SRC, kSolveScan4, 2>(st, P, tracers);
    default: return launch_steps_variant<S, SRC, kSolveScan, 1>(st, P, tracers);
    }
}

// CROMA_CUDA_TRIDIAG (src/fp_cuda_solver.cu:41-63 of the reference): "thomas"
// keeps the scan solvers, "pcr" forces PCR, unset lets the tuner choose.
int tridiag_env()
{
    const char *e = getenv("CROMA_CUDA_TRIDIAG");
    if (!e) e = getenv("FP_GPU_CUDA_TRIDIAG");
    if (!e) return 0;
    if (strcmp(e, "thomas") == 0) return 1;
    if (strcmp(e, "pcr") == 0) return 2;
    return 0;
}

// The autotuner of runs below the packed kernel's line, and of PCR at any size:
// on the first chunk a context evolves, each variant of the family tune_family
// names runs the chunk's tracers (fewer than 64; under PCR, whose one variant is
// timed to be reported, at most kTuneTracers) for their first 16 sub-steps on a
// copy of their spectra, timed with CUDA events; the fastest is kept for the
// context's species.  Results are recorded in
// ctx.tune.  CROMA_B200_STEPS_VARIANT = 0..8 fixes the variant (scan x1, scan
// x2, shared scan x1, shared scan x2, PCR, rhs-shared scan x1, rhs-shared scan
// x2, short-chain scan x1, short-chain scan x2) without calibrating, for
// reproducible profiles; unset or out of range: tune.
constexpr int kTuneTracers = 16384;

int fixed_variant_env()
{
    const char *e = getenv("CROMA_B200_STEPS_VARIANT");
    if (!e || !*e) return -1;
    const int v = atoi(e);
    return (v >= 0 && v < kStepVariants) ? v : -1;
}

// Which runs take the packed kernel: all of the FP64 on-chip path from
// kPackedMin tracers on, unless the environment asks for PCR or names a
// variant.  The line is on the run's tracers, not the chunk's, so that no
// result depends on how a run is cut into chunks; across it a tracer's spectra
// agree to rounding (a run of 63 is another arithmetic than one of 64).  The line
// is not where the kernels cross.  A snapshot of both species, alone, by the
// tuned variants and by the packed kernel (us): 1 tracer 445 and 387 (128 bins),
// 505 and 451 (256), 520 and 514 (512); 63 tracers 447 and 414, 507 and 481, 533
// and 537; the first snapshot, calibration included, 1260 and 480, 1360 and 560,
// 890 and 640.  Below it the tuner stays because its record is part of the
// interface (croma_b200_get_tuning: the times of a family's variants).
constexpr int kPackedMin = 64;
bool packed_rule(const Context &ctx, const FusedParams &P)
{
    return ctx.cfg.path == CROMA_PATH_FUSED && P.a.ntracer >= kPackedMin && fixed_variant_env() < 0 &&
           tridiag_env() != 2;
}

template <int S>
int tune_steps(Context &ctx, const FusedParams &P, bool src)
{
    TuneState &tu = ctx.tune[S];
    const int fixed = fixed_variant_env();
    if (fixed >= 0) {
        tu.variant = fixed;
        tu.tuned = 1;
        return 0;
    }
    const int env = tridiag_env();
    const int T = min(P.nt, kTuneTracers), steps = 16;
    double *scratch = nullptr;
    CROMA_CUDA(dev_alloc(ctx, &scratch, (size_t)T * NB * sizeof(double)));
    struct Free {
        Context &c;
        double *p;
        ~Free() { dev_free(c, p); }
    } guard{ctx, scratch};
    const double *real = (S == 0 ? P.a.crp : P.a.cre) + (size_t)P.t0 * NB;
    FusedParams Q = P;
    Q.cal_spec = scratch;
    Q.cal_steps = steps;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    CROMA_CUDA(cudaEventCreate(&e0));
    CROMA_CUDA(cudaEventCreate(&e1));
    int best = -1;
    const int family = tune_family(env);
    for (int v = 0; v < kStepVariants; v++) {
        tu.ms[v] = -1.0;
        if (kVariantFamily[v] != family) continue;
        double ms_best = 1e30;
        for (int rep = 0; rep < 2; rep++) {   // the first run warms the code and L2
            CROMA_CUDA(cudaMemcpyAsync(scratch, real, (size_t)T * NB * sizeof(double), cudaMemcpyDeviceToDevice,
                                       ctx.stream));
            CROMA_CUDA(cudaEventRecord(e0, ctx.stream));
            CROMA_CUDA((src ? launch_variant<S, true>(ctx.stream, Q, v, T) : launch_variant<S, false>(ctx.stream, Q, v, T)));
            CROMA_CUDA(cudaEventRecord(e1, ctx.stream));
            CROMA_CUDA(cudaEventSynchronize(e1));
            float ms = 0.0f;
            CROMA_CUDA(cudaEventElapsedTime(&ms, e0, e1));
            if (rep == 1) ms_best = ms;
        }
        tu.ms[v] = ms_best;
        if (best < 0 || ms_best < tu.ms[best]) best = v;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    tu.variant = best < 0 ? 0 : best;
    tu.tuned = 1;
    tu.tracers = T;
    tu.steps = steps;
    return 0;
}

template <int S>
cudaError_t launch_steps(Context &ctx, const FusedParams &P, bool src, bool perstep)
{
    if (perstep) {
        if (src) plain_steps_kernel<S, true><<<P.nt, 32, 0, ctx.stream>>>(P);
        else plain_steps_kernel<S, false><<<P.nt, 32, 0, ctx.stream>>>(P);
        return cudaGetLastError();
    }
    if (ctx.cfg.path == CROMA_PATH_FUSED_FP32R) {
        if (src) return launch_steps_variant<S, true, kSolveRefined, 1>(ctx.stream, P, 0);
        return launch_steps_variant<S, false, kSolveRefined, 1>(ctx.stream, P, 0);
    }
    if (packed_rule(ctx, P)) {
        TuneState &tu = ctx.tune[S];
        if (tu.variant != kPackedVariant) {
            tu = TuneState{};
            tu.variant = kPackedVariant;
        }
        tu.tuned = 1;
        return src ? launch_packed<S, true>(ctx.stream, P) : launch_packed<S, false>(ctx.stream, P);
    }
    if (!ctx.tune[S].tuned || ctx.tune[S].variant == kPackedVariant) {
        const int rc = tune_steps<S>(ctx, P, src);
        if (rc) return cudaErrorUnknown;
    }
    const int v = ctx.tune[S].variant;
    return src ? launch_variant<S, true>(ctx.stream, P, v, 0) : launch_variant<S, false>(ctx.stream, P, v, 0);
}

// Workspace budget of the fused path (factored matrices, segment-start
// proton spectra, segment sources); CROMA_B200_WORKSPACE_GB overrides it.
double workspace_budget_bytes()
{
    const char *s = getenv("CROMA_B200_WORKSPACE_GB");
    double gb = s ? atof(s) : 0.0;
    if (!(gb > 0.0)) gb = 24.0;
    return gb * 1e9;
}

}  // namespace

namespace {

struct WorkspaceShape {
    int nseg, sets;
    long long chunk;
    double per_tracer;
};

// The per-step path holds one segment slot at a time; the on-chip path all
// of a snapshot's slots.
WorkspaceShape workspace_shape(const ModelParams &mp, int cap, double workspace_cap, bool perstep)
{
    WorkspaceShape w;
    w.nseg = perstep ? 1
                     : (mp.interp_max_segments < 1 ? 1 : (mp.interp_max_segments > 64 ? 64 : mp.interp_max_segments));
    w.sets = mp.window_centred ? 2 : 1;
    w.per_tracer = 8.0 * NB * ((double)2 * w.nseg * w.sets * 3 + 2.0 * w.nseg) + (double)w.nseg * sizeof(SegPre);
    const double budget = workspace_cap > 0.0 ? workspace_cap : workspace_budget_bytes();
    w.chunk = (long long)(budget / w.per_tracer);
    if (w.chunk < 1) w.chunk = 1;
    if (w.chunk > cap) w.chunk = cap;
    return w;
}

}  // namespace

double fused_workspace_bytes(const ModelParams &mp, int cap, double workspace_cap, int path)
{
    const WorkspaceShape w = workspace_shape(mp, cap, workspace_cap, path == CROMA_PATH_PLAIN);
    return (double)w.chunk * (w.per_tracer + sizeof(int)) + 8.0 * cap + 2.0 * kOrderBins * sizeof(unsigned);
}

int fused_reserve(Context &ctx, int cap)
{
    const WorkspaceShape w = workspace_shape(ctx.mp, cap, ctx.workspace_bytes, ctx.cfg.path == CROMA_PATH_PLAIN);
    const int nseg = w.nseg, sets = w.sets;
    const long long chunk = w.chunk;
    dev_free(ctx, ctx.d_inje);
    dev_free(ctx, ctx.d_eta_scale);
    dev_free(ctx, ctx.d_fac);
    dev_free(ctx, ctx.d_np_seg);
    dev_free(ctx, ctx.d_segpre);
    dev_free(ctx, ctx.d_order);
    ctx.d_inje = ctx.d_eta_scale = ctx.d_fac = ctx.d_np_seg = nullptr;
    ctx.d_segpre = nullptr;
    ctx.d_order = nullptr;
    ctx.fused_chunk = ctx.fused_nseg = ctx.fused_sets = 0;
    const size_t rows = (size_t)nseg * chunk * NB;
    CROMA_CUDA(dev_alloc(ctx, &ctx.d_fac, (size_t)2 * sets * rows * 3 * sizeof(double)));
    CROMA_CUDA(dev_alloc(ctx, &ctx.d_np_seg, rows * sizeof(double)));
    CROMA_CUDA(dev_alloc(ctx, &ctx.d_inje, rows * sizeof(double)));
    CROMA_CUDA(dev_alloc(ctx, &ctx.d_eta_scale, (size_t)cap * sizeof(double)));
    CROMA_CUDA(dev_alloc(ctx, &ctx.d_segpre, (size_t)nseg * chunk * sizeof(SegPre)));
    CROMA_CUDA(dev_alloc(ctx, &ctx.d_order, (2 * kOrderBins + (size_t)chunk) * sizeof(int)));
    ctx.fused_chunk = (int)chunk;
    ctx.fused_nseg = nseg;
    ctx.fused_sets = sets;
    return 0;
}

// Segments [g0, g1) of one tracer chunk: the eta-cap scales (if the cap is
// on), the factored matrices of both species, the proton steps, the
// secondary source, the electron steps.  perstep (the plain path, one slot):
// the raw rows of both species, the secondary source from the protons at the
// slot start, then the per-step kernels.
// Host-pipeline copies of one chunk's rows of one species: after an event on
// the compute stream, on the d2h stream.
static int pipe_download(Context &ctx, const FusedParams &P, cudaEvent_t ev, double *host, const double *dev)
{
    CROMA_CUDA(cudaEventRecord(ev, ctx.stream));
    CROMA_CUDA(cudaStreamWaitEvent(ctx.d2h_stream, ev, 0));
    const size_t off = (size_t)P.t0 * NB, bytes = (size_t)P.nt * NB * sizeof(double);
    CROMA_CUDA(cudaMemcpyAsync(host + off, dev + off, bytes, cudaMemcpyDeviceToHost, ctx.d2h_stream));
    return 0;
}

static void launch_seg_pre(Context &ctx, const FusedParams &P)
{
    const long long total = (long long)(P.g1 - P.g0) * P.nt;
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    long long blocks = (total + 255) / 256;
    if (blocks > 8LL * nsm) blocks = 8LL * nsm;
    seg_pre_kernel<<<(unsigned)blocks, 256, 0, ctx.stream>>>(P);
}

// pk >= 0 (host pipeline, all segments in one launch): the chunk's upload is
// awaited only before the first steps kernel -- the per-segment scalars and
// the factored rows do not read the spectra -- and the proton rows go back as
// soon as the proton steps are done.  scalars_done: the slots' scalars are
// there already, P.pre at this slot's.
static int fused_range(Context &ctx, FusedParams &P, int g0, int g1, bool perstep, int pk = -1, bool scalars_done = false)
{
    const SnapArgs &a = P.a;
    const int protons = ctx.mp.species_mask & CROMA_SPECIES_PROTON;
    const int electrons = ctx.mp.species_mask & CROMA_SPECIES_ELECTRON;
    const bool secondaries = protons && electrons;
    const bool cap = ctx.mp.eta_dpp_cap > 0.0 && isfinite(ctx.mp.eta_dpp_cap) && ctx.mp.dpp_model != kDppOff;
    if ((cap || perstep) && g1 != g0 + 1) {
        set_error("internal: the eta cap and the per-step path need one segment per launch");
        return -1;
    }
    P.g0 = g0;
    P.g1 = g1;
    P.eta_scale = nullptr;
    // protons at the segment start: recorded by the steps kernel, or (per
    // step, one slot) the chunk's resident rows themselves
    P.np_seg = !secondaries ? nullptr : (perstep ? a.crp + (size_t)P.t0 * NB : ctx.d_np_seg);
    P.inje = secondaries ? ctx.d_inje : nullptr;
    cudaEvent_t ev = nullptr;
    timed_begin(ctx, kKindCoeff, &ev);
    if (cap) {
        eta_scale_kernel<<<(P.nt + 3) / 4, 128, 0, ctx.stream>>>(P, ctx.d_eta_scale);
        ctx.last_launches += 1;
        P.eta_scale = ctx.d_eta_scale;
    }
    if ((protons || electrons) && !scalars_done) {
        launch_seg_pre(ctx, P);
        ctx.last_launches += 1;
    }
    if (protons) {
        CROMA_CUDA((perstep ? launch_factor<0, true>(ctx, P) : launch_factor<0, false>(ctx, P)));
        ctx.last_launches += 1;
    }
    if (electrons) {
        CROMA_CUDA((perstep ? launch_factor<1, true>(ctx, P) : launch_factor<1, false>(ctx, P)));
        ctx.last_launches += 1;
    }
    timed_end(ctx, kKindCoeff, ev);
    if (pk >= 0) CROMA_CUDA(cudaStreamWaitEvent(ctx.stream, ctx.pipe_up[pk], 0));
    if (secondaries && perstep) {
        timed_begin(ctx, kKindSecondary, &ev);
        CROMA_CUDA(launch_secondary(ctx, P));
        timed_end(ctx, kKindSecondary, ev);
        ctx.last_launches += 1;
    }
    if (protons) {
        timed_begin(ctx, kKindEvolve, &ev);
        CROMA_CUDA(launch_steps<0>(ctx, P, a.qpi != nullptr, perstep));
        timed_end(ctx, kKindEvolve, ev);
        ctx.last_launches += 1;
    }
    if (pk >= 0 && ctx.pipe->down_p) {
        const int rc = pipe_download(ctx, P, ctx.pipe_done_p[pk], ctx.pipe->crp, a.crp);
        if (rc) return rc;
    }
    if (secondaries && !perstep) {
        timed_begin(ctx, kKindSecondary, &ev);
        CROMA_CUDA(launch_secondary(ctx, P));
        timed_end(ctx, kKindSecondary, ev);
        ctx.last_launches += 1;
    }
    if (electrons) {
        timed_begin(ctx, kKindEvolve, &ev);
        CROMA_CUDA(launch_steps<1>(ctx, P, secondaries || a.qepri != nullptr, perstep));
        timed_end(ctx, kKindEvolve, ev);
        ctx.last_launches += 1;
    }
    CROMA_CUDA(cudaGetLastError());
    return 0;
}

// Every segment slot of every tracer chunk.
static int fused_chunks(Context &ctx, FusedParams &P, int nslots, bool perstep)
{
    if (ctx.fused_chunk <= 0 || !ctx.d_fac) {
        set_error("fused workspace not reserved");
        return -1;
    }
    if ((perstep ? 1 : nslots) > ctx.fused_nseg) {
        set_error("internal: more segment slots than the fused workspace holds");
        return -1;
    }
    const bool windows = P.explicit_seg ? P.ex.windowed != 0 : ctx.mp.window_centred != 0;
    if (windows && ctx.fused_sets < 2) {
        set_error("internal: windowed segments without an off-coefficient workspace");
        return -1;
    }
    // the evolve kernels access rows with 32-byte vector loads and stores
    auto misaligned = [](const void *p) { return ((uintptr_t)p & 31u) != 0; };
    if (misaligned(P.a.crp) || misaligned(P.a.cre) || misaligned(P.a.qpi) || misaligned(P.a.qepri) ||
        misaligned(ctx.d_fac) || misaligned(ctx.d_inje) || misaligned(ctx.d_np_seg)) {
        set_error("internal: spectra, sources or workspace not 32-byte aligned");
        return -1;
    }
    const bool cap = ctx.mp.eta_dpp_cap > 0.0 && isfinite(ctx.mp.eta_dpp_cap) && ctx.mp.dpp_model != kDppOff;
    P.sets = ctx.fused_sets;
    P.fac = ctx.d_fac;
    P.pre = static_cast<SegPre *>(ctx.d_segpre);
    // chunks: the workspace's uniform split, or the host pipeline's bounds
    // (each within the workspace chunk), whose uploads gate the chunk and
    // whose downloads follow it
    const HostPipe *pipe = ctx.pipe;
    const int nchunk = pipe ? (int)pipe->bounds.size() - 1
                            : (P.a.ntracer + ctx.fused_chunk - 1) / ctx.fused_chunk;
    for (int k = 0; k < nchunk; k++) {
        P.t0 = pipe ? pipe->bounds[k] : k * ctx.fused_chunk;
        const int t1 = pipe ? pipe->bounds[k + 1]
                            : (P.a.ntracer - P.t0 < ctx.fused_chunk ? P.a.ntracer : P.t0 + ctx.fused_chunk);
        P.nt = t1 - P.t0;
        if (P.nt <= 0 || P.nt > ctx.fused_chunk) {
            set_error("internal: tracer chunk outside the fused workspace");
            return -1;
        }
        P.order = nullptr;
        if (!perstep && !P.explicit_seg && packed_rule(ctx, P)) {
            int *order = ctx.d_order + 2 * kOrderBins;
            CROMA_CUDA(launch_order(ctx.stream, P.nt, P.a.sched.nsub + P.t0, reinterpret_cast<unsigned *>(ctx.d_order),
                                    order));
            P.order = order;
            ctx.last_launches += P.nt <= kOrderOneBlock ? 1 : 2;
        }
        if (!cap && !perstep) {
            // one launch per kernel for the chunk: the upload wait and the
            // proton download sit inside, next to the kernels they gate
            const int rc = fused_range(ctx, P, 0, nslots, false, pipe ? k : -1);
            if (rc) return rc;
        } else {
            if (pipe) CROMA_CUDA(cudaStreamWaitEvent(ctx.stream, ctx.pipe_up[k], 0));
            // one slot per launch; the on-chip path's workspace holds the scalars
            // of all slots, which do not depend on the spectra, so they take one
            // launch: 21 us at 16 slots of 10,000 windowed tracers, 16 of 7.3 before
            const bool once = !perstep && (ctx.mp.species_mask & 3);
            SegPre *const base = P.pre;
            if (once) {
                P.g0 = 0;
                P.g1 = nslots;
                cudaEvent_t ev = nullptr;
                timed_begin(ctx, kKindCoeff, &ev);
                launch_seg_pre(ctx, P);
                timed_end(ctx, kKindCoeff, ev);
                ctx.last_launches += 1;
            }
            for (int g = 0; g < nslots; g++) {
                P.pre = once ? base + (size_t)g * P.nt : base;
                const int rc = fused_range(ctx, P, g, g + 1, perstep, -1, once);
                if (rc) {
                    P.pre = base;
                    return rc;
                }
            }
            P.pre = base;
            if (pipe && pipe->down_p) {
                const int rc = pipe_download(ctx, P, ctx.pipe_done_p[k], pipe->crp, P.a.crp);
                if (rc) return rc;
            }
        }
        if (pipe && pipe->down_e) {
            const int rc = pipe_download(ctx, P, ctx.pipe_done[k], pipe->cre, P.a.cre);
            if (rc) return rc;
        }
    }
    return 0;
}

int run_fused(Context &ctx, const SnapArgs &a)
{
    FusedParams P{};
    P.a = a;
    P.gt = ctx.gt;
    P.mp = ctx.mp;
    P.np_min_qe = ctx.d_np_min_qe;
    P.explicit_seg = 0;
    P.ex = SegInfo{};
    P.ic_stride = 0;
    const int nslots = ctx.mp.interp_max_segments < 1 ? 1
                     : (ctx.mp.interp_max_segments > 64 ? 64 : ctx.mp.interp_max_segments);
    return fused_chunks(ctx, P, nslots, ctx.cfg.path == CROMA_PATH_PLAIN);
}

int tuning_info(const Context &ctx, int species, int *solver, int *wpb)
{
    if (species < 0 || species > 1) return -1;
    const TuneState &t = ctx.tune[species];
    if (solver) *solver = kVariantSolver[t.variant];
    if (wpb) *wpb = kVariantWpb[t.variant];
    return t.tuned;
}

int run_fused_segment(Context &ctx, const SnapArgs &a, const SegInfo &ex, int ic_stride)
{
    FusedParams P{};
    P.a = a;
    P.gt = ctx.gt;
    P.mp = ctx.mp;
    P.np_min_qe = ctx.d_np_min_qe;
    P.explicit_seg = 1;
    P.ex = ex;
    P.ic_stride = ic_stride;
    return fused_chunks(ctx, P, 1, false);
}

}  // namespace croma
