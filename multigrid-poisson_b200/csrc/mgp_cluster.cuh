// mgp_cluster.cuh -- the coarse levels of a cycle in one thread-block cluster (included by
// mgp_engine.cu).
//
// From the first level T whose fields, and those of every coarser level, fit in the shared
// memory of one cluster, a visit of the cycle to level T (include/vcycle.h:14-98,
// include/fcycle.h:13-97) is ONE launch of one cluster of up to 16 CTAs.  Each CTA holds a slab
// of consecutive x planes of every level (u, f, r and the Neumann face rows, with one halo plane
// on each side) in its shared memory for the whole visit, and runs the visit as a host-written
// program of level operations.
//
// What bounds it: these levels are a chain of short dependent operations.  As separate kernels
// each costs 2.5-3 us (a launch boundary plus one or two round trips to L2); here an operation
// reads only the CTA's own shared memory and sends its boundary planes straight into the
// neighbours' halos.  A cluster barrier with release semantics costs 380-600 cycles on B200 and
// more with remote stores in flight (1000-2000 measured here), against 115 for the barrier alone,
// so the sweeps and residuals synchronise with their two neighbours only: every boundary value
// is an asynchronous remote store that counts down the receiver's mbarrier (st.async), and a CTA
// waits for the bytes of the two planes it needs (670 cycles for the exchange alone; remote stores
// followed by an mbarrier arrival took 1300-2900).  A plane that has arrived complete also tells
// that its sender is done reading the halo on that side, since the threads that read a halo
// plane are the ones that send.  Cluster barriers remain where data go beyond the neighbours:
// after a restriction and before a prolongation.
//
// Arithmetic: operand for operand that of the grid kernels (stencil_tile, k_resid_restrict,
// prolong_tile, bc_restrict_value), and the same values are left behind: u in both Jacobi
// buffers, f and the Neumann face data of the coarser levels, r at the unrelaxed points (the
// residual at relaxed points stays unstored, as in the one-kernel set-up).
#pragma once

namespace mgp {

constexpr int kClMaxLevels = 8;
constexpr int kClMaxOps = 160;
constexpr int kClMaxThreads = 640;
constexpr int kErrCluster = 2;  // the error word's value (the wavefront passes set 1)

template <typename T>
struct ClLevel {
    Geom G;
    T* ub[2];  // global u buffers (ub[1] null for Gauss-Seidel)
    T* f;
    T* r;
    T* g[6];
    int neumann[6];
    T two_h, hsq, inv_hsq, one_omega, omega_sixth, h;
    int pow2;
    int P, nact;       // planes per CTA; CTAs that own planes
    int rp, pl;            // row pitch in shared memory (even) and elements of a plane
    unsigned m_nz, m_ny, m_yz, m_rp, m_pl, m_P;  // cl_div's magic numbers
    int ncol;          // relaxed columns (points of a plane inside the y and z bounds)
    int nitem;         // work items of a relaxation: columns, or pairs of columns (red-black)
    int nseg, seglen;  // an item's planes are split over nseg threads, seglen planes each
    int rseg, rlen;    // the same for the residual's columns
    unsigned m_item, m_col;  // cl_div's magic numbers of nitem and ncol
    int so_tab, so_pair;  // byte offsets of the column table and the column-pair table
    int so_u[2], so_f, so_r, so_g[6];  // shared-memory offsets (elements), equal in every CTA
};

enum ClOp : unsigned char { CL_RELAX = 0, CL_RELAX_SKIP1 = 1, CL_SETUP = 2, CL_PROLONG = 3, CL_NORM = 4 };

template <typename T>
struct ClArgs {
    ClLevel<T> L[kClMaxLevels];
    int nl, ns, fw, alt, nops;
    int so_gather;  // scratch: the coarse planes a CTA's prolongation reads
    unsigned cur;   // bit l: the current u buffer of level l
    unsigned long long* norm;
    int* err;        // set when a wait for a neighbour's planes ran out
    unsigned polls;  // bound of such a wait
    unsigned char op[kClMaxOps], lv[kClMaxOps];
};

__device__ __forceinline__ unsigned cl_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Every thread of every CTA: all shared-memory writes before it, remote ones included, are
// visible to the whole cluster after it.  The block barrier orders the CTA's threads before the
// one thread whose cluster-scope fence then covers them all (a fence by every thread, as
// arrive.release makes it, costs 600 cycles at 1024 threads).
__device__ __forceinline__ void cl_sync() {
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("fence.acq_rel.cluster;" ::: "memory");
    __syncwarp();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// The same before data of a level go to another one, unless both levels sit in one CTA.
__device__ __forceinline__ void cl_sync_levels(int nact_a, int nact_b) {
    if (nact_a == 1 && nact_b == 1) __syncthreads();
    else cl_sync();
}
__device__ __forceinline__ unsigned cl_map(unsigned addr, unsigned rank) {
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
__device__ __forceinline__ void cl_st(unsigned addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void cl_st(unsigned addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void cl_ld(unsigned addr, double& v) {
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
}
__device__ __forceinline__ void cl_ld(unsigned addr, float& v) {
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
}
// asynchronous remote store; its bytes count towards the mbarrier `mb` of the same CTA
__device__ __forceinline__ void cl_send(unsigned addr, double v, unsigned mb) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
                 "l"(__double_as_longlong(v)), "r"(mb)
                 : "memory");
}
__device__ __forceinline__ void cl_send(unsigned addr, float v, unsigned mb) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
                 "r"(__float_as_uint(v)), "r"(mb)
                 : "memory");
}
__device__ __forceinline__ void cl_mbar_init(unsigned mb) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
}
__device__ __forceinline__ void cl_mbar_expect(unsigned mb, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool cl_mbar_test(unsigned mb, unsigned phase) {
    unsigned ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                 "selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(mb), "r"(phase)
                 : "memory");
    return ok;
}
__device__ __forceinline__ bool cl_mbar_try(unsigned mb, unsigned phase) {
    unsigned ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                 "selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(mb), "r"(phase)
                 : "memory");
    return ok;
}
// The bound of a wait, and whether any CTA's wait ran out; in shared memory, read only by waits that
// have to wait (the bound in a register cost 1.5% of the smallest solve: 33x17x17 318 -> 325 us).
// Red-black kernels exist for the default bound too, with waits that block from their first poll:
// the form below costs them 1-2% (65^3 FP32 F-cycles 1097 -> 1106 us, 17x25x9 414 -> 425), which
// Jacobi gains (33x17x17 322 -> 311).
struct ClWait {
    unsigned polls;
    int dead;
};
// Waits for the barrier's phase; false after `polls` polls, or once `dead` is set.  The first poll
// does not block, so that a bound of one fails on any plane still on its way.
__device__ __forceinline__ bool cl_mbar_wait(unsigned mb, unsigned phase, const volatile ClWait* w) {
    if (cl_mbar_test(mb, phase)) return true;
    const unsigned polls = w->polls;
    for (unsigned n = 1; n < polls && !w->dead; n++)
        if (cl_mbar_try(mb, phase)) return true;
    return false;
}
// Sets the int at shared-memory address `flag` in every CTA of the cluster.
__device__ __noinline__ void cl_raise(unsigned flag) {
    unsigned n;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
    for (unsigned r = 0; r < n; r++)
        asm volatile("st.shared::cluster.u32 [%0], 1;" ::"r"(cl_map(flag, r)) : "memory");
}
__device__ __forceinline__ void cl_copy(double* s, const double* g) { cp_async_elem(s, g); }
__device__ __forceinline__ void cl_copy(float* s, const float* g) { cp_async_elem(s, g); }
// n / d by the magic number ceil(2^32/d) (0 stands for d = 1); exact while n*d < 2^32
__device__ __forceinline__ int cl_div(int n, unsigned magic) {
    return magic ? (int)__umulhi((unsigned)n, magic) : n;
}

// What a sweep of a level needs in this CTA, in shared memory (read with a few vector loads: an
// operation costs a few hundred instructions per warp, so its set-up counts).
template <typename T>
struct __align__(16) ClCta {
    int u[2], f, r;               // offsets of the slab's first plane (elements)
    int nitem, nseg, seglen, tab; // relaxation items; tab: byte offset of their table
    int ncol, rseg, rlen, rtab;   // the residual's columns
    int lo, hi, np, i0;           // planes [i0, i0 + np), of which [lo, hi) (counted from i0) are relaxed
    int pl, rp, nz, ny, nx;
    unsigned la, ra;              // cluster addresses (offset 0) of the halo planes it fills, 0: no neighbour
    unsigned lmb, rmb;            // the neighbours' mbarriers for them
    unsigned bl[3], br[3];        // bytes expected from each side: colour 0, colour 1, every relaxed point
    unsigned m_item, m_col;
    int pow2;
    T two_h, hsq, inv_hsq, one_omega, omega_sixth;
};

// This CTA's share of level L: planes [i0, i0 + np).
template <typename T>
struct ClSlab {
    int i0, np;
    __device__ __forceinline__ ClSlab(const ClLevel<T>& L, int rank) {
        i0 = rank * L.P;
        np = min(L.P, L.G.nx - i0);
        if (np < 0) np = 0;
    }
};

// Column table entries: the column's index in the plane and the faces it lies on.  Columns off
// the faces come first, so whole warps take the ghost-free stencil.  Red-black relaxations work on
// pairs of columns (j, j+1), of which one point per plane has the colour, so every lane has work:
// the entry is the first column's, with the parity of j + k + poff, whether the second column is
// on the north face and whether there is one.  A warp's lanes run along k and alternate between
// the two rows; with an even row pitch their addresses fall into different banks.
enum : unsigned {
    CL_SOUTH = 1u << 16, CL_NORTH = 1u << 17, CL_BOTTOM = 1u << 18, CL_TOP = 1u << 19,
    CL_ODD = 1u << 20, CL_NORTH2 = 1u << 21, CL_ONE = 1u << 22
};
constexpr unsigned kClEdge = CL_SOUTH | CL_NORTH | CL_BOTTOM | CL_TOP;

// Bytes of plane i that an operation writes (and sends): its relaxed points (what = 2), or those
// of one colour in a red-black half-sweep.
template <typename T>
__device__ __forceinline__ unsigned cl_bytes(const ClLevel<T>& L, int i, int what) {
    if (i < L.G.x0 || i >= L.G.x1) return 0u;
    if (what == 2) return (unsigned)L.ncol * (unsigned)sizeof(T);
    const bool first = ((i + L.G.y0 + L.G.z0 + L.G.poff) & 1) == what;  // the box's first point is of the colour
    return (unsigned)((L.ncol + (first ? 1 : 0)) >> 1) * (unsigned)sizeof(T);
}

template <typename T, bool JAC>
__device__ __forceinline__ void cl_tables(const ClArgs<T>& a, unsigned char* smem, unsigned sbase, unsigned mb, ClCta<T>* S,
                                          int rank) {
    if ((int)threadIdx.x < a.nl) {
        const ClLevel<T>& L = a.L[threadIdx.x];
        ClCta<T> c;
        c.i0 = rank * L.P;
        c.np = max(0, min(L.P, L.G.nx - c.i0));
        c.u[0] = L.so_u[0] + L.pl;
        c.u[1] = L.so_u[1] + L.pl;
        c.f = L.so_f;
        c.r = L.so_r + L.pl;
        c.nitem = L.nitem;
        c.nseg = L.nseg;
        c.seglen = L.seglen;
        c.tab = JAC ? L.so_tab : L.so_pair;
        c.ncol = L.ncol;
        c.rseg = L.rseg;
        c.rlen = L.rlen;
        c.rtab = L.so_tab;
        c.lo = max(0, L.G.x0 - c.i0);
        c.hi = min(c.np, L.G.x1 - c.i0);
        c.pl = L.pl;
        c.rp = L.rp;
        c.nz = L.G.nz;
        c.ny = L.G.ny;
        c.nx = L.G.nx;
        c.la = c.ra = c.lmb = c.rmb = 0u;
        const unsigned plane = (unsigned)L.pl * (unsigned)sizeof(T);
        if (rank > 0 && rank < L.nact) {  // past the last plane of the left neighbour's slab
            c.la = cl_map(sbase + (unsigned)L.P * plane, rank - 1);
            c.lmb = cl_map(mb + 16, rank - 1);
        }
        if (rank + 1 < L.nact) {  // before the first plane of the right neighbour's slab
            c.ra = cl_map(sbase, rank + 1) - plane;
            c.rmb = cl_map(mb, rank + 1);
        }
        for (int q = 0; q < 3; q++) {
            c.bl[q] = c.la ? cl_bytes(L, c.i0 - 1, q) : 0u;
            c.br[q] = c.ra ? cl_bytes(L, c.i0 + c.np, q) : 0u;
        }
        c.m_item = L.m_item;
        c.m_col = L.m_col;
        c.pow2 = L.pow2;
        c.two_h = L.two_h;
        c.hsq = L.hsq;
        c.inv_hsq = L.inv_hsq;
        c.one_omega = L.one_omega;
        c.omega_sixth = L.omega_sixth;
        S[threadIdx.x] = c;
    }
    for (int l = 0; l < a.nl; l++) {
        const ClLevel<T>& L = a.L[l];
        const Geom& G = L.G;
        unsigned* tab = reinterpret_cast<unsigned*>(smem + L.so_tab);
        // the box of columns off the faces, then the relaxed ones on rows j = 0 and ny-1, then
        // those on k = 0 and nz-1
        const int ya = max(G.y0, 1), yb = min(G.y1, G.ny - 1), za = max(G.z0, 1), zb = min(G.z1, G.nz - 1);
        const int wz = max(0, zb - za), wy = max(0, yb - ya), ni = wz * wy, w = G.z1 - G.z0;
        const int rows = (G.y0 == 0) + (G.y1 == G.ny);
        const bool south = G.y0 == 0, bottom = G.z0 == 0;
        const int sides = (G.z0 == 0) + (G.z1 == G.nz);
        for (int c = threadIdx.x; c < L.ncol; c += blockDim.x) {
            int j, k;
            if (c < ni) {
                j = ya + c / wz;
                k = za + c % wz;
            } else if (c < ni + rows * w) {
                const int q = c - ni;
                j = q < w && south ? 0 : G.ny - 1;
                k = G.z0 + q % w;
            } else {
                const int q = c - ni - rows * w;
                j = ya + q / sides;
                k = q % sides == 0 && bottom ? 0 : G.nz - 1;
            }
            tab[c] = (unsigned)(j * L.rp + k) | (j == 0 ? CL_SOUTH : 0u) | (j == G.ny - 1 ? CL_NORTH : 0u) |
                     (k == 0 ? CL_BOTTOM : 0u) | (k == G.nz - 1 ? CL_TOP : 0u);
        }
        if (JAC) continue;
        unsigned* pair = reinterpret_cast<unsigned*>(smem + L.so_pair);
        for (int c = threadIdx.x; c < L.nitem; c += blockDim.x) {
            const int j = G.y0 + c / w * 2, k = G.z0 + c % w;
            pair[c] = (unsigned)(j * L.rp + k) | (j == 0 ? CL_SOUTH : 0u) | (j == G.ny - 1 ? CL_NORTH : 0u) |
                      (k == 0 ? CL_BOTTOM : 0u) | (k == G.nz - 1 ? CL_TOP : 0u) |
                      (j + 1 == G.ny - 1 ? CL_NORTH2 : 0u) | (j + 1 >= G.y1 ? CL_ONE : 0u) |
                      (((j + k + G.poff) & 1) ? CL_ODD : 0u);
        }
    }
}

// Stores v at row entry `idx` of x plane I of a halo-padded array (rows of `len` elements, `off`
// its shared-memory offset) in the CTA that owns the plane and in the neighbours' halos.
template <typename T>
__device__ __forceinline__ void cl_put(const ClLevel<T>& L, unsigned sbase, int off, int len, int I, int idx, T v) {
    const int rank = cl_div(I, L.m_P);
    const int slot = I - rank * L.P + 1;
    cl_st(cl_map(sbase + (unsigned)(off + slot * len + idx) * (unsigned)sizeof(T), rank), v);
    if (slot == 1 && rank > 0)
        cl_st(cl_map(sbase + (unsigned)(off + (L.P + 1) * len + idx) * (unsigned)sizeof(T), rank - 1), v);
    if (slot == L.P && I + 1 < L.G.nx) cl_st(cl_map(sbase + (unsigned)(off + idx) * (unsigned)sizeof(T), rank + 1), v);
}

// The CTA's exchange state: mbarriers 0/1 count the bytes from the left neighbour, 2/3 those from
// the right one, alternating from one exchange to the next (`n`, counted in program order by
// every CTA): a neighbour cannot be two exchanges of a level ahead, as each needs the other's
// planes.  phase: bit b is the phase of barrier b this CTA waits for next.
//
// A thread whose wait runs out (never seen but with a bound set for it) goes through the rest of
// the program without announcing, waiting or sending, and raises the flag in every CTA, which ends
// the others' waits: without its values its neighbours' waits cannot complete either.  An
// mbarrier takes one arrival per phase; the announcing thread makes it, after its own wait for
// the barrier's phase before came to its end, so none is one too many.  A CTA that no longer
// announces gets two planes more from a neighbour at most (until that one's waits fail), far from
// the 2^20 bytes a barrier may be ahead.
struct ClXchg {
    unsigned mb;
    unsigned n, phase;
    ClWait* w;
    bool dead;  // this thread's wait ran out, or was ended by another's
    template <bool BOUND>
    __device__ __forceinline__ bool wait(unsigned q) {
        if (BOUND) {
            if (cl_mbar_wait(mb + 8 * q, (phase >> q) & 1, w)) return true;
        } else {
            for (unsigned n = 0; n < kWaitPolls; n++) {
                if (cl_mbar_try(mb + 8 * q, (phase >> q) & 1)) return true;
                if (*(const volatile int*)&w->dead) break;
            }
        }
        cl_raise((unsigned)__cvta_generic_to_shared(&w->dead));
        return false;
    }
};

// Where an operation's results go: the slab, and the neighbours' halos.
template <typename T>
struct ClOut {
    unsigned la, ra, lmb, rmb;
    int last;
    __device__ __forceinline__ ClOut(const ClCta<T>& s, int dst, unsigned b)
        : la(s.la ? s.la + (unsigned)dst * (unsigned)sizeof(T) : 0u),
          ra(s.ra ? s.ra + (unsigned)dst * (unsigned)sizeof(T) : 0u), lmb(s.lmb + b), rmb(s.rmb + b), last(s.np - 1) {}
    __device__ __forceinline__ void put(T* d, int ii, int rem, T v) const {
        *d = v;
        if (ii == 0 && la) cl_send(la + (unsigned)rem * (unsigned)sizeof(T), v, lmb);
        if (ii == last && ra) cl_send(ra + (unsigned)rem * (unsigned)sizeof(T), v, rmb);
    }
};

// The in-plane neighbours of a point on a face (flags e): Neumann ghosts where there is none.
template <typename T>
__device__ __forceinline__ void cl_edge(const ClArgs<T>& a, int l, const ClCta<T>& s, const T* sm, const T* u, int ii,
                                        int rem, unsigned e, T& ym, T& yp, T& zm, T& zp) {
    const int* g = a.L[l].so_g;
    const int j = cl_div(rem, a.L[l].m_rp), k = rem - j * s.rp;
    const T h2 = s.two_h, m2h = -s.two_h;
    ym = !(e & CL_SOUTH) ? u[-s.rp] : m2h * sm[g[F_SOUTH] + (ii + 1) * s.nz + k] + u[s.rp];
    yp = !(e & CL_NORTH) ? u[s.rp] : h2 * sm[g[F_NORTH] + (ii + 1) * s.nz + k] + u[-s.rp];
    zm = !(e & CL_BOTTOM) ? u[-1] : m2h * sm[g[F_BOTTOM] + (ii + 1) * s.ny + j] + u[1];
    zp = !(e & CL_TOP) ? u[1] : h2 * sm[g[F_TOP] + (ii + 1) * s.ny + j] + u[-1];
}

template <typename T, int OP>
__device__ __forceinline__ T cl_value(const ClCta<T>& s, T vm, T vp, T ym, T yp, T zm, T zp, T c, T fv) {
    const T sum = vm + vp + ym + yp + zm + zp;
    return OP == OP_RESIDUAL ? residual_pt(fv, sum, c, s.hsq, s.inv_hsq, s.pow2)
                             : s.one_omega * c + s.omega_sixth * (sum - s.hsq * fv);
}

// Jacobi or the residual on the planes [lo, hi) of one column, u(i-1), u(i), u(i+1) in registers.
template <typename T, int OP>
__device__ __forceinline__ void cl_march(const ClArgs<T>& a, int l, const ClCta<T>& s, T* sm, int src, int dst, unsigned e,
                                         int lo, int hi, const ClOut<T>& out) {
    const int rem = (int)(e & 0xffffu);
    const T* u = sm + src + rem + lo * s.pl;
    T* d = sm + dst + rem + lo * s.pl;
    const T* f = sm + s.f + rem + lo * s.pl;
    T vm = s.i0 + lo > 0 ? u[-s.pl] : -s.two_h * sm[a.L[l].so_g[F_WEST] + rem] + u[s.pl];
    T c = u[0];
    const bool edge = (e & kClEdge) != 0u;
    for (int ii = lo; ii < hi; ii++) {
        const T fv = f[0];
        const T vp = s.i0 + ii < s.nx - 1 ? u[s.pl] : s.two_h * sm[a.L[l].so_g[F_EAST] + rem] + u[-s.pl];
        T ym, yp, zm, zp;
        if (!edge) {
            ym = u[-s.rp];
            yp = u[s.rp];
            zm = u[-1];
            zp = u[1];
        } else {
            cl_edge(a, l, s, sm, u, ii, rem, e, ym, yp, zm, zp);
        }
        out.put(d, ii, rem, cl_value<T, OP>(s, vm, vp, ym, yp, zm, zp, c, fv));
        vm = c;
        c = vp;
        u += s.pl;
        d += s.pl;
        f += s.pl;
    }
}

// A red-black half-sweep on the planes [lo, hi) of a pair of columns.
template <typename T>
__device__ __forceinline__ void cl_march_pair(const ClArgs<T>& a, int l, const ClCta<T>& s, T* sm, int src, unsigned e,
                                              int lo, int hi, int colour, const ClOut<T>& out) {
    const int rem0 = (int)(e & 0xffffu);
    int second = ((s.i0 + lo + (int)((e >> 20) & 1u)) & 1) != colour;  // the pair's point of the colour in plane lo
    const int base = src + rem0 + lo * s.pl;
    for (int ii = lo, p = base; ii < hi; ii++, p += s.pl, second ^= 1) {
        if (second && (e & CL_ONE)) continue;
        const int rem = second ? rem0 + s.rp : rem0;
        T* u = sm + (second ? p + s.rp : p);
        const T fv = sm[s.f + rem + ii * s.pl];
        const T vm = s.i0 + ii > 0 ? u[-s.pl] : -s.two_h * sm[a.L[l].so_g[F_WEST] + rem] + u[s.pl];
        const T vp = s.i0 + ii < s.nx - 1 ? u[s.pl] : s.two_h * sm[a.L[l].so_g[F_EAST] + rem] + u[-s.pl];
        T ym, yp, zm, zp;
        const unsigned ee = second ? (e & (CL_BOTTOM | CL_TOP)) | ((e & CL_NORTH2) ? CL_NORTH : 0u) : e & kClEdge;
        if (!ee) {
            ym = u[-s.rp];
            yp = u[s.rp];
            zm = u[-1];
            zp = u[1];
        } else {
            cl_edge(a, l, s, sm, u, ii, rem, ee, ym, yp, zm, zp);
        }
        out.put(u, ii, rem, cl_value<T, OP_GS>(s, vm, vp, ym, yp, zm, zp, u[0], fv));
    }
}

// Announces the bytes the neighbours will send for the exchange that begins: one thread of the
// last warp, which has the least to do.
template <typename T>
__device__ __forceinline__ void cl_expect(const ClCta<T>& s, const ClXchg& X, int what) {
    if (threadIdx.x == blockDim.x - 1 && !X.dead) {
        const unsigned b = (X.n & 1) * 8;
        if (s.la) cl_mbar_expect(X.mb + b, s.bl[what]);
        if (s.ra) cl_mbar_expect(X.mb + 16 + b, s.br[what]);
    }
}

// Ends a sweep or residual of level L: the CTA's own values, and the neighbours' planes in its
// halos, are there.  Every CTA calls it; those without planes of the level only count.
template <typename T, bool BOUND>
__device__ __forceinline__ void cl_exchange(const ClCta<T>& S, ClXchg& X) {
    const unsigned b = X.n & 1;
    X.n++;
    if (S.np == 0) return;
    const bool from_left = S.la != 0u, from_right = S.ra != 0u;
    __syncthreads();
    if (from_left) {
        if (!X.dead) X.dead = !X.wait<BOUND>(b);
        X.phase ^= 1u << b;
    }
    if (from_right) {
        if (!X.dead) X.dead = !X.wait<BOUND>(2 + b);
        X.phase ^= 4u << b;
    }
}

// r = f - A u over this CTA's planes of level l; ends the exchange unless the caller does.
template <typename T>
__device__ __forceinline__ void cl_residual(const ClArgs<T>& a, int l, const ClCta<T>& S, T* sm, int src, const ClXchg& X) {
    const ClCta<T> s = S;
    if (s.np == 0) return;
    cl_expect(S, X, 2);
    const ClOut<T> out(s, s.r, (X.n & 1) * 8);
    const unsigned* tab = reinterpret_cast<const unsigned*>(reinterpret_cast<const unsigned char*>(sm) + s.rtab);
    const int seg = s.rseg > 1 ? cl_div((int)threadIdx.x, s.m_col) : 0;
    const int step = s.rseg > 1 ? s.ncol : (int)blockDim.x;
    const int lo = max(seg * s.rlen, s.lo), hi = seg < s.rseg ? min(s.hi, (seg + 1) * s.rlen) : lo;
    if (lo >= hi || X.dead) return;
    for (int c = (int)threadIdx.x - seg * s.ncol; c < s.ncol; c += step)
        cl_march<T, OP_RESIDUAL>(a, l, s, sm, src, s.r, tab[c], lo, hi, out);
}

// Relaxation<T>::relax of level l: nsmooth Jacobi sweeps (swapping the buffers) or 2*nsmooth
// red-black half-sweeps, the first one skipped on request.  What a thread needs for the level
// stays in registers from sweep to sweep.
template <typename T, bool JAC, bool BOUND>
__device__ __forceinline__ void cl_relax(const ClArgs<T>& a, int l, const ClCta<T>& S, T* sm, bool skip, unsigned& cur,
                                         int& alt, ClXchg& X) {
    const ClCta<T> s = S;
    const int sweeps = JAC ? a.ns : 2 * a.ns;
    const unsigned* tab = reinterpret_cast<const unsigned*>(reinterpret_cast<const unsigned char*>(sm) + s.tab);
    const int seg = s.nseg > 1 ? cl_div((int)threadIdx.x, s.m_item) : 0;
    const int step = s.nseg > 1 ? s.nitem : (int)blockDim.x;
    const int lo = max(seg * s.seglen, s.lo), hi = seg < s.nseg ? min(s.hi, (seg + 1) * s.seglen) : lo;
    const int c0 = lo < hi ? (int)threadIdx.x - seg * s.nitem : s.nitem;
    const unsigned e0 = c0 < s.nitem ? tab[c0] : 0u;
    for (int it = 0; it < sweeps; it++) {
        int src, dst;
        const int colour = alt ? 0 : 1;
        if (JAC) {
            cur ^= 1u << l;  // swap_u
            const bool one = (cur >> l) & 1u;
            dst = one ? s.u[1] : s.u[0];
            src = one ? s.u[0] : s.u[1];
        } else {
            alt = !alt;
            src = dst = s.u[0];
        }
        if (it == 0 && skip) continue;
        if (s.np > 0) {
            cl_expect(S, X, JAC ? 2 : colour);
            const ClOut<T> out(s, dst, (X.n & 1) * 8);
            unsigned e = e0;
            for (int c = X.dead ? s.nitem : c0; c < s.nitem; e = (c += step) < s.nitem ? tab[c] : 0u) {
                if (JAC) cl_march<T, OP_JACOBI>(a, l, s, sm, src, dst, e, lo, hi, out);
                else cl_march_pair(a, l, s, sm, src, e, lo, hi, colour, out);
            }
        }
        cl_exchange<T, BOUND>(S, X);
    }
}

// Neumann::restrict_to of every Neumann face (bc_restrict_value's arithmetic): the CTA that owns
// fine plane 2I forms row I of the coarse north/south/top/bottom faces; the CTAs of the first and
// the last plane form the west and the east face.
template <typename T>
__device__ __forceinline__ void cl_face_restrict(const ClArgs<T>& a, int l, T* sm, unsigned sbase, int so_u, int rank) {
    const ClLevel<T>& F = a.L[l];
    const ClLevel<T>& C = a.L[l + 1];
    const Geom& G = F.G;
    const Geom& Gc = C.G;
    const ClSlab<T> S(F, rank);
    if (S.np == 0) return;
    const int I0 = (S.i0 + 1) >> 1, I1 = (S.i0 + S.np + 1) >> 1;  // coarse planes I with 2I in the slab
    // the warps are dealt out to the Neumann faces, so that the faces' chains run side by side
    int nf = 0;
#pragma unroll
    for (int q = 0; q < 6; q++) nf += C.neumann[q] != 0;
    if (nf == 0) return;
    const int warp = (int)threadIdx.x >> 5, group = warp % nf;
    const int nthr = (((int)blockDim.x >> 5) - group + nf - 1) / nf * 32;  // threads of this face
    const int t0 = warp / nf * 32 + ((int)threadIdx.x & 31);
    int fc = -1;
    for (int q = 0, g = group; q < 6; q++)
        if (C.neumann[q] && g-- == 0) fc = q;
    const T* gf = sm + F.so_g[fc];
    const bool upper = fc == F_EAST || fc == F_NORTH || fc == F_TOP;
    const T c1 = upper ? T(3.0 / 2.0) : T(-3.0 / 2.0), c2 = upper ? T(-2.0) : T(2.0), c3 = upper ? T(0.5) : T(-0.5);
    const int d = upper ? -1 : 1;
    if (fc == F_EAST || fc == F_WEST) {
        const int x = upper ? G.nx - 1 : 0;
        if (x < S.i0 || x >= S.i0 + S.np) return;
        for (int t = t0; t < Gc.ny * Gc.nz; t += nthr) {
            const int J = cl_div(t, C.m_nz), K = t - J * Gc.nz;
            T g;
            if (a.fw) {
                const int jj = min(G.ny - 1, 2 * J), kk = min(G.nz - 1, 2 * K);
                auto A = [&](int, int y, int z) -> double { return (double)gf[y * F.rp + z]; };
                g = fw_sum<T>(A, 0, 0, 0, max(0, jj - 1), jj, min(G.ny - 1, jj + 1), max(0, kk - 1), kk,
                              min(G.nz - 1, kk + 1));
            } else {
                g = gf[2 * J * F.rp + 2 * K];
            }
            const int idx = 2 * J * F.rp + 2 * K;
            // planes x, x+d and x+2d: in the slab or its halo, as slabs hold at least two planes
            const T* up = sm + so_u + (x - S.i0 + 1) * F.pl + idx;
            g -= (c1 * up[0] + c2 * up[d * F.pl] + c3 * up[2 * d * F.pl]) / F.h;
            const int owner = upper ? C.nact - 1 : 0;
            cl_st(cl_map(sbase + (unsigned)(C.so_g[fc] + J * C.rp + K) * (unsigned)sizeof(T), owner), g);
        }
    } else {
        const bool ns = fc == F_NORTH || fc == F_SOUTH;  // rows along k, else rows along j
        const int len = ns ? G.nz : G.ny, clen = ns ? Gc.nz : Gc.ny;
        const unsigned m_clen = ns ? C.m_nz : C.m_ny;
        const int n = (I1 - I0) * clen;
        for (int t = t0; t < n; t += nthr) {
            const int row = cl_div(t, m_clen), q = t - row * clen, I = I0 + row;
            const int sl = 2 * I - S.i0 + 1;  // slot of fine row 2I
            T g;
            if (a.fw) {
                const int im = 2 * I > 0 ? sl - 1 : sl, ip = 2 * I < G.nx - 1 ? sl + 1 : sl;
                const int qq = min(len - 1, 2 * q);
                auto A = [&](int x, int y, int z) -> double { return (double)gf[x * len + (ns ? z : y)]; };
                const int qm = max(0, qq - 1), qp = min(len - 1, qq + 1);
                if (ns) g = fw_sum<T>(A, im, sl, ip, 0, 0, 0, qm, qq, qp);
                else g = fw_sum<T>(A, im, sl, ip, qm, qq, qp, 0, 0, 0);
            } else {
                g = gf[sl * len + 2 * q];
            }
            const int at = ns ? (upper ? (G.ny - 1) * F.rp : 0) + 2 * q : 2 * q * F.rp + (upper ? G.nz - 1 : 0);
            const T* up = sm + so_u + sl * F.pl + at;
            const int s = d * (ns ? F.rp : 1);
            g -= (c1 * up[0] + c2 * up[s] + c3 * up[2 * s]) / F.h;
            cl_put(C, sbase, C.so_g[fc], clen, I, q, g);
        }
    }
}

// residual of level l, restriction into f_{l+1}, u_{l+1} = 0, Neumann face restriction
template <typename T, bool JAC, bool BOUND>
__device__ __forceinline__ void cl_setup(const ClArgs<T>& a, int l, T* sm, unsigned sbase, unsigned cur, int rank,
                                         const ClCta<T>* S, ClXchg& X) {
    const ClLevel<T>& F = a.L[l];
    const ClLevel<T>& C = a.L[l + 1];
    const Geom& G = F.G;
    const int so_u = F.so_u[(cur >> l) & 1u];
    cl_residual(a, l, S[l], sm, so_u + F.pl, X);
    // Zeroing: a red-black neighbour may write into this CTA's halo in its first coarse sweep, so
    // the zeros are there before the barrier below; a Jacobi CTA far away may still be reading this
    // one's coarse planes for its last prolongation, so they wait until after the barrier.
    auto zero_coarse = [&]() {
        T* uc = sm + C.so_u[(cur >> (l + 1)) & 1u];
        const int n = (C.P + 2) * C.pl;
        for (int t = threadIdx.x; t < n; t += blockDim.x) uc[t] = T(0);
    };
    if (!JAC) zero_coarse();
    cl_face_restrict(a, l, sm, sbase, so_u, rank);
    cl_exchange<T, BOUND>(S[l], X);
    // the CTA that owns fine plane 2I restricts into coarse plane I
    const int i0 = S[l].i0, np = S[l].np;
    if (np > 0) {
        const int I0 = (i0 + 1) >> 1, I1 = (i0 + np + 1) >> 1;
        const T* r = sm + F.so_r;
        const int yz = C.G.ny * C.G.nz, n = (I1 - I0) * yz;
        for (int t = threadIdx.x; t < n; t += blockDim.x) {
            const int q = cl_div(t, C.m_yz), d = t - q * yz;
            const int I = I0 + q, J = cl_div(d, C.m_nz), K = d - J * C.G.nz;
            const int rem = J * C.rp + K;
            const int sl = 2 * I - i0 + 1;
            T v;
            if (a.fw) {
                const int im = (2 * I > 0 ? sl - 1 : sl) * F.pl, ic = sl * F.pl, ip = (2 * I < G.nx - 1 ? sl + 1 : sl) * F.pl;
                const int jj = min(G.ny - 1, 2 * J), kk = min(G.nz - 1, 2 * K);
                const int jm = max(0, jj - 1) * F.rp, jp = min(G.ny - 1, jj + 1) * F.rp;
                auto A = [&](int x, int y, int z) -> double { return (double)r[x + y + z]; };
                v = fw_sum<T>(A, im, ic, ip, jm, jj * F.rp, jp, max(0, kk - 1), kk, min(G.nz - 1, kk + 1));
            } else {
                v = r[sl * F.pl + 2 * J * F.rp + 2 * K];
            }
            const int owner = cl_div(I, C.m_P);
            cl_st(cl_map(sbase + (unsigned)(C.so_f + (I - owner * C.P) * C.pl + rem) * (unsigned)sizeof(T), owner), v);
        }
    }
    cl_sync_levels(F.nact, C.nact);
    if (JAC) {
        zero_coarse();
        __syncthreads();
    }
}

// u_l += P u_{l+1} on the slab and its halo planes (the neighbours form the same values there),
// r_l = P u_{l+1} at the unrelaxed points.  x, then y, then z midpoints, as prolong_tile.
template <typename T>
__device__ __forceinline__ void cl_prolong(const ClArgs<T>& a, int l, T* sm, unsigned sbase, unsigned cur, int rank) {
    const ClLevel<T>& F = a.L[l];
    const ClLevel<T>& C = a.L[l + 1];
    const int i0 = rank * F.P, nx = F.G.nx, np = min(F.P, nx - i0);
    T* sc = sm + a.so_gather;
    const int ia = max(0, i0 - 1), ib = min(nx, i0 + np + 1);           // planes written
    const int Ia = ia >> 1, Ib = min(C.G.nx - 1, ((ib - 1) >> 1) + 1);  // coarse planes read
    const int plc = C.pl, so_c = C.so_u[(cur >> (l + 1)) & 1u];
    cl_sync_levels(F.nact, C.nact);  // every CTA's last sweep of the coarse level
    if (np > 0) {
        const int n = (Ib - Ia + 1) * plc, Pc = C.P;
        const unsigned m_pl = C.m_pl, m_P = C.m_P;
        for (int t = threadIdx.x; t < n; t += blockDim.x) {
            const int q = cl_div(t, m_pl), rem = t - q * plc;
            const int I = Ia + q, owner = cl_div(I, m_P);
            T v;
            cl_ld(cl_map(sbase + (unsigned)(so_c + (I - owner * Pc + 1) * plc + rem) * (unsigned)sizeof(T), owner), v);
            sc[t] = v;
        }
    }
    __syncthreads();
    if (np > 0) {
        T* u = sm + F.so_u[(cur >> l) & 1u];
        T* r = sm + F.so_r;
        // an item is a pair of columns (k even, k+1): both interpolate between the same coarse rows
        const int pl = F.pl, rpf = F.rp, rpc = C.rp, ny = F.G.ny, nzc = C.G.nz;
        const int x0 = F.G.x0, x1 = F.G.x1, y0b = F.G.y0, y1b = F.G.y1, z0 = F.G.z0, z1 = F.G.z1;
        const int items = ny * nzc;  // nz = 2*nzc - 1: the last column of a row is alone
        const unsigned m_nzc = C.m_nz;
        const int nseg = max(1, (int)blockDim.x / items);
        const int seg = nseg > 1 ? (int)threadIdx.x / items : 0;
        const int step = nseg > 1 ? items : (int)blockDim.x;
        const int len = nseg > 1 ? (ib - ia + nseg - 1) / nseg : ib - ia;
        const int sa = ia + seg * len, sb = seg < nseg ? min(ib, sa + len) : sa;
        for (int it = (int)threadIdx.x - seg * items; it < items && sa < sb; it += step) {
            const int j = cl_div(it, m_nzc), kc = it - j * nzc, k = 2 * kc;
            const int jp = j & 1;
            const bool pair = kc + 1 < nzc;
            const bool jin = j >= y0b && j < y1b, in0 = jin && k >= z0 && k < z1, in1 = jin && k + 1 < z1;
            const T* c = sc + (j >> 1) * rpc + kc;
            const int dj = jp ? rpc : 0, dk = pair ? 1 : 0;  // what is not interpolated repeats a value (unused)
            T c0[2][2], c1[2][2];
            auto load = [&](T (&d)[2][2], int I) {
                const T* q = c + (I - Ia) * plc;
                d[0][0] = q[0];
                d[0][1] = q[dk];
                d[1][0] = q[dj];
                d[1][1] = q[dj + dk];
            };
            load(c0, sa >> 1);
            T* up = u + (sa - i0 + 1) * pl + j * rpf + k;
            T* rp = r + (sa - i0 + 1) * pl + j * rpf + k;
            for (int i = sa; i < sb; i++, up += pl, rp += pl) {
                T x[2][2];
                if (i & 1) {
                    load(c1, (i >> 1) + 1);
#pragma unroll
                    for (int y = 0; y < 2; y++)
#pragma unroll
                        for (int z = 0; z < 2; z++) {
                            x[y][z] = half_sum(c0[y][z], c1[y][z]);
                            c0[y][z] = c1[y][z];
                        }
                } else {
#pragma unroll
                    for (int y = 0; y < 2; y++)
#pragma unroll
                        for (int z = 0; z < 2; z++) x[y][z] = c0[y][z];
                }
                const T e0 = jp ? half_sum(x[0][0], x[1][0]) : x[0][0];
                const T e1 = jp ? half_sum(x[0][1], x[1][1]) : x[0][1];
                const bool xin = i >= x0 && i < x1;
                up[0] = up[0] + e0;
                if (!(xin && in0)) rp[0] = e0;
                if (pair) {
                    const T e = half_sum(e0, e1);
                    up[1] = up[1] + e;
                    if (!(xin && in1)) rp[1] = e;
                }
            }
        }
    }
}

// Slab copies between the pitched global arrays and shared memory.
// Loading is asynchronous (cp.async), so all arrays of all levels share one memory round trip.
// Coarser levels need only what the set-ups do not write before it is read: the other u buffer
// of a Jacobi pair and the stored r, both at unrelaxed points.
template <typename T>
__device__ __forceinline__ void cl_load(const ClArgs<T>& a, T* sm, int rank) {
    for (int l = 0; l < a.nl; l++) {
        const ClLevel<T>& L = a.L[l];
        const int nx = L.G.nx, ny = L.G.ny, nz = L.G.nz, pl = L.pl, i0 = rank * L.P, np = min(L.P, nx - i0);
        const int x0 = L.G.x0, x1 = L.G.x1, y0 = L.G.y0, y1 = L.G.y1, z0 = L.G.z0, z1 = L.G.z1;
        const long long sx = L.G.sx, sy = L.G.sy;
        const int rp = L.rp;
        const unsigned m_nz = L.m_nz, m_yz = L.m_yz;
        if (np <= 0) continue;
        const int ia = max(0, i0 - 1), ib = min(nx, i0 + np + 1);
        const int c = (a.cur >> l) & 1;
        const T* gu = L.ub[c];
        const T* gp = L.ub[1] ? L.ub[c ^ 1] : nullptr;
        const T* gf = L.f;
        const T* gr = L.r;
        T* su = sm + L.so_u[c];
        T* sp = sm + L.so_u[c ^ 1];
        T* sf = sm + L.so_f;
        T* sr = sm + L.so_r;
        const int yz = ny * nz, n = (ib - ia) * yz;
        for (int t = threadIdx.x; t < n; t += blockDim.x) {
            const int q = cl_div(t, m_yz), rem = t - q * yz;
            const int i = ia + q, j = cl_div(rem, m_nz), k = rem - j * nz;
            const int p = (i - i0 + 1) * pl + j * rp + k;
            const long long o = (long long)i * sx + j * sy + k;
            const bool unrelaxed = i < x0 || i >= x1 || j < y0 || j >= y1 || k < z0 || k >= z1;
            if (l == 0) {
                cl_copy(su + p, gu + o);
                if (i >= i0 && i < i0 + np) cl_copy(sf + p - pl, gf + o);
            }
            if (gp && (l == 0 || unrelaxed)) cl_copy(sp + p, gp + o);
            if (unrelaxed) cl_copy(sr + p, gr + o);
        }
        if (l > 0) continue;  // coarser faces are written by the set-ups
        for (int fc = 0; fc < 6; fc++) {
            if (!L.neumann[fc]) continue;
            T* sg = sm + L.so_g[fc];
            const T* gg = L.g[fc];
            if (fc == F_EAST || fc == F_WEST) {
                for (int t = threadIdx.x; t < ny * nz; t += blockDim.x) {
                    const int j = cl_div(t, L.m_nz);
                    cl_copy(sg + t + j * (rp - nz), gg + t);
                }
            } else {
                const int len = (fc == F_NORTH || fc == F_SOUTH) ? nz : ny;
                const int m = (ib - ia) * len;
                for (int t = threadIdx.x; t < m; t += blockDim.x) cl_copy(sg + (ia - i0 + 1) * len + t, gg + ia * len + t);
            }
        }
    }
    cp_async_commit();
    cp_async_wait<0>();
}

template <typename T>
__device__ __forceinline__ void cl_store(const ClArgs<T>& a, const T* sm, int rank) {
    for (int l = 0; l < a.nl; l++) {
        const ClLevel<T>& L = a.L[l];
        const int nx = L.G.nx, ny = L.G.ny, nz = L.G.nz, pl = L.pl, i0 = rank * L.P, np = min(L.P, nx - i0);
        const int x0 = L.G.x0, x1 = L.G.x1, y0 = L.G.y0, y1 = L.G.y1, z0 = L.G.z0, z1 = L.G.z1;
        const long long sx = L.G.sx, sy = L.G.sy;
        const int rp = L.rp;
        const unsigned m_nz = L.m_nz, m_yz = L.m_yz;
        if (np <= 0) continue;
        T* g0 = L.ub[0];
        T* g1 = L.ub[1];
        T* gf = L.f;
        T* gr = L.r;
        const T* s0 = sm + L.so_u[0];
        const T* s1 = sm + L.so_u[1];
        const T* sf = sm + L.so_f;
        const T* sr = sm + L.so_r;
        const int yz = ny * nz, n = np * yz;
        for (int t = threadIdx.x; t < n; t += blockDim.x) {
            const int q = cl_div(t, m_yz), rem = t - q * yz;
            const int i = i0 + q, j = cl_div(rem, m_nz), k = rem - j * nz;
            const int p = (q + 1) * pl + j * rp + k;
            const long long o = (long long)i * sx + j * sy + k;
            g0[o] = s0[p];
            if (g1) g1[o] = s1[p];
            if (i < x0 || i >= x1 || j < y0 || j >= y1 || k < z0 || k >= z1) gr[o] = sr[p];
            if (l > 0) gf[o] = sf[p - pl];
        }
        if (l == 0) continue;
        for (int fc = 0; fc < 6; fc++) {
            if (!L.neumann[fc]) continue;
            const T* sg = sm + L.so_g[fc];
            T* gg = L.g[fc];
            if (fc == F_EAST || fc == F_WEST) {
                if (rank != (fc == F_EAST ? L.nact - 1 : 0)) continue;
                for (int t = threadIdx.x; t < ny * nz; t += blockDim.x) gg[t] = sg[t + cl_div(t, L.m_nz) * (rp - nz)];
            } else {
                const int len = (fc == F_NORTH || fc == F_SOUTH) ? nz : ny;
                for (int t = threadIdx.x; t < np * len; t += blockDim.x) gg[i0 * len + t] = sg[len + t];
            }
        }
    }
}

// BOUND: the waits take their bound from the arguments, else the default one.
template <typename T, bool JAC, bool BOUND>
__global__ void __launch_bounds__(kClMaxThreads, 1) k_cluster(const __grid_constant__ ClArgs<T> args) {
    extern __shared__ __align__(16) unsigned char cl_smem[];
    __shared__ ClArgs<T> a;
    T* sm = reinterpret_cast<T*>(cl_smem);
    const unsigned sbase = (unsigned)__cvta_generic_to_shared(cl_smem);
    const int rank = (int)cl_rank();
    {
        const int* src = reinterpret_cast<const int*>(&args);
        int* dst = reinterpret_cast<int*>(&a);
        for (int w = threadIdx.x; w < (int)(sizeof(ClArgs<T>) / sizeof(int)); w += blockDim.x) dst[w] = src[w];
    }
    __shared__ ClCta<T> S[kClMaxLevels];
    __shared__ __align__(8) unsigned long long mbar[4];
    __shared__ ClWait wt;
    ClXchg X;
    X.mb = (unsigned)__cvta_generic_to_shared(mbar);
    X.n = X.phase = 0u;
    X.w = &wt;
    X.dead = false;
    if (threadIdx.x == 0) {
        wt.polls = args.polls;
        wt.dead = 0;
        for (int q = 0; q < 4; q++) cl_mbar_init(X.mb + 8 * q);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    cl_tables<T, JAC>(a, cl_smem, sbase, X.mb, S, rank);
    pdl_begin();
    cl_load(a, sm, rank);
    cl_sync();  // every CTA has started and filled its own slab before a neighbour writes into it
    unsigned cur = a.cur;
    int alt = a.alt;
    for (int q = 0; q < a.nops; q++) {
        const int l = a.lv[q], op = a.op[q];
        if (op == CL_RELAX || op == CL_RELAX_SKIP1) {
            cl_relax<T, JAC, BOUND>(a, l, S[l], sm, op == CL_RELAX_SKIP1, cur, alt, X);
        } else if (op == CL_SETUP) {
            cl_setup<T, JAC, BOUND>(a, l, sm, sbase, cur, rank, S, X);
        } else if (op == CL_PROLONG) {
            cl_prolong(a, l, sm, sbase, cur, rank);
            // Jacobi's next sweep only reads this CTA's u and writes the other buffer; an in-place
            // sweep of a neighbour would write halo points still being updated here
            if (JAC || a.L[l].nact == 1) __syncthreads();
            else cl_sync();
        } else {  // the solve loop's residual of level 0, stored, and its max-norm over the shape
            cl_residual(a, l, S[l], sm, S[l].u[(cur >> l) & 1u], X);
            cl_exchange<T, BOUND>(S[l], X);
            const ClLevel<T>& L = a.L[l];
            const int i0 = S[l].i0, np = S[l].np;
            const Geom& G = L.G;
            unsigned long long mx = 0ull;
            for (int rem = threadIdx.x; rem < L.pl; rem += blockDim.x) {
                const int j = cl_div(rem, L.m_rp), k = rem - j * L.rp;
                if (k >= G.nz) continue;
                for (int ii = 0; ii < np; ii++) {
                    const T v = sm[L.so_r + (ii + 1) * L.pl + rem];
                    mx = max(mx, abs_bits(v));
                    L.r[(long long)(i0 + ii) * G.sx + (long long)j * G.sy + k] = v;
                }
            }
            block_max_to(mx, a.norm);
        }
    }
    cl_store(a, sm, rank);
    cl_sync();  // no CTA leaves while a neighbour may still read or write its shared memory
    if (*(volatile int*)&wt.dead) {
        // the results are invalid, the host is told; planes sent that nobody waited for land (all
        // were sent before the barrier) before this CTA leaves
        if (threadIdx.x == 0) *a.err = kErrCluster;
        const long long t = clock64();
        while (clock64() - t < (1ll << 22)) {
        }
    }
}

}  // namespace mgp
