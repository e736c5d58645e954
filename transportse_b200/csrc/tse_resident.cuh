// Resident red-black solves: the pieces the FP32 correction form
// (tse_dc_resident.cuh) and the FP64 form (tse_rbsolve_res.cuh) share.
//
// A grid whose solver state fits on the chip (registers and shared memory of
// the SMs) needs no memory traffic during its iterations but the values on
// the tiles' edges.  The grid's (i, j) columns are cut into gx x gy tiles of
// whole columns, one thread block each, all co-resident (cooperative launch).
// A block keeps its cells' coefficients and both colours of the solution, with
// a ring of neighbour columns around them, for the whole solve.
//
// What bounds it: a half-sweep of such a grid is latency.  The staged sweeps
// pay a device-wide barrier, the restart of their copy pipelines and a
// release fence a half-sweep (about 3.6 us for any grid that fits in L2).
// Here tiles exchange only their edges, and without a barrier: each edge value
// goes to memory as one 8-byte word {value, tag} (two for a double), the tag
// counting half-sweeps, and the neighbour polls the word itself until its tag
// arrives -- one write and one read through L2, no fence, no flag, and no tile
// waits for any tile but its neighbours (the flag-in-word exchange that NCCL's
// LL protocol uses).  A word is overwritten only after its reader is done with
// it: a tile writes colour c again only after it has read its neighbours' next
// values of the other colour, which they write after reading c.
//
// Every wait is bounded: a poll that runs out of time raises the launch's
// error flag, which ends every other poll.  A block whose wait ran out leaves
// without storing its part of the result while its neighbours may go on to a
// good end, so the last block to leave says whether the solve is good
// (res_last).
#pragma once

#include "tse_common.cuh"

namespace tse {

// Cells are held in groups of 16 bytes along a column (four floats or two
// doubles of one colour), so a thread loads, relaxes and stores a group with
// vector accesses; a column of H cells per colour is Hg groups, the last one
// filled up with cells whose coefficients are zero.
//
// Tiling of a resident solve: tile (bi, bj) = block bi * gy + bj holds the
// columns [bi nx / gx, (bi + 1) nx / gx) x [bj ny / gy, (bj + 1) ny / gy).
struct ResPlan {
    int gx, gy, nb;
    int ti, tj;       // the largest tile, in columns
    int pitch;        // columns of a padded tile row (tj + 2)
    int Hg;           // groups of a column and colour
    int groups;       // groups per colour of the largest tile
    int pad;          // padded groups per colour: (ti + 2) pitch Hg + 2
    int halo;         // most edge groups a tile reads per half-sweep
    int smem;         // dynamic shared memory
};

// Blocks of one resident launch at most, and their threads at most.
constexpr int kResMaxBlocks = 256;
constexpr int kResMaxThreads = 512;

// A plan for the layout (vals cells a group) on at most maxb blocks, at most
// max_groups groups per colour and tile, dynamic shared memory smem(plan) <=
// smem_max.  The plan with the smallest largest tile, edges weighed against
// cells; one block when one_first and everything fits in it, since a
// half-sweep of one block exchanges nothing.
template <class SmemFn, class ThreadsFn>
inline bool res_plan(const Layout& L, int vals, int maxb, int max_groups, int smem_max, SmemFn smem,
                     ThreadsFn threads, bool one_first, ResPlan& best) {
    double best_cost = 0.0;
    bool found = false;
    const int Hg = (L.H + vals - 1) / vals;
    for (int gx0 = 1; gx0 <= L.nx && gx0 <= maxb; ++gx0) {
        const int ti = (L.nx + gx0 - 1) / gx0, gx = (L.nx + ti - 1) / ti;
        const int cap = maxb / gx;
        const int gy0 = L.ny < cap ? L.ny : cap;
        for (int one = 0; one < 2; ++one) {
            const int gyt = one ? 1 : gy0;
            const int tj = (L.ny + gyt - 1) / gyt, gy = (L.ny + tj - 1) / tj;
            ResPlan P;
            P.gx = gx;
            P.gy = gy;
            P.nb = gx * gy;
            P.ti = ti;
            P.tj = tj;
            P.pitch = tj + 2;
            P.Hg = Hg;
            const long long pad = (long long)(ti + 2) * P.pitch * Hg + 2;
            const long long groups = (long long)ti * tj * Hg;
            if (groups > max_groups || pad > 65535 || ti > 250) continue;
            P.groups = (int)groups;
            P.pad = (int)pad;
            P.halo = ((gx > 1 ? 2 * tj : 0) + (gy > 1 ? 2 * ti : 0)) * Hg;
            P.smem = smem(P);
            if (P.smem > smem_max) continue;
            // a second round of polling costs about what 250 groups' sweep does
            const double cost =
                P.nb == 1 && one_first ? -1.0 : (double)groups + 0.5 * P.halo + (P.halo > threads(P) ? 250.0 : 0.0);
            if (!found || cost < best_cost) {
                best = P;
                best_cost = cost;
                found = true;
            }
        }
    }
    return found;
}

// A block's tile.  Groups of a colour are numbered u = 0 .. groups - 1, columns
// on the tile's edge first, so that their new values leave before the inside
// is computed; column(ci, cj) is the grid column, p a group's place in the
// padded shared-memory arrays (one guard group at either end).
struct ResTile {
    int i0, j0, ti, tj, Hg, ny, pitch, groups;

    __device__ __forceinline__ void init(const Layout& L, const ResPlan& P, int b) {
        const int bi = b / P.gy, bj = b - bi * P.gy;
        i0 = (int)((long long)bi * L.nx / P.gx);
        ti = (int)((long long)(bi + 1) * L.nx / P.gx) - i0;
        j0 = (int)((long long)bj * L.ny / P.gy);
        tj = (int)((long long)(bj + 1) * L.ny / P.gy) - j0;
        Hg = P.Hg;
        ny = L.ny;
        pitch = P.pitch;
        groups = ti * tj * Hg;
    }
    __device__ __forceinline__ void decode(int u, int& ci, int& cj, int& g) const {
        int o = u / Hg;
        g = u - o * Hg;
        if (o < tj) { ci = 0; cj = o; return; }
        o -= tj;
        if (o < tj) { ci = ti - 1; cj = o; return; }   // reached only when ti > 1
        o -= tj;
        const int mid = ti - 2;
        if (o < mid) { ci = 1 + o; cj = 0; return; }
        o -= mid;
        if (o < mid) { ci = 1 + o; cj = tj - 1; return; }   // only when tj > 1
        o -= mid;
        const int w = tj - 2;
        ci = 1 + o / w;
        cj = 1 + (o - (ci - 1) * w);
    }
    __device__ __forceinline__ int column(int ci, int cj) const { return (i0 + ci) * ny + j0 + cj; }
    __device__ __forceinline__ int p(int ci, int cj, int g) const {
        return ((ci + 1) * pitch + cj + 1) * Hg + g + 1;
    }
    // a group's record among the exchange records (column(ci, cj) Hg + g) is
    // p + ci * rec_row() + rec_base()
    __device__ __forceinline__ int rec_row() const { return (ny - pitch) * Hg; }
    __device__ __forceinline__ int rec_base() const { return column(0, 0) * Hg - (pitch + 1) * Hg - 1; }
    // edge group h of the tile's surroundings: its record and padded place;
    // the sides that exist in the order x-, x+, y-, y+
    __device__ __forceinline__ int halo_groups(int nx) const {
        int n = 0;
        if (i0 > 0) n += tj * Hg;
        if (i0 + ti < nx) n += tj * Hg;
        if (j0 > 0) n += ti * Hg;
        if (j0 + tj < ny) n += ti * Hg;
        return n;
    }
    __device__ __forceinline__ void halo(int h, int nx, int& rec, int& pp) const {
        const int row = tj * Hg, col = ti * Hg;
        if (i0 > 0) {
            if (h < row) { rec = column(-1, 0) * Hg + h; pp = p(-1, 0, h); return; }
            h -= row;
        }
        if (i0 + ti < nx) {
            if (h < row) { rec = column(ti, 0) * Hg + h; pp = p(ti, 0, h); return; }
            h -= row;
        }
        int cj = -1;
        if (j0 == 0 || h >= col) {
            if (j0 > 0) h -= col;
            cj = tj;
        }
        const int ci = h / Hg, g = h - ci * Hg;
        rec = column(ci, cj) * Hg + g;
        pp = p(ci, cj, g);
    }
};

// A group's word in a thread's registers (or in shared memory): padded place
// (16 bits), (i + j) & 1 (bit 16), in use (bit 17), the sides on which another
// tile reads it (bits 18-21: x-, x+, y-, y+), tile row ci (bits 24 up).
enum : unsigned {
    RS_PAR = 1u << 16, RS_USED = 1u << 17, RS_XM = 1u << 18, RS_XP = 1u << 19, RS_YM = 1u << 20,
    RS_YP = 1u << 21, RS_SHARED = RS_XM | RS_XP | RS_YM | RS_YP
};

__device__ __forceinline__ unsigned res_group_word(const ResTile& T, int u, int nx, bool exchange) {
    if (u >= T.groups) return 0u;
    int ci, cj, g;
    T.decode(u, ci, cj, g);
    unsigned f = (unsigned)T.p(ci, cj, g) | RS_USED | ((unsigned)ci << 24);
    if ((T.i0 + ci + T.j0 + cj) & 1) f |= RS_PAR;
    if (exchange) {
        if (ci == 0 && T.i0 > 0) f |= RS_XM;
        if (ci == T.ti - 1 && T.i0 + T.ti < nx) f |= RS_XP;
        if (cj == 0 && T.j0 > 0) f |= RS_YM;
        if (cj == T.tj - 1 && T.j0 + T.tj < T.ny) f |= RS_YP;
    }
    return f;
}

// --------------------------------------------------------- tagged exchange
// An exchange record: a group's 16 bytes as four 8-byte words {32 bits of the
// group, tag}, each written and read whole.  The first two words of all
// records lie together and the last two `plane` words further on, so a warp's
// 16-byte stores and loads are contiguous.
__device__ __forceinline__ uint64_t ld_word(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(uint64_t* p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void ld_words2(const uint64_t* p, uint64_t& a, uint64_t& b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_words2(uint64_t* p, uint64_t a, uint64_t b) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ uint64_t tagged(unsigned v, unsigned tag) {
    return ((uint64_t)tag << 32) | v;
}
__device__ __forceinline__ void res_publish(uint64_t* recs, int plane, int rec, unsigned a, unsigned b,
                                            unsigned c, unsigned d, unsigned tag) {
    uint64_t* r = recs + 2 * rec;
    st_words2(r, tagged(a, tag), tagged(b, tag));
    st_words2(r + plane, tagged(c, tag), tagged(d, tag));
}

// Bounded polling: every 256th try looks at the launch's error flag, the
// block's own and the time.
struct ResWait {
    GridBarrier* bar;
    volatile int* err;
    unsigned tries;
    uint64_t t0;
    unsigned long long timeout_ns;
    __device__ __forceinline__ bool go_on() {
        if ((++tries & 255u) != 0u) return true;
        const uint64_t now = globaltimer();
        if (tries == 256u) t0 = now;
        if (*err || *(volatile int*)&bar->error || now - t0 > timeout_ns) {
            *err = 1;
            atomicExch(&bar->error, 1);
            return false;
        }
        return true;
    }
};

// The tile's edge groups with tag `tag` into the ring of the padded array s.
// (Two groups in flight a thread: 10 % slower for tiles of at most NT edge
// groups, 5 % faster above; plans with more are avoided instead.)
template <int NT>
__device__ __forceinline__ void res_poll(const uint64_t* recs, int plane, unsigned tag, uint4* s,
                                         const int* hrec, const unsigned short* hp, int nh, GridBarrier* bar,
                                         volatile int* err,
                                         unsigned long long timeout_ns = kBarrierTimeoutNs) {
    for (int h = threadIdx.x; h < nh; h += NT) {
        const uint64_t* r = recs + 2 * hrec[h];
        uint64_t a, b, c, d;
        ResWait wt = {bar, err, 0u, 0, timeout_ns};
        for (;;) {
            ld_words2(r, a, b);
            ld_words2(r + plane, c, d);
            if ((unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag && (unsigned)(c >> 32) == tag &&
                (unsigned)(d >> 32) == tag)
                break;
            if (!wt.go_on()) break;
        }
        s[hp[h]] = make_uint4((unsigned)a, (unsigned)b, (unsigned)c, (unsigned)d);
    }
}

// How the tiles of a launch exchange edges and sums: through tagged records
// in memory (any co-resident blocks), or, when the launch is one thread-block
// cluster, by writing into each other's shared memory with the hardware
// cluster barrier between half-sweeps.
enum ResMode { RES_GRID = 0, RES_CLUSTER = 1 };

// cluster barrier, also a block barrier: orders shared (own and peers') and
// global accesses of all the cluster's threads
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of `p` (this block's shared memory) in block `rank` of the cluster
__device__ __forceinline__ unsigned peer_smem(const void* p, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;"
        : "=r"(r)
        : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_peer(unsigned addr, unsigned a, unsigned b, unsigned c, unsigned d) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c),
                 "r"(d)
                 : "memory");
}

// The four neighbours of a tile in a cluster launch: the shared-memory
// distance (bytes) from a group's own address to its place in that
// neighbour's ring, cluster addresses (the peers' windows differ by a constant)
struct ResPeers {
    unsigned xm, xp, ym, yp;
    __device__ __forceinline__ void init(const ResTile& T, const Layout& L, const ResPlan& P, int b,
                                         const void* smem) {
        const unsigned own = (unsigned)__cvta_generic_to_shared(smem);
        const int bi = b / P.gy, bj = b - bi * P.gy;
        xm = xp = ym = yp = 0u;
        // p(ti', cj, g) of the tile before, p(-1, cj, g) of the tile after
        if (bi > 0) {
            const int tn = T.i0 - (int)((long long)(bi - 1) * L.nx / P.gx);
            xm = peer_smem(smem, (unsigned)(b - P.gy)) - own + 16u * (unsigned)(tn * T.pitch * T.Hg);
        }
        if (bi + 1 < P.gx) xp = peer_smem(smem, (unsigned)(b + P.gy)) - own - 16u * (unsigned)(T.ti * T.pitch * T.Hg);
        if (bj > 0) {
            const int tn = T.j0 - (int)((long long)(bj - 1) * L.ny / P.gy);
            ym = peer_smem(smem, (unsigned)(b - 1)) - own + 16u * (unsigned)(tn * T.Hg);
        }
        if (bj + 1 < P.gy) yp = peer_smem(smem, (unsigned)(b + 1)) - own - 16u * (unsigned)(T.tj * T.Hg);
    }
    // a group's new value (at shared address `at`) into the rings it is read from
    __device__ __forceinline__ void publish(unsigned f, const void* at, unsigned a, unsigned b, unsigned c,
                                            unsigned d) const {
        const unsigned own = (unsigned)__cvta_generic_to_shared(at);
        if (f & RS_XM) st_peer(own + xm, a, b, c, d);
        if (f & RS_XP) st_peer(own + xp, a, b, c, d);
        if (f & RS_YM) st_peer(own + ym, a, b, c, d);
        if (f & RS_YP) st_peer(own + yp, a, b, c, d);
    }
};

// Sums of two values over all threads of all blocks, the same bits in every
// thread: warps and blocks in a fixed order.  Memory form: every block writes
// one record, block 0 polls and adds them and writes the totals back as
// kResCopies records, which the other blocks poll (all blocks polling all
// records kept the memory's few hot sectors so busy that a sum took 7 us at
// 148 blocks).  Two sets of records alternate with `count`, tagged with count
// + 1.  Contains block barriers; a caller has one between two calls.  False, in
// all of a block's threads, when a wait of this block ran out here or before.
constexpr int kResCopies = 8;
constexpr int kResSetWords = kResMaxBlocks * 4 + kResCopies * 16;   // copies on lines of their own
struct ResSumShared {
    double a[kResMaxThreads / 32], b[kResMaxThreads / 32];
    double total[2];
    double2 peers[2][16];   // cluster form: the blocks' sums, two sets
};

__device__ __forceinline__ bool res_poll_pair(const uint64_t* s, unsigned tag, double& A, double& B,
                                              GridBarrier* bar, volatile int* err,
                                              unsigned long long timeout_ns = kBarrierTimeoutNs) {
    ResWait wt = {bar, err, 0u, 0, timeout_ns};
    uint64_t v0, v1, v2, v3;
    for (;;) {
        ld_words2(s, v0, v1);
        ld_words2(s + 2, v2, v3);
        if ((unsigned)(v0 >> 32) == tag && (unsigned)(v1 >> 32) == tag && (unsigned)(v2 >> 32) == tag &&
            (unsigned)(v3 >> 32) == tag)
            break;
        if (!wt.go_on()) return false;
    }
    A = __longlong_as_double((long long)((v0 & 0xffffffffu) | (v1 << 32)));
    B = __longlong_as_double((long long)((v2 & 0xffffffffu) | (v3 << 32)));
    return true;
}
__device__ __forceinline__ void res_write_pair(uint64_t* s, unsigned tag, double A, double B) {
    const uint64_t x = __double_as_longlong(A), y = __double_as_longlong(B);
    st_words2(s, tagged((unsigned)x, tag), tagged((unsigned)(x >> 32), tag));
    st_words2(s + 2, tagged((unsigned)y, tag), tagged((unsigned)(y >> 32), tag));
}

template <int NT, int MODE>
__device__ __forceinline__ bool res_team_sum(double& va, double& vb, ResSumShared& sh, uint64_t* slots,
                                             unsigned nb, unsigned b, unsigned count, GridBarrier* bar,
                                             volatile int* err,
                                             unsigned long long timeout_ns = kBarrierTimeoutNs) {
    constexpr int NW = NT / 32;
    static_assert(NT <= kResMaxThreads && NT >= kResMaxBlocks && NW <= 32, "one polling thread a block");
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        va = va + __shfl_down_sync(0xffffffffu, va, o);
        vb = vb + __shfl_down_sync(0xffffffffu, vb, o);
    }
    if (lane == 0) {
        sh.a[w] = va;
        sh.b[w] = vb;
    }
    __syncthreads();
    if (MODE == RES_GRID && nb == 1) {
        va = 0.0;
        vb = 0.0;
        for (int q = 0; q < NW; ++q) {
            va = va + sh.a[q];
            vb = vb + sh.b[q];
        }
        return true;
    }
    double A = 0.0, B = 0.0;
    if (w == 0) {
        A = lane < NW ? sh.a[lane] : 0.0;
        B = lane < NW ? sh.b[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            A = A + __shfl_down_sync(0xffffffffu, A, o);
            B = B + __shfl_down_sync(0xffffffffu, B, o);
        }
    }
    if (MODE == RES_CLUSTER) {
        if (w == 0) {
            A = __shfl_sync(0xffffffffu, A, 0);
            B = __shfl_sync(0xffffffffu, B, 0);
            if (lane < (int)nb) {
                const uint64_t x = __double_as_longlong(A), y = __double_as_longlong(B);
                st_peer(peer_smem(&sh.peers[count & 1u][b], (unsigned)lane), (unsigned)x,
                        (unsigned)(x >> 32), (unsigned)y, (unsigned)(y >> 32));
            }
        }
        cluster_sync();
        va = 0.0;
        vb = 0.0;
        for (unsigned q = 0; q < nb; ++q) {
            va = va + sh.peers[count & 1u][q].x;
            vb = vb + sh.peers[count & 1u][q].y;
        }
        return true;
    }
    uint64_t* set = slots + (size_t)(count & 1u) * kResSetWords;
    uint64_t* copies = set + kResMaxBlocks * 4;
    const unsigned tag = count + 1u;
    if (b != 0) {
        if (threadIdx.x == 0) {
            res_write_pair(set + 4 * b, tag, A, B);
            res_poll_pair(copies + 16 * (b % kResCopies), tag, A, B, bar, err, timeout_ns);
            sh.total[0] = A;
            sh.total[1] = B;
        }
    } else {
        // warps in order, a block a lane; this block's own sum is lane 0's
        __syncthreads();   // sh.a, sh.b read above
        const unsigned q = threadIdx.x;
        double x = 0.0, y = 0.0;
        if (q == 0) {
            x = A;
            y = B;
        } else if (q < nb) {
            res_poll_pair(set + 4 * q, tag, x, y, bar, err, timeout_ns);
        }
        if ((q & ~31u) < nb) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                x = x + __shfl_down_sync(0xffffffffu, x, o);
                y = y + __shfl_down_sync(0xffffffffu, y, o);
            }
            if (lane == 0) {
                sh.a[w] = x;
                sh.b[w] = y;
            }
        }
        __syncthreads();
        if (w == 0) {
            double ta = 0.0, tb = 0.0;
            for (unsigned k = 0; k * 32 < nb; ++k) {
                ta = ta + sh.a[k];
                tb = tb + sh.b[k];
            }
            if (lane < kResCopies) res_write_pair(copies + 16 * lane, tag, ta, tb);
            if (lane == 0) {
                sh.total[0] = ta;
                sh.total[1] = tb;
            }
        }
    }
    const bool ok = __syncthreads_and(*err == 0);   // the same for all threads
    va = sh.total[0];
    vb = sh.total[1];
    return ok;
}

// The end of a launch's solve: every block comes here last, with `failed` if a
// wait of its own ran out.  True in one thread of the launch, thread 0 of the
// last block to come, with `failed` then if any block's did: it writes the
// status.  No wait: the blocks count themselves.  (A barrier there slowed the
// solves' loops by 1 %, by the registers' allocation.)
template <int MODE>
__device__ __forceinline__ bool res_last(unsigned* counter, unsigned nb, unsigned b, bool& failed) {
    if (threadIdx.x != 0) return false;
    if (MODE == RES_CLUSTER || nb == 1) return b == 0;
    return last_out(counter, nb, failed);
}

// A launch's exchange memory: two counters, the sum slots, and per colour one
// record a group.
constexpr size_t kResSlotBytes = (size_t)2 * kResSetWords * sizeof(uint64_t);
struct ResMem {
    unsigned* counter;   // count_sync's
    unsigned* leavers;   // res_last's
    uint64_t* slots;
    uint64_t* recs[2];
    int plane;
};
inline size_t res_mem_bytes(const Layout& L, int vals) {
    const size_t groups = (size_t)L.nx * L.ny * ((L.H + vals - 1) / vals);
    return 256 + kResSlotBytes + 2 * groups * 32;
}
inline ResMem res_mem(void* at, const Layout& L, int vals) {
    const size_t groups = (size_t)L.nx * L.ny * ((L.H + vals - 1) / vals);
    ResMem m;
    m.counter = (unsigned*)at;
    m.leavers = m.counter + 32;
    m.slots = (uint64_t*)((char*)at + 256);
    m.recs[0] = (uint64_t*)((char*)at + 256 + kResSlotBytes);
    m.recs[1] = m.recs[0] + 4 * groups;
    m.plane = (int)(2 * groups);
    return m;
}

// Can this plan run: `fn` co-resident, or as one cluster?
inline bool res_can_launch(const void* fn, const ResPlan& P, int threads, int room, bool cluster) {
    int per_sm = 0;
    bool ok = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, room) == cudaSuccess;
    if (cluster) {
        int n = 0;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        cfg.gridDim = dim3((unsigned)P.nb);
        cfg.blockDim = dim3((unsigned)threads);
        cfg.dynamicSmemBytes = (size_t)P.smem;
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)P.nb;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        ok = ok && cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
             cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n > 0;
    } else {
        ok = ok &&
             cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, (size_t)P.smem) == cudaSuccess &&
             per_sm > 0;
    }
    if (!ok) cudaGetLastError();
    return ok;
}

inline bool res_launch(const void* fn, const ResPlan& P, int threads, bool cluster, void** args,
                       cudaStream_t stream) {
    if (!cluster)
        return cudaLaunchCooperativeKernel(fn, dim3((unsigned)P.nb), dim3((unsigned)threads), args,
                                           (size_t)P.smem, stream) == cudaSuccess;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cfg.gridDim = dim3((unsigned)P.nb);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)P.smem;
    cfg.stream = stream;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)P.nb;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, args) == cudaSuccess;
}

}  // namespace tse
