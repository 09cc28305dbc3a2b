// The cell loop with four lanes per cell, plain mode (included by cells.cu).
//
// What bounds the loop while every cell can hold a place at once is the
// dependency chain: the DAG's depth times one link, i.e. detecting the
// dependency, the update's own serial program, and publishing.  With a lane
// per cell a link took 8-9 us: one warp issues an update's instructions about
// five cycles apart, the IEEE divisions one after another, and a warp of 32
// cells that become ready at different times runs its passes one after
// another.  Here a cell has four lanes, and what a link need not do is left
// out of it:
//   - lane p < 3 gathers, averages and scatters species 4p..4p+3 (one 16-byte
//     load and store per face);
//   - the rounds in which transporters and effectors may run side by side, the
//     first secretions, the maintenance factors and the list of reactions that
//     run are worked out while the cell waits for its dependencies;
//   - a reaction's substrate, catalyst and cofactor terms are divided by three
//     lanes at once and exchanged by shuffles;
//   - dependencies are polled with acquire loads, one or two per lane, so no
//     fence follows the last of them.
// A warp holds 8 cells, so a pass that runs for one of them delays 7 others
// instead of 31.
//
// The result is the lane-per-cell loop's bit for bit: each operation that can
// change a value is the same IEEE operation on the same operands in the same
// order.  What is left out changes nothing as long as the cell's values are
// ordinary (see quad_plan); a cell with any other value runs quad_serial.

constexpr int kQuadThreads = 128;
constexpr int kQuadCells = kQuadThreads / 4;
// Blocks per SM the register budget allows: 80 registers.  With 7 blocks (72)
// the update spills, which cost 210 against 200 us at 38k cells, and with 8
// (64) 252: the polls' acquire loads invalidate L1, so a spilled value comes
// back from L2.
constexpr int kQuadBlocksPerSM = 6;

// Where a cell's update reads and writes: its run's arrays.  A single run's are
// the kernel's parameters; a batch's cells carry theirs, because the
// descriptors in global memory would be read from L2 at every poll (the polls'
// acquire loads invalidate L1).
struct QuadAt {
    float* field;
    const float* light;
    uint32_t* done;
    float* internal;
    uint32_t* age;
    uint32_t* state;
    uint8_t* events;
    uint32_t cap, epoch;
    int X, Y;
    uint32_t j;  // index in its run
};
__device__ __forceinline__ QuadAt quad_at(const CellTable& t, const Grid& g, float* field, const float* light,
                                          uint32_t epoch, uint32_t j) {
    return QuadAt{field, light, t.done, t.internal, t.age, t.state, t.events, t.cap, epoch, g.X, g.Y, j};
}

// The same, member by member where it is used, so that nothing of it stays in
// registers meanwhile.
struct QuadOfLaunch {  // a single run's
    const CellLaunch& a;
    uint32_t j_;
    __device__ float* field() const { return a.field; }
    __device__ const float* light() const { return a.light; }
    __device__ uint32_t* done() const { return a.t.done; }
    __device__ uint32_t epoch() const { return a.epoch; }
    __device__ int X() const { return a.g.X; }
    __device__ int Y() const { return a.g.Y; }
    __device__ uint32_t j() const { return j_; }
    __device__ QuadAt all() const { return quad_at(a.t, a.g, a.field, a.light, a.epoch, j_); }
};
struct QuadOfCell {  // a batch's, from the staged record
    const QuadAt& r;
    __device__ float* field() const { return r.field; }
    __device__ const float* light() const { return r.light; }
    __device__ uint32_t* done() const { return r.done; }
    __device__ uint32_t epoch() const { return r.epoch; }
    __device__ int X() const { return r.X; }
    __device__ int Y() const { return r.Y; }
    __device__ uint32_t j() const { return r.j; }
    __device__ QuadAt all() const { return r; }
};

// One staged cell: the copy of its table entries, then what its group derives
// from them before the cell is ready.  784 bytes = 49 x 16: an odd number of
// 16-byte pieces, so the same member of a warp's 8 cells lies in different
// banks.
struct __align__(16) QuadCell {
    uint4 rx[MARL_R_MAX];  // the plan moves the reactions that run to the front, in order
    float2 tp[MARL_S_TRANSPORTERS];
    float2 ef[MARL_S_EFFECTORS];
    uint4 idx[2];  // transporter pairs (ext | int << 8), effector pairs (int | ext << 8)
    float4 fate;
    float x[MARL_M_INT + 2];  // x[16] is 0, read for "no cofactor"; x[17] is written by lanes that store nothing
    float keep, cost;   // maintenance: energy = max(energy * keep - cost, 0)
    float ext[MARL_S_EXT];
    float del[MARL_S_EXT];
    uint32_t pos, state, age, nb;
    int32_t dep[6];  // dependencies by face; after the plan the different ones, then -1
    uint32_t info;  // reactions that run | transporter rounds << 8 | effector rounds << 16 | flags
    uint32_t rounds[4];  // lane p's slots, a byte each: transporters p, p + 4, effectors p, p + 4 (kQuadOut: left out)
    uint32_t vox;  // the cell's voxel
    float2 secretion[4];  // lane p's transporters' secretion where their round is 0: nothing changes their species before
    QuadAt at;  // batch only
};
static_assert(sizeof(QuadCell) == 784, "49 pieces of 16 bytes");
constexpr int kQuadSmem = kQuadCells * (int)sizeof(QuadCell);
constexpr uint32_t kQuadOut = 0xFFu;
constexpr int kQuadZero = MARL_M_INT, kQuadTrash = MARL_M_INT + 1;  // indices into x

constexpr uint32_t kQuadPlain = 1u << 24;     // the rounds and the parallel reactions apply (see quad_plan)
constexpr uint32_t kQuadCofactor = 1u << 25;  // a running reaction has a cofactor

// Bounds within which products of rates and values cannot overflow.
constexpr float kQuadRateMax = 1e30f, kQuadValueMax = 1e6f;

__device__ __forceinline__ uint32_t pair_of(const uint4& w, int i) {
    const uint32_t q = (i >> 1) == 0 ? w.x : ((i >> 1) == 1 ? w.y : ((i >> 1) == 2 ? w.z : w.w));
    return (q >> ((i & 1) * 16)) & 0xFFFFu;
}
// Pair p + 4 i for a lane's p.
__device__ __forceinline__ uint32_t own_pair(const uint4& w, int p, int i) {
    const uint32_t lo = i ? w.z : w.x, hi = i ? w.w : w.y;
    return ((p & 2 ? hi : lo) >> ((p & 1) * 16)) & 0xFFFFu;
}

// The group's nibble of a ballot of the whole warp.
__device__ __forceinline__ uint32_t group_ballot(bool b) {
    return (__ballot_sync(0xFFFFFFFFu, b) >> (threadIdx.x & 28)) & 0xFu;
}

// a / b, IEEE round-to-nearest, for a >= +0 and b > 0: div_rn without its
// cases of sign and zero or NaN divisors.
__device__ __forceinline__ float div_pos(float a, float b) {
    const bool zero = a == 0.0f;
    float num;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\tselp.f32 %0, %1, %2, p;\n\t}"
        : "=f"(num)
        : "f"(1.5f), "f"(a), "r"((unsigned)zero));
    const float q = num / b;
    return zero ? 0.0f : q;
}

// The four values' quotients by n = 1..6 (n = 0: unchanged zeros).  For a power
// of two c = 1/n is exact, the remainder r is exact, and q0 + r c is x / n
// exactly before its one rounding; for 3, 5 and 6 as div_small_n, with the
// IEEE operator where that needs it.
__device__ __forceinline__ void quad_divide(float (&v)[4], int n) {
    const float nf = (float)(n > 0 ? n : 1);
    const float c = n == 2 ? 0.5f : (n == 4 ? 0.25f : (n < 2 ? 1.0f : small_divisor_inverse(n)));
    bool bad = false;
    float q[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const uint32_t u = __float_as_uint(v[s]) & 0x7FFFFFFFu;
        bad = bad || u - 1u < 0x00FFFFFFu || u > 0x7F7FFFFFu;  // not 0, below 2^-125; not finite
        q[s] = div_small_n(v[s], c, nf);
    }
    if (bad) {
#pragma unroll
        for (int s = 0; s < 4; ++s) q[s] = div_rn(v[s], nf);
    }
#pragma unroll
    for (int s = 0; s < 4; ++s) v[s] = q[s];
}

// Copies cell j's record into C, a quarter of it per lane (one commit group);
// with schedule_here lane p also computes the schedule of faces p and p + 4.
// All four lanes of the group take part.
__device__ __forceinline__ void quad_stage(const CellRunView& v, QuadCell& C, uint32_t j, int p, bool schedule_here) {
    const CellTable& t = *v.t;
    const size_t cap = t.cap;
#pragma unroll
    for (int i = 0; i < MARL_R_MAX / 4; ++i) cp_async16(&C.rx[p + 4 * i], &t.rx[(p + 4 * i) * cap + j]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        cp_async8(&C.tp[p + 4 * i], &t.tp_rate[(p + 4 * i) * cap + j]);
        cp_async8(&C.ef[p + 4 * i], &t.ef_par[(p + 4 * i) * cap + j]);
    }
#pragma unroll
    for (int i = 0; i < MARL_M_INT / 4; ++i) cp_async4(&C.x[p + 4 * i], &t.internal[(p + 4 * i) * cap + j]);
    if (p == 0) {
        cp_async16(&C.idx[0], &t.tp_idx[j]);
        cp_async4(&C.pos, &t.pos[j]);
    } else if (p == 1) {
        cp_async16(&C.idx[1], &t.ef_idx[j]);
        cp_async4(&C.state, &t.state[j]);
    } else if (p == 2) {
        cp_async16(&C.fate, &t.fate[j]);
        cp_async4(&C.age, &t.age[j]);
    }
    if (schedule_here) {
        const uint32_t P = t.pos[j];
        const Grid g = v.g;
        uint32_t nb = 0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int f = p + 4 * i;
            if (f >= 6) break;
            const int s = (f & 1) ? -1 : 1;
            const int nx = pos_x(P) + (f < 2 ? s : 0), ny = pos_y(P) + ((f >> 1) == 1 ? s : 0),
                      nz = pos_z(P) + (f >= 4 ? s : 0);
            int dep = -1;
            if (nx >= 0 && nx < g.X && ny >= 0 && ny < g.Y && nz >= 0 && nz < g.Z &&
                v.cmap[((size_t)nz * g.Y + ny) * g.X + nx] < 0) {
                nb |= 1u << f;
#pragma unroll
                for (int h = 0; h < 6; ++h) {
                    const int ux = nx + c_face[h][0], uy = ny + c_face[h][1], uz = nz + c_face[h][2];
                    if (ux >= 0 && ux < g.X && uy >= 0 && uy < g.Y && uz >= 0 && uz < g.Z) {
                        const int32_t q = v.cmap[((size_t)uz * g.Y + uy) * g.X + ux];
                        if (q >= 0 && (uint32_t)q < j && q > dep) dep = q;
                    }
                }
            }
            C.dep[f] = dep;
        }
        const unsigned gmask = 0xFu << (threadIdx.x & 28);
        nb |= __shfl_xor_sync(gmask, nb, 1);
        nb |= __shfl_xor_sync(gmask, nb, 2);
        if (p == 3) C.nb = nb;
    } else {
        if (p == 3) cp_async4(&C.nb, &t.nb[j]);
        cp_async4(&C.dep[p], &t.dep[(size_t)p * cap + j]);
        if (p < 2) cp_async4(&C.dep[p + 4], &t.dep[(size_t)(p + 4) * cap + j]);
    }
    cp_async_commit();
}

// Rounds of eight slots with species pairs w, of which `part` take part: a
// slot's round comes after those of every earlier slot it shares a species
// with.  Returns the number of rounds; own[i] is slot p + 4i's round.  The
// whole warp takes part.
__device__ __forceinline__ uint32_t quad_rounds(const uint4& w, uint32_t part, int p, uint32_t (&own)[2]) {
    uint32_t before[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int s = p + 4 * i;
        const uint32_t mine = own_pair(w, p, i);
        uint32_t m = 0;
#pragma unroll
        for (int o = 0; o < 7; ++o) {
            const uint32_t d = pair_of(w, o) ^ mine;
            m |= (o < s && ((d & 0xFFu) == 0 || (d & 0xFF00u) == 0) ? 1u : 0u) << o;
        }
        before[i] = m & part;
        own[i] = kQuadOut;
    }
    uint32_t done = 0, rounds = 0;
    while (__any_sync(0xFFFFFFFFu, done != part)) {
        uint32_t now = 0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int s = p + 4 * i;
            const bool run = ((part & ~done) >> s & 1u) && !(before[i] & ~done);
            if (run) own[i] = rounds;
            now |= group_ballot(run) << (4 * i);
        }
        done |= now;
        if (now) ++rounds;
    }
    return rounds;
}

// Face f's voxel from the voxel at `at` (spatial.rs:8-15).
__device__ __forceinline__ float* quad_face(float* at, int X, int Y, int f) {
    const uint32_t row = (uint32_t)X * 12, slab = (uint32_t)Y * row;
    const size_t off = f < 2 ? 12u : (f < 4 ? row : slab);
    return f & 1 ? at - off : at + off;
}
__device__ __forceinline__ size_t quad_voxel(int X, int Y, uint32_t P) {
    return ((size_t)pos_z(P) * Y + pos_y(P)) * X + pos_x(P);
}

// Derives the plan of a staged cell (groups with `fresh`; the whole warp takes
// part, other groups compute on what lies in their record and store nothing).
//
// The plan leaves out transporters and effectors whose rates are zero.  Such a
// slot changes nothing if
//   - every internal value lies in [+0, c_max] and every gathered one in
//     [+0, 1e6] (so no product is NaN and no clamp or maximum acts);
//   - rates, v_max, k_m and k_cat are below 1e30 and not negative, so
//     quotients lie in [0, 1], a reaction's flux in [0, substrate], and the
//     internal values stay in [+0, c_max];
//   - dt, epsilon and c_max are ordinary numbers.
// kQuadPlain says that all of this holds but for the gathered values and the
// light, which the update checks.
__device__ __forceinline__ void quad_plan(const CellConsts& c, QuadCell& C, int p, bool fresh, int X, int Y) {
    // Lane p waits for the p-th and the (p + 4)-th different dependency: more
    // than four are rare, and a lane's two acquire loads follow one another.
    int32_t wait[2] = {-1, -1};
    {
        int32_t d[6];
        int found = 0;
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            d[f] = C.dep[f];
            bool is_new = d[f] >= 0;
#pragma unroll
            for (int e = 0; e < f; ++e) is_new = is_new && d[e] != d[f];
            if (is_new) {
                if (found == p) wait[0] = d[f];
                if (found == p + 4) wait[1] = d[f];
                ++found;
            }
        }
    }
    const float inf = __uint_as_float(0x7F800000u);
    bool plain = c.dt >= 0.0f && c.dt < inf && c.epsilon >= 0.0f && c.epsilon < kQuadRateMax && c.c_max > 0.0f &&
                 c.c_max <= kQuadValueMax;
    const uint32_t top = __float_as_uint(c.c_max);
    const float4 x4 = *reinterpret_cast<const float4*>(&C.x[4 * p]);
    // Non-negative floats order like their bits; -0, negative values and NaN are above them.
    plain = plain && __float_as_uint(x4.x) <= top && __float_as_uint(x4.y) <= top && __float_as_uint(x4.z) <= top &&
            __float_as_uint(x4.w) <= top;

    // Reactions (the tests of cell.rs:246-262): those that run move to the front.
    uint4 rec[MARL_R_MAX / 4];
    uint32_t act = 0, run = 0;
    bool cof = false;
#pragma unroll
    for (int i = 0; i < MARL_R_MAX / 4; ++i) {
        rec[i] = C.rx[p + 4 * i];
        const uint32_t si = rec[i].x & 0xFF, pi = (rec[i].x >> 8) & 0xFF, ci = (rec[i].x >> 16) & 0xFF;
        const float km = __uint_as_float(rec[i].y), vmax = __uint_as_float(rec[i].z), kcat = __uint_as_float(rec[i].w);
        act += __popc(group_ballot(fabsf(vmax) > c.thr && si != pi));
        const bool runs =
            !(fabsf(vmax) < c.thr) && si != pi && si < MARL_M_INT && pi < MARL_M_INT && ci < MARL_M_INT;
        run |= group_ballot(runs) << (4 * i);
        if (runs) {
            plain = plain && km >= 0.0f && km < kQuadRateMax && kcat >= 0.0f && kcat < kQuadRateMax && vmax >= 0.0f &&
                    vmax < kQuadRateMax;
            if ((rec[i].x >> 24) >= (uint32_t)MARL_M_INT)
                rec[i].x = (rec[i].x & 0xFFFFFFu) | (uint32_t)kQuadZero << 24;
            else
                cof = true;
        }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < MARL_R_MAX / 4; ++i) {
        const uint32_t r = p + 4 * i;
        if (fresh && (run >> r & 1u)) C.rx[__popc(run & ((1u << r) - 1u))] = rec[i];
    }

    // Transporters and effectors
    const uint4 tw = C.idx[0], ew = C.idx[1];
    uint32_t tpart = 0, epart = 0;
    float2 tr[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const uint32_t a = own_pair(tw, p, i), b = own_pair(ew, p, i);
        tr[i] = C.tp[p + 4 * i];
        const float2 er = C.ef[p + 4 * i];
        tpart |= group_ballot((a & 0xFF) < MARL_S_EXT && (a >> 8) < MARL_M_INT && (tr[i].x != 0.0f || tr[i].y != 0.0f))
                 << (4 * i);
        epart |= group_ballot((b & 0xFF) < MARL_M_INT && (b >> 8) < MARL_S_EXT && er.y != 0.0f) << (4 * i);
        plain = plain && tr[i].x >= 0.0f && tr[i].x < kQuadRateMax && tr[i].y >= 0.0f && tr[i].y < kQuadRateMax &&
                er.y >= 0.0f && er.y < kQuadRateMax;
    }
    uint32_t to[2], eo[2];
    const uint32_t nt = quad_rounds(tw, tpart, p, to);
    const uint32_t ne = quad_rounds(ew, epart, p, eo);
    float sec[2] = {0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < 2; ++i)
        if (to[i] == 0) {
            const float xk = C.x[own_pair(tw, p, i) >> 8];
            sec[i] = div_rn(tr[i].y * xk, 1.0f + xk);
        }

    // Maintenance (cell.rs:291-311)
    float pm = 1.0f;
    if ((C.state & 0xFFFFu) > 0) {
        const float evolved = fmaxf(C.fate.w, 1.0f);
        const float rush = fmaxf(c.base_division_prep - evolved, 0.0f);
        pm = c.prep_maintenance_multiplier + rush * c.rush_penalty_rate;
    }
    const float keep = 1.0f - c.lambda_maintenance * pm * c.dt;
    const float cost = (float)act * c.reaction_maintenance * c.dt;
    plain = plain && keep >= 0.0f && keep <= 1.0f && cost >= 0.0f && cost < inf;
    plain = group_ballot(plain) == 0xFu;
    cof = group_ballot(cof) != 0;
    if (fresh) {
        C.dep[p] = wait[0];
        if (p < 2) C.dep[p + 4] = wait[1];
        C.rounds[p] = to[0] | to[1] << 8 | eo[0] << 16 | eo[1] << 24;
        C.secretion[p] = make_float2(sec[0], sec[1]);
        if (p == 0) {
            C.x[kQuadZero] = 0.0f;
            C.vox = (uint32_t)quad_voxel(X, Y, C.pos);
            C.keep = keep;
            C.cost = cost;
            C.info = __popc(run) | nt << 8 | ne << 16 | (plain ? kQuadPlain : 0u) | (cof ? kQuadCofactor : 0u);
        }
    }
    __syncwarp();
}

// Fate (cell.rs:332-366) of an updated cell; its internal values are stored by
// the caller.
__device__ __forceinline__ void quad_fate(const CellConsts& c, const QuadAt& t, const QuadCell& C) {
    const float energy = C.x[0];
    const uint32_t st = C.state;
    uint32_t prep = st & 0xFFFFu, quiescent = (st >> 16) & 1u;
    const float4 fate = C.fate;
    const float eff_death = fmaxf(fate.y, c.hard_death_floor);
    uint8_t event;
    if (energy < eff_death) {
        prep = 0;
        event = MARL_EVENT_DEATH;
    } else if (prep > 0) {
        prep -= 1;
        event = prep == 0 ? MARL_EVENT_DIVISION : MARL_EVENT_NONE;
    } else if (energy > fate.x) {
        const float pt = fmaxf(fate.w, 1.0f);  // `as u16` saturates
        prep = pt >= 65535.0f ? 65535u : (uint32_t)pt;
        quiescent = 0;
        event = MARL_EVENT_NONE;
    } else if (energy < fate.z) {
        quiescent = 1;
        event = MARL_EVENT_QUIESCENCE;
    } else {
        quiescent = 0;
        event = MARL_EVENT_NONE;
    }
    t.age[t.j] = C.age + 1;
    t.state[t.j] = (st & 0xFF000000u) | (quiescent << 16) | prep;
    t.events[t.j] = event;
}

// The whole update of cell j by one lane, for any values.
__device__ __noinline__ void quad_serial(const QuadAt t, const CellConsts& c, QuadCell& C) {
    const uint32_t nb = C.nb;
    const int n = __popc(nb);
    const size_t vox = quad_voxel(t.X, t.Y, C.pos);
    float* const at = t.field + vox * 12;
#pragma unroll 1
    for (int s = 0; s < MARL_S_EXT; ++s) {
        float m = 0.0f;
#pragma unroll
        for (int f = 0; f < 6; ++f)
            if ((nb >> f) & 1u) m = m + __ldcg(quad_face(at, t.X, t.Y, f) + s);
        C.ext[s] = n > 1 ? div_rn(m, (float)n) : m;
        C.del[s] = 0.0f;
    }
    const float dt = c.dt;
    const uint4 tw = C.idx[0], ew = C.idx[1];
#pragma unroll 1
    for (int i = 0; i < MARL_S_TRANSPORTERS; ++i) {
        const uint32_t pair = pair_of(tw, i), e = pair & 0xFF, k = pair >> 8;
        if (e >= MARL_S_EXT || k >= MARL_M_INT) continue;
        const float2 r = C.tp[i];
        const float ev = C.ext[e], xk = C.x[k];
        const float uptake = div_rn(r.x * ev, 1.0f + ev);
        const float secretion = div_rn(r.y * xk, 1.0f + xk);
        C.x[k] = rclamp(xk + (uptake - secretion) * dt, 0.0f, c.c_max);
        C.del[e] = C.del[e] + (secretion - uptake) * dt;
    }
    C.x[MARL_M_INT - 1] = t.light[vox];
    const float feps = 1.1920928955078125e-07f;
    const int runs = (int)(C.info & 0xFFu);
#pragma unroll 1
    for (int r = 0; r < runs; ++r) {
        const uint4 q = C.rx[r];
        const uint32_t si = q.x & 0xFF, pi = (q.x >> 8) & 0xFF, ci = (q.x >> 16) & 0xFF, fi = q.x >> 24;
        const float km = __uint_as_float(q.y), vmax = __uint_as_float(q.z), kcat = __uint_as_float(q.w);
        const float substrate_term = div_rn(C.x[si], km + C.x[si] + feps);
        const float catalyst_term = c.epsilon + div_rn(C.x[ci], kcat + C.x[ci] + feps);
        float rate = vmax * substrate_term * catalyst_term;
        if (fi < MARL_M_INT) {
            const float cof = C.x[fi];
            rate *= div_rn(cof, 1.0f + cof);
            C.x[fi] = cof - fminf(0.5f * rate * dt, cof);
        }
        const float flux = fminf(rate * dt, C.x[si]);
        C.x[si] = C.x[si] - flux;
        C.x[pi] = fminf(C.x[pi] + flux, c.c_max);
    }
    C.x[0] = fmaxf(C.x[0] * C.keep - C.cost, 0.0f);
    const bool quiescent = (C.state >> 16) & 1u;
#pragma unroll 1
    for (int i = 0; i < MARL_S_EFFECTORS; ++i) {
        const uint32_t pair = pair_of(ew, i), k = pair & 0xFF, e = pair >> 8;
        if (quiescent || k >= MARL_M_INT || e >= MARL_S_EXT) continue;
        const float2 pr = C.ef[i];
        const float xk = C.x[k];
        if (xk > pr.x) {
            const float amount = div_rn(pr.y * xk, 1.0f + xk) * dt;
            C.x[k] = fmaxf(xk - amount, 0.0f);
            C.del[e] = C.del[e] + amount;
        }
    }
#pragma unroll 1
    for (int s = 0; n > 0 && s < MARL_S_EXT; ++s) {
        const float split = div_rn(C.del[s], (float)n);
#pragma unroll
        for (int f = 0; f < 6; ++f)
            if ((nb >> f) & 1u) {
                float* const q = quad_face(at, t.X, t.Y, f) + s;
                __stcg(q, fmaxf(__ldcg(q) + split, 0.0f));
            }
    }
    st_release_u32(&t.done[t.j], t.epoch);
    quad_fate(c, t, C);
    for (int k = 0; k < MARL_M_INT; ++k) t.internal[(size_t)k * t.cap + t.j] = C.x[k];
}

// The reactions (cell.rs:246-285) of the warp's cells side by side, each
// cell's in slot order; `runs` of this lane's cell, `most` over the warp.
// Lane 0 holds the substrate, 1 the catalyst, 2 the cofactor, 3 the product.
// Every lane loads one value, divides once and stores once: lanes with nothing
// to store write to the trash slot, so the loop has no branch but its own.
template <bool COF>
__device__ __forceinline__ void quad_reactions(const CellConsts& c, QuadCell& C, int p, uint32_t runs, uint32_t most) {
    const unsigned FULL = 0xFFFFFFFFu;
    const int shift = p == 0 ? 0 : (p == 1 ? 16 : (p == 2 ? 24 : 8));
    const float tail = p < 2 ? 1.1920928955078125e-07f : 0.0f;  // f32::EPSILON
    const float eps = p == 1 ? c.epsilon : 0.0f;
    const bool stores = p == 0 || p == 3;
    uint4 q = C.rx[0];
#pragma unroll 1
    for (uint32_t r = 0; r < most; ++r) {
        const bool live = r < runs;
        const uint32_t own = (q.x >> shift) & 0x1Fu;
        const uint32_t load_at = live ? own : (uint32_t)kQuadZero;
        uint32_t store_at = live && stores ? own : (uint32_t)kQuadTrash;
        const float k0 = p == 0 ? __uint_as_float(q.y) : (p == 1 ? __uint_as_float(q.w) : 1.0f);
        const float vmax = __uint_as_float(q.z);
        const uint32_t word = q.x;
        q = C.rx[(r + 1) & (MARL_R_MAX - 1)];
        float val = C.x[load_at];
        const float term = eps + div_pos(val, k0 + val + tail);  // 0 + t is t: t >= +0
        float s_now = __shfl_sync(FULL, val, 0, 4);
        float rate = vmax * __shfl_sync(FULL, term, 0, 4) * __shfl_sync(FULL, term, 1, 4);
        float left = 0.0f;
        if constexpr (COF) {
            const float cof = __shfl_sync(FULL, val, 2, 4);
            const float cof_term = __shfl_sync(FULL, term, 2, 4);
            const uint32_t fi = word >> 24;
            if (fi != (uint32_t)kQuadZero) {
                rate *= cof_term;
                left = cof - fminf(0.5f * rate * c.dt, cof);
                const bool is_s = fi == (word & 0xFFu), is_p = fi == ((word >> 8) & 0xFFu);
                s_now = is_s ? left : s_now;
                val = is_p ? left : val;  // lane 3's product
                if (live && p == 2 && !is_s && !is_p) store_at = fi;
            }
        }
        const float flux = fminf(rate * c.dt, s_now);
        float out = p == 0 ? s_now - flux : fminf(val + flux, c.c_max);
        if constexpr (COF) out = p == 2 ? left : out;
        C.x[store_at] = out;
        __syncwarp();
    }
}

// Transport and reactions of the groups with `on`, whose plan is plain and
// whose gathered values are ordinary.  The whole warp takes part; the other
// groups change nothing.
__device__ __forceinline__ void quad_kinetics(const CellConsts& c, QuadCell& C, int p, float light, bool on) {
    const unsigned FULL = 0xFFFFFFFFu;
    const float dt = c.dt;
    const uint32_t info = on ? C.info : 0u;
    const uint32_t mine = on ? C.rounds[p] : 0xFFFFFFFFu;
    // Transport (cell.rs:223-238): uptake from the gathered environment, all
    // slots at once; then each slot's sums in its round.
    {
        const uint4 w = C.idx[0];
        const float2 sec = C.secretion[p];
        uint32_t e[2], k[2];
        float uptake[2] = {0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const bool in = ((mine >> (8 * i)) & 0xFFu) != kQuadOut;
            const uint32_t pr = own_pair(w, p, i);
            e[i] = in ? pr & 0xFFu : 0u;
            k[i] = in ? pr >> 8 : 0u;
            if (i == 0 || __any_sync(FULL, in)) {
                const float ev = C.ext[e[i]];
                uptake[i] = div_pos(in ? C.tp[p + 4 * i].x * ev : 0.0f, 1.0f + ev);
            }
        }
        const uint32_t most = __reduce_max_sync(FULL, (info >> 8) & 0xFFu);
#pragma unroll 1
        for (uint32_t r = 0; r < most; ++r) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const bool now = ((mine >> (8 * i)) & 0xFFu) == r;
                if (i == 1 && !__any_sync(FULL, now)) continue;
                const float xk = C.x[k[i]];
                const float de = C.del[e[i]];
                float secretion = i ? sec.y : sec.x;
                if (r > 0) secretion = div_pos(now ? C.tp[p + 4 * i].y * xk : 0.0f, 1.0f + xk);
                const float x_new = rclamp(xk + (uptake[i] - secretion) * dt, 0.0f, c.c_max);
                const float d_new = de + (secretion - uptake[i]) * dt;
                if (now) {
                    C.x[k[i]] = x_new;
                    C.del[e[i]] = d_new;
                }
            }
            __syncwarp();
        }
    }
    if (on && p == 3) C.x[MARL_M_INT - 1] = light;  // cell.rs:243
    __syncwarp();

    const uint32_t runs = info & 0xFFu, most = __reduce_max_sync(FULL, runs);
    if (__any_sync(FULL, (info & kQuadCofactor) != 0))
        quad_reactions<true>(c, C, p, runs, most);
    else
        quad_reactions<false>(c, C, p, runs, most);
}

// Maintenance and effectors, likewise.
__device__ __forceinline__ void quad_effects(const CellConsts& c, QuadCell& C, int p, bool on) {
    const unsigned FULL = 0xFFFFFFFFu;
    const float dt = c.dt;
    const uint32_t info = on ? C.info : 0u;
    const uint32_t mine = on ? C.rounds[p] : 0xFFFFFFFFu;
    // Maintenance (cell.rs:291-311)
    if (on && p == 0) C.x[0] = fmaxf(C.x[0] * C.keep - C.cost, 0.0f);
    __syncwarp();

    // Effectors (cell.rs:314-329): nothing to do unless one of them fires,
    // because their internal values only change by firing.
    {
        const bool awake = on && !((C.state >> 16) & 1u);
        const uint4 w = C.idx[1];
        uint32_t k[2], e[2], round[2];
        bool fires = false;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            round[i] = awake ? (mine >> (16 + 8 * i)) & 0xFFu : kQuadOut;
            const uint32_t pr = own_pair(w, p, i);
            k[i] = round[i] != kQuadOut ? pr & 0xFFu : 0u;
            e[i] = round[i] != kQuadOut ? pr >> 8 : 0u;
            fires = fires || (round[i] != kQuadOut && C.x[k[i]] > C.ef[p + 4 * i].x);
        }
        const uint32_t firing = group_ballot(fires);
        const uint32_t most = __reduce_max_sync(FULL, firing ? (info >> 16) & 0xFFu : 0u);
#pragma unroll 1
        for (uint32_t r = 0; r < most; ++r) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float2 pr = C.ef[p + 4 * i];
                const float xk = C.x[k[i]];
                const bool now = round[i] == r && xk > pr.x;
                if (!__any_sync(FULL, now)) continue;
                const float amount = div_pos(now ? pr.y * xk : 0.0f, 1.0f + xk) * dt;
                const float x_new = fmaxf(xk - amount, 0.0f), d_new = C.del[e[i]] + amount;
                if (now) {
                    C.x[k[i]] = x_new;
                    C.del[e[i]] = d_new;
                }
            }
            __syncwarp();
        }
    }
}

// Gather -> tick -> scatter (spatial.rs:56-110, cell.rs:193-369; update_cell is
// the same update with one lane) of the cells of the groups that are `ready`:
// all their dependencies are done.  The whole warp takes part; the other
// groups change nothing.  False for the lanes of a ready group whose values
// are not ordinary: nothing of its cell is changed then but C.ext and C.del.
template <class View>
__device__ __forceinline__ bool quad_update(const View& v, const CellConsts& c, QuadCell& C, int p, bool ready) {
    const uint32_t nb = ready ? C.nb : 0u;
    const int n = __popc(nb);
    const size_t vox = ready ? C.vox : 0u;
    float* const at = v.field() + vox * 12 + 4 * p;

    // Gather (spatial.rs:56-77), summed in face order from 0.0; a face that is
    // not an empty voxel adds +0.0, which changes nothing.
    float4 nv[6];
    auto load_faces = [&] {
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            nv[f] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (p < 3 && ((nb >> f) & 1u)) nv[f] = ld4(quad_face(at, v.X(), v.Y(), f));
        }
    };
    load_faces();
    const float light = ready && p == 3 ? __ldg(v.light() + vox) : 0.0f;
    float m[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int f = 0; f < 6; ++f) m[0] += nv[f].x, m[1] += nv[f].y, m[2] += nv[f].z, m[3] += nv[f].w;
    quad_divide(m, n);
    if (ready && p < 3) {
        *reinterpret_cast<float4*>(&C.ext[4 * p]) = make_float4(m[0], m[1], m[2], m[3]);
        *reinterpret_cast<float4*>(&C.del[4 * p]) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    bool ordinary = __float_as_uint(light) <= __float_as_uint(c.c_max);
#pragma unroll
    for (int s = 0; s < 4; ++s) ordinary = ordinary && __float_as_uint(m[s]) <= __float_as_uint(kQuadValueMax);
    const uint32_t all = group_ballot(ordinary);  // by the whole warp, ready or not
    const bool fast = ready && all == 0xFu && (C.info & kQuadPlain);
    __syncwarp();
    quad_kinetics(c, C, p, light, fast);
    // The scatter's starting values, which no other cell has touched: read again
    // (from L2, behind the effectors) rather than held in 24 registers.
    load_faces();
    quad_effects(c, C, p, fast);

    // Scatter (spatial.rs:87-110, field.rs:57-62): the deltas split over the
    // gathered neighbours, clamped after each add.
    if (fast && p < 3) {
        const float4 d = *reinterpret_cast<const float4*>(&C.del[4 * p]);
        float split[4] = {d.x, d.y, d.z, d.w};
        quad_divide(split, n);
#pragma unroll
        for (int f = 0; f < 6; ++f)
            if ((nb >> f) & 1u)
                st4(quad_face(at, v.X(), v.Y(), f),
                    make_float4(fmaxf(nv[f].x + split[0], 0.0f), fmaxf(nv[f].y + split[1], 0.0f),
                                fmaxf(nv[f].z + split[2], 0.0f), fmaxf(nv[f].w + split[3], 0.0f)));
    }
    __syncwarp();
    if (fast) {
        // Publish: the group's stores are ordered before lane 0's release by
        // the warp barrier.  Only later kernels read the cell's own state.
        if (p == 0) st_release_u32(&v.done()[v.j()], v.epoch());
        const QuadAt t = v.all();
        if (p == 0) quad_fate(c, t, C);
#pragma unroll
        for (int i = 0; i < MARL_M_INT / 4; ++i) t.internal[(size_t)(p + 4 * i) * t.cap + t.j] = C.x[p + 4 * i];
    }
    return fast || !ready;
}

// Rounds of a warp: poll the dependencies of its staged cells, update the
// ready ones together, give every free group the next index from the ticket
// counter (in group order, so indices go out in ascending order) and stage it.
// A warp with no free group left to fill keeps polling.  Progress is as in the
// lane-per-cell loop: a cell waits only for smaller indices, whose tickets
// were taken earlier by warps that run; every wait is bounded.
template <class Stage, class Look>
__device__ __forceinline__ void quad_loop(QuadCell* cells, const CellConsts& c, uint32_t total, uint32_t* ticket,
                                          uint32_t* err, Stage stage, Look look) {
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, p = lane & 3;
    // Cells a warp holds: as few as the grid's warps need to hold all of them,
    // so that they wait on one another's passes as little as possible.
    const uint32_t warps = gridDim.x * (kQuadThreads / 32), per_warp = min((total + warps - 1) / warps, 8u);
    if ((blockIdx.x * (kQuadThreads / 32) + (threadIdx.x >> 5)) * per_warp >= total) return;  // earlier warps hold them
    const bool usable = (uint32_t)(lane >> 2) < per_warp;
    QuadCell& C = cells[threadIdx.x >> 2];
    bool pending = false, fresh = false, more = true;
    uint32_t gi = 0, waiting = 0, spins = 0;
    for (;;) {
        if (__any_sync(FULL, fresh)) {
            cp_async_wait_all();
            __syncwarp();
            const auto w = look(C, gi);
            quad_plan(c, C, p, fresh, w.X(), w.Y());
            if (fresh) {
                waiting = (pending && C.dep[p] >= 0 ? 1u : 0u) | (pending && p < 2 && C.dep[p + 4] >= 0 ? 2u : 0u);
                fresh = false;
            }
        }
        const auto v = look(C, gi);  // not used where the group has no cell
        bool ready = false;
        if (pending) {
            const uint32_t *done = v.done(), epoch = v.epoch();
            if ((waiting & 1u) && ld_acquire_u32(&done[C.dep[p]]) == epoch) waiting &= ~1u;
            if ((waiting & 2u) && ld_acquire_u32(&done[C.dep[p + 4]]) == epoch) waiting &= ~2u;
            ready = waiting == 0;
        }
        ready = group_ballot(ready) == 0xFu;
        const unsigned run = __ballot_sync(FULL, ready);
        const unsigned free_lanes = __ballot_sync(FULL, usable && (!pending || ready));
        uint32_t base = 0;
        if (more && free_lanes && lane == 0) base = atomicAdd(ticket, (uint32_t)__popc(free_lanes) >> 2);
        if (run) {  // an update publishes its cell itself
            // Passes each lane's acquires on to the lanes that gather: a vote orders no memory.
            __syncwarp();
            const bool updated = quad_update(v, c, C, p, ready);
            if (__any_sync(FULL, !updated)) {
                if (!updated && p == 0) quad_serial(v.all(), c, C);
                __syncwarp();
            }
        }
        if (ready) {
            pending = false;
        } else if (pending && ++spins > c.wait_limit) {
            if (p == 0) {
                atomicOr(err, kErrTimeoutDeps);
                v.all().events[v.j()] = MARL_EVENT_NONE;
                st_release_u32(&v.done()[v.j()], v.epoch());
            }
            pending = false;
        }
        if (more && free_lanes) {
            base = __shfl_sync(FULL, base, 0);
            if (base >= total) {
                more = false;
            } else if ((free_lanes >> lane) & 1u) {
                __syncwarp(free_lanes);  // the group's reads of the record it replaces
                const uint32_t next = base + ((uint32_t)__popc(free_lanes & ((1u << (lane & 28)) - 1u)) >> 2);
                if (next < total) {
                    gi = next;
                    stage(C, gi, p);
                    pending = fresh = true;
                    spins = 0;
                }
            }
        }
        if (!__any_sync(FULL, pending)) break;
        // Back off only when no group of the warp made progress this round.
        if (!run && !__any_sync(FULL, fresh)) __nanosleep(32);
    }
}

__global__ void __launch_bounds__(kQuadThreads, kQuadBlocksPerSM)
    k_cell_tick_quad(const __grid_constant__ CellLaunch a) {
    extern __shared__ __align__(16) unsigned char tick_smem[];
    const uint32_t total = a.n_dev ? *a.n_dev : a.n;
    if (a.split && total > a.split) return;
    quad_loop(
        reinterpret_cast<QuadCell*>(tick_smem), a.k, total, a.ticket, a.err,
        [&](QuadCell& C, uint32_t gi, int p) {
            const CellRunView v{&a.t, a.g, a.field, a.light, a.epoch, nullptr, nullptr, a.cmap};
            quad_stage(v, C, gi, p, a.k.schedule_here != 0);
        },
        [&](const QuadCell&, uint32_t gi) { return QuadOfLaunch{a, gi}; });
}

__global__ void __launch_bounds__(kQuadThreads, kQuadBlocksPerSM)
    k_cell_tick_quad_batch(const RunDesc* __restrict__ runs, int n_runs, BatchScalars* __restrict__ bs,
                           const __grid_constant__ CellConsts c, int parity, uint32_t split) {
    extern __shared__ __align__(16) unsigned char tick_smem[];
    const uint32_t total = batch_total(runs, n_runs);
    if (total > split) return;
    quad_loop(
        reinterpret_cast<QuadCell*>(tick_smem), c, total, &bs->ticket, &bs->err,
        [&](QuadCell& C, uint32_t gi, int p) {
            const RunDesc& R = runs[find_run(runs, n_runs, gi)];
            const uint32_t j = gi - R.cell_base;
            const CellRunView v{&R.t, R.g, R.field[parity], R.light, R.epoch, nullptr, nullptr, R.cmap};
            quad_stage(v, C, j, p, c.schedule_here != 0);
            if (p == 0) C.at = quad_at(R.t, R.g, v.field, v.light, v.epoch, j);  // read after the plan's warp barrier
        },
        [&](const QuadCell& C, uint32_t) { return QuadOfCell{C.at}; });
}
