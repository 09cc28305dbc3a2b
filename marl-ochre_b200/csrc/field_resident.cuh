// All substeps of a small grid in one cooperative kernel (included by field.cu).
//
// What bounds small grids in k_diffuse is not the stencil: a substep of 10,000
// voxels takes 3.3 us of launch, fill and drain, and the host spends 3.6 us on
// each launch.  Here every block keeps a brick of the grid in shared memory (two
// copies, with a halo of one voxel) through all substeps.  Per substep it
// computes the brick's surface first and sends it to its neighbours, computes
// the inside while that travels, and receives their surfaces into its halo.  The
// whole brick goes to global memory after the last substep only.
//
// A surface voxel travels as four 16-byte words of three species and the
// substep's tag, written and read as single 128-bit accesses: a word whose tag
// is there has its data, so a substep costs one trip through L2 (with flags,
// release and acquire it cost three, 3 us, no less than a dependent launch).
// Words alternate between two sets by substep; a set is written again only after
// the neighbour that read it has sent the next substep's surface.
//
// Blocks wait on one another, so the launch is cooperative (all resident or
// none) and every wait is bounded.
//
// The arithmetic is stencil_pairwise()'s operation for operation; a wall, a
// grid edge or an occupied neighbour reads as the centre voxel.

constexpr int kResThreads = 512;
constexpr uint32_t kResSmemMax = 220 * 1024;

// Shared memory: two copies of the brick with its halo, a word per brick voxel
// (place in the copy | walls << 16), two words per halo voxel, the occupancy of
// brick and halo.
__host__ __device__ inline uint32_t resident_halo(int bx, int by, int bz) { return 2u * (bx * by + by * bz + bx * bz); }
__host__ __device__ inline uint32_t resident_words(int bx, int by, int bz) {
    return ((uint32_t)bx * by * bz + 1) & ~1u;  // even: what follows is 8-byte aligned
}
__host__ __device__ inline uint32_t resident_smem(int bx, int by, int bz) {
    const uint32_t full = (uint32_t)(bx + 2) * (by + 2) * (bz + 2);
    return full * 96 + resident_words(bx, by, bz) * 4 + resident_halo(bx, by, bz) * 8 + ((full + 15) & ~15u);
}

// First word of face f's part of a brick's mailbox (in voxels), and its size: a
// face is bx x by, by x bz or bx x bz voxels.
__host__ __device__ inline uint32_t resident_face(const ResidentPlan& p, int f) {
    const uint32_t yz = p.by * p.bz, xz = p.bx * p.bz;
    return f < 2 ? f * yz : (f < 4 ? 2 * yz + (f - 2) * xz : 2 * (yz + xz) + (f - 4) * p.bx * p.by);
}
size_t resident_mail_bytes(const ResidentPlan& p) {
    return (size_t)p.nx * p.ny * p.nz * resident_halo(p.bx, p.by, p.bz) * 64 * 2;
}

struct ResidentArgs {
    float* field;           // the grid, updated in place
    const uint8_t* mask;    // [z][y][pitch]
    int pitch;
    Grid g;
    ResidentPlan p;
    FieldConsts k;
    int substeps;
    uint4* mail;            // [2][brick][resident_halo][4], zeroed; substep s sends tag s + 1
    uint32_t* err;
};

// Single 128-bit accesses at GPU scope.
__device__ __forceinline__ void mail_send(uint4* p, float a, float b, float c, uint32_t tag) {
    asm volatile(
        "{\n\t.reg .b128 w;\n\t.reg .b64 lo, hi;\n\t"
        "mov.b64 lo, {%1, %2};\n\tmov.b64 hi, {%3, %4};\n\tmov.b128 w, {lo, hi};\n\t"
        "st.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p),
        "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(__float_as_uint(c)), "r"(tag)
        : "memory");
}
__device__ __forceinline__ uint4 mail_read(const uint4* p) {
    uint4 v;
    asm volatile(
        "{\n\t.reg .b128 w;\n\t.reg .b64 lo, hi;\n\t"
        "ld.relaxed.gpu.global.b128 w, [%4];\n\tmov.b128 {lo, hi}, w;\n\t"
        "mov.b64 {%0, %1}, lo;\n\tmov.b64 {%2, %3}, hi;\n\t}"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p)
        : "memory");
    return v;
}

__device__ __forceinline__ void stencil_at(float out[12], const Vox& c, const float* const (&nb)[6],
                                           const FieldConsts& k) {
    const float structural = c.v[3].y;  // species 7
    const float niche = 1.0f - div_rn(k.alpha_eps * structural, k.k_eps + structural);
#pragma unroll
    for (int w = 0; w < 3; ++w) {
        float4 n[6];
#pragma unroll
        for (int f = 0; f < 6; ++f) n[f] = reinterpret_cast<const float4*>(nb[f])[w];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int q = 2 * w + h;
            const float2 cc = c.v[q];
            auto at = [&](int f) { return h ? make_float2(n[f].z, n[f].w) : make_float2(n[f].x, n[f].y); };
            const float2 d = make_float2(__fmul_rn(k.d_voxel[2 * q], niche), __fmul_rn(k.d_voxel[2 * q + 1], niche));
            float2 lap = add2_rn(at(0), at(1));  // -x, +x, -y, +y, -z, +z: the reference's order
            lap = add2_rn(lap, at(2));
            lap = add2_rn(lap, at(3));
            lap = add2_rn(lap, at(4));
            lap = add2_rn(lap, at(5));
            lap = add2_rn(lap, make_float2(__fmul_rn(-6.0f, cc.x), __fmul_rn(-6.0f, cc.y)));
            const float2 ndecay = make_float2(__fmul_rn(-k.lambda_decay[2 * q], cc.x),
                                              __fmul_rn(-k.lambda_decay[2 * q + 1], cc.y));
            const float2 t = add2_rn(make_float2(__fmul_rn(d.x, lap.x), __fmul_rn(d.y, lap.y)), ndecay);
            const float2 nc = add2_rn(cc, make_float2(__fmul_rn(k.dt_sub, t.x), __fmul_rn(k.dt_sub, t.y)));
            out[2 * q] = fmaxf(nc.x, 0.0f);
            out[2 * q + 1] = fmaxf(nc.y, 0.0f);
        }
    }
}

__global__ void __launch_bounds__(kResThreads, 1) k_diffuse_resident(const __grid_constant__ ResidentArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint32_t s_front, s_back, s_halo;
    __shared__ int s_abort;
    const ResidentPlan p = a.p;
    const Grid g = a.g;
    const int tid = threadIdx.x, lane = tid & 31;
    const int ix = blockIdx.x % p.nx, iy = (blockIdx.x / p.nx) % p.ny, iz = blockIdx.x / (p.nx * p.ny);
    const int x0 = ix * p.bx, y0 = iy * p.by, z0 = iz * p.bz;
    const int ex = min(p.bx, g.X - x0), ey = min(p.by, g.Y - y0), ez = min(p.bz, g.Z - z0);  // this brick's extent
    const int row = p.bx + 2, slab = row * (p.by + 2), full = slab * (p.bz + 2);
    float* const copy0 = reinterpret_cast<float*>(smem);
    float* const copy1 = copy0 + (size_t)full * 12;
    uint32_t* const list = reinterpret_cast<uint32_t*>(copy1 + (size_t)full * 12);
    uint2* const halo = reinterpret_cast<uint2*>(list + resident_words(p.bx, p.by, p.bz));
    uint8_t* const occ = reinterpret_cast<uint8_t*>(halo + resident_halo(p.bx, p.by, p.bz));
    const int voxels = ex * ey * ez;

    const uint32_t mail_brick = resident_halo(p.bx, p.by, p.bz);  // voxels of a brick's mailbox
    const size_t mail_set = (size_t)gridDim.x * mail_brick * 4;

    if (tid == 0) s_front = 0, s_back = (uint32_t)voxels, s_halo = 0, s_abort = 0;
    // Occupancy (outside the grid: occupied, a wall either way) and values of the
    // brick and its halo.  Halo edges and corners are not read by anyone.
    for (int i = tid; i < full; i += kResThreads) {
        const int lx = i % row - 1, ly = (i / row) % (p.by + 2) - 1, lz = i / slab - 1;
        const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
        const bool in = lx <= ex && ly <= ey && lz <= ez && x >= 0 && x < g.X && y >= 0 && y < g.Y && z >= 0 && z < g.Z;
        occ[i] = in ? a.mask[((size_t)z * g.Y + y) * a.pitch + x] != 0 : 1;
    }
    for (int i = tid; i < full * 3; i += kResThreads) {
        const int v = i / 3, q = i % 3;
        const int lx = v % row - 1, ly = (v / row) % (p.by + 2) - 1, lz = v / slab - 1;
        const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
        if (lx <= ex && ly <= ey && lz <= ez && x >= 0 && x < g.X && y >= 0 && y < g.Y && z >= 0 && z < g.Z)
            reinterpret_cast<float4*>(copy0)[i] =
                __ldcg(reinterpret_cast<const float4*>(a.field + (((size_t)z * g.Y + y) * g.X + x) * 12) + q);
    }
    __syncthreads();

    // The brick's voxels: the surface that a neighbour reads from the front of
    // the list, the inside from its back; the halo voxels that are read.
    for (int i0 = tid - lane; i0 < voxels; i0 += kResThreads) {
        const int i = i0 + lane;
        bool surface = false;
        uint32_t word = 0;
        if (i < voxels) {
            const int lx = i % ex, ly = (i / ex) % ey, lz = i / (ex * ey);
            const int at = (lz + 1) * slab + (ly + 1) * row + lx + 1;
            const uint32_t walls = (uint32_t)(occ[at - 1] != 0) | (uint32_t)(occ[at + 1] != 0) << 1 |
                                   (uint32_t)(occ[at - row] != 0) << 2 | (uint32_t)(occ[at + row] != 0) << 3 |
                                   (uint32_t)(occ[at - slab] != 0) << 4 | (uint32_t)(occ[at + slab] != 0) << 5 |
                                   (uint32_t)(occ[at] != 0) << 6;
            word = (uint32_t)at | walls << 16;
            surface = (lx == 0 && ix > 0) || (lx == ex - 1 && ix < p.nx - 1) || (ly == 0 && iy > 0) ||
                      (ly == ey - 1 && iy < p.ny - 1) || (lz == 0 && iz > 0) || (lz == ez - 1 && iz < p.nz - 1);
        }
        const unsigned front = __ballot_sync(0xFFFFFFFFu, surface), back = __ballot_sync(0xFFFFFFFFu, i < voxels && !surface);
        uint32_t f0 = 0, b0 = 0;
        if (lane == 0) {
            f0 = atomicAdd(&s_front, (uint32_t)__popc(front));
            b0 = atomicSub(&s_back, (uint32_t)__popc(back)) - (uint32_t)__popc(back);
        }
        f0 = __shfl_sync(0xFFFFFFFFu, f0, 0);
        b0 = __shfl_sync(0xFFFFFFFFu, b0, 0);
        const unsigned below = (1u << lane) - 1u;
        if (surface)
            list[f0 + __popc(front & below)] = word;
        else if (i < voxels)
            list[b0 + __popc(back & below)] = word;
    }
    for (int i = tid; i < full; i += kResThreads) {
        const int lx = i % row - 1, ly = (i / row) % (p.by + 2) - 1, lz = i / slab - 1;
        const bool ox = lx < 0 || lx == ex, oy = ly < 0 || ly == ey, oz = lz < 0 || lz == ez;
        const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
        // Occupied voxels too, although nothing reads them: that a neighbour's
        // surface has arrived is what allows the next one to be sent to it.
        if (lx <= ex && ly <= ey && lz <= ez && (int)ox + (int)oy + (int)oz == 1 && x >= 0 && x < g.X && y >= 0 &&
            y < g.Y && z >= 0 && z < g.Z) {
            // The neighbour's opposite face: its f ^ 1 is toward this brick.
            const int f = ox ? (lx < 0 ? 0 : 1) : (oy ? (ly < 0 ? 2 : 3) : (lz < 0 ? 4 : 5));
            const int jx = ix + (f == 0 ? -1 : (f == 1 ? 1 : 0)), jy = iy + (f == 2 ? -1 : (f == 3 ? 1 : 0)),
                      jz = iz + (f == 4 ? -1 : (f == 5 ? 1 : 0));
            const uint32_t in_face = f < 2 ? (uint32_t)(lz * p.by + ly)
                                           : (f < 4 ? (uint32_t)(lz * p.bx + lx) : (uint32_t)(ly * p.bx + lx));
            halo[atomicAdd(&s_halo, 1u)] =
                make_uint2((uint32_t)i, (uint32_t)((jz * p.ny + jy) * p.nx + jx) * mail_brick +
                                            resident_face(p, f ^ 1) + in_face);
        }
    }
    __syncthreads();
    const uint32_t n_surface = s_front, n_halo = s_halo;
    for (int s = 0; s < a.substeps; ++s) {
        const float* const from = s & 1 ? copy1 : copy0;
        float* const to = s & 1 ? copy0 : copy1;
        uint4* const mail = a.mail + (s & 1 ? mail_set : 0);
        const uint32_t tag = (uint32_t)s + 1;
        const bool final_step = s == a.substeps - 1;
        auto update = [&](uint32_t i, bool send) {
            const uint32_t word = list[i], at = word & 0xFFFFu;
            const float* P = from + (size_t)at * 12;
            Vox c;
            load_vox(c, P);
            float out[12];
            if (word >> 22 & 1u) {  // occupied: copied unchanged (field.rs:130-136)
#pragma unroll
                for (int q = 0; q < 6; ++q) out[2 * q] = c.v[q].x, out[2 * q + 1] = c.v[q].y;
            } else {
                const float* const nb[6] = {P - (word >> 16 & 1u ? 0 : 12),       P + (word >> 17 & 1u ? 0 : 12),
                                            P - (word >> 18 & 1u ? 0 : row * 12),  P + (word >> 19 & 1u ? 0 : row * 12),
                                            P - (word >> 20 & 1u ? 0 : slab * 12), P + (word >> 21 & 1u ? 0 : slab * 12)};
                stencil_at(out, c, nb, a.k);
            }
            float4* T = reinterpret_cast<float4*>(to + (size_t)at * 12);
            T[0] = make_float4(out[0], out[1], out[2], out[3]);
            T[1] = make_float4(out[4], out[5], out[6], out[7]);
            T[2] = make_float4(out[8], out[9], out[10], out[11]);
            if (send) {
                const int lx = (int)at % row - 1, ly = ((int)at / row) % (p.by + 2) - 1, lz = (int)at / slab - 1;
                auto to_face = [&](int f, uint32_t in_face) {
                    uint4* w = mail + ((size_t)blockIdx.x * mail_brick + resident_face(p, f) + in_face) * 4;
#pragma unroll
                    for (int q = 0; q < 4; ++q) mail_send(w + q, out[3 * q], out[3 * q + 1], out[3 * q + 2], tag);
                };
                if (lx == 0 && ix > 0) to_face(0, (uint32_t)(lz * p.by + ly));
                if (lx == ex - 1 && ix < p.nx - 1) to_face(1, (uint32_t)(lz * p.by + ly));
                if (ly == 0 && iy > 0) to_face(2, (uint32_t)(lz * p.bx + lx));
                if (ly == ey - 1 && iy < p.ny - 1) to_face(3, (uint32_t)(lz * p.bx + lx));
                if (lz == 0 && iz > 0) to_face(4, (uint32_t)(ly * p.bx + lx));
                if (lz == ez - 1 && iz < p.nz - 1) to_face(5, (uint32_t)(ly * p.bx + lx));
            }
        };
        for (uint32_t i = tid; i < n_surface; i += kResThreads) update(i, !final_step);
        for (uint32_t i = n_surface + tid; i < (uint32_t)voxels; i += kResThreads) update(i, false);
        if (final_step) break;
        // The neighbours' surfaces of this substep, word by word.
        for (uint32_t i = tid; i < n_halo * 4; i += kResThreads) {
            const uint2 h = halo[i >> 2];
            const uint32_t q = i & 3u;
            const uint4* w = mail + (size_t)h.y * 4 + q;
            uint4 v = mail_read(w);
            for (uint32_t spins = 0; v.w != tag; v = mail_read(w))
                if (++spins > kFlagSpinLimit || *(volatile int*)&s_abort) {
                    atomicOr(a.err, kErrTimeoutMbar);
                    s_abort = 1;
                    break;
                }
            float* d = to + (size_t)h.x * 12 + 3 * q;
            d[0] = __uint_as_float(v.x), d[1] = __uint_as_float(v.y), d[2] = __uint_as_float(v.z);
        }
        __syncthreads();
        if (*(volatile int*)&s_abort) return;  // set before the barrier or not at all in this substep
    }
    // The result.  With two substeps or more every neighbour has sent a surface,
    // so it has long read its first halo from the grid.
    __syncthreads();
    const float* const result = a.substeps & 1 ? copy1 : copy0;
    for (int i = tid; i < voxels * 3; i += kResThreads) {
        const int v = i / 3, q = i % 3;
        const int lx = v % ex, ly = (v / ex) % ey, lz = v / (ex * ey);
        const float4 val = reinterpret_cast<const float4*>(
            result + (size_t)((lz + 1) * slab + (ly + 1) * row + lx + 1) * 12)[q];
        const size_t at = ((size_t)(z0 + lz) * g.Y + y0 + ly) * g.X + x0 + lx;
        __stcg(reinterpret_cast<float4*>(a.field + at * 12) + q, val);
    }
}

// The largest grid that runs this way.  A whole call of 10 substeps on device pointers, this kernel / 10
// tile launches: 10k voxels 49 / 59 us, 16k 51 / 59, 36k 61 / 73, 38k 63 / 72, 66k
// 75 / 71, 131k 100 / 84: with more than a voxel a thread the brick's own
// arithmetic (seven voxels read from shared memory for each one written) takes
// longer than a launch.
constexpr size_t kResidentVoxels = 40000;
// The fewest substeps: loading the bricks costs about three launches.  38k voxels,
// 4 / 5 / 20 substeps: 49 / 50 / 95 us here, 42 / 48 / 112 us in tiles; 10k voxels:
// 37 / 39 / 73 here, 40 / 47 / 88; 768 voxels: 35 / 35 / 59 here, 32 / 40 / 79.
constexpr uint32_t kResidentSubsteps = 5, kResidentSubstepsMax = 1u << 30;  // tags are 32-bit

// A plan with at most num_sms bricks, or false.  The smallest largest brick
// wins; among equals the one with the smaller surface.
bool resident_plan(const Grid& g, uint32_t substeps, int num_sms, ResidentPlan* plan) {
    if (g.V() > kResidentVoxels || substeps < kResidentSubsteps || substeps > kResidentSubstepsMax) return false;
    double best = 1e300;
    for (int nz = 1; nz <= num_sms && nz <= g.Z; ++nz)
        for (int ny = 1; ny * nz <= num_sms && ny <= g.Y; ++ny) {
            const int nx = std::min(num_sms / (ny * nz), g.X);
            const int bx = (g.X + nx - 1) / nx, by = (g.Y + ny - 1) / ny, bz = (g.Z + nz - 1) / nz;
            const uint64_t full = (uint64_t)(bx + 2) * (by + 2) * (bz + 2);
            if (full > 0xFFFFu || full * 101 > kResSmemMax) continue;  // places are 16-bit
            const uint32_t smem = resident_smem(bx, by, bz);
            if (smem > kResSmemMax) continue;
            const double cost = (double)bx * by * bz + 0.25 * resident_halo(bx, by, bz);
            if (cost < best) {
                best = cost;
                // Bricks that would be empty are left out.
                *plan = ResidentPlan{bx, by, bz, (g.X + bx - 1) / bx, (g.Y + by - 1) / by, (g.Z + bz - 1) / bz, smem};
            }
        }
    return best < 1e300;
}

cudaError_t launch_diffuse_resident(const ResidentPlan& plan, float* field, const uint8_t* mask, int pitch, const Grid& g,
                                    const FieldConsts& k, int substeps, void* mail, uint32_t* err, cudaStream_t s) {
    static std::atomic<int> setup[kSetupDevices];
    cudaError_t e = set_smem_once(setup, k_diffuse_resident, kResSmemMax);
    if (e != cudaSuccess) return e;
    ResidentArgs a{field, mask, pitch, g, plan, k, substeps, (uint4*)mail, err};
    void* args[] = {&a};
    return cudaLaunchCooperativeKernel((const void*)k_diffuse_resident, dim3(plan.nx * plan.ny * plan.nz),
                                       dim3(kResThreads), args, plan.smem, s);
}
