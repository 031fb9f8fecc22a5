// mesh.cu -- marching cubes over all allocated blocks (src/voxel_hashing/
// scene_mesh.cu:14-643, tables include/voxel_hashing/device_tables.h).
//
// GB300 design: passes over the allocated-block list (ids 0..n-1 of the pool;
// the reference instead compacts the whole hash table, scene_mesh.cu:24-52).
//   count  one 128-thread CTA per block: the signs and the validity of the block
//          and its +x/+y/+z halo as bit rows (7 neighbour lookups, ballots), every
//          row's eight cubes classified from four bit rows, the block's triangles
//          summed, and those of its chunk of blocks.
//   scan   offsets of the blocks, a CTA per chunk on top of the chunks before it.
//   emit   restages with the values, lists the block's triangles in voxel order in
//          shared memory, then a lane per vertex: ten triangles per warp at a time,
//          written through shared memory as whole rows of floats.
// Output order is deterministic (block id, voxel index, table order); the
// reference appends with one global atomicAdd per triangle (scene_mesh.cu:231).
// Vertex arithmetic follows make_vertex (scene_mesh.cu:119-209) exactly.
//
// What bounds it: latency and issue, not memory (48,000 blocks of a scanned room
// read 98 MB of voxels and write 310 MB of triangles: 60 us at the measured
// bandwidth).  A 512-thread CTA per block with a thread per voxel held four
// blocks per SM through two dependent lookups, and interpolated twelve edges per
// voxel for all lanes of a warp, with the reference's thresholds in double: 36
// FP64 comparisons of 64 cycles each.  They are the same tests on floats (below).
// 48,000 blocks, 4.1 M triangles with normals: 2,513 -> 541 us a call (count 0.50 ->
// 0.11 ms, scan 50 -> 5 us, emit 1.9 -> 0.36 ms).
#include "gbf_device.cuh"
#include "gbf_kernels.h"

namespace gbf {

namespace {

// Triangle table of classic marching cubes (the public-domain Lorensen-Cline /
// Bourke table, identical to the reference's triangle_table so that the mesh
// topology matches bit for bit).  Packed: low nibble = number of triangles,
// then one nibble per edge index, three per triangle, in table order.  In global
// memory: the lanes of a warp look up different cubes, which the constant bank
// would serve one after the other.
__device__ const unsigned long long kTriPacked[256] = {
    0x0000000000000000ull, 0x0000000000003801ull, 0x0000000000009101ull, 0x0000000001893812ull,
    0x000000000000a211ull, 0x000000000a213802ull, 0x000000000920a292ull, 0x00000089a8a23823ull,
    0x0000000000002b31ull, 0x0000000000b82b02ull, 0x000000000b320912ull, 0x000000b89b912b13ull,
    0x0000000003ab1a32ull, 0x000000ab8a801a03ull, 0x0000009ab9b30933ull, 0x000000000b8aa892ull,
    0x0000000000008741ull, 0x0000000004370342ull, 0x0000000007489102ull, 0x0000001371749143ull,
    0x000000000748a212ull, 0x000000a214037433ull, 0x000000748209a293ull, 0x0004973727929a24ull,
    0x0000000002b37482ull, 0x00000040242b74b3ull, 0x000000b327481093ull, 0x0001292b9b49b744ull,
    0x000000487ab31a33ull, 0x0004b7401b41ab14ull, 0x00030bab9b098744ull, 0x000000ab99b4b743ull,
    0x0000000000004591ull, 0x0000000003804592ull, 0x0000000000514502ull, 0x0000005135384583ull,
    0x000000000459a212ull, 0x000000594a218033ull, 0x000000204245a253ull, 0x0008434535235a24ull,
    0x000000000b324592ull, 0x000000594b802b03ull, 0x000000b325104503ull, 0x000584b828525124ull,
    0x00000045931ab3a3ull, 0x000ab81a81805944ull, 0x00030bab5b050454ull, 0x000000b8aa858453ull,
    0x0000000009758792ull, 0x0000003753590393ull, 0x0000007517108703ull, 0x0000000007533512ull,
    0x00000021a7598793ull, 0x00037503505921a4ull, 0x00025a7585282084ull, 0x0000007533525a23ull,
    0x0000002b39875973ull, 0x000b720292797594ull, 0x000751871810b324ull, 0x00000051771b12b3ull,
    0x000b3a31a7588594ull, 0x0aba010b79050755ull, 0x07570805a30b0ab5ull, 0x0000000005b75ab2ull,
    0x00000000000056a1ull, 0x0000000006a53802ull, 0x0000000006a51092ull, 0x0000006a58913813ull,
    0x0000000001625612ull, 0x0000008036215613ull, 0x0000006206095693ull, 0x0008236252858954ull,
    0x00000000056ab322ull, 0x00000056a02b80b3ull, 0x0000006a5b329103ull, 0x000b892b92916a54ull,
    0x000000315356b363ull, 0x0006b51505b0b804ull, 0x0009505606306b34ull, 0x00000089bb969563ull,
    0x0000000008746a52ull, 0x000000a563740343ull, 0x0000007486a50913ull, 0x00049737179156a4ull,
    0x0000008741562163ull, 0x0007434036255214ull, 0x0006205605097484ull, 0x9626959234979375ull,
    0x00000056a4872b33ull, 0x000b720242746a54ull, 0x0006a5b328749104ull, 0x6a54b7b492b91295ull,
    0x0006b51535b37484ull, 0xb404b7b016b5b155ull, 0x74836b6305609505ull, 0x0009b7974b969564ull,
    0x000000000a4694a2ull, 0x000000380a946a43ull, 0x00000004606a10a3ull, 0x000a164686181384ull,
    0x0000004624219413ull, 0x0004629429218034ull, 0x0000000006244202ull, 0x0000006244282383ull,
    0x00000032b46a94a3ull, 0x0006a4a94b822804ull, 0x000a164606102b34ull, 0x1b8b12184a161465ull,
    0x00036b3196394694ull, 0x14641916b0181b85ull, 0x0000004600636b33ull, 0x00000000086b8462ull,
    0x000000a98a876a73ull, 0x000a76a907a03704ull, 0x0000818717a176a4ull, 0x00000037117a76a3ull,
    0x0007689818616214ull, 0x9373909761929625ull, 0x0000002066070873ull, 0x0000000002762372ull,
    0x00076898a86ab324ull, 0x7a9a76790b727025ull, 0xb32a767a18710815ull, 0x00017616a71b12b4ull,
    0x63136b6197686985ull, 0x00000000076b1902ull, 0x00006b0b36070874ull, 0x0000000000006b71ull,
    0x000000000000b671ull, 0x00000000067b8032ull, 0x00000000067b9102ull, 0x00000067b1389183ull,
    0x0000000007b621a2ull, 0x0000007b6803a213ull, 0x0000007b69a20923ull, 0x00089a38a3a27b64ull,
    0x0000000007263272ull, 0x0000000260678073ull, 0x0000009107326723ull, 0x0006788916812614ull,
    0x00000073171a67a3ull, 0x000801781a7167a4ull, 0x0007a69a0a707304ull, 0x0000009a88a7a673ull,
    0x00000000068b4862ull, 0x000000640603b633ull, 0x000000109648b683ull, 0x00063b1393696494ull,
    0x0000001a28b64863ull, 0x000640b60b03a214ull, 0x0009a2920b648b44ull, 0x36463b34923a39a5ull,
    0x0000002642483283ull, 0x0000000002642402ull, 0x0008346424320914ull, 0x0000006422414913ull,
    0x0001a66481683184ull, 0x00000040660a01a3ull, 0x39a9303a68343645ull, 0x0000000004a649a2ull,
    0x000000000b675942ull, 0x00000067b5943803ull, 0x000000b670451053ull, 0x00051345343867b4ull,
    0x000000b6721a4593ull, 0x000594380a217b64ull, 0x000204a24a45b674ull, 0x67b25a5234538435ull,
    0x0000009452673273ull, 0x0007862606804594ull, 0x0000450516732634ull, 0x8515848127868265ull,
    0x00073167161a4594ull, 0x459078701671a615ull, 0xa737a6a305a4a045ull, 0x000a84a458a7a674ull,
    0x00000098b9b65963ull, 0x000590650360b634ull, 0x000b65510b508b04ull, 0x0000001355363b63ull,
    0x00065b8b9b59a214ull, 0xa21965690b603b05ull, 0x52025a50865b58b5ull, 0x00035a3a25363b64ull,
    0x0002832658259854ull, 0x0000002600696593ull, 0x8262838650818515ull, 0x0000000006126512ull,
    0x698965683a616315ull, 0x00006505960a01a4ull, 0x000000000a658302ull, 0x00000000000065a1ull,
    0x000000000b57a5b2ull, 0x00000003857ba5b3ull, 0x000000091ba57b53ull, 0x0001381897ba57a4ull,
    0x00000015717b21b3ull, 0x000b275717213804ull, 0x0007b22097295794ull, 0x289823295b272575ull,
    0x000000573532a523ull, 0x00052a5782580284ull, 0x0002a37353a51094ull, 0x25752a2781292895ull,
    0x0000000005735312ull, 0x0000005711707803ull, 0x0000007355393093ull, 0x0000000007957892ull,
    0x0000008ba8a54853ull, 0x00003bba50b54054ull, 0x00054aba8a489104ull, 0x41314943b54a4ba5ull,
    0x0008548b25821524ull, 0xb151b2b543b0b405ull, 0x58b8545b29505205ull, 0x0000000003b25492ull,
    0x000483543253a524ull, 0x0000000244252a53ull, 0x910854583a532a35ull, 0x0002492914252a54ull,
    0x0000001533585483ull, 0x0000000005015402ull, 0x0005305093585484ull, 0x0000000000005491ull,
    0x000000ba9b947b43ull, 0x000ba97b97943804ull, 0x000b470414b1ba14ull, 0x4bab474a18434135ull,
    0x000219b294b97b44ull, 0x3801b2b197b94795ull, 0x00000004224b47b3ull, 0x00042343824b47b4ull,
    0x000947732972a924ull, 0x70207872a4797a95ull, 0xa040a1a472a3a735ull, 0x0000000004782a12ull,
    0x0000003177141943ull, 0x0001781807141944ull, 0x0000000003473042ull, 0x0000000000007841ull,
    0x0000000008ba8a92ull, 0x000000a9bb939033ull, 0x000000ba88a0a103ull, 0x000000000a3ba132ull,
    0x0000008b99b1b213ull, 0x0009b2921b939034ull, 0x000000000b08b202ull, 0x000000000000b231ull,
    0x00000098aa828323ull, 0x0000000002902a92ull, 0x0008a1810a828324ull, 0x0000000000002a11ull,
    0x0000000008198312ull, 0x0000000000001901ull, 0x0000000000008301ull, 0x0000000000000000ull,
};

constexpr int kHaloSide = 9;
constexpr int kHaloCells = kHaloSide * kHaloSide * kHaloSide;
constexpr int kHaloRows = kHaloSide * kHaloSide;
constexpr int kHaloExtra = kHaloCells - kBlockVoxels;  // 217 cells of the neighbours
constexpr int kMeshThreads = 128;
constexpr int kMeshMaxTris = kBlockVoxels * 5;

// Signs and validity of a block and its halo: row z * 9 + y has x = 0..7 in the
// low byte and x = 8 in `end`.
struct MeshBits {
    unsigned char ok[kHaloRows], ok_end[kHaloRows], neg[kHaloRows], neg_end[kHaloRows];
    int nb[8];
};

// Halo cell i < 217: the +x, +y and +z faces (64 each), the edges (8, 8, z), (8, y, 8), (x, 8, 8), the corner.
__device__ __forceinline__ void halo_cell(int i, int &x, int &y, int &z) {
    const int a = i & 7, b = (i >> 3) & 7;
    x = i < 64 ? 8 : a;
    y = i < 64 ? a : i < 128 ? 8 : b;
    z = i < 128 ? b : 8;
    if (i >= 192) {
        const int e = i - 192;
        x = e < 16 ? 8 : e < 24 ? a : 8;
        y = e < 8 || e >= 16 ? 8 : a;
        z = e < 8 ? a : 8;
    }
}

// The sdf of a voxel and whether it counts: weight != 0 (scene_mesh.cu:58), or weight > 1e-3 for colour
// (scene_mesh.cu:397; of the floats, those from 1e-3f, which lies just above 1e-3).
template <int LAYOUT>
__device__ __forceinline__ float mesh_sdf(const SessionView &sv, int id, int x, int y, int z, int mode, bool &ok, int &vi) {
    ok = false;
    vi = 0;
    if (id < 0) return 0.f;
    vi = id * kBlockVoxels + (z & 7) * 64 + (y & 7) * 8 + (x & 7);
    float w;
    const float s = load_sdf<LAYOUT>(sv, (size_t)vi, w);
    ok = mode == GBF_MESH_COLOUR ? w >= 1e-3f : w != 0.f;
    return s;
}

// Block `id` and its halo into the bit rows, and with VALUES the sdf (and for
// colour the colours) of every cell.  All threads; barriers at both ends.
template <int LAYOUT, bool VALUES>
__device__ __forceinline__ void stage_block(const SessionView &sv, int id, int mode, MeshBits &m, float *sdf,
                                            uchar4 *rgb) {
    const int tid = threadIdx.x, lane = tid & 31;
    __syncthreads();  // the previous block's use of the shared arrays
    if (tid < 8) {
        const int4 bc = sv.bcoord[id];
        m.nb[tid] = tid == 0 ? id : find_block(sv, bc.x + (tid & 1), bc.y + ((tid >> 1) & 1), bc.z + (tid >> 2));
    }
    __syncwarp();
    // the block itself: its loads go out beside the lookups
#pragma unroll
    for (int j = 0; j < kBlockVoxels / kMeshThreads; ++j) {
        const int li = tid + j * kMeshThreads, x = li & 7, y = (li >> 3) & 7, z = li >> 6;
        bool ok;
        int vi;
        const float s = mesh_sdf<LAYOUT>(sv, id, x, y, z, mode, ok, vi);
        const unsigned oks = __ballot_sync(0xffffffffu, ok), negs = __ballot_sync(0xffffffffu, s < 0);
        if (x == 0) {  // a warp covers four rows
            m.ok[z * 9 + y] = (unsigned char)(oks >> lane);
            m.neg[z * 9 + y] = (unsigned char)(negs >> lane);
        }
        if (VALUES) {
            const int c = x + 9 * y + 81 * z;
            sdf[c] = s;
            if (mode == GBF_MESH_COLOUR) rgb[c] = sv.vox_rgb[vi];
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int i = tid + j * kMeshThreads;
        const bool in = i < kHaloExtra;
        int x, y, z;
        halo_cell(min(i, kHaloExtra - 1), x, y, z);
        bool ok = false;
        int vi = 0, id2 = -1;
        float s = 0.f;
        if (in) {
            id2 = m.nb[(x >> 3) | ((y >> 3) << 1) | ((z >> 3) << 2)];
            s = mesh_sdf<LAYOUT>(sv, id2, x, y, z, mode, ok, vi);
        }
        const unsigned oks = __ballot_sync(0xffffffffu, ok), negs = __ballot_sync(0xffffffffu, s < 0);
        if (in) {
            const int row = z * 9 + y;
            if (x == 8) {
                m.ok_end[row] = ok;
                m.neg_end[row] = s < 0;
            } else if (x == 0) {  // the faces' rows of eight lie in lanes of a multiple of eight
                m.ok[row] = (unsigned char)(oks >> lane);
                m.neg[row] = (unsigned char)(negs >> lane);
            }
            if (VALUES) {
                const int c = x + 9 * y + 81 * z;
                sdf[c] = s;
                if (mode == GBF_MESH_COLOUR) rgb[c] = id2 >= 0 ? sv.vox_rgb[vi] : make_uchar4(0, 0, 0, 0);
            }
        }
    }
    __syncthreads();
}

// The cubes of voxel row r = 8 z + y (a thread each of the first 64): which of the
// eight have all their corners, and the four rows of signs that make them up.
struct CubeRow {
    unsigned valid, n00, n10, n01, n11;
    // corner order of make_vertex (scene_mesh.cu:73-101): (0,0) (1,0) (1,1) (0,1) below, then above
    __device__ __forceinline__ int cube(int x) const {
        const unsigned a = n00 >> x, b = n10 >> x, c = n01 >> x, d = n11 >> x;
        return (int)((a & 3u) | ((b & 2u) << 1) | ((b & 1u) << 3) | ((c & 3u) << 4) | ((d & 2u) << 5) | ((d & 1u) << 7));
    }
};
__device__ __forceinline__ CubeRow cube_row(const MeshBits &m, int r) {
    const int q = (r >> 3) * 9 + (r & 7);
    auto bits = [](const unsigned char *lo, const unsigned char *end, int i) { return (unsigned)lo[i] | ((unsigned)end[i] << 8); };
    CubeRow c;
    const unsigned ok = bits(m.ok, m.ok_end, q) & bits(m.ok, m.ok_end, q + 1) & bits(m.ok, m.ok_end, q + 9) &
                        bits(m.ok, m.ok_end, q + 10);
    c.valid = ok & (ok >> 1) & 0xffu;
    c.n00 = bits(m.neg, m.neg_end, q);
    c.n10 = bits(m.neg, m.neg_end, q + 1);
    c.n01 = bits(m.neg, m.neg_end, q + 9);
    c.n11 = bits(m.neg, m.neg_end, q + 10);
    // cubes with all corners on one side have no triangles
    const unsigned any = c.n00 | c.n10 | c.n01 | c.n11, all = c.n00 & c.n10 & c.n01 & c.n11;
    c.valid &= (any | (any >> 1)) & ~(all & (all >> 1));
    return c;
}

// The CTAs of a launch take its n blocks from a counter: a block has from none to some
// 300 triangles, and with the blocks shared out beforehand the CTAs that started last
// worked on while the others' places stood empty (48,000 blocks: 407 -> 354 us).  The
// counter is read a block ahead, so that its answer is there in time; a launch with
// a CTA per block needs none.
struct BlockQueue {
    int *counter;
    int n;
    bool lead;
    int ahead = 0, turn = 0;
    __device__ __forceinline__ BlockQueue(int *c, int blocks, bool l) : counter(c), n(blocks), lead(l && blocks > (int)gridDim.x) {
        if (lead) ahead = (int)gridDim.x + atomicAdd(counter, 1);
    }
    // all threads; slot: two words of shared memory (a thread that is late to read one
    // has passed no further barrier, and the word is written again only after two)
    __device__ __forceinline__ int next(int *slot) {
        if (n <= (int)gridDim.x) return n;
        if (lead) {
            slot[turn] = ahead;
            ahead = (int)gridDim.x + atomicAdd(counter, 1);
        }
        __syncthreads();
        const int b = slot[turn];
        turn ^= 1;
        return b;
    }
};

// Blocks per chunk of the offset scan (at most kMeshChunks chunks).
__host__ __device__ __forceinline__ int mesh_chunk(int pool) {
    const int c = (pool + kMeshChunks - 1) / kMeshChunks;
    return c <= 1024 ? 1024 : (c + 1023) / 1024 * 1024;
}

template <int LAYOUT>
__global__ void __launch_bounds__(kMeshThreads, 16) mesh_count_kernel(const SessionView *__restrict__ svs, int mode, int *counts) {
    chain_begin();
    const SessionView &sv = svs[0];
    const int n = min(sv.ctr[C_NUSED], sv.pool), chunk = mesh_chunk(sv.pool);
    __shared__ MeshBits m;
    __shared__ unsigned char tris[256];
    __shared__ int part[2];
    for (int i = threadIdx.x; i < 256; i += kMeshThreads) tris[i] = (unsigned char)(kTriPacked[i] & 0xf);
    for (int b = blockIdx.x; b < n; b += gridDim.x) {
        stage_block<LAYOUT, false>(sv, b, mode, m, nullptr, nullptr);
        if (threadIdx.x < 64) {
            const CubeRow row = cube_row(m, threadIdx.x);
            int t = 0;
            for (unsigned v = row.valid; v; v &= v - 1) t += tris[row.cube(__ffs(v) - 1)];
            __syncwarp();
            t = __reduce_add_sync(0xffffffffu, t);
            if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = t;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const int total = part[0] + part[1];
            counts[b] = total;
            if (total) atomicAdd(sv.mesh_sums + b / chunk, total);
        }
    }
}

// Exclusive scan of counts[0..n) in place, the total into counts[n] and
// C_MESH_TRIS.  A CTA per chunk: the sums of the chunks before it, then its own
// counts, 1024 at a time.  (One CTA over all the blocks took 6.3 us for 6,000.)
__global__ void __launch_bounds__(1024) mesh_scan_kernel(const SessionView *__restrict__ svs, int *counts) {
    chain_begin();
    const SessionView &sv = svs[0];
    const int n = min(sv.ctr[C_NUSED], sv.pool), chunk = mesh_chunk(sv.pool);
    const int first = blockIdx.x * chunk, end = min(n, first + chunk);
    if (first >= n && blockIdx.x > 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ int wsum[32];
    __shared__ int carry;
    const int *sums = sv.mesh_sums;
    int before = tid < (int)blockIdx.x ? sums[tid] : 0;
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) wsum[warp] = before;
    __syncthreads();
    if (warp == 0) {
        const int t = __reduce_add_sync(0xffffffffu, wsum[lane]);
        if (lane == 0) carry = t;
    }
    __syncthreads();
    for (int base = first; base < end; base += 1024) {
        const int i = base + tid, v = i < end ? counts[i] : 0;
        int x = v;  // inclusive warp scan
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, off);
            if (lane >= off) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        int w = wsum[lane];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, off);
            if (lane >= off) w += y;
        }
        const int c = carry, total = __shfl_sync(0xffffffffu, w, 31);
        const int prior = __shfl_sync(0xffffffffu, w, warp ? warp - 1 : 0);
        if (i < end) counts[i] = c + (warp ? prior : 0) + (x - v);
        __syncthreads();
        if (tid == 0) carry = c + total;
        __syncthreads();
    }
    if (tid == 0 && end >= n) {
        counts[n] = carry;
        sv.ctr[C_MESH_TRIS] = carry;
    }
}

// interpolate_sdf (scene_mesh.cu:108-117).  The reference's thresholds compare in
// double against 1e-6; of the floats, 1e-6f is the largest below it.
__device__ __forceinline__ float edge_point(float v1, float v2) {
    if (fabsf(0 - v1) <= 1e-6f) return 0.f;
    if (fabsf(0 - v2) <= 1e-6f) return 1.f;
    if (fabsf(v1 - v2) <= 1e-6f) return 0.f;
    return (0 - v1) / (v2 - v1);
}

struct MeshEmit {
    MeshBits bits;
    float sdf[kHaloCells];
    unsigned short tri[kMeshMaxTris];  // voxel | triangle of its cube << 9
    unsigned char cube[kBlockVoxels];
    int part[2], next[2];
    float out[kMeshThreads / 32][2][90];  // a warp's ten triangles: vertices, normals
};

template <int LAYOUT, int MODE>
__global__ void __launch_bounds__(kMeshThreads, 10) mesh_emit_kernel(const SessionView *__restrict__ svs, const int *offsets,
                                                                     float *vtx, void *attr, long long max_tris) {
    chain_begin();
    const SessionView &sv = svs[0];
    const int n = min(sv.ctr[C_NUSED], sv.pool);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ MeshEmit sm;
    __shared__ uchar4 rgb[MODE == GBF_MESH_COLOUR ? kHaloCells : 1];
    BlockQueue queue(sv.mesh_sums + kMeshChunks, n, tid == 0);
    for (int b = blockIdx.x; b < n; b = queue.next(sm.next)) {
        const int first = offsets[b];
        const int count = (int)min((long long)(offsets[b + 1] - first), max_tris - first);
        if (count <= 0) continue;  // uniform per CTA
        stage_block<LAYOUT, true>(sv, b, MODE, sm.bits, sm.sdf, rgb);
        // the block's triangles in voxel order
        CubeRow row;
        int t = 0, x = 0;
        if (tid < 64) {
            row = cube_row(sm.bits, tid);
            for (unsigned v = row.valid; v; v &= v - 1) {
                const int at = __ffs(v) - 1, ci = row.cube(at);
                sm.cube[tid * 8 + at] = (unsigned char)ci;
                t += (int)(kTriPacked[ci] & 0xf);
            }
            __syncwarp();
            x = t;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, off);
                if (lane >= off) x += y;
            }
            if (lane == 31) sm.part[warp] = x;
        }
        __syncthreads();
        if (tid < 64) {
            int at = x - t + (warp ? sm.part[0] : 0);
            for (unsigned v = row.valid; v; v &= v - 1) {
                const int li = tid * 8 + __ffs(v) - 1, k = (int)(kTriPacked[sm.cube[li]] & 0xf);
                for (int i = 0; i < k; ++i) sm.tri[at++] = (unsigned short)(li | (i << 9));
            }
        }
        __syncthreads();
        const int4 bc = sv.bcoord[b];
        const float voxel = sv.voxel;
        for (int base = warp * 10; base < count; base += 10 * (kMeshThreads / 32)) {
            // lane 3 k + q < 30: vertex q of triangle base + k
            const int k = lane / 3, q = lane - 3 * k, last = min(10, count - base);
            const bool on = lane < 30 && k < last;
            const unsigned entry = sm.tri[base + (on ? k : 0)];
            const int li = entry & 511, lx = li & 7, ly = (li >> 3) & 7, lz = li >> 6;
            const unsigned long long packed = kTriPacked[sm.cube[li]];
            const int e = (int)(packed >> (4 + 12 * (entry >> 9) + 4 * (on ? q : 0))) & 0xf;
            // edge e runs from corner c0 to c1 (scene_mesh.cu:147-205)
            const int c0 = e < 8 ? e : e - 8, c1 = e < 8 ? (e & 4) | ((e + 1) & 3) : e - 4;
            auto cell = [&](int c) {
                const int dx = ((c & 3) == 1 || (c & 3) == 2) ? 1 : 0, dy = (c & 3) >> 1, dz = c >> 2;
                return (lx + dx) + 9 * (ly + dy) + 81 * (lz + dz);
            };
            const int cell0 = cell(c0);
            const float val = edge_point(sm.sdf[cell0], sm.sdf[cell(c1)]);
            const int kind = e & 3;
            const float far = (kind == 1 || kind == 2) ? 1.f : 0.f;  // corner x of the edges along z, and of edges 1, 2
            float ox, oy, oz;
            if (e < 8) {
                ox = kind == 0 ? val : kind == 2 ? 1 - val : far;
                oy = kind == 1 ? val : kind == 3 ? 1 - val : kind == 2 ? 1.f : 0.f;
                oz = e < 4 ? 0.f : 1.f;
            } else {
                ox = far;
                oy = kind >= 2 ? 1.f : 0.f;
                oz = val;
            }
            const float px = ((float)(bc.x * 8 + lx) + ox) * voxel, py = ((float)(bc.y * 8 + ly) + oy) * voxel,
                        pz = ((float)(bc.z * 8 + lz) + oz) * voxel;
            float *out = sm.out[warp][0];
            if (lane < 30) {
                out[3 * lane] = px;
                out[3 * lane + 1] = py;
                out[3 * lane + 2] = pz;
            }
            __syncwarp();
            const long long at = (long long)first + base;  // the warp's first triangle
            for (int i = lane; i < 9 * last; i += 32) vtx[at * 9 + i] = out[i];
            if (MODE == GBF_MESH_NORMAL) {
                const float *A = out + 9 * min(k, 9);
                const float3 u = make_float3(A[3] - A[0], A[4] - A[1], A[5] - A[2]);
                const float3 v = make_float3(A[6] - A[0], A[7] - A[1], A[8] - A[2]);
                const float3 nn = cross3(u, v);
                const float l = norm3(nn.x, nn.y, nn.z);
                // lane q divides component q, which is component q of all three vertices' normals
                const float c = (q == 0 ? nn.x : q == 1 ? nn.y : nn.z) / l;
                float *nrm = sm.out[warp][1];
                if (lane < 30) nrm[9 * k + q] = nrm[9 * k + 3 + q] = nrm[9 * k + 6 + q] = c;
                __syncwarp();
                float *na = static_cast<float *>(attr);
                for (int i = lane; i < 9 * last; i += 32) na[at * 9 + i] = nrm[i];
            } else if (MODE == GBF_MESH_COLOUR && on) {
                // edges 0-7 take corner e's colour, 8-11 corner e-8 (scene_mesh.cu:526-549)
                const uchar4 col = rgb[cell0];
                unsigned char *ca = static_cast<unsigned char *>(attr) + (at * 3 + lane) * 3;
                ca[0] = col.x;
                ca[1] = col.y;
                ca[2] = col.z;
            }
            __syncwarp();
        }
    }
}

template <int LAYOUT>
void launch_mesh_layout(const SessionView *d_sv, const Extent &ex, int mode, float *vtx, void *attr, long long max_tris,
                        int *counts, cudaStream_t st) {
    // the device alone knows how many blocks there are: 16 CTAs per SM, all resident,
    // stride over them to count, twice as many as are resident queue for them to emit
    // (2,000 blocks, a pass over 2,432 CTAs with the blocks shared out 57 us, 1,520 with the queue 67, 3,040 55)
    const int g = min(max(ex.max_pool, 1), 152 * 16), ge = min(max(ex.max_pool, 1), 152 * 20);
    const int chunks = (ex.max_pool + mesh_chunk(ex.max_pool) - 1) / mesh_chunk(ex.max_pool);
    launch_kernel(mesh_count_kernel<LAYOUT>, g, kMeshThreads, ex.chain, st, d_sv, mode, counts);
    launch_kernel(mesh_scan_kernel, max(chunks, 1), 1024, ex.chain, st, d_sv, counts);
    if (mode == GBF_MESH_VERTEX)
        launch_kernel(mesh_emit_kernel<LAYOUT, GBF_MESH_VERTEX>, ge, kMeshThreads, ex.chain, st, d_sv, counts, vtx, attr,
                      max_tris);
    else if (mode == GBF_MESH_NORMAL)
        launch_kernel(mesh_emit_kernel<LAYOUT, GBF_MESH_NORMAL>, ge, kMeshThreads, ex.chain, st, d_sv, counts, vtx, attr,
                      max_tris);
    else
        launch_kernel(mesh_emit_kernel<LAYOUT, GBF_MESH_COLOUR>, ge, kMeshThreads, ex.chain, st, d_sv, counts, vtx, attr,
                      max_tris);
}

}  // namespace

void launch_mesh(const SessionView *d_sv, const Extent &ex, int layout, int mode, float *vtx, void *attr,
                 long long max_tris, int *counts, int *chunk_sums, cudaStream_t st) {
    cudaMemsetAsync(chunk_sums, 0, kMeshWords * sizeof(int), st);
    if (layout == GBF_VOXEL_REF) launch_mesh_layout<GBF_VOXEL_REF>(d_sv, ex, mode, vtx, attr, max_tris, counts, st);
    else if (layout == GBF_VOXEL_HALF) launch_mesh_layout<GBF_VOXEL_HALF>(d_sv, ex, mode, vtx, attr, max_tris, counts, st);
    else launch_mesh_layout<GBF_VOXEL_SNORM>(d_sv, ex, mode, vtx, attr, max_tris, counts, st);
}

}  // namespace gbf
