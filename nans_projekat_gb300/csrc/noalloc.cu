// Allocation-free sequential-impulse solve of one scene's contact list.
//
// Who needs this: callers that must not allocate GPU memory after start-up. The reference's
// own host is the model case -- its platform layer reserves all memory once and hands it to
// the hot-reloaded simulation library every frame, and the library is not supposed to grab
// memory of its own while a frame runs. Engines with a fixed GPU memory budget owned by the
// application's pool, and real-time loops that forbid allocation after initialisation for
// latency reasons, are in the same position. nans_world_* cannot serve them: a world
// allocates its buffers with cudaMalloc.
//
// This entry point runs the same solve as the world's solver (waves of contacts that touch
// disjoint bodies, the reference's operation order, bit-identical results) on device
// buffers that the caller owns, and keeps all of its scratch in one file-scope device
// array of fixed size. It never calls cudaMalloc, cudaFree or an allocating library routine.
//
// Limits: at most kMaxBodies bodies and kMaxContacts contacts per call (larger requests are
// rejected with NANS_ERR_INVALID_ARGUMENT). The array lives on every GPU that loads the
// library until the process exits, and every call shares it: calls whose kernels overlap on
// the GPU (two streams, two threads) race on it, so callers must serialise them. What must
// start at zero is cleared on every call.
#include <cuda_runtime.h>
#include <mutex>

#include "../../include/nans_gb300.h"
#include "nans_solve.cuh"

namespace
{

constexpr int kMaxBodies = 16384;
constexpr int kMaxContacts = 16384;
constexpr int kThreads = 512;

// Scratch layout (4-byte words):
//   [0]                          error word (bit 0: a contact names a body outside the scene)
//   [1]                          waves of the last ordered list
//   ab[kMaxContacts]             the contact's bodies: A, (B + 1) << 16 (B = -1: the floor), ~0: skipped
//   next[2 * kMaxContacts]       the next contact in list order that touches A / B, or -1; in a list
//                                that is ordered first: the contacts in wave order, then the waves' ends
//   k[kMaxContacts * 36]         velocity-independent constants, 9 float4 per contact (ordered lists:
//                                9 rows of kMaxContacts, in wave order)
constexpr size_t kOffAb = 4;
constexpr size_t kOffNext = kOffAb + kMaxContacts;
constexpr size_t kOffOrder = kOffNext, kOffWend = kOffNext + kMaxContacts;
constexpr size_t kOffK = kOffNext + 2 * (size_t)kMaxContacts; // multiple of 4 words: float4-aligned
constexpr size_t kScratchWords = kOffK + (size_t)36 * kMaxContacts;
constexpr unsigned kSkipped = 0xffffffffu;
static_assert(kOffK % 4 == 0, "constants must be 16-byte aligned");

// About 2.5 MB, resident on each device that loads the library.
static __device__ __align__(256) unsigned g_solve_scratch[kScratchWords];

// Lists of up to kOneLaunch contacts are solved by one launch (k_solve_static), longer ones by four:
// decode, order, constants, waves. In a long list one block's gathers of 96-byte records and 144-byte
// constants cost more than the launches. A call in one launch and in four: 80 and 88 us at 600 contacts,
// 91 and 89 at 1,000, 103 and 96 at 2,000, 164 and 111 at 5,000, 362 and 173 at 14,161.
constexpr int kOneLaunch = 1024;

// Dynamic shared memory of the single launch: while the order is worked out, per body the end of its
// contacts in the list that follows, both sides of every contact grouped by body; while the waves run,
// two wave lists and, for up to kSmallCache bodies, the velocities. The contacts' open predecessors
// in both.
constexpr int kSmallCache = 6000;
size_t one_launch_smem(int nbodies, int npairs)
{
    const size_t order = (size_t)(nbodies + 1) * sizeof(int) + 2 * (size_t)npairs * sizeof(unsigned short);
    const size_t waves = 2 * (size_t)npairs * sizeof(unsigned short) +
                         (nbodies <= kSmallCache ? (size_t)nbodies * 6 * sizeof(float) : 0) + 16;
    return (((size_t)npairs + 15) & ~(size_t)15) + (order > waves ? order : waves);
}
// Of the ordering: the open predecessors, the neighbours of both sides, per body the end of its
// contacts, and both sides grouped by body (then the order).
size_t order_smem(int nbodies, int npairs)
{
    return (((size_t)npairs + 15) & ~(size_t)15) + 4 * (size_t)npairs * sizeof(unsigned short) +
           (size_t)(nbodies + 1) * sizeof(int);
}
// Of the waves: the velocities of up to kWaveCache bodies.
constexpr int kWaveCache = 9000;
size_t waves_smem(int nbodies) { return nbodies <= kWaveCache ? (size_t)nbodies * 6 * sizeof(float) : 0; }
constexpr size_t kSmemMax = 227 * 1024, kDynamicMax = kSmemMax - 4096; // some is static
static_assert(kMaxContacts + 4 * (size_t)kMaxContacts * 2 + (kMaxBodies + 1) * 4 <= kDynamicMax, "ordering's shared memory");
static_assert((size_t)kWaveCache * 24 <= kDynamicMax, "waves' shared memory");

// Device address of g_solve_scratch per device, looked up once with that device current. A
// cudaDeviceReset destroys the device's context, and the library's module, with the array in
// it, is loaded again in the next context, possibly at another address. So each entry also keeps
// the id of the context it was taken in, and the address is looked up again when the device's
// current context has another id.
struct ScratchAddr
{
    void *ptr;
    unsigned long long ctx;
};
std::mutex g_setup_mutex;
ScratchAddr g_scratch_addr[64] = {};

typedef int (*CtxGetCurrentFn)(void **);
typedef int (*CtxGetIdFn)(void *, unsigned long long *);

// Id of the calling thread's current context through the driver's cuCtxGetCurrent and
// cuCtxGetId (CUDA 12.0 and later); 0 when the driver does not provide them. Call with
// g_setup_mutex held.
unsigned long long current_context_id()
{
    static bool looked_up = false;
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    if (!looked_up)
    {
        looked_up = true;
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = (CtxGetCurrentFn)f;
        f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = (CtxGetIdFn)f;
    }
    void *ctx = nullptr;
    unsigned long long id = 0;
    if (get_current && get_id && get_current(&ctx) == 0 && ctx && get_id(ctx, &id) == 0)
        return id;
    return 0;
}

struct Floor
{
    v3 p, v, w;
    float invm, invi;
};

struct Bodies
{
    const float *pos, *mass, *moi;
    float *vel, *omg;
    int nbodies, ncubes;
};

__device__ __forceinline__ v3 ld3(const float *a, int i) { return mk3(a[3 * i], a[3 * i + 1], a[3 * i + 2]); }
__device__ __forceinline__ void st3(float *a, int i, v3 v)
{
    a[3 * i] = v.x;
    a[3 * i + 1] = v.y;
    a[3 * i + 2] = v.z;
}

// Body index of each side of a contact record (code/nans.h:338-372); -1 = the floor,
// -2 = a contact that is skipped and reported: an index outside the scene, or both sides the
// same body.
__device__ __forceinline__ void sides(const Bodies &B, const nans_contact_pair &c, int &a, int &b)
{
    int t = c.Type;
    bool a_sphere = (t == NANS_SS || t == NANS_SF);
    bool b_floor = (t == NANS_CF || t == NANS_SF);
    bool b_sphere = (t == NANS_CS || t == NANS_SS);
    a = a_sphere ? B.ncubes + c.IndexA : c.IndexA;
    b = b_floor ? -1 : (b_sphere ? B.ncubes + c.IndexB : c.IndexB);
    int nsph = B.nbodies - B.ncubes;
    bool a_ok = c.IndexA >= 0 && (a_sphere ? c.IndexA < nsph : c.IndexA < B.ncubes);
    bool b_ok = b_floor || (c.IndexB >= 0 && (b_sphere ? c.IndexB < nsph : c.IndexB < B.ncubes));
    // a contact whose two sides are one body: the sequential solve would interleave the two
    // sides' updates on that body, which the per-side loads and stores below cannot reproduce
    if (t < 0 || t > 4 || !a_ok || !b_ok || (b >= 0 && a == b))
        a = b = -2;
}

// Constants of contact c between bodies a and b (-1: the floor).
__device__ __forceinline__ void contact_record(const Bodies &B, const Floor &F, const nans_contact_pair &c, int a, int b,
                                               float dt, float4 *q)
{
    // velocity-independent part of Constraint (code/nans.cpp:1023-1174)
    v3 n = normalize3(mk3(c.N[0], c.N[1], c.N[2]));
    v3 pa = ld3(B.pos, a);
    v3 pb = (b >= 0) ? ld3(B.pos, b) : F.p;
    float invi1 = 1.0f / B.moi[a], invm1 = 1.0f / B.mass[a];
    float invi2 = (b >= 0) ? 1.0f / B.moi[b] : F.invi;
    float invm2 = (b >= 0) ? 1.0f / B.mass[b] : F.invm;
    if (eq3(n, mk3(0.0f, 0.0f, 0.0f)))
        n = normalize3(pb - pa);
    v3 r1 = mk3(c.PointA[0], c.PointA[1], c.PointA[2]) - pa;
    v3 r2 = mk3(c.PointB[0], c.PointB[1], c.PointB[2]) - pb;
    v3 t1 = (n.x >= 0.57735f) ? mk3(n.y, -n.x, 0.0f) : mk3(0.0f, n.z, -n.y);
    v3 t2 = cross3(n, t1);
    float depth = dot3((pa + r1) - (pb + r2), n);
    v3 rn1 = cross3(r1, n), rn2 = cross3(r2, n);
    float jn = invm1 + invm2;
    jn = jn + (invi1 * dot3(rn1, rn1) - invi2 * dot3(-rn2, -rn2));
    jn = 1.0f / jn;
    float bias0 = (-0.3f) / dt * depth;
    v3 r1t1 = cross3(r1, t1), r2t1 = cross3(r2, t1), r1t2 = cross3(r1, t2), r2t2 = cross3(r2, t2);
    float jt1 = invm1 + invm2;
    jt1 = jt1 + (invi1 * dot3(r1t1, r1t1) - invi2 * dot3(-r2t1, -r2t1));
    jt1 = 1.0f / jt1;
    float jt2 = invm1 + invm2;
    jt2 = jt2 + (invi1 * dot3(r1t2, r1t2) - invi2 * dot3(-r2t2, -r2t2));
    jt2 = 1.0f / jt2;
    q[0] = make_float4(n.x, n.y, n.z, jn);
    q[1] = make_float4(t1.x, t1.y, t1.z, jt1);
    q[2] = make_float4(t2.x, t2.y, t2.z, jt2);
    q[3] = make_float4(rn1.x, rn1.y, rn1.z, bias0);
    q[4] = make_float4(rn2.x, rn2.y, rn2.z, invm1);
    q[5] = make_float4(r1t1.x, r1t1.y, r1t1.z, invm2);
    q[6] = make_float4(r2t1.x, r2t1.y, r2t1.z, invi1);
    q[7] = make_float4(r1t2.x, r1t2.y, r1t2.z, invi2);
    q[8] = make_float4(r2t2.x, r2t2.y, r2t2.z, 0.0f);
}

// One contact's impulses on the velocities V, W (Constraint, code/nans.cpp:1149-1328).
__device__ __forceinline__ void solve_one(const Floor &F, const float4 (&q)[9], float *V, float *W, int a, int b, float cr,
                                          double c2, const nans::FBound &fb, int iters)
{
    const v3 n3 = xyz(q[0]), t1 = xyz(q[1]), t2 = xyz(q[2]);
    const float jn = q[0].w, jt1 = q[1].w, jt2 = q[2].w;
    const float invm1 = q[4].w, invm2 = q[5].w, invi1 = q[6].w, invi2 = q[7].w;
    v3 V1 = ld3(V, a), W1 = ld3(W, a);
    v3 V2 = (b >= 0) ? ld3(V, b) : F.v;
    v3 W2 = (b >= 0) ? ld3(W, b) : F.w;
    const float jdvn = dot3(((V1 + cross3(W1, n3)) - V2) - cross3(W2, n3), n3);
    const float jdvt1 = dot3(((V1 + cross3(W1, t1)) - V2) - cross3(W2, t1), t1);
    const float jdvt2 = dot3(((V1 + cross3(W1, t2)) - V2) - cross3(W2, t2), t2);
    const float bias = q[3].w + cr * jdvn;
    float sn = 0.0f, st1 = 0.0f, st2 = 0.0f, dn = 0.0f, dt1 = 0.0f, dt2 = 0.0f;
    if (!nans::impulse_direct((-jdvn + bias) * jn, (-jdvt1) * jt1, (-jdvt2) * jt2, c2, fb, iters, dn, dt1, dt2))
    {
        sn = st1 = st2 = dn = dt1 = dt2 = 0.0f;
        nans::impulse_loop<false>(jdvn, jdvt1, jdvt2, bias, jn, jt1, jt2, c2, fb, iters, sn, st1, st2, dn, dt1,
                                  dt2);
    }
    const v3 li = dn * n3, lt1 = dt1 * t1, lt2 = dt2 * t2;
    V1 = V1 + invm1 * li;
    W1 = W1 + invi1 * (dn * xyz(q[3]));
    V1 = V1 + invm1 * lt1;
    W1 = W1 + invi1 * (dt1 * xyz(q[5]));
    V1 = V1 + invm1 * lt2;
    W1 = W1 + invi1 * (dt2 * xyz(q[7]));
    st3(V, a, V1);
    st3(W, a, W1);
    if (b >= 0)
    {
        V2 = V2 - invm2 * li;
        W2 = W2 - invi2 * (dn * xyz(q[4]));
        V2 = V2 - invm2 * lt1;
        W2 = W2 - invi2 * (dt1 * xyz(q[6]));
        V2 = V2 - invm2 * lt2;
        W2 = W2 - invi2 * (dt2 * xyz(q[8]));
        st3(V, b, V2);
        st3(W, b, W2);
    }
}

// The solve by waves without labels: a contact may run when the contacts before it in the list that
// touch its bodies have run, and contacts that touch disjoint bodies commute exactly (the floor is
// never written), so every contact whose open predecessors reach zero joins the next wave. One block:
//   (1) the contacts' bodies, and per body how many contacts touch it;
//   (2) each body's contacts side by side (a counting sort by body, order within a body free);
//   (3) per contact and side, its neighbours in list order among its body's contacts, by looking
//       through them (a few, at most kOneLaunch), and the velocity-independent constants;
//   (4) the waves, on a shared-memory copy of the velocities where they fit.
// Bound by the waves' chain: a barrier, the constants' load (L2) and the impulses each. The form before
// labelled the waves by one thread from global memory and ran the loop's friction bound in double
// precision: 325 contacts of 125 bodies (18 waves) took 193 us a call with the caller's two copies and
// now take 85.
__global__ void __launch_bounds__(kThreads) k_solve_static(unsigned *scratch, Bodies B, Floor F,
                                                            const nans_contact_pair *pairs, int npairs, float cr,
                                                            float cf, int iters, float dt)
{
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned char *const open = smem; // predecessors a contact still waits for
    unsigned char *const rest = smem + (((size_t)npairs + 15) & ~(size_t)15);
    unsigned *ab = scratch + kOffAb;
    int *next = reinterpret_cast<int *>(scratch + kOffNext);
    float4 *K = reinterpret_cast<float4 *>(scratch + kOffK);
    __shared__ int sh[32];
    __shared__ int s_n[2];
    const int tid = threadIdx.x, nb = B.nbodies;
    int *const end = reinterpret_cast<int *>(rest); // per body: where its contacts end (then begin)
    unsigned short *const of = reinterpret_cast<unsigned short *>(end + nb + 1);
    if (tid == 0)
        scratch[0] = 0u;
    for (int i = tid; i <= nb; i += kThreads)
        end[i] = 0;
    __syncthreads();
    // (1)
    bool bad = false;
#pragma unroll 4
    for (int k = tid; k < npairs; k += kThreads)
    {
        int a, b;
        sides(B, pairs[k], a, b);
        unsigned v = kSkipped;
        if (a == -2)
            bad = true;
        else
        {
            v = (unsigned)a | ((unsigned)(b + 1) << 16);
            atomicAdd(end + a, 1);
            if (b >= 0)
                atomicAdd(end + b, 1);
        }
        ab[k] = v;
    }
    if (bad)
        scratch[0] = 1u;
    __syncthreads();
    // (2) exclusive prefix of the counts; the placement moves each body's cursor to its end
    int carry = 0;
    for (int base = 0; base < nb; base += kThreads)
    {
        const int i = base + tid;
        int tot;
        const int pre = nans::block_scan_excl(i < nb ? end[i] : 0, sh, &tot);
        if (i < nb)
            end[i] = carry + pre;
        carry += tot;
    }
    __syncthreads();
    for (int k = tid; k < npairs; k += kThreads)
    {
        const unsigned v = ab[k];
        if (v == kSkipped)
            continue;
        const int a = v & 0xffffu, b = (int)(v >> 16) - 1;
        of[atomicAdd(end + a, 1)] = (unsigned short)k;
        if (b >= 0)
            of[atomicAdd(end + b, 1)] = (unsigned short)k;
    }
    __syncthreads();
    // (3)
    for (int k = tid; k < npairs; k += kThreads)
    {
        const unsigned v = ab[k];
        if (v == kSkipped)
        {
            open[k] = 255;
            continue;
        }
        const int a = v & 0xffffu, b = (int)(v >> 16) - 1;
        int before = 0;
        for (int side = 0; side < 2; ++side)
        {
            const int body = side ? b : a;
            int nx = 0x7fffffff;
            bool has = false;
            if (body >= 0)
                for (int j = body ? end[body - 1] : 0; j < end[body]; ++j)
                {
                    const int o = of[j];
                    has = has || o < k;
                    if (o > k && o < nx)
                        nx = o;
                }
            before += has;
            next[2 * k + side] = nx == 0x7fffffff ? -1 : nx;
        }
        open[k] = (unsigned char)before;
        float4 q[9];
        contact_record(B, F, pairs[k], a, b, dt, q);
#pragma unroll
        for (int j = 0; j < 9; ++j)
            K[(size_t)9 * k + j] = q[j];
    }
    __syncthreads(); // the bodies' contact lists' memory becomes the wave lists and the velocities
    // (4)
    unsigned short *list = reinterpret_cast<unsigned short *>(rest), *list2 = list + npairs;
    float *const vel = reinterpret_cast<float *>(rest + ((4 * (size_t)npairs + 15) & ~(size_t)15)), *const omg = vel + 3 * nb;
    const bool cached = nb <= kSmallCache;
    float *const V = cached ? vel : B.vel, *const W = cached ? omg : B.omg;
    if (cached)
        for (int i = tid; i < 3 * nb; i += kThreads)
        {
            vel[i] = B.vel[i];
            omg[i] = B.omg[i];
        }
    if (tid < 2)
        s_n[tid] = 0;
    __syncthreads();
    for (int k = tid; k < npairs; k += kThreads)
        if (open[k] == 0)
            list[atomicAdd(&s_n[0], 1)] = (unsigned short)k;
    __syncthreads();
    const double c2 = nans::friction_scale(cf);
    const nans::FBound fb = nans::fbound_split(c2);
    for (int cur = 0;; cur ^= 1)
    {
        const int n = s_n[cur];
        if (n == 0)
            break;
        for (int i = tid; i < n; i += kThreads)
        {
            const int k = list[i];
            const unsigned v = ab[k];
            const int a = v & 0xffffu, b = (int)(v >> 16) - 1;
            const int na = next[2 * k], nx = next[2 * k + 1];
            float4 q[9];
#pragma unroll
            for (int j = 0; j < 9; ++j)
                q[j] = K[(size_t)9 * k + j];
            solve_one(F, q, V, W, a, b, cr, c2, fb, iters);
            // the contacts that waited for this one alone make the next wave
            for (int side = 0; side < 2; ++side)
            {
                const int s = side ? nx : na;
                if (s < 0)
                    continue;
                // a byte of the word that holds it: no borrow, a waiting contact's count is at least 1
                const unsigned shift = 8u * (s & 3);
                const unsigned old = atomicSub(reinterpret_cast<unsigned *>(open) + (s >> 2), 1u << shift);
                if (((old >> shift) & 255u) == 1u)
                    list2[atomicAdd(&s_n[cur ^ 1], 1)] = (unsigned short)s;
            }
        }
        __syncthreads();
        if (tid == 0)
            s_n[cur] = 0;
        unsigned short *const t = list;
        list = list2;
        list2 = t;
        __syncthreads();
    }
    if (cached)
        for (int i = tid; i < 3 * nb; i += kThreads)
        {
            B.vel[i] = vel[i];
            B.omg[i] = omg[i];
        }
}

// The same for longer lists in four launches. The bodies of each contact, coalesced for the next one.
__global__ void __launch_bounds__(256) k_static_decode(unsigned *scratch, Bodies B, const nans_contact_pair *pairs,
                                                        int npairs)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= npairs)
        return;
    int a, b;
    sides(B, pairs[k], a, b);
    if (a == -2)
        scratch[0] = 1u;
    scratch[kOffAb + k] = a == -2 ? kSkipped : ((unsigned)a | ((unsigned)(b + 1) << 16));
}

// The contacts in wave order and the waves' ends, one block: steps (1) to (3) of k_solve_static without
// the constants, then its waves without the solving, all in shared memory. Bound by the waves' chain of
// two barriers and an atomic each.
//
// A body of more than kHubContacts contacts (a ground plate modelled as a body, a container) has its
// contacts marked in a bitmap, where the next one is a bit scan away, in place of a look through them
// all for each: a call of 16,384 contacts of one pair 44.4 -> 30.8 ms, of one body with the ground 22.4
// -> 15.6, of 4,000 4.25 -> 3.86. The line is where a bitmap (some 2 us a body) costs what the looks do
// (43 us at 1,024 contacts, 3 at 256).
constexpr int kOrderThreads = 1024;
constexpr int kHubContacts = 256, kMaxHubs = 2 * kMaxContacts / (kHubContacts + 1);
__global__ void __launch_bounds__(kOrderThreads) k_static_order(unsigned *scratch, int nb, int npairs)
{
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned char *const open = smem;
    unsigned short *const next = reinterpret_cast<unsigned short *>(smem + (((size_t)npairs + 15) & ~(size_t)15));
    unsigned short *const of = next + 2 * npairs, *const order = of; // the order takes the lists' place
    int *const end = reinterpret_cast<int *>(of + 2 * npairs);
    const unsigned *ab = scratch + kOffAb;
    int *const out = reinterpret_cast<int *>(scratch + kOffOrder), *const wend = reinterpret_cast<int *>(scratch + kOffWend);
    __shared__ int sh[32];
    __shared__ int s_tail, s_hubs, s_first;
    __shared__ unsigned short s_hub[kMaxHubs];
    __shared__ unsigned s_bits[kMaxContacts / 32];
    const int tid = threadIdx.x;
    if (tid == 0)
        s_hubs = 0;
    for (int i = tid; i <= nb; i += kOrderThreads)
        end[i] = 0;
    __syncthreads();
    for (int k = tid; k < npairs; k += kOrderThreads)
    {
        const unsigned v = ab[k];
        if (v == kSkipped)
            continue;
        atomicAdd(end + (v & 0xffffu), 1);
        if (v >> 16)
            atomicAdd(end + (v >> 16) - 1, 1);
    }
    __syncthreads();
    int carry = 0;
    for (int base = 0; base < nb; base += kOrderThreads)
    {
        const int i = base + tid;
        int tot;
        const int own = i < nb ? end[i] : 0;
        const int pre = nans::block_scan_excl(own, sh, &tot);
        if (i < nb)
            end[i] = carry + pre;
        if (own > kHubContacts)
            s_hub[atomicAdd(&s_hubs, 1)] = (unsigned short)i;
        carry += tot;
    }
    __syncthreads();
    for (int k = tid; k < npairs; k += kOrderThreads)
    {
        const unsigned v = ab[k];
        if (v == kSkipped)
            continue;
        of[atomicAdd(end + (v & 0xffffu), 1)] = (unsigned short)k;
        if (v >> 16)
            of[atomicAdd(end + (v >> 16) - 1, 1)] = (unsigned short)k;
    }
    __syncthreads();
    const int hubs = s_hubs;
    if (hubs > 0)
    {
        for (int k = tid; k < npairs; k += kOrderThreads)
            open[k] = 0;
        for (int h = 0; h < hubs; ++h)
        {
            const int body = s_hub[h], j0 = body ? end[body - 1] : 0, j1 = end[body];
            for (int i = tid; i < kMaxContacts / 32; i += kOrderThreads)
                s_bits[i] = 0u;
            if (tid == 0)
                s_first = 0x7fffffff;
            __syncthreads();
            for (int j = j0 + tid; j < j1; j += kOrderThreads)
            {
                const int k = of[j];
                atomicOr(s_bits + (k >> 5), 1u << (k & 31));
                atomicMin(&s_first, k);
            }
            __syncthreads();
            for (int j = j0 + tid; j < j1; j += kOrderThreads)
            {
                const int k = of[j], side = (ab[k] & 0xffffu) == (unsigned)body ? 0 : 1;
                int i = k >> 5;
                unsigned m = s_bits[i] & ~((2u << (k & 31)) - 1u);
                while (m == 0u && ++i < kMaxContacts / 32)
                    m = s_bits[i];
                next[2 * k + side] = m ? (unsigned short)(32 * i + __ffs(m) - 1) : 0xffffu;
                if (k != s_first)
                    ++open[k];
            }
            __syncthreads(); // the bitmap is the next body's
        }
    }
    for (int k = tid; k < npairs; k += kOrderThreads)
    {
        const unsigned v = ab[k];
        int before = v == kSkipped ? 255 : (hubs > 0 ? open[k] : 0);
        for (int side = 0; side < 2 && v != kSkipped; ++side)
        {
            const int body = side ? (int)(v >> 16) - 1 : (int)(v & 0xffffu);
            int nx = 0xffff;
            bool has = false;
            const int j0 = body > 0 ? end[body - 1] : 0, j1 = body >= 0 ? end[body] : 0;
            if (j1 - j0 > kHubContacts)
                continue;
            if (body >= 0)
                for (int j = j0; j < j1; ++j)
                {
                    const int o = of[j];
                    has = has || o < k;
                    if (o > k && o < nx)
                        nx = o;
                }
            before += has;
            next[2 * k + side] = (unsigned short)nx;
        }
        open[k] = (unsigned char)before;
    }
    if (tid == 0)
        s_tail = 0;
    __syncthreads();
    for (int k = tid; k < npairs; k += kOrderThreads)
        if (open[k] == 0)
            order[atomicAdd(&s_tail, 1)] = (unsigned short)k;
    __syncthreads();
    int lo = 0, wave = 0;
    for (;;)
    {
        const int hi = s_tail;
        if (hi == lo)
            break;
        if (tid == 0)
            wend[wave] = hi;
        __syncthreads(); // the length is read before the wave's contacts add to it
        for (int i = lo + tid; i < hi; i += kOrderThreads)
        {
            const int k = order[i];
            for (int side = 0; side < 2; ++side)
            {
                const int s = next[2 * k + side];
                if (s == 0xffff)
                    continue;
                const unsigned shift = 8u * (s & 3);
                const unsigned old = atomicSub(reinterpret_cast<unsigned *>(open) + (s >> 2), 1u << shift);
                if (((old >> shift) & 255u) == 1u)
                    order[atomicAdd(&s_tail, 1)] = (unsigned short)s;
            }
        }
        __syncthreads();
        lo = hi;
        ++wave;
    }
    for (int i = tid; i < lo; i += kOrderThreads)
        out[i] = order[i];
    if (tid == 0)
        scratch[1] = (unsigned)wave;
}

// The constants in wave order, row by row, with the bodies in place of the contact: a warp of the waves
// reads 512 bytes of each row instead of 32 records 144 bytes apart. Bound by the latency of the
// contacts' and bodies' gathers, which the whole chip takes on here instead of one block.
__global__ void __launch_bounds__(128) k_static_constants(unsigned *scratch, Bodies B, Floor F,
                                                           const nans_contact_pair *pairs, float dt)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, waves = (int)scratch[1];
    const int *wend = reinterpret_cast<const int *>(scratch + kOffWend);
    if (waves == 0 || i >= wend[waves - 1])
        return;
    int *order = reinterpret_cast<int *>(scratch + kOffOrder);
    float4 *K = reinterpret_cast<float4 *>(scratch + kOffK);
    const int k = order[i];
    const unsigned v = scratch[kOffAb + k];
    float4 q[9];
    contact_record(B, F, pairs[k], v & 0xffffu, (int)(v >> 16) - 1, dt, q);
#pragma unroll
    for (int j = 0; j < 9; ++j)
        K[(size_t)j * kMaxContacts + i] = q[j];
    order[i] = (int)v;
}

// The waves, one block, each thread's next contact (of this wave or the next) read ahead, so that a
// wave's chain is a barrier, the velocities' reads and writes in shared memory and the impulses.
__global__ void __launch_bounds__(kThreads) k_static_waves(const unsigned *scratch, Bodies B, Floor F, float cr, float cf,
                                                            int iters)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, nb = B.nbodies, waves = (int)scratch[1];
    const int *ab = reinterpret_cast<const int *>(scratch + kOffOrder), *wend = reinterpret_cast<const int *>(scratch + kOffWend);
    const float4 *K = reinterpret_cast<const float4 *>(scratch + kOffK);
    float *const vel = reinterpret_cast<float *>(smem), *const omg = vel + 3 * nb;
    const bool cached = nb <= kWaveCache;
    float *const V = cached ? vel : B.vel, *const W = cached ? omg : B.omg;
    if (waves == 0)
        return;
    if (cached)
        for (int i = tid; i < 3 * nb; i += kThreads)
        {
            vel[i] = B.vel[i];
            omg[i] = B.omg[i];
        }
    const double c2 = nans::friction_scale(cf);
    const nans::FBound fb = nans::fbound_split(c2);
    __syncthreads();
    int hi = wend[0], hin = waves > 1 ? wend[1] : hi;
    int i = tid; // this thread's current slot
    bool have = false;
    unsigned v = 0u;
    float4 q[9] = {};
    for (int wv = 0; wv < waves; ++wv)
    {
        const int hinn = wv + 2 < waves ? wend[wv + 2] : hin;
        const bool in_next = wv + 1 < waves && hi + tid < hin;
        while (i < hi || !have)
        {
            if (!have)
            {
                // the slot's record, or with none in this wave the next wave's first
                const int j = i < hi ? i : hi + tid;
                have = true;
                if (i < hi || in_next)
                {
                    v = ab[j];
#pragma unroll
                    for (int r = 0; r < 9; ++r)
                        q[r] = K[(size_t)r * kMaxContacts + j];
                }
                continue;
            }
            const int nx = i + kThreads < hi ? i + kThreads : hi + tid;
            unsigned vn = 0u;
            float4 qn[9] = {};
            if (i + kThreads < hi || in_next)
            {
                vn = ab[nx];
#pragma unroll
                for (int r = 0; r < 9; ++r)
                    qn[r] = K[(size_t)r * kMaxContacts + nx];
            }
            solve_one(F, q, V, W, v & 0xffffu, (int)(v >> 16) - 1, cr, c2, fb, iters);
            v = vn;
#pragma unroll
            for (int r = 0; r < 9; ++r)
                q[r] = qn[r];
            if (i + kThreads >= hi)
            {
                have = in_next;
                break;
            }
            i += kThreads;
        }
        if (!in_next)
            have = false;
        __syncthreads();
        i = hi + tid;
        hi = hin;
        hin = hinn;
    }
    if (cached)
        for (int k = tid; k < 3 * nb; k += kThreads)
        {
            B.vel[k] = vel[k];
            B.omg[k] = omg[k];
        }
}

int static_fail(int code, const char *msg)
{
    nans::set_last_error(msg);
    return code;
}

} // namespace

extern "C" int nans_solve_contacts_static(uint32_t nbodies, uint32_t ncubes, const float *d_position,
                                          const float *d_mass, const float *d_moi, float *d_velocity,
                                          float *d_angular_velocity, const float *floor,
                                          const nans_contact_pair *d_pairs, uint32_t npairs, float cr, float cf,
                                          int32_t iterations, float dt, void *stream)
{
    if (nbodies > (uint32_t)kMaxBodies)
        return static_fail(NANS_ERR_INVALID_ARGUMENT,
                           "nans_solve_contacts_static: more than 16384 bodies (static scratch limit)");
    if (npairs > (uint32_t)kMaxContacts)
        return static_fail(NANS_ERR_INVALID_ARGUMENT,
                           "nans_solve_contacts_static: more than 16384 contacts (static scratch limit)");
    if (ncubes > nbodies || !floor || (npairs > 0 && (!d_pairs || nbodies == 0)) ||
        (nbodies > 0 && (!d_position || !d_mass || !d_moi || !d_velocity || !d_angular_velocity)))
        return static_fail(NANS_ERR_INVALID_ARGUMENT, "nans_solve_contacts_static: null or inconsistent argument");
    if (!(dt > 0.0f) || iterations < 0)
        return static_fail(NANS_ERR_INVALID_ARGUMENT, "nans_solve_contacts_static: dt must be positive");
    if (npairs == 0)
        return NANS_OK;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64)
        return static_fail(NANS_ERR_CUDA, "nans_solve_contacts_static: no current CUDA device");
    void *scratch = nullptr;
    {
        // set-up, once per device (again after a reset of that device), with that device
        // current: the device address of the scratch array. cudaSetDevice makes the device's
        // primary context current on this thread, so that its id can be read.
        std::lock_guard<std::mutex> lock(g_setup_mutex);
        e = cudaSetDevice(dev);
        if (e != cudaSuccess)
            return static_fail(NANS_ERR_CUDA, "nans_solve_contacts_static: cudaSetDevice failed");
        const unsigned long long ctx = current_context_id();
        if (!g_scratch_addr[dev].ptr || ctx == 0 || ctx != g_scratch_addr[dev].ctx)
        {
            void *p = nullptr;
            e = cudaGetSymbolAddress(&p, g_solve_scratch);
            if (e != cudaSuccess || !p)
                return static_fail(NANS_ERR_CUDA, "nans_solve_contacts_static: cudaGetSymbolAddress failed");
            // Every kernel is loaded here (kernels load lazily, and one's code takes device memory), and
            // those with large dynamic shared memory get their limit, which belongs to the device's
            // context as well.
            const struct
            {
                const void *fn;
                bool large;
            } kernels[] = {{(const void *)k_solve_static, true},
                           {(const void *)k_static_decode, false},
                           {(const void *)k_static_order, true},
                           {(const void *)k_static_constants, false},
                           {(const void *)k_static_waves, true}};
            for (const auto &k : kernels)
            {
                cudaFuncAttributes attr;
                if (e == cudaSuccess)
                    e = cudaFuncGetAttributes(&attr, k.fn);
                if (e == cudaSuccess && k.large)
                    e = cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDynamicMax);
            }
            if (e != cudaSuccess)
                return static_fail(NANS_ERR_CUDA, "nans_solve_contacts_static: kernel set-up");
            g_scratch_addr[dev].ptr = p;
            g_scratch_addr[dev].ctx = ctx;
        }
        scratch = g_scratch_addr[dev].ptr;
    }
    Bodies B{d_position, d_mass, d_moi, d_velocity, d_angular_velocity, (int)nbodies, (int)ncubes};
    // floor: Position[3], V[3], W[3], Mass, MOI
    Floor F{mk3(floor[0], floor[1], floor[2]), mk3(floor[3], floor[4], floor[5]), mk3(floor[6], floor[7], floor[8]),
            1.0f / floor[9], 1.0f / floor[10]};
    cudaStream_t st = (cudaStream_t)stream;
    unsigned *const S = (unsigned *)scratch;
    const int n = (int)npairs;
    if (n <= kOneLaunch)
        k_solve_static<<<1, kThreads, one_launch_smem((int)nbodies, n), st>>>(S, B, F, d_pairs, n, cr, cf, iterations, dt);
    else
    {
        e = cudaMemsetAsync(scratch, 0, sizeof(unsigned), st);
        if (e != cudaSuccess)
            return static_fail(NANS_ERR_CUDA, "nans_solve_contacts_static: clearing the status word failed");
        k_static_decode<<<(n + 255) / 256, 256, 0, st>>>(S, B, d_pairs, n);
        k_static_order<<<1, kOrderThreads, order_smem((int)nbodies, n), st>>>(S, (int)nbodies, n);
        k_static_constants<<<(n + 127) / 128, 128, 0, st>>>(S, B, F, d_pairs, dt);
        k_static_waves<<<1, kThreads, waves_smem((int)nbodies), st>>>(S, B, F, cr, cf, iterations);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess)
        return static_fail(NANS_ERR_CUDA, "nans_solve_contacts_static: kernel launch failed");
    // the status word (scratch word 0), read on the caller's stream
    unsigned err = 0;
    e = cudaMemcpyAsync(&err, scratch, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(st);
    if (e != cudaSuccess)
        return static_fail(NANS_ERR_CUDA, "nans_solve_contacts_static: kernel failed");
    if (err & 1u)
        return static_fail(NANS_ERR_INVALID_ARGUMENT,
                           "nans_solve_contacts_static: a contact names a body outside the scene, or the same "
                           "body on both sides (skipped)");
    return NANS_OK;
}
