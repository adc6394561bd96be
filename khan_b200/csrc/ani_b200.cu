// C ABI of libani_b200.so: argument checks, launch configuration and the per-device scratch
// cache.  All kernels live in the .cuh files included below (one translation unit, so the
// device status word and the constant tables exist exactly once).
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <initializer_list>
#include <new>
#include <mutex>
#include <vector>

#include "ani_common.cuh"

#include "ani_featurize.cuh"
#include "ani_featurize_mol.cuh"
#include "ani_featurize_large.cuh"
#include "ani_grad.cuh"
#include "ani_grad_mol.cuh"
#include "ani_grad_large.cuh"
#include "ani_grad_inverse.cuh"
#include "ani_tangent_mol.cuh"
#include "ani_mlp_forward.cuh"
#include "ani_mlp_backward.cuh"
#include "ani_mlp_wgrad.cuh"
#include "ani_mlp_chain.cuh"
#include "ani_mlp_small.cuh"
#include "ani_force_fit.cuh"
#include "ani_charge.cuh"
#include "ani_optim.cuh"
#include "ani_energy.cuh"
#include "ani_sort.cuh"
#include "ani_host_pack.h"
#include "ani_driver.h"
#include "ani_feeder.h"
#include "ani_peer.cuh"

namespace {

using namespace ani;

thread_local cudaError_t t_last_error = cudaSuccess;

int cuda_fail(cudaError_t e)
{
    t_last_error = e;
    return ANI_ERR_CUDA;
}

#define ANI_CUDA(call)                                  \
    do {                                                \
        cudaError_t e_ = (call);                        \
        if (e_ != cudaSuccess) return cuda_fail(e_);    \
    } while (0)

constexpr int kMaxDevices = 64;

// Scratch of the large-batch sort (per-tile element counts), one buffer per (device, stream): two
// calls that overlap on the GPU are on different streams and so never share a buffer.  A buffer
// that has become too small is replaced but NEVER freed -- its address may be recorded in a CUDA
// graph that is replayed later -- so the old ones stay allocated until the process ends (they are
// a few KiB each and grow geometrically).
struct SortScratch {
    int dev;
    cudaStream_t stream;
    int* ptr;
    size_t bytes;
};
std::mutex g_scratch_mutex;
std::vector<SortScratch> g_sort_scratch;

// True when work given to `stream` is being recorded into a graph instead of run.
int stream_is_capturing(cudaStream_t stream, bool* capturing)
{
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    ANI_CUDA(cudaStreamIsCapturing(stream, &status));
    *capturing = status != cudaStreamCaptureStatusNone;
    return ANI_OK;
}

int sort_scratch(size_t bytes, cudaStream_t stream, int** out)
{
    int dev = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    SortScratch* slot = nullptr;
    for (SortScratch& s : g_sort_scratch)
        if (s.dev == dev && s.stream == stream) slot = &s;
    if (slot && slot->bytes >= bytes) {
        *out = slot->ptr;
        return ANI_OK;
    }
    // an allocation is not something a stream capture can record
    bool capturing = false;
    if (int rc = stream_is_capturing(stream, &capturing)) return rc;
    if (capturing) return ANI_ERR_CAPTURE;
    const size_t want = bytes < (1u << 16) ? (1u << 16) : bytes * 2;
    int* ptr = nullptr;
    ANI_CUDA(cudaMalloc(&ptr, want));
    if (slot) {
        slot->ptr = ptr;       // the previous buffer stays allocated (see above)
        slot->bytes = want;
    } else {
        g_sort_scratch.push_back(SortScratch{dev, stream, ptr, want});
    }
    *out = ptr;
    return ANI_OK;
}

// Fixed scratch for ani_sort_noalloc: per-tile element counts for batches of up to
// kSortStaticMaxAtoms atoms ((tiles + 1) x 4 ints = 64 KiB + 16 B).  It lives in the module's
// static device data, so every GPU that loads this library holds it until the process exits.
constexpr int kSortStaticMaxAtoms = 1 << 22;  // 4,194,304 atoms
constexpr int kSortStaticMaxTiles = kSortStaticMaxAtoms / kSortTile;
static __device__ __align__(256) int g_sort_static_scratch[(kSortStaticMaxTiles + 1) * kTypes];

// Device address of g_sort_static_scratch on each device, resolved on first use.  In host code
// the array's name is only a handle for the runtime, not a device address, so it is never
// passed to a kernel; the pointer obtained here is.
int* g_sort_static_ptr[kMaxDevices] = {};
std::mutex g_sort_static_mutex;

int sort_static_scratch(cudaStream_t stream, int** out)
{
    int dev = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return ANI_ERR_BAD_SIZE;
    std::lock_guard<std::mutex> lock(g_sort_static_mutex);
    if (!g_sort_static_ptr[dev]) {
        // The look-up may load the module's data on this device: not something to do while the stream
        // is being captured.  Make the first call on a device outside any capture.
        bool capturing = false;
        if (int rc = stream_is_capturing(stream, &capturing)) return rc;
        if (capturing) return ANI_ERR_CAPTURE;
        int* ptr = nullptr;
        ANI_CUDA(cudaGetSymbolAddress((void**)&ptr, g_sort_static_scratch));  // current device = dev
        g_sort_static_ptr[dev] = ptr;
    }
    *out = g_sort_static_ptr[dev];
    return ANI_OK;
}

// Featurizer launch shapes: NW warps per CTA, (slots per molecule) / NW CTAs per molecule, one warp
// per central atom.  The capacities bound the neighbours of one element kept in shared memory
// per central atom (atoms with more take the streaming path).
#ifndef ANI_NW
#define ANI_NW 4
#endif
constexpr int kNW = ANI_NW;   // warps per CTA of the featurizer kernels (a power of two <= 32)
constexpr int kCapT = 24;  // angular (r < 3.1 A) neighbours per element
constexpr int kCapR = 48;  // radial (r < 4.6 A) neighbours per element

// Persistent grid: as many CTAs as fit on the device at once (rounded to a multiple of
// kSlotsPerMol / kNW so that the warp count is a multiple of kSlotsPerMol), or fewer when the
// batch is small.
template <typename K> int featurizer_grid(K kernel, size_t smem, int n_mols, int* grid)
{
    int dev = 0, sms = 0, per_sm = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    ANI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    ANI_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kNW * kWarp, smem));
    constexpr int kGroup = kSlotsPerMol / kNW;
    long long resident = (long long)sms * (per_sm > 0 ? per_sm : 1);
    resident = (resident / kGroup) * kGroup;
    if (resident < kGroup) resident = kGroup;
    const long long needed = (long long)n_mols * kGroup;
    *grid = (int)(needed < resident ? needed : resident);
    return ANI_OK;
}

// Work list of a launch, packed into one kernel argument: bits 0-4 = log2 of the slots per
// molecule (the smallest power of two that is not below the mean atoms per molecule, between kNW
// and kSlotsPerMol: few empty items, and larger molecules simply give some slots a second atom);
// bit 5 = slot-major order, used when molecules are small (see next_work).
constexpr int kSlotMajorFlag = 32;
int pick_slot_shift(long long n_atoms, int n_mols)
{
    const long long mean = n_mols > 0 ? (n_atoms + n_mols - 1) / n_mols : 1;
    int shift = 0;
    while ((1 << shift) < kNW) shift++;   // at least one slot per warp of a CTA
    while ((1 << shift) < mean && (1 << shift) < kSlotsPerMol) shift++;
    return shift | (mean <= kSlotsPerMol ? kSlotMajorFlag : 0);
}

template <typename K> int set_smem(K kernel, size_t bytes)
{
    ANI_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return ANI_OK;
}

// Batches whose MEAN molecule size is at most this take the kernels for small molecules (their fast path covers
// molecules of up to kMolMaxAtoms atoms; a larger molecule in such a batch is still handled, slowly).  Batches of
// larger molecules take featurize_large_kernel and featurize_grad_large_kernel (a few central atoms per warp, the
// molecule scanned from global memory); the one-warp-per-atom forward kernel remains for outputs that are not 16-byte
// aligned.
constexpr int kMolMeanLimit = 24;
constexpr int kSms = 148;
bool small_molecules(long long n_atoms, int n_mols) { return n_mols > 0 && n_atoms <= (long long)n_mols * kMolMeanLimit; }

// True when every non-null pointer of the list is 16-byte aligned.
bool all_aligned16(std::initializer_list<const void*> ptrs)
{
    for (const void* q : ptrs)
        if (reinterpret_cast<uintptr_t>(q) & 15) return false;
    return true;
}

int check_acs(const int* acs_host, long long* n_atoms)
{
    if (!acs_host) return ANI_ERR_NULL_POINTER;
    long long n = 0;
    for (int t = 0; t < kTypes; t++) {
        if (acs_host[t] < 0) return ANI_ERR_BAD_SIZE;
        n += acs_host[t];
    }
    if (n > 0x7fffffffLL) return ANI_ERR_TOO_MANY_ATOMS;
    *n_atoms = n;
    return ANI_OK;
}

template <typename T, int CAPT = kCapT, int CAPR = kCapR>
int featurize_impl(const T* xs, const T* ys, const T* zs, const int* types, const int* mos,
                   const int* macs, int n_mols, const int* sis, T* oh, T* oc, T* on, T* oo,
                   const int* acs_host, void* stream, bool after_sort = false)
{
    long long n_atoms = 0;
    if (int rc = check_acs(acs_host, &n_atoms)) return rc;
    if (n_mols < 0) return ANI_ERR_BAD_SIZE;
    if (n_mols == 0 || n_atoms == 0) return ANI_OK;
    if (!xs || !ys || !zs || !types || !mos || !macs || !sis) return ANI_ERR_NULL_POINTER;
    T* outs[kTypes] = {oh, oc, on, oo};
    for (int t = 0; t < kTypes; t++)
        if (acs_host[t] > 0 && !outs[t]) return ANI_ERR_NULL_POINTER;

    int dev = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    // small molecules with outputs that take 16-byte stores: one warp (= one CTA) per round of one to four
    // central atoms
    if (small_molecules(n_atoms, n_mols) && all_aligned16({oh, oc, on, oo}) &&
        (long long)n_mols * kMolMaxAtoms <= 0x7fffffffLL) {
        // As few central atoms per warp as still find all warps resident at once (28 per SM in float, 20 in double): with
        // four, the scans and triplets of one warp are a chain of 12 us (float; double 25 us), however small the batch.
        // Few atoms per warp cost more instructions (load, sort and table per round), so not beyond that.  Microseconds
        // with 4 / 2 / 1 atoms in float, 64 molecules 12.9 / 9.8 / 8.3, 256: 16.0 / 12.8 / 12.0, 512: 18.7 / 16.0 / 18.9,
        // 1024: 24.0 / 25.3 / 31.1, 8192: 118 / 153 / 238; in double, 64: 26 / 19 / 17, 256: 34 / 27 / 31, 512: 39 / 41 /
        // 49, 1024: 60 / 64 / 84.  (32 float warps are resident, but with that line 1024 molecules take three atoms per
        // warp: 27.3 us when four took 25.2, and 1.5 more a batch with eight streams.)
        const int resident = kSms * (sizeof(T) == 4 ? 28 : 20);
        const int per_round = (int)std::min<long long>((n_atoms + resident - 1) / resident, kMolCentrals);
        const int rounds = (kMolMaxAtoms + per_round - 1) / per_round;
        ANI_CUDA(launch_chain(featurize_mol_kernel<T>, n_mols * rounds, kWarp, 0, (cudaStream_t)stream, 1, xs, ys, zs,
                              types, mos, macs, n_mols, (int)n_atoms, sis, oh, oc, on, oo, acs_host[0], acs_host[1],
                              acs_host[2], acs_host[3], per_round, 65536 / per_round + 1, after_sort));
        return ANI_OK;
    }

    // larger molecules: the same rounds of one to four central atoms, the molecule scanned from global memory;
    // a CTA takes every rounds_in_grid-th round of its molecule
    if (n_mols > 0 && all_aligned16({oh, oc, on, oo})) {
        const int resident = kSms * (sizeof(T) == 4 ? 22 : 14);
        const int per_round = (int)std::min<long long>((n_atoms + resident - 1) / resident, kMolCentrals);
        const long long mean_rounds = (n_atoms / n_mols + per_round) / per_round;
        const long long rounds = std::min(std::min<long long>(mean_rounds, 256), 0x7fffffffLL / n_mols);
        ANI_CUDA(launch_chain(featurize_large_kernel<T>, (int)(n_mols * rounds), kWarp, 0, (cudaStream_t)stream, 1, xs, ys, zs,
                              types, mos, macs, n_mols, (int)n_atoms, per_round, sis, oh, oc, on, oo, acs_host[0],
                              acs_host[1], acs_host[2], acs_host[3]));
        return ANI_OK;
    }

    auto kernel = featurize_kernel<T, kNW, CAPT, CAPR>;
    const size_t smem = kNW * sizeof(FeaturizeWarpShared<T, CAPT, CAPR>);
    static thread_local int configured_dev = -1;
    if (configured_dev != dev) {
        if (int rc = set_smem(kernel, smem)) return rc;
        configured_dev = dev;
    }
    static thread_local int cached_grid_dev = -1, cached_resident = 0;
    if (cached_grid_dev != dev) {
        if (int rc = featurizer_grid(kernel, smem, 1 << 24, &cached_resident)) return rc;
        cached_grid_dev = dev;
    }
    const int slot_shift = pick_slot_shift(n_atoms, n_mols);
    const long long needed = (long long)n_mols * ((1 << (slot_shift & 31)) / kNW);
    const int grid = (int)(needed < cached_resident ? needed : cached_resident);
    kernel<<<grid, kNW * kWarp, smem, (cudaStream_t)stream>>>(
        xs, ys, zs, types, mos, macs, n_mols, (int)n_atoms, slot_shift, sis, oh, oc, on, oo, acs_host[0],
        acs_host[1], acs_host[2], acs_host[3]);
    ANI_CUDA(cudaGetLastError());
    return ANI_OK;
}

// The coordinate gradients of such a batch are computed a molecule per CTA (and molecule energies with them).
bool grad_per_molecule(long long n_atoms, int n_mols, std::initializer_list<const void*> rows)
{
    return n_mols > 0 && small_molecules(n_atoms, n_mols) && all_aligned16(rows) && n_mols <= 0x7fffffff - kWarp;
}

template <typename T>
int featurize_grad_impl(const T* xs, const T* ys, const T* zs, const int* types, const int* mos,
                        const int* macs, int n_mols, const int* sis, const T* gh, const T* gc,
                        const T* gn, const T* go, T* gx, T* gy, T* gz, const int* acs_host,
                        void* stream, const MolEnergySums<T>& sums = MolEnergySums<T>{}, bool early_inputs = false)
{
    long long n_atoms = 0;
    if (int rc = check_acs(acs_host, &n_atoms)) return rc;
    if (n_mols < 0) return ANI_ERR_BAD_SIZE;
    if (n_atoms == 0) return ANI_OK;
    if (!gx || !gy || !gz) return ANI_ERR_NULL_POINTER;
    cudaStream_t st = (cudaStream_t)stream;
    const T* gin[kTypes] = {gh, gc, gn, go};
    // One CTA per molecule when the molecules are small and the upstream rows can be fetched with
    // 16-byte copies: writes every output itself, so no zero fill.
    if (grad_per_molecule(n_atoms, n_mols, {gh, gc, gn, go})) {
        if (!xs || !ys || !zs || !types || !mos || !macs || !sis) return ANI_ERR_NULL_POINTER;
        for (int t = 0; t < kTypes; t++)
            if (acs_host[t] > 0 && !gin[t]) return ANI_ERR_NULL_POINTER;
        auto launch = [&](auto warps, auto ctas) -> int {
            constexpr int NW = decltype(warps)::value, CTAS = decltype(ctas)::value;
            constexpr size_t smem = sizeof(MolGradShared<T, NW, CTAS>);
            static thread_local int configured_dev = -1;     // one per variant
            int dev = 0;
            ANI_CUDA(cudaGetDevice(&dev));
            if (configured_dev != dev) {
                if (int rc = set_smem(featurize_grad_mol_kernel<T, NW, CTAS>, smem)) return rc;
                configured_dev = dev;
            }
            // more molecules than are resident at once: the larger ones start first (figures at kMolGradOrder)
            const bool in_order = n_mols > kSms * CTAS;
            const dim3 grid = in_order ? dim3((n_mols + kMolGradOrder - 1) / kMolGradOrder, kMolGradOrder) : dim3(n_mols);
            ANI_CUDA(launch_chain(featurize_grad_mol_kernel<T, NW, CTAS>, grid, NW * kWarp, smem, st, 1, xs, ys, zs, types, mos,
                                  macs, n_mols, (int)n_atoms, sis, gh, gc, gn, go, gx, gy, gz, acs_host[0], acs_host[1],
                                  acs_host[2], acs_host[3], sums, early_inputs));
            return ANI_OK;
        };
        // Few molecules: all of an SM for one (molecules for every other SM at most: the next batch's find a free SM then),
        // or half of one.  Microseconds alone / with two / with eight streams in flight, float, one CTA of twelve warps per SM |
        // two of them | four of eight: 64 molecules 10.6 / 5.4 / 2.6 | 11.7 / 6.0 / 2.1 | -, 148: 11.3 / 6.7 / 5.5 | 12.5 /
        // 7.1 / 3.6 | -, 296: - | 15.8 / 8.8 / 7.3 | 19.8 / 11.2 / 5.5, 592: - | 18.9 / 14.6 / 14.6 | 24.3 / 14.0 / 10.5, 740: - |
        // 22.3 / 18.0 / 18.1 | 23.8 / 14.2 / 13.5.  The second line is drawn where a batch alone stops gaining.  (With central
        // atoms dealt to warps, as it was once, 14.6 / 7.5 / 2.5, 17.1 / 9.2 / 4.0, 19.2 / 10.7 /
        // 8.1, 20.5 / 16.0 / 16.1 and 24.1 / 19.8 / 20.0.)  Double, one of twelve | two of eight: 296: 27.4 / 21.1 / 21.2 | 40.7 /
        // 22.2 / 16.5, 512: 40.2 / 35.4 / 35.5 | 42.4 / 28.3 / 28.2, 592: 46.2 / 40.9 / 41.0 | 43.7 / 32.5 / 32.5.
        using One = std::integral_constant<int, 1>;
        using Two = std::integral_constant<int, 2>;
        using Twelve = std::integral_constant<int, 12>;
        using Eight = std::integral_constant<int, 8>;
        if constexpr (sizeof(T) == 8) return 2 * n_mols <= 7 * kSms ? launch(Twelve{}, One{}) : launch(Eight{}, Two{});
        if (2 * n_mols <= kSms) return launch(Twelve{}, One{});
        if (n_mols <= 5 * kSms) return launch(Twelve{}, Two{});
        return launch(Eight{}, std::integral_constant<int, 4>{});
    }
    {
        const int threads = 256;
        long long blocks = (n_atoms + threads - 1) / threads;
        if (blocks > 1184) blocks = 1184;
        ANI_CUDA(launch_chain(zero3_kernel<T>, (int)blocks, threads, 0, st, 1, gx, gy, gz, (int)n_atoms));
    }
    if (n_mols == 0) return ANI_OK;
    if (!xs || !ys || !zs || !types || !mos || !macs || !sis) return ANI_ERR_NULL_POINTER;
    for (int t = 0; t < kTypes; t++)
        if (acs_host[t] > 0 && !gin[t]) return ANI_ERR_NULL_POINTER;

    // one to three central atoms per warp, as in the features: few while all warps are resident anyway
    const auto kernel = featurize_grad_large_kernel<T>;
    const size_t smem = sizeof(LargeGradWarpShared<T>);
    static thread_local int configured_dev = -1;
    int dev = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    if (configured_dev != dev) {
        if (int rc = set_smem(kernel, smem)) return rc;
        configured_dev = dev;
    }
    const int resident = kSms * (sizeof(T) == 4 ? 20 : 12);
    const int per_round = (int)std::min<long long>((n_atoms + resident - 1) / resident, kLargeGradCentrals);
    const long long mean_rounds = (n_atoms / n_mols + per_round) / per_round;
    const long long rounds = std::min(std::min<long long>(mean_rounds, 256), 0x7fffffffLL / n_mols);
    ANI_CUDA(launch_chain(kernel, (int)(n_mols * rounds), kWarp, smem, st, 1, xs, ys, zs, types, mos, macs, n_mols,
                          (int)n_atoms, per_round, all_aligned16({gh, gc, gn, go}), sis, gh, gc, gn, go, gx, gy, gz,
                          acs_host[0], acs_host[1], acs_host[2], acs_host[3]));
    return ANI_OK;
}

template <typename T>
int featurize_grad_inverse_impl(const T* xs, const T* ys, const T* zs, const int* types,
                                const int* mos, const int* macs, int n_mols, const int* sis,
                                const T* vx, const T* vy, const T* vz, T* oh, T* oc, T* on, T* oo,
                                const int* acs_host, void* stream)
{
    long long n_atoms = 0;
    if (int rc = check_acs(acs_host, &n_atoms)) return rc;
    if (n_mols < 0) return ANI_ERR_BAD_SIZE;
    if (n_mols == 0 || n_atoms == 0) return ANI_OK;
    if (!xs || !ys || !zs || !types || !mos || !macs || !sis || !vx || !vy || !vz)
        return ANI_ERR_NULL_POINTER;
    T* outs[kTypes] = {oh, oc, on, oo};
    for (int t = 0; t < kTypes; t++)
        if (acs_host[t] > 0 && !outs[t]) return ANI_ERR_NULL_POINTER;

    // small molecules with outputs that take 16-byte stores: rounds of one to four central atoms per warp, as few as still
    // find all warps resident at once, as in the features.  Microseconds with 4 / 3 / 2 / 1 in float, 32 molecules 14.6 /
    // 13.0 / 10.9 / 8.8, 128: 17.2 / 15.6 / 13.3 / 11.5, 256: 22.5 / 19.1 / 16.2 / 18.0, 512: 25.1 / 25.8 / 24.5 / 29.9,
    // 1024: 39.7 / 39.8 / 43.8 / 57.3; in double, 64: 36 / 34 / 26 / 20, 256: 42 / 36 / 40 / 44, 1024: 92 / 95 / 110 / 143.
    // Three lose to four in float where the rule would take them, and do in both types with eight streams in flight.
    if (small_molecules(n_atoms, n_mols) && all_aligned16({oh, oc, on, oo}) &&
        (long long)n_mols * kMolMaxAtoms <= 0x7fffffffLL) {
        const int resident = kSms * (sizeof(T) == 4 ? 16 : 10);
        int per_round = (int)std::min<long long>((n_atoms + resident - 1) / resident, kMolCentrals);
        if (sizeof(T) == 4 && per_round == 3) per_round = 4;
        const int rounds = (kMolMaxAtoms + per_round - 1) / per_round;
        ANI_CUDA(launch_chain(featurize_tangent_mol_kernel<T>, n_mols * rounds, kWarp, 0, (cudaStream_t)stream, 1, xs, ys,
                              zs, types, mos, macs, n_mols, (int)n_atoms, sis, vx, vy, vz, oh, oc, on, oo, acs_host[0],
                              acs_host[1], acs_host[2], acs_host[3], per_round, 65536 / per_round + 1));
        return ANI_OK;
    }

    auto kernel = featurize_grad_inverse_kernel<T, kNW>;
    const size_t smem = kNW * sizeof(JvpWarpShared<T>);
    static thread_local int configured_dev = -1, cached_resident = 0;
    int dev = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    if (configured_dev != dev) {
        if (int rc = set_smem(kernel, smem)) return rc;
        if (int rc = featurizer_grid(kernel, smem, 1 << 24, &cached_resident)) return rc;
        configured_dev = dev;
    }
    const int slot_shift = pick_slot_shift(n_atoms, n_mols);
    const long long needed = (long long)n_mols * ((1 << (slot_shift & 31)) / kNW);
    const int grid = (int)(needed < cached_resident ? needed : cached_resident);
    kernel<<<grid, kNW * kWarp, smem, (cudaStream_t)stream>>>(
        xs, ys, zs, types, mos, macs, n_mols, (int)n_atoms, slot_shift, sis, vx, vy, vz, oh, oc, on, oo,
        acs_host[0], acs_host[1], acs_host[2], acs_host[3]);
    ANI_CUDA(cudaGetLastError());
    return ANI_OK;
}

// Grid of the one-warp-per-molecule charge kernels: every molecule gets a warp, up to 16 CTAs per SM.
int charge_grid(int n_mols, int* grid)
{
    int dev = 0, sms = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    ANI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int needed = (n_mols + kNW - 1) / kNW;
    *grid = needed < sms * 16 ? needed : sms * 16;
    return ANI_OK;
}

template <typename T>
int charge_impl(const T* xs, const T* ys, const T* zs, const T* qs, const int* mos, const int* macs,
                int n_mols, int n_atoms, T* energies, void* stream)
{
    if (n_mols < 0 || n_atoms < 0) return ANI_ERR_BAD_SIZE;
    if (n_mols == 0) return ANI_OK;
    if (!mos || !macs || !energies) return ANI_ERR_NULL_POINTER;
    if (n_atoms > 0 && (!xs || !ys || !zs || !qs)) return ANI_ERR_NULL_POINTER;
    int grid = 0;
    if (int rc = charge_grid(n_mols, &grid)) return rc;
    charge_energy_kernel<T, kNW><<<grid, kNW * kWarp, 0, (cudaStream_t)stream>>>(
        xs, ys, zs, qs, mos, macs, n_mols, n_atoms, energies);
    ANI_CUDA(cudaGetLastError());
    return ANI_OK;
}

template <typename T>
int charge_grad_impl(const T* xs, const T* ys, const T* zs, const T* qs, const int* mos,
                     const int* macs, int n_mols, int n_atoms, const T* energy_grads, T* q_grads,
                     void* stream)
{
    if (n_mols < 0 || n_atoms < 0) return ANI_ERR_BAD_SIZE;
    if (n_atoms == 0) return ANI_OK;
    if (!xs || !ys || !zs || !qs || !q_grads) return ANI_ERR_NULL_POINTER;
    cudaStream_t st = (cudaStream_t)stream;
    ANI_CUDA(cudaMemsetAsync(q_grads, 0, (size_t)n_atoms * sizeof(T), st));
    if (n_mols == 0) return ANI_OK;
    if (!mos || !macs || !energy_grads) return ANI_ERR_NULL_POINTER;
    int grid = 0;
    if (int rc = charge_grid(n_mols, &grid)) return rc;
    charge_grad_kernel<T, kNW><<<grid, kNW * kWarp, 0, st>>>(xs, ys, zs, qs, mos, macs, n_mols, n_atoms,
                                                             energy_grads, q_grads);
    ANI_CUDA(cudaGetLastError());
    return ANI_OK;
}

template <int ACT, bool SPLIT> int mlp_launch(const MlpParams& p, int n_tiles, cudaStream_t st)
{
    auto kernel = mlp_forward_kernel<ACT, SPLIT>;
    const size_t smem = sizeof(MlpShared) + 1024;
    static thread_local int configured_dev = -1;
    int dev = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    if (configured_dev != dev) {
        if (int rc = set_smem(kernel, smem)) return rc;
        configured_dev = dev;
    }
    ANI_CUDA(launch_chain(kernel, n_tiles, kMlpAllThreads, smem, st, 1, p));
    return ANI_OK;
}

template <bool SPLIT> int mlp_backward_launch(const MlpBackwardParams& p, int n_tiles, cudaStream_t st)
{
    auto kernel = mlp_backward_kernel<SPLIT>;
    const size_t smem = sizeof(MlpShared) + 1024;
    static thread_local int configured_dev = -1;
    int dev = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    if (configured_dev != dev) {
        if (int rc = set_smem(kernel, smem)) return rc;
        configured_dev = dev;
    }
    ANI_CUDA(launch_chain(kernel, n_tiles, kMlpAllThreads, smem, st, 1, p));
    return ANI_OK;
}

template <int ACT, bool SPLIT, int MODE> int mlp_chain_launch(const MlpChainParams& p, cudaStream_t st)
{
    auto kernel = mlp_chain_kernel<ACT, SPLIT, MODE>;
    const size_t smem = sizeof(ChainShared);
    static thread_local int configured_dev = -1;
    int dev = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    if (configured_dev != dev) {
        if (int rc = set_smem(kernel, smem)) return rc;
        configured_dev = dev;
    }
    ANI_CUDA(launch_chain(kernel, p.tile_start[kTypes], kChainThreads, smem, st, 1, p));
    return ANI_OK;
}
template <int ACT, int MODE> int mlp_chain_split(const MlpChainParams& p, bool split, cudaStream_t st)
{
    return split ? mlp_chain_launch<ACT, true, MODE>(p, st) : mlp_chain_launch<ACT, false, MODE>(p, st);
}
template <int MODE> int mlp_chain_act(const MlpChainParams& p, int activation, bool split, cudaStream_t st)
{
    if constexpr (MODE == kChainBackward) {      // no activation in it
        return mlp_chain_split<kActCelu, MODE>(p, split, st);
    } else {
        switch (activation) {
            case kActCelu: return mlp_chain_split<kActCelu, MODE>(p, split, st);
            case kActGaussian: return mlp_chain_split<kActGaussian, MODE>(p, split, st);
            case kActNormal: return mlp_chain_split<kActNormal, MODE>(p, split, st);
            default: return mlp_chain_split<kActSoftplus, MODE>(p, split, st);
        }
    }
}

template <bool SPLIT> int mlp_wgrad_launch(const MlpWgradSets& p, int n_ranges, int n_sets, cudaStream_t st)
{
    auto kernel = mlp_wgrad_kernel<SPLIT>;
    const size_t smem = sizeof(WgradShared);
    static thread_local int configured_dev = -1;
    int dev = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    if (configured_dev != dev) {
        if (int rc = set_smem(kernel, smem)) return rc;
        configured_dev = dev;
    }
    ANI_CUDA(launch_chain(kernel, dim3(n_ranges, kWgradBlocks, n_sets), kMlpAllThreads, smem, st, 1, p));
    return ANI_OK;
}

int pack_params(const float* const* w1, const float* const* w2, const float* const* w3, void* const* packed, MlpPackParams* p,
                bool* any)
{
    for (int t = 0; t < kTypes; t++) {
        p->w1[t] = w1[t]; p->w2[t] = w2[t]; p->w3[t] = w3[t];
        p->packed[t] = (unsigned char*)packed[t];
        if (!packed[t]) continue;
        if (!w1[t] || !w2[t] || !w3[t]) return ANI_ERR_NULL_POINTER;
        if (reinterpret_cast<uintptr_t>(packed[t]) & 15) return ANI_ERR_MISALIGNED;
        *any = true;
    }
    return ANI_OK;
}
int pack_launch(const MlpPackParams& p, cudaStream_t st)
{
    ANI_CUDA(launch_chain(mlp_pack_kernel, dim3(kPackChunks, kTypes), kMlpThreads, 0, st, 1, p));
    return ANI_OK;
}

// Batches whose networks take mlp_small_kernel: every tile of 16 atoms is a cluster of 8 CTAs, which share the columns of
// a layer, where the chain kernel needs 22 us (forward) or 37 us (with backward) for one tile or for 148.  Measured,
// forward / with backward: 4 to 14 tiles 6.8 / 11.4 us, 28: 9.3 / 16.8, 39: 16.7 / 30.9, 53: 17.2 / 32.0, 84: 25.3 / 47.7.
constexpr int kFewTiles = 56;
bool few_atoms(const int* acs)
{
    int tiles = 0;
    for (int t = 0; t < kTypes; t++) tiles += (acs[t] + kSmallTile - 1) / kSmallTile;
    return tiles <= kFewTiles;
}

template <typename T>
int energy_launch(const T* atom_energy_sorted, const int* gather, const int* mos, const int* macs, int n_mols, int n_atoms,
                  const T* labels, T grad_scale, T* mol_energy, T* l2s, T* grad_atom_energy_sorted, cudaStream_t st)
{
    int grid = 0;
    if (int rc = charge_grid(n_mols, &grid)) return rc;
    ANI_CUDA(launch_chain(molecule_energy_kernel<T, kNW>, grid, kNW * kWarp, 0, st, 1, atom_energy_sorted, gather, mos, macs,
                          n_mols, n_atoms, labels, grad_scale, mol_energy, l2s, grad_atom_energy_sorted));
    return ANI_OK;
}

// Networks of few atoms / of double precision: forward and (grad_feat != NULL) backward to the features.
template <typename T>
int mlp_small_launch(const T* feat, const int* acs, const T* const* w1, const T* const* b1, const T* const* w2,
                     const T* const* b2, const T* const* w3, const T* const* b3, const T* const* w4, const T* const* b4,
                     const T* grad_energy, T* energy, T* grad_feat, int activation, bool early_weights, cudaStream_t st,
                     const MlpPackParams* pack = nullptr)
{
    if (activation < 0 || activation > 3) return ANI_ERR_BAD_SIZE;
    MlpSmallParams<T> p;
    p.feat = feat;
    p.grad_energy = grad_energy;
    p.energy = energy;
    p.grad_feat = grad_feat;
    p.activation = activation;
    p.early_weights = early_weights;
    int tiles = 0, row = 0;
    if (!feat || !energy) return ANI_ERR_NULL_POINTER;
    if (!all_aligned16({feat, grad_feat})) return ANI_ERR_MISALIGNED;
    for (int t = 0; t < kTypes; t++) {
        p.tile_start[t] = tiles;
        p.row_start[t] = row;
        p.count[t] = acs[t];
        tiles += (acs[t] + kSmallTile - 1) / kSmallTile;
        row += acs[t];
        if (acs[t] > 0) {
            if (!w1[t] || !b1[t] || !w2[t] || !b2[t] || !w3[t] || !b3[t] || !w4[t] || !b4[t]) return ANI_ERR_NULL_POINTER;
            if (!all_aligned16({w1[t], w2[t], w3[t]})) return ANI_ERR_MISALIGNED;
        }
        p.w1[t] = w1[t]; p.b1[t] = b1[t]; p.w2[t] = w2[t]; p.b2[t] = b2[t];
        p.w3[t] = w3[t]; p.b3[t] = b3[t]; p.w4[t] = w4[t]; p.b4[t] = b4[t];
    }
    p.tile_start[kTypes] = tiles;
    if (tiles == 0) return ANI_OK;
    auto kernel = mlp_small_kernel<T>;
    const size_t smem = sizeof(MlpSmallShared<T>);
    static thread_local int configured_dev = -1;
    int dev = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    if (configured_dev != dev) {
        if (int rc = set_smem(kernel, smem)) return rc;
        configured_dev = dev;
    }
    static_assert(kPackChunks * kTypes % kSmallCtas == 0, "whole clusters pack");
    ANI_CUDA(launch_chain(kernel, tiles * kSmallCtas + (pack ? kPackChunks * kTypes : 0), kSmallThreads, smem, st, kSmallCtas, p,
                          pack ? *pack : MlpPackParams{}));
    return ANI_OK;
}

// Pre-activations of the hidden layers with celu, in plain float32 products.
int celu_preactivations_launch(const ani_pass_args* a, const int* acs, float* z1, float* z2, float* z3, cudaStream_t st)
{
    CeluPreParams p = {};
    p.feat = a->features;
    p.z[0] = z1; p.z[1] = z2; p.z[2] = z3;
    p.aligned = all_aligned16({a->features});
    int tiles = 0, row = 0;
    for (int t = 0; t < kTypes; t++) {
        const float* const w[3] = {a->w1[t], a->w2[t], a->w3[t]};
        const float* const b[3] = {a->b1[t], a->b2[t], a->b3[t]};
        for (int l = 0; l < 3; l++) {
            if (acs[t] > 0 && (!w[l] || !b[l])) return ANI_ERR_NULL_POINTER;
            p.aligned = p.aligned && (acs[t] == 0 || all_aligned16({w[l]}));
            p.w[l][t] = w[l];
            p.bias[l][t] = b[l];
        }
        p.count[t] = acs[t];
        p.row_start[t] = row;
        p.tile_start[t] = tiles;
        row += acs[t];
        tiles += (acs[t] + kCeluRows - 1) / kCeluRows;
    }
    p.tile_start[kTypes] = tiles;
    if (tiles == 0) return ANI_OK;
    if (!all_aligned16({z1, z2, z3})) return ANI_ERR_MISALIGNED;
    static thread_local int configured_dev = -1;
    int dev = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    if (configured_dev != dev) {
        if (int rc = set_smem(celu_preactivations_kernel, sizeof(CeluPreShared))) return rc;
        configured_dev = dev;
    }
    ANI_CUDA(launch_chain(celu_preactivations_kernel, tiles, kCeluThreads, sizeof(CeluPreShared), st, 1, p));
    return ANI_OK;
}

// True when every element that has atoms comes with packed weights.
bool all_packed(const void* const* packed, const int* acs)
{
    for (int t = 0; t < kTypes; t++)
        if (acs[t] > 0 && !packed[t]) return false;
    return true;
}

// Adds the weight gradients of the first n_sets sets of p (counts and ranges are set here).
int wgrad_call(MlpWgradSets& p, const int* acs, int n_sets, int split_precision, cudaStream_t st)
{
    // atoms per CTA: the smallest multiple of 32 for which the grid fits the SMs once (the kernel runs one CTA per
    // SM, so a second partial wave would double the time), but no fewer than a chunk for each of its four groups
    int dev = 0, sms = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    ANI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    int range = kChainGroups * kPipeK;
    for (;; range += kPipeK) {
        long long ctas = 0;
        for (int t = 0; t < kTypes; t++) ctas += (acs[t] + range - 1) / range;
        if (ctas * kWgradBlocks * n_sets <= sms || range >= (1 << 20)) break;
    }
    p.range = range;
    int ranges = 0;
    for (int t = 0; t < kTypes; t++) {
        p.count[t] = acs[t];
        p.range_start[t] = ranges;
        ranges += (acs[t] + range - 1) / range;
    }
    p.range_start[kTypes] = ranges;
    return split_precision ? mlp_wgrad_launch<true>(p, ranges, n_sets, st) : mlp_wgrad_launch<false>(p, ranges, n_sets, st);
}

// ani_mlp_backward_f32, with dL/dA_l of the two inner layers in r1 and r2 (element-sorted rows) when given.
int backward_call(const ani_mlp_backward_args* a, const int* acs_host, int split_precision, float* r1, float* r2,
                  cudaStream_t st)
{
    long long n_atoms = 0;
    if (!a) return ANI_ERR_NULL_POINTER;
    if (int rc = check_acs(acs_host, &n_atoms)) return rc;
    if (n_atoms == 0) return ANI_OK;
    MlpBackwardParams p;
    int tiles = 0, row = 0;
    for (int t = 0; t < kTypes; t++) {
        p.tile_start[t] = tiles;
        p.count[t] = acs_host[t];
        tiles += (acs_host[t] + kMlpTile - 1) / kMlpTile;
        if (acs_host[t] > 0 && (!a->grad_energy[t] || !a->w1[t] || !a->w2[t] || !a->w3[t] || !a->w4[t] ||
                                !a->dact1[t] || !a->dact2[t] || !a->dact3[t] || !a->dz1[t] || !a->dz2[t] ||
                                !a->dz3[t]))
            return ANI_ERR_NULL_POINTER;
        if (acs_host[t] > 0 && !all_aligned16({a->w1[t], a->w2[t], a->w3[t], a->dact1[t], a->dact2[t], a->dact3[t],
                                               a->dz1[t], a->dz2[t], a->dz3[t], a->grad_features[t]}))
            return ANI_ERR_MISALIGNED;
        p.grad_energy[t] = a->grad_energy[t];
        p.w1[t] = a->w1[t]; p.w2[t] = a->w2[t]; p.w3[t] = a->w3[t]; p.w4[t] = a->w4[t];
        p.dact1[t] = a->dact1[t]; p.dact2[t] = a->dact2[t]; p.dact3[t] = a->dact3[t];
        p.dz1[t] = a->dz1[t]; p.dz2[t] = a->dz2[t]; p.dz3[t] = a->dz3[t];
        p.grad_feat[t] = a->grad_features[t];
        p.r1[t] = r1 && acs_host[t] > 0 ? r1 + (size_t)row * kMlpH1 : nullptr;
        p.r2[t] = r2 && acs_host[t] > 0 ? r2 + (size_t)row * kMlpH2 : nullptr;
        row += acs_host[t];
        if (reinterpret_cast<uintptr_t>(a->packed[t]) & 15) return ANI_ERR_MISALIGNED;
    }
    p.tile_start[kTypes] = tiles;
    if (all_packed(a->packed, acs_host)) {
        MlpChainParams c = {};
        for (int t = 0; t <= kTypes; t++) c.tile_start[t] = p.tile_start[t];
        for (int t = 0; t < kTypes; t++) {
            c.count[t] = p.count[t];
            c.packed[t] = (const unsigned char*)a->packed[t];
            c.w4[t] = p.w4[t];
            c.grad_energy[t] = p.grad_energy[t];
            c.dact1[t] = const_cast<float*>(p.dact1[t]);
            c.dact2[t] = const_cast<float*>(p.dact2[t]);
            c.dact3[t] = const_cast<float*>(p.dact3[t]);
            c.dz1[t] = p.dz1[t]; c.dz2[t] = p.dz2[t]; c.dz3[t] = p.dz3[t];
            c.r1[t] = p.r1[t]; c.r2[t] = p.r2[t];
            c.grad_feat[t] = p.grad_feat[t];
        }
        return mlp_chain_act<kChainBackward>(c, kActCelu, split_precision != 0, st);
    }
    return split_precision ? mlp_backward_launch<true>(p, tiles, st) : mlp_backward_launch<false>(p, tiles, st);
}

template <int ACT> int mlp_launch_act(const MlpParams& p, int n_tiles, bool split, cudaStream_t st)
{
    return split ? mlp_launch<ACT, true>(p, n_tiles, st) : mlp_launch<ACT, false>(p, n_tiles, st);
}

}  // namespace

extern "C" {

int ani_feature_size(void) { return ani::kTotal; }

const char* ani_status_string(int status)
{
    switch (status) {
        case ANI_OK: return "ok";
        case ANI_ERR_NULL_POINTER: return "a required pointer argument is NULL";
        case ANI_ERR_BAD_SIZE: return "negative or inconsistent size argument";
        case ANI_ERR_CUDA: return "CUDA runtime error (see ani_last_cuda_error)";
        case ANI_ERR_BAD_ELEMENT: return "element id outside 0..3 in atomic_numbers";
        case ANI_ERR_BAD_INDEX: return "molecule offset/count or scatter index out of range";
        case ANI_ERR_TOO_MANY_ATOMS: return "size beyond what this entry point supports";
        case ANI_ERR_TIMEOUT: return "a bounded device-side wait ran out";
        case ANI_ERR_MISALIGNED: return "a pointer that must be 16-byte aligned is not";
        case ANI_ERR_CAPTURE:
            return "first-use set-up (scratch allocation or address look-up) cannot run while the stream is being "
                   "captured: make the same call once outside the capture";
        default: return "unknown status";
    }
}

const char* ani_last_cuda_error(void) { return cudaGetErrorString(t_last_error); }

int ani_device_status(void* stream)
{
    ANI_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    int v = 0;
    ANI_CUDA(cudaMemcpyFromSymbol(&v, ani::g_status, sizeof(int)));
    if (v != 0) {
        const int zero = 0;
        ANI_CUDA(cudaMemcpyToSymbol(ani::g_status, &zero, sizeof(int)));
    }
    return v;
}

int ani_sort(const int* atomic_numbers, int n_atoms, int* scatter_idxs, int* gather_idxs,
             int* atom_counts, void* stream)
{
    if (n_atoms < 0) return ANI_ERR_BAD_SIZE;
    if (!atom_counts) return ANI_ERR_NULL_POINTER;
    cudaStream_t st = (cudaStream_t)stream;
    if (n_atoms == 0) {
        sort_empty_kernel<<<1, 32, 0, st>>>(atom_counts);
        ANI_CUDA(cudaGetLastError());
        return ANI_OK;
    }
    if (!atomic_numbers || !scatter_idxs || !gather_idxs) return ANI_ERR_NULL_POINTER;
    const int n_tiles = (n_atoms + kSortTile - 1) / kSortTile;
    if (n_atoms <= kSortSingleLaunchMax) {
        ANI_CUDA(launch_chain(sort_single_kernel, n_tiles, kSortThreads, 0, st, 1, atomic_numbers, n_atoms, scatter_idxs,
                              gather_idxs, atom_counts));
        return ANI_OK;
    }
    int* scratch = nullptr;
    if (int rc = sort_scratch((size_t)(n_tiles + 1) * kTypes * sizeof(int), st, &scratch)) return rc;
    sort_histogram_kernel<<<n_tiles, kSortThreads, 0, st>>>(atomic_numbers, n_atoms, scratch);
    ANI_CUDA(cudaGetLastError());
    sort_scan_kernel<<<1, kSortThreads, 0, st>>>(scratch, n_tiles);
    ANI_CUDA(cudaGetLastError());
    sort_rank_kernel<<<n_tiles, kSortThreads, 0, st>>>(atomic_numbers, n_atoms, scratch, n_tiles,
                                                       scatter_idxs, gather_idxs, atom_counts);
    ANI_CUDA(cudaGetLastError());
    return ANI_OK;
}

int ani_sort_noalloc(const int* atomic_numbers, int n_atoms, int* scatter_idxs, int* gather_idxs,
                     int* atom_counts, void* stream)
{
    if (n_atoms < 0) return ANI_ERR_BAD_SIZE;
    if (n_atoms > kSortStaticMaxAtoms) return ANI_ERR_TOO_MANY_ATOMS;
    if (!atom_counts) return ANI_ERR_NULL_POINTER;
    cudaStream_t st = (cudaStream_t)stream;
    if (n_atoms == 0) {
        sort_empty_kernel<<<1, 32, 0, st>>>(atom_counts);
        ANI_CUDA(cudaGetLastError());
        return ANI_OK;
    }
    if (!atomic_numbers || !scatter_idxs || !gather_idxs) return ANI_ERR_NULL_POINTER;
    int* scratch = nullptr;
    if (int rc = sort_static_scratch(st, &scratch)) return rc;
    // Every scratch entry that is read is written first by the same call (the histogram kernel
    // fills entries [0, n_tiles), the scan kernel entry n_tiles), so nothing has to be cleared.
    const int n_tiles = (n_atoms + kSortTile - 1) / kSortTile;
    sort_histogram_kernel<<<n_tiles, kSortThreads, 0, st>>>(atomic_numbers, n_atoms, scratch);
    ANI_CUDA(cudaGetLastError());
    sort_scan_kernel<<<1, kSortThreads, 0, st>>>(scratch, n_tiles);
    ANI_CUDA(cudaGetLastError());
    sort_rank_kernel<<<n_tiles, kSortThreads, 0, st>>>(atomic_numbers, n_atoms, scratch, n_tiles,
                                                       scatter_idxs, gather_idxs, atom_counts);
    ANI_CUDA(cudaGetLastError());
    return ANI_OK;
}

int ani_sort_noalloc_max_atoms(void) { return kSortStaticMaxAtoms; }

int ani_featurize_f32(const float* xs, const float* ys, const float* zs, const int* atomic_numbers,
                      const int* mol_offsets, const int* mol_atom_counts, int n_mols,
                      const int* scatter_idxs, float* out_h, float* out_c, float* out_n,
                      float* out_o, const int* acs_host, void* stream)
{
    return featurize_impl<float>(xs, ys, zs, atomic_numbers, mol_offsets, mol_atom_counts, n_mols,
                                 scatter_idxs, out_h, out_c, out_n, out_o, acs_host, stream);
}

int ani_featurize_f64(const double* xs, const double* ys, const double* zs,
                      const int* atomic_numbers, const int* mol_offsets, const int* mol_atom_counts,
                      int n_mols, const int* scatter_idxs, double* out_h, double* out_c,
                      double* out_n, double* out_o, const int* acs_host, void* stream)
{
    return featurize_impl<double>(xs, ys, zs, atomic_numbers, mol_offsets, mol_atom_counts, n_mols,
                                  scatter_idxs, out_h, out_c, out_n, out_o, acs_host, stream);
}

int ani_featurize_grad_f32(const float* xs, const float* ys, const float* zs,
                           const int* atomic_numbers, const int* mol_offsets,
                           const int* mol_atom_counts, int n_mols, const int* scatter_idxs,
                           const float* grad_h, const float* grad_c, const float* grad_n,
                           const float* grad_o, float* x_grads, float* y_grads, float* z_grads,
                           const int* acs_host, void* stream)
{
    return featurize_grad_impl<float>(xs, ys, zs, atomic_numbers, mol_offsets, mol_atom_counts,
                                      n_mols, scatter_idxs, grad_h, grad_c, grad_n, grad_o,
                                      x_grads, y_grads, z_grads, acs_host, stream);
}

int ani_featurize_grad_f64(const double* xs, const double* ys, const double* zs,
                           const int* atomic_numbers, const int* mol_offsets,
                           const int* mol_atom_counts, int n_mols, const int* scatter_idxs,
                           const double* grad_h, const double* grad_c, const double* grad_n,
                           const double* grad_o, double* x_grads, double* y_grads,
                           double* z_grads, const int* acs_host, void* stream)
{
    return featurize_grad_impl<double>(xs, ys, zs, atomic_numbers, mol_offsets, mol_atom_counts,
                                       n_mols, scatter_idxs, grad_h, grad_c, grad_n, grad_o,
                                       x_grads, y_grads, z_grads, acs_host, stream);
}

int ani_featurize_grad_inverse_f32(const float* xs, const float* ys, const float* zs,
                                   const int* atomic_numbers, const int* mol_offsets,
                                   const int* mol_atom_counts, int n_mols, const int* scatter_idxs,
                                   const float* x_grads, const float* y_grads, const float* z_grads,
                                   float* out_h, float* out_c, float* out_n, float* out_o,
                                   const int* acs_host, void* stream)
{
    return featurize_grad_inverse_impl<float>(xs, ys, zs, atomic_numbers, mol_offsets,
                                              mol_atom_counts, n_mols, scatter_idxs, x_grads,
                                              y_grads, z_grads, out_h, out_c, out_n, out_o,
                                              acs_host, stream);
}

int ani_featurize_grad_inverse_f64(const double* xs, const double* ys, const double* zs,
                                   const int* atomic_numbers, const int* mol_offsets,
                                   const int* mol_atom_counts, int n_mols, const int* scatter_idxs,
                                   const double* x_grads, const double* y_grads,
                                   const double* z_grads, double* out_h, double* out_c,
                                   double* out_n, double* out_o, const int* acs_host, void* stream)
{
    return featurize_grad_inverse_impl<double>(xs, ys, zs, atomic_numbers, mol_offsets,
                                               mol_atom_counts, n_mols, scatter_idxs, x_grads,
                                               y_grads, z_grads, out_h, out_c, out_n, out_o,
                                               acs_host, stream);
}

int ani_mlp_forward_f32(const ani_mlp_args* a, const int* acs_host, int activation,
                        int split_precision, void* stream)
{
    long long n_atoms = 0;
    if (!a) return ANI_ERR_NULL_POINTER;
    if (int rc = check_acs(acs_host, &n_atoms)) return rc;
    if (activation < 0 || activation > 3) return ANI_ERR_BAD_SIZE;
    if (n_atoms == 0) return ANI_OK;
    MlpParams p;
    int tiles = 0;
    for (int t = 0; t < kTypes; t++) {
        p.tile_start[t] = tiles;
        p.count[t] = acs_host[t];
        tiles += (acs_host[t] + kMlpTile - 1) / kMlpTile;
        if (acs_host[t] > 0 && (!a->features[t] || !a->w1[t] || !a->b1[t] || !a->w2[t] || !a->b2[t] ||
                                !a->w3[t] || !a->b3[t] || !a->w4[t] || !a->b4[t] || !a->energy[t]))
            return ANI_ERR_NULL_POINTER;
        if (acs_host[t] > 0 && !all_aligned16({a->features[t], a->w1[t], a->w2[t], a->w3[t], a->act1[t], a->act2[t],
                                               a->act3[t], a->dact1[t], a->dact2[t], a->dact3[t]}))
            return ANI_ERR_MISALIGNED;
        p.feat[t] = a->features[t];
        p.w1[t] = a->w1[t]; p.b1[t] = a->b1[t];
        p.w2[t] = a->w2[t]; p.b2[t] = a->b2[t];
        p.w3[t] = a->w3[t]; p.b3[t] = a->b3[t];
        p.w4[t] = a->w4[t];   p.b4[t] = a->b4[t];
        p.energy[t] = a->energy[t];
        p.act1[t] = a->act1[t]; p.act2[t] = a->act2[t]; p.act3[t] = a->act3[t];
        p.dact1[t] = a->dact1[t]; p.dact2[t] = a->dact2[t]; p.dact3[t] = a->dact3[t];
        if (reinterpret_cast<uintptr_t>(a->packed[t]) & 15) return ANI_ERR_MISALIGNED;
    }
    p.tile_start[kTypes] = tiles;
    cudaStream_t st = (cudaStream_t)stream;
    const bool split = split_precision != 0;
    if (all_packed(a->packed, acs_host)) {
        MlpChainParams c = {};
        for (int t = 0; t <= kTypes; t++) c.tile_start[t] = p.tile_start[t];
        for (int t = 0; t < kTypes; t++) {
            c.count[t] = p.count[t];
            c.packed[t] = (const unsigned char*)a->packed[t];
            c.feat[t] = p.feat[t];
            c.b1[t] = p.b1[t]; c.b2[t] = p.b2[t]; c.b3[t] = p.b3[t]; c.b4[t] = p.b4[t];
            c.w4[t] = p.w4[t];
            c.energy[t] = p.energy[t];
            c.act1[t] = p.act1[t]; c.act2[t] = p.act2[t]; c.act3[t] = p.act3[t];
            c.dact1[t] = p.dact1[t]; c.dact2[t] = p.dact2[t]; c.dact3[t] = p.dact3[t];
        }
        return mlp_chain_act<kChainForward>(c, activation, split, st);
    }
    switch (activation) {
        case kActCelu: return mlp_launch_act<kActCelu>(p, tiles, split, st);
        case kActGaussian: return mlp_launch_act<kActGaussian>(p, tiles, split, st);
        case kActNormal: return mlp_launch_act<kActNormal>(p, tiles, split, st);
        default: return mlp_launch_act<kActSoftplus>(p, tiles, split, st);
    }
}

size_t ani_mlp_packed_bytes(void) { return (size_t)kPackChunks * kPackedChunkBytes; }

int ani_mlp_pack_weights_f32(const ani_mlp_pack_args* a, void* stream)
{
    if (!a) return ANI_ERR_NULL_POINTER;
    MlpPackParams p;
    bool any = false;
    if (int rc = pack_params(a->w1, a->w2, a->w3, a->packed, &p, &any)) return rc;
    return any ? pack_launch(p, (cudaStream_t)stream) : ANI_OK;
}

int ani_mlp_backward_f32(const ani_mlp_backward_args* a, const int* acs_host, int split_precision,
                         void* stream)
{
    return backward_call(a, acs_host, split_precision, nullptr, nullptr, (cudaStream_t)stream);
}
int ani_mlp_weight_grad_f32(const ani_mlp_weight_grad_args* a, const int* acs_host, int split_precision,
                            void* stream)
{
    long long n_atoms = 0;
    if (!a) return ANI_ERR_NULL_POINTER;
    if (int rc = check_acs(acs_host, &n_atoms)) return rc;
    if (n_atoms == 0) return ANI_OK;
    MlpWgradSets sets = {};
    MlpWgradParams& p = sets.set[0];
    for (int t = 0; t < kTypes; t++) {
        if (acs_host[t] > 0 && (!a->features[t] || !a->act1[t] || !a->act2[t] || !a->dz1[t] || !a->dz2[t] ||
                                !a->dz3[t] || !a->dw1[t] || !a->dw2[t] || !a->dw3[t] || !a->db1[t] ||
                                !a->db2[t] || !a->db3[t] || !a->act3[t] || !a->grad_energy[t] ||
                                !a->dw4[t] || !a->db4[t]))
            return ANI_ERR_NULL_POINTER;
        if (acs_host[t] > 0) {
            const void* vec[] = {a->features[t], a->act1[t], a->act2[t], a->act3[t], a->dz1[t], a->dz2[t],
                                 a->dz3[t], a->dw1[t], a->dw2[t], a->dw3[t]};
            for (const void* ptr : vec)
                if (reinterpret_cast<uintptr_t>(ptr) & 15) return ANI_ERR_MISALIGNED;
        }
        p.feat[t] = a->features[t]; p.act1[t] = a->act1[t]; p.act2[t] = a->act2[t];
        p.dz1[t] = a->dz1[t]; p.dz2[t] = a->dz2[t]; p.dz3[t] = a->dz3[t];
        p.dw1[t] = a->dw1[t]; p.dw2[t] = a->dw2[t]; p.dw3[t] = a->dw3[t];
        p.db1[t] = a->db1[t]; p.db2[t] = a->db2[t]; p.db3[t] = a->db3[t];
        p.act3[t] = a->act3[t]; p.grad_energy[t] = a->grad_energy[t];
        p.dw4[t] = a->dw4[t]; p.db4[t] = a->db4[t];
    }
    return wgrad_call(sets, acs_host, 1, split_precision, (cudaStream_t)stream);
}

int ani_molecule_energy_f32(const float* atom_energy_sorted, const int* gather_idxs, const int* mol_offsets,
                            const int* mol_atom_counts, int n_mols, int n_atoms, const float* labels,
                            float grad_scale, float* mol_energy, float* l2s, float* grad_atom_energy_sorted,
                            void* stream)
{
    if (n_mols < 0 || n_atoms < 0) return ANI_ERR_BAD_SIZE;
    if (n_mols == 0) return ANI_OK;
    if (!mol_offsets || !mol_atom_counts || !mol_energy) return ANI_ERR_NULL_POINTER;
    if (n_atoms > 0 && (!atom_energy_sorted || !gather_idxs)) return ANI_ERR_NULL_POINTER;
    return energy_launch<float>(atom_energy_sorted, gather_idxs, mol_offsets, mol_atom_counts, n_mols, n_atoms, labels,
                                grad_scale, mol_energy, l2s, grad_atom_energy_sorted, (cudaStream_t)stream);
}

int ani_nadam_step_f32(float* params, const float* grads, float* m, float* v, float* ema,
                       long long n, const float* hyper, void* state, void* stream)
{
    if (n < 0) return ANI_ERR_BAD_SIZE;
    if (n == 0) return ANI_OK;
    if (!params || !grads || !m || !v || !hyper || !state) return ANI_ERR_NULL_POINTER;
    int dev = 0, sms = 0;
    ANI_CUDA(cudaGetDevice(&dev));
    ANI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const long long want = (n + 4 * kOptimThreads - 1) / (4 * kOptimThreads);
    const int grid = (int)(want < (long long)sms * 4 ? want : (long long)sms * 4);
    cudaStream_t st = (cudaStream_t)stream;
    if (want > 0x7fffffffLL) return ANI_ERR_BAD_SIZE;
    ANI_CUDA(launch_chain(grad_sumsq_kernel, grid, kOptimThreads, 0, st, 1, grads, n, (OptimState*)state));
    ANI_CUDA(launch_chain(nadam_update_kernel, (int)want, kOptimThreads, 0, st, 1, params, grads, m, v, ema, n,
                          (const OptimHyper*)hyper, (OptimState*)state));
    return ANI_OK;
}

int ani_clip_rows_f32(float* params, const int* row_offsets, const int* row_lengths, int n_rows, float max_norm,
                      void* stream)
{
    if (n_rows < 0 || !(max_norm > 0.0f)) return ANI_ERR_BAD_SIZE;
    if (n_rows == 0) return ANI_OK;
    if (!params || !row_offsets || !row_lengths) return ANI_ERR_NULL_POINTER;
    const int per_block = kOptimThreads / kWarp;
    const int grid = (n_rows + per_block - 1) / per_block;
    ANI_CUDA(launch_chain(clip_rows_kernel, grid, kOptimThreads, 0, (cudaStream_t)stream, 1, params, row_offsets, row_lengths,
                          n_rows, max_norm));
    return ANI_OK;
}

int ani_scale_by_loss_f32(float* grads, long long n, const float* l2s, int n_mols, int kind, float* rmse_out,
                          void* stream)
{
    if (n < 0 || n_mols <= 0 || (kind != 1 && kind != 2)) return ANI_ERR_BAD_SIZE;
    if (!l2s || (n > 0 && !grads)) return ANI_ERR_NULL_POINTER;
    const long long blocks = std::max<long long>(1, std::min<long long>((n + kOptimThreads - 1) / kOptimThreads, 296));
    ANI_CUDA(launch_chain(loss_scale_kernel, (int)blocks, kOptimThreads, 0, (cudaStream_t)stream, 1, grads, n, l2s, n_mols,
                          kind, rmse_out));
    return ANI_OK;
}

int ani_charge_f32(const float* xs, const float* ys, const float* zs, const float* qs,
                   const int* mol_offsets, const int* mol_atom_counts, int n_mols, int n_atoms,
                   float* charge_energies, void* stream)
{
    return charge_impl<float>(xs, ys, zs, qs, mol_offsets, mol_atom_counts, n_mols, n_atoms,
                              charge_energies, stream);
}

int ani_charge_f64(const double* xs, const double* ys, const double* zs, const double* qs,
                   const int* mol_offsets, const int* mol_atom_counts, int n_mols, int n_atoms,
                   double* charge_energies, void* stream)
{
    return charge_impl<double>(xs, ys, zs, qs, mol_offsets, mol_atom_counts, n_mols, n_atoms,
                               charge_energies, stream);
}

int ani_charge_grad_f32(const float* xs, const float* ys, const float* zs, const float* qs,
                        const int* mol_offsets, const int* mol_atom_counts, int n_mols, int n_atoms,
                        const float* grads, float* q_grads, void* stream)
{
    return charge_grad_impl<float>(xs, ys, zs, qs, mol_offsets, mol_atom_counts, n_mols, n_atoms,
                                   grads, q_grads, stream);
}

int ani_charge_grad_f64(const double* xs, const double* ys, const double* zs, const double* qs,
                        const int* mol_offsets, const int* mol_atom_counts, int n_mols, int n_atoms,
                        const double* grads, double* q_grads, void* stream)
{
    return charge_grad_impl<double>(xs, ys, zs, qs, mol_offsets, mol_atom_counts, n_mols, n_atoms,
                                    grads, q_grads, stream);
}

int ani_host_pack_batch(const ani_host_pack_args* args)
{
    if (!args) return ANI_ERR_NULL_POINTER;
    return ani::host_pack_batch(*args);
}

struct ani_feeder {
    ani::Feeder impl;
    ani_feeder(int device, const ani_feeder_slot* slots, int n) : impl(device, slots, n) {}
};

int ani_feeder_create(int device, const ani_feeder_slot* slots, int n_slots, ani_feeder** out)
{
    if (!slots || !out) return ANI_ERR_NULL_POINTER;
    if (n_slots <= 0) return ANI_ERR_BAD_SIZE;
    for (int s = 0; s < n_slots; s++)
        if (!slots[s].host_arena || (device >= 0 && !slots[s].dev_arena)) return ANI_ERR_NULL_POINTER;
    ani_feeder* f = new (std::nothrow) ani_feeder(device, slots, n_slots);
    if (!f) return ANI_ERR_CUDA;
    if (int rc = f->impl.init()) {
        delete f;
        return rc;
    }
    *out = f;
    return ANI_OK;
}

int ani_feeder_begin(ani_feeder* f, const long long* order, long long n_order, int batch_size)
{
    return f ? f->impl.begin(order, n_order, batch_size, nullptr, 0, 0.0) : ANI_ERR_NULL_POINTER;
}

int ani_feeder_begin_fuzz(ani_feeder* f, const long long* order, long long n_order, int batch_size, const unsigned* key,
                          int pos, double fuzz)
{
    return f && key ? f->impl.begin(order, n_order, batch_size, key, pos, fuzz) : ANI_ERR_NULL_POINTER;
}

int ani_feeder_random_state(ani_feeder* f, unsigned* key, int* pos)
{
    return f && key && pos ? f->impl.random_state(key, pos) : ANI_ERR_NULL_POINTER;
}

int ani_feeder_next(ani_feeder* f, ani_feeder_batch* out)
{
    return f && out ? f->impl.next(out) : ANI_ERR_NULL_POINTER;
}

int ani_feeder_wait(ani_feeder* f, int slot, void* stream)
{
    return f ? f->impl.wait(slot, static_cast<cudaStream_t>(stream)) : ANI_ERR_NULL_POINTER;
}

int ani_feeder_release(ani_feeder* f, int slot, void* stream)
{
    return f ? f->impl.release(slot, static_cast<cudaStream_t>(stream)) : ANI_ERR_NULL_POINTER;
}

int ani_feeder_end(ani_feeder* f)
{
    if (!f) return ANI_ERR_NULL_POINTER;
    f->impl.end();
    return ANI_OK;
}

int ani_feeder_destroy(ani_feeder* f)
{
    if (!f) return ANI_OK;
    f->impl.end();
    const int rc = f->impl.drain();
    delete f;
    return rc;
}

int ani_feeder_set_slots(ani_feeder* f, const ani_feeder_slot* slots, int n_slots)
{
    if (!f || !slots) return ANI_ERR_NULL_POINTER;
    for (int s = 0; s < n_slots; s++)
        if (!slots[s].host_arena) return ANI_ERR_NULL_POINTER;
    return f->impl.set_slots(slots, n_slots);
}

struct ani_driver {
    ani::Driver impl;
    explicit ani_driver(const ani_driver_args& a) : impl(a) {}
};

size_t ani_driver_weights_bytes(int double_precision) { return ani::weights_bytes(double_precision != 0); }

int ani_driver_create(const ani_driver_args* a, ani_driver** out)
{
    if (!a || !out || !a->slots || !a->streams[0]) return ANI_ERR_NULL_POINTER;
    if (a->n_slots <= 0 || a->mode < ANI_DRIVER_ENERGIES || a->mode > ANI_DRIVER_TRAIN) return ANI_ERR_BAD_SIZE;
    const bool train = a->mode == ANI_DRIVER_TRAIN;
    if (!train && !a->streams[1]) return ANI_ERR_NULL_POINTER;
    for (int k = 0; k < 2; k++)
        if (!a->pass[k] && (train || !a->pass64[k])) return ANI_ERR_NULL_POINTER;
    if (train && (!a->params || !a->grads || (a->loss_kind && !a->rmse))) return ANI_ERR_NULL_POINTER;
    if (a->mode == ANI_DRIVER_GRADIENTS || (a->mode == ANI_DRIVER_ENERGIES && !a->energies))
        for (void* p : a->ring_host)
            if (!p) return ANI_ERR_NULL_POINTER;
    if (a->mode == ANI_DRIVER_GRADIENTS)
        for (void* p : a->weights) {
            if (!p != !a->weights[0]) return ANI_ERR_NULL_POINTER;
            if (reinterpret_cast<uintptr_t>(p) & 255) return ANI_ERR_MISALIGNED;
        }
    ani_driver* d = new (std::nothrow) ani_driver(*a);
    if (!d) return ANI_ERR_CUDA;
    if (int rc = d->impl.init()) {
        delete d;
        return rc;
    }
    *out = d;
    return ANI_OK;
}

int ani_driver_step(ani_driver* d, ani_feeder* f, void* stream, ani_feeder_batch* batch)
{
    return d && f && batch ? d->impl.step(f->impl, static_cast<cudaStream_t>(stream), batch) : ANI_ERR_NULL_POINTER;
}

int ani_driver_wait(ani_driver* d, int place) { return d ? d->impl.wait(place) : ANI_ERR_NULL_POINTER; }

int ani_driver_join(ani_driver* d, void* stream)
{
    return d ? d->impl.join(static_cast<cudaStream_t>(stream)) : ANI_ERR_NULL_POINTER;
}

int ani_driver_destroy(ani_driver* d)
{
    delete d;
    return ANI_OK;
}

struct ani_peer {
    int device = 0, rank = 0, world = 1, grid = 1;
    int two_halves = 0;                  // slice means + exchange (more than four ranks)
    long long capacity = 0;              // floats per staging buffer
    unsigned char* block = nullptr;      // local: [flags | staging 0 | staging 1]
    ani::PeerState* state = nullptr;     // local
    unsigned char* peer_block[ani::kPeerMaxRanks] = {};
    bool mapped[ani::kPeerMaxRanks] = {};   // opened through CUDA IPC (to be closed)
};

int ani_peer_create(int rank, int world, long long n_floats, ani_peer** out)
{
    if (!out) return ANI_ERR_NULL_POINTER;
    if (world < 1 || world > ani::kPeerMaxRanks || rank < 0 || rank >= world || n_floats <= 0) return ANI_ERR_BAD_SIZE;
    ani_peer* p = new (std::nothrow) ani_peer();
    if (!p) return ANI_ERR_CUDA;
    p->rank = rank;
    p->world = world;
    p->capacity = (n_floats + 3) / 4 * 4;
    cudaDeviceProp prop;
    cudaError_t e = cudaGetDevice(&p->device);
    if (e == cudaSuccess) e = cudaGetDeviceProperties(&prop, p->device);
    // [flags | staging 0, 1 (every rank's contribution) | staging 2, 3 (this rank's slice means)]
    const size_t bytes = ani::kPeerFlagBytes + 4 * (size_t)p->capacity * sizeof(float);
    if (e == cudaSuccess) e = cudaMalloc(&p->block, bytes);
    if (e == cudaSuccess) e = cudaMemset(p->block, 0, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&p->state, sizeof(ani::PeerState));
    if (e == cudaSuccess) {
        ani::PeerState init{0ull, 0ull, 0ull, 0u, ani::kPeerSpinLimit};
        e = cudaMemcpy(p->state, &init, sizeof(init), cudaMemcpyHostToDevice);
    }
    if (e != cudaSuccess) {
        if (p->block) cudaFree(p->block);
        if (p->state) cudaFree(p->state);
        delete p;
        return cuda_fail(e);
    }
    const long long groups = p->capacity / 4;
    p->grid = (int)std::max<long long>(1, std::min<long long>((groups + ani::kPeerThreads - 1) / ani::kPeerThreads,
                                                               std::min(prop.multiProcessorCount, ani::kPeerMaxBlocks)));
    p->peer_block[rank] = p->block;
    p->two_halves = world > 4 ? 1 : 0;
    *out = p;
    return ANI_OK;
}

int ani_peer_handle(ani_peer* p, void* out64)
{
    if (!p || !out64) return ANI_ERR_NULL_POINTER;
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "the handle is exchanged as 64 bytes");
    cudaIpcMemHandle_t h;
    ANI_CUDA(cudaIpcGetMemHandle(&h, p->block));
    memcpy(out64, &h, sizeof(h));
    return ANI_OK;
}

int ani_peer_connect(ani_peer* p, int q, const void* handle64)
{
    if (!p || !handle64) return ANI_ERR_NULL_POINTER;
    if (q < 0 || q >= p->world || q == p->rank || p->peer_block[q]) return ANI_ERR_BAD_INDEX;
    cudaIpcMemHandle_t h;
    memcpy(&h, handle64, sizeof(h));
    void* ptr = nullptr;
    ANI_CUDA(cudaIpcOpenMemHandle(&ptr, h, cudaIpcMemLazyEnablePeerAccess));
    p->peer_block[q] = static_cast<unsigned char*>(ptr);
    p->mapped[q] = true;
    return ANI_OK;
}

int ani_peer_connect_raw(ani_peer* p, int q, void* block)
{
    if (!p || !block) return ANI_ERR_NULL_POINTER;
    if (q < 0 || q >= p->world || q == p->rank || p->peer_block[q]) return ANI_ERR_BAD_INDEX;
    p->peer_block[q] = static_cast<unsigned char*>(block);
    return ANI_OK;
}

void* ani_peer_block(ani_peer* p) { return p ? p->block : nullptr; }

int ani_peer_set_two_halves(ani_peer* p, int on)
{
    if (!p) return ANI_ERR_NULL_POINTER;
    p->two_halves = on ? 1 : 0;
    return ANI_OK;
}

int ani_peer_set_spin_limit(ani_peer* p, unsigned tries)
{
    if (!p) return ANI_ERR_NULL_POINTER;
    ANI_CUDA(cudaMemcpy(&p->state->spin_limit, &tries, sizeof(tries), cudaMemcpyHostToDevice));
    return ANI_OK;
}

int ani_peer_mean_f32(ani_peer* p, float* buffer, long long n, void* stream)
{
    if (!p || !buffer) return ANI_ERR_NULL_POINTER;
    if (n < 0 || n > p->capacity || (n & 3)) return ANI_ERR_BAD_SIZE;
    if (reinterpret_cast<uintptr_t>(buffer) & 15) return ANI_ERR_MISALIGNED;
    ani::PeerParams a{};
    a.buffer = buffer;
    a.n4 = n / 4;
    a.stage_floats = p->capacity;
    a.rank = p->rank;
    a.world = p->world;
    for (int q = 0; q < p->world; q++) {
        if (!p->peer_block[q]) return ANI_ERR_NULL_POINTER;   // a rank that was never connected
        a.flags[q] = reinterpret_cast<unsigned*>(p->peer_block[q]);
        a.stage[q] = reinterpret_cast<float*>(p->peer_block[q] + ani::kPeerFlagBytes);
    }
    a.state = p->state;
    a.inv_world = 1.0f / (float)p->world;
    a.two_halves = p->two_halves;
    ani::peer_mean_kernel<<<p->grid, ani::kPeerThreads, 0, (cudaStream_t)stream>>>(a);
    ANI_CUDA(cudaGetLastError());
    return ANI_OK;
}

int ani_peer_destroy(ani_peer* p)
{
    if (!p) return ANI_OK;
    cudaDeviceSynchronize();
    for (int q = 0; q < p->world; q++)
        if (p->mapped[q]) cudaIpcCloseMemHandle(p->peer_block[q]);
    cudaFree(p->block);
    cudaFree(p->state);
    delete p;
    return ANI_OK;
}

int ani_network_pass_f32(const ani_pass_args* a, void* stream)
{
    if (!a) return ANI_ERR_NULL_POINTER;
    long long n_atoms = 0;
    if (int rc = check_acs(a->acs_host, &n_atoms)) return rc;
    if (a->n_atoms < 0 || a->n_mols < 0 || n_atoms != a->n_atoms) return ANI_ERR_BAD_SIZE;
    const int* acs = a->acs_host;
    size_t start[kTypes];   // first row of each element
    size_t at = 0;
    for (int t = 0; t < kTypes; t++) {
        start[t] = at;
        at += (size_t)acs[t];
    }
    auto rows = [&](float* base, int t, int width) -> float* {
        return base && acs[t] > 0 ? base + start[t] * (size_t)width : nullptr;
    };
    const bool transient = (a->phases & ANI_PASS_TRANSIENT) != 0;
    const bool small_networks = (a->phases & ANI_PASS_FORWARD) && transient && few_atoms(acs) &&
                                !(a->phases & ANI_PASS_WEIGHT_GRAD) && !a->labels;
    bool sorted = false, pack_later = false;
    MlpPackParams p = {};
    if (a->phases & ANI_PASS_PACK) {
        bool any = false;
        if (int rc = pack_params(a->w1, a->w2, a->w3, a->packed, &p, &any)) return rc;
        // networks of few atoms do not read the packed weights: packed beside them, on SMs that have nothing to do
        if (any && small_networks && n_atoms > 0) {
            pack_later = true;
            any = false;
        }
        // with a sort of one launch in the same pass: both in one kernel
        if (any && (a->phases & ANI_PASS_FEATURIZE) && n_atoms > 0 && n_atoms <= kSortSingleLaunchMax) {
            if (!a->atomic_numbers || !a->scatter_idxs || !a->gather_idxs || !a->atom_counts) return ANI_ERR_NULL_POINTER;
            const int n_tiles = (int)((n_atoms + kSortTile - 1) / kSortTile);
            ANI_CUDA(launch_chain(sort_and_pack_kernel, n_tiles + kPackChunks * kTypes, kSortThreads, 0, (cudaStream_t)stream,
                                  1, a->atomic_numbers, (int)n_atoms, n_tiles, a->scatter_idxs, a->gather_idxs,
                                  a->atom_counts, p));
            sorted = true;
        } else if (any) {
            if (int rc = pack_launch(p, (cudaStream_t)stream)) return rc;
        }
    }
    if (a->phases & ANI_PASS_FEATURIZE) {
        if (!sorted)
            if (int rc = ani_sort(a->atomic_numbers, a->n_atoms, a->scatter_idxs, a->gather_idxs, a->atom_counts, stream))
                return rc;
        if (int rc = featurize_impl<float>(a->xs, a->ys, a->zs, a->atomic_numbers, a->mol_offsets, a->mol_atom_counts,
                                           a->n_mols, a->scatter_idxs, rows(a->features, 0, kTotal),
                                           rows(a->features, 1, kTotal), rows(a->features, 2, kTotal),
                                           rows(a->features, 3, kTotal), acs, stream, n_atoms <= kSortSingleLaunchMax))
            return rc;
    }
    bool backward_done = false;
    if (small_networks) {
        const bool backward = (a->phases & ANI_PASS_BACKWARD) && a->feature_grads;
        if (n_atoms > 0)
            if (int rc = mlp_small_launch<float>(a->features, acs, a->w1, a->b1, a->w2, a->b2, a->w3, a->b3, a->w4, a->b4,
                                                 a->grad_energy_sorted, a->energy_sorted,
                                                 backward ? a->feature_grads : nullptr, a->activation,
                                                 (a->phases & ANI_PASS_FEATURIZE) != 0, (cudaStream_t)stream,
                                                 pack_later ? &p : nullptr))
                return rc;
        backward_done = true;
    } else if ((a->phases & ANI_PASS_FORWARD) && (a->phases & ANI_PASS_BACKWARD) && transient && a->feature_grads &&
               !(a->phases & ANI_PASS_WEIGHT_GRAD) && !a->labels && n_atoms > 0 && all_packed(a->packed, acs)) {
        // energies + forces: forward and backward of a tile in one kernel, nothing of the networks in global memory
        if (a->activation < 0 || a->activation > 3) return ANI_ERR_BAD_SIZE;
        if (!a->features || !a->energy_sorted) return ANI_ERR_NULL_POINTER;
        if (!all_aligned16({a->features, a->feature_grads})) return ANI_ERR_MISALIGNED;
        MlpChainParams c = {};
        int tiles = 0;
        for (int t = 0; t < kTypes; t++) {
            c.tile_start[t] = tiles;
            c.count[t] = acs[t];
            tiles += (acs[t] + kMlpTile - 1) / kMlpTile;
            if (acs[t] == 0) continue;
            if (!a->b1[t] || !a->b2[t] || !a->b3[t] || !a->w4[t] || !a->b4[t]) return ANI_ERR_NULL_POINTER;
            if (!all_aligned16({a->packed[t]})) return ANI_ERR_MISALIGNED;
            c.packed[t] = (const unsigned char*)a->packed[t];
            c.feat[t] = rows(a->features, t, kTotal);
            c.b1[t] = a->b1[t]; c.b2[t] = a->b2[t]; c.b3[t] = a->b3[t]; c.b4[t] = a->b4[t];
            c.w4[t] = a->w4[t];
            c.energy[t] = rows(a->energy_sorted, t, 1);
            c.grad_energy[t] = rows(a->grad_energy_sorted, t, 1);
            c.grad_feat[t] = rows(a->feature_grads, t, kTotal);
        }
        c.tile_start[kTypes] = tiles;
        c.early_weights = (a->phases & ANI_PASS_FEATURIZE) != 0 && a->n_mols > 0;     // the features lie behind the packing
        if (int rc = mlp_chain_act<kChainForces>(c, a->activation, a->split_precision != 0, (cudaStream_t)stream)) return rc;
        backward_done = true;
    } else if (a->phases & ANI_PASS_FORWARD) {
        // what only the backward steps read is not written when they do not follow
        const bool save = !transient || (a->phases & (ANI_PASS_BACKWARD | ANI_PASS_WEIGHT_GRAD));
        const bool save_act = save && (!transient || (a->phases & ANI_PASS_WEIGHT_GRAD));
        ani_mlp_args f;
        for (int t = 0; t < kTypes; t++) {
            f.features[t] = rows(a->features, t, kTotal);
            f.w1[t] = a->w1[t]; f.b1[t] = a->b1[t]; f.w2[t] = a->w2[t]; f.b2[t] = a->b2[t];
            f.w3[t] = a->w3[t]; f.b3[t] = a->b3[t]; f.w4[t] = a->w4[t]; f.b4[t] = a->b4[t];
            f.energy[t] = rows(a->energy_sorted, t, 1);
            f.act1[t] = save_act ? rows(a->act1, t, kMlpH1) : nullptr;
            f.act2[t] = save_act ? rows(a->act2, t, kMlpH2) : nullptr;
            f.act3[t] = save_act ? rows(a->act3, t, kMlpH3) : nullptr;
            f.dact1[t] = save ? rows(a->dact1, t, kMlpH1) : nullptr;
            f.dact2[t] = save ? rows(a->dact2, t, kMlpH2) : nullptr;
            f.dact3[t] = save ? rows(a->dact3, t, kMlpH3) : nullptr;
            f.packed[t] = a->packed[t];
        }
        if (int rc = ani_mlp_forward_f32(&f, acs, a->activation, a->split_precision, stream)) return rc;
    }
    const bool sums_with_grads = (a->phases & ANI_PASS_ENERGY) && (a->phases & ANI_PASS_COORD_GRAD) && !a->labels &&
                                 grad_per_molecule(n_atoms, a->n_mols, {a->feature_grads}) && n_atoms > 0;
    if (sums_with_grads && (!a->energy_sorted || !a->gather_idxs || !a->mol_energy)) return ANI_ERR_NULL_POINTER;
    if ((a->phases & ANI_PASS_ENERGY) && !sums_with_grads) {
        if (int rc = ani_molecule_energy_f32(a->energy_sorted, a->gather_idxs, a->mol_offsets, a->mol_atom_counts,
                                             a->n_mols, a->n_atoms, a->labels, a->grad_scale, a->mol_energy,
                                             a->labels ? a->l2s : nullptr,
                                             a->labels ? a->grad_energy_sorted : nullptr, stream))
            return rc;
    }
    if ((a->phases & ANI_PASS_BACKWARD) && !backward_done) {
        ani_mlp_backward_args b;
        for (int t = 0; t < kTypes; t++) {
            b.grad_energy[t] = rows(a->grad_energy_sorted, t, 1);
            b.w1[t] = a->w1[t]; b.w2[t] = a->w2[t]; b.w3[t] = a->w3[t]; b.w4[t] = a->w4[t];
            b.dact1[t] = rows(a->dact1, t, kMlpH1); b.dact2[t] = rows(a->dact2, t, kMlpH2);
            b.dact3[t] = rows(a->dact3, t, kMlpH3);
            b.dz1[t] = rows(a->dz1, t, kMlpH1); b.dz2[t] = rows(a->dz2, t, kMlpH2); b.dz3[t] = rows(a->dz3, t, kMlpH3);
            b.grad_features[t] = rows(a->feature_grads, t, kTotal);
            b.packed[t] = a->packed[t];
        }
        if (int rc = ani_mlp_backward_f32(&b, acs, a->split_precision, stream)) return rc;
    }
    if (a->phases & ANI_PASS_WEIGHT_GRAD) {
        if (a->zero_ptr && a->zero_bytes)
            ANI_CUDA(cudaMemsetAsync(a->zero_ptr, 0, a->zero_bytes, (cudaStream_t)stream));
        ani_mlp_weight_grad_args w;
        for (int t = 0; t < kTypes; t++) {
            w.features[t] = rows(a->features, t, kTotal);
            w.act1[t] = rows(a->act1, t, kMlpH1); w.act2[t] = rows(a->act2, t, kMlpH2); w.act3[t] = rows(a->act3, t, kMlpH3);
            w.dz1[t] = rows(a->dz1, t, kMlpH1); w.dz2[t] = rows(a->dz2, t, kMlpH2); w.dz3[t] = rows(a->dz3, t, kMlpH3);
            w.dw1[t] = a->dw1[t]; w.dw2[t] = a->dw2[t]; w.dw3[t] = a->dw3[t]; w.dw4[t] = a->dw4[t];
            w.db1[t] = a->db1[t]; w.db2[t] = a->db2[t]; w.db3[t] = a->db3[t]; w.db4[t] = a->db4[t];
            w.grad_energy[t] = rows(a->grad_energy_sorted, t, 1);
        }
        if (int rc = ani_mlp_weight_grad_f32(&w, acs, a->split_precision, stream)) return rc;
    }
    if (a->phases & ANI_PASS_COORD_GRAD) {
        // the kernel before is one of the networks', launched above: it has waited for what came before it
        const bool after_networks = backward_done && n_atoms > 0 && !(a->phases & ANI_PASS_WEIGHT_GRAD) &&
                                    ((a->phases & ANI_PASS_ENERGY) == 0 || sums_with_grads);
        MolEnergySums<float> sums = {};
        if (sums_with_grads) sums = {a->energy_sorted, a->gather_idxs, a->mol_energy};
        if (int rc = featurize_grad_impl<float>(a->xs, a->ys, a->zs, a->atomic_numbers, a->mol_offsets, a->mol_atom_counts,
                                                a->n_mols, a->scatter_idxs, rows(a->feature_grads, 0, kTotal),
                                                rows(a->feature_grads, 1, kTotal), rows(a->feature_grads, 2, kTotal),
                                                rows(a->feature_grads, 3, kTotal), a->x_grads, a->y_grads, a->z_grads,
                                                acs, stream, sums, after_networks))
            return rc;
    }
    return ANI_OK;
}

int ani_energy_pass_f64(const ani_energy_args_f64* a, void* stream)
{
    if (!a) return ANI_ERR_NULL_POINTER;
    long long n_atoms = 0;
    if (int rc = check_acs(a->acs_host, &n_atoms)) return rc;
    if (a->n_atoms < 0 || a->n_mols < 0 || n_atoms != a->n_atoms) return ANI_ERR_BAD_SIZE;
    if ((a->phases & ANI_PASS_BACKWARD) && !(a->phases & ANI_PASS_FORWARD)) return ANI_ERR_BAD_SIZE;
    const int* acs = a->acs_host;
    double *rows[kTypes], *grad_rows[kTypes];
    size_t at = 0;
    for (int t = 0; t < kTypes; t++) {
        rows[t] = a->features && acs[t] > 0 ? a->features + at * kTotal : nullptr;
        grad_rows[t] = a->feature_grads && acs[t] > 0 ? a->feature_grads + at * kTotal : nullptr;
        at += (size_t)acs[t];
    }
    if (a->phases & ANI_PASS_FEATURIZE) {
        if (int rc = ani_sort(a->atomic_numbers, a->n_atoms, a->scatter_idxs, a->gather_idxs, a->atom_counts, stream))
            return rc;
        if (int rc = featurize_impl<double>(a->xs, a->ys, a->zs, a->atomic_numbers, a->mol_offsets, a->mol_atom_counts,
                                            a->n_mols, a->scatter_idxs, rows[0], rows[1], rows[2], rows[3], acs, stream,
                                            n_atoms <= kSortSingleLaunchMax))
            return rc;
    }
    if ((a->phases & ANI_PASS_FORWARD) && n_atoms > 0) {
        const bool backward = (a->phases & ANI_PASS_BACKWARD) != 0;
        if (backward && !a->feature_grads) return ANI_ERR_NULL_POINTER;
        if (int rc = mlp_small_launch<double>(a->features, acs, a->w1, a->b1, a->w2, a->b2, a->w3, a->b3, a->w4, a->b4,
                                              nullptr, a->energy_sorted, backward ? a->feature_grads : nullptr,
                                              a->activation, (a->phases & ANI_PASS_FEATURIZE) != 0,
                                              (cudaStream_t)stream))
            return rc;
    }
    const bool sums_with_grads = (a->phases & ANI_PASS_ENERGY) && (a->phases & ANI_PASS_COORD_GRAD) && n_atoms > 0 &&
                                 grad_per_molecule(n_atoms, a->n_mols, {a->feature_grads});
    if (sums_with_grads && (!a->energy_sorted || !a->gather_idxs || !a->mol_energy)) return ANI_ERR_NULL_POINTER;
    if ((a->phases & ANI_PASS_ENERGY) && a->n_mols > 0 && !sums_with_grads) {
        if (!a->mol_offsets || !a->mol_atom_counts || !a->mol_energy) return ANI_ERR_NULL_POINTER;
        if (n_atoms > 0 && (!a->energy_sorted || !a->gather_idxs)) return ANI_ERR_NULL_POINTER;
        if (int rc = energy_launch<double>(a->energy_sorted, a->gather_idxs, a->mol_offsets, a->mol_atom_counts, a->n_mols,
                                           a->n_atoms, nullptr, 0.0, a->mol_energy, nullptr, nullptr, (cudaStream_t)stream))
            return rc;
    }
    if (a->phases & ANI_PASS_COORD_GRAD) {
        MolEnergySums<double> sums = {};
        if (sums_with_grads) sums = {a->energy_sorted, a->gather_idxs, a->mol_energy};
        if (int rc = featurize_grad_impl<double>(a->xs, a->ys, a->zs, a->atomic_numbers, a->mol_offsets, a->mol_atom_counts,
                                                 a->n_mols, a->scatter_idxs, grad_rows[0], grad_rows[1], grad_rows[2],
                                                 grad_rows[3], a->x_grads, a->y_grads, a->z_grads, acs, stream, sums,
                                                 (a->phases & ANI_PASS_FORWARD) && ((a->phases & ANI_PASS_ENERGY) == 0 || sums_with_grads)))
            return rc;
    }
    return ANI_OK;
}

int ani_request(const ani_request_args* a, void* stream)
{
    if (!a || !a->in_host || !a->in_dev || !a->out_dev || !a->out_host || (!a->pass && !a->pass64)) return ANI_ERR_NULL_POINTER;
    const cudaStream_t st = (cudaStream_t)stream;
    ANI_CUDA(cudaMemcpyAsync(a->in_dev, a->in_host, a->in_bytes, cudaMemcpyHostToDevice, st));
    if (int rc = a->pass64 ? ani_energy_pass_f64(a->pass64, stream) : ani_network_pass_f32(a->pass, stream)) return rc;
    ANI_CUDA(cudaMemcpyAsync(a->out_host, a->out_dev, a->out_bytes, cudaMemcpyDeviceToHost, st));
    ANI_CUDA(cudaStreamSynchronize(st));
    return ANI_OK;
}

int ani_bias_celu_f32(float* z, float* a, const float* const* bias, const int* acs_host, int width, void* stream)
{
    long long n_atoms = 0;
    if (int rc = check_acs(acs_host, &n_atoms)) return rc;
    if (width <= 0 || (width & 3) || n_atoms * width > 0x7fffffffLL) return ANI_ERR_BAD_SIZE;
    if (n_atoms == 0) return ANI_OK;
    if (!z || !bias) return ANI_ERR_NULL_POINTER;
    BiasCeluParams p;
    p.z = z;
    p.a = a;
    p.rows = (int)n_atoms;
    p.width = width;
    int row = 0;
    for (int t = 0; t < kTypes; t++) {
        if (acs_host[t] > 0 && !bias[t]) return ANI_ERR_NULL_POINTER;
        if (!all_aligned16({bias[t]})) return ANI_ERR_MISALIGNED;
        p.bias[t] = bias[t];
        row += acs_host[t];
        p.row_end[t] = row;
    }
    if (!all_aligned16({z, a})) return ANI_ERR_MISALIGNED;
    ANI_CUDA(launch_chain(bias_celu_kernel, (int)((n_atoms * (width / 4) + 255) / 256), 256, 0, (cudaStream_t)stream, 1, p));
    return ANI_OK;
}

// Work on a side stream that a call has not waited for yet: where the call gives up, the caller's stream waits for it all the
// same, so that the caller may take back the buffers in the order of its own stream.
struct SideWork {
    cudaStream_t stream = nullptr;
    cudaEvent_t done = nullptr;
    ~SideWork()
    {
        if (done) cudaStreamWaitEvent(stream, done, 0);
    }
};

static int force_fit_pass(const ani_force_fit_args* f, void* side_stream, void* features_ready, void* stream)
{
    const ani_pass_args* a = &f->pass;
    const int* acs = a->acs_host;
    long long n_atoms = 0;
    if (int rc = check_acs(acs, &n_atoms)) return rc;
    if (n_atoms == 0) return ANI_OK;
    if (!f->fx || !f->fy || !f->fz || !f->vx || !f->vy || !f->vz || !f->feature_rates || !f->r1 || !f->r2 || !f->adot1 ||
        !f->adot2 || !f->adot3 || !f->q1 || !f->q2 || !f->q3 || !f->partial || !f->rmse || !a->feature_grads || !a->features ||
        !a->act1 || !a->act2 || !a->act3 || !a->dact1 || !a->dact2 || !a->dact3 || !a->dz1 || !a->dz2 || !a->dz3)
        return ANI_ERR_NULL_POINTER;
    if (a->activation < 0 || a->activation > 3 || f->part < 0 || f->part > 2) return ANI_ERR_BAD_SIZE;
    for (int t = 0; t < kTypes; t++)
        if (acs[t] > 0 && (!a->packed[t] || !a->w4[t] || !a->dw1[t] || !a->dw2[t] || !a->dw3[t] || !a->dw4[t] || !a->db1[t] ||
                           !a->db2[t] || !a->db3[t]))
            return ANI_ERR_NULL_POINTER;
    if (!all_aligned16({f->feature_rates, f->r1, f->r2, f->adot1, f->adot2, f->adot3, f->q1, f->q2, f->q3}))
        return ANI_ERR_MISALIGNED;
    const bool signs_here = side_stream && a->activation == kActCelu;      // else they are the caller's
    if (signs_here && (!f->z1 || !f->z2 || !f->z3 || !features_ready || !f->z_ready)) return ANI_ERR_NULL_POINTER;
    cudaStream_t st = (cudaStream_t)stream;
    const int n = (int)n_atoms;
    SideWork in_flight;

    // coordinate gradients of the energy: the first-order pass, which also leaves dE/dA_l
    if (f->part != 2) {
        ani_pass_args first = *a;
        first.labels = nullptr;
        const int before = a->phases & (ANI_PASS_PACK | ANI_PASS_FEATURIZE);
        if (signs_here) {
            // beside the networks, on the stream that the caller keeps for it
            first.phases = before;
            if (int rc = ani_network_pass_f32(&first, stream)) return rc;
            const cudaStream_t side = (cudaStream_t)side_stream;
            ANI_CUDA(cudaEventRecord((cudaEvent_t)features_ready, st));
            ANI_CUDA(cudaStreamWaitEvent(side, (cudaEvent_t)features_ready, 0));
            if (int rc = celu_preactivations_launch(a, acs, const_cast<float*>(f->z1), const_cast<float*>(f->z2),
                                                    const_cast<float*>(f->z3), side))
                return rc;
            ANI_CUDA(cudaEventRecord((cudaEvent_t)f->z_ready, side));
            in_flight.stream = st;
            in_flight.done = (cudaEvent_t)f->z_ready;
        }
        first.phases = (signs_here ? 0 : before) | ANI_PASS_FORWARD;
        if (int rc = ani_network_pass_f32(&first, stream)) return rc;
        {
            ani_mlp_backward_args b;
            size_t row = 0;
            for (int t = 0; t < kTypes; t++) {
                b.grad_energy[t] = a->grad_energy_sorted + row;
                b.w1[t] = a->w1[t]; b.w2[t] = a->w2[t]; b.w3[t] = a->w3[t]; b.w4[t] = a->w4[t];
                b.dact1[t] = a->dact1 + row * kMlpH1; b.dact2[t] = a->dact2 + row * kMlpH2; b.dact3[t] = a->dact3 + row * kMlpH3;
                b.dz1[t] = a->dz1 + row * kMlpH1; b.dz2[t] = a->dz2 + row * kMlpH2; b.dz3[t] = a->dz3 + row * kMlpH3;
                b.grad_features[t] = a->feature_grads + row * kTotal;
                b.packed[t] = a->packed[t];
                row += (size_t)acs[t];
            }
            if (int rc = backward_call(&b, acs, a->split_precision, f->r1, f->r2, st)) return rc;
        }
        first.phases = ANI_PASS_COORD_GRAD;
        if (int rc = ani_network_pass_f32(&first, stream)) return rc;
        // the loss, its derivative with respect to those gradients, and the rates of the features along it
        ANI_CUDA(launch_chain(force_residual_kernel, kForceLossBlocks, kForceLossThreads, 0, st, 1, a->x_grads, a->y_grads,
                              a->z_grads, f->fx, f->fy, f->fz, n, f->partial));
        ANI_CUDA(launch_chain(force_loss_kernel, (n + kForceLossThreads - 1) / kForceLossThreads, kForceLossThreads, 0, st, 1,
                              a->x_grads, a->y_grads, a->z_grads, f->fx, f->fy, f->fz, n, f->partial, f->vx, f->vy, f->vz,
                              f->rmse));
    }
    float* rates[kTypes];
    MlpChainParams p = {};
    MlpWgradSets sets = {};
    MlpWgradParams &w1 = sets.set[0], &w2 = sets.set[1];      // F^T Q and U^T P
    size_t row = 0;
    int tiles = 0;
    for (int t = 0; t < kTypes; t++) {
        auto at = [&](float* base, int width) { return base + row * (size_t)width; };
        rates[t] = at(f->feature_rates, kTotal);
        p.count[t] = acs[t];
        p.tile_start[t] = tiles;
        tiles += (acs[t] + kMlpTile - 1) / kMlpTile;
        p.feat[t] = w2.feat[t] = rates[t];
        p.w4[t] = a->w4[t];
        p.packed[t] = (const unsigned char*)a->packed[t];
        w1.act1[t] = p.act1[t] = at(a->act1, kMlpH1);
        w1.act2[t] = p.act2[t] = at(a->act2, kMlpH2);
        p.act3[t] = at(a->act3, kMlpH3);
        if (a->activation == kActCelu && f->z1 && f->z2 && f->z3) {
            p.act1[t] = const_cast<float*>(f->z1) + row * kMlpH1;
            p.act2[t] = const_cast<float*>(f->z2) + row * kMlpH2;
            p.act3[t] = const_cast<float*>(f->z3) + row * kMlpH3;
        }
        p.dact1[t] = at(a->dact1, kMlpH1); p.dact2[t] = at(a->dact2, kMlpH2); p.dact3[t] = at(a->dact3, kMlpH3);
        p.r1[t] = at(f->r1, kMlpH1); p.r2[t] = at(f->r2, kMlpH2);
        p.adot1[t] = at(f->adot1, kMlpH1); p.adot2[t] = at(f->adot2, kMlpH2); p.adot3[t] = at(f->adot3, kMlpH3);
        p.q1[t] = at(f->q1, kMlpH1); p.q2[t] = at(f->q2, kMlpH2); p.q3[t] = at(f->q3, kMlpH3);
        w1.feat[t] = at(a->features, kTotal);
        w1.dz1[t] = p.q1[t]; w1.dz2[t] = p.q2[t]; w1.dz3[t] = p.q3[t];
        w2.act1[t] = p.adot1[t]; w2.act2[t] = p.adot2[t];
        w2.dz1[t] = at(a->dz1, kMlpH1); w2.dz2[t] = at(a->dz2, kMlpH2); w2.dz3[t] = at(a->dz3, kMlpH3);
        w1.act3[t] = w2.act3[t] = p.adot3[t];
        w1.dw1[t] = w2.dw1[t] = a->dw1[t]; w1.dw2[t] = w2.dw2[t] = a->dw2[t]; w1.dw3[t] = w2.dw3[t] = a->dw3[t];
        w1.db1[t] = a->db1[t]; w1.db2[t] = a->db2[t]; w1.db3[t] = a->db3[t];
        w2.db1[t] = w2.db2[t] = w2.db3[t] = nullptr;
        w1.dw4[t] = a->dw4[t];
        w2.dw4[t] = nullptr;
        w1.db4[t] = w2.db4[t] = nullptr;
        w1.grad_energy[t] = w2.grad_energy[t] = nullptr;
        row += (size_t)acs[t];
    }
    p.tile_start[kTypes] = tiles;
    if (f->part != 2)
        if (int rc = ani_featurize_grad_inverse_f32(a->xs, a->ys, a->zs, a->atomic_numbers, a->mol_offsets, a->mol_atom_counts,
                                                    a->n_mols, a->scatter_idxs, f->vx, f->vy, f->vz, rates[0], rates[1],
                                                    rates[2], rates[3], acs, stream))
            return rc;
    in_flight.done = nullptr;      // part 2 waits
    if (f->part == 1) return ANI_OK;
    if (f->z_ready) ANI_CUDA(cudaStreamWaitEvent(st, (cudaEvent_t)f->z_ready, 0));
    if (int rc = mlp_chain_act<kChainTangent>(p, a->activation, a->split_precision != 0, st)) return rc;
    if (a->zero_ptr && a->zero_bytes) ANI_CUDA(cudaMemsetAsync(a->zero_ptr, 0, a->zero_bytes, st));
    return wgrad_call(sets, acs, 2, a->split_precision, st);
}

int ani_force_fit_pass_f32(const ani_force_fit_args* f, void* stream)
{
    return f ? force_fit_pass(f, nullptr, nullptr, stream) : ANI_ERR_NULL_POINTER;
}

int ani_force_fit_pass_beside_f32(const ani_force_fit_args* f, void* side_stream, void* features_ready, void* stream)
{
    return f && side_stream ? force_fit_pass(f, side_stream, features_ready, stream) : ANI_ERR_NULL_POINTER;
}

}  // extern "C"
