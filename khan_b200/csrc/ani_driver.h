// The work on one batch of a fed data set as ONE call: take the batch from the feeder, enqueue sort, features, networks
// and what the pass is for -- energies, gradients to a pinned host ring, or a training update -- and give its slot back.
//
// The reference drives its batches from Python through session.run
// (khan/training/trainer_multi_tower.py:580-678,710-828).  Here a batch of 1024 molecules is 80 to 120 us of GPU
// work, and the Python of a batch (a dozen tensor views, four or five calls, stream and event objects) was 150 to
// 200 us: predict, coordinate_gradients and feed_dataset were bound by it.  A step of this class is 25 to 40 us of
// host time, nearly all of it launches.
//
// Two batches are in flight, each in a set of buffers of its own:
//   * energies: batch b on stream b & 1.  The networks take whole waves of 128-atom tiles (220 tiles on 148
//     SMs for 2048 molecules), and the other batch's kernels fill what the last wave leaves idle.
//   * gradients: the same, but their consumer takes the results batch by batch and may enqueue anything in between, a
//     training step among it.  So every batch has a copy of the weights of its own, made on the caller's stream at the
//     batch's step: one small kernel, beside the batches in flight.  (With the weights themselves the caller's stream
//     would have to wait for every batch and the next networks for that stream: 8 batches of 1024 molecules took 2500 us
//     that way, 2360 with copies, 2290 without either: 9 us a batch, which the host takes for the launch and the events.)
//   * training: sort + featurize of the next batch on a side stream beside this one's networks; each update waits for
//     everything of its own batch.
#pragma once

#include <type_traits>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/ani_b200.h"
#include "ani_feeder.h"
#include "ani_launch.cuh"

namespace ani {

// (n, 3) rows from three arrays, straight into pinned host memory: 170 kB take 4 us that way, under the next
// batch's kernels, and a copy after the kernel would hold those up for 9.
template <typename T>
__global__ void __launch_bounds__(256) interleave3_kernel(const T* __restrict__ x, const T* __restrict__ y,
                                                          const T* __restrict__ z, int n, T* __restrict__ out)
{
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * 256 + threadIdx.x;      // one value of the output per thread: coalesced stores
    if (i >= 3 * n) return;
    const int atom = i / 3, axis = i - 3 * atom;
    out[i] = (axis == 0 ? x : (axis == 1 ? y : z))[atom];
}

// The arrays of the four networks, one after another.
constexpr int kWeightArrays = 8 * kTypes;       // w1, b1, ... w4, b4 of every element
constexpr int weight_array_length(int k)
{
    return k == 0 ? kMlpIn * kMlpH1 : (k == 2 ? kMlpH1 * kMlpH2 : (k == 4 ? kMlpH2 * kMlpH3 : (k == 1 || k == 3 ? kMlpH1 :
           (k == 7 ? 1 : kMlpH3))));
}
constexpr int weight_array_start(int i)         // in values; every array starts on 16 bytes
{
    int at = 0;
    for (int j = 0; j < i; j++) at += (weight_array_length(j % 8) + 3) / 4 * 4;
    return at;
}
template <typename T> struct WeightCopyParams {
    const T* from[kWeightArrays];
    int length[kWeightArrays];       // 0 where there is none
    T* to[kWeightArrays];
};
// kCopyCtas CTAs for each array, and in float behind them one for each packed chunk.
constexpr int kCopyCtas = 6;
template <typename T>
__global__ void __launch_bounds__(kMlpThreads) copy_weights_kernel(const WeightCopyParams<T> p, const MlpPackParams pack)
{
    if ((int)blockIdx.x >= kCopyCtas * kWeightArrays) {
        const int c = (int)blockIdx.x - kCopyCtas * kWeightArrays;
        pack_chunk(pack, c % kPackChunks, c / kPackChunks);
        return;
    }
    const int i = blockIdx.x / kCopyCtas;
    const T* from = p.from[i];
    T* to = p.to[i];
    for (int k = (blockIdx.x % kCopyCtas) * kMlpThreads + threadIdx.x; k < p.length[i]; k += kCopyCtas * kMlpThreads) to[k] = from[k];
}
constexpr size_t weights_bytes(bool f64)        // of a copy; in float with the packed form behind it
{
    const size_t values = (size_t)weight_array_start(kWeightArrays) * (f64 ? 8 : 4);
    return (values + 255) / 256 * 256 + (f64 ? 0 : (size_t)kTypes * kPackChunks * kPackedChunkBytes);
}

class Driver {
  public:
    explicit Driver(const ani_driver_args& a) : a_(a) {}
    ~Driver()
    {
        for (cudaEvent_t e : {side_done_, main_done_, ring_done_[0], ring_done_[1], ring_done_[2]})
            if (e) cudaEventDestroy(e);
    }
    int init()
    {
        slots_.assign(a_.slots, a_.slots + a_.n_slots);
        for (int k = 0; k < 2; k++) streams_[k] = static_cast<cudaStream_t>(a_.streams[k]);
        for (cudaEvent_t* e : {&side_done_, &main_done_, &ring_done_[0], &ring_done_[1], &ring_done_[2]})
            if (cudaEventCreateWithFlags(e, cudaEventDisableTiming) != cudaSuccess) return ANI_ERR_CUDA;
        return ANI_OK;
    }
    // 1: *out describes the batch whose work has been enqueued; 0: the pass is over; negative: an error.
    int step(Feeder& feeder, cudaStream_t main, ani_feeder_batch* out)
    {
        const int rc = a_.mode == ANI_DRIVER_TRAIN ? train_step(feeder, main, out) : evaluate_step(feeder, main, out);
        if (rc == 1) {
            molecules_ += out->n_mols;
            index_++;
        }
        return rc;
    }
    // `main` waits for everything enqueued so far.
    int join(cudaStream_t main)
    {
        for (cudaStream_t s : streams_)
            if (s && (cudaEventRecord(side_done_, s) != cudaSuccess || cudaStreamWaitEvent(main, side_done_, 0) != cudaSuccess))
                return ANI_ERR_CUDA;
        return ANI_OK;
    }
    // Host wait for the results of ring place r.
    int wait(int r)
    {
        if (r < 0 || r >= kRing) return ANI_ERR_BAD_INDEX;
        return cudaEventSynchronize(ring_done_[r]) == cudaSuccess ? ANI_OK : ANI_ERR_CUDA;
    }

  private:
    static constexpr int kRing = ANI_DRIVER_RING;
    // every batch has its own copy of the weights
    bool copies() const { return a_.mode == ANI_DRIVER_GRADIENTS && a_.weights[0]; }

    // Where the energies of this batch go: an array of all molecules, the host ring, or (null) the pass's own array.
    void* energies(size_t size) const
    {
        if (a_.energies) return static_cast<char*>(a_.energies) + (size_t)molecules_ * size;
        return a_.mode == ANI_DRIVER_ENERGIES ? a_.ring_host[index_ % kRing] : nullptr;
    }
    template <typename P> void describe(P& p, const ani_feeder_batch& b)
    {
        const ani_driver_slot& s = slots_[b.slot];
        p.n_atoms = b.n_atoms;
        p.n_mols = b.n_mols;
        p.acs_host = b.acs;
        using Real = std::remove_const_t<std::remove_pointer_t<decltype(p.xs)>>;
        p.xs = static_cast<const Real*>(s.xs);
        p.ys = static_cast<const Real*>(s.ys);
        p.zs = static_cast<const Real*>(s.zs);
        p.atomic_numbers = s.atomic_numbers;
        p.mol_offsets = s.mol_offsets;
        p.mol_atom_counts = s.mol_counts;
    }
    int pass(int which, const ani_feeder_batch& b, int phases, cudaStream_t stream)
    {
        if (a_.pass64[which]) {
            ani_energy_args_f64 p = *a_.pass64[which];
            describe(p, b);
            p.phases = phases & ~(ANI_PASS_PACK | ANI_PASS_TRANSIENT);
            own_weights(p);
            if (void* out = energies(sizeof(double))) p.mol_energy = static_cast<double*>(out);
            return ani_energy_pass_f64(&p, stream);
        }
        ani_pass_args p = *a_.pass[which];
        describe(p, b);
        p.phases = phases;
        own_weights(p);
        if (void* out = energies(sizeof(float))) p.mol_energy = static_cast<float*>(out);
        if (a_.mode == ANI_DRIVER_TRAIN) {
            p.labels = static_cast<const float*>(slots_[b.slot].labels);
            p.grad_scale = 1.0f / (float)(b.n_mols > 0 ? b.n_mols : 1);
            p.feature_grads = nullptr;
        }
        return ani_network_pass_f32(&p, stream);
    }
    int evaluate_step(Feeder& feeder, cudaStream_t main, ani_feeder_batch* out)
    {
        const int which = (int)(index_ & 1), r = (int)(index_ % kRing);
        cudaStream_t stream = streams_[which];
        int rc = ANI_OK;
        const bool forces = a_.mode == ANI_DRIVER_GRADIENTS;
        // without copies nobody else may have a turn during the pass, and the weights are packed once
        if (index_ == 0 && !copies() && (rc = weights(main))) return rc;
        const int more = feeder.next(out);
        if (more <= 0) return more;
        if (copies() && (rc = weights(main))) return rc;
        if ((copies() || index_ < 2) && cudaStreamWaitEvent(stream, main_done_, 0) != cudaSuccess) return ANI_ERR_CUDA;
        if ((rc = feeder.wait(out->slot, stream))) return rc;
        if ((rc = pass(which, *out, ANI_PASS_FEATURIZE | ANI_PASS_FORWARD | ANI_PASS_ENERGY | ANI_PASS_TRANSIENT |
                                        (forces ? ANI_PASS_BACKWARD | ANI_PASS_COORD_GRAD : 0), stream))) {
            feeder.used(out->slot, stream);
            return rc;
        }
        if ((rc = feeder.release(out->slot, stream))) return rc;
        cudaError_t e = cudaSuccess;
        if (forces && out->n_atoms > 0)
            e = a_.pass64[which] ? rows_to_host(*a_.pass64[which], out->n_atoms, static_cast<double*>(a_.ring_host[r]), stream)
                                 : rows_to_host(*a_.pass[which], out->n_atoms, static_cast<float*>(a_.ring_host[r]), stream);
        if (e == cudaSuccess) e = cudaEventRecord(ring_done_[r], stream);
        return e == cudaSuccess ? 1 : ANI_ERR_CUDA;
    }
    // The weights as the work on `main` so far leaves them, in the batch's copy if it has one, packed; what comes after
    // main_done_ may read them.
    int weights(cudaStream_t main)
    {
        if (copies()) {
            // the batch that had this copy before has ended: the caller has read its results
            const cudaError_t e = a_.pass64[0] ? copy_weights<double>(*a_.pass64[0], main) : copy_weights<float>(*a_.pass[0], main);
            if (e != cudaSuccess) return ANI_ERR_CUDA;
        } else if (!a_.pass64[0]) {
            ani_pass_args p = *a_.pass[0];
            const int none[4] = {0, 0, 0, 0};
            p.n_atoms = p.n_mols = 0;
            p.acs_host = none;
            p.phases = ANI_PASS_PACK;
            if (int rc = ani_network_pass_f32(&p, main)) return rc;
        }
        return cudaEventRecord(main_done_, main) == cudaSuccess ? ANI_OK : ANI_ERR_CUDA;
    }
    int train_step(Feeder& feeder, cudaStream_t main, ani_feeder_batch* out)
    {
        int rc = ANI_OK;
        // Everything enqueued on the main stream so far: the last use of the buffers that the next batch gets among it.
        if (cudaEventRecord(main_done_, main) != cudaSuccess) return ANI_ERR_CUDA;
        if (!started_) {
            started_ = true;
            have_ = feeder.next(&now_);
            if (have_ > 0 && (rc = featurize(feeder, now_, 0))) return rc;
        }
        if (have_ <= 0) return have_;        // the pass is over, or failed behind the batch of the step before
        if (cudaStreamWaitEvent(main, side_done_, 0) != cudaSuccess) return ANI_ERR_CUDA;      // this batch's features
        // The next batch's features first, so that they run beside this one's networks; but the GPU does not wait
        // for a batch that is still being packed.
        ani_feeder_batch next;
        const int which = (int)(index_ & 1);
        int more = feeder.next(&next, false);
        if (more > 0 && more != Feeder::kNotYet && (rc = featurize(feeder, next, 1 - which))) return rc;
        if ((rc = update(now_, which, main))) return rc;
        if ((rc = feeder.release(now_.slot, main))) return rc;
        if (more == Feeder::kNotYet) {
            more = feeder.next(&next);
            if (more > 0 && (rc = featurize(feeder, next, 1 - which))) return rc;
        }
        *out = now_;
        now_ = next;
        have_ = more;
        return 1;
    }
    int featurize(Feeder& feeder, const ani_feeder_batch& b, int which)
    {
        cudaStream_t side = streams_[0];
        if (cudaStreamWaitEvent(side, main_done_, 0) != cudaSuccess) return ANI_ERR_CUDA;
        if (int rc = feeder.wait(b.slot, side)) return rc;
        const int rc = pass(which, b, ANI_PASS_FEATURIZE, side);
        const int used = feeder.used(b.slot, side);
        if (rc || used) return rc ? rc : used;
        return cudaEventRecord(side_done_, side) == cudaSuccess ? ANI_OK : ANI_ERR_CUDA;
    }
    int update(const ani_feeder_batch& b, int which, cudaStream_t main)
    {
        if (a_.clip_n_rows > 0)
            if (int rc = ani_clip_rows_f32(a_.params, a_.clip_row_offsets, a_.clip_row_lengths, a_.clip_n_rows,
                                           a_.clip_max_norm, main))
                return rc;
        if (int rc = pass(which, b, ANI_PASS_PACK | ANI_PASS_FORWARD | ANI_PASS_ENERGY | ANI_PASS_BACKWARD |
                                        ANI_PASS_WEIGHT_GRAD, main))
            return rc;
        if (a_.loss_kind)
            if (int rc = ani_scale_by_loss_f32(a_.grads, a_.n_params, a_.pass[which]->l2s, b.n_mols, a_.loss_kind, a_.rmse,
                                               main))
                return rc;
        if (!a_.update) return ANI_OK;
        return ani_nadam_step_f32(a_.params, a_.grads, a_.m, a_.v, a_.ema, a_.n_params, a_.hyper, a_.state, main);
    }
    template <typename T, typename P> cudaError_t copy_weights(const P& p, cudaStream_t stream)
    {
        WeightCopyParams<T> c = {};
        const T* const* arrays[8] = {p.w1, p.b1, p.w2, p.b2, p.w3, p.b3, p.w4, p.b4};
        for (int i = 0; i < kWeightArrays; i++) {
            c.from[i] = arrays[i % 8][i / 8];
            c.length[i] = c.from[i] ? weight_array_length(i % 8) : 0;
            c.to[i] = static_cast<T*>(a_.weights[index_ % kRing]) + weight_array_start(i);
        }
        MlpPackParams pack = {};
        if constexpr (sizeof(T) == 4) {
            P own = p;
            own_weights(own);
            for (int t = 0; t < kTypes; t++) {
                pack.w1[t] = p.w1[t]; pack.w2[t] = p.w2[t]; pack.w3[t] = p.w3[t];
                pack.packed[t] = p.w1[t] && p.w2[t] && p.w3[t] ? static_cast<unsigned char*>(own.packed[t]) : nullptr;
            }
        }
        const int grid = kCopyCtas * kWeightArrays + (sizeof(T) == 4 ? kPackChunks * kTypes : 0);
        copy_weights_kernel<T><<<grid, kMlpThreads, 0, stream>>>(c, pack);
        return cudaGetLastError();
    }
    // Points the pass at the batch's copy of the weights, if it has one.
    template <typename P> void own_weights(P& p)
    {
        if (!copies()) return;
        using Real = std::remove_const_t<std::remove_pointer_t<decltype(p.xs)>>;
        char* copy = static_cast<char*>(a_.weights[index_ % kRing]);
        const Real* values = reinterpret_cast<const Real*>(copy);
        const Real** arrays[8] = {p.w1, p.b1, p.w2, p.b2, p.w3, p.b3, p.w4, p.b4};
        for (int t = 0; t < kTypes; t++)
            for (int k = 0; k < 8; k++)
                if (arrays[k][t]) arrays[k][t] = values + weight_array_start(8 * t + k);
        if constexpr (sizeof(Real) == 4) {
            constexpr size_t kPacked = (size_t)kPackChunks * kPackedChunkBytes;
            char* packed = copy + weights_bytes(false) - kTypes * kPacked;
            for (int t = 0; t < kTypes; t++)
                if (p.packed[t]) p.packed[t] = packed + t * kPacked;
        }
    }
    template <typename P, typename T> cudaError_t rows_to_host(const P& p, int n, T* to, cudaStream_t stream)
    {
        return launch_chain(interleave3_kernel<T>, (3 * n + 255) / 256, 256, 0, stream, 1, p.x_grads, p.y_grads, p.z_grads, n,
                            to);
    }

    ani_driver_args a_;
    std::vector<ani_driver_slot> slots_;
    cudaStream_t streams_[2] = {};
    cudaEvent_t side_done_ = nullptr, main_done_ = nullptr, ring_done_[kRing] = {};
    ani_feeder_batch now_{};
    bool started_ = false;
    int have_ = 0;             // of now_: what feeder.next() said
    long long index_ = 0, molecules_ = 0;
};

}  // namespace ani
