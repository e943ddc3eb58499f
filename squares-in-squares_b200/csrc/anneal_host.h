// Host-side helpers shared by the batch entry point (anneal_host.cu) and the
// serving runtime (serve_host.cu).
#pragma once
#include <string>
#include <vector>

#include "anneal.cuh"
#include "common.cuh"

namespace sqs {
namespace ann {

struct Plan {
    int cs, Rl, Gmax;
    int64_t rb;   // shared-memory bytes of one replica
    float cell;   // minimum cell side
};

// A launch shape chosen by the autotuner (cs = 0: none, use the default plan).
struct Shape {
    int cs = 0;
    float cell = kCellSide;
};

int prime_anneal();
int launch_init(cudaStream_t stream, int njobs, const InitRec* rec, const double* start, float4* pos);
int launch_trace(cudaStream_t stream, int items, const int2* list, const JobDev* jdev, const JobMut* jmut,
                 float4* pos, TraceRec* out, size_t smem);
// FP64 kernels, one CTA a packing, its width by its size.  `n` holds the sizes in
// launch order: as they come up to one packing an SM, else descending, as
// width_order sorts them (it returns the permutation, empty in the first
// case), and `order` is that permutation on the device (null in the first case).
std::vector<int32_t> width_order(sqs_ctx* ctx, std::vector<int32_t>& n);
int launch_energy_states(sqs_ctx* ctx, const std::vector<int32_t>& n, const int32_t* order, const int32_t* n_of,
                         const int64_t* row0, const double* side, const double* xya, double* energy_out, double* grad);

// One launch of the anneal kernel: the jobs job_list[0 .. njobs) sharing a
// cluster shape, with the shared memory of the largest.
struct Group {
    int njobs, cs, Rl;
    size_t smem;
    const int32_t* list;
    bool moves;  // the jobs use move-set options (the kernel instance with them)
};
// Launch every group for one slice.  Several groups run concurrently on the
// context's side streams, forked from and joined back to its main stream
// (under stream capture they become parallel branches of the graph).
int launch_groups(sqs_ctx* ctx, const std::vector<Group>& groups, const JobDev* jdev, JobMut* jmut, float4* pos,
                  double* best, int slice);
int anneal_max_clusters(int cs, int Rl, size_t smem, bool moves, int* out);
// Shared memory to launch with: the replicas, and the quench scratch when it fits
// without lowering the resident clusters.
size_t anneal_smem(int cs, int Rl, int64_t rb, int n_max, bool moves, int need = 1 << 30);
int launch_anneal(cudaStream_t stream, int njobs, int cs, int Rl, size_t smem, bool moves, const int32_t* job_list,
                  const JobDev* jdev, JobMut* jmut, float4* pos, double* best, int slice);
// job_list: the jobs in the order of `n`
int launch_polish(sqs_ctx* ctx, const std::vector<int32_t>& n, const int32_t* job_list, const JobDev* jdev, JobMut* jmut,
                  double* best);
int launch_polish_states(sqs_ctx* ctx, const std::vector<int32_t>& n, const int32_t* order, const int32_t* n_of,
                         const int64_t* row0, int iters, double* xya, double* res);

void put(char* dst, size_t cap, const std::string& s);
// Validate one job and fill its device records (offsets left to the caller).
// `shape` (optional) fixes the cluster size and cell side instead of the
// default (smallest cluster that fits, cells of side kCellSide).
int prepare_job(const sqs_job& J, int j, JobDev& d, JobMut& m, Plan& p, const Shape* shape = nullptr);
// Another launch shape for a prepared job: about `rl` replicas a CTA (at most
// the default plan's; the cell side stays).  True when the plan changed; a
// shape of which the device cannot hold one cluster is not taken.
bool replan(const sqs_job& J, int rl, JobDev& d, Plan& p);
// Resolve SQS_JOB_AUTOTUNE: the tuned shape of the job's class (tuning it on
// first sight) and, when the job leaves exchange_every at 0, the tuned
// interval written into `eff` (a copy of the job).  No flag: eff = job.
int resolve_job(sqs_ctx* ctx, const sqs_job& job, int mode, sqs_job& eff, Shape& shape);
// float4 elements of a job's state region: R*n replica squares and kQuenchScr n scratch a replica.
int64_t job_pos_elems(const sqs_job& J);
// Proposals per replica in a job's budget (sweeps * n, or -sweeps), and that
// budget in whole sweeps, rounded up.
int64_t job_props(const sqs_job& J);
int64_t job_sweeps(const sqs_job& J);
// Every replica starts from the job's initial state (angles wrapped to [0, pi/2)).
void init_replicas(const sqs_job& J, float4* dst);
void fill_result(const sqs_job& J, const JobDev& d, const JobMut& m, float dev_ms, sqs_job_result& o);
// A finished job that certified no state during its anneal would return
// nothing: its coldest replica's final state is polished from scratch
// instead (the sqs_polish_batch path: overlaps resolved in a spread box,
// then the compress-and-descend attempts, `iters` gradient steps), and a
// certified side found that way becomes the job's best (*m, best[3n]).
struct Rescue {
    int n, iters;
    const float4* d_state;  // the replica's final (x, y, angle, -) on the device
    double* best;           // host, n x 3
    JobMut* m;              // host copy of the job's record
};
int rescue_uncertified(sqs_ctx* ctx, const std::vector<Rescue>& items);
// The rescue candidates among finished jobs: annealed (sweeps > 0), best
// side still unset, polish requested.
void add_rescue(std::vector<Rescue>& out, const sqs_job& J, const JobDev& d, JobMut& m, const float4* d_pos,
                double* best);
int certify_states(sqs_ctx* ctx, const std::vector<int>& ns, const std::vector<const double*>& best,
                   const std::vector<sqs_job_result*>& out, const std::vector<double*>& xya_out);

}  // namespace ann
}  // namespace sqs
