// The launches of a host-sized FemPIC step up to its move, in one call (oppb_step_begin).

#include "oppb_common.cuh"
#include "oppb_dh.h"

extern "C" int oppb_step_begin(const oppb_step* st, const oppb_particles* parts, void* stream) {
    using namespace oppb;
    if (!st || !parts || !st->status || !st->status_host || !st->node_charge || st->n_inject < 0 ||
        st->n_inject > parts->size || st->n_nodes < 0)
        return OPPB_ERR_ARG;
    int rc = oppb_inject_f64(st->mesh, st->inlet, parts, parts->size - st->n_inject, st->n_inject, st->rnd,
                             st->rnd_stride, st->rnd_dim, st->ion_velocity, st->move.qm, st->move.dt, stream);
    if (rc) return rc;
    if ((rc = oppb_fill(st->node_charge, st->n_nodes, 8, 0, stream))) return rc;
    if (st->separate_push) {
        rc = st->move.precision == OPPB_PRECISION_MIXED
                 ? oppb_push_mixed(st->mesh, parts, st->move.qm, st->move.dt, stream)
                 : oppb_push_f64(st->mesh, parts, st->move.qm, st->move.dt, stream);
        if (rc) return rc;
    }
    rc = oppb_move_ex(st->mesh, parts, &st->move, st->node_charge, st->status, st->max_hops, st->workspace,
                      st->workspace_bytes, stream);
    if (rc) return rc;
    cudaStream_t s = as_stream(stream);
    if (cudaMemcpyAsync(st->status_host, st->status, sizeof(oppb_move_status), cudaMemcpyDeviceToHost, s) !=
            cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return OPPB_ERR_LAUNCH;
    return OPPB_OK;
}
