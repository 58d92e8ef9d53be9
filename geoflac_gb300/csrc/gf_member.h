// Library-internal view of a context, for the ensemble driver (gf_batch.cu).
#pragma once

#include <memory>

#include "gf_ctx.h"

struct GfMemberView {
    const DevParams *P;
    DevClock *C;
    DevArrays A;
    GfDims d;
    int mode, idt_scale, movegrid, itherm, nmarkers;
    int nloop, nsrate;
    int ifreq_rmasses, ifreq_visc, ifreq_imasses, ifreq_avgsr;
    double z0, rzbo, g;
    cudaStream_t s;
    const gf_params *hp; // host parameters of the context
    gf_layout *L;        // host arrays registered with the context
};

// Order between a batch's stream and the members' streams.
struct GfEvent {
    cudaEvent_t e = nullptr;
    ~GfEvent() {
        if (e) cudaEventDestroy(e);
    }
};

extern "C" {
int gf_ctx_view(gf_ctx *c, GfMemberView *v);
unsigned gf_ctx_signature(const gf_ctx *c);
void gf_ctx_advance(gf_ctx *c, unsigned sig); // host bookkeeping after one step
int gf_ctx_take_status(gf_ctx *c);
// the member's stresses or mesh were changed outside its own calls
void gf_ctx_invalidate_forces(gf_ctx *c);
// the device-side part of rsflac.f90:197-236 once the restart files are
// uploaded and marker2elem has run: init_areas, temp0 = temp, heating and
// strain-rate accumulators reset, rmasses, init_visc, dt_mass, dtavg /
// nsrate reset
int gf_ctx_restart_finish(gf_ctx *c);
// what the member's own calls enqueued and did not wait for has run; stream s
// waits for other batches that still read the member (own: not this one's event)
int gf_ctx_settle(gf_ctx *c, cudaStream_t s, const GfEvent *own);
// the member's state is read on another stream until the event: the next call
// that changes the state waits for it (on the device)
int gf_ctx_read_until(gf_ctx *c, const std::shared_ptr<GfEvent> &until);
}
