// A stretch of a context's work beside the rest of it (ctx.cu); internal to the library.
#pragma once

struct zkb_ctx;

namespace zk {

// From side_begin to side_end what the host enqueues goes to a second stream of the context, after everything enqueued before; what
// follows side_end runs beside it until side_join. In between only kernels that read and write memory of their own may be
// enqueued on either side of the fork: the scratch buffer belongs to the work outside. A fork at a time.
int side_begin(zkb_ctx* ctx);
int side_end(zkb_ctx* ctx);
int side_join(zkb_ctx* ctx);  // nothing to do: no fork since the last one

// Joins on the way out, whatever the way: memory of the fork may be given back (and used again by later work) from then on.
struct SideScope {
    zkb_ctx* ctx;
    explicit SideScope(zkb_ctx* c) : ctx(c) {}
    ~SideScope() { side_join(ctx); }
};

}  // namespace zk
