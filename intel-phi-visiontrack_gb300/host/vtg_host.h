/* vtg_host.h -- what the served loop (server.c, serve.c) and the tracker code (api.cu) share beside the public headers. */
#ifndef VTG_HOST_H
#define VTG_HOST_H

#include "vtg_serve.h"

#ifdef __cplusplus
extern "C" {
#endif

/* vtg_tracker_create, and with `compact` a tracker whose rows lie as far apart as each level's width asks, so that it holds what it
 * is charged, in whatever context. */
int vtg_tracker_create_as(vtg_ctx *ctx, const struct vtg_config *cfg, int compact, vtg_tracker **out);
/* Device bytes such a tracker may hold without `compact`. */
size_t vtg_tracker_held(const struct vtg_config *cfg);
/* The streams that the server opens from now on get compact trackers. */
void vtg_server_compact(vtg_server *s);

#ifdef __cplusplus
}
#endif

#endif
