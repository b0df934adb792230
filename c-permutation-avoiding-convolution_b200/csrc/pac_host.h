/* pac_host.h -- what the fft.h drop-in (pac_dropin.c) needs from the library
 * beyond pac.h: pinned host memory, events and the current device for its
 * copy threads, the plan's status word with the results.  Not exported. */
#ifndef PAC_HOST_H
#define PAC_HOST_H

#include <stddef.h>

#include "pac.h"

#ifdef __cplusplus
extern "C" {
#endif

int pac_host_alloc(void** p, size_t bytes); /* pinned, for every device */
void pac_host_free(void* p);
int pac_host_device(void);            /* the calling thread's device ... */
void pac_host_set_device(int device); /* ... for a thread it started */
/* 0 ordinary host memory, 1 pinned, 2 not host memory alone (device, managed) */
int pac_host_kind(const void* p);
int pac_host_event_create(void** ev);
void pac_host_event_destroy(void* ev);
int pac_host_event_record(void* ev, pac_stream_t stream);
int pac_host_event_wait(void* ev);
/* queue a copy of the plan's status word to *word (pinned) */
int pac_host_fetch_status(pac_plan_t plan, int* word, pac_stream_t stream);

#ifdef __cplusplus
}
#endif
#endif
