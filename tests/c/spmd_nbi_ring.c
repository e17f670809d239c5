/*
 * Non-blocking fetches that stay outstanding while the program queues more
 * requests than the serving ring has slots, run as 2 PEs by shmemx_b200_run:
 * every fetch still gets its own old value.  First PE 0 alone (one quiet
 * after NOPS fetch-adds); then PE 1 keeps NKEEP fetches of its own
 * outstanding while PE 0 queues NOPS puts.  Exits 0 when every value is right.
 */
#include <sched.h>
#include <stdatomic.h>
#include <stdint.h>
#include <stdio.h>

#include "shmem.h"
#include "shmemx.h"

#define NOPS 10000 /* the ring has 4096 slots */
#define NKEEP 100

static atomic_int turn, wrong;
static int64_t fetched[NOPS], kept[NKEEP];

static void wait_for(int t) {
  while (atomic_load(&turn) < t) sched_yield();
}
static void expect(int64_t got, int64_t want, const char *what, int k) {
  if (got != want && atomic_fetch_add(&wrong, 1) < 5)
    fprintf(stderr, "%s %d: %lld, expected %lld\n", what, k, (long long)got, (long long)want);
}

static void pe_main(void *arg) {
  (void)arg;
  shmem_init();
  const int me = shmem_my_pe();
  int64_t *from = shmem_calloc(NOPS, sizeof(int64_t));
  int64_t *to = shmem_calloc(NOPS, sizeof(int64_t));
  int64_t *many = shmem_calloc(NOPS, sizeof(int64_t));
  for (int k = 0; k < NOPS; k++) many[k] = from[k] = 7 * (int64_t)k + me;
  shmem_barrier_all();
  if (me == 0) {
    /* each fetch meets a counter of its own, so the order does not matter */
    for (int k = 0; k < NOPS; k++) shmem_int64_atomic_fetch_add_nbi(&fetched[k], many + k, 1, 1);
    shmem_quiet();
    for (int k = 0; k < NOPS; k++) expect(fetched[k], 7 * (int64_t)k + 1, "one PE, fetch", k);
    atomic_store(&turn, 1);
    wait_for(2);
    for (int k = 0; k < NOPS; k++) shmem_int64_put_nbi(to + k, from + k, 1, 1);
    shmem_quiet();
    atomic_store(&turn, 3);
  } else if (me == 1) {
    wait_for(1);
    for (int k = 0; k < NKEEP; k++) shmem_int64_atomic_fetch_add_nbi(&kept[k], many + k, 5, 0);
    atomic_store(&turn, 2);
    wait_for(3);
    shmem_quiet();
    for (int k = 0; k < NKEEP; k++) expect(kept[k], 7 * (int64_t)k, "two PEs, fetch", k);
  }
  shmem_barrier_all();
  if (me == 1)
    for (int k = 0; k < NOPS; k++) expect(to[k], 7 * (int64_t)k, "put", k);
  shmem_finalize();
}

int main(void) {
  if (shmemx_b200_run(2, pe_main, NULL) != 0) {
    fprintf(stderr, "shmemx_b200_run: %s\n", shmemx_b200_last_error());
    return 5;
  }
  return atomic_load(&wrong) ? 1 : 0;
}
