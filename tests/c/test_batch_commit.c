/*
 * Batch commits on a stand-in for the CUDA layer.
 *
 * Links the library's C host files (api.c, batch.c, tables.c, numbers.c,
 * tuning.c) against the fakes below: device memory is host memory that is
 * never reused after a free, so a job that points into freed memory is seen
 * when it is launched, and allocations, copies and captures fail on request.
 * No GPU and no CUDA call.  One scenario per run: argv[1]; exit 0 when it holds.
 */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "../../vkhel_gb300/csrc/internal.h"

/* ---- the fake device ---- */
#define MAX_BLOCKS 4096
static struct block {
	char *p;
	size_t bytes;
	int live;
} blocks[MAX_BLOCKS];
static int nblocks;
static size_t used, mem_limit;   /* mem_limit 0: unlimited */
static int fail_captures;        /* the next captures fail */
static int failures;
static int fused_launches, composed_launches;

#define CHECK(cond)                                                        \
	do {                                                                   \
		if (!(cond)) {                                                     \
			fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #cond);     \
			failures++;                                                    \
		}                                                                  \
	} while (0)

static int live(const void *p, size_t bytes) {
	for (int i = 0; i < nblocks; i++)
		if (blocks[i].live && (const char *) p >= blocks[i].p &&
				(const char *) p + bytes <= blocks[i].p + blocks[i].bytes)
			return 1;
	return 0;
}

int vkcu_alloc(void *pool, void *stream, size_t bytes, void **ptr) {
	*ptr = NULL;
	if (nblocks == MAX_BLOCKS || (mem_limit && used + bytes > mem_limit))
		return 2;
	struct block *b = &blocks[nblocks++];
	b->p = aligned_alloc(256, (bytes + 255) & ~(size_t) 255);
	memset(b->p, 0, bytes);
	b->bytes = bytes;
	b->live = 1;
	used += bytes;
	*ptr = b->p;
	return 0;
}

int vkcu_free(void *stream, void *ptr) {
	for (int i = 0; ptr && i < nblocks; i++) {
		if (blocks[i].p == ptr) {
			CHECK(blocks[i].live);
			blocks[i].live = 0;
			used -= blocks[i].bytes;
		}
	}
	return 0;
}

static int copy(void *dst, const void *src, size_t bytes) {
	memcpy(dst, src, bytes);
	return 0;
}
int vkcu_h2d(void *stream, void *dst, const void *src, size_t bytes) { return copy(dst, src, bytes); }
int vkcu_d2h(void *stream, void *dst, const void *src, size_t bytes) { return copy(dst, src, bytes); }
int vkcu_d2d(void *stream, void *dst, const void *src, size_t bytes) { return copy(dst, src, bytes); }
int vkcu_memset0(void *stream, void *ptr, size_t bytes) {
	memset(ptr, 0, bytes);
	return 0;
}

int vkcu_device_count(int *count) {
	*count = 1;
	return 0;
}
int vkcu_set_device(int device) { return 0; }
int vkcu_sm_count(int device, int *sms) {
	*sms = 152;
	return 0;
}
static int handle(void **h) {
	*h = malloc(1);
	return 0;
}
int vkcu_stream_create(void **stream) { return handle(stream); }
int vkcu_stream_destroy(void *stream) {
	free(stream);
	return 0;
}
int vkcu_event_create(void **ev) { return handle(ev); }
int vkcu_event_destroy(void *ev) {
	free(ev);
	return 0;
}
int vkcu_pool_create(int device, void **pool) { return handle(pool); }
int vkcu_pool_destroy(void *pool) {
	free(pool);
	return 0;
}
int vkcu_event_record(void *ev, void *stream) { return 0; }
int vkcu_stream_wait(void *stream, void *ev) { return 0; }
int vkcu_sync(void *stream) { return 0; }
int vkcu_host_alloc(void **ptr, size_t bytes) {
	*ptr = malloc(bytes);
	return 0;
}
int vkcu_host_free(void *ptr) {
	free(ptr);
	return 0;
}
const char *vkcu_error_string(int code) { return "fake"; }
static uint64_t launches;
uint64_t vkcu_launch_count(void) { return launches; }
void vkcu_count_launches(uint64_t n) { launches += n; }
void vkcu_range_push(const char *name) {}
void vkcu_range_pop(void) {}
int vkcu_capture_begin(void *stream) { return fail_captures > 0 ? (fail_captures--, 1) : 0; }
int vkcu_capture_end(void *stream, void **exec) { return handle(exec); }
int vkcu_graph_launch(void *exec, void *stream) { return 0; }
int vkcu_graph_destroy(void *exec) {
	free(exec);
	return 0;
}

#define ELEMENTWISE(name, ...) \
	int name(void *stream, uint64_t *res, const uint64_t *a, __VA_ARGS__) { return 0; }
ELEMENTWISE(vkcu_elemmul, const uint64_t *b, uint64_t len, uint64_t mod, uint64_t mu, uint32_t bits)
ELEMENTWISE(vkcu_elemmulconst, uint64_t len, uint64_t c, uint64_t cs, uint64_t mod)
ELEMENTWISE(vkcu_elemfma, const uint64_t *b, uint64_t len, uint64_t m, uint64_t ms, uint64_t mod)
ELEMENTWISE(vkcu_elemfma_canonical, const uint64_t *b, uint64_t len, uint64_t m, uint64_t ms, uint64_t mod, uint64_t mu,
		uint32_t bits)
ELEMENTWISE(vkcu_elemgtsub, uint64_t len, uint64_t bound, uint64_t d, uint64_t mod, uint64_t mu, uint32_t bits)
ELEMENTWISE(vkcu_elemgtadd, uint64_t len, uint64_t bound, uint64_t diff)
ELEMENTWISE(vkcu_elemmodbytwo, uint64_t len, uint64_t bound)
int vkcu_lift_range(void *stream, uint64_t *p, uint64_t len, uint64_t q, int sms, const vkcu_lift *lift) { return 0; }
int vkcu_twiddles(void *stream, uint64_t *fwd, uint64_t *inv, const uint64_t *phi, const uint64_t *plo, uint32_t log_n,
		uint32_t lb, uint64_t q, uint64_t mu, uint32_t qbits) {
	return 0;
}
int vkcu_measure_int_peak(void *stream, int sms, double *b, double *i) { return 1; }
int vkcu_ntt_forward(void *stream, const vkcu_ntt_job *jobs, int njobs, const vkcu_ntt_job *one, uint32_t log_n,
		int qclass, int sms, int avail) {
	return 0;
}
int vkcu_ntt_inverse_lift(void *stream, const vkcu_ntt_job *jobs, int njobs, const vkcu_ntt_job *one, uint32_t log_n,
		int qclass, int sms, int avail, const vkcu_lift *lift) {
	return 0;
}
int vkcu_polymul_ragged(void *stream, const vkcu_ragged_item *items, int n_cluster_items, int n_items,
		const vkcu_poly_job *jobs, unsigned *counters, int qclass) {
	return 0;
}
uint32_t vkcu_max_fused_log_n(void) { return 17; }
uint32_t vkcu_max_log_n(void) { return 26; }
int vkcu_few_composed(long njobs, uint32_t log_n, int qclass, int avail) {
	return qclass != VKCU_Q63 && log_n == 17 && njobs * 16 <= avail;
}

/* every pointer of a launched product lies in memory that is allocated now */
static void check_jobs(const vkcu_poly_job *jobs, int njobs, uint32_t log_n) {
	const size_t bytes = sizeof(uint64_t) << log_n;
	CHECK(live(jobs, sizeof(*jobs) * (size_t) njobs));
	for (int i = 0; i < njobs; i++) {
		CHECK(live(jobs[i].a, bytes));
		CHECK(live(jobs[i].b, bytes));
		CHECK(live(jobs[i].c, bytes));
		CHECK(live(jobs[i].scratch, bytes));
	}
}

int vkcu_polymul_lift(void *stream, const vkcu_poly_job *jobs, int njobs, const vkcu_poly_job *one, uint32_t log_n,
		int qclass, int sms, int avail, const vkcu_lift *lift, int b_ntt) {
	if (jobs)
		check_jobs(jobs, njobs, log_n);
	fused_launches++;
	return 0;
}

int vkcu_polymul_composed(void *stream, const vkcu_poly_job *jobs, const vkcu_ntt_job *b, const vkcu_ntt_job *a,
		const vkcu_ntt_job *c, int njobs, const vkcu_poly_job *one, uint32_t log_n, int qclass, int sms,
		const vkcu_lift *lift, int b_ntt) {
	if (jobs) {
		check_jobs(jobs, njobs, log_n);
		for (int i = 0; i < njobs; i++) /* NTT(b) must not be overwritten by a's transform */
			CHECK(jobs[i].scratch != jobs[i].c);
	}
	composed_launches++;
	return 0;
}

/* ---- scenarios: products of 2^17 words, the prime and its root in argv[2] and argv[3] ---- */
#define LOG_N 17
#define N ((uint64_t) 1 << LOG_N)

static struct vkhel_ctx *ctx;
static struct vkhel_ntt_tables *tab;
static struct vkhel_vector *a, *b, *c;
static struct vkhel_batch *bt;

static void setup(uint64_t q, uint64_t w) {
	ctx = vkhel_ctx_create();
	tab = vkhel_ntt_tables_create(N, q, w);
	a = vkhel_vector_create2(ctx, N, true);
	b = vkhel_vector_create2(ctx, N, true);
	c = vkhel_vector_create2(ctx, N, true);
	bt = vkhel_batch_create(ctx);
	CHECK(ctx && tab && a && b && c && bt);
	struct vkhel_ntt_tables *const tabs[1] = {tab};
	CHECK(vkhel_batch_add_polymul(bt, tabs, 1, a, b, c) == VKHEL_OK);
}

/* A commit that fails after it took the passes' scratch, and one that cannot
 * have it: the fused kernel parks NTT(b) in c, not in what was given back. */
static void retry_without_scratch(void) {
	fail_captures = 1;
	CHECK(vkhel_batch_commit(bt, VKHEL_BATCH_GRAPH) != VKHEL_OK);
	mem_limit = used - N * sizeof(uint64_t) + 4096; /* room for the job table alone */
	CHECK(vkhel_batch_commit(bt, VKHEL_BATCH_GRAPH) == VKHEL_OK);
	CHECK(fused_launches == 1 && composed_launches == 0);
}

/* The same where the retry's tuning keeps the fused kernel. */
static void retry_with_other_tuning(void) {
	fail_captures = 1;
	CHECK(vkhel_batch_commit(bt, VKHEL_BATCH_GRAPH) != VKHEL_OK);
	CHECK(vkhel_tune_set(3, 2, 1) == VKHEL_OK);
	CHECK(vkhel_batch_commit(bt, VKHEL_BATCH_GRAPH) == VKHEL_OK);
	CHECK(fused_launches == 1 && composed_launches == 0);
}

/* Room for the passes' scratch or the job table, not both: the batch runs fused. */
static void no_room_beside_the_table(void) {
	mem_limit = used + N * sizeof(uint64_t) + 64;
	CHECK(vkhel_batch_commit(bt, VKHEL_BATCH_GRAPH) == VKHEL_OK);
	CHECK(fused_launches == 1 && composed_launches == 0);
}

/* What a budget leaves beside the job table stays free for later vectors. */
static void budget_for_a_later_vector(void) {
	const uint64_t before = vkhel_ctx_bytes_in_use(ctx);
	CHECK(vkhel_ctx_set_budget(ctx, before + N * sizeof(uint64_t) + 4096) == VKHEL_OK);
	CHECK(vkhel_batch_commit(bt, VKHEL_BATCH_GRAPH) == VKHEL_OK);
	struct vkhel_vector *v = vkhel_vector_create2(ctx, N, true);
	CHECK(v != NULL);
	vkhel_vector_destroy(v);
	CHECK(fused_launches == 1 && composed_launches == 0);
}

static void composed_where_there_is_room(void) {
	CHECK(vkhel_batch_commit(bt, VKHEL_BATCH_GRAPH) == VKHEL_OK);
	CHECK(fused_launches == 0 && composed_launches == 1);
}

int main(int argc, char **argv) {
	static const struct {
		const char *name;
		void (*run)(void);
	} scenarios[] = {
		{"retry_without_scratch", retry_without_scratch},
		{"retry_with_other_tuning", retry_with_other_tuning},
		{"no_room_beside_the_table", no_room_beside_the_table},
		{"budget_for_a_later_vector", budget_for_a_later_vector},
		{"composed_where_there_is_room", composed_where_there_is_room},
	};
	if (argc != 4)
		return 2;
	for (size_t i = 0; i < sizeof scenarios / sizeof scenarios[0]; i++) {
		if (strcmp(argv[1], scenarios[i].name))
			continue;
		setup(strtoull(argv[2], NULL, 10), strtoull(argv[3], NULL, 10));
		scenarios[i].run();
		mem_limit = 0;
		vkhel_batch_destroy(bt);
		vkhel_vector_destroy(a);
		vkhel_vector_destroy(b);
		vkhel_vector_destroy(c);
		vkhel_ntt_tables_destroy(tab);
		vkhel_ctx_destroy(ctx);
		CHECK(used == 0);
		return failures ? 1 : 0;
	}
	return 2;
}
