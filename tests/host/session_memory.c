/* The library's handling of device memory against a driver that has little of it: session.c and core.c as they are, linked
 * with the few runtime calls below instead of the CUDA runtime.  Prints nothing and returns 0, or the line that failed. */
#include <stdlib.h>
#include <string.h>
#include "internal.h"

static size_t total, used;
static cudaError_t last;
static struct { void* p; size_t bytes; } block[256];

cudaError_t cudaMalloc(void** p, size_t bytes) {
    if (used + bytes > total) return last = cudaErrorMemoryAllocation;
    for (int i = 0; i < 256; i++)
        if (!block[i].p) {
            used += block[i].bytes = bytes;
            *p = block[i].p = malloc(1);
            return cudaSuccess;
        }
    abort();
}
cudaError_t cudaFree(void* p) {
    for (int i = 0; p && i < 256; i++)
        if (block[i].p == p) {
            used -= block[i].bytes;
            free(p);
            block[i].p = NULL;
            return cudaSuccess;
        }
    abort();
}
cudaError_t cudaGetLastError(void) { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { (void)e; return "no memory"; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
static int graphs;
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t g) { (void)g; graphs--; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) { (void)d; (void)s; (void)n; (void)k; (void)st; return cudaSuccess; }

size_t s2p_kv_vec_bytes(const s2p_model* m) { return m->kv8 ? S2P_HEAD_DIM : S2P_HEAD_DIM * 2; }
size_t s2p_kv_plane_bytes(const s2p_model* m) { return (size_t)m->ctx_len * s2p_kv_vec_bytes(m); }
size_t s2p_kvs_plane_bytes(const s2p_model* m) { return m->kv8 ? (size_t)m->ctx_len * 8 : 0; }
void s2p_sampler_init(s2p_sampler* sp, const s2p_sampling_cfg* cfg, uint64_t entropy) { (void)cfg; (void)entropy; memset(sp, 0, sizeof(*sp)); }

static s2p_model* model(int device) {
    s2p_model* m = calloc(1, sizeof(*m));
    m->n_slow = 2; m->ctx_len = 1024; m->kv8 = 1; m->max_sessions = 64; m->device = device;
    return m;
}
static size_t session_bytes(void) { /* of one session of such a model */
    s2p_model* m = model(0);
    s2p_session* s;
    total = (size_t)1 << 40;
    if (s2p_session_create(m, NULL, &s) != S2P_OK) abort();
    const size_t n = used;
    s2p_session_destroy(s);
    s2p_session_pool_clear(m);
    free(m);
    return n;
}
#define CHECK(x) do { if (!(x)) return __LINE__; } while (0)

int main(void) {
    const size_t one = session_bytes();
    CHECK(used == 0);
    s2p_model *a = model(0), *b = model(0), *elsewhere = model(1);
    s2p_session* s[8];
    s2p_tensor t;

    /* a refused session leaves no error behind that a healthy session's next launch would return */
    total = 2 * one;
    CHECK(s2p_session_create(a, NULL, &s[0]) == S2P_OK && s2p_session_create(a, NULL, &s[1]) == S2P_OK);
    CHECK(s2p_session_create(a, NULL, &s[2]) == S2P_ERR_OOM && a->n_sessions == 2);
    CHECK(cudaGetLastError() == cudaSuccess);
    const int64_t too_many[1] = {(int64_t)one};
    CHECK(s2p_tensor_device_alloc(&t, S2P_DT_U8, 1, too_many) == S2P_ERR_OOM && !t.data);
    CHECK(cudaGetLastError() == cudaSuccess);

    /* closed sessions' blocks wait for the next session ... */
    s2p_session_destroy(s[0]);
    s2p_session_destroy(s[1]);
    CHECK(used == 2 * one && a->n_pool == 2);
    CHECK(s2p_session_create(a, NULL, &s[0]) == S2P_OK && used == 2 * one && a->n_pool == 1);
    /* ... unless another buffer, or another model's session, needs the memory; a session's own block stays */
    CHECK(s2p_tensor_device_alloc(&t, S2P_DT_U8, 1, too_many) == S2P_OK && a->n_pool == 0 && used == 2 * one);
    CHECK(cudaGetLastError() == cudaSuccess);
    s2p_tensor_free(&t);
    CHECK(s2p_session_create(a, NULL, &s[1]) == S2P_OK);
    s2p_session_destroy(s[1]);
    CHECK(s2p_session_create(b, NULL, &s[1]) == S2P_OK && a->n_pool == 0 && used == 2 * one);

    /* a pool on another GPU would not help */
    total = 3 * one;
    CHECK(s2p_session_create(elsewhere, NULL, &s[2]) == S2P_OK);
    s2p_session_destroy(s[2]);
    CHECK(s2p_session_create(b, NULL, &s[2]) == S2P_ERR_OOM && elsewhere->n_pool == 1);

    /* freed models leave the list */
    s2p_session_pool_clear(elsewhere);
    free(elsewhere);
    s2p_session_destroy(s[0]);
    s2p_session_pool_clear(a);
    free(a);
    CHECK(used == one);
    total = 2 * one;
    CHECK(s2p_session_create(b, NULL, &s[0]) == S2P_OK && s2p_session_create(b, NULL, &s[2]) == S2P_ERR_OOM);
    s2p_session_destroy(s[0]);
    s2p_session_destroy(s[1]);
    s2p_session_pool_clear(b);

    /* resident copies of the weights give way to sessions: the bf16 ones, then the tiles and the graphs that read them */
    total = 4 * one;
    CHECK(cudaMalloc(&b->wide_weights, one) == cudaSuccess && cudaMalloc(&b->tc_weights, one / 2) == cudaSuccess && cudaMalloc(&b->xt_norm, one / 2) == cudaSuccess);
    b->slow[1].wide[2] = b->wide_weights;
    b->slow[1].tc[2] = b->fast[3].tc[0] = b->tc_fast_out = b->tc_weights;
    b->xt_attn = b->xt_ffn = b->xt_norm;
    b->gready[1] = b->gready[32] = 1;
    graphs = 2;
    CHECK(s2p_session_create(b, NULL, &s[0]) == S2P_OK && s2p_session_create(b, NULL, &s[1]) == S2P_OK && b->wide_weights);
    CHECK(s2p_session_create(b, NULL, &s[2]) == S2P_OK && !b->wide_weights && !b->slow[1].wide[2] && b->tc_weights && graphs == 2);
    CHECK(s2p_session_create(b, NULL, &s[3]) == S2P_OK && !b->tc_weights && !b->xt_norm && !b->xt_ffn && !b->xt_attn && !b->tc_fast_out);
    CHECK(!b->slow[1].tc[2] && !b->fast[3].tc[0] && graphs == 0 && !b->gready[1] && !b->gready[32]);
    CHECK(s2p_session_create(b, NULL, &s[4]) == S2P_ERR_OOM && cudaGetLastError() == cudaSuccess);
    for (int i = 0; i < 4; i++) s2p_session_destroy(s[i]);
    s2p_session_pool_clear(b);
    CHECK(used == 0);
    free(b);
    return 0;
}
