/* The host side of the layer (picoforge_b200/csrc/moe_host.c) on a stand-in for the CUDA shim, so that what it does with host
 * memory, threads and copies can be looked at without a GPU (tests/test_host_rows.py drives it).
 *
 * The stand-in's stream is a queue: copies, events and layer launches are carried out, one at a time and in order, only when
 * somebody asks about an event or waits for the stream.  A slot of the ring that is filled or emptied too early therefore shows up as
 * wrong rows.  The "layer" writes y = 2 x + 1, ids and weights that name their token. */
#include "../picoforge_b200/csrc/moe_host.c"

#include <dirent.h>
#include <signal.h>
#include <sys/syscall.h>

static size_t host_bytes_live, host_bytes_peak;
enum { OP_COPY, OP_EVENT, OP_LAYER };
typedef struct { int kind; void *dst; const void *src; size_t dst_pitch, src_pitch, width, rows; int *event; QW4ShWork work; size_t tokens; float *y; } Op;
static Op queue[1 << 16];
static size_t q_head, q_tail;
static unsigned max_threads, unblocked_threads;
static size_t top_k, hidden;

static void look_at_threads(void) {                     /* the helpers' signal masks, while they live */
    DIR *dir = opendir("/proc/self/task");
    unsigned n = 0, open_masks = 0;
    for (struct dirent *e; dir && (e = readdir(dir));) {
        const long tid = atol(e->d_name);
        if (!tid) continue;
        n++;
        if (tid == (long)getpid()) continue;
        char path[64], line[256];
        snprintf(path, sizeof path, "/proc/self/task/%ld/status", tid);
        FILE *f = fopen(path, "r");
        unsigned long long mask = 0;
        bool seen = false;
        while (f && fgets(line, sizeof line, f)) if (sscanf(line, "SigBlk: %llx", &mask) == 1) seen = true;
        if (f) fclose(f);
        if (seen && !(mask & 1ull << (SIGUSR1 - 1) && mask & 1ull << (SIGINT - 1) && mask & 1ull << (SIGTERM - 1))) open_masks++;
    }
    if (dir) closedir(dir);
    if (n > max_threads) max_threads = n;
    if (open_masks > unblocked_threads) unblocked_threads = open_masks;
}
static void run_one(void) {
    Op *o = &queue[q_head++ % (sizeof queue / sizeof *queue)];
    if (o->kind == OP_COPY)
        for (size_t r = 0; r < o->rows; r++) memcpy((char *)o->dst + r * o->dst_pitch, (const char *)o->src + r * o->src_pitch, o->width);
    else if (o->kind == OP_EVENT) --*o->event;
    else
        for (size_t t = 0; t < o->tokens; t++) {
            for (size_t c = 0; c < hidden; c++) o->y[t * hidden + c] = 2.0f * o->work.x[t * hidden + c] + 1.0f;
            for (size_t s = 0; s < top_k; s++) { o->work.ids[t * top_k + s] = (uint32_t)(t * 16 + s); o->work.weights[t * top_k + s] = (float)t + 0.25f * (float)s; }
        }
}
static void enqueue(Op o) {
    if (q_tail - q_head == sizeof queue / sizeof *queue) run_one();
    queue[q_tail++ % (sizeof queue / sizeof *queue)] = o;
}
int qw4sh_device_count(void) { return 1; }
int qw4sh_current_device(void) { return 0; }
const char *qw4sh_last_error(void) { return "stand-in"; }
void *qw4sh_malloc(size_t bytes) { return malloc(bytes); }
void qw4sh_free(void *p) { free(p); }
void *qw4sh_host_alloc(size_t bytes) {
    size_t *p = malloc(bytes + 64);
    p[0] = bytes;
    host_bytes_live += bytes;
    if (host_bytes_live > host_bytes_peak) host_bytes_peak = host_bytes_live;
    return p + 8;
}
void qw4sh_host_free(void *p) { if (p) { size_t *q = (size_t *)p - 8; host_bytes_live -= q[0]; free(q); } }
int qw4sh_memcpy(void *dst, const void *src, size_t bytes, int to_device) { (void)to_device; memcpy(dst, src, bytes); return 0; }
int qw4sh_memcpy2d_async(void *dst, size_t dst_pitch, const void *src, size_t src_pitch, size_t width, size_t rows, int to_device, void *stream) {
    (void)stream;
    if (to_device == 1) look_at_threads();
    enqueue((Op){.kind = OP_COPY, .dst = dst, .src = src, .dst_pitch = dst_pitch, .src_pitch = src_pitch, .width = width, .rows = rows});
    return 0;
}
int qw4sh_memset_async(void *dst, int value, size_t bytes, void *stream) { (void)stream; memset(dst, value, bytes); return 0; }
int qw4sh_shared_stream(void **stream) { static int s; *stream = &s; return 0; }
int qw4sh_current_stream(void **stream) { return qw4sh_shared_stream(stream); }
void *qw4sh_graph_cache_create(void) { return malloc(1); }
void qw4sh_graph_cache_destroy(void *cache) { free(cache); }
int qw4sh_prepare_mma(void) { return 0; }
int qw4sh_stream_sync(void *stream) { (void)stream; while (q_head < q_tail) run_one(); return 0; }
int qw4sh_stream_query(void *stream) { (void)stream; if (q_head < q_tail) run_one(); return q_head < q_tail; }
int qw4sh_event_create(void **event) { *event = calloc(1, sizeof(int)); return 0; }
void qw4sh_event_destroy(void *event) { free(event); }
int qw4sh_event_record(void *event, void *stream) { (void)stream; ++*(int *)event; enqueue((Op){.kind = OP_EVENT, .event = event}); return 0; }
int qw4sh_event_query(void *event) { if (q_head < q_tail) run_one(); return *(int *)event != 0; }
int qw4sh_upload_tensor(const void *host, size_t bytes, uint32_t type, size_t k_storage, size_t n_out, size_t n_experts, void **device) {
    (void)host; (void)bytes; (void)type; (void)k_storage; (void)n_out; (void)n_experts;
    *device = malloc(16);
    return 0;
}
int qw4sh_tile_prepare(QW4ShLayer *layer) { (void)layer; return 0; }
void qw4sh_tile_release(QW4ShLayer *layer) { (void)layer; }
int qw4sh_fused_prepare(QW4ShLayer *layer) { (void)layer; return 0; }
void qw4sh_fused_release(QW4ShLayer *layer) { (void)layer; }
void qw4sh_fused_scratch_sizes(const QW4ShLayer *layer, size_t *a, size_t *b, size_t *c) { (void)layer; *a = *b = *c = 64; }
int qw4sh_takes_fused(const QW4ShLayer *l, const QW4ShWork *w, const float *x, const float *y, size_t t) { (void)l; (void)w; (void)x; (void)y; (void)t; return 0; }
int qw4sh_layer_forward(const QW4ShLayer *layer, const QW4ShWork *work, const float *x, float *y, size_t tokens, uint32_t *ids, float *weights, int mode) {
    (void)layer; (void)x; (void)ids; (void)weights; (void)mode;
    enqueue((Op){.kind = OP_LAYER, .work = *work, .tokens = tokens, .y = y});
    return 0;
}

/* A handle of `experts` experts with F32 tensors of h columns, i intermediate, whose bytes nobody reads. */
static Qwen4Moe *make_moe(size_t h, size_t experts, size_t k, size_t i) {
    static float bytes[16];
    const size_t shape[8][3] = {{h, experts, 1}, {h, i, experts}, {h, i, experts}, {i, h, experts}, {h, i, 1}, {h, i, 1}, {i, h, 1}, {h, 1, 1}};
    QW4PackedCpuView v[8];
    for (int a = 0; a < 8; a++) {
        const size_t row = shape[a][0] * 4, expert = row * shape[a][1], tensor = expert * shape[a][2];
        v[a] = (QW4PackedCpuView){{(const unsigned char *)bytes, tensor}, {0, shape[a][0], shape[a][0], shape[a][1], shape[a][2], row, expert, tensor}};
    }
    const Qwen4MoeConfig c = {(uint32_t)h, (uint32_t)experts, (uint32_t)k, (uint32_t)i, (uint32_t)i, (uint32_t)i, true, {0, 0, 0}};
    const Qwen4MoeWeights w = {v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]};
    Qwen4Moe *m = NULL;
    Qwen4Error err;
    if (qwen4_moe_create(&c, &w, &m, &err)) { fprintf(stderr, "create: %s\n", err.detail); exit(2); }
    hidden = h; top_k = k;
    return m;
}
static Qwen4F32 view(const float *p, size_t rows, size_t cols, size_t pitch) {
    Qwen4F32 v;
    memset(&v, 0, sizeof v);
    v.data = p; v.capacity_bytes = rows * pitch * 4; v.rank = 2;
    v.dim[0] = rows; v.dim[1] = cols; v.stride_bytes[0] = pitch * 4; v.stride_bytes[1] = 4;
    return v;
}
static Qwen4F32Mut view_mut(float *p, size_t rows, size_t cols, size_t pitch) {
    const Qwen4F32 v = view(p, rows, cols, pitch);
    Qwen4F32Mut m;
    memcpy(&m, &v, sizeof m);
    return m;
}

/* budget CAP HIDDEN: the bytes asked for, the bytes held at the most, the status with one byte less. */
static int budget(size_t cap, size_t h) {
    Qwen4Moe *m = make_moe(h, 16, 4, 1);
    size_t asked = 0;
    Qwen4MoeWork *work = NULL;
    Qwen4Error err;
    if (qwen4_moe_work_size(m, cap, &asked, &err)) return 3;
    const int refused = qwen4_moe_work_create(m, cap, asked - 1, &work, &err);
    if (qwen4_moe_work_create(m, cap, asked, &work, &err)) return 4;
    printf("%zu %zu %d\n", asked, host_bytes_peak + sizeof(Qwen4MoeWork), refused);
    qwen4_moe_work_destroy(work);
    qwen4_moe_destroy(m);
    return host_bytes_live ? 5 : 0;
}
/* rows TOKENS HIDDEN XPAD YPAD CALLS: wrong values, threads seen, threads with open signal masks, whether the caller's mask changed. */
static int rows(size_t t, size_t h, size_t xpad, size_t ypad, int calls) {
    Qwen4Moe *m = make_moe(h, 16, 4, 1);
    size_t asked = 0, wrong = 0;
    Qwen4MoeWork *work = NULL;
    Qwen4Error err;
    if (qwen4_moe_work_size(m, t, &asked, &err) || qwen4_moe_work_create(m, t, asked, &work, &err)) return 3;
    const size_t xp = h + xpad, yp = h + ypad;
    float *x = malloc(t * xp * 4), *y = malloc(t * yp * 4), *w = malloc(t * 4 * 4);
    uint32_t *ids = malloc(t * 4 * 4);
    sigset_t before, after;
    pthread_sigmask(SIG_BLOCK, NULL, &before);
    for (int call = 0; call < calls; call++) {
        for (size_t i = 0; i < t * xp; i++) x[i] = (float)((i * 2654435761u + (size_t)call * 977u) % 1000003u) - 500000.0f;
        for (size_t i = 0; i < t * yp; i++) y[i] = -7.0f;
        Qwen4MoeRoutes routes;
        memset(&routes, 0, sizeof routes);
        routes.ids.data = ids; routes.ids.capacity_bytes = t * 16; routes.ids.rows = t; routes.ids.cols = 4; routes.ids.row_stride_bytes = 16;
        routes.weights = view_mut(w, t, 4, 4);
        if (qwen4_moe_forward(m, view(x, t, h, xp), view_mut(y, t, h, yp), &routes, work, &err)) { fprintf(stderr, "forward: %s\n", err.detail); return 4; }
        for (size_t r = 0; r < t; r++) {
            for (size_t c = 0; c < yp; c++) wrong += y[r * yp + c] != (c < h ? 2.0f * x[r * xp + c] + 1.0f : -7.0f);
            const size_t row = r % 4096;                 /* launch sequences of 4096 tokens */
            for (size_t s = 0; s < 4; s++) wrong += ids[r * 4 + s] != row * 16 + s || w[r * 4 + s] != (float)row + 0.25f * (float)s;
        }
    }
    pthread_sigmask(SIG_BLOCK, NULL, &after);
    int changed = 0;
    for (int s = 1; s < 32; s++) changed |= sigismember(&before, s) != sigismember(&after, s);
    printf("%zu %u %u %d\n", wrong, max_threads, unblocked_threads, changed);
    qwen4_moe_work_destroy(work);
    qwen4_moe_destroy(m);
    free(x); free(y); free(w); free(ids);
    return host_bytes_live ? 5 : 0;
}
/* device CAP HIDDEN EXPERTS TOPK INTER: bytes of the workspace's device block. */
static int device(size_t cap, size_t h, size_t e, size_t k, size_t i) {
    Qwen4Moe *m = make_moe(h, e, k, i);
    size_t chunk;
    Plan plan;
    Qwen4Error err;
    if (plan_work(m, cap, &chunk, &plan, &err)) return 3;
    printf("%zu\n", plan.total);
    qwen4_moe_destroy(m);
    return 0;
}
int main(int argc, char **argv) {
    if (argc == 4 && !strcmp(argv[1], "budget")) return budget(strtoul(argv[2], NULL, 10), strtoul(argv[3], NULL, 10));
    if (argc == 7 && !strcmp(argv[1], "rows"))
        return rows(strtoul(argv[2], NULL, 10), strtoul(argv[3], NULL, 10), strtoul(argv[4], NULL, 10), strtoul(argv[5], NULL, 10), atoi(argv[6]));
    if (argc == 7 && !strcmp(argv[1], "device"))
        return device(strtoul(argv[2], NULL, 10), strtoul(argv[3], NULL, 10), strtoul(argv[4], NULL, 10), strtoul(argv[5], NULL, 10), strtoul(argv[6], NULL, 10));
    return 1;
}
