// Host-callable launchers of the non-fused kernels.  All take raw device pointers and a
// stream so the translation units that define them do not need the PyTorch headers.
#pragma once
#include <cuda_runtime.h>
#include "tn_types.h"

namespace tn {

// pooling.cu
void launch_pool_fwd(const RowSource& src, const int* inverse, const int* offsets, int B, int S, int pd, int combiner, float* out,
                     int out_ld, cudaStream_t st);
void launch_pool_bwd(float* gU, int gstride, const int* inverse, const int* offsets, int B, int S, int pd, int dim,
                     int combiner, const float* gout, int gout_ld, cudaStream_t st);
void launch_seq_fwd(const RowSource& src, const int* inverse, const int* offsets, int B, int T, int pd, float* out, int* lengths,
                    cudaStream_t st);
void launch_seq_bwd(float* gU, int gstride, const int* inverse, const int* offsets, int B, int T, int pd, int dim,
                    const float* gout, cudaStream_t st);
void launch_expand_bag_labels(const float* y, const int* offsets, int B, int nbags, float* out, int room, cudaStream_t st);
// Up to kPackColumns id columns of a batch -> packed values and offsets (columns `first`, `first` + 1, ... of the result).
constexpr int kPackColumns = 64;
struct PackColumns {
  int n, B, first;
  const void* values[kPackColumns];      // int64 or int32 ids
  const void* offsets[kPackColumns];     // [B + 1] int64 or int32, or null: every example has len[c] ids
  int room[kPackColumns];                // ids the column's buffer can hold
  int len[kPackColumns];
  unsigned char val64[kPackColumns], off64[kPackColumns];
  long long* out_values;
  int* out_offsets;
  long long total_room;                  // entries of out_values
};
void launch_pack_columns(const PackColumns& a, cudaStream_t st);

// table_ops.cu
void launch_table_insert_keys(const TableView& t, const long long* keys, int n, int* out_rows, int* status, cudaStream_t st);
void launch_table_lookup(const TableView& t, const long long* keys, int n, int* out_rows, cudaStream_t st);
void launch_table_decay(const TableView& t, int kind, float rate, int delta_days, cudaStream_t st);
void launch_table_rebuild_index(const TableView& t, int n, int* status, cudaStream_t st);
void launch_table_keep_mask(const TableView& t, int kind, const ExportRule& rule, int n, unsigned char* keep, cudaStream_t st);
void launch_table_export(const TableView& t, int kind, const ExportRule& rule, int r0, int r1, int* counts, int* cursors,
                         unsigned long long* out_keys, float* out_rows, int rf, cudaStream_t st);

// elementwise.cu
constexpr int kMaxPieces = 6;
struct ConcatArgs {
  int B;
  int n_pieces;
  const void* ptr[kMaxPieces];   // piece p: [B, width[p]] with row stride ld[p], fp32 or bf16
  int width[kMaxPieces];
  int ld[kMaxPieces];
  int is_bf16[kMaxPieces];
  void* out;                     // bf16 [B, ld_out]; columns past the pieces are 0, ones_col is 1
  int ld_out;
  int ones_col;                  // -1 for none
};
void launch_fm_fwd(const float* E, int ld, int B, int F, int D, float* out, cudaStream_t st);
void launch_fm_bwd(const float* E, int ld, int B, int F, int D, const float* gout, float* gE, int gld, int accumulate, cudaStream_t st);
void launch_concat_cast(const ConcatArgs& a, cudaStream_t st);
void launch_split_cast(const ConcatArgs& a, cudaStream_t st);
void launch_gemv_fwd(const void* Z, int ld, int B, int K, const float* w, float* y, cudaStream_t st);
void launch_gemv_bwd(const void* Z, int ld, int B, int K, const float* w, const float* dy, void* dZ, float* gw, int relu_cols,
                     cudaStream_t st);
void launch_bce(const float* logit, const float* label, int B, float* pred, float* dlogit, float grad_scale, float* sums,
                int nbins, cudaStream_t st);
void launch_cross_v1_fwd(const float* x0, const float* xl, const float* w, const float* bias, int B, int D, float* y, float* dot,
                         cudaStream_t st);
constexpr int kCrossV1OneTile = 1024;   // wider rows take `row_scratch`: fp32 [B]
void launch_cross_v1_bwd(const float* x0, const float* xl, const float* w, const float* dot, const float* gy, int B, int D,
                         float* gx0, float* gxl, float* gw, float* gb, float* row_scratch, cudaStream_t st);
void launch_relu_mask(const void* g, const void* y, void* out, long long n, cudaStream_t st);
void launch_cross_v2_bwd_elem(const void* g, const void* u, const void* x0, float* gx0, void* du, long long n, int first, cudaStream_t st);
constexpr int kMaxCrossLayers = 8;
struct CrossTerms {              // gradient of each layer's output and its u, last layer first; bf16
  const void* g[kMaxCrossLayers];
  const void* u[kMaxCrossLayers];
  int n;
};
struct CrossNet {                // a DCN-v1 cross network of up to kMaxCrossLayers layers, every vector [D]
  const float* w[kMaxCrossLayers];
  const float* b[kMaxCrossLayers];
  float* gw[kMaxCrossLayers];    // added to by the backward pass
  float* gb[kMaxCrossLayers];
  int layers;
};
constexpr int kCrossNetColumns = 1024;   // widest input
// dots, t_row: [layers][B], each layer's x_l . w_l and (backward, scratch) its gradient . x0
void launch_cross_v1_net_fwd(const CrossNet& n, const float* x0, int B, int D, float* y, float* dots, cudaStream_t st);
void launch_cross_v1_net_bwd(const CrossNet& n, const float* x0, int B, int D, const float* dots, const float* gy, float* gx0, float* t_row,
                             cudaStream_t st);
void launch_cross_v2_du(const void* g, const void* x0, void* du, long long n, cudaStream_t st);
void launch_cross_v2_bwd_sum(const CrossTerms& t, const void* g0, void* out, long long n, cudaStream_t st);
void launch_cross_v2_bwd_final(const float* gx0, const void* g, void* out, long long n, cudaStream_t st);

// head.cu  (return nullptr or a static error string)
constexpr int kMaxHeadPieces = 4;
constexpr int kMaxHeadSpan = 4096;      // weights that fit, every piece's rounded up to eight
constexpr int kHeadCopies = 16;         // partial copies of the weight gradient in the scratch
enum HeadKind { kHeadBf16, kHeadF32, kHeadF32x4 };
struct HeadArgs {
  int B, n, K;                          // rows, pieces, weights without the bias (w[K])
  const void* src[kMaxHeadPieces];      // piece p: [B, width[p]] with row stride ld[p]
  void* grad[kMaxHeadPieces];           // its gradient, row stride gld[p] (bf16: zeros behind width[p]); null: not wanted
  int width[kMaxHeadPieces], ld[kMaxHeadPieces], gld[kMaxHeadPieces], kind[kMaxHeadPieces];
  int relu_first;                       // piece 0 is a ReLU's output: its gradient comes masked
  const float* w;
  const float* label;
  float* gw;                            // added to
  float* sums;                          // [0] += mean loss, [1] += sum(label), [2] += sum(pred), [3] += B, then the histograms
  int nbins;
  float* pred;                          // head_loss: probabilities (may be null); head_score: logits
  float* loss_out;
  float* scratch;                       // 4 + kHeadCopies * (span + 8) floats, zero between calls
  int at[kMaxHeadPieces], first[kMaxHeadPieces], units[kMaxHeadPieces], span, groups, copies;      // filled in by the launch
};
const char* launch_head_loss(HeadArgs a, cudaStream_t st);
const char* launch_head_score(HeadArgs a, cudaStream_t st);

// embed_input.cu  (return nullptr or a static error string)
constexpr int kEmbedInputColumns = 128;
struct EmbedInput {
  const int* inverse;
  const int* offsets;        // as in pool_fwd; null: one id a bag
  int B, S, D, combiner;     // columns of a pooled slot
  const float* dense;        // [B, Dd], row stride ld_dense
  int Dd, ld_dense;
  void* X0;                  // bf16 [B, ld]
  int ld;
  float* E;                  // pooled columns [B, S * D] in fp32, or with the dense features behind them; may be null
  int ldE;                   // S * D or S * D + Dd
  float* fm;                 // [B]; may be null
  float* fsum;               // [B, 4 * ceil(D / 4)], the field sums of the FM term for the backward pass; may be null
  float* Lout;               // [B, S]: column lin_col of the rows; lin_col < 0: not wanted
  int lin_col;
};
struct EmbedGrad {
  const int* inverse;
  const int* offsets;
  int B, S, D, dim, combiner;      // the first `dim` columns of a slot have a gradient
  const void* dX0;                 // bf16 [B, ld]
  int ld;
  const float* E;                  // with gfm: what the forward pass has left
  const float* fsum;
  const float* gfm;                // [B], or null
  const float* gE;                 // gradient of the pooled columns, or null
  int ldE;                         // row stride of E and gE
  const float* dL;                 // [B, S], or null
  int lin_col;
  float* gU;
  int gstride;
};
const char* launch_embed_input_fwd(const RowSource& src, const EmbedInput& a, cudaStream_t st);
const char* launch_embed_input_bwd(const EmbedGrad& a, cudaStream_t st);

// stage.cu
constexpr int kStagePieces = 96;
constexpr int kStageBlockBytes = 8192;
struct StagePieces {
  int n;
  const void* src[kStagePieces];       // page-locked host memory as the device sees it
  void* dst[kStagePieces];
  int bytes[kStagePieces];             // above zero
  int first[kStagePieces];             // filled in by the launch
};
cudaError_t launch_stage_inputs(StagePieces& a, cudaStream_t st);

// unique.cu
void launch_unique_assign(const long long* ids, int n, const float* labels, unsigned long long* dd_keys, int* dd_vals,
                          unsigned scratch_cap, unsigned long long* uniq, int cap, int* inverse, float* show, float* click,
                          int* count, int* status, cudaStream_t st);

// bn.cu
struct BnInput {                 // columns [0, nh) of a bf16 matrix of rows ldh long, then those of an fp32 matrix
  const void* h;
  int ldh, nh;
  const float* x;
  int ldx;
};
void launch_bn_batch_stats(const BnInput& in, int B, int C, const float* center, double* batch, cudaStream_t st);
void launch_bn_table_append(const BnTableView& t, double* batch, bool drop_inc, cudaStream_t st);
void launch_bn_join_fwd(const BnInput& in, int B, int C, const float* mean, const float* var, const float* gamma, const float* beta, float eps,
                        void* z, int ldz, float* mean_out, float* var_out, cudaStream_t st);
// the three above for a batch of up to a few thousand rows, whole rows of z written; `batch` (zeroed) is left so
bool bn_join_train_fits(int B, int C, int ldz);
void launch_bn_join_train(const BnTableView& t, const BnInput& in, int B, const float* gamma, const float* beta, float eps, bool drop_inc,
                          void* z, int ldz, float* mean_out, float* var_out, double* batch, cudaStream_t st);
void launch_bn_join_bwd(const void* dz, int ldz, const BnInput& in, int B, int C, const float* mean, const float* var, const float* gamma,
                        float eps, int mask, void* gh, float* gx, int ldg, float* gg, float* gb, cudaStream_t st);
void launch_bn_table_refresh(const BnTableView& t, cudaStream_t st);
void launch_bn_table_sync(const BnTableView& t, const BnSyncView& s, double* scratch, cudaStream_t st);
void launch_bn_apply_fwd(const float* x, int ldx, int B, int C, const float* mean, const float* var, const float* gamma,
                         const float* beta, float eps, float* y, int ldy, cudaStream_t st);
void launch_bn_apply_bwd(const float* dy, int ldd, const float* x, int ldx, int B, int C, const float* mean, const float* var,
                         const float* gamma, float eps, float* dx, int ldo, float* gg, float* gb, cudaStream_t st);

// serving.cu
void launch_dict_lookup_pool(const TableView& t, const long long* ids, const int* offsets, int B, int S, int combiner, void* out,
                             int ld_out, int ones_col, cudaStream_t st);
// The kernels of InferenceEngine's request path (in launch order); `ids` / `offsets` may be pinned host memory.
constexpr int kServeMaxLayers = 8;
constexpr int kServeSkinnyRows = 2;      // requests of up to this many rows take launch_serve_skinny for their layers
struct ServeCast {
  int n;
  const float* src[kServeMaxLayers];
  void* dst[kServeMaxLayers];
  long long n8[kServeMaxLayers];         // groups of eight elements
};
void launch_serve_cast(const ServeCast& a, cudaStream_t st);
// `read` (may be null): recorded once ids and offsets have been read
void launch_serve_lookup_single(const TableView& t, const long long* ids, int B, int S, void* out, int ld_out, int ones_col, bool behind_cast,
                                cudaEvent_t read, cudaStream_t st);
void launch_serve_lookup_ragged(const TableView& t, const long long* ids, int n, const int* offsets, int B, int S, int combiner, int* rows,
                                int* offsets_dev, void* out, int ld_out, int ones_col, bool behind_cast, cudaEvent_t read, cudaStream_t st);
void launch_serve_skinny(const void* x, int ldx, const void* w, int w_f32, int ldw, int M, int N, int K, int relu, void* y, int ldy, int n_store,
                         cudaStream_t st);
void launch_serve_head(const void* z, int ld, int B, int K, const float* w, float* prob, cudaStream_t st);
void launch_sigmoid(const float* x, float* y, int n, cudaStream_t st);

}  // namespace tn
