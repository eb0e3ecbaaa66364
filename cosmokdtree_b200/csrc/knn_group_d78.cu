// knn_group_d78.cu -- the kNN kernel with a group of lanes per query, d = 7 and 8.
#include "ckd_knn_group.cuh"

namespace ckd {
CKD_KNN_GROUP(7)
CKD_KNN_GROUP(8)
}  // namespace ckd
